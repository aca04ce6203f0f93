"""The bf16 causal backward at every geometry race_b200_causal_bwd_heads grants (S = 64, 128, 256, 512; d_k = 64, 128)."""
from __future__ import annotations

import pytest
import torch

from oracle import race_oracle as ro

pytestmark = pytest.mark.gpu

GEOMETRIES = [(L, R, dk) for L, R in ((4, 16), (2, 64), (4, 64), (8, 64)) for dk in (64, 128)]


def _inputs(N, T, L, R, dk, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    pq, pk = (torch.softmax(torch.randn(N, T, L, R, device="cuda", generator=g), -1).bfloat16() for _ in range(2))
    v, dO = (torch.randn(N, T, dk, device="cuda", generator=g).bfloat16() for _ in range(2))
    return pq, pk, v, dO


@pytest.mark.parametrize("L,R,dk", GEOMETRIES)
@pytest.mark.parametrize("B,H,T", [(1, 2, 300), (2, 3, 129)])
def test_operator_layout_has_the_bits_of_the_flat_one(L, R, dk, B, H, T):
    import race_attention_kernel_b200.ops as ops
    N = B * H
    pq, pk, v, dO = _inputs(N, T, L, R, dk, seed=T + dk)
    assert ops.causal_bwd_takes_heads(N, T, L, R, dk, torch.bfloat16, H)

    def operator_layout(x):
        return x.view(1, B, H, T, dk).permute(0, 1, 3, 2, 4).contiguous()

    flat = ops.race_causal_backward(pq, pk, v, dO)
    heads = ops.race_causal_backward(pq, pk, operator_layout(v), operator_layout(dO))
    assert torch.equal(heads[0], flat[0]) and torch.equal(heads[1], flat[1])
    assert torch.equal(heads[2], operator_layout(flat[2]))


@pytest.mark.parametrize("L,R,dk", [(4, 16, 64), (4, 16, 128), (2, 64, 64), (8, 64, 128)])
def test_outputs_that_begin_between_two_sectors(L, R, dk):
    """The ABI promises to take any 16-byte boundary; outputs carved out of one buffer often begin on an odd one."""
    import ctypes

    import race_attention_kernel_b200.ops as ops
    from race_attention_kernel_b200 import _lib
    N, T = 3, 200
    pq, pk, v, dO = _inputs(N, T, L, R, dk, seed=7)
    want = ops.race_causal_backward(pq, pk, v, dO)
    got = [torch.empty(t.numel() + 8, device="cuda", dtype=t.dtype)[8:].view_as(t) for t in want]
    assert all(t.data_ptr() % 32 == 16 for t in got)
    sh = ops.make_shape(N, T, L, R, dk, torch.bfloat16, 1e-6)
    n = _lib.lib().race_b200_causal_bwd_workspace_bytes(ctypes.byref(sh))
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    rc = _lib.lib().race_b200_causal_bwd(*map(ops._ptr, (pq, pk, v, dO)), *map(ops._ptr, got), ops._ptr(ws), n,
                                         ctypes.byref(sh), ops._stream(), None)
    assert rc == 0
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def _reference(pq, pk, v, dO, A0, B0, d_state):
    """Gradients in 64 bits of one chunk (src/race_baseline.py:45-51 with the state of the tokens before it)."""
    q, k, x, a, b = (t.double().requires_grad_(True) for t in (pq.flatten(2), pk.flatten(2), v, A0.flatten(1), B0.flatten(1, 2)))
    w = q / (a.unsqueeze(1) + k.cumsum(1) + 1e-6)
    out = torch.tril(w @ k.transpose(1, 2)) @ x + w @ b
    state = torch.cat([(b + k.transpose(1, 2) @ x).flatten(1), a + k.sum(1)], 1)
    dq, dk, dx, da, db = torch.autograd.grad((out, state), (q, k, x, a, b), (dO.double(), d_state.double()))
    return dq.view_as(pq), dk.view_as(pk), dx, torch.cat([db.flatten(1), da], 1)


@pytest.mark.parametrize("L,R,dk", GEOMETRIES)
@pytest.mark.parametrize("T", [1, 128, 129, 1500])
def test_chunk_of_a_longer_sequence(L, R, dk, T):
    import race_attention_kernel_b200.ops as ops
    N, S = 4, L * R
    pq, pk, v, dO = _inputs(N, T, L, R, dk, seed=T + S + dk)
    g = torch.Generator(device="cuda").manual_seed(T)
    A0 = torch.rand(N, L, R, device="cuda", generator=g) * 20 + 1
    B0 = torch.randn(N, L, R, dk, device="cuda", generator=g) * 5
    d_state = torch.randn(N, S * (dk + 1), device="cuda", generator=g)
    kw = dict(carry_in=ops.pack_state(A0, B0), grad_state=d_state)
    ref = _reference(pq, pk, v, dO, A0, B0, d_state)
    for got in (ops.race_causal_backward(pq, pk, v, dO, **kw),
                ops.race_causal_backward(pq, pk, v, dO, return_grad_carry=True, **kw)):
        for a, b in zip(got[:3], ref):      # nothing but the results is rounded to bf16: 2^-9
            assert ro.rel_l2(a, b) <= 4e-3
    # the gradient of the carry is an fp32 tensor: fp32 products and sums of T terms
    assert ro.rel_l2(got[3][:, S * dk:], ref[3][:, S * dk:]) <= 1e-6
    assert ro.rel_l2(got[3][:, :S * dk], ref[3][:, :S * dk]) <= 1e-6
    # V and the gradient in the operator's layout, as two heads

    def operator_layout(x):
        return x.view(1, 2, 2, T, dk).permute(0, 1, 3, 2, 4).contiguous()

    heads = ops.race_causal_backward(pq, pk, operator_layout(v), operator_layout(dO), return_grad_carry=True, **kw)
    for a, b in zip(heads, (got[0], got[1], operator_layout(got[2]), got[3])):
        assert torch.equal(a, b)
