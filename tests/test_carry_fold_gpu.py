"""The state before each tile formed by the output kernels themselves (few tiles per stream) against the scan launch
(many), and the totals that are left out when nobody needs them."""
from __future__ import annotations

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(N, T, dk, dt, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    pQ, pK = (torch.softmax(torch.randn(N, T, 4, 16, device="cuda", generator=g), -1).to(dt) for _ in range(2))
    V = torch.randn(N, T, dk, device="cuda", generator=g).to(dt)
    carry = torch.rand(N, 64 * (dk + 1), device="cuda", generator=g) + 0.5
    return pQ, pK, V, carry


# 12 streams of 20 tiles take the scan launch, 2 fold; seven tiles are one more than a batch of loads
@pytest.mark.parametrize("dt,dk", [(torch.float32, 64), (torch.bfloat16, 64), (torch.bfloat16, 128)])
@pytest.mark.parametrize("norm", ["bucket", "global"])
@pytest.mark.parametrize("with_state", [False, True])
def test_folded_prefix_has_the_bits_of_the_scan(dt, dk, norm, with_state):
    import race_attention_kernel_b200 as rk
    pQ, pK, V, carry = _inputs(12, 20 * 64 - 5, dk, dt)

    def run(n, c):
        res = rk.race_causal_prefix(pQ[:n], pK[:n], V[:n], carry_in=carry[:n] if c else None, return_state=with_state,
                                    normalization=norm, tile_tokens=64, variant="tensor")
        return res if with_state else (res,)

    for c in (False, True):
        for many, few in zip(run(12, c), run(2, c)):
            assert torch.equal(many[:2], few)


@pytest.mark.parametrize("dt,dk", [(torch.float32, 64), (torch.bfloat16, 64)])
@pytest.mark.parametrize("T", [1, 64, 65, 128, 7 * 64 + 1])
def test_outputs_do_not_depend_on_the_state_being_asked_for(dt, dk, T):
    """Without a final state the last tile's totals are not formed."""
    import race_attention_kernel_b200 as rk
    pQ, pK, V, carry = _inputs(3, T, dk, dt, seed=T)
    for c in (None, carry):
        a = rk.race_causal_prefix(pQ, pK, V, carry_in=c, tile_tokens=64, variant="tensor")
        b, A, B = rk.race_causal_prefix(pQ, pK, V, carry_in=c, return_state=True, tile_tokens=64, variant="tensor")
        assert torch.equal(a, b)
        ref = pK.double().sum(1) + (0 if c is None else c[:, 64 * dk:].view(3, 4, 16).double())
        assert (A - ref).norm() / ref.norm() <= 1e-6


@pytest.mark.parametrize("dt,dk,T", [(torch.float32, 64, 500), (torch.bfloat16, 64, 500), (torch.float32, 64, 50)])
def test_state_over_its_own_carry(dt, dk, T):
    import race_attention_kernel_b200 as rk
    from race_attention_kernel_b200 import _lib, ops
    pQ, pK, V, carry = _inputs(4, T, dk, dt, seed=T)
    want = rk.race_causal_prefix(pQ, pK, V, carry_in=carry, return_state=True, tile_tokens=64, variant="tensor")
    state, out = carry.clone(), torch.empty_like(V)
    sh = ops.make_shape(4, T, 4, 16, dk, dt, 1e-6, 1)
    L = _lib.lib()
    var = _lib.VARIANTS["tensor"]
    ws = torch.empty(L.race_b200_causal_workspace_bytes(ctypes.byref(sh), 64, var), dtype=torch.uint8, device="cuda")
    rc = L.race_b200_causal_fwd(ops._ptr(pQ), ops._ptr(pK), ops._ptr(V), ops._ptr(out), ops._ptr(state), ops._ptr(state),
                                ops._ptr(ws), ws.numel(), ctypes.byref(sh), 64, var, ops._stream(), None)
    assert rc == 0
    assert torch.equal(out, want[0])
    assert torch.equal(state, ops.pack_state(want[1], want[2]).view_as(state))
