"""Gradients on the GPU: the backward of the producer and the operator under autograd at the geometries that run on the
kernels alone, against torch.autograd through the restated forward (src/race_baseline.py:41-51) in fp64."""
from __future__ import annotations

import pytest
import torch

from oracle import race_oracle as ro

pytestmark = pytest.mark.gpu

# fp32: three-limb projections, two-limb products elsewhere (2^-17 per factor); bf16: the outputs' own rounding (2^-9)
# and that of the probabilities and their gradients, each of which enters a result once
TOL = {torch.float32: 3e-5, torch.bfloat16: 1e-2}
GEOMETRIES = [(64, 4, 4, torch.float32), (64, 4, 4, torch.bfloat16), (128, 6, 8, torch.bfloat16)]   # d_k, K, L, type


def _probs64(x, planes, L, K):
    """[M,B,T,H,d_k] fp64 -> [N,T,L,R] (src/race_baseline.py:35-44)."""
    M, B, T, H, dk = x.shape
    corners = torch.tensor([[2.0 * ((r >> (K - 1 - k)) & 1) - 1 for r in range(1 << K)] for k in range(K)],
                           dtype=torch.float64, device=x.device)
    x2 = x.permute(0, 1, 3, 2, 4).reshape(M * B * H, T, dk)
    proj = (x2 @ planes.double().T).view(M * B * H, T, L, K)
    return torch.softmax(proj.tanh() / dk ** 0.5 @ corners, -1)


def _leaf(x):
    return x.detach().double().requires_grad_(True)


@pytest.mark.parametrize("dk,K,L,dt", GEOMETRIES + [(128, 6, 8, torch.float32)])
@pytest.mark.parametrize("B,T,H", [(1, 1, 1), (2, 37, 3), (1, 1003, 4)])
def test_producer_backward(dk, K, L, dt, B, T, H):
    import race_attention_kernel_b200.ops as ops
    g = torch.Generator(device="cuda").manual_seed(T + dk)
    x = torch.randn(1, B, T, H, dk, device="cuda", generator=g).to(dt)
    planes = torch.randn(L * K, dk, device="cuda", generator=g)
    dp = torch.randn(B * H, T, L, 1 << K, device="cuda", generator=g).to(dt)
    got = ops.bucket_probs_streams_bwd(x, planes, dp, L, K)
    x64 = _leaf(x)
    (ref,) = torch.autograd.grad(_probs64(x64, planes, L, K), x64, dp.double())
    # nothing but the result is rounded here: 2^-9 for bf16
    assert ro.rel_l2(got, ref) <= (2e-5 if dt == torch.float32 else 4e-3)


@pytest.mark.parametrize("dk,K,L,dt", GEOMETRIES + [(128, 6, 8, torch.float32), (32, 3, 4, torch.float32)])
@pytest.mark.parametrize("B,T,H", [(1, 1, 1), (2, 37, 3), (3, 1003, 16)])
def test_two_tensors_in_one_launch(dk, K, L, dt, B, T, H):
    """The pair entries give the bits of the single ones (the last geometry has no kernel for two tensors)."""
    import race_attention_kernel_b200.ops as ops
    from race_attention_kernel_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(T + dk)
    x = [torch.randn(1, B, T, H, dk, device="cuda", generator=g).to(dt) for _ in range(2)]
    planes = torch.randn(L * K, dk, device="cuda", generator=g)
    dims = (B, T, H, dk, L, K, ops._DTYPES[dt])
    for exact in (0, 1):
        p = [torch.empty(B * H, T, L, 1 << K, device="cuda", dtype=dt) for _ in range(2)]
        assert _lib.lib().race_b200_bucket_probs_streams_pair(
            *map(ops._ptr, x), ops._ptr(planes), *map(ops._ptr, p), *dims, exact, ops._stream()) == 0
        for a, b in zip(x, p):
            assert torch.equal(b, ops.bucket_probs_streams(a, planes, L, K, exact=bool(exact)))
    if not ops.bucket_probs_bwd_is_supported(dk, L, K, dt):
        return
    dp = [torch.randn_like(t) for t in p]
    dx = [torch.empty_like(t) for t in x]
    assert _lib.lib().race_b200_bucket_probs_streams_bwd_pair(
        *map(ops._ptr, x), ops._ptr(planes), *map(ops._ptr, dp), *map(ops._ptr, dx), *dims, ops._stream()) == 0
    for a, b, c in zip(x, dp, dx):
        assert torch.equal(c, ops.bucket_probs_streams_bwd(a, planes, b, L, K))


@pytest.mark.parametrize("dk,K,L,dt", GEOMETRIES)
@pytest.mark.parametrize("B,T,H", [(1, 1, 2), (2, 127, 3), (1, 128, 2), (1, 129, 1), (1, 2500, 2)])
def test_operator_gradients(dk, K, L, dt, B, T, H):
    """Edges of the 64- and 128-token chunks, one token, several state tiles."""
    import race_attention_kernel_b200 as rk
    torch.manual_seed(T)
    ace = rk.BatchedACE(dk, K, L, 1).cuda()
    Kh, Vh, Qh, dO = (torch.randn(1, B, T, H, dk, device="cuda").to(dt) for _ in range(4))
    for t in (Kh, Vh, Qh):
        t.requires_grad_(True)
    out = ace(Kh, Vh, Qh)
    got = (out, *torch.autograd.grad(out, (Kh, Vh, Qh), dO))
    k, v, q = _leaf(Kh), _leaf(Vh), _leaf(Qh)
    planes = ace.planes_T.T
    pK, pQ = _probs64(k, planes, L, K).flatten(2), _probs64(q, planes, L, K).flatten(2)
    v2 = v.permute(0, 1, 3, 2, 4).reshape(B * H, T, dk)
    o = torch.tril((pQ / (pK.cumsum(1) + ace.eps)) @ pK.transpose(1, 2)) @ v2
    o = o.view(1, B, H, T, dk).permute(0, 1, 3, 2, 4)
    ref = (o, *torch.autograd.grad(o, (k, v, q), dO.double()))
    for name, a, b in zip(("out", "dK", "dV", "dQ"), got, ref):
        assert a.shape == b.shape and a.dtype == dt
        if name in ("dK", "dQ") and T == 1:
            # with one token the output does not depend on the probabilities (pQ_1 B_1 / A_1 = pQ_1 (x) V_1 summed over
            # a softmax): both gradients cancel to O(eps).  What is left are rounding errors of terms of size
            # |V . dO| <= 40, 2^-17 of them in fp32 and 2^-9 in bf16, through a Jacobian below 1.
            assert float(a.double().abs().max()) <= {torch.float32: 1e-3, torch.bfloat16: 0.5}[dt]
            continue
        assert ro.rel_l2(a, b) <= TOL[dt], (name, ro.rel_l2(a, b))


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,T", [(1, 1), (2, 127), (3, 128), (40, 300), (300, 130), (2, 20000)])
def test_noncausal_shares(N, T, dt):
    """The non-causal token kernel deals the 128-token chunks of all streams out to the SMs in equal shares: one chunk,
    remainders, fewer and more chunks than SMs, shares that begin and end inside a stream."""
    import race_attention_kernel_b200.ops as ops
    g = torch.Generator(device="cuda").manual_seed(T)
    pq, pk = (torch.softmax(torch.randn(N, T, 4, 16, device="cuda", generator=g), -1).to(dt).requires_grad_(True)
              for _ in range(2))
    v, dO = (torch.randn(N, T, 64, device="cuda", generator=g).to(dt) for _ in range(2))
    v.requires_grad_(True)
    out = ops.race_noncausal(pq, pk, v)
    got = (out, *torch.autograd.grad(out, (pq, pk, v), dO))
    a, b, c = (_leaf(t) for t in (pq, pk, v))
    o = a.flatten(2) @ ((b.flatten(2).transpose(1, 2) @ c) / (b.flatten(2).sum(1).unsqueeze(-1) + 1e-6))
    for name, x, y in zip(("out", "dPQ", "dPK", "dV"), got, (o, *torch.autograd.grad(o, (a, b, c), dO.double()))):
        if name == "dPK" and T == 1:
            continue    # cancels to O(eps): only rounding errors are left
        assert ro.rel_l2(x, y) <= (2e-5 if dt == torch.float32 else 4e-3), (name, ro.rel_l2(x, y))
