"""Errors against 64 bits where a step for speed could cost some: sums of whole tiles, and gradients of fp32 tensors."""
from __future__ import annotations

import pytest
import torch

from oracle import race_oracle as ro

pytestmark = pytest.mark.gpu


# An accumulator rounds each of its additions down: of a tile of n tokens it takes n / 16 per limb product (three in fp32,
# one in bf16), each half a unit of 2^-23 off on average, on a sum that has grown to two thirds of its end by then.  The
# tile of 64 streams of 8192 tokens has at most 1024: 64 x 2^-24 x 2/3 = 2.5e-6 in bf16, three times that in fp32.
@pytest.mark.parametrize("dt,bound", [(torch.bfloat16, 2.5e-6), (torch.float32, 7.6e-6)])
def test_state_of_many_streams(dt, bound):
    import race_attention_kernel_b200.ops as ops
    N, T = 64, 8192
    g = torch.Generator(device="cuda").manual_seed(0)
    pq, pk = (torch.softmax(torch.randn(N, T, 4, 16, device="cuda", generator=g), -1).to(dt) for _ in range(2))
    v = torch.randn(N, T, 64, device="cuda", generator=g).to(dt)
    out, A, B = ops.race_causal_prefix(pq, pk, v, return_state=True)
    p64, v64 = pk.flatten(2).double(), v.double()
    assert ro.rel_l2(A.flatten(1), p64.sum(1)) <= 5e-7
    assert ro.rel_l2(B.flatten(1, 2), p64.transpose(1, 2) @ v64) <= bound
    if dt == torch.bfloat16:   # outputs alone take longer tiles: the same but for their rounding
        assert ro.rel_l2(ops.race_causal_prefix(pq, pk, v), out) <= 1e-3


def _probs64(x, planes, L, K):
    """[1,B,T,H,d_k] fp64 -> [B*H,T,L,R] (src/race_baseline.py:35-44)."""
    _, B, T, H, dk = x.shape
    corners = torch.tensor([[2.0 * ((r >> (K - 1 - k)) & 1) - 1 for r in range(1 << K)] for k in range(K)],
                           dtype=torch.float64, device=x.device)
    proj = (x.permute(0, 1, 3, 2, 4).reshape(B * H, T, dk) @ planes.double().T).view(B * H, T, L, K)
    return torch.softmax(proj.tanh() / dk ** 0.5 @ corners, -1)


def _rows(dk, L, K, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(1, 2, 500, 4, dk, device="cuda", generator=g), torch.randn(L * K, dk, device="cuda", generator=g),
            torch.randn(8, 500, L, 1 << K, device="cuda", generator=g))


@pytest.mark.parametrize("dk,L,K", [(64, 4, 4), (128, 8, 6)])
def test_gradient_of_the_producer_in_fp32(dk, L, K):
    """As exact as fp32 arithmetic: both products have three limbs of both operands and no long chain in an accumulator, and
    what is left are about ten roundings of 2^-24 (a result off by 2^-17 of a limb left out is ten times that)."""
    import race_attention_kernel_b200.ops as ops
    x, planes, dp = _rows(dk, L, K)
    x64 = x.double().requires_grad_(True)
    (ref,) = torch.autograd.grad(_probs64(x64, planes, L, K), x64, dp.double())
    assert ro.rel_l2(ops.bucket_probs_streams_bwd(x, planes, dp, L, K), ref) <= 10 * 2.0 ** -24


@pytest.mark.parametrize("dk,L,K", [(64, 4, 4), (128, 8, 6)])
def test_probabilities_of_a_training_step_in_fp32(dk, L, K):
    """Rounded once: at most 2^-24, a little over half of that in the mean square, and 1e-8 from the projections."""
    import race_attention_kernel_b200.ops as ops
    x, planes, _ = _rows(dk, L, K)
    assert ro.rel_l2(ops.bucket_probs_streams(x, planes, L, K, exact=True), _probs64(x.double(), planes, L, K)) <= 4.5e-8
