"""Calls of the operator in the forms user programs make them: what they accept, and what they must not depend on."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ace(dk=64, K=4, L=4, seed=0):
    import race_attention_kernel_b200 as rk
    torch.manual_seed(seed)
    return rk.BatchedACE(dk, K, L, 1).cuda()


def _inputs(B, T, H, dk, dt, n=3, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(1, B, T, H, dk, device="cuda", generator=g).to(dt) for _ in range(n)]


@pytest.mark.parametrize("T", [40, 777, 4096])
def test_planes_written_by_the_kernel_before(T):
    """Planes that are not stored as rows are copied by a kernel directly before the first launch of the call."""
    ace, x = _ace(), _inputs(1, T, 8, 64, torch.float32)
    for i in range(10):
        planes = torch.randn(16, 64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(i))
        ace.planes_T = planes.T
        torch.cuda.synchronize()
        with torch.no_grad():
            want = ace(*x)
        torch.cuda.synchronize()
        ace.planes_T = planes.T.contiguous()
        with torch.no_grad():
            assert torch.equal(ace(*x), want)
