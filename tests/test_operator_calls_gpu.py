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


def test_steps_of_different_lengths_from_two_threads():
    """The wide step's shared memory grows with the number of new tokens; the limit is an attribute of the process."""
    import ctypes
    import threading

    import race_attention_kernel_b200.ops as ops
    from race_attention_kernel_b200 import _lib
    ace = _ace(128, 6, 8)
    planes = ace.planes_T.T.contiguous()
    codes = {}

    def steps(T):
        x = _inputs(1, T, 2, 128, torch.bfloat16, n=4)
        state = torch.zeros(2, 512 * 129, device="cuda")
        sh = ops.make_shape(2, T, 8, 64, 128, torch.bfloat16, 1e-6, 2)
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        codes[T] = {_lib.lib().race_b200_decode_step_qkv(*map(ops._ptr, x[:3]), ops._ptr(planes), ops._ptr(x[3]),
                                                         ops._ptr(state), ops._ptr(state), ctypes.byref(sh), 6,
                                                         ctypes.c_void_p(stream.cuda_stream)) for _ in range(3000)}
        stream.synchronize()

    threads = [threading.Thread(target=steps, args=(T,)) for T in (64, 20)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert codes == {64: {0}, 20: {0}}
