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


def _off_boundary(x):
    """The same values in a contiguous tensor that begins 4 bytes (bf16: 2) after a 16-byte boundary."""
    y = torch.empty(x.numel() + 1, device=x.device, dtype=x.dtype)[1:].view_as(x).copy_(x)
    assert y.is_contiguous() and y.data_ptr() % 16
    return y


@pytest.mark.parametrize("dk,K,L,dt", [(64, 4, 4, torch.float32), (64, 4, 4, torch.bfloat16), (128, 6, 8, torch.bfloat16),
                                       (128, 6, 8, torch.float32)])
def test_training_takes_rows_off_the_boundary(dk, K, L, dt):
    ace, x = _ace(dk, K, L), _inputs(1, 150, 3, dk, dt, n=4)

    def grads(inputs, g):
        leaves = [t.requires_grad_(True) for t in inputs]
        out = ace(*leaves)
        return (out.detach(), *torch.autograd.grad(out, leaves, g))

    want = grads([t.clone() for t in x[:3]], x[3])
    for i in range(3):
        got = grads([_off_boundary(t) if i == j else t.clone() for j, t in enumerate(x[:3])], x[3])
        assert all(map(torch.equal, got, want))
    assert all(map(torch.equal, grads([t.clone() for t in x[:3]], _off_boundary(x[3])), want))
    ace.planes_T = _off_boundary(ace.planes_T.T.contiguous()).T
    assert all(map(torch.equal, grads([t.clone() for t in x[:3]], x[3]), want))


def test_v_off_the_boundary_where_it_was_always_copied():
    ace, (k, v, q) = _ace(), _inputs(1, 150, 3, 64, torch.bfloat16)
    with torch.no_grad():
        assert torch.equal(ace(k, _off_boundary(v), q), ace(k, v, q))
        with pytest.raises(RuntimeError, match="aligned"):
            ace(_off_boundary(k), v, q)
    states = [torch.zeros(3, 64 * 65, device="cuda") for _ in range(2)]
    k, v, q = (t[:, :, :5].contiguous() for t in (k, v, q))
    assert torch.equal(ace.step(k, _off_boundary(v), q, states[0]), ace.step(k, v, q, states[1]))
    assert torch.equal(*states)
    with pytest.raises(RuntimeError, match="aligned"):
        ace.step(_off_boundary(k), v, q, states[0])


def test_training_honours_other_prototypes():
    """Assigned, written in place or loaded; and the corners again, however they come back."""
    import copy
    ace, x = _ace(), _inputs(1, 70, 2, 64, torch.float32)

    def out(module=ace):
        return module(x[0].clone().requires_grad_(True), x[1], x[2]).detach()

    def by_hand(protos):
        p = [torch.softmax(((t.double().permute(0, 1, 3, 2, 4).reshape(2, 70, 64) @ ace.planes_T.double()).view(2, 70, 4, 4).tanh() / 8)
                           @ protos.double(), -1).flatten(2) for t in (x[0], x[2])]
        v = x[1].double().permute(0, 1, 3, 2, 4).reshape(2, 70, 64)
        o = torch.tril((p[1] / (p[0].cumsum(1) + ace.eps)) @ p[0].transpose(1, 2)) @ v
        return o.view(1, 1, 2, 70, 64).permute(0, 1, 3, 2, 4)

    def close(a, b):
        return float((a - b).norm() / b.norm()) < 3e-5

    corners = ace.protos_T.clone()
    other = corners * torch.linspace(8.0, 12.0, 16, device="cuda")
    want, want_other = out(), by_hand(other)
    assert close(want, by_hand(corners)) and not close(want, want_other)
    ace.protos_T = other
    assert close(out(), want_other)
    ace.protos_T = corners.clone()
    assert torch.equal(out(), want)
    with torch.no_grad():
        ace.protos_T.copy_(other)
    assert close(out(), want_other) and close(out(copy.deepcopy(ace)), want_other)
    ace.load_state_dict({**ace.state_dict(), "protos_T": corners})
    assert torch.equal(out(), want) and torch.equal(out(copy.deepcopy(ace)), want)
    ace.load_state_dict({**ace.state_dict(), "protos_T": other})
    assert close(out(), want_other)


@pytest.mark.parametrize("kind", ["forward", "training", "prefix"])
def test_other_threads_run_while_a_call_waits(kind, monkeypatch):
    """The call synchronises here (RACE_B200_CHECK_STATUS=1) behind a kernel that keeps the GPU busy for half a second."""
    import threading
    import time

    import race_attention_kernel_b200.ops as ops
    monkeypatch.setenv("RACE_B200_CHECK_STATUS", "1")
    ace, (k, v, q) = _ace(), _inputs(1, 64, 2, 64, torch.float32)
    p = torch.softmax(torch.randn(2, 64, 4, 16, device="cuda"), -1)
    call = {"forward": lambda: ace(k, v, q), "training": lambda: ace(k.requires_grad_(True), v, q),
            "prefix": lambda: ops.race_causal_prefix(p, p, v[0, 0].permute(1, 0, 2).contiguous())}[kind]
    call()
    stamps, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            stamps.append(time.perf_counter())
            time.sleep(0.005)

    t = threading.Thread(target=tick)
    t.start()
    torch.cuda._sleep(int(1e9))
    t0 = time.perf_counter()
    call()
    waited = time.perf_counter() - t0
    stop.set()
    t.join()
    assert waited > 0.2
    assert max(b - a for a, b in zip(stamps, stamps[1:])) < 0.5 * waited


@pytest.mark.parametrize("shape", [(0, 5, 3), (2, 0, 3), (2, 5, 0)])
def test_training_on_nothing(shape):
    B, T, H = shape
    x = [t.requires_grad_(True) for t in _inputs(B, T, H, 64, torch.float32)]
    out = _ace()(*x)
    assert out.shape == (1, B, T, H, 64)
    for g, t in zip(torch.autograd.grad(out, x, torch.zeros_like(out)), x):
        assert g.shape == t.shape


def test_training_refuses_mixed_types_in_words():
    k, v, q = _inputs(1, 5, 2, 64, torch.float32)
    with pytest.raises(RuntimeError, match="dtype"):
        _ace()(k.requires_grad_(True), v.double(), q)


def test_a_tensor_subclass_gets_its_type_back():
    class Tagged(torch.Tensor):
        pass

    ace, x = _ace(), _inputs(1, 70, 2, 64, torch.float32)
    with torch.no_grad():
        out = ace(*(t.as_subclass(Tagged) for t in x))
        assert type(out) is Tagged and torch.equal(out.as_subclass(torch.Tensor), ace(*x))
