"""The operator's training node in Python, which runs where the one in C++ does not apply: host tensors, inputs that are not
contiguous, fp32 at d_k = 128."""
from __future__ import annotations

import pytest
import torch

from oracle import race_oracle as ro

pytestmark = pytest.mark.gpu

GEOMETRIES = [(64, 4, 4, torch.float32), (64, 4, 4, torch.bfloat16), (128, 6, 8, torch.bfloat16)]   # d_k, K, L, type


def _call(ace, inputs, g):
    leaves = [t.detach().requires_grad_(True) for t in inputs]
    out = ace(*leaves)
    return (out.detach(), *torch.autograd.grad(out, leaves, g))


def _setup(dk, K, L, dt, B=2, T=150, H=3):
    import race_attention_kernel_b200 as rk
    torch.manual_seed(dk)
    ace = rk.BatchedACE(dk, K, L, 1).cuda()
    return ace, [torch.randn(1, B, T, H, dk, device="cuda").to(dt) for _ in range(4)]


@pytest.mark.parametrize("dk,K,L,dt", GEOMETRIES)
def test_host_tensors_and_strides_have_the_bits_of_the_plain_call(dk, K, L, dt):
    ace, x = _setup(dk, K, L, dt)
    want = _call(ace, x[:3], x[3])
    on_host = _call(ace, [t.cpu() for t in x[:3]], x[3].cpu())
    assert all(t.device.type == "cpu" for t in on_host)
    assert all(torch.equal(a.cuda(), b) for a, b in zip(on_host, want))
    strided = [t.transpose(2, 3).contiguous().transpose(2, 3) for t in x]
    assert not strided[0].is_contiguous()
    assert all(map(torch.equal, _call(ace, strided[:3], strided[3]), want))
    expanded = torch.ones((), device="cuda", dtype=dt).expand(x[3].shape)
    assert all(map(torch.equal, _call(ace, strided[:3], expanded), _call(ace, x[:3], expanded.contiguous())))


def test_only_some_inputs_need_a_gradient():
    ace, x = _setup(64, 4, 4, torch.float32)
    want = _call(ace, x[:3], x[3])
    for i in range(3):
        for call in (x, [t.cpu() for t in x]):
            leaves = [t.detach().requires_grad_(i == j) for j, t in enumerate(call[:3])]
            (got,) = torch.autograd.grad(ace(*leaves), leaves[i], call[3])
            assert torch.equal(got.cuda(), want[i + 1])


@pytest.mark.parametrize("B,T,H", [(1, 37, 1), (2, 200, 3)])
def test_fp32_with_wide_rows(B, T, H):
    """Against 64 bits; fp32 products all the way.  The gradients of K and Q are differences of terms that nearly cancel (a
    gradient of the probabilities against its mean): measured 6e-7, and 20 roundings of 2^-24 allow twice that."""
    dk, K, L = 128, 6, 8
    ace, x = _setup(dk, K, L, torch.float32, B, T, H)
    k, v, q = (t.double().requires_grad_(True) for t in x[:3])
    corners = torch.tensor([[2.0 * ((r >> (K - 1 - j)) & 1) - 1 for r in range(1 << K)] for j in range(K)],
                           dtype=torch.float64, device="cuda")

    def streams(t):
        return t.permute(0, 1, 3, 2, 4).reshape(B * H, T, dk)

    pk, pq = (torch.softmax((streams(t) @ ace.planes_T.double()).view(B * H, T, L, K).tanh() / dk ** 0.5 @ corners, -1).flatten(2)
              for t in (k, q))
    o = torch.tril((pq / (pk.cumsum(1) + ace.eps)) @ pk.transpose(1, 2)) @ streams(v)
    o = o.view(1, B, H, T, dk).permute(0, 1, 3, 2, 4)
    ref = (o, *torch.autograd.grad(o, (k, v, q), x[3].double()))
    for a, b in zip(_call(ace, x[:3], x[3]), ref):
        assert ro.rel_l2(a, b) <= 20 * 2.0 ** -24


@pytest.mark.parametrize("dk,K,L,dt", GEOMETRIES)
def test_saved_tensors_that_go_elsewhere(dk, K, L, dt):
    """Hooks, checkpoints and dispatch modes around the node in C++: what comes back may lie in memory differently."""
    from torch.autograd.graph import save_on_cpu, saved_tensors_hooks
    from torch.utils.checkpoint import checkpoint
    from torch.utils._python_dispatch import TorchDispatchMode

    class Through(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    ace, x = _setup(dk, K, L, dt)
    want = _call(ace, x[:3], x[3])
    strided = saved_tensors_hooks(lambda t: t.transpose(0, 1).contiguous(), lambda t: t.transpose(0, 1))
    for context in (save_on_cpu(), save_on_cpu(pin_memory=True), strided, Through()):
        with context:
            got = _call(ace, x[:3], x[3])
        assert all(map(torch.equal, got, want))
    leaves = [t.detach().requires_grad_(True) for t in x[:3]]
    out = checkpoint(ace, *leaves, use_reentrant=False)
    out.backward(x[3])
    assert all(map(torch.equal, (out, *(t.grad for t in leaves)), want))
    # planes that are stored the other way round, through the same hooks
    ace.planes_T = ace.planes_T.contiguous()
    for context in (save_on_cpu(pin_memory=True), strided):
        with context:
            got = _call(ace, x[:3], x[3])
        assert all(map(torch.equal, got, want))
