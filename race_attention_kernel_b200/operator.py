"""Drop-in operator: ``BatchedACE`` with the reference's constructor and call signature.

    ace = BatchedACE(d_k, K, L, M)            # buffers drawn like the reference (CPU RNG)
    ace = ace.cuda()
    out = ace(Khf, Vhf, Qhf)                  # argument order K, V, Q; each [M,B,T,H,d_k]

(src/race_baseline.py:21-52).  Buffers keep the reference's names and shapes (``planes_T``
[d_k, L*K], ``protos_T`` [K, R]) so code that overwrites ``ace.planes_T`` keeps working.
The forward runs on the GPU only: bucket probabilities come from the producer kernel and the
cumsum/divide/bmm of the reference is replaced by the prefix kernel.  Host tensors are
accepted and streamed through the device; there is no CPU compute path.

Gradients: the reference module is differentiable through K, V and Q (plain autograd over
src/race_baseline.py:41-51).  Here, when autograd is recording and an input requires a gradient,
``forward`` is one autograd node over the kernels: the producer, the prefix forward, and for the gradients
the causal backward and the backward of the producer (in C++ where every kernel takes the operator's layout).  Geometries the producer's backward does not cover, planes with a gradient and other prototypes form
the bucket probabilities with differentiable torch ops and run the prefix path through ``ops.race_causal``.
"""
from __future__ import annotations

import itertools

import torch
from torch import nn

from . import _lib, ops


class _CausalOperator(torch.autograd.Function):
    """``BatchedACE.forward`` with gradients for K, V and Q ([M,B,T,H,d_k], contiguous, on the GPU; planes [L*K, d_k]).
    Saved: the inputs and the two probability tensors; the backward recomputes the prefix states tile by tile."""

    @staticmethod
    def forward(ctx, Khf, Vhf, Qhf, planes, L, K, eps):
        M, B, T, H, dk = Khf.shape
        Khf, Qhf, planes = (_on_boundary(t) for t in (Khf, Qhf, planes))
        pK = ops.bucket_probs_streams(Khf, planes, L, K, exact=True)
        pQ = ops.bucket_probs_streams(Qhf, planes, L, K, exact=True)
        shape = (M * B * H, T, L, 1 << K, dk, Vhf.dtype)
        if H > 1 and T > 1:
            Vhf = _on_boundary(Vhf)
        V2 = None
        if ops.is_supported(*shape, "auto", heads=H):
            out = ops.race_causal_prefix(pQ, pK, Vhf, eps)
        else:
            V2 = _streams(Vhf)
            out = _unstreams(ops.race_causal_prefix(pQ, pK, V2, eps), M, B, H)
        ctx.bwd_heads = ops.causal_bwd_takes_heads(*shape, H)
        if ctx.bwd_heads or V2 is None:
            V2 = Vhf
        ctx.save_for_backward(Khf, V2, Qhf, pK, pQ, planes)
        ctx.dims, ctx.eps = (M, B, H, L, K), eps
        return out

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, grad_out):
        Khf, V, Qhf, pK, pQ, planes = ctx.saved_tensors
        M, B, H, L, K = ctx.dims
        want_k, want_v, want_q = ctx.needs_input_grad[:3]
        grad_out = grad_out.to(V.dtype)
        if ctx.bwd_heads:
            dpq, dpk, dV = ops.race_causal_backward(pQ, pK, V, _on_boundary(grad_out.contiguous()), ctx.eps)
        else:
            V2 = V if V.dim() == 3 else _streams(V)
            dpq, dpk, dV = ops.race_causal_backward(pQ, pK, V2, _streams(grad_out), ctx.eps)
            dV = _unstreams(dV, M, B, H)
        dK = ops.bucket_probs_streams_bwd(Khf, planes, dpk, L, K) if want_k else None
        dQ = ops.bucket_probs_streams_bwd(Qhf, planes, dpq, L, K) if want_q else None
        return dK, dV if want_v else None, dQ, None, None, None, None


def _on_boundary(x: torch.Tensor) -> torch.Tensor:
    """The kernels want 16-byte boundaries; gradients are also given for rows that begin elsewhere."""
    return x if x.data_ptr() % 16 == 0 else x.clone()


def _streams(x: torch.Tensor) -> torch.Tensor:
    """[M,B,T,H,d_k] -> [M*B*H, T, d_k] (src/race_baseline.py:35-40)."""
    M, B, T, H, dk = x.shape
    return x.permute(0, 1, 3, 2, 4).contiguous().view(M * B * H, T, dk)


def _unstreams(x2: torch.Tensor, M: int, B: int, H: int) -> torch.Tensor:
    return x2.view(M, B, H, *x2.shape[1:]).permute(0, 1, 3, 2, 4)


class BatchedACE(nn.Module):
    def __init__(self, d_k, K, L, M, device="cpu", share_planes=True):
        super().__init__()
        assert share_planes, "reference config uses shared planes"
        self.d_k, self.K, self.L, self.M = d_k, K, L, M
        self.R = 1 << K
        # drawn exactly like the reference (src/race_baseline.py:27-32) so that a seeded
        # construction gives the same planes
        planes = torch.randn(L, K, d_k, device=device)
        self.register_buffer("planes_T", planes.view(L * K, d_k).T)
        corners = torch.tensor(list(itertools.product([-1.0, 1.0], repeat=K)), device=device)
        self.register_buffer("protos_T", corners.T)
        self._protos_hold_corners()
        self.eps = 1e-6
        self.variant = "auto"
        # form the bucket probabilities inside the prefix kernels where that path exists (fp32, d_k = 64, L = 4,
        # K = 4); False keeps the producer kernel and the probabilities in device memory
        self.fuse_producer = True

    def _streams(self, x: torch.Tensor) -> torch.Tensor:
        return _streams(x)

    def bucket_probs(self, x2: torch.Tensor) -> torch.Tensor:
        """[N,T,d_k] -> [N,T,L,R] with this module's planes."""
        planes = self.planes_T.T.contiguous().float()
        return ops.bucket_probs(x2, planes, self.L, self.K)

    def _probs_autograd(self, x2: torch.Tensor) -> torch.Tensor:
        """src/race_baseline.py:41-44 with torch ops (differentiable); x2 [N,T,d_k] on the GPU."""
        N, T, dk = x2.shape
        planes_T = self.planes_T.to(device=x2.device, dtype=torch.float32)
        protos_T = self.protos_T.to(device=x2.device, dtype=torch.float32)
        proj = (x2.float() @ planes_T).view(N, T, self.L, self.K)
        logits = proj.tanh().div(dk ** 0.5) @ protos_T
        return torch.softmax(logits, dim=-1).to(x2.dtype)

    def _protos_unchanged(self, p) -> bool:
        """The buffer is the tensor last found to hold the corners, and has not been written to since."""
        seen = self.__dict__.get("_protos_seen")
        return seen is not None and seen[0] is p and not p.is_inference() and seen[1:] == (p._version, p.data_ptr())

    def _protos_are_corners(self) -> bool:
        """Whether ``protos_T`` holds what the kernels are built on: training honours other prototypes, with torch ops.
        Compared by value, which reads back from the GPU, when the buffer is another tensor than at the last comparison or
        has been written to since (its version counter; writes through ``.data`` are not counted by torch)."""
        p = self.protos_T
        if self._protos_unchanged(p):
            return not p.requires_grad
        same = p.dim() == 2 and p.T.tolist() == [list(c) for c in itertools.product([-1.0, 1.0], repeat=self.K)]
        if same:
            self._protos_hold_corners()
        return same and not p.requires_grad

    def _protos_hold_corners(self) -> None:
        p = self.protos_T
        if type(p) is torch.Tensor and not p.is_meta and not p.is_inference():
            self.__dict__["_protos_seen"] = (p, p._version, p.data_ptr())

    def _move(self, move, *args, **kwargs):
        known = self._protos_unchanged(self.protos_T)
        move(*args, **kwargs)
        if known:   # the same values elsewhere: nothing to read back
            self._protos_hold_corners()
        return self

    def to(self, *args, **kwargs):
        return self._move(super().to, *args, **kwargs)

    def cuda(self, *args, **kwargs):
        return self._move(super().cuda, *args, **kwargs)

    def _forward_autograd(self, Khf, Vhf, Qhf):
        M, B, T, H, dk = Khf.shape
        dev = self.planes_T.device if self.planes_T.is_cuda else torch.device("cuda", torch.cuda.current_device())
        if (Khf.numel() and Khf.dtype == Vhf.dtype == Qhf.dtype and ops.bucket_probs_bwd_is_supported(dk, self.L, self.K, Khf.dtype)
                and not self.planes_T.requires_grad and self._protos_are_corners()):
            planes = self.planes_T.T.contiguous().float().to(dev)
            out = _CausalOperator.apply(*(t.to(dev).contiguous() for t in (Khf, Vhf, Qhf)), planes, self.L, self.K, self.eps)
            return out if Khf.is_cuda else out.cpu()
        K2, V2, Q2 = (self._streams(t.to(dev)) for t in (Khf, Vhf, Qhf))
        out2 = ops.race_causal(self._probs_autograd(Q2), self._probs_autograd(K2), V2, self.eps)
        out = out2.view(M, B, H, T, dk).permute(0, 1, 3, 2, 4)
        return out if Khf.is_cuda else out.cpu()

    def forward(self, Khf, Vhf, Qhf, *, carry_in=None, return_state=False):
        grad = torch.is_grad_enabled() and (Khf.requires_grad or Vhf.requires_grad or Qhf.requires_grad)
        if not grad and self.variant == "auto" and Khf.is_cuda:
            # the plain call in C++ (None: something about the arguments needs the general path below)
            if isinstance(carry_in, (tuple, list)):
                carry_in = ops.pack_state(*carry_in)
            res = _lib.native().forward(self.planes_T, Khf, Vhf, Qhf, self.L, self.K, self.eps, carry_in, bool(return_state),
                                        bool(self.fuse_producer), ops._status_ptr(Khf.get_device()))
            if res is not None:
                return res
        if not (Khf.shape == Vhf.shape == Qhf.shape) or Khf.dim() != 5:
            raise RuntimeError("expected K, V, Q of identical shape [M,B,T,H,d_k]")
        M, B, T, H, dk = Khf.shape
        if dk != self.d_k:
            raise RuntimeError(f"d_k mismatch: module {self.d_k}, input {dk}")
        if grad:
            if carry_in is not None or return_state:
                raise RuntimeError("carry_in / return_state are inference-only; chain ops.race_causal_chunk "
                                   "for differentiable chunked sequences")
            if Khf.is_cuda and self._protos_are_corners():
                out = _lib.native().train_forward(self.planes_T, Khf, Vhf, Qhf, self.L, self.K, self.eps,
                                                  ops._status_ptr(Khf.get_device()))
                if out is not None:
                    return out
            if Khf.dtype not in (torch.float32, torch.bfloat16):
                raise RuntimeError("fp32 or bf16 inputs only")
            return self._forward_autograd(Khf, Vhf, Qhf)
        with torch.no_grad():
            return self._forward_kernels(Khf, Vhf, Qhf, carry_in, return_state)

    def _forward_kernels(self, Khf, Vhf, Qhf, carry_in, return_state):
        M, B, T, H, dk = Khf.shape
        host = not Khf.is_cuda
        dev = self.planes_T.device if self.planes_T.is_cuda else torch.device("cuda", torch.cuda.current_device())
        if host:
            Khf, Vhf, Qhf = (t.to(dev, non_blocking=True) for t in (Khf, Vhf, Qhf))
        if Khf.dtype not in (torch.float32, torch.bfloat16):
            raise RuntimeError("fp32 or bf16 inputs only")
        planes = self.planes_T.T.contiguous().float()
        if self.fuse_producer and self.variant == "auto" and ops.qkv_is_supported(M * B * H, T, self.L, self.K, dk, Khf.dtype, heads=H):
            # the prefix kernels form the bucket probabilities themselves: Q, K, V in, out back, nothing else
            res = ops.race_causal_qkv(Qhf.contiguous(), Khf.contiguous(), Vhf.contiguous(), planes, self.L, self.K,
                                      self.eps, carry_in=carry_in, return_state=return_state)
            out = res[0] if return_state else res
            if host:
                out = out.cpu()
            return (out, res[1], res[2]) if return_state else out
        # K and Q are only read by the producer, which flattens [M,B,T,H,d_k] -> streams on the fly;
        # V is consumed by the prefix kernels as [N,T,d_k] and is copied once
        pK = ops.bucket_probs_streams(Khf.contiguous(), planes, self.L, self.K)
        pQ = ops.bucket_probs_streams(Qhf.contiguous(), planes, self.L, self.K)
        N, S_l, S_r = M * B * H, self.L, 1 << self.K
        if self.variant == "auto" and ops.is_supported(N, T, S_l, S_r, dk, Vhf.dtype, "auto", heads=H):
            # the prefix kernels read V and write the output in [M,B,T,H,d_k] directly
            res = ops.race_causal_prefix(pQ, pK, Vhf.contiguous(), self.eps, carry_in=carry_in,
                                         return_state=return_state, variant=self.variant)
            out = res[0] if return_state else res
        else:
            V2 = self._streams(Vhf)
            res = ops.race_causal_prefix(pQ, pK, V2, self.eps, carry_in=carry_in,
                                         return_state=return_state, variant=self.variant)
            out2 = res[0] if return_state else res
            out = out2.view(M, B, H, T, dk).permute(0, 1, 3, 2, 4)
        if host:
            out = out.cpu()
        return (out, res[1], res[2]) if return_state else out

    def step(self, Khf, Vhf, Qhf, state: torch.Tensor):
        """Token-by-token generation: outputs for the ``t`` <= 64 NEW tokens ``[M,B,t,H,d_k]`` given the
        packed running state ``[M*B*H, S*(d_k+1)]`` of everything before them (``torch.zeros`` or
        ``ops.pack_state(A, B)`` of a ``forward(..., return_state=True)`` prefill); ``state`` is advanced
        in place.  Equals continuing the reference's chunked evaluation (src/race_chunked.py:54-63) by a
        chunk of ``t`` tokens."""
        if Khf.is_cuda:   # one launch where the geometry has it (None: the general path below)
            out = _lib.native().step(self.planes_T, Khf, Vhf, Qhf, state, self.L, self.K, self.eps)
            if out is not None:
                return out
        with torch.no_grad():
            return self._step(Khf, Vhf, Qhf, state)

    def _step(self, Khf, Vhf, Qhf, state: torch.Tensor):
        if not (Khf.shape == Vhf.shape == Qhf.shape) or Khf.dim() != 5:
            raise RuntimeError("expected K, V, Q of identical shape [M,B,t,H,d_k]")
        M, B, T, H, dk = Khf.shape
        if dk != self.d_k:
            raise RuntimeError(f"d_k mismatch: module {self.d_k}, input {dk}")
        if not (Khf.is_cuda and state.is_cuda):
            raise RuntimeError("step() takes CUDA tensors (there is no CPU path)")
        planes = self.planes_T.T.contiguous().float()
        pK = ops.bucket_probs_streams(Khf.contiguous(), planes, self.L, self.K)
        pQ = ops.bucket_probs_streams(Qhf.contiguous(), planes, self.L, self.K)
        out2 = ops.race_decode_step(pQ, pK, self._streams(Vhf), state, self.eps)
        return out2.view(M, B, H, T, dk).permute(0, 1, 3, 2, 4)
