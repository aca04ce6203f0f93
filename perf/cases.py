"""What a user of this package runs, as a list of measurable cases and a generator of more of the same kind.

Five kinds of call, each through the public entry points and in the types and geometries of the repository's own
configurations (d_k = 64, L = 4, K = 4 in fp32 and bf16; d_k = 128, L = 8, K = 6 in bf16):

  step       ``BatchedACE.step``: token-by-token generation against a running state that is advanced in place
  forward    ``BatchedACE.forward`` without gradients: prompts and long documents, also continued from a carried state
  train      ``BatchedACE.forward`` and the gradients of K, V and Q for a given gradient of the output
  prefix     ``race_causal_prefix`` on probabilities the caller has: the sweep configuration and sequence shards
  noncausal  ``race_noncausal`` forward and backward on probabilities: the full-sequence (vision) configuration
"""
from __future__ import annotations

import math

import torch

import race_attention_kernel_b200 as rk
from race_attention_kernel_b200 import ops

_DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
# (type, d_k, K hyperplanes, L tables) of the configurations
_F32 = dict(dtype="f32", dk=64, K=4, L=4)
_BF16 = dict(dtype="bf16", dk=64, K=4, L=4)
_WIDE = dict(dtype="bf16", dk=128, K=6, L=8)


def _case(kind, geometry, B, H, T, carry=False, **more):
    return dict(kind=kind, B=B, H=H, T=T, carry=carry, **geometry, **more)


def listed():
    return [
        # one user's chat, the next token: eight heads, one token each (the incremental step's latency workload)
        _case("step", _F32, 1, 8, 1, name="step_f32_b1"),
        # a server's decoding batch at the multi-head configuration (B = 8, H = 32): the state read and written is 2 x 67 MB
        _case("step", _WIDE, 8, 32, 1, name="step_bf16_wide_b8"),
        # a further turn of a conversation: a short ragged prompt on top of the state of earlier turns, the state returned
        _case("forward", _F32, 1, 8, 777, carry=True, name="turn_f32_t777"),
        # the CPU configuration's size (B = 1, H = 8, T = 4096) as one prompt
        _case("forward", _F32, 1, 8, 4096, name="prompt_f32_t4096"),
        # one very long document: the operator at the headline length of 2^20 tokens
        _case("forward", _F32, 1, 8, 1 << 20, name="document_f32_t1m"),
        # a batch of ragged prompts in bf16 at the small geometry, twelve heads
        _case("forward", _BF16, 4, 12, 5003, name="prompts_bf16_t5003"),
        # a long prompt at the multi-head bf16 configuration (H = 32, S = 512 buckets)
        _case("forward", _WIDE, 1, 32, 32768, name="prompt_bf16_wide_t32k"),
        # training steps of one attention layer: long sequences in fp32, a batch of 4096-token sequences in bf16,
        # and one sequence of the multi-head bf16 configuration
        _case("train", _F32, 4, 8, 16384, name="train_f32_t16k"),
        _case("train", _BF16, 8, 12, 4096, name="train_bf16_t4096"),
        _case("train", _WIDE, 1, 32, 4096, name="train_bf16_wide_t4096"),
        # the non-causal forward + backward configuration (B = 64, H = 12, T = 4096, fp32)
        _case("noncausal", _F32, 64, 12, 4096, name="noncausal_f32_b64"),
        # one rank's shard of a long sequence at the probabilities boundary: carry in, state out, 131072 tokens
        _case("prefix", _F32, 1, 8, 131072, carry=True, name="shard_f32_t131072"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# kind -> geometry -> (shortest T, longest T, most stream-tokens B*H*T)
_RANGES = {
    "step": ((_F32, 1, 8, 4096), (_BF16, 1, 8, 4096), (_WIDE, 1, 8, 256)),
    "forward": ((_F32, 16, 1 << 20, 1 << 23), (_BF16, 16, 1 << 20, 1 << 23), (_WIDE, 16, 1 << 17, 1 << 20)),
    "train": ((_F32, 64, 65536, 1 << 19), (_BF16, 64, 65536, 1 << 19), (_WIDE, 64, 16384, 1 << 17)),
    "prefix": ((_F32, 1024, 1 << 20, 1 << 23), (_BF16, 1024, 1 << 20, 1 << 23), (_WIDE, 1024, 1 << 17, 1 << 20)),
    "noncausal": ((_F32, 64, 16384, 3 << 20), (_BF16, 64, 16384, 3 << 20)),
}


def draw(rng):
    kind = rng.choice(("step", "forward", "forward", "train", "train", "prefix", "noncausal"))
    geometry, t_lo, t_hi, most = rng.choice(_RANGES[kind])
    H = rng.choice((4, 8, 12, 16, 32))
    if kind == "step":       # one new token mostly, sometimes a few (several guesses checked at once)
        T = rng.choice((1, 1, 1, 2, 3, t_hi))
        B = _log_uniform(rng, 1, max(1, most // H))
    else:
        T = _log_uniform(rng, t_lo, min(t_hi, most // H))
        if rng.random() < 0.3:
            T = max(t_lo, T // 64 * 64)
        B = _log_uniform(rng, 1, max(1, min(64, most // (H * T))))
    carry = kind in ("forward", "prefix") and rng.random() < 0.3
    return _case(kind, geometry, B, H, T, carry=carry)


def prepare(case, seed):
    dev = torch.device("cuda")
    dt = _DTYPES[case["dtype"]]
    B, H, T, dk, K, L = (case[k] for k in ("B", "H", "T", "dk", "K", "L"))
    N, R = B * H, 1 << K
    g = torch.Generator(device=dev).manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, device=dev, generator=g).to(dt)

    st = {"kind": case["kind"], "carry": None}
    if case["kind"] in ("step", "forward", "train"):
        with torch.random.fork_rng(devices=[]):
            torch.manual_seed(seed)
            ace = rk.BatchedACE(dk, K, L, 1)
        st["ace"] = ace.to(dev)
        st["K"], st["V"], st["Q"] = (normal(1, B, T, H, dk) for _ in range(3))
        if case["kind"] == "step" or case["carry"]:
            # what the conversation left behind: the state after a 100-token prompt
            with torch.no_grad():
                _, A, Bs = ace(*(normal(1, B, 100, H, dk) for _ in range(3)), return_state=True)
            st["carry"] = ops.pack_state(A, Bs)
        if case["kind"] == "train":
            for name in ("K", "V", "Q"):
                st[name].requires_grad_(True)
            st["dO"] = normal(1, B, T, H, dk)
        return st
    # probabilities-level calls: softmax rows of N(0,1) logits, as the sweep configuration has them
    st["pQ"], st["pK"] = (torch.softmax(torch.randn(N, T, L, R, device=dev, generator=g), -1).to(dt) for _ in range(2))
    st["V"] = normal(N, T, dk)
    if case["carry"]:
        p = torch.softmax(torch.randn(N, 500, L, R, device=dev, generator=g), -1)
        v = torch.randn(N, 500, dk, device=dev, generator=g)
        st["carry"] = ops.pack_state(p.sum(1), (p.reshape(N, 500, -1).transpose(1, 2) @ v).view(N, L, R, dk))
    if case["kind"] == "noncausal":
        for name in ("pQ", "pK", "V"):
            st[name].requires_grad_(True)
        st["dO"] = normal(N, T, dk)
    return st


def run(st):
    kind = st["kind"]
    if kind == "step":
        return st["ace"].step(st["K"], st["V"], st["Q"], st["carry"]), st["carry"]
    if kind == "forward":
        with torch.no_grad():
            if st["carry"] is None:
                return st["ace"](st["K"], st["V"], st["Q"])
            return st["ace"](st["K"], st["V"], st["Q"], carry_in=st["carry"], return_state=True)
    if kind == "train":
        out = st["ace"](st["K"], st["V"], st["Q"])
        return (out.detach(), *torch.autograd.grad(out, (st["K"], st["V"], st["Q"]), st["dO"]))
    if kind == "prefix":
        if st["carry"] is None:
            return ops.race_causal_prefix(st["pQ"], st["pK"], st["V"])
        return ops.race_causal_prefix(st["pQ"], st["pK"], st["V"], carry_in=st["carry"], return_state=True)
    out = ops.race_noncausal(st["pQ"], st["pK"], st["V"])
    return (out.detach(), *torch.autograd.grad(out, (st["pQ"], st["pK"], st["V"]), st["dO"]))


def work(case):
    """Each input read once, each output written once; the multiply-adds of the projections, of the state's sums and
    of the query against it (twice more of each for gradients)."""
    elt = 4 if case["dtype"] == "f32" else 2
    dk, S = case["dk"], case["L"] << case["K"]
    tokens = case["B"] * case["H"] * case["T"]
    state = case["B"] * case["H"] * S * (dk + 1) * 4
    project, sums = 4 * dk * case["L"] * case["K"], 4 * S * dk
    kind = case["kind"]
    if kind == "noncausal":     # pQ, pK, V, dO in; out and three gradients back
        return {"bytes": tokens * elt * (4 * S + 4 * dk), "flops": tokens * 3 * sums}
    if kind == "train":         # K, V, Q, dO in; out and three gradients back
        return {"bytes": tokens * elt * 8 * dk, "flops": tokens * 3 * (project + sums)}
    if kind == "prefix":
        nbytes, flops = tokens * elt * (2 * S + 2 * dk), tokens * sums
    else:
        nbytes, flops = tokens * elt * 4 * dk, tokens * (project + sums)
    return {"bytes": nbytes + (2 * state if kind == "step" or case["carry"] else 0), "flops": flops}


def tolerance(case):
    # fp32 results come from 16-bit limb products with fp32 accumulation and sums over up to 2^20 tokens; bf16 results
    # carry the rounding of bf16 probabilities and outputs.  Gradients of the first tokens are differences of terms
    # that nearly cancel, hence the wider bound on single values.
    if case["dtype"] == "f32":
        return {"rel": 3e-5, "max": 2e-3}
    return {"rel": 1e-2, "max": 0.4}
