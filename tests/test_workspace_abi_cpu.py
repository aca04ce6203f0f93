"""Workspaces smaller than the library asks for are refused before anything is launched, also where the kernels of the one
call would need less."""
from __future__ import annotations

import ctypes

import pytest

from race_attention_kernel_b200 import _lib

P = ctypes.c_void_p(1 << 20)      # never dereferenced
TOO_SMALL = -4


@pytest.mark.parametrize("N,T", [(400, 128), (2, 20000)])
def test_noncausal_forward(N, T):
    """With one tile per stream its totals are the state, and no kernel needs a workspace."""
    L, sh = _lib.lib(), _lib.RaceShape(N, T, 4, 16, 64, 0, 1e-6, 0)
    assert L.race_b200_noncausal_fwd(P, P, P, P, P, P, 16, ctypes.byref(sh), None) == TOO_SMALL


@pytest.mark.parametrize("L_,R,dk", [(4, 16, 64), (8, 64, 128)])
def test_bf16_forward_without_a_state(L_, R, dk):
    """Outputs alone take longer tiles than the ones the workspace is sized for."""
    L, sh = _lib.lib(), _lib.RaceShape(64, 8192, L_, R, dk, 1, 1e-6, 0)
    need = L.race_b200_causal_workspace_bytes(ctypes.byref(sh), 0, 0)
    assert L.race_b200_causal_fwd(P, P, P, P, None, None, P, need - 1, ctypes.byref(sh), 0, 0, None, None) == TOO_SMALL
