"""The module's buffers on the host: what it notices about its prototypes, and that moving it works in every form."""
from __future__ import annotations

import copy

import torch


def _ace(**kw):
    import race_attention_kernel_b200 as rk
    return rk.BatchedACE(64, 4, 4, 1, **kw)


def test_prototypes_are_compared_by_value():
    ace = _ace()
    corners = ace.protos_T.clone()
    assert ace._protos_are_corners() and copy.deepcopy(ace)._protos_are_corners()
    assert ace.double()._protos_are_corners() and ace.bfloat16()._protos_are_corners()
    ace.float()
    for other in (corners * 2, corners.flip(0), corners[:2], corners.flatten()):
        ace.protos_T = other
        assert not ace._protos_are_corners()
        ace.protos_T = corners.clone()
        assert ace._protos_are_corners()
    ace.protos_T[0, 0] = 1.0
    assert not ace._protos_are_corners()
    ace.load_state_dict({**ace.state_dict(), "protos_T": corners})
    assert ace._protos_are_corners()
    ace.protos_T.data = corners * 3
    assert not ace._protos_are_corners()


def test_moving_a_module_that_has_no_values_to_compare():
    from torch._subclasses.fake_tensor import FakeTensorMode
    assert not _ace(device="meta").to_empty(device="cpu").to(torch.float64)._protos_are_corners()
    with FakeTensorMode():
        _ace().double().to("cpu")
    ace = _ace()
    ace.protos_T = None
    ace.double().to("cpu")


def test_moved_prototypes_are_not_read_back(monkeypatch):
    ace = _ace()
    monkeypatch.setattr(torch.Tensor, "tolist", None)
    assert ace.to(torch.float64)._protos_are_corners() and ace.to("cpu")._protos_are_corners()
    monkeypatch.undo()
    ace.protos_T = ace.protos_T * 2
    assert not ace.to(torch.float32)._protos_are_corners()
