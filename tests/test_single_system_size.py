"""The largest system of a call of one system is the call: nothing is counted or read."""

import torch

from tsb import _lib as L


def test_one_system_is_not_counted(monkeypatch):
    idx = torch.zeros(70, dtype=torch.int64)
    two = torch.tensor([0] * 30 + [1] * 40)
    assert L.max_system_atoms(two, 2) == 40

    def count(*_a, **_k):
        raise AssertionError("counted")

    monkeypatch.setattr(torch, "bincount", count)
    assert L.max_system_atoms(idx, 1) == 70
    assert L.max_system_atoms(idx[:0], 1) == 0
