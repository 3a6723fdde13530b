"""Lists that cannot be made longer for want of memory keep the capacity that they have: a
later call must not be given a larger one than was allocated."""

import pytest
import torch

from tsb import models


class _Full(RuntimeError):
    pass


@pytest.fixture
def model(monkeypatch):
    m = models.VerletListModel(models.kob_andersen_model(device="cpu"), skin=1.0)
    m.cap, m.list = 40, torch.empty(400, dtype=torch.int32)
    m.s_cap, m.s_list = 50, torch.empty(500, dtype=torch.int32)
    monkeypatch.setattr(m, "_reset", lambda *_: None)

    def full(*_a, **_k):
        raise _Full

    monkeypatch.setattr(torch, "empty", full)
    return m


class _State:
    n_atoms, n_systems = 10, 1
    positions = torch.zeros((10, 3))


@pytest.mark.parametrize("grow", [lambda m: m._grow_lists(90, 10, 1, "cpu"),
                                  lambda m: m.grow(90, _State)])
def test_a_list_that_does_not_grow(model, grow):
    model._key = ("a batch",)
    with pytest.raises(_Full):
        grow(model)
    assert model.cap * 10 <= model.list.numel()
    assert model._key is None  # (its lists may be cut short)


def test_the_single_list_does_not_grow(model, monkeypatch):
    from tsb import _lib as L

    class Overflowed:
        def item(self):
            return 90

    state = type("S", (), {"n_atoms": 10, "device": torch.device("cpu"),
                           "cell": torch.eye(3)[None]})
    monkeypatch.setattr(L, "call", lambda *_: None)
    monkeypatch.setattr(L, "ptr", lambda _: None)
    monkeypatch.setattr(L, "stream_ptr", lambda _: None)
    model.s_counts = model.s_ref = model.s_wraps = None
    model.s_status, model.s_ws = Overflowed(), torch.zeros(1)
    with pytest.raises(_Full):
        model._s_build(state, torch.zeros((10, 3), dtype=torch.float64))
    assert model.s_cap * 10 <= model.s_list.numel() and not model._s_built


def test_a_new_batch_without_room_is_not_taken_for_the_old_one(model):
    model._key = ("an old batch",)
    model._seen, model._seen_pbc = (), None
    z = torch.ones(10, dtype=torch.int64)
    state = type("S", (), {"n_atoms": 10, "n_systems": 1, "system_idx": 0 * z,
                           "atomic_numbers": z, "pbc": torch.ones(3, dtype=torch.bool)})
    with pytest.raises(_Full):
        model._ensure(state, torch.zeros((10, 3)), 9.0 * torch.eye(3)[None])
    assert model._key is None and model.cap * 10 <= model.list.numel()
