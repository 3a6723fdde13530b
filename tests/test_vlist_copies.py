"""A VerletListModel that has been called can be copied and pickled: nothing of the copy
is tied to the process or to page-locked memory that it does not have."""

import copy
import pickle

import pytest
import torch


def _copies(model):
    return [copy.deepcopy(model), copy.copy(model), pickle.loads(pickle.dumps(model))]


def test_the_host_buffer_stays_behind():
    from tsb import models

    model = models.VerletListModel(models.kob_andersen_model(device="cpu"), skin=1.2)
    for buffer in (None, torch.zeros(2, dtype=torch.int32)):
        model._flags_host = buffer  # (what a call leaves, page-locked there)
        for other in _copies(model):
            assert other._flags_host is None and other.skin == 1.2
        assert model._flags_host is buffer


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [[900], [300, 500]])  # the single engine and the batched
@pytest.mark.parametrize("unread", [False, True])
def test_copies_of_a_called_model(sizes, unread, monkeypatch):
    from test_gpu_vlist_frozen import _batch
    from tsb import models

    if unread:
        monkeypatch.setattr(models.VerletListModel, "UNREAD_ATOMS", 0)
    st = _batch(sizes)
    model = models.VerletListModel(
        models.kob_andersen_model(compute_stress=True, device="cuda"), skin=1.0)
    want = {}
    for _ in range(3):  # (a first call, and ones that read the flags late)
        want = {k: v.clone() for k, v in model(st).items()}
        for other in _copies(model):
            for _ in range(2):
                got = other(st)
                assert all(torch.equal(got[k], want[k]) for k in want)
                assert other._flags_host is None or other._flags_host.is_pinned()
            st2 = _batch(sizes)
            assert all(torch.equal(v, want[k]) for k, v in other(st2).items())
