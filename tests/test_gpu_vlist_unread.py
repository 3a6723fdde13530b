"""Lists are rebuilt unread (without waiting for the check) only where that touches no
more than the marked systems: no system above the size that is binned one block each."""

import pytest
import torch

from test_gpu_vlist_frozen import _batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(("sizes", "unread"), [([4096, 64], True), ([4097, 64], False),
                                               ([300, 500], True), ([9000], False)])
def test_what_is_rebuilt_unread(sizes, unread, monkeypatch):
    from tsb import _lib as L
    from tsb import models

    limit = models.VerletListModel.UNREAD_ATOMS
    assert sum(sizes) < limit
    monkeypatch.setattr(models.VerletListModel, "UNREAD_ATOMS", 0)
    st = _batch(sizes)
    pair = models.kob_andersen_model(compute_stress=True, device="cuda", precision="fp64")
    model, names, call = models.VerletListModel(pair, skin=1.0), [], L.call
    want = {k: v.clone() for k, v in model(st).items()}
    monkeypatch.setattr(L, "call", lambda name, *a: names.append(name) or call(name, *a))
    got = model(st)
    assert ("tsb_vlist_build_pairs" in names) is unread
    assert all(torch.equal(got[k], want[k]) for k in want) and model.n_builds == 1
    # atoms that move are listed anew either way
    st.positions = st.positions + 0.7 * torch.sin(st.positions)
    names.clear()
    got, want = model(st), models.VerletListModel(pair, skin=1.0)(st)
    assert "tsb_vlist_build_pairs" in names and model.n_builds == 2
    assert all(torch.equal(got[k], want[k]) for k in want)
