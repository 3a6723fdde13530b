"""A cell that has become narrower than cutoff + skin is refused before anything is
written, in every call until it is wide again; a list that overflows after the forces
have been launched is grown and the call evaluated again.  Whatever came before, a call's
results are those of a model that has just been made (the same bits: the lists are
built from the same positions)."""

import pytest
import torch

from test_gpu_vlist_frozen import _batch, _into, _model

pytestmark = pytest.mark.gpu

# the single engine (FP32 pair arithmetic), the batched one for one system, and for two
CASES = [([1000], "mixed"), ([1000], "fp64"), ([1000, 800], "mixed")]


def _fresh(st, precision):
    return _into(_model(precision), st, None)


@pytest.mark.parametrize(("sizes", "precision"), CASES)
@pytest.mark.parametrize("unread", [False, True])
def test_a_narrow_cell_is_refused_with_the_buffers_untouched(sizes, precision, unread,
                                                             monkeypatch):
    from tsb import models

    if unread:
        monkeypatch.setattr(models.VerletListModel, "UNREAD_ATOMS", 0)
    st, model = _batch(sizes), _model(precision)
    wide, out = st.cell.clone(), _into(model, st, None)
    for a, b in zip(out, _fresh(st, precision), strict=True):
        assert torch.equal(a, b)
    x = st.positions.clone()
    for _ in range(2):
        st.cell = wide.clone()
        st.cell[0, 0, 0] *= 0.25  # 32 A: now below 8.5 + 1
        st.positions = x * (st.cell[0].diagonal() / wide[0].diagonal())
        for _ in range(3):
            n, ns = st.n_atoms, st.n_systems
            out = [torch.full(s, 7.0, dtype=st.dtype, device="cuda")
                   for s in ((ns,), (n, 3), (ns, 3, 3))]
            with pytest.raises(ValueError, match="cell width"):
                model.forward_into(st, energy=out[0], forces=out[1], stress=out[2])
            assert all(bool((t == 7.0).all()) for t in out)
        st.cell, st.positions = wide, x
        for a, b in zip(_into(model, st, None), _fresh(st, precision), strict=True):
            assert torch.equal(a, b)


@pytest.mark.parametrize(("sizes", "precision"), CASES)
@pytest.mark.parametrize("unread", [False, True])
def test_an_overflow_found_behind_the_launch(sizes, precision, unread, monkeypatch):
    from tsb import models

    if unread:
        monkeypatch.setattr(models.VerletListModel, "UNREAD_ATOMS", 0)
    st, model = _batch(sizes), _model(precision)
    _into(model, st, None)
    x, cell = st.positions.clone(), st.cell.clone()
    # the systems shrink by a third of their volume: the lists' estimate does not hold
    st.positions, st.cell = 0.87 * x, 0.87 * cell
    wide = bool((st.cell.diagonal(dim1=1, dim2=2) >= 9.5).all())
    assert wide
    for a, b in zip(_into(model, st, None), _fresh(st, precision), strict=True):
        assert torch.equal(a, b)
    st.positions, st.cell = x, cell
    for a, b in zip(_into(model, st, None), _fresh(st, precision), strict=True):
        assert torch.equal(a, b)
