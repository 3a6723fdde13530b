"""Batched Verlet-list forces read nothing of systems that take no part: a first call in
which every system is frozen leaves the buffers as they were, frozen systems beside
others change nothing, and systems may stand in any order.  A system's results are the
same bits whatever stands beside it."""

import pytest
import torch

from test_gpu_vlist_staged import _state

pytestmark = pytest.mark.gpu


def _batch(sizes, order=None):
    """The systems 0, 1, ... of these sizes, their atoms in the given order of systems."""
    order = list(range(len(sizes))) if order is None else order
    states = [_state([n], 10 + k) for k, n in enumerate(sizes)]
    st = _state([1], 0)
    for name in ("positions", "masses", "atomic_numbers"):
        setattr(st, name, torch.cat([getattr(states[k], name) for k in order]))
    st.cell = torch.cat([s.cell for s in states])
    st.system_idx = torch.cat([torch.full((sizes[k],), k, device="cuda") for k in order])
    st._n_systems = None
    return st


def _model(precision="mixed"):
    from tsb import models

    return models.VerletListModel(models.kob_andersen_model(
        compute_stress=True, device="cuda", precision=precision), skin=1.0)


def _into(model, st, active):
    n, ns = st.n_atoms, st.n_systems
    out = [torch.full(shape, 7.0, dtype=st.dtype, device="cuda")
           for shape in ((ns,), (n, 3), (ns, 3, 3))]
    flags = None if active is None else torch.tensor(active, dtype=torch.uint8, device="cuda")
    model.forward_into(st, energy=out[0], forces=out[1], stress=out[2], sys_active=flags)
    return out


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("filler", [0, 70_000])  # four lanes per slot, one lane
def test_frozen_systems(precision, filler):
    sizes = [300, 900, 64, 1500] + [700] * (filler // 700)
    st, model = _batch(sizes), _model(precision)
    for t in _into(model, st, [0] * len(sizes)):
        assert bool((t == 7.0).all())
    want = _into(_model(precision), st, None)
    active = [k in (1, 3) for k in range(len(sizes))]
    got = _into(model, st, active)
    on = torch.tensor(active, device="cuda")
    for a, b, mine in zip(got, want, (on, on[st.system_idx], on), strict=True):
        assert torch.equal(a[mine], b[mine]) and bool((a[~mine] == 7.0).all())
    for a, b in zip(_into(model, st, None), want, strict=True):
        assert torch.equal(a, b)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("sizes", [[64, 70, 65], [300, 64, 900], [1700, 1000, 1793]])
@pytest.mark.parametrize("filler", [0, 70_000])
def test_systems_in_any_order(precision, sizes, filler):
    sizes = sizes + [700] * (filler // 700)
    rest = list(range(3, len(sizes)))
    want = _into(_model(precision), _batch(sizes), None)
    for order in ([2, 0, 1], [1, 2, 0], [2, 1, 0]):
        got = _into(_model(precision), _batch(sizes, order + rest), None)
        assert torch.equal(got[0], want[0]) and torch.equal(got[2], want[2])
        starts = [sum(sizes[:k]) for k in range(len(sizes))]
        rows = torch.cat([torch.arange(starts[k], starts[k] + sizes[k]) for k in order + rest])
        assert torch.equal(got[1], want[1][rows.cuda()])
