"""Systems whose atoms lie together, numbered in any order: dilute ones fill all the bins
that they may have (2 per atom), so the bins of two systems must not touch."""

import numpy as np
import pytest
import torch

from tsb import _lib as L
from tsb import models, neighbors
from tsb.state import SimState

DEV = "cuda"
N, LENGTH, CUTOFF = 4, 20.0, 3.0  # 2 x 2 x 2 bins for 4 atoms


def _batch(systems, order, seed=0):
    """(positions, cells by number, system_idx) of boxes of two pairs of near atoms."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, LENGTH, (systems, 2, 1, 3)) + np.concatenate(
        [np.zeros((systems, 2, 1, 3)), rng.uniform(0.6, 1.4, (systems, 2, 1, 3))], 2)
    cells = LENGTH * np.eye(3) * rng.uniform(1.0, 1.05, (systems, 1, 1))
    cells[order] = cells.copy()
    return (torch.as_tensor(x.reshape(-1, 3), device=DEV), torch.as_tensor(cells, device=DEV),
            torch.as_tensor(np.repeat(order, N), device=DEV))


def _orders(systems):
    yield np.arange(systems)[::-1].copy()
    for seed in range(3):
        yield np.random.default_rng(seed).permutation(systems)


@pytest.mark.gpu
@pytest.mark.parametrize("systems", [2, 5, 60, 1000])
@pytest.mark.parametrize("pbc", [True, False])
def test_neighbour_list(systems, pbc):
    p = torch.tensor([pbc] * 3, device=DEV)
    up = np.arange(systems)
    x, cell, idx = _batch(systems, up)
    m, _, sh = neighbors.torchsim_nl(x, cell, p, CUTOFF, idx)
    assert m.shape[1] >= 4 * systems  # the two pairs, from either end
    for order in _orders(systems):
        x1, cell1, idx1 = _batch(systems, order)
        assert torch.equal(x1, x) and torch.equal(cell1[idx1], cell[idx])
        m1, s1, sh1 = neighbors.torchsim_nl(x1, cell1, p, CUTOFF, idx1)
        assert torch.equal(m1, m) and torch.equal(sh1, sh) and torch.equal(s1, idx1[m1[0]])


@pytest.mark.gpu
@pytest.mark.parametrize("systems", [5, 60, 1000])
@pytest.mark.parametrize("lists", [False, True])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_forces(systems, lists, precision):
    out = []
    for order in [np.arange(systems), *_orders(systems)]:
        x, cell, idx = _batch(systems, order)
        model = models.LennardJonesModel(1.0, 0.1, cutoff=CUTOFF, device=DEV,
                                         precision=precision, compute_stress=True)
        if lists:
            model = models.VerletListModel(model, skin=0.5)
        st = SimState(positions=x, masses=torch.ones_like(x[:, 0]), cell=cell.mT.contiguous(),
                      pbc=True, atomic_numbers=torch.ones_like(idx), system_idx=idx)
        got = model(st)
        first = idx[::N]
        out.append((got["forces"], got["energy"][first], got["stress"][first]))
    assert bool((out[0][0] != 0).all())
    for o in out[1:]:
        assert all(torch.equal(a, b) for a, b in zip(o, out[0], strict=True))


def test_the_lists_size_hint():
    up = torch.repeat_interleave(torch.arange(3), torch.tensor([5, 5000, 20]))
    assert L.list_size_hint(up, 3, 5000) == 5000
    assert L.list_size_hint(2 - up, 3, 5000) == 4096
    assert L.list_size_hint(2 - up, 3, 900) == 900
    assert L.list_size_hint(torch.zeros(5000, dtype=torch.int64), 1, 5000) == 5000


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("filler", [0, 70_000])
def test_lists_of_large_systems(precision, filler):
    """(the batch-wide bins against those of one block per system: the same bits)"""
    from test_gpu_vlist_frozen import _batch as batch
    from test_gpu_vlist_frozen import _into, _model

    sizes = [300, 4500, 900] + [700] * (filler // 700)
    rest = list(range(3, len(sizes)))
    starts = [sum(sizes[:k]) for k in range(len(sizes))]
    st, model = batch(sizes), _model(precision)
    for order in ([2, 0, 1], [1, 0, 2], [2, 1, 0]):
        rows = torch.cat([torch.arange(starts[k], starts[k] + sizes[k])
                          for k in order + rest]).cuda()
        other, again = batch(sizes, order + rest), _model(precision)
        st.positions[:] = batch(sizes).positions
        for _ in range(3):
            want, got = _into(model, st, None), _into(again, other, None)
            assert torch.equal(got[0], want[0]) and torch.equal(got[2], want[2])
            assert torch.equal(got[1], want[1][rows])
            st.positions[:300] += 0.7  # (one system's lists expire)
            other.positions[:] = st.positions[rows]
