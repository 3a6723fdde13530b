"""Neighbour lists where the kernel changes: one warp per atom up to 28,672 atoms of large
systems and 49,152 of small ones, tiles of 32 atoms beyond.  Rows are the same in both,
in the same order, bit for bit."""

import numpy as np
import pytest
import torch

from test_gpu_window import DEV, SIZES, _batch
from tsb import _lib as L
from tsb import neighbors

pytestmark = pytest.mark.gpu
LARGE, SMALL = 28672, 49152  # largest calls by warps: large systems, small ones
FLAGS = [{}, {"self_interaction": True}, {"half": True}]


def _rows(x, cell, pbc, idx, flags):
    """(mapping, system mapping, shifts) of a call."""
    got = neighbors.torchsim_nl(x, cell, torch.tensor(pbc, device=DEV), 5.0, idx, **flags)
    assert got[0].is_contiguous()
    return got


def _same_as_alone(x, cell, pbc, idx, flags, check):
    m, s, sh = _rows(x, cell, pbc, idx, flags)
    lo, row = 0, 0
    order, counts = torch.unique_consecutive(idx, return_counts=True)
    for k, (system, n) in enumerate(zip(order.tolist(), counts.tolist(), strict=True)):
        if k < check or k == len(order) - 1:
            m1, _, sh1 = _rows(x[lo:lo + n], cell[system:system + 1], pbc,
                               torch.zeros(n, dtype=torch.int64, device=DEV), flags)
            c = m1.shape[1]
            assert torch.equal(m[:, row:row + c], m1 + lo)
            assert torch.equal(sh[row:row + c], sh1)
            assert bool((s[row:row + c] == system).all())
        lo += n
        row = int(torch.searchsorted(m[0].contiguous(), torch.tensor(lo, device=DEV)))
    assert row == m.shape[1]


@pytest.mark.parametrize("pbc", [(True, True, True), (True, False, True), (False,) * 3])
@pytest.mark.parametrize("flags", FLAGS)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_tiles_list_the_rows_of_each_system_alone(pbc, flags, dtype):
    x, cell, idx, _ = _batch([*SIZES, *[410] * 80], 0.04, True, dtype, 3)
    assert len(x) > SMALL
    _same_as_alone(x, cell, pbc, idx, flags, len(SIZES))


@pytest.mark.parametrize("flags", FLAGS)
@pytest.mark.parametrize("n", [SMALL, SMALL + 1])
def test_small_systems_on_either_side_of_the_limit(n, flags):
    x, cell, idx, _ = _batch([*SIZES, *[300] * 107, n - sum(SIZES) - 32100], 0.04, True,
                             torch.float64, 4)
    assert len(x) == n
    _same_as_alone(x, cell, (True,) * 3, idx, flags, len(SIZES))


@pytest.mark.parametrize("flags", FLAGS)
@pytest.mark.parametrize("n", [LARGE, LARGE + 1])
def test_one_large_system_on_either_side_of_the_limit(n, flags):
    x, cell, idx, _ = _batch([n], 0.04, True, torch.float64, 5)
    m, _, sh = _rows(x, cell, (True,) * 3, idx, flags)
    # beside seven single atoms, with no pairs, the call counts as one of small systems
    y, c, s, _ = _batch([1] * 7, 1e-4, False, torch.float64, 6)
    m1, _, sh1 = _rows(torch.cat([x, y]), torch.cat([cell, c]), (True,) * 3,
                       torch.cat([idx, s + 1]), flags)
    p = m.shape[1]
    assert torch.equal(m1[:, :p], m) and torch.equal(sh1[:p], sh)
    assert p == int((m1[0] < n).sum())


def test_tiles_of_systems_in_any_order():
    """The atoms of a system lie together; the systems need not ascend."""
    sizes = [*SIZES, *[410] * 80]
    x, cell, idx, _ = _batch(sizes, 0.04, True, torch.float64, 7)
    number = torch.as_tensor(np.random.default_rng(1).permutation(len(sizes)), device=DEV)
    back = torch.argsort(number)
    _same_as_alone(x, cell[back], (True,) * 3, number[idx], {}, len(SIZES))


@pytest.mark.parametrize("less", [1, 0])
def test_capacity_of_a_call_of_tiles(less):
    n = LARGE + 1
    x, cell, idx, _ = _batch([n], 0.03, False, torch.float64, 5)
    pbc = torch.ones((1, 3), dtype=torch.uint8, device=DEV)
    ws = torch.empty(L.load().tsb_nl_workspace_size(n, 1), dtype=torch.uint8, device=DEV)
    want = neighbors.torchsim_nl(x, cell, pbc, 5.0, idx)[0].shape[1]
    cap = want - less
    mapping = torch.full((2 * cap,), -7, dtype=torch.int64, device=DEV)
    sysmap = torch.full((cap,), -7, dtype=torch.int64, device=DEV)
    shifts = torch.full((cap, 3), -7.0, dtype=torch.float64, device=DEV)
    count = torch.zeros(1, dtype=torch.int64, device=DEV)
    L.call("tsb_nl_build_packed", L.ptr(x), L.ptr(cell), L.ptr(pbc), L.ptr(idx), n, 1, L.F64,
           5.0, 0, L.ptr(mapping), L.ptr(sysmap), L.ptr(shifts), cap, L.ptr(count), L.ptr(ws),
           ws.numel(), L.stream_ptr(x.device))
    assert int(count) == want
    assert bool((mapping == -7).all()) == bool(less)
    assert bool((sysmap == -7).any()) == bool(less)


def test_lost_atoms_in_tiles():
    """NaN coordinates fall into the bins of ordinary atoms: those keep their pairs."""
    n = LARGE + 2000
    x, cell, idx, _ = _batch([n], 0.03, True, torch.float64, 6)
    m, _, sh = _rows(x, cell, (True,) * 3, idx, {})
    lost = torch.tensor([5, n // 2], device=DEV)
    keep = ~torch.isin(m[0], lost) & ~torch.isin(m[1], lost)
    x[lost[0]] = float("nan")
    x[lost[1], 1] = float("nan")
    m2, _, sh2 = _rows(x, cell, (True,) * 3, idx, {})
    assert torch.equal(m[:, keep], m2)
    assert torch.equal(sh[keep], sh2)
