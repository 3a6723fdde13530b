"""What does not fit a block is found out once, before anything is allocated where that can
be known, and the general path then answers alone.  Reference: the step-by-step path
(``use_graphs=False``); tolerance as in test_gpu_adjoint_blocks."""

import pytest
import torch

from test_gpu_adjoint_blocks import _close, _problem
from test_gpu_adjoint_sizes import _trajectory

pytestmark = pytest.mark.gpu
BLOCKS = {"tsb_adj_trajectory", "tsb_adj_sweep"}


@pytest.fixture
def launched(monkeypatch):
    """Names of the block kernels' calls, in order."""
    from tsb import _lib as L

    names, call = [], L.call
    monkeypatch.setattr(L, "call", lambda name, *a: (names.append(name) if name in BLOCKS
                                                     else None) or call(name, *a))
    return names


def _check(P, s, e, q, p):
    from tsb import adjoint

    got = adjoint.loss_and_grad(s, e, q, p, P)
    want = adjoint.loss_and_grad(s, e, q, p, P, use_graphs=False)
    for a, b in zip(got, want, strict=True):
        _close(a, b)


def test_a_narrow_cell_is_found_once(launched):
    args = _problem([9, 40], 3, width=6.5)
    _check(*args)
    assert len(launched) > 0
    launched.clear()
    _check(*args)
    assert launched == []


def test_too_many_atoms_are_known_beforehand(launched):
    from tsb import adjoint

    P, s, e, q, p = _problem([513], 3)
    _check(P, s, e, q, p)
    P.n_steps = 10**5  # 1.2 GB of positions
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    with pytest.raises(adjoint._NoBlocks):
        adjoint._Blocks.loss_and_grad(adjoint.lj_table(s, e), q, p, P)
    assert torch.cuda.max_memory_allocated() - before < 2**20 and launched == []


def test_lists_beyond_a_block_are_found_once(launched):
    P, s, e, q, p = _problem([512], 3)
    P.cutoff = 11.0  # ~180 neighbours within 12 A; a block holds ~165
    _check(P, s, e, q, p)
    assert launched == ["tsb_adj_trajectory", "tsb_adj_sweep"]
    launched.clear()
    _check(P, s, e, q, p)
    assert launched == []


def test_lists_that_fit_the_trajectory_alone(launched, monkeypatch):
    from tsb import _lib as L
    from tsb import adjoint

    P, s, e, q, p = _problem([300], 6)
    lib = L.load()
    sweep, alone = (lib.tsb_adj_block_max_neighbors(300, 2, k) for k in (1, 0))
    assert 0 < sweep < alone
    monkeypatch.setattr(adjoint._Blocks, "CAP", alone)
    _check(P, s, e, q, p)
    assert launched == ["tsb_adj_trajectory"]  # the general path's own trajectory
    monkeypatch.setattr(adjoint._Blocks, "CAP", sweep)
    P.__dict__.pop("_block_cap")
    launched.clear()
    _check(P, s, e, q, p)
    assert launched == ["tsb_adj_trajectory", "tsb_adj_sweep"]
    assert lib.tsb_adj_block_max_neighbors(513, 2, 1) == 0
    assert lib.tsb_adj_block_max_neighbors(300, 5, 1) == 0


def test_a_system_left_out_keeps_its_positions():
    P, s, e, q, p = _problem([30, 9, 28], 4)
    from tsb import adjoint

    full = _trajectory(P, adjoint.lj_table(s, e), q, p, 30)
    assert full[0] == 0
    P.cell_row = P.cell_row.clone()
    P.cell_row[1] *= 0.5  # narrower than cutoff + skin
    part = _trajectory(P, adjoint.lj_table(s, e), q, p, 30)
    assert part[0] == 1 << 30
    for a, b, start in ((part[1], full[1], q), (part[2], full[2], p)):
        assert torch.equal(a[30:39], start[30:39])
        assert torch.equal(a[:30], b[:30]) and torch.equal(a[39:], b[39:])
