"""One-block-per-system trajectories and adjoint sweeps against the step-by-step path
(``use_graphs=False``: per-call searches, one launch per piece).  Same pairs and
formulas, other summation orders: a few FP64 roundings per step, amplified over the
steps, far below the 1e-10 of the largest value asked for here."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _problem(sizes, n_steps, n_species=2, pbc=True, seed=0, width=None):
    from tsb import adjoint, workloads
    from tsb.state import SimState

    rng = np.random.default_rng(seed)
    pos, cell, idx = [], [], []
    for k, n in enumerate(sizes):
        length = max((n / 0.025) ** (1 / 3), 10.0) if width is None else width
        m = int(np.ceil(n ** (1 / 3)))
        at = np.sort(rng.permutation(m**3)[:n])
        g = (np.stack([at // (m * m), at // m % m, at % m], -1) + 0.5) / m
        pos.append(g * length + rng.normal(0, 0.05, (n, 3)) + 3 * length * (k % 2))
        cell.append(np.eye(3) * length)
        idx += [k] * n
    n = len(idx)
    t = lambda v: torch.as_tensor(v, device=DEV)  # noqa: E731
    st = SimState(positions=t(np.concatenate(pos)), masses=t(np.full(n, 39.948)),
                  cell=t(np.stack(cell)), pbc=pbc, system_idx=t(np.array(idx)),
                  atomic_numbers=t(rng.integers(1, n_species + 1, n)))
    P = adjoint.make_problem(st, n_steps, 0.002 * workloads.METAL_TIME, cutoff=6.0,
                             species_atomic_numbers=tuple(range(1, n_species + 1)))
    P.target = adjoint.histogram(st.positions, P)
    s, e = adjoint.argon_pair_params(n_species, perturb=0.05, seed=1)
    p = t(rng.normal(0, np.sqrt(39.948 * 60 * workloads.KB_EV), (n, 3)))
    return P, s, e, st.positions, p


def _close(a, b, rel=1e-10):
    scale = float(b.abs().max())
    assert float((a - b).abs().max()) <= rel * max(scale, 1e-30)


def _same(P, s, e, q, p):
    from tsb import adjoint

    got = adjoint.loss_and_grad(s, e, q, p, P)
    assert "_graphs" not in P.__dict__  # the blocks took it
    want = adjoint.loss_and_grad(s, e, q, p, P, use_graphs=False)
    for a, b in zip(got, want, strict=True):
        _close(a, b)


# four, two and one thread per atom, and the edges between them
@pytest.mark.parametrize("sizes", [[1, 2], [128, 3], [129], [256, 33], [257], [512]])
def test_block_sizes(sizes):
    _same(*_problem(sizes, 6))


@pytest.mark.parametrize("n_species", [1, 3, 4])
def test_species(n_species):
    _same(*_problem([60, 61], 5, n_species))


@pytest.mark.parametrize("pbc", [[True, True, False], [False, False, False]])
def test_open_axes(pbc):
    _same(*_problem([60, 40], 5, pbc=pbc))


def test_lists_are_rebuilt_and_segments_match(monkeypatch):
    """Fast atoms outrun the skin several times; sweeps over re-integrated segments
    give what the whole stored trajectory gives."""
    from tsb import adjoint

    P, s, e, q, p = _problem([64, 50], 60)
    p = 6.0 * p
    whole = adjoint.loss_and_grad(s, e, q, p, P)
    want = adjoint.loss_and_grad(s, e, q, p, P, use_graphs=False)
    # 60 steps at 2000 K: 1e-16 grows by the trajectory's own instability
    for a, b in zip(whole, want, strict=True):
        _close(a, b, 1e-8)
    monkeypatch.setattr(adjoint._Blocks, "TRAJ_BYTES", 0)
    P.checkpoint_every = 7
    for a, b in zip(adjoint.loss_and_grad(s, e, q, p, P), whole, strict=True):
        _close(a, b, 1e-8)
    qT, pT, ckpt = adjoint.integrate(q, p, adjoint.lj_table(s, e), P)
    qR, pR, ref = adjoint.integrate(q, p, adjoint.lj_table(s, e), P, use_graphs=False)
    _close(qT, qR, 1e-10)
    _close(pT, pR, 1e-8)
    assert sorted(ckpt) == sorted(ref)


def test_short_lists_grow(monkeypatch):
    from tsb import adjoint

    monkeypatch.setattr(adjoint._Blocks, "CAP", 3)
    args = _problem([70, 64], 4)
    _same(*args)
    assert args[0].__dict__["_block_cap"] > 3


def test_what_does_not_fit_takes_the_general_path():
    """A cell narrower than cutoff + skin, and a system beyond a block."""
    from tsb import adjoint

    for sizes, width in (([9], 6.5), ([adjoint.L.load().tsb_adj_block_max_atoms() + 1], None)):
        P, s, e, q, p = _problem(sizes, 3, width=width)
        got = adjoint.loss_and_grad(s, e, q, p, P)
        assert "_graphs" in P.__dict__
        want = adjoint.loss_and_grad(s, e, q, p, P, use_graphs=False)
        for a, b in zip(got, want, strict=True):
            _close(a, b)
