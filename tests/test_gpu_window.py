"""Cooperative search kernels (neighbour list and pair forces): one warp per atom for
small calls, one warp per tile of 32 atoms for large ones.  The same systems, alone and
in a large batch, take the two; lists must agree row by row, forces to rounding."""

import numpy as np
import pytest
import torch

from tsb import models, neighbors
from tsb.state import SimState

pytestmark = pytest.mark.gpu
DEV = "cuda"
WARP_MAX = 16384  # largest call of the one-warp-per-atom kernels


def _system(rng, n, density, triclinic, dtype):
    length = (n / density) ** (1 / 3)
    cell = np.diag(length * rng.uniform(0.8, 1.25, 3))
    if triclinic:
        cell = cell + rng.uniform(-0.25, 0.25, (3, 3)) * length
    m = int(np.ceil(n ** (1 / 3)))
    at = np.sort(rng.permutation(m**3)[:n])
    frac = (np.stack([at // (m * m), at // m % m, at % m], -1) + 0.5
            + rng.uniform(-0.2, 0.2, (n, 3))) / m
    frac += rng.integers(-2, 3, (n, 3)) * (rng.random((n, 1)) < 0.2)
    return (torch.as_tensor(frac @ cell, device=DEV).to(dtype),
            torch.as_tensor(cell, device=DEV).to(dtype))


def _batch(sizes, density, triclinic, dtype, seed):
    rng = np.random.default_rng(seed)
    got = [_system(rng, n, density, triclinic, dtype) for n in sizes]
    sys_idx = torch.repeat_interleave(torch.arange(len(sizes), device=DEV),
                                      torch.tensor(sizes, device=DEV))
    return (torch.cat([x for x, _ in got]), torch.stack([c for _, c in got]), sys_idx,
            torch.as_tensor(rng.integers(1, 3, sum(sizes)), device=DEV))


# sizes around 32 (a tile), one atom, cells smaller than the cutoff, and one system of
# more columns of bins than tiles are joined across
SIZES = [1, 2, 31, 32, 33, 64, 65, 300, 7, 4097, 12000]


@pytest.mark.parametrize("pbc", [(True, True, True), (True, False, True), (False,) * 3])
@pytest.mark.parametrize("flags", [{}, {"self_interaction": True}, {"half": True}])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_large_and_small_calls_list_the_same_rows(pbc, flags, dtype):
    x, cell, sys_idx, _ = _batch(SIZES, 0.04, True, dtype, 3)
    assert len(x) > WARP_MAX
    p = torch.tensor(pbc, device=DEV)
    m, s, sh = neighbors.torchsim_nl(x, cell, p, 5.0, sys_idx, **flags)
    assert m.is_contiguous()
    lo, row = 0, 0
    for k, n in enumerate(SIZES):
        one = torch.zeros(n, dtype=torch.int64, device=DEV)
        m1, _, sh1 = neighbors.torchsim_nl(x[lo:lo + n], cell[k:k + 1], p, 5.0, one, **flags)
        c = m1.shape[1]
        assert torch.equal(m[:, row:row + c], m1 + lo)
        assert torch.equal(sh[row:row + c], sh1)
        assert bool((s[row:row + c] == k).all())
        lo, row = lo + n, row + c
    assert row == m.shape[1]


@pytest.mark.parametrize("n", [WARP_MAX, WARP_MAX + 1])
def test_capacity_is_never_exceeded(n):
    from tsb import _lib as L

    x, cell, sys_idx, _ = _batch([n], 0.03, False, torch.float64, 5)
    pbc = torch.ones((1, 3), dtype=torch.uint8, device=DEV)
    ws = torch.empty(L.load().tsb_nl_workspace_size(n, 1), dtype=torch.uint8, device=DEV)
    want = neighbors.torchsim_nl(x, cell, pbc, 5.0, sys_idx)[0].shape[1]
    for cap in (want - 1, want):
        mapping = torch.full((2 * cap,), -7, dtype=torch.int64, device=DEV)
        sysmap = torch.full((cap,), -7, dtype=torch.int64, device=DEV)
        shifts = torch.full((cap, 3), -7.0, dtype=torch.float64, device=DEV)
        count = torch.zeros(1, dtype=torch.int64, device=DEV)
        L.call("tsb_nl_build_packed", L.ptr(x), L.ptr(cell), L.ptr(pbc), L.ptr(sys_idx), n, 1,
               L.F64, 5.0, 0, L.ptr(mapping), L.ptr(sysmap), L.ptr(shifts), cap, L.ptr(count),
               L.ptr(ws), ws.numel(), L.stream_ptr(x.device))
        assert int(count) == want
        assert bool((mapping == -7).all()) == (cap < want)
        assert bool((sysmap == -7).any()) == (cap < want)


def _forces(x, cell, sys_idx, z, kind, precision):
    kw = dict(device=DEV, dtype=x.dtype, precision=precision, compute_stress=True,
              per_atom_energies=True)
    model = {"lj": lambda: models.LennardJonesModel(2.6, 0.01, cutoff=6.0, **kw),
             "morse": lambda: models.MorseModel(2.8, 0.34, 1.36, cutoff=6.0, **kw),
             "soft": lambda: models.SoftSphereModel(5.0, 1.0, 2.5, **kw),
             "ka": lambda: models.kob_andersen_model(2.2, **kw)}[kind]()
    return model(SimState(positions=x, masses=torch.ones_like(x[:, 0]),
                          cell=cell.mT.contiguous(), pbc=True, atomic_numbers=z,
                          system_idx=sys_idx))


@pytest.mark.parametrize("kind", ["lj", "morse", "soft", "ka"])
@pytest.mark.parametrize("dtype,precision", [(torch.float64, "fp64"), (torch.float64, "mixed"),
                                             (torch.float32, "mixed")])
def test_large_and_small_calls_give_the_same_forces(kind, dtype, precision):
    """An atom's pairs are the same, so FP64 sums differ by their order alone (100 terms:
    below 1e-13 of the largest) and FP32 sums by 100 * 2^-24 of the terms' size."""
    sizes = SIZES + [300] * 200
    x, cell, sys_idx, z = _batch(sizes, 0.04, True, dtype, 8)
    assert len(x) > 65536  # also the larger limit of FP32 pair math with FP64 results
    full = _forces(x, cell, sys_idx, z, kind, precision)
    tol = 1e-12 if precision == "fp64" else 2e-5
    lo = 0
    for k, n in enumerate(sizes[:len(SIZES)]):
        one = _forces(x[lo:lo + n], cell[k:k + 1], torch.zeros_like(sys_idx[lo:lo + n]),
                      z[lo:lo + n], kind, precision)
        for name, a in (("forces", full["forces"][lo:lo + n]),
                        ("energies", full["energies"][lo:lo + n]),
                        ("energy", full["energy"][k:k + 1]), ("stress", full["stress"][k:k + 1])):
            b = one[name]
            # forces of one or two atoms cancel to rounding of the pair terms
            scale = max(float(b.abs().max()), 1e-2)
            assert float((a - b).abs().max()) <= tol * scale, (name, n)
        lo += n


def test_lost_atoms_do_not_touch_their_neighbours():
    """NaN coordinates fall into the bins of ordinary atoms: those keep their pairs."""
    for n in (3000, WARP_MAX + 2000):
        x, cell, sys_idx, _ = _batch([n], 0.03, True, torch.float64, 6)
        pbc = torch.ones(3, dtype=torch.bool, device=DEV)
        lost = torch.tensor([5, n // 2], device=DEV)
        m, _, sh = neighbors.torchsim_nl(x, cell, pbc, 5.0, sys_idx)
        keep = ~torch.isin(m[0], lost) & ~torch.isin(m[1], lost)
        y = x.clone()
        y[lost[0]] = float("nan")
        y[lost[1], 1] = float("nan")
        m2, _, sh2 = neighbors.torchsim_nl(y, cell, pbc, 5.0, sys_idx)
        # (an atom that moves to another bin changes only its own rows)
        assert torch.equal(m[:, keep], m2)
        assert torch.equal(sh[keep], sh2)
