"""Pair forces where the kernel changes: warps per atom against tiles, tiles of 16 against
tiles of 32 atoms, atoms with no pairs and with more than one chunk of them.

FP32 force sums keep the order of the search in tiles of either width, so a system's
forces are the same bits in both.  FP64 sums of ~100 terms differ by their order alone:
1e-12 of the largest component is asked for (100 * 1.1e-16 * a sum of terms up to ~30
times their total)."""

import numpy as np
import pytest
import torch

from oracle import pair as opair
from test_gpu_window import DEV, _batch, _forces, _system

pytestmark = pytest.mark.gpu


def _close(a, b, tol=1e-12):
    assert float((a - b).abs().max()) <= tol * max(float(b.abs().max()), 1e-2)


@pytest.mark.parametrize("kind", ["lj", "ka"])
@pytest.mark.parametrize("dtype,precision,first,more", [
    (torch.float32, "mixed", 70_000, 60_000), (torch.float64, "mixed", 70_000, 60_000),
    (torch.float64, "fp64", 70_000, 10_000)])
def test_tiles_of_16_and_of_32_atoms(kind, dtype, precision, first, more):
    sizes = [33, 300, 1, 17, 500, 64, 700] * (first // 1615 + 1)
    n, lo = sum(sizes), len(sizes)
    x, cell, idx, z = _batch(sizes + [400] * (more // 400), 0.04, True, dtype, 4)
    small = _forces(x[:n], cell[:lo], idx[:n], z[:n], kind, precision)
    large = _forces(x, cell, idx, z, kind, precision)
    if precision == "mixed":
        assert torch.equal(small["forces"], large["forces"][:n])
    _close(small["forces"], large["forces"][:n])
    _close(small["energy"], large["energy"][:lo])
    _close(small["stress"], large["stress"][:lo])


@pytest.mark.parametrize("kind", ["lj", "soft"])
@pytest.mark.parametrize("n", [24_576, 24_577])  # by warps, and (lj) by tiles
def test_one_large_system_in_fp64(kind, n):
    x, cell, idx, z = _batch([n], 0.04, False, torch.float64, 6)
    one = _forces(x, cell, idx, z, kind, "fp64")
    # beside seven single atoms the batch counts as one of small systems: by warps
    y, c, s, zz = _batch([1] * 7, 0.01, False, torch.float64, 7)
    both = _forces(torch.cat([x, y]), torch.cat([cell, c]), torch.cat([idx, s + 1]),
                   torch.cat([z, zz]), kind, "fp64")
    _close(one["forces"], both["forces"][:n])
    _close(one["energies"], both["energies"][:n])
    _close(one["stress"], both["stress"][:1])


@pytest.mark.parametrize("dtype,precision", [(torch.float32, "mixed"), (torch.float64, "mixed"),
                                             (torch.float64, "fp64")])
@pytest.mark.parametrize("stress", [False, True])
@pytest.mark.parametrize("n,density,cutoff", [
    (5, 1e-5, 5.0),        # no pairs at all
    (1, 0.04, 9.0),        # images of itself: spans of one atom, one partial sum
    (3, 0.04, 9.0), (40, 0.02, 7.0), (200, 0.04, 7.0),
    (150, 0.08, 9.0),      # ~244 pairs: two chunks
    (90, 0.08, 11.5),      # ~510 pairs
])
def test_few_and_many_pairs_against_the_oracle(dtype, precision, stress, n, density, cutoff):
    from tsb import models
    from tsb.state import SimState

    x, cell = _system(np.random.default_rng(n), n, density, True, dtype)
    model = models.LennardJonesModel(1.8, 0.05, cutoff=cutoff, device=DEV, dtype=dtype,
                                     precision=precision, compute_stress=stress,
                                     per_atom_energies=True)
    out = model(SimState(positions=x, masses=torch.ones_like(x[:, 0]), cell=cell.mT[None],
                         pbc=True, atomic_numbers=torch.ones(n, dtype=torch.int64, device=DEV)))
    want = opair.pair_forward(opair.LJ, opair.single_table(opair.LJ, 1.8, 0.05),
                              np.zeros(n, dtype=int), x.double().cpu().numpy(),
                              cell.double().cpu().numpy()[None], np.array([True] * 3),
                              np.zeros(n, dtype=np.int64), cutoff, per_atom=True)
    # FP32: 2^-24 per operation, ~20 of them in a term with its powers, on terms whose
    # sum of magnitudes is up to a few hundred times a component that cancels: 1e-4 of
    # the largest; FP64 the same with 2^-53
    tol = 1e-4 if precision == "mixed" else 1e-11
    for k in ("forces", "energies", "energy") + (("stress",) if stress else ()):
        w = want[k]
        scale = max(np.abs(w).max(), 1e-6 if n > 1 else 1e-2)
        assert np.abs(out[k].double().cpu().numpy() - w).max() <= tol * scale, k
