"""Pair forces by tiles: directed pairs, systems left out, systems in any order."""

import numpy as np
import pytest
import torch

from test_gpu_window import DEV, SIZES, _batch
from tsb import models
from tsb.state import SimState

pytestmark = pytest.mark.gpu
LARGE = [*SIZES, *[300] * 200]  # 76,632 atoms: by tiles in every precision


def _state(x, cell, idx, z):
    return SimState(positions=x, masses=torch.ones_like(x[:, 0]), cell=cell.mT.contiguous(),
                    pbc=True, atomic_numbers=z, system_idx=idx)


def _model(kind, dtype, precision):
    kw = dict(device=DEV, dtype=dtype, precision=precision, compute_stress=True)
    if kind == "life":
        return models.ParticleLifeModel(sigma=4.0, epsilon=1.0, beta=0.4, cutoff=5.0, **kw)
    if kind == "lives":  # the force on a of b is not that on b of a
        a, b, s = [[1.0, -0.7], [0.4, 1.3]], [[0.3, 0.2], [0.4, 0.3]], [[4.0, 3.0], [4.5, 5.0]]
        return models.ParticleLifeMultiModel([1, 2], a, b, s, cutoff=5.0, **kw)
    return models.kob_andersen_model(2.2, **kw)


@pytest.mark.parametrize("kind", ["life", "lives"])
@pytest.mark.parametrize("dtype,precision", [(torch.float64, "fp64"), (torch.float64, "mixed"),
                                             (torch.float32, "mixed")])
def test_directed_pairs(kind, dtype, precision):
    """A system alone goes by warps.  Sums of ~20 terms in another order: below 1e-13 of
    the largest in FP64, 2^-24 per operation of them (some 30) in FP32."""
    x, cell, idx, z = _batch(LARGE, 0.04, True, dtype, 8)
    model = _model(kind, dtype, precision)
    full = model(_state(x, cell, idx, z))
    tol, lo = 1e-12 if precision == "fp64" else 2e-5, 0
    for k, n in enumerate(SIZES):
        one = model(_state(x[lo:lo + n], cell[k:k + 1], torch.zeros_like(idx[lo:lo + n]),
                           z[lo:lo + n]))
        for a, b in ((full["forces"][lo:lo + n], one["forces"]),
                     (full["stress"][k:k + 1], one["stress"])):
            assert float((a - b).abs().max()) <= tol * max(float(b.abs().max()), 1e-2), n
        lo += n


@pytest.mark.parametrize("dtype,precision", [(torch.float64, "fp64"), (torch.float32, "mixed")])
def test_systems_left_out_keep_their_entries(dtype, precision):
    x, cell, idx, z = _batch(LARGE, 0.04, True, dtype, 9)
    model, st = _model("ka", dtype, precision), _state(x, cell, idx, z)
    want = model(st)
    rng = np.random.default_rng(2)
    for on in (rng.random(len(LARGE)) < 0.5, np.zeros(len(LARGE), bool),
               np.arange(len(LARGE)) == len(SIZES) - 1):
        on = torch.as_tensor(on, device=DEV)
        e, f, s = (torch.full_like(want[k], 7.0) for k in ("energy", "forces", "stress"))
        model.forward_into(st, energy=e, forces=f, stress=s, sys_active=on.to(torch.uint8))
        for got, all_, rows in ((e, want["energy"], on), (f, want["forces"], on[idx]),
                                (s, want["stress"], on)):
            assert torch.equal(got[rows], all_[rows])
            assert bool((got[~rows] == 7.0).all())


@pytest.mark.parametrize("dtype,precision", [(torch.float64, "fp64"), (torch.float32, "mixed")])
def test_systems_in_any_order(dtype, precision):
    """The atoms of a system lie together; the systems need not ascend."""
    x, cell, idx, z = _batch(LARGE, 0.04, True, dtype, 10)
    model = _model("ka", dtype, precision)
    want = model(_state(x, cell, idx, z))
    number = torch.as_tensor(np.random.default_rng(1).permutation(len(LARGE)), device=DEV)
    got = model(_state(x, cell[torch.argsort(number)], number[idx], z))
    assert torch.equal(got["forces"], want["forces"])
    assert torch.equal(got["energy"][number], want["energy"])
    assert torch.equal(got["stress"][number], want["stress"])
