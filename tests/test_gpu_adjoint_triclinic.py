"""One-block-per-system trajectories and sweeps in sheared cells, against the step-by-step
path.  Same pairs and formulas, other summation orders: a few FP64 roundings per step,
amplified over the steps, far below the 1e-10 of the largest value asked for here."""

import numpy as np
import pytest
import torch

from test_gpu_adjoint_blocks import DEV, _close, _problem, _same

pytestmark = pytest.mark.gpu
SHEARS = [[[1, 0, 0], [0.3, 1, 0], [-0.25, 0.2, 1]],   # lower triangular
          [[1, 0.3, -0.2], [0, 1, 0.35], [0, 0, 1]],   # upper
          [[1, 0.2, 0.1], [-0.15, 1.1, 0.25], [0.3, -0.1, 0.95]],
          [[0, 1, 0], [0, 0.2, 1], [1, 0, 0.1]]]       # axes in another order


def _sheared(sizes, steps, shear, pbc=True, **kw):
    """The problem with its cells sheared, the atoms with them, some cells away."""
    P, s, e, q, p = _problem(sizes, steps, **kw)
    m = torch.as_tensor(np.array(shear), device=DEV)
    shift = torch.as_tensor(np.random.default_rng(1).integers(-2, 3, q.shape).astype(float),
                            device=DEV)
    q = q @ m
    P.cell_row = (P.cell_row @ m).contiguous()
    P.pbc = torch.as_tensor(np.broadcast_to(pbc, tuple(P.pbc.shape)).astype(np.uint8),
                            device=DEV).contiguous()
    q = q + torch.einsum("ik,ikm->im", shift * P.pbc[P.system_idx], P.cell_row[P.system_idx])
    return P, s, e, q.contiguous(), p


@pytest.mark.parametrize("shear", SHEARS)
@pytest.mark.parametrize("sizes", [[128, 60], [200], [300]])  # four, two, one thread per atom
def test_sheared_cells(sizes, shear):
    _same(*_sheared(sizes, 12, shear))


@pytest.mark.parametrize("shear", SHEARS)
@pytest.mark.parametrize("pbc", [(True, True, False), (False, True, True), (True, False, False)])
def test_sheared_cells_with_open_axes(pbc, shear):
    _same(*_sheared([90, 150], 8, shear, pbc=pbc))


@pytest.mark.parametrize("shear", SHEARS[:3])
def test_lists_rebuilt_in_sheared_cells(shear):
    P, s, e, q, p = _sheared([100, 64], 30, shear)
    _same(P, s, e, q, 12.0 * p)  # (drifts of more than half the skin)


@pytest.mark.parametrize("wide", [False, True])
def test_a_plane_spacing_decides(wide):
    """Edges of 14 A, sheared so that the spacing of one pair of planes is just below or
    above cutoff + skin = 7 A: the narrow one goes the general way."""
    from tsb import adjoint

    c = 0.98 if wide else 1.02
    shear = [[1, 0, 0], [c * np.sqrt(3), 1, 0], [0, 0, 1]]  # |b_0| = sqrt(1 + 3 c^2) / 14
    P, s, e, q, p = _sheared([100], 8, shear, width=14.0)
    got = adjoint.loss_and_grad(s, e, q, p, P)
    assert ("_graphs" not in P.__dict__) == wide
    want = adjoint.loss_and_grad(s, e, q, p, P, use_graphs=False)
    for a, b in zip(got, want, strict=True):
        _close(a, b)
