"""Single-system Verlet lists on FP32 positions: gathered as given or in the frame."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = a.double(), b.double()
    return float((a - b).abs().max() / b.abs().max())


@pytest.mark.parametrize("n_cells,images", [(3, 0), (3, 1), (3, 5), (7, 0), (7, 1), (7, 40)])
def test_fp32_positions_as_given_and_in_the_frame_agree(n_cells, images):
    """FP32 positions are gathered as they are while the shifts between them stay
    within one cell, else mapped into the build's frame.  Coordinates and cell are
    multiples of 2^-12, so moving atoms by lattice vectors is exact and both forms see
    the same displacements up to FP64 rounding: FP32 results agree within 1e-6 of the
    largest (a few of their own last places)."""
    from tsb import models
    from tsb.state import SimState

    rng = np.random.default_rng(n_cells)
    a = 5.25
    length = n_cells * a
    g = np.stack(np.meshgrid(*[np.arange(n_cells)] * 3, indexing="ij"), -1).reshape(-1, 3)
    basis = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    x = ((g[:, None] + basis).reshape(-1, 3) * a + rng.normal(0, 0.1, (4 * len(g), 3)))
    x = np.round(x * 4096) / 4096
    moved = x + length * rng.integers(-images, images + 1, x.shape)
    t = lambda v, d=torch.float32: torch.as_tensor(v, dtype=d, device="cuda")  # noqa: E731
    z = torch.full((len(x),), 18, device="cuda")

    def run(pos, dtype):
        base = models.LennardJonesModel(3.405, 0.0104, cutoff=8.5, compute_stress=True,
                                        dtype=dtype, device="cuda")
        vm = models.VerletListModel(base, skin=1.0)
        st = SimState(positions=t(pos, dtype), masses=t(np.ones(len(x)), dtype),
                      cell=t(np.eye(3) * length, dtype)[None], pbc=True, atomic_numbers=z)
        first = vm(st)
        st.positions = st.positions + 0.25
        return first, vm(st)

    for a1, b1 in zip(run(x, torch.float32), run(moved, torch.float32), strict=True):
        for name in ("energy", "forces", "stress"):
            assert _rel(b1[name], a1[name]) <= 1e-6, name
    # and FP64 positions, always in the frame
    for a1, b1 in zip(run(moved, torch.float32), run(moved, torch.float64), strict=True):
        assert _rel(a1["forces"], b1["forces"]) <= 1e-6
