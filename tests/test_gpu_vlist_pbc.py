"""Kept lists follow the periodic axes: the same positions and cell evaluated with other
flags, given by tensors that come and go or written in place, are those of the per-call
model.  Both engines decide pairs in FP64, so the pair sets are equal; forces in FP32
pair arithmetic differ by the rounding of ~100 terms (1e-5 of the largest is asked for,
a lost or a spurious image changes them by percents)."""

import pytest
import torch

from test_gpu_vlist_staged import _state

pytestmark = pytest.mark.gpu

FLAGS = [[True] * 3, [True, True, False], [False] * 3, [True] * 3, [False, True, True]]


def _close(got, want):
    for k in ("energy", "forces", "stress"):
        scale = float(want[k].abs().max())
        assert float((got[k] - want[k]).abs().max()) <= 1e-5 * scale, k


@pytest.mark.parametrize("sizes", [[900], [900, 1000]])  # the single engine and the batched
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("given", ["tensor", "in place", "host"])
def test_axes_switched_between_calls(sizes, precision, given):
    from tsb import models

    st = _state(sizes[:1], 3)
    if len(sizes) > 1:
        other = _state(sizes[1:], 4)
        for name in ("positions", "masses", "cell", "atomic_numbers"):
            setattr(st, name, torch.cat([getattr(st, name), getattr(other, name)]))
        st.system_idx = torch.cat([st.system_idx, other.system_idx + 1])
        st._n_systems = None
    st.positions = st.positions * 1.02  # (a little apart, so that no pair dominates)
    st.cell = st.cell * 1.02
    model = models.kob_andersen_model(compute_stress=True, device="cuda", precision=precision)
    kept = models.VerletListModel(model, skin=1.0)
    st.pbc = torch.tensor(FLAGS[0], device="cuda")
    for flags in FLAGS * 2:
        if given == "tensor":
            st.pbc = None
            st.pbc = torch.tensor(flags, device="cuda")
        elif given == "host":
            st.pbc = flags
        else:
            st.pbc.copy_(torch.tensor(flags))
        _close(kept(st), model(st))


def test_equal_axes_in_a_new_tensor_keep_the_lists():
    from tsb import models

    st = _state([900], 3)
    kept = models.VerletListModel(
        models.kob_andersen_model(compute_stress=True, device="cuda", precision="fp64"))
    for _ in range(4):
        st.pbc = torch.tensor([True] * 3, device="cuda")
        kept(st)
    assert kept.n_builds == 1
