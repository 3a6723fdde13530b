"""The single-system forces need no per-atom energy and virial buffers."""

import pytest
import torch

from test_gpu_vlist_frozen import _batch, _model

pytestmark = pytest.mark.gpu


def test_forces_without_scratch():
    from tsb import _lib as L

    st, model = _batch([900]), _model()
    want = model(st)
    assert not hasattr(model, "s_e_atom") and not hasattr(model, "s_vir_atom")
    out = [torch.empty_like(want[k]) for k in ("energy", "forces", "stress")]
    m, cell = model.model, st.cell[0].mT.contiguous()
    L.call("tsb_verlet_forces", m.kind, L.ptr(m.table), m.n_species, L.ptr(model.s_list),
           L.ptr(model.s_counts), st.n_atoms, L.ptr(cell), L.F64, m.cutoff,
           L.OUT_FORCES | L.OUT_STRESS, *(L.ptr(t) for t in out), None, None,
           L.ptr(model.s_ws), model.s_ws.numel(), L.stream_ptr(st.device))
    for t, k in zip(out, ("energy", "forces", "stress"), strict=True):
        assert torch.equal(t, want[k])
