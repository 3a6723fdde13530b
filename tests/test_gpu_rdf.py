"""Pair-distance histogram and its gradient (one warp per atom) against plain FP64
tensor operations over the package's neighbour list.  ~100 positive terms per bin and
exp within 1 ulp: 1e-12 of the largest value."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# bins below, at and above the shared-memory limit of 128, odd ones among them; a
# window wider than 16 bins; one atom; cells of one and of several bins
@pytest.mark.parametrize("n_bins,width", [(1, 0.5), (17, 0.3), (64, 0.05), (128, 0.2),
                                          (129, 0.05), (300, 0.02)])
def test_histogram_and_gradient(n_bins, width):
    from tsb import adjoint, neighbors, workloads
    from tsb.state import state_from_arrays

    d = workloads.argon_species_batch(3, (3, 2, 1), seed=2, jitter=0.3)
    one = workloads.argon_species_batch(1, (2, 2, 2), seed=1, jitter=0.3)
    for k in ("positions", "masses", "atomic_numbers"):
        d[k] = np.concatenate([d[k], one[k][:1]])
    d["cell"] = np.concatenate([d["cell"], 3 * one["cell"]])
    d["system_idx"] = np.concatenate([d["system_idx"], [3]])
    st = state_from_arrays(d, device="cuda")
    P = adjoint.make_problem(st, 1, 1.0)
    P.n_bins, P.width, P.r_max = n_bins, width, 8.0
    q = st.positions.contiguous()
    m, s, sh = neighbors.torchsim_nl(q, P.cell_row, P.pbc, P.r_max, st.system_idx)
    dr = q[m[1]] + torch.einsum("pi,pij->pj", sh, P.cell_row[s]) - q[m[0]]
    r = dr.norm(dim=1)
    c = (torch.arange(n_bins, device="cuda", dtype=torch.float64) + 0.5) * (P.r_max / n_bins)
    e = torch.exp(-((r[:, None] - c) ** 2) / (2 * width**2))
    want = torch.zeros((4, n_bins), dtype=torch.float64, device="cuda").index_add_(0, s, 0.5 * e)
    got = adjoint.histogram(q, P)
    assert float((got - want).abs().max()) <= 1e-12 * float(want.abs().max())
    g = torch.Generator(device="cuda").manual_seed(3)
    w = torch.randn((4, n_bins), dtype=torch.float64, device="cuda", generator=g)
    dl = (w[s] * e * -(r[:, None] - c) / width**2).sum(1)
    grad = torch.zeros_like(q).index_add_(0, m[0], -dr * (dl / r)[:, None])
    err = (adjoint._hist_grad(q, w, P) - grad).abs().max()
    # the sum over bins of terms of either sign
    terms = (w[s].abs() * e * (r[:, None] - c).abs() / width**2).sum(1).max()
    assert float(err) <= 1e-12 * max(float(terms), 1e-30) * 100
