"""Block trajectories take the systems' sizes from the batch, not from what they are told:
a system beyond the size given is reported and left out, and nothing else changes.
The general path (``use_graphs=False``) is the reference; tolerances as in
test_gpu_adjoint_blocks (FP64 sums in another order over a few steps)."""

import pytest
import torch

from test_gpu_adjoint_blocks import DEV, _close, _problem

pytestmark = pytest.mark.gpu


def _trajectory(P, table, q, p, max_system_atoms, cap=200, steps=4):
    from tsb import _lib as L

    ws = L.Workspace.get(q.device, L.load().tsb_adj_block_workspace_size(P.n_systems))
    inv_m = (1.0 / P.masses).contiguous()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    qT, pT = torch.zeros_like(q), torch.zeros_like(p)
    traj = torch.zeros((steps, *q.shape), dtype=q.dtype, device=DEV)
    system = (L.ptr(table), P.n_species, L.ptr(P.species), L.ptr(P.cell_row), L.ptr(P.pbc),
              L.ptr(P.system_idx), P.n_atoms, P.n_systems, max_system_atoms, P.cutoff, 1.0, cap,
              L.ptr(inv_m))
    end = (L.ptr(status), L.ptr(ws), ws.numel(), L.stream_ptr(q.device))
    L.call("tsb_adj_trajectory", *system, L.ptr(q), L.ptr(p), P.dt, steps, 1, L.ptr(qT),
           L.ptr(pT), None, None, L.ptr(traj), *end)
    lam_q, lam_p = q.sin(), torch.zeros_like(q)
    grad = torch.zeros((P.n_systems, P.n_species, P.n_species, 2), dtype=q.dtype, device=DEV)
    L.call("tsb_adj_sweep", *system, L.ptr(traj), P.dt, steps, 1, L.ptr(lam_q), L.ptr(lam_p),
           L.ptr(grad), *end)
    return int(status.item()), qT, pT, traj, lam_q, lam_p, grad


# the middle system is one atom, and many, beyond what the call says: with four, two and
# one threads per atom
@pytest.mark.parametrize(("sizes", "said"), [([24, 26, 10], 25), ([32, 60, 31], 32),
                                             ([130, 200, 130], 140), ([260, 300, 3], 299)])
def test_an_understated_size_leaves_the_system_out(sizes, said):
    from tsb import adjoint

    P, s, e, q, p = _problem(sizes, 4)
    table, lo, hi = adjoint.lj_table(s, e), sizes[0], sizes[0] + sizes[1]
    full = _trajectory(P, table, q, p, max(sizes))
    part = _trajectory(P, table, q, p, said)
    assert full[0] == 0 and part[0] == 1 << 30
    for a, b in zip(part[1:], full[1:], strict=True):
        per_atom = a.shape[-2] == q.shape[0]
        first, last = (slice(0, lo), slice(hi, None)) if per_atom else (slice(0, 1),
                                                                        slice(2, None))
        a, b = (t if t.ndim != 3 or not per_atom else t.transpose(0, 1) for t in (a, b))
        assert torch.equal(a[first], b[first]) and torch.equal(a[last], b[last])


def test_problems_of_other_sizes_in_turn():
    from tsb import adjoint

    for sizes in ([25, 25, 25, 25], [10, 30, 30, 30], [40, 20, 20, 20]) * 3:
        args = _problem(sizes, 5, seed=len(sizes))
        P, s, e, q, p = args
        got = adjoint.loss_and_grad(s, e, q, p, P)
        want = adjoint.loss_and_grad(s, e, q, p, P, use_graphs=False)
        for a, b in zip(got, want, strict=True):
            _close(a, b)
        del P, args, s, e, q, p, got, want
