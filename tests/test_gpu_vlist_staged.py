"""Batched Verlet-list forces with the neighbours' positions staged in shared memory
(blocks whose systems fit 1792 slots) and gathered from global memory (others), one and
four lanes per slot.  Both read the same values and sum them in the same order, so a
system's results are equal bit for bit, whatever its neighbours in the batch."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _state(sizes, seed):
    from tsb.state import SimState

    rng = np.random.default_rng(seed)
    pos, cell, z = [], [], []
    for n in sizes:
        length = (n * 3.4**3 / 1.2) ** (1 / 3)
        m = int(np.ceil(n ** (1 / 3)))
        at = np.sort(rng.permutation(m**3)[:n])
        g = np.stack([at // (m * m), at // m % m, at % m], -1) + 0.5
        pos.append((g + rng.uniform(-0.1, 0.1, (n, 3))) / m * length)
        cell.append(np.eye(3) * length)
        z.append(1 + (rng.random(n) < 0.2))
    t = lambda v: torch.as_tensor(v, device="cuda")  # noqa: E731
    n = sum(sizes)
    return SimState(positions=t(np.concatenate(pos)), masses=torch.ones(n, device="cuda").double(),
                    cell=t(np.stack(cell)), pbc=True, atomic_numbers=t(np.concatenate(z)),
                    system_idx=t(np.repeat(np.arange(len(sizes)), sizes)))


# the system under test, and what shares its blocks: systems that still fit the
# staged range, and ones that do not
@pytest.mark.parametrize("n", [64, 70, 892, 893, 1000, 1791, 1792, 1793])
@pytest.mark.parametrize("filler", [0, 70_000])  # four lanes per slot, one lane
def test_staged_and_gathered_positions(n, filler):
    from tsb import models

    pad = [700] * (filler // 700)  # the last: its blocks do not touch the others
    got = []
    for before, after in (([], [64]), ([], [900]), ([100], [3000]), ([1793], [100])):
        sizes = before + [n] + after + pad
        states = [_state([k], k) for k in before] + [_state([n], 1)]
        states += [_state([k], k) for k in after + pad]
        st = _state([1], 0)
        for name in ("positions", "masses", "cell", "atomic_numbers"):
            setattr(st, name, torch.cat([getattr(s, name) for s in states]))
        st.system_idx = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"),
                                                torch.tensor(sizes, device="cuda"))
        st._n_systems = None
        vm = models.VerletListModel(
            models.kob_andersen_model(compute_stress=True, device="cuda"), skin=1.0)
        out, k, lo = vm(st), len(before), sum(before)
        got.append((out["forces"][lo:lo + n], out["energy"][k], out["stress"][k]))
    for other in got[1:]:
        for a, b in zip(got[0], other, strict=True):
            assert torch.equal(a, b)
