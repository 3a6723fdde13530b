"""Rebuilding part of a batch: the offsets of the marked systems' atoms come from one
block up to 4096 systems, in passes of 1024, and from the general scan above.  Pairs of
atoms in cells of their own, so that every force is known in closed form."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
SIGMA, EPS, CUTOFF, SKIN, L = 1.0, 0.5, 2.5, 0.3, 6.0


@pytest.mark.parametrize("ns", [2, 31, 1023, 1024, 1025, 4096, 4097])
def test_marked_systems(ns):
    from tsb import models
    from tsb.state import SimState

    rng = np.random.default_rng(ns)
    sizes = rng.integers(2, 4, ns) if ns > 2 else np.array([2, 2])
    first = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    n = int(sizes.sum())
    sysi = np.repeat(np.arange(ns), sizes)
    pos = rng.uniform(0, L, (n, 3))
    # the second atom at 1 to 2.2 sigma, the third (if any) out of reach of both
    d = rng.standard_normal((ns, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    third = first[sizes == 3] + 2
    pos[third] = pos[third - 2] + L / 2
    model = models.VerletListModel(
        models.LennardJonesModel(sigma=SIGMA, epsilon=EPS, cutoff=CUTOFF, dtype=torch.float64,
                                 device="cuda", precision="fp64"), skin=SKIN)
    st = None
    r = rng.uniform(1.0, 1.4, ns)
    for step in range(3):
        if step == 1:  # some systems expire, the first and the last among them
            r[1:-1][rng.random(ns - 2) < 0.3] += 0.7
            r[0] += 0.7
        if step == 2:
            r[-1] += 0.7
        pos[first + 1] = pos[first] + r[:, None] * d
        t = torch.as_tensor(pos, device="cuda")
        if st is None:
            st = SimState(positions=t, masses=torch.ones(n, device="cuda").double(),
                          cell=(torch.eye(3, device="cuda").double() * L).repeat(ns, 1, 1),
                          pbc=True, atomic_numbers=torch.ones(n, device="cuda").long(),
                          system_idx=torch.as_tensor(sysi, device="cuda"))
        st.positions = t
        got = model(st)["forces"].cpu().numpy()
        want = np.zeros((n, 3))
        i6 = (SIGMA / r) ** 6
        f = (24 * EPS * (2 * i6 * i6 - i6) / r)[:, None] * d
        want[first + 1], want[first] = f, -f
        # positions of up to 6 rounded to 1e-16 of that, a force gradient of some 30
        # per unit length at r = 1: some 1e-13 absolute
        np.testing.assert_allclose(got, want, rtol=0, atol=1e-11)


def test_systems_in_any_order():
    """The atoms of a system lie together; the systems need not ascend."""
    from tsb import neighbors

    rng = np.random.default_rng(3)
    pos = torch.as_tensor(rng.uniform(0, 8, (70, 3)), device="cuda")
    cell = torch.eye(3, device="cuda").double().repeat(3, 1, 1) * 8.0
    pbc = torch.ones(3, dtype=torch.bool, device="cuda")
    idx = torch.tensor([2] * 30 + [0] * 25 + [1] * 15, device="cuda")
    m, s, _ = neighbors.torchsim_nl(pos, cell, pbc, 3.0, idx)
    for k in range(3):
        at = (idx == k).nonzero()[:, 0]
        one, _, _ = neighbors.torchsim_nl(pos[at], cell[:1], pbc, 3.0, torch.zeros_like(at))
        here = m[:, s == k]
        assert torch.equal(here[0].sort()[0], at[one[0]].sort()[0])
        assert {tuple(p) for p in here.T.tolist()} == {tuple(p) for p in at[one].T.tolist()}
