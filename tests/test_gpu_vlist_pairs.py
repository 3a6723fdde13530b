"""Verlet lists that hold each pair within its own cutoff + skin: results equal those of
the search per call while the lists stay valid, and the lists follow the species."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _state(n, seed):
    from tsb.state import SimState

    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1 / 3)))
    length = (n * 3.4**3 / 1.2) ** (1 / 3)
    at = np.sort(rng.permutation(m**3)[:n])
    g = (np.stack([at // (m * m), at // m % m, at % m], -1) + 0.5) / m * length
    t = lambda v: torch.as_tensor(v, device="cuda")  # noqa: E731
    return SimState(positions=t(np.concatenate([g, g]) + rng.uniform(-0.3, 0.3, (2 * n, 3))),
                    masses=torch.ones(2 * n, device="cuda").double(),
                    cell=torch.eye(3, device="cuda").double().repeat(2, 1, 1) * length,
                    pbc=True, atomic_numbers=t(1 + (rng.random(2 * n) < 0.4)),
                    system_idx=t(np.repeat([0, 1], n)))


def _check(vm, model, st):
    got, want = vm(st), model(st)
    for k in ("forces", "energy", "stress"):
        # FP64 sums of some 100 terms each in two orders: 1e-13 of the largest term
        scale = float(want[k].abs().max())
        assert float((got[k] - want[k]).abs().max()) <= 1e-11 * scale, k


@pytest.mark.parametrize("prune", [None, 0.4])
@pytest.mark.parametrize("n", [600, 1100])
@pytest.mark.parametrize("kind", ["lj", "morse"])
def test_species_cutoffs(kind, n, prune):
    from tsb import models

    if kind == "lj":
        model = models.kob_andersen_model(compute_stress=True, device="cuda", precision="fp64",
                                          dtype=torch.float64)
    else:
        model = models.MorseModel(2.6, 0.3, 1.4, cutoff=6.0, compute_stress=True, device="cuda",
                                  precision="fp64", dtype=torch.float64)
    vm = models.VerletListModel(model, skin=1.0, prune=prune)
    st = _state(n, n)
    _check(vm, model, st)
    # every atom up to just short of the distance at which the lists expire
    g = torch.Generator(device="cuda").manual_seed(1)
    for reach in (0.3, 0.495):
        d = torch.randn(st.positions.shape, generator=g, device="cuda").double()
        d = d / d.norm(dim=1, keepdim=True) * reach
        base = st.positions
        st.positions = base + d
        _check(vm, model, st)
        st.positions = base
    assert vm.n_builds == 1 or prune is not None
    if kind == "lj":  # species exchanged, in place and in tensors that come and go
        st.atomic_numbers.copy_(3 - st.atomic_numbers)
        _check(vm, model, st)
        for _ in range(4):
            z = (3 - st.atomic_numbers).tolist()
            st.atomic_numbers = None
            st.atomic_numbers = torch.tensor(z, device="cuda")
            _check(vm, model, st)
