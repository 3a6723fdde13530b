"""The work whose speed is followed, through the package's public entry points.

Kinds of case (field ``kind``) and what each stands for:

``nl``       ``torchsim_nl``: the neighbour list a user's own potential, analysis or
             descriptor starts from
``model``    one model call on fresh positions (energy, forces and, by choice, stress
             and per-atom energies): scoring a batch, or a custom integrator's force call
``nve``      velocity-Verlet steps of one large system over a kept Verlet list
``langevin`` per-call NVT-Langevin steps of a small batch: a loop driven from Python,
             where launches and latency count
``fire``     FIRE steps with the Frechet cell filter in the middle of a batched relaxation
``fused``    ``run_md``: a chunk of many MD steps of a whole batch in one call
``adjoint``  loss and gradients of a differentiable NVE trajectory (forward and backward)

Structures (field ``matter``): ``argon`` is fcc Lennard-Jones argon (a = 5.26 A),
``copper`` strained and sheared fcc Morse copper supercells, ``ka`` the 80:20
Kob-Andersen mixture at its number density, all with thermal or random displacements.
Batches are ragged: sizes spread over [atoms_min, atoms_max], with vacancies.
"""

from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "torch-sim_b200"))

from tsb import adjoint, integrators, models, neighbors, optimizers, workloads  # noqa: E402
from tsb.state import SimState  # noqa: E402

DEV = "cuda"
KB, PS = workloads.KB_EV, workloads.METAL_TIME
SIGMA, EPS = 3.405, 0.0104                   # argon
MORSE = (2.866, 0.3429, 1.3588)              # copper: r0, depth, alpha
KA_SIGMA = 3.4
BASIS = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])


def _case(name, kind, matter, systems, lo, hi, **more):
    d = {"name": name, "kind": kind, "matter": matter, "systems": systems, "atoms_min": lo,
         "atoms_max": hi, "cutoff": 8.5, "dtype": "float64", "precision": "mixed",
         "stress": False, "per_atom": False, "half": False, "potential": "lj", "steps": 1,
         "integrator": "nve"}
    d.update(more)
    return d


def listed():
    return [
        # the smallest list: one unit of argon, latency only
        _case("nl_argon_256", "nl", "argon", 1, 256, 256),
        # lists of a ragged batch, as a batched model would ask for them
        _case("nl_copper_512", "nl", "copper", 512, 8, 512, cutoff=6.0, dtype="float32"),
        # the list of one large system: 36 bytes written per pair
        _case("nl_argon_500k", "nl", "argon", 1, 500000, 500000, dtype="float32"),
        # the smallest model call, everything in 64 bits
        _case("lj_256", "model", "argon", 1, 256, 256, precision="fp64", stress=True),
        # forces of a whole ragged batch with 32-bit state
        _case("morse_2048", "model", "copper", 2048, 8, 512, cutoff=6.0, dtype="float32",
              potential="morse"),
        # a species-matrix potential in 64 bits with stress and per-atom energies
        _case("ka_1024", "model", "ka", 1024, 64, 1000, precision="fp64", stress=True,
              per_atom=True, potential="ka"),
        # one large system, 10 steps per pass, lists rebuilt as the atoms drift
        _case("nve_500k", "nve", "argon", 1, 500000, 500000, dtype="float32", steps=10,
              stress=True),
        # a small batch stepped from Python
        _case("langevin_64", "langevin", "argon", 64, 32, 256, steps=5,
              integrator="nvt_langevin"),
        # 20 steps in the middle of a batched relaxation
        _case("fire_ka_1024", "fire", "ka", 1024, 64, 1000, steps=20, stress=True,
              potential="ka"),
        # a chunk of a batched thermostatted run
        _case("fused_copper_2048", "fused", "copper", 2048, 8, 512, cutoff=6.0, dtype="float32",
              potential="morse", steps=100, integrator="nvt_langevin"),
        # a chunk of a small batch in the microcanonical ensemble
        _case("fused_argon_48", "fused", "argon", 48, 32, 256, steps=100),
        # parameter gradients through a trajectory
        _case("adjoint_256", "adjoint", "argon", 256, 108, 108, cutoff=8.5125, steps=200,
              precision="fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["nl", "nl", "model", "model", "model", "nve", "langevin", "fire", "fused",
                       "fused", "adjoint"])
    matter = rng.choice(["argon", "copper", "ka"])
    dtype, precision = rng.choice([("float32", "mixed"), ("float64", "mixed"),
                                   ("float64", "fp64")])
    more = {"stress": rng.random() < 0.5, "per_atom": rng.random() < 0.3}
    if kind in ("nl", "model"):
        if rng.random() < 0.4:
            systems, lo, hi = 1, 0, _log(rng, 33, 500000)
            lo, matter = hi, "argon" if matter == "copper" else matter
        else:
            systems, lo, hi = _log(rng, 2, 512), 8, _log(rng, 40, 512)
        more["half"] = kind == "nl" and rng.random() < 0.3
    elif kind == "nve":
        systems, lo, hi = 1, 0, _log(rng, 4000, 500000)
        lo, matter, dtype, precision = hi, "argon", rng.choice(["float32", "float64"]), "mixed"
        more.update(steps=rng.randint(4, 10), per_atom=False)
    elif kind == "langevin":
        systems, lo, hi = _log(rng, 1, 256), 20, _log(rng, 40, 400)
        more.update(steps=rng.randint(1, 8), integrator="nvt_langevin", per_atom=False)
    elif kind == "fire":
        systems, lo, hi = _log(rng, 8, 1024), 64, _log(rng, 100, 1000)
        matter, dtype, precision = "ka", "float64", rng.choice(["mixed", "fp64"])
        more = {"steps": rng.randint(5, 20), "stress": True}
    elif kind == "fused":
        systems, lo, hi = _log(rng, 16, 2048), 20, _log(rng, 64, 500)
        matter = rng.choice(["argon", "copper"])
        dtype, precision = rng.choice(["float32", "float64"]), "mixed"
        more = {"steps": rng.randint(20, 100),
                "integrator": rng.choice(["nve", "nvt_langevin"])}
    else:
        systems, n = _log(rng, 4, 256), rng.randint(60, 200)
        lo, hi, matter, dtype, precision = n, n + rng.randint(0, 40), "argon", "float64", "fp64"
        more = {"steps": rng.randint(20, 200)}
        if systems * hi * more["steps"] > 5.0e6:
            more["steps"] = max(20, int(5.0e6 / (systems * hi)))
    more["cutoff"] = {"copper": 6.0, "ka": 2.5 * KA_SIGMA}.get(
        matter, 8.5125 if kind == "adjoint" else round(rng.uniform(6.8, 8.5), 3))
    more["potential"] = {"copper": "morse", "ka": "ka"}.get(
        matter, "soft_sphere" if kind == "model" and rng.random() < 0.25 else "lj")
    d = _case("", kind, matter, systems, lo, hi, dtype=dtype, precision=precision, **more)
    del d["name"]
    return d


# ------------------------------------------------------------------ structures
def _crystal(n, a, rng, jitter, strain=0.0, shear=0.0):
    """(positions, row cell) of n atoms of an fcc supercell just large enough."""
    units = max(1, math.ceil(n / 4))
    m1 = max(1, round(units ** (1 / 3)))
    m2 = max(1, round(math.sqrt(units / m1)))
    m3 = math.ceil(units / (m1 * m2))
    shape = np.array([m1, m2, m3])[rng.permutation(3)]
    deform = np.eye(3) + np.diag(rng.uniform(-strain, strain, 3))
    deform[0, 1], deform[0, 2], deform[1, 2] = np.tan(
        np.deg2rad(rng.uniform(-shear, shear, 3)))
    cell = np.diag(shape * a) @ deform
    g = np.stack(np.meshgrid(*(np.arange(k) for k in shape), indexing="ij"), -1).reshape(-1, 3)
    frac = ((g[:, None, :] + BASIS[None]).reshape(-1, 3)) / shape
    if len(frac) > n:                        # vacancies
        frac = frac[np.sort(rng.permutation(len(frac))[:n])]
    return frac @ cell + rng.normal(0.0, jitter, (n, 3)), cell


def _mixture(n, rng):
    """n atoms at the Kob-Andersen density on a displaced, partly filled grid."""
    length = (n * KA_SIGMA ** 3 / 1.2) ** (1 / 3)
    m = math.ceil(n ** (1 / 3))
    at = np.sort(rng.permutation(m ** 3)[:n])
    grid = np.stack([at // (m * m), at // m % m, at % m], -1) + 0.5
    return (grid / m + rng.uniform(-0.08, 0.08, (n, 3)) / m) * length, np.eye(3) * length


def _arrays(case, seed):
    """positions, row cells, masses, numbers, system index and normals, in 64 bits.
    The sizes follow from the case.  So do a list's structures, which a seed only
    mirrors, turns and renumbers: the number of pairs is the shape of the result."""
    fixed = np.random.default_rng([case["systems"], case["atoms_min"], case["atoms_max"]])
    sizes = fixed.integers(case["atoms_min"], case["atoms_max"] + 1, case["systems"])
    rng = np.random.default_rng(seed)
    pos, cells, z = [], [], []
    for n in sizes.tolist():
        rng, own = (fixed, rng) if case["kind"] == "nl" else (rng, None)
        if case["matter"] == "ka":
            x, c = _mixture(n, rng)
            zz = np.ones(n, dtype=np.int64)
            zz[rng.permutation(n)[: round(0.2 * n)]] = 2
        elif case["matter"] == "copper":
            x, c = _crystal(n, 3.61, rng, 0.08, 0.02, 3.0)
            zz = np.full(n, 29)
        else:
            x, c = _crystal(n, 5.26, rng, 0.05 if case["kind"] == "adjoint" else 0.1)
            zz = rng.integers(1, 3, n) if case["kind"] == "adjoint" else np.full(n, 18)
        if own is not None:
            rng = own
            axes, sign = rng.permutation(3), rng.choice([-1.0, 1.0], 3)
            x, c = np.roll(x[:, axes] * sign, rng.integers(n), axis=0), c[:, axes] * sign
        pos.append(x)
        cells.append(c)
        z.append(zz)
    z = np.concatenate(z)
    mass = np.where(z == 29, 63.546, 39.948)
    n = len(z)
    t = lambda v: torch.as_tensor(v, device=DEV)  # noqa: E731
    return (t(np.concatenate(pos)), t(np.stack(cells)), t(mass), t(z),
            t(np.repeat(np.arange(len(sizes)), sizes)), t(rng.standard_normal((n, 3))))


def _temperature(case):
    return {"copper": 1000.0, "argon": 80.0 if case["kind"] == "adjoint" else 50.0,
            "ka": 50.0}[case["matter"]]


def _momenta(case, mass, system_idx, normals):
    """Maxwell-Boltzmann momenta without the systems' drift."""
    p = normals * torch.sqrt(mass * KB * _temperature(case)).unsqueeze(-1)
    size = torch.bincount(system_idx)
    ends = size.cumsum(0)
    total = torch.cat([torch.zeros_like(p[:1]), p.cumsum(0)])
    return p - ((total[ends] - total[ends - size]) / size.unsqueeze(-1))[system_idx]


def _model(case, dtype):
    kw = {"dtype": dtype, "device": DEV, "precision": case["precision"],
          "compute_stress": case["stress"], "per_atom_energies": case["per_atom"]}
    if case["potential"] == "morse":
        return models.MorseModel(*MORSE, cutoff=case["cutoff"], **kw)
    if case["potential"] == "ka":
        return models.kob_andersen_model(sigma_aa=KA_SIGMA, **kw)
    if case["potential"] == "soft_sphere":
        return models.SoftSphereModel(case["cutoff"], 1.0, 2.5, **kw)
    return models.LennardJonesModel(SIGMA, EPS, cutoff=case["cutoff"], **kw)


# ------------------------------------------------------------------ the passes
def prepare(case, seed):
    x, cell, mass, z, sys_idx, normals = _arrays(case, seed)
    dtype = getattr(torch, case["dtype"])
    st = SimState(positions=x.to(dtype), masses=mass.to(dtype), cell=cell.mT.to(dtype).contiguous(),
                  pbc=True, atomic_numbers=z, system_idx=sys_idx)
    s = {"case": case, "state": st}
    kind = case["kind"]
    if kind == "nl":
        s["cell"], s["pbc"] = st.cell.mT.contiguous(), st.pbc
        return s
    if kind == "adjoint":
        p = _momenta(case, mass, sys_idx, normals)
        prob = adjoint.make_problem(st, case["steps"], 0.002 * PS, cutoff=case["cutoff"])
        sg, ep = adjoint.argon_pair_params(device=DEV)
        prob.target = adjoint.histogram(st.positions, prob)
        return s | {"problem": prob, "p": p, "sigma": sg * 1.01, "epsilon": ep * 0.98}
    s["model"] = model = _model(case, dtype)
    if kind == "model":
        return s
    if kind == "fire":
        s["model"] = model = models.VerletListModel(model, skin=1.5)
        fs = optimizers.fire_init(st, model, cell_filter="frechet")
        for _ in range(30):
            fs = optimizers.fire_step(fs, model)
        return s | {"state": fs, "start": {k: getattr(fs, k).clone() for k in _FIRE_FIELDS}}
    if kind == "nve":
        s["model"] = model = models.VerletListModel(model, skin=1.0)
    st.momenta = _momenta(case, mass, sys_idx, normals).to(dtype)
    init = integrators.nvt_langevin_init if case["integrator"] == "nvt_langevin" else (
        integrators.nve_init)
    st.rng = 7
    s["state"] = init(st, model, kT=_temperature(case) * KB)
    return s


_FIRE_FIELDS = ("positions", "velocities", "forces", "energy", "stress", "dt", "alpha", "n_pos",
                "cell", "cell_positions", "cell_velocities", "cell_forces")


def run(s):
    case, st = s["case"], s["state"]
    kind, dt, kT = case["kind"], 0.002 * PS, _temperature(case) * KB
    if kind == "nl":
        return neighbors.torchsim_nl(st.positions, s["cell"], s["pbc"], case["cutoff"],
                                     st.system_idx, half=case["half"])
    if kind == "model":
        return s["model"](st)
    if kind == "adjoint":
        out = adjoint.loss_and_grad(s["sigma"], s["epsilon"], st.positions, s["p"], s["problem"])
        return dict(zip(("loss", "sigma", "epsilon", "q", "p"), out, strict=True))
    if kind == "fire":
        # every pass takes the same stretch of the relaxation: left to run on, the
        # batch converges and stops moving
        for k, v in s["start"].items():
            getattr(st, k).copy_(v)
        for _ in range(case["steps"]):
            st = optimizers.fire_step(st, s["model"])
        return {k: getattr(st, k) for k in _FIRE_FIELDS}
    if kind == "fused":
        st = integrators.run_md(st, s["model"], case["steps"], integrator=case["integrator"],
                                dt=dt, kT=kT if case["integrator"] != "nve" else None,
                                gamma=10.0 / PS if case["integrator"] != "nve" else None,
                                skin=1.0)
    elif kind == "nve":
        for _ in range(case["steps"]):
            st = integrators.nve_step(st, s["model"], dt=dt)
    else:
        for _ in range(case["steps"]):
            st = integrators.nvt_langevin_step(st, s["model"], dt=dt, kT=kT, gamma=1.0 / PS)
    return {k: getattr(st, k) for k in ("positions", "momenta", "forces", "energy")}


def work(case):
    """Atoms, their half-list pairs within the cutoff and about 45 flops per pair
    evaluation; state read and written once per step (nothing per step for the
    chunk of a fused run, whose state can stay on the chip)."""
    n = case["systems"] * (case["atoms_min"] + case["atoms_max"]) / 2
    rho = {"copper": 4 / 3.61 ** 3, "ka": 1.2 / KA_SIGMA ** 3}.get(case["matter"], 4 / 5.26 ** 3)
    pairs = n * 2 / 3 * math.pi * case["cutoff"] ** 3 * rho
    size = 4 if case["dtype"] == "float32" else 8
    kind, steps = case["kind"], case["steps"]
    if kind == "nl":
        rows = pairs if case["half"] else 2 * pairs
        return {"bytes": n * (3 * size + 8) + rows * (24 + 3 * size), "flops": 9 * pairs}
    if kind == "model":
        return {"bytes": n * ((6 + case["per_atom"]) * size + 16), "flops": 45 * pairs}
    if kind == "adjoint":
        # forces forward, forces again and a Hessian-vector product backward
        return {"bytes": n * 160, "flops": steps * pairs * (45 + 45 + 110)}
    if kind == "fused":
        return {"bytes": n * 18 * size, "flops": 45 * pairs * steps}
    per_atom = 24 if kind == "fire" else 18
    return {"bytes": steps * n * per_atom * size, "flops": 45 * pairs * steps}


# ------------------------------------------------------- the same in 64 bits
def _pairs_small(x, cell, lo, reach):
    """Every ordered pair within reach of one small system (all images, dense)."""
    width = 1.0 / torch.linalg.inv(cell).norm(dim=0)
    k = [int(v) for v in torch.ceil(reach / width).tolist()]
    grid = torch.cartesian_prod(*(torch.arange(-v - 1, v + 2, device=DEV) for v in k)).double()
    i, j, sh = [], [], []
    for part in grid.split(max(1, int(6e7 / len(x) ** 2))):
        d = (x[None, None] + (part @ cell)[:, None, None]) - x[None, :, None]
        hit = (d * d).sum(-1) < reach * reach
        hit &= ~((part == 0).all(-1)[:, None, None] & torch.eye(len(x), dtype=torch.bool,
                                                                device=DEV))
        m, a, b = torch.nonzero(hit, as_tuple=True)
        i.append(a + lo)
        j.append(b + lo)
        sh.append(part[m] @ cell)
    return torch.cat(i), torch.cat(j), torch.cat(sh)


def _pairs_large(x, cell, reach):
    """Every ordered pair within reach of one large system (cells of that width)."""
    inv = torch.linalg.inv(cell)
    nb = torch.floor(1.0 / inv.norm(dim=0) / reach).long().clamp_min(1)
    u = x @ inv
    wrap = torch.floor(u)
    b3 = ((u - wrap) * nb).long().clamp_min(0).minimum(nb - 1)
    b = (b3[:, 0] * nb[1] + b3[:, 1]) * nb[2] + b3[:, 2]
    order = torch.argsort(b, stable=True)
    count = torch.bincount(b, minlength=int(nb.prod()))
    slot = torch.arange(len(x), device=DEV) - (count.cumsum(0) - count)[b[order]]
    table = torch.full((len(count), int(count.max())), -1, device=DEV)
    table[b[order], slot] = order
    w = x - wrap @ cell
    c3 = torch.cartesian_prod(*(torch.arange(int(v), device=DEV) for v in nb))
    i, j, sh = [], [], []
    for o in torch.cartesian_prod(*[torch.arange(-1, 2, device=DEV)] * 3):
        to = c3 + o
        image = torch.div(to, nb, rounding_mode="floor")
        to = to - image * nb
        other = table[(to[:, 0] * nb[1] + to[:, 1]) * nb[2] + to[:, 2]]
        move = image.double() @ cell
        step = max(1, int(3e7 / table.shape[1] ** 2))
        for k in range(0, len(table), step):
            a, c, mv = table[k:k + step], other[k:k + step], move[k:k + step]
            d = (w[c] + mv[:, None])[:, None, :] - w[a][:, :, None]
            hit = ((d * d).sum(-1) < reach * reach) & (a >= 0)[:, :, None] & (c >= 0)[:, None, :]
            hit &= (a[:, :, None] != c[:, None, :]) | (mv != 0).any(-1)[:, None, None]
            m, p, q = torch.nonzero(hit, as_tuple=True)
            ai, cj = a[m, p], c[m, q]
            i.append(ai)
            j.append(cj)
            sh.append(mv[m] + (wrap[ai] - wrap[cj]) @ cell)
    return torch.cat(i), torch.cat(j), torch.cat(sh)


def _pairs(x, cell, sys_idx, reach):
    """(i, j, lattice vector): the ordered pairs |x_j + vector - x_i| < reach."""
    size = torch.bincount(sys_idx).tolist()
    if len(size) == 1 and size[0] > 3000:
        return _pairs_large(x, cell[0], reach)
    got, lo = [], 0
    for s, n in enumerate(size):
        got.append(_pairs_small(x[lo:lo + n], cell[s], lo, reach))
        lo += n
    return tuple(torch.cat(v) for v in zip(*got, strict=True))


class _Exact:
    """Pair energies and forces of a case by plain tensor operations in 64 bits."""

    def __init__(self, case, x, cell, z, sys_idx, margin=0.0):
        self.case, self.cell, self.sys_idx = case, cell, sys_idx
        self.i, self.j, self.sh = _pairs(x, cell, sys_idx, case["cutoff"] + margin)
        one = torch.ones((), dtype=torch.float64, device=DEV)
        sg, ep, self.rc, self.shift = SIGMA * one, EPS * one, case["cutoff"] * one, 0.0 * one
        if case["potential"] == "ka":
            sg = torch.tensor([[1.0, 0.8], [0.8, 0.88]], dtype=torch.float64, device=DEV) * KA_SIGMA
            ep = torch.tensor([[1.0, 1.5], [1.5, 0.5]], dtype=torch.float64, device=DEV) * EPS
            self.rc = 2.5 * sg
            self.shift = 4 * ep * (2.5 ** -12 - 2.5 ** -6)
        self.of = None
        if sg.ndim == 2:
            self.of = (z[self.i] - 1, z[self.j] - 1)
        self.sg, self.ep = sg, ep

    def at(self, t):
        return t if self.of is None or t.ndim == 0 else t[self.of]

    def __call__(self, x, full=False):
        d = x[self.j] + self.sh - x[self.i]
        r2 = (d * d).sum(-1)
        inside = r2 < self.at(self.rc) ** 2
        r = r2.sqrt()
        pot = self.case["potential"]
        if pot == "morse":
            r0, depth, alpha = MORSE
            ex = torch.exp(-alpha * (r - r0))
            e, dv = depth * (1 - ex) ** 2 - depth, 2 * alpha * depth * ex * (1 - ex)
        elif pot == "soft_sphere":
            base = (1 - r / self.case["cutoff"]).clamp_min(0.0)
            e, dv = base ** 2.5 / 2.5, -base ** 1.5 / self.case["cutoff"]
        else:
            ep, s6 = self.at(self.ep), (self.at(self.sg) ** 2 / r2) ** 3
            e, dv = 4 * ep * (s6 * s6 - s6) - self.at(self.shift), -24 * ep * (2 * s6 * s6 - s6) / r
        e, dv = torch.where(inside, e, 0.0), torch.where(inside, dv, 0.0)
        f = torch.zeros_like(x).index_add_(0, self.i, d * (dv / r).unsqueeze(-1))
        per_atom = torch.zeros_like(x[:, 0]).index_add_(0, self.i, e)
        ns = len(self.cell)
        energy = 0.5 * torch.zeros(ns, dtype=x.dtype, device=DEV).index_add_(
            0, self.sys_idx, per_atom)
        if not full:
            return energy, f
        out = {"energy": energy, "forces": f}
        if self.case["stress"]:
            w = (d.unsqueeze(2) * (d * (dv / r).unsqueeze(-1)).unsqueeze(1)).reshape(-1, 9)
            v = torch.zeros((ns, 9), dtype=x.dtype, device=DEV).index_add_(
                0, self.sys_idx[self.i], w)
            out["stress"] = (0.5 * v / torch.linalg.det(self.cell).abs()[:, None]).view(ns, 3, 3)
        if self.case["per_atom"]:
            out["energies"] = per_atom
        return out


def _exact_nve(case, ex, x, p, mass):
    dt, m = 0.002 * PS, mass.unsqueeze(-1)
    e, f = ex(x)
    for _ in range(case["steps"]):
        p = p + f * (dt / 2)
        x = x + p / m * dt
        e, f = ex(x)
        p = p + f * (dt / 2)
    return {"positions": x, "momenta": p, "forces": f, "energy": e}


def _exact_adjoint(case, x0, p0, cell, mass, z, sys_idx):
    """The trajectory step by step, its loss, and the reversed sweep with each
    step's Hessian and parameter products taken by differentiating the forces."""
    i, j, sh = _pairs(x0, cell, sys_idx, case["cutoff"] + 2.0)
    kind = (z[i] - 1) * 2 + z[j] - 1
    ns, m, dt, steps = len(cell), mass.unsqueeze(-1), 0.002 * PS, case["steps"]
    par0 = torch.tensor([[SIGMA * 1.01], [EPS * 0.98]], dtype=torch.float64,
                        device=DEV).repeat(1, 4)
    rc2 = case["cutoff"] ** 2

    def forces(x, par):
        d = x[j] + sh - x[i]
        r2 = (d * d).sum(-1)
        s6 = (par[0][kind] ** 2 / r2) ** 3
        g = torch.where(r2 < rc2, -24 * par[1][kind] * (2 * s6 * s6 - s6) / r2, 0.0)
        return torch.zeros_like(x).index_add(0, i, d * g.unsqueeze(-1))

    def histogram(x):
        d = x[j] + sh - x[i]
        r = (d * d).sum(-1).sqrt()
        centre = (torch.arange(64, device=DEV, dtype=torch.float64) + 0.5) * (8.0 / 64)
        h = torch.zeros((ns, 64), dtype=torch.float64, device=DEV)
        keep = torch.nonzero(r < 8.0).flatten()
        for part in keep.split(1_000_000):
            g = 0.5 * torch.exp(-((r[part, None] - centre) ** 2) / (2 * 0.05 ** 2))
            h = h.index_add(0, sys_idx[i[part]], g)
        return h

    target = histogram(x0)
    x, p, f = x0, p0, forces(x0, par0)
    path = []
    for _ in range(steps):
        path.append(x)
        p = p + f * (dt / 2)
        x = x + p / m * dt
        f = forces(x, par0)
        p = p + f * (dt / 2)
    xt = x.clone().requires_grad_(True)
    loss = ((histogram(xt) - target) ** 2).sum()
    lq = torch.autograd.grad(loss, xt)[0]
    lp, gp = torch.zeros_like(lq), torch.zeros_like(par0)
    for k in range(steps - 1, -1, -1):
        lp = lp + lq / m * dt
        xk, par = path[k].clone().requires_grad_(True), par0.clone().requires_grad_(True)
        gx, gpar = torch.autograd.grad((forces(xk, par) * lp).sum(), (xk, par))
        c = dt / 2 if k == 0 else dt
        lq, gp = lq + c * gx, gp + c * gpar
    gp = gp.view(2, 2, 2)
    gp = gp + gp.mT - torch.diag_embed(torch.diagonal(gp, dim1=1, dim2=2))
    return {"loss": loss.detach(), "sigma": gp[0], "epsilon": gp[1], "q": lq, "p": lp}


def exact(case, seed):
    kind = case["kind"]
    # lists are whole numbers; Langevin noise is drawn by the package; relaxations
    # are held to the bound of their type
    if kind in ("nl", "langevin", "fire") or case["integrator"] == "nvt_langevin":
        return None
    dtype = getattr(torch, case["dtype"])
    x, cell, mass, z, sys_idx, normals = _arrays(case, seed)
    x, cell, mass = (t.to(dtype).double() for t in (x, cell, mass))
    if kind == "model":
        return _Exact(case, x, cell, z, sys_idx)(x, full=True)
    p = _momenta(case, _arrays(case, seed)[2], sys_idx, normals).to(dtype).double()
    if kind == "adjoint":
        return _exact_adjoint(case, x, p, cell, mass, z, sys_idx)
    if case["systems"] * case["atoms_max"] * case["steps"] > 6e6 and kind == "fused":
        return None
    return _exact_nve(case, _Exact(case, x, cell, z, sys_idx, margin=2.0), x, p, mass)
