"""Verlet-list model wrapper: neighbour lists kept between calls.

``VerletListModel(model, skin=1.0)`` wraps a tsb ``PairTableModel`` (LJ, Morse,
soft sphere).  Each system's list holds every pair within cutoff + skin and is
rebuilt, per system, only when its atoms' drift and its cell's deformation since
the build could have brought a pair from beyond cutoff + skin to inside the
cutoff (C ABI: tsb_vlist_check / tsb_vlist_build / tsb_vlist_forces).  The
reference rebuilds its list in every call (torch_sim/models/pair_potential.py:
168-174); the pairs inside the cutoff, and therefore energy, forces and stress,
are the same.  Works for one large system (500,000 atoms) and for batches of
small ones whose atoms and cells move (FIRE with a cell filter, NPT, MD).

Every periodic cell must be at least cutoff + skin wide (image shifts in
{-1,0,1}^3); narrower cells raise ValueError.  The wrapper keeps its own device
workspace (the list frame) and reads two flags from the device per call, while the
force kernel runs: the flags leave for pinned memory before it is launched.  Where the
lists turn out to have overflowed (or, for one large system, expired) that kernel has
written nothing, and the call evaluates again before it returns or raises.

One fully periodic system with FP32 pair arithmetic and no per-atom outputs (the
500,000-atom workload) takes the single-system kernels (tsb_verlet_build /
tsb_verlet_check / tsb_verlet_forces: atom order, per-block sums fused into the
force kernel), about 10 % faster there; its list expires when an atom moved more
than skin/2 or the cell changed.
"""

from __future__ import annotations

import torch

from .. import _lib as L
from .. import ops as _ops  # noqa: F401  (registers torch.ops.tsb.*)
from .interface import ModelInterface
from .pair_potential import PairTableModel


class VerletListModel(ModelInterface):
    # Batches of this many atoms have their lists rebuilt (the marked systems') without
    # waiting for the check, smaller ones after reading its answer: below it the launches
    # of a build that does nothing cost more than the wait, which leaves the GPU idle.  A
    # FIRE step of Kob-Andersen systems of 64 to 1000 atoms, unread against read: 229 and
    # 200 us at 6,000 atoms, 239 and 222 at 177,000, 290 and 290 at 312,000, 403 and 432 at
    # 550,000 on one host; 239 and 253 at 211,000, 283 and 286 at 266,000, 294 and 314 at
    # 330,000, 399 and 427 at 550,000 on another (FP64: 312 and 327, 378 and 399, 436 and
    # 457, 637 and 666).
    # Only with systems of at most UNREAD_SYSTEM_ATOMS, which are binned one block each, the
    # marked ones alone (tsb_vlist_build): a larger one bins the whole batch in every call.
    # NVE steps, unread against read: one system of 500,000 atoms in FP64 533 and 468 us,
    # two of 200,000 335 and 275; 100 of 4,000 259 to 306 and 342 to 373.
    UNREAD_ATOMS = 262144
    UNREAD_SYSTEM_ATOMS = 4096

    def __init__(self, model: PairTableModel, *, skin: float = 1.0, max_neighbors: int = 0,
                 prune: float | None = None):
        """``prune`` (Angstrom, batched lists only): between rebuilds each atom
        evaluates only the list entries that were within its pair cutoff +
        ``prune`` at the system's last pruning; a system is pruned again when its
        atoms' drift or its cell's deformation could bring a left-out pair inside
        the cutoff.  Results equal those of the whole list to FP64 rounding.
        Default 0 (off): on the FIRE + Frechet relax workload the non-affine
        steps use up the drift allowance within a few steps and the re-prunings
        cost more than the shorter lists save (0.54 against 0.47 ms per step
        with 0.2 to 0.45 A)."""
        super().__init__()
        if not isinstance(model, PairTableModel):
            raise TypeError("VerletListModel wraps a tsb PairTableModel")
        if model.kind not in (L.POT_LJ, L.POT_MORSE, L.POT_SOFT):
            raise TypeError("VerletListModel supports LJ, Morse and soft-sphere tables")
        self.model = model
        self._device, self._dtype = model.device, model.dtype
        self._compute_forces, self._compute_stress = True, model.compute_stress
        self.per_atom_energies = getattr(model, "per_atom_energies", False)
        self.per_atom_stresses = getattr(model, "per_atom_stresses", False)
        self.skin = float(skin)
        self.prune = 0.0 if prune is None else float(prune)
        if not (0.0 <= self.prune):
            raise ValueError("prune must be >= 0")
        if self.prune >= self.skin:
            self.prune = 0.0  # the whole list is within cutoff + skin anyway
        self.max_neighbors = int(max_neighbors)
        self.n_builds = 0
        self._key = None          # what the batched lists are for
        self._pbc_of_single = L.SeenPbc()  # the flags that _pbc_all says it for
        self._last_single = False
        # graph-safe mode: the rebuild is decided on the device (no host reads),
        # list overflow is recorded in a sticky device flag (see set_graph_safe)
        self.graph_safe = False
        self.sticky = None
        self._built = False       # the batched lists have been built once
        self._flags_host = None   # pinned copy of the flags

    # -------------------------------------------------------------- buffers
    def _ensure(self, state, pos, cell_row):
        n, ns = state.n_atoms, state.n_systems
        sysi, z = state.system_idx, state.atomic_numbers
        # the systems, the species, the table's cutoffs and the periodic axes decide which
        # pairs are listed
        key, of = (n, ns, pos.dtype, pos.device), (sysi, z, self.model.table)
        if (self._key == key and all(a.same(b) for a, b in zip(self._seen, of, strict=True))
                and self._seen_pbc.same(state.pbc)):
            return
        dev = pos.device
        self._key = None  # (until every buffer is there)
        rcs = self.model.cutoff + self.skin
        counts = torch.bincount(sysi, minlength=ns).double()
        self.max_system_atoms = L.list_size_hint(sysi, ns, int(counts.max()) if ns else 0)
        vol = torch.linalg.det(cell_row.double()).abs().clamp_min(1e-30)
        dens = float((counts / vol).max())
        est = int(4.19 * rcs ** 3 * dens * 1.35) + 16
        if not (est < 4096):
            est = 4096
        self._allot(max(self.max_neighbors, est), n, dev)
        self.counts = torch.empty(n, dtype=torch.int32, device=dev)
        self.flags = torch.zeros(2, dtype=torch.int32, device=dev)
        self.ws = torch.empty(L.load().tsb_vlist_workspace_size(n, ns), dtype=torch.uint8,
                              device=dev)
        self._reset(n, ns, dev)
        self._built = False
        self._key, self._seen = key, tuple(map(L.Seen, of))
        self._seen_pbc = L.SeenPbc(state.pbc)

    def _allot(self, cap, n, dev):
        """Room for ``cap`` neighbours per atom.  The capacity is what the kernels may
        write, so it changes after the allocation has succeeded; where it does not, the
        lists that are there (cut short, perhaps) are no good for a later call."""
        key, self._key = self._key, None
        self.list = torch.empty(cap * n, dtype=torch.int32, device=dev)
        self.cap, self._key = cap, key

    def _reset(self, n, ns, dev):
        L.call("tsb_vlist_reset", n, ns, L.ptr(self.ws), self.ws.numel(), L.stream_ptr(dev))

    def set_graph_safe(self, on: bool = True) -> None:
        """Graph-safe mode for CUDA-graph capture of step loops: every call checks
        the lists and launches the rebuild unconditionally (the rebuild kernels
        only touch the systems the check marked as expired), and nothing is read
        back to the host.  A list that overflows or a cell narrower than cutoff +
        skin is recorded in ``self.sticky`` (device int32 [1], maximum over
        calls); ``check_overflow()`` reads it after a replay."""
        self.graph_safe = bool(on)

    def check_overflow(self) -> int:
        """0, or the neighbour count that overflowed the lists since the last
        reset (1 << 30 for a cell narrower than cutoff + skin)."""
        return 0 if self.sticky is None else int(self.sticky.item())

    def grow(self, needed: int, state) -> None:
        """Regrow the lists to hold ``needed`` neighbours per atom and mark every
        system for a rebuild (after an overflow seen by check_overflow)."""
        if needed >= (1 << 30):
            raise ValueError("VerletListModel needs every periodic cell width >= cutoff + skin")
        dev = state.positions.device
        self._allot(int(needed * 1.2) + 8, state.n_atoms, dev)
        self._reset(state.n_atoms, state.n_systems, dev)
        self._built = False
        if self.sticky is not None:
            self.sticky.zero_()

    # ---------------------------------------------------------------- flags
    def _publish(self, flags):
        """Device flags into pinned memory, on the current stream."""
        if self._flags_host is None:
            self._flags_host = torch.zeros(2, dtype=torch.int32).pin_memory()
        stream = torch.cuda.current_stream(flags.device)
        L.call("tsb_publish_flags", L.ptr(flags), flags.numel(), L.ptr(self._flags_host),
               stream.cuda_stream)
        return stream

    def _flags_now(self, flags) -> list[int]:
        self._publish(flags).synchronize()
        return self._flags_host.tolist()

    def _send_flags(self, flags) -> torch.cuda.Event:
        """The flags on their way: an event for _read_flags."""
        sent = torch.cuda.Event()
        sent.record(self._publish(flags))
        return sent

    def _read_flags(self, sent) -> list[int]:
        sent.synchronize()
        return self._flags_host.tolist()

    def __getstate__(self):
        # a copied or loaded model pins a buffer of its own (a copy of this one would be
        # pageable memory, which the kernel must not write to)
        return self.__dict__ | {"_flags_host": None}

    # ---------------------------------------------------------------- lists
    def _update_lists(self, state, pos, cell_row, pbc, sysi, species, active,
                      table):
        """None, or the event of flags on their way, which have to be read after the
        forces have been launched."""
        n, ns, dev = state.n_atoms, state.n_systems, pos.device
        m, cutoff = self.model, self.model.cutoff

        def build():
            torch.ops.tsb.vlist_build_(pos, cell_row, pbc, sysi, species, ns, cutoff, self.skin,
                                       self.list, self.counts, self.cap, self.max_system_atoms,
                                       self.flags, self.ws, table, m.kind, m.n_species)

        if self.graph_safe:
            if self.sticky is None or self.sticky.device != dev:
                self.sticky = torch.zeros(1, dtype=torch.int32, device=dev)
            torch.ops.tsb.vlist_check_(pos, cell_row, sysi, active, ns, cutoff, self.skin,
                                       self.prune, self.flags, self.ws)
            build()
            torch.maximum(self.sticky, self.flags[1:], out=self.sticky)
            return None
        if (self._built and n >= self.UNREAD_ATOMS
                and self.max_system_atoms <= self.UNREAD_SYSTEM_ATOMS):
            # (the rebuild touches only the systems that the check marked)
            torch.ops.tsb.vlist_check_(pos, cell_row, sysi, active, ns, cutoff, self.skin,
                                       self.prune, self.flags, self.ws)
            build()
            return self._send_flags(self.flags)
        while True:
            torch.ops.tsb.vlist_check_(pos, cell_row, sysi, active, ns, cutoff, self.skin,
                                       self.prune, self.flags, self.ws)
            if not self._flags_now(self.flags)[0]:
                break
            build()
            self.n_builds += 1
            st = int(self.flags[1].item())
            if st == 0:
                break
            self._grow_lists(st, n, ns, dev)
        self._built = True
        return None

    def _grow_lists(self, needed, n, ns, dev):
        """A list overflowed: regrow it and mark every system for a rebuild."""
        if needed >= (1 << 30):
            self._key = None  # (what has been listed is no good for a later call either)
            raise ValueError("VerletListModel needs every periodic cell width >= "
                             "cutoff + skin")
        self._allot(int(needed * 1.2) + 8, n, dev)
        self._reset(n, ns, dev)
        self._built = False

    def _run(self, state, energy, forces, stress, energies, stresses, active):
        if state.dtype != self._dtype:
            raise TypeError(f"SimState dtype {state.dtype} does not match model dtype "
                            f"{self._dtype}.")
        pos = state.positions.contiguous()
        L.require_cuda(pos, "state.positions")
        n_sys = state.n_systems
        cell_row = state.cell.mT.contiguous()
        pbc = L.pbc_rows(state.pbc, n_sys, pos.device)
        sysi = state.system_idx.contiguous()
        species = self.model._species(state.atomic_numbers)
        m = self.model
        table = m.table if m.table.device == pos.device else m.table.to(pos.device)
        self._ensure(state, pos, cell_row)
        pending = self._update_lists(state, pos, cell_row, pbc, sysi, species, active, table)
        flags = 0
        if forces is not None:
            flags |= L.OUT_FORCES
        if stress is not None:
            flags |= L.OUT_STRESS
        if energies is not None:
            flags |= L.OUT_ENERGIES
        if stresses is not None:
            flags |= L.OUT_STRESSES
        if m.precision == "fp64":
            flags |= L.MATH_FP64

        def evaluate(skip=None):
            torch.ops.tsb.vlist_forces_(m.kind, table, m.n_species, species, self.list,
                                        self.counts, pos, cell_row, sysi, active, n_sys,
                                        m.cutoff, self.prune, flags, energy, forces, stress,
                                        energies, stresses, self.ws, skip)

        try:
            evaluate(self.flags[1:] if pending else None)
        finally:  # (the host buffer is in use until it has been read)
            marked, overflow = self._read_flags(pending) if pending else (0, 0)
        self.n_builds += 1 if marked else 0
        if overflow:
            self._grow_lists(overflow, state.n_atoms, n_sys, pos.device)
            self._update_lists(state, pos, cell_row, pbc, sysi, species, active, table)
            evaluate()

    # ------------------------------------------------- one large system
    def _single_ok(self, state):
        if (state.n_systems != 1 or self.model.precision == "fp64" or self.per_atom_energies
                or self.per_atom_stresses):
            return False
        pbc = state.pbc
        if not self._pbc_of_single.same(pbc):  # one device read per pbc tensor
            self._pbc_of_single = L.SeenPbc(pbc)
            self._pbc_all = bool(L.pbc_rows(pbc, 1, state.positions.device).all())
        return self._pbc_all

    def _s_ensure(self, state):
        n = state.n_atoms
        key = (n, state.positions.dtype, state.positions.device)
        if getattr(self, "_s_key", None) == key:
            return
        dev = state.device
        self._s_key = None  # (until every buffer is there)
        rcs = self.model.cutoff + self.skin
        vol = float(torch.det(state.cell[0].double()).abs())
        est = int(4.2 * rcs ** 3 * n / vol * 1.35) + 16
        self._s_allot(max(self.max_neighbors, est), n, dev)
        self.s_counts = torch.empty(n, dtype=torch.int32, device=dev)
        self.s_ref = torch.empty((n, 3), dtype=torch.float64, device=dev)
        self.s_wraps = torch.empty((n, 3), dtype=torch.int32, device=dev)
        self.s_status = torch.zeros(1, dtype=torch.int32, device=dev)
        self.s_expired = torch.zeros(1, dtype=torch.int32, device=dev)
        self.s_ws = torch.empty(L.load().tsb_verlet_workspace_size(n), dtype=torch.uint8,
                                device=dev)
        self._s_key = key
        self._s_built = False

    def _s_allot(self, cap, n, dev):
        self.s_list = torch.empty(cap * n, dtype=torch.int32, device=dev)
        self.s_cap = cap

    def _s_check(self, state, pos, cell64):
        L.call("tsb_verlet_check", L.ptr(pos), L.ptr(self.s_ref), L.ptr(self.s_wraps),
               L.ptr(cell64), L.ptr(self.model._species(state.atomic_numbers)), state.n_atoms,
               L.dtype_code(pos.dtype), self.skin, L.ptr(self.s_expired), L.ptr(self.s_ws),
               self.s_ws.numel(), L.stream_ptr(state.device))

    def _s_build(self, state, pos):
        cell = state.cell[0].mT.to(pos.dtype).contiguous()
        self._s_built = False
        while True:
            L.call("tsb_verlet_build", L.ptr(pos), L.ptr(cell), state.n_atoms,
                   L.dtype_code(pos.dtype), self.model.cutoff, self.skin, L.ptr(self.s_list),
                   L.ptr(self.s_counts), self.s_cap, L.ptr(self.s_ref), L.ptr(self.s_wraps),
                   L.ptr(self.s_status), L.ptr(self.s_ws), self.s_ws.numel(),
                   L.stream_ptr(state.device))
            st = int(self.s_status.item())
            if st == 0:
                break
            if st >= (1 << 30):
                raise ValueError("VerletListModel needs every periodic cell width >= "
                                 "cutoff + skin")
            self._s_allot(int(st * 1.2) + 8, state.n_atoms, state.device)
        self.n_builds += 1
        self._s_built = True

    def _single_forward(self, state, energy=None, forces=None, stress=None):
        """Results in the given contiguous buffers of the positions' dtype, or in new
        ones."""
        if state.dtype != self._dtype:
            raise TypeError(f"SimState dtype {state.dtype} does not match model dtype "
                            f"{self._dtype}.")
        L.require_cuda(state.positions, "state.positions")
        self._s_ensure(state)
        pos = state.positions.contiguous()
        # (one launch: type and layout in the same copy)
        cell64 = torch.empty((3, 3), dtype=torch.float64, device=pos.device)
        cell64.copy_(state.cell[0].mT)
        fresh = not self._s_built
        if fresh:
            self._s_build(state, pos)
        self._s_check(state, pos, cell64)
        sent = None if fresh else self._send_flags(self.s_expired)
        dt = pos.dtype
        energy = torch.empty(1, dtype=dt, device=state.device) if energy is None else energy
        forces = torch.empty_like(pos) if forces is None else forces
        if not self._compute_stress:
            stress = None
        elif stress is None:
            stress = torch.empty((1, 3, 3), dtype=dt, device=state.device)
        flags = L.OUT_FORCES | (L.OUT_STRESS if stress is not None else 0)
        m = self.model

        def evaluate(skip=None):
            L.call("tsb_verlet_forces_unless", m.kind, L.ptr(m.table), m.n_species,
                   L.ptr(self.s_list), L.ptr(self.s_counts), state.n_atoms, L.ptr(cell64),
                   L.dtype_code(dt), m.cutoff, flags, L.ptr(energy), L.ptr(forces),
                   L.ptr(stress), L.ptr(skip), L.ptr(self.s_ws), self.s_ws.numel(),
                   L.stream_ptr(state.device))

        try:
            evaluate(None if fresh else self.s_expired)
        finally:  # (the host buffer is in use until it has been read)
            expired = sent is not None and self._read_flags(sent)[0]
        if expired:
            self._s_build(state, pos)
            self._s_check(state, pos, cell64)
            evaluate()
        out = {"energy": energy, "forces": forces}
        if stress is not None:
            out["stress"] = stress
        return out

    # ------------------------------------------------------------------ API
    @property
    def list_counts(self) -> torch.Tensor:
        """Neighbour-list entries per atom (slot order on the batched path) of the
        engine used by the last call."""
        return self.s_counts if self._last_single else self.counts

    def forward(self, state, **_kw) -> dict[str, torch.Tensor]:
        self._last_single = self._single_ok(state)
        if self._last_single:
            return self._single_forward(state)
        dev, dt = state.positions.device, state.positions.dtype
        n, n_sys = state.n_atoms, state.n_systems
        energy = torch.empty(n_sys, dtype=dt, device=dev)
        forces = torch.empty((n, 3), dtype=dt, device=dev)
        stress = (torch.empty((n_sys, 3, 3), dtype=dt, device=dev)
                  if self._compute_stress else None)
        energies = torch.empty(n, dtype=dt, device=dev) if self.per_atom_energies else None
        stresses = (torch.empty((n, 3, 3), dtype=dt, device=dev)
                    if self.per_atom_stresses else None)
        self._run(state, energy, forces, stress, energies, stresses, None)
        out = {"energy": energy, "forces": forces}
        if stress is not None:
            out["stress"] = stress
        if energies is not None:
            out["energies"] = energies
        if stresses is not None:
            out["stresses"] = stresses
        return out

    def forward_into(self, state, *, energy, forces, stress=None, sys_active=None):
        """Write energy/forces(/stress) of the systems with ``sys_active`` != 0 into
        existing contiguous buffers; the other systems' entries are left untouched."""
        for t in (energy, forces, stress):
            if t is not None and not t.is_contiguous():
                raise ValueError("forward_into needs contiguous output buffers")
        if sys_active is None and self._single_ok(state):
            # one large system: its own kernels, writing into the buffers (or copied
            # into ones of another dtype)
            self._last_single = True
            shapes = ((energy, (1,)), (forces, tuple(state.positions.shape)),
                      (stress, (1, 3, 3)))
            if all(t is None or (t.dtype == state.positions.dtype and tuple(t.shape) == shape
                                 and t.device == state.positions.device)
                   for t, shape in shapes):
                self._single_forward(state, energy, forces, stress)
                return
            out = self._single_forward(state)
            energy.copy_(out["energy"])
            forces.copy_(out["forces"])
            if stress is not None and "stress" in out:
                stress.copy_(out["stress"])
            return
        self._last_single = False
        self._run(state, energy, forces, stress if self._compute_stress else None, None, None,
                  sys_active)
