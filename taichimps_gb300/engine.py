"""
The fused step engine behind ``Simulation.run``.

One step of Simulation._sub_step_inner (simulation.py:205-247) with fix
nve/sphere, optionally damping/cundall and deform/pressure, becomes three
kernels (tmps_fused_a, tmps_fused_c, tmps_fused_servo; two where no servo runs)
that decide on the device whether the step needs a neighbor rebuild; in the
FP64 form without a servo, fixed granular walls add a kernel after the contacts
(tmps_fused_walls).  Steps are queued in
chunks (replayed as CUDA graphs) with one host synchronisation per chunk.
When a step finds it needs a rebuild, every later launch of the chunk does
nothing; the host then rebuilds exactly as the reference does at that step
(save history, wrap, build, restore history), finishes the step, and
carries on.

Two precisions:
  "fp64"  every operation FP64 (the plain FP64 form);
  "mixed" FP32 contact arithmetic and per-atom force accumulation;
          positions (offsets from each atom's cell origin), velocities and
          angular velocities as double-word FP32 (hi + lo, ~48 bits) updated
          with error-free transforms; the contact histories as double words
          too while the run lasts (doubles before a rebuild carries them over
          and at the end); virial partials as double words, their totals --
          what the servo reads -- in FP64.
"""

from __future__ import annotations

import ctypes
import weakref

import numpy as np
import torch

from . import _device, _lib
from .EXTRA_FIX.damping_cundall import FixDampingCundall
from .EXTRA_FIX.deform_pressure import FixDeformPressure
from .EXTRA_FIX.wall_gran import FixWallGran
from .EXTRA_FIX.wall_gran_region import FixWallGranRegion


def fusable(sim, walls: bool = False) -> bool:
    """The configurations the fused step covers.  `walls`: granular walls too, where they stand still,
    follow any damping in the list of fixes (their force is not damped) and no servo reads the virial;
    up to the number one kernel takes."""
    if sim.integrator is None or sim.pair_style is None or sim.neighbor is None or sim.history is None:
        return False
    kinds = [type(f) for f in sim.fixes]
    on_walls = [i for i, k in enumerate(kinds) if k in (FixWallGran, FixWallGranRegion)] if walls else []
    if on_walls:
        if len(on_walls) > _lib.MAX_FUSED_WALLS or FixDeformPressure in kinds:
            return False
        if FixDampingCundall in kinds[on_walls[0]:]:
            return False
        if any(getattr(sim.fixes[i], "wiggle_amplitude", 0.0) != 0.0 for i in on_walls):
            return False
        kinds = [k for i, k in enumerate(kinds) if i not in on_walls]
    if any(k not in (FixDampingCundall, FixDeformPressure) for k in kinds):
        return False
    if kinds.count(FixDampingCundall) > 1 or kinds.count(FixDeformPressure) > 1:
        return False
    # damping must act on the pair force before the servo reads the virial: the
    # reference calls post_force hooks (Cundall) and end_of_step hooks (servo) in
    # that order regardless of insertion order, so any order is fine here.
    return True


class FusedEngine:
    # kernels per step: A, C, S (C is two launches on the pair path; walls add one, no servo takes S off)
    LAUNCHES_PER_STEP = 3
    MAX_PAIRS = 2**31 - 64  # pair indices carry one more bit

    def __init__(self, sim, precision: str = "fp64", chunk: int = 64, graphs: bool = True,
                 cull: bool = True, launch_shape: tuple[int, int] | None = None,
                 contact_path: str | None = None) -> None:
        if precision not in ("fp64", "mixed"):
            raise ValueError("precision must be 'fp64' or 'mixed'")
        if contact_path is None:
            contact_path = getattr(sim, "contact_path", "auto")
        if contact_path not in ("auto", "screened", "rows"):
            raise ValueError("contact_path must be 'auto', 'screened' or 'rows'")
        # the Simulation keeps its last engine (Simulation.last_engine); the engine refers back
        # weakly, so a finished run's device memory goes with the Simulation instead of waiting
        # for the cycle collector
        self._sim = weakref.ref(sim)
        self.precision = precision
        self.mixed = precision == "mixed"
        self.chunk = int(chunk)
        self.dev = _device.device()
        self.cundall = next((f for f in sim.fixes if isinstance(f, FixDampingCundall)), None)
        self.deform = next((f for f in sim.fixes if isinstance(f, FixDeformPressure)), None)
        self.walls = [f for f in sim.fixes if type(f) in (FixWallGran, FixWallGranRegion)]
        self._eng = _device.struct_buffer(_lib.Engine())
        self.status = torch.zeros(1, dtype=torch.int32, device=self.dev)
        self._dummy_servo = _device.struct_buffer(_lib.Servo())
        self._n = -1
        self.rebuilds = 0
        self._target = 0  # the step run() goes to
        self._stepped = False  # whether run() was called since begin()
        self._interval = self.chunk  # steps between the last two builds
        # A chunk of `chunk` steps is captured once as a CUDA graph and replayed;
        # a rebuild swaps buffers, so the graph is captured again after one.
        self.graphs = bool(graphs)
        # C skips 32-atom groups whose gap bound rules out any contact (exact;
        # off screens every group, with bit-identical results)
        self.cull = bool(cull)
        # C's path: "screened" (tmps_fused_c) rules contact-free 32-atom groups out and runs the contacts
        # of the rest 32 at a time, each for both of its atoms; "rows" (tmps_fused_c_pairs) runs every
        # contact once and sums every atom's row from the pairs' records.  "auto" picks rows at a build
        # where more than half of the atoms touch or overlap at the build positions (their gap bound is
        # <= 0): there the screen rules out little and half of the contact arithmetic is saved; on dilute
        # states the screen reads a few bytes per group where rows would read every list entry.  Steps
        # screened and by rows, jammed packings with 95, 76, 57 and 47 % of the atoms touching (the others
        # shrunk out of contact above a height): a million spheres, mixed 331, 281, 218, 194 and 223, 197,
        # 169, 148 us, FP64 2.86, 2.28, 1.76, 1.47 and 1.15, 0.98, 0.77, 0.66 ms; 15,600, mixed 32, 30, 30,
        # 30 and 25, 24, 24, 23 us, FP64 107, 83, 82, 83 and 54, 56, 53, 52 us; 343 spheres alike.  Both
        # paths sum each atom's contacts in slot order with the same per-contact code; only the order of
        # the virial sums differs.
        self.contact_path = contact_path
        self.rows = contact_path == "rows"
        # launch shape (tmps_fused_shape): 32-atom groups per warp of A and of C, 0 = the default grid;
        # it fixes the order of the virial sum, so equal shapes give bit-identical runs
        shape = getattr(sim, "launch_shape", (0, 0)) if launch_shape is None else launch_shape
        self.launch_shape = (int(shape[0]), int(shape[1]))
        self._graph = None
        self._graph_key = None
        # the arguments of the last chunk that ran as plain launches; the next chunk with the same
        # arguments is captured (`capture_first`: capture at the first chunk instead)
        self._seen_key = None
        self.capture_first = False
        self._hist_dw = False
        # the rows path's buffer (tmps_pairs_*): the pairs of the current build and, while `_in_pairs`,
        # the contact histories
        self.pairs: torch.Tensor | None = None
        self.npairs = 0
        self._in_pairs = False
        self.graph_replays = 0
        self.graph_kernel_launches = 0
        # (engine record, status) as the last run() left them, while nothing has been launched since:
        # the next run() starts from it instead of another synchronisation
        self._known = None

    @property
    def sim(self):
        sim = self._sim()
        if sim is None:
            raise RuntimeError("the Simulation of this fused engine no longer exists")
        return sim

    # ------------------------------------------------------------ storage

    def _alloc(self, n: int) -> None:
        if n == self._n:
            return
        # every per-atom array here is written in full by tmps_fused_prepare before any kernel reads
        # it: left unset, in one allocation for the mixed form's eleven
        self.rinv = None if self.mixed else torch.empty((2, n), dtype=torch.float64, device=self.dev)
        style, mixed = int(self.sim.pair_style.params.style), 1 if self.mixed else 0
        self._shape(n)
        self.part = torch.zeros(int(_device.lib().tmps_fused_scratch_bytes(n, style, mixed)), dtype=torch.uint8,
                                device=self.dev)
        if self.mixed:
            # (name, FP32 words per atom, shape); each slice starts on a 256-byte boundary
            parts = [("pos32", 4, (n, 4)), ("pos32lo", 4, (n, 4)), ("lo32", 4, (n, 4)), ("wlz32", 1, (n,)),
                     ("inv32", 2, (n, 2)), ("vel32", 4, (n, 4)), ("om32", 4, (n, 4)), ("f32", 3, (3, n)),
                     ("t32", 3, (3, n)), ("o0", 3, (3, n)), ("cell32", 1, (n,))]
            r64 = lambda w: (w + 63) // 64 * 64
            flat = torch.empty(sum(r64(w * n) for _, w, _ in parts), dtype=torch.float32, device=self.dev)
            off = 0
            for name, w, shape in parts:
                t = flat[off:off + w * n].view(shape)
                setattr(self, name, t.view(torch.int32) if name == "cell32" else t)
                off += r64(w * n)
        self._n = n

    def _shape(self, n: int) -> None:
        """Grids of A and C for n atoms under this engine's launch shape; nblocks = virial partials."""
        a_b, c_b = ctypes.c_int32(), ctypes.c_int32()
        style, mixed = int(self.sim.pair_style.params.style), 1 if self.mixed else 0
        _lib.check(_device.lib().tmps_fused_shape(n, style, mixed, self.launch_shape[0], self.launch_shape[1],
                                                  ctypes.byref(a_b), ctypes.byref(c_b)), "tmps_fused_shape")
        self.a_blocks, self.c_blocks = a_b.value, c_b.value
        self.nblocks = self.a_blocks + self.c_blocks

    def set_launch_shape(self, shape: tuple[int, int]) -> None:
        """Change the launch shape between steps (the scratch holds any shape's partials)."""
        self._known = None
        self.launch_shape = (int(shape[0]), int(shape[1]))
        if self._n < 0:
            return
        self._shape(self._n)
        e = self._engine_state()
        e.nblocks, e.ablocks = self.nblocks, self.a_blocks
        _device.push_struct(self._eng, e)
        self._graph = None

    def atoms(self) -> _lib.Atoms:
        s = self.sim.atom.cstruct()
        s.rinv = None if self.rinv is None else self.rinv.data_ptr()
        if self.mixed:
            s.pos32, s.vel32, s.om32 = self.pos32.data_ptr(), self.vel32.data_ptr(), self.om32.data_ptr()
            s.f32, s.torque32, s.o0_32 = self.f32.data_ptr(), self.t32.data_ptr(), self.o0.data_ptr()
            s.cell32 = self.cell32.data_ptr()
            s.pos32lo = self.pos32lo.data_ptr()
            s.lo32, s.wlz32, s.inv32 = self.lo32.data_ptr(), self.wlz32.data_ptr(), self.inv32.data_ptr()
        return s

    def _servo_ptr(self) -> int:
        return self.deform._dservo.data_ptr() if self.deform is not None else self._dummy_servo.data_ptr()

    # ------------------------------------------------------------ lifecycle

    def begin(self, stop_step: int | None = None, steps: int | None = None) -> None:
        """After Simulation.init_simulation(): hand the state to the fused step.  `stop_step`: fused
        launches do nothing once the step count reaches it (batched runs).  `steps`: how many steps
        will follow, where the caller knows."""
        self._known = None
        sim = self.sim
        atom, nl = sim.atom, sim.neighbor
        n = atom.nlocal
        self._alloc(n)
        self._stepped = False
        if sim.pair_style.params.rolling_id:
            sim.history.enable_rolling()
        if self.mixed:
            g = nl.grid_dim
            if np.any(g > 1023):
                raise NotImplementedError("the mixed form packs cell coordinates in 10 bits (<= 1023 bins per axis)")
        e = _lib.Engine()
        e.step = self._begun = sim.timestep
        e.last_build_step = nl.last_build_step
        e.delay, e.every, e.check = int(nl.delay), max(1, int(nl.every)), 1 if nl.check else 0
        e.cundall = 1 if self.cundall is not None else 0
        e.servo = 1 if self.deform is not None else 0
        # without a servo the contact kernel itself ends the step (two launches a step, not three)
        self.fold = self.deform is None and n > 0
        e.fold = 1 if self.fold else 0
        e.walls = 1 if self.walls else 0
        self._wall_args = (_lib.FusedWall * len(self.walls))() if self.walls else None
        for k, f in enumerate(self.walls):
            f.ready(atom)
            self._wall_args[k] = _lib.FusedWall(f.params(), f.shear.data_ptr(), f.touch.data_ptr(), f.max_atoms,
                                                1 if f.history_update else 0)
        e.mixed = 1 if self.mixed else 0
        e.nblocks, e.ablocks = self.nblocks, self.a_blocks
        e.dt = float(sim.dt)
        if self.cundall is not None:
            e.gamma_lin, e.gamma_ang = self.cundall.gamma_lin, self.cundall.gamma_ang
        e.trigger_sq = 0.25 * nl.skin * nl.skin
        e.remap_scale[0] = e.remap_scale[1] = e.remap_scale[2] = 1.0
        e.stop_step = (1 << 62) if stop_step is None else int(stop_step)
        _device.push_struct(self._eng, e)
        if self.deform is not None:
            # the run counters only; the rest of the servo record stays as the device has it
            fx = self.deform
            sv = _lib.Servo()
            sv.nsteps, sv.nsteps_total, sv.step_count, sv.nevery = fx.nsteps, fx.nsteps_total, fx.step_count, fx.nevery
            _device.push_fields(fx._dservo, sv, "nsteps", "nevery")
        self._prepare(self.chunk if steps is None else int(steps))
        log = self.deform.pressure_log if self.deform is not None else None
        rc = _device.lib().tmps_fused_pressure_log(self._eng.data_ptr(), None if log is None else log.data_ptr(),
                                                   0 if log is None else len(log), _device.stream())
        _lib.check(rc, "tmps_fused_pressure_log")
        # (the mixed form's first half-kick takes the setup forces, which tmps_fused_prepare copied
        # into f32, t32)
        self.status.zero_()
        # the record as pushed above, in the fields run() reads (step, aborted), and a clear status:
        # the first run() starts without a synchronisation
        self._known = (e, 0)

    def _prepare(self, steps: int) -> None:
        """Split state and per-step constants for the current list, then the per-group
        contact bounds C uses to skip groups that cannot touch.  `steps`: as many will be made on it."""
        self._known = None
        sim = self.sim
        nl = sim.neighbor
        L, st = _device.lib(), _device.stream()
        atoms = self.atoms()
        rc = L.tmps_fused_prepare(atoms, sim.domain.dbox, self._eng.data_ptr(), nl.cell_of.data_ptr(), st)
        _lib.check(rc, "tmps_fused_prepare")
        rc = L.tmps_fused_bounds(atoms, sim.history.cstruct(nl), sim.domain.dbox, self._eng.data_ptr(),
                                 sim.pair_style.params, 1 if self.cull else 0, self.part.data_ptr(), st)
        _lib.check(rc, "tmps_fused_bounds")
        # one synchronisation for what the host needs before the steps: the counts of touching atoms
        # and of pairs (the contact path) and the status of a neighbor build that did not wait for the
        # device.  The FP64 form asks for the counts once a list, with that status: a run of a few steps
        # on the same list would wait longer for them (90 us a call) than for its steps.  The mixed form
        # asks again, as contacts that formed since the build change its path.  On a jammed packing its
        # pairs are numbered in 50-180 us and save 6 us a step of 15,600 spheres, 17 of 125,000 and 108
        # of a million: the fewest steps stay screened and do not ask (one step of 15,600 spheres on the
        # list of the run before 0.80 -> 0.63 ms, of a million 1.64 -> 1.53).
        path = self.contact_path
        if path == "auto" and self.mixed and steps < 5 and steps * self._n <= 1_000_000:
            path = "screened"
        ask = path != "screened" and (self.mixed or nl.counts is None)
        items = []
        if ask:
            off = _lib.Engine.touching.offset
            items.append((self._eng[off:], None))
        if nl.status_pending:
            items.append((nl.status, None))
        got = _device.pull_many(items) if items else []
        if nl.status_pending:
            nl.check_status(int(got[-1].view(np.int32)[0]))
        if ask:
            # the bounds kernel counted the atoms whose gap bound is <= 0, and the pairs, into the
            # engine record
            at = _lib.Engine.pairs.offset - off
            nl.counts = int(got[0][:4].view(np.int32)[0]), int(got[0][at:at + 8].view(np.int64)[0])
        self.rows = False
        if path != "screened":
            touching, self.npairs = nl.counts
            self.rows = path == "rows" or touching * 2 > self._n
            self.rows = self.rows and 0 < self._n and self.npairs <= self.MAX_PAIRS and self._build_pairs()
        if not self.rows:
            self._history_form(True)

    def _build_pairs(self) -> bool:
        """The rows path's pair buffer for the current list, with the contact histories; False (and nothing
        changed) where the device has no room for it: the screened path, which keeps no records, has the
        same results."""
        sim = self.sim
        nl, par, L = sim.neighbor, sim.pair_style.params, _device.lib()
        mixed = 1 if self.mixed else 0
        need = int(L.tmps_pairs_bytes(self._n, nl.slots, self.npairs, int(par.style), mixed, int(par.rolling_id)))
        if self.pairs is None or self.pairs.numel() < need:
            self.pairs = None
            try:
                self.pairs = torch.empty(need, dtype=torch.uint8, device=self.dev)
            except torch.OutOfMemoryError:
                return False
        _lib.check(L.tmps_pairs_build(sim.history.cstruct(nl), par, self.npairs, mixed, self.pairs.data_ptr(),
                                      _device.stream()), "tmps_pairs_build")
        self._in_pairs = True
        return True

    def _history_back(self) -> None:
        """The contact histories back in the list's rows as doubles, both copies of each."""
        if self._in_pairs:
            sim = self.sim
            _lib.check(_device.lib().tmps_pairs_history(sim.history.cstruct(sim.neighbor), sim.pair_style.params,
                                                        self.npairs, 1 if self.mixed else 0, self.pairs.data_ptr(),
                                                        _device.stream()), "tmps_pairs_history")
            self._in_pairs = False
        self._history_form(False)

    def _history_form(self, dw: bool) -> None:
        """The mixed form keeps the contact histories as FP32 double words while it runs, and
        hands them back as doubles (before a rebuild carries them over, and at the end)."""
        if not self.mixed or self._hist_dw == dw:
            return
        sim = self.sim
        rc = _device.lib().tmps_mixed_history(sim.history.cstruct(sim.neighbor), 1 if dw else 0, _device.stream())
        _lib.check(rc, "tmps_mixed_history")
        self._hist_dw = dw

    def _launch_step(self, L, st, atoms, nl_struct, params) -> None:
        self._known = None
        dbox, eng = self.sim.domain.dbox, self._eng.data_ptr()
        with _device.timed("fused_a"):
            rc = L.tmps_fused_a(atoms, dbox, eng, self.a_blocks, self.part.data_ptr(), st)
        _lib.check(rc, "tmps_fused_a")
        with _device.timed("fused_c"):
            self._launch_c(L, st, atoms, nl_struct, params)
        if self.fold:
            return
        with _device.timed("fused_s"):
            rc = L.tmps_fused_servo(dbox, self._servo_ptr(), eng, self.part.data_ptr(), self.status.data_ptr(), st)
        _lib.check(rc, "tmps_fused_servo")

    def _launch_c(self, L, st, atoms, nl_struct, params) -> None:
        dbox, eng, part = self.sim.domain.dbox, self._eng.data_ptr(), self.part.data_ptr()
        if self.rows:
            _lib.check(L.tmps_fused_c_pairs(atoms, nl_struct, dbox, eng, params, self.c_blocks, part, self.npairs,
                                            self.pairs.data_ptr(), st), "tmps_fused_c_pairs")
        else:
            _lib.check(L.tmps_fused_c(atoms, nl_struct, dbox, eng, params, self.c_blocks, part, st), "tmps_fused_c")
        if self.walls:
            with _device.timed("wall"):
                rc = L.tmps_fused_walls(atoms, eng, self._wall_args, len(self.walls), part, st)
            _lib.check(rc, "tmps_fused_walls")

    def instance(self, a_first: int, a_blocks: int, c_first: int, c_blocks: int) -> _lib.Instance:
        """This system's descriptor for a batched run (tmps_instance)."""
        sim = self.sim
        d = _lib.Instance()
        d.a = self.atoms()
        d.nl = sim.history.cstruct(sim.neighbor)
        d.p = sim.pair_style.params
        d.box = sim.domain.dbox
        d.eng = self._eng.data_ptr()
        d.servo = self._servo_ptr()
        d.scratch = self.part.data_ptr()
        d.a_first, d.a_blocks, d.c_first, d.c_blocks = a_first, a_blocks, c_first, c_blocks
        return d

    def _engine_state(self) -> _lib.Engine:
        return _device.pull_struct(self._eng, _lib.Engine)

    def _engine_and_status(self) -> tuple[_lib.Engine, int]:
        """The engine record and the status word with one synchronisation (two copies into
        page-locked memory)."""
        nbytes = self._eng.numel()
        if getattr(self, "_pull_host", None) is None or self._pull_host.numel() != nbytes + 4:
            self._pull_host = torch.empty(nbytes + 4, dtype=torch.uint8, pin_memory=True)
        h = self._pull_host
        h[:nbytes].copy_(self._eng, non_blocking=True)
        h[nbytes:].copy_(self.status.view(torch.uint8), non_blocking=True)
        torch.cuda.current_stream().synchronize()
        raw = h.numpy()
        return _lib.Engine.from_buffer_copy(raw[:nbytes].tobytes()), int(raw[nbytes:].view(np.int32)[0])

    def run(self, nsteps: int) -> None:
        """Advance `nsteps` steps."""
        sim = self.sim
        L = _device.lib()
        st = _device.stream()
        if self._stepped and not self.mixed and self._n > 0:
            # the FP64 update's kept kinetic sums (none since the last bounds, if no step has been made)
            # hold while only its own steps change a velocity
            _lib.check(L.tmps_fused_forget_kinetic(self._n, self.part.data_ptr(), st), "tmps_fused_forget_kinetic")
        self._stepped = True
        start = sim.timestep
        target = self._target = start + int(nsteps)
        while True:
            if self._known is not None:
                e, status = self._known
                self._known = None
            else:
                e, status = self._engine_and_status()  # after a chunk: its status too, in the same copy
            self._check_status(status)
            done = int(e.step)
            if e.aborted:
                self._rebuild_step(done + 1)
                continue
            if done >= target:
                self._known = (e, status)
                break
            count = min(self.chunk, target - done)
            if self._interval < self.chunk:
                # rebuilds come sooner than a chunk ends, and every launch queued past one is idle work: as
                # many steps as the last interval held and an eighth more, then half of what has passed
                since, held = done - int(e.last_build_step), self._interval + self._interval // 8 + 1
                count = min(count, held - since if since < held else max(4, since // 2))
            if self.graphs and count == self.chunk and _device.TIMED is None:
                self._replay_chunk(L)
            else:
                atoms = self.atoms()
                nl_struct = sim.history.cstruct(sim.neighbor)
                params = sim.pair_style.params
                for _ in range(count):
                    self._launch_step(L, st, atoms, nl_struct, params)
        sim.timestep = target

    def _replay_chunk(self, L) -> None:
        """One chunk of steps as a CUDA graph (captured on first use and after a rebuild; the launch
        arguments are built only for a capture)."""
        self._known = None
        sim = self.sim
        key = (sim.neighbor.build_count, sim.atom.buffers.xr.data_ptr(), sim.history.touch.data_ptr(),
               sim.neighbor.nbr.data_ptr(), self.rows, self.pairs.data_ptr() if self.rows else 0, self.chunk)
        if self._graph is None or self._graph_key != key:
            self._graph = None
            atoms = self.atoms()
            nl_struct = sim.history.cstruct(sim.neighbor)
            params = sim.pair_style.params
            if self._seen_key != key and not self.capture_first:
                # a chunk whose arguments have not been seen before runs as plain launches: the device
                # starts on it at once, where a capture would hold it idle, and a run of one chunk
                # (or one chunk between rebuilds) never pays for a graph it would replay once
                self._seen_key = key
                st = _device.stream()
                for _ in range(self.chunk):
                    self._launch_step(L, st, atoms, nl_struct, params)
                return

            def chunk():
                st = _device.stream()
                for _ in range(self.chunk):
                    self._launch_step(L, st, atoms, nl_struct, params)

            self._graph, self._graph_key = _device.capture_graph(chunk), key
        self._graph.replay()
        self.graph_replays += 1
        self.graph_kernel_launches += self.chunk * (self.LAUNCHES_PER_STEP + (1 if self.rows else 0) - (1 if self.fold else 0)
                                                    + (1 if self.walls else 0))

    def cull_stats(self) -> tuple[int, int]:
        """(32-atom groups, groups the contact bound rules out right now), from the
        device state.  No reference counterpart; for reports and tests."""
        n = self._n
        ng = (n + 31) // 32
        e = self._engine_state()
        if not e.cull or ng == 0:
            return ng, 0
        # scratch layout: flag words (ng + 1, 256-byte aligned), then the gaps
        off = ((ng + 1) * 4 + 255) // 256 * 256
        gap = self.part[off:off + 4 * ng].view(torch.float32).cpu().numpy()
        f32 = np.float32
        md = np.sqrt(np.array([e.maxd2_bits], dtype=np.uint32).view(np.float32)[0])
        thr = (f32(2.0) * md) * f32(1.0001) + f32(e.shift_bound) + f32(e.cull_tol)
        return ng, int(np.count_nonzero(gap > thr))

    def flagged_count(self) -> int:
        """Atoms C flagged (some neighbor within reach of contact) in the last step, from the flag
        words.  No reference counterpart; for reports and tests."""
        ng = (self._n + 31) // 32
        if ng == 0:
            return 0
        w = self.part[:4 * ng].view(torch.int32).cpu().numpy().view(np.uint32)
        return int(np.unpackbits(w.view(np.uint8)).sum())

    def _check_status(self, st: int | None = None) -> None:
        st = int(self.status.item()) if st is None else st
        if st & _lib.STATUS_BOX_NONPOSITIVE and self.deform is not None:
            self.deform.status.fill_(st)
            self.deform.status_clean = False
            self.deform.check_status()

    def _rebuild_step(self, s: int) -> None:
        """Step `s` has had its first half-kick and drift; rebuild, then finish it."""
        self._known = None
        sim = self.sim
        L = _device.lib()
        st = _device.stream()
        atom, nl = sim.atom, sim.neighbor
        self.rebuilds += 1
        sim.timestep = s
        nl.current_step = s
        if self.mixed:
            _lib.check(L.tmps_mixed_unpack(self.atoms(), sim.domain.dbox, st), "tmps_mixed_unpack")
        self._history_back()
        sim.domain.mark_device_authoritative()
        sim.domain.pull()
        sim.history.save_state(atom, nl)
        sim.domain.pbc(atom)
        nl.build(atom, defer_check=True)  # its status is read with the engine's next pull
        sim.history.restore_state(atom, nl)
        e = self._engine_state()
        e.aborted = 0
        e.disp_stamp = 0
        self._interval = s - int(e.last_build_step)
        e.last_build_step = s
        _device.push_struct(self._eng, e)
        if atom.nlocal != self._n:
            raise RuntimeError("atom count changed during a fused run")
        self._prepare(max(1, min(self._interval, self._target - s)))
        atoms = self.atoms()
        nl_struct = sim.history.cstruct(nl)
        dbox, eng = sim.domain.dbox, self._eng.data_ptr()
        self._launch_c(L, st, atoms, nl_struct, sim.pair_style.params)
        if not self.fold:
            _lib.check(L.tmps_fused_servo(dbox, self._servo_ptr(), eng, self.part.data_ptr(),
                                          self.status.data_ptr(), st), "tmps_fused_servo")

    def finish(self) -> None:
        """Settle pending updates and hand the state back to the per-hook path."""
        self._known = None
        # the captured graph goes now, not whenever the engine is collected (which may be
        # during a later capture)
        self._graph = self._graph_key = None
        sim = self.sim
        L = _device.lib()
        st = _device.stream()
        atoms = self.atoms()
        _lib.check(L.tmps_fused_settle(atoms, sim.domain.dbox, self._eng.data_ptr(), st), "tmps_fused_settle")
        if self.mixed:
            _lib.check(L.tmps_mixed_unpack(atoms, sim.domain.dbox, st), "tmps_mixed_unpack")
        self._history_back()
        sim.domain.mark_device_authoritative()
        # the engine record, the status word, the box and the servo record: one synchronisation
        items = [(self._eng, _lib.Engine), (self.status, None), (sim.domain.dbox_tensor, _lib.Box)]
        if self.deform is not None:
            items.append((self.deform._dservo, _lib.Servo))
        got = _device.pull_many(items)
        e, status, box = got[0], int(got[1].view(np.int32)[0]), got[2]
        sim.domain.take_pulled(box)
        for f in self.walls:
            f.passed(int(e.step) - self._begun, float(sim.dt))
        self._begun = int(e.step)
        sim.timestep = int(e.step)
        sim.neighbor.current_step = int(e.step)
        sim.neighbor.last_build_step = int(e.last_build_step)
        for fx in sim.fixes:
            fx.timestep = sim.timestep
        if self.deform is not None:
            sv = got[3]
            self.deform.nsteps, self.deform.step_count = int(sv.nsteps), int(sv.step_count)
        if sim.integrator is not None:
            sim.integrator.timestep = sim.timestep
        self._check_status(status)
