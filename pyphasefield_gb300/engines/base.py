"""GB300Engine: the device half of every engine in this package.

Mixed into a Simulation subclass (this package's, or the reference's own
pyphasefield.simulation.Simulation through make_engines), it replaces the
reference's per-step loop (Simulation.simulate, simulation.py:245-271) and
its numba device utilities (ppf_gpu_utils.send_fields_to_GPU /
retrieve_fields_from_GPU / apply_boundary_conditions, ppf_gpu_utils.py:
396-514):

* fields live on the device as float32 (default) or float64, interior only,
  in two ping-pong buffer sets; the boundary rule is fused into every
  kernel's tile load, so apply_boundary_conditions is a no-op on device;
* simulate(n) advances n steps in captured CUDA graphs of `graph_chunk`
  steps (each launch with programmatic dependent launch), split at
  autosave boundaries so autosave cadence and time_step_counter behave as in
  the reference;
* send_fields_to_GPU / retrieve_fields_from_GPU move the interiors between
  Field.data (float64, ghosts refilled on the host) and the device.

User-data keys added to the reference's: precision ("fp32" | "fp64"),
temporal_depth (steps per HBM pass, 2-D Diffusion/Allen-Cahn; 1, the
default, leaves the steps per pass to the engine), tile
((tile_x, tile_y) or None; Warren1995: (0, rows per warp band), chosen by
grid size when None), zchunk (planes per warp or CTA, 3-D), autotune (bool: time the
launch shapes on scratch copies and cache the fastest), bulk_shortcut
(bool, Warren1995), pdl (bool), use_graph (bool), graph_chunk (int),
check_status (bool, default True).

Failure detection: after every chunk of steps (inside the captured graph)
the engine runs the NaN/Inf sentinel over its fields,
moves the library's status bits (a bounded barrier wait that gave up, a
Cahn-Hilliard range overflow) into its own sticky status word and writes
that word to pinned host memory, in one launch (ppf_watch_*). The host
reads the copy at the next chunk boundary (waiting for the chunk before the
last, so the device stays a chunk ahead), at every autosave and in
retrieve_fields_from_GPU, and raises EngineFault on any set bit: a run never
carries on from a state a kernel reported as corrupt. The library's word is
shared by every engine on a device; whichever engine collects it first
reports the fault.
"""
from __future__ import annotations

import collections
import contextlib
import ctypes as C
import gc
import hashlib
import inspect
from pathlib import Path

import numpy as np
import torch

from .. import _lib as L
from ..device import DeviceGrid, boundary_struct, ptr, require_cuda, tiling_struct
from ..simulation import fill_ghosts_host

COMMON_DEFAULTS = dict(precision="fp32", temporal_depth=1, tile=None, pdl=True,
                       use_graph=True, graph_chunk=64, check_status=True)

#: captured graphs kept per engine (one per distinct parameter set)
MAX_GRAPHS = 8

#: user_data values that stand for themselves in a graph's key
_PLAIN = frozenset((bool, int, float, str, type(None)))

_STATUS_NAMES = ((L.PPF_STATUS_TIMEOUT, "a bounded barrier wait timed out (tile not written)"),
                 (L.PPF_STATUS_NONFINITE, "a field holds NaN or Inf"),
                 (L.PPF_STATUS_RANGE, "a value left the kernel's representable range"),
                 (L.PPF_STATUS_NOT_CONVERGED, "an iterative solve did not converge"))


try:
    from torch.cuda import nvtx as _nvtx
except Exception:  # pragma: no cover - torch without NVTX
    _nvtx = None


@contextlib.contextmanager
def nvtx_range(name: str):
    """NVTX range on the host timeline (shown by Nsight Systems / ncu
    --nvtx): simulate calls, graph replays, eager passes, transfers."""
    if _nvtx is None:
        yield
        return
    _nvtx.range_push(name)
    try:
        yield
    finally:
        _nvtx.range_pop()


def _device_of(stream):
    """Context of a launch into `stream`, whose device has to be current; nothing
    where it is (entering a device or a stream costs the host 10 us)."""
    if torch.cuda.current_device() == stream.device.index:
        return contextlib.nullcontext()
    return torch.cuda.device(stream.device)


def _save_npz(sim, step: int) -> None:
    """The reference's checkpoint format: np.savez of every field's interior
    keyed by field name, to <save_path>/step_<step>.npz."""
    if not sim._save_path:
        print("self._save_path not defined, aborting save!")
        return
    loc = Path(sim._save_path)
    loc.mkdir(parents=True, exist_ok=True)
    np.savez(str(loc) + "/step_" + str(int(step)), **{f.name: f.get_cells() for f in sim.fields})


class EngineFault(RuntimeError):
    """A kernel reported a fault through the device status word."""

    def __init__(self, bits: int, where: str):
        self.bits = bits
        names = [n for b, n in _STATUS_NAMES if bits & b] or [f"status bits {bits:#x}"]
        super().__init__(f"{where}: " + "; ".join(names))


class GB300Engine:
    #: number of fields the engine advances together
    NFIELDS = 1

    # ------------------------------------------------------------ subclass API
    def _ppf_params(self):
        """Return the ctypes params struct for the library call."""
        raise NotImplementedError

    def _ppf_step(self, src, dst, depth: int, step: int, step_base, stream_ptr):
        """Launch one pass advancing `depth` steps from buffers src to dst."""
        raise NotImplementedError

    #: whether a step reads the step counter (noise drawn per step). An engine
    #: that states False gets step_base = None, also in captured runs.
    USES_STEP = True

    def _ppf_run(self):
        """PpfRun of the engine's steps (model, params, tiling and the model's
        own buffers; the fields and the step are filled in), or None for an
        engine whose steps are launched one by one. A run issues the same
        passes as _ppf_step does."""
        return None

    def __init_subclass__(cls, **kwargs):
        """A class with a _ppf_step of its own is stepped through it: what it
        inherits for another step (_ppf_run, _ppf_auto_depth, USES_STEP =
        False) does not hold for it unless it states it again."""
        super().__init_subclass__(**kwargs)

        def owner(name):
            return next(i for i, c in enumerate(cls.__mro__) if name in c.__dict__)

        step = owner("_ppf_step")
        for name in ("_ppf_run", "_ppf_auto_depth", "USES_STEP"):
            if step < owner(name):
                setattr(cls, name, GB300Engine.__dict__[name])

    def _ppf_max_depth(self) -> int:
        return 1

    def _ppf_auto_depth(self) -> int:
        """Steps a pass takes on its own account while temporal_depth is 1:
        more than 1 where the kernels advance several steps per pass with the
        results of single steps, bit for bit."""
        return 1

    def _ppf_encode(self, j: int, x: np.ndarray) -> np.ndarray:
        """Host value -> stored value of field j (identity by default)."""
        return x

    def _ppf_decode(self, j: int, x: np.ndarray) -> np.ndarray:
        return x

    def _ppf_prepare(self):
        """Engine-specific set-up before the device copy (derived params)."""

    def _ppf_segment_begin(self, nsteps: int, stream):
        """Launches issued before a run of steps (captured in graphs)."""

    def _ppf_segment_end(self, nsteps: int, stream):
        """Host bookkeeping after a run of steps (not captured)."""

    # ------------------------------------------------------------ helpers
    def _ppf_defaults(self):
        for k, v in COMMON_DEFAULTS.items():
            self.user_data.setdefault(k, v)

    @property
    def _ppf_dtype(self):
        p = self.user_data.get("precision", "fp32")
        if p not in ("fp32", "fp64"):
            raise ValueError(f"precision must be 'fp32' or 'fp64', got {p!r}")
        return torch.float32 if p == "fp32" else torch.float64

    def _ppf_ready(self) -> bool:
        return getattr(self, "_ppf_bufs", None) is not None

    def _ppf_setup(self):
        dev = require_cuda()
        if not self.fields or len(self.fields) != self.NFIELDS:
            raise RuntimeError(f"{type(self).__name__} needs {self.NFIELDS} field(s); "
                               "call initialize_fields_and_imported_data() first")
        shape = self.fields[0].get_cells().shape
        self._ppf_release_graphs()
        self._ppf_grid = DeviceGrid(shape, self._ppf_dtype, dev)
        self._ppf_bufs = [[self._ppf_grid.empty() for _ in range(self.NFIELDS)] for _ in range(2)]
        self._ppf_cur = 0
        self._ppf_stream = torch.cuda.Stream(dev)
        self._ppf_bc = boundary_struct(self, self._ppf_grid, self.NFIELDS)
        # step counter; status word and the watch's arrival counter
        words = torch.zeros(2, dtype=torch.int64, device=dev)
        self._ppf_stepctr = words[:1]
        self._ppf_status, self._ppf_watch_counter = words[1:].view(torch.int32).split(1)
        # the buffers' zero fills ran on the current stream
        self._ppf_stream.wait_stream(torch.cuda.current_stream(dev))
        self._ppf_graphs = collections.OrderedDict()
        self._ppf_staging = []
        self._ppf_status_host = torch.zeros(1, dtype=torch.int32, pin_memory=True)
        self._ppf_status_events = collections.deque()
        self._ppf_event_pool = []
        self._uses_gpu = True

    def _ppf_release_graphs(self):
        for g in getattr(self, "_ppf_graphs", {}).values():
            L.call("ppf_graph_destroy", g)
        self._ppf_graphs = collections.OrderedDict()

    # ------------------------------------------------------------ status
    def _ppf_watch(self, stream):
        """The launch issued after a chunk of steps (captured with it): the
        NaN/Inf sentinel on the current fields, the library status bits
        moved into the engine's word, and the word written to pinned host
        memory."""
        if not self.user_data.get("check_status", True):
            return
        bufs = self._ppf_bufs[self._ppf_cur]
        L.call("ppf_watch_f32" if self._ppf_dtype == torch.float32 else "ppf_watch_f64",
               (C.c_void_p * len(bufs))(*[t.data_ptr() for t in bufs]), len(bufs),
               C.byref(self._ppf_grid.grid), self._ppf_status.data_ptr(),
               self._ppf_watch_counter.data_ptr(), self._ppf_status_host.data_ptr(),
               stream.cuda_stream)

    def _ppf_watch_launches(self) -> int:
        """Kernels _ppf_watch launches."""
        return 1 if self.user_data.get("check_status", True) else 0

    def _ppf_mark(self):
        """Records the point after a chunk's status word (host side)."""
        if self.user_data.get("check_status", True):
            ev = self._ppf_event_pool.pop() if self._ppf_event_pool else torch.cuda.Event()
            ev.record(self._ppf_stream)
            self._ppf_status_events.append(ev)

    def _ppf_check_status(self, block: bool, where: str = "simulate"):
        """Raises EngineFault if a chunk reported a fault. block=False waits
        only for chunks two or more behind the newest, so the device keeps
        one chunk queued; block=True waits for everything issued."""
        if not self._ppf_ready():
            return
        evs = self._ppf_status_events
        if block:
            if evs:
                evs[-1].synchronize()
                self._ppf_event_pool.extend(evs)
                evs.clear()
        else:
            while len(evs) > 1:
                ev = evs.popleft()
                ev.synchronize()
                self._ppf_event_pool.append(ev)
        bits = int(self._ppf_status_host.item())
        if bits:
            self.synchronize()
            bits = int(self._ppf_status_host.item())
            with torch.cuda.stream(self._ppf_stream):
                self._ppf_status.zero_()
            self._ppf_stream.synchronize()
            self._ppf_status_host.zero_()
            raise EngineFault(bits, f"{type(self).__name__} {where} (step "
                                    f"{self.time_step_counter})")

    def __del__(self):
        try:
            if getattr(self, "_ppf_stream", None) is not None:
                # work in flight still reads the buffers freed with the engine
                self._ppf_stream.synchronize()
            self._ppf_checkpoint_wait()
            ck = getattr(self, "_ppf_ckpt", None)
            if ck is not None:
                ck["pool"].shutdown(wait=True)
            self._ppf_release_graphs()
        except Exception:
            pass

    def _ppf_tune_candidates(self) -> list:
        """Launch shapes the autotuner may try (user_data updates)."""
        return []

    #: part of the autotuner's cache key, changed with the kernels behind the
    #: candidates: a choice cached for others is made anew
    TUNE_KERNELS = ""

    def _ppf_autotune(self):
        """Pick tile / temporal depth by timing candidates on scratch copies
        of the current fields (user_data["autotune"] = True); the choice is
        cached per kernel, shape, dtype and device (autotune.py)."""
        from .. import autotune

        cands = self._ppf_tune_candidates()
        if len(cands) < 2:
            return
        key = autotune.make_key(type(self).__name__, self._ppf_grid.kshape, self._ppf_dtype,
                                str(len(self.dimensions)) + self.TUNE_KERNELS)
        s = self._ppf_stream
        sp = C.c_void_p(s.cuda_stream)
        with torch.cuda.stream(s):
            scratch = [[t.clone() for t in self._ppf_bufs[self._ppf_cur]] for _ in range(2)]
        saved = {k: self.user_data.get(k) for c in cands for k in c}

        timed = {}  # seconds per step of the passes timed so far

        def measure(cand):
            self.user_data.update(cand)
            # the passes a long run consists of
            depth = max(1, min(int(self.user_data.get("temporal_depth", 1)), self._ppf_max_depth()))
            if depth == 1:
                depth = self._ppf_auto_depth()
            flip = [0]

            def run():
                self._ppf_step(scratch[flip[0]], scratch[1 - flip[0]], depth, 0, None, sp)
                flip[0] ^= 1

            # candidates of the same passes (a depth that is the engine's own) tie,
            # and the first of them is taken
            passes = repr((depth, self.user_data.get("tile"), self.user_data.get("zchunk")))
            if passes not in timed:
                with torch.cuda.stream(s):
                    run()  # a shape the kernel refuses ends here
                timed[passes] = self._ppf_time(run) / depth
            return timed[passes]

        try:
            best = autotune.pick(key, cands, measure)
        finally:
            self.user_data.update(saved)
        self.user_data.update(best)
        self._ppf_graphs_reset()

    def _ppf_time(self, run, passes: int = 8) -> float:
        """Seconds of one run() on the engine's stream, `passes` of them issued
        as a captured graph where the engine's runs are: launched one by one a
        small grid's passes would be timed by the host."""
        from .. import autotune
        if not self.user_data.get("use_graph", True):
            return autotune.time_candidate(run, self._ppf_stream)
        g = self._ppf_capture(lambda: [run() for _ in range(passes)])
        try:
            sp = C.c_void_p(self._ppf_stream.cuda_stream)
            return autotune.time_candidate(lambda: L.call("ppf_graph_launch", g, sp),
                                           self._ppf_stream, reps=5) / passes
        finally:
            L.call("ppf_graph_destroy", g)

    def _ppf_graphs_reset(self):
        self._ppf_release_graphs()

    def _ppf_tiling(self, depth: int):
        ud = self.user_data
        flags = 0 if ud.get("bulk_shortcut", True) else L.PPF_TILING_FULL_EVAL
        return tiling_struct(depth, ud.get("tile"), ud.get("pdl", True), flags, ud.get("zchunk", 0))

    # ------------------------------------------------------------ lifecycle
    def just_before_simulating(self):
        t = self._temperature_type
        if t not in (None, "ISOTHERMAL", "LINEAR_GRADIENT"):
            raise NotImplementedError(f"temperature type {t!r} is not supported (XDMF input "
                                      "needs meshio)")
        self._ppf_prepare()
        self._ppf_setup()
        fill_ghosts_host(self)
        self.send_fields_to_GPU()
        if self.user_data.get("autotune", False):
            self._ppf_autotune()

    def send_fields_to_GPU(self):
        if not self._ppf_ready():
            self._ppf_setup()
        s = self._ppf_stream
        with nvtx_range("ppf.send_fields_to_GPU"):
            self._ppf_send(s)

    def _ppf_send(self, s):
        self._ppf_staging = [
            self._ppf_grid.upload(self._ppf_bufs[self._ppf_cur][j],
                                  self._ppf_encode(j, f.get_cells()), s)
            for j, f in enumerate(self.fields)]

    def retrieve_fields_from_GPU(self):
        if not self._ppf_ready():
            return
        self._ppf_check_status(True, "retrieve_fields_from_GPU")
        s = self._ppf_stream
        with nvtx_range("ppf.retrieve_fields_from_GPU"):
            for j, f in enumerate(self.fields):
                f.data[f._slice] = self._ppf_decode(
                    j, self._ppf_grid.download(self._ppf_bufs[self._ppf_cur][j], s))
        self._ppf_staging = []
        fill_ghosts_host(self)

    def apply_boundary_conditions(self):
        if self._ppf_ready():
            return  # fused into every kernel's tile load
        fill_ghosts_host(self)

    def update_temperature_field(self, force_cpu=False):
        """One step of the temperature law (simulation.py:303-333). None of the
        four engines reads the temperature field (Warren1995 takes the scalar
        T of user_data), so it stays a host field that advances with the
        step count."""
        self._ppf_advance_temperature(1)

    def _ppf_advance_temperature(self, nsteps: int):
        t = self._temperature_type
        if t == "LINEAR_GRADIENT" and self.temperature is not None and self._dTdt:
            # closed form of nsteps per-step increments dTdt * dt
            self.temperature.data += nsteps * self._dTdt * self.dt
        elif t not in (None, "ISOTHERMAL", "LINEAR_GRADIENT"):
            raise NotImplementedError(f"temperature type {t!r} is not supported")

    def simulation_loop(self):
        """Advance one step on the device (the reference's engine call)."""
        if not self._ppf_ready():
            self.just_before_simulating()
        self._ppf_advance(1, self.time_step_counter)

    def simulate(self, number_of_timesteps):
        with nvtx_range(f"ppf.simulate {type(self).__name__} n={int(number_of_timesteps)}"):
            self._ppf_simulate(number_of_timesteps)

    def _ppf_simulate(self, number_of_timesteps):
        if not self._begun_simulation or not self._ppf_ready():
            self._begun_simulation = True
            self.just_before_simulating()
        n = int(number_of_timesteps)
        rate = self._autosave_rate if self._autosave_flag else None
        while n > 0:
            chunk = n
            if rate:
                chunk = min(chunk, rate - self.time_step_counter % rate)
            # the reference increments the counter before each engine call;
            # the step index keyed into the noise is the counter before it
            try:
                self._ppf_advance(chunk, self.time_step_counter)
            except EngineFault:
                # the counter covers the steps launched before the fault
                self.time_step_counter += self._ppf_done
                raise
            self.time_step_counter += chunk
            self._ppf_advance_temperature(chunk)
            n -= chunk
            if rate and self.time_step_counter % rate == 0:
                self._ppf_check_status(True, "autosave")
                self._ppf_checkpoint()
        self._ppf_checkpoint_wait()

    # ------------------------------------------------------------ autosave
    def _ppf_checkpoint(self):
        """Autosave without stopping the device (simulation.py:267-271 saves
        synchronously): the state is copied on the device into one of two
        snapshot slots, then to pinned host memory on a copy stream, and a
        writer thread fills Field.data and writes step_<counter>.npz while
        the next steps run. simulate() returns after every write finished,
        with Field.data holding the last autosaved state, as in the
        reference."""
        with nvtx_range(f"ppf.autosave step {self.time_step_counter}"):
            self._ppf_checkpoint_issue()

    def _ppf_checkpoint_issue(self):
        import concurrent.futures as cf
        ck = getattr(self, "_ppf_ckpt", None)
        g = self._ppf_grid
        if ck is None:
            ck = self._ppf_ckpt = {
                "pool": cf.ThreadPoolExecutor(max_workers=1), "stream": torch.cuda.Stream(g.device),
                "slots": [{"dev": [g.empty() for _ in range(self.NFIELDS)],
                           "host": [torch.empty(g.alloc_shape, dtype=g.dtype, pin_memory=True)
                                    for _ in range(self.NFIELDS)], "job": None}
                          for _ in range(2)], "next": 0}
        slot = ck["slots"][ck["next"]]
        ck["next"] ^= 1
        if slot["job"] is not None:
            slot["job"].result()  # the slot's previous write is done with its buffers
        s, cs = self._ppf_stream, ck["stream"]
        with torch.cuda.stream(s):
            for j in range(self.NFIELDS):
                slot["dev"][j].copy_(self._ppf_bufs[self._ppf_cur][j])
        taken = torch.cuda.Event()
        taken.record(s)
        cs.wait_event(taken)
        with torch.cuda.stream(cs):
            for j in range(self.NFIELDS):
                slot["host"][j].copy_(slot["dev"][j], non_blocking=True)
        done = torch.cuda.Event()
        done.record(cs)
        slot["job"] = ck["pool"].submit(self._ppf_write_checkpoint, slot, done,
                                        self.time_step_counter)

    def _ppf_write_checkpoint(self, slot, done, step):
        done.synchronize()
        g = self._ppf_grid
        for j, f in enumerate(self.fields):
            host = slot["host"][j][..., : g.kshape[-1]].numpy().astype(np.float64)
            f.data[f._slice] = self._ppf_decode(j, host.reshape(g.user_shape))
        fill_ghosts_host(self)
        if "step" in inspect.signature(self.save_simulation).parameters:
            self.save_simulation(step=step)
        else:
            # the reference's save_simulation (simulation.py:399-420) names the
            # file by the live counter, which has moved on by now: write the
            # same file under the step that was snapshotted
            _save_npz(self, step)

    def _ppf_checkpoint_wait(self):
        ck = getattr(self, "_ppf_ckpt", None)
        if ck is not None:
            for slot in ck["slots"]:
                if slot["job"] is not None:
                    slot["job"].result()
                    slot["job"] = None

    # ------------------------------------------------------------ stepping
    def _ppf_passes(self, nsteps: int, even: bool = False) -> list[int]:
        """Steps of each pass of a run of nsteps. temporal_depth > 1: passes
        of that depth and a remainder; else as few passes as the engine's own
        depth allows, of equal depth within one step (even: an even number of
        them, so that the field ends in the buffers it began in)."""
        k = max(1, min(int(self.user_data.get("temporal_depth", 1)), self._ppf_max_depth()))
        if k == 1:
            m = -(-nsteps // self._ppf_auto_depth())
            if even:
                m += m & 1
            return [nsteps // m + (i < nsteps % m) for i in range(m)]
        passes = [k] * (nsteps // k)
        if nsteps % k:
            passes.append(nsteps % k)
        return passes

    def _ppf_launch_passes(self, depths, step, step_base):
        """Launch the passes of a run of steps from absolute step `step` (plus
        *step_base on the device): one native call, or one call per pass."""
        cur = self._ppf_cur
        sp = self._ppf_stream.cuda_stream
        run = self._ppf_run()
        if run is None:
            for d in depths:
                self._ppf_step(self._ppf_bufs[self._ppf_cur], self._ppf_bufs[1 - self._ppf_cur], d,
                               step, step_base, C.c_void_p(sp))
                self._ppf_cur ^= 1
                step += d
            return
        run.elem_bytes = 4 if self._ppf_dtype == torch.float32 else 8
        run.grid = C.pointer(self._ppf_grid.grid)
        run.boundary = C.pointer(self._ppf_bc)
        for j, (t, u) in enumerate(zip(self._ppf_bufs[cur], self._ppf_bufs[1 - cur])):
            run.a[j], run.b[j] = t.data_ptr(), u.data_ptr()
        run.step = step
        run.step_base = step_base.data_ptr() if step_base is not None else None
        it = C.c_int32()
        n = len(depths)
        try:
            L.call("ppf_run", C.byref(run), (C.c_int32 * n)(*depths), n, C.byref(it), sp)
        except L.PpfError:
            # the passes before the refused one ran
            done = C.c_int32()
            L.call("ppf_run_passes", C.byref(done))
            self._ppf_cur ^= done.value & 1
            raise
        self._ppf_iterations = it.value
        self._ppf_cur ^= n & 1

    def _ppf_state_key(self):
        """What a captured graph bakes in besides the buffers: every
        user_data value (parameters, tiling, seed, ...), dt, dx and the
        boundary struct. A graph is reused only while all of it is unchanged,
        so editing user_data between simulate() calls never replays stale
        constants."""
        items = []
        for k, v in self.user_data.items():
            t = type(v)
            if t in _PLAIN:
                v = (t, v or repr(v))  # 0.0 == -0.0, which are not the same constant
            elif isinstance(v, np.ndarray):
                v = (v.shape, v.dtype.str,
                     hashlib.sha1(np.ascontiguousarray(v).tobytes()).hexdigest())
            elif isinstance(v, torch.Tensor):
                v = ("tensor", v.data_ptr(), tuple(v.shape), v._version)
            else:
                v = repr(v)
            items.append((str(k), v))
        return (tuple(items), repr(self.dt), repr(self.dx), bytes(self._ppf_bc))

    def _ppf_capture(self, issue):
        """Executable graph of the launches issue() makes on the engine's stream."""
        s = self._ppf_stream
        sp = C.c_void_p(s.cuda_stream)
        # No Python garbage collection while capturing: collecting another
        # engine would free its pinned staging buffers and graphs, and those
        # CUDA calls would invalidate the capture.
        gc_was_enabled = gc.isenabled()
        gc.disable()
        L.call("ppf_graph_begin", sp)
        exec_ = C.c_void_p()
        try:
            with torch.cuda.stream(s):
                issue()
        finally:
            try:
                L.call("ppf_graph_end", sp, C.byref(exec_))
            finally:
                if gc_was_enabled:
                    gc.enable()
        return exec_

    def _ppf_graph(self, depths: tuple[int, ...]):
        key = (self._ppf_cur, depths, self._ppf_state_key())
        g = self._ppf_graphs.get(key)
        if g is not None:
            self._ppf_graphs.move_to_end(key)
            return g
        while len(self._ppf_graphs) >= MAX_GRAPHS:
            L.call("ppf_graph_destroy", self._ppf_graphs.popitem(last=False)[1])
        s = self._ppf_stream
        cur0 = self._ppf_cur
        total = sum(depths)

        def issue():
            self._ppf_segment_begin(total, s)
            self._ppf_launch_passes(depths, 0, self._ppf_stepctr if self.USES_STEP else None)
            if self.USES_STEP:
                L.call("ppf_counter_add_u64", ptr(self._ppf_stepctr), C.c_uint64(total),
                       C.c_void_p(s.cuda_stream))
            self._ppf_watch(s)

        try:
            exec_ = self._ppf_capture(issue)
        finally:
            self._ppf_cur = cur0
        self._ppf_graphs[key] = exec_
        return exec_

    def _ppf_advance(self, nsteps: int, step0: int):
        """Advance nsteps from absolute step index step0 (noise key)."""
        if nsteps <= 0:
            return
        self._ppf_done = 0
        ud = self.user_data
        chunk = max(2, int(ud.get("graph_chunk", 64)) // 2 * 2)
        s = self._ppf_stream
        sp = C.c_void_p(s.cuda_stream)
        step = step0
        # a graph holds `chunk` passes of temporal_depth steps, or `chunk`
        # steps in passes of the engine's own depth
        k = max(1, min(int(ud.get("temporal_depth", 1)), self._ppf_max_depth()))
        span = chunk * k
        if ud.get("use_graph", True) and nsteps >= span:
            g = self._ppf_graph(tuple(self._ppf_passes(span, even=True)))
            if self.USES_STEP:
                with _device_of(s):
                    L.call("ppf_counter_set_u64", ptr(self._ppf_stepctr), C.c_uint64(step), sp)
            while nsteps >= span:
                self._ppf_check_status(False)
                with nvtx_range(f"ppf.graph {span} steps from {step}"):
                    L.call("ppf_graph_launch", g, sp)
                self._ppf_mark()
                self._ppf_segment_end(span, s)
                nsteps -= span
                step += span
                self._ppf_done += span
        if nsteps:
            self._ppf_check_status(False)
            with torch.cuda.stream(s), nvtx_range(f"ppf.eager {nsteps} steps from {step}"):
                self._ppf_segment_begin(nsteps, s)
                self._ppf_launch_passes(self._ppf_passes(nsteps), step, None)
                self._ppf_watch(s)
            self._ppf_mark()
            self._ppf_segment_end(nsteps, s)

    # ------------------------------------------------------------ access
    def device_fields(self) -> list[torch.Tensor]:
        """Views of the current device fields (interior only, stored values)."""
        return [self._ppf_grid.view(t) for t in self._ppf_bufs[self._ppf_cur]]

    def synchronize(self):
        if self._ppf_ready():
            self._ppf_stream.synchronize()
