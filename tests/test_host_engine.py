"""The engines' host side with the library calls recorded (no GPU)."""
import contextlib
import types

import pytest
import torch

from pyphasefield_gb300 import _lib as L
from pyphasefield_gb300.engines import base


class Stream:
    cuda_stream = 7
    device = types.SimpleNamespace(index=1)


class Engine(base.GB300Engine):
    """An engine of a few fields, without device buffers."""

    def __init__(self, **user_data):
        self.user_data = dict(user_data)
        self._ppf_stream = Stream()
        self._ppf_stepctr = torch.zeros(1, dtype=torch.int64)
        self._ppf_cur = 0

    def _ppf_graph(self, depths):
        return "graph"

    def _ppf_check_status(self, block, where=""):
        pass

    def _ppf_mark(self):
        pass


@pytest.mark.parametrize("current", [0, 1])
def test_counter_is_set_with_the_engines_device_current(monkeypatch, current):
    """A launch into a stream of another device than the current one is refused."""
    class Noisy(Engine):
        USES_STEP = True

    log, devices = [], [current]

    @contextlib.contextmanager
    def enter(s):
        devices.append(getattr(s, "device", s).index)
        yield
        devices.pop()

    monkeypatch.setattr(base.torch.cuda, "current_device", lambda: devices[-1])
    monkeypatch.setattr(base.torch.cuda, "device", enter)
    monkeypatch.setattr(base.torch.cuda, "stream", enter)
    monkeypatch.setattr(base.L, "call", lambda name, *a: log.append((name, devices[-1])))
    e = Noisy(graph_chunk=4, check_status=False)
    e._ppf_advance(8, 3)
    assert [n for n, _ in log] == ["ppf_counter_set_u64", "ppf_graph_launch", "ppf_graph_launch"]
    assert log[0][1] == 1 and devices == [current]


@pytest.mark.parametrize("done", [0, 1, 2, 3])
def test_a_run_that_stops_leaves_its_last_complete_state_current(monkeypatch, done):
    class Native(Engine):
        def _ppf_run(self):
            return L.PpfRun()

    def call(name, *args):
        if name == "ppf_run":
            raise L.PpfError(L.PPF_ERR_INVALID, name, "refused")
        assert name == "ppf_run_passes"
        args[0]._obj.value = done

    e = Native()
    e._ppf_bufs = [[torch.zeros(4)], [torch.zeros(4)]]
    e._ppf_grid = types.SimpleNamespace(grid=L.PpfGrid())
    e._ppf_bc = L.PpfBoundary()
    monkeypatch.setattr(base.L, "call", call)
    with pytest.raises(L.PpfError, match="refused"):
        e._ppf_launch_passes([1] * 5, 0, None)
    assert e._ppf_cur == done % 2


def test_a_step_of_its_own_is_not_bypassed():
    """A subclass that overrides _ppf_step alone is stepped one step a pass,
    through it, and is given the step counter."""
    from pyphasefield_gb300 import DiffusionGB300, Warren1995GB300

    class Sourced(DiffusionGB300):
        def _ppf_step(self, *a):
            pass

    class Further(Sourced):
        pass

    class Mixed(type("Step", (), {"_ppf_step": lambda self, *a: None}), DiffusionGB300):
        pass

    class Stated(DiffusionGB300):
        USES_STEP = False
        _ppf_auto_depth = DiffusionGB300._ppf_auto_depth

        def _ppf_step(self, *a):
            pass

    for cls in (Sourced, Further, Mixed):
        e = cls.__new__(cls)
        e._ppf_grid = types.SimpleNamespace(kshape=(64, 64))
        assert e._ppf_run() is None and e._ppf_auto_depth() == 1 and e.USES_STEP
    assert not Stated.USES_STEP and Stated._ppf_auto_depth is DiffusionGB300._ppf_auto_depth
    assert not DiffusionGB300.USES_STEP and Warren1995GB300.USES_STEP

    class Renamed(DiffusionGB300):
        """No step of its own: everything is inherited."""

    for cls in (Renamed, Warren1995GB300):
        assert cls._ppf_run is not base.GB300Engine._ppf_run
    assert Renamed._ppf_auto_depth is DiffusionGB300._ppf_auto_depth and not Renamed.USES_STEP


@pytest.mark.parametrize("shape", [(64, 64), (24, 24, 24)])
@pytest.mark.parametrize("name", ["DiffusionGB300", "CahnAllenGB300"])
def test_the_engines_own_choice_is_a_tuning_candidate(name, shape):
    import pyphasefield_gb300 as P
    cls = getattr(P, name)
    e = cls(dimensions=list(shape), dx=1.0, dt=0.1, boundary_conditions="PERIODIC")
    e._ppf_grid = types.SimpleNamespace(kshape=shape)
    default = {"temporal_depth": e.user_data["temporal_depth"], "tile": e.user_data["tile"],
               "zchunk": 0}
    cands = e._ppf_tune_candidates()
    assert all(default[k] == v for k, v in cands[0].items())
    # every candidate sets the same keys: none is timed with another's left-overs
    assert len({frozenset(c) for c in cands}) == 1


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_candidates_are_timed_at_the_depth_they_run_at(monkeypatch, precision):
    import pyphasefield_gb300 as P
    from pyphasefield_gb300 import autotune
    e = P.DiffusionGB300(dimensions=[64, 64], dx=1.0, dt=0.1, boundary_conditions="PERIODIC",
                         user_data={"precision": precision, "use_graph": False})
    e._ppf_grid = types.SimpleNamespace(kshape=(64, 64))
    e._ppf_bc, e._ppf_stream, e._ppf_cur = L.PpfBoundary(), Stream(), 0
    e._ppf_bufs = [[torch.zeros(4)], [torch.zeros(4)]]
    timed = []
    e._ppf_step = lambda src, dst, depth, *a: timed.append(depth)
    monkeypatch.setattr(base.torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(autotune, "time_candidate", lambda run, s: [run(), 1.0][1])

    def pick(key, cands, measure):
        seen = set()
        for c in cands:
            seconds = measure(c)
            e.user_data.update(c)
            depth = max(e._ppf_passes(64))
            assert seconds == 1.0 / depth, c
            if (depth, c["tile"]) not in seen:
                assert timed == [depth, depth], c  # once before it is timed
                timed.clear()
            seen.add((depth, c["tile"]))
        return cands[0]

    monkeypatch.setattr(autotune, "pick", pick)
    e._ppf_autotune()
    assert not timed


def test_the_engines_own_choice_wins_against_its_own_passes(monkeypatch, tmp_path):
    """In 2-D float the own choice and temporal_depth 8 are the same passes, in
    other graphs; the timer's spread does not decide between them."""
    import pyphasefield_gb300 as P
    from pyphasefield_gb300 import autotune
    monkeypatch.setenv("PPF_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(autotune, "_memory", {})
    monkeypatch.setattr(base.torch.cuda, "stream", lambda s: contextlib.nullcontext())
    e = P.DiffusionGB300(dimensions=[64, 64], dx=1.0, dt=0.1, boundary_conditions="PERIODIC",
                         user_data={"use_graph": False})
    e._ppf_grid, e._ppf_bc = types.SimpleNamespace(kshape=(64, 64)), L.PpfBoundary()
    e._ppf_stream, e._ppf_cur = Stream(), 0
    e._ppf_bufs = [[torch.zeros(4)], [torch.zeros(4)]]
    e._ppf_step = lambda *a: None
    spread = iter([2.0, 1.9])

    def time_candidate(run, s):
        own = e.user_data["tile"] is None and e.user_data["temporal_depth"] in (1, 8)
        return next(spread) if own else 100.0

    monkeypatch.setattr(autotune, "time_candidate", time_candidate)
    e._ppf_autotune()
    assert e.user_data["temporal_depth"] == 1 and e.user_data["tile"] is None


def test_choices_cached_for_other_kernels_are_not_taken(monkeypatch):
    """The Diffusion and Allen-Cahn kernels changed; the others' choices stay."""
    import pyphasefield_gb300 as P
    from pyphasefield_gb300 import autotune
    keys = {}
    monkeypatch.setattr(autotune, "pick", lambda key, cands, m: keys.update({name: key}) or cands[0])
    monkeypatch.setattr(base.torch.cuda, "stream", lambda s: contextlib.nullcontext())
    for name in ("DiffusionGB300", "CahnAllenGB300", "Warren1995GB300"):
        e = getattr(P, name)(dimensions=[64, 64], dx=1.0, dt=0.1, boundary_conditions="PERIODIC")
        e._ppf_grid = types.SimpleNamespace(kshape=(64, 64))
        e._ppf_stream, e._ppf_cur = Stream(), 0
        e._ppf_bufs = [[torch.zeros(4)], [torch.zeros(4)]]
        e._ppf_autotune()
        old = autotune.make_key(name, (64, 64), torch.float32, "2")
        assert (keys[name] == old) == (name == "Warren1995GB300")


def test_the_state_key_tells_zeros_apart():
    e = Engine()
    e.dt, e.dx, e._ppf_bc = 0.1, 1.0, L.PpfBoundary()
    keys = []
    for v in (0.0, -0.0, 0, False, None, "", "0.0", 1, 1.0, True):
        e.user_data["v"] = v
        keys.append(e._ppf_state_key())
    assert len(set(keys)) == len(keys)


def test_candidates_are_timed_as_graphs(monkeypatch):
    """Passes launched one by one would be timed by the host on a small grid."""
    import pyphasefield_gb300 as P
    from pyphasefield_gb300 import autotune
    e = P.DiffusionGB300(dimensions=[64, 64, 64], dx=1.0, dt=0.1, boundary_conditions="PERIODIC")
    e._ppf_grid, e._ppf_bc = types.SimpleNamespace(kshape=(64, 64, 64)), L.PpfBoundary()
    e._ppf_stream, e._ppf_cur = Stream(), 0
    e._ppf_bufs = [[torch.zeros(4)], [torch.zeros(4)]]
    log = []
    e._ppf_step = lambda *a: log.append("step")
    monkeypatch.setattr(base.torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(base.L, "call", lambda name, *a: log.append(name))
    monkeypatch.setattr(autotune, "time_candidate", lambda run, s, reps: [run(), 16.0][1])

    def pick(key, cands, measure):
        assert measure(cands[0]) == 2.0
        return cands[0]

    monkeypatch.setattr(autotune, "pick", pick)
    e._ppf_autotune()
    assert log == ["step", "ppf_graph_begin"] + ["step"] * 8 + [
        "ppf_graph_end", "ppf_graph_launch", "ppf_graph_destroy"]
