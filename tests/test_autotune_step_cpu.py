"""The autotuner judges the step that the engine runs: whole steps are timed with
the profiler off, and a shape found from pass times is kept only if its step is
faster than the default's.  A stand-in handle, no GPU: a profiled step is slower
than an unprofiled one, and shapes other than the default give up a merged
launch."""
import pytest

from rocflupicl_gb300 import autotune as AT
from rocflupicl_gb300 import engine as E


class Handle:
    """Pass times favour faceBlock 256; whole steps do what step_ms says."""

    def __init__(self, step_ms, profiled_ms):
        self.step_ms, self.profiled_ms = step_ms, profiled_ms
        self.shape = {k: 0 for k in E.TUNING_KEYS}
        self.on, self.timer, self.prof, self.steps = False, 0.0, {}, 0

    def set_tuning(self, **kw):
        self.shape = dict(self.shape, **kw)

    def step(self, *args):
        self.steps += 1
        self.timer += (self.profiled_ms if self.on else self.step_ms)(self.shape)
        if self.on:
            t, n = self.prof.get("face_flux", (0.0, 0))
            self.prof["face_flux"] = (t + (0.9 if self.shape["faceBlock"] == 256 else 1.0), n + 1)

    def sync(self):
        pass

    def profile(self, on=True):
        self.on = on
        if on:
            self.prof = {}

    def profile_read(self):
        return dict(self.prof)

    def timer_start(self):
        self.timer = 0.0

    def timer_stop(self):
        return self.timer


def _tune(kind, h, monkeypatch):
    monkeypatch.setattr(AT.E, "sm_count", lambda: 152)
    return (AT.tune_region(h, 0.5, 1.0, steps=2) if kind == "region" else
            AT.tune_batch(h, 0.5, steps=2))


@pytest.mark.parametrize("kind", ["region", "batch"])
def test_shape_slower_than_the_default_is_not_kept(kind, monkeypatch):
    # profiled, every step launches every pass alone: the shapes cost nothing
    h = Handle(lambda s: (12.0 if s["faceBlock"] not in (0, 128) else 9.0) + bool(s["gridCap"]) +
               5.0 * s["persistentStage"], lambda s: 13.0 if s["faceBlock"] != 256 else 12.9)
    out = _tune(kind, h, monkeypatch)
    assert out["shape"] == {k: 0 for k in E.TUNING_KEYS} == h.shape
    assert out["ms"]["shape"] == {"default": 9.0, "tuned": 12.0}
    assert out["steps_taken"] == h.steps


@pytest.mark.parametrize("kind", ["region", "batch"])
def test_faster_shape_is_kept(kind, monkeypatch):
    h = Handle(lambda s: 9.0 - 0.2 * (s["faceBlock"] == 256), lambda s: 13.0)
    out = _tune(kind, h, monkeypatch)
    assert out["shape"]["faceBlock"] == 256 and h.shape == out["shape"]


def test_persistent_stage_competes_with_the_unprofiled_step(monkeypatch):
    # 10 beats the profiled 13, not the 9 that the engine runs
    h = Handle(lambda s: 10.0 if s["persistentStage"] else 9.0,
               lambda s: 10.0 if s["persistentStage"] else 13.0)
    assert _tune("region", h, monkeypatch)["shape"]["persistentStage"] == 0


def test_batch_keeps_the_grid_cap_that_helps(monkeypatch):
    h = Handle(lambda s: (12.0 if s["faceBlock"] == 256 else 9.0) - (s["gridCap"] == 152 * 8),
               lambda s: 13.0)
    out = _tune("batch", h, monkeypatch)
    assert out["shape"] == dict({k: 0 for k in E.TUNING_KEYS}, gridCap=152 * 8)
    assert out["grid_cap"] == 152 * 8
