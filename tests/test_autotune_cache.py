"""What the tuner keeps on disk: a choice is used again for the same kernels and
candidates, and timed anew when either has changed (no GPU: the simulations
that are timed are stand-ins).
"""
import json

import numpy as np
import pytest

from phonomena_gb300 import autotune, batch

SHAPE = (33, 21, 17)


class Sim:
    timed = []  # tile shapes timed, in order
    nx = SHAPE[0]

    def __init__(self):
        self.shape = (0, 0)

    def set_tiling(self, tj, xs):
        self.shape = (tj, xs)

    def step(self, n):
        pass

    sync = close = lambda self: None

    def last_step_ms(self):
        Sim.timed.append(self.shape)
        return 1.0 if self.shape == (0, 0) else 2.0


class Batch:
    def __init__(self, n, **kw):
        self.kw = kw

    def __enter__(self):
        return self

    __exit__ = add = step = sync = lambda self, *a: None

    def last_step_ms(self):
        Sim.timed.append(self.kw["tile_j"])
        return 1.0


@pytest.fixture
def cache(tmp_path, monkeypatch):
    monkeypatch.setattr(autotune, "CACHE", tmp_path / "autotune.json")
    monkeypatch.setattr(autotune, "_scratch", lambda *a, **k: Sim())
    monkeypatch.setattr(batch, "Batch", Batch)
    Sim.timed = []
    return autotune.CACHE


def tuned(**kw):
    before = len(Sim.timed)
    best = autotune.tune(None, np.zeros(SHAPE, np.uint8), None, 1e-10, precision="f64", **kw)
    return best, len(Sim.timed) - before


def test_a_choice_of_other_kernels_is_not_used(cache):
    """Entries as they were written before the kernels and the candidates were
    part of the key."""
    name = autotune._device_name()
    cache.write_text(json.dumps({f"f64:{'x'.join(map(str, SHAPE))}:{name}": {"best": [8, 24]}}))
    best, timed = tuned()
    assert best == (0, 0) and timed > 1
    assert tuned() == ((0, 0), 0)  # the new entry is


@pytest.mark.parametrize("changed", ["fdtd_step.cu", "split_step.cu", "soft_f64.cuh", "api.cu"])
def test_a_changed_kernel_is_timed_anew(cache, monkeypatch, tmp_path, changed):
    copy = tmp_path / "csrc"
    copy.mkdir()
    for f in autotune.build.CSRC.iterdir():
        (copy / f.name).write_bytes(f.read_bytes())
    monkeypatch.setattr(autotune.build, "CSRC", copy)
    autotune._kernels.cache_clear()
    try:
        mix = lambda: autotune.tune_batch([SHAPE], "f32k", tile_js=(16,))
        assert tuned()[1] > 0 and tuned()[1] == 0
        mix()
        n = len(Sim.timed)
        assert mix() and len(Sim.timed) == n
        with open(copy / changed, "a") as f:
            f.write("// changed\n")
        autotune._kernels.cache_clear()
        assert tuned()[1] > 0
        n = len(Sim.timed)
        assert mix() and len(Sim.timed) > n
    finally:
        autotune._kernels.cache_clear()


def test_other_candidates_are_timed(cache):
    assert tuned(candidates=[(8, 32)])[1] == 2  # the library's own choice and it
    assert tuned(candidates=[(8, 32), (16, 32)])[1] == 3
    assert tuned(candidates=[(8, 32)])[1] == 0
