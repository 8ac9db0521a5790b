"""thysea.run's own preparation, before the call of thy_run: any simulated time
and snapshot interval that the library takes reaches it."""
import numpy as np
import pytest

import thysea
from thysea import synth


@pytest.mark.parametrize("sim_time,save_time", [
    (-5.0, 1.0), (-1e30, 1.0), (0.0, 1.0), (float("nan"), 1.0), (float("inf"), 1.0), (100.0, 1e-30),
    (100.0, float("inf")), (100.0, float("nan")), (100.0, 0.0)])
def test_times_reach_the_library(sim_time, save_time, monkeypatch):
    calls = []

    class Lib:
        def __getattr__(self, name):
            if name != "thy_run":
                return getattr(real, name)
            return lambda *a: calls.append(a) or 0

    prep = thysea.Prepared(synth.plain_small(24, 20, sim_time=sim_time, save_time=save_time, npoints=0))
    real = thysea._ffi.lib()
    monkeypatch.setattr(thysea._ffi, "lib", lambda: Lib())
    r = thysea.run(prep)
    assert len(calls) == 1 and r["snapshots"]["eta"].shape == (0,)


def test_no_room_for_the_stacks(monkeypatch):
    prep = thysea.Prepared(synth.plain_small(24, 20, sim_time=100.0, save_time=10.0, npoints=0))
    empty = np.empty
    calls = []

    class Lib:
        def __getattr__(self, name):
            if name != "thy_run":
                return getattr(real, name)
            return lambda *a: calls.append(a) or 0

    def short(shape, *a, **k):
        if np.size(shape) == 3:
            raise MemoryError
        return empty(shape, *a, **k)

    real = thysea._ffi.lib()
    monkeypatch.setattr(thysea._ffi, "lib", lambda: Lib())
    monkeypatch.setattr(np, "empty", short)
    thysea.run(prep)
    assert len(calls) == 1
