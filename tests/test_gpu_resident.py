"""Chunks of steps that stay resident on the device (kernels/resident.cu)
against the launched kernels: the same code of every cell, so bitwise the same
fields, samples, step counts and unit counts, at sizes around the edges of
strips (28 columns), tiles (112), units (16 rows) and of the task splits, up to
the largest resident work."""
import dataclasses
import os
import subprocess
import sys

import numpy as np
import pytest

import thysea
from thysea import synth

pytestmark = pytest.mark.gpu

FIELDS = ("max_height", "arrival", "deformed_bathy", "eta", "ux", "uy")


def _problem(nx, ny, kind, sim_time):
    rng = np.random.default_rng(nx * 10007 + ny)
    lon, lat = synth.lonlat_grid(nx, ny, lat_centre=12.0)
    z = synth.shelf_bathymetry(nx, ny, rng) if kind != "shallow" else (
        -15.0 + 20.0 * synth.gaussian_random_field(nx, ny, 4.0, rng)).astype(np.float32)
    p = synth.Problem(name="resident", lon=lon, lat=lat, z=z, sim_time=sim_time)
    if kind in ("file", "shallow"):
        p.eta_init = synth.gaussian_random_field(nx, ny, 5.0, rng).astype(np.float32)
    else:
        c = synth.random_fault(lon, lat, z, rng)
        p.faults = [c]
        if kind == "late":
            p.faults = [c, synth.random_fault(lon, lat, z, rng, time=0.5 * sim_time)]
    p.borders = {"file": (-1.0, -1.0, -1.0, -1.0), "periodic": (1.0, -1.0, 2.0, 2.0)}.get(kind, (1.0, 1.0, 1.0, 1.0))
    if kind == "late":
        p.points = np.stack([lon[rng.integers(0, nx, 5)], lat[rng.integers(0, ny, 5)]], axis=1)
        p.series_time, p.save_time = sim_time / 20.0, sim_time / 3.0
    return p


def _run(prep):
    r = thysea.run(prep)
    return {k: r[k].copy() for k in FIELDS}, r


@pytest.mark.parametrize("nx,ny,kind,sim_time", [
    (2, 2, "file", 30.0), (3, 17, "file", 60.0), (28, 16, "shallow", 120.0), (29, 33, "shallow", 200.0),
    (112, 48, "periodic", 300.0), (113, 95, "late", 400.0), (229, 160, "late", 400.0), (336, 337, "open", 400.0),
    (500, 411, "shallow", 400.0), (641, 512, "periodic", 500.0), (1024, 700, "late", 300.0), (1700, 1790, "open", 120.0),
])
def test_resident_chunks_match_the_launched_kernels(gpu, nx, ny, kind, sim_time):
    prep = thysea.Prepared(_problem(nx, ny, kind, sim_time))
    thysea.force_tiling((0, 0, 0))   # a forced tiling names the launched kernels
    try:
        ref, r0 = _run(prep)
    finally:
        thysea.force_tiling(None)
    got, r = _run(prep)
    assert r["kernel_launches"] < r["iterations"] < r0["kernel_launches"]   # one launch a chunk against six a step
    for k in ("iterations", "final_time", "deep_tiles", "dry_tiles", "nseries", "nsnaps"):
        assert r[k] == r0[k], k
    for k in FIELDS:
        assert np.array_equal(got[k], ref[k], equal_nan=True), k
    for part in ("snapshots", "series"):
        for k in r0[part]:
            assert np.array_equal(r[part][k], r0[part][k], equal_nan=True), (part, k)


def test_resident_batch_matches_alone(gpu):
    """several scenarios in one resident chunk, each with its own dt, end and
    gauges-free events, against their launched runs"""
    probs = [_problem(nx, ny, kind, t) for nx, ny, kind, t in
             ((120, 100, "open", 300.0), (257, 130, "periodic", 500.0), (64, 64, "shallow", 100.0), (300, 222, "file", 350.0))]
    thysea.force_tiling((0, 0, 0))
    try:
        alone = [_run(thysea.Prepared(p)) for p in probs]
    finally:
        thysea.force_tiling(None)
    srv = thysea.Server(hbm_budget_bytes=2 << 30, max_scenarios=8)
    ids = [srv.submit(p) for p in probs]
    srv.drain()
    srv.close()
    for rid, (ref, r) in zip(ids, alone):
        assert srv.results[rid]["status"] == 0
        assert srv.results[rid]["stats"]["steps"] == r["iterations"]
        for k in FIELDS:
            assert np.array_equal(srv.results[rid]["outputs"][k], ref[k], equal_nan=True), k


@pytest.mark.parametrize("ngauges", [1, 33, 700])
@pytest.mark.parametrize("launched", [False, True])
def test_gauge_samples_on_the_device(gpu, launched, ngauges):
    """samples taken at a step's end by a resident chunk's first CTA and by the
    last CTA of a launched step, a thread a gauge, also with more gauges than
    threads: the eta of a snapshot of the same step at the gauge's cell (each one
    rounding of the same product, hence two units of the last place)"""
    nx, ny = 180, 150
    p = _problem(nx, ny, "open", 300.0)
    rng = np.random.default_rng(ngauges)
    ix, iy = rng.integers(0, nx, ngauges), rng.integers(0, ny, ngauges)
    p.points = np.stack([p.lon[ix], p.lat[iy]], axis=1)
    p.series_time = p.save_time = 25.0
    prep = thysea.Prepared(p)
    thysea.force_tiling((0, 0, 0) if launched else None)
    try:
        r = thysea.run(prep)
    finally:
        thysea.force_tiling(None)
    s, f = r["series"], r["snapshots"]
    assert r["nseries"] == r["nsnaps"] > 5
    assert np.array_equal(s["time"], f["time"])
    # (points of one cell are one gauge)
    cells = np.ctypeslib.as_array(prep.c.point_cell, (prep.npoints,))
    assert set(cells) == set(iy * nx + ix)
    for k in range(r["nseries"]):
        at = f["eta"][k].reshape(-1)[cells]
        wet = np.abs(at) < 1e3
        assert wet.any()
        np.testing.assert_allclose(np.asarray(s["eta"][k])[wet], at[wet], rtol=2.4e-7, atol=0)
    assert np.abs(np.asarray(s["eta"])).max() > 1e-3


def test_largest_resident_work(gpu):
    """close to the largest work of a resident chunk (25 x 148 units)"""
    prep = thysea.Prepared(_problem(2640, 2360, "open", 60.0))
    thysea.force_tiling((0, 0, 0))
    try:
        ref, r0 = _run(prep)
    finally:
        thysea.force_tiling(None)
    got, r = _run(prep)
    assert r["kernel_launches"] < r["iterations"] < r0["kernel_launches"]
    assert r["iterations"] == r0["iterations"] and r["deep_tiles"] == r0["deep_tiles"]
    for k in FIELDS:
        assert np.array_equal(got[k], ref[k], equal_nan=True), k


def _spike(nx, ny):
    """a finite initial state whose fluxes overflow in the first step"""
    p = _problem(nx, ny, "file", 300.0)
    p.eta_init[ny // 2, nx // 3] = 1e30
    return p


def test_scenarios_that_fail_in_a_resident_batch(gpu):
    """values that are not finite end their scenario in the same step for every
    CTA: a chunk whose last running scenarios fail ends, the others of a chunk
    finish as alone, and the batch's next chunks find the barriers in order"""
    goods = [_problem(256, 240, "open", 900.0), _problem(230, 256, "file", 900.0)]
    alone = [_run(thysea.Prepared(p)) for p in goods]
    spikes = [_spike(96, 80), _spike(113, 64), _spike(200, 190)]
    srv = thysea.Server(hbm_budget_bytes=2 << 30, max_scenarios=8)
    bad = [srv.submit(p) for p in spikes]   # no other scenario in these chunks
    srv.drain()
    before = srv.stats()["chunks"]
    bad += [srv.submit(p) for p in spikes[:1]]
    ids = [srv.submit(p) for p in goods]
    bad += [srv.submit(p) for p in spikes[1:]]
    srv.drain()
    chunks = srv.stats()["chunks"] - before
    srv.close()
    for rid in bad:
        assert srv.results[rid]["status"] == thysea.THY_ERR_NONFINITE
        assert srv.results[rid]["stats"]["steps"] == 1
    for rid, (ref, r) in zip(ids, alone):
        assert srv.results[rid]["status"] == 0
        assert srv.results[rid]["stats"]["steps"] == r["iterations"]
        for k in FIELDS:
            assert np.array_equal(srv.results[rid]["outputs"][k], ref[k], equal_nan=True), k
    # (launched chunks of a queue are 16 steps long)
    assert chunks < max(r["iterations"] for _, r in alone) / 16


def test_scenario_that_fails_late_in_a_resident_batch(gpu):
    """a second fault whose deformation overflows single precision, in mid-run: the
    scenario ends at the same step alone and in a batch, whose other scenarios, one
    that ends before and one after it, finish as alone"""
    bad = _problem(200, 190, "late", 600.0)
    bad.points, bad.series_time, bad.save_time = None, -1.0, -1.0
    bad.faults[1] = dataclasses.replace(bad.faults[1], slip=1e300)
    goods = [_problem(120, 100, "open", 200.0), _problem(230, 256, "file", 900.0)]
    alone = [_run(thysea.Prepared(p)) for p in goods]
    srv = thysea.Server(hbm_budget_bytes=2 << 30, max_scenarios=8)
    first = srv.submit(bad)
    srv.drain()
    ids = [srv.submit(p) for p in (goods[0], bad, goods[1])]
    srv.drain()
    srv.close()
    steps = srv.results[first]["stats"]["steps"]
    assert srv.results[first]["status"] == srv.results[ids[1]]["status"] == thysea.THY_ERR_NONFINITE
    assert steps > 64 and srv.results[ids[1]]["stats"]["steps"] == steps
    for rid, (ref, r) in zip((ids[0], ids[2]), alone):
        assert srv.results[rid]["status"] == 0
        assert srv.results[rid]["stats"]["steps"] == r["iterations"]
        for k in FIELDS:
            assert np.array_equal(srv.results[rid]["outputs"][k], ref[k], equal_nan=True), k


def test_barrier_timeout_is_reported_and_the_chunk_can_be_stepped_again(gpu):
    """one block that stays away from a resident chunk's barriers: the others'
    waits run out, the steps fail with THY_ERR_TIMEOUT, and the next chunk starts
    on cleared barrier words from the state of the last good one"""
    prep = thysea.Prepared(_problem(641, 512, "open", 3600.0))
    ref = thysea.Session(prep)
    ref.steps(16)
    ref.steps(48)
    want = ref.fetch()
    s = thysea.Session(prep)
    _, k = s.steps(16)
    before, t = s.launches(), s.time()
    assert k == 16 and before < 16   # resident
    s.inject(2)
    for _ in range(2):
        with pytest.raises(thysea.ThyError) as e:
            s.steps(16)
        assert e.value.code == thysea.THY_ERR_TIMEOUT
        assert s.time() == t
    s.inject(0)
    _, k = s.steps(48)
    assert k == 48
    assert s.time() == ref.time() and s.tiles() == ref.tiles()
    got = s.fetch()
    for key in want:
        assert np.array_equal(got[key], want[key], equal_nan=True), key
    s.close()
    ref.close()


def test_unstepped_resident_chunk_takes_the_launched_kernels(gpu):
    """a resident chunk that its blocks leave unstepped (too few of them found a
    free SM): separate launches step it, with the same results"""
    prep = thysea.Prepared(_problem(500, 411, "open", 3600.0))
    ref, s = thysea.Session(prep), thysea.Session(prep)
    ref.steps(16)
    ref.steps(40)
    s.steps(16)
    assert s.launches() < 16
    s.inject(4)
    n = s.launches()
    _, k = s.steps(40)
    assert k == 40 and s.launches() - n == 5 * 40   # five launches a step
    assert ref.launches() < 16
    assert s.time() == ref.time() and s.tiles() == ref.tiles()
    got, want = s.fetch(), ref.fetch()
    for key in want:
        assert np.array_equal(got[key], want[key], equal_nan=True), key
    s.close()
    ref.close()


_BESIDE = """
import sys, time
import numpy as np
import torch
import thysea
import test_gpu_resident as t

prep = thysea.Prepared(t._problem(256, 240, "late", 900.0))
ref, r0 = t._run(prep)
streams, side = [torch.cuda.Stream() for _ in range(int(sys.argv[1]))], torch.cuda.Stream()
x = torch.zeros(1024, device="cuda")
x.add_(1.0)
torch.cuda.synchronize()
t0 = time.perf_counter()
for st in streams:
    with torch.cuda.stream(st):
        torch.cuda._sleep(int(7.6e9))   # one block, four seconds
got, r = t._run(prep)
with torch.cuda.stream(side):
    x.add_(1.0)
side.synchronize()
waited = time.perf_counter() - t0
assert not any(st.query() for st in streams)   # they are still running
torch.cuda.synchronize()
assert waited < 2.0, waited   # (a run takes 0.01 s; a host may stall)
assert r["iterations"] == r0["iterations"] and r["kernel_launches"] < r["iterations"]
for k in t.FIELDS:
    assert np.array_equal(got[k], ref[k], equal_nan=True), k
"""


@pytest.mark.parametrize("blocks", [1, 3])
def test_resident_chunks_beside_another_streams_long_kernels(gpu, blocks):
    """SMs held by other streams' kernels for seconds: a run does not wait for
    their end (its chunks are stepped by the blocks that find a free SM), other
    kernels are not held back by it, and the results are the same.  (In a process
    with a hardware queue for each of its streams.)"""
    env = dict(os.environ, CUDA_DEVICE_MAX_CONNECTIONS="32",
               PYTHONPATH=os.pathsep.join([os.path.dirname(os.path.abspath(__file__)), *sys.path]))
    r = subprocess.run([sys.executable, "-c", _BESIDE, str(blocks)], env=env, capture_output=True, text=True, timeout=200)
    assert r.returncode == 0, r.stderr[-3000:]


def test_runs_of_several_threads_share_the_gpu(gpu):
    """runs of several host threads at a time, each on its share of the SMs: the
    results of each alone"""
    import threading

    sizes = [(96, 80, "file"), (256, 240, "late"), (500, 411, "open"), (113, 95, "late"), (1024, 700, "open"), (200, 640, "file")]
    preps = [thysea.Prepared(_problem(nx, ny, kind, 400.0)) for nx, ny, kind in sizes]
    alone = [_run(p) for p in preps]
    out = [[] for _ in preps]
    start = threading.Barrier(len(preps))

    def work(k):
        start.wait()
        for _ in range(4):
            out[k].append(_run(preps[k]))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(preps))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (ref, r0), runs in zip(alone, out):
        assert len(runs) == 4
        for got, r in runs:
            assert r["iterations"] == r0["iterations"] and r["deep_tiles"] == r0["deep_tiles"]
            for k in FIELDS:
                assert np.array_equal(got[k], ref[k], equal_nan=True), k
