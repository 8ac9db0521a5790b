"""Performance cases of the time stepper: what a user of the library has it do.

A case is one call (or one short program) through the public entry points:
whole simulations through thysea.run(), a queue of scenarios through
thysea.Server, step-level use through thysea.Session, and the Okada stage on
device memory through thy_apply_okada.  `listed()` names the cases that are
timed, `draw()` gives further ones of the same ranges, and `exact()` restates
the FP64 scheme with torch for the accuracy of the results.

Sizes are those of the seeded workloads in thysea.synth (sides 256 to 4096, one
arc-minute cells, 600 to 3600 s simulated) and of the tests (small grids, odd
sizes, walls, periodic longitudes, crops, faults at two times, initial states
from a file, gauges and snapshots).
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "tsunami-hysea_b200"))

import thysea  # noqa: E402
from thysea import _ffi, synth  # noqa: E402

BORDERS = {"open": (1.0, 1.0, 1.0, 1.0), "wall": (-1.0, -1.0, -1.0, -1.0), "channel": (1.0, -1.0, 2.0, 2.0)}
EARTH_RADIUS_M = 6378136.6
FIELDS = thysea.OUTPUT_FIELDS


def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def run_case(name, nx, ny, sim_time, **more):
    """A thysea.run() case: `coast` "ramp" (linear shelf), "shelf" (random-field
    ocean, shelf and about 10 % land) or "basin" (no land); `faults` Okada
    sources (0: initial surface from a file), `late` moves the last of them to
    mid-run; snapshots and gauges by their counts over the run."""
    c = dict(name=name, kind="run", nx=nx, ny=ny, sim_time=float(sim_time), arcmin=1.0, lat=0.0, coast="shelf",
             borders="open", faults=1, late=False, crop=0, snapshots=0, gauges=0)
    assert set(more) <= set(c)
    c.update(more)
    return c


def listed():
    return [
        # the smallest simulations: a harbour-sized basin started from a surface
        # file, a few dozen steps; fixed costs per call and per step
        run_case("basin_96x80_file", 96, 80, 240.0, coast="ramp", borders="wall", faults=0, gauges=6),
        # a small regional run with two sources (one late), crop, gauges; odd sides
        run_case("coast_289x211_late_fault", 289, 211, 600.0, faults=2, late=True, crop=1, gauges=8, snapshots=2),
        # the plain small problem: 512^2, ten minutes, snapshots every 300 s, 16 gauges every minute
        run_case("plain_512", 512, 512, 600.0, coast="ramp", snapshots=2, gauges=16),
        # a periodic channel of odd sides (wrap in longitude, wall below, sponge above)
        run_case("channel_733x517", 733, 517, 900.0, borders="channel", crop=2),
        # an ordinary regional run
        run_case("shelf_1024", 1024, 1024, 900.0, snapshots=1),
        # one scenario of the uniform batch: 2048^2, half an hour
        run_case("batch_member_2048", 2048, 2048, 1800.0),
        # a periodic belt of the globe at 4 arc-minutes, two hours
        run_case("belt_5400x1801", 5400, 1801, 7200.0, arcmin=4.0, borders="channel", faults=2),
        # the headline: 4096^2, four subfaults, one hour
        run_case("large_4096", 4096, 4096, 3600.0, faults=4),
        # a queue of mixed-size scenarios handed to the server at once
        dict(name="server_mixed_12", kind="server", count=12, side_lo=256, side_hi=1100, time_lo=600.0, time_hi=1200.0),
        # many small scenarios of one size in one batch
        dict(name="server_uniform_24x256", kind="server", count=24, side_lo=256, side_hi=256, time_lo=600.0, time_hi=600.0),
        # step-level use: 128 steps of a 1500 x 1100 grid, then the fields
        dict(name="session_1500x1100", kind="session", nx=1500, ny=1100, steps=128, coast="shelf", borders="open"),
        # the Okada stage alone, on a caller's device state
        dict(name="okada_2048", kind="okada", nx=2048, ny=2048, crop=1, noalloc=False),
    ]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "server", "session", "okada"])
    if kind == "okada":
        noalloc = rng.random() < 0.4
        return dict(kind=kind, nx=log_uniform(rng, 200, 1000 if noalloc else 4000),
                    ny=log_uniform(rng, 200, 1000 if noalloc else 4000), crop=rng.choice([0, 1, 2]), noalloc=noalloc)
    if kind == "session":
        return dict(kind=kind, nx=log_uniform(rng, 120, 3000), ny=log_uniform(rng, 120, 3000),
                    steps=rng.randrange(20, 200), coast=rng.choice(["shelf", "ramp", "basin"]),
                    borders=rng.choice(["open", "wall", "channel"]))
    if kind == "server":
        lo = log_uniform(rng, 150, 500)
        return dict(kind=kind, count=rng.randrange(4, 25), side_lo=lo, side_hi=log_uniform(rng, lo, 1100),
                    time_lo=600.0, time_hi=float(rng.randrange(600, 1300)))
    nx, ny = log_uniform(rng, 80, 4096), log_uniform(rng, 80, 4096)
    faults = rng.choice([0, 1, 1, 2, 4])
    c = run_case("", nx, ny, rng.randrange(600, 1800) if nx * ny > 200000 else rng.randrange(200, 1200),
                 coast=rng.choice(["shelf", "shelf", "ramp", "basin"]),
                 lat=rng.choice([0.0, 30.0, -45.0]) if ny < 1500 else 0.0,
                 borders=rng.choice(["open", "open", "wall", "channel"]), faults=faults,
                 late=faults > 1 and rng.random() < 0.5, crop=rng.choice([0, 0, 1, 2]) if faults else 0,
                 snapshots=rng.choice([0, 0, 1, 3]), gauges=rng.choice([0, 0, 8, 16]))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def bathymetry(nx, ny, coast, seed):
    """Topobathymetry (m, positive up) as synth makes it, on the device."""
    dev = device()
    gen = torch.Generator(device=dev).manual_seed(seed)
    noise = torch.randn((ny, nx), generator=gen, device=dev, dtype=torch.float64)
    x = torch.arange(nx, device=dev, dtype=torch.float64)
    if coast == "ramp":
        x0 = int(round(0.85 * nx))
        prof = torch.where(x >= x0, -4000.0 + (x - x0) * (4200.0 / max(nx - 1 - x0, 1)), torch.full_like(x, -4000.0))
        return (prof[None, :] + 20.0 * noise).to(torch.float32).cpu().numpy()
    corr = min(50.0, max(nx, ny) / 4.0)
    kx = torch.fft.rfftfreq(nx, device=dev, dtype=torch.float64)
    ky = torch.fft.fftfreq(ny, device=dev, dtype=torch.float64)
    k2 = ky[:, None] ** 2 + kx[None, :] ** 2
    f = torch.fft.irfft2(torch.fft.rfft2(noise) * torch.exp(-2.0 * (math.pi * corr) ** 2 * k2), s=(ny, nx))
    f = f - f.mean()
    f = f / f.std()
    ocean = (-3000.0 + 800.0 * f).clamp(-7000.0, -50.0)
    if coast == "basin":
        return ocean.to(torch.float32).cpu().numpy()
    s = ((x / max(nx - 1, 1) - 0.75) / 0.25).clamp(0.0, 1.0)[None, :]
    lo, hi = 0.0, 20000.0
    for _ in range(20):
        land = 0.5 * (lo + hi)
        if float((ocean * (1.0 - s) + s * land > 0).double().mean()) < 0.10:
            lo = land
        else:
            hi = land
    return (ocean * (1.0 - s) + s * 0.5 * (lo + hi)).to(torch.float32).cpu().numpy()


def make_problem(case, seed):
    nx, ny, rng = case["nx"], case["ny"], np.random.default_rng(seed)
    lon, lat = synth.lonlat_grid(nx, ny, case["arcmin"] * synth.ARCMIN, lat_centre=case["lat"])
    z = bathymetry(nx, ny, case["coast"], seed)
    p = synth.Problem(name="case", lon=lon, lat=lat, z=z, borders=BORDERS[case["borders"]], sim_time=case["sim_time"])
    for k in range(case["faults"]):
        # contiguous 100 x 50 km subfaults along strike, as in the single large problem
        c_lon = float(lon[0] + rng.uniform(0.3, 0.5) * (lon[-1] - lon[0]))
        c_lat = float(0.5 * (lat[0] + lat[-1])) + (k - 0.5 * (case["faults"] - 1)) * 100.0 / synth.KM_PER_DEG
        late = case["late"] and k == case["faults"] - 1
        p.faults.append(synth.Fault(0.4 * case["sim_time"] if late else 0.0, c_lon, c_lat,
                                    synth.centroid_depth(10.0, 50.0, 15.0), 100.0, 50.0, float(rng.uniform(0.0, 40.0)),
                                    15.0, 90.0, float(rng.uniform(2.0, 8.0))))
    if not p.faults:
        x0, y0 = rng.uniform(0.3, 0.6) * nx, rng.uniform(0.3, 0.6) * ny
        r2 = (np.arange(ny)[:, None] - y0) ** 2 + (np.arange(nx)[None, :] - x0) ** 2
        p.eta_init = (rng.uniform(1.0, 3.0) * np.exp(-r2 / (0.1 * min(nx, ny)) ** 2)).astype(np.float32)
    p.crop_flag = case["crop"]
    p.crop_value = {0: 0.0, 1: 5e-3, 2: 0.05}[case["crop"]]
    if case["snapshots"]:
        p.save_time = case["sim_time"] / case["snapshots"]
    if case["gauges"]:
        ocean = np.flatnonzero(z.ravel() < -100.0)
        pick = ocean[rng.choice(len(ocean), size=case["gauges"], replace=False)]
        p.points = np.stack([lon[pick % nx], lat[pick // nx]], axis=1)
        p.series_time = case["sim_time"] / 10.0
    return p


def server_members(case, seed):
    """The scenarios of a server case: sides log-spaced over the range, one
    random fault each (the mixed batch)."""
    out = []
    for k in range(case["count"]):
        f = k / max(case["count"] - 1, 1)
        side = int(round(case["side_lo"] * (case["side_hi"] / case["side_lo"]) ** f))
        out.append(run_case("m", side, side, case["time_lo"] + (case["time_hi"] - case["time_lo"]) * ((k * 7) % 5) / 4.0))
    return [(c, make_problem(c, seed * 64 + k)) for k, c in enumerate(out)]


def session_case(case):
    """A session steps on for as long as it is asked: its simulated time has no end here."""
    return run_case("s", case["nx"], case["ny"], 1e8, coast=case["coast"], borders=case["borders"])


def okada_inputs(case, seed):
    gen = torch.Generator(device=device()).manual_seed(seed)
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    dep = 0.5 + 5.5 * torch.rand(nx * ny, generator=gen, device=device(), dtype=torch.float64)
    state = torch.stack([(dep - 0.3).clamp(min=0.0), dep], dim=1).contiguous()
    f = np.array([0.0, 9.0 + rng.uniform(0.3, 0.7) * nx / 60.0, 3.5 + rng.uniform(0.3, 0.7) * ny / 60.0,
                  16.47, 100.0, 50.0, rng.uniform(0.0, 360.0), rng.uniform(10.0, 30.0), 90.0, rng.uniform(2.0, 8.0)])
    return state, torch.zeros(nx * ny, device=device(), dtype=torch.float64), f


# ---------------------------------------------------------------------------
# a pass
# ---------------------------------------------------------------------------

class PageLocked:
    """Field arrays the program keeps for its outputs, page-locked for as long as it lives."""

    def __init__(self, shapes):
        self.flat = {k: np.zeros(sum(a * b for a, b in shapes), np.float32) for k in FIELDS}
        for v in self.flat.values():
            assert _ffi.lib().thy_host_register(v.ctypes.data, v.nbytes) == 0
        self.views, at = [], 0
        for a, b in shapes:
            self.views.append({k: v[at:at + a * b].reshape(a, b) for k, v in self.flat.items()})
            at += a * b

    def __del__(self):
        for v in self.flat.values():
            _ffi.lib().thy_host_unregister(v.ctypes.data)


def prepare(case, seed):
    if case["kind"] == "run":
        prep = thysea.Prepared(make_problem(case, seed)).pin()
        return case, prep, PageLocked([(case["ny"], case["nx"])])
    if case["kind"] == "server":
        preps = [thysea.Prepared(p).pin() for _, p in server_members(case, seed)]
        outs = PageLocked([(int(p.c.ny), int(p.c.nx)) for p in preps])
        return case, thysea.Server(hbm_budget_bytes=8 << 30, max_scenarios=32), preps, outs
    if case["kind"] == "session":
        return case, thysea.Session(make_problem(session_case(case), seed))
    return case, okada_inputs(case, seed)


def run(state):
    case = state[0]
    if case["kind"] == "run":
        _, prep, outs = state
        r = thysea.run(prep, snapshots=case["snapshots"] > 0, series=case["gauges"] > 0, out=outs.views[0])
        got = {k: r[k] for k in FIELDS}
        got["iterations"], got["final_time"] = int(r["iterations"]), float(r["final_time"])
        if case["snapshots"]:
            got["snapshots"] = r["snapshots"]
        if case["gauges"]:
            got["series"] = r["series"]
        return got
    if case["kind"] == "server":
        _, srv, preps, outs = state
        ids = [srv.submit(p, out=v) for p, v in zip(preps, outs.views)]
        srv.drain()
        res = [srv.results.pop(i) for i in ids]
        got = dict(outs.flat)
        got["status"] = np.array([r["status"] for r in res])
        got["steps"] = np.array([r["stats"]["steps"] for r in res])
        return got
    if case["kind"] == "session":
        _, ses = state
        ses.steps(case["steps"])
        return ses.fetch()
    _, (dev_state, eta0, fault) = state
    f = _ffi.lib().thy_apply_okada_noalloc if case["noalloc"] else _ffi.lib().thy_apply_okada
    crop_value = {0: 0.0, 1: 5e-3, 2: 5e-5}[case["crop"]]
    rc = f(case["nx"], case["ny"], 9.0, 1.0 / 60.0, 3.5, 1.0 / 60.0, fault.ctypes.data_as(_ffi.f64p), 1000.0,
           case["crop"], crop_value, ctypes.c_void_p(dev_state.data_ptr()), ctypes.c_void_p(eta0.data_ptr()),
           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    return {"state": dev_state, "eta_initial": eta0}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def expected_steps(nx, ny, sim_time, arcmin=1.0, lat=0.0, coast="shelf"):
    """Time steps of a run, from the CFL condition over its deepest water."""
    depth = 4070.0 if coast == "ramp" else 6300.0
    dy = EARTH_RADIUS_M * math.radians(arcmin / 60.0)
    edge = min(89.0, abs(lat) + 0.5 * ny * arcmin / 60.0)
    dx = dy * math.cos(math.radians(edge))
    return max(1.0, sim_time / (0.5 / (math.sqrt(9.81 * depth) * (1.0 / dx + 1.0 / dy))))


def work(case):
    """A step of a cell reads the surface, the depth and two discharges and
    writes the new surface, discharges and, as it grows, the maximum height
    (in phases: 36 + 24 bytes) in about 350 operations; a run also reads its
    FP64 problem and writes its fields."""
    if case["kind"] == "okada":
        n = case["nx"] * case["ny"]
        return {"bytes": 32.0 * n, "flops": 700.0 * n}
    if case["kind"] == "session":
        n = case["nx"] * case["ny"]
        return {"bytes": n * (60.0 * case["steps"] + 16.0), "flops": 350.0 * n * case["steps"]}
    if case["kind"] == "server":
        total = {"bytes": 0.0, "flops": 0.0}
        for k in range(case["count"]):
            side = case["side_lo"] * (case["side_hi"] / case["side_lo"]) ** (k / max(case["count"] - 1, 1))
            t = case["time_lo"] + (case["time_hi"] - case["time_lo"]) * ((k * 7) % 5) / 4.0
            steps = expected_steps(side, side, t)
            total["bytes"] += side * side * (60.0 * steps + 56.0)
            total["flops"] += 350.0 * side * side * steps
        return total
    n = case["nx"] * case["ny"]
    steps = expected_steps(case["nx"], case["ny"], case["sim_time"], case["arcmin"], case["lat"], case["coast"])
    return {"bytes": n * (60.0 * steps + 56.0 + 12.0 * case["snapshots"]), "flops": 350.0 * n * steps}


# ---------------------------------------------------------------------------
# the FP64 scheme
# ---------------------------------------------------------------------------

EPS = 2.220446049250313e-16


def inv_depth(h, eps):
    return math.sqrt(2.0) * h / torch.sqrt(h ** 4 + h.clamp(min=eps) ** 4)


def limiter(pm, p0, p1, pp, wave):
    mid = p1 - p0
    up = torch.where(wave < 0, pp - p1, torch.where(wave > 0, p0 - pm, 0.5 * (pp - pm)))
    same = (mid * up >= 0).double()
    mid, up = mid.abs(), up.abs()
    a = ((up - mid) / (up + mid)).abs()
    u = 0.5 * (up + mid) * (1.0 - a ** 3)
    r = torch.where(mid > u, u / (mid + EPS), mid / (u + EPS))
    return torch.where(mid < EPS, torch.ones_like(mid), same * r * (1.0 + r) / (1.0 + r * r))


def spread(v, dim, periodic):
    """v with two cells more on each side of `dim`: wrapped or repeated."""
    n = v.shape[dim]
    if periodic:
        return torch.cat([v.narrow(dim, n - 2, 2), v, v.narrow(dim, 0, 2)], dim)
    first, last = v.narrow(dim, 0, 1), v.narrow(dim, n - 1, 1)
    return torch.cat([first, first, v, last, last], dim)


class Scheme:
    """One scenario in FP64: the 2s / 2s+WAF step, Okada sources, metrics and outputs."""

    def __init__(self, p):
        dev, f8 = device(), torch.float64
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=f8, device=dev)  # noqa: E731
        self.p, self.ny, self.nx = p, p.ny, p.nx
        self.H, self.Q = p.H, math.sqrt(9.81 * p.H ** 3)
        self.T = p.L * p.H / self.Q
        self.eps, self.hpos, self.cvis = p.eps_h / p.H, p.hpos / p.H, 1.0 - p.stability
        self.mf0 = p.manning * (9.81 * p.manning * p.L / p.H ** (4.0 / 3.0))
        self.vmax, self.dif_at = p.vmax / (self.Q / p.H), p.dif_at / p.H
        self.b = p.borders
        self.periodic = p.borders[2] == 2.0 and p.borders[3] == 2.0
        self.sponge = [4 if v == 1.0 else 0 for v in p.borders]   # up, low, left, right
        self.D = t(-p.z.astype(np.float64) / p.H)
        if p.eta_init is None:
            self.h = self.D.clamp(min=0.0)
        else:
            self.h = (t(p.eta_init.astype(np.float64) / p.H) + self.D).clamp(min=0.0)
        self.qx, self.qy = torch.zeros_like(self.h), torch.zeros_like(self.h)
        dlat = np.abs(np.diff(p.lat))
        dlat = np.append(dlat, dlat[-1])
        dlon = abs(p.lon[1] - p.lon[0])
        self.dlat, self.cos = t(dlat)[:, None], t(np.cos(p.lat * (math.pi / 180.0)))[:, None]
        self.area = t(EARTH_RADIUS_M / p.L * dlon * dlat * (math.pi / 180.0))[:, None]
        self.dlon = float(dlon)
        em = torch.where(self.h < self.eps, torch.full_like(self.h, -1e30), self.h - self.D)
        self.top, self.first, self.arr = em, em.clone(), torch.full_like(em, -1.0)
        self.sponge_tables(dev, f8)

    def sponge_tables(self, dev, f8):
        up, low, left, right = self.sponge
        x = torch.arange(self.nx, device=dev, dtype=f8)[None, :]
        y = torch.arange(self.ny, device=dev, dtype=f8)[:, None]
        far = lambda d: torch.where(d <= 0, torch.full_like(d, 1e30), d)  # noqa: E731
        one = torch.ones((self.ny, self.nx), device=dev, dtype=f8)
        dx, dy = self.dlon * one, self.dlat * one
        parts = [((left - x - 0.5) * dx, dx * left), ((x - (self.nx - 1 - right) - 0.5) * dx, dx * right),
                 ((up - y - 0.5) * dy, dy * up), ((y - (self.ny - 1 - low) - 0.5) * dy, dy * low)]
        dist, ls = far(parts[0][0]), parts[0][1]
        for d, n in parts[1:]:
            nearer = far(d) < dist
            dist, ls = torch.where(nearer, far(d), dist), torch.where(nearer, n, ls)
        inside = ((x < left) | (x >= self.nx - right) | (y < up) | (y >= self.ny - low)) & (one > 0)
        self.any_sponge = any(self.sponge)
        self.relax = torch.where(inside, 0.9 * (dist / ls.clamp(min=1e-300)) ** 2, torch.zeros_like(one))
        damp = lambda d, n, use: torch.where(use & (one > 0), 1.0 - 0.9 * (d / n.clamp(min=1e-300)) ** 2, one)  # noqa: E731
        self.damp_x = damp(*parts[0], x < left) * damp(*parts[1], x >= self.nx - right)
        self.damp_y = damp(*parts[2], y < up) * damp(*parts[3], y >= self.ny - low)

    def edges(self, dim):
        """The four stencil cells of every edge along `dim`, ghost sides set up:
        where the ghost is on the low side the sides change places."""
        per = self.periodic and dim == 1
        n = self.nx if dim == 1 else self.ny
        u, v = (self.qx, self.qy) if dim == 1 else (self.qy, self.qx)
        e = {}
        for key, f in (("h", self.h), ("D", self.D), ("u", u), ("v", v)):
            s = spread(f, dim, per)
            e[key] = [s.narrow(dim, k, n + 1) for k in range(4)]
        if dim == 1:
            e["a"], e["c"] = [self.area, self.area], [self.cos, self.cos]
            e["len"] = self.dlat / self.cos
        else:
            for key, f in (("a", self.area), ("c", self.cos)):
                s = spread(f, 0, False)
                e[key] = [s.narrow(0, 1, n + 1), s.narrow(0, 2, n + 1)]
            e["len"] = torch.full_like(e["c"][0], self.dlon)
        at = torch.arange(n + 1, device=self.h.device)
        at = at[None, :] if dim == 1 else at[:, None]
        e["nolim"] = (at < 2) | (at > n - 2)
        e["ghost"] = (at == 0) & (not per)
        e["normal"] = torch.where(e["ghost"], -1.0, 1.0).double()
        if not per:
            lo, hi = (self.b[2], self.b[3]) if dim == 1 else (self.b[0], self.b[1])
            u0 = torch.where(at == 0, e["u"][1] * lo, e["u"][1])
            u1 = torch.where(at == n, e["u"][2] * hi, e["u"][2])
            e["u"] = [e["u"][0], u0, u1, e["u"][3]]
            for key in ("h", "D", "u", "v"):
                w = [x.clone() for x in e[key]]
                for k in range(4):
                    w[k].narrow(dim, 0, 1).copy_(e[key][3 - k].narrow(dim, 0, 1))
                e[key] = w
        e["deep"] = (e["h"][0] > self.hpos) & (e["h"][1] > self.hpos) & (e["h"][2] > self.hpos) & (e["h"][3] > self.hpos)
        e["deep"] = e["deep"] & ~e["nolim"]
        return e

    def wet_dry(self, e):
        (_, h0, h1, _), (_, D0, D1, _) = e["h"], e["D"]
        w0, w1 = e["u"][1] * e["normal"], e["u"][2] * e["normal"]
        e0, e1 = h0 - D0, h1 - D1
        w1 = torch.where((h0 < self.eps) & (-e1 > D0), torch.zeros_like(w1), w1)
        w0 = torch.where((h1 < self.eps) & (-e0 > D1), torch.zeros_like(w0), w0)
        return w0, w1

    def waf(self, e, uij, u0n, u1n, s0, s1, c0, dt):
        el = [h - D for h, D in zip(e["h"], e["D"])]
        val = 2.0 * e["len"] * dt / (e["a"][0] + e["a"][1])
        lo, hi = torch.minimum(uij - c0, u0n - s0), torch.maximum(uij + c0, u1n + s1)
        zero = torch.zeros_like(lo)
        xl = torch.where(e["nolim"], zero, limiter(*el, lo))
        xr = torch.where(e["nolim"], zero, limiter(*el, hi))
        al = torch.sign(lo) * (1.0 - xl) + val * lo * xl
        bl = torch.sign(hi) * (1.0 - xr) + val * hi * xr
        maxa = torch.maximum(hi.abs(), lo.abs())
        split = (lo - hi).abs() >= EPS
        inv = 1.0 / torch.where(split, hi - lo, torch.ones_like(lo))
        a0 = torch.where(split, (al - bl) * (lo * hi) * inv, maxa)
        a1 = torch.where(split, (bl * hi - al * lo) * inv, zero)
        return val, maxa, a0, a1

    def jump(self, e):
        Hm = torch.minimum(e["D"][1], e["D"][2])
        return (e["h"][2] - e["D"][2] + Hm).clamp(min=0.0) - (e["h"][1] - e["D"][1] + Hm).clamp(min=0.0)

    def blend(self, e, hij):
        w = torch.where(hij < self.hpos, 1.0 / (1.0 + torch.exp(-15.0 * (1.0 - 0.5 * self.hpos / (hij + EPS)))),
                        torch.ones_like(hij))
        return torch.where(e["nolim"], torch.zeros_like(w), w)

    def mass(self, dim, dt):
        """Mass flux of every edge along `dim`, and its share in each row's terms."""
        e = self.edges(dim)
        (_, h0, h1, _), (c0s, c1s), y = e["h"], e["c"], dim == 0
        w0, w1 = self.wet_dry(e)
        u0n, u1n = inv_depth(h0, self.eps) * w0, inv_depth(h1, self.eps) * w1
        w0, w1 = u0n * h0, u1n * h1
        s0, s1, hij = h0.sqrt(), h1.sqrt(), 0.5 * (h0 + h1)
        uij = (s0 * u0n + s1 * u1n) / (s0 + s1 + EPS)
        _, _, a0, _ = self.waf(e, uij, u0n, u1n, s0, s1, hij.sqrt(), dt)
        wc0, wc1 = (c0s, c1s) if y else (1.0, 1.0)
        deta = self.jump(e)
        if y:
            deta = 0.5 * (c0s + c1s) * deta - uij * uij * (c1s - c0s)
        f2s = e["len"] * w0 * wc0 * e["normal"]
        fwaf = 0.5 * (w0 * wc0 + w1 * wc1 - a0 * deta) * e["len"]
        k = self.blend(e, hij)
        F = torch.where(e["deep"], e["len"] * e["u"][1] * wc0, k * f2s + (1.0 - k) * fwaf)
        F = torch.where((h0 > EPS) | (h1 > EPS), F, torch.zeros_like(F))
        cap = torch.where(F > 0, 0.25 * h0 * wc0 * e["a"][0], 0.25 * h1 * wc1 * e["a"][1]) / (F.abs() + EPS)
        F = torch.where(dt > cap, F * cap / (dt + EPS), F)
        lo, hi = (-F / c0s, F / c1s) if y else (-F, F)
        hi = torch.where(e["ghost"], lo, hi)
        n = self.ny if y else self.nx
        return lo.narrow(dim, 1, n) + hi.narrow(dim, 0, n)

    def momentum(self, dim, dt):
        """Shares of every cell in the momentum fluxes along `dim`: (qx, qy, wave speed)."""
        e = self.edges(dim)
        (hm, h0, h1, hp), (c0s, c1s), y, ln, nr = e["h"], e["c"], dim == 0, e["len"], e["normal"]
        w0, w1 = self.wet_dry(e)
        r0, r1 = inv_depth(h0, self.eps), inv_depth(h1, self.eps)
        u0n, u1n = r0 * w0, r1 * w1
        if not y:
            w0, w1 = u0n * h0, u1n * h1
        s0, s1, hij = h0.sqrt(), h1.sqrt(), 0.5 * (h0 + h1)
        uij = (s0 * u0n + s1 * u1n) / (s0 + s1 + EPS)
        val, maxa, a0, a1 = self.waf(e, uij, u0n, u1n, s0, s1, hij.sqrt(), dt)
        deep = e["deep"]
        maxa = torch.where(deep, uij.abs() + hij.sqrt(), maxa)
        deta, i0, i1, wc0, wc1 = self.jump(e), 1.0, 1.0, 1.0, 1.0
        if y:
            i0, i1, wc0, wc1 = 1.0 / c0s, 1.0 / c1s, c0s, c1s
            deta = 0.5 * (c0s + c1s) * deta - uij * uij * (c1s - c0s)
        left = uij < 0
        un, uw, ut = (torch.where(left, b, a) for a, b in ((u0n, u1n), (w0, w1), (e["v"][1], e["v"][2])))
        base = un * uw * ln * nr
        s_n0 = torch.where(left, base * (wc1 * i0), base) + hij * deta * ln * i0
        s_n1 = torch.where(left, -base, -base * (wc0 * i1))
        s_t0 = un * ut * ln
        f0, f1 = w0 * wc0, w1 * wc1
        dq = f1 - f0
        soft = torch.where(deep, torch.ones_like(hij), 1.0 / (1.0 + torch.exp(-20.0 * (1.0 - self.hpos / hij))))
        des = 0.5 * (1.0 - self.cvis * soft) * val * maxa * maxa * dq * ln * (1.0 if y else nr)
        s_n0, s_n1 = s_n0 - des * i0, s_n1 + des * i1
        mx = 0.5 * dq
        my = 0.5 * (u1n * f1 - u0n * f0 + hij * deta)
        dx_, dy_ = 0.5 * a0 * deta, 0.5 * a0 * dq + a1 * my
        fx = (mx + f0 - dx_) * ln
        t_n0, t_n1 = (my + u0n * f0 - dy_) * ln, (my + dy_ - u1n * f1) * ln
        sg = -nr if y else nr
        q = [inv_depth(h, self.eps) * v * sg for h, v in zip((hm, h0, h1, hp), e["v"])]
        side = torch.sign(fx)
        speed = uij.abs() * side
        xi = torch.where(e["nolim"], torch.zeros_like(fx), limiter(*q, speed))
        ut = 0.5 * (q[1] * i0 + q[2] * i1) - 0.5 * ((1.0 - xi) * side + xi * speed * val) * (q[2] * i1 - q[1] * i0)
        t_t0 = fx * ut * sg
        k = torch.where(deep, torch.ones_like(hij), self.blend(e, hij))
        mix = lambda a, b: torch.where(deep, a, k * a + (1.0 - k) * b)  # noqa: E731
        n0, n1 = mix(s_n0, t_n0 * nr * i0), mix(s_n1, t_n1 * nr * i1)
        t0, t1 = mix(s_t0, t_t0), mix(-s_t0, -t_t0)
        lam = ln * torch.where(~deep & (maxa < self.eps), maxa + self.eps, maxa)
        wet = (h0 > EPS) | (h1 > EPS)
        n = self.ny if y else self.nx
        out = []
        for a, b in ((n0, n1), (t0, t1), (lam, lam)):
            a, b = torch.where(wet, a, torch.zeros_like(a)), torch.where(wet, b, torch.zeros_like(b))
            out.append(a.narrow(dim, 1, n) + torch.where(e["ghost"], a, b).narrow(dim, 0, n))
        return (out[1], out[0], out[2]) if y else (out[0], out[1], out[2])

    def first_dt(self):
        total = 0.0
        for dim in (1, 0):
            e = self.edges(dim)
            h0, h1 = e["h"][1], e["h"][2]
            u0n, u1n = inv_depth(h0, self.eps) * e["u"][1], inv_depth(h1, self.eps) * e["u"][2]
            s0, s1 = h0.sqrt(), h1.sqrt()
            a = ((s0 * u0n + s1 * u1n) / (s0 + s1 + EPS)).abs() + (0.5 * (h0 + h1)).sqrt()
            lam = e["len"] * torch.where(a < self.eps, a + self.eps, a)
            n = self.nx if dim else self.ny
            total = total + lam.narrow(dim, 1, n) + lam.narrow(dim, 0, n)
        return self.bound(total)

    def bound(self, lam):
        s = 2.0 * self.p.cfl * self.area / torch.where(lam < EPS, torch.ones_like(lam), lam)
        return float(torch.where(lam < EPS, torch.full_like(s, 1e30), s).min())

    def step(self, dt):
        """One time step; the next dt."""
        p = self.p
        h = self.h + dt / self.area * (self.mass(1, dt) + self.mass(0, dt))
        h = h.clamp(min=0.0)
        if self.any_sponge:
            h = (h - self.relax * (h - self.D.clamp(min=0.0))).clamp(min=0.0)
        self.h = h
        ax, bx, lx = self.momentum(1, dt)
        ay, by, ly = self.momentum(0, dt)
        nxt = self.bound(lx + ly)
        old = torch.sqrt(self.qx ** 2 + self.qy ** 2)
        qx, qy = self.qx - dt / self.area * (ax + ay), self.qy - dt / self.area * (bx + by)
        if self.any_sponge:
            qx, qy = qx * self.damp_x, qy * self.damp_y
        damp = torch.exp(-dt / ((h / self.eps) ** 4 + EPS))
        fac = inv_depth(h, self.eps)
        fx, fy = qx * damp, qy * damp
        if p.vmax > 0:
            ux, uy = fac * fx, fac * fy
            u = torch.sqrt(ux * ux + uy * uy)
            cut = torch.where(u > self.vmax, self.vmax / u.clamp(min=1e-300), torch.ones_like(u))
            fx, fy = ux * cut * h, uy * cut * h
        fr = h / (1.0 + dt * self.mf0 * (fac * old) / (h ** (4.0 / 3.0) + EPS))
        wet = h > 0
        fx, fy = torch.where(wet, fr * fac * fx, fx), torch.where(wet, fr * fac * fy, fy)
        near = h <= self.hpos
        self.qx, self.qy = torch.where(near, fx, qx), torch.where(near, fy, qy)
        return nxt

    def metrics(self, t):
        e = self.h - self.D
        self.top = torch.where((e > self.top) & (self.h > self.eps), e, self.top)
        self.arr = torch.where((self.arr < 0) & ((e - self.first).abs() > self.dif_at), torch.full_like(e, t), self.arr)

    def deform(self, f):
        p = self.p
        lon = p.lon[0] + np.arange(p.nx) * ((p.lon[-1] - p.lon[0]) / (p.nx - 1))
        lat = p.lat[0] + np.arange(p.ny) * ((p.lat[-1] - p.lat[0]) / (p.ny - 1))
        U = okada_uplift(torch.as_tensor(lon, device=self.h.device)[None, :],
                         torch.as_tensor(lat, device=self.h.device)[:, None], f) / p.H
        U = crop(U, p.crop_flag, p.crop_value / p.H if p.crop_flag == 2 else p.crop_value)
        self.D, self.first = self.D - U, self.first + U

    def velocity(self):
        h, eps = self.h, self.eps
        f = torch.where(h < eps, math.sqrt(2.0) * h / torch.sqrt(h ** 4 + eps ** 4), 1.0 / h.clamp(min=eps)) * (self.Q / self.H)
        return self.qx * f, self.qy * f

    def state(self):
        eta = torch.where(self.h < self.eps, torch.full_like(self.h, -9999.0), (self.h - self.D) * self.H)
        return (eta, *self.velocity())

    def peak(self):
        return torch.where(self.top < -1e20, torch.full_like(self.top, -9999.0), self.top * self.H)

    def simulate(self, max_steps=None):
        p, T = self.p, self.T
        faults = sorted((f.as_row() for f in p.faults), key=lambda r: r[0])
        tf = [f[0] for f in faults]
        t, end, due, jumping, steps = 0.0, p.sim_time / T, 0, False, 0
        snaps, series, next_nc, next_ts = [], [], 0.0, 0.0
        cells = None
        if p.points is not None:
            ix = np.abs(p.lon[None, :] - p.points[:, :1]).argmin(1)
            iy = np.abs(p.lat[None, :] - p.points[:, 1:]).argmin(1)
            cells = torch.as_tensor(iy * p.nx + ix, device=self.h.device)

        def clip(dt, jumping):
            """dt shortened to land on the next fault time (of another time than
            the pending one, when the last step landed on it)."""
            k = due
            if jumping:
                while k < len(tf) and tf[k] - tf[due] <= EPS:
                    k += 1
            if k < len(tf) and (t + dt) * T > tf[k]:
                return tf[k] / T - t, True
            return dt, False

        dt = self.first_dt()
        if tf:
            dt, jumping = clip(dt, tf[0] < EPS)
        while t < end and (max_steps is None or steps < max_steps):
            while due < len(tf) and t * T >= tf[due]:
                self.deform(faults[due])
                due += 1
            if p.save_time >= 0 and t >= next_nc:
                next_nc += p.save_time / T
                snaps.append((t * T, *self.state()))
            if cells is not None and t >= next_ts:
                next_ts += p.series_time / T
                u, v = self.velocity()
                series.append((t * T, ((self.h - self.D) * self.H).reshape(-1)[cells], u.reshape(-1)[cells],
                               v.reshape(-1)[cells]))
            self.metrics(t)
            nxt = self.step(dt)
            t += dt
            dt, jumping = clip(nxt, jumping)
            steps += 1
        eta, ux, uy = self.state()
        arr = torch.where(self.arr < 0, torch.full_like(self.arr, -1.0), self.arr * T)
        out = {"max_height": self.peak(), "arrival": arr, "deformed_bathy": self.D * self.H, "eta": eta, "ux": ux, "uy": uy,
               "iterations": steps, "final_time": t * T}
        stack = lambda rows, k: torch.stack([r[k] for r in rows])  # noqa: E731
        if snaps:
            out["snapshots"] = {"time": np.array([r[0] for r in snaps]), "eta": stack(snaps, 1), "ux": stack(snaps, 2),
                                "uy": stack(snaps, 3)}
        if series:
            e = stack(series, 1)
            out["series"] = {"time": np.array([r[0] for r in series]), "eta": e, "ux": stack(series, 2),
                             "uy": stack(series, 3), "min": e.min(0).values, "max": e.max(0).values,
                             "bathy": (self.D * self.H).reshape(-1)[cells]}
        return out


def crop(U, flag, value):
    if flag == 1:
        return torch.where(U.abs() < value * float(U.abs().max().float()), torch.zeros_like(U), U)
    if flag == 2:
        return torch.where(U.abs() < value, torch.zeros_like(U), U)
    return U


def okada_uplift(lon, lat, fault):
    """Vertical displacement (m) of one rectangular source (Okada 1985), at
    lon/lat projected about the source's centre (Gauss-Krueger)."""
    _, lon0, lat0, depth, L, W, strike, dip, rake, slip = (float(v) for v in fault)
    deg = 0.017453292371619689
    rlat = lat * deg
    dl = lon - lon0
    clat = torch.cos(rlat)
    ph1 = lat + (clat * 0.0067397251 * clat + 1.0) * 0.5 * dl * dl * torch.sin(rlat) * clat * deg
    d = torch.sqrt(1.0 - torch.sin((ph1 + lat0) * 0.5 * deg) ** 2 * 0.0066946053)
    rn = 6378.16 / torch.sqrt(1.0 - torch.sin(ph1 * deg) ** 2 * 0.0066946053)
    north = (ph1 - lat0) / (57.29578 / (6335.4607362597517 / d ** 3))
    east = dl * clat / (57.29578 / rn) * (dl * dl * torch.cos(rlat * 2.0) / 19696.838434850401 + 1.0)
    ss, cs = math.sin(math.radians(strike)), math.cos(math.radians(strike))
    x, y = east * ss + north * cs, -east * cs + north * ss
    sd, cd = math.sin(math.radians(dip)), math.cos(math.radians(dip))
    U1, U2 = slip * math.cos(math.radians(rake)), slip * math.sin(math.radians(rake))
    p, q = y * cd + depth * sd, y * sd - depth * cd
    uz = 0.0
    for j, X in enumerate((x + 0.5 * L, x - 0.5 * L)):
        for k, E in enumerate((p + 0.5 * W, p - 0.5 * W)):
            R = torch.sqrt(X * X + E * E + q * q)
            b = E * sd - q * cd
            theta = torch.atan(X * E / (q * R))
            Xs = torch.sqrt(X * X + q * q)
            I4 = 0.5 / cd * (torch.log(R + b) - sd * torch.log(R + E))
            I5 = 1.0 / cd * torch.atan((E * (Xs + q * cd) + Xs * (R + Xs) * sd) / (X * (R + Xs) * cd))
            fss = b * q / R / (R + E) + q * sd / (R + E) + I4 * sd
            fds = b * q / R / (R + X) + sd * theta - I5 * sd * cd
            uz = uz + (-1.0 if j != k else 1.0) * (-U1 * fss - U2 * fds) / (2.0 * math.pi)
    return uz


def exact(case, seed):
    """What run() returns, in FP64; None where that would take too long (cells x steps)."""
    if case["kind"] == "okada":
        state, eta0, fault = okada_inputs(case, seed)
        i, j = torch.arange(case["nx"], device=device()).double(), torch.arange(case["ny"], device=device()).double()
        U = okada_uplift(9.0 + i[None, :] / 60.0, 3.5 + j[:, None] / 60.0, fault) / 1000.0
        U = crop(U, case["crop"], {0: 0.0, 1: 5e-3, 2: 5e-5}[case["crop"]]).reshape(-1)
        return {"state": torch.stack([state[:, 0], state[:, 1] - U], dim=1), "eta_initial": eta0 + U}
    if work(case)["flops"] > 350.0 * 5.0e9:
        return None
    if case["kind"] == "session":
        r = Scheme(make_problem(session_case(case), seed)).simulate(case["steps"])
        return {k: r[k] for k in ("max_height", "eta", "ux", "uy")}
    if case["kind"] == "server":
        got = [Scheme(p).simulate() for _, p in server_members(case, seed)]
        out = {k: torch.cat([r[k].reshape(-1) for r in got]) for k in FIELDS}
        return {**out, "status": None, "steps": None}
    r = Scheme(make_problem(case, seed)).simulate()
    return {**r, "iterations": None}
