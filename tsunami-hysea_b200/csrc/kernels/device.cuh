// Device-side data structures and FP32 edge-flux arithmetic of the B200
// time stepper.
//
// State of one scenario in HBM (all FP32, row-major with a padded pitch):
//   eta[2]  free-surface elevation above the undisturbed sea level (m / H)
//   dep     still-water depth, positive down, Okada-deformed (m / H);
//           water depth h = eta + dep (h = 0 exactly on dry cells: eta = -dep)
//   qx[2], qy[2]  discharges (x: along longitude, y: along latitude)
//   eta_max, arr, eta_ini   max-height / arrival-time diagnostics
// eta and q are double-buffered: phase 1 reads eta[p] and writes eta[p^1],
// phase 2 reads eta[p^1], q[p] and writes q[p^1]; the controller flips p.
//
// Storing eta instead of h keeps ~1e-10 resolution on the wave itself
// (h ~ 4 in units of H would quantise the surface to ~0.5 mm); every place
// where the reference forms a surface difference from h - H uses eta.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace thy {

constexpr float kEps = 2.220446049250313e-16f;  // the reference's EPSILON (DBL_EPSILON)
constexpr float kSqrt2 = 1.41421356237309505f;
constexpr int kSponge = 4;

// scenario status (ScenarioCtl::status)
enum : int {
    kRunning = 0,
    kPaused = 1,   // an event (fault, snapshot, gauge sample) is due at time t
    kDone = 2,     // t >= t_end or the step budget is used
    kFailed = 3,   // non-finite state or time step
    kIdle = 4,     // slot not in use / not started
};

// pause reasons (bit mask, ScenarioCtl::events)
enum : int { kEvFault = 1, kEvSnapshot = 2, kEvSeries = 4, kEvStepBudget = 8 };

struct RowMetrics {
    // per row y (ny entries unless noted), FP64 on the host, rounded once
    const float *cosphi;     // cos(lat)
    const float *ilcos;      // x-edge length / cos(lat)  (dlat / cos)
    const float *area;       // cell area
    const float *dlon;       // y-edge length at edge row y (ny+1 entries); sponge dx
    const float *dlat;       // sponge dy
};

// Mutable per-scenario control block; written by the host between chunks and by
// the step controller that ends each step (phase 2's last CTA, or a launch of its
// own; a resident chunk's CTAs each advance a copy, stored at the chunk's end).
struct ScenarioCtl {
    double t;            // simulated time (dimensionless)
    double dt;           // time step of the next step
    double t_end;
    double save_nc, next_nc;   // snapshot interval / next snapshot time (< 0: off)
    double save_ts, next_ts;   // gauge interval / next gauge time
    double T;                  // time scale (s)
    long long step;            // completed steps
    long long max_steps;       // < 0: unlimited
    int status;
    int events;
    int parity;
    int fault_next;            // index of the next fault to apply
    int jumping;               // the reference's saltar_deformacion
    int nfaults;
    unsigned int dt_bits;      // atomicMin target (positive float bits)
    unsigned int tiles_done;   // phase-0 tiles finished (initial dt)
    unsigned int errors;       // bit 0 non-finite values, bit 1 a bounded wait ran out, bit 2 misaligned staging
    int inject;                // test hook: bit 0 = the deep kernels issue none of this scenario's copies,
                               // bit 1 = a CTA of its resident chunks stays away from the barriers,
                               // bit 2 = its resident chunks are not stepped
    const double *fault_times; // nfaults fault times (s), sorted, device memory
    unsigned long long units_deep;   // work units stepped by the deep-water kernels (phase 2)
    unsigned long long units_dry;    // work units skipped as dry land (classifications)
    unsigned int gauge_count;  // gauge samples the controller took (ring slot = count % kGaugeRing)
};

// Gauge samples taken on the device between two reads by the host: at most
// one per step, and the host reads them after every chunk of at most
// kGaugeRing steps.
constexpr int kGaugeRing = 64;

// Opaque 128-byte TMA tensor map (CUtensorMap), 64-byte aligned in device memory.
struct alignas(64) TmaMap {
    unsigned long long opaque[16];
};

// tensor maps of a scenario: state planes boxed kStageW x kStageRows (the
// staged window of a half tile), diagnostics boxed kTileX x kHalfRows
enum : int {
    kMapEta0 = 0, kMapEta1, kMapQx0, kMapQx1, kMapQy0, kMapQy1, kMapDep, kMapEtaMax, kMapArr, kMapEtaIni, kNumMaps
};
constexpr int kHalfRows = 16;                 // rows of a half tile
constexpr int kStageW = 120;                  // staged columns: x0-4 .. x0+115 (16-byte aligned start)
constexpr int kStageRows = kHalfRows + 2;     // staged rows: one above and one below the half tile

// Depth summary of a work unit for one state: {min, max} of eta + dep over
// the unit, over its two-cell border strips (left, right, top, bottom: the
// unit's first / last two columns or rows inside the grid) and over its four
// 2 x 2 corners - exactly the cells the two-cell stencil ring of a
// neighbouring unit reaches into.
struct UnitSum {
    float2 all, L, R, T, B, TL, TR, BL, BR;
};

struct ScenarioDev {
    int nx, ny, pitch;
    int tiles_x, tiles_y, ntiles;
    int x_org;   // grid column of tile 0's first column (tile_origin: 0 or -4 .. -108)
    int periodic;
    float b_up, b_low, b_left, b_right;
    int sp_up, sp_low, sp_left, sp_right;
    float cfl, eps_h, hpos, cvis, mf0, vmax, dif_at, sea;
    double eps_h64;   // eps_h in double for the FP64 set-up / output thresholds
    float *eta[2];
    float *qx[2];
    float *qy[2];
    float *dep;
    float *eta_max;
    float *arr;
    float *eta_ini;
    // per work unit (half tile of kTileX x kHalfRows cells from column
    // x_org + tx kTileX; unit (tx, uy) at uy * tiles_x + tx): depth summary of the state phase 1 produces (index
    // parity^1); NaN = unknown
    UnitSum *usum[2];
    // per unit: consecutive classifications that found its 3 x 3 unit
    // neighbourhood dry (saturating)
    unsigned char *dry_age;
    // per unit: the largest |dep1 - dep0| between the two cells of an edge of
    // the unit's cells (x edges x0 .. x0+112 of its rows, y edges yb .. yb+16
    // of its columns, inside the grid); fixed between faults.  A deep unit
    // whose unit and two-cell ring are all deeper than this steps its
    // surface jumps as the plain difference (see surface_jump)
    float *unit_gmax;
    // TMA tensor maps of the field planes (kMap* order), null when the grid
    // is too small to have deep tiles
    const struct TmaMap *tmap;
    // per row y (ny+1 entries): {cos, ilcos, area, dlon} (dlon of edge row y;
    // the other three unused in entry ny)
    const float4 *rowpack;
    RowMetrics row;
    ScenarioCtl *ctl;
    // gauges (time-series points), sampled by the step controller at each
    // gauge time that does not coincide with a fault
    const int *gauge_cells;   // ngauges cell indices (y nx + x; -1: outside the grid)
    int ngauges;
    float *gauge_ring;        // kGaugeRing samples of ngauges x {eta, ux, uy, depth} (m, m/s)
    double *gauge_ring_t;     // their times (s)
    float2 *gauge_minmax;     // per gauge {min, max} of eta over every sample (-9999 outside the grid)
    double Hs, Qs;            // depth and discharge scales (dimensional outputs)
};

// One gauge of the state at `parity` in dimensional units (eta, ux, uy,
// depth: src/GPU/Volumen_kernel.cu:223-254 with the output scaling of
// src/GPU/netcdfSeries.cu), -9999 for a point outside the grid; folds eta into
// the gauge's {min, max} when minmax is not null (the running extremes of
// src/GPU/netcdfSeries.cu:125,138).
__device__ __forceinline__ void gauge_values(const ScenarioDev &s, int parity, int cell, float *out4, float2 *minmax)
{
    if (cell < 0) {
        out4[0] = out4[1] = out4[2] = out4[3] = -9999.0f;
        return;
    }
    const int x = cell % s.nx, y = cell / s.nx;
    const size_t idx = (size_t)y * s.pitch + x;
    const double eta = (double)s.eta[parity][idx], D = (double)s.dep[idx];
    const double h = eta + D, eps_h = s.eps_h64;
    double f;
    if (h < eps_h) {
        const double e4 = eps_h * eps_h * eps_h * eps_h;
        f = 1.41421356237309505 * h / sqrt(h * h * h * h + e4);
    } else {
        f = 1.0 / h;
    }
    const float e = (float)(eta * s.Hs);
    out4[0] = e;
    out4[1] = (float)(f * (double)s.qx[parity][idx] * s.Qs / s.Hs);
    out4[2] = (float)(f * (double)s.qy[parity][idx] * s.Qs / s.Hs);
    out4[3] = (float)(D * s.Hs);
    if (minmax) {
        float2 m = *minmax;
        m.x = (m.x < e) ? m.x : e;
        m.y = (e < m.y) ? m.y : e;
        *minmax = m;
    }
}

// The control of one scenario after a step (src/GPU/ShallowWater.cu:397-450
// loop body after the step; src/GPU/Timestep.cu:35-68 dt truncation to fault
// times): time, next dt (dmin: the step's CFL minimum), status and events in
// c.  Returns the ring slot of a gauge sample to take at this step (at c.t), or -1.
__device__ __forceinline__ int advance_scenario(ScenarioCtl &c, const ScenarioDev &s, float dmin, unsigned errs)
{
    int sample = -1;
    c.t += c.dt;
    double dt = (double)dmin;
    // truncation so that t lands on the next fault time
    const int nf = c.nfaults;
    const int f = c.fault_next;
    const double *tf = c.fault_times;
    if (!c.jumping) {
        if (f < nf && (c.t + dt) * c.T > tf[f]) {
            dt = tf[f] / c.T - c.t;
            c.jumping = 1;
        }
    } else {
        c.jumping = 0;
        if (f < nf) {
            int i = f + 1;
            while (i < nf && !(fabs(tf[i] - tf[f]) > 2.220446049250313e-16)) i++;
            if (i < nf && (c.t + dt) * c.T > tf[i]) {
                dt = tf[i] / c.T - c.t;
                c.jumping = 1;
            }
        }
    }
    c.dt = dt;
    c.step += 1;
    c.parity ^= 1;
    c.dt_bits = 0x7f7fffffu;
    c.tiles_done = 0u;
    int ev = 0;
    if (errs || !(dmin > 0.f) || isnan(dmin)) {
        c.status = kFailed;
    } else if (!(c.t < c.t_end)) {
        c.status = kDone;
    } else if (c.max_steps >= 0 && c.step >= c.max_steps) {
        c.events = kEvStepBudget;
        c.status = kDone;
    } else {
        if (f < nf && c.t * c.T >= tf[f]) ev |= kEvFault;
        if (c.save_nc >= 0.0 && c.t >= c.next_nc) ev |= kEvSnapshot;
        if (c.save_ts >= 0.0 && c.t >= c.next_ts) {
            if (s.ngauges > 0 && !(ev & kEvFault)) {
                // the loop's gauge event on the device: same time test
                // and interval update as the host's
                sample = (int)(c.gauge_count % kGaugeRing);
                c.next_ts += c.save_ts;
                c.gauge_count += 1;
            } else {
                ev |= kEvSeries;
            }
        }
        if (ev) {
            c.events = ev;
            c.status = kPaused;
        }
    }
    return sample;
}

// the fields advance_scenario changes, back to the scenario's control block
__device__ __forceinline__ void store_advanced(ScenarioCtl *cp, const ScenarioCtl &c)
{
    cp->t = c.t;
    cp->dt = c.dt;
    cp->step = c.step;
    cp->parity = c.parity;
    cp->jumping = c.jumping;
    cp->dt_bits = c.dt_bits;
    cp->tiles_done = c.tiles_done;
    cp->events = c.events;
    cp->status = c.status;
    cp->next_ts = c.next_ts;
    cp->gauge_count = c.gauge_count;
}

__host__ __device__ inline float fmax_(float a, float b) { return (a < b) ? b : a; }
__host__ __device__ inline float fmin_(float a, float b) { return (b < a) ? b : a; }

__device__ __forceinline__ float sgnf(float a) { return (a > 0.f) ? 1.f : ((a < 0.f) ? -1.f : 0.f); }
__device__ __forceinline__ float pow4f(float a) { float b = a * a; return b * b; }

// Approximate reciprocal square root and square root of the stepping
// kernels.  The square root is x * rsqrt(x), an approximate reciprocal square
// root and one multiply, written out so that every call site computes it
// with the same two instructions: an approximate sqrtf is not lowered alike
// at every site, and then two warp tilings of the same cells, which reach the
// same formula through different code, differ in the last bit.
// sqrt_ap(0) = 0; a negative or NaN argument gives NaN.
__device__ __forceinline__ float rsqrt_ap(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sqrt_ap(float x)
{
    return x == 0.f ? 0.f : __fmul_rn(x, rsqrt_ap(x));
}

// Desingularised 1/h (src/GPU/Arista_kernel.cu:164): sqrt2 h / sqrt(h^4 + max(h,eps)^4),
// which is exactly 1/h for h >= eps.
__device__ __forceinline__ float inv_depth(float h, float eps)
{
    if (h >= eps) return __frcp_rn(h);
    return kSqrt2 * h * rsqrt_ap(pow4f(h) + pow4f(eps));
}

// Limits a mass flux so that neither side loses more than 1/4 of its water in
// one step (src/GPU/Arista_kernel.cu:79-114; c0/c1 = cos(lat) for y edges).
// dt > dt0 = cap / (|F| + eps) is tested as dt (|F| + eps) > cap, so the
// divisions only run when the limit applies.
__device__ __forceinline__ float limit_outflow(float F, float h0, float h1, float c0, float c1, float dt, float a0, float a1)
{
    const float cap = (F > 0.f) ? 0.25f * h0 * c0 * a0 : 0.25f * h1 * c1 * a1;
    const float aF = fabsf(F) + kEps;
    if (dt * aF > cap) F *= (cap / aF) / (dt + kEps);
    return F;
}

// Surface-gradient term max(eta1+Hm,0) - max(eta0+Hm,0) with Hm = min(D0,D1),
// evaluated as eta1 - eta0 whenever both sides are wet at the lower bed so that
// FP32 does not lose the wave to the depth's magnitude.  With h0, h1 > |D1 - D0|
// both sides are (eta1 + Hm >= h1 - |D1 - D0| and eta0 + Hm >= h0 - |D1 - D0|),
// and the term is eta1 - eta0 without the tests.
__device__ __forceinline__ float surface_jump(float e0, float e1, float D0, float D1)
{
    float Hm = fmin_(D0, D1);
    float a = e1 + Hm, b = e0 + Hm;
    if (a > 0.f && b > 0.f) return e1 - e0;
    return fmax_(a, 0.f) - fmax_(b, 0.f);
}

__device__ __forceinline__ void swapf(float &a, float &b) { float t = a; a = b; b = t; }

// ---------------------------------------------------------------------------
// Edges whose four stencil cells are all deeper than hpos and which lie at
// least two cells from a boundary: the 2s blend weight is exactly 1, so the
// flux is the 2s flux alone (the WAF part, the wet/dry tests and the limiter
// drop out).  The general units call these fluxes; the deep units evaluate the
// formulas two edges at a time in packed FP32x2 arithmetic (mass_pair, pair_update in
// step_parts.cuh), the momentum fluxes with roundings of their own.
// ---------------------------------------------------------------------------

// x edge: F = q0 len, outflow-limited (src/GPU/Arista_kernel.cu:118-219, alfa = 1)
__device__ __forceinline__ float mass_2s_x(float q0, float len, float h0, float h1, float dt, float a0, float a1)
{
    return limit_outflow(q0 * len, h0, h1, 1.f, 1.f, dt, a0, a1);
}

// y edge: F = len q0 cos0 (src/GPU/Arista_kernel.cu:674-778, alfa = 1)
__device__ __forceinline__ float mass_2s_y(float q0, float len, float cos0, float cos1, float h0, float h1, float dt,
                                           float a0, float a1)
{
    return limit_outflow(len * q0 * cos0, h0, h1, cos0, cos1, dt, a0, a1);
}

// Per-cell factors of the 2s fluxes, computed once per cell and shared by
// its four edges: 1/h (approximate reciprocal) and sqrt(h).
__device__ __forceinline__ float rcp_depth(float h) { return __fdividef(1.f, h); }

// Constants of the 2s momentum flux that depend only on the edge's row (its
// metrics), the step's dt and the scenario's viscosity: the deep-water kernels
// form them once per row of a unit, the general kernel per edge, with the same
// expressions.
struct XRowK {
    float ilcos;   // len / cos of the row
    float kdes;    // cd * val * ilcos, val = 2 ilcos dt / (area0 + area1), cd = (1 - cvis) / 2
};
__device__ __forceinline__ XRowK make_xrow(float ilcos, float asum, float dt, float cvis)
{
    XRowK k;
    const float val = (2.f * ilcos * dt) / asum;
    k.ilcos = ilcos;
    k.kdes = (0.5f * (1.f - cvis)) * val * ilcos;
    return k;
}
struct YRowK {
    float len, cmid, cdiff, c10;   // len; (cos0 + cos1) / 2; cos1 - cos0; cos1 / cos0
    float c01, li0, kdes0, kdes1;  // cos0 / cos1; len / cos0; cd val len / cos0; cd val len / cos1
    float cos0, cos1;
};
__device__ __forceinline__ YRowK make_yrow(float cos0, float cos1, float icos0, float icos1, float len, float asum,
                                           float dt, float cvis)
{
    YRowK k;
    const float val = (2.f * len * dt) / asum;
    const float kd = (0.5f * (1.f - cvis)) * val * len;
    k.len = len;
    k.cmid = 0.5f * (cos0 + cos1);
    k.cdiff = cos1 - cos0;
    k.c10 = cos1 * icos0;
    k.c01 = cos0 * icos1;
    k.li0 = len * icos0;
    k.kdes0 = kd * icos0;
    k.kdes1 = kd * icos1;
    k.cos0 = cos0;
    k.cos1 = cos1;
    return k;
}

// ---------------------------------------------------------------------------
// Roundings.  The edge fluxes below and the cell updates are written with
// explicit operations (add, sub, mul, fma2p, ...), never left to the
// compiler's contraction: the same cell is stepped by code copies in several
// kernels (tilings, launched and resident steps), and every copy must round
// alike.  Which products are fused is part of the formula.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fadd_rn(a, -b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// a b + c d and a b - c d, the second product rounded first (fma2p, fma2m) or
// the first one (fma2q, fma2n)
__device__ __forceinline__ float fma2p(float a, float b, float c, float d) { return fma_(a, b, mul(c, d)); }
__device__ __forceinline__ float fma2m(float a, float b, float c, float d) { return fma_(a, b, -mul(c, d)); }
__device__ __forceinline__ float fma2q(float a, float b, float c, float d) { return fma_(c, d, mul(a, b)); }
__device__ __forceinline__ float fma2n(float a, float b, float c, float d) { return fma_(-c, d, mul(a, b)); }

// inv_depth with every rounding explicit: the general units' (inv_depth is the
// initial dt's, one code copy).
__device__ __forceinline__ float inv_depth_x(float h, float eps)
{
    if (h >= eps) return __frcp_rn(h);
    const float h2 = mul(h, h), e2 = mul(eps, eps);
    return mul(mul(kSqrt2, h), rsqrt_ap(fma2p(h2, h2, e2, e2)));
}

// Monotone limiter of the WAF correction from the difference across the edge
// and the one upwind of it (src/GPU/Arista_kernel.cu:45-68)
__device__ __forceinline__ float limiter_of(float d_mid, float d_up)
{
    const float same = (mul(d_mid, d_up) >= 0.f) ? 1.f : 0.f;
    const float m = fabsf(d_mid), u = fabsf(d_up);
    const float a = fabsf(__fdividef(sub(u, m), add(u, m)));
    const float v = mul(mul(0.5f, add(u, m)), fma_(-mul(a, a), a, 1.f));
    const bool big = m > v;
    const float r = __fdividef(big ? v : m, add(big ? m : v, kEps));
    const float x = mul(mul(same, r), __fdividef(add(1.f, r), fma_(r, r, 1.f)));
    return m < kEps ? 1.f : x;
}

// Blend weight of the 2s flux against the WAF flux (src/GPU/Arista_kernel.cu:208).
__device__ __forceinline__ float blend_weight(float hij, float hpos, bool no_lim)
{
    const float x = __frcp_rn(add(1.f, __expf(mul(-15.f, fma_(-mul(0.5f, hpos), __fdividef(1.f, add(hij, kEps)), 1.f)))));
    return no_lim ? 0.f : (hij < hpos) ? x : 1.f;
}

// The two sides of an edge along its normal, low side 0 and high side 1: depth,
// surface, still-water depth, sqrt(h), discharge and velocity along the normal
// (velocity: desingularised discharge / h).  A ghost side repeats the cell's
// with the discharge times the border value; where the ghost is on the low side
// the edge is computed mirrored: side 0 is the cell, normal -1.
struct Sides {
    float h0, h1, e0, e1, D0, D1, s0, s1, u0, u1, t0, t1;
    float em, ep;          // surface of the cells next to sides 0 and 1
    float area0, area1, cos0, cos1, len;   // len: x edges len / cos
    float normal;
    bool no_lim;           // within two cells of a boundary: first order, no 2s blend
};

// What both phases form of an edge first: the velocities and discharges without
// flow into a dry cell above the wet neighbour's surface, the Roe velocity, the
// wave speeds and the WAF coefficients' limiters.
struct EdgeWaves {
    float t0, t1, uij, val, lo, hi, maxa, alr, blr, jump, hij;
    bool z0, z1, split;
};
template <bool X_FUSED>   // the mass flux of x edges fuses the Roe velocity's quotient into the wave speeds
__device__ __forceinline__ EdgeWaves edge_waves(const Sides &e, float dt, float eps_h)
{
    EdgeWaves w;
    w.z1 = (e.h0 < eps_h) && (-e.e1 > e.D0);
    w.z0 = (e.h1 < eps_h) && (-e.e0 > e.D1);
    w.t0 = w.z0 ? 0.f : mul(e.t0, e.normal);
    w.t1 = w.z1 ? 0.f : mul(e.t1, e.normal);
    w.hij = mul(0.5f, add(e.h0, e.h1));
    const float c = sqrt_ap(w.hij);
    const float num = fma2p(e.s0, w.t0, e.s1, w.t1), den = add(add(e.s0, e.s1), kEps);
    w.uij = __fdividef(num, den);
    const float rden = __fdividef(1.f, den);
    w.val = __fdividef(mul(mul(2.f, e.len), dt), add(e.area0, e.area1));
    w.lo = fmin_(X_FUSED ? fma_(num, rden, -c) : sub(w.uij, c), sub(w.t0, e.s0));
    w.hi = fmax_(X_FUSED ? fma_(num, rden, c) : add(w.uij, c), add(w.t1, e.s1));
    w.maxa = fmax_(fabsf(w.hi), fabsf(w.lo));
    const float mid = sub(e.e1, e.e0), below = sub(e.e0, e.em), above = sub(e.ep, e.e1), both = mul(0.5f, sub(e.ep, e.em));
    float xl = limiter_of(mid, (w.lo < 0.f) ? above : (w.lo > 0.f) ? below : both);
    float xr = limiter_of(mid, (w.hi < 0.f) ? above : (w.hi > 0.f) ? below : both);
    xl = e.no_lim ? 0.f : xl;
    xr = e.no_lim ? 0.f : xr;
    w.split = fabsf(sub(w.lo, w.hi)) >= kEps;
    w.alr = fma_(mul(w.val, w.lo), xl, mul(sgnf(w.lo), sub(1.f, xl)));
    w.blr = fma_(mul(w.val, w.hi), xr, mul(sgnf(w.hi), sub(1.f, xr)));
    w.jump = surface_jump(e.e0, e.e1, e.D0, e.D1);
    return w;
}

// ---------------------------------------------------------------------------
// phase 1: mass flux through one edge that is not all deep
// (src/GPU/Arista_kernel.cu:118-219 for x edges, 674-778 for y edges).  Returns
// F; the caller applies it as cell0 -= F (/cos0 for y), cell1 += F (/cos1).
// ---------------------------------------------------------------------------
template <bool LAT>
__device__ __forceinline__ float mass_waf(const Sides &e, float dt, float eps_h, float hpos)
{
    const EdgeWaves w = edge_waves<!LAT>(e, dt, eps_h);
    const float q0 = mul(w.t0, e.h0), q1 = mul(w.t1, e.h1);
    const float F2s = LAT ? mul(mul(mul(e.len, q0), e.cos0), e.normal) : mul(mul(e.len, q0), e.normal);
    const float a0 = w.split ? __fdividef(mul(sub(w.alr, w.blr), mul(w.lo, w.hi)), sub(w.hi, w.lo)) : w.maxa;
    float Fwaf;
    if (!LAT) {
        Fwaf = mul(mul(0.5f, fma_(-a0, w.jump, fma_(w.t1, e.h1, q0))), e.len);
    } else {
        const float deta = fma2m(mul(0.5f, add(e.cos0, e.cos1)), w.jump, mul(w.uij, w.uij), sub(e.cos1, e.cos0));
        Fwaf = mul(mul(0.5f, fma_(-a0, deta, fma2p(q0, e.cos0, q1, e.cos1))), e.len);
    }
    const float alfa = blend_weight(w.hij, hpos, e.no_lim);
    const float F = fma2p(alfa, F2s, sub(1.f, alfa), Fwaf);
    const float Fl = limit_outflow(F, e.h0, e.h1, LAT ? e.cos0 : 1.f, LAT ? e.cos1 : 1.f, dt, e.area0, e.area1);
    return ((e.h0 > kEps) || (e.h1 > kEps)) ? Fl : 0.f;
}

// Result of a momentum flux, to be subtracted: components along the normal (n)
// and the tangent (t) for side 0 and side 1, and the wave-speed term for the
// time step (added to both).
struct MomFlux {
    float n0, t0, n1, t1, lam;
};

// Edges whose four stencil cells are all deeper than hpos and which lie at
// least two cells from a boundary: the 2s flux alone (alfa = 1).
// x edge (src/GPU/Arista_kernel.cu:221-280); rh = 1/h (approximate), sh = sqrt(h),
// u normal and v tangential discharge, k = the row's constants
__device__ __forceinline__ MomFlux momentum_2s_x(float h0, float h1, float rh0, float rh1, float s0, float s1, float u0,
                                                 float u1, float v0, float v1, float jump, const XRowK &k)
{
    MomFlux r;
    const float hij = mul(0.5f, add(h0, h1));
    const float u0n = mul(u0, rh0), u1n = mul(u1, rh1);
    const float uij = __fdividef(fma2p(s0, u0n, s1, u1n), add(add(s0, s1), kEps));
    const float maxa = add(fabsf(uij), sqrt_ap(hij));
    const bool neg = uij < 0.f;
    const float un = neg ? u1n : u0n, uu = neg ? u1 : u0, vv = neg ? v1 : v0;
    const float m = mul(mul(un, uu), k.ilcos);
    const float c = mul(k.kdes, mul(maxa, maxa)), du = sub(u1, u0);
    r.n0 = fma_(-c, du, fma_(mul(hij, jump), k.ilcos, m));
    r.n1 = fma_(c, du, -m);
    r.t0 = mul(mul(un, vv), k.ilcos);
    r.t1 = -r.t0;
    r.lam = mul(k.ilcos, maxa);
    return r;
}

// y edge (src/GPU/Arista_kernel.cu:780-843); k = the constants of its row pair
__device__ __forceinline__ MomFlux momentum_2s_y(float h0, float h1, float rh0, float rh1, float s0, float s1, float u0,
                                                 float u1, float v0, float v1, float jump, const YRowK &k)
{
    MomFlux r;
    const float hij = mul(0.5f, add(h0, h1));
    const float u0n = mul(u0, rh0), u1n = mul(u1, rh1);
    const float uij = __fdividef(fma2p(s0, u0n, s1, u1n), add(add(s0, s1), kEps));
    const float maxa = add(fabsf(uij), sqrt_ap(hij));
    const float deta = fma2m(k.cmid, jump, mul(uij, uij), k.cdiff);
    const float g = mul(hij, deta);
    const float m2 = mul(mul(maxa, maxa), fma2m(u1, k.cos1, u0, k.cos0));
    const bool neg = uij < 0.f;
    const float un = neg ? u1n : u0n, uu = neg ? u1 : u0, vv = neg ? v1 : v0;
    const float f = mul(mul(un, uu), k.len);
    // (a factor 1 leaves a product as it is)
    r.n0 = fma_(-k.kdes0, m2, fma2p(g, k.li0, f, neg ? k.c10 : 1.f));
    r.n1 = fma2p(k.kdes1, m2, -f, neg ? 1.f : k.c01);
    r.t0 = mul(mul(un, vv), k.len);
    r.t1 = -r.t0;
    r.lam = mul(k.len, maxa);
    return r;
}

// ---------------------------------------------------------------------------
// phase 2: momentum flux of an edge that is not all deep
// (src/GPU/Arista_kernel.cu:282-464 for x edges, 845-1026 for y edges).  v0, v1:
// tangential discharges; pm, p0, p1, pp: tangential velocities of the four
// stencil cells.
// ---------------------------------------------------------------------------
template <bool LAT>
__device__ __forceinline__ MomFlux momentum_waf(const Sides &e, float v0, float v1, float pm, float p0, float p1, float pp,
                                                float icos0, float icos1, float dt, float eps_h, float hpos, float cvis)
{
    MomFlux r;
    const EdgeWaves w = edge_waves<false>(e, dt, eps_h);
    const float n = e.normal;
    const float w0 = LAT ? (w.z0 ? 0.f : mul(e.u0, n)) : mul(w.t0, e.h0);
    const float w1 = LAT ? (w.z1 ? 0.f : mul(e.u1, n)) : mul(w.t1, e.h1);
    const float deta = LAT ? fma2m(mul(0.5f, add(e.cos0, e.cos1)), w.jump, mul(w.uij, w.uij), sub(e.cos1, e.cos0)) : w.jump;
    const bool neg = w.uij < 0.f;
    const float un = neg ? w.t1 : w.t0;
    const float s = mul(mul(mul(un, neg ? w1 : w0), e.len), n);
    const float f0 = LAT ? mul(w0, e.cos0) : w0, f1 = LAT ? mul(w1, e.cos1) : w1;
    const float g0 = mul(w.t0, f0), g1 = mul(w.t1, f1);
    const float dq = sub(f1, f0);
    const float ex = add(1.f, __expf(mul(-20.f, fma_(-hpos, __fdividef(1.f, w.hij), 1.f))));
    const float cd = mul(0.5f, fma_(-cvis, __fdividef(1.f, ex), 1.f));
    const float des = mul(mul(mul(mul(mul(cd, w.val), w.maxa), w.maxa), dq), e.len);
    float sn0, sn1;
    if (!LAT) {
        sn0 = sub(fma_(mul(w.hij, deta), e.len, s), mul(des, n));
        sn1 = add(-s, mul(des, n));
    } else {
        const float grav = mul(mul(w.hij, deta), e.len);
        sn0 = fma_(-des, icos0, fma_(grav, icos0, neg ? mul(s, mul(e.cos1, icos0)) : s));
        sn1 = fma_(des, icos1, neg ? -s : mul(mul(-s, e.cos0), icos1));
    }
    const float st = mul(mul(un, neg ? v1 : v0), e.len);
    const float aux = __fdividef(1.f, sub(w.hi, w.lo));
    const float a0 = w.split ? mul(mul(sub(w.alr, w.blr), mul(w.lo, w.hi)), aux) : w.maxa;
    const float a1 = w.split ? mul(fma2m(w.blr, w.hi, w.alr, w.lo), aux) : 0.f;
    const float hm = mul(0.5f, dq), hn = mul(0.5f, add(sub(g1, g0), mul(w.hij, deta)));
    const float ha = mul(0.5f, a0);
    const float dn = fma2p(ha, dq, a1, hn);
    const float mx = mul(add(hm, fma_(-ha, deta, f0)), e.len);
    const float my = mul(add(hn, sub(g0, dn)), e.len);
    const float py = mul(add(hn, sub(dn, g1)), e.len);
    // transverse momentum carried with a limited tangential velocity
    const float sg = LAT ? -n : n;
    const float ym = mul(pm, sg), y0 = mul(p0, sg), y1 = mul(p1, sg), yp = mul(pp, sg);
    const float side = sgnf(mx);
    const float speed = mul(fabsf(w.uij), side);
    const float up = (speed < 0.f) ? sub(yp, y1) : (speed > 0.f) ? sub(y0, ym) : mul(0.5f, sub(yp, ym));
    const float xi = e.no_lim ? 0.f : limiter_of(sub(y1, y0), up);
    const float coef = add(mul(sub(1.f, xi), side), mul(mul(xi, speed), w.val));
    const float sum = LAT ? fma2p(y0, icos0, y1, icos1) : add(y0, y1);
    const float dif = LAT ? fma2n(y1, icos1, y0, icos0) : sub(y1, y0);
    const float ut = sub(mul(0.5f, sum), mul(mul(0.5f, coef), dif));
    const float tt = mul(mul(mx, ut), sg);
    const float alfa = blend_weight(w.hij, hpos, e.no_lim), be = sub(1.f, alfa);
    const float tn0 = LAT ? mul(mul(my, n), icos0) : mul(my, n), tn1 = LAT ? mul(mul(py, n), icos1) : mul(py, n);
    r.n0 = fma2p(alfa, sn0, be, tn0);
    r.n1 = fma2p(alfa, sn1, be, tn1);
    r.t0 = fma2q(alfa, st, be, tt);
    r.t1 = -r.t0;
    r.lam = mul(e.len, (w.maxa < eps_h) ? add(w.maxa, eps_h) : w.maxa);
    const bool wet = (e.h0 > kEps) || (e.h1 > kEps);
    r.n0 = wet ? r.n0 : 0.f;
    r.n1 = wet ? r.n1 : 0.f;
    r.t0 = wet ? r.t0 : 0.f;
    r.t1 = wet ? r.t1 : 0.f;
    r.lam = wet ? r.lam : 0.f;
    return r;
}

}  // namespace thy
