// Device code shared by the stepping kernels: cells and their loads, the unit
// classes and depth summaries, the row marching of the general units, and the
// packed pair arithmetic of the deep-water units.  Included by the kernels
// that launch once per phase (step.cu) and by the kernel that keeps a chunk of
// steps on the device (resident.cu); both give bitwise the same results.
#pragma once
#include "device.cuh"
#include "kernels.h"

#include <cfloat>

namespace thy {

constexpr int STRIPS = kStepThreads / 32;   // column strips of a tile
constexpr int OUTW = 28;              // output columns per strip
constexpr int TY = kTileY;            // output rows per tile
static_assert(kTileX == STRIPS * OUTW, "tile width = strips x 28 columns");
static_assert(STRIPS == 4, "deep and general kernels: 4 column-strip warps per row group");

// one cell of a lane's column: depth, surface elevation, still-water depth, discharges
struct Cell {
    float h, e, D, qx, qy;
};

// Column of a loaded cell: periodic wrap or clamp (src/GPU/Arista_kernel.cu:6-21).
// Halo lanes beyond the grid load a valid column (modulo / clamp); only the
// columns the reference would read are used by an edge.
__device__ __forceinline__ int map_col(int gx, int nx, int periodic)
{
    if (gx >= 0 && gx < nx) return gx;
    if (periodic) {
        const int m = gx % nx;
        return m < 0 ? m + nx : m;
    }
    return gx < 0 ? 0 : nx - 1;
}

__device__ __forceinline__ int clamp_row(int gy, int ny) { return gy < 0 ? 0 : (gy >= ny ? ny - 1 : gy); }

// A load of a field.  LIVE: other CTAs of the same launch may have written the
// value (in an earlier phase, ordered by a grid barrier), so it must not take
// the read-only path, whose lines no barrier refreshes.
template <bool LIVE>
__device__ __forceinline__ float ldf(const float *p)
{
    return LIVE ? *p : __ldg(p);
}

template <bool LIVE>
__device__ __forceinline__ Cell load_cell(const float *eta, const float *dep, const float *qx, const float *qy, size_t idx)
{
    Cell c;
    c.e = ldf<LIVE>(eta + idx);
    c.D = ldf<LIVE>(dep + idx);
    c.qx = ldf<LIVE>(qx + idx);
    c.qy = ldf<LIVE>(qy + idx);
    c.h = c.e + c.D;
    return c;
}

// raw loads of a row that is still in flight (prefetch two rows ahead); in
// phase 1 also the cell's max-height / arrival-time / initial-surface values
struct RawCell {
    float e, D, qx, qy;
    float em, ar, ei;
};

template <bool DIAG, bool LIVE>
__device__ __forceinline__ RawCell load_raw(const ScenarioDev &s, const float *eta, const float *qx, const float *qy,
                                            size_t idx, bool diag)
{
    RawCell r;
    r.e = ldf<LIVE>(eta + idx);
    r.D = ldf<LIVE>(s.dep + idx);
    r.qx = ldf<LIVE>(qx + idx);
    r.qy = ldf<LIVE>(qy + idx);
    r.em = r.ar = r.ei = 0.f;
    if (DIAG && diag) {
        r.em = s.eta_max[idx];
        r.ar = s.arr[idx];
        r.ei = ldf<LIVE>(s.eta_ini + idx);
    }
    return r;
}

// Max-height / arrival-time update of one cell from the state the step starts
// from (src/GPU/Metrics.cu:23-77).
__device__ __forceinline__ void diagnostics(const ScenarioDev &s, const RawCell &r, size_t idx, float t_sec)
{
    const float h = r.e + r.D;
    if (r.e > r.em && h > s.eps_h) s.eta_max[idx] = r.e;
    if (r.ar < 0.f && fabsf(r.e - r.ei) > s.dif_at) s.arr[idx] = t_sec;
}

__device__ __forceinline__ float shup(float v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
__device__ __forceinline__ float shdn(float v, int d) { return __shfl_down_sync(0xffffffffu, v, d); }

// Wave-speed term of one edge for the initial dt (src/GPU/Arista_kernel.cu:1237-1280);
// x edges carry len/cos in e.len.
struct SpeedEdge {
    float h0, h1, u0, u1, len, normal;
    bool front;     // ghost on the low side: sides swapped
};
__device__ __forceinline__ float initial_speed(SpeedEdge &e, const ScenarioDev &s)
{
    if (e.front) {
        swapf(e.h0, e.h1);
        swapf(e.u0, e.u1);
    }
    const float w0 = e.u0 * e.normal, w1 = e.u1 * e.normal;
    const float h0 = e.h0, h1 = e.h1, hij = 0.5f * (h0 + h1);
    const float u0n = inv_depth(h0, s.eps_h) * w0, u1n = inv_depth(h1, s.eps_h) * w1;
    const float s0 = sqrt_ap(h0), s1 = sqrt_ap(h1);
    const float uij = (s0 * u0n + s1 * u1n) / (s0 + s1 + kEps);
    float maxa = fabsf(uij) + sqrt_ap(hij);
    if (maxa < s.eps_h) maxa += s.eps_h;
    return e.len * maxa;
}

// the initial speed of the edge between rows gy-1 (a) and gy (b) of a column
__device__ __forceinline__ float initial_speed_y(const ScenarioDev &s, const Cell &a, const Cell &b, int gy, float dlon)
{
    SpeedEdge e{a.h, b.h, a.qy, b.qy, dlon, 1.f, false};
    if (gy == 0) {
        e.u0 *= s.b_up;
        e.normal = -1.f;
        e.front = true;
    }
    if (gy == s.ny) e.u1 *= s.b_low;
    return initial_speed(e, s);
}

// ---------------------------------------------------------------------------
// Work units and their classes.  A unit is a half tile (kTileX x kHalfRows
// cells; tile column tx starts at grid column x_org + tx kTileX, so tile 0
// and the last tile may hold fewer columns); work-list entry w (scenario,
// tile) holds units 2w (upper half) and 2w+1 (lower half).  Phase 1 records each unit's depth summary (UnitSum);
// from the unit's own cells and the border strips and corners of its eight
// neighbours - exactly its two-cell stencil ring -
//   deep:  every cell of unit and ring deeper than hpos, and the unit at
//          least two cells from the boundaries and outside the sponge
//          layers - every edge is a pure 2s edge and no cell is dried,
//          damped or relaxed;
//   dry:   every cell of unit and ring dry (depth 0) at three consecutive
//          classifications - then both state buffers hold the scheme's
//          fixed point (eta = -dep, q = 0), which a step would write again,
//          so the unit is skipped;
//   general: the rest.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int units_y(const ScenarioDev &s) { return (s.ny + kHalfRows - 1) / kHalfRows; }

// The geometric tests imply 1 <= tx <= tiles_x - 2 and 1 <= uy <= units_y - 2.
// *hmin: the smallest depth over the unit and its two-cell ring (when deep).
__device__ __forceinline__ bool unit_deep(const ScenarioDev &s, const UnitSum *sum, int tx, int uy,
                                          float *hmin)
{
    if (!s.tmap) return false;
    const int x0 = s.x_org + tx * kTileX, yb = uy * kHalfRows;
    if (x0 < max(2, s.sp_left) || x0 + kTileX > s.nx - max(2, s.sp_right)) return false;
    if (yb < max(2, s.sp_up) || yb + kHalfRows > s.ny - max(2, s.sp_low)) return false;
    const int W = s.tiles_x;
    const UnitSum *c = sum + (size_t)uy * W + tx;
    const float hp = s.hpos;
    // all nine loads first and no short-circuit, so that they are in flight
    // together (a NaN, an unknown summary, fails its test as before)
    const float v0 = c->all.x, v1 = c[-1].R.x, v2 = c[1].L.x, v3 = c[-W].B.x, v4 = c[W].T.x;
    const float v5 = c[-W - 1].BR.x, v6 = c[-W + 1].BL.x, v7 = c[W - 1].TR.x, v8 = c[W + 1].TL.x;
    *hmin = fminf(fminf(fminf(v0, v1), fminf(v2, v3)), fminf(fminf(v4, v5), fminf(fminf(v6, v7), v8)));
    return (v0 > hp) & (v1 > hp) & (v2 > hp) & (v3 > hp) & (v4 > hp) & (v5 > hp) & (v6 > hp) & (v7 > hp) & (v8 > hp);
}

// Deep-list entries: the unit code (2 x work-list index + half) and, in bit
// kJumpPlain, whether every surface jump of the unit's edges in the state
// the list was made for is the plain difference of the elevations (its unit
// and ring deeper than unit_gmax, with a margin for the FP32 rounding of the
// test itself).
constexpr int kJumpPlain = 30;
__device__ __forceinline__ int unit_code(int entry) { return entry & ((1 << kJumpPlain) - 1); }
__device__ __forceinline__ bool jump_plain(int entry) { return (entry >> kJumpPlain) & 1; }

// Outside the grid counts as dry (ghost cells copy the boundary cell), except
// across a periodic x boundary, where the wrapped unit counts.
__device__ __forceinline__ bool unit_dry(const ScenarioDev &s, const UnitSum *sum, int tx, int uy)
{
    const int ny_u = units_y(s), nx_u = s.tiles_x;
    bool dry = true;
    // every neighbour's load issued without waiting for the previous test
#pragma unroll
    for (int dy = -1; dy <= 1; dy++) {
        const int y = uy + dy;
        if (y < 0 || y >= ny_u) continue;
#pragma unroll
        for (int dx = -1; dx <= 1; dx++) {
            int x = tx + dx;
            if (x < 0 || x >= nx_u) {
                if (!s.periodic) continue;
                x = (x + nx_u) % nx_u;
            }
            const UnitSum &u = sum[(size_t)y * nx_u + x];
            // the part of neighbour (dx, dy) inside the ring
            const float2 v = (dx == 0 && dy == 0) ? u.all
                           : (dy == 0) ? (dx < 0 ? u.R : u.L)
                           : (dx == 0) ? (dy < 0 ? u.B : u.T)
                           : (dy < 0) ? (dx < 0 ? u.BR : u.BL)
                                      : (dx < 0 ? u.TR : u.TL);
            dry &= (v.y <= 0.f);
        }
    }
    return dry;
}

// Per-lane depth accumulators of a unit: every row, the unit's first two
// rows and its last two rows.
struct DepthAcc {
    float amin, amax, tmin, tmax, bmin, bmax;
    __device__ __forceinline__ void init()
    {
        amin = tmin = bmin = FLT_MAX;
        amax = tmax = bmax = -FLT_MAX;
    }
    __device__ __forceinline__ void add(float h, bool top, bool bot)
    {
        amin = fminf(amin, h);
        amax = fmaxf(amax, h);
        if (top) { tmin = fminf(tmin, h); tmax = fmaxf(tmax, h); }
        if (bot) { bmin = fminf(bmin, h); bmax = fmaxf(bmax, h); }
    }
};

// {min, max} over the lanes of a warp that are members, of depths: >= 0, so
// that their bits order as integers (a -0 counts as +0), and a warp reduction
// is one instruction.  The empty value is {FLT_MAX, -FLT_MAX}.
__device__ __forceinline__ float2 warp_minmax(float mn, float mx, bool member)
{
    const int lo = __float_as_int(member ? mn + 0.f : FLT_MAX), hi = __float_as_int(member ? mx + 0.f : -FLT_MAX);
    return make_float2(__int_as_float(__reduce_min_sync(0xffffffffu, lo)), __int_as_float(__reduce_max_sync(0xffffffffu, hi)));
}

constexpr int kDryAge = 3;   // classifications a unit must stay dry before it is skipped

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

struct DeepRow {
    float4 m;      // cos, ilcos, area, dlon (edge row)
    float icos;    // 1/cos, correctly rounded
    // phase 2, for the unit's dt: dt / area, 1 / (2 cfl area), the x edges'
    // XRowK::kdes, and the YRowK of the y edge above the row (y0: len, cmid,
    // cdiff, c10; y1: c01, li0, kdes0, kdes1)
    float dtA, kcfl, kdx;
    float4 y0, y1;
};
static_assert(sizeof(DeepRow) == 64, "row metrics: four float4");

// ---------------------------------------------------------------------------
// Deep phase 2 in pairs: a lane steps two adjacent columns, and the 2s
// momentum fluxes, y edges and updates of the pair run in packed FP32x2
// arithmetic (two lanes of FP32 per instruction, explicit round-to-nearest,
// so no compiler contraction changes a result between code copies).  The
// formulas are those of momentum_2s_x / momentum_2s_y.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 bc2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 sel2(bool px, bool py, float2 a, float2 b)
{
    return make_float2(px ? a.x : b.x, py ? a.y : b.y);
}
// Square roots of a pair (sqrt_ap per component, with its zero test: written
// as a packed x * rsqrt(x) without it, the 16-warp deep phase 2 no longer
// rounded like the other tilings), and 1/h and sqrt(h) of a cell pair from one
// reciprocal square root per cell (deep cells: h > hpos >= 0)
__device__ __forceinline__ float2 sqrt2(float2 h) { return make_float2(sqrt_ap(h.x), sqrt_ap(h.y)); }
struct Depth2 {
    float2 rh, sh;
};
__device__ __forceinline__ Depth2 depth2(float2 h)
{
    const float2 rs = make_float2(rsqrt_ap(h.x), rsqrt_ap(h.y));
    return Depth2{mul2(rs, rs), make_float2(h.x == 0.f ? 0.f : __fmul_rn(h.x, rs.x), h.y == 0.f ? 0.f : __fmul_rn(h.y, rs.y))};
}

// two cells of a staged row (columns i, i + 1; i even)
struct Cell2 {
    float2 h, e, D, qx, qy;
};

struct MomFlux2 {
    float2 m_x, m_y, p_x, p_y, lam;
};
// an edge's fluxes into one of its cells, as momentum_2s_* returns them (the
// cell's update subtracts dt/area times their sum), and its wave-speed term
struct Contrib2 {
    float2 a, b, lam;
};

// momentum_2s_x for two edges at once
__device__ __forceinline__ void momentum_2s_x2(MomFlux2 &r, float2 h0, float2 h1, float2 rh0, float2 rh1, float2 s0,
                                               float2 s1, float2 u0, float2 u1, float2 v0, float2 v1, float2 jump,
                                               const XRowK &k)
{
    const float2 hij = mul2(bc2(0.5f), add2(h0, h1));
    const float2 u0n = mul2(u0, rh0), u1n = mul2(u1, rh1);
    const float2 num = fma2(s0, u0n, mul2(s1, u1n));
    const float2 den = add2(add2(s0, s1), bc2(kEps));
    const float2 uijn = make_float2(__fdividef(num.x, den.x), __fdividef(num.y, den.y));
    const float2 maxa = add2(make_float2(fabsf(uijn.x), fabsf(uijn.y)), sqrt2(hij));
    const bool nx_ = uijn.x < 0.f, ny_ = uijn.y < 0.f;
    const float2 un = sel2(nx_, ny_, u1n, u0n), uu = sel2(nx_, ny_, u1, u0), vv = sel2(nx_, ny_, v1, v0);
    const float2 il = bc2(k.ilcos);
    const float2 mx0 = mul2(mul2(un, uu), il);
    const float2 mx = fma2(mul2(hij, jump), il, mx0);
    const float2 my = mul2(mul2(un, vv), il);
    const float2 des = mul2(mul2(bc2(k.kdes), mul2(maxa, maxa)), sub2(u1, u0));
    r.m_x = sub2(mx, des);
    r.m_y = my;
    r.p_x = sub2(des, mx0);
    r.p_y = neg2(my);
    r.lam = mul2(il, maxa);
}

// momentum_2s_y for two edges at once (one row pair: the constants are shared)
__device__ __forceinline__ void momentum_2s_y2(MomFlux2 &r, float2 h0, float2 h1, float2 rh0, float2 rh1, float2 s0,
                                               float2 s1, float2 u0, float2 u1, float2 v0, float2 v1, float2 jump,
                                               const YRowK &k)
{
    const float2 hij = mul2(bc2(0.5f), add2(h0, h1));
    const float2 u0n = mul2(u0, rh0), u1n = mul2(u1, rh1);
    const float2 num = fma2(s0, u0n, mul2(s1, u1n));
    const float2 den = add2(add2(s0, s1), bc2(kEps));
    const float2 uijn = make_float2(__fdividef(num.x, den.x), __fdividef(num.y, den.y));
    const float2 maxa = add2(make_float2(fabsf(uijn.x), fabsf(uijn.y)), sqrt2(hij));
    const float2 deta = fma2(neg2(mul2(uijn, uijn)), bc2(k.cdiff), mul2(bc2(k.cmid), jump));
    const bool nx_ = uijn.x < 0.f, ny_ = uijn.y < 0.f;
    const float2 un = sel2(nx_, ny_, u1n, u0n), uu = sel2(nx_, ny_, u1, u0), vv = sel2(nx_, ny_, v1, v0);
    const float2 len = bc2(k.len);
    const float2 fym0 = mul2(mul2(un, uu), len);
    // upwind from below: fyp = -fym0, fym = fym0 cos1/cos0; from above: fyp = -fym0 cos0/cos1, fym = fym0
    const float2 fyp = mul2(neg2(fym0), sel2(nx_, ny_, bc2(1.f), bc2(k.c01)));
    const float2 fym = fma2(mul2(hij, deta), bc2(k.li0), mul2(fym0, sel2(nx_, ny_, bc2(k.c10), bc2(1.f))));
    const float2 fxm = mul2(mul2(un, vv), len);
    const float2 m2 = mul2(mul2(maxa, maxa), fma2(u1, bc2(k.cos1), neg2(mul2(u0, bc2(k.cos0)))));
    r.m_x = fxm;
    r.m_y = fma2(bc2(-k.kdes0), m2, fym);
    r.p_x = neg2(fxm);
    r.p_y = fma2(bc2(k.kdes1), m2, fyp);
    r.lam = mul2(len, maxa);
}

// surface jumps of two edges (e0 -> e1); PLAIN: the unit's depths exceed its
// depth steps, so each is the plain difference (the same value)
template <bool PLAIN>
__device__ __forceinline__ float2 jump2(float2 e0, float2 e1, float2 D0, float2 D1)
{
    if (PLAIN) return sub2(e1, e0);
    return make_float2(surface_jump(e0.x, e1.x, D0.x, D1.x), surface_jump(e0.y, e1.y, D0.y, D1.y));
}

// y edge of phase 2 between rows a (metrics ra) and b (rb) for two columns
template <bool PLAIN>
__device__ __forceinline__ void y_edge_deep2(const Cell2 &a, const Cell2 &b, float2 rha, float2 sha, float2 rhb,
                                             float2 shb, const DeepRow &ra, const DeepRow &rb, Contrib2 &lo,
                                             Contrib2 &hi)
{
    YRowK k;
    k.len = rb.y0.x; k.cmid = rb.y0.y; k.cdiff = rb.y0.z; k.c10 = rb.y0.w;
    k.c01 = rb.y1.x; k.li0 = rb.y1.y; k.kdes0 = rb.y1.z; k.kdes1 = rb.y1.w;
    k.cos0 = ra.m.x; k.cos1 = rb.m.x;
    const float2 jump = jump2<PLAIN>(a.e, b.e, a.D, b.D);
    MomFlux2 f;
    momentum_2s_y2(f, a.h, b.h, rha, rhb, sha, shb, a.qy, b.qy, a.qx, b.qx, jump, k);
    lo = {f.m_x, f.m_y, f.lam};
    hi = {f.p_x, f.p_y, f.lam};
}

// Phase 2 of a row of pairs in a deep unit: the x edges left of each lane's
// first column (its left neighbour, with its 1/h and sqrt h, is lane-1's second
// column) and between its two columns, and the momentum update with the shares
// top and below of the y edges.  Lane 0 is halo: its left edge is not used.
// w: the pair's largest lam / (2 cfl area) (0 for lam < eps).
template <bool PLAIN>
__device__ __forceinline__ void pair_update(const Cell2 &c, const Depth2 &f, const DeepRow &rc, const Contrib2 &top,
                                            const Contrib2 &below, float2 &qx, float2 &qy, float &w)
{
    const float le = shup(c.e.y, 1), lh = shup(c.h.y, 1);
    const float lqx = shup(c.qx.y, 1), lqy = shup(c.qy.y, 1);
    const float rhL = shup(f.rh.y, 1), shL = shup(f.sh.y, 1);
    // (the left depth D only for the wet/dry tests of the jump)
    const float2 jump = PLAIN ? sub2(c.e, make_float2(le, c.e.x))
                              : jump2<false>(make_float2(le, c.e.x), c.e, make_float2(shup(c.D.y, 1), c.D.x), c.D);
    MomFlux2 m;
    momentum_2s_x2(m, make_float2(lh, c.h.x), c.h, make_float2(rhL, f.rh.x), f.rh, make_float2(shL, f.sh.x), f.sh,
                   make_float2(lqx, c.qx.x), c.qx, make_float2(lqy, c.qy.x), c.qy, jump, XRowK{rc.m.y, rc.kdx});
    // first column: right cell of the left edge, left cell of the middle edge;
    // second column: right cell of the middle edge, left cell of lane+1's left edge
    const Contrib2 xr = {m.p_x, m.p_y, m.lam};
    const Contrib2 xrr = {make_float2(m.m_x.y, shdn(m.m_x.x, 1)), make_float2(m.m_y.y, shdn(m.m_y.x, 1)),
                          make_float2(m.lam.y, shdn(m.lam.x, 1))};
    const float2 lam = add2(add2(add2(xr.lam, xrr.lam), top.lam), below.lam);
    const float2 k = mul2(lam, bc2(rc.kcfl));
    w = fmaxf(lam.x < kEps ? 0.f : k.x, lam.y < kEps ? 0.f : k.y);
    // q - dtA * (sum of the fluxes), bitwise the sum of the negated fluxes times
    // dtA (negation is exact)
    const float2 val = bc2(-rc.dtA);
    qx = fma2(val, add2(add2(add2(xr.a, xrr.a), top.a), below.a), c.qx);
    qy = fma2(val, add2(add2(add2(xr.b, xrr.b), top.b), below.b), c.qy);
}

// row constants of a deep unit's window: m the row's metrics, above those of the
// row above it, dt folded in
__device__ __forceinline__ DeepRow deep_row(const float4 &m, const float4 &above, float dt, float cfl, float cvis)
{
    DeepRow r;
    r.m = m;
    r.icos = __frcp_rn(m.x);
    r.dtA = __fdividef(dt, m.z);
    r.kcfl = 1.f / (2.f * cfl * m.z);
    r.kdx = make_xrow(m.y, m.z + m.z, dt, cvis).kdes;
    const YRowK k = make_yrow(above.x, m.x, __frcp_rn(above.x), r.icos, m.w, above.z + m.z, dt, cvis);
    r.y0 = make_float4(k.len, k.cmid, k.cdiff, k.c10);
    r.y1 = make_float4(k.c01, k.li0, k.kdes0, k.kdes1);
    return r;
}

// Mass fluxes of two deep edges: len q [cos], outflow-limited (mass_2s_x / _y).
// The limit is tested in pairs with a margin (0.24 of the smaller depth instead
// of 0.25 of the upwind one; km: the smaller cos area of the two sides), the
// exact test and the limit themselves run only where an edge may be limited.
__device__ __forceinline__ float2 limit2(float2 F, float2 h0, float2 h1, float c0, float c1, float a0, float a1, float dt,
                                         float km)
{
    const float2 lhs = mul2(bc2(dt), add2(make_float2(fabsf(F.x), fabsf(F.y)), bc2(kEps)));
    const float2 cap = mul2(bc2(0.24f * km), make_float2(fminf(h0.x, h1.x), fminf(h0.y, h1.y)));
    if (__any_sync(0xffffffffu, !(lhs.x <= cap.x) || !(lhs.y <= cap.y))) {
        F.x = limit_outflow(F.x, h0.x, h1.x, c0, c1, dt, a0, a1);
        F.y = limit_outflow(F.y, h0.y, h1.y, c0, c1, dt, a0, a1);
    }
    return F;
}
__device__ __forceinline__ float2 mass_y2(const Cell2 &a, const Cell2 &b, const float4 &ka, const float4 &kb, float dt)
{
    const float2 F = mul2(mul2(bc2(kb.w), a.qy), bc2(ka.x));
    return limit2(F, a.h, b.h, ka.x, kb.x, ka.z, kb.z, dt, fminf(ka.x, kb.x) * fminf(ka.z, kb.z));
}

// Phase 1 of a pair: its new surface elevations (src/GPU/Volumen_kernel.cu:111-157).
// c and n: its row and the row below with their metrics (1/cos in icos, dt/area in
// dtA); top: the share of the edge above, then of the edge below in its cells
__device__ __forceinline__ float2 mass_pair(const Cell2 &c, const Cell2 &n, const DeepRow &rc, const DeepRow &rn, float dt,
                                            float2 &top)
{
    const float4 m = rc.m;
    // mass fluxes below the row, left of and between the lane's columns
    const float2 Fb = mass_y2(c, n, m, rn.m, dt);
    const float2 lq = make_float2(shup(c.qx.y, 1), c.qx.x), lh = make_float2(shup(c.h.y, 1), c.h.x);
    const float2 F = limit2(mul2(lq, bc2(m.y)), lh, c.h, 1.f, 1.f, m.z, m.z, dt, m.z);
    const float2 Fr = make_float2(F.y, shdn(F.x, 1));
    const float2 acc = fma2(neg2(Fb), bc2(rc.icos), add2(sub2(F, Fr), top));
    top = mul2(Fb, bc2(rn.icos));
    const float2 e = fma2(bc2(rc.dtA), acc, c.e);
    const float2 h = add2(e, c.D);
    return sel2(h.x > 0.f, h.y > 0.f, e, neg2(c.D));
}

// General units: those that are not deep water (boundaries, sponge layers,
// coasts, wet/dry fronts).  A unit's work is split into tasks of one warp
// each: column strip `strip` (28 output columns and a two-column halo on
// each side) and a group of rows.
//
// The bound is instruction latency (16 warps an SM at 128 registers, about 0.3
// instructions a cycle and scheduler), so the path is kept short: what the four
// edges of a cell share (sqrt h, 1/h, velocities) is formed once per cell instead
// of once per edge side, there is one copy of the y-edge code (the first
// iteration only produces the edge above the group), the flux functions select
// instead of branching, and a warp whose lanes are all deep, or all not, skips the
// other formula.  Against one evaluation per edge side with branches: general
// phase 1 / 2 at 4096^2 52.9 / 61.0 -> 49.5 / 59.4 us launched alone, a step at
// 2048^2 122.5 -> 113.3 us.

// a cell of a lane's column with what its four edges share: sqrt(h), 1/h
// (desingularised) and the velocities
struct EdgeCell {
    float h, e, D, qx, qy, s, inv, tx, ty;
};
__device__ __forceinline__ EdgeCell edge_cell(const RawCell &r, float eps_h)
{
    EdgeCell c;
    c.e = r.e;
    c.D = r.D;
    c.qx = r.qx;
    c.qy = r.qy;
    c.h = r.e + r.D;
    c.s = sqrt_ap(c.h);
    c.inv = inv_depth_x(c.h, eps_h);
    c.tx = mul(c.inv, c.qx);
    c.ty = mul(c.inv, c.qy);
    return c;
}

// Phase PHASE (1 or 2) of one task: rows y0 .. y_end-1 of column strip `strip`
// of unit (tx, uy) (y_end within the unit and the grid), for the state at
// parity p.  Marches the edges between rows y0-1 | y0 to y_end-1 | y_end; each
// iteration computes the y edge below row a (between rows a and b) and, from
// the second on, the x edges of row a and its cells.  Returns the lane's dt
// bound (phase 2), depth summary (phase 1) and error flag; cell: the lane
// holds one of the strip's output cells, gx_out its grid column.
template <int PHASE, bool LIVE>
__device__ __forceinline__ void general_rows(const ScenarioDev &s, int p, float dt, float t_sec, int tx, int uy, int strip,
                                             int y0, int y_end, float &local_min, DepthAcc &hacc, bool &bad, bool &cell,
                                             int &gx_out)
{
    constexpr bool DIAG = (PHASE == 1);
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int nx = s.nx, ny = s.ny;
    const int uy0 = uy * kHalfRows;
    const int unit_end = min(uy0 + kHalfRows, ny);
    const int x0 = s.x_org + tx * kTileX + strip * OUTW;
    const int gx = x0 - 2 + lane;
    const int col = map_col(gx, nx, s.periodic);
    const bool has_edge = (lane >= 2) && (lane <= 30) && (gx >= 0) && (gx <= nx);
    const bool has_cell = (lane >= 2) && (lane <= 29) && (gx >= 0) && (gx < nx);
    const float *eta_in = (PHASE == 2) ? s.eta[p ^ 1] : s.eta[p];
    const float *qx_in = s.qx[p], *qy_in = s.qy[p];
    const size_t pitch = (size_t)s.pitch;
    const bool x_ghost_lo = !s.periodic && gx == 0, x_ghost_hi = !s.periodic && gx == nx;
    const bool x_nolim = (gx < 2) || (gx > nx - 2);
    const bool sponge = (s.sp_left | s.sp_right | s.sp_up | s.sp_low) != 0;
    const float eps_h = s.eps_h, hpos = s.hpos;
    local_min = FLT_MAX;
    hacc.init();
    bad = false;
    gx_out = gx;
    cell = has_cell && x0 < nx && x0 + OUTW > 0;
    if (x0 >= nx || x0 + OUTW <= 0 || y0 >= y_end) return;

    auto load = [&](int y, bool diag) {
        return load_raw<DIAG, LIVE>(s, eta_in, qx_in, qy_in, clamp_row(y, ny) * pitch + col, diag);
    };
    // rows y0-2 .. y0+2 (the last still raw); the diagnostics of rows y0 .. y_end-1
    const RawCell rm = load(y0 - 2, false), ra = load(y0 - 1, false), rb = load(y0, has_cell);
    const RawCell rp = load(y0 + 1, has_cell && y0 + 1 < y_end);
    RawCell r1 = load(y0 + 2, has_cell && y0 + 2 < y_end);
    if (DIAG && has_cell) {
        diagnostics(s, rb, (size_t)y0 * pitch + col, t_sec);
        if (y0 + 1 < y_end) diagnostics(s, rp, (size_t)(y0 + 1) * pitch + col, t_sec);
    }
    float em = rm.e, txm = 0.f;   // row m: what the edge between a and b needs of it
    unsigned dm, da, db, dp;      // lanes deeper than hpos, per row
    EdgeCell a = edge_cell(ra, eps_h), b = edge_cell(rb, eps_h), c = edge_cell(rp, eps_h);
    {
        const EdgeCell m = edge_cell(rm, eps_h);
        txm = m.tx;
        dm = __ballot_sync(FULL, m.h > hpos);
    }
    da = __ballot_sync(FULL, a.h > hpos);
    db = __ballot_sync(FULL, b.h > hpos);
    dp = __ballot_sync(FULL, c.h > hpos);
    // row metrics {cos, ilcos, area, dlon}: ka of row a, kn of row b (entry ny: dlon only)
    const float4 *__restrict__ rows = s.rowpack;
    float4 ka = __ldg(rows + clamp_row(y0 - 1, ny)), kn = __ldg(rows + y0);
    float icos_a = (PHASE == 2) ? __frcp_rn(ka.x) : 0.f;
    // shares of the edge above row a in its cells: mass, or {qx, qy, wave speed}
    float top0 = 0.f, top1 = 0.f, topl = 0.f;

#pragma unroll 1
    for (int ye = y0; ye <= y_end; ye++) {
        const float4 knn = __ldg(rows + min(ye + 1, ny));
        const RawCell r2 = load(ye + 3, has_cell && ye + 3 < y_end);
        const float4 kb = (ye < ny) ? kn : ka;
        const float icos_b = (PHASE == 2) ? __frcp_rn(kb.x) : 0.f;

        // ---- y edge between rows a (ye - 1) and b (ye) ----
        const bool y_ghost_lo = ye == 0, y_nolim = (ye < 2) || (ye > ny - 2);
        const bool deep_y = !y_nolim && ((dm & da & db & dp) >> lane & 1u);
        float lo0 = 0.f, lo1 = 0.f, hi0 = 0.f, hi1 = 0.f, laml = 0.f;
        Sides e;
        const auto y_sides = [&]() {
            e.h0 = a.h; e.h1 = b.h;
            e.e0 = a.e; e.e1 = b.e;
            e.D0 = a.D; e.D1 = b.D;
            e.s0 = a.s; e.s1 = b.s;
            e.u0 = a.qy; e.u1 = b.qy;
            e.t0 = a.ty; e.t1 = b.ty;
            e.em = em; e.ep = c.e;
            e.area0 = ka.z; e.area1 = kb.z;
            e.cos0 = ka.x; e.cos1 = kb.x;
            e.len = kn.w;
            e.normal = y_ghost_lo ? -1.f : 1.f;
            e.no_lim = y_nolim;
            if (y_ghost_lo || ye == ny) {
                e.u1 = mul(b.qy, y_ghost_lo ? s.b_up : s.b_low);
                e.t1 = mul(b.inv, e.u1);
            }
        };
        if (PHASE == 1) {
            float F = 0.f;
            if (__any_sync(FULL, deep_y)) F = mass_2s_y(a.qy, kn.w, ka.x, kb.x, a.h, b.h, dt, ka.z, kb.z);
            if (__any_sync(FULL, !deep_y)) {
                y_sides();
                const float Fw = mass_waf<true>(e, dt, eps_h, hpos);
                F = deep_y ? F : Fw;
            }
            lo0 = -__fdividef(F, ka.x);
            hi0 = y_ghost_lo ? lo0 : __fdividef(F, kb.x);
        } else {
            MomFlux f = {0.f, 0.f, 0.f, 0.f, 0.f};
            if (__any_sync(FULL, deep_y))
                f = momentum_2s_y(a.h, b.h, rcp_depth(a.h), rcp_depth(b.h), a.s, b.s, a.qy, b.qy, a.qx, b.qx,
                                  surface_jump(a.e, b.e, a.D, b.D),
                                  make_yrow(ka.x, kb.x, icos_a, icos_b, kn.w, ka.z + kb.z, dt, s.cvis));
            if (__any_sync(FULL, !deep_y)) {
                y_sides();
                const MomFlux g = momentum_waf<true>(e, a.qx, b.qx, txm, a.tx, b.tx, c.tx, icos_a, icos_b, dt, eps_h, hpos,
                                                     s.cvis);
                f.n0 = deep_y ? f.n0 : g.n0;
                f.t0 = deep_y ? f.t0 : g.t0;
                f.n1 = deep_y ? f.n1 : g.n1;
                f.t1 = deep_y ? f.t1 : g.t1;
                f.lam = deep_y ? f.lam : g.lam;
            }
            lo0 = f.t0;
            lo1 = f.n0;
            hi0 = y_ghost_lo ? lo0 : f.t1;
            hi1 = y_ghost_lo ? lo1 : f.n1;
            laml = f.lam;
        }

        // ---- row a: x edges (each lane its left one) and cells ----
        if (ye > y0) {
            const int yo = ye - 1;
            const size_t idx = (size_t)yo * pitch + col;
            const float area = ka.z;
            const bool deep_x = !x_nolim && lane >= 2 && lane <= 30 && ((da >> (lane - 2)) & 0xfu) == 0xfu;
            const bool waf_x = has_edge && !deep_x;
            const float lh = shup(a.h, 1), lu = shup(a.qx, 1);
            const float ls = shup(a.s, 1), le = shup(a.e, 1), lD = shup(a.D, 1), lt = shup(a.tx, 1);
            const float lem = shup(a.e, 2), rep = shdn(a.e, 1);
            const auto x_sides = [&]() {
                e.h0 = lh; e.h1 = a.h;
                e.e0 = le; e.e1 = a.e;
                e.D0 = lD; e.D1 = a.D;
                e.s0 = ls; e.s1 = a.s;
                e.u0 = lu; e.u1 = a.qx;
                e.t0 = lt; e.t1 = a.tx;
                e.em = lem; e.ep = rep;
                e.area0 = e.area1 = area;
                e.cos0 = e.cos1 = ka.x;
                e.len = ka.y;
                e.normal = x_ghost_lo ? -1.f : 1.f;
                e.no_lim = x_nolim;
                if (x_ghost_lo || x_ghost_hi) {
                    e.u1 = mul(a.qx, x_ghost_lo ? s.b_left : s.b_right);
                    e.t1 = mul(a.inv, e.u1);
                }
            };
            if (PHASE == 1) {
                float F = 0.f;
                if (__any_sync(FULL, deep_x)) F = mass_2s_x(lu, ka.y, lh, a.h, dt, area, area);
                if (__any_sync(FULL, waf_x)) {
                    x_sides();
                    const float Fw = mass_waf<false>(e, dt, eps_h, hpos);
                    F = deep_x ? F : Fw;
                }
                const float Fr = shdn(F, 1);
                if (has_cell) {
                    // mass update (src/GPU/Volumen_kernel.cu:111-157); the
                    // diagnostics run when a row's loads complete
                    const float acc = add(add(sub(x_ghost_lo ? -F : F, Fr), top0), lo0);
                    const float D = a.D;
                    float eta = fma_(__fdividef(dt, area), acc, a.e);
                    if (!(add(eta, D) > 0.f)) eta = -D;
                    if (sponge && ((gx < s.sp_left) || (gx >= nx - s.sp_right) || (yo < s.sp_up) ||
                                   (yo >= ny - s.sp_low))) {
                        const float dx = __ldg(s.row.dlon + yo), dy = __ldg(s.row.dlat + yo);
                        float dl = (s.sp_left - gx - 0.5f) * dx, dr = (gx - (nx - 1 - s.sp_right) - 0.5f) * dx;
                        float du = (s.sp_up - yo - 0.5f) * dy, dd = (yo - (ny - 1 - s.sp_low) - 0.5f) * dy;
                        if (dl <= 0.f) dl = 1e30f;
                        if (dr <= 0.f) dr = 1e30f;
                        if (du <= 0.f) du = 1e30f;
                        if (dd <= 0.f) dd = 1e30f;
                        float dist, ls2;
                        if ((dl <= dr) && (dl <= du) && (dl <= dd)) { dist = dl; ls2 = dx * s.sp_left; }
                        else if ((dr <= dl) && (dr <= du) && (dr <= dd)) { dist = dr; ls2 = dx * s.sp_right; }
                        else if ((du <= dl) && (du <= dr) && (du <= dd)) { dist = du; ls2 = dy * s.sp_up; }
                        else { dist = dd; ls2 = dy * s.sp_low; }
                        const float rr = dist / ls2, co = mul(mul(0.9f, rr), rr);
                        // relax h towards max(D + sea level, 0), expressed on eta
                        const float eta_rest = (D + s.sea > 0.f) ? s.sea : -D;
                        eta = fma_(-co, sub(eta, eta_rest), eta);
                        if (!(add(eta, D) >= 0.f)) eta = -D;
                    }
                    if (!isfinite(eta)) bad = true;
                    s.eta[p ^ 1][idx] = eta;
                    hacc.add(add(eta, D), yo - uy0 < 2, unit_end - yo <= 2);
                }
            } else {
                const float lv = shup(a.qy, 1), ltt = shup(a.ty, 1), lttm = shup(a.ty, 2), rtt = shdn(a.ty, 1);
                MomFlux f = {0.f, 0.f, 0.f, 0.f, 0.f};
                if (__any_sync(FULL, deep_x))
                    f = momentum_2s_x(lh, a.h, rcp_depth(lh), rcp_depth(a.h), ls, a.s, lu, a.qx, lv, a.qy,
                                      surface_jump(le, a.e, lD, a.D), make_xrow(ka.y, area + area, dt, s.cvis));
                if (__any_sync(FULL, waf_x)) {
                    x_sides();
                    const MomFlux g = momentum_waf<false>(e, lv, a.qy, lttm, ltt, a.ty, rtt, 0.f, 0.f, dt, eps_h, hpos, s.cvis);
                    f.n0 = deep_x ? f.n0 : g.n0;
                    f.t0 = deep_x ? f.t0 : g.t0;
                    f.n1 = deep_x ? f.n1 : g.n1;
                    f.t1 = deep_x ? f.t1 : g.t1;
                    f.lam = deep_x ? f.lam : g.lam;
                }
                // the right edge of this cell is the left edge of lane+1
                const float rn = shdn(f.n0, 1), rt = shdn(f.t0, 1), rl = shdn(f.lam, 1);
                if (has_cell) {
                    // momentum update (src/GPU/Volumen_kernel.cu:175-219); the
                    // fluxes are summed as they are subtracted (negation is exact)
                    const float lam = add(add(add(f.lam, rl), topl), laml);
                    const float step = (lam < kEps) ? 1e30f : __fdividef(2.f * s.cfl * area, lam);
                    local_min = fminf(local_min, step);
                    const float val = -__fdividef(dt, area);
                    const float qx_old = a.qx, qy_old = a.qy, h = a.h;
                    float qx = fma_(val, add(add(add(x_ghost_lo ? f.n0 : f.n1, rn), top0), lo0), qx_old);
                    float qy = fma_(val, add(add(add(x_ghost_lo ? f.t0 : f.t1, rt), top1), lo1), qy_old);
                    if (sponge) {
                        const float dx = __ldg(s.row.dlon + yo), dy = __ldg(s.row.dlat + yo);
                        if (gx < s.sp_left) {
                            const float rr = ((s.sp_left - gx - 0.5f) * dx) / (dx * s.sp_left);
                            qx = fma_(-mul(mul(0.9f, rr), rr), qx, qx);
                        }
                        if (gx >= nx - s.sp_right) {
                            const float rr = ((gx - (nx - 1 - s.sp_right) - 0.5f) * dx) / (dx * s.sp_right);
                            qx = fma_(-mul(mul(0.9f, rr), rr), qx, qx);
                        }
                        if (yo < s.sp_up) {
                            const float rr = ((s.sp_up - yo - 0.5f) * dy) / (dy * s.sp_up);
                            qy = fma_(-mul(mul(0.9f, rr), rr), qy, qy);
                        }
                        if (yo >= ny - s.sp_low) {
                            const float rr = ((yo - (ny - 1 - s.sp_low) - 0.5f) * dy) / (dy * s.sp_low);
                            qy = fma_(-mul(mul(0.9f, rr), rr), qy, qy);
                        }
                    }
                    if (h <= hpos) {
                        // damping of almost-dry cells and velocity cap (filtroEstado)
                        const float f1 = h / eps_h, f2 = mul(f1, f1);
                        const float damp = __expf(-dt * (1.f / fma_(f2, f2, kEps)));
                        qx *= damp;
                        qy *= damp;
                        const float fac = a.inv;
                        if (s.vmax > 0.f) {
                            float ux = fac * qx, uyv = fac * qy;
                            const float uu = sqrt_ap(fma2p(ux, ux, uyv, uyv));
                            if (uu > s.vmax) { ux *= s.vmax / uu; uyv *= s.vmax / uu; }
                            qx = ux * h;
                            qy = uyv * h;
                        }
                        // semi-implicit Manning friction with the pre-update speed (disImplicita)
                        const float u1x = fac * qx, u1y = fac * qy;
                        const float u1 = sqrt_ap(fma2q(qx_old, qx_old, qy_old, qy_old)) * fac;
                        if (h > 0.f) {
                            const float c1 = __fdividef(1.f, add(exp2f(log2f(h) * (4.f / 3.f)), kEps));
                            const float fr = h / fma_(dt * s.mf0 * fabsf(u1), c1, 1.f);
                            qx = fr * u1x;
                            qy = fr * u1y;
                        }
                    }
                    if (!isfinite(qx) || !isfinite(qy)) bad = true;
                    s.qx[p ^ 1][idx] = qx;
                    s.qy[p ^ 1][idx] = qy;
                }
            }
        }
        top0 = hi0;
        top1 = hi1;
        topl = laml;
        em = a.e;
        txm = a.tx;
        a = b;
        b = c;
        c = edge_cell(r1, eps_h);
        if (DIAG && has_cell && ye + 2 < y_end) diagnostics(s, r1, (size_t)(ye + 2) * pitch + col, t_sec);
        dm = da;
        da = db;
        db = dp;
        dp = __ballot_sync(FULL, c.h > hpos);
        r1 = r2;
        ka = kb;
        icos_a = icos_b;
        kn = knn;
    }
}

// Phase 0 of one task: the lane's initial dt bound.
__device__ __forceinline__ void initial_rows(const ScenarioDev &s, int p, int tx, int uy, int strip, int y0, int y_end,
                                             float &local_min)
{
    const int lane = threadIdx.x & 31;
    const int nx = s.nx, ny = s.ny;
    const int x0 = s.x_org + tx * kTileX + strip * OUTW;
    const int gx = x0 - 2 + lane;
    const int col = map_col(gx, nx, s.periodic);
    const bool has_edge = (lane >= 2) && (lane <= 30) && (gx >= 0) && (gx <= nx);
    const bool has_cell = (lane >= 2) && (lane <= 29) && (gx >= 0) && (gx < nx);
    const float *eta = s.eta[p], *qx = s.qx[p], *qy = s.qy[p];
    const size_t pitch = (size_t)s.pitch;
    local_min = FLT_MAX;
    if (x0 >= nx || x0 + OUTW <= 0 || y0 >= y_end) return;
    const float4 *__restrict__ rp = s.rowpack;
    Cell c1 = load_cell<false>(eta, s.dep, qx, qy, clamp_row(y0 - 1, ny) * pitch + col);
    Cell c2 = load_cell<false>(eta, s.dep, qx, qy, (size_t)y0 * pitch + col);
    float top = initial_speed_y(s, c1, c2, y0, __ldg(rp + y0).w);
    for (int yo = y0; yo < y_end; yo++) {
        const float4 k = __ldg(rp + yo);
        const Cell c3 = load_cell<false>(eta, s.dep, qx, qy, clamp_row(yo + 1, ny) * pitch + col);
        const float below = initial_speed_y(s, c2, c3, yo + 1, __ldg(rp + yo + 1).w);
        SpeedEdge e{shup(c2.h, 1), c2.h, shup(c2.qx, 1), c2.qx, k.y, 1.f, false};
        if (!s.periodic && gx == 0) {
            e.u0 *= s.b_left;
            e.normal = -1.f;
            e.front = true;
        }
        if (!s.periodic && gx == nx) e.u1 *= s.b_right;
        float xl = 0.f;
        if (has_edge) xl = initial_speed(e, s);
        const float xr = shdn(xl, 1);
        if (has_cell) {
            const float lam = ((xl + xr) + top) + below;
            const float step = (lam < kEps) ? 1e30f : __fdividef(2.f * s.cfl * k.z, lam);
            local_min = fminf(local_min, step);
        }
        top = below;
        c2 = c3;
    }
}

// general_rows over row group `group` (of NG) of a unit, from the control block
template <int PHASE, int NG>
__device__ __forceinline__ void general_part(const ScenarioDev &s, const ScenarioCtl *ctl, int tx, int uy, int strip,
                                             int group, float &local_min, DepthAcc &hacc, bool &bad, bool &cell,
                                             int &gx_out)
{
    constexpr int GROWS = kHalfRows / NG;
    static_assert(kHalfRows % NG == 0, "row groups of equal height");
    const int y0 = uy * kHalfRows + group * GROWS;
    general_rows<PHASE, false>(s, ctl->parity, (float)ctl->dt, (float)(ctl->t * ctl->T), tx, uy, strip, y0,
                               min(y0 + GROWS, min(uy * kHalfRows + kHalfRows, s.ny)), local_min, hacc, bad, cell, gx_out);
}

// Folds one warp's share of a unit's depth summary (nine {min, max}, UnitSum
// order; a field the warp holds no cell of is left alone) into the unit's
// summary with integer atomics on the float bits (see warp_minmax; min and max
// are exact in any order), lane f the field f, so the summary does not depend on
// which warp came first.  The classification resets the summaries of the general
// units it lists to the empty value (FLT_MAX, -FLT_MAX) before this phase runs.
__device__ __forceinline__ void fold_unit_summary(const DepthAcc &a, bool cell, bool is_l, bool is_r, UnitSum *dst)
{
    const int lane = threadIdx.x & 31;
    const float2 none = make_float2(FLT_MAX, -FLT_MAX);
    const bool has_t = __any_sync(0xffffffffu, cell && a.tmin != FLT_MAX);
    const bool has_b = __any_sync(0xffffffffu, cell && a.bmin != FLT_MAX);
    const bool has_l = __any_sync(0xffffffffu, is_l), has_r = __any_sync(0xffffffffu, is_r);
    float2 mine = none;
    const auto put = [&](int k, const float2 &v) { mine = lane == k ? v : mine; };
    put(0, warp_minmax(a.amin, a.amax, cell));
    if (has_l) put(1, warp_minmax(a.amin, a.amax, is_l));
    if (has_r) put(2, warp_minmax(a.amin, a.amax, is_r));
    if (has_t) {
        put(3, warp_minmax(a.tmin, a.tmax, cell));
        if (has_l) put(5, warp_minmax(a.tmin, a.tmax, is_l));
        if (has_r) put(6, warp_minmax(a.tmin, a.tmax, is_r));
    }
    if (has_b) {
        put(4, warp_minmax(a.bmin, a.bmax, cell));
        if (has_l) put(7, warp_minmax(a.bmin, a.bmax, is_l));
        if (has_r) put(8, warp_minmax(a.bmin, a.bmax, is_r));
    }
    if (mine.x != FLT_MAX) {
        int *d = reinterpret_cast<int *>(dst) + 2 * lane;
        atomicMin(d, __float_as_int(mine.x));
        atomicMax(d + 1, __float_as_int(mine.y));
    }
}

// smallest of the lanes' positive dt bounds
__device__ __forceinline__ float warp_min_bound(float v)
{
    return __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(v)));
}

}  // namespace thy
