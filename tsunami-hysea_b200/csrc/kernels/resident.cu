// A chunk of time steps in one launch, for work that does not fill the GPU.
//
// What bounds such work is latency, not throughput: as separate launches
// (step.cu) a step is a chain of kernels, each of which reads
// its lists, work items, descriptors and control words one after the other
// before its first cell.  Here one CTA per SM stays on the device for the whole
// chunk with the scenarios' descriptors in shared memory, and a step is
//     phase 1 | grid barrier | classes, phase 2 | grid barrier, control
// A task is a column strip of a unit and a few of its rows.  The tasks are dealt
// to the CTAs once per chunk, by falling cost (shallow general units, the other
// general ones, deep units), and a CTA's
// warps claim them from shared memory.  The classes that the classification
// launch would list are evaluated in place, one thread per task of the CTA, so
// that a step has no list to build; a unit that changes class during the chunk is
// stepped by the same tasks, each step by the class it has.  Every CTA advances
// the control blocks for itself from the barrier's dt minimum, which saves a hop
// through a controlling CTA.
//
// What bounds it now: the chain of a task's edges (about 3.8 us a row of WAF
// edges in both phases on an otherwise idle SM), two barriers of 1.3 us, and the
// spread of the tasks' costs over the SMs; from 1024^2 on also the loads of the
// deep rows, which are issued a row ahead (a second row ahead: 1 % slower).  us a
// step, launched -> resident: 96 x 80 28 -> 14, 512^2 48 -> 23, 1024^2 70 -> 38,
// 1600^2 94 -> 64, 2048^2 111 -> 95.  Deep rows go in column pairs in both phases:
// packed arithmetic and half the loads and stores of one column a lane (phase 1
// with one column a lane: 1024^2 44.5, 2048^2 126; with a row's diagnostics loaded
// in the iteration that uses them: 40, 103).
//
// Arithmetic, classes, depth summaries, dry counts and the control are those
// of the launches in step.cu; results are bitwise the same.
//
// Reference: src/GPU/Timestep.cu:11-120 (the launches of a step),
// src/GPU/ShallowWater.cu:396-450 (the loop around it).
#include "step_parts.cuh"

#include <algorithm>

namespace thy {

namespace {

constexpr int kResWarps = kResidentWarps, kResThreads = 32 * kResWarps;
constexpr int kMaxDeepRows = 8;     // rows of a deep task at most
constexpr int kTaskRows = kMaxDeepRows + 2;
constexpr int kDealStep = 61;       // odd: units of one column of a grid alternate in the lists

// classes of a unit; kClsPlain: a flag of deep units; kClsShallow: a flag of
// general units with water no deeper than hpos (their edges take the costly path)
enum : int { kClsGeneral = 0, kClsDeep = 1, kClsDry = 2, kClsPlain = 4, kClsShallow = 8 };

// the step state of a scenario
struct alignas(16) StepState {
    float dt, t_sec;
    int parity, status;
};

// A task of one warp: unit (tx, uy) of scenario `slot`, its sub-task and the rows
// of one.  Sub-tasks are (strip of 28 columns) + 4 (row group), or, of the units
// that were deep when the tasks were dealt (kPairTask in rows), (strip of 56
// columns) + 2 (row group).  A unit whose class has changed is covered by the
// same sub-tasks: a deep unit by strips of 56 and half the rows, a general one by
// both strips of 28 in turn.
constexpr int kPairTask = 0x80;
struct Task {
    short slot, tx, uy;
    unsigned char sub, rows;
    __device__ __forceinline__ bool pair() const { return (rows & kPairTask) != 0; }
    __device__ __forceinline__ int nrows() const { return rows & (kPairTask - 1); }
};
// the deep rows of a task: first row in the unit and rows (0: covered by others)
__device__ __forceinline__ int2 deep_rows(const Task &t)
{
    if (t.pair()) return make_int2((t.sub >> 1) * t.nrows(), t.nrows());
    const int half = max(t.nrows() >> 1, 1), y = (t.sub >> 1) * half;   // (a single row is not halved)
    return make_int2(y, y < kHalfRows ? half : 0);
}

// A scenario in shared memory.  (One array of them behind the CTA's tables, so that
// every address is a constant, a slot and a field: pointers to an array each took
// registers that the row loops need.)
struct alignas(16) Slot {
    ScenarioDev dev;
    ScenarioCtl ctl;     // every CTA advances its own copy
    StepState state;
    unsigned dt_bits;    // the block's smallest dt bound of the step
};
struct Shared {
    DeepRow rows[kResWarps * kTaskRows];
    Task tasks[kResThreads];           // this CTA's tasks, one thread evaluates the class of each
    unsigned char cls[kResThreads];
    Slot slots[1];                     // nslots
};
__host__ __device__ inline size_t shared_bytes(int nslots) { return sizeof(Shared) + (nslots - 1) * sizeof(Slot); }

// ---------------------------------------------------------------------------
// Grid barriers: one thread per CTA adds to a counter and polls it.  Arrivals
// release, waits acquire (which also drops the SM's L1 lines, so that plain
// loads after a barrier see what other SMs wrote before it).  Measured on 148
// CTAs: 1.27 us a barrier; a tag per CTA that every CTA polls 6.0 us, a
// gathering CTA that answers with one word 2.9 us.  The dt bounds lie in words of
// their own, read after the wait: one more load than a bound in the counter's word
// (0.15 to 0.35 us a step), but accesses of two sizes to one word have no defined
// order in the PTX memory model.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned ld_acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned *p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// arrives at w and waits for n arrivals; false after wait_ns of global time (or
// 2^28 polls), so that no wait is endless
__device__ __forceinline__ bool arrive_and_wait(ResidentSync::Word &w, unsigned n, unsigned long long wait_ns)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&w.arrived) : "memory");
    unsigned long long t0 = 0;
    for (int i = 0; i < (1 << 28); i++) {
        if (ld_acquire(&w.arrived) == n) return true;
        if ((i & 63) == 63) {
            const unsigned long long now = global_ns();
            if (!t0) t0 = now;
            else if (now - t0 > wait_ns) break;
        }
    }
    return false;
}

// ---------------------------------------------------------------------------
// The team: the CTAs that step the chunk.  Each CTA counts itself in as it starts;
// the team is all of the launch once they have, or those that have started kTeamNs
// after the first one, which then closes it.  A CTA that comes later (its SM was
// held by another stream's kernel) leaves, so a barrier waits for running CTAs only.
// (A cooperative launch guarantees as much by starting only when every SM is free:
// beside one block of a long kernel it waited for that kernel's end, and while it
// was pending no other kernel of the process started.)
// ---------------------------------------------------------------------------
constexpr unsigned long long kTeamNs = 50000;   // all CTAs of a launch on a free GPU start within some us
constexpr unsigned kTeamClosed = 0x80000000u;
// this CTA's {rank, CTAs of the team}; {-, 0}: too late; {-, -1}: no answer within
// wait_ns.  The ranks of a whole team are the block indices, which the device spreads
// over its SMs (by arrival 1 % slower at 96 x 80 and 733 x 517).
__device__ __forceinline__ int2 join_team(ResidentSync *sync, int launch, unsigned grid, unsigned long long wait_ns)
{
    ResidentSync::Word &w = sync->team[launch];
    unsigned *size = &sync->team_size[launch];
    const unsigned rank = atomicAdd(&w.arrived, 1u);   // by arrival
    if (rank & kTeamClosed) return make_int2(0, 0);
    if (rank == 0) {
        // the next launch's words; the last one's are read by no one any more
        const int next = launch == 2 ? 0 : launch + 1;
        sync->team[next].arrived = 0u;
        sync->team_size[next] = 0u;
    }
    const unsigned long long t0 = global_ns();
    for (int i = 0; i < (1 << 28); i++) {
        const unsigned v = ld_acquire(&w.arrived);
        if (v == grid) return make_int2(blockIdx.x, grid);
        if (v & kTeamClosed) {
            const unsigned n = ld_acquire(size);
            if (n) return make_int2(n == grid ? blockIdx.x : rank, n);
        }
        const unsigned long long waited = global_ns() - t0;
        if (rank == 0 && waited > kTeamNs) {
            const unsigned n = atomicOr(&w.arrived, kTeamClosed);
            st_release(size, n);   // (all of them after all: some may have seen it)
            return make_int2(n == grid ? blockIdx.x : rank, n);
        }
        if (waited > wait_ns) break;
    }
    return make_int2(rank, -1);
}

// ---------------------------------------------------------------------------
// Deep units.  The formulas and roundings are those of the deep-water kernels
// (step.cu), with the rows loaded straight from global memory: a task has a
// few rows, and the state of most of this work (up to about 1700^2) stays in L2.
// ---------------------------------------------------------------------------

// the loads of a row of column pairs that is still in flight
struct Raw2 {
    float2 e, D, qx, qy;
};
__device__ __forceinline__ Raw2 load_raw2(const float *eta, const float *dep, const float *qx, const float *qy, size_t off)
{
    Raw2 c;
    c.e = *reinterpret_cast<const float2 *>(eta + off);
    c.D = *reinterpret_cast<const float2 *>(dep + off);
    c.qx = *reinterpret_cast<const float2 *>(qx + off);
    c.qy = *reinterpret_cast<const float2 *>(qy + off);
    return c;
}
__device__ __forceinline__ Cell2 cell2(const Raw2 &r)
{
    return Cell2{add2(r.e, r.D), r.e, r.D, r.qx, r.qy};
}

// the diagnostics of a cell pair
struct Diag2 {
    float2 em, ar, ei;
};
__device__ __forceinline__ Diag2 load_diag2(const ScenarioDev &s, size_t off, bool cell)
{
    Diag2 d{};
    if (cell) {
        d.em = *reinterpret_cast<const float2 *>(s.eta_max + off);
        d.ar = *reinterpret_cast<const float2 *>(s.arr + off);
        d.ei = *reinterpret_cast<const float2 *>(s.eta_ini + off);
    }
    return d;
}

// Column pairs: lane l holds columns x0 - 2 + 2l and the next one (x0 even) of a
// strip of 56 columns; lanes 1..28 are cells, lanes 0 and 29 the halo, lanes 30
// and 31 repeat lane 29.

// phase 1: columns x0 .. x0+55, rows y0 .. y0+nrows-1; the warp's depth {min, max}
__device__ __forceinline__ void mass_rows(const ScenarioDev &s, int p, float dt, float t_sec, int x0, int y0, int nrows,
                                          DeepRow *rows, float &mn, float &mx, bool &bad)
{
    const int lane = threadIdx.x & 31;
    const size_t pitch = (size_t)s.pitch;
    const bool out_lane = (lane >= 1) && (lane <= 28);
    const float *eta = s.eta[p], *qx = s.qx[p], *qy = s.qy[p];
    float *out = s.eta[p ^ 1];
    size_t off = (size_t)y0 * pitch + x0 - 2 + 2 * min(lane, 29);
    const Raw2 ra = load_raw2(eta, s.dep, qx, qy, off - pitch), rc = load_raw2(eta, s.dep, qx, qy, off);
    Raw2 rn = load_raw2(eta, s.dep, qx, qy, off + pitch);
    Diag2 dg = load_diag2(s, off, out_lane);
    // row y0 - 1 + t of the window at rows[t]
    if (lane < nrows + 2) {
        const float4 m = __ldg(s.rowpack + y0 - 1 + lane);
        rows[lane].m = m;
        rows[lane].icos = __frcp_rn(m.x);
        rows[lane].dtA = __fdividef(dt, m.z);
    }
    __syncwarp();
    Cell2 c = cell2(rc);
    float2 top = mul2(mass_y2(cell2(ra), c, rows[0].m, rows[1].m, dt), bc2(rows[1].icos));
    mn = FLT_MAX;
    mx = -FLT_MAX;
    float2 fin = make_float2(0.f, 0.f);   // running sum: non-finite iff a new value is
#pragma unroll 1
    for (int k = 0; k < nrows; k++, off += pitch) {
        // the row after the next one; the next row's diagnostics
        Raw2 rnn = rn;
        if (k + 1 < nrows) rnn = load_raw2(eta, s.dep, qx, qy, off + 2 * pitch);
        Diag2 dn = dg;
        if (k + 1 < nrows) dn = load_diag2(s, off + pitch, out_lane);
        const Cell2 n = cell2(rn);
        const float2 e = mass_pair(c, n, rows[k + 1], rows[k + 2], dt, top);
        if (out_lane) {
            const float2 h = add2(e, c.D);
            fin = add2(fin, e);
            *reinterpret_cast<float2 *>(out + off) = e;
            mn = fminf(mn, fminf(h.x, h.y));
            mx = fmaxf(mx, fmaxf(h.x, h.y));
            // diagnostics of the state the step starts from (src/GPU/Metrics.cu:23-77)
            if (c.e.x > dg.em.x && c.h.x > s.eps_h) s.eta_max[off] = c.e.x;
            if (c.e.y > dg.em.y && c.h.y > s.eps_h) s.eta_max[off + 1] = c.e.y;
            if (dg.ar.x < 0.f && fabsf(c.e.x - dg.ei.x) > s.dif_at) s.arr[off] = t_sec;
            if (dg.ar.y < 0.f && fabsf(c.e.y - dg.ei.y) > s.dif_at) s.arr[off + 1] = t_sec;
        }
        c = n;
        rn = rnn;
        dg = dn;
    }
    bad = !isfinite(fin.x) || !isfinite(fin.y);
    const float2 v = warp_minmax(mn, mx, out_lane);
    mn = v.x;
    mx = v.y;
    __syncwarp();   // rows is reused by the warp's next task
}

// phase 2: columns x0 .. x0+55, rows y0 .. y0+nrows-1; the warp's largest lam /
// (2 cfl area)
template <bool PLAIN>
__device__ __forceinline__ float momentum_rows(const ScenarioDev &s, int p, float dt, int x0, int y0, int nrows, DeepRow *rows,
                                               bool &bad)
{
    const int lane = threadIdx.x & 31;
    const size_t pitch = (size_t)s.pitch;
    const bool out_lane = (lane >= 1) && (lane <= 28);
    const float *eta = s.eta[p ^ 1], *qx_in = s.qx[p], *qy_in = s.qy[p];
    float *qx_out = s.qx[p ^ 1], *qy_out = s.qy[p ^ 1];
    size_t off = (size_t)y0 * pitch + x0 - 2 + 2 * min(lane, 29);
    const Raw2 ra = load_raw2(eta, s.dep, qx_in, qy_in, off - pitch), rc = load_raw2(eta, s.dep, qx_in, qy_in, off);
    Raw2 rn = load_raw2(eta, s.dep, qx_in, qy_in, off + pitch);
    if (lane < nrows + 2)
        rows[lane] = deep_row(__ldg(s.rowpack + y0 - 1 + lane), __ldg(s.rowpack + y0 - 2 + lane), dt, s.cfl, s.cvis);
    __syncwarp();
    Cell2 c = cell2(rc);
    Depth2 fc = depth2(c.h);
    Contrib2 top;
    {
        Contrib2 dummy;
        const Cell2 a = cell2(ra);
        const Depth2 fa = depth2(a.h);
        y_edge_deep2<PLAIN>(a, c, fa.rh, fa.sh, fc.rh, fc.sh, rows[0], rows[1], dummy, top);
    }
    float local_max = 0.f;
    float2 fin = make_float2(0.f, 0.f);   // running sum: non-finite iff a new value is
#pragma unroll 1
    for (int k = 0; k < nrows; k++, off += pitch) {
        Raw2 rnn = rn;
        if (k + 1 < nrows) rnn = load_raw2(eta, s.dep, qx_in, qy_in, off + 2 * pitch);
        const Cell2 n = cell2(rn);
        const Depth2 fn = depth2(n.h);
        Contrib2 below, next_top;
        y_edge_deep2<PLAIN>(c, n, fc.rh, fc.sh, fn.rh, fn.sh, rows[k + 1], rows[k + 2], below, next_top);
        float2 qx, qy;
        float wm;
        pair_update<PLAIN>(c, fc, rows[k + 1], top, below, qx, qy, wm);
        if (out_lane) {
            local_max = fmaxf(local_max, wm);
            fin = add2(fin, add2(qx, qy));
            *reinterpret_cast<float2 *>(qx_out + off) = qx;
            *reinterpret_cast<float2 *>(qy_out + off) = qy;
        }
        top = next_top;
        c = n;
        rn = rnn;
        fc = fn;
    }
    bad = !isfinite(fin.x) || !isfinite(fin.y);
    local_max = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(local_max)));   // (>= 0)
    __syncwarp();   // rows is reused by the warp's next task
    return local_max;
}

// Class of a unit for the state its summaries `sum` describe, as unit_deep and
// unit_dry find it, from one round of nine loads; *age: its dry count
// (advance: the classification of a step, which moves the count); gmax: the
// unit's depth step.
__device__ __forceinline__ int unit_class(const ScenarioDev &s, const UnitSum *sum, int tx, int uy, float gmax, bool advance,
                                          int &age)
{
    const int W = s.tiles_x, ny_u = units_y(s);
    const int x0 = s.x_org + tx * kTileX, yb = uy * kHalfRows;
    const bool inside = s.tmap && x0 >= max(2, s.sp_left) && x0 + kTileX <= s.nx - max(2, s.sp_right) &&
                        yb >= max(2, s.sp_up) && yb + kHalfRows <= s.ny - max(2, s.sp_low);
    const bool l = tx > 0 || s.periodic, r = tx + 1 < W || s.periodic, t = uy > 0, b = uy + 1 < ny_u;
    const UnitSum *c = sum + (size_t)uy * W + tx;
    // neighbours: the wrapped unit across a periodic boundary; the unit itself
    // where there is none (outside counts as dry, and the unit is not inside)
    const int dl = !l ? 0 : tx > 0 ? -1 : W - 1, dr = !r ? 0 : tx + 1 < W ? 1 : 1 - W;
    const int dt = t ? -W : 0, db = b ? W : 0;
    const float2 v0 = c->all, v1 = c[dl].R, v2 = c[dr].L, v3 = c[dt].B, v4 = c[db].T;
    const float2 v5 = c[dt + dl].BR, v6 = c[dt + dr].BL, v7 = c[db + dl].TR, v8 = c[db + dr].TL;
    const float hp = s.hpos;
    const bool deep = inside & (v0.x > hp) & (v1.x > hp) & (v2.x > hp) & (v3.x > hp) & (v4.x > hp) & (v5.x > hp) &
                      (v6.x > hp) & (v7.x > hp) & (v8.x > hp);
    const bool dry = (v0.y <= 0.f) & (!l | (v1.y <= 0.f)) & (!r | (v2.y <= 0.f)) & (!t | (v3.y <= 0.f)) &
                     (!b | (v4.y <= 0.f)) & (!(t & l) | (v5.y <= 0.f)) & (!(t & r) | (v6.y <= 0.f)) &
                     (!(b & l) | (v7.y <= 0.f)) & (!(b & r) | (v8.y <= 0.f));
    if (advance) age = (!deep && dry) ? min(age + 1, 255) : 0;
    if (age >= kDryAge) return kClsDry;
    if (!deep) return kClsGeneral | (v0.x > hp ? 0 : kClsShallow);
    const float hmin = fminf(fminf(fminf(v0.x, v1.x), fminf(v2.x, v3.x)),
                             fminf(fminf(v4.x, v5.x), fminf(fminf(v6.x, v7.x), v8.x)));
    return kClsDeep | (hmin > 1.001f * gmax + 1e-6f ? kClsPlain : 0);
}

__device__ __forceinline__ void clear_summary(UnitSum *u)
{
    float2 *e = reinterpret_cast<float2 *>(u);
#pragma unroll
    for (int f = 0; f < 9; f++) e[f] = make_float2(FLT_MAX, -FLT_MAX);
}

__device__ __forceinline__ StepState step_state(const ScenarioCtl &c)
{
    return StepState{(float)c.dt, (float)(c.t * c.T), c.parity, c.status};
}

// A value of the scenario is not finite: besides the error bit for the host, no
// valid dt (0) among the block's bounds.  What ends the scenario is that bound, which
// reaches every CTA through the step's barrier; the error bit would reach a CTA that
// reads it late together with the next step's, and the CTAs would part.
__device__ __forceinline__ void fail(const ScenarioDev &s, unsigned *dt_bits)
{
    atomicOr(&s.ctl->errors, 1u);
    atomicMin(dt_bits, 0u);
}

// the warp's next task of the CTA
__device__ __forceinline__ int claim(int *next)
{
    int j = 0;
    if ((threadIdx.x & 31) == 0) j = atomicAdd(next, 1);
    return __shfl_sync(0xffffffffu, j, 0);
}

__global__ void __launch_bounds__(kResThreads, 1) resident_kernel(const ResidentLaunch L)
{
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ bool s_ok;            // no wait has run out
    __shared__ int s_next[2];        // the CTA's next task of phase 1 and 2
    __shared__ int s_sample[kResidentSlots];   // rank 0: the step's gauge samples (ring slots)
    __shared__ bool s_sampled, s_any;          // some; some scenario still runs
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ int s_rank, s_team;   // this CTA's place in the team, its CTAs
    Shared &h = *reinterpret_cast<Shared *>(dsm);
    Slot *slots = h.slots;
    ResidentSync *sync = L.sync;
    Task *tasks = h.tasks;
    unsigned char *cls = h.cls;
    DeepRow *rows = h.rows + warp * kTaskRows;

    // ---- the scenarios' descriptors and states ----
    {
        constexpr int words = sizeof(ScenarioDev) / 4;
        const unsigned *src = reinterpret_cast<const unsigned *>(L.tab);
        for (int k = tid; k < L.nslots * words; k += kResThreads)
            reinterpret_cast<unsigned *>(&slots[k / words].dev)[k % words] = __ldg(src + k);
    }
    if (tid == 0) {
        const int2 t = join_team(sync, L.launch, gridDim.x, L.wait_ns);
        s_rank = t.x;
        s_team = t.y;
        s_ok = true;
    }
    __syncthreads();
    if (s_team <= 0) {
        // (no answer: the others' waits for this CTA run out, too)
        if (s_team < 0 && tid < L.nslots) atomicOr(&slots[tid].dev.ctl->errors, 2u);
        return;
    }
    const bool absent = L.drop && s_rank == s_team - 1;   // test hook: this CTA takes part in no barrier of the steps
    for (int k = tid; k < L.nslots; k += kResThreads) {
        slots[k].ctl = *slots[k].dev.ctl;
        slots[k].state = step_state(slots[k].ctl);
        slots[k].dt_bits = 0x7f7fffffu;
        s_sample[k] = -1;
        if (s_rank == 0) sync->dt_bits[0][k] = sync->dt_bits[1][k] = sync->dt_bits[2][k] = 0x7f7fffffu;
    }
    __syncthreads();

    // ---- the units by class (as the classification before a chunk) ----
    for (int base = (s_rank * kResWarps + warp) * 32; base < L.nunits; base += s_team * kResThreads) {
        const int u = base + lane;
        int c = -1;
        if (u < L.nunits) {
            const int2 item = L.units[u];
            const ScenarioDev &s = slots[item.x].dev;
            const int uy = item.y / s.tiles_x, tx = item.y - uy * s.tiles_x;
            const int par = slots[item.x].state.parity;
            int age = s.dry_age[item.y];
            c = unit_class(s, s.usum[par], tx, uy, 0.f, false, age);
            // phase 1 folds its summary into the other parity's entry
            if (c != kClsDry) clear_summary(&s.usum[par ^ 1][item.y]);
            c = (c & kClsShallow) ? 0 : 1 + (c & 3);   // the list
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const unsigned m = __ballot_sync(0xffffffffu, c == k);
            if (!m) continue;
            int at = 0;
            if (lane == 0) at = atomicAdd(&sync->counts[k], __popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (c == k) L.order[k * L.cap + at + __popc(m & ((1u << lane) - 1u))] = u;
        }
    }
    int at = __ldcg(&sync->next);   // this launch's first barrier words
    __syncthreads();
    if (tid == 0 && !arrive_and_wait(sync->start, s_team, L.wait_ns)) s_ok = false;
    __syncthreads();

    // ---- this CTA's tasks, dealt in rounds: the shallow general units' first,
    // then the other general units', the deep units' and the dry ones' (by falling
    // cost); consecutive tasks are the same rows of different units and strips, and
    // each round starts at another CTA, so that no CTA gets the boundary strips of
    // all its units.  Its warps claim them in this order. ----
    int ntask, age = 0;
    float gmax = 0.f;
    int counted_deep = 0, counted_dry = 0;
    {
        int n[4], per[4], total = 0;
        for (int k = 0; k < 4; k++) {
            n[k] = sync->counts[k];
            per[k] = k == 2 ? 2 * (kHalfRows / L.rows_deep) : STRIPS * (kHalfRows / L.rows_general);
            total += n[k] * per[k];
        }
        // a team too small for the tasks, or for their time, leaves the chunk to
        // the launched kernels: the host finds that nothing was stepped
        if (s_ok && (L.decline || total > s_team * kResThreads || 4 * s_team < (int)gridDim.x)) return;
        // round k gives this CTA task k n + (rank + kDealStep k) mod n, n CTAs in the team
        const auto dealt = [&](int k) { return k * s_team + (int)((s_rank + (unsigned)kDealStep * k) % s_team); };
        ntask = total / s_team;
        ntask = min(kResThreads, ntask + (dealt(ntask) < total ? 1 : 0));
        if (s_ok && tid < ntask) {
            int i = dealt(tid), k = 0;
            while (i >= n[k] * per[k]) {
                i -= n[k] * per[k];
                k++;
            }
            const int u = i % n[k], sub = i / n[k];
            const int2 item = L.units[L.order[k * L.cap + u]];
            const ScenarioDev &s = slots[item.x].dev;
            Task t;
            t.slot = (short)item.x;
            t.uy = (short)(item.y / s.tiles_x);
            t.tx = (short)(item.y - t.uy * s.tiles_x);
            t.sub = (unsigned char)(k == 2 ? sub : (sub & ~3) | ((sub + u) & 3));
            t.rows = (unsigned char)(k == 2 ? L.rows_deep | kPairTask : L.rows_general);
            tasks[tid] = t;
            age = s.dry_age[item.y];
            gmax = s.unit_gmax[item.y];
            cls[tid] = (unsigned char)unit_class(s, s.usum[slots[item.x].state.parity], t.tx, t.uy, gmax, false, age);
        }
        if (tid < 2) s_next[tid] = kResWarps;
    }
    __syncthreads();

    for (int step = 0; step < L.steps && s_ok && !absent; step++) {
        // ---- phase 1 ----
        for (int j = warp; j < ntask; j = claim(&s_next[0])) {
            const Task t = tasks[j];
            const StepState q = slots[t.slot].state;
            const int c = cls[j];
            if (q.status != kRunning || (c & 3) == kClsDry) continue;
            const ScenarioDev &s = slots[t.slot].dev;
            UnitSum *dst = &s.usum[q.parity ^ 1][t.uy * s.tiles_x + t.tx];
            bool bad = false;
            if (c & kClsDeep) {
                const int2 y = deep_rows(t);
                if (!y.y) continue;
                float mn, mx;
                mass_rows(s, q.parity, q.dt, q.t_sec, s.x_org + t.tx * kTileX + (t.sub & 1) * 2 * OUTW,
                          t.uy * kHalfRows + y.x, y.y, rows, mn, mx, bad);
                // a deep unit reports its whole-unit {min, max} for its strips and
                // corners too: lane f folds float f of the summary
                if (lane < 18) {
                    int *d = reinterpret_cast<int *>(dst) + lane;
                    if (lane & 1) atomicMax(d, __float_as_int(mx));
                    else atomicMin(d, __float_as_int(mn));
                }
            } else {
                const int y0 = t.uy * kHalfRows + (t.pair() ? t.sub >> 1 : t.sub >> 2) * t.nrows();
                const int y1 = min(y0 + t.nrows(), min(t.uy * kHalfRows + kHalfRows, s.ny));
                const int tx0 = s.x_org + t.tx * kTileX, ux0 = max(tx0, 0), ux1 = min(tx0 + kTileX, s.nx);
                int strip = t.pair() ? 2 * (t.sub & 1) : t.sub & 3;
                const int last = t.pair() ? strip + 1 : strip;
#pragma unroll 1
                for (; strip <= last; strip++) {
                    float local_min;
                    DepthAcc hacc;
                    bool cell, b;
                    int gx;
                    general_rows<1, true>(s, q.parity, q.dt, q.t_sec, t.tx, t.uy, strip, y0, y1, local_min, hacc, b, cell, gx);
                    bad |= b;
                    fold_unit_summary(hacc, cell, cell && gx < ux0 + 2, cell && gx >= ux1 - 2, dst);
                }
            }
            if (bad) fail(s, &slots[t.slot].dt_bits);
        }
        __syncthreads();
        if (tid == 0) {
            s_next[0] = kResWarps;
            if (!arrive_and_wait(sync->phase1[at], s_team, L.wait_ns)) s_ok = false;
        }
        __syncthreads();
        if (!s_ok) break;

        // ---- classes for the state phase 1 produced (for phase 2 of this
        // step and phase 1 of the next), one thread per task ----
        if (tid < ntask) {
            const Task t = tasks[tid];
            const StepState q = slots[t.slot].state;
            if (q.status == kRunning) {
                const ScenarioDev &s = slots[t.slot].dev;
                const int c = unit_class(s, s.usum[q.parity ^ 1], t.tx, t.uy, gmax, true, age);
                cls[tid] = (unsigned char)c;
                if (t.sub == 0) {
                    // the next phase 1 folds this unit's summary into the entry
                    // that the last classification read
                    if (c != kClsDry) clear_summary(&s.usum[q.parity][t.uy * s.tiles_x + t.tx]);
                    counted_deep += (c & kClsDeep) ? 1 : 0;
                    counted_dry += c == kClsDry ? 1 : 0;
                }
            }
        }
        __syncthreads();

        // ---- phase 2 ----
        for (int j = warp; j < ntask; j = claim(&s_next[1])) {
            const Task t = tasks[j];
            const StepState q = slots[t.slot].state;
            const int c = cls[j];
            if (q.status != kRunning || (c & 3) == kClsDry) continue;
            const ScenarioDev &s = slots[t.slot].dev;
            bool bad = false;
            float bound;
            if (c & kClsDeep) {
                const int2 y = deep_rows(t);
                if (!y.y) continue;
                const int x0 = s.x_org + t.tx * kTileX + (t.sub & 1) * 2 * OUTW, y0 = t.uy * kHalfRows + y.x;
                const float m = (c & kClsPlain) ? momentum_rows<true>(s, q.parity, q.dt, x0, y0, y.y, rows, bad)
                                                : momentum_rows<false>(s, q.parity, q.dt, x0, y0, y.y, rows, bad);
                // (the reciprocal is monotone, so the smallest over the tasks is
                // that of the unit's largest lam / (2 cfl area))
                bound = (m > 0.f) ? 1.f / m : 1e30f;
            } else {
                const int y0 = t.uy * kHalfRows + (t.pair() ? t.sub >> 1 : t.sub >> 2) * t.nrows();
                const int y1 = min(y0 + t.nrows(), min(t.uy * kHalfRows + kHalfRows, s.ny));
                int strip = t.pair() ? 2 * (t.sub & 1) : t.sub & 3;
                const int last = t.pair() ? strip + 1 : strip;
                bound = FLT_MAX;
#pragma unroll 1
                for (; strip <= last; strip++) {
                    float local_min;
                    DepthAcc hacc;
                    bool cell, b;
                    int gx;
                    general_rows<2, true>(s, q.parity, q.dt, q.t_sec, t.tx, t.uy, strip, y0, y1, local_min, hacc, b, cell, gx);
                    bad |= b;
                    bound = fminf(bound, warp_min_bound(local_min));
                }
            }
            if (lane == 0) atomicMin(&slots[t.slot].dt_bits, __float_as_uint(bound));
            if (bad) fail(s, &slots[t.slot].dt_bits);
        }
        __syncthreads();
        // the block's bounds into the step's words
        unsigned *gmin = sync->dt_bits[at];
        for (int k = tid; k < L.nslots; k += kResThreads)
            if (slots[k].dt_bits != 0x7f7fffffu) {
                atomicMin(gmin + k, slots[k].dt_bits);
                slots[k].dt_bits = 0x7f7fffffu;
            }
        if (L.nslots > 1) __syncthreads();   // (one scenario: the arriving thread's own)

        // ---- the step's control, by every CTA for itself: warp 0, a lane per
        // scenario (the gauge samples by rank 0) ----
        if (warp == 0) {
            bool go = lane != 0 || arrive_and_wait(sync->phase2[at], s_team, L.wait_ns);
            go = __all_sync(0xffffffffu, go);
            __syncwarp();   // (the bounds are read after lane 0's wait)
            const int clear = at == 0 ? 2 : at - 1;   // the words every CTA is done with
            bool any = false, sampled = false;
            for (int k = lane; go && k < L.nslots; k += 32) {
                ScenarioCtl &c = slots[k].ctl;
                if (c.status != kRunning) continue;
                const ScenarioDev &s = slots[k].dev;
                const int sample = advance_scenario(c, s, __uint_as_float(__ldcg(gmin + k)), 0u);
                slots[k].state = step_state(c);
                any |= c.status == kRunning;
                if (s_rank == 0) {
                    sync->dt_bits[clear][k] = 0x7f7fffffu;
                    s_sample[k] = sample;
                    if (sample >= 0) s.gauge_ring_t[sample] = c.t * c.T;
                    sampled |= sample >= 0;
                }
            }
            any = __any_sync(0xffffffffu, any);
            sampled = __any_sync(0xffffffffu, sampled);
            if (lane == 0) {
                s_next[1] = kResWarps;
                s_ok = go;
                s_any = any;
                s_sampled = sampled;
                if (s_rank == 0 && go) {
                    sync->phase1[clear].arrived = sync->phase2[clear].arrived = sync->start.arrived = 0u;
                    sync->counts[0] = sync->counts[1] = sync->counts[2] = sync->counts[3] = 0;
                    sync->next = at == 2 ? 0 : at + 1;
                }
            }
        }
        at = at == 2 ? 0 : at + 1;
        __syncthreads();
        if (!s_ok) break;
        if (s_sampled) {
            for (int k = 0; k < L.nslots; k++) {
                const int sample = s_sample[k];
                if (sample < 0) continue;
                const ScenarioDev &s = slots[k].dev;
                float *dst = s.gauge_ring + (size_t)sample * 4 * s.ngauges;
                for (int g = tid; g < s.ngauges; g += kResThreads)
                    gauge_values(s, slots[k].state.parity, s.gauge_cells[g], dst + 4 * g, s.gauge_minmax + g);
            }
            __syncthreads();
            if (tid < kResidentSlots) s_sample[tid] = -1;
            __syncthreads();
        }
        if (!s_any) break;   // nothing left to step: every scenario of the chunk is paused or done
    }

    // ---- the end of the chunk: counts and control blocks back ----
    const bool whole = s_ok && !absent;
    if (whole && tid < ntask) {
        const Task t = tasks[tid];
        if (t.sub == 0) {
            const ScenarioDev &s = slots[t.slot].dev;
            s.dry_age[t.uy * s.tiles_x + t.tx] = (unsigned char)age;
            if (counted_deep) atomicAdd(&s.ctl->units_deep, (unsigned long long)counted_deep);
            if (counted_dry) atomicAdd(&s.ctl->units_dry, (unsigned long long)counted_dry);
        }
    }
    // A CTA whose wait ran out has stepped less than the others and kept its counts:
    // whichever it is, it reports every scenario that it has not seen end, and the
    // host fails those and clears the barrier words.
    for (int k = tid; k < L.nslots; k += kResThreads) {
        ScenarioCtl *c = slots[k].dev.ctl;
        const int status = slots[k].state.status;
        const bool ended = status == kDone || status == kFailed;
        if (!whole && !ended) atomicOr(&c->errors, 2u);
        if (s_rank == 0 && (whole || ended)) store_advanced(c, slots[k].ctl);
    }
}

}  // namespace

cudaError_t configure_resident_kernel(int device, bool *usable)
{
    *usable = false;
    int smem = 0, ctas = 0;
    cudaError_t e;
    if ((e = cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device))) return e;
    const size_t need = shared_bytes(kResidentSlots);
    if (need > (size_t)smem) return cudaSuccess;
    if ((e = cudaFuncSetAttribute(resident_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need)) ||
        (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, resident_kernel, kResThreads, need)))
        return e;
    *usable = ctas > 0;
    return cudaSuccess;
}

void launch_resident(const ResidentLaunch &L, int ctas, cudaStream_t st)
{
    resident_kernel<<<ctas, kResThreads, shared_bytes(L.nslots), st>>>(L);
}

}  // namespace thy
