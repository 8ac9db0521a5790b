// Time-step kernels of the B200 stepper.
//
// One launched time step (work too large for resident.cu) = five launches over a
// work list of (scenario, tile) items:
//   phase 1  mass fluxes -> new surface elevation, fused with the
//            max-height / arrival-time diagnostics of the state the step
//            starts from (src/GPU/Metrics.cu:23-77) and with the depth
//            summary of each work unit of the new state (deep and general
//            kernels, concurrent);
//   classification of the units for the state phase 1 produced;
//   phase 2  momentum fluxes with the phase-1 depths -> new discharges,
//            sponge, shallow-water filter, Manning friction, local CFL dt,
//            one atomicMin per deep unit or general warp task (deep and
//            general kernels, concurrent);
//   control  (the last CTA of phase 2) time, next dt, events, gauges.
// Phases 1 and 2 are each a deep-water kernel and a general kernel.  A tile
// is deep when every cell within two cells of it is deeper than hpos and it
// is at least two cells from the boundaries and outside the sponge layers:
// then every edge flux is the pure 2s flux and no cell is dried, damped or
// relaxed, and the deep kernel marches the tile with a two-row window and
// a fraction of the instructions and registers.  Both kernels evaluate the
// same predicate on per-tile minimum depths that no launch of the phase
// writes, so every tile is stepped by exactly one of them.
// Phase 0 (the general kernel's arithmetic, one unit per CTA) computes the
// initial dt.
//
// Row marching (general kernel, step_parts.cuh): a unit is 4 column strips side by
// side, each in row groups (a tiling: 1, 2 or 8), and each (strip, row group) is a task
// of one warp, claimed independently of the others; each lane owns one
// column and the warp marches down its rows keeping a four-row window of its
// column in registers.  The y edge below the current
// row needs nothing but that window; x edges take their left/right
// neighbours from warp shuffles.  The 32 lanes cover 28 output columns plus
// a two-column halo on each side (the x stencil reaches two cells), so the
// loads of a strip are whole rows and need no shared memory.  Rows are
// loaded two ahead of the one being computed.  Each edge flux is evaluated once
// per strip: the lane right of an x edge computes it and hands the left
// cell's share to its neighbour with one shuffle; the y edge below row y is
// carried to row y+1 in registers.  No accumulator arrays, no edge
// colouring, no atomics on cells.
//
// Reference: src/GPU/Timestep.cu:11-120 (launch sequence),
// src/GPU/Arista_kernel.cu (edge fluxes), src/GPU/Volumen_kernel.cu (cell
// updates), src/GPU/Reduccion_kernel.cu (dt min).
#include "step_parts.cuh"

#include <algorithm>
#include <type_traits>
#include <cfloat>

namespace thy {

// ---------------------------------------------------------------------------
// TMA staging: one elected thread issues 2D tensor copies of a half tile's
// window into shared memory, completing on an mbarrier that every thread
// waits on with an iteration limit.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// try_wait that may suspend the thread for up to hint_ns while the phase is
// incomplete (it resumes as soon as the phase completes), so that waiting
// warps do not take issue slots from the warps that compute
__device__ __forceinline__ bool mbar_try_wait_hint(uint64_t *bar, uint32_t parity, uint32_t hint_ns)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity), "r"(hint_ns)
        : "memory");
    return ok != 0;
}
constexpr uint32_t kSuspendNs = 1000000;   // at most 1 ms per try
// Waits for the phase with this parity to complete; false when it has not
// after kWaitNs or 2^28 tries.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity)
{
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (int i = 0; i < (1 << 28); i++) {
        if (mbar_try_wait_hint(bar, parity, kSuspendNs)) return true;
        if (global_ns() - t0 > kWaitNs) return false;
    }
    return false;
}

// 2D tile load; x must be a multiple of 4 floats (16 bytes)
__device__ __forceinline__ void tma_load_2d(float *dst, const TmaMap *map, int x, int y, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

// untiled bulk copy global -> shared (no multicast): both addresses 16-byte
// aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ void tmap_acquire(const TmaMap *map)
{
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
}

// Compute warps of a deep-kernel CTA: 2 strips of column pairs x 2 NG row groups (the
// tiling's variant: by default NG = 1 in both phases, 4 warps and the producer; two
// CTAs per SM in phase 1, whose double-buffered staging is larger, three in phase 2).
constexpr int SPLANE = (kStageRows * kStageW + 31) / 32 * 32;   // floats per staged plane (128-byte multiple)
constexpr int DPLANE = kHalfRows * kTileX;          // floats per staged diagnostics plane
constexpr uint32_t kStateBytes = kStageRows * kStageW * 4;
constexpr uint32_t kDiagBytes = kHalfRows * kTileX * 4;
// x0 = x_org + tx kTileX with x_org a multiple of 4 (tile_origin)
static_assert(kTileX % 4 == 0, "TMA x coordinates x0 - 4 and x0 must be 16-byte aligned");
static_assert(kTileY == 2 * kHalfRows, "two half tiles per tile");
static_assert((SPLANE * 4) % 128 == 0 && (DPLANE * 4) % 128 == 0, "staged planes 128-byte aligned");

// Shared memory of a deep kernel CTA: two staging buffers (double buffering
// across work units), then the two mbarriers, the claimed next unit (index
// and descriptor, one slot per buffer parity) and the error flag, the staged
// row metrics of the current unit and the reduction scratch (one set per
// buffer parity).
constexpr size_t kNextBytes = 16 + 3 * 112;   // s_next[2], s_err, pad, s_unit[3]
// A staging buffer also receives the unit's packed row metrics, rows
// yb-2 .. yb+16 (a deep unit lies at least two rows inside the grid), copied
// with the planes so that they arrive one unit ahead too; each phase derives
// its row constants from them in shared memory.
constexpr int kRawRows = kStageRows + 1;
constexpr uint32_t kRawRowBytes = kRawRows * 16;
__host__ __device__ constexpr size_t deep_raw_rows_offset(int phase)
{
    return (size_t)(4 * SPLANE + (phase == 1 ? 3 * DPLANE : 0)) * sizeof(float);
}
__host__ __device__ constexpr size_t deep_stage_bytes(int phase)
{
    return deep_raw_rows_offset(phase) + (kRawRowBytes + 127) / 128 * 128;   // 128-byte aligned
}
__host__ __device__ constexpr size_t deep_misc_offset(int phase) { return 2 * deep_stage_bytes(phase); }
static size_t deep_smem_bytes(int phase, int ng)
{
    return deep_misc_offset(phase) + 16 + kNextBytes + kStageRows * sizeof(DeepRow) + 2 * 2 * 4 * ng * sizeof(float);
}

// Work lists of a step (device memory, cap entries each): lists[0] = deep
// count, lists[1] = general count, deep work-list indices at lists + 2,
// general ones at lists + 2 + cap.
__device__ __forceinline__ const int *deep_items(const int *lists) { return lists + 2; }
__device__ __forceinline__ const int *general_items(const int *lists, int cap) { return lists + 2 + cap; }

// Splits the work units into deep and general lists (dry units go to
// neither) for the state the next phase reads.  In the step (before_step = 0,
// after phase 1): for a running scenario that is the state phase 1 produced
// (summaries at parity^1), which phase 2 of this step and phase 1 of the next
// step both read, and the dry counts advance; for a scenario that is not
// running it is the state at its current parity.  From the host before a
// chunk (before_step = 1, the work list or a state changed): the state at the
// current parity for every scenario, dry counts unchanged; a state the host
// changed has unknown (NaN) summaries, so its units are general.  Units below
// the grid (the lower half of a last tile row of <= 16 rows) are not listed.
// The counts are zero before the launch (lists_read, or the host).
constexpr int kClassifyThreads = 128, kClassifyWarps = kClassifyThreads / 32;
__global__ void __launch_bounds__(kClassifyThreads) classify_kernel(const ScenarioDev *__restrict__ scen,
                                                                   const int2 *__restrict__ work,
                                const int *__restrict__ nwork_ptr, int *__restrict__ lists, int cap, int before_step,
                                int *__restrict__ claims)
{
    const int n = 2 * *nwork_ptr;
    // the deep kernels that read these lists claim units from zero (the
    // previous ones are done: this kernel runs after phase 1)
    if (blockIdx.x == 0 && threadIdx.x < 4) claims[threadIdx.x] = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ int cnt[2][kClassifyWarps];   // per warp: deep and general units of this round
    __shared__ int base2[2];                 // the block's first deep and general list slots
    for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const int u = base + threadIdx.x;
        bool listed = false, deep = false, plain = false;
        ScenarioCtl *dry_ctl = nullptr;   // the scenario of a unit skipped as dry land this step
        if (u < n) {
            const int2 item = work[u >> 1];
            const ScenarioDev &s = scen[item.x];
            const int ty = item.y / s.tiles_x, tx = item.y - ty * s.tiles_x;
            const int uy = 2 * ty + (u & 1);
            listed = uy * kHalfRows < s.ny;
            if (listed) {
                ScenarioCtl *ctl = s.ctl;
                const bool running = !before_step && ctl->status == kRunning;
                const int par = running ? (ctl->parity ^ 1) : ctl->parity;
                const UnitSum *sum = s.usum[par];
                float hmin = 0.f;
                deep = unit_deep(s, sum, tx, uy, &hmin);
                const size_t k = (size_t)uy * s.tiles_x + tx;
                plain = deep && hmin > 1.001f * s.unit_gmax[k] + 1e-6f;
                int age = s.dry_age[k];
                if (running) {
                    age = (!deep && unit_dry(s, sum, tx, uy)) ? min(age + 1, 255) : 0;
                    s.dry_age[k] = (unsigned char)age;
                }
                if (age >= kDryAge) {
                    listed = false;
                    if (running) dry_ctl = ctl;
                } else if (!deep) {
                    // a general unit: the general kernel of the next phase 1
                    // folds its summary into the other parity's entry, from
                    // the empty value (nothing reads that entry before then)
                    float2 *e = reinterpret_cast<float2 *>(&s.usum[par ^ 1][k]);
#pragma unroll
                    for (int f = 0; f < 9; f++) e[f] = make_float2(FLT_MAX, -FLT_MAX);
                }
            }
        }
        // dry units counted with one atomic per scenario and warp (the lanes
        // of a warp can belong to different scenarios of a batch)
        {
            const unsigned peers = __match_any_sync(0xffffffffu, (unsigned long long)dry_ctl);
            if (dry_ctl && lane == __ffs(peers) - 1) atomicAdd(&dry_ctl->units_dry, (unsigned long long)__popc(peers));
        }
        // block-aggregated appends: one atomic per list and block (the
        // counters are two words that every block appends to)
        const unsigned dm = __ballot_sync(0xffffffffu, listed && deep);
        const unsigned gm = __ballot_sync(0xffffffffu, listed && !deep);
        if (lane == 0) {
            cnt[0][warp] = __popc(dm);
            cnt[1][warp] = __popc(gm);
        }
        __syncthreads();
        if (threadIdx.x < 2) {
            int tot = 0;
            for (int w = 0; w < kClassifyWarps; w++) tot += cnt[threadIdx.x][w];
            base2[threadIdx.x] = tot ? atomicAdd(&lists[threadIdx.x], tot) : 0;
        }
        __syncthreads();
        int dbase = base2[0], gbase = base2[1];
        for (int w = 0; w < warp; w++) {
            dbase += cnt[0][w];
            gbase += cnt[1][w];
        }
        const unsigned below = (1u << lane) - 1u;
        if (listed) {
            if (deep) lists[2 + dbase + __popc(dm & below)] = u | (plain ? 1 << kJumpPlain : 0);
            else lists[2 + cap + gbase + __popc(gm & below)] = u;
        }
        __syncthreads();   // cnt and base2 are reused by the next round
    }
}

__device__ __forceinline__ Cell2 staged_cell2(const float *st, int i)
{
    Cell2 c;
    c.e = *reinterpret_cast<const float2 *>(st + i);
    c.D = *reinterpret_cast<const float2 *>(st + SPLANE + i);
    c.qx = *reinterpret_cast<const float2 *>(st + 2 * SPLANE + i);
    c.qy = *reinterpret_cast<const float2 *>(st + 3 * SPLANE + i);
    c.h = add2(c.e, c.D);
    return c;
}

// A deep work unit: unit code u = 2 * (work-list index) + half.
// A deep unit and what its compute warps read of its scenario (read by the
// producer when it claims the unit, so that the compute warps start the unit
// from shared memory): dt, time and parity are fixed during a launch.
struct DeepUnit {
    const ScenarioDev *s;
    ScenarioCtl *ctl;
    float *out0, *out1;       // phase 1: eta at the new parity; phase 2: qx, qy at the new parity
    float *eta_max, *arr;     // phase 1 diagnostics
    const float4 *rowpack;    // phase 2 row metrics
    UnitSum *sum;             // phase 1: the unit's summary at the new parity
    int x0, yb, p;
    int pitch;
    float dt, t_sec, eps_h, dif_at, cfl, cvis;
    bool run;
    bool drop;                // test hook: issue no copy for it (its wait runs out)
    bool plain;               // phase 2: every surface jump of the unit is the plain difference
};
static_assert(3 * sizeof(DeepUnit) + 16 <= kNextBytes, "claimed units' slots in shared memory");

template <int PHASE>
__device__ __forceinline__ DeepUnit deep_unit(const ScenarioDev *__restrict__ scen, const int2 *__restrict__ work,
                                              const int *__restrict__ lists, int i)
{
    DeepUnit d;
    const int entry = deep_items(lists)[i];
    const int u = unit_code(entry);
    d.plain = jump_plain(entry);
    const int2 item = work[u >> 1];
    d.s = &scen[item.x];
    const int ty = item.y / d.s->tiles_x, tx = item.y - ty * d.s->tiles_x;
    const int uy = 2 * ty + (u & 1);
    d.x0 = d.s->x_org + tx * kTileX;
    d.yb = uy * kHalfRows;
    const ScenarioDev &s = *d.s;
    ScenarioCtl *ctl = s.ctl;
    d.ctl = ctl;
    d.p = ctl->parity;
    d.run = *((volatile const int *)&ctl->status) == kRunning;
    d.drop = (ctl->inject & 1) != 0;
    d.pitch = s.pitch;
    d.dt = (float)ctl->dt;
    d.t_sec = (PHASE == 1) ? (float)(ctl->t * ctl->T) : 0.f;
    d.eps_h = s.eps_h;
    d.dif_at = s.dif_at;
    d.cfl = s.cfl;
    d.cvis = s.cvis;
    d.sum = &s.usum[d.p ^ 1][uy * s.tiles_x + tx];
    d.out0 = (PHASE == 1) ? s.eta[d.p ^ 1] : s.qx[d.p ^ 1];
    d.out1 = s.qy[d.p ^ 1];
    d.eta_max = s.eta_max;
    d.arr = s.arr;
    d.rowpack = s.rowpack;
    return d;
}

// TMA copies of a unit's window into one staging buffer (one thread).  The
// maps are written by host copies before the launch; a CTA acquires a
// scenario's maps once, when it first copies from that scenario (acq).
template <int PHASE>
__device__ __forceinline__ void deep_issue(const DeepUnit &d, float *stage, uint64_t *bar, const TmaMap *&acq)
{
    const TmaMap *m = d.s->tmap;
    const int p = d.p;
    const int me = (PHASE == 2) ? kMapEta0 + (p ^ 1) : kMapEta0 + p;
    if (m != acq) {
        for (int k = 0; k < kNumMaps; k++) tmap_acquire(m + k);
        acq = m;
    }
    mbar_expect_tx(bar, 4 * kStateBytes + kRawRowBytes + (PHASE == 1 ? 3 * kDiagBytes : 0));
    bulk_load(reinterpret_cast<unsigned char *>(stage) + deep_raw_rows_offset(PHASE), d.s->rowpack + d.yb - 2,
              kRawRowBytes, bar);
    tma_load_2d(stage, m + me, d.x0 - 4, d.yb - 1, bar);
    tma_load_2d(stage + SPLANE, m + kMapDep, d.x0 - 4, d.yb - 1, bar);
    tma_load_2d(stage + 2 * SPLANE, m + kMapQx0 + p, d.x0 - 4, d.yb - 1, bar);
    tma_load_2d(stage + 3 * SPLANE, m + kMapQy0 + p, d.x0 - 4, d.yb - 1, bar);
    if (PHASE == 1) {
        tma_load_2d(stage + 4 * SPLANE, m + kMapEtaMax, d.x0, d.yb, bar);
        tma_load_2d(stage + 4 * SPLANE + DPLANE, m + kMapArr, d.x0, d.yb, bar);
        tma_load_2d(stage + 4 * SPLANE + 2 * DPLANE, m + kMapEtaIni, d.x0, d.yb, bar);
    }
}

// What the CTAs of a phase's two launches do together: phase 1's zero the lists'
// lengths for the classification once all have read them, and the last one to
// finish phase 2 runs the step controller: two nodes less in a step's chain (us a
// step, 4096^2 255 -> 253, 5400 x 1801 belt 187 -> 184.5, 2048^2 112.5 -> 110.5).
constexpr int kStepMaxThreads = 128 * 4 + 32;   // of a deep or general CTA
struct StepEnds {
    int *count;   // CTAs so far; left zero
    int ctas;     // of both launches
    int nslots;   // phase 2: scenario slots to control, 0: the controller is a launch of its own
};

// Every thread of the CTA calls it after its read of the lengths.
__device__ __forceinline__ void lists_read(int *lists, const StepEnds &e)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(e.count, 1) == e.ctas - 1) {
            lists[0] = lists[1] = 0;
            *e.count = 0;
        }
    }
}

// the step controller of every slot (controller_kernel), by one CTA
__device__ __noinline__ void control_slots(const ScenarioDev *scen, int nslots, int *s_sample)
{
    for (int base = 0; base < nslots; base += blockDim.x) {
        const int k = base + threadIdx.x;
        int sample = -1;
        if (k < nslots && scen[k].ctl && scen[k].ctl->status == kRunning) {
            const ScenarioDev &s = scen[k];
            ScenarioCtl c = *s.ctl;
            // (what phase 2 changes, not from this SM's cache)
            sample = advance_scenario(c, s, __uint_as_float(__ldcg(&s.ctl->dt_bits)), __ldcg(&s.ctl->errors));
            if (sample >= 0) s.gauge_ring_t[sample] = c.t * c.T;
            store_advanced(s.ctl, c);
        }
        s_sample[threadIdx.x] = sample;
        if (!__syncthreads_or(sample >= 0)) continue;
        for (int j = 0; j < (int)blockDim.x && base + j < nslots; j++) {
            if (s_sample[j] < 0) continue;
            const ScenarioDev &s = scen[base + j];
            const int parity = *(volatile const int *)&s.ctl->parity;
            float *dst = s.gauge_ring + (size_t)s_sample[j] * 4 * s.ngauges;
            for (int g = threadIdx.x; g < s.ngauges; g += blockDim.x)
                gauge_values(s, parity, s.gauge_cells[g], dst + 4 * g, s.gauge_minmax + g);
        }
        __syncthreads();   // s_sample is reused by the next round
    }
}

__device__ __forceinline__ void phase2_done(const ScenarioDev *scen, const StepEnds &e)
{
    if (e.nslots == 0) return;
    __shared__ int s_last, s_sample[kStepMaxThreads];
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(e.count, 1) == e.ctas - 1;
        if (s_last) *e.count = 0;
        __threadfence();
    }
    __syncthreads();
    if (s_last) control_slots(scen, e.nslots, s_sample);
}

// Phase 1 / 2 of the deep tiles, persistent, over the units of the deep list
// (two per tile: its upper and lower half).  A unit's window - its rows plus
// one above and one below, columns x0-4 .. x0+115 of eta, dep, qx, qy, and in
// phase 1 the diagnostics of its own cells and the row metrics - is staged by
// TMA, the next unit's copy in flight while the current one is computed.
// Compute warp w marches its row group (w >> 1) of column strip w & 1 (56 output
// columns, two a lane) with a two-row window; one more warp is the producer.
//
// What bounds it (4096^2, 8074 units): phase 1 memory, 476 MB in 92 us, 80 % of
// the measured copy rate (one column a lane: 99 us; a third of its instructions
// went with the pairs); phase 2 issue, 57 M warp instructions at 0.64 a scheduler
// and cycle in 86 us (89 with the next unit's descriptor read only when its buffer
// was free).
template <int PHASE, int NG>
__device__ __forceinline__ void deep_units(const ScenarioDev *__restrict__ scen, const int2 *__restrict__ work, int *lists,
                                           int *claim, const StepEnds &ends)
{
    extern __shared__ __align__(1024) unsigned char dsm[];
    constexpr size_t SB = deep_stage_bytes(PHASE);
    constexpr int NW = 4 * NG;      // compute warps
    constexpr int PT = NW * 32;     // the producer: lane 0 of warp NW
    // staging buffer b at dsm + b * SB
    unsigned char *misc = dsm + deep_misc_offset(PHASE);
    uint64_t *bars = reinterpret_cast<uint64_t *>(misc);
    int *s_next = reinterpret_cast<int *>(misc + 16);          // [parity]: the unit after the current one
    int &s_err = *reinterpret_cast<int *>(misc + 24);          // a copy did not land in time
    DeepUnit *s_unit = reinterpret_cast<DeepUnit *>(misc + 32);   // descriptors, unit k of the CTA in slot k % 3
    DeepRow *rows = reinterpret_cast<DeepRow *>(misc + 16 + kNextBytes);
    float *red0 = reinterpret_cast<float *>(rows + kStageRows);   // [parity][2 NW]: per warp dt, or depth min and max
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool producer = warp == NW;
    const int nunits = lists[0];
    if (PHASE == 1) lists_read(lists, ends);
    if (blockIdx.x >= nunits) return;
    // TMA destinations must be 128-byte aligned: a misaligned buffer is
    // reported on every scenario of the CTA's units and nothing is copied
    if (smem_addr(dsm) & 127u) {
        if (threadIdx.x == PT)
            for (int u = blockIdx.x; u < nunits; u += gridDim.x)
                atomicOr(&scen[work[unit_code(deep_items(lists)[u]) >> 1].x].ctl->errors, 4u);
        return;
    }
    if (threadIdx.x == PT) {
        mbar_init(&bars[0]);
        mbar_init(&bars[1]);
        s_err = 0;
    }
    __syncthreads();
    uint32_t phase_bits = 0;     // bit b: parity of the next completion of bars[b]
    const TmaMap *acq = nullptr; // maps acquired by this CTA (producer)
    // The first two waves take units blockIdx.x and blockIdx.x + gridDim.x;
    // after that each CTA claims its units from the counter (2 gridDim.x,
    // 2 gridDim.x + 1, ...), so a CTA that started late, or whose units took
    // longer, takes fewer.  A producer warp issues the copies of the next unit,
    // reduces the previous unit's results, and claims the unit after the next one
    // and reads its descriptor (a chain of five loads, done by the time its buffer
    // is free), while the compute warps step the current unit; they meet once per
    // unit, and the producer publishes the next unit there.
    DeepUnit d = deep_unit<PHASE>(scen, work, lists, blockIdx.x);
    int next = blockIdx.x + gridDim.x, slot = 1;   // producer: the next unit; its descriptor's slot
    if (threadIdx.x == PT) {
        if (d.run && !d.drop) deep_issue<PHASE>(d, reinterpret_cast<float *>(dsm), &bars[0], acq);
        if (next < nunits) s_unit[1] = deep_unit<PHASE>(scen, work, lists, next);
    }
    // a unit's results from its warps' (thread PT)
    auto reduce = [&](const DeepUnit &q, const float *red) {
        float m = red[0];
        for (int k = 1; k < NW; k++) m = (PHASE == 1) ? fminf(m, red[k]) : fmaxf(m, red[k]);
        if (PHASE == 1) {
            // a deep unit reports its whole-unit {min, max} for its strips
            // and corners too: conservative for a neighbour's deep test,
            // and a wet unit fails a neighbour's dry test either way
            float mx = red[NW];
            for (int k = 1; k < NW; k++) mx = fmaxf(mx, red[NW + k]);
            const float2 v = make_float2(m, mx);
            *q.sum = UnitSum{v, v, v, v, v, v, v, v, v};
        } else {
            // the unit's dt bound from its largest lam / (2 cfl area), inverted
            // once per unit so that it does not depend on the warps' rows
            m = (m > 0.f) ? 1.f / m : 1e30f;
            atomicMin(&q.ctl->dt_bits, __float_as_uint(m));
            atomicAdd(&q.ctl->units_deep, 1ull);
        }
    };
    DeepUnit prev;   // thread PT: the previous unit
    prev.run = false;
    int buf = 0;
    for (int u = blockIdx.x; u < nunits; buf ^= 1) {
        float *red = red0 + buf * 2 * NW;
        if (producer) {
            // the next unit's copy goes to the other buffer, free since the
            // compute warps passed the end of the previous unit
            if (lane == 0) {
                s_next[buf ^ 1] = next;
                if (next < nunits) {
                    const DeepUnit &dn = s_unit[slot];
                    if (dn.run && !dn.drop)
                        deep_issue<PHASE>(dn, reinterpret_cast<float *>(dsm + (buf ^ 1) * SB), &bars[buf ^ 1], acq);
                    next = 2 * (int)gridDim.x + atomicAdd(claim, 1);
                    // (three slots: the compute warps may still be reading the current unit's)
                    if (next < nunits) s_unit[slot == 2 ? 0 : slot + 1] = deep_unit<PHASE>(scen, work, lists, next);
                }
                if (prev.run) reduce(prev, red0 + (buf ^ 1) * 2 * NW);
            }
        } else if (d.run) {
            ScenarioCtl *ctl = d.ctl;
            const int x0 = d.x0, yb = d.yb;
            const float dt = d.dt;
            if (!mbar_wait_bounded(&bars[buf], (phase_bits >> buf) & 1u)) s_err = 1;
            const float4 *raw = reinterpret_cast<const float4 *>(dsm + buf * SB + deep_raw_rows_offset(PHASE));
            if (PHASE == 2 && threadIdx.x < kStageRows) {
                // row constants of the window with the unit's dt folded in, from
                // the staged row metrics (row t of the window at t + 1; staged
                // row t is grid row yb - 1 + t)
                rows[threadIdx.x] = deep_row(raw[threadIdx.x + 1], raw[threadIdx.x], dt, d.cfl, d.cvis);
            }
            if (PHASE == 1 && threadIdx.x < kStageRows) {
                // phase 1 row constants from the staged row metrics: 1/cos for
                // the y edges, dt/area
                DeepRow r;
                r.m = raw[threadIdx.x + 1];
                r.icos = __frcp_rn(r.m.x);
                r.dtA = __fdividef(dt, r.m.z);
                rows[threadIdx.x] = r;
            }
            // the compute warps only: the row constants are written, every copy checked
            asm volatile("bar.sync 1, %0;" ::"r"(PT) : "memory");
            if (!s_err) {
              // in pairs: two column strips of 56 cells; lane l steps staged
              // columns sc0 and sc0 + 1 (lanes 1..28 are cells, lanes 0 and 29 the
              // halo, lanes 30 and 31 repeat lane 29)
              constexpr int NG2 = 2 * NG, nrows = kHalfRows / NG2;   // row groups, rows per warp
              static_assert(kHalfRows % NG2 == 0, "row groups of equal height");
              const int strip2 = warp & 1, prow0 = nrows * (warp >> 1);
              const int sc0 = strip2 * 56 + 2 + 2 * min(lane, 29);
              const bool out_lane = (lane >= 1) && (lane <= 28);
              if constexpr (PHASE == 1) {
                const float *stage = reinterpret_cast<const float *>(dsm + buf * SB);
                const float t_sec = d.t_sec;
                float local_min = FLT_MAX, local_max = -FLT_MAX;   // depths
                int i = prow0 * kStageW + sc0;                     // staged cells of the row above
                const float *dg = stage + 4 * SPLANE + prow0 * kTileX + strip2 * 56 + 2 * (lane - 1);   // (of output lanes)
                int off = (yb + prow0) * d.pitch + x0 - 4 + sc0;
                Cell2 a = staged_cell2(stage, i), c = staged_cell2(stage, i + kStageW);
                float2 top = mul2(mass_y2(a, c, rows[prow0].m, rows[prow0 + 1].m, dt), bc2(rows[prow0 + 1].icos));
                float2 fin = make_float2(0.f, 0.f);   // running sum: non-finite iff a new value is
#pragma unroll 1
                for (int k = prow0 + 1; k <= prow0 + nrows; k++, off += d.pitch, dg += kTileX) {
                    i += kStageW;
                    const Cell2 n = staged_cell2(stage, i + kStageW);
                    const float2 e = mass_pair(c, n, rows[k], rows[k + 1], dt, top);
                    if (out_lane) {
                        // diagnostics of the state the step starts from (src/GPU/Metrics.cu:23-77)
                        const float2 em = *reinterpret_cast<const float2 *>(dg);
                        const float2 ar = *reinterpret_cast<const float2 *>(dg + DPLANE);
                        const float2 ei = *reinterpret_cast<const float2 *>(dg + 2 * DPLANE);
                        if (c.e.x > em.x && c.h.x > d.eps_h) d.eta_max[off] = c.e.x;
                        if (c.e.y > em.y && c.h.y > d.eps_h) d.eta_max[off + 1] = c.e.y;
                        if (ar.x < 0.f && fabsf(c.e.x - ei.x) > d.dif_at) d.arr[off] = t_sec;
                        if (ar.y < 0.f && fabsf(c.e.y - ei.y) > d.dif_at) d.arr[off + 1] = t_sec;
                        const float2 h = add2(e, c.D);
                        fin = add2(fin, e);
                        *reinterpret_cast<float2 *>(d.out0 + off) = e;
                        local_min = fminf(local_min, fminf(h.x, h.y));
                        local_max = fmaxf(local_max, fmaxf(h.x, h.y));
                    }
                    c = n;
                }
                if (!isfinite(fin.x) || !isfinite(fin.y)) atomicOr(&ctl->errors, 1u);
                const float2 mm = warp_minmax(local_min, local_max, out_lane);
                local_min = mm.x;
                local_max = mm.y;
                if (lane == 0) {
                    red[warp] = local_min;
                    red[NW + warp] = local_max;
                }
              } else {
                float local_max = -FLT_MAX;                        // max of lam / (2 cfl area)
                float2 fin = make_float2(0.f, 0.f);   // running sum: non-finite iff a new value is
                // the row loop in two copies: surface jumps with their wet/dry
                // tests, or as plain differences (a unit the classification
                // found deeper than its depth steps); a uniform branch per unit
                auto pair_rows = [&](auto plain_tag) {
                    constexpr bool PLAIN = decltype(plain_tag)::value;
                    const float *stage = reinterpret_cast<const float *>(dsm + buf * SB);
                    const int pitch = d.pitch;
                    const int r_first = prow0 + 1;                    // staged row of this warp's first output row
                    int i = r_first * kStageW + sc0;
                    Cell2 c = staged_cell2(stage, i);
                    const Depth2 fc = depth2(c.h);
                    float2 rh_c = fc.rh, sh_c = fc.sh;
                    DeepRow rc = rows[r_first];
                    Contrib2 top;
                    {
                        const Cell2 a = staged_cell2(stage, i - kStageW);
                        Contrib2 dummy;
                        const Depth2 fa = depth2(a.h);
                        y_edge_deep2<PLAIN>(a, c, fa.rh, fa.sh, rh_c, sh_c, rows[r_first - 1], rc, dummy, top);
                    }
                    float *out0 = d.out0, *out1 = d.out1;
                    int off = (yb + r_first - 1) * pitch + x0 - 4 + sc0;
                    // two rows an iteration, so that the row window is renamed
                    // rather than copied (every operation here is explicitly
                    // rounded: the copies compute alike)
    #pragma unroll 2
                    for (int k = 0; k < nrows; k++, i += kStageW, off += pitch) {
                        const DeepRow rn = rows[r_first + k + 1];
                        const Cell2 n = staged_cell2(stage, i + kStageW);
                        const Depth2 fn = depth2(n.h);
                        const float2 rh_n = fn.rh, sh_n = fn.sh;
                        // y edges below this row
                        Contrib2 below, next_top;
                        y_edge_deep2<PLAIN>(c, n, rh_c, sh_c, rh_n, sh_n, rc, rn, below, next_top);
                        // x edges and update
                        float2 qx, qy;
                        float wm;
                        pair_update<PLAIN>(c, Depth2{rh_c, sh_c}, rc, top, below, qx, qy, wm);
                        if (out_lane) local_max = fmaxf(local_max, wm);
                        if (out_lane) {
                            fin = add2(fin, add2(qx, qy));
                            *reinterpret_cast<float2 *>(out0 + off) = qx;
                            *reinterpret_cast<float2 *>(out1 + off) = qy;
                        }
                        top = next_top;
                        rc = rn;
                        c = n;
                        rh_c = rh_n;
                        sh_c = sh_n;
                    }
                };
                if (d.plain) pair_rows(std::true_type{});
                else pair_rows(std::false_type{});
                if (!isfinite(fin.x) || !isfinite(fin.y)) atomicOr(&ctl->errors, 1u);
                for (int o = 16; o > 0; o >>= 1) local_max = fmaxf(local_max, __shfl_xor_sync(0xffffffffu, local_max, o));
                if (lane == 0) red[warp] = local_max;
              }
            }
        }
        if (d.run) phase_bits ^= 1u << buf;
        // every compute warp is done with the staged window, the row metrics
        // and its results; the next unit and the error flag are published
        __syncthreads();
        if (s_err) {
            // a copy did not land in time: report; the producer gives both
            // buffers' copies one more bounded wait so none is still writing; stop
            if (threadIdx.x == PT) {
                atomicOr(&d.s->ctl->errors, 2u);
                if (!d.drop) mbar_wait_bounded(&bars[buf], ((phase_bits >> buf) & 1u) ^ 1u);
                if (s_next[buf ^ 1] < nunits && s_unit[slot].run && !s_unit[slot].drop)
                    mbar_wait_bounded(&bars[buf ^ 1], (phase_bits >> (buf ^ 1)) & 1u);
            }
            return;
        }
        if (threadIdx.x == PT) prev = d;
        u = s_next[buf ^ 1];
        d = s_unit[slot];   // valid when u < nunits
        slot = slot == 2 ? 0 : slot + 1;
    }
    if (threadIdx.x == PT && prev.run) reduce(prev, red0 + (buf ^ 1) * 2 * NW);
}

template <int PHASE, int NG, int MINB>
__global__ void __launch_bounds__(128 * NG + 32, MINB) deep_kernel(const ScenarioDev *__restrict__ scen,
                                                                const int2 *__restrict__ work, int *lists, int *claim,
                                                                const StepEnds ends)
{
    deep_units<PHASE, NG>(scen, work, lists, claim, ends);
    if (PHASE == 2) phase2_done(scen, ends);
}

// Phase 0 (the initial dt) over every unit of the work list, one unit per CTA
// iteration, 4 x NG warps; the last unit of a scenario stores its dt.
template <int NG>
__global__ void __launch_bounds__(128 * NG) initial_dt_kernel(const ScenarioDev *__restrict__ scen,
                                                              const int2 *__restrict__ work,
                                                              const int *__restrict__ nwork_ptr)
{
    constexpr int GWARPS = 4 * NG;
    __shared__ float red[GWARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int strip = warp % STRIPS, group = warp / STRIPS;
    const int nitems = 2 * *nwork_ptr;
    for (int u = blockIdx.x; u < nitems; u += gridDim.x) {
        const int2 item = work[u >> 1];
        const ScenarioDev &s = scen[item.x];
        ScenarioCtl *ctl = s.ctl;
        const int ty = item.y / s.tiles_x, tx = item.y - ty * s.tiles_x;
        const int uy = 2 * ty + (u & 1);
        if (uy * kHalfRows >= s.ny) continue;   // a unit below the grid (CTA-uniform)
        constexpr int GROWS = kHalfRows / NG;
        const int y0 = uy * kHalfRows + group * GROWS;
        float local_min;
        initial_rows(s, ctl->parity, tx, uy, strip, y0, min(y0 + GROWS, min(uy * kHalfRows + kHalfRows, s.ny)), local_min);
        for (int o = 16; o > 0; o >>= 1) local_min = fminf(local_min, __shfl_xor_sync(0xffffffffu, local_min, o));
        if (lane == 0) red[warp] = local_min;
        __syncthreads();
        if (threadIdx.x == 0) {
            float m = red[0];
            for (int k = 1; k < GWARPS; k++) m = fminf(m, red[k]);
            atomicMin(&ctl->dt_bits, __float_as_uint(m));
            // the last unit stores the min and resets the counters
            __threadfence();
            const unsigned prev = atomicAdd(&ctl->tiles_done, 1u);
            if (prev == (unsigned)(s.tiles_x * units_y(s) - 1)) {
                __threadfence();
                ctl->dt = (double)__uint_as_float(atomicOr(&ctl->dt_bits, 0u));
                ctl->dt_bits = 0x7f7fffffu;
                ctl->tiles_done = 0u;
            }
        }
        __syncthreads();   // red[] is reused by the next unit
    }
}

// Phases 1 and 2 over the general list of the step.  Every warp runs tasks on
// its own: the first wave takes tasks by warp index, then each warp claims
// its next task from *claim (zeroed by the classification), so no warp waits
// for another and a unit's strips outside the grid (in the first and last
// tile columns) cost nothing.  The tasks of a unit are consecutive, so that
// its strips and row groups run side by side and share their halo rows in L2.
constexpr int kGeneralThreads = 128;
template <int PHASE, int NG>
__global__ void __launch_bounds__(kGeneralThreads, 4) general_kernel(const ScenarioDev *__restrict__ scen,
                                                                    const int2 *__restrict__ work,
                                                                    int *lists, int cap, int *claim,
                                                                    const StepEnds ends)
{
    constexpr int TASKS = STRIPS * NG;   // tasks per unit
    constexpr int WPB = kGeneralThreads / 32;
    const int lane = threadIdx.x & 31;
    const int ntasks = lists[1] * TASKS;
    if (PHASE == 1) lists_read(lists, ends);
    const int first_wave = (int)gridDim.x * WPB;
    int t = blockIdx.x * WPB + (threadIdx.x >> 5);
    while (t < ntasks) {
        const int g = t / TASKS, r = t - g * TASKS;
        const int group = r / STRIPS, strip = r - group * STRIPS;
        const int u = general_items(lists, cap)[g];
        const int2 item = work[u >> 1];
        const ScenarioDev &s = scen[item.x];
        ScenarioCtl *ctl = s.ctl;
        if (*((volatile int *)&ctl->status) == kRunning) {
            const int ty = item.y / s.tiles_x, tx = item.y - ty * s.tiles_x;
            const int uy = 2 * ty + (u & 1);
            float local_min;
            DepthAcc hacc;
            bool bad, cell;
            int gx;
            general_part<PHASE, NG>(s, ctl, tx, uy, strip, group, local_min, hacc, bad, cell, gx);
            if (bad) atomicOr(&ctl->errors, 1u);
            if (PHASE == 1) {
                // the unit's first two and last two columns inside the grid
                const int tx0 = s.x_org + tx * kTileX, ux0 = max(tx0, 0), ux1 = min(tx0 + kTileX, s.nx);
                fold_unit_summary(hacc, cell, cell && gx < ux0 + 2, cell && gx >= ux1 - 2,
                                  &s.usum[ctl->parity ^ 1][(size_t)uy * s.tiles_x + tx]);
            } else {
                // the minimum is exact in any order
                local_min = warp_min_bound(local_min);
                if (lane == 0) atomicMin(&ctl->dt_bits, __float_as_uint(local_min));
            }
        }
        int next = 0;
        if (lane == 0) next = first_wave + atomicAdd(claim, 1);
        t = __shfl_sync(0xffffffffu, next, 0);
    }
    if (PHASE == 2) phase2_done(scen, ends);
}

template <int PHASE>
static StepEnds step_ends(const StepLaunch &L)
{
    return StepEnds{L.claims + 3 + PHASE, L.deep_grid[PHASE - 1] + L.grid, PHASE == 2 && L.control ? L.nslots : 0};
}

// One launch of deep phase PHASE / the general kernel in variant V.
template <int PHASE, int V>
static void launch_deep(const StepLaunch &L, cudaStream_t st)
{
    constexpr int NG = deep_ng(V);
    deep_kernel<PHASE, NG, deep_minb(PHASE, V)>
        <<<L.deep_grid[PHASE - 1], 128 * NG + 32, deep_smem_bytes(PHASE, NG), st>>>(L.scen, L.work, L.lists,
                                                                            L.claims + (PHASE - 1), step_ends<PHASE>(L));
}
template <int PHASE>
static void launch_deep_any(const StepLaunch &L, cudaStream_t st)
{
    switch (PHASE == 1 ? L.tiling.deep1 : L.tiling.deep2) {
    case 1: launch_deep<PHASE, 1>(L, st); break;
    case 2: launch_deep<PHASE, 2>(L, st); break;
    default: launch_deep<PHASE, 0>(L, st); break;
    }
}
template <int PHASE, int V>
static void launch_general_v(const StepLaunch &L, cudaStream_t st)
{
    general_kernel<PHASE, general_ng(V)><<<L.grid, kGeneralThreads, 0, st>>>(L.scen, L.work, L.lists, L.cap,
                                                                            L.claims + 2 + (PHASE - 1), step_ends<PHASE>(L));
}
template <int PHASE>
static void launch_general(const StepLaunch &L, cudaStream_t st)
{
    switch (L.tiling.general) {
    case 1: launch_general_v<PHASE, 1>(L, st); break;
    case 2: launch_general_v<PHASE, 2>(L, st); break;
    default: launch_general_v<PHASE, 0>(L, st); break;
    }
}

void launch_step_kernel(int k, const StepLaunch &L, cudaStream_t st)
{
    switch (k) {
    case 0: launch_deep_any<1>(L, st); break;
    case 1: launch_general<1>(L, st); break;
    case 2:
        classify_kernel<<<L.classify_grid, kClassifyThreads, 0, st>>>(L.scen, L.work, L.nwork, L.lists, L.cap, 0, L.claims);
        break;
    case 3: launch_deep_any<2>(L, st); break;
    case 4: launch_general<2>(L, st); break;
    default: launch_controller(L, st); break;
    }
}

// phase 0 (initial dt) runs once per scenario: default tiling, the grid of L
void launch_initial_dt(const StepLaunch &L, cudaStream_t st)
{
    initial_dt_kernel<general_ng(0)><<<L.grid, 128 * general_ng(0), 0, st>>>(L.scen, L.work, L.nwork);
}

void launch_lists_current(const StepLaunch &L, cudaStream_t st)
{
    cudaMemsetAsync(L.lists, 0, 2 * sizeof(int), st);
    classify_kernel<<<L.classify_grid, kClassifyThreads, 0, st>>>(L.scen, L.work, L.nwork, L.lists, L.cap, 1, L.claims);
}

template <int PHASE, int V>
static cudaError_t configure_deep()
{
    constexpr int NG = deep_ng(V);
    auto *f = deep_kernel<PHASE, NG, deep_minb(PHASE, V)>;
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)deep_smem_bytes(PHASE, NG));
    if (e) return e;
    return cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
}

// Loads every step kernel now (module loading is otherwise lazy, at a
// kernel's first launch or graph instantiation: inside the first run's loop).
template <typename F>
static cudaError_t preload(F *f)
{
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, f);
}

cudaError_t configure_step_kernels()
{
    cudaError_t e;
    if ((e = preload(initial_dt_kernel<general_ng(0)>)) || (e = preload(general_kernel<1, general_ng(0)>)) ||
        (e = preload(general_kernel<1, general_ng(1)>)) || (e = preload(general_kernel<1, general_ng(2)>)) ||
        (e = preload(general_kernel<2, general_ng(0)>)) || (e = preload(general_kernel<2, general_ng(1)>)) ||
        (e = preload(general_kernel<2, general_ng(2)>)) || (e = preload(classify_kernel)))
        return e;
    if ((e = configure_deep<1, 0>()) || (e = configure_deep<1, 1>()) || (e = configure_deep<1, 2>()) ||
        (e = configure_deep<2, 0>()) || (e = configure_deep<2, 1>()) || (e = configure_deep<2, 2>()))
        return e;
    return cudaSuccess;
}

// Resident CTAs per SM of the phase-2 general kernel / a deep kernel in a variant.
int step_blocks_per_sm(int v)
{
    int n = 0;
    switch (v) {
    case 1: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, general_kernel<2, general_ng(1)>, kGeneralThreads, 0); break;
    case 2: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, general_kernel<2, general_ng(2)>, kGeneralThreads, 0); break;
    default: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, general_kernel<2, general_ng(0)>, kGeneralThreads, 0); break;
    }
    return n;
}

template <int PHASE, int V>
static int deep_occupancy()
{
    constexpr int NG = deep_ng(V);
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, deep_kernel<PHASE, NG, deep_minb(PHASE, V)>, 128 * NG + 32,
                                                  deep_smem_bytes(PHASE, NG));
    return n;
}

int deep_blocks_per_sm(int phase, int v)
{
    if (phase == 1) return v == 1 ? deep_occupancy<1, 1>() : v == 2 ? deep_occupancy<1, 2>() : deep_occupancy<1, 0>();
    return v == 1 ? deep_occupancy<2, 1>() : v == 2 ? deep_occupancy<2, 2>() : deep_occupancy<2, 0>();
}

}  // namespace thy
