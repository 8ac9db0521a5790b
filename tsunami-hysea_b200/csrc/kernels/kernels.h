// Launch wrappers of the device kernels (host-callable, no CUDA types beyond
// cudaStream_t / int2 in the signatures).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cuda_runtime.h>

namespace thy {

struct ScenarioDev;

constexpr int kStepThreads = 128;           // 4 warps = 4 column strips per tile
constexpr int kTileX = 28 * (kStepThreads / 32);   // tile width: 28 output columns per warp
constexpr int kTileY = 32;                  // tile height: rows one warp marches through

// Grid column where tile 0 starts: 0 or a negative multiple of 4 above
// -kTileX (tile 0 then holds its last 4 .. 108 columns), so that the deep
// kernels' boxes at x0 - 4 and x0 stay 16-byte aligned.  Tiles that reach
// within two cells of the left or right boundary, or into a sponge layer,
// take the general kernel, whose cost is one warp per 28-column strip holding
// a cell; the origin is the first of the 28 aligned shifts that minimises
// those strips (origin 0 when no shift does better).  Periodic grids and
// grids narrower than 2 kTileX + 4 keep origin 0.
inline int tile_origin(int nx, bool periodic, int sp_left, int sp_right)
{
    if (periodic || nx < 2 * kTileX + 4) return 0;
    const int need_l = sp_left > 2 ? sp_left : 2, need_r = sp_right > 2 ? sp_right : 2;
    int best = 0, best_cost = -1;
    for (int org = 0; org > -kTileX; org -= 4) {
        const int tiles = (nx - org + kTileX - 1) / kTileX;
        int cost = 0;
        for (int t = 0; t < tiles; t++) {
            const int x0 = org + t * kTileX;
            if (x0 >= need_l && x0 + kTileX <= nx - need_r) continue;   // may run deep
            for (int k = 0; k < kTileX / 28; k++) cost += (x0 + 28 * k + 28 > 0 && x0 + 28 * k < nx) ? 1 : 0;
        }
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = org;
        }
    }
    return best;
}

// Warp tilings of the stepping kernels, picked per workload by the autotuner
// (runtime/tuner.cu).  A work unit is always kTileX x kHalfRows cells, its
// column strips marched by warps; a tiling says into how many row groups a
// unit's rows are split (deep kernels: compute warps per CTA = 4 x groups of
// the variant, and the CTAs an SM keeps resident follow; general kernel: one
// warp task per strip and row group).  Every cell's arithmetic is the same
// under every tiling (a warp recomputes the y edge above its first row from
// the same inputs), so results do not depend on the tiling.  Variant 0 is the
// default.
constexpr int kTilingVariants = 3;
struct Tiling {
    int deep1 = 0, deep2 = 0, general = 0;   // variant of deep phase 1, deep phase 2, the general kernel
    bool operator==(const Tiling &o) const { return deep1 == o.deep1 && deep2 == o.deep2 && general == o.general; }
    bool operator!=(const Tiling &o) const { return !(*this == o); }
};
// compute warps per CTA = 4 x deep_ng {1, 2, 4}: 2 column strips of column pairs x
// twice that many row groups; general {2, 1, 8} row groups (one warp task per strip
// and row group; 8 groups of 2 rows for short chains).  (4096^2, us a launch: deep
// phase 1 95 / 98 / 107, deep phase 2 86 / 98 / 146, general 48 / 51 / 59.)
__host__ __device__ constexpr int deep_ng(int v) { return v == 0 ? 1 : v == 1 ? 2 : 4; }
// resident CTAs per SM the deep kernels are compiled for: phase 1 is held to two
// by its staging buffers (one of the largest variant, by its registers), phase 2
// to three, two or one
__host__ __device__ constexpr int deep_minb(int phase, int v) { return v == 0 ? (phase == 1 ? 2 : 3) : v == 1 ? 2 : 1; }
__host__ __device__ constexpr int general_ng(int v) { return v == 0 ? 2 : v == 1 ? 1 : 8; }

// Limit of every wait on the device (global time; each also has a limit of
// polls): what is waited for takes microseconds; the limit is seconds so that a
// context that is time-sliced or pre-empted on a shared GPU does not take a
// healthy copy or barrier for a lost one.
constexpr unsigned long long kWaitNs = 4000000000ull;

// step.cu
cudaError_t configure_step_kernels();
int step_blocks_per_sm(int general_variant);
// Launch parameters of the stepping kernels of a batch.
struct StepLaunch {
    const ScenarioDev *scen;   // scenario table (nslots entries)
    const int2 *work;          // work list: (scenario slot, tile)
    const int *nwork;          // its length (device)
    int *lists;                // deep / general lists of the step: 2 counts + 2 x cap indices
    int *claims;               // units claimed beyond the first wave by deep phase 1 / 2 and the general
                               // kernel of phase 1 / 2 (zeroed by classification); CTAs that have read the
                               // lists' lengths in phase 1, CTAs that have finished phase 2
    int cap;                   // list capacity (>= work-list length)
    int grid;                  // general kernel grid
    int deep_grid[2];          // persistent deep kernel grids, phase 1 and 2
    int classify_grid;
    int nslots;
    Tiling tiling;
    bool control;              // phase 2's last CTA runs the step controller (launch 5 is left out)
};

// The kLaunchesPerStep launches of a time step, in order: 0 deep phase 1,
// 1 general phase 1, 2 work-list classification, 3 deep phase 2, 4 general
// phase 2, 5 step controller.  Launches 0/1 and 3/4 may run concurrently; 0 and 1,
// and 3 and 4, are always launched both.
constexpr int kLaunchesPerStep = 6;
constexpr int kClaims = 6;   // words of StepLaunch::claims
void launch_step_kernel(int k, const StepLaunch &L, cudaStream_t st);
void launch_initial_dt(const StepLaunch &L, cudaStream_t st);
// lists for the current states of the work list's scenarios (from the host,
// before a chunk: after the work list or a state changed)
void launch_lists_current(const StepLaunch &L, cudaStream_t st);
// resident.cu: a chunk of steps in one launch, at most one CTA per SM, for
// work whose steps are bound by the latency of their launches
constexpr int kResidentSlots = 64;      // scenarios of such a chunk at most
// Barrier words, zero before the first launch and after one that gave up a wait
// (else the kernel leaves the ones of its next launch zero), and the scenarios'
// smallest dt bounds of a step (float bits).
struct ResidentSync {
    struct alignas(128) Word {
        unsigned arrived, pad[31];
    };
    Word team[3];                       // by launch modulo 3: CTAs that have started
    unsigned team_size[3];              // of a team closed before all had
    Word start, phase1[3], phase2[3];   // by step modulo 3, counted on from launch to launch
    unsigned int dt_bits[3][kResidentSlots];
    int next;                           // the next launch's first step, modulo 3
    int counts[4];                      // units per list at the start of the chunk
};
struct ResidentLaunch {
    const ScenarioDev *tab;    // the stepped scenarios (nslots of them)
    const int2 *units;         // their work units: (index into tab, unit)
    int *order;                // scratch, 4 x cap: the units by class
    ResidentSync *sync;
    int nslots, nunits, cap, steps;
    int rows_general, rows_deep;   // rows of a task: 1, 2, 4 or 8
    unsigned long long wait_ns;    // limit of a barrier's wait
    int launch;                    // counted from launch to launch, modulo 3
    bool drop, decline;            // test hooks: a CTA stays away from the steps' barriers; the chunk is not stepped
};
constexpr int kResidentWarps = 16;       // warps of a CTA
constexpr int resident_warps(int sms) { return sms * kResidentWarps; }           // of a launch
constexpr int resident_tasks_capacity(int warps) { return warps * 32; }          // tasks they can hold
// Largest work of a resident chunk, in units (us a step resident / launched: 640
// units 38 / 70, 1500 units 64 / 94, 2560 units 95 / 111, 3168 units 120 / 127,
// 3768 units 135 / 136, 4394 units 153 / 147, 5264 units 197 / 172: the launched
// kernels stage the deep units, which pays once every SM has enough of them to
// hide the launches).  Measured on 148 SMs; a device with fewer has as much less of
// a resident chunk's tasks and registers.
constexpr int kResidentUnits = 3712;
constexpr int resident_units(int sms) { return sms < 148 ? kResidentUnits * sms / 148 : kResidentUnits; }
static_assert(resident_units(1) * 8 <= resident_tasks_capacity(resident_warps(1)), "in rows of 8: 8 tasks a unit");
// CTAs of a resident chunk of `units`, while the process steps all_units on the
// device: its share of the SMs, at least an eighth of them and what holds its tasks.
// A chunk on every SM would make the others wait for its end (one alone has them
// all).  (Turns -> shares, ms for a run of each thread: 4 / 8 threads of 128^2 23.6 /
// 48.1 -> 9.2 / 20.4, of 512^2 40 / 81 -> 29 / 59, of 1024^2 74 / 155 -> 64 / 142; a
// 4096^2 run of 214 ms beside back-to-back runs of 128^2 to 1024^2 690..810 -> 247..257.)
inline int resident_ctas(int units, int sms, long long all_units)
{
    const int per_cta = resident_tasks_capacity(kResidentWarps);
    const int share = (int)((long long)sms * units / all_units);
    return std::min(sms, std::max({share, (sms + 7) / 8, (8 * units + per_cta - 1) / per_cta}));
}
// Rows of the tasks of a resident chunk: r = 1, 2, 4 or 8 general rows, the
// first with at most 3 r^2 / 64 units a warp, and twice as many deep rows.  Short
// tasks shorten a step's chain while warps are idle; each evaluates one y edge
// row more than it has rows, which costs more once every warp has several.  (us
// per step, 2368 warps, r = 1 / 2 / 4 / 8: 88 units 19.7 / 21.3 / 28.8 / 46.1; 108
// units 21.8 / 22.6 / 29.7 / 47.0; 240 units 30.4 / 26.3 / 31.8 / 49.1; 456 units
// 42.0 / 34.9 / 35.6 / 51.1; 640 units 52.2 / 42.8 / 40.7 / 54.2; 984 units 72.5 /
// 56.9 / 51.5 / 58.6; 1500 units r = 4 / 8 69.3 / 71.8; 1921 units 84.9 / 82.8.)
// Work the tuner searches takes its variants of the general kernel and of deep
// phase 2 as half and double the rows.
inline void resident_rows(int units, int warps, const Tiling &t, int *general, int *deep)
{
    int r = 1;
    while (r < 8 && units * 64 > 3 * r * r * warps) r *= 2;
    const auto variant = [](int rows, int v) { return std::min(8, std::max(1, v == 1 ? 2 * rows : v == 2 ? rows / 2 : rows)); };
    *general = variant(r, t.general);
    *deep = variant(std::min(8, 2 * r), t.deep2);
    // (a CTA holds one task a thread; resident_units() fit in rows of 8)
    while (std::min(*general, *deep) < 8 && units * (64 / std::min(*general, *deep)) > resident_tasks_capacity(warps)) {
        *general = std::min(8, 2 * *general);
        *deep = std::min(8, 2 * *deep);
    }
}
cudaError_t configure_resident_kernel(int device, bool *usable);   // usable: the device has room for its CTAs
void launch_resident(const ResidentLaunch &L, int ctas, cudaStream_t st);
// init_extract.cu: the step controller of every slot (launch 5 of a step)
void launch_controller(const StepLaunch &L, cudaStream_t st);
// init_extract.cu: per-unit depth steps (ScenarioDev::unit_gmax), after the
// depths change
void launch_unit_gmax(const ScenarioDev *s_host, cudaStream_t st);
// init_extract.cu / okada.cu: load their kernels now rather than at first use
cudaError_t preload_output_kernels();
cudaError_t preload_okada_kernels();
int deep_blocks_per_sm(int phase, int variant);

// init.cu: double-precision host state (reference layout, dimensionless) to
// the FP32 device state; metrics initialised as in src/GPU/ShallowWater.cu:305-309
void launch_init_state(const ScenarioDev *s_host, const ScenarioDev *s_dev, const double *h, const double *Hs,
                       const double *qx, const double *qy, double Hmin, cudaStream_t st);

// okada.cu: FP64 Okada deformation of one fault into a double scratch field,
// |U_Z| max (for relative cropping), crop and apply
struct OkadaFault {
    double lon_c, lat_c, depth_c, length, width, strike, dip, rake, slip;
};
void launch_okada(const ScenarioDev *s_host, double *def, double lon0, double dlon, double lat0, double dlat,
                  const OkadaFault &f, double Hs, cudaStream_t st);
void launch_absmax(const double *def, long long n, unsigned int *max_bits, cudaStream_t st);
void launch_apply_deformation(const ScenarioDev *s_host, const double *def, int crop_flag, double crop_value,
                              const unsigned int *max_bits, cudaStream_t st);
// Split of a row over blocks of kOkadaThreads: `segs` blocks a row of `per` cells a
// thread - up to 4, which share the row's sines, as long as every SM has its 5
// blocks.  Unsigned: the first column behind a row may lie beyond the largest int.
constexpr unsigned kOkadaThreads = 128;
struct OkadaSplit {
    unsigned per, segs;
};
inline OkadaSplit okada_split(int nx, int ny, int sms)
{
    const long long n = (long long)nx * ny;
    const unsigned per = (unsigned)std::min(4ll, std::max(1ll, n / ((long long)sms * 5 * kOkadaThreads)));
    return OkadaSplit{per, ((unsigned)nx + per * kOkadaThreads - 1) / (per * kOkadaThreads)};
}
__host__ __device__ inline unsigned okada_first_cell(const OkadaSplit &s, unsigned seg) { return seg * s.per * kOkadaThreads; }
// the whole stage on the reference's device state; crop_flag 1 uses max_bits (one
// word) and, if given, def (nx*ny doubles), otherwise both may be null
void launch_okada_reference(int nx, int ny, int sms, double lon0, double dlon, double lat0, double dlat, const OkadaFault &f,
                            double Hs, int crop_flag, double crop_value, double *state, double *eta_initial,
                            unsigned int *max_bits, double *def, cudaStream_t st);

// extract.cu: dimensional output fields (src/GPU/netcdf_kernel.cu)
enum Field { kFieldEta = 0, kFieldUx = 1, kFieldUy = 2, kFieldMaxHeight = 3, kFieldArrival = 4, kFieldDeformed = 5 };
void launch_extract(const ScenarioDev *s_host, int field, int parity, float *out, double Hs, double Qs, double Hmin,
                    cudaStream_t st);
// gauges: eta (m), ux, uy (m/s) and depth at nP cells (cell index or -1);
// fold_minmax: a sample of the series, its eta folded into the scenario's
// gauge extremes (not for the final read of the depths)
void launch_gauges(const ScenarioDev *s_host, int parity, const int *cells, int nP, float *out4, bool fold_minmax,
                   cudaStream_t st);

}  // namespace thy
