// Host-side engine: device state of scenarios, the time loop in chunks and its
// event handling.  Shared by thy_run (one scenario), the session API
// (benchmarking) and the server runtime (many scenarios in one batch).
#pragma once
#include <cstdint>
#include <memory>
#include <string>
#include <utility>
#include <vector>

#include <cuda_runtime.h>

#include "../../../include/thysea.h"
#include "../kernels/device.cuh"
#include "../kernels/kernels.h"
#include "tuner.h"

namespace thy {

#define THY_CK(expr)                                                          \
    do {                                                                      \
        cudaError_t _e = (expr);                                              \
        if (_e != cudaSuccess) {                                              \
            set_last_cuda_error(_e, #expr, __FILE__, __LINE__);               \
            return (_e == cudaErrorMemoryAllocation) ? THY_ERR_GPU_MEMORY : THY_ERR_CUDA; \
        }                                                                     \
    } while (0)

void set_last_cuda_error(cudaError_t e, const char *what, const char *file, int line);
const char *last_error_text();

// Device bytes one scenario of nx*ny cells needs (fields, row tables, control,
// Okada scratch when it has faults).
size_t scenario_bytes(int nx, int ny, bool has_faults);

class OutputPipe;   // asynchronous snapshot / gauge delivery (engine.cu)

// One scenario on the device.
struct DevScenario {
    int nx = 0, ny = 0, pitch = 0;
    size_t plane = 0;              // floats per field plane
    float *fields = nullptr;       // 10 planes: eta0 eta1 qx0 qx1 qy0 qy1 dep emax arr eini
    float *rows = nullptr;         // row tables
    double *def = nullptr;         // Okada scratch (nx*ny doubles)
    unsigned int *maxbits = nullptr;
    int *d_cells = nullptr;        // gauge cells
    float *d_gauge = nullptr;      // 4 floats per gauge
    float *d_gring = nullptr;      // kGaugeRing device samples x 4 floats per gauge (desc.gauge_ring)
    double *d_gring_t = nullptr;   // their times (desc.gauge_ring_t)
    float2 *d_gminmax = nullptr;   // per gauge extremes of eta (desc.gauge_minmax)
    unsigned gauges_read = 0;      // device samples handed to the outputs so far
    float *d_out = nullptr;        // 3 planes nx*ny for snapshots / outputs
    double *fault_times_d = nullptr;
    UnitSum *usum = nullptr;       // 2 parities x 2 ntiles unit depth summaries (desc.usum)
    unsigned char *dry_age = nullptr;   // 2 ntiles (desc.dry_age)
    float *gmax = nullptr;              // 2 ntiles depth steps per unit (desc.unit_gmax)
    TmaMap *tmaps = nullptr;       // kNumMaps tensor maps of the field planes (desc.tmap)
    float4 *rowpack = nullptr;     // ny+1 packed row metrics (desc.rowpack)
    ScenarioCtl *ctl = nullptr;    // device control block (owned by the batch slot)
    cudaStream_t ast = nullptr;    // stream the buffers were allocated on (stream-ordered pool)
    ScenarioDev desc{};            // descriptor (device pointers), host copy
    // problem data kept on the host
    double Hs = 1, Qs = 1, Ts = 1, Hmin = 0, Ls = 1;
    double lon0 = 0, dlon = 0, lat0 = 0, dlat = 0;
    double t_end = 0, save_nc = -1, save_ts = -1;
    long long max_steps = -1;
    int crop_flag = 0;
    double crop_value = 0;
    std::vector<double> faults;    // 10 per fault, sorted by time
    std::vector<int> cells;        // gauge cells
    int okada_flag = 0;
    // host mirror of the control block
    ScenarioCtl hctl{};
    // run bookkeeping
    int snapshots = 0, series = 0;
    double first_dt_s = 0;
    // work mix of the last chunk it stepped (per step): deep units, skipped
    // dry units; the autotuner's key for the chunks that follow
    double mix_deep = 0, mix_dry = 0;
    bool mix_known = false;
    std::unique_ptr<OutputPipe> pipe;   // created at the first snapshot / gauge sample
    // what the set-up's copies read
    std::vector<double> h_tf;
    std::vector<float2> h_mm;
    std::vector<float> h_rows;
    std::vector<float4> h_pk;
    std::vector<TmaMap> h_maps;

    long long units() const { return (long long)desc.tiles_x * ((ny + kHalfRows - 1) / kHalfRows); }   // work units
    DevScenario();
    ~DevScenario();
    int setup(const thy_problem *p, cudaStream_t st);   // allocate, upload (enqueued)
    int enqueue_setup(const thy_problem *p, cudaStream_t st);
    int upload_ctl(cudaStream_t st);
    int download_ctl(cudaStream_t st);                   // async into hctl (pinned by the batch)
    int apply_due_faults(cudaStream_t st);               // faults with time <= t (the loop's first action)
    cudaError_t invalidate_tile_minima(cudaStream_t st);
    int encode_tensor_maps(cudaStream_t st);
    int extract(int field, float *host_out, cudaStream_t st);   // enqueued
    int open_outputs(const thy_outputs *o, cudaStream_t st);
    int snapshot(const thy_outputs *o, cudaStream_t st);
    int sample_gauges(const thy_outputs *o, cudaStream_t st);
    int read_device_gauges(const thy_outputs *o, cudaStream_t st);   // the controller's samples since the last call
    int finish(const thy_outputs *o, cudaStream_t st);
};

// A set of scenarios stepped together: one work list over all their tiles,
// resident launches of the work that is small enough, and one CUDA graph of `chunk`
// steps per warp tiling the autotuner has run it with (tuner.h).
struct Batch {
    std::vector<DevScenario *> members;
    ScenarioDev *d_table = nullptr;
    int2 *d_work = nullptr;
    int *d_nwork = nullptr;
    int2 *d_work0 = nullptr;           // work list of scenarios joining (their initial dt)
    int *d_nwork0 = nullptr;
    int *d_lists = nullptr;            // deep / general lists of the current step (StepLaunch::lists)
    int *d_claims = nullptr;           // StepLaunch::claims
    // resident chunks (kernels/resident.cu), for work of up to kResidentUnits
    // units: the stepped members' descriptors and units, packed; scratch
    ScenarioDev *d_rtab = nullptr;
    int2 *d_runits = nullptr;
    int *d_rorder = nullptr;
    ResidentSync *d_rsync = nullptr;
    int res_slots = 0, res_units = 0;  // of the current work list (0: too much work)
    int res_launch = 0;                // ResidentLaunch::launch
    int res_hold = 0;                  // chunks to launch step by step, after a resident one that could not be stepped
    bool lists_stale = false;          // d_lists not made for the current states (made when a step is launched)
    ScenarioCtl *d_ctl = nullptr;      // slots
    ScenarioCtl *h_ctl = nullptr;      // pinned mirror
    int capacity = 0;
    int work_capacity = 0;
    int nwork = 0;
    int chunk = 16;
    int device = 0;
    Tiling tiling;                     // of gexec
    // step graphs captured for the current capacity, per tiling and length:
    // the full chunk, and one step, launched as often as a shorter chunk
    // needs (a session's last steps, the steps before an event)
    struct Graph {
        Tiling tiling;
        int len;
        cudaGraphExec_t exec;
    };
    std::vector<Graph> graphs;
    long long tune_samples = 0;        // chunks timed for the autotuner
    cudaStream_t st = nullptr;
    cudaStream_t st_side = nullptr;    // second branch of the captured graph (deep-water kernels)
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    cudaGraphExec_t gexec = nullptr;   // graph of the current tiling
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    double device_ms = 0;
    long long launches = 0;
    long long chunks_run = 0;
    long long captures = 0;            // graphs captured
    double capture_s = 0;              // host time spent capturing and instantiating them
    bool owns_stream = false;          // st was created for the batch (pooled batches of thy_run)
    void reset_counters();             // the per-run counters above, and the tuning samples

    ~Batch();
    int init(int capacity, int max_work, cudaStream_t stream);
    int attach(DevScenario *s);      // gives s a control slot
    int detach(DevScenario *s);
    // upload the member table and the work list (of the members with
    // selected[slot] != 0, all of them without a selection)
    int update(const std::vector<char> *selected = nullptr);
    // (re)capture the `len`-step graph of `tiling` for the current capacity
    // (len 0: the full chunk, which becomes gexec)
    int capture(int len = 0);
    int use_tiling(const Tiling &t);  // switch graphs (capturing the tiling's graph if it has none)
    void drop_graphs();
    int rebuild();                    // update(), and capture() when there is no graph yet
    int initial_dt_of(const std::vector<DevScenario *> &joining);   // initial dt of some members (phase 0 over their units only)
    // `len` steps (0 or more than max_chunk(): `chunk`; one launch for a resident
    // chunk, else a graph launch per `chunk` steps and one of the 1-step graph for
    // each of the rest) + control download (synchronous); the tiling is the
    // autotuner's pick, and a timed chunk of `chunk` steps is one of its samples
    int run_chunk(bool timed, int len = 0);
    // steps a member can take before its next event or its end, estimated
    // from its current dt (at least 1)
    static long long steps_to_event(const DevScenario &s);
    // the chunk length for `steps` steps: at least 1, at most `chunk` for a sample
    // of the tuner's, else kMaxChunk
    int chunk_for(long long steps) const;
    int max_chunk() const;
    // the autotuner's key of the next chunk: this device, its kind, the deep and
    // general units per step estimated from each stepping member's last
    // chunk (members with status running; every member when all_members);
    // *known: each of them has been measured
    TuneKey tune_key(bool *known = nullptr, bool all_members = false) const;
    StepLaunch params() const;
    void reset_lists() { lists_stale = true; }   // classify again: after the host changed a member's state
    int fresh_lists();               // the classification, if it is due (before a launch of the stepping kernels)
    class Stepping *stepping = nullptr;   // while its owner steps it
    bool resident() const;           // the next chunk is one resident launch
    int run_resident(int len, const Tiling &rows, long long all_units);
};

// A batch that is being stepped, for as long as the object lives: its units count
// among those that the process's batches step on the device, so that a resident
// chunk takes its share of the SMs only (resident_ctas) and leaves room for the
// others', and the tuner takes no sample of a device that is shared.
class Stepping {
public:
    explicit Stepping(Batch &b);
    ~Stepping();
    Stepping(const Stepping &) = delete;
    long long set(long long units);   // of the coming chunk; those of every batch on the device

private:
    Batch &b_;
    long long units_ = 0;
};

// Longest chunk that is no sample of the autotuner.  Between chunks the GPU waits
// for the host (the control blocks' copy, a launch: about 40 us before a resident
// chunk, more with a graph launch); the gauge ring keeps the samples of the steps
// between.  A queue's launched chunks stay at `chunk` steps, after which it
// admits and retires.  (Loop less device time of runs whose chunks after tuning have
// 16 / 64 steps: 1024^2, 443 steps, 0.88 / 0.44 ms; 2048^2, 986 steps, 2.0 / 1.1 ms.)
constexpr int kMaxChunk = 64;
constexpr int kResidentHold = 4;   // Batch::res_hold after a chunk that was not stepped
static_assert(kMaxChunk <= kGaugeRing, "at most one gauge sample a step");

// Single-scenario batches of thy_run, kept per device between runs with
// their buffers, stream and captured graphs, so that a run of a grid size the
// process has run before captures no graph.  A lease hands a batch with at
// least `max_work` work items to one caller at a time.
Batch *lease_run_batch(int device, int max_work, int *rc);
void return_run_batch(Batch *b, bool healthy);   // healthy = false: destroy it instead

int ensure_device();
int device_sm_count();
// the THY_ERR_* code of a scenario the controller stopped as failed
int failure_code(const ScenarioCtl &c);
// page-locked host blocks, reused across runs (engine.cu)
cudaError_t pinned_alloc(void **p, size_t bytes);
void pinned_free(void *p);

}  // namespace thy
