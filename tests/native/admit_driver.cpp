// Admission of the multi-scenario runtime (runtime/server.cu) on the host, with the
// batch and the CUDA runtime replaced by stand-ins: a batch whose common set-up of the
// joining requests fails, as out of memory, while a scenario wider than 500 columns
// is attached.  Prints each request's completion.  Used by tests/test_server_admit.py;
// no GPU needed.
#include <cuda_runtime.h>

#include <cstdio>

static cudaError_t fake_last() { return cudaSuccess; }
static cudaError_t fake_mem(size_t *f, size_t *t) { *f = *t = (size_t)8 << 30; return cudaSuccess; }
static cudaError_t fake_create(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
static cudaError_t fake_stream(cudaStream_t) { return cudaSuccess; }
#define cudaGetLastError fake_last
#define cudaMemGetInfo fake_mem
#define cudaStreamCreateWithFlags fake_create
#define cudaStreamDestroy fake_stream
#define cudaStreamSynchronize fake_stream
#include "runtime/server.cu"

extern "C" int thy_set_device(int) { return THY_OK; }

namespace thy {
void set_last_cuda_error(cudaError_t, const char *, const char *, int) {}
int ensure_device() { return THY_OK; }
int failure_code(const ScenarioCtl &) { return THY_ERR_CUDA; }
size_t scenario_bytes(int nx, int ny, bool) { return (size_t)nx * ny * 60; }
int handle_events_ex(DevScenario &, const thy_outputs *, cudaStream_t, bool *) { return THY_OK; }

class OutputPipe {};
DevScenario::DevScenario() = default;
DevScenario::~DevScenario() {}
int DevScenario::setup(const thy_problem *p, cudaStream_t)
{
    nx = p->nx;
    ny = p->ny;
    t_end = 1.0;
    max_steps = -1;
    return nx == 13 ? THY_ERR_INVALID : THY_OK;
}
int DevScenario::upload_ctl(cudaStream_t) { return THY_OK; }
int DevScenario::read_device_gauges(const thy_outputs *, cudaStream_t) { return THY_OK; }
int DevScenario::finish(const thy_outputs *, cudaStream_t) { return THY_OK; }

Batch::~Batch() {}
int Batch::init(int cap, int, cudaStream_t)
{
    capacity = cap;
    members.assign(cap, nullptr);
    return THY_OK;
}
int Batch::attach(DevScenario *s)
{
    for (auto &m : members)
        if (!m) {
            m = s;
            return THY_OK;
        }
    return THY_ERR_BUDGET;
}
int Batch::detach(DevScenario *s)
{
    for (auto &m : members)
        if (m == s) m = nullptr;
    return THY_OK;
}
int Batch::rebuild() { return THY_OK; }
int Batch::update(const std::vector<char> *)
{
    for (auto *m : members)
        if (m && m->nx > 500) return THY_ERR_GPU_MEMORY;
    return THY_OK;
}
int Batch::initial_dt_of(const std::vector<DevScenario *> &joining)
{
    for (auto *s : joining) s->hctl.dt = 0.25;
    return THY_OK;
}
bool Batch::resident() const { return true; }
int Batch::max_chunk() const { return 64; }
int Batch::chunk_for(long long steps) const { return (int)steps; }
long long Batch::steps_to_event(const DevScenario &) { return 4; }
int Batch::run_chunk(bool, int len)
{
    for (auto *m : members)
        if (m && m->hctl.status == kRunning) {
            m->hctl.t += len * m->hctl.dt;
            m->hctl.step += len;
        }
    return THY_OK;
}
Stepping::Stepping(Batch &b) : b_(b) {}
Stepping::~Stepping() {}
}  // namespace thy

static void done(void *, long long id, int status, const thy_stats *st)
{
    std::printf("%lld %d %lld\n", id, status, st ? st->steps : -1ll);
}

int main(int argc, char **argv)
{
    thy_server_opts o{};
    thy_server *S = nullptr;
    if (thy_server_open(&o, &S)) return 1;
    double cell = 0.0;
    std::vector<thy_problem> p(argc);
    for (int i = 1; i < argc; i++) {
        p[i] = thy_problem{};
        p[i].nx = std::atoi(argv[i]);
        p[i].ny = 100;
        p[i].h = p[i].Hs = &cell;
        long long id = 0;
        if (thy_server_submit(S, &p[i], nullptr, done, nullptr, &id)) return 1;
    }
    if (thy_server_drain(S)) return 1;
    thy_server_close(S);
    return 0;
}
