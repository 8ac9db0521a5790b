// C ABI of the Okada stage on its own: the reference's aplicarOkada()
// (src/GPU/Deformacion.cu:118-143) on device memory in the reference's state
// layout (double2 (h, H) per cell, dimensionless): the FP64 vertical
// deformation of one fault, optional relative / absolute cropping, then
// H -= U_Z and eta_initial += U_Z (src/GPU/Deformacion.cu:38-53).
//
// Two entry points run the same kernels.  Neither allocates device memory,
// except that more than 64 overlapping calls of thy_apply_okada with relative
// cropping on a device take a word each from cudaMalloc.  Relative cropping needs
// the largest deformation before any is applied: thy_apply_okada evaluates the
// deformation twice (any grid size), thy_apply_okada_noalloc keeps it in the
// fixed-size device array below (and only enqueues its work).
#include <atomic>
#include <mutex>

#include <cuda.h>

#include "engine.h"

namespace thy {

// Scratch of thy_apply_okada_noalloc.  File-scope device arrays: every GPU
// that loads the library holds them (8 MiB) until the process
// exits, and every call shares them.
static __device__ __align__(256) double g_okada_scratch[THY_OKADA_NOALLOC_MAX_CELLS];
static __device__ __align__(256) unsigned int g_okada_scratch_max;

namespace {
// Device addresses of the two arrays, looked up once per device and context:
// a device reset (cudaDeviceReset) or a new primary context can load the
// module at other addresses, so a cached address is only used while the
// context it was looked up in is still the current one.
struct ScratchAddr {
    CUcontext ctx = nullptr;
    double *def = nullptr;
    unsigned int *max = nullptr;
};
std::mutex g_scratch_mu;
ScratchAddr g_scratch[64];

using CtxGetCurrentFn = CUresult (*)(CUcontext *);
CtxGetCurrentFn ctx_get_current_fn()
{
    static CtxGetCurrentFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<CtxGetCurrentFn>(p);
        else
            cudaGetLastError();
    }
    return fn;
}
}  // namespace

namespace {
// Cropping maxima of thy_apply_okada calls in progress: a call holds a word of its
// device from its start until its stream is idle.
constexpr int kMaxWords = 64;
__device__ unsigned int g_okada_max[kMaxWords];
std::atomic<unsigned long long> g_words_held[64];

class MaxWord {
public:
    ~MaxWord()
    {
        if (bit_) g_words_held[dev_].fetch_and(~bit_);
        else if (word_) cudaFree(word_);
    }
    cudaError_t claim(int dev)
    {
        if (dev < 64) {
            unsigned long long held = g_words_held[dev].load();
            while (~held) {
                const unsigned long long bit = ~held & (held + 1);   // the lowest free one
                if (!g_words_held[dev].compare_exchange_weak(held, held | bit)) continue;
                dev_ = dev;
                bit_ = bit;
                void *p = nullptr;
                const cudaError_t e = cudaGetSymbolAddress(&p, g_okada_max);
                if (e == cudaSuccess) word_ = (unsigned int *)p + __builtin_ctzll(bit);
                return e;
            }
        }
        return cudaMalloc(&word_, sizeof(unsigned int));
    }
    unsigned int *get() const { return word_; }

private:
    int dev_ = 0;
    unsigned long long bit_ = 0;
    unsigned int *word_ = nullptr;
};

int enqueue(int nx, int ny, double lon0, double dlon, double lat0, double dlat, const double *fault, double H, int crop_flag,
            double crop_value, void *state, double *eta_initial, unsigned int *max_bits, double *def, cudaStream_t st)
{
    int dev = 0, sms = 0;
    THY_CK(cudaGetDevice(&dev));
    THY_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const OkadaFault f{fault[1], fault[2], fault[3], fault[4], fault[5], fault[6], fault[7], fault[8], fault[9]};
    launch_okada_reference(nx, ny, sms, lon0, dlon, lat0, dlat, f, H, crop_flag, crop_value, (double *)state, eta_initial, max_bits,
                           def, st);
    THY_CK(cudaGetLastError());
    return THY_OK;
}
}  // namespace

int check_okada_args(int nx, int ny, const double *fault, int crop_flag, const void *state)
{
    if (nx < 2 || ny < 2 || !fault || !state || crop_flag < 0 || crop_flag > 2) return THY_ERR_INVALID;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return THY_ERR_NO_DEVICE;
    }
    return THY_OK;
}

}  // namespace thy

using namespace thy;

extern "C" int thy_apply_okada(int nx, int ny, double lon0, double dlon, double lat0, double dlat, const double *fault,
                               double H, int crop_flag, double crop_value, void *d_state1, double *d_eta_initial,
                               void *stream)
{
    int rc = check_okada_args(nx, ny, fault, crop_flag, d_state1);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    MaxWord word;
    if (crop_flag == 1) {
        int dev = 0;
        THY_CK(cudaGetDevice(&dev));
        THY_CK(word.claim(dev));
    }
    rc = enqueue(nx, ny, lon0, dlon, lat0, dlat, fault, H, crop_flag, crop_value, d_state1, d_eta_initial, word.get(), nullptr, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (rc) return rc;
    THY_CK(e);
    return THY_OK;
}

// Same computation with the library's fixed device scratch and without waiting
// for the work: for callers that cannot allocate device memory (a caching or
// budgeted allocator owns the GPU, or an allocation's implicit device-wide
// synchronisation is not acceptable).  Up to THY_OKADA_NOALLOC_MAX_CELLS
// cells; larger grids return THY_ERR_TOO_LARGE before any work.  The first
// call on a device looks up the scratch's device address there
// (cudaGetSymbolAddress), so make that first call before any stream capture;
// after a device reset the next call looks it up again (and is then again a
// first call).  The work is only enqueued on `stream`.  The scratch is shared
// by every call and keeps the last call's contents (the cropping maximum is
// cleared at the start of each call); calls whose work overlaps on the GPU
// (other streams, other host threads) race on it.
extern "C" int thy_apply_okada_noalloc(int nx, int ny, double lon0, double dlon, double lat0, double dlat,
                                       const double *fault, double H, int crop_flag, double crop_value,
                                       void *d_state1, double *d_eta_initial, void *stream)
{
    // the size first, before anything touches the device
    if (nx > 0 && ny > 0 && (long long)nx * ny > (long long)THY_OKADA_NOALLOC_MAX_CELLS) return THY_ERR_TOO_LARGE;
    int rc = check_okada_args(nx, ny, fault, crop_flag, d_state1);
    if (rc) return rc;
    int dev = 0;
    THY_CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return THY_ERR_INVALID;
    // the context the work will run in (none yet before the runtime's first
    // use of the device: the look-up below creates it)
    CtxGetCurrentFn get_ctx = ctx_get_current_fn();
    if (!get_ctx) return THY_ERR_CUDA;
    CUcontext ctx = nullptr;
    if (get_ctx(&ctx) != CUDA_SUCCESS) return THY_ERR_CUDA;
    double *def;
    unsigned int *mx;
    {
        std::lock_guard<std::mutex> lock(g_scratch_mu);
        ScratchAddr &a = g_scratch[dev];
        if (!ctx || a.ctx != ctx || !a.def || !a.max) {
            void *pd = nullptr, *pm = nullptr;
            THY_CK(cudaGetSymbolAddress(&pd, g_okada_scratch));
            THY_CK(cudaGetSymbolAddress(&pm, g_okada_scratch_max));
            if (!ctx && (get_ctx(&ctx) != CUDA_SUCCESS || !ctx)) return THY_ERR_CUDA;
            a.ctx = ctx;
            a.def = (double *)pd;
            a.max = (unsigned int *)pm;
        }
        def = a.def;
        mx = a.max;
    }
    return enqueue(nx, ny, lon0, dlon, lat0, dlat, fault, H, crop_flag, crop_value, d_state1, d_eta_initial, mx, def,
                   (cudaStream_t)stream);
}
