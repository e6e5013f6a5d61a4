// lfts_step_fwd_noalloc: the contour step (step::fwd) for callers that must
// not allocate device memory -- code running where cudaMalloc is off limits
// (a host framework that owns every device allocation through its own pool,
// a real-time loop that may not call into the allocator, or a library layered
// under an allocator-free API).  The caller passes device inputs and outputs;
// the step's scratch, the two chains' fields, lives in one file-scope device array
// of fixed size, so this path makes no allocation at all.  The kernels make their
// own twiddle and Boltzmann-weight tables in shared memory: a kernel of one CTA
// that wrote them to memory first, with a plain launch for each of the others,
// took 14.3 us a call at 24^3 against 9.9.
//
// Limits and sharing rules, stated once here and in include/lfts_b200.h:
//  * FP64 only; 2 * mx * my * (mz/2 + 1) <= LFTS_NOALLOC_MAX_SPECTRUM complex
//    values (covers every mesh up to 64^3); each dimension one of the compiled
//    FFT lengths (<= 128).
//  * The array is one per device and shared by every call: two calls whose
//    kernels overlap on a GPU (different streams, or different host threads)
//    race on it.  Serialise them (one stream, or events).
//  * Nothing in the array has to start at zero: every call rewrites the fields
//    before reading them.  The array keeps the last call's contents.
//  * The first call on a device looks up the array's device address (with
//    that device current); make that first call before any stream capture.
#include <cmath>
#include <cstdio>
#include <mutex>
#include <string>

#include <cuda_runtime.h>

#include "../../include/lfts_b200.h"
#include "axis_dispatch.h"

using namespace lfts;

// error text reported by lfts_last_error_string (lfts_capi.cu)
void lfts_internal_set_error(const char *msg);

namespace {

constexpr long long kMaxSpec = LFTS_NOALLOC_MAX_SPECTRUM;  // complex values, both chains
constexpr int kMaxLen = 128;                               // largest compiled FFT length

// the scratch: one per device, shared by all calls (see the rules above)
static __device__ __align__(256) unsigned char g_step_scratch[sizeof(cpx<double>) * kMaxSpec];

constexpr int kMaxDevices = 64;
// device address of g_step_scratch per device, looked up once per device
// (std::call_once: host threads making their first calls together wait for
// one lookup).  The address belongs to the device's primary context: after
// cudaDeviceReset on a device it is stale, like every other handle of this
// library on that device.
unsigned char *g_scratch_addr[kMaxDevices] = {};
std::once_flag g_scratch_once[kMaxDevices];
cudaError_t g_scratch_err[kMaxDevices] = {};

int fail(int code, const char *msg)
{
    lfts_internal_set_error(msg);
    return code;
}

// Per-device set-up, done by the first call on each device with that device
// current: the scratch array's device address.
int device_setup(int dev)
{
    std::call_once(g_scratch_once[dev], [dev] {
        void *p = nullptr;
        g_scratch_err[dev] = cudaGetSymbolAddress(&p, g_step_scratch);
        if (g_scratch_err[dev] == cudaSuccess && p) g_scratch_addr[dev] = static_cast<unsigned char *>(p);
    });
    if (g_scratch_err[dev] != cudaSuccess || !g_scratch_addr[dev])
        return fail(LFTS_ERR_CUDA, "cudaGetSymbolAddress(g_step_scratch) failed");
    return LFTS_OK;
}

// one launch of the step, with the kernel's dynamic shared-memory limit; one after
// the first may be scheduled while its predecessor drains (pdl_wait): its tables
// are made by then
bool launch(const AxisFn<double> &f, dim3 grid, cudaStream_t st, bool after, const AxisArgs<double> &a)
{
    if (cudaFuncSetAttribute(f.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f.smem) != cudaSuccess)
        return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(f.nt);
    cfg.dynamicSmemBytes = f.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = after ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, f.fn, a) == cudaSuccess;
}

}  // namespace

extern "C" {

int lfts_step_fwd_noalloc(const lfts_params *p, const double *q_in, double *q_out, const double *h, int i,
                          void *stream)
{
    if (!p || !q_in || !q_out || !h) return fail(LFTS_ERR_ARG, "null pointer");
    const int mx = p->m[0], my = p->m[1], mz = p->m[2];
    if (p->N < 2 || i < 1 || i >= p->N || p->NA < 0 || p->NA > p->N)
        return fail(LFTS_ERR_ARG, "chain lengths or monomer index out of range");
    if (mx < 1 || my < 1 || mz < 1 || mx > kMaxLen || my > kMaxLen || mz > kMaxLen)
        return fail(LFTS_ERR_ARG, "mesh dimension above the no-alloc limit of 128");
    for (int d = 0; d < 3; d++)
        if (!(p->L[d] > 0.0) || !std::isfinite(p->L[d]))
            return fail(LFTS_ERR_ARG, "box lengths must be positive and finite");
    const long long KZ = mz / 2 + 1;
    if (2LL * mx * my * KZ > kMaxSpec)
        return fail(LFTS_ERR_ARG, "mesh above the no-alloc scratch limit: 2*mx*my*(mz/2+1) must be <= "
                                  "LFTS_NOALLOC_MAX_SPECTRUM (64^3 meshes fit)");
    AxisStepSet ax;
    if (!axis_step_kernels(mx, my, mz, &ax))
        return fail(LFTS_ERR_UNSUPPORTED, "mesh size without an FFT kernel");
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return fail(LFTS_ERR_CUDA, "no current CUDA device");
    int rc = device_setup(dev);
    if (rc) return rc;

    unsigned char *base = g_scratch_addr[dev];
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long M = (long long)mx * my * mz;
    const int NB = p->N - p->NA;

    AxisArgs<double> a{};
    a.S = reinterpret_cast<double *>(base);
    for (int d = 0; d < 3; d++) a.L[d] = p->L[d];
    a.mx = mx;
    a.my = my;
    a.mz = mz;
    a.M = M;
    a.Nd = (double)p->N;
    a.src[0] = q_in;
    a.src[1] = q_in + M;
    a.h = h;
    a.q[0] = q_out;
    a.q[1] = q_out + M;
    a.hsel[0] = i < p->NA ? 0 : 1;  // src/step.cc:53-57
    a.hsel[1] = i < NB ? 1 : 0;     // src/step.cc:60-64
    // z and y lines, then x lines and the product with h (axis_conv.cuh)
    const AxisFn<double> &f = ax.first, &x = ax.out;
    bool ok = launch(f, dim3(ax.planes ? mx : (mx * my / 2 + f.per - 1) / f.per, 1, 2), st, false, a);
    if (!ax.planes) ok = ok && launch(ax.y, dim3((mz / 2 + ax.y.per - 1) / ax.y.per, mx, 2), st, true, a);
    ok = ok && launch(x, dim3((my * mz / 2 + x.per - 1) / x.per, 1, 2), st, true, a);
    if (!ok) return fail(LFTS_ERR_CUDA, cudaGetErrorString(cudaGetLastError()));

    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(LFTS_ERR_CUDA, cudaGetErrorString(e));
    return LFTS_OK;
}

}  // extern "C"
