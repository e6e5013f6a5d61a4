// C ABI of the B200 L-FTS step (include/lfts_b200.h): device state, launch
// orchestration and the small host-side pieces (Anderson least squares,
// S(k) bin tables) around the kernels in fft_kernels.cuh / field_kernels.cuh.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <tuple>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/lfts_b200.h"
#include "anderson_device.cuh"
#include "ctx.h"
#include "field_kernels.cuh"

using namespace lfts;

namespace {

thread_local std::string g_last_error = "";

int cuda_fail(cudaError_t e, const char *what)
{
    char buf[512];
    snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
    g_last_error = buf;
    return LFTS_ERR_CUDA;
}

#define CK(call)                                           \
    do {                                                   \
        cudaError_t e_ = (call);                           \
        if (e_ != cudaSuccess) return cuda_fail(e_, #call); \
    } while (0)

constexpr double kTwoPi = 6.283185307179586476925286766559005768;
// x-pencil tile widths used when autotuning is off (the usual winners at 128^3)
constexpr int kDefaultCwFp32 = 16, kDefaultCwFp64 = 16;

// Gaussian elimination with partial pivoting (first maximal |pivot|,
// reciprocal scaling of the sub-column, right-looking rank-1 updates), then
// forward/back substitution: the LU solve the reference does with GSL at
// src/anderson.cc:106-127.  Returns false for an exactly singular matrix,
// where GSL's solve reports an error.
bool lu_solve(std::vector<double> A, std::vector<double> y, double *x, int n)
{
    std::vector<int> perm(n);
    std::iota(perm.begin(), perm.end(), 0);
    for (int j = 0; j < n; j++) {
        int piv = j;
        double amax = std::fabs(A[j * n + j]);
        for (int i = j + 1; i < n; i++) {
            double v = std::fabs(A[i * n + j]);
            if (v > amax) { amax = v; piv = i; }
        }
        if (piv != j) {
            for (int k = 0; k < n; k++) std::swap(A[j * n + k], A[piv * n + k]);
            std::swap(perm[j], perm[piv]);
        }
        if (j + 1 < n) {
            const double ajj = A[j * n + j];
            if (std::fabs(ajj) >= 2.2250738585072014e-308) {
                const double inv = 1.0 / ajj;
                for (int i = j + 1; i < n; i++) A[i * n + j] *= inv;
            } else {
                for (int i = j + 1; i < n; i++) A[i * n + j] /= ajj;
            }
            for (int i = j + 1; i < n; i++) {
                const double lij = A[i * n + j];
                for (int k = j + 1; k < n; k++) A[i * n + k] -= lij * A[j * n + k];
            }
        }
    }
    for (int i = 0; i < n; i++)
        if (A[i * n + i] == 0.0) return false;
    for (int i = 0; i < n; i++) x[i] = y[perm[i]];
    for (int i = 0; i < n; i++) {
        double t = x[i];
        for (int j = 0; j < i; j++) t -= A[i * n + j] * x[j];
        x[i] = t;
    }
    for (int i = n - 1; i >= 0; i--) {
        double t = x[i];
        for (int j = i + 1; j < n; j++) t -= A[i * n + j] * x[j];
        x[i] = t / A[i * n + i];
    }
    return true;
}

// signed wavenumber of index K in [0, m): -(m-1)/2 .. m/2 (src/step.cc:69-79)
inline int signed_k(int K, int m) { return (K <= m / 2) ? K : K - m; }

}  // namespace

// shared with lfts_noalloc.cu, which reports through lfts_last_error_string
void lfts_internal_set_error(const char *msg) { g_last_error = msg; }


namespace {

template <typename T>
AxisSet<T> &axis_of(lfts_ctx *c);
template <>
AxisSet<double> &axis_of<double>(lfts_ctx *c) { return c->ax64; }
template <>
AxisSet<float> &axis_of<float>(lfts_ctx *c) { return c->ax32; }

template <typename T>
int set_smem(const AxisFn<T> &f)
{
    if (f.fn) CK(cudaFuncSetAttribute(f.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f.smem));
    return LFTS_OK;
}

// the axis kernels of this context's mesh with x and y tiles of cw columns
template <typename T>
int set_axis(lfts_ctx *c, int cw)
{
    AxisSet<T> ax;
    if (!axis_kernels(c->mx, c->my, c->mz, cw, &ax)) return LFTS_ERR_UNSUPPORTED;
    int rc = set_smem(ax.y);
    for (int m = 0; m < kAxisModes && !rc; m++) {
        rc = set_smem(ax.x[m]);
        if (!rc) rc = set_smem(ax.z[m]);
        if (!rc) rc = set_smem(ax.plane[m]);
    }
    if (!rc) axis_of<T>(c) = ax;
    return rc;
}

template <typename T>
int upload_tables(lfts_ctx *c, void **tw, void **gt)
{
    const int m[3] = {c->mx, c->my, c->mz};
    for (int d = 0; d < 3; d++) {
        std::vector<cpx<T>> t(m[d]);
        for (int k = 0; k < m[d]; k++) {
            long double a = -(long double)kTwoPi * (long double)k / (long double)m[d];
            t[k].x = (T)(double)cosl(a);
            t[k].y = (T)(double)sinl(a);
        }
        CK(cudaMalloc(&tw[d], sizeof(cpx<T>) * m[d]));
        CK(cudaMemcpy(tw[d], t.data(), sizeof(cpx<T>) * m[d], cudaMemcpyHostToDevice));
    }
    if (!gt) return LFTS_OK;
    // g = exp(-(2 pi)^2 (kx^2/Lx^2 + ky^2/Ly^2 + kz^2/Lz^2)/(6N)) / M, factorised;
    // over each axis's signed wavenumbers, 1/M shared out by axis_scale
    const int sx = axis_scale(c->mx), sy = axis_scale(c->my);
    const double share[3] = {(double)sx, (double)sy, (double)c->M / (sx * sy)};
    for (int d = 0; d < 3; d++) {
        std::vector<T> g(m[d]);
        for (int K = 0; K < m[d]; K++) {
            const int k = signed_k(K, m[d]);
            const double ksq = (double)k * k / (c->p.L[d] * c->p.L[d]);
            g[K] = (T)(std::exp(-kTwoPi * kTwoPi * ksq / (6.0 * c->N)) / share[d]);
        }
        CK(cudaMalloc(&gt[d], sizeof(T) * m[d]));
        CK(cudaMemcpy(gt[d], g.data(), sizeof(T) * m[d], cudaMemcpyHostToDevice));
    }
    return LFTS_OK;
}

inline dim3 stream_grid(const lfts_ctx *c) { return dim3(c->red_blocks); }
// element-wise passes with no cross-block reduction (the Anderson w+ update,
// the Langevin update): a full wave of 256-thread CTAs, so more loads are in
// flight per SM
inline dim3 update_grid(const lfts_ctx *c) { return dim3(c->sms * 8); }

// ---- contour chain ----------------------------------------------------------
template <typename T>
AxisArgs<T> axis_args(lfts_ctx *c)
{
    AxisArgs<T> a{};
    a.S = static_cast<T *>(c->field);
    a.twx = static_cast<const cpx<T> *>(c->tw[0]);
    a.twy = static_cast<const cpx<T> *>(c->tw[1]);
    a.twz = static_cast<const cpx<T> *>(c->tw[2]);
    a.gx = static_cast<const T *>(c->gtab[0]);
    a.gy = static_cast<const T *>(c->gtab[1]);
    a.gz = static_cast<const T *>(c->gtab[2]);
    a.mx = c->mx;
    a.my = c->my;
    a.mz = c->mz;
    a.M = c->M;
    a.w = c->w;
    a.Nd = (double)c->N;
    a.h = static_cast<const T *>(c->q);  // slot 1
    a.qpart = c->qpart;
    a.ticket = c->ticket;
    a.Qd = c->Qd;
    return a;
}

// Chain kernels go out with programmatic stream serialisation (see pdl_wait in
// fft_kernels.cuh): each may be scheduled while its predecessor drains.
template <typename K, typename A>
void launch_pdl(lfts_ctx *c, K kernel, dim3 grid, int nt, size_t smem, const A &args, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(nt);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = c->use_pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args);
    c->launches++;
}

// The kernels over x lines and over yz planes (one kernel, or z and y lines
// apart), of the chains from a.cbase on: all of them, or `chains` (FP64)
template <typename T>
void launch_x(lfts_ctx *c, int mode, const AxisArgs<T> &a, int chains, cudaStream_t st)
{
    const AxisFn<T> &f = axis_of<T>(c).x[mode];
    const int ncol = c->my * c->mz / kChains<T>;
    launch_pdl(c, f.fn, dim3((ncol + f.per - 1) / f.per, 1, chains), f.nt, f.smem, a, st);
}

// y lines on their own, for the meshes without plane kernels
template <typename T>
void launch_y(lfts_ctx *c, const AxisArgs<T> &a, int chains, cudaStream_t st)
{
    const AxisSet<T> &ax = axis_of<T>(c);
    if (ax.planes) return;
    const int ncol = c->mz / kChains<T>;
    launch_pdl(c, ax.y.fn, dim3((ncol + ax.y.per - 1) / ax.y.per, c->mx, chains), ax.y.nt, ax.y.smem, a, st);
}

// what follows h in a yz kernel's mode ends with the z convolution only where
// the y lines have a kernel of their own: launch_y comes before and after it
template <typename T>
void launch_yz(lfts_ctx *c, int mode, const AxisArgs<T> &a, int chains, cudaStream_t st)
{
    const AxisSet<T> &ax = axis_of<T>(c);
    if (ax.planes) {
        const AxisFn<T> &f = ax.plane[mode];
        launch_pdl(c, f.fn, dim3(c->mx, 1, chains), f.nt, f.smem, a, st);
        return;
    }
    const AxisFn<T> &f = ax.z[mode];
    const int nlines = c->mx * c->my / kChains<T>;
    launch_pdl(c, f.fn, dim3((nlines + f.per - 1) / f.per, 1, chains), f.nt, f.smem, a, st);
}

inline int hsel_chain0(const lfts_ctx *c, int i) { return i < c->NA ? 0 : 1; }  // src/step.cc:53-57
inline int hsel_chain1(const lfts_ctx *c, int i) { return i < c->NB ? 1 : 0; }  // src/step.cc:60-64

template <typename T>
void enqueue_chain_launches(lfts_ctx *c);

// The chain's launches have fixed arguments for the life of the context, so
// they are captured once into a CUDA graph (programmatic-launch edges
// included) and replayed: one launch per calc_concs instead of ~2N.
template <typename T>
void enqueue_chain(lfts_ctx *c)
{
    if (!c->use_graph) {
        enqueue_chain_launches<T>(c);
        return;
    }
    if (!c->chain_exec) {
        const long long before = c->launches;
        cudaError_t e = cudaStreamBeginCapture(c->st, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            enqueue_chain_launches<T>(c);
            cudaGraph_t g = nullptr;
            e = cudaStreamEndCapture(c->st, &g);
            if (e == cudaSuccess && g) e = cudaGraphInstantiate(&c->chain_exec, g, 0);
            if (e == cudaSuccess && c->chain_exec) {
                c->chain_graph = g;
                c->chain_kernels = c->launches - before;
                // upload before the first replay and let both streams drain
                e = cudaGraphUpload(c->chain_exec, c->st);
                if (e == cudaSuccess) e = cudaStreamSynchronize(c->st);
                if (e == cudaSuccess) e = cudaStreamSynchronize(c->st1);
            } else {
                if (g) cudaGraphDestroy(g);
                c->chain_exec = nullptr;
            }
        }
        if (e != cudaSuccess) cuda_fail(e, "chain graph capture");
        c->launches = before;
        cudaGetLastError();  // a failed capture falls back to direct launches below
        if (!c->chain_exec) {
            c->use_graph = false;
            enqueue_chain_launches<T>(c);
            return;
        }
    }
    cudaError_t e = cudaGraphLaunch(c->chain_exec, c->st);
    if (e != cudaSuccess) {
        cuda_fail(e, "cudaGraphLaunch(chain)");
        fprintf(stderr, "lfts: %s\n", g_last_error.c_str());
    }
    c->launches += c->chain_kernels;
}

// ---- FP32-mixed chain by 3-D transforms ---------------------------------------
// What a context runs once lfts_set_tiles has been called on it, and what the
// ensemble's replicas run (lfts_ensemble.cu): fft_packed.cuh, fft_plane3.cuh.
PlaneArgs<float> plane_args(lfts_ctx *c)
{
    PlaneArgs<float> a{};
    a.w = c->w;
    a.spec = static_cast<cpx<float> *>(c->field);
    a.twy = static_cast<const cpx<float> *>(c->tw[1]);
    a.twz = static_cast<const cpx<float> *>(c->tw[2]);
    a.qpart = c->qpart;
    a.Nd = (double)c->N;
    a.gx = static_cast<const float *>(c->gtab[0]);
    a.gy = static_cast<const float *>(c->gtab[1]);
    a.gz = static_cast<const float *>(c->gtab[2]);
    return a;
}

PencilArgs<float> pencil_args(lfts_ctx *c)
{
    PencilArgs<float> a{};
    a.spec = static_cast<cpx<float> *>(c->field);
    a.twx = static_cast<const cpx<float> *>(c->tw[0]);
    a.gx = static_cast<const float *>(c->gtab[0]);
    a.gy = static_cast<const float *>(c->gtab[1]);
    a.gz = static_cast<const float *>(c->gtab[2]);
    a.ncol = c->my * c->mz;
    a.KZ = c->mz;
    a.w = c->w;
    a.h = static_cast<const float *>(c->q);  // slot 1: the (hA, hB) pairs
    a.M = c->M;
    a.Nd = (double)c->N;
    return a;
}

void launch_plane(lfts_ctx *c, int mode, const PlaneArgs<float> &a)
{
    if (mode == PLANE_G && c->plane_split > 1) {
        launch_pdl(c, c->psplit.fn, dim3(c->mx * c->psplit.cl), c->psplit.nt, c->psplit.smem, a, c->st);
        return;
    }
    const int extra = mode == PLANE_G ? a.pf_ctas : 0;
    launch_pdl(c, c->pl32.fn[mode], dim3(c->mx + extra), c->pl32.nt, c->pl32.smem, a, c->st);
}

void launch_pencil(lfts_ctx *c, int mode, const PencilArgs<float> &a)
{
    launch_pdl(c, c->pe32.fn[mode], dim3((a.ncol + c->pe32.cw - 1) / c->pe32.cw), c->pe32.nt, c->pe32.smem, a, c->st);
}

void enqueue_transform_chain(lfts_ctx *c)
{
    float *q = static_cast<float *>(c->q);
    const long long M = c->M;
    PlaneArgs<float> a = plane_args(c);
    PencilArgs<float> pa = pencil_args(c);
    if (c->xh_chain) {
        // One step is q_{i+1} = h . F^-1[g . F[q_i]].  g is even in every
        // wavenumber, so F^-1[g F[q]] = F[g F^-1[q]]; with D_i = F_x^-1[q_i]
        // in the spectrum buffer a step is
        //   yz-plane (PLANE_G):  E_i = F_yz[g . F_yz^-1[D_i]]  (the STEP flow, g for h)
        //   x-pencil (PENCIL_H): q_{i+1} = h . F_x[E_i], stored; D_{i+1} = F_x^-1[q_{i+1}]
        // which puts the h loads and q stores in the pencil's several CTAs
        // per SM instead of the plane kernel's one.
        PencilArgs<float> pi = pa;
        pi.qout = q;  // slot 1 = (hA, hB)
        launch_pencil(c, PENCIL_INIT_W, pi);
        // With phi in the chain, the concentration sums are formed as the
        // slots are made: slot i+1 = (q_{i+1}, q^_{N-i}) pairs with slot
        // N-i = (q_{N-i}, q^_{i+1}).  From the middle of the chain on that
        // partner is already stored, so the pencil adds the two products
        // into acc and slot i+1 need not be stored (except slot N, for Q);
        // the middle slot of an odd chain pairs with itself.
        const bool acc = c->phi_in_chain;
        bool first_acc = true;
        for (int i = 1; i < c->N; i++) {
            PlaneArgs<float> ag = a;
            if (acc && c->N - i < i + 1) {
                ag.pf = q + (long long)(c->N - i - 1) * 2 * M;  // the partner slot
                if (c->plane_split == 1) ag.pf_ctas = c->pf_ctas;
            }
            launch_plane(c, PLANE_G, ag);
            PencilArgs<float> ph = pa;
            ph.qout = q + (long long)i * 2 * M;  // slot i+1
            ph.hsel0 = hsel_chain0(c, i);
            ph.hsel1 = hsel_chain1(c, i);
            const int p = c->N - i;  // partner slot
            if (!acc || p > i + 1) {
                launch_pencil(c, i + 1 < c->N ? PENCIL_H : PENCIL_H_LAST, ph);
                continue;
            }
            ph.partner = p < i + 1 ? q + (long long)(p - 1) * 2 * M : nullptr;
            ph.acc = static_cast<float *>(c->acc);
            ph.acc_init = first_acc ? 1 : 0;
            ph.a_is_A = i + 1 <= c->NA;
            ph.b_is_A = p <= c->NA;
            first_acc = false;
            launch_pencil(c, i + 1 < c->N ? PENCIL_HA : PENCIL_HA_LAST, ph);
        }
        plane_q_sums_kernel<<<c->mx, 256, 0, c->st>>>(
            reinterpret_cast<const float2 *>(q + (long long)(c->N - 1) * 2 * M), (long long)c->my * c->mz,
            c->qpart);
        q_finalize_kernel<<<1, 256, 0, c->st>>>(c->qpart, c->mx, M, c->Qd);
        c->launches += 2;
        return;
    }
    a.qout = q;  // slot 1 = [hA | hB]
    launch_plane(c, PLANE_INIT_W, a);
    a.h = q;
    for (int i = 1; i < c->N; i++) {
        launch_pencil(c, PENCIL_CONV, pa);
        a.qout = q + (long long)i * 2 * M;  // slot i+1
        a.hsel0 = hsel_chain0(c, i);
        a.hsel1 = hsel_chain1(c, i);
        launch_plane(c, i + 1 < c->N ? PLANE_STEP : PLANE_LAST, a);
    }
    q_finalize_kernel<<<1, 256, 0, c->st>>>(c->qpart, c->mx, M, c->Qd);
    c->launches++;
}

// ---- chain one axis at a time -------------------------------------------------
// One contour step of the chains from a.cbase on: step i makes slot i+1 from
// the field that the step before left convolved along z and y (i odd) or
// along x (i even); a holds what the step's kernel needs.
template <typename T>
void launch_step(lfts_ctx *c, int i, int mode, const AxisArgs<T> &a, int chains, cudaStream_t st)
{
    launch_y<T>(c, a, chains, st);
    if (i & 1)
        launch_x<T>(c, mode, a, chains, st);
    else
        launch_yz<T>(c, mode, a, chains, st);
}

// slot i+1 and the h halves of step i (src/step.cc:53-64)
template <typename T>
void set_slot(lfts_ctx *c, AxisArgs<T> &a, int i)
{
    a.q[0] = static_cast<T *>(c->q) + (long long)i * 2 * c->M;
    a.q[1] = a.q[0] + c->M;
    a.hsel[0] = hsel_chain0(c, i);
    a.hsel[1] = hsel_chain1(c, i);
}

// Propagators of both chains for all N monomers, then Q (src/diblock.cc:36-48),
// one axis at a time (axis_conv.cuh): INIT_W leaves h convolved along z and y;
// odd steps end along x and begin the next step there, even steps end and begin
// along z and y.  FP64 chains are independent until the concentrations: with
// two_streams each runs its own launches on its own stream, else both share
// every launch.
template <typename T>
void enqueue_chain_launches(lfts_ctx *c)
{
    if constexpr (kPairs<T>) {
        if (c->transform_chain) {
            enqueue_transform_chain(c);
            return;
        }
    }
    const int N = c->N;
    const AxisArgs<T> a = axis_args<T>(c);
    const bool two = !kPairs<T> && c->two_streams;
    const int chains = two ? 1 : kChains<T>;
    cudaStream_t sc[2] = {c->st, c->st1};
    AxisArgs<T> ac[2] = {a, a};
    ac[1].cbase = 1;
    if (two) {
        cudaEventRecord(c->ev_fork, c->st);
        cudaStreamWaitEvent(c->st1, c->ev_fork, 0);
    }
    for (int k = 0; k <= (two ? 1 : 0); k++) {
        set_slot(c, ac[k], 0);
        launch_yz<T>(c, AX_INIT_W, ac[k], chains, sc[k]);
    }
    if (two) {
        // Each stream's INIT_W writes its own half of h (hA from chain 1, hB from
        // chain 2), and each chain's steps read the other half once i >= NA
        // (chain 1) or i >= NB (chain 2): both halves are complete before either
        // chain's first step.
        for (int k = 0; k < 2; k++) cudaEventRecord(c->ev_h[k], sc[k]);
        for (int k = 0; k < 2; k++) cudaStreamWaitEvent(sc[k], c->ev_h[1 - k], 0);
    }
    bool first_acc = true;
    for (int i = 1; i < N; i++) {
        for (int k = 0; k <= (two ? 1 : 0); k++) {
            set_slot(c, ac[k], i);
            int mode = i + 1 < N ? AX_H : AX_H_LAST;
            // With phi in the chain (FP32), the concentration sums are formed as the
            // slots are made: slot i+1 = (q_{i+1}, q^_{N-i}) pairs with slot
            // N-i = (q_{N-i}, q^_{i+1}).  From the middle of the chain on that
            // partner is already stored, so the kernel adds the two products
            // into acc and slot i+1 need not be stored (except slot N, for Q);
            // the middle slot of an odd chain pairs with itself.
            const int p = N - i;  // partner slot
            if (kPairs<T> && c->phi_in_chain && p <= i + 1) {
                mode = i + 1 < N ? AX_HA : AX_HA_LAST;
                ac[k].partner = p < i + 1 ? static_cast<const T *>(c->q) + (long long)(p - 1) * 2 * c->M : nullptr;
                ac[k].acc = static_cast<T *>(c->acc);
                ac[k].acc_init = first_acc ? 1 : 0;
                ac[k].a_is_A = i + 1 <= c->NA;
                ac[k].b_is_A = p <= c->NA;
                first_acc = false;
            }
            launch_step<T>(c, i, mode, ac[k], chains, sc[k]);
        }
    }
    if (two) {
        cudaEventRecord(c->ev_join, c->st1);
        cudaStreamWaitEvent(c->st, c->ev_join, 0);
    }
}

// phi from the stored slots, and with Dh0 the residual and its dot products
template <typename T>
void launch_concs(lfts_ctx *c, void *Dh0, int nh, const HistPtrs &hist)
{
    auto *fn = conc_slices<T>(c->M, c->N, c->red_blocks) > 1 ? concentrations_kernel<T, true>
                                                             : concentrations_kernel<T, false>;
    fn<<<stream_grid(c), kRedThreads, 0, c->st>>>(static_cast<const T *>(c->q), c->M, c->N, c->NA, c->w, c->w + 2 * c->M,
                                                  c->w + 3 * c->M, c->Qd, static_cast<T *>(Dh0), nh, hist, c->partials,
                                                  c->Q_host);
}

template <typename T>
void enqueue_concs(lfts_ctx *c, void *Dh0, int nh, const HistPtrs &hist)
{
    enqueue_chain<T>(c);
    if (c->phi_in_chain)
        concentrations_acc_kernel<<<stream_grid(c), kRedThreads, 0, c->st>>>(
            static_cast<const float *>(c->acc), static_cast<const float *>(c->q), c->M, c->N, c->w + 2 * c->M,
            c->w + 3 * c->M, c->Qd, static_cast<float *>(Dh0), nh, hist, c->partials, c->Q_host);
    else
        launch_concs<T>(c, Dh0, nh, hist);
    c->launches++;
    if (Dh0) {
        reduce_partials_kernel<<<nh + 1, 256, 0, c->st>>>(c->partials, c->red_blocks, nh + 1, c->red_host);
        c->launches++;
    }
}

void enqueue_chain_any(lfts_ctx *c)
{
    if (c->prec == LFTS_FP64)
        enqueue_chain<double>(c);
    else
        enqueue_chain<float>(c);
}

void enqueue_concs_any(lfts_ctx *c, void *Dh0, int nh, const HistPtrs &hist)
{
    if (c->prec == LFTS_FP64)
        enqueue_concs<double>(c, Dh0, nh, hist);
    else
        enqueue_concs<float>(c, Dh0, nh, hist);
}

// ---- tile choices and their autotuner ------------------------------------------
// The axis-by-axis chain has these free choices, none of which changes what is
// computed (phi_in_chain within the FP32-mixed tolerance, the others not at all):
//   pencil_cw     columns per CTA of the x- and y-line kernels (8, 16, 32)
//   phi_in_chain  FP32-mixed, 96- and 128-point lines: concentration sums formed
//                 in the chain
//   two_streams   FP64: each chain on its own stream, or both chains per launch
// autotune() times the whole chain for every combination on the context's own
// buffers (a tile's cost depends on how it overlaps its neighbours in the chain,
// so it is timed in place) and keeps the fastest, once per precision, mesh, chain
// length within a factor of two (it decides how much of the slots stays in L2) and
// candidates (chain and tiles, which the environment restricts) per process -- the
// reference's analogue is planning its FFTs with FFTW_PATIENT (src/step.cc:15-16).
// lfts_set_tiles on an FP32-mixed context installs the transform chain instead,
// whose choices change how values are rounded:
//   plane_stages  yz-plane transform stages per axis: 3 (fft_plane3.cuh, 64 / 96 /
//                 128 square planes) or 2 (fft_packed.cuh)
//   h_in_pencil   h and the propagator stores in the x-pencil and g in the
//                 yz-plane kernel (96- and 128-point x lines, three-stage planes),
//                 or both in the yz-plane kernel
std::mutex g_tune_mu;
std::map<std::tuple<int, int, int, int, int, std::vector<int>>, lfts_tiles> g_tuned;

// the captured chain and the Anderson-loop graph that holds it (rebuilt on
// the next use with the new tiles)
void drop_chain_graph(lfts_ctx *c)
{
    if (c->chain_exec) cudaGraphExecDestroy(c->chain_exec);
    if (c->chain_graph) cudaGraphDestroy(c->chain_graph);
    c->chain_exec = nullptr;
    c->chain_graph = nullptr;
    if (c->mix_exec) cudaGraphExecDestroy(c->mix_exec);
    if (c->mix_graph) cudaGraphDestroy(c->mix_graph);
    c->mix_exec = nullptr;
    c->mix_graph = nullptr;
    if (c->mix_graph_state == 1) c->mix_graph_state = 0;
}

// FP32-mixed meshes whose default chain is the one by transforms:
//  * what an ensemble runs with one layout of it only, so that a replica computes
//    what a context of its mesh does (16^3 ... 48^3: as replicas' Anderson loops
//    amplify rounding, the ensemble keeps the arithmetic of its chain; 64^3 and 96^3 have
//    several layouts there, and a context equals a replica only with set_tiles anyway);
//  * meshes of up to 16384 points, where a Langevin step with a capped Anderson loop
//    moves by up to 6e-5 with any change of rounding (20^3 3.6e-5, 80 x 12 x 12 5.9e-5;
//    of 52 systems of 17 to 66 thousand points three moved by 2.3e-5 to 4.0e-5, the
//    others by less than 2e-5): they keep their arithmetic too, at 20^3 N = 64 for
//    295 us a calc_concs (308 before the loads were moved ahead) against 174 axis by axis.
bool transform_by_default(const lfts_ctx *c)
{
    auto ens = [](int n) { return n == 16 || n == 24 || n == 32 || n == 48; };
    return c->prec == LFTS_FP32_MIXED &&
           (c->M <= 16384 || (c->my == c->mz && ens(c->my) && (ens(c->mx) || c->mx == 64 || c->mx == 96)));
}

// square planes with a three-stage kernel
bool has_three_stages(const lfts_ctx *c) { return c->my == c->mz && (c->my == 64 || c->my == 96 || c->my == 128); }
bool has_h_in_pencil(const lfts_ctx *c)
{
    return has_three_stages(c) && c->my != 64 && (c->mx == 96 || c->mx == 128);
}
bool has_plane_split(const lfts_ctx *c)
{
    PlaneSplitKernel ps{};
    return has_h_in_pencil(c) && plane_split_kernel(c->my, c->mz, &ps) && ps.cl == 8;
}

// LFTS_XH_CHAIN=0|1 and LFTS_PLANE_SPLIT=8 name a layout of the transform chain: where
// it has that layout, they select that chain
bool transform_by_environment(const lfts_ctx *c)
{
    const char *split = std::getenv("LFTS_PLANE_SPLIT");
    return c->prec == LFTS_FP32_MIXED && ((std::getenv("LFTS_XH_CHAIN") && has_h_in_pencil(c)) ||
                                          (split && std::atoi(split) == 8 && has_plane_split(c)));
}

// the (A, B) concentration sums, FP32 pairs per mesh point
int alloc_sums(lfts_ctx *c)
{
    if (c->acc) return LFTS_OK;
    if (cudaMalloc(&c->acc, sizeof(float) * 2 * (size_t)c->M) == cudaSuccess) return LFTS_OK;
    cudaGetLastError();
    c->acc = nullptr;
    g_last_error = "device allocation of the concentration sums failed";
    return LFTS_ERR_NOMEM;
}

// the axis-by-axis chain with the choices of t (autotune's, so valid)
int apply_axis_tiles(lfts_ctx *c, const lfts_tiles &t)
{
    int rc = t.phi_in_chain ? alloc_sums(c) : LFTS_OK;
    if (!rc) rc = c->prec == LFTS_FP64 ? set_axis<double>(c, t.pencil_cw) : set_axis<float>(c, t.pencil_cw);
    if (rc) return rc;
    c->transform_chain = false;
    c->two_streams = t.two_streams == 1;
    c->phi_in_chain = t.phi_in_chain == 1;
    c->tiles = t;
    drop_chain_graph(c);
    return LFTS_OK;
}

// lfts_set_tiles' choice, validated first; the chain graph is captured anew
int apply_tiles(lfts_ctx *c, const lfts_tiles &t)
{
    if (t.pencil_cw != 8 && t.pencil_cw != 16 && t.pencil_cw != 32) return LFTS_ERR_ARG;
    const int split = t.plane_split == 0 ? 1 : t.plane_split;
    if (split != 1 && split != 8) return LFTS_ERR_ARG;
    lfts_tiles now = t;
    now.plane_split = split;
    if (c->prec == LFTS_FP64) {
        if (t.plane_stages != 2 || t.h_in_pencil != 0 || (t.two_streams != 0 && t.two_streams != 1) ||
            t.phi_in_chain != 0 || split != 1)
            return LFTS_ERR_ARG;
        return apply_axis_tiles(c, now);
    }
    if ((t.plane_stages != 2 && t.plane_stages != 3) || (t.h_in_pencil != 0 && t.h_in_pencil != 1) ||
        t.two_streams != 0 || (t.phi_in_chain != 0 && t.phi_in_chain != 1) || (t.phi_in_chain && !t.h_in_pencil))
        return LFTS_ERR_ARG;
    PlaneKernels<float> pl{};
    const bool ok = t.plane_stages == 3 ? plane3_kernels(c->my, c->mz, &pl) : plane_c_kernels(c->my, c->mz, &pl);
    if (!ok) return LFTS_ERR_UNSUPPORTED;
    PencilKernels<float> pk{};
    if (!pencil_kernels(c->mx, t.pencil_cw, &pk)) return LFTS_ERR_UNSUPPORTED;
    if (t.h_in_pencil && !(pl.fn[PLANE_G] && pk.fn[PENCIL_H])) return LFTS_ERR_UNSUPPORTED;
    if (t.phi_in_chain && !(pk.fn[PENCIL_HA] && pk.fn[PENCIL_HA_LAST])) return LFTS_ERR_UNSUPPORTED;
    PlaneSplitKernel ps{};
    if (split > 1) {
        // the cluster kernel replaces PLANE_G of the three-stage plane
        if (!(t.h_in_pencil && t.plane_stages == 3 && plane_split_kernel(c->my, c->mz, &ps) && ps.cl == split))
            return LFTS_ERR_UNSUPPORTED;
        CK(cudaFuncSetAttribute(ps.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ps.smem));
    }
    if (t.phi_in_chain) {
        int rc = alloc_sums(c);
        if (rc) return rc;
    }
    for (int m = 0; m < kPlaneModes; m++)
        if (pl.fn[m]) CK(cudaFuncSetAttribute(pl.fn[m], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
    for (int m = 0; m < kPencilModes; m++)
        if (pk.fn[m]) CK(cudaFuncSetAttribute(pk.fn[m], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pk.smem));
    c->transform_chain = true;
    c->pl32 = pl;
    c->pe32 = pk;
    c->psplit = ps;
    c->plane_split = split;
    c->xh_chain = t.h_in_pencil == 1;
    c->phi_in_chain = t.phi_in_chain == 1;
    c->tiles = now;
    drop_chain_graph(c);
    return LFTS_OK;
}

// a choice of tile_candidates, for the chain that the context runs by default
int apply_default_tiles(lfts_ctx *c, const lfts_tiles &t)
{
    return c->default_transform ? apply_tiles(c, t) : apply_axis_tiles(c, t);
}

// every combination of the default chain, restricted by the environment
// (LFTS_PENCIL_CW, LFTS_ONE_STREAM, LFTS_PHI_IN_CHAIN, and of the transform chain
// LFTS_XH_CHAIN and LFTS_PLANE_SPLIT, fix one choice each).  For the axis-by-axis
// chain plane_stages and h_in_pencil are those of a transform chain with such tiles.
// The width that was the fastest on none of the cubic meshes is not tried: FP64 32
// (64^3 460 us a call against 423, 128^3 2562 against 2223), FP32 8 (354 against 326,
// 1405 against 1273); it costs a context's first creation as much as the others.
std::vector<lfts_tiles> tile_candidates(const lfts_ctx *c)
{
    std::vector<lfts_tiles> out;
    const char *fcw = std::getenv("LFTS_PENCIL_CW");
    const char *fxh = std::getenv("LFTS_XH_CHAIN");
    const char *fone = std::getenv("LFTS_ONE_STREAM");
    const char *fphi = std::getenv("LFTS_PHI_IN_CHAIN");
    const char *fsplit = std::getenv("LFTS_PLANE_SPLIT");
    const int cw_forced = fcw ? std::atoi(fcw) : 0, split_forced = fsplit ? std::atoi(fsplit) : 0;
    const bool by_env = transform_by_environment(c);
    for (int cw : {8, 16, 32}) {
        if (cw_forced > 0 ? cw != cw_forced : cw == (c->prec == LFTS_FP64 ? 32 : 8)) continue;
        if (c->prec == LFTS_FP64) {
            for (int two : {1, 0}) {
                if (fone && ((fone[0] == '1') == (two == 1))) continue;
                out.push_back({cw, 2, 0, two, 0, 1});
            }
            continue;
        }
        const int xh = has_h_in_pencil(c) && !(fxh && fxh[0] == '0') ? 1 : 0;
        const bool splits = by_env && xh && has_plane_split(c);
        for (int stages : {3, 2}) {
            // two stages where there are three: h in the plane kernel, as asked for
            if (stages == 3 ? !has_three_stages(c) : has_three_stages(c) && !(by_env && !xh)) continue;
            for (int phi : {0, 1}) {
                if (phi && !xh) continue;
                if (fphi && xh && ((fphi[0] != '0') != (phi == 1))) continue;
                for (int split : {1, 8}) {
                    if (split == 8 && !splits) continue;
                    if (splits && split_forced > 0 && split != split_forced) continue;
                    out.push_back({cw, stages, xh, 0, phi, split});
                }
            }
        }
    }
    return out;
}

// the choice used when autotuning is off: the usual tile winners, two FP64
// streams, the separate concentration pass
lfts_tiles default_tiles(const lfts_ctx *c)
{
    std::vector<lfts_tiles> cand = tile_candidates(c);
    const int cw = c->prec == LFTS_FP64 ? kDefaultCwFp64 : kDefaultCwFp32;
    for (const lfts_tiles &t : cand)
        if (t.pencil_cw == cw) return t;  // candidates come best-guess first
    return cand.empty() ? lfts_tiles{cw, 2, 0, c->prec == LFTS_FP64 ? 1 : 0, 0, 1} : cand.front();
}

// a tile choice is timed on whole calc_concs, replayed from the chain's graph as
// calls run it (launched one by one, a chain of 3 us kernels takes the host's time:
// 64^3 FP64 then got 460 us a call where the best choice takes 423)
int time_chain(lfts_ctx *c, cudaEvent_t e0, cudaEvent_t e1, float *ms)
{
    HistPtrs none{};
    enqueue_concs_any(c, nullptr, 0, none);  // warm-up
    CK(cudaEventRecord(e0, c->st));
    for (int r = 0; r < 3; r++) enqueue_concs_any(c, nullptr, 0, none);
    CK(cudaEventRecord(e1, c->st));
    CK(cudaEventSynchronize(e1));
    CK(cudaGetLastError());
    CK(cudaEventElapsedTime(ms, e0, e1));
    return LFTS_OK;
}

int tune_tiles(lfts_ctx *c, lfts_tiles *best)
{
    const long long launches0 = c->launches;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    float best_ms = 0.f;
    bool found = false;
    int rc = LFTS_OK;
    for (const lfts_tiles &t : tile_candidates(c)) {
        if (apply_default_tiles(c, t) != LFTS_OK) continue;
        float ms = 0.f;
        if ((rc = time_chain(c, e0, e1, &ms))) break;
        if (!found || ms < best_ms) {
            best_ms = ms;
            *best = t;
            found = true;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    c->launches = launches0;
    if (rc) return rc;
    CK(cudaStreamSynchronize(c->st));
    CK(cudaStreamSynchronize(c->st1));
    return found ? LFTS_OK : LFTS_ERR_UNSUPPORTED;
}

int autotune(lfts_ctx *c)
{
    lfts_tiles t = default_tiles(c);
    const char *e = std::getenv("LFTS_AUTOTUNE");
    if (!(e && e[0] == '0')) {
        std::vector<int> cand;
        for (const lfts_tiles &a : tile_candidates(c))
            cand.insert(cand.end(), {a.pencil_cw, a.plane_stages, a.h_in_pencil, a.two_streams, a.phi_in_chain,
                                     a.plane_split});
        cand.push_back(c->default_transform);
        const auto key = std::make_tuple(c->prec, c->mx, c->my, c->mz, (int)std::log2(c->N), cand);
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tuned.find(key);
        if (it != g_tuned.end()) {
            t = it->second;
        } else {
            int rc = tune_tiles(c, &t);
            if (rc) return rc;
            g_tuned[key] = t;
            // the timed calls left their concentrations: back to a new context's
            CK(cudaMemsetAsync(c->w + 2 * c->M, 0, sizeof(double) * 2 * c->M, c->st));
        }
    }
    return apply_default_tiles(c, t);
}

// One chain on one stream with CUDA events around every contour-step kernel
// (mean duration of a yz-plane STEP and an x-pencil CONV launch, both chains
// per launch), then the production chain timed as a whole (first launch to Q).
int profile_transform_chain(lfts_ctx *c, double *ms_plane, double *ms_pencil, double *ms_chain)
{
    const int n = c->N - 1;
    std::vector<cudaEvent_t> ev(4 * n + 2);
    for (auto &e : ev) CK(cudaEventCreate(&e));
    float *q = static_cast<float *>(c->q);
    const long long M = c->M;
    PlaneArgs<float> a = plane_args(c);
    PencilArgs<float> pa = pencil_args(c);
    // per step j: pencil between ev[4j] and ev[4j+1], plane between ev[4j+2] and ev[4j+3]
    CK(cudaEventRecord(ev[4 * n], c->st));
    if (c->xh_chain) {
        // the chain of enqueue_transform_chain: pencil INIT_W, (N-1) x (plane G, pencil H)
        PencilArgs<float> pi = pa;
        pi.qout = q;
        launch_pencil(c, PENCIL_INIT_W, pi);
        for (int i = 1; i < c->N; i++) {
            const int j = i - 1;
            CK(cudaEventRecord(ev[4 * j + 2], c->st));
            launch_plane(c, PLANE_G, a);
            CK(cudaEventRecord(ev[4 * j + 3], c->st));
            PencilArgs<float> ph = pa;
            ph.qout = q + (long long)i * 2 * M;
            ph.hsel0 = hsel_chain0(c, i);
            ph.hsel1 = hsel_chain1(c, i);
            CK(cudaEventRecord(ev[4 * j], c->st));
            launch_pencil(c, i + 1 < c->N ? PENCIL_H : PENCIL_H_LAST, ph);
            CK(cudaEventRecord(ev[4 * j + 1], c->st));
        }
        plane_q_sums_kernel<<<c->mx, 256, 0, c->st>>>(
            reinterpret_cast<const float2 *>(q + (long long)(c->N - 1) * 2 * M), (long long)c->my * c->mz,
            c->qpart);
    } else {
        a.qout = q;
        launch_plane(c, PLANE_INIT_W, a);
        a.h = q;
        for (int i = 1; i < c->N; i++) {
            const int j = i - 1;
            CK(cudaEventRecord(ev[4 * j], c->st));
            launch_pencil(c, PENCIL_CONV, pa);
            CK(cudaEventRecord(ev[4 * j + 1], c->st));
            a.qout = q + (long long)i * 2 * M;
            a.hsel0 = hsel_chain0(c, i);
            a.hsel1 = hsel_chain1(c, i);
            CK(cudaEventRecord(ev[4 * j + 2], c->st));
            launch_plane(c, i + 1 < c->N ? PLANE_STEP : PLANE_LAST, a);
            CK(cudaEventRecord(ev[4 * j + 3], c->st));
        }
    }
    q_finalize_kernel<<<1, 256, 0, c->st>>>(c->qpart, c->mx, M, c->Qd);
    c->launches += c->xh_chain ? 2 : 1;
    CK(cudaEventRecord(ev[4 * n + 1], c->st));
    CK(cudaEventSynchronize(ev[4 * n + 1]));
    // means over the full-step launches (the last step's short launch left out)
    double pl = 0.0, pe = 0.0;
    int npl = 0, npe = 0;
    for (int j = 0; j < n; j++) {
        float t = 0.f;
        if (j + 1 < n || !c->xh_chain) {
            CK(cudaEventElapsedTime(&t, ev[4 * j], ev[4 * j + 1]));
            pe += t;
            npe++;
        }
        if (j + 1 < n || c->xh_chain) {
            CK(cudaEventElapsedTime(&t, ev[4 * j + 2], ev[4 * j + 3]));
            pl += t;
            npl++;
        }
    }
    // the production chain (both streams, PDL), timed as a whole
    CK(cudaEventRecord(ev[0], c->st));
    enqueue_chain<float>(c);
    CK(cudaEventRecord(ev[1], c->st));
    CK(cudaEventSynchronize(ev[1]));
    float tc = 0.f;
    CK(cudaEventElapsedTime(&tc, ev[0], ev[1]));
    for (auto &e : ev) cudaEventDestroy(e);
    *ms_pencil = npe ? pe / npe : 0.0;
    *ms_plane = npl ? pl / npl : 0.0;
    *ms_chain = tc;
    return LFTS_OK;
}

// The chain on one stream with CUDA events around its launches: mean duration
// per contour step of the kernels over yz planes (y and z lines) and over x
// lines, both chains per launch; then the production chain timed as a whole.
template <typename T>
int profile_chain(lfts_ctx *c, double *ms_plane, double *ms_pencil, double *ms_chain)
{
    const int n = c->N - 1;
    std::vector<cudaEvent_t> ev(3 * n + 2);
    for (auto &e : ev) CK(cudaEventCreate(&e));
    AxisArgs<T> a = axis_args<T>(c);
    set_slot(c, a, 0);
    launch_yz<T>(c, AX_INIT_W, a, kChains<T>, c->st);
    for (int i = 1; i <= n; i++) {
        set_slot(c, a, i);
        const int mode = i < n ? AX_H : AX_H_LAST;
        CK(cudaEventRecord(ev[3 * i - 3], c->st));
        launch_y<T>(c, a, kChains<T>, c->st);
        CK(cudaEventRecord(ev[3 * i - 2], c->st));
        if (i & 1)
            launch_x<T>(c, mode, a, kChains<T>, c->st);
        else
            launch_yz<T>(c, mode, a, kChains<T>, c->st);
        CK(cudaEventRecord(ev[3 * i - 1], c->st));
    }
    CK(cudaEventSynchronize(ev[3 * n - 1]));
    double pl = 0.0, pe = 0.0;
    for (int i = 1; i <= n; i++) {
        float ty = 0.f, t = 0.f;
        if (!axis_of<T>(c).planes) CK(cudaEventElapsedTime(&ty, ev[3 * i - 3], ev[3 * i - 2]));
        CK(cudaEventElapsedTime(&t, ev[3 * i - 2], ev[3 * i - 1]));
        pl += ty + (i & 1 ? 0.f : t);
        pe += i & 1 ? t : 0.f;
    }
    // the production chain (streams, PDL), timed as a whole
    CK(cudaEventRecord(ev[3 * n], c->st));
    enqueue_chain<T>(c);
    CK(cudaEventRecord(ev[3 * n + 1], c->st));
    CK(cudaEventSynchronize(ev[3 * n + 1]));
    float tc = 0.f;
    CK(cudaEventElapsedTime(&tc, ev[3 * n], ev[3 * n + 1]));
    for (auto &e : ev) cudaEventDestroy(e);
    *ms_pencil = pe / n;
    *ms_plane = pl / n;
    *ms_chain = tc;
    return LFTS_OK;
}

int calc_concs_sync(lfts_ctx *c, double *lnQ)
{
    HistPtrs none{};
    enqueue_concs_any(c, nullptr, 0, none);
    CK(cudaGetLastError());
    if (lnQ) {
        CK(cudaStreamSynchronize(c->st));
        *lnQ = c->Q_host[1];
    }
    c->have_concs = true;
    return LFTS_OK;
}

// anderson::mix (src/anderson.cc:24-93) with the history kept as a ring of
// physical buffers addressed through the reference's logical slot numbers:
// the host-driven loop (one round trip per iteration for the dot products and
// the least squares).  anderson_mix below runs the same loop on the device.
int anderson_mix_host(lfts_ctx *c, int maxIter, double errTol, int *k_out)
{
    const int nhMax = kMaxHist;
    const long long M = c->M;
    double err = 1.0;
    int k;
    for (k = 1; k < maxIter && err > errTol; k++) {
        const int nh = (k < nhMax + 1) ? k - 1 : nhMax;
        HistPtrs Dhp{}, whp{};
        for (int m = 1; m <= nh; m++) {
            Dhp.p[m - 1] = c->Dh[c->phys[m]];
            whp.p[m - 1] = c->wh[c->phys[m]];
        }
        void *Dh0 = c->Dh[c->cur];
        enqueue_concs_any(c, Dh0, nh, Dhp);
        CK(cudaStreamSynchronize(c->st));
        const double S1 = c->red_host[0];
        err = std::pow(S1 / (double)M, 0.5);
        if (!std::isfinite(err)) {
            // stop before w+ is updated with it; k_out is what the reference's
            // loop would return (NaN > tol ends it after this iteration)
            g_last_error = "NaN or infinite Anderson residual (non-finite fields or concentrations)";
            c->mix_calls++;
            if (k_out) *k_out = k + 1;
            return LFTS_ERR_NONFINITE;
        }
        const double lambda = 1.0 - std::pow(0.9, double(k));
        for (int m = 0; m <= nh; m++) c->DD[0][m] = c->red_host[m];

        Coefs C{};
        int simple = 1;
        if (k >= 2) {
            simple = 0;
            std::vector<double> U((size_t)nh * nh), V(nh);
            for (int m = 1; m <= nh; m++) {
                V[m - 1] = c->DD[0][0] - c->DD[0][m];
                for (int n = 1; n <= m; n++) {
                    const double u = c->DD[0][0] - c->DD[0][m] - c->DD[0][n] + c->DD[n][m];
                    U[(m - 1) * nh + n - 1] = u;
                    U[(n - 1) * nh + m - 1] = u;
                }
            }
            if (!lu_solve(U, V, C.c, nh)) {
                g_last_error = "Anderson least-squares matrix is singular";
                return LFTS_ERR_SINGULAR;
            }
        }
        if (c->prec == LFTS_FP64)
            anderson_update_kernel<double><<<update_grid(c), 256, 0, c->st>>>(
                c->w + M, static_cast<double *>(c->wh[c->cur]), static_cast<const double *>(Dh0), M, lambda, nh,
                simple, Dhp, whp, C);
        else
            anderson_update_kernel<float><<<update_grid(c), 256, 0, c->st>>>(
                c->w + M, static_cast<float *>(c->wh[c->cur]), static_cast<const float *>(Dh0), M, lambda, nh,
                simple, Dhp, whp, C);
        c->launches++;
        CK(cudaGetLastError());

        // the current field and deviation become history slot n (src/anderson.cc:82-89)
        const int n = 1 + (k - 1) % nhMax;
        const int evicted = c->phys[n];
        c->phys[n] = c->cur;
        c->cur = evicted;
        c->DD[n][n] = c->DD[0][0];
        for (int m = 1; m < n; m++) c->DD[m][n] = c->DD[0][m];
        for (int m = n + 1; m <= nh; m++) c->DD[n][m] = c->DD[0][m];
        c->mix_iters++;
    }
    c->mix_calls++;
    if (k_out) *k_out = k;
    c->have_concs = true;
    if (err > errTol) {  // the loop ended at maxIter
        g_last_error = "Anderson mixing stopped at maxIter with the error above the tolerance";
        return LFTS_ERR_NOTCONV;
    }
    return LFTS_OK;
}

// ---- the Anderson loop on the device ---------------------------------------------
// One graph per context: begin -> WHILE { contour chain (the chain's own
// launches, programmatic edges included), concentrations + dot products,
// reduce + least squares (one warp, the host LU's operation order), w+
// update, control }.  Bit for bit what anderson_mix_host computes; the host
// sees the loop once per mix (state in, state out) instead of once per
// iteration.
template <typename T>
int capture_mix_graph(lfts_ctx *c, cudaGraph_t *g_out)
{
    MixState *S = static_cast<MixState *>(c->d_mix);
    cudaGraph_t g = nullptr;
    CK(cudaGraphCreate(&g, 0));
    auto fail = [&](cudaError_t e, const char *what) {
        cudaGraphDestroy(g);
        cudaGetLastError();
        return cuda_fail(e, what);
    };
    cudaGraphConditionalHandle loop;
    cudaError_t e = cudaGraphConditionalHandleCreate(&loop, g, 1, cudaGraphCondAssignDefault);
    if (e != cudaSuccess) return fail(e, "conditional handle");
    e = cudaStreamBeginCaptureToGraph(c->st, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return fail(e, "mix graph capture");
    mix_begin_kernel<<<1, 32, 0, c->st>>>(S);
    cudaGraph_t cap = nullptr;
    e = cudaStreamEndCapture(c->st, &cap);
    if (e != cudaSuccess) return fail(e, "mix graph capture");
    size_t nn = 1;
    cudaGraphNode_t begin = nullptr;
    e = cudaGraphGetNodes(g, &begin, &nn);
    if (e != cudaSuccess) return fail(e, "mix graph nodes");
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = loop;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t cond = nullptr;
    e = cudaGraphAddNode(&cond, g, &begin, 1, &cp);
    if (e != cudaSuccess) return fail(e, "mix graph WHILE node");
    e = cudaStreamBeginCaptureToGraph(c->st, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                      cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return fail(e, "mix graph body capture");
    const long long launches0 = c->launches;
    enqueue_chain_launches<T>(c);
    if (c->phi_in_chain)
        mix_conc_acc_kernel<<<stream_grid(c), kRedThreads, 0, c->st>>>(S, static_cast<const float *>(c->acc),
                                                                        static_cast<const float *>(c->q), c->N, c->Qd);
    else
        mix_conc_kernel<T><<<stream_grid(c), kRedThreads, 0, c->st>>>(S, static_cast<const T *>(c->q), c->N, c->NA,
                                                                        c->Qd);
    mix_solve_kernel<<<1, 256, 0, c->st>>>(S);
    mix_update_kernel<T><<<update_grid(c), 256, 0, c->st>>>(S);
    mix_control_kernel<<<1, 32, 0, c->st>>>(S, loop);
    c->mix_body_kernels = c->launches - launches0 + 4;
    c->launches = launches0;
    e = cudaStreamEndCapture(c->st, &cap);
    if (e != cudaSuccess) return fail(e, "mix graph body capture");
    *g_out = g;
    return LFTS_OK;
}

// builds the graph (with the chain's programmatic edges; without them if the
// body refuses them); on failure the context keeps the host loop
int ensure_mix_graph(lfts_ctx *c, int maxIter)
{
    if (c->mix_graph_state < 0) return LFTS_ERR_UNSUPPORTED;
    if (!c->d_mix) CK(cudaMalloc(&c->d_mix, sizeof(MixState)));
    if (maxIter + 2 > c->lambda_cap) {
        // lambda_k = 1 - 0.9^k (src/anderson.cc:44), host pow as in anderson_mix_host
        const int cap = std::max(maxIter + 2, 256);
        std::vector<double> lam(cap);
        for (int k = 0; k < cap; k++) lam[k] = 1.0 - std::pow(0.9, double(k));
        cudaFree(c->d_lambda);
        c->d_lambda = nullptr;
        CK(cudaMalloc(&c->d_lambda, sizeof(double) * cap));
        CK(cudaMemcpy(c->d_lambda, lam.data(), sizeof(double) * cap, cudaMemcpyHostToDevice));
        c->lambda_cap = cap;
    }
    if (c->mix_graph_state == 1) return LFTS_OK;
    const bool pdl = c->use_pdl;
    int rc = LFTS_ERR_CUDA;
    for (int attempt = 0; attempt < 2 && rc; attempt++) {
        c->use_pdl = pdl && attempt == 0;
        cudaGraph_t g = nullptr;
        rc = c->prec == LFTS_FP64 ? capture_mix_graph<double>(c, &g) : capture_mix_graph<float>(c, &g);
        if (!rc) {
            cudaError_t e = cudaGraphInstantiate(&c->mix_exec, g, 0);
            if (e == cudaSuccess) e = cudaGraphUpload(c->mix_exec, c->st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(c->st);
            if (e != cudaSuccess) {
                if (c->mix_exec) cudaGraphExecDestroy(c->mix_exec);
                c->mix_exec = nullptr;
                cudaGraphDestroy(g);
                cudaGetLastError();
                rc = cuda_fail(e, "mix graph instantiate");
            } else {
                c->mix_graph = g;
                c->mix_pdl = c->use_pdl;
            }
        }
    }
    c->use_pdl = pdl;
    c->mix_graph_state = rc ? -1 : 1;
    if (const char *v = getenv("LFTS_VERBOSE"))
        if (v[0] == '1')
            fprintf(stderr, "lfts: Anderson-loop graph %s%s\n", rc ? "not built: " : "built, chain ",
                    rc ? g_last_error.c_str() : (c->mix_pdl ? "with programmatic edges" : "without programmatic edges"));
    return rc;
}

int anderson_mix(lfts_ctx *c, int maxIter, double errTol, int *k_out)
{
    if (!c->mix_on_device || maxIter < 2 || ensure_mix_graph(c, maxIter) != LFTS_OK)
        return anderson_mix_host(c, maxIter, errTol, k_out);
    MixState h{};
    h.M = c->M;
    h.red_blocks = c->red_blocks;
    h.maxIter = maxIter;
    h.tol = errTol;
    h.w = c->w;
    h.partials = c->partials;
    h.lambda = c->d_lambda;
    for (int i = 0; i < kRedWidth; i++) {
        h.Dh[i] = c->Dh[i];
        h.wh[i] = c->wh[i];
        h.phys[i] = c->phys[i];
    }
    h.cur = c->cur;
    MixState *S = static_cast<MixState *>(c->d_mix);
    CK(cudaMemcpyAsync(S, &h, sizeof(MixState), cudaMemcpyHostToDevice, c->st));
    CK(cudaGraphLaunch(c->mix_exec, c->st));
    CK(cudaMemcpyAsync(&h, S, sizeof(MixState), cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    for (int i = 0; i < kRedWidth; i++) c->phys[i] = h.phys[i];
    c->cur = h.cur;
    std::memcpy(c->DD, h.DD, sizeof(c->DD));
    const bool failed = h.nonfinite || h.singular;
    c->mix_iters += h.iters - 1 - (failed ? 1 : 0);
    c->mix_calls++;
    c->launches += (long long)(h.iters - 1) * c->mix_body_kernels + 1;
    if (h.nonfinite) {
        g_last_error = "NaN or infinite Anderson residual (non-finite fields or concentrations)";
        if (k_out) *k_out = h.iters;
        return LFTS_ERR_NONFINITE;
    }
    if (h.singular) {
        g_last_error = "Anderson least-squares matrix is singular";
        return LFTS_ERR_SINGULAR;
    }
    if (k_out) *k_out = h.iters;
    c->have_concs = true;
    if (h.notconv) {
        g_last_error = "Anderson mixing stopped at maxIter with the error above the tolerance";
        return LFTS_ERR_NOTCONV;
    }
    return LFTS_OK;
}

// ---- structure function -------------------------------------------------------
int sk_sample(lfts_ctx *c)
{
    FwdArgs a{};
    a.src[0][0] = c->w;  // W-
    a.spec = static_cast<cpx<double> *>(c->skspec);
    const bool fp64 = c->prec == LFTS_FP64;
    a.twy = static_cast<const cpx<double> *>(fp64 ? c->tw[1] : c->sktw[1]);
    a.twz = static_cast<const cpx<double> *>(fp64 ? c->tw[2] : c->sktw[2]);
    c->fwd_yz.fn<<<dim3(c->mx, 1), c->fwd_yz.nt, c->fwd_yz.smem, c->st>>>(a);
    PencilArgs<double> pa{};
    pa.spec = a.spec;
    pa.twx = static_cast<const cpx<double> *>(fp64 ? c->tw[0] : c->sktw[0]);
    pa.S = c->S;
    pa.ncol = c->my * c->KZ;
    const int ncol = pa.ncol;
    c->power_x.fn<<<(ncol + c->power_x.cw - 1) / c->power_x.cw, c->power_x.nt, c->power_x.smem, c->st>>>(pa);
    c->launches += 2;
    CK(cudaGetLastError());
    c->nsamples++;
    return LFTS_OK;
}

// |K| of every half-spectrum index (src/strFunc.cc:80-103) and bin tables
int sk_prepare_bins(lfts_ctx *c, double dK)
{
    const int m[3] = {c->mx, c->my, c->mz};
    const double *L = c->p.L;
    const long long Mk = c->Mk;
    std::vector<double> K(Mk);
    std::vector<int> wt(Mk, 2), P(Mk);
    for (int k0 = -(m[0] - 1) / 2; k0 <= m[0] / 2; k0++) {
        const int K0 = (k0 < 0) ? (k0 + m[0]) : k0;
        const double kx_sq = k0 * k0 / (L[0] * L[0]);
        for (int k1 = -(m[1] - 1) / 2; k1 <= m[1] / 2; k1++) {
            const int K1 = (k1 < 0) ? (k1 + m[1]) : k1;
            const double ky_sq = k1 * k1 / (L[1] * L[1]);
            for (int k2 = 0; k2 <= m[2] / 2; k2++) {
                const double kz_sq = k2 * k2 / (L[2] * L[2]);
                const long long k = k2 + (long long)(m[2] / 2 + 1) * (K1 + (long long)m[1] * K0);
                K[k] = kTwoPi * std::pow(kx_sq + ky_sq + kz_sq, 0.5);
                if (k2 == 0 || k2 == m[2] / 2) wt[k] = 1;
            }
        }
    }
    std::iota(P.begin(), P.end(), 0);
    std::stable_sort(P.begin(), P.end(), [&](int i, int j) { return K[i] < K[j]; });
    std::vector<int> bins;
    c->sk_K.clear();
    bins.push_back(0);
    for (long long k = 0; k < Mk; k++) {
        if (k == Mk - 1 || std::fabs(K[P[k + 1]] - K[P[k]]) > dK) {
            bins.push_back((int)k + 1);
            c->sk_K.push_back(K[P[k]]);
        }
    }
    cudaFree(c->sk_order);
    cudaFree(c->sk_wt);
    cudaFree(c->sk_bins);
    cudaFree(c->sk_out);
    c->sk_nbins = (int)bins.size() - 1;
    CK(cudaMalloc(&c->sk_order, sizeof(int) * Mk));
    CK(cudaMalloc(&c->sk_wt, sizeof(int) * Mk));
    CK(cudaMalloc(&c->sk_bins, sizeof(int) * bins.size()));
    CK(cudaMalloc(&c->sk_out, sizeof(double) * c->sk_nbins));
    CK(cudaMemcpy(c->sk_order, P.data(), sizeof(int) * Mk, cudaMemcpyHostToDevice));
    CK(cudaMemcpy(c->sk_wt, wt.data(), sizeof(int) * Mk, cudaMemcpyHostToDevice));
    CK(cudaMemcpy(c->sk_bins, bins.data(), sizeof(int) * bins.size(), cudaMemcpyHostToDevice));
    c->sk_dK = dK;
    return LFTS_OK;
}

int ctx_alloc(lfts_ctx *c)
{
    const long long M = c->M;
    CK(cudaMalloc(&c->w, sizeof(double) * 4 * M));
    CK(cudaMemset(c->w, 0, sizeof(double) * 4 * M));
    CK(cudaMalloc(&c->q, c->tsize * 2 * M * (size_t)c->N));
    CK(cudaMalloc(&c->field, c->tsize * 2 * 2 * (size_t)c->mx * c->my * c->KZ));
    CK(cudaMalloc(&c->qpart, sizeof(double) * kMaxQparts));
    CK(cudaMalloc(&c->ticket, sizeof(unsigned)));
    CK(cudaMemset(c->ticket, 0, sizeof(unsigned)));
    CK(cudaMalloc(&c->Qd, sizeof(double) * 2));
    CK(cudaMalloc(&c->partials, sizeof(double) * kRedWidth * c->red_blocks));
    CK(cudaMallocHost(&c->red_host, sizeof(double) * (kRedWidth + 2)));
    c->Q_host = c->red_host + kRedWidth;
    for (int i = 0; i < 2; i++) {
        CK(cudaMalloc(&c->eta[i], sizeof(double) * M));
        CK(cudaMemset(c->eta[i], 0, sizeof(double) * M));
    }
    for (int i = 0; i < kRedWidth; i++) {
        CK(cudaMalloc(&c->Dh[i], c->tsize * M));
        CK(cudaMalloc(&c->wh[i], c->tsize * M));
        CK(cudaMemset(c->Dh[i], 0, c->tsize * M));
        CK(cudaMemset(c->wh[i], 0, c->tsize * M));
    }
    // logical slots 1..10 -> buffers 1..10, buffer 0 is the first current one
    for (int i = 0; i < kRedWidth; i++) c->phys[i] = i;
    c->cur = 0;
    CK(cudaMalloc(&c->S, sizeof(double) * c->Mk));
    CK(cudaMemset(c->S, 0, sizeof(double) * c->Mk));
    if (c->prec == LFTS_FP64) {
        c->skspec = c->field;
    } else {
        CK(cudaMalloc(&c->skspec, sizeof(cpx<double>) * (size_t)c->Mk));
        c->sk_own_spec = true;
    }
    return LFTS_OK;
}

void ctx_free(lfts_ctx *c)
{
    if (c->st) cudaStreamSynchronize(c->st);
    cudaFree(c->w);
    cudaFree(c->q);
    cudaFree(c->field);
    for (int d = 0; d < 3; d++) {
        cudaFree(c->tw[d]);
        cudaFree(c->gtab[d]);
        cudaFree(c->sktw[d]);
    }
    cudaFree(c->qpart);
    cudaFree(c->ticket);
    cudaFree(c->Qd);
    cudaFree(c->partials);
    if (c->red_host) cudaFreeHost(c->red_host);
    for (int i = 0; i < 2; i++) cudaFree(c->eta[i]);
    for (int i = 0; i < kRedWidth; i++) {
        cudaFree(c->Dh[i]);
        cudaFree(c->wh[i]);
    }
    cudaFree(c->S);
    if (c->sk_own_spec) cudaFree(c->skspec);
    cudaFree(c->sk_order);
    cudaFree(c->sk_wt);
    cudaFree(c->sk_bins);
    cudaFree(c->sk_out);
    cudaFree(c->sf_buf);
    cudaFree(c->adj_partial);
    cudaFree(c->adj_buf);
    cudaFree(c->adj_spec);
    drop_chain_graph(c);
    cudaFree(c->acc);
    cudaFree(c->d_mix);
    cudaFree(c->d_lambda);
    if (c->st1) cudaStreamSynchronize(c->st1);
    if (c->ev_fork) cudaEventDestroy(c->ev_fork);
    if (c->ev_join) cudaEventDestroy(c->ev_join);
    for (int k = 0; k < 2; k++)
        if (c->ev_h[k]) cudaEventDestroy(c->ev_h[k]);
    if (c->st1) cudaStreamDestroy(c->st1);
    if (c->st) cudaStreamDestroy(c->st);
}

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev)
    {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard()
    {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

namespace {
template <typename T>
int step_fwd_impl(lfts_ctx *c, const double *q_in, double *q_out, const double *h, int i)
{
    const long long M = c->M;
    double *dq = static_cast<double *>(c->sf_buf);
    double *dout = dq + 2 * M, *dh = dq + 4 * M;
    T *tq = reinterpret_cast<T *>(dh + 2 * M);  // T copies when T != double
    T *th = tq + 2 * M;
    T *tout = th + 2 * M;
    CK(cudaMemcpyAsync(dq, q_in, sizeof(double) * 2 * M, cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(dh, h, sizeof(double) * 2 * M, cudaMemcpyHostToDevice, c->st));
    const T *src = reinterpret_cast<const T *>(dq), *hh = reinterpret_cast<const T *>(dh);
    T *dst = reinterpret_cast<T *>(dout);
    if (sizeof(T) != sizeof(double)) {
        convert_kernel<double, T><<<stream_grid(c), 256, 0, c->st>>>(dq, tq, 2 * M);
        to_pairs_kernel<double, T><<<stream_grid(c), 256, 0, c->st>>>(dh, th, M);  // pairs, as slot 1
        c->launches += 2;
        src = tq;
        hh = th;
        dst = tout;
    }
    AxisArgs<T> a = axis_args<T>(c);
    a.src[0] = src;
    a.src[1] = src + M;
    a.h = hh;
    a.q[0] = dst;
    a.q[1] = dst + M;
    a.hsel[0] = hsel_chain0(c, i);
    a.hsel[1] = hsel_chain1(c, i);
    launch_yz<T>(c, AX_INIT_Q, a, kChains<T>, c->st);
    launch_step<T>(c, 1, AX_OUT, a, kChains<T>, c->st);
    if (sizeof(T) != sizeof(double)) {
        from_pairs_kernel<T, double><<<stream_grid(c), 256, 0, c->st>>>(tout, dout, M);
        c->launches++;
    }
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(q_out, dout, sizeof(double) * 2 * M, cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    return LFTS_OK;
}

}  // namespace

namespace {

// Adjoint terms: forward transforms of q_i (field 0) and q^_{i+1} (field 1) of n
// monomers i, then the k^2-weighted products summed into c->adj_partial.
void adjoint_terms(lfts_ctx *c, const FwdArgs &f, int n)
{
    c->fwd_yz.fn<<<dim3(c->mx, 2, n), c->fwd_yz.nt, c->fwd_yz.smem, c->st>>>(f);
    AdjArgs aa{};
    aa.spec = f.spec;
    aa.twx = static_cast<const cpx<double> *>(c->tw[0]);
    aa.gx = static_cast<const double *>(c->gtab[0]);
    aa.gy = static_cast<const double *>(c->gtab[1]);
    aa.gz = static_cast<const double *>(c->gtab[2]);
    aa.ncol = c->my * c->KZ;
    aa.KZ = c->KZ;
    aa.mx = c->mx;
    aa.my = c->my;
    aa.mz = c->mz;
    aa.partial = c->adj_partial;
    c->adj.fn<<<dim3((aa.ncol + c->adj.cw - 1) / c->adj.cw, n), c->adj.nt, c->adj.smem, c->st>>>(aa);
    c->launches += 2;
}

// Device scratch of lfts_backward: K rows a segment for the recomputed propagators
// (K = 0: all are stored), the spectra of the terms of one launch, their partial
// sums.  The rows come first, since nothing else can stand in for them, and the
// spectra give way to them; without room for spectra of their own one term at a
// time goes through the chain's field, which is free between the chain and the
// next recomputed segments.
int adjoint_scratch(lfts_ctx *c, int nblk, int K, int *segs)
{
    auto try_alloc = [](auto **p, size_t bytes) {
        if (cudaMalloc(reinterpret_cast<void **>(p), bytes) == cudaSuccess) return true;
        cudaGetLastError();
        *p = nullptr;
        return false;
    };
    if (c->adj_buf_slots < *segs * K) {
        const size_t row = sizeof(double) * (size_t)c->M;
        cudaFree(c->adj_buf);
        c->adj_buf = nullptr;
        c->adj_buf_slots = 0;
        if (*segs == 2 && !try_alloc(&c->adj_buf, 2 * K * row)) *segs = 1;
        if (!c->adj_buf && !try_alloc(&c->adj_buf, K * row)) {
            cudaFree(c->adj_spec);
            c->adj_spec = nullptr;
            CK(cudaMalloc(&c->adj_buf, K * row));
        }
        c->adj_buf_slots = *segs * K;
    }
    // terms per launch: about four CTAs per SM of 2 mx planes a term
    const int batch = std::max(1, std::min(kFwdBatch, (4 * c->sms + 2 * c->mx - 1) / (2 * c->mx)));
    if (!c->adj_partial) CK(cudaMalloc(&c->adj_partial, sizeof(double) * 3 * nblk * batch));
    if (!c->adj_spec) try_alloc(&c->adj_spec, sizeof(cpx<double>) * 2 * (size_t)c->Mk * batch);
    c->adj_batch = c->adj_spec ? batch : 1;
    return LFTS_OK;
}

// Terms given one by one, launched c->adj_batch at a time
struct AdjointBatch {
    lfts_ctx *c;
    FwdArgs f{};
    int n = 0;
    explicit AdjointBatch(lfts_ctx *ctx) : c(ctx)
    {
        f.spec = static_cast<cpx<double> *>(c->adj_spec ? c->adj_spec : c->field);
        f.twy = static_cast<const cpx<double> *>(c->tw[1]);
        f.twz = static_cast<const cpx<double> *>(c->tw[2]);
    }
    void add(const double *q_i, const double *qh_ip1)
    {
        f.src[0][n] = q_i;
        f.src[1][n] = qh_ip1;
        if (++n == c->adj_batch) flush();
    }
    void flush()
    {
        if (n) adjoint_terms(c, f, n);
        n = 0;
    }
};

// Propagators of both chains with q stored only at monomers 1, 1+K, 1+2K, ...
// (q^ in full); returns after Q is reduced.
int chain_checkpointed(lfts_ctx *c, int K)
{
    AxisArgs<double> a = axis_args<double>(c);
    set_slot(c, a, 0);
    launch_yz<double>(c, AX_INIT_W, a, 2, c->st);  // slot 1 = [hA | hB]
    for (int i = 1; i < c->N; i++) {
        set_slot(c, a, i);
        if (i % K) a.q[0] = nullptr;
        launch_step<double>(c, i, i + 1 < c->N ? AX_H : AX_H_LAST, a, 2, c->st);
    }
    return LFTS_OK;
}

// Two segments recomputed side by side, as the two FP64 fields of the axis
// kernels: segment s's q_{c0+1} .. q_{c0+n[s]} from its checkpoint q_{c0} (row 0)
// into rows 1 .. n[s], n[0] >= n[1]
void recompute_segments(lfts_ctx *c, const double *const row0[2], double *const rows[2], const int c0[2],
                        const int n[2])
{
    AxisArgs<double> a = axis_args<double>(c);
    const int nseg = n[1] > 0 ? 2 : 1;
    for (int s = 0; s < nseg; s++) a.src[s] = row0[s];
    a.ticket = nullptr;
    launch_yz<double>(c, AX_INIT_Q, a, nseg, c->st);
    for (int j = 1; j <= n[0]; j++) {
        for (int s = 0; s < nseg; s++) {
            a.hsel[s] = hsel_chain0(c, c0[s] + j - 1);  // monomer step i = c0 + j - 1 makes q_{i+1}
            a.q[s] = j <= n[s] ? rows[s] + (long long)j * c->M : nullptr;
        }
        launch_step<double>(c, j, j < n[0] ? AX_H : AX_H_LAST, a, nseg, c->st);
    }
}

}  // namespace

}  // namespace

// =============================================================================
extern "C" {

const char *lfts_version(void) { return "lfts_b200 0.1 (sm_100a)"; }

const char *lfts_status_string(int s)
{
    switch (s) {
        case LFTS_OK: return "ok";
        case LFTS_ERR_ARG: return "invalid argument";
        case LFTS_ERR_UNSUPPORTED: return "mesh size not supported by the FFT kernels";
        case LFTS_ERR_CUDA: return "CUDA error";
        case LFTS_ERR_NOMEM: return "device allocation failed";
        case LFTS_ERR_SINGULAR: return "Anderson least-squares matrix singular";
        case LFTS_ERR_STATE: return "call out of order";
        case LFTS_ERR_NOTCONV: return "Anderson iteration cap reached above the tolerance";
        case LFTS_ERR_NONFINITE: return "non-finite Anderson residual";
        default: return "unknown status";
    }
}

const char *lfts_last_error_string(void) { return g_last_error.c_str(); }

int lfts_mesh_supported(int n) { return fft_length_supported(n) ? 1 : 0; }

int lfts_create(const lfts_params *p, int precision, int device, lfts_ctx **out)
{
    if (!p || !out) return LFTS_ERR_ARG;
    *out = nullptr;
    if (p->N < 2 || p->NA < 0 || p->NA > p->N || p->C <= 0.0 || p->XbN == 0.0) return LFTS_ERR_ARG;
    if (precision != LFTS_FP64 && precision != LFTS_FP32_MIXED) return LFTS_ERR_ARG;
    for (int d = 0; d < 3; d++)
        if (p->m[d] < 1 || !(p->L[d] > 0.0)) return LFTS_ERR_ARG;
    // even my and mz (row pairs, packed Nyquist column) also make M a multiple
    // of 4, which the vectorised concentration pass relies on
    if (!fft_length_supported(p->m[0]) || !plane_pair_supported(p->m[1], p->m[2]) || (p->m[1] % 2) ||
        (p->m[2] % 2)) {
        g_last_error = "mesh not supported: each dimension must be one of the compiled FFT lengths";
        return LFTS_ERR_UNSUPPORTED;
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        g_last_error = "no CUDA device";
        return LFTS_ERR_CUDA;
    }
    DeviceGuard g(device);
    lfts_ctx *c = new lfts_ctx;
    c->p = *p;
    c->prec = precision;
    c->dev = device;
    c->N = p->N;
    c->NA = p->NA;
    c->NB = p->N - p->NA;
    c->mx = p->m[0];
    c->my = p->m[1];
    c->mz = p->m[2];
    c->KZ = c->mz / 2 + 1;
    c->M = (long long)c->mx * c->my * c->mz;
    c->Mk = (long long)c->mx * c->my * c->KZ;
    c->tsize = precision == LFTS_FP64 ? sizeof(double) : sizeof(float);
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) == cudaSuccess) c->sms = prop.multiProcessorCount;
    c->red_blocks = c->sms * 4;
    if (const char *e = getenv("LFTS_NO_PDL")) c->use_pdl = !(e[0] == '1');
    // SMs the one-CTA-per-plane PLANE_G leaves idle take its L2 prefetch of the
    // partner slot (LFTS_PREFETCH_CTAS=0: the plane CTAs issue it themselves).
    // Only for 128 x 128 planes, whose CTA fills an SM's shared memory: at 96 x 96
    // two plane CTAs share an SM and the extra CTAs measured slower
    c->pf_ctas = (c->my == 128 && c->mz == 128 && c->sms > c->mx) ? std::min(c->sms - c->mx, 64) : 0;
    if (const char *e = getenv("LFTS_PREFETCH_CTAS")) c->pf_ctas = std::max(0, std::min(std::atoi(e), c->pf_ctas));
    if (const char *e = getenv("LFTS_ONE_STREAM")) c->two_streams = !(e[0] == '1');
    if (const char *e = getenv("LFTS_NO_GRAPH")) c->use_graph = !(e[0] == '1');
    if (const char *e = getenv("LFTS_DEVICE_MIX")) c->mix_on_device = e[0] == '1';
    if (!c->use_graph) c->mix_on_device = false;
    int rc = LFTS_OK;
    auto fail = [&](int code) {
        ctx_free(c);
        delete c;
        return code;
    };
    if (cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&c->st1, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&c->ev_fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&c->ev_join, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&c->ev_h[0], cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&c->ev_h[1], cudaEventDisableTiming) != cudaSuccess)
        return fail(LFTS_ERR_CUDA);
    if (!fwd_plane_kernel(c->my, c->mz, &c->fwd_yz) || !power_pencil_kernel(c->mx, &c->power_x))
        return fail(LFTS_ERR_UNSUPPORTED);
    if (cudaFuncSetAttribute(c->fwd_yz.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c->fwd_yz.smem) !=
            cudaSuccess ||
        cudaFuncSetAttribute(c->power_x.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c->power_x.smem) !=
            cudaSuccess)
        return fail(LFTS_ERR_CUDA);
    if ((rc = ctx_alloc(c))) return fail(rc == LFTS_ERR_CUDA ? LFTS_ERR_NOMEM : rc);
    if (precision == LFTS_FP64)
        rc = upload_tables<double>(c, c->tw, c->gtab);
    else {
        rc = upload_tables<float>(c, c->tw, c->gtab);
        if (!rc) rc = upload_tables<double>(c, c->sktw, nullptr);
    }
    if (rc) return fail(rc);
    if (precision == LFTS_FP32_MIXED && (rc = set_axis<float>(c, kDefaultCwFp32))) return fail(rc);  // step_fwd
    c->default_transform = transform_by_default(c) || transform_by_environment(c);
    if ((rc = autotune(c))) return fail(rc);
    c->default_tiles = c->tiles;
    *out = c;
    return LFTS_OK;
}

int lfts_destroy(lfts_ctx *c)
{
    if (!c) return LFTS_OK;
    DeviceGuard g(c->dev);
    ctx_free(c);
    delete c;
    return LFTS_OK;
}

int lfts_device_bytes(const lfts_ctx *c, size_t *bytes)
{
    if (!c || !bytes) return LFTS_ERR_ARG;
    const size_t M = c->M;
    size_t b = 4 * M * 8 + c->tsize * 2 * M * c->N + c->tsize * 4 * (size_t)c->mx * c->my * c->KZ;
    b += 2 * M * 8 + 2 * kRedWidth * M * c->tsize + c->Mk * 8;
    if (c->sk_own_spec) b += c->Mk * 16;
    if (c->acc) b += 8 * M;
    *bytes = b;
    return LFTS_OK;
}

int lfts_set_fields(lfts_ctx *c, const double *w_host)
{
    if (!c || !w_host) return LFTS_ERR_ARG;
    DeviceGuard g(c->dev);
    CK(cudaMemcpyAsync(c->w, w_host, sizeof(double) * 2 * c->M, cudaMemcpyHostToDevice, c->st));
    CK(cudaStreamSynchronize(c->st));
    c->fields_set = true;
    return LFTS_OK;
}

int lfts_get_fields(lfts_ctx *c, double *w_host)
{
    if (!c || !w_host) return LFTS_ERR_ARG;
    DeviceGuard g(c->dev);
    CK(cudaMemcpyAsync(w_host, c->w, sizeof(double) * 4 * c->M, cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    return LFTS_OK;
}

int lfts_fields_device(lfts_ctx *c, double **w_dev)
{
    if (!c || !w_dev) return LFTS_ERR_ARG;
    *w_dev = c->w;
    c->fields_set = true;  // the caller may fill the array directly
    return LFTS_OK;
}

int lfts_calc_concs(lfts_ctx *c, double *lnQ)
{
    if (!c) return LFTS_ERR_ARG;
    if (!c->fields_set) return LFTS_ERR_STATE;
    DeviceGuard g(c->dev);
    return calc_concs_sync(c, lnQ);
}

int lfts_anderson_mix(lfts_ctx *c, int maxIter, double errTol, int *k_out)
{
    if (!c) return LFTS_ERR_ARG;
    if (!c->fields_set) return LFTS_ERR_STATE;
    DeviceGuard g(c->dev);
    return anderson_mix(c, maxIter, errTol, k_out);
}

int lfts_langevin_init(lfts_ctx *c, const double *noise_prev_host)
{
    if (!c || !noise_prev_host) return LFTS_ERR_ARG;
    DeviceGuard g(c->dev);
    c->eta_prev = 0;
    CK(cudaMemcpyAsync(c->eta[0], noise_prev_host, sizeof(double) * c->M, cudaMemcpyHostToDevice, c->st));
    CK(cudaStreamSynchronize(c->st));
    c->eta_set = true;
    return LFTS_OK;
}

static int langevin_device(lfts_ctx *c, const double *eta_new_dev)
{
    const int nb = 1 - c->eta_prev;
    if (eta_new_dev != c->eta[nb])
        CK(cudaMemcpyAsync(c->eta[nb], eta_new_dev, sizeof(double) * c->M, cudaMemcpyDeviceToDevice, c->st));
    langevin_kernel<<<update_grid(c), 256, 0, c->st>>>(c->w, c->M, c->eta[c->eta_prev], c->eta[nb], c->p.XbN,
                                                       c->p.dt);
    c->launches++;
    CK(cudaGetLastError());
    c->eta_prev = nb;  // the new noise is the next step's previous noise (src/langevin.cc:34-36)
    return LFTS_OK;
}

int lfts_langevin_step(lfts_ctx *c, const double *noise_new_host)
{
    if (!c || !noise_new_host) return LFTS_ERR_ARG;
    if (!c->fields_set || !c->eta_set || !c->have_concs) return LFTS_ERR_STATE;
    DeviceGuard g(c->dev);
    const int nb = 1 - c->eta_prev;
    CK(cudaMemcpyAsync(c->eta[nb], noise_new_host, sizeof(double) * c->M, cudaMemcpyHostToDevice, c->st));
    int rc = langevin_device(c, c->eta[nb]);
    if (rc) return rc;
    CK(cudaStreamSynchronize(c->st));
    return LFTS_OK;
}

int lfts_langevin_step_device(lfts_ctx *c, const double *noise_new_dev)
{
    if (!c || !noise_new_dev) return LFTS_ERR_ARG;
    if (!c->fields_set || !c->eta_set || !c->have_concs) return LFTS_ERR_STATE;
    DeviceGuard g(c->dev);
    return langevin_device(c, noise_new_dev);
}

int lfts_langevin_full_step(lfts_ctx *c, const double *noise_new_dev, int maxIter, double errTol, int *k_out,
                            double *lnQ)
{
    if (!c || !noise_new_dev) return LFTS_ERR_ARG;
    if (!c->fields_set || !c->eta_set || !c->have_concs) return LFTS_ERR_STATE;
    DeviceGuard g(c->dev);
    int rc = langevin_device(c, noise_new_dev);
    if (rc) return rc;
    rc = anderson_mix(c, maxIter, errTol, k_out);
    if (rc && rc != LFTS_ERR_NOTCONV) return rc;
    const int rc2 = calc_concs_sync(c, lnQ);  // the step completes past the cap, as in the reference
    return rc2 ? rc2 : rc;
}

int lfts_sk_sample(lfts_ctx *c)
{
    if (!c) return LFTS_ERR_ARG;
    if (!c->fields_set) return LFTS_ERR_STATE;
    DeviceGuard g(c->dev);
    int rc = sk_sample(c);
    if (rc) return rc;
    CK(cudaStreamSynchronize(c->st));
    return LFTS_OK;
}

int lfts_sk_get(lfts_ctx *c, double *S_host, int *nsamples)
{
    if (!c) return LFTS_ERR_ARG;
    DeviceGuard g(c->dev);
    if (S_host) {
        CK(cudaMemcpyAsync(S_host, c->S, sizeof(double) * c->Mk, cudaMemcpyDeviceToHost, c->st));
        CK(cudaStreamSynchronize(c->st));
    }
    if (nsamples) *nsamples = c->nsamples;
    return LFTS_OK;
}

int lfts_sk_reset(lfts_ctx *c)
{
    if (!c) return LFTS_ERR_ARG;
    DeviceGuard g(c->dev);
    CK(cudaMemsetAsync(c->S, 0, sizeof(double) * c->Mk, c->st));
    CK(cudaStreamSynchronize(c->st));
    c->nsamples = 0;
    return LFTS_OK;
}

int lfts_sk_bin(lfts_ctx *c, double dK, double *K_out, double *S_out, int *nbins)
{
    // with no samples the averages come out NaN, as the reference's division
    // by nsamples_ = 0 does
    if (!c || !K_out || !S_out || !nbins || !(dK >= 0.0)) return LFTS_ERR_ARG;
    DeviceGuard g(c->dev);
    if (dK != c->sk_dK) {
        int rc = sk_prepare_bins(c, dK);
        if (rc) return rc;
    }
    // coeff_ = CV/(chi_b^2 M^2) (src/strFunc.cc:21), with CV = C*V
    const double V = c->p.L[0] * c->p.L[1] * c->p.L[2];
    const double CV = c->p.C * V;
    const double M = (double)c->M;
    const double coeff = CV / (c->p.XbN * c->p.XbN * M * M);
    sk_bin_kernel<<<(c->sk_nbins + 7) / 8, 256, 0, c->st>>>(c->S, c->sk_order, c->sk_wt, c->sk_bins,
                                                               c->sk_nbins, coeff / (double)c->nsamples,
                                                               0.5 / c->p.XbN, c->sk_out);
    c->launches++;
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(S_out, c->sk_out, sizeof(double) * c->sk_nbins, cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    std::memcpy(K_out, c->sk_K.data(), sizeof(double) * c->sk_nbins);
    *nbins = c->sk_nbins;
    return LFTS_OK;
}

int lfts_get_H(lfts_ctx *c, double *H)
{
    if (!c || !H) return LFTS_ERR_ARG;
    if (!c->fields_set) return LFTS_ERR_STATE;
    DeviceGuard g(c->dev);
    int rc = calc_concs_sync(c, nullptr);
    if (rc) return rc;
    h_sums_kernel<<<stream_grid(c), kRedThreads, 0, c->st>>>(c->w, c->M, c->partials);
    reduce_partials_kernel<<<2, 256, 0, c->st>>>(c->partials, c->red_blocks, 2, c->red_host);
    c->launches += 2;
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(c->st));
    const double wp_sum = c->red_host[0], wm2_sum = c->red_host[1], lnQ = c->Q_host[1];
    *H = -lnQ + (wm2_sum / c->p.XbN - wp_sum) / (double)c->M;
    return LFTS_OK;
}

int lfts_step_fwd(lfts_ctx *c, const double *q_in, double *q_out, const double *h, int i)
{
    if (!c || !q_in || !q_out || !h || i < 1 || i >= c->N) return LFTS_ERR_ARG;
    DeviceGuard g(c->dev);
    if (!c->sf_buf) CK(cudaMalloc(&c->sf_buf, sizeof(double) * 6 * c->M + c->tsize * 6 * c->M));
    if (c->prec == LFTS_FP64) return step_fwd_impl<double>(c, q_in, q_out, h, i);
    return step_fwd_impl<float>(c, q_in, q_out, h, i);
}

int lfts_g_lookup(lfts_ctx *c, double *g_host)
{
    if (!c || !g_host) return LFTS_ERR_ARG;
    // the factorised weights the kernels multiply by, expanded to the Mk layout
    const int m[3] = {c->mx, c->my, c->mz};
    std::vector<double> g[3];
    const int n[3] = {c->mx, c->my, c->KZ};
    for (int d = 0; d < 3; d++) {
        g[d].resize(n[d]);
        for (int K = 0; K < n[d]; K++) {
            const int k = (d == 2) ? K : signed_k(K, m[d]);
            const double ksq = (double)k * k / (c->p.L[d] * c->p.L[d]);
            double v = std::exp(-kTwoPi * kTwoPi * ksq / (6.0 * c->N));
            if (d == 2) v /= (double)c->M;
            g[d][K] = (c->prec == LFTS_FP64) ? v : (double)(float)v;
        }
    }
    for (int a = 0; a < c->mx; a++)
        for (int b = 0; b < c->my; b++)
            for (int k = 0; k < c->KZ; k++)
                g_host[((long long)a * c->my + b) * c->KZ + k] = g[0][a] * g[1][b] * g[2][k];
    return LFTS_OK;
}

int lfts_backward(lfts_ctx *c, int ckpt_every, double *dH_dL, double *dH_dXbN, double *H)
{
    if (!c || !dH_dL || ckpt_every < 0) return LFTS_ERR_ARG;
    if (!c->fields_set) return LFTS_ERR_STATE;
    if (c->prec != LFTS_FP64) {
        g_last_error = "the adjoint runs on FP64 contexts";
        return LFTS_ERR_UNSUPPORTED;
    }
    DeviceGuard g(c->dev);
    if (!c->adj.fn && !adjoint_kernel(c->mx, &c->adj)) return LFTS_ERR_UNSUPPORTED;
    CK(cudaFuncSetAttribute(c->adj.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c->adj.smem));
    const long long M = c->M;
    const int nblk = (c->my * c->KZ + c->adj.cw - 1) / c->adj.cw;
    const int K = std::min(ckpt_every, c->N);
    int segs = 1 + K < c->N ? 2 : 1;  // segments side by side; one alone if there is no second or no room
    int rc = adjoint_scratch(c, nblk, K, &segs);
    if (rc) return rc;
    CK(cudaMemsetAsync(c->adj_partial, 0, sizeof(double) * 3 * nblk * c->adj_batch, c->st));
    const int nrows = nblk * c->adj_batch;
    double *q = static_cast<double *>(c->q);
    const int N = c->N;
    // q_i is the first half of slot i, q^_{i+1} the second half of slot N-i
    auto qh = [&](int i1) { return q + (long long)(N - i1) * 2 * M + M; };  // q^_{i1}
    AdjointBatch terms(c);
    if (K == 0) {
        rc = calc_concs_sync(c, nullptr);
        if (rc) return rc;
        for (int i = 1; i < N; i++) terms.add(q + (long long)(i - 1) * 2 * M, qh(i + 1));
    } else {
        chain_checkpointed(c, K);
        // `segs` segments (terms i = c0 .. c0 + n) at a time
        for (int c1 = 1; c1 < N; c1 += segs * K) {
            int c0[2], n[2];
            const double *row0[2];
            double *rows[2];
            for (int s = 0; s < 2; s++) {
                c0[s] = c1 + s * K;
                n[s] = s < segs ? std::min(c0[s] + K - 1, N - 1) - c0[s] : -1;
                row0[s] = q + (long long)(c0[s] - 1) * 2 * M;
                rows[s] = c->adj_buf + (long long)s * K * M;
            }
            if (n[0] > 0) recompute_segments(c, row0, rows, c0, n);
            for (int s = 0; s < 2; s++)
                for (int j = 0; j <= n[s]; j++)
                    terms.add(j ? rows[s] + (long long)j * M : row0[s], qh(c0[s] + j + 1));
            if (K > 1) terms.flush();  // before the rows are written again
        }
        c->have_concs = false;  // phi was not recomputed
    }
    terms.flush();
    h_sums_kernel<<<stream_grid(c), kRedThreads, 0, c->st>>>(c->w, M, c->partials);
    reduce_partials_kernel<<<2, 256, 0, c->st>>>(c->partials, c->red_blocks, 2, c->red_host);
    c->launches += 2;
    CK(cudaGetLastError());
    std::vector<double> part(3 * (size_t)nrows);
    CK(cudaMemcpyAsync(part.data(), c->adj_partial, sizeof(double) * part.size(), cudaMemcpyDeviceToHost, c->st));
    CK(cudaMemcpyAsync(c->Q_host, c->Qd, 2 * sizeof(double), cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    const double wp_sum = c->red_host[0], wm2_sum = c->red_host[1], Q = c->Q_host[0], lnQ = c->Q_host[1];
    double S[3] = {0.0, 0.0, 0.0};
    for (int b = 0; b < nrows; b++)
        for (int d = 0; d < 3; d++) S[d] += part[3 * (size_t)b + d];
    // dH/dL = -(1/Q) dQ/dL, dQ/dL_a = (1/M) 4 pi^2 S_a / (3 N L_a^3)
    for (int d = 0; d < 3; d++) {
        const double L = c->p.L[d];
        dH_dL[d] = -(kTwoPi * kTwoPi * S[d] / (3.0 * N * L * L * L)) / ((double)M * Q);
    }
    const double X = c->p.XbN;
    if (dH_dXbN) *dH_dXbN = -wm2_sum / (X * X * (double)M);
    if (H) *H = -lnQ + (wm2_sum / X - wp_sum) / (double)M;
    return LFTS_OK;
}

void *lfts_stream(lfts_ctx *c) { return c ? (void *)c->st : nullptr; }

int lfts_profile_chain(lfts_ctx *c, double *ms_plane, double *ms_pencil, double *ms_chain)
{
    if (!c || !ms_plane || !ms_pencil || !ms_chain) return LFTS_ERR_ARG;
    if (!c->fields_set) return LFTS_ERR_STATE;
    DeviceGuard g(c->dev);
    CK(cudaStreamSynchronize(c->st));
    if (c->prec == LFTS_FP64) return profile_chain<double>(c, ms_plane, ms_pencil, ms_chain);
    if (c->transform_chain) return profile_transform_chain(c, ms_plane, ms_pencil, ms_chain);
    return profile_chain<float>(c, ms_plane, ms_pencil, ms_chain);
}

int lfts_profile_iteration(lfts_ctx *c, int reps, double *ms_chain, double *ms_concs, double *ms_update)
{
    if (!c || reps < 1 || !ms_chain || !ms_concs || !ms_update) return LFTS_ERR_ARG;
    if (!c->fields_set) return LFTS_ERR_STATE;
    DeviceGuard g(c->dev);
    CK(cudaStreamSynchronize(c->st));
    const long long M = c->M;
    // a full history: every ring buffer in use, as from the 11th iteration on
    HistPtrs Dhp{}, whp{};
    for (int m = 1; m <= kMaxHist; m++) {
        Dhp.p[m - 1] = c->Dh[c->phys[m]];
        whp.p[m - 1] = c->wh[c->phys[m]];
    }
    Coefs zero{};  // lambda = 0 and zero coefficients leave w+ bitwise unchanged
    cudaEvent_t ev[4];
    for (auto &e : ev) CK(cudaEventCreate(&e));
    enqueue_chain_any(c);  // warm
    CK(cudaEventRecord(ev[0], c->st));
    for (int r = 0; r < reps; r++) enqueue_chain_any(c);
    CK(cudaEventRecord(ev[1], c->st));
    for (int r = 0; r < reps; r++) {
        if (c->prec == LFTS_FP64)
            launch_concs<double>(c, c->Dh[c->cur], kMaxHist, Dhp);
        else if (c->phi_in_chain)
            concentrations_acc_kernel<<<stream_grid(c), kRedThreads, 0, c->st>>>(
                static_cast<const float *>(c->acc), static_cast<const float *>(c->q), M, c->N, c->w + 2 * M,
                c->w + 3 * M, c->Qd, static_cast<float *>(c->Dh[c->cur]), kMaxHist, Dhp, c->partials, c->Q_host);
        else
            launch_concs<float>(c, c->Dh[c->cur], kMaxHist, Dhp);
        reduce_partials_kernel<<<kRedWidth, 256, 0, c->st>>>(c->partials, c->red_blocks, kRedWidth, c->red_host);
    }
    CK(cudaEventRecord(ev[2], c->st));
    for (int r = 0; r < reps; r++) {
        if (c->prec == LFTS_FP64)
            anderson_update_kernel<double><<<update_grid(c), 256, 0, c->st>>>(
                c->w + M, static_cast<double *>(c->wh[c->cur]), static_cast<const double *>(c->Dh[c->cur]), M, 0.0,
                kMaxHist, 0, Dhp, whp, zero);
        else
            anderson_update_kernel<float><<<update_grid(c), 256, 0, c->st>>>(
                c->w + M, static_cast<float *>(c->wh[c->cur]), static_cast<const float *>(c->Dh[c->cur]), M, 0.0,
                kMaxHist, 0, Dhp, whp, zero);
    }
    CK(cudaEventRecord(ev[3], c->st));
    CK(cudaEventSynchronize(ev[3]));
    CK(cudaGetLastError());
    float t[3];
    for (int i = 0; i < 3; i++) CK(cudaEventElapsedTime(&t[i], ev[i], ev[i + 1]));
    for (auto &e : ev) cudaEventDestroy(e);
    c->launches += (long long)reps * 3;
    *ms_chain = t[0] / reps;
    *ms_concs = t[1] / reps;
    *ms_update = t[2] / reps;
    return LFTS_OK;
}

int lfts_get_tiles(const lfts_ctx *c, lfts_tiles *out)
{
    if (!c || !out) return LFTS_ERR_ARG;
    *out = c->tiles;
    return LFTS_OK;
}

int lfts_set_tiles(lfts_ctx *c, const lfts_tiles *t)
{
    if (!c || !t) return LFTS_ERR_ARG;
    DeviceGuard g(c->dev);
    CK(cudaStreamSynchronize(c->st));
    CK(cudaStreamSynchronize(c->st1));
    int rc = apply_tiles(c, *t);  // an invalid choice leaves the context as it was
    if (rc) g_last_error = "tile choice not valid for this context's precision and mesh";
    return rc;
}

int lfts_reset_tiles(lfts_ctx *c)
{
    if (!c) return LFTS_ERR_ARG;
    DeviceGuard g(c->dev);
    CK(cudaStreamSynchronize(c->st));
    CK(cudaStreamSynchronize(c->st1));
    return apply_default_tiles(c, c->default_tiles);
}

int lfts_chain_by_transforms(const lfts_ctx *c, int *by_transforms)
{
    if (!c || !by_transforms) return LFTS_ERR_ARG;
    *by_transforms = c->transform_chain ? 1 : 0;
    return LFTS_OK;
}

int lfts_tuning(const lfts_ctx *c, int *pencil_cw, int *plane_stages)
{
    if (!c) return LFTS_ERR_ARG;
    if (pencil_cw) *pencil_cw = c->tiles.pencil_cw;
    if (plane_stages) *plane_stages = c->tiles.plane_stages;
    return LFTS_OK;
}

long long lfts_kernel_launches(const lfts_ctx *c) { return c ? c->launches : 0; }

int lfts_anderson_stats(const lfts_ctx *c, long long *calls, long long *iterations)
{
    if (!c) return LFTS_ERR_ARG;
    if (calls) *calls = c->mix_calls;
    if (iterations) *iterations = c->mix_iters;
    return LFTS_OK;
}

int lfts_get_propagators(lfts_ctx *c, double *q_host)
{
    if (!c || !q_host) return LFTS_ERR_ARG;
    DeviceGuard g(c->dev);
    const long long n = 2 * c->M * (long long)c->N;
    std::memset(q_host, 0, sizeof(double) * 2 * c->M);
    if (c->prec == LFTS_FP64) {
        CK(cudaMemcpyAsync(q_host + 2 * c->M, c->q, sizeof(double) * n, cudaMemcpyDeviceToHost, c->st));
        CK(cudaStreamSynchronize(c->st));
    } else {
        if (c->phi_in_chain && c->fields_set) {
            // the chain that forms the concentration sums leaves the later slots
            // unstored: run the storing chain on the same fields
            c->phi_in_chain = false;
            enqueue_chain_launches<float>(c);
            c->phi_in_chain = true;
            CK(cudaGetLastError());
        }
        // FP32 slots hold (q_i, q^_{N+1-i}) pairs: back to the [q_i | q^] halves
        std::vector<float> tmp(n);
        CK(cudaMemcpyAsync(tmp.data(), c->q, sizeof(float) * n, cudaMemcpyDeviceToHost, c->st));
        CK(cudaStreamSynchronize(c->st));
        const long long M = c->M;
        for (int sl = 0; sl < c->N; sl++) {
            const float *src = tmp.data() + (long long)sl * 2 * M;
            double *dst = q_host + (long long)(sl + 1) * 2 * M;
            for (long long r = 0; r < M; r++) {
                dst[r] = src[2 * r];
                dst[M + r] = src[2 * r + 1];
            }
        }
    }
    return LFTS_OK;
}

}  // extern "C"
