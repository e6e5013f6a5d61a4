// Contour-chain kernels that apply the Gaussian bond one axis at a time.
//
// The Boltzmann weight of a bond is separable, g(k) = gx gy gz, so one contour
// step of the reference (step::fwd, src/step.cc:35-65)
//     q' = h . F^-1[g . F[q]] = h . Cx Cy Cz q,    Ca = Fa^-1 ga Fa,
// is three one-dimensional convolutions, which commute and keep real fields
// real.  They are therefore free to be grouped across the multiplication by h:
//     ... h . Cx | Cx . (Cy Cz) . h . (Cz Cy) | Cx . h . Cx | (Cy Cz) . h ...
// A kernel that holds whole x lines does [Cx h Cx], the end of one step and the
// start of the next, and one that holds whole yz planes does [Cy Cz h Cz Cy]:
// one kernel and one pass over the field per contour step, where a forward and
// a backward 3-D transform take two.  Where a plane is too much work for one
// CTA, the y lines get a kernel of their own: [Cz h Cz], [Cy], [Cx h Cx], [Cy].
// Both groupings do the same arithmetic on every value in the same order, so
// they agree bit for bit.
//
// What is transformed as one complex line.  FP32: the two chains, Z = q_i + i
// q^_{N+1-i}, stored as pairs.  FP64: two neighbouring real lines of one chain
// (Ca is real, so it acts on the two parts alike), the chains apart: columns z
// and z + 1 along x and y, rows y and y + 1 along z.
//
// A line of n = R1 R2 points is transformed in two register stages with one
// exchange through shared memory between them (stage A: points j2 + R2 a;
// stage B: outputs k1 + R1 k2), and a convolution is A | B ga B' | A': every
// thread ends with the natural-order points that it started with, so h is
// applied, the propagator slot stored and the next convolution begun without
// leaving registers.
//
// Every kernel lets its dependent launch only ahead of its final stores.  A
// dependent launched at the start takes SM slots that it can only wait in, and
// its CTAs pile up on the SMs that happen to have room: the chain of a 96^3
// FP32 system (N = 64) took 964 us so, 596 us with the late release.
#pragma once
#include "dft.cuh"
#include "fft_kernels.cuh"

namespace lfts {

enum AxisMode : int {
    AX_H = 0,        // convolve, times h, store the slot, convolve
    AX_H_LAST = 1,   // convolve, times h, store slot N, sum chain 1 for Q
    AX_HA = 2,       // AX_H with the concentration sums in place of the stored slot
    AX_HA_LAST = 3,  // AX_H_LAST with the concentration sums
    AX_CONV = 4,     // convolve (y lines)
    AX_INIT_W = 5,   // h = exp(-w/N) from the fields, stored as slot 1, convolve (z, plane)
    AX_INIT_Q = 6,   // the given rows, convolve (z, plane)
    AX_OUT = 7,      // convolve, times h, store to the caller's arrays (x lines; FP64: 8-byte aligned)
};
constexpr int kAxisModes = 8;

// The share of 1/M in an axis's weights: the largest power of two up to its length on
// x and y, the rest on z, so that every convolution leaves values of the size that it
// found.  With all of it on z an FP32 field was 1/(mx my) of itself between the axes,
// and propagators below exp(-80) lost digits there (128^3, w+ shifted by 86: q_N 8.4e-5
// off, 5.8e-7 so).  Powers of two change no other value.
__host__ __device__ constexpr int axis_scale(int n)
{
    int s = 1;
    while (2 * s <= n) s *= 2;
    return s;
}

template <typename T>
struct AxisArgs {
    T *S;                      // the field: FP32 M pairs (chain 1, chain 2); FP64 two fields of M
    const cpx<T> *twx, *twy, *twz;  // exp(-2 pi i t/n)
    const T *gx, *gy, *gz;     // axis weights over signed wavenumbers, 1/M in their product (axis_scale)
    int mx, my, mz;
    int cbase;                 // chain of the grid's first chain index (FP64)
    long long M;
    const double *w;           // INIT_W: W- (M) and w+ (M)
    double Nd;                 // N as a double (h = exp(-w/N))
    double L[3];               // SELF kernels: box, for the tables that they make themselves
    const T *h;                // FP32: (hA, hB) pairs; FP64: [hA | hB]
    const T *src[2];           // INIT_Q: the chains' real rows
    T *q[2];                   // FP32: q[0] = the slot's pairs; FP64: each chain's half (null: not stored)
    int hsel[2];               // h half of each chain (0 = hA, 1 = hB)
    const T *partner;          // HA: the partner slot's pairs (null: the slot pairs with itself)
    T *acc;                    // HA: (A, B) sums per mesh point
    int acc_init, a_is_A, b_is_A;
    double *qpart;             // LAST: one chain-1 sum per CTA
    unsigned *ticket;          // LAST: CTAs done, zero between launches (null: no Q)
    double *Qd;                // LAST: Q, ln Q
};

// R1 points per stage-A task, R2 per stage-B task
template <int N>
struct AxPlan;
template <> struct AxPlan<8> { static constexpr int R1 = 4, R2 = 2; };
template <> struct AxPlan<12> { static constexpr int R1 = 4, R2 = 3; };
template <> struct AxPlan<16> { static constexpr int R1 = 4, R2 = 4; };
template <> struct AxPlan<20> { static constexpr int R1 = 5, R2 = 4; };
template <> struct AxPlan<24> { static constexpr int R1 = 6, R2 = 4; };
template <> struct AxPlan<32> { static constexpr int R1 = 8, R2 = 4; };
template <> struct AxPlan<40> { static constexpr int R1 = 8, R2 = 5; };
template <> struct AxPlan<48> { static constexpr int R1 = 8, R2 = 6; };
template <> struct AxPlan<64> { static constexpr int R1 = 8, R2 = 8; };
template <> struct AxPlan<80> { static constexpr int R1 = 10, R2 = 8; };
template <> struct AxPlan<96> { static constexpr int R1 = 12, R2 = 8; };
template <> struct AxPlan<128> { static constexpr int R1 = 16, R2 = 8; };

// z lines apart (zline_kernel): R1, R2 and the lines a warp works on
template <int N>
struct AxPlanZ {
    static constexpr int R1 = AxPlan<N>::R1, R2 = AxPlan<N>::R2, LPW = 32 / R2;
};
// 128: 16 lanes of a warp then take 16 neighbouring points, a whole 128-byte row
// (FP32; Z kernel 11.7 -> 10.0 us with lines of 128^3; at 80 and 96 the wider
// stage B costs more than the rows give: 4.6 -> 5.2, 6.3 -> 6.5 us)
template <> struct AxPlanZ<128> { static constexpr int R1 = 8, R2 = 16, LPW = 4; };

// R values of a 16-byte aligned shared-memory row, read 16 bytes at a time (the
// row is padded to whole 16 bytes)
template <int R, typename E>
__device__ __forceinline__ void ax_row(const E *row, E (&out)[R])
{
    constexpr int V = 16 / (int)sizeof(E);
#pragma unroll
    for (int i = 0; i < (R + V - 1) / V; i++) {
        const float4 q = reinterpret_cast<const float4 *>(row)[i];
        const E *e = reinterpret_cast<const E *>(&q);
#pragma unroll
        for (int j = 0; j < V; j++)
            if (V * i + j < R) out[V * i + j] = e[j];
    }
}

// Axis tables in shared memory, a row per k1: twiddles exp(-2 pi i k1 u/n) over
// u, then g(k1 + R1 k2) over k2.  The twiddles are applied in stage B, where a
// task needs R2 of them for both directions, and not in stage A, which would read
// R1 for each; rows are an odd number of 16-byte units, so that lanes on
// different rows read different banks.
template <typename T, int R1, int R2>
struct AxTables {
    static constexpr int N = R1 * R2;
    static constexpr int TP = (R2 * (int)sizeof(cpx<T>) + 15) / 16 | 1, GP = (R2 * (int)sizeof(T) + 15) / 16 | 1;
    static constexpr size_t BYTES = 16 * (size_t)R1 * (TP + GP);
    unsigned char *at;
    __device__ __forceinline__ cpx<T> *tw(int k1) const { return reinterpret_cast<cpx<T> *>(at + 16 * k1 * TP); }
    __device__ __forceinline__ T *g(int k1) const { return reinterpret_cast<T *>(at + 16 * (R1 * TP + k1 * GP)); }
    __device__ __forceinline__ void load(const cpx<T> *__restrict__ twg, const T *__restrict__ gg, int tid, int nt)
    {
        for (int i = tid; i < N; i += nt) {
            const int k1 = i % R1, r = i / R1;
            tw(k1)[r] = twg[k1 * r];
            g(k1)[r] = gg[i];
        }
    }
    // the same from the axis's length and box side, for callers without tables in
    // memory: chain length nc, g divided by div
    __device__ __forceinline__ void make(double L, int nc, double div, int tid, int nt)
    {
        const double two_pi = 6.283185307179586476925286766559005768;
        for (int i = tid; i < N; i += nt) {
            const int k1 = i % R1, r = i / R1, k = i <= N / 2 ? i : i - N;
            double sn, cs;
            sincospi(-2.0 * (k1 * r) / N, &sn, &cs);
            tw(k1)[r] = {(T)cs, (T)sn};
            const double ksq = (double)k * k / (L * L);
            g(k1)[r] = (T)(exp(-two_pi * two_pi * ksq / (6.0 * nc)) / div);
        }
    }
    // stage B of one task: v[u], the inputs of outputs k1 + R1 k2, there and back
    __device__ __forceinline__ void convolve(cpx<T> (&v)[R2], int k1) const
    {
        cpx<T> w[R2];
        T gk[R2];
        ax_row(tw(k1), w);
        ax_row(g(k1), gk);
#pragma unroll
        for (int u = 1; u < R2; u++) v[u] = ctw<-1>(v[u], w[u]);
        Dft<R2, -1, T>::run(v);
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) v[k2] = cscale(v[k2], gk[k2]);
        Dft<R2, 1, T>::run(v);
#pragma unroll
        for (int u = 1; u < R2; u++) v[u] = ctw<1>(v[u], w[u]);
    }
};

// One group of threads (a block or a warp) convolving NL lines of N points.
// LF: neighbouring threads take neighbouring lines (strided axes), else
// neighbouring points of one line (the contiguous axis).  Idx maps (line,
// point) to shared memory.
template <typename T, int R1, int R2, int NL, int NTG, bool LF, class Idx>
struct LineConv {
    static constexpr int RA = (NL * R2 + NTG - 1) / NTG, RB = (NL * R1 + NTG - 1) / NTG;
    static __device__ __forceinline__ bool okA(int t) { return (NL * R2) % NTG == 0 || t < NL * R2; }
    static __device__ __forceinline__ bool okB(int t) { return (NL * R1) % NTG == 0 || t < NL * R1; }
    static __device__ __forceinline__ int lineA(int t) { return LF ? t % NL : t / R2; }
    static __device__ __forceinline__ int ptA(int t) { return LF ? t / NL : t % R2; }
    static __device__ __forceinline__ int lineB(int t) { return LF ? t % NL : t / R1; }
    static __device__ __forceinline__ int ptB(int t) { return LF ? t / NL : t % R1; }

    // stage A: DFT, to shared memory
    static __device__ __forceinline__ void A(cpx<T> (&v)[RA][R1], cpx<T> *sm, int tid)
    {
#pragma unroll
        for (int s = 0; s < RA; s++) {
            const int t = tid + s * NTG;
            if (!okA(t)) continue;
            const int l = lineA(t), j2 = ptA(t);
            Dft<R1, -1, T>::run(v[s]);
#pragma unroll
            for (int k1 = 0; k1 < R1; k1++) sm[Idx::at(l, j2 + R2 * k1)] = v[s][k1];
        }
    }
    // stage B in place: twiddles, spectrum times g, and back
    static __device__ __forceinline__ void B(cpx<T> *sm, const AxTables<T, R1, R2> &tab, int tid)
    {
#pragma unroll
        for (int s = 0; s < RB; s++) {
            const int t = tid + s * NTG;
            if (!okB(t)) continue;
            const int l = lineB(t), k1 = ptB(t);
            cpx<T> v[R2];
#pragma unroll
            for (int u = 0; u < R2; u++) v[u] = sm[Idx::at(l, R2 * k1 + u)];
            tab.convolve(v, k1);
#pragma unroll
            for (int u = 0; u < R2; u++) sm[Idx::at(l, R2 * k1 + u)] = v[u];
        }
    }
    // stage A back: v[s][j1] = the line's point j2 + R2 j1
    static __device__ __forceinline__ void Ainv(cpx<T> (&v)[RA][R1], const cpx<T> *sm, int tid)
    {
#pragma unroll
        for (int s = 0; s < RA; s++) {
            const int t = tid + s * NTG;
            if (!okA(t)) continue;
            const int l = lineA(t), j2 = ptA(t);
#pragma unroll
            for (int k1 = 0; k1 < R1; k1++) v[s][k1] = sm[Idx::at(l, j2 + R2 * k1)];
            Dft<R1, 1, T>::run(v[s]);
        }
    }
};

// ------------------------------------------------ h, slots, concentration sums --
// real fields in one complex value: FP32 pairs, one field of them; FP64 the
// chain's own field, whose points o and o + 1 (x and y lines) make one value
template <typename T>
inline constexpr bool kPairs = sizeof(T) == sizeof(float);
template <typename T>
inline constexpr int kChains = kPairs<T> ? 1 : 2;  // fields of a context

// complex value o of the field, chain c
template <typename T>
__device__ __forceinline__ cpx<T> *ax_field(const AxisArgs<T> &a, int c)
{
    return reinterpret_cast<cpx<T> *>(a.S + (kPairs<T> ? 0 : (long long)c * a.M));
}

// h at complex value o (x and y lines); WIDE: FP64 as one 16-byte load
template <bool WIDE, typename T>
__device__ __forceinline__ cpx<T> ax_h(const AxisArgs<T> &a, int c, int o)
{
    if constexpr (kPairs<T>) {
        const float2 h = __ldg(reinterpret_cast<const float2 *>(a.h) + o);
        return {a.hsel[0] ? h.y : h.x, a.hsel[1] ? h.y : h.x};
    } else {
        const double *p = a.h + (a.hsel[c] ? a.M : 0);
        if constexpr (!WIDE) return {__ldg(p + 2 * o), __ldg(p + 2 * o + 1)};
        const double2 h = __ldg(reinterpret_cast<const double2 *>(p) + o);
        return {h.x, h.y};
    }
}

// the slots go out with evict-first stores: they are read again only by the
// concentration pass
template <bool WIDE, typename T>
__device__ __forceinline__ void ax_store(const AxisArgs<T> &a, int c, int o, cpx<T> v)
{
    if constexpr (kPairs<T>) {
        __stcs(reinterpret_cast<float2 *>(a.q[0]) + o, make_float2(v.x, v.y));
    } else if constexpr (WIDE) {
        if (a.q[c]) __stcs(reinterpret_cast<double2 *>(a.q[c]) + o, make_double2(v.x, v.y));
    } else {
        a.q[c][2 * o] = v.x;
        a.q[c][2 * o + 1] = v.y;
    }
}

// The same for z lines.  FP64: a value is (point o of a row, point o + mz, the
// row after it); o counts reals.
template <typename T>
__device__ __forceinline__ cpx<T> axz_field(const AxisArgs<T> &a, int c, int o)
{
    if constexpr (kPairs<T>) return ax_field(a, c)[o];
    const T *p = a.S + (long long)c * a.M + o;
    return {p[0], p[a.mz]};
}
template <typename T>
__device__ __forceinline__ void axz_field_store(const AxisArgs<T> &a, int c, int o, cpx<T> v)
{
    if constexpr (kPairs<T>) {
        ax_field(a, c)[o] = v;
    } else {
        T *p = a.S + (long long)c * a.M + o;
        p[0] = v.x;
        p[a.mz] = v.y;
    }
}
template <typename T>
__device__ __forceinline__ cpx<T> axz_h(const AxisArgs<T> &a, int c, int o)
{
    if constexpr (kPairs<T>) return ax_h<true>(a, c, o);
    const T *p = a.h + (a.hsel[c] ? a.M : 0) + o;
    return {__ldg(p), __ldg(p + a.mz)};
}
template <typename T>
__device__ __forceinline__ void axz_store(const AxisArgs<T> &a, int c, int o, cpx<T> v)
{
    if constexpr (kPairs<T>) {
        ax_store<true>(a, c, o, v);
    } else if (a.q[c]) {
        __stcs(a.q[c] + o, v.x);
        __stcs(a.q[c] + o + a.mz, v.y);
    }
}

// h = exp(-w/N) at a z-line value (src/diblock.cc:64-72), stored as slot 1: hA
// for chain 1, hB for chain 2.  FP32: the exponential is that of the transform
// chain's INIT_W on the same mesh (fft_plane3.cuh: single precision on 64, 96 and
// 128 square planes; fft_packed.cuh: double, rounded, elsewhere), so both chains
// start from the same h.
template <typename T>
__device__ __forceinline__ cpx<T> axz_init_w(const AxisArgs<T> &a, int c, int o)
{
    cpx<T> v;
    if constexpr (kPairs<T>) {
        const double wm = a.w[o], wp = a.w[a.M + o];
        const double eA = -(wm + wp) / a.Nd, eB = -(-wm + wp) / a.Nd;
        if (a.my == a.mz && (a.my == 64 || a.my == 96 || a.my == 128))
            v = {expf((float)eA), expf((float)eB)};
        else
            v = {(float)exp(eA), (float)exp(eB)};
        reinterpret_cast<cpx<T> *>(a.q[0])[o] = v;
    } else {
        const double sgn = c == 0 ? 1.0 : -1.0;
        const double *wm = a.w + o, *wp = a.w + a.M + o;
        v = {exp(-(sgn * wm[0] + wp[0]) / a.Nd), exp(-(sgn * wm[a.mz] + wp[a.mz]) / a.Nd)};
        a.q[c][o] = v.x;
        a.q[c][o + a.mz] = v.y;
    }
    return v;
}

// given rows: FP32 the two chains' (the field pairs them), FP64 two of chain c's
template <typename T>
__device__ __forceinline__ cpx<T> axz_init_q(const AxisArgs<T> &a, int c, int o)
{
    if constexpr (kPairs<T>) return {a.src[0][o], a.src[1][o]};
    return {a.src[c][o], a.src[c][o + a.mz]};
}

// concentration sums in the chain: FP32 lines long enough for the sums to pay
// (the separate pass reads what is then still in L2 at smaller meshes)
template <typename T, int N>
inline constexpr bool kAxisSums = kPairs<T> && (N == 96 || N == 128);

// chain-1 part of a value of slot N, for Q
template <typename T>
__device__ __forceinline__ double ax_q_part(cpx<T> v)
{
    return kPairs<T> ? (double)v.x : (double)v.x + (double)v.y;
}

// Concentration sums (AX_HA, AX_HA_LAST, FP32).  The new slot i+1 = (q_{i+1},
// q^_{N-i}) and its partner, slot N-i = (q_{N-i}, q^_{i+1}), give q_{i+1}
// q^_{i+1} = v.x p.y and q_{N-i} q^_{N-i} = p.x v.y; the middle slot of an odd
// chain has no partner and gives the one product v.x v.y.
template <typename T>
__device__ __forceinline__ float2 ax_partner(const AxisArgs<T> &a, int o)
{
    return a.partner ? __ldcs(reinterpret_cast<const float2 *>(a.partner) + o) : make_float2(0.f, 0.f);
}
template <typename T>
__device__ __forceinline__ float2 ax_sums(const AxisArgs<T> &a, int o)
{
    return a.acc_init ? make_float2(0.f, 0.f) : reinterpret_cast<const float2 *>(a.acc)[o];
}
template <typename T>
__device__ __forceinline__ void ax_acc(const AxisArgs<T> &a, int o, cpx<T> v, float2 p, float2 s)
{
    static_assert(kPairs<T>, "FP32 pairs only");
    float pa, pb = 0.f;
    if (a.partner) {
        pa = v.x * p.y;
        pb = p.x * v.y;
    } else {
        pa = v.x * v.y;
    }
    if (a.a_is_A)
        s.x += pa;
    else
        s.y += pa;
    if (a.b_is_A)
        s.x += pb;
    else
        s.y += pb;
    reinterpret_cast<float2 *>(a.acc)[o] = s;
}

// Q from the chain-1 values of slot N: one partial per CTA, and the CTA that
// finishes last adds the partials up in order, so the sum does not depend on
// the order in which CTAs run.  (src/diblock.cc:46-48,59)
template <int NT>
__device__ __forceinline__ void ax_q_sum(double qs, double *qpart, unsigned *ticket, double *Qd, double M, int cta,
                                         int nctas)
{
    constexpr int NW = (NT + 31) / 32;
    __shared__ double red[NW];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr unsigned mask = 0xffffffffu;
    static_assert(NT % 32 == 0, "whole warps");
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) qs += __shfl_xor_sync(mask, qs, o);
    if (lane == 0) red[wid] = qs;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < NW; i++) s += red[i];
        qpart[cta] = s;
        __threadfence();
        last = atomicAdd(ticket, 1u) + 1u == (unsigned)nctas;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double s = 0.0;
    for (int i = threadIdx.x; i < nctas; i += NT) s += __ldcg(qpart + i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(mask, s, o);
    if (lane == 0) red[wid] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int i = 0; i < NW; i++) t += red[i];
        const double Q = t / M;
        Qd[0] = Q;
        Qd[1] = log(Q);
        *ticket = 0;
    }
}

// --------------------------------------------------------------- strided lines --
// x lines (stride my mz, all columns) and y lines (stride mz, one x-plane per
// blockIdx.y): CTAs of CW neighbouring columns, so a warp's global accesses are
// whole 128-byte rows.
template <typename T, int N, int CW>
struct StridedCfg {
    static constexpr int R1 = AxPlan<N>::R1, R2 = AxPlan<N>::R2;
    static constexpr int NT = (CW * R2 + 31) / 32 * 32;
    // a row of 64 bytes (FP32, 8 columns) puts stage B's rows, R2 apart, on the
    // same half of the banks: one pad row per R2 rows moves them apart
    static constexpr int PADROW = (sizeof(cpx<T>) * CW == 64 && R2 % 2 == 0) ? 1 : 0;
    struct Idx {
        static __device__ __forceinline__ int at(int l, int p) { return (p + PADROW * (p / R2)) * CW + l; }
    };
    static constexpr size_t TILE = (sizeof(cpx<T>) * (size_t)CW * (N + PADROW * (N / R2)) + 15) / 16 * 16;
    using Tables = AxTables<T, R1, R2>;
    static constexpr size_t SMEM = TILE + Tables::BYTES;
    using Conv = LineConv<T, R1, R2, CW, NT, true, Idx>;
};

// (SELF: the CTA makes its tables, AxTables::make)
template <typename T, int N, int CW, int MODE, bool SELF, int AXIS>
__device__ __forceinline__ void strided_body(const AxisArgs<T> &a, const int c, const int stride, const int ncol, const int tile, const int base,
                                             const int nctas)
{
    using C = StridedCfg<T, N, CW>;
    using V = typename C::Conv;
    constexpr bool kH = MODE != AX_CONV, kAcc = MODE == AX_HA || MODE == AX_HA_LAST;
    constexpr bool kLast = MODE == AX_H_LAST || MODE == AX_HA_LAST;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cpx<T> *sm = reinterpret_cast<cpx<T> *>(smem_raw);
    const int tid = threadIdx.x, col0 = tile * CW;
    typename C::Tables tab{smem_raw + C::TILE};
    if constexpr (SELF)
        tab.make(a.L[AXIS], (int)a.Nd, (double)axis_scale(N), tid, C::NT);
    else
        tab.load(AXIS == 0 ? a.twx : a.twy, AXIS == 0 ? a.gx : a.gy, tid, C::NT);
    pdl_wait();

    // complex value of stage-A task t's point j
    cpx<T> *S = ax_field(a, c);
    auto live = [&](int t) { return V::okA(t) && col0 + V::lineA(t) < ncol; };
    auto at = [&](int t, int j) { return base + (V::ptA(t) + j * C::R2) * stride + col0 + V::lineA(t); };
    cpx<T> v[V::RA][C::R1];
#pragma unroll
    for (int s = 0; s < V::RA; s++) {
        const int t = tid + s * C::NT;
#pragma unroll
        for (int j = 0; j < C::R1; j++) v[s][j] = live(t) ? S[at(t, j)] : cpx<T>{(T)0, (T)0};
    }
    __syncthreads();
    V::A(v, sm, tid);
    // h comes in while stage B works from shared memory: the registers that
    // held the line's points are free until Ainv.  With the sums, so do the
    // partner slot and the sums: loaded at their use they made the 128^3 chain
    // 1565 us, loaded here 1204 (the fewer CTAs per SM cost less than the waits).
    cpx<T> h[kH ? V::RA : 1][C::R1];
    float2 pv[kAcc ? V::RA : 1][C::R1], sv[kAcc ? V::RA : 1][C::R1];
    if constexpr (kH) {
#pragma unroll
        for (int s = 0; s < V::RA; s++) {
            const int t = tid + s * C::NT;
            if (!live(t)) continue;
#pragma unroll
            for (int j = 0; j < C::R1; j++) h[s][j] = ax_h<MODE != AX_OUT>(a, c, at(t, j));
        }
    }
    if constexpr (kAcc) {
#pragma unroll
        for (int s = 0; s < V::RA; s++) {
            const int t = tid + s * C::NT;
            if (!live(t)) continue;
#pragma unroll
            for (int j = 0; j < C::R1; j++) {
                pv[s][j] = ax_partner(a, at(t, j));
                sv[s][j] = ax_sums(a, at(t, j));
            }
        }
    }
    __syncthreads();
    V::B(sm, tab, tid);
    __syncthreads();
    V::Ainv(v, sm, tid);
    if constexpr (kH) {
        double qs = 0.0;
#pragma unroll
        for (int s = 0; s < V::RA; s++) {
            const int t = tid + s * C::NT;
            if (!live(t)) continue;
#pragma unroll
            for (int j = 0; j < C::R1; j++) {
                v[s][j] = {v[s][j].x * h[s][j].x, v[s][j].y * h[s][j].y};
                if (MODE != AX_HA) ax_store<MODE != AX_OUT>(a, c, at(t, j), v[s][j]);
                if constexpr (kAcc) ax_acc(a, at(t, j), v[s][j], pv[s][j], sv[s][j]);
                if (kLast) qs += ax_q_part(v[s][j]);
            }
        }
        if constexpr (kLast) {
            if (a.ticket && c == 0) ax_q_sum<C::NT>(qs, a.qpart, a.ticket, a.Qd, (double)a.M, tile, nctas);
            return;
        }
        if constexpr (MODE == AX_OUT) return;
        V::A(v, sm, tid);
        __syncthreads();
        V::B(sm, tab, tid);
        __syncthreads();
        V::Ainv(v, sm, tid);
    }
    pdl_launch_dependents();
#pragma unroll
    for (int s = 0; s < V::RA; s++) {
        const int t = tid + s * C::NT;
        if (!live(t)) continue;
#pragma unroll
        for (int j = 0; j < C::R1; j++) S[at(t, j)] = v[s][j];
    }
}

// x lines: tile of CW columns of chain c's field (FP64: pairs of real columns)
template <typename T, int N, int CW, int MODE, bool SELF = false>
__device__ __forceinline__ void xline_body(const AxisArgs<T> &a, int tile, int c, int nctas)
{
    const int ncol = a.my * a.mz / kChains<T>;
    strided_body<T, N, CW, MODE, SELF, 0>(a, c, ncol, ncol, tile, 0, nctas);
}
// y lines of x-plane x
template <typename T, int N, int CW, bool SELF = false>
__device__ __forceinline__ void yline_body(const AxisArgs<T> &a, int tile, int x, int c)
{
    const int ncol = a.mz / kChains<T>;
    strided_body<T, N, CW, AX_CONV, SELF, 1>(a, c, ncol, ncol, tile, x * N * ncol, 0);
}

template <typename T, int N, int CW, int MODE, bool SELF = false>
__global__ void __launch_bounds__(StridedCfg<T, N, CW>::NT) xline_kernel(AxisArgs<T> a)
{
    xline_body<T, N, CW, MODE, SELF>(a, blockIdx.x, blockIdx.z + a.cbase, gridDim.x);
}
template <typename T, int N, int CW, bool SELF = false>
__global__ void __launch_bounds__(StridedCfg<T, N, CW>::NT) yline_kernel(AxisArgs<T> a)
{
    yline_body<T, N, CW, SELF>(a, blockIdx.x, blockIdx.y, blockIdx.z + a.cbase);
}

// ------------------------------------------------------------- contiguous lines --
// z lines, LPW whole lines per warp, so the exchanges need no block barrier
template <typename T, int N>
struct ZCfg {
    static constexpr int R1 = AxPlanZ<N>::R1, R2 = AxPlanZ<N>::R2;
    static constexpr int LPW = AxPlanZ<N>::LPW;
    static constexpr int NW = 4, NT = 32 * NW;
    // one pad slot per R2 points: stage B's tasks, R2 apart, start on different banks
    static constexpr int SPAN = N + N / R2;
    static constexpr int PITCH = (SPAN + 7) / 16 * 16 + 8;
    struct Idx {
        static __device__ __forceinline__ int at(int l, int p) { return l * PITCH + p + p / R2; }
    };
    static constexpr size_t TILE = (sizeof(cpx<T>) * (size_t)NW * LPW * PITCH + 15) / 16 * 16;
    using Tables = AxTables<T, R1, R2>;
    static constexpr size_t SMEM = TILE + Tables::BYTES;
    using Conv = LineConv<T, R1, R2, LPW, 32, false, Idx>;
    static_assert(PITCH >= SPAN, "pitch covers the padded line");
};

template <typename T, int N, int MODE, bool SELF = false>
__device__ __forceinline__ void zline_body(const AxisArgs<T> &a, const int cta, const int c, const int nctas)
{
    using C = ZCfg<T, N>;
    using V = typename C::Conv;
    constexpr bool kInit = MODE == AX_INIT_W || MODE == AX_INIT_Q;
    constexpr bool kAcc = MODE == AX_HA || MODE == AX_HA_LAST;
    constexpr bool kLast = MODE == AX_H_LAST || MODE == AX_HA_LAST;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    cpx<T> *sm = reinterpret_cast<cpx<T> *>(smem_raw) + wid * C::LPW * C::PITCH;
    const int nlines = a.mx * a.my / kChains<T>;
    const int line0 = (cta * C::NW + wid) * C::LPW;
    typename C::Tables tab{smem_raw + C::TILE};
    if constexpr (SELF)
        tab.make(a.L[2], (int)a.Nd, (double)a.M / (axis_scale(a.mx) * axis_scale(a.my)), threadIdx.x, C::NT);
    else
        tab.load(a.twz, a.gz, threadIdx.x, C::NT);
    pdl_wait();

    auto live = [&](int t) { return V::okA(t) && line0 + V::lineA(t) < nlines; };
    auto at = [&](int t, int j) {  // FP64: the first row's point, two rows a line
        return (line0 + V::lineA(t)) * (kChains<T> * N) + V::ptA(t) + j * C::R2;
    };
    cpx<T> v[V::RA][C::R1];
#pragma unroll
    for (int s = 0; s < V::RA; s++) {
        const int t = lane + s * 32;
#pragma unroll
        for (int j = 0; j < C::R1; j++) {
            if (!live(t))
                v[s][j] = {(T)0, (T)0};
            else if constexpr (MODE == AX_INIT_W)
                v[s][j] = axz_init_w(a, c, at(t, j));
            else if constexpr (MODE == AX_INIT_Q)
                v[s][j] = axz_init_q(a, c, at(t, j));
            else
                v[s][j] = axz_field(a, c, at(t, j));
        }
    }
    __syncthreads();
    V::A(v, sm, lane);
    cpx<T> h[kInit ? 1 : V::RA][C::R1];  // as in strided_body
    float2 pv[kAcc ? V::RA : 1][C::R1], sv[kAcc ? V::RA : 1][C::R1];
    if constexpr (!kInit) {
#pragma unroll
        for (int s = 0; s < V::RA; s++) {
            const int t = lane + s * 32;
            if (!live(t)) continue;
#pragma unroll
            for (int j = 0; j < C::R1; j++) h[s][j] = axz_h(a, c, at(t, j));
        }
    }
    if constexpr (kAcc) {
#pragma unroll
        for (int s = 0; s < V::RA; s++) {
            const int t = lane + s * 32;
            if (!live(t)) continue;
#pragma unroll
            for (int j = 0; j < C::R1; j++) {
                pv[s][j] = ax_partner(a, at(t, j));
                sv[s][j] = ax_sums(a, at(t, j));
            }
        }
    }
    __syncwarp();
    V::B(sm, tab, lane);
    __syncwarp();
    V::Ainv(v, sm, lane);
    if constexpr (!kInit) {
        double qs = 0.0;
#pragma unroll
        for (int s = 0; s < V::RA; s++) {
            const int t = lane + s * 32;
            if (!live(t)) continue;
#pragma unroll
            for (int j = 0; j < C::R1; j++) {
                v[s][j] = {v[s][j].x * h[s][j].x, v[s][j].y * h[s][j].y};
                if (MODE != AX_HA) axz_store(a, c, at(t, j), v[s][j]);
                if constexpr (kAcc) ax_acc(a, at(t, j), v[s][j], pv[s][j], sv[s][j]);
                if (kLast) qs += ax_q_part(v[s][j]);
            }
        }
        if constexpr (kLast) {
            if (a.ticket && c == 0) ax_q_sum<C::NT>(qs, a.qpart, a.ticket, a.Qd, (double)a.M, cta, nctas);
            return;
        }
        V::A(v, sm, lane);
        __syncwarp();
        V::B(sm, tab, lane);
        __syncwarp();
        V::Ainv(v, sm, lane);
    }
    pdl_launch_dependents();
#pragma unroll
    for (int s = 0; s < V::RA; s++) {
        const int t = lane + s * 32;
        if (!live(t)) continue;
#pragma unroll
        for (int j = 0; j < C::R1; j++) axz_field_store(a, c, at(t, j), v[s][j]);
    }
}

template <typename T, int N, int MODE, bool SELF = false>
__global__ void __launch_bounds__(ZCfg<T, N>::NT) zline_kernel(AxisArgs<T> a)
{
    zline_body<T, N, MODE, SELF>(a, blockIdx.x, blockIdx.z + a.cbase, gridDim.x);
}

// -------------------------------------------------------------------- yz planes --
// One CTA per x-plane (and, in FP64, chain), the plane in shared memory: a warp
// convolves whole y lines, then (after a block barrier) whole z lines, then y
// lines again; the exchanges inside a line are the warp's own.
template <typename T, int NY, int NZ>
struct PlaneAxCfg {
    static constexpr int RY1 = AxPlan<NY>::R1, RY2 = AxPlan<NY>::R2, RZ1 = AxPlan<NZ>::R1, RZ2 = AxPlan<NZ>::R2;
    static constexpr int MY = RY1 > RY2 ? RY1 : RY2, MZ = RZ1 > RZ2 ? RZ1 : RZ2;
    static constexpr int CPW = 32 / MY, LPW = 32 / MZ;  // y and z lines per warp, one task per lane
    static constexpr int NCOL = NZ / kChains<T>, NROW = NY / kChains<T>;  // y and z lines of a plane
    static constexpr int WY = (NCOL + CPW - 1) / CPW, WZ = (NROW + LPW - 1) / LPW;
    static constexpr int NW0 = WY > WZ ? WY : WZ;
    static constexpr int NW = NW0 > 16 ? 16 : NW0, NT = 32 * NW;
    // rows of NCOL values; pads: one value per RZ2, 4 values per RY2 rows, and a
    // pitch of 4 (mod 8) values
    static constexpr int SPAN = NCOL + (NCOL - 1) / RZ2;
    static constexpr int PITCH = (SPAN + 3) / 8 * 8 + 4;
    static __device__ __forceinline__ int zpos(int z) { return z + z / RZ2; }
    static __device__ __forceinline__ int ypos(int y) { return y * PITCH + 4 * (y / RY2); }
    static constexpr size_t TILE = (sizeof(cpx<T>) * (size_t)(NY * PITCH + 4 * (NY / RY2)) + 15) / 16 * 16;
    using TabY = AxTables<T, RY1, RY2>;
    using TabZ = AxTables<T, RZ1, RZ2>;
    static constexpr size_t SMEM = TILE + TabY::BYTES + TabZ::BYTES;
    static_assert(PITCH >= SPAN, "pitch covers the padded row");
};

template <typename T, int NY, int NZ, int MODE, bool SELF = false>
__device__ __forceinline__ void planeax_body(const AxisArgs<T> &a, const int x, const int c, const int nctas)
{
    using C = PlaneAxCfg<T, NY, NZ>;
    constexpr bool kInit = MODE == AX_INIT_W || MODE == AX_INIT_Q;
    constexpr bool kLast = MODE == AX_H_LAST;
    static_assert(MODE != AX_HA && MODE != AX_HA_LAST && MODE != AX_CONV, "not a plane mode");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cpx<T> *P = reinterpret_cast<cpx<T> *>(smem_raw);
    T *Pr = reinterpret_cast<T *>(smem_raw);
    typename C::TabY taby{smem_raw + C::TILE};
    typename C::TabZ tabz{smem_raw + C::TILE + C::TabY::BYTES};
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if constexpr (SELF) {
        taby.make(a.L[1], (int)a.Nd, (double)axis_scale(NY), threadIdx.x, C::NT);
        tabz.make(a.L[2], (int)a.Nd, (double)a.M / (axis_scale(a.mx) * axis_scale(NY)), threadIdx.x, C::NT);
    } else {
        taby.load(a.twy, a.gy, threadIdx.x, C::NT);
        tabz.load(a.twz, a.gz, threadIdx.x, C::NT);
    }
    pdl_wait();
    cpx<T> *S = ax_field(a, c) + x * NY * C::NCOL;

    // y lines: a lane's tasks are (column, j2) and (column, k1), column fastest
    const int ycl = lane % C::CPW, yj = lane / C::CPW;
    // z lines: (line, j2) and (line, k1), point fastest
    const int zlA = lane / C::RZ2, zjA = lane % C::RZ2, zlB = lane / C::RZ1, zjB = lane % C::RZ1;

    auto y_conv = [&](cpx<T>(&v)[C::RY1], int col, bool okA, bool okB) {
        if (okA) {
            Dft<C::RY1, -1, T>::run(v);
#pragma unroll
            for (int k = 0; k < C::RY1; k++) P[C::ypos(yj + C::RY2 * k) + col] = v[k];
        }
        __syncwarp();
        if (okB) {
            cpx<T> u[C::RY2];
#pragma unroll
            for (int i = 0; i < C::RY2; i++) u[i] = P[C::ypos(C::RY2 * yj + i) + col];
            taby.convolve(u, yj);
#pragma unroll
            for (int i = 0; i < C::RY2; i++) P[C::ypos(C::RY2 * yj + i) + col] = u[i];
        }
        __syncwarp();
        if (okA) {
#pragma unroll
            for (int k = 0; k < C::RY1; k++) v[k] = P[C::ypos(yj + C::RY2 * k) + col];
            Dft<C::RY1, 1, T>::run(v);
        }
    };
    // point p of z line l in flight: FP32 in its row; FP64 in the two rows of
    // the line (2l, 2l + 1) as one run of complex values
    auto zat = [&](int l, int p) {
        if constexpr (kPairs<T>)
            return C::ypos(l) + C::zpos(p);
        else
            return p < NZ / 2 ? C::ypos(2 * l) + C::zpos(p) : C::ypos(2 * l + 1) + C::zpos(p - NZ / 2);
    };
    auto z_conv = [&](cpx<T>(&v)[C::RZ1], int l0, bool okA, bool okB) {
        if (okA) {
            Dft<C::RZ1, -1, T>::run(v);
#pragma unroll
            for (int k = 0; k < C::RZ1; k++) P[zat(l0 + zlA, zjA + C::RZ2 * k)] = v[k];
        }
        __syncwarp();
        if (okB) {
            cpx<T> u[C::RZ2];
#pragma unroll
            for (int i = 0; i < C::RZ2; i++) u[i] = P[zat(l0 + zlB, C::RZ2 * zjB + i)];
            tabz.convolve(u, zjB);
#pragma unroll
            for (int i = 0; i < C::RZ2; i++) P[zat(l0 + zlB, C::RZ2 * zjB + i)] = u[i];
        }
        __syncwarp();
        if (okA) {
#pragma unroll
            for (int k = 0; k < C::RZ1; k++) v[k] = P[zat(l0 + zlA, zjA + C::RZ2 * k)];
            Dft<C::RZ1, 1, T>::run(v);
        }
    };

    if constexpr (!kInit) {
        for (int w = wid; w < C::WY || w == wid; w += C::NW) {
            const int z = w * C::CPW + ycl;
            const bool okA = w < C::WY && yj < C::RY2 && z < C::NCOL, okB = w < C::WY && yj < C::RY1 && z < C::NCOL;
            cpx<T> v[C::RY1];
            if (okA) {
#pragma unroll
                for (int j = 0; j < C::RY1; j++) v[j] = S[(yj + C::RY2 * j) * C::NCOL + z];
            }
            if (w == wid) __syncthreads();  // tables
            y_conv(v, C::zpos(z), okA, okB);
            if (okA) {
#pragma unroll
                for (int j = 0; j < C::RY1; j++) P[C::ypos(yj + C::RY2 * j) + C::zpos(z)] = v[j];
            }
        }
    }
    __syncthreads();

    double qs = 0.0;
    for (int w = wid; w < C::WZ; w += C::NW) {
        const int l0 = w * C::LPW, l = l0 + zlA;
        const bool okA = zlA < C::LPW && l < C::NROW, okB = zlB < C::LPW && l0 + zlB < C::NROW;
        const int o0 = x * NY * NZ + l * (kChains<T> * NZ) + zjA;
        cpx<T> v[C::RZ1];
        if (okA) {
#pragma unroll
            for (int j = 0; j < C::RZ1; j++) {
                const int z = zjA + C::RZ2 * j;
                if constexpr (MODE == AX_INIT_W) {
                    v[j] = axz_init_w(a, c, o0 + C::RZ2 * j);
                } else if constexpr (MODE == AX_INIT_Q) {
                    v[j] = axz_init_q(a, c, o0 + C::RZ2 * j);
                } else if constexpr (kPairs<T>) {
                    v[j] = P[zat(l, z)];
                } else {
                    const int at = 2 * C::zpos(z / 2) + (z & 1);
                    v[j] = {Pr[2 * C::ypos(2 * l) + at], Pr[2 * C::ypos(2 * l + 1) + at]};
                }
            }
        }
        if constexpr (!kPairs<T>) __syncwarp();  // rows read before complex values go over them
        if constexpr (!kInit) {
            cpx<T> h[C::RZ1];
            if (okA) {
#pragma unroll
                for (int j = 0; j < C::RZ1; j++) h[j] = axz_h(a, c, o0 + C::RZ2 * j);
            }
            z_conv(v, l0, okA, okB);
            if (okA) {
#pragma unroll
                for (int j = 0; j < C::RZ1; j++) {
                    v[j] = {v[j].x * h[j].x, v[j].y * h[j].y};
                    axz_store(a, c, o0 + C::RZ2 * j, v[j]);
                    if (kLast) qs += ax_q_part(v[j]);
                }
            }
        }
        if constexpr (!kLast) {
            z_conv(v, l0, okA, okB);
            if constexpr (!kPairs<T>) __syncwarp();  // complex values read before rows go over them
            if (okA) {
#pragma unroll
                for (int j = 0; j < C::RZ1; j++) {
                    const int z = zjA + C::RZ2 * j;
                    if constexpr (kPairs<T>) {
                        P[zat(l, z)] = v[j];
                    } else {
                        const int at = 2 * C::zpos(z / 2) + (z & 1);
                        Pr[2 * C::ypos(2 * l) + at] = v[j].x;
                        Pr[2 * C::ypos(2 * l + 1) + at] = v[j].y;
                    }
                }
            }
        }
    }
    if constexpr (kLast) {
        if (a.ticket && c == 0) ax_q_sum<C::NT>(qs, a.qpart, a.ticket, a.Qd, (double)a.M, x, nctas);
        return;
    }
    __syncthreads();
    pdl_launch_dependents();

    for (int w = wid; w < C::WY; w += C::NW) {
        const int z = w * C::CPW + ycl;
        const bool okA = yj < C::RY2 && z < C::NCOL, okB = yj < C::RY1 && z < C::NCOL;
        cpx<T> v[C::RY1];
        if (okA) {
#pragma unroll
            for (int j = 0; j < C::RY1; j++) v[j] = P[C::ypos(yj + C::RY2 * j) + C::zpos(z)];
        }
        y_conv(v, C::zpos(z), okA, okB);
        if (okA) {
#pragma unroll
            for (int j = 0; j < C::RY1; j++) S[(yj + C::RY2 * j) * C::NCOL + z] = v[j];
        }
    }
}

template <typename T, int NY, int NZ, int MODE, bool SELF = false>
__global__ void __launch_bounds__(PlaneAxCfg<T, NY, NZ>::NT) planeax_kernel(AxisArgs<T> a)
{
    planeax_body<T, NY, NZ, MODE, SELF>(a, blockIdx.x, blockIdx.z + a.cbase, gridDim.x);
}

}  // namespace lfts
