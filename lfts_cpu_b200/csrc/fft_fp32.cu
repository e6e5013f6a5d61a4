// FP32 kernels of the transform chain (the FP32-mixed chain by 3-D transforms).
#include "fft_dispatch.h"
#include "fft_lengths.h"
#include "fft_packed.cuh"
#include "fft_plane3.cuh"
#include "fft_plane3c.cuh"

namespace lfts {

template <typename T, int NY, int NZ>
static void fill_plane_c(PlaneKernels<T> *o)
{
    using C = PlaneCCfg<T, NY, NZ>;
    o->fn[PLANE_INIT_W] = plane_c_kernel<T, NY, NZ, PLANE_INIT_W>;
    o->fn[PLANE_STEP] = plane_c_kernel<T, NY, NZ, PLANE_STEP>;
    o->fn[PLANE_LAST] = plane_c_kernel<T, NY, NZ, PLANE_LAST>;
    o->fn[PLANE_G] = nullptr;
    o->nt = C::NT;
    o->smem = C::SMEM;
}

template <typename T, int NX, int CW>
static void fill_pencil(PencilKernels<T> *o)
{
    using C = PencilCfg<T, NX, CW>;
    o->fn[PENCIL_CONV] = pencil_kernel<T, NX, CW, PENCIL_CONV>;
    o->fn[PENCIL_POWER] = nullptr;  // S(k) samples run in FP64 in both precisions
    // the h-in-pencil chain: FP32 packed field, 96- and 128-point x lines (at 64
    // the pencil's added h and q traffic cost more than the plane kernel saves)
    if constexpr (NX == 96 || NX == 128) {
        o->fn[PENCIL_H] = pencil_kernel<T, NX, CW, PENCIL_H>;
        o->fn[PENCIL_H_LAST] = pencil_kernel<T, NX, CW, PENCIL_H_LAST>;
        o->fn[PENCIL_INIT_W] = pencil_kernel<T, NX, CW, PENCIL_INIT_W>;
        o->fn[PENCIL_HA] = pencil_kernel<T, NX, CW, PENCIL_HA>;
        o->fn[PENCIL_HA_LAST] = pencil_kernel<T, NX, CW, PENCIL_HA_LAST>;
    } else {
        o->fn[PENCIL_H] = o->fn[PENCIL_H_LAST] = o->fn[PENCIL_INIT_W] = nullptr;
        o->fn[PENCIL_HA] = o->fn[PENCIL_HA_LAST] = nullptr;
    }
    o->nt = C::NT;
    o->smem = C::SMEM;
    o->cw = CW;
}

bool pencil_kernels(int nx, int cw, PencilKernels<float> *o)
{
#define LFTS_PENCIL_CW_CASE(a)                                         \
    if (nx == a) {                                                     \
        if (cw == 8) { fill_pencil<float, a, 8>(o); return true; }     \
        if (cw == 16) { fill_pencil<float, a, 16>(o); return true; }   \
        if (cw == 32) { fill_pencil<float, a, 32>(o); return true; }   \
        return false;                                                  \
    }
    LFTS_FOR_EACH_LEN(LFTS_PENCIL_CW_CASE)
#undef LFTS_PENCIL_CW_CASE
    return false;
}

}  // namespace lfts

#define LFTS_PLANE_C_CASE(a, b) \
    if (ny == a && nz == b) { fill_plane_c<float, a, b>(o); return true; }
namespace lfts {
bool plane_c_kernels(int ny, int nz, PlaneKernels<float> *o)
{
    LFTS_FOR_EACH_PAIR(LFTS_PLANE_C_CASE)
    return false;
}
template <typename C>
static void fill_plane3(PlaneKernels<float> *o)
{
    o->fn[PLANE_INIT_W] = plane3_kernel<C, PLANE_INIT_W>;
    o->fn[PLANE_STEP] = plane3_kernel<C, PLANE_STEP>;
    o->fn[PLANE_LAST] = plane3_kernel<C, PLANE_LAST>;
    // the h-in-pencil chain runs on 96 x 96 and 128 x 128 planes
    if constexpr (C::NY == 96 || C::NY == 128)
        o->fn[PLANE_G] = plane3_kernel<C, PLANE_G>;
    else
        o->fn[PLANE_G] = nullptr;
    o->nt = C::NT;
    o->smem = C::SMEM;
}
bool plane3_kernels(int ny, int nz, PlaneKernels<float> *o)
{
    if (ny != nz) return false;
    if (ny == 128) { fill_plane3<Plane3_128>(o); return true; }
    if (ny == 96) { fill_plane3<Plane3_96>(o); return true; }
    if (ny == 64) { fill_plane3<Plane3_64>(o); return true; }
    return false;
}
bool plane_split_kernel(int ny, int nz, PlaneSplitKernel *o)
{
    if (ny != 128 || nz != 128) return false;
    o->fn = plane3_split_g_kernel<Plane3Split128>;
    o->cl = Plane3Split128::CL;
    o->nt = Plane3Split128::NT;
    o->smem = Plane3Split128::SMEM;
    return true;
}
}  // namespace lfts
