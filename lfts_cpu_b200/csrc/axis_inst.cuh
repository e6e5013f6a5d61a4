// Instantiation of the axis kernels, shared by axis_fp64.cu / axis_fp32.cu.
#pragma once
#include "axis_dispatch.h"
#include "fft_lengths.h"

namespace lfts {

template <typename T, int N, int CW>
static void fill_x(AxisSet<T> *o)
{
    using C = StridedCfg<T, N, CW>;
    using L = StridedCfg<T, N, kLastCw>;
    o->x[AX_H] = {xline_kernel<T, N, CW, AX_H>, C::NT, C::SMEM, CW};
    o->x[AX_H_LAST] = {xline_kernel<T, N, kLastCw, AX_H_LAST>, L::NT, L::SMEM, kLastCw};
    o->x[AX_OUT] = {xline_kernel<T, N, kLastCw, AX_OUT>, L::NT, L::SMEM, kLastCw};
    if constexpr (kAxisSums<T, N>) {
        o->x[AX_HA] = {xline_kernel<T, N, CW, AX_HA>, C::NT, C::SMEM, CW};
        o->x[AX_HA_LAST] = {xline_kernel<T, N, kLastCw, AX_HA_LAST>, L::NT, L::SMEM, kLastCw};
    }
}

template <typename T, int N, int CW>
static void fill_y(AxisSet<T> *o)
{
    using C = StridedCfg<T, N, CW>;
    o->y = {yline_kernel<T, N, CW>, C::NT, C::SMEM, CW};
}

template <typename T, int N>
static void fill_z(AxisSet<T> *o)
{
    using C = ZCfg<T, N>;
    constexpr int per = C::NW * C::LPW;
    o->z[AX_INIT_W] = {zline_kernel<T, N, AX_INIT_W>, C::NT, C::SMEM, per};
    o->z[AX_INIT_Q] = {zline_kernel<T, N, AX_INIT_Q>, C::NT, C::SMEM, per};
    o->z[AX_H] = {zline_kernel<T, N, AX_H>, C::NT, C::SMEM, per};
    o->z[AX_H_LAST] = {zline_kernel<T, N, AX_H_LAST>, C::NT, C::SMEM, per};
    if constexpr (kAxisSums<T, N>) {
        o->z[AX_HA] = {zline_kernel<T, N, AX_HA>, C::NT, C::SMEM, per};
        o->z[AX_HA_LAST] = {zline_kernel<T, N, AX_HA_LAST>, C::NT, C::SMEM, per};
    }
}

template <typename T, int NY, int NZ>
static void fill_plane(AxisSet<T> *o)
{
    if constexpr (axis_planes<T>(NY, NZ)) {
        using C = PlaneAxCfg<T, NY, NZ>;
        o->plane[AX_INIT_W] = {planeax_kernel<T, NY, NZ, AX_INIT_W>, C::NT, C::SMEM, 1};
        o->plane[AX_INIT_Q] = {planeax_kernel<T, NY, NZ, AX_INIT_Q>, C::NT, C::SMEM, 1};
        o->plane[AX_H] = {planeax_kernel<T, NY, NZ, AX_H>, C::NT, C::SMEM, 1};
        o->plane[AX_H_LAST] = {planeax_kernel<T, NY, NZ, AX_H_LAST>, C::NT, C::SMEM, 1};
        o->planes = true;
    }
}

template <typename T>
static bool fill_axis(int mx, int my, int mz, int cw, AxisSet<T> *o)
{
    *o = AxisSet<T>{};
    o->cw = cw;
    bool x = false, p = false;
#define LFTS_X(n)                                      \
    if (mx == n) {                                     \
        x = true;                                      \
        if (cw == 8) fill_x<T, n, 8>(o);               \
        else if (cw == 16) fill_x<T, n, 16>(o);        \
        else if (cw == 32) fill_x<T, n, 32>(o);        \
        else return false;                             \
    }
    LFTS_FOR_EACH_LEN(LFTS_X)
#undef LFTS_X
#define LFTS_P(a, b)                                   \
    if (my == a && mz == b) {                          \
        p = true;                                      \
        if constexpr (axis_planes<T>(a, b)) {             \
            fill_plane<T, a, b>(o);                    \
        } else {                                       \
            if (cw == 8) fill_y<T, a, 8>(o);           \
            else if (cw == 16) fill_y<T, a, 16>(o);    \
            else fill_y<T, a, 32>(o);                  \
            fill_z<T, b>(o);                           \
        }                                              \
    }
    LFTS_FOR_EACH_PAIR(LFTS_P)
#undef LFTS_P
    return x && p;
}

}  // namespace lfts
