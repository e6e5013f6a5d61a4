// The compiled axis kernels (axis_conv.cuh) of one mesh, looked up by size:
// axis_fp64.cu and axis_fp32.cu instantiate them.
#pragma once
#include "axis_conv.cuh"

namespace lfts {

template <typename T>
struct AxisFn {
    void (*fn)(AxisArgs<T>);  // null: not compiled
    int nt;
    size_t smem;
    int per;  // x, y: columns per CTA; z: lines per CTA; plane: 1 (the plane)
};

template <typename T>
struct AxisSet {
    AxisFn<T> x[kAxisModes], y, z[kAxisModes], plane[kAxisModes];
    bool planes;  // [Cy Cz h Cz Cy] in one kernel; else z lines and y lines apart
    int cw;
};

// fills *o for an mx x my x mz mesh with x and y tiles of cw columns (8, 16, 32);
// false without kernels for it
bool axis_kernels(int mx, int my, int mz, int cw, AxisSet<double> *o);
bool axis_kernels(int mx, int my, int mz, int cw, AxisSet<float> *o);

// The kernels of one contour step on the caller's arrays that make their own
// tables (FP64): z lines or planes from the caller's rows, y lines, x lines out
struct AxisStepSet {
    AxisFn<double> first, y, out;
    bool planes;
};
bool axis_step_kernels(int mx, int my, int mz, AxisStepSet *o);

// Columns per CTA of the x-line kernel that ends a chain, whatever the tile
// choice: its CTAs' partial sums for Q then do not depend on the tiles.
constexpr int kLastCw = 16;

// Whether y and z lines share a kernel, one CTA per x-plane (and FP64 chain): one
// launch less a step while a CTA has little of a plane to work through.  Chain with
// one kernel / two, N = 64, us: 32^3 FP64 194 / 285, 40^3 267 / 315, FP32 221 / 244;
// 48^3 FP64 385 / 322, 64^3 FP32 363 / 273.  FP64 planes of 64 x 64, whose stages
// are all of 8 points and fill their warps: calc_concs 467 / 476, with 128 of them
// 710 / 765.
template <typename T>
constexpr bool axis_planes(int my, int mz)
{
    return my * mz <= 2048 || (!kPairs<T> && my == 64 && mz == 64);
}

}  // namespace lfts
