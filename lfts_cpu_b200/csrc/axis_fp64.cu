// FP64 axis kernels (the FP64 contour chain, the allocation-free contour step).
#include "axis_inst.cuh"

namespace lfts {
bool axis_kernels(int mx, int my, int mz, int cw, AxisSet<double> *o) { return fill_axis<double>(mx, my, mz, cw, o); }

template <int N>
static void step_x(AxisStepSet *o)
{
    using C = StridedCfg<double, N, kLastCw>;
    o->out = {xline_kernel<double, N, kLastCw, AX_OUT, true>, C::NT, C::SMEM, kLastCw};
}

template <int NY, int NZ>
static void step_yz(AxisStepSet *o)
{
    if constexpr (axis_planes<double>(NY, NZ)) {
        using C = PlaneAxCfg<double, NY, NZ>;
        o->first = {planeax_kernel<double, NY, NZ, AX_INIT_Q, true>, C::NT, C::SMEM, 1};
        o->planes = true;
    } else {
        using Z = ZCfg<double, NZ>;
        using Y = StridedCfg<double, NY, kLastCw>;
        o->first = {zline_kernel<double, NZ, AX_INIT_Q, true>, Z::NT, Z::SMEM, Z::NW * Z::LPW};
        o->y = {yline_kernel<double, NY, kLastCw, true>, Y::NT, Y::SMEM, kLastCw};
    }
}

bool axis_step_kernels(int mx, int my, int mz, AxisStepSet *o)
{
    *o = AxisStepSet{};
    bool x = false, yz = false;
#define LFTS_X(n) if (mx == n) { step_x<n>(o); x = true; }
    LFTS_FOR_EACH_LEN(LFTS_X)
#undef LFTS_X
#define LFTS_P(a, b) if (my == a && mz == b) { step_yz<a, b>(o); yz = true; }
    LFTS_FOR_EACH_PAIR(LFTS_P)
#undef LFTS_P
    return x && yz;
}
}  // namespace lfts
