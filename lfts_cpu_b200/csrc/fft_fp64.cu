// FP64 forward-transform kernels: S(k) samples and the adjoint.
#include "fft_dispatch.h"
#include "fft_lengths.h"

namespace lfts {

bool fwd_plane_kernel(int ny, int nz, PlaneKernel *o)
{
#define LFTS_PLANE_CASE(a, b)                                                                  \
    if (ny == a && nz == b) {                                                                  \
        *o = {fwd_plane_kernel_t<a, b>, PlaneCfg<double, a, b>::NT, PlaneCfg<double, a, b>::SMEM}; \
        return true;                                                                           \
    }
    LFTS_FOR_EACH_PAIR(LFTS_PLANE_CASE)
#undef LFTS_PLANE_CASE
    return false;
}

bool power_pencil_kernel(int nx, PencilKernel *o)
{
    constexpr int CW = 32;
#define LFTS_POWER_CASE(a)                                                                \
    if (nx == a) {                                                                        \
        using C = PencilCfg<double, a, CW>;                                               \
        *o = {pencil_kernel<double, a, CW, PENCIL_POWER>, C::NT, C::SMEM, CW};            \
        return true;                                                                      \
    }
    LFTS_FOR_EACH_LEN(LFTS_POWER_CASE)
#undef LFTS_POWER_CASE
    return false;
}

bool adjoint_kernel(int nx, AdjKernel *o)
{
    constexpr int CW = 16;
#define LFTS_ADJ_CASE(a)                                       \
    if (nx == a) {                                             \
        o->fn = pencil_adj_kernel<a, CW>;                      \
        o->nt = AdjCfg<a, CW>::NT;                             \
        o->smem = AdjCfg<a, CW>::SMEM;                         \
        o->cw = CW;                                            \
        return true;                                           \
    }
    LFTS_FOR_EACH_LEN(LFTS_ADJ_CASE)
#undef LFTS_ADJ_CASE
    return false;
}

bool fft_length_supported(int n)
{
#define LFTS_LEN_CASE(a) if (n == a) return true;
    LFTS_FOR_EACH_LEN(LFTS_LEN_CASE)
#undef LFTS_LEN_CASE
    return false;
}
bool plane_pair_supported(int ny, int nz)
{
#define LFTS_PAIR_CASE(a, b) if (ny == a && nz == b) return true;
    LFTS_FOR_EACH_PAIR(LFTS_PAIR_CASE)
#undef LFTS_PAIR_CASE
    return false;
}

}  // namespace lfts
