// FP64 axis kernels (the FP64 contour chain, the allocation-free contour step).
#include "axis_inst.cuh"

namespace lfts {
bool axis_kernels(int mx, int my, int mz, int cw, AxisSet<double> *o) { return fill_axis<double>(mx, my, mz, cw, o); }
}  // namespace lfts
