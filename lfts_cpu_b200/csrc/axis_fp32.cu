// FP32 axis kernels (the FP32-mixed contour chain).
#include "axis_inst.cuh"

namespace lfts {
bool axis_kernels(int mx, int my, int mz, int cw, AxisSet<float> *o) { return fill_axis<float>(mx, my, mz, cw, o); }
}  // namespace lfts
