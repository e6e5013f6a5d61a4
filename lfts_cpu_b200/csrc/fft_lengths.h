// Mesh sizes with compiled kernels.
#pragma once

// line lengths (each needs an AxPlan<> in axis_conv.cuh and a Plan<> in dft.cuh)
#define LFTS_FOR_EACH_LEN(X) X(8) X(12) X(16) X(20) X(24) X(32) X(40) X(48) X(64) X(80) X(96) X(128)
// (ny, nz) plane pairs: the cubic ones plus a few boxes used by tests
#define LFTS_FOR_EACH_PAIR(X)                                                                  \
    X(8, 8) X(12, 12) X(16, 16) X(20, 20) X(24, 24) X(32, 32) X(40, 40) X(48, 48) X(64, 64)   \
    X(80, 80) X(96, 96) X(128, 128) X(12, 20) X(24, 16) X(16, 32) X(32, 64)
