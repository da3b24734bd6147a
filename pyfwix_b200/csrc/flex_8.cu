// Run-time-length passes (flex.cuh) with a thread-resident stage of radix 8.
// Kernels of their own: lines of 48, 72, 80, 112, 360, 400, 432, 480 samples.
#define FWIX_FLEX_RT 8
#define FWIX_FLEX_FIXED X(6, 1) X(9, 1) X(10, 1) X(14, 1) X(9, 5) X(10, 5) X(9, 6) X(10, 6)
// Row passes: lines of 64, 96, 128, 384, 512, 640 samples.
#define FWIX_FLEX_ROWS X(8, 1) X(8, 8) X(12, 1) X(16, 1) X(8, 6) X(10, 8)
#include "flex_unit.cuh"
