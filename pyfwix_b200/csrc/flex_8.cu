// Run-time-length passes (flex.cuh) with a thread-resident stage of radix 8.
// Kernels of their own: lines of 48, 72, 80, 112, 360, 400, 432, 480 samples.
#define FWIX_FLEX_RT 8
#define FWIX_FLEX_FIXED X(6, 1) X(9, 1) X(10, 1) X(14, 1) X(9, 5) X(10, 5) X(9, 6) X(10, 6)
#include "flex_unit.cuh"
