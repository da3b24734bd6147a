// Run-time-length passes (flex.cuh) with a thread-resident stage of radix 15.
// Kernels of their own: lines of 75, 225, 240, 270, 300 samples.
#define FWIX_FLEX_RT 15
#define FWIX_FLEX_FIXED X(5, 1) X(15, 1) X(16, 1) X(18, 1) X(20, 1)
#include "flex_unit.cuh"
