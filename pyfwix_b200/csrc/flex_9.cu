// Run-time-length passes (flex.cuh) with a thread-resident stage of radix 9.
// Kernels of their own: lines of 54, 81, 90, 108, 126, 135, 162 samples.
#define FWIX_FLEX_RT 9
#define FWIX_FLEX_FIXED X(6, 1) X(9, 1) X(10, 1) X(12, 1) X(14, 1) X(15, 1) X(18, 1)
#include "flex_unit.cuh"
