// Run-time-length passes (flex.cuh) with a thread-resident stage of radix 14.
// Kernels of their own: lines of 196, 210, 224, 252, 280 samples.
#define FWIX_FLEX_RT 14
#define FWIX_FLEX_FIXED X(14, 1) X(15, 1) X(16, 1) X(18, 1) X(20, 1)
#include "flex_unit.cuh"
