// Run-time-length passes (flex.cuh) with a thread-resident stage of radix 16.
// Kernels of their own: lines of 288 samples.
#define FWIX_FLEX_RT 16
#define FWIX_FLEX_FIXED X(18, 1)
// Row passes: lines of 320 samples.
#define FWIX_FLEX_ROWS X(20, 1)
#include "flex_unit.cuh"
