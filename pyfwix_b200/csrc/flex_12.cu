// Run-time-length passes (flex.cuh) with a thread-resident stage of radix 12.
// Kernels of their own: lines of 144, 168, 180, 216 samples.
#define FWIX_FLEX_RT 12
#define FWIX_FLEX_FIXED X(12, 1) X(14, 1) X(15, 1) X(18, 1)
// Row passes: lines of 192 samples.
#define FWIX_FLEX_ROWS X(16, 1)
#include "flex_unit.cuh"
