// Run-time-length passes (flex.cuh) with a thread-resident stage of radix 10.
// Kernels of their own: lines of 50, 60, 100, 120, 140, 150, 200, 250, 500 samples.
#define FWIX_FLEX_RT 10
#define FWIX_FLEX_FIXED X(5, 1) X(6, 1) X(10, 1) X(12, 1) X(14, 1) X(15, 1) X(20, 1) X(5, 5) X(10, 5)
// Row passes: lines of 160 samples.
#define FWIX_FLEX_ROWS X(16, 1)
#include "flex_unit.cuh"
