// Run-time-length passes (flex.cuh) with a thread-resident stage of radix 7.
// Kernels of their own: lines of 49, 56, 63, 70, 84, 98, 105, 336, 420, 448, 504 samples.
#define FWIX_FLEX_RT 7
#define FWIX_FLEX_FIXED X(7, 1) X(8, 1) X(9, 1) X(10, 1) X(12, 1) X(14, 1) X(15, 1) X(8, 6) X(10, 6) X(8, 8) X(9, 8)
#include "flex_unit.cuh"
