// Lines of any other 7-smooth length: the plan of the run-time-length passes
// (flex.cuh) and their host entry points.
#pragma once
#include "internal.h"

namespace fwix {
namespace flex {

// A line of n samples as two or three radix stages (mixed-radix Stockham).  rt is
// the radix a kernel is compiled for, the stage whose samples a thread keeps in
// registers across the terms; ra and rb (1: none) are chosen at run time.  Rows
// run rt, rb, ra forward (rt on the space side, where the weights are applied),
// columns ra, rb, rt (rt on the wavenumber side, where the phase factors are);
// the inverse transforms run the stages in reverse order.
struct Line {
  int n = 0, rt = 0, ra = 0, rb = 1;
};

// Whether length n has such a plan (every 7-smooth length from 14 to 1024 except
// 15, 25, 125, 625 and 875), and the plan.
bool line_plan(int n, Line* out);
inline bool has_plan(int n) {
  Line l;
  return line_plan(n, &l);
}

cudaError_t row_forward(const SpecArgs& a, int pre, cudaStream_t s);
cudaError_t row_inverse(const SpecArgs& a, int post, int post_taper, cudaStream_t s);
cudaError_t col_type_a(const SpecArgs& a, int qmode, cudaStream_t s);
cudaError_t col_type_b(const SpecArgs& a, int qmode, cudaStream_t s);
cudaError_t col_fft(const SpecArgs& a, int inverse, const float2* in, float2* out, int add, float scale,
                    cudaStream_t s);

}  // namespace flex
}  // namespace fwix
