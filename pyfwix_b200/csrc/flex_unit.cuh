// The host entry points of one compile-time radix FWIX_FLEX_RT (flex.cuh): the
// lengths of FWIX_FLEX_FIXED, listed as X(ra, rb), run kernels compiled for their
// radices, those of FWIX_FLEX_ROWS only their row passes (their columns have a
// compile-time plan), every other one the kernels with run-time radices.
#include "flex.cuh"

#ifndef FWIX_FLEX_ROWS
#define FWIX_FLEX_ROWS
#endif

#define FWIX_FLEX_JOIN2(a, b) a##b
#define FWIX_FLEX_JOIN(a, b) FWIX_FLEX_JOIN2(a, b)

namespace fwix {
namespace flex {

#define X(ra_, rb_) \
  if (p.ra == ra_ && p.rb == rb_) return row_forward_s<Fixed<FWIX_FLEX_RT, ra_, rb_>>(a, p, pre, s);
cudaError_t FWIX_FLEX_JOIN(row_forward_, FWIX_FLEX_RT)(const SpecArgs& a, const Line& p, int pre, cudaStream_t s) {
  FWIX_FLEX_FIXED
  FWIX_FLEX_ROWS
  return row_forward_s<Run<FWIX_FLEX_RT>>(a, p, pre, s);
}
#undef X
#define X(ra_, rb_) \
  if (p.ra == ra_ && p.rb == rb_) return row_inverse_s<Fixed<FWIX_FLEX_RT, ra_, rb_>>(a, p, post, pt, s);
cudaError_t FWIX_FLEX_JOIN(row_inverse_, FWIX_FLEX_RT)(const SpecArgs& a, const Line& p, int post, int pt,
                                                       cudaStream_t s) {
  FWIX_FLEX_FIXED
  FWIX_FLEX_ROWS
  return row_inverse_s<Run<FWIX_FLEX_RT>>(a, p, post, pt, s);
}
#undef X
#define X(ra_, rb_) \
  if (p.ra == ra_ && p.rb == rb_) return col_type_a_s<Fixed<FWIX_FLEX_RT, ra_, rb_>>(a, p, q, s);
cudaError_t FWIX_FLEX_JOIN(col_type_a_, FWIX_FLEX_RT)(const SpecArgs& a, const Line& p, int q, cudaStream_t s) {
  FWIX_FLEX_FIXED
  return col_type_a_s<Run<FWIX_FLEX_RT>>(a, p, q, s);
}
#undef X
#define X(ra_, rb_) \
  if (p.ra == ra_ && p.rb == rb_) return col_type_b_s<Fixed<FWIX_FLEX_RT, ra_, rb_>>(a, p, q, s);
cudaError_t FWIX_FLEX_JOIN(col_type_b_, FWIX_FLEX_RT)(const SpecArgs& a, const Line& p, int q, cudaStream_t s) {
  FWIX_FLEX_FIXED
  return col_type_b_s<Run<FWIX_FLEX_RT>>(a, p, q, s);
}
#undef X
// (plain transforms: the run-time radices serve every length)
cudaError_t FWIX_FLEX_JOIN(col_fft_, FWIX_FLEX_RT)(const SpecArgs& a, const Line& p, int inv, const float2* in,
                                                   float2* out, int add, float sc, cudaStream_t s) {
  return col_fft_s<Run<FWIX_FLEX_RT>>(a, p, inv, in, out, add, sc, s);
}

}  // namespace flex
}  // namespace fwix
