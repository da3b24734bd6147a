// The host entry points of one compile-time radix FWIX_FLEX_RT (flex.cuh): the
// lengths of FWIX_FLEX_FIXED, listed as X(ra, rb), run kernels compiled for their
// radices, those of FWIX_FLEX_ROWS only their row passes (their columns have a
// compile-time plan), every other one the kernels with run-time radices.
//
// Kernels of their own have every two-stage length from 48 up and ten three-stage lengths
// between 250 and 504 that round grid sizes and paddings give: a depth step and adjoint
// of both kinds on n x n takes 1.2 - 1.7 times as long with the run-time radices on two
// stages, 1.45 - 1.95 times on three (144: 447 us and 596; 336: 551 and 967; row passes alone,
// 128: 349 and 456).  A length's kernels cost some ten seconds of compilation and half a
// megabyte, so the shorter lengths, whose steps are bound by launches, and the other
// three-stage ones run the run-time radices, there 1.15 - 3.2 times as fast as the per-warp
// passes of spectral.cu (147: 1015 us and 1207; 486: 926 and 1894; 1024: 1388 and 4174).
//
// A file that includes this is compiled once as it is (the dispatch and the run-time
// radices) and once more for every listed length, with FWIX_FLEX_RA and FWIX_FLEX_RB
// defined (pyfwix_b200/build.py): a length's kernels are a module of their own, so that a
// program loads those of its own lengths and not those of the whole radix.
#include "flex.cuh"

#ifndef FWIX_FLEX_ROWS
#define FWIX_FLEX_ROWS
#endif

#define FWIX_FLEX_JOIN2(a, b) a##b
#define FWIX_FLEX_JOIN(a, b) FWIX_FLEX_JOIN2(a, b)
#define FWIX_FLEX_ROW_PASSES(KW, ra_, rb_)                                                                         \
  KW template cudaError_t row_forward_s<Fixed<FWIX_FLEX_RT, ra_, rb_>>(const SpecArgs&, const Line&, int, cudaStream_t); \
  KW template cudaError_t row_inverse_s<Fixed<FWIX_FLEX_RT, ra_, rb_>>(const SpecArgs&, const Line&, int, int,     \
                                                                       cudaStream_t);
#define FWIX_FLEX_COL_PASSES(KW, ra_, rb_)                                                                         \
  KW template cudaError_t col_type_a_s<Fixed<FWIX_FLEX_RT, ra_, rb_>>(const SpecArgs&, const Line&, int, cudaStream_t);  \
  KW template cudaError_t col_type_b_s<Fixed<FWIX_FLEX_RT, ra_, rb_>>(const SpecArgs&, const Line&, int, cudaStream_t);

namespace fwix {
namespace flex {

#ifdef FWIX_FLEX_RA

FWIX_FLEX_ROW_PASSES(, FWIX_FLEX_RA, FWIX_FLEX_RB)
#ifndef FWIX_FLEX_ROWS_ONLY
FWIX_FLEX_COL_PASSES(, FWIX_FLEX_RA, FWIX_FLEX_RB)
#endif

#else

#define X(ra_, rb_) FWIX_FLEX_ROW_PASSES(extern, ra_, rb_)
FWIX_FLEX_FIXED
FWIX_FLEX_ROWS
#undef X
#define X(ra_, rb_) FWIX_FLEX_COL_PASSES(extern, ra_, rb_)
FWIX_FLEX_FIXED
#undef X

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

#endif

}  // namespace flex
}  // namespace fwix
