// Rows dispatch on NX, columns on NY: compile-time plans (fast.cuh), run-time ones
// (flex.cuh), and the per-warp Stockham passes of spectral.cu for the few lengths
// that have neither.
#include "flex.h"
#include "internal.h"

#define FWIX_FAST_DECL_ROWS(TAG)                                                                       \
  cudaError_t row_forward_##TAG(const SpecArgs& a, int pre, cudaStream_t s);                           \
  cudaError_t row_inverse_##TAG(const SpecArgs& a, int post, int pt, cudaStream_t s);
#define FWIX_FAST_DECL(TAG)                                                                            \
  cudaError_t col_type_a_##TAG(const SpecArgs& a, int q, cudaStream_t s);                              \
  cudaError_t col_type_b_##TAG(const SpecArgs& a, int q, cudaStream_t s);                              \
  cudaError_t col_fft_##TAG(const SpecArgs& a, int inv, const float2* in, float2* out, int add, float sc, \
                            cudaStream_t s);

namespace fwix {
namespace fast {
FWIX_FAST_DECL(64)
FWIX_FAST_DECL(96)
FWIX_FAST_DECL(128)
FWIX_FAST_DECL(160)
FWIX_FAST_DECL(192)
FWIX_FAST_DECL(256)
FWIX_FAST_DECL(320)
FWIX_FAST_DECL(384)
FWIX_FAST_DECL(512)
FWIX_FAST_DECL(640)
FWIX_FAST_DECL_ROWS(256)
}  // namespace fast

bool fast_length(int n) {
  switch (n) {
    case 64:
    case 96:
    case 128:
    case 160:
    case 192:
    case 256:
    case 320:
    case 384:
    case 512:
    case 640:
      return true;
    default:
      return false;
  }
}

bool resident_length(int n) { return fast_length(n) || flex::has_plan(n); }

// Rows run the compile-time plan (fast.cuh) at 256 only, one conflict-free exchange
// in a warp's own shared memory: the Born pair at 256 x 256 x 128 takes 12.6 ms so and
// 13.9 with flex.cuh's rows.  At the other planned lengths flex.cuh's split saves an
// exchange (128 = 8 16 for 8 4 4, 320 = 16 20 for 20 4 4, 384 = 8 8 6 for 12 4 4 2) or its
// CTAs of 128 threads hold more warps (64 = 8 8, 512 = 8 8 8); us per pass at 320 x 320 x
// 80 with six references, compile-time against flex: inverse with labels 185 and 143,
// forward with labels 148 and 101, plain forward 50 and 42; at 384 x 384 x 96 the
// smooth step's 308 and 233, its adjoint's 252 and 198; the packed Born pair at
// 512 x 512 x 64 27.9 and 26.7 ms.
cudaError_t row_forward(const SpecArgs& a, int pre, cudaStream_t s) {
  switch (a.d.NX) {
    case 256: return fast::row_forward_256(a, pre, s);
    default: return flex::has_plan(a.d.NX) ? flex::row_forward(a, pre, s) : generic_row_forward(a, pre, s);
  }
}

cudaError_t row_inverse(const SpecArgs& a, int post, int post_taper, cudaStream_t s) {
  switch (a.d.NX) {
    case 256: return fast::row_inverse_256(a, post, post_taper, s);
    default: return flex::has_plan(a.d.NX) ? flex::row_inverse(a, post, post_taper, s) : generic_row_inverse(a, post, post_taper, s);
  }
}

cudaError_t col_type_a(const SpecArgs& a, int qmode, cudaStream_t s) {
  switch (a.d.NY) {
    case 64: return fast::col_type_a_64(a, qmode, s);
    case 96: return fast::col_type_a_96(a, qmode, s);
    case 128: return fast::col_type_a_128(a, qmode, s);
    case 160: return fast::col_type_a_160(a, qmode, s);
    case 192: return fast::col_type_a_192(a, qmode, s);
    case 256: return fast::col_type_a_256(a, qmode, s);
    case 320: return fast::col_type_a_320(a, qmode, s);
    case 384: return fast::col_type_a_384(a, qmode, s);
    case 512: return fast::col_type_a_512(a, qmode, s);
    case 640: return fast::col_type_a_640(a, qmode, s);
    default: return flex::has_plan(a.d.NY) ? flex::col_type_a(a, qmode, s) : generic_col_type_a(a, qmode, s);
  }
}

cudaError_t col_type_b(const SpecArgs& a, int qmode, cudaStream_t s) {
  switch (a.d.NY) {
    case 64: return fast::col_type_b_64(a, qmode, s);
    case 96: return fast::col_type_b_96(a, qmode, s);
    case 128: return fast::col_type_b_128(a, qmode, s);
    case 160: return fast::col_type_b_160(a, qmode, s);
    case 192: return fast::col_type_b_192(a, qmode, s);
    case 256: return fast::col_type_b_256(a, qmode, s);
    case 320: return fast::col_type_b_320(a, qmode, s);
    case 384: return fast::col_type_b_384(a, qmode, s);
    case 512: return fast::col_type_b_512(a, qmode, s);
    case 640: return fast::col_type_b_640(a, qmode, s);
    default: return flex::has_plan(a.d.NY) ? flex::col_type_b(a, qmode, s) : generic_col_type_b(a, qmode, s);
  }
}

cudaError_t col_fft(const SpecArgs& a, int inverse, const float2* in, float2* out, int add, float scale,
                    cudaStream_t s) {
  switch (a.d.NY) {
    case 64: return fast::col_fft_64(a, inverse, in, out, add, scale, s);
    case 96: return fast::col_fft_96(a, inverse, in, out, add, scale, s);
    case 128: return fast::col_fft_128(a, inverse, in, out, add, scale, s);
    case 160: return fast::col_fft_160(a, inverse, in, out, add, scale, s);
    case 192: return fast::col_fft_192(a, inverse, in, out, add, scale, s);
    case 256: return fast::col_fft_256(a, inverse, in, out, add, scale, s);
    case 320: return fast::col_fft_320(a, inverse, in, out, add, scale, s);
    case 384: return fast::col_fft_384(a, inverse, in, out, add, scale, s);
    case 512: return fast::col_fft_512(a, inverse, in, out, add, scale, s);
    case 640: return fast::col_fft_640(a, inverse, in, out, add, scale, s);
    default: return flex::has_plan(a.d.NY) ? flex::col_fft(a, inverse, in, out, add, scale, s) : generic_col_fft(a, inverse, in, out, add, scale, s);
  }
}

}  // namespace fwix
