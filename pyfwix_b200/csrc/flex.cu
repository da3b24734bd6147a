// Plans of the run-time-length lines (flex.h) and their dispatch on the
// compile-time radix.
#include "flex.h"

#include <vector>

#define FWIX_FLEX_DECL(RT)                                                                              \
  cudaError_t row_forward_##RT(const SpecArgs& a, const Line& p, int pre, cudaStream_t s);              \
  cudaError_t row_inverse_##RT(const SpecArgs& a, const Line& p, int post, int pt, cudaStream_t s);     \
  cudaError_t col_type_a_##RT(const SpecArgs& a, const Line& p, int q, cudaStream_t s);                 \
  cudaError_t col_type_b_##RT(const SpecArgs& a, const Line& p, int q, cudaStream_t s);                 \
  cudaError_t col_fft_##RT(const SpecArgs& a, const Line& p, int inv, const float2* in, float2* out, int add, \
                           float sc, cudaStream_t s);
#define FWIX_FLEX_DISPATCH(RT, FN, ...) \
  switch (RT) {                         \
    case 7: return FN##_7(__VA_ARGS__); \
    case 8: return FN##_8(__VA_ARGS__); \
    case 9: return FN##_9(__VA_ARGS__); \
    case 10: return FN##_10(__VA_ARGS__); \
    case 12: return FN##_12(__VA_ARGS__); \
    case 14: return FN##_14(__VA_ARGS__); \
    case 15: return FN##_15(__VA_ARGS__); \
    case 16: return FN##_16(__VA_ARGS__); \
    default: return cudaErrorInvalidValue; \
  }

namespace fwix {
namespace flex {

FWIX_FLEX_DECL(7)
FWIX_FLEX_DECL(8)
FWIX_FLEX_DECL(9)
FWIX_FLEX_DECL(10)
FWIX_FLEX_DECL(12)
FWIX_FLEX_DECL(14)
FWIX_FLEX_DECL(15)
FWIX_FLEX_DECL(16)

namespace {

bool find_plan(int n, Line* out) {
  static const int rts[] = {7, 8, 9, 10, 12, 14, 15, 16};
  static const int ras[] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16, 18, 20};
  static const int mids[] = {5, 6, 7, 8, 9, 10, 12, 14, 15, 16};
  Line best;
  int spread = 1 << 30;
  // two stages (one exchange per transform) where the length allows, else three;
  // of those the most even split (the largest radix sets the registers, the smallest
  // the threads), with the smaller radix where the samples stay in registers
  for (int rt : rts) {
    for (int ra : ras) {
      if (rt * ra != n) continue;
      const int d = rt > ra ? rt - ra : ra - rt;
      if (d < spread) {
        spread = d;
        best.n = n, best.rt = rt, best.ra = ra, best.rb = 1;
      }
    }
  }
  if (!best.n) {
    for (int rt : rts)
      for (int rb : mids)
        for (int ra : ras) {
          if (rt * rb * ra != n) continue;
          int lo = rt < rb ? rt : rb, hi = rt < rb ? rb : rt;
          lo = lo < ra ? lo : ra, hi = hi > ra ? hi : ra;
          if (hi - lo < spread) {
            spread = hi - lo;
            best.n = n, best.rt = rt, best.ra = ra, best.rb = rb;
          }
        }
  }
  if (!best.n) return false;
  *out = best;
  return true;
}

}  // namespace

bool line_plan(int n, Line* out) {
  // all lengths once: the launches look their plan up
  static const std::vector<Line> plans = [] {
    std::vector<Line> v(FWIX_MAX_N + 1);
    for (int i = 1; i <= FWIX_MAX_N; ++i) find_plan(i, &v[i]);
    return v;
  }();
  if (n < 1 || n > FWIX_MAX_N || !plans[n].n) return false;
  *out = plans[n];
  return true;
}

cudaError_t row_forward(const SpecArgs& a, int pre, cudaStream_t s) {
  Line p;
  if (!line_plan(a.d.NX, &p)) return cudaErrorInvalidValue;
  FWIX_FLEX_DISPATCH(p.rt, row_forward, a, p, pre, s)
}
cudaError_t row_inverse(const SpecArgs& a, int post, int post_taper, cudaStream_t s) {
  Line p;
  if (!line_plan(a.d.NX, &p)) return cudaErrorInvalidValue;
  FWIX_FLEX_DISPATCH(p.rt, row_inverse, a, p, post, post_taper, s)
}
cudaError_t col_type_a(const SpecArgs& a, int qmode, cudaStream_t s) {
  Line p;
  if (!line_plan(a.d.NY, &p)) return cudaErrorInvalidValue;
  FWIX_FLEX_DISPATCH(p.rt, col_type_a, a, p, qmode, s)
}
cudaError_t col_type_b(const SpecArgs& a, int qmode, cudaStream_t s) {
  Line p;
  if (!line_plan(a.d.NY, &p)) return cudaErrorInvalidValue;
  FWIX_FLEX_DISPATCH(p.rt, col_type_b, a, p, qmode, s)
}
cudaError_t col_fft(const SpecArgs& a, int inverse, const float2* in, float2* out, int add, float scale,
                    cudaStream_t s) {
  Line p;
  if (!line_plan(a.d.NY, &p)) return cudaErrorInvalidValue;
  FWIX_FLEX_DISPATCH(p.rt, col_fft, a, p, inverse, in, out, add, scale, s)
}

}  // namespace flex
}  // namespace fwix
