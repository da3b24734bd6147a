// Row and column passes for line lengths without a compile-time plan (fast.cuh):
// any 7-smooth length that splits into two or three radix stages (flex.h).
//
// A CTA owns a group of lines and runs every stage over all of its threads, one
// butterfly per thread and turn; the samples cross shared memory once per
// stage boundary (two-stage lines: one exchange per transform, as in the
// compile-time plans).  The first stage reads HBM, and the last one writes it,
// straight from registers.  One stage, of the compile-time radix RT, has a fixed
// butterfly per thread, so that what must live across the terms of a pass (the
// row's samples, the sum over references, the column's spectrum) stays in
// registers; the other stages' radices are uniform run-time switches.
//
// Rows: lanes run along the line, so HBM is read in row segments; between the
// stages a line is a matrix of odd pitch (RowPlace), free of bank conflicts.
// Columns: a tile of LX neighbouring columns is kept row by row, and
// lanes run across the columns, so that every access of every stage, whatever
// its stride, is a contiguous 8 LX bytes (no bank conflicts without a swizzle)
// and HBM is touched in segments of the same length.
//
// What bounds them: the latency of a term's global loads at 14 - 24 warps per SM, then
// the L1 data pipe (8-byte accesses), 20 - 37 % of DRAM bandwidth.  us per pass, with
// the per-warp passes of spectral.cu that these replace (7 to 9 shared-memory crossings
// per sample and term, radix 8 at most, a part of the lanes idle): PSPI continuation and
// its adjoint over six levels at 200 x 168 x 40 1569 -> 720; four uneven shots (270, 216,
// 160, 135) imaged 11580 -> 5830; the Born pair at 135 x 120 x 40 on two shots 6240 ->
// 3060.
#pragma once
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <utility>

#include "flex.h"
#include "ops.cuh"

namespace fwix {
namespace flex {

constexpr int kMaxThreads = 512;

// Geometry of a launch (kernel parameter; what a Fixed line knows is not read).
struct Geo {
  int n;           // line length
  int ra, rb;      // run-time radices (rb 1: two stages)
  int nt, na, nb;  // butterflies per line of the stages RT, ra, rb
  int lines;       // lines per CTA (columns: a power of two)
  int sh;          // columns: log2(lines)
  int nchunk;      // CTAs per slice
  unsigned mt, ma, mb;  // multipliers of q = idx / n{t,a,b} as umulhi(idx, m)
};

// Rows per CTA (about 128 threads) and columns per CTA (16, whole 128-byte lines,
// while the tile takes at most 160 threads, else 8 or fewer) of a line whose stage
// RT has nt butterflies.  Small CTAs: every stage ends in a CTA barrier, so that
// several CTAs at different stages keep an SM busy, and the last wave is short.
constexpr int row_lines(int nt) { return 128 / nt < 1 ? 1 : 128 / nt > 64 ? 64 : 128 / nt; }
constexpr int col_shift(int nt) {
  int sh = nt * 16 <= 160 ? 4 : 3;
  while (sh > 1 && (nt << sh) > kMaxThreads) --sh;
  return sh;
}
// Twiddles of the stages in the order A, B, C (fill_twiddles).
constexpr int table_size(int A, int B, int C) { return (B - 1) * A + (C - 1) * A * B; }

// A line whose radices are known at compile time (the lengths listed in
// flex_*.cu): registers are those of its own radices and every index is a
// constant or a multiplication by one.
template <int RT_, int RA_, int RB_>
struct Fixed {
  static constexpr bool kFixed = true;
  static constexpr int RT = RT_, RA = RA_, RB = RB_, N = RT_ * RA_ * RB_;
  static constexpr int NT = N / RT, NA = N / RA, NB = N / RB;
  static constexpr int ROW_LINES = row_lines(NT), COL_SH = col_shift(NT);
  static constexpr int ROW_THREADS = (ROW_LINES * NT + 31) / 32 * 32;
  static constexpr int COL_THREADS = ((NT << COL_SH) + 31) / 32 * 32;
  static constexpr int MAXR = RT > RA ? (RT > RB ? RT : RB) : (RA > RB ? RA : RB);
};
// A line with run-time radices ra, rb.
template <int RT_>
struct Run {
  static constexpr bool kFixed = false;
  static constexpr int RT = RT_;
  static constexpr int ROW_THREADS = kMaxThreads, COL_THREADS = kMaxThreads, MAXR = 20;
};

__device__ __forceinline__ int fdiv(int i, unsigned m) { return (int)__umulhi((unsigned)i, m); }

// The line's numbers, from the type where it has them, else from the geometry.
template <class S>
struct Dim {
  const Geo& g;
#define FWIX_FLEX_NUM(name, fixed, run)              \
  __device__ __forceinline__ int name() const {      \
    if constexpr (S::kFixed) return fixed;           \
    else return run;                                 \
  }
  FWIX_FLEX_NUM(n, S::N, g.n)
  FWIX_FLEX_NUM(ra, S::RA, g.ra)
  FWIX_FLEX_NUM(rb, S::RB, g.rb)
  FWIX_FLEX_NUM(nt, S::NT, g.nt)
  FWIX_FLEX_NUM(na, S::NA, g.na)
  FWIX_FLEX_NUM(nb, S::NB, g.nb)
  FWIX_FLEX_NUM(rows, S::ROW_LINES, g.lines)
  FWIX_FLEX_NUM(row_threads, S::ROW_THREADS, blockDim.x)
  FWIX_FLEX_NUM(sh, S::COL_SH, g.sh)
  FWIX_FLEX_NUM(col_threads, S::COL_THREADS, blockDim.x)
  FWIX_FLEX_NUM(cols, 1 << S::COL_SH, g.lines)
  FWIX_FLEX_NUM(fwd_rows_tw, table_size(S::RT, S::RB, S::RA), (g.rb - 1) * S::RT + (g.ra - 1) * g.na)
  FWIX_FLEX_NUM(inv_rows_tw, table_size(S::RA, S::RB, S::RT), (g.rb - 1) * g.ra + (S::RT - 1) * g.nt)
#undef FWIX_FLEX_NUM
  __device__ __forceinline__ int div_nt(int i) const {
    if constexpr (S::kFixed) return (unsigned)i / (unsigned)S::NT;
    else return fdiv(i, g.mt);
  }
  __device__ __forceinline__ int div_na(int i) const {
    if constexpr (S::kFixed) return (unsigned)i / (unsigned)S::NA;
    else return fdiv(i, g.ma);
  }
  __device__ __forceinline__ int div_nb(int i) const {
    if constexpr (S::kFixed) return (unsigned)i / (unsigned)S::NB;
    else return fdiv(i, g.mb);
  }
};

// Resident CTAs that a Fixed line's registers are held to.  `sets` counts what a
// thread holds across a stage of the largest radix, in units of RT registers (a
// complex set is 2, labels or hat indices 1); with that stage's samples and some
// 30 registers of addresses and temporaries it bounds the threads an SM can hold.
template <class S>
constexpr int min_blocks(int threads, int sets) {
  if constexpr (!S::kFixed) {
    return 1;
  } else {
    const int regs = (32 + sets * S::RT + 2 * S::MAXR + 7) / 8 * 8;
    const int fit = 65536 / (regs * threads);
    const int most = 1536 / threads;  // (more warps than that never paid)
    return fit < 1 ? 1 : fit > most ? (most < 1 ? 1 : most) : fit;
  }
}

// Calls f(std::integral_constant<int, R>) for the run-time radix R.
template <class F>
__device__ __forceinline__ void with_radix(int R, F&& f) {
#define FWIX_FLEX_R(r) \
  case r: f(std::integral_constant<int, r>()); break;
  switch (R) {
    FWIX_FLEX_R(2)
    FWIX_FLEX_R(3)
    FWIX_FLEX_R(4)
    FWIX_FLEX_R(5)
    FWIX_FLEX_R(6)
    FWIX_FLEX_R(7)
    FWIX_FLEX_R(8)
    FWIX_FLEX_R(9)
    FWIX_FLEX_R(10)
    FWIX_FLEX_R(12)
    FWIX_FLEX_R(14)
    FWIX_FLEX_R(15)
    FWIX_FLEX_R(16)
    FWIX_FLEX_R(18)
    FWIX_FLEX_R(20)
    default: break;
  }
#undef FWIX_FLEX_R
}
// The same for the middle stage of a three-stage line.
template <class F>
__device__ __forceinline__ void with_mid_radix(int R, F&& f) {
#define FWIX_FLEX_R(r) \
  case r: f(std::integral_constant<int, r>()); break;
  switch (R) {
    FWIX_FLEX_R(5)
    FWIX_FLEX_R(6)
    FWIX_FLEX_R(7)
    FWIX_FLEX_R(8)
    FWIX_FLEX_R(9)
    FWIX_FLEX_R(10)
    FWIX_FLEX_R(12)
    FWIX_FLEX_R(14)
    FWIX_FLEX_R(15)
    FWIX_FLEX_R(16)
    default: break;
  }
#undef FWIX_FLEX_R
}

// The stage of radix ra and the middle stage of line S.
template <class S, class F>
__device__ __forceinline__ void stage_a(const Dim<S>& d, F&& f) {
  if constexpr (S::kFixed) f(std::integral_constant<int, S::RA>());
  else with_radix(d.ra(), f);
}
template <class S, class F>
__device__ __forceinline__ void stage_b(const Dim<S>& d, F&& f) {
  if constexpr (!S::kFixed) with_mid_radix(d.rb(), f);
  else if constexpr (S::RB > 1) f(std::integral_constant<int, S::RB>());
}

template <bool INV>
__device__ __forceinline__ float2 twid(float2 v, float2 w) {
  return INV ? cmul_conj(v, w) : cmul(v, w);
}

// Twiddles of the stages in the order A, B, C from the plain table tw[m] = exp(-2 pi i m / n): radix B with span A,
// W_n^(k r n / (A B)) at (r - 1) A + k, then radix C with span A B, so that
// the lanes of a warp read consecutive entries.
__device__ __forceinline__ void fill_twiddles(float2* dst, const float2* __restrict__ tw, int A, int B, int C,
                                              int nthreads) {
  for (int i = threadIdx.x; i < (B - 1) * A; i += nthreads) {
    const int r = i / A, k = i - r * A;
    dst[i] = tw[k * (r + 1) * C];
  }
  dst += (B - 1) * A;
  const int nc = A * B;
  for (int i = threadIdx.x; i < (C - 1) * nc; i += nthreads) {
    const int r = i / nc, k = i - r * nc;
    dst[i] = tw[k * (r + 1)];
  }
}

// ---------------------------------------------------------------- rows

// Placement of a row's samples between its stages: the line as a matrix whose rows
// are one butterfly of the first stage (its radix P, an even one padded to P + 1).
// The first stage's stores, P apart, then hit different banks, and the next
// stage's loads run along a row.  Lines follow one another without a gap, so that
// the first stage's stores stay conflict-free across lines too.
template <class S, bool INV>
struct RowPlace {
  int P, pitch, ls;
  __device__ __forceinline__ RowPlace(const Dim<S>& d) {
    P = INV ? d.ra() : S::RT;
    pitch = P | 1;
    ls = d.n() / P * pitch;
  }
  __device__ __forceinline__ int first(int j, int r) const { return j * pitch + r; }   // sample j P + r
  __device__ __forceinline__ int at(int p) const { return p + p / P * (pitch - P); }
  // sample j + r m, m butterflies per line of the reading stage (m = P: two stages)
  __device__ __forceinline__ int next(const Dim<S>& d, int j, int r, int m) const {
    return d.rb() == 1 ? j + r * pitch : at(j + r * m);
  }
};
constexpr int row_ls(int n, int P) { return n / P * (P | 1); }

// Middle stage over the CTA's lines, src -> dst; the span is the first stage's radix.
template <bool INV, class S>
__device__ __forceinline__ void row_mid(const Dim<S>& d, const RowPlace<S, INV>& w, const float2* tw,
                                        const float2* src, float2* dst) {
  stage_b(d, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int span = w.P;
    for (int i = threadIdx.x; i < d.rows() * d.nb(); i += d.row_threads()) {
      const int l = d.div_nb(i), j = i - l * d.nb();
      const int q = j / span, k = j - q * span;
      float2 u[R];
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = src[l * w.ls + w.at(j + r * d.nb())];
#pragma unroll
      for (int r = 1; r < R; ++r) u[r] = twid<INV>(u[r], tw[(r - 1) * span + k]);
      Dft<R, INV>::run(u);
#pragma unroll
      for (int r = 0; r < R; ++r) dst[l * w.ls + (q * R + r) * w.pitch + k] = u[r];
    }
  });
}

// Bitwise or over the CTA's threads (every thread calls it, once per kernel).
__device__ __forceinline__ unsigned cta_or(unsigned v) {
  __shared__ unsigned all;
  if (threadIdx.x == 0) all = 0;
  v = __reduce_or_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0 && v) atomicOr(&all, v);
  __syncthreads();
  return all;
}

// What a thread of a row pass works on: line l of the CTA, butterfly j of stage RT.
template <class S>
struct RowCtx {
  int l, j, y, y0, iw;
  bool live;
  long long bl, b;
  __device__ __forceinline__ RowCtx(const SpecArgs& a, const Dim<S>& d) {
    l = d.div_nt(threadIdx.x);
    j = threadIdx.x - l * d.nt();
    bl = blockIdx.x / d.g.nchunk;
    b = a.b0 + bl;
    y0 = (int)(blockIdx.x - bl * d.g.nchunk) * d.rows();
    y = y0 + l;
    live = l < d.rows() && y < a.d.NY;
    iw = (int)(b % a.d.nw);
  }
};

// Classes of row weights that share a kernel (the weight itself is a uniform
// run-time switch within a class).
enum RowClass { C_ONE, C_MASK, C_SCAT, C_SMOOTH, C_PAIR, C_DERIV };
// What a row pass's thread holds across the terms (min_blocks).
constexpr int row_sets(int cls) {
  return cls == C_ONE ? 0 : cls == C_SCAT ? 2 : cls == C_PAIR || cls == C_DERIV ? 5 : 3;
}

// t1[term] = F_x(pre_term * in) for each term.  The row's samples are read once
// into registers; a term whose weight vanishes on all of the CTA's rows (masks,
// smooth weights) is written as zeros.
template <class S, int CLS>
__global__ void __launch_bounds__(S::ROW_THREADS, min_blocks<S>(S::ROW_THREADS, row_sets(CLS)))
    k_row_fwd(const SpecArgs a, const __grid_constant__ Geo g, int pre) {
  constexpr int RT = S::RT;
  const Dim<S> d{g};
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* const buf0 = sm + d.fwd_rows_tw();
  float2* const buf1 = buf0 + d.rows() * row_ls(d.n(), S::RT);
  const RowCtx<S> c(a, d);
  const RowPlace<S, false> w(d);
  if (a.early) chain_next();
  fill_twiddles(tw, a.twx, RT, d.rb(), d.ra(), d.row_threads());
  chain_wait();
  constexpr bool kSmooth = CLS == C_SMOOTH;
  __shared__ typename std::conditional<kSmooth, HatTables, int>::type hat;
  PhaseUnit unit = {0.f, 0.f};
  if constexpr (kSmooth) {
    unit = phase_unit(a, c.iw);
    stage_hat(hat, a, c.iw, unit);
  }
  const long long roff = (c.b * a.d.NY + (c.live ? c.y : 0)) * d.n();
  float2 raw[RT];
#pragma unroll
  for (int r = 0; r < RT; ++r) raw[r] = c.live ? a.in[roff + c.j + r * d.nt()] : make_float2(0.f, 0.f);
  if (a.in2 && c.live) {
#pragma unroll
    for (int r = 0; r < RT; ++r) raw[r] = cadd(raw[r], a.in2[roff + c.j + r * d.nt()]);
  }
  if (CLS == C_ONE || CLS == C_MASK) {
    if (a.rf_at == 1 && c.live && c.y < a.d.ny) {
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const int x = c.j + r * d.nt();
        if (x < a.d.nx) raw[r] = cadd(raw[r], refl_term(a, roff, c.y, x));
      }
    }
  }
  if (CLS == C_ONE && c.live) {
    if (pre == W_TAPER) {
#pragma unroll
      for (int r = 0; r < RT; ++r) raw[r] = row_weight<W_TAPER>(a, 0, c.iw, c.y, c.j + r * d.nt(), raw[r]);
    } else if (pre == W_IC) {
#pragma unroll
      for (int r = 0; r < RT; ++r) raw[r] = row_weight<W_IC>(a, 0, c.iw, c.y, c.j + r * d.nt(), raw[r]);
    }
  }
  int lab[CLS == C_MASK ? RT : 1];
  unsigned used = 0xffffffffu;
  if (CLS == C_MASK) {
    const uint8_t* lrow = a.lab + (long long)c.iw * a.lab_w + (long long)(c.live ? c.y : 0) * d.n();
    unsigned mine = 0;
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      lab[r] = c.live ? lrow[c.j + r * d.nt()] : 255;
      if (lab[r] < 32) mine |= 1u << lab[r];
    }
    used = a.nterm > 32 ? 0xffffffffu : cta_or(mine);
  } else {
    __syncthreads();
  }
  // smooth weights: a cell's place between the references, and the cell part conj(B(s))
  // of every reference's weight once per cell
  HatCells<kSmooth ? RT : 1> hc;
  if constexpr (kSmooth) {
    unsigned mine = 0;
    const float* srow = a.sm_s + (long long)(c.live ? c.y : 0) * d.n();
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const float sv = c.live ? srow[c.j + r * d.nt()] : 0.f;
      const HatPos hp = hat_pos(hat, a.sm_n, sv);
      hc.set(r, hp);
      if (c.live) {
        mine |= hat_support(a.sm_n, hp.j);
        raw[r] = cmul_conj(raw[r], smooth_cell_phase(unit, sv));
      }
    }
    used = cta_or(mine);
  }
  const int nterm = CLS == C_ONE ? 1 : a.nterm;
  int k = 0;  // terms transformed so far
  for (int term = 0; term < nterm; ++term) {
    float2* const dst = a.t1 + (long long)term * a.tstride + (c.bl * a.d.NY + c.y0) * d.n();
    if (!((used >> (term & 31)) & 1u)) {
      const int cnt = min(d.rows(), a.d.NY - c.y0) * d.n();
      for (int i = threadIdx.x; i < cnt; i += d.row_threads()) dst[i] = make_float2(0.f, 0.f);
      continue;
    }
    float2* src = (d.rb() == 1 && (k & 1)) ? buf1 : buf0;
    ++k;
    if (c.l < d.rows()) {
      float2 v[RT];
      if (CLS == C_MASK) {
#pragma unroll
        for (int r = 0; r < RT; ++r) v[r] = lab[r] == term ? raw[r] : make_float2(0.f, 0.f);
      } else if (CLS == C_SCAT) {
#pragma unroll
        for (int r = 0; r < RT; ++r)
          v[r] = c.live ? row_weight<W_SCAT_CONJ>(a, term, c.iw, c.y, c.j + r * d.nt(), raw[r]) : raw[r];
      } else if constexpr (kSmooth) {
        const float2 C = hat.C[term];
#pragma unroll
        for (int r = 0; r < RT; ++r) v[r] = cmul_conj(cscale(raw[r], hc.w(r, term)), C);
      } else {
#pragma unroll
        for (int r = 0; r < RT; ++r) v[r] = raw[r];
      }
      Dft<RT, false>::run(v);
#pragma unroll
      for (int r = 0; r < RT; ++r) src[c.l * w.ls + w.first(c.j, r)] = v[r];
    }
    __syncthreads();
    if (d.rb() > 1) {
      row_mid<false>(d, w, tw, src, buf1);
      __syncthreads();
      src = buf1;
    }
    if (term + 1 == nterm) chain_next();
    const float2* twl = tw + (d.rb() - 1) * RT;
    stage_a(d, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int i = threadIdx.x; i < d.rows() * d.na(); i += d.row_threads()) {
        const int l = d.div_na(i), j = i - l * d.na();
        if (c.y0 + l >= a.d.NY) break;
        float2 u[R];
#pragma unroll
        for (int r = 0; r < R; ++r) u[r] = src[l * w.ls + w.next(d, j, r, d.na())];
#pragma unroll
        for (int r = 1; r < R; ++r) u[r] = cmul(u[r], twl[(r - 1) * d.na() + j]);
        Dft<R, false>::run(u);
#pragma unroll
        for (int r = 0; r < R; ++r) dst[l * d.n() + j + r * d.na()] = u[r];
      }
    });
  }
}

// out (+)= post * sum_term W_term * F_x^-1(t2[term]); terms that no sample of the
// CTA's rows selects are skipped.
template <class S, int CLS>
__global__ void __launch_bounds__(S::ROW_THREADS, min_blocks<S>(S::ROW_THREADS, row_sets(CLS)))
    k_row_inv(const SpecArgs a, const __grid_constant__ Geo g, int post, int post_taper) {
  constexpr int RT = S::RT;
  const Dim<S> d{g};
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* const buf0 = sm + d.inv_rows_tw();
  float2* const buf1 = buf0 + d.rows() * row_ls(d.n(), d.ra());
  const RowCtx<S> c(a, d);
  const RowPlace<S, true> w(d);
  if (a.early) chain_next();
  fill_twiddles(tw, a.twx, d.ra(), d.rb(), RT, d.row_threads());
  chain_wait();
  // kDeriv: the sum of w_r' C_r T_r beside the step's own
  constexpr bool kDeriv = CLS == C_PAIR || CLS == C_DERIV, kSmooth = CLS == C_SMOOTH || kDeriv;
  __shared__ typename std::conditional<kSmooth, HatTables, int>::type hat;
  PhaseUnit unit = {0.f, 0.f};
  if constexpr (kSmooth) {
    unit = phase_unit(a, c.iw);
    stage_hat(hat, a, c.iw, unit);
  }
  float2 acc[RT];
  float2 acc2[kDeriv ? RT : 1];
#pragma unroll
  for (int r = 0; r < RT; ++r) acc[r] = make_float2(0.f, 0.f);
  if constexpr (kDeriv) {
#pragma unroll
    for (int r = 0; r < RT; ++r) acc2[r] = make_float2(0.f, 0.f);
  }
  int lab[CLS == C_MASK ? RT : 1];
  unsigned used = 0xffffffffu;
  if (CLS == C_MASK) {
    const uint8_t* lrow = a.lab + (long long)c.iw * a.lab_w + (long long)(c.live ? c.y : 0) * d.n();
    unsigned mine = 0;
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      lab[r] = c.live ? lrow[c.j + r * d.nt()] : 255;
      if (lab[r] < 32) mine |= 1u << lab[r];
    }
    used = a.nterm > 32 ? 0xffffffffu : cta_or(mine);
  } else {
    __syncthreads();
  }
  HatCells<kSmooth ? RT : 1> hc;
  if constexpr (kSmooth) {
    unsigned mine = 0;
    const float* srow = a.sm_s + (long long)(c.live ? c.y : 0) * d.n();
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      const HatPos hp = hat_pos(hat, a.sm_n, c.live ? srow[c.j + r * d.nt()] : 0.f);
      hc.set(r, hp);
      if (c.live) mine |= hat_support(a.sm_n, hp.j);
    }
    used = cta_or(mine);
  }
  const int nterm = CLS == C_ONE ? 1 : a.nterm;
  int k = 0;
  for (int term = 0; term < nterm; ++term) {
    if (!((used >> (term & 31)) & 1u)) continue;
    float2* src = (d.rb() == 1 && (k & 1)) ? buf1 : buf0;
    ++k;
    const float2* in = a.t2 + (long long)term * a.tstride + (c.bl * a.d.NY + c.y0) * d.n();
    stage_a(d, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      for (int i = threadIdx.x; i < d.rows() * d.na(); i += d.row_threads()) {
        const int l = d.div_na(i), j = i - l * d.na();
        if (c.y0 + l >= a.d.NY) break;
        float2 u[R];
#pragma unroll
        for (int r = 0; r < R; ++r) u[r] = in[l * d.n() + j + r * d.na()];
        Dft<R, true>::run(u);
#pragma unroll
        for (int r = 0; r < R; ++r) src[l * w.ls + w.first(j, r)] = u[r];
      }
    });
    __syncthreads();
    if (d.rb() > 1) {
      row_mid<true>(d, w, tw, src, buf1);
      __syncthreads();
      src = buf1;
    }
    if (!c.live) continue;
    const float2* twl = tw + (d.rb() - 1) * d.ra();
    float2 v[RT];
#pragma unroll
    for (int r = 0; r < RT; ++r) v[r] = src[c.l * w.ls + w.next(d, c.j, r, d.nt())];
#pragma unroll
    for (int r = 1; r < RT; ++r) v[r] = cmul_conj(v[r], twl[(r - 1) * d.nt() + c.j]);
    Dft<RT, true>::run(v);
    if (CLS == C_MASK) {
#pragma unroll
      for (int r = 0; r < RT; ++r)
        if (lab[r] == term) acc[r] = v[r];
    } else if (CLS == C_SCAT) {
#pragma unroll
      for (int r = 0; r < RT; ++r)
        acc[r] = cadd(acc[r], row_weight<W_SCAT>(a, term, c.iw, c.y, c.j + r * d.nt(), v[r]));
    } else if constexpr (kSmooth) {
      // reference part of the weights here, the cell part B(s) once after the sum
      const float2 C = hat.C[term];
      const float below = term > 0 ? hat.inv[term - 1] : 0.f, above = hat.inv[term];
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const float2 u = cmul(v[r], C);
        acc[r] = cfma(u, hc.w(r, term), acc[r]);
        if constexpr (kDeriv) acc2[r] = cfma(u, hc.dw(r, term, below, above), acc2[r]);
      }
    } else {
#pragma unroll
      for (int r = 0; r < RT; ++r) acc[r] = v[r];
    }
  }
  chain_next();
  if (!c.live) return;
  const long long roff = (c.b * a.d.NY + c.y) * d.n();
  const float ty = post_taper ? a.tapy[c.y] : 1.f;
  const float wdz = a.w[c.iw] * a.dz;
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    const int x = c.j + r * d.nt();
    float2 v = acc[r];
    float2 cell = make_float2(1.f, 0.f);
    if constexpr (kSmooth) {
      cell = smooth_cell_phase(unit, a.sm_s[(long long)c.y * d.n() + x]);
      if constexpr (kDeriv) acc2[r] = cfma(rot90<false>(v), wdz, acc2[r]);  // S1 - i w dz S
      v = cmul(CLS == C_DERIV ? acc2[kDeriv ? r : 0] : v, cell);
    }
    if (CLS == C_ONE && post == W_ONE_DIRECT) v = cadd(v, scat_direct(a, c.b, c.iw, c.y, x));
    if (post_taper) v = cscale(v, a.tapx[x] * ty);
    if (a.add) v = cadd(a.out[roff + x], v);
    if ((CLS == C_ONE || CLS == C_MASK) && a.rf_at == 2 && c.y < a.d.ny && x < a.d.nx)
      v = cadd(v, refl_term(a, roff, c.y, x));
    a.out[roff + x] = v;
    if (a.ic_img && c.y < a.d.ny && x < a.d.nx) {
      const float2 bg = a.ic_bg[roff + x];
      atomicAdd(a.ic_img + (long long)c.y * a.d.nx + x, bg.x * v.x + bg.y * v.y);
    }
    if (CLS == C_PAIR) {
      float2 u = cmul(acc2[kDeriv ? r : 0], cell);
      if (post_taper) u = cscale(u, a.tapx[x] * ty);
      if (a.add) u = cadd(a.out2[roff + x], u);
      a.out2[roff + x] = u;
    }
  }
}

// ---------------------------------------------------------------- columns

// What a thread of a column pass works on: column x0 + c of the tile, butterfly j
// of stage RT.
template <class S>
struct ColCtx {
  int c, j, x0, x, iw;
  bool ok;  // the thread's column exists
  long long b;
  __device__ __forceinline__ ColCtx(const SpecArgs& a, const Dim<S>& d) {
    c = threadIdx.x & (d.cols() - 1);
    j = threadIdx.x >> d.sh();
    b = blockIdx.x / d.g.nchunk;
    x0 = (int)(blockIdx.x - b * d.g.nchunk) * d.cols();
    x = x0 + c;
    iw = (int)((a.b0 + b) % a.d.nw);
    ok = j < d.nt() && x < a.d.NX;
  }
};

// Both directions' twiddles: the forward order ra, rb, RT, then RT, rb, ra.
template <class S>
__device__ __forceinline__ void col_twiddles(const SpecArgs& a, const Dim<S>& d, float2* tw) {
  fill_twiddles(tw, a.twy, d.ra(), d.rb(), S::RT, d.col_threads());
  fill_twiddles(tw + d.inv_rows_tw(), a.twy, S::RT, d.rb(), d.ra(), d.col_threads());
}

// First stage of the forward transform (radix ra, from HBM) of the CTA's columns of
// slice-local b.  With `copy` the samples also go there, scaled.
template <class S>
__device__ __forceinline__ void col_first(const SpecArgs& a, const Dim<S>& d, const ColCtx<S>& c, const float2* in,
                                          float2* dst, float2* copy = nullptr, float scale = 1.f) {
  const float2* src = in + c.b * a.d.slice + c.x0;
  float2* cp = copy ? copy + c.b * a.d.slice + c.x0 : nullptr;
  stage_a(d, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int i = threadIdx.x; i < d.cols() * d.na(); i += d.col_threads()) {
      const int cc = i & (d.cols() - 1), j = i >> d.sh();
      if (c.x0 + cc >= a.d.NX) continue;
      const int o = j * a.d.NX + cc, step = d.na() * a.d.NX;
      float2 u[R];
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = src[o + r * step];
      if (cp) {
#pragma unroll
        for (int r = 0; r < R; ++r) cp[o + r * step] = cscale(u[r], scale);
      }
      Dft<R, false>::run(u);
#pragma unroll
      for (int r = 0; r < R; ++r) dst[((j * R + r) << d.sh()) + cc] = u[r];
    }
  });
}
// Hints into L2 the CTA's columns of slice-local b of a later term: one hint per row
// segment.
template <class S>
__device__ __forceinline__ void col_prefetch(const SpecArgs& a, const Dim<S>& d, const ColCtx<S>& c,
                                             const float2* in) {
  const float2* p = in + c.b * a.d.slice + c.x0;
  for (int y = threadIdx.x; y < d.n(); y += d.col_threads())
    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p + y * a.d.NX));
}
// Middle stage, src -> dst; span = the first stage's radix.
template <bool INV, class S>
__device__ __forceinline__ void col_mid(const Dim<S>& d, const float2* tw, const float2* src, float2* dst, int span) {
  stage_b(d, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int i = threadIdx.x; i < d.cols() * d.nb(); i += d.col_threads()) {
      const int cc = i & (d.cols() - 1), j = i >> d.sh();
      const int q = j / span, k = j - q * span;
      float2 u[R];
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = src[((j + r * d.nb()) << d.sh()) + cc];
#pragma unroll
      for (int r = 1; r < R; ++r) u[r] = twid<INV>(u[r], tw[(r - 1) * span + k]);
      Dft<R, INV>::run(u);
#pragma unroll
      for (int r = 0; r < R; ++r) dst[((q * span * R + k + r * span) << d.sh()) + cc] = u[r];
    }
  });
}
// Last stage of the inverse transform (radix ra), to HBM.
template <class S>
__device__ __forceinline__ void col_last(const SpecArgs& a, const Dim<S>& d, const ColCtx<S>& c, const float2* twl,
                                         const float2* src, float2* out, int add, float scale) {
  float2* dst = out + c.b * a.d.slice + c.x0;
  stage_a(d, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    for (int i = threadIdx.x; i < d.cols() * d.na(); i += d.col_threads()) {
      const int cc = i & (d.cols() - 1), j = i >> d.sh();
      if (c.x0 + cc >= a.d.NX) continue;
      float2 u[R];
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = src[((j + r * d.na()) << d.sh()) + cc];
#pragma unroll
      for (int r = 1; r < R; ++r) u[r] = cmul_conj(u[r], twl[(r - 1) * d.na() + j]);
      Dft<R, true>::run(u);
      float2* const o = dst + j * a.d.NX + cc;
      const int step = d.na() * a.d.NX;
      if (add) {
#pragma unroll
        for (int r = 0; r < R; ++r) o[r * step] = cadd(o[r * step], cscale(u[r], scale));
      } else if (scale != 1.f) {
#pragma unroll
        for (int r = 0; r < R; ++r) o[r * step] = cscale(u[r], scale);
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) o[r * step] = u[r];
      }
    }
  });
}
// Last stage of the forward transform (radix RT) into registers: the spectrum
// samples j + r nt of the thread's column.
template <class S, int RT = S::RT>
__device__ __forceinline__ void col_spectrum(const Dim<S>& d, const ColCtx<S>& c, const float2* twl, const float2* src,
                                             float2 (&v)[RT]) {
#pragma unroll
  for (int r = 0; r < RT; ++r) v[r] = src[((c.j + r * d.nt()) << d.sh()) + c.c];
#pragma unroll
  for (int r = 1; r < RT; ++r) v[r] = cmul(v[r], twl[(r - 1) * d.nt() + c.j]);
  Dft<RT, false>::run(v);
}
// Column multipliers of term t at the thread's spectrum samples (qmult's values).
template <class S, int RT = S::RT>
__device__ __forceinline__ void col_factors(const SpecArgs& a, const Dim<S>& d, const ColCtx<S>& c, int qm, int t,
                                            float2 (&q)[RT]) {
  if ((qm == Q_PS_FWD || qm == Q_PS_ADJ) && a.ptab) {
    const int kxq = min(c.x, a.d.NX - c.x);
    const float2* p = a.ptab + ((long long)t * a.d.nw + c.iw) * a.ptab_nx * a.ptab_ny + (long long)kxq * a.ptab_sx;
    bool flip = false;
    if (qm == Q_PS_ADJ) {
      const float2 sr = a.sref[t * a.d.nw + c.iw];
      flip = !(a.w2[c.iw] * (sr.y - a.eps * sr.x) > 0.f);
    }
    // a thread's j < nt, so most of its rows know their side of n / 2: they step from
    // two bases by a multiple of the row pitch instead of a minimum and a product each
    const int step = d.nt() * a.ptab_sy;
    const float2* const up = p + c.j * a.ptab_sy;
    const float2* const down = p + (d.n() - c.j) * a.ptab_sy;
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      if (2 * r + 2 <= RT)  // j + r nt < (r + 1) nt <= n / 2
        q[r] = up[r * step];
      else if (2 * r >= RT)
        q[r] = down[-(r * step)];
      else
        q[r] = p[min(c.j + r * d.nt(), d.n() - c.j - r * d.nt()) * a.ptab_sy];
    }
    if (flip) {
#pragma unroll
      for (int r = 0; r < RT; ++r) q[r] = cconj(q[r]);
    }
  } else if (qm == Q_PS_FWD) {
#pragma unroll 1
    for (int r = 0; r < RT; ++r) q[r] = qmult<Q_PS_FWD>(a, t, c.iw, c.x, c.j + r * d.nt());
  } else if (qm == Q_PS_ADJ) {
#pragma unroll 1
    for (int r = 0; r < RT; ++r) q[r] = qmult<Q_PS_ADJ>(a, t, c.iw, c.x, c.j + r * d.nt());
  } else if (qm == Q_KPOW) {
    const KPow k(a, t, c.iw, c.x);
#pragma unroll
    for (int r = 0; r < RT; ++r) q[r] = make_float2(k.at(c.j + r * d.nt()), 0.f);
  } else {
#pragma unroll
    for (int r = 0; r < RT; ++r) q[r] = make_float2(a.norm, 0.f);
  }
}

// t2[term] = F_y^-1(Q_term * F_y(t1[0])); the spectrum stays in registers.
template <class S>
__global__ void __launch_bounds__(S::COL_THREADS, min_blocks<S>(S::COL_THREADS, 2))
    k_col_a(const SpecArgs a, const __grid_constant__ Geo g, int qm) {
  constexpr int RT = S::RT;
  const Dim<S> d{g};
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* const buf0 = sm + d.fwd_rows_tw() + d.inv_rows_tw();
  float2* const buf1 = buf0 + (d.n() << d.sh());
  const ColCtx<S> c(a, d);
  if (a.early) chain_next();
  col_twiddles(a, d, tw);
  chain_wait();
  // the zeroth Born order's filter is the identity: its output is the input,
  // scaled as the transform pair would
  const int first = qm == Q_KPOW && a.term0 == 0 ? 1 : 0;
  col_first(a, d, c, a.t1, buf1, first ? a.t2 : nullptr, a.norm * (float)d.n());
  __syncthreads();
  const float2* src = buf1;
  if (d.rb() > 1) {
    col_mid<false>(d, tw, buf1, buf0, d.ra());
    __syncthreads();
    src = buf0;
  }
  float2 psi[RT];
  if (c.ok) col_spectrum(d, c, tw + (d.rb() - 1) * d.ra(), src, psi);
  if (d.rb() > 1) __syncthreads();  // the terms start in buf0
  const float2* itw = tw + d.inv_rows_tw();
  for (int term = first; term < a.nterm; ++term) {
    float2* dst = (d.rb() == 1 && ((term - first) & 1)) ? buf1 : buf0;
    if (c.ok) {
      float2 v[RT];
      col_factors(a, d, c, qm, term, v);
#pragma unroll
      for (int r = 0; r < RT; ++r) v[r] = cmul(psi[r], v[r]);
      Dft<RT, true>::run(v);
#pragma unroll
      for (int r = 0; r < RT; ++r) dst[((c.j * RT + r) << d.sh()) + c.c] = v[r];
    }
    __syncthreads();
    if (d.rb() > 1) {
      col_mid<true>(d, itw, buf0, buf1, RT);
      __syncthreads();
      dst = buf1;
    }
    if (term + 1 == a.nterm) chain_next();
    col_last(a, d, c, itw + (d.rb() - 1) * RT, dst, a.t2 + (long long)term * a.tstride, 0, 1.f);
  }
}

// t2[0] = F_y^-1(sum_term Q_term * F_y(t1[term])).
template <class S>
__global__ void __launch_bounds__(S::COL_THREADS, min_blocks<S>(S::COL_THREADS, 2))
    k_col_b(const SpecArgs a, const __grid_constant__ Geo g, int qm) {
  constexpr int RT = S::RT;
  const Dim<S> d{g};
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* const buf0 = sm + d.fwd_rows_tw() + d.inv_rows_tw();
  float2* const buf1 = buf0 + (d.n() << d.sh());
  const ColCtx<S> c(a, d);
  if (a.early) chain_next();
  col_twiddles(a, d, tw);
  chain_wait();
  float2 acc[RT];
#pragma unroll
  for (int r = 0; r < RT; ++r) acc[r] = make_float2(0.f, 0.f);
  for (int term = 0; term < a.nterm; ++term) {
    float2* src = (d.rb() == 1 && (term & 1)) ? buf1 : buf0;
    col_first(a, d, c, a.t1 + (long long)term * a.tstride, src);
    if (term + 1 < a.nterm) col_prefetch(a, d, c, a.t1 + (long long)(term + 1) * a.tstride);
    __syncthreads();
    if (d.rb() > 1) {
      col_mid<false>(d, tw, buf0, buf1, d.ra());
      __syncthreads();
      src = buf1;
    }
    if (c.ok) {
      float2 v[RT], q[RT];
      col_factors(a, d, c, qm, term, q);
      col_spectrum(d, c, tw + (d.rb() - 1) * d.ra(), src, v);
#pragma unroll
      for (int r = 0; r < RT; ++r) acc[r] = cadd(acc[r], cmul(v[r], q[r]));
    }
  }
  chain_next();
  // the last term left its samples in buf1 (three stages) or in buf[(nterm - 1) & 1]
  float2* dst = (d.rb() == 1 && (a.nterm & 1)) ? buf1 : buf0;
  if (c.ok) {
    Dft<RT, true>::run(acc);
#pragma unroll
    for (int r = 0; r < RT; ++r) dst[((c.j * RT + r) << d.sh()) + c.c] = acc[r];
  }
  __syncthreads();
  const float2* itw = tw + d.inv_rows_tw();
  if (d.rb() > 1) {
    col_mid<true>(d, itw, buf0, buf1, RT);
    __syncthreads();
    dst = buf1;
  }
  col_last(a, d, c, itw + (d.rb() - 1) * RT, dst, a.t2, 0, 1.f);
}

// out (+)= scale * F_y^{-+1}(in): the column half of a plain 2D transform.
template <class S, bool INV>
__global__ void __launch_bounds__(S::COL_THREADS, min_blocks<S>(S::COL_THREADS, 2))
    k_col_fft(const SpecArgs a, const __grid_constant__ Geo g, const float2* in, float2* out, int add, float scale) {
  constexpr int RT = S::RT;
  const Dim<S> d{g};
  extern __shared__ float2 sm[];
  float2* tw = sm;
  float2* const buf0 = sm + d.fwd_rows_tw() + d.inv_rows_tw();
  float2* const buf1 = buf0 + (d.n() << d.sh());
  const ColCtx<S> c(a, d);
  if (a.early) chain_next();
  col_twiddles(a, d, tw);
  chain_wait();
  const long long off = c.b * a.d.slice + c.x;
  float2 v[RT];
  if (!INV) {
    col_first(a, d, c, in, buf0);
    __syncthreads();
    const float2* src = buf0;
    if (d.rb() > 1) {
      col_mid<false>(d, tw, buf0, buf1, d.ra());
      __syncthreads();
      src = buf1;
    }
    if (!c.ok) return;
    col_spectrum(d, c, tw + (d.rb() - 1) * d.ra(), src, v);
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      float2* q = out + off + (c.j + r * d.nt()) * a.d.NX;
      const float2 u = cscale(v[r], scale);
      *q = add ? cadd(*q, u) : u;
    }
    return;
  }
  if (c.ok) {
#pragma unroll
    for (int r = 0; r < RT; ++r) v[r] = in[off + (c.j + r * d.nt()) * a.d.NX];
    Dft<RT, true>::run(v);
#pragma unroll
    for (int r = 0; r < RT; ++r) buf0[((c.j * RT + r) << d.sh()) + c.c] = v[r];
  }
  __syncthreads();
  const float2* itw = tw + d.inv_rows_tw();
  const float2* src = buf0;
  if (d.rb() > 1) {
    col_mid<true>(d, itw, buf0, buf1, RT);
    __syncthreads();
    src = buf1;
  }
  col_last(a, d, c, itw + (d.rb() - 1) * RT, src, out, add, scale);
}

// ---------------------------------------------------------------- launches

inline unsigned magic(int d) { return (unsigned)((0x100000000ull + d - 1) / (unsigned)d); }

inline Geo base_geo(const Line& p) {
  Geo g;
  memset(&g, 0, sizeof(g));
  g.n = p.n;
  g.ra = p.ra;
  g.rb = p.rb;
  g.nt = p.n / p.rt;
  g.na = p.n / p.ra;
  g.nb = p.n / p.rb;
  g.mt = magic(g.nt);
  g.ma = magic(g.na);
  g.mb = magic(g.nb);
  return g;
}
inline Geo row_geo(const SpecArgs& a, const Line& p, bool inverse, unsigned* threads, size_t* smem) {
  Geo g = base_geo(p);
  g.lines = row_lines(g.nt);
  g.nchunk = (a.d.NY + g.lines - 1) / g.lines;
  *threads = (unsigned)((g.lines * g.nt + 31) / 32 * 32);
  const int tw = inverse ? table_size(p.ra, p.rb, p.rt) : table_size(p.rt, p.rb, p.ra);
  *smem = ((size_t)tw + 2 * (size_t)g.lines * row_ls(p.n, inverse ? p.ra : p.rt)) * sizeof(float2);
  return g;
}
inline Geo col_geo(const SpecArgs& a, const Line& p, unsigned* threads, size_t* smem) {
  Geo g = base_geo(p);
  g.sh = col_shift(g.nt);
  g.lines = 1 << g.sh;
  g.nchunk = (a.d.NX + g.lines - 1) / g.lines;
  *threads = (unsigned)(((g.nt << g.sh) + 31) / 32 * 32);
  const size_t tw = (size_t)table_size(p.rt, p.rb, p.ra) + table_size(p.ra, p.rb, p.rt);
  *smem = (tw + 2 * ((size_t)g.n << g.sh)) * sizeof(float2);
  return g;
}

// Opts a kernel in to the shared memory of its launch, once per (kernel, device, size),
// and gives the CTAs of it that the device holds at once.
template <class K>
cudaError_t opt_in(K kernel, unsigned threads, size_t bytes, int* resident) {
  static std::mutex mu;
  static std::map<std::tuple<const void*, int, size_t>, int> done;
  static std::map<std::pair<const void*, int>, size_t> most;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const auto key = std::make_tuple((const void*)kernel, dev, bytes * 2048 + threads);
  std::lock_guard<std::mutex> lock(mu);
  auto it = done.find(key);
  if (it != done.end()) {
    *resident = it->second;
    return cudaSuccess;
  }
  size_t& m = most[std::make_pair((const void*)kernel, dev)];
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e == cudaSuccess && bytes > 48 * 1024 && bytes > m)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  m = std::max(m, bytes);
  int per = 0, sms = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, (int)threads, bytes) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    per = 0;
  }
  *resident = done[key] = per * sms;
  return cudaSuccess;
}

template <class K, class... Args>
cudaError_t launch(K kernel, unsigned grid, unsigned threads, size_t smem, cudaStream_t s, const SpecArgs& a,
                   Args... args) {
  int res = 0;
  cudaError_t e = opt_in(kernel, threads, smem, &res);
  SpecArgs b = a;
  b.early = res > 0 && grid > (unsigned)res;
  if (e == cudaSuccess) e = launch_chained(a.d.chained, kernel, grid, threads, smem, s, b, args...);
  if (e == cudaSuccess) count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

template <class S>
cudaError_t row_forward_s(const SpecArgs& a, const Line& p, int pre, cudaStream_t s) {
  unsigned th;
  size_t sm;
  const Geo g = row_geo(a, p, false, &th, &sm);
  const unsigned grid = (unsigned)(a.nb * g.nchunk);
  if (a.rf_at == 1 && pre != W_ONE && pre != W_MASK) return cudaErrorInvalidValue;
  switch (pre) {
    case W_ONE:
    case W_TAPER:
    case W_IC: return launch(k_row_fwd<S, C_ONE>, grid, th, sm, s, a, g, pre);
    case W_MASK: return launch(k_row_fwd<S, C_MASK>, grid, th, sm, s, a, g, pre);
    case W_SCAT_CONJ: return launch(k_row_fwd<S, C_SCAT>, grid, th, sm, s, a, g, pre);
    case W_SMOOTH_CONJ: return launch(k_row_fwd<S, C_SMOOTH>, grid, th, sm, s, a, g, pre);
    default: return cudaErrorInvalidValue;
  }
}
template <class S>
cudaError_t row_inverse_s(const SpecArgs& a, const Line& p, int post, int pt, cudaStream_t s) {
  unsigned th;
  size_t sm;
  const Geo g = row_geo(a, p, true, &th, &sm);
  const unsigned grid = (unsigned)(a.nb * g.nchunk);
  if (a.rf_at == 2 && post != W_ONE && post != W_MASK) return cudaErrorInvalidValue;
  switch (post) {
    case W_ONE:
    case W_ONE_DIRECT: return launch(k_row_inv<S, C_ONE>, grid, th, sm, s, a, g, post, pt);
    case W_MASK: return launch(k_row_inv<S, C_MASK>, grid, th, sm, s, a, g, post, pt);
    case W_SCAT: return launch(k_row_inv<S, C_SCAT>, grid, th, sm, s, a, g, post, pt);
    case W_SMOOTH: return launch(k_row_inv<S, C_SMOOTH>, grid, th, sm, s, a, g, post, pt);
    case W_SMOOTH_DERIV: return launch(k_row_inv<S, C_DERIV>, grid, th, sm, s, a, g, post, pt);
    case W_SMOOTH_PAIR: return launch(k_row_inv<S, C_PAIR>, grid, th, sm, s, a, g, post, pt);
    default: return cudaErrorInvalidValue;
  }
}
inline bool col_mode(int qm) { return qm == Q_PS_FWD || qm == Q_PS_ADJ || qm == Q_KPOW || qm == Q_ONE; }
template <class S>
cudaError_t col_type_a_s(const SpecArgs& a, const Line& p, int qm, cudaStream_t s) {
  unsigned th;
  size_t sm;
  const Geo g = col_geo(a, p, &th, &sm);
  if (!col_mode(qm)) return cudaErrorInvalidValue;
  return launch(k_col_a<S>, (unsigned)(a.nb * g.nchunk), th, sm, s, a, g, qm);
}
template <class S>
cudaError_t col_type_b_s(const SpecArgs& a, const Line& p, int qm, cudaStream_t s) {
  unsigned th;
  size_t sm;
  const Geo g = col_geo(a, p, &th, &sm);
  if (!col_mode(qm)) return cudaErrorInvalidValue;
  return launch(k_col_b<S>, (unsigned)(a.nb * g.nchunk), th, sm, s, a, g, qm);
}
template <class S>
cudaError_t col_fft_s(const SpecArgs& a, const Line& p, int inverse, const float2* in, float2* out, int add,
                       float scale, cudaStream_t s) {
  unsigned th;
  size_t sm;
  const Geo g = col_geo(a, p, &th, &sm);
  const unsigned grid = (unsigned)(a.nb * g.nchunk);
  return inverse ? launch(k_col_fft<S, true>, grid, th, sm, s, a, g, in, out, add, scale)
                 : launch(k_col_fft<S, false>, grid, th, sm, s, a, g, in, out, add, scale);
}

}  // namespace flex
}  // namespace fwix
