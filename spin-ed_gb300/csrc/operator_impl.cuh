// operator_impl.cuh — device-side pieces of the matvec shared by the
// operator and eigensolver translation units (see operator.cu for the
// mathematics of the pull form and the stream form).
#pragma once

#include <type_traits>

#include "sed_internal.hpp"
#include "util.cuh"

namespace sed {

constexpr uint32_t kNull = 0xFFFFFFFFu;
constexpr unsigned kMaxCodes = 65535;

struct StreamView {
  uint64_t const* slice_ptr;
  uint32_t const* entries;
  uint16_t const* codes;  // unpacked form only
  void const* diag;       // double[D] or double2[D]
  uint8_t const* row_class;
  void const* table;      // double or double2 [n_codes]
  double const* inv_sqrt_s;
  uint32_t col_bits;
  uint32_t n_codes;
};

struct CodeView {
  uint32_t const* divisors;  // ascending divisors of |G|
  uint32_t n_div;
  uint32_t n_ph;             // 2 (real: sign) or L
  uint32_t real_phase;       // 1 if phases are encoded as sign
};

__device__ __forceinline__ uint32_t divisor_class(uint32_t S, CodeView const& C) {
  uint32_t lo = 0, hi = C.n_div;
  while (lo < hi) {
    uint32_t const mid = (lo + hi) >> 1;
    if (C.divisors[mid] < S)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

__device__ __forceinline__ uint32_t element_code(uint32_t vid, uint32_t phase, uint32_t S_j,
                                                 CodeView const& C) {
  uint32_t const ph = C.real_phase ? (phase != 0u) : phase;
  return (vid * C.n_ph + ph) * C.n_div + divisor_class(S_j, C);
}

template <class V>
__device__ __forceinline__ V load_table(void const* t, uint32_t i, bool real_table);
template <>
__device__ __forceinline__ double load_table<double>(void const* t, uint32_t i, bool) {
  return static_cast<double const*>(t)[i];
}
template <>
__device__ __forceinline__ cplx load_table<cplx>(void const* t, uint32_t i, bool real_table) {
  if (real_table) return {static_cast<double const*>(t)[i], 0.0};
  double2 const v = static_cast<double2 const*>(t)[i];
  return {v.x, v.y};
}

template <class V>
__device__ __forceinline__ V row_value(V diag_x, double f, V acc) {
  return addv(diag_x, mulv(f, acc));
}

// Number of off-diagonal elements of row r.
__device__ __forceinline__ uint32_t row_count(uint64_t r, TermsView const& T) {
  uint32_t c = 0;
  for (uint32_t u = 0; u < T.n_tuples; ++u) {
    uint32_t const tk = T.tuple_term[u];
    uint32_t const t = tk & 0xFFFFu, k = tk >> 16;
    c += T.n_off[t * 16 + local_index(r, T.tuple_sites[u], k)];
  }
  return c;
}

// Walks the elements of row r in canonical order: f(e, s, vid).
template <class F>
__device__ __forceinline__ void walk_row(uint64_t r, TermsView const& T, F&& f) {
  uint32_t e = 0;
  for (uint32_t u = 0; u < T.n_tuples; ++u) {
    uint32_t const tk = T.tuple_term[u];
    uint32_t const t = tk & 0xFFFFu, k = tk >> 16;
    uint32_t const sites = T.tuple_sites[u];
    uint32_t const a = local_index(r, sites, k);
    uint32_t const n = T.n_off[t * 16 + a];
    for (uint32_t q = 0; q < n; ++q) {
      uint32_t const a2 = T.off_col[(t * 16 + a) * 16 + q];
      uint32_t const vid = T.off_vid[(t * 16 + a) * 16 + q];
      f(e++, replace_local(r, sites, k, a2), vid);
    }
  }
}

template <class V>
__device__ __forceinline__ V row_diag(uint64_t r, TermsView const& T);
template <>
__device__ __forceinline__ double row_diag<double>(uint64_t r, TermsView const& T) {
  double d = 0.0;
  for (uint32_t u = 0; u < T.n_tuples; ++u) {
    uint32_t const tk = T.tuple_term[u];
    uint32_t const t = tk & 0xFFFFu, k = tk >> 16;
    d = __dadd_rn(d, T.diag[2 * (t * 16 + local_index(r, T.tuple_sites[u], k))]);
  }
  return d;
}
template <>
__device__ __forceinline__ cplx row_diag<cplx>(uint64_t r, TermsView const& T) {
  cplx d{0.0, 0.0};
  for (uint32_t u = 0; u < T.n_tuples; ++u) {
    uint32_t const tk = T.tuple_term[u];
    uint32_t const t = tk & 0xFFFFu, k = tk >> 16;
    uint32_t const a = local_index(r, T.tuple_sites[u], k);
    d.re = __dadd_rn(d.re, T.diag[2 * (t * 16 + a)]);
    d.im = __dadd_rn(d.im, T.diag[2 * (t * 16 + a) + 1]);
  }
  return d;
}


// ------------------------------------------ exact fixed-point accumulation --
// For a real operator with real characters (chi = +-1) the off-diagonal part
// of row i is (1/sqrt(S_i)) sum_v c_v sum_{e: value v} chi_e sqrt(S_j) x_j.
// With u_j = round(sqrt(S_j) x_j 2^F) held as int64 (one pass over x before
// the matvec, F chosen per vector from max|x_j| so that no row sum can
// overflow), the inner sums are exact integer sums of +-u_j: one integer
// accumulator per distinct value c_v, converted and scaled by c_v 2^-F once
// per row. The only rounding before the row's FP64 epilogue is that of u_j
// (half an integer step, at most 2^-61 of the largest |u|), and integer sums
// do not depend on their order, so every form of the matvec agrees bit for
// bit. The integer pipe is 64x wider than GB300's FP64 pipe, which otherwise
// bounds the matvec at one FMA per element.
constexpr unsigned kFixMaxValues = 4;   // accumulators per row
constexpr unsigned kFixMaxClasses = 256;
constexpr int64_t kFixBad = INT64_MIN;  // x held a NaN or an infinity

struct FixView {
  uint8_t const* code;   // [n_codes]: value index << 1 | character sign
  double const* sqrt_s;  // [n_div]: sqrt(S) per stabiliser class
  uint32_t n_codes;
  uint32_t n_div;
  double bound;          // (largest row count) x sqrt(largest S), rounded up
  double sqrt_s_max;     // sqrt(largest S), rounded up
  double c[kFixMaxValues];
  uint32_t one_sign;     // every character of the group is +1
  uint32_t second;       // codes from here on carry the second value or a later one
};

// Nearest integer of a finite d with |d| < 2^62 (halves away from zero),
// from the bit pattern: integer instructions only.
__device__ __forceinline__ int64_t fix_round(double d) {
  uint64_t const b = (uint64_t)__double_as_longlong(d);
  int const e = (int)((b >> 52) & 0x7FF);
  uint64_t const m = (b & 0xFFFFFFFFFFFFFull) | (e ? (1ull << 52) : 0ull);
  int const sh = 1075 - e;  // |d| = m 2^-sh for normal d
  uint64_t mag;
  if (sh <= 0)
    mag = m << (-sh);
  else if (sh >= 64)
    mag = 0;
  else
    mag = ((m >> (sh - 1)) + 1) >> 1;  // (m + 2^(sh-1)) >> sh
  return (b >> 63) ? -(int64_t)mag : (int64_t)mag;
}

// Scale exponent F for a vector whose largest |x_j| has bit pattern
// max_bits: bound * max|x| * 2^F < 2^62, so a row's sum of at most
// (row count) terms |u_j| <= sqrt(S_max) max|x| 2^F stays below 2^62.
__device__ __forceinline__ int64_t fix_exponent(uint64_t max_bits, double bound) {
  if (max_bits >= 0x7FF0000000000000ull) return kFixBad;
  if (max_bits == 0) return 0;
  double const t = __longlong_as_double((long long)max_bits) * bound;
  int const e = (int)(((uint64_t)__double_as_longlong(t) >> 52) & 0x7FF) - 1023;  // t < 2^(e+1)
  return 61 - e;  // in [-963, 1084]: t is finite, at least 2^-1074 before the bound
}

// The same for 32-bit u (the FP32-stored form): |u_j| < 2^30, sums in int64.
__device__ __forceinline__ int64_t fix_exponent32(uint64_t max_bits, double sqrt_s_max) {
  if (max_bits >= 0x7FF0000000000000ull) return kFixBad;
  if (max_bits == 0) return 0;
  double const t = __longlong_as_double((long long)max_bits) * sqrt_s_max;
  int const e = (int)(((uint64_t)__double_as_longlong(t) >> 52) & 0x7FF) - 1023;  // t < 2^(e+1)
  int64_t F = 29 - e;
  return F > 1000 ? 1000 : (F < -1000 ? -1000 : F);
}

// 2^p for |p| <= 1000 (a normal double), built from its bits.
__device__ __forceinline__ double fix_pow2(int64_t p) {
  return __longlong_as_double((long long)((uint64_t)(1023 + p) << 52));
}

// a 2^p for any exponent F can produce (|p| <= 1100): one multiplication
// when 2^p is a normal double, else two by halves of p (each exact unless
// the result is subnormal).
__device__ __forceinline__ double fix_ldexp(double a, int64_t p) {
  if (p >= -1000 && p <= 1000) return a * fix_pow2(p);
  int64_t const h = p / 2;
  return (a * fix_pow2(h)) * fix_pow2(p - h);
}

// Adds +-g to the accumulator of value index t >> 1 (sign t & 1).
template <int NV>
__device__ __forceinline__ void fix_add(int64_t (&acc)[NV], uint32_t t, int64_t g) {
  int64_t const v = (t & 1u) ? -g : g;
  if constexpr (NV == 1) {
    acc[0] += v;
  } else {
    uint32_t const q = t >> 1;
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (q == (uint32_t)k) acc[k] += v;
  }
}

// The row factors g[cls NV + v] = (c_v / sqrt(S_cls)) 2^-min(F, 1000), one
// table per block in shared memory (one rounding of c_v / sqrt(S), then an
// exact power of two). F above 1000 only occurs for vectors whose largest
// entry is below about 1e-290; the rest of the scaling is then applied by
// fix_row after the sum, so that g stays a normal number. Every thread of
// the block calls it; the caller synchronises.
template <int NV>
__device__ __forceinline__ void fix_row_factors(FixView const& fv, double const* __restrict__ inv_sqrt_s, int64_t F,
                                                double* g) {
  int64_t const Fa = F > 1000 ? 1000 : F;
  for (uint32_t t = threadIdx.x; t < fv.n_div * NV; t += blockDim.x)
    g[t] = F == kFixBad ? 0.0 : fix_ldexp(__dmul_rn(inv_sqrt_s[t / NV], fv.c[t % NV]), -Fa);
}

// (double)f from the bits: the conversion instruction runs on the FP64 pipe.
__device__ __forceinline__ double widen(float f) {
  uint32_t const b = __float_as_uint(f), e = (b >> 23) & 0xFFu;
  if (e == 0 || e == 0xFF) return (double)f;
  return __hiloint2double((int)((b & 0x80000000u) | ((e + 896u) << 20) | ((b & 0x7FFFFFu) >> 3)), (int)(b << 29));
}

// (double)v to nearest (ties to even) with integer instructions: the
// conversion runs on the FP64 pipe.
__device__ __forceinline__ double fix_to_double(int64_t v) {
  uint64_t m = (uint64_t)(v < 0 ? -v : v);  // |v| < 2^62
  int const z = __clzll((long long)m);
  m <<= z & 63;
  uint32_t const rest = (uint32_t)m & 0x7FFu;
  uint64_t const top = m >> 11;
  uint64_t b = ((uint64_t)(1085 - z) << 52) + top + ((rest > 0x400u || (rest == 0x400u && (top & 1))) ? 1u : 0u);
  if (m == 0) b = 0;
  return __longlong_as_double((long long)(b | (uint64_t)(v < 0) << 63));
}

// The row's epilogue, shared by every fixed-point kernel so that all of them
// round identically: y_i = d_i x_i + sum_v g[cls][v] acc_v (times
// 2^-(F - 1000) when F > 1000), with g from fix_row_factors (g points at the
// row's class).
template <int NV>
__device__ __forceinline__ double fix_row(int64_t const (&acc)[NV], double const* g, int64_t F, double dg, double xi) {
  if (F == kFixBad) return __longlong_as_double(0x7FF8000000000000ll);  // NaN in x gives NaN out
  if (F > 1000) {
    double o = 0.0;
#pragma unroll
    for (int k = 0; k < NV; ++k) o = __fma_rn(g[k], fix_to_double(acc[k]), o);
    return __fma_rn(o, fix_pow2(1000 - F), __dmul_rn(dg, xi));
  }
  double s = __dmul_rn(dg, xi);
#pragma unroll
  for (int k = 0; k < NV; ++k) s = __fma_rn(g[k], fix_to_double(acc[k]), s);
  return s;
}

// The code bytes and the zero byte behind them, by every thread of the block.
__device__ __forceinline__ void fix_stage_codes(FixView const& fv, uint8_t* code8) {
  for (uint32_t c = threadIdx.x; c <= fv.n_codes; c += blockDim.x) code8[c] = c < fv.n_codes ? fv.code[c] : 0;
}

// The integer sums of one row: N gathered columns per element, U elements in
// flight; gather(col, g) fetches g[0..N). Where the gather copy stays in L2
// the integer ALU limits it (64 lanes per clock and SM; about 40 instructions
// per warp and element with the sign and the value looked up), so the loop
// does without what an operator does not need:
//  - characters all +1 (!Signed): no sign; one value: no code at all, two: a
//    comparison of the entry;
//  - a padding slot reads the zero row `zero_row` that every gather copy has
//    behind its last row: no branch and no selection.
// One column, 6x6 torus (585 M elements): 1147 -> 1116 us; 30-site J1-J2 ring
// (40 M elements) 80 -> 72 us, eight columns of it 515 -> 345 us. Loading the
// next step's entries before this step's sums gained nothing (72 to 76 us;
// more copies in flight evict one another).
template <bool Packed, int NV, bool Signed, int N, uint32_t U, class T, class Entry, class Gather>
__device__ __forceinline__ void fix_row_sums(StreamView const& S, FixView const& fv, uint8_t const* code8,
                                             uint16_t const* codes, uint32_t width, uint32_t zero_row,
                                             int64_t (&acc)[N][NV], Entry&& entry, Gather&& gather, T) {
  uint32_t const mask = Packed ? ((1u << S.col_bits) - 1u) : 0xFFFFFFFFu;
  uint32_t const second = Packed ? fv.second << S.col_bits : fv.second;
  constexpr bool kCodes = !Packed && (NV > 1 || Signed);
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[n][k] = 0;
  auto step = [&](uint32_t e, auto guarded) {
    uint32_t v[U], c[U];
    T g[U][N];
#pragma unroll
    for (uint32_t p = 0; p < U; ++p) {
      bool const in = !decltype(guarded)::value || e + p < width;
      v[p] = in ? entry(e + p) : kNull;
      if constexpr (kCodes) c[p] = in ? (uint32_t)__ldcs(codes + (uint64_t)(e + p) * 32) : 0u;
    }
#pragma unroll
    for (uint32_t p = 0; p < U; ++p) gather(min(v[p] & mask, zero_row), g[p]);
#pragma unroll
    for (uint32_t p = 0; p < U; ++p) {
      if constexpr (Signed) {
        uint32_t const t = code8[Packed ? min(v[p] >> S.col_bits, fv.n_codes) : c[p]];
#pragma unroll
        for (int n = 0; n < N; ++n) fix_add<NV>(acc[n], t, (int64_t)g[p][n]);
      } else if constexpr (NV == 1) {
#pragma unroll
        for (int n = 0; n < N; ++n) acc[n][0] += g[p][n];
      } else {
        bool const later = (Packed ? v[p] : c[p]) >= second;
#pragma unroll
        for (int n = 0; n < N; ++n) {
          if (later) acc[n][1] += g[p][n];
          else acc[n][0] += g[p][n];
        }
      }
    }
  };
  uint32_t e = 0;
  for (; e + U <= width; e += U) step(e, std::false_type{});
  if (e < width) step(e, std::true_type{});
}

// The streamed matvec of an operator with complex elements on complex64
// vectors in integers (spmv_cols.cu). An element's factor and the gathered part are numbers of two
// 32-bit limbs (the low one signed, so that the high one is rounded):
// w = round(value x character x 2^-shift), |w| <= 2^54, and u as for real
// operators, |u| <= 2^62 / R with R the largest row count. A row keeps two
// 64-bit sums per part,
//   hi = sum w_h u_h,   lo = sum w_h u_l + w_l u_h + w_l u_l / 2^32,
// |hi| <= 2^53 and |lo| <= 2 R (2^61 / R + 2^53 + 2^30) < 2^63 up to R = 128;
// its value is (hi 2^32 + lo) 2^(32 + shift - F).
struct CplxView {
  int4 const* w;  // [n_codes]: limbs of Re w (high, low) and of Im w
  int shift;
};
constexpr uint64_t kCplxMaxRow = 128;
constexpr uint32_t kCplxMaxCodes = 2048;  // 32 KB of shared memory

struct OperatorTables {
  DeviceBuffer buf;      // holds all of them
  DevicePart divisors;
  DevicePart table;    // double[n_codes], real operators only
  DevicePart table_c;  // double2[n_codes], every operator
  DevicePart inv_sqrt_s;
  CodeView code{};
  uint32_t n_codes = 0;
  // fixed-point form (fix_ok: the operator qualifies)
  bool fix_ok = false;
  uint32_t fix_nv = 1;   // accumulators per row: 1, 2 or 4
  DevicePart fix_code;
  DevicePart fix_sqrt_s;
  FixView fix{};
  // integer form of a complex operator (cplx_ok: it qualifies; fix then holds
  // sqrt_s, n_div, n_codes and bound)
  bool cplx_ok = false;
  DevicePart cplx_w;
  CplxView cplx{};
};

// One row of the streamed SpMV over a SELL-32 slice (lane = row in slice).
template <class V, class X, bool RealOp, bool Packed>
__device__ __forceinline__ V stream_row_acc(StreamView const& S, void const* table, uint64_t s,
                                            uint32_t lane, X const* __restrict__ x) {
  uint64_t const base = S.slice_ptr[s];
  uint32_t const width = (uint32_t)((S.slice_ptr[s + 1] - base) >> 5);
  uint32_t const col_mask = Packed ? ((1u << S.col_bits) - 1u) : 0xFFFFFFFFu;
  V acc = zero<V>();
  uint32_t const* ent = S.entries + base + lane;
  for (uint32_t e = 0; e < width; ++e) {
    uint32_t const v = __ldcs(ent + (uint64_t)e * 32);
    if (v != kNull) {
      uint32_t const col = v & col_mask;
      uint32_t const code =
          Packed ? (v >> S.col_bits) : (uint32_t)__ldcs(S.codes + base + lane + (uint64_t)e * 32);
      mac(acc, load_table<V>(table, code, RealOp), Store<X>::load(x, col));
    }
  }
  return acc;
}

template <class V, bool RealOp>
__device__ __forceinline__ V stream_diag(StreamView const& S, uint64_t i) {
  if constexpr (std::is_same<V, double>::value) {
    return static_cast<double const*>(S.diag)[i];
  } else {
    if (RealOp) return cplx{static_cast<double const*>(S.diag)[i], 0.0};
    double2 const d2 = static_cast<double2 const*>(S.diag)[i];
    return cplx{d2.x, d2.y};
  }
}

// Stages the value table in shared memory when it fits (32 KB); returns the
// table to read from. Must be called by every thread of the block.
template <bool RealOp>
__device__ __forceinline__ void const* stage_table(StreamView const& S, unsigned char* smem) {
  bool const in_smem = S.n_codes * (RealOp ? 8u : 16u) <= 32768u;
  if (in_smem) {
    if (RealOp) {
      double* t = reinterpret_cast<double*>(smem);
      for (uint32_t c = threadIdx.x; c < S.n_codes; c += blockDim.x)
        t[c] = static_cast<double const*>(S.table)[c];
    } else {
      double2* t = reinterpret_cast<double2*>(smem);
      for (uint32_t c = threadIdx.x; c < S.n_codes; c += blockDim.x)
        t[c] = static_cast<double2 const*>(S.table)[c];
    }
    __syncthreads();
    return smem;
  }
  return S.table;
}

StreamView stream_view(OperatorData const& op);

// The fixed-point workspace of an operator (column 0), for kernels that
// prepare u and F themselves.
struct FixSlots {
  unsigned long long* max_bits;  // max |x| bit pattern (zero before use)
  int64_t* F;
  int64_t* u;
  uint8_t const* row_class;
  FixView view;
};
// True (and *out filled) when the FP64 matvec of `op` runs in fixed point
// through the stream form.
bool fix_slots(OperatorData& op, FixSlots* out);
// The matvec's pre-pass on its own: max |x|, then u and F, for x = base (+ k
// ld in Krylov mode).
int fix_prescale(OperatorData& op, double const* base, Indirect ind, cudaStream_t stream);
// Calls f(packed, nv, signed) with the integral constants of the
// fixed-point kernel an operator takes. Unsigned variants exist where they
// save the look-up: one value, or two in packed entries.
template <class F>
void fix_dispatch(OperatorTables const& tb, bool packed, F&& f) {
  using Yes = std::true_type;
  using No = std::false_type;
  std::integral_constant<int, 1> n1;
  std::integral_constant<int, 2> n2;
  std::integral_constant<int, 4> n4;
  bool const one = tb.fix.one_sign != 0;
  if (packed) {
    switch (tb.fix_nv) {
      case 1: one ? f(Yes{}, n1, No{}) : f(Yes{}, n1, Yes{}); break;
      case 2: one ? f(Yes{}, n2, No{}) : f(Yes{}, n2, Yes{}); break;
      default: f(Yes{}, n4, Yes{}); break;
    }
  } else {
    switch (tb.fix_nv) {
      case 1: one ? f(No{}, n1, No{}) : f(No{}, n1, Yes{}); break;
      case 2: f(No{}, n2, Yes{}); break;
      default: f(No{}, n4, Yes{}); break;
    }
  }
}
// Shared memory of a fixed-point kernel over K columns: the row factors, then
// the code bytes and a zero byte for padding slots.
inline size_t fix_smem_bytes(OperatorTables const& tb, unsigned K) {
  return (size_t)K * tb.fix.n_div * tb.fix_nv * 8 + tb.fix.n_codes + 1;
}

// FP32 streamed SpMV in Krylov-indirect mode (x = base + k ld, y = base +
// (k+1) ld); FP32 arithmetic, per-block partial sums of x_i y_i in FP64.
int operator_apply_krylov32(OperatorData& op, float* base, Indirect ind, cudaStream_t stream);
// The same SpMV on explicit FP32 vectors; prescaled: u and F of x are in the
// workspace already.
int operator_apply32(OperatorData& op, float const* x, float* y, cudaStream_t stream, bool prescaled = false);
// The fixed-point workspace of that SpMV (true if it has one), and y = H x in
// FP64 with u and F of x in the workspace already (fix_slots).
struct FixSlots32 {
  int64_t* F;
  int32_t* u;
  uint8_t const* row_class;
  FixView view;
};
bool fix_slots32(OperatorData& op, FixSlots32* out);
int operator_apply_prescaled(OperatorData& op, double const* x, double* y, cudaStream_t stream);
// Krylov-indirect apply (see Indirect), on at most ceil(D / kBlock) blocks.
int operator_apply_krylov(OperatorData& op, int dtype, void* base, Indirect ind, cudaStream_t stream);
int operator_ensure_ready(OperatorData& op);

// Whether complex64 matvecs of a recorded complex operator take integer sums.
bool cplx_sums(OperatorData const& op);
// Whether streamed matvecs of this dtype take the integer sums of
// fix_cols_blocks, and the first `block` columns through it (spmv_cols.cu);
// *done counts the columns taken.
bool fix_cols_apply(OperatorData const& op, int dtype, bool use_stream, cudaStream_t stream);
int fix_cols_blocks(OperatorData& op, int dtype, uint64_t block, char const* x, uint64_t ldx, char* y, uint64_t ldy,
                    size_t es, cudaStream_t stream, uint64_t* done);

// V[:, 0..kk) <- V[:, 0..m) Y on the tensor cores (rotate_tc.cu): V FP64,
// D x m with column stride ld, Y m x kk row-major FP64, both on the device;
// *error_flag (device int) is set to 1 if a bounded wait ran out.
bool rotate_tc_eligible(uint32_t m, uint32_t kk);
int rotate_tc(double* V, uint64_t ld, uint32_t m, double const* Y, uint32_t kk, uint64_t D, cudaStream_t stream,
              int* error_flag);
// Path of the thick restart's basis rotation (sed_set_rotate_path).
extern int g_rotate_path;

}  // namespace sed
