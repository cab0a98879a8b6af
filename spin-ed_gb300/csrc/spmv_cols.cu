// spmv_cols.cu — the streamed fixed-point matvec on blocks of columns, on FP32
// vectors (real or complex) of real operators and on complex FP32 vectors of
// complex operators (src/SpinED/Internal.hs:411-429; the mathematics is at
// FixView and CplxView in operator_impl.cuh).
//
// A pass covers K real columns; a complex column is two. The gather copy u
// holds the K columns of a row next to each other.
//
// FP32 vectors of any range of entries: the integer sums of a row err by at
// most half a unit per element, and a part of a row's result that is below 2^30
// times that is summed again as k_spmv does (general_entry), so that every part
// of every entry is within 2^-30 of the FP64 value before it is rounded to FP32.
// In a vector of normal numbers these are 10^-4 of the rows or fewer (4.7 M FP32
// rows: 163 us a call with and without the rule); where nearly all entries are
// zero or below 2^-26 of the largest they are nearly all rows, 484 us a call for
// the 395 of k_spmv.
//
// complex128 vectors stay with the FP64 sums of k_spmv, whose errors are those
// of each entry: a fixed point of the vector's largest entry gives rows that
// couple to entries far below it fewer digits, or none.
#include "operator_impl.cuh"

namespace sed {
namespace {

constexpr int64_t kFixZero = 1000;  // F of an FP32 column of zeros (those of others are below 300)

// FP32 vectors of a real operator take the same integer sums as FP64 ones: the
// FP64 operations per element of k_spmv (one or two multiply-adds on a pipe of
// 1.75 per clock and SM, and after an FP32 load a conversion on the same pipe)
// bound it at 395 us a call where these take 163
// (ring of 32 sites, FP32).
struct Columns {
  void const* x;
  void* y;
  uint64_t ldx, ldy;  // in vector elements
  uint32_t cols;      // real columns of this pass (the rest of K is padding)
  bool f32, cx;       // complex columns are FP32 ones
  // offset of entry i of real column q, in reals
  __device__ __forceinline__ uint64_t at(uint32_t q, uint64_t i, uint64_t ld) const {
    return cx ? 2 * ((uint64_t)(q >> 1) * ld + i) + (q & 1u) : (uint64_t)q * ld + i;
  }
  __device__ __forceinline__ double load(uint32_t q, uint64_t i) const {
    uint64_t const o = at(q, i, ldx);
    return f32 ? (double)__ldcs(static_cast<float const*>(x) + o) : __ldcs(static_cast<double const*>(x) + o);
  }
  __device__ __forceinline__ void store(uint32_t q, uint64_t i, double v) const {
    uint64_t const o = at(q, i, ldy);
    if (f32) __stcs(static_cast<float*>(y) + o, (float)v);
    else __stcs(static_cast<double*>(y) + o, v);
  }
};

// k_fix_max for Columns: blockIdx.y is the vector column.
__global__ void __launch_bounds__(kBlock) k_fix_max_cols(Columns c, uint64_t D, unsigned long long* __restrict__ max_bits) {
  __shared__ unsigned long long red[2][kBlock / 32];
  unsigned long long m[2] = {0, 0};
  uint64_t const n = c.cx ? 2 * D : D, o = (uint64_t)blockIdx.y * (c.cx ? 2 : 1) * c.ldx;
  // blockDim and the stride are even: a thread sees one part of a complex column
  uint64_t const first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
  unsigned long long v = 0;
  if (c.f32) {
    float const* p = static_cast<float const*>(c.x) + o;
    uint32_t w = 0;
    uint64_t i = first;
    for (; i + 3 * step < n; i += 4 * step)
#pragma unroll
      for (int k = 0; k < 4; ++k) w = max(w, __float_as_uint(p[i + k * step]) & 0x7FFFFFFFu);
    for (; i < n; i += step) w = max(w, __float_as_uint(p[i]) & 0x7FFFFFFFu);
    v = (unsigned long long)__double_as_longlong((double)__uint_as_float(w));  // keeps the order, infinities and NaN
  } else {
    double const* p = static_cast<double const*>(c.x) + o;
    uint64_t i = first;
    for (; i + 3 * step < n; i += 4 * step)
#pragma unroll
      for (int k = 0; k < 4; ++k) v = max(v, (unsigned long long)__double_as_longlong(p[i + k * step]) & 0x7FFFFFFFFFFFFFFFull);
    for (; i < n; i += step) v = max(v, (unsigned long long)__double_as_longlong(p[i]) & 0x7FFFFFFFFFFFFFFFull);
  }
  m[c.cx ? (threadIdx.x & 1u) : 0u] = v;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    for (int d = 16; d > 0; d >>= 1) m[p] = max(m[p], __shfl_xor_sync(0xffffffffu, m[p], d));
    if ((threadIdx.x & 31) == 0) red[p][threadIdx.x >> 5] = m[p];
  }
  __syncthreads();
  if (threadIdx.x < (c.cx ? 2u : 1u)) {
    unsigned long long t = 0;
    for (unsigned w = 0; w < kBlock / 32; ++w) t = max(t, red[threadIdx.x][w]);
    atomicMax(max_bits + blockIdx.y * (c.cx ? 2 : 1) + threadIdx.x, t);
  }
}

// k_fix_convert for Columns: u row by row, the K columns of a row next to
// each other, so that an element's gather is one run of 8 K bytes instead of
// K sectors. K / 2 lanes share a row, two columns each, so that a warp writes
// 512 bytes in a row (a lane that wrote a whole row took 59 us for 8 columns
// of 1.3 M rows); a thread keeps its columns, and what belongs to them, over
// its rows, since the integer ALU bounds it. Cplx (K = 2): one scale for both
// parts, and u in two limbs (CplxView).
template <int K, bool Cplx>
__global__ void __launch_bounds__(kBlock) k_fix_convert_cols(Columns c, uint64_t D, uint8_t const* __restrict__ row_class,
                                                             FixView fv, unsigned long long const* __restrict__ max_bits,
                                                             int64_t* __restrict__ F_out, int64_t* __restrict__ u) {
  constexpr uint32_t N = K > 1 ? 2 : 1, L = K / N;  // columns per lane, lanes per row
  extern __shared__ double fac[];                    // [K][n_div]
  auto exponent = [&](uint32_t q) {
    return fix_exponent(Cplx ? max(max_bits[0], max_bits[1]) : max_bits[q], fv.bound);
  };
  for (uint32_t t = threadIdx.x; t < K * fv.n_div; t += blockDim.x) {
    uint32_t const q = t / fv.n_div;
    double f = 0.0;
    if (q < c.cols) {
      int64_t const F = exponent(q);
      int64_t const F1 = (F == kFixBad || (F >= -1000 && F <= 1000)) ? 0 : F / 2;
      if (F != kFixBad) f = fv.sqrt_s[t % fv.n_div] * fix_pow2(F - F1);
      if (blockIdx.x == 0 && t % fv.n_div == 0) F_out[q] = !Cplx && c.f32 && max_bits[q] == 0 ? kFixZero : F;
    }
    fac[t] = f;
  }
  // blockDim and the stride are multiples of L: the columns of a thread
  uint32_t const q0 = (threadIdx.x % L) * N;
  uint64_t const first = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / L, step = (uint64_t)gridDim.x * blockDim.x / L;
  uint64_t const es = c.cx ? 2 : 1;
  bool on[N];        // a column, and not one with a NaN or an infinity
  double p1[N];      // the first of two factors (F beyond +-1000)
  bool two = false;
  uint64_t at[N];
#pragma unroll
  for (uint32_t n = 0; n < N; ++n) {
    uint32_t const q = q0 + n;
    int64_t const F = q < c.cols ? exponent(q) : kFixBad;
    on[n] = F != kFixBad;
    int64_t const F1 = (F == kFixBad || (F >= -1000 && F <= 1000)) ? 0 : F / 2;
    p1[n] = fix_pow2(F1);
    two = two || F1 != 0;
    at[n] = c.at(q, 0, c.ldx);
  }
  __syncthreads();
  auto load = [&](uint64_t i, double (&xv)[N]) -> uint32_t {
#pragma unroll
    for (uint32_t n = 0; n < N; ++n) {
      uint64_t const o = at[n] + i * es;
      xv[n] = !on[n] ? 0.0 : c.f32 ? widen(static_cast<float const*>(c.x)[o]) : static_cast<double const*>(c.x)[o];
    }
    return row_class[i];
  };
  auto store = [&](uint64_t i, uint32_t cls, double const (&xv)[N]) {
    int64_t v[N];
#pragma unroll
    for (uint32_t n = 0; n < N; ++n) {
      v[n] = fix_round((two ? xv[n] * p1[n] : xv[n]) * fac[(q0 + n) * fv.n_div + cls]);
      if constexpr (Cplx) v[n] += (v[n] & 0x80000000ll) << 1;  // high limb | low limb
    }
    if constexpr (N == 1) u[i] = v[0];
    else reinterpret_cast<longlong2*>(u)[i * L + q0 / 2] = make_longlong2(v[0], v[N - 1]);
  };
  // four rows' loads together: one at a time left a load's latency per row (4.7 M
  // FP32 rows 32 -> 23 us, 1.3 M rows of 8 columns 61 -> 47)
  uint64_t i = first;
  for (; i + 3 * step < D; i += 4 * step) {
    double xv[4][N];
    uint32_t cls[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) cls[m] = load(i + m * step, xv[m]);
#pragma unroll
    for (int m = 0; m < 4; ++m) store(i + m * step, cls[m], xv[m]);
  }
  for (; i <= D; i += step) {  // row D is the zero row of fix_row_sums
    double xv[N] = {};
    uint32_t const cls = i < D ? load(i, xv) : 0u;
    store(i, cls, xv);
  }
}

__device__ __forceinline__ int exponent_bits(double v) { return __double2hiint(v) >> 20 & 0x7FF; }

// Entry i of FP32 column q (V real), or of the complex column whose real part
// is q, as k_spmv gives it: four elements' loads in flight (a warp that came
// here late with one at a time ended some 70 us after the others), and no sums
// over zeros of x, which most rows of a sparse vector have only.
template <class V, bool RealOp>
__device__ __forceinline__ V general_entry(StreamView const& S, Columns const& c, uint32_t const* ent, uint16_t const* codes,
                                           uint32_t width, bool packed, uint32_t q, uint64_t i) {
  constexpr bool kReal = std::is_same<V, double>::value;
  constexpr uint32_t U = 4;
  uint32_t const mask = packed ? ((1u << S.col_bits) - 1u) : 0xFFFFFFFFu;
  float const* const x = static_cast<float const*>(c.x) + c.at(q, 0, c.ldx);
  uint64_t const es = c.cx ? 2 : 1;
  auto widened = [&](float re, float im) -> V {
    if constexpr (kReal) return (double)re;
    else return cplx{(double)re, (double)im};
  };
  V acc = zero<V>();
  for (uint32_t e0 = 0; e0 < width; e0 += U) {
    uint32_t v[U];
    float re[U], im[U];
#pragma unroll
    for (uint32_t p = 0; p < U; ++p) v[p] = e0 + p < width ? ent[(uint64_t)(e0 + p) * 32] : kNull;
#pragma unroll
    for (uint32_t p = 0; p < U; ++p) {
      uint64_t const at = v[p] == kNull ? 0 : (uint64_t)(v[p] & mask) * es;
      re[p] = x[at];
      im[p] = kReal ? 0.0f : x[at + 1];
    }
#pragma unroll
    for (uint32_t p = 0; p < U; ++p) {
      if (v[p] == kNull || ((__float_as_uint(re[p]) | __float_as_uint(im[p])) & 0x7FFFFFFFu) == 0) continue;
      uint32_t const code = packed ? (v[p] >> S.col_bits) : (uint32_t)codes[(uint64_t)(e0 + p) * 32];
      mac(acc, load_table<V>(S.table, code, RealOp), widened(re[p], im[p]));
    }
  }
  V const xi = widened(x[i * es], kReal ? 0.0f : x[i * es + 1]);
  return row_value<V>(mulv(stream_diag<V, RealOp>(S, i), xi), S.inv_sqrt_s[S.row_class[i]], acc);
}

// Streamed SpMV on K interleaved columns (u row i at u + i K): K / 4 lanes
// share a row, four columns (one 32-byte sector of u) each, and a slice of 32
// rows is K / 4 warps. Column by column every element took K sectors, one per
// column; 16-byte loads by K / 2 lanes took 345 us where 32-byte loads took
// 319: 8 FP64 columns of the 30-site J1-J2 ring (1.3 M rows, 40 M elements,
// 2.6 GB of gathered sectors), 515 column by column. FP32 columns: 304 (with
// the registers held to four blocks a multiprocessor).
// x, y and the entries pass through L2 once (evict first), so that u stays.
// The registers of FP32 columns are held to what the sums alone need: without
// the bound, general_entry's took the occupancy that hides the gathers (32-site
// ring, one column: 40 registers, 180 us a call; 32 and a few spills there, 163).
template <bool Packed, int NV, bool Signed, int K, bool F32>
__global__ void __launch_bounds__(kBlock, !F32 || NV > 2 ? 0 : K == 1 ? 8 : K == 2 ? 6 : K == 4 ? 5 : 4)
    k_spmv_fix_cols(StreamView S, FixView fv, uint64_t D, Columns c, int64_t const* __restrict__ u,
                    int64_t const* __restrict__ F_in, unsigned long long* __restrict__ clear) {
  constexpr uint32_t N = K < 4 ? K : 4, L = K / N;  // columns per lane, lanes per row
  extern __shared__ double fix_smem[];                 // g[K][n_div NV], then the code bytes
  if (blockIdx.x == 0 && threadIdx.x < K) clear[threadIdx.x] = 0;  // max |x| for the next call's pre-pass
  uint8_t* code8 = reinterpret_cast<uint8_t*>(fix_smem + K * fv.n_div * NV);
  if constexpr (Signed) fix_stage_codes(fv, code8);
  for (uint32_t q = 0; q < c.cols; ++q) fix_row_factors<NV>(fv, S.inv_sqrt_s, F_in[q], fix_smem + q * fv.n_div * NV);
  __syncthreads();
  uint64_t const gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint64_t const s = gw / L;
  if ((s << 5) >= D) return;
  uint32_t const lane = threadIdx.x & 31, row = (uint32_t)(gw % L) * (32 / L) + lane / L, q0 = (lane % L) * N;
  uint64_t const base = S.slice_ptr[s], i = s * 32 + row;
  uint32_t const width = (uint32_t)((S.slice_ptr[s + 1] - base) >> 5);
  uint32_t const* ent = S.entries + base + row;
  uint16_t const* codes = S.codes + base + row;
  int64_t acc[N][NV];
  fix_row_sums<Packed, NV, Signed, (int)N, 8>(
      S, fv, code8, codes, width, (uint32_t)D, acc,
      [&](uint32_t e) { return __ldcs(ent + (uint64_t)e * 32); },
      [&](uint32_t col, int64_t* g) {
        int64_t const* src = u + (uint64_t)col * K + q0;
        if constexpr (N == 1) {
          g[0] = *src;
        } else if constexpr (N == 2) {
          longlong2 const v = *reinterpret_cast<longlong2 const*>(src);
          g[0] = v.x;
          g[1] = v.y;
        } else {
          asm("ld.global.nc.v4.s64 {%0, %1, %2, %3}, [%4];" : "=l"(g[0]), "=l"(g[1]), "=l"(g[2]), "=l"(g[3]) : "l"(src));
        }
      },
      int64_t{});
  if (i >= D) return;
  uint32_t const cls = __ldcs(S.row_class + i);
  double const dg = __ldcs(static_cast<double const*>(S.diag) + i);
  uint32_t again = 0;  // columns to sum again
  // 2^30 width max |g_v| is below 2^wide times the power of two below max |g_v|
  int const wide = 31 + (32 - __clz((int)width));
#pragma unroll
  for (uint32_t n = 0; n < N; ++n) {
    uint32_t const q = q0 + n;
    if (q >= c.cols) continue;
    double const* g = fix_smem + (q * fv.n_div + cls) * NV;
    double const y = fix_row<NV>(acc[n], g, F_in[q], dg, c.load(q, i));
    c.store(q, i, y);
    if constexpr (F32) {
      int e = 0;
#pragma unroll
      for (int k = 0; k < NV; ++k) e = max(e, exponent_bits(g[k]));
      if ((exponent_bits(y) < e + wide && F_in[q] != kFixZero) || F_in[q] == kFixBad || (c.cx && F_in[q ^ 1u] == kFixBad)) again |= 1u << n;
    }
  }
  if constexpr (F32)
    for (; again; again &= again - 1) {
      uint32_t const q = q0 + __ffs((int)again) - 1;
      if (c.cx && (F_in[q] == kFixBad || F_in[q ^ 1u] == kFixBad)) {  // either part spoils both
        cplx const y = general_entry<cplx, true>(S, c, ent, codes, width, Packed, q & ~1u, i);
        c.store(q, i, (q & 1u) ? y.im : y.re);
      } else {
        c.store(q, i, general_entry<double, true>(S, c, ent, codes, width, Packed, q, i));
      }
    }
}

// hi 2^32 + lo as a double, rounded to nearest even (|hi| < 2^55).
__device__ __forceinline__ double limbs_to_double(int64_t hi, int64_t lo) {
  hi += lo >> 32;
  uint32_t l = (uint32_t)lo;
  bool const neg = hi < 0;
  if (neg) {
    l = 0u - l;
    hi = ~hi + (l == 0u ? 1 : 0);
  }
  int const z = __clzll(hi);
  uint64_t m = (uint64_t)hi << 32 | l;
  uint64_t b = 0;
  if (z < 32) {  // 2^64 and above: the 64 leading bits, the rest as a sticky one
    m = (uint64_t)hi << z | l >> (32 - z) | ((l << z) != 0u ? 1u : 0u);
    b = (uint64_t)(32 - z) << 52;
  }
  int const y = __clzll((long long)m);
  m <<= y & 63;
  uint32_t const rest = (uint32_t)m & 0x7FFu;
  uint64_t const top = m >> 11;
  b += ((uint64_t)(1085 - y) << 52) + top + ((rest > 0x400u || (rest == 0x400u && (top & 1))) ? 1u : 0u);
  if (m == 0) b = 0;
  return __longlong_as_double((long long)(b | (uint64_t)neg << 63));
}

// Streamed SpMV of a complex operator on a complex64 column, sums in integers
// (CplxView). The four FP64 multiply-adds per element of k_spmv and the
// conversions of its loads take 159 us on the 28-site ring at k = 3 (10.4 M
// elements, FP64 pipe of 1.75 per clock and SM); here an element is 16 wide
// integer multiply-adds and one 16-byte gather: 57 us. A call takes 92 us for 178.
// Factors are staged with their position's low three bits swizzled: codes of
// one stabiliser class are n_div apart, which would put them all in one bank
// group. Eight elements in flight: 20.8 M elements in 109 us for 112 with four.
template <bool Packed>
__global__ void __launch_bounds__(kBlock, 5) k_spmv_cplx(StreamView S, FixView fv, CplxView cw, uint64_t D, Columns c,
                                                      int4 const* __restrict__ u, int64_t const* __restrict__ F_in,
                                                      unsigned long long* __restrict__ clear) {
  extern __shared__ int4 w_smem[];  // [n_codes], swizzled within groups of 8; then g[n_div]
  auto place = [](uint32_t code) { return code ^ ((code >> 3) & 7u); };
  uint32_t const n8 = (fv.n_codes + 7u) & ~7u;
  double* g = reinterpret_cast<double*>(w_smem + n8);
  if (blockIdx.x == 0 && threadIdx.x < 2) clear[threadIdx.x] = 0;  // max |x| for the next call's pre-pass
  int64_t const F = F_in[0];
  // 2^(32 + shift - F): F is in -100 .. 215 for FP32 entries, shift in -254 .. 146
  int64_t const e = F == kFixBad ? 0 : 32 + cw.shift - F;
  for (uint32_t t = threadIdx.x; t < fv.n_codes; t += blockDim.x) w_smem[place(t)] = cw.w[t];
  for (uint32_t t = threadIdx.x; t < fv.n_div; t += blockDim.x) g[t] = S.inv_sqrt_s[t] * fix_pow2(e);
  __syncthreads();
  uint64_t const i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, s = i >> 5;
  if ((s << 5) >= D) return;
  uint32_t const lane = threadIdx.x & 31;
  uint64_t const base = S.slice_ptr[s];
  uint32_t const width = (uint32_t)((S.slice_ptr[s + 1] - base) >> 5);
  uint32_t const mask = Packed ? ((1u << S.col_bits) - 1u) : 0xFFFFFFFFu;
  uint32_t const* ent = S.entries + base + lane;
  uint16_t const* codes = S.codes + base + lane;
  int64_t hr = 0, lr = 0, hi = 0, li = 0;
  auto add = [](int64_t& h, int64_t& l, int wh, int wl, int uh, int ul) {
    h += (int64_t)wh * uh;
    l += (int64_t)wh * ul;
    l += (int64_t)wl * uh;
    l += (int64_t)(wl >> 16) * (ul >> 16);  // the last 2^-68 of the largest product is not kept
  };
  // the products are subtracted: a low limb can be -2^31, which has no negative in 32 bits
  auto sub = [](int64_t& h, int64_t& l, int wh, int wl, int uh, int ul) {
    h -= (int64_t)wh * uh;
    l -= (int64_t)wh * ul;
    l -= (int64_t)wl * uh;
    l -= (int64_t)(wl >> 16) * (ul >> 16);
  };
  constexpr uint32_t U = 8;
  auto step = [&](uint32_t e0, auto guarded) {
    uint32_t v[U], cd[U];
    int4 x[U];
#pragma unroll
    for (uint32_t p = 0; p < U; ++p) {
      bool const in = !decltype(guarded)::value || e0 + p < width;
      v[p] = in ? __ldcs(ent + (uint64_t)(e0 + p) * 32) : kNull;
      if constexpr (Packed) cd[p] = min(v[p] >> S.col_bits, fv.n_codes - 1);
      else cd[p] = in ? (uint32_t)__ldcs(codes + (uint64_t)(e0 + p) * 32) : 0u;
    }
#pragma unroll
    for (uint32_t p = 0; p < U; ++p) x[p] = __ldg(u + min(v[p] & mask, (uint32_t)D));  // row D is zero
#pragma unroll
    for (uint32_t p = 0; p < U; ++p) {
      int4 const w = w_smem[place(cd[p])];
      // little endian: x low, y high limb of the real part, z and w of the imaginary
      add(hr, lr, w.x, w.y, x[p].y, x[p].x);
      sub(hr, lr, w.z, w.w, x[p].w, x[p].z);
      add(hi, li, w.x, w.y, x[p].w, x[p].z);
      add(hi, li, w.z, w.w, x[p].y, x[p].x);
    }
  };
  uint32_t e0 = 0;
  for (; e0 + U <= width; e0 += U) step(e0, std::false_type{});
  if (e0 < width) step(e0, std::true_type{});
  if (i >= D) return;
  double const f = g[__ldcs(S.row_class + i)];
  double2 const dg = __ldcs(static_cast<double2 const*>(S.diag) + i);
  double const xr = c.load(0, i), xi = c.load(1, i);
  double yr = __dmul_rn(dg.x, xr), yi = __dmul_rn(dg.x, xi);
  if (dg.y != 0.0) {
    yr = __fma_rn(-dg.y, xi, yr);
    yi = __fma_rn(dg.y, xr, yi);
  }
  yr = __fma_rn(f, limbs_to_double(hr, lr), yr);
  yi = __fma_rn(f, limbs_to_double(hi, li), yi);
  // The sums err by less than 2^32 units of f: each element by 2^22 (u of two
  // parts, half a unit each, times |w| 2^-32) and 2^17 (low products), the
  // factors (half a unit times |u| 2^-32) by 2^30 in all.
  int const least = exponent_bits(f) + 63;
  bool const again_r = exponent_bits(yr) < least || F == kFixBad, again_i = exponent_bits(yi) < least || F == kFixBad;
  if (again_r || again_i) {
    cplx const y = general_entry<cplx, false>(S, c, ent, codes, width, Packed, 0, i);
    if (again_r) yr = y.re;
    if (again_i) yi = y.im;
  }
  c.store(0, i, yr);
  c.store(1, i, yi);
}

int launch_cplx(OperatorData& op, Columns const& c, cudaStream_t stream) {
  BasisData& b = *op.basis;
  OperatorTables const& tb = *op.tables;
  StreamForm const& sf = op.stream;
  uint64_t const D = b.D;
  if (D == 0) return LS_SUCCESS;
  auto* mx = op.fix_slots.as<unsigned long long>();
  auto* F = reinterpret_cast<int64_t*>(mx + op.fix_cols);
  int64_t* u = op.fix_u.as<int64_t>();
  if (int st = fix_enter(op, stream)) return st;
  if (!op.fix_clean) SED_TRY_CUDA(cudaMemsetAsync(mx, 0, (size_t)op.fix_cols * 8, stream));
  op.fix_clean = false;
  k_fix_max_cols<<<grid_size(2 * D, b.device, 8), kBlock, 0, stream>>>(c, D, mx);
  k_fix_convert_cols<2, true><<<grid_size(D + 1, b.device, 8), kBlock, (size_t)2 * tb.fix.n_div * 8, stream>>>(
      c, D, sf.row_class.as<uint8_t>(), tb.fix, mx, F, u);
  StreamView const S = stream_view(op);
  unsigned const grid = (unsigned)((sf.n_slices * 32 + kBlock - 1) / kBlock);
  size_t const smem = (size_t)((tb.n_codes + 7) & ~7u) * 16 + (size_t)tb.fix.n_div * 8;
  auto const* u4 = reinterpret_cast<int4 const*>(u);
  if (sf.packed) k_spmv_cplx<true><<<grid, kBlock, smem, stream>>>(S, tb.fix, tb.cplx, D, c, u4, F, mx);
  else k_spmv_cplx<false><<<grid, kBlock, smem, stream>>>(S, tb.fix, tb.cplx, D, c, u4, F, mx);
  note_launches(3);
  SED_TRY_CUDA(cudaGetLastError());
  op.fix_clean = !op.fix_captured;  // the SpMV has cleared the words again
  return fix_leave(op, stream);
}

// A pass of the fixed-point SpMV over c.cols <= K real columns (K = 1, 2, 4,
// 8, 16; the workspace holds K).
int launch_fix_cols(OperatorData& op, unsigned K, Columns const& c, cudaStream_t stream) {
  BasisData& b = *op.basis;
  OperatorTables const& tb = *op.tables;
  StreamForm const& sf = op.stream;
  uint64_t const D = b.D;
  auto* mx = op.fix_slots.as<unsigned long long>();
  auto* F = reinterpret_cast<int64_t*>(mx + op.fix_cols);
  int64_t* u = op.fix_u.as<int64_t>();
  if (int st = fix_enter(op, stream)) return st;
  if (!op.fix_clean) SED_TRY_CUDA(cudaMemsetAsync(mx, 0, (size_t)op.fix_cols * 8, stream));
  op.fix_clean = false;
  unsigned const vg = std::max(1u, grid_size(c.cx ? 2 * D : D, b.device, 8) / (c.cols > 2 ? 4 : 1));
  uint8_t const* cls = sf.row_class.as<uint8_t>();
  k_fix_max_cols<<<dim3(vg, c.cx ? c.cols / 2 : c.cols), kBlock, 0, stream>>>(c, D, mx);
  StreamView const S = stream_view(op);
  size_t const smem = fix_smem_bytes(tb, K);
  if (smem > 48 * 1024) return fail(LS_SYSTEM_ERROR, "fixed-point block matvec: tables exceed shared memory");
  auto pass = [&](auto k_tag) {
    constexpr int KK = decltype(k_tag)::value;
    constexpr int LL = KK > 4 ? KK / 4 : 1;
    uint64_t const warps = sf.n_slices * LL;
    unsigned const grid = (unsigned)((warps * 32 + kBlock - 1) / kBlock);
    unsigned const cg = grid_size((D + 1) * (KK > 2 ? KK / 2 : 1), b.device, 8);
    k_fix_convert_cols<KK, false><<<cg, kBlock, (size_t)KK * tb.fix.n_div * 8, stream>>>(c, D, cls, tb.fix, mx, F, u);
    fix_dispatch(tb, sf.packed, [&](auto packed, auto nv, auto sign) {
      if (c.f32) k_spmv_fix_cols<packed.value, nv.value, sign.value, KK, true><<<grid, kBlock, smem, stream>>>(S, tb.fix, D, c, u, F, mx);
      else k_spmv_fix_cols<packed.value, nv.value, sign.value, KK, false><<<grid, kBlock, smem, stream>>>(S, tb.fix, D, c, u, F, mx);
    });
  };
  switch (K) {
    case 1: pass(std::integral_constant<int, 1>{}); break;
    case 2: pass(std::integral_constant<int, 2>{}); break;
    case 4: pass(std::integral_constant<int, 4>{}); break;
    case 8: pass(std::integral_constant<int, 8>{}); break;
    default: pass(std::integral_constant<int, 16>{}); break;
  }
  note_launches(3);
  SED_TRY_CUDA(cudaGetLastError());
  op.fix_clean = !op.fix_captured;  // the SpMV has cleared the words again
  return fix_leave(op, stream);
}

// The gather copy stays with the operator. FP32 vectors took no memory before
// they took this path, so theirs is bounded: 1 GiB, 8 columns of 15.8 M rows
// (a single FP32 column uses the copy that every real operator has).
constexpr uint64_t kKeptCopy = 1ull << 30;
uint64_t copy_bytes(OperatorData const& op, unsigned K) { return (op.basis->D + 1) * K * 8; }
}  // namespace

// Below this size the two launches more per column cost what the sums save.
// Calls of 1 / 7 / 16 columns in us, general kernels and this one: 0.7 M
// elements 35 / 142 / 280 and 34 / 159 / 346, 1.4 M 47 / 227 / 465 and
// 37 / 175 / 378.
bool cplx_sums(OperatorData const& op) {
  return op.tables->cplx_ok && op.stream.n_elements >= ((uint64_t)1 << 20) && copy_bytes(op, 2) <= kKeptCopy;
}

// Whether vectors of this dtype go through launch_fix_cols. FP64 columns
// always do. FP32 and complex64 ones do from 2^21 and 2^20 elements on: below,
// the three launches more cost what the sums save (290 000 elements of a
// complex column: 30 us in the general kernel, 37 here; 77 M FP32 ones: 397 and
// 164). The rule does not look at the width of the block, so that a column's
// product does not depend on the columns beside it. They do not where one
// column's gather copy would be larger than kKeptCopy, nor while the caller's
// stream is being captured, where the shared workspace could be overwritten
// between replays (the general kernels use none), nor when a captured FP64
// product holds the workspace.
bool fix_cols_apply(OperatorData const& op, int dtype, bool use_stream, cudaStream_t stream) {
  if (!use_stream || dtype == 3 || (dtype != 1 && op.fix_captured)) return false;
  if (op.tables->cplx_ok) {
    if (dtype != 2 || !cplx_sums(op)) return false;
  } else {
    if (!op.tables->fix_ok || op.fix_cols < 1) return false;
    if (dtype == 1) return true;
    if (op.stream.n_elements < ((uint64_t)1 << (dtype == 2 ? 20 : 21))) return false;
    if (dtype == 2 && copy_bytes(op, 2) > kKeptCopy) return false;
  }
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return cap == cudaStreamCaptureStatusNone;
}

// The first `block` columns in passes of fixed width, widest first; *done
// counts the columns taken. A pass is padded to a power of two (three
// columns to 4, 5 to 7 to 8, 13 to 15 to 16): an element costs 4 + 8 K bytes
// of stream and gather, so that one padded pass moves less than two exact
// ones (7 columns: 68 against 36 + 20 + 12 bytes and three reads of the
// entries), except at 9 to 12 (8 + 4: 104 against 132). Stops early, with
// success, where the workspace for even the narrowest pass cannot be had:
// the caller's general path does the rest.
int fix_cols_blocks(OperatorData& op, int dtype, uint64_t block, char const* x, uint64_t ldx, char* y, uint64_t ldy,
                    size_t es, cudaStream_t stream, uint64_t* done) {
  if (op.tables->cplx_ok) {
    if (int st = fix_reserve(op, 2)) return st == LS_OUT_OF_MEMORY ? LS_SUCCESS : st;
    for (; *done < block; ++*done)
      if (int st = launch_cplx(op, {x + *done * ldx * es, y + *done * ldy * es, ldx, ldy, 2, true, true}, stream))
        return st;
    return LS_SUCCESS;
  }
  // a pass keeps K tables of row factors in shared memory: at most kmax
  // columns fit in 48 KB
  size_t const table = (size_t)op.tables->fix.n_div * op.tables->fix_nv * 8;
  unsigned const kmax = (unsigned)std::min<size_t>(16, (48 * 1024 - op.tables->fix.n_codes - 1) / table);
  bool const cx = dtype == 2;
  unsigned const per = cx ? 2 : 1;  // real columns per column
  while (*done < block) {
    uint64_t const left = (block - *done) * per;
    unsigned K = 1;
    while (K < left && K < 16) K *= 2;
    if (left >= 9 && left <= 12) K = 8;
    while (K > per && (K > kmax || (dtype != 1 && copy_bytes(op, K) > kKeptCopy))) K /= 2;
    if (K > kmax) return LS_SUCCESS;
    while (int st = fix_reserve(op, K)) {
      if (st != LS_OUT_OF_MEMORY) return st;
      if (K <= per) return LS_SUCCESS;
      K /= 2;
    }
    if (K == 1 && dtype == 1) return LS_SUCCESS;  // launch_apply_fix
    unsigned const cols = (unsigned)std::min<uint64_t>(left, K);
    Columns const c{x + *done * ldx * es, y + *done * ldy * es, ldx, ldy, cols, dtype == 0 || dtype == 2, cx};
    if (int st = launch_fix_cols(op, K, c, stream)) return st;
    *done += cols / per;
  }
  return LS_SUCCESS;
}

}  // namespace sed
