// lanczos.cu — the device eigensolver behind sed_eigh, replacing the PRIMME
// call at src/SpinED.hs:404 (options at src/SpinED.hs:383-394: smallest
// eigenvalues, tolerance, basis and block sizes, per-iteration monitor).
//
// Single-vector Lanczos with every Krylov vector resident in HBM:
//   w = H v_k (streamed SpMV; its epilogue also yields alpha_k = <v_k, w>)
//   w -= alpha_k v_k + beta_{k-1} v_{k-1}      (+ CGS2 against V when nev > 1)
//   beta_k = ||w||, v_{k+1} = w / beta_k
// The step index lives in device memory, so one CUDA graph holding `check`
// steps is replayed for the whole run; the sums (alpha, beta) are finished by
// the last block of the kernel that forms them, so a step is three kernels.
// Every `check` steps the host solves the tridiagonal T_k for its lowest
// eigenpair(s) while the next replay runs (Rayleigh-quotient iteration seeded
// with the previous Ritz vector and certified by a Sturm count; Sturm
// multisection and inverse iteration otherwise) and ends the cycle when
// beta_k |s_k| <= tol / 2. The Ritz vector psi = V s is then formed in one
// pass and its true residual ||H psi - E psi|| recomputed in FP64; the run
// restarts from psi until that residual meets the tolerance.
//
// Precision SED_PRECISION_MIXED runs the bulk of the iterations with FP32
// Krylov vectors and FP32 SpMV arithmetic (reductions, alpha/beta, the
// tridiagonal solve stay FP64), then refines the FP32 Ritz vector with the
// FP64 iteration above.
#include <chrono>
#include <cmath>
#include <cstring>

#include "operator_impl.cuh"
#include "tridiagonal.hpp"

namespace sed {
namespace {

constexpr unsigned kMaxNev = 16;

// What the step kernels share in device memory. alpha and beta follow it in
// the same buffer (state_bytes), so that one copy per chunk of steps shows
// the host all it needs.
struct LzHeader {
  uint32_t k;       // newest normalised Krylov vector
  uint32_t stop;    // kRunning, kFull or kBreakdown
  uint32_t m_max;   // stored vectors
  uint32_t size;    // order of T so far
  uint32_t steps;   // Lanczos steps taken
  uint32_t pad[11];
};
static_assert(sizeof(LzHeader) == 64, "alpha starts on a 64-byte boundary");

enum : uint32_t { kRunning = 0, kConverged = 1, kFull = 2, kBreakdown = 3 };

size_t state_bytes(uint32_t m) { return sizeof(LzHeader) + (size_t)m * 16; }

// ------------------------------------------------------------ vector ops --

template <class X>
__device__ __forceinline__ typename Store<X>::V ld(X const* p, uint64_t i) { return Store<X>::load(p, i); }

template <class X>
__device__ __forceinline__ double norm2(X const* p, uint64_t i) {
  auto const v = Store<X>::load(p, i);
  return dot_re(v, v);
}

// The sum of the matvec's partials where its grid is too large to finish it
// (finish_sum): ind.sum[k]. Virtual thread t of 1024 adds partials t, t +
// 1024, ... in eight running sums; then a butterfly per warp, and the 32
// warps in order by the last block to finish. One warp per block: on one SM
// the 61 738 FP64 additions of a 15.8 M-row SpMV take 17 us of its FP64 pipe
// alone (30 us in all as one block of 1024 threads), on 32 SMs 4 us.
__global__ void __launch_bounds__(32) k_sum_partials(unsigned n, Indirect ind, double* warp_sum, uint32_t* done) {
  if (*ind.stop) return;
  double const* partial = ind.partial;
  double a[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  unsigned i = blockIdx.x * 32 + threadIdx.x;
  for (; i + 31 * 1024 < n; i += 32 * 1024) {
    double v[32];
#pragma unroll
    for (unsigned q = 0; q < 32; ++q) v[q] = partial[i + q * 1024];
#pragma unroll
    for (unsigned q = 0; q < 32; ++q) a[q & 7] += v[q];
  }
  for (; i + 7 * 1024 < n; i += 8 * 1024) {
    double v[8];
#pragma unroll
    for (unsigned q = 0; q < 8; ++q) v[q] = partial[i + q * 1024];
#pragma unroll
    for (unsigned q = 0; q < 8; ++q) a[q] += v[q];
  }
  for (; i < n; i += 1024) a[0] += partial[i];
  double s = ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  uint32_t last = 0;
  if (threadIdx.x == 0) {
    warp_sum[blockIdx.x] = s;
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return;
  __threadfence();
  double const mine = __ldcg(warp_sum + threadIdx.x);
  s = 0.0;
  for (int w = 0; w < 32; ++w) s += __shfl_sync(0xffffffffu, mine, w);
  if (threadIdx.x == 0) {
    *done = 0;
    ind.sum[*ind.k] = s;
    if (ind.clear) *ind.clear = 0;
  }
}

// One Krylov matvec with alpha_k; ind.partial holds ceil(D / kBlock) + 32
// doubles.
template <class Apply>
int apply_with_alpha(Indirect ind, uint64_t D, cudaStream_t stream, Apply&& apply) {
  uint64_t const blocks = (D + kBlock - 1) / kBlock;
  uint32_t* const done = ind.done;
  if (blocks > kFusedSumBlocks) ind.done = nullptr;
  if (int st = apply(ind)) return st;
  if (!ind.done) { k_sum_partials<<<32, 32, 0, stream>>>((unsigned)blocks, ind, ind.partial + blocks, done); note_launches(1); }
  return LS_SUCCESS;
}

// Fused fixed-point Lanczos step (FP64): the last kernel that changes w leaves max |w|
// (bit pattern) in *wmax and k_scale_next writes, next to v_{k+1} = w /
// beta_k, the next matvec's gather copy u = round(sqrt(S) v_{k+1} 2^F) and
// F, so that matvec skips its own pre-pass. `on` is false otherwise.
struct FixStep {
  bool on;
  unsigned long long* wmax;
  int64_t* F;
  int64_t* u;
  uint8_t const* row_class;
  FixView fv;
};

// *out = max(*out, the block's largest m); red holds one word per warp.
__device__ __forceinline__ void block_max_to(unsigned long long m, unsigned long long* red, unsigned long long* out) {
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (unsigned q = 1; q < kBlock / 32; ++q) m = max(m, red[q]);
    atomicMax(out, m);
  }
}

// w = w - alpha_k v_k - beta_{k-1} v_{k-1}; with Norm also beta_k = ||w|| (by
// the last block) and max |w| (otherwise the Gram-Schmidt passes follow).
template <class X, bool Norm>
__global__ void k_update(X* __restrict__ V, uint64_t ld_v, uint64_t D, LzHeader const* h,
                         double const* __restrict__ alpha, double* __restrict__ beta,
                         double* __restrict__ partial, uint32_t* __restrict__ done,
                         unsigned long long* __restrict__ wmax) {
  using Vt = typename Store<X>::V;
  __shared__ double red[kBlock / 32];
  __shared__ unsigned long long redm[kBlock / 32];
  if (h->stop) return;
  unsigned long long m = 0;
  uint32_t const k = h->k;
  X* w = V + (uint64_t)(k + 1) * ld_v;
  X const* v = V + (uint64_t)k * ld_v;
  X const* vp = k ? V + (uint64_t)(k - 1) * ld_v : v;
  double const a = alpha[k];
  double const b = k ? beta[k - 1] : 0.0;
  double part = 0.0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x) {
    Vt wi = Store<X>::load(w, i);
    Vt const vi = Store<X>::load(v, i), vpi = Store<X>::load(vp, i);
    if constexpr (std::is_same<Vt, double>::value) {
      wi = fma(-a, vi, fma(-b, vpi, wi));
    } else {
      wi.re = fma(-a, vi.re, fma(-b, vpi.re, wi.re));
      wi.im = fma(-a, vi.im, fma(-b, vpi.im, wi.im));
    }
    Store<X>::store(w, i, wi);
    if constexpr (!Norm) continue;
    part += dot_re(wi, wi);
    if constexpr (std::is_same<Vt, double>::value)
      m = max(m, (unsigned long long)__double_as_longlong(wi) & 0x7FFFFFFFFFFFFFFFull);
  }
  if constexpr (!Norm) return;
  double const tot = block_sum(part, red);
  if (wmax) block_max_to(m, redm, wmax);
  finish_sum(tot, partial, done, [&](double s) { beta[k] = sqrt(s); });
}

// Classical Gram-Schmidt pass against V[0..k]: c_j = <V_j, w> (partials per
// block and vector, 16 vectors per blockIdx.y). FP64 issue bounds it (1.75
// lanes per clock and SM): one FMA per element, and one addition per element
// to add a block's 256 products where each thread has about one row (D near
// 304 000). The 16 sums of a warp are transposed while they are added (8 + 4
// + 2 + 1 + 1 additions per lane instead of 16 x 5; each pair of lanes adds
// the same two numbers as a butterfly of one sum, so the bits are the same):
// 251 -> 103 us per pass over 56 vectors of 361 270 rows on average. The
// vector count NJ of the block's group is a template parameter of the loop
// body, chosen on the device from k: a predicated-off FP64 FMA still takes
// its issue slot, so the body never pads to 16.
template <int NJ, class X>
__device__ __forceinline__ void cgs_dots_body(X const* __restrict__ V, uint64_t ld_v, uint64_t D, X const* w,
                                              uint32_t j0, double (*red)[16], double* __restrict__ partial) {
  double acc[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) acc[j] = 0.0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x) {
    auto const wi = Store<X>::load(w, i);
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[j] += dot_re(Store<X>::load(V + (uint64_t)(j0 + j) * ld_v, i), wi);
  }
  // after the step with offset o a lane holds the sums j whose bit o / 2 is
  // set as its own lane bit o is
  uint32_t const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o >= 2; o >>= 1) {
    bool const up = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (j >= o / 2) break;
      double const give = up ? acc[j] : acc[j + o / 2], keep = up ? acc[j + o / 2] : acc[j];
      acc[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
  if (!(lane & 1)) red[warp][lane >> 1] = acc[0];
  __syncthreads();
  if (threadIdx.x < NJ) {
    double t = 0.0;
    for (int q = 0; q < (int)kBlock / 32; ++q) t += red[q][threadIdx.x];
    partial[(uint64_t)(j0 + threadIdx.x) * gridDim.x + blockIdx.x] = t;
  }
}

template <class X>
__global__ void k_cgs_dots(X const* __restrict__ V, uint64_t ld_v, uint64_t D, LzHeader const* h,
                           double* __restrict__ partial /* [m_max][gridDim.x] */) {
  __shared__ double red[kBlock / 32][16];
  if (h->stop) return;
  uint32_t const k = h->k;
  uint32_t const j0 = blockIdx.y * 16;
  if (j0 > k) return;  // uniform per block
  uint32_t const nj = min(16u, k + 1 - j0);
  X const* w = V + (uint64_t)(k + 1) * ld_v;
  switch (nj) {
#define SED_CGS(N) \
  case N: cgs_dots_body<N, X>(V, ld_v, D, w, j0, red, partial); break;
    SED_CGS(1) SED_CGS(2) SED_CGS(3) SED_CGS(4) SED_CGS(5) SED_CGS(6) SED_CGS(7) SED_CGS(8)
    SED_CGS(9) SED_CGS(10) SED_CGS(11) SED_CGS(12) SED_CGS(13) SED_CGS(14) SED_CGS(15) SED_CGS(16)
#undef SED_CGS
  }
}

// c_j = the sum of vector j's partials, one block per vector (as one block
// for all of them: 190 us at 56 vectors on average; 5 us so).
__global__ void __launch_bounds__(1024) k_cgs_reduce(double const* __restrict__ partial, unsigned nb,
                                                     LzHeader const* h, double* __restrict__ coef,
                                                     double* __restrict__ alpha) {
  __shared__ double red[1024 / 32];
  uint32_t const k = h->k, j = blockIdx.x;
  if (h->stop || j > k) return;
  double s = 0.0;
  for (unsigned i = threadIdx.x; i < nb; i += blockDim.x) s += partial[(uint64_t)j * nb + i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) {
    coef[j] = s;
    if (j == k) alpha[k] += s;  // the projection on v_k corrects alpha_k
  }
}

// w -= sum_j c_j V_j; on the last pass also beta_k = ||w|| and (wmax not
// null) max |w|.
template <class X, bool Last>
__global__ void __launch_bounds__(kBlock) k_cgs_update(X* __restrict__ V, uint64_t ld_v, uint64_t D, LzHeader const* h,
                             double const* __restrict__ coef, double* __restrict__ beta,
                             double* __restrict__ partial, uint32_t* __restrict__ done,
                             unsigned long long* __restrict__ wmax) {
  using Vt = typename Store<X>::V;
  __shared__ double red[kBlock / 32];
  __shared__ unsigned long long redm[kBlock / 32];
  __shared__ double c[2048];
  if (h->stop) return;
  uint32_t const k = h->k;
  for (uint32_t j = threadIdx.x; j <= k; j += blockDim.x) c[j] = coef[j];
  __syncthreads();
  X* w = V + (uint64_t)(k + 1) * ld_v;
  double part = 0.0;
  unsigned long long m = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x) {
    Vt wi = Store<X>::load(w, i);
#pragma unroll 8
    for (uint32_t j = 0; j <= k; ++j) {
      Vt const vj = Store<X>::load(V + (uint64_t)j * ld_v, i);
      if constexpr (std::is_same<Vt, double>::value) {
        wi = fma(-c[j], vj, wi);
      } else {
        wi.re = fma(-c[j], vj.re, wi.re);
        wi.im = fma(-c[j], vj.im, wi.im);
      }
    }
    Store<X>::store(w, i, wi);
    if constexpr (Last) {
      part += dot_re(wi, wi);
      if constexpr (std::is_same<Vt, double>::value)
        m = max(m, (unsigned long long)__double_as_longlong(wi) & 0x7FFFFFFFFFFFFFFFull);
    }
  }
  if constexpr (Last) {
    double const tot = block_sum(part, red);
    if (wmax) block_max_to(m, redm, wmax);
    finish_sum(tot, partial, done, [&](double t) { beta[k] = sqrt(t); });
  }
}

// Ends the step: the last block to get here advances k, or stops the run
// when the storage is full or the Krylov space is exhausted. Every block has
// read the header before its thread 0 is counted.
__device__ __forceinline__ void advance_step(LzHeader* h, double b, uint32_t* done) {
  __syncthreads();
  if (threadIdx.x != 0 || atomicAdd(done, 1u) != gridDim.x - 1) return;
  *done = 0;
  uint32_t const k = h->k;
  h->size = k + 1;
  h->steps += 1;
  if (!(b > 0.0) || !isfinite(b))
    h->stop = kBreakdown;
  else if (k + 2 >= h->m_max)
    h->stop = kFull;
  else
    h->k = k + 1;
}

// v_{k+1} = w / beta_k (and the next matvec's gather copy), then the next step.
template <class X>
__global__ void k_scale_next(X* __restrict__ V, uint64_t ld_v, uint64_t D, LzHeader* h,
                             double const* __restrict__ beta, uint32_t* __restrict__ done, FixStep fx) {
  __shared__ double fac[kFixMaxClasses];
  if (h->stop) return;
  uint32_t const k = h->k;
  double const b = beta[k];
  if (!(b > 0.0)) {
    advance_step(h, b, done);
    return;
  }
  double const inv = 1.0 / b;
  X* w = V + (uint64_t)(k + 1) * ld_v;
  if constexpr (std::is_same<X, double>::value) {
    if (fx.on) {
      // max |v_j| = fl(max |w_j| inv): the rounding of v_j = w_j inv is
      // monotone in |w_j|, so this bounds every |v_j| exactly
      double const vmax = __longlong_as_double((long long)*fx.wmax) * inv;
      int64_t const F = fix_exponent((uint64_t)__double_as_longlong(fabs(vmax)), fx.fv.bound);
      if (blockIdx.x == 0 && threadIdx.x == 0) *fx.F = F;
      int64_t const F1 = (F == kFixBad || (F >= -1000 && F <= 1000)) ? 0 : F / 2;
      double const p1 = fix_pow2(F1);
      double const p2 = F == kFixBad ? 0.0 : fix_pow2(F - F1);
      for (uint32_t c = threadIdx.x; c < fx.fv.n_div; c += blockDim.x) fac[c] = fx.fv.sqrt_s[c] * p2;
      __syncthreads();
      for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
           i += (uint64_t)gridDim.x * blockDim.x) {
        double const v = inv * w[i];
        w[i] = v;
        fx.u[i] = F == kFixBad ? 0 : fix_round((F1 ? v * p1 : v) * fac[fx.row_class[i]]);
      }
      advance_step(h, b, done);
      return;
    }
  }
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x) {
    auto v = Store<X>::load(w, i);
    Store<X>::store(w, i, mulv(inv, v));
  }
  advance_step(h, b, done);
}

// out_i = sum_{j < n} s_j V_j[i]
template <class X, class Y>
__global__ void k_ritz(X const* __restrict__ V, uint64_t ld_v, uint64_t D, double const* __restrict__ s,
                       uint32_t n, Y* __restrict__ out) {
  __shared__ double c[2048];
  for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) c[j] = s[j];
  __syncthreads();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x) {
    typename Store<Y>::V acc = zero<typename Store<Y>::V>();
    for (uint32_t j = 0; j < n; ++j) {
      auto const v = Store<X>::load(V + (uint64_t)j * ld_v, i);
      if constexpr (std::is_same<typename Store<Y>::V, double>::value) {
        acc = fma(c[j], v, acc);
      } else {
        acc.re = fma(c[j], v.re, acc.re);
        acc.im = fma(c[j], v.im, acc.im);
      }
    }
    Store<Y>::store(out, i, acc);
  }
}

// partial dots for <x,x>, <x,y> and ||y - e x||^2 (mode 0: first two; 1: last)
template <class X>
__global__ void k_dots(X const* __restrict__ x, X const* __restrict__ y, uint64_t D, double e,
                       int mode, double* __restrict__ partial) {
  __shared__ double red[kBlock / 32];
  double p0 = 0.0, p1 = 0.0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x) {
    auto const xi = Store<X>::load(x, i);
    auto const yi = Store<X>::load(y, i);
    if (mode == 0) {
      p0 += dot_re(xi, xi);
      p1 += dot_re(xi, yi);
    } else {
      auto const r = addv(yi, mulv(-e, xi));
      p0 += dot_re(r, r);
    }
  }
  double const t0 = block_sum(p0, red);
  double const t1 = block_sum(p1, red);
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = t0;
    partial[2 * blockIdx.x + 1] = t1;
  }
}

template <class X>
__global__ void k_scale(X* __restrict__ x, uint64_t D, double f) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x)
    Store<X>::store(x, i, mulv(f, Store<X>::load(x, i)));
}

template <class X, class Y>
__global__ void k_convert(X const* __restrict__ x, uint64_t D, Y* __restrict__ y) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x) {
    auto const v = Store<X>::load(x, i);
    if constexpr (std::is_same<decltype(v), typename Store<Y>::V const>::value) {
      Store<Y>::store(y, i, v);
    } else if constexpr (std::is_same<typename Store<Y>::V, cplx>::value) {
      Store<Y>::store(y, i, cplx{(double)v, 0.0});
    } else {
      Store<Y>::store(y, i, v.re);
    }
  }
}

// Element i of the start vector is uniform in [-1, 1) from Philox block i/2.
template <class X>
__global__ void k_random(X* __restrict__ x, uint64_t D, uint64_t seed) {
  for (uint64_t blk = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; blk < (D + 1) / 2;
       blk += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t c[4] = {(uint32_t)blk, (uint32_t)(blk >> 32), 0u, 0u};
    philox(c, (uint32_t)seed, (uint32_t)(seed >> 32));
    double const v0 = 2.0 * u01_53(c[0], c[1]) - 1.0;
    double const v1 = 2.0 * u01_53(c[2], c[3]) - 1.0;
    if constexpr (std::is_same<typename Store<X>::V, double>::value) {
      Store<X>::store(x, 2 * blk, v0);
      if (2 * blk + 1 < D) Store<X>::store(x, 2 * blk + 1, v1);
    } else {
      Store<X>::store(x, 2 * blk, cplx{v0, 0.0});
      if (2 * blk + 1 < D) Store<X>::store(x, 2 * blk + 1, cplx{v1, 0.0});
    }
  }
}

// ----------------------------------------------------------------- cycle --
// Host side of one Krylov cycle: replays the graph of `check` steps and
// solves T after each replay until the pairs converge, the device stops or
// `max_steps` are used up.
class Cycle {
 public:
  cudaGraphExec_t graph = nullptr;
  LzHeader* hdr = nullptr;   // device: header, alpha[m], beta[m]
  uint32_t m = 0, check = 1;
  uint32_t stop = kRunning;  // how the cycle ended (kRunning: out of steps)
  uint32_t steps = 0;        // steps of the cycle

  Cycle() = default;
  Cycle(Cycle const&) = delete;
  Cycle& operator=(Cycle const&) = delete;
  ~Cycle() {
    if (stream_) cudaStreamSynchronize(stream_);  // a replay and its copy may be in flight
    if (graph) cudaGraphExecDestroy(graph);
    for (cudaEvent_t e : ready_)
      if (e) cudaEventDestroy(e);
    pinned_give(pinned_);
  }

  double* alpha() const { return reinterpret_cast<double*>(hdr + 1); }
  double* beta() const { return alpha() + m; }

  int init(LzHeader* device_state, uint32_t m_max, uint32_t check_every) {
    hdr = device_state;
    m = m_max;
    check = check_every;
    if (int st = pinned_take(2 * state_bytes(m), pinned_)) return st;
    host_ = static_cast<char*>(pinned_.ptr);
    for (cudaEvent_t& e : ready_) SED_TRY_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return LS_SUCCESS;
  }

  // Captures `check` steps on `stream`.
  template <class Step>
  int capture(cudaStream_t stream, Step&& step) {
    stream_ = stream;
    cudaGraph_t g;
    SED_TRY_CUDA(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
    set_capturing(true);
    int st = LS_SUCCESS;
    for (uint32_t i = 0; i < check && st == LS_SUCCESS; ++i) st = step();
    set_capturing(false);
    cudaError_t e = cudaStreamEndCapture(stream, &g);
    if (st) {
      if (e == cudaSuccess) cudaGraphDestroy(g);
      return st;
    }
    SED_TRY_CUDA(e);
    cudaGraphGetNodes(g, nullptr, &nodes_);
    e = cudaGraphInstantiate(&graph, g, 0);
    cudaGraphDestroy(g);
    SED_TRY_CUDA(e);
    return LS_SUCCESS;
  }

  // Resets the header: the cycle starts from v_k0 (alpha and beta below k0
  // are the caller's). The copy leaves host_[0], which no replay uses yet.
  int start(cudaStream_t stream, uint32_t k0) {
    LzHeader h{};
    h.k = k0;
    h.m_max = m;
    h.size = k0;
    stream_ = stream;
    std::memcpy(host_, &h, sizeof(h));
    SED_TRY_CUDA(cudaMemcpyAsync(hdr, host_, sizeof(h), cudaMemcpyHostToDevice, stream));
    SED_TRY_CUDA(cudaStreamSynchronize(stream));
    return LS_SUCCESS;
  }

  // The next replay is queued before the host looks at the last one, so the
  // device does not wait for the host's solve, as long as the estimates are
  // more than 1000 times the tolerance: four steps gain less than that, so
  // the replay in flight when the cycle ends (its steps are not counted) is
  // at most the rare one.
  template <class Progress>
  int run(cudaStream_t stream, Tridiagonal& T, double tol_est, uint64_t max_steps, Progress&& progress) {
    T.restart();
    stop = kRunning;
    steps = 0;
    bool far = false;
    uint64_t launched = 0, seen = 0;
    while (true) {
      while (launched < seen + (far ? 2 : 1) && (launched == 0 || launched * check < max_steps)) {
        SED_TRY_CUDA(cudaGraphLaunch(graph, stream));
        note_launches(nodes_);
        SED_TRY_CUDA(cudaMemcpyAsync(slot(launched), hdr, state_bytes(m), cudaMemcpyDeviceToHost, stream));
        SED_TRY_CUDA(cudaEventRecord(ready_[launched & 1], stream));
        ++launched;
      }
      if (seen == launched) return LS_SUCCESS;  // out of steps
      SED_TRY_CUDA(cudaEventSynchronize(ready_[seen & 1]));
      LzHeader const& h = *reinterpret_cast<LzHeader const*>(slot(seen));
      double const* a = reinterpret_cast<double const*>(slot(seen) + sizeof(LzHeader));
      ++seen;
      steps = h.steps;
      bool const halted = h.stop != kRunning;
      uint32_t const n = halted ? h.size : h.size - h.size % check;
      bool const done = n > 0 && T.solve(a, a + m, n, h.stop == kBreakdown, tol_est);
      progress(steps);
      if (halted || done) {
        stop = h.stop == kBreakdown ? (uint32_t)kBreakdown : done ? (uint32_t)kConverged : (uint32_t)kFull;
        steps -= h.size - n;  // steps past the solved order
        return LS_SUCCESS;
      }
      far = n > 0;
      if (far) far = *std::max_element(T.est.begin(), T.est.end()) > 1e3 * tol_est;
    }
  }

 private:
  PinnedBuffer pinned_;
  char* host_ = nullptr;  // two copies of the state, pinned
  cudaStream_t stream_ = nullptr;
  cudaEvent_t ready_[2] = {nullptr, nullptr};
  size_t nodes_ = 0;
  char* slot(uint64_t i) const { return host_ + (i & 1) * state_bytes(m); }
};

// ------------------------------------------------------------- driver ----

struct Workspace {
  DeviceBuffer V, buf, scratch;
  DevicePart state, s, partial, done, cgs_partial, coef, ritz, y;  // in buf
};

int elem_bytes(int dtype) { return dtype == 0 ? 4 : dtype == 1 ? 8 : dtype == 2 ? 8 : 16; }

template <class X>
double host_sum(DevicePart const& partial, unsigned n, unsigned stride, unsigned off, cudaStream_t s,
                int* st) {
  std::vector<double> h((size_t)n * stride);
  cudaError_t e = cudaMemcpyAsync(h.data(), partial.ptr, h.size() * 8, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    *st = fail(LS_CUDA_ERROR, std::string("reading partial sums: ") + cudaGetErrorString(e));
    return 0.0;
  }
  double t = 0.0;
  for (unsigned i = 0; i < n; ++i) t += h[(size_t)i * stride + off];
  return t;
}

template <class X>
struct Solver {
  OperatorData& op;
  int dtype;  // storage dtype of X
  uint64_t D;
  cudaStream_t stream;
  Workspace ws;
  uint32_t m_max = 0;
  unsigned vblocks = 0;
  bool reorth = false;
  Cycle cycle;
  FixStep fx{};            // fused fixed-point step (FP64, stream form)

  Solver(OperatorData& o, int dt, cudaStream_t s) : op(o), dtype(dt), D(o.basis->D), stream(s) {}
  ~Solver() {
    cudaStreamSynchronize(stream);  // a replay may be in flight on an early exit
    krylov_give(ws.V);
  }

  X* V() const { return ws.V.as<X>(); }
  LzHeader* hdr() const { return cycle.hdr; }

  int init(uint32_t m, uint32_t check, bool reorthogonalise) {
    m_max = m;
    reorth = reorthogonalise;
    int dev = op.basis->device;
    vblocks = grid_size(D, dev, 8);
    if (int st = krylov_take((size_t)m_max * D * sizeof(X), ws.V)) return st;
    uint64_t const nb = std::max<uint64_t>((D + kBlock - 1) / kBlock, vblocks) + 32;
    DeviceParts parts;
    parts.add(ws.state, state_bytes(m_max));
    parts.add(ws.s, (size_t)m_max * 8);
    parts.add(ws.partial, nb * 16);
    parts.add(ws.done, 16);
    if (reorth) {
      parts.add(ws.cgs_partial, (size_t)m_max * vblocks * 8);
      parts.add(ws.coef, (size_t)m_max * 8);
    }
    parts.add(ws.ritz, D * sizeof(X));
    parts.add(ws.y, D * sizeof(X));
    if (int st = parts.allocate(ws.buf)) return st;
    if (int st = cycle.init(ws.state.as<LzHeader>(), m_max, check)) return st;
    SED_TRY_CUDA(cudaMemsetAsync(ws.state.ptr, 0, state_bytes(m_max), stream));
    SED_TRY_CUDA(cudaMemsetAsync(ws.done.ptr, 0, 16, stream));
    FixSlots fs;
    if (std::is_same<X, double>::value && fix_slots(op, &fs))
      fx = FixStep{true, fs.max_bits, fs.F, fs.u, fs.row_class, fs.view};
    return LS_SUCCESS;
  }

  // Fused step: the matvec's pre-pass for the current v_k, needed whenever
  // v_k was not produced by k_scale_next (the start and every restart) or
  // the workspace was used by another matvec since.
  int prescale() {
    if (!fx.on) return LS_SUCCESS;
    Indirect ind;
    ind.k = &hdr()->k;
    ind.stop = &hdr()->stop;
    ind.ld = D;
    return fix_prescale(op, reinterpret_cast<double const*>(V()), ind, stream);
  }

  // One Lanczos step (all kernels read k from the header).
  int enqueue_step() {
    LzHeader* h = hdr();
    double *alpha = cycle.alpha(), *beta = cycle.beta(), *partial = ws.partial.template as<double>();
    uint32_t* done = ws.done.template as<uint32_t>();
    Indirect ind;
    ind.k = &h->k;
    ind.stop = &h->stop;
    ind.ld = D;
    ind.partial = partial;
    ind.done = done;
    ind.sum = alpha;
    ind.clear = fx.on ? fx.wmax : nullptr;  // the step's max |w| starts at zero
    ind.prescaled = fx.on;
    if (int st = apply_with_alpha(ind, D, stream, [&](Indirect i) { return operator_apply_krylov(op, dtype, V(), i, stream); }))
      return st;
    unsigned long long* const wmax = fx.on ? fx.wmax : nullptr;
    if (!reorth) {
      { k_update<X, true><<<vblocks, kBlock, 0, stream>>>(V(), D, D, h, alpha, beta, partial, done, wmax); note_launches(1); }
    } else {
      double *cp = ws.cgs_partial.template as<double>(), *coef = ws.coef.template as<double>();
      { k_update<X, false><<<vblocks, kBlock, 0, stream>>>(V(), D, D, h, alpha, beta, partial, done, nullptr); note_launches(1); }
      for (int pass = 0; pass < 2; ++pass) {
        dim3 grid(vblocks, (m_max + 15) / 16);
        { k_cgs_dots<X><<<grid, kBlock, 0, stream>>>(V(), D, D, h, cp); note_launches(1); }
        { k_cgs_reduce<<<m_max, 1024, 0, stream>>>(cp, vblocks, h, coef, alpha); note_launches(1); }
        if (pass == 0) { k_cgs_update<X, false><<<vblocks, kBlock, 0, stream>>>(V(), D, D, h, coef, beta, partial, done, nullptr); }
        else { k_cgs_update<X, true><<<vblocks, kBlock, 0, stream>>>(V(), D, D, h, coef, beta, partial, done, wmax); }
        note_launches(1);
      }
    }
    { k_scale_next<X><<<vblocks, kBlock, 0, stream>>>(V(), D, D, h, beta, done, fx); note_launches(1); }
    SED_TRY_CUDA(cudaGetLastError());
    return LS_SUCCESS;
  }

  int capture() {
    return cycle.capture(stream, [&] { return enqueue_step(); });
  }

  // Writes x (device, type X) to dst (host or device) as `out_dtype`.
  int store(X const* x, int out_dtype, void* dst) {
    int const own = std::is_same<X, double>::value ? 1 : 3;
    if (out_dtype == own) {
      SED_TRY_CUDA(cudaMemcpyAsync(dst, x, D * sizeof(X), cudaMemcpyDefault, stream));
      SED_TRY_CUDA(cudaStreamSynchronize(stream));
      return LS_SUCCESS;
    }
    size_t const es = (size_t)elem_bytes(out_dtype);
    if (!ws.scratch.ptr || ws.scratch.bytes < D * es)
      if (int st = ws.scratch.allocate(D * es)) return st;
    switch (out_dtype) {
      case 0: { k_convert<X, float><<<vblocks, kBlock, 0, stream>>>(x, D, ws.scratch.as<float>()); note_launches(1); } break;
      case 1: { k_convert<X, double><<<vblocks, kBlock, 0, stream>>>(x, D, ws.scratch.as<double>()); note_launches(1); } break;
      case 2: { k_convert<X, float2><<<vblocks, kBlock, 0, stream>>>(x, D, ws.scratch.as<float2>()); note_launches(1); } break;
      default: { k_convert<X, double2><<<vblocks, kBlock, 0, stream>>>(x, D, ws.scratch.as<double2>()); note_launches(1); } break;
    }
    SED_TRY_CUDA(cudaGetLastError());
    SED_TRY_CUDA(cudaMemcpyAsync(dst, ws.scratch.ptr, D * es, cudaMemcpyDefault, stream));
    SED_TRY_CUDA(cudaStreamSynchronize(stream));
    return LS_SUCCESS;
  }

  // ||x||, normalises x in place.
  int normalise_vec(X* x, double* out_norm) {
    { k_dots<X><<<vblocks, kBlock, 0, stream>>>(x, x, D, 0.0, 0, ws.partial.as<double>()); note_launches(1); }
    SED_TRY_CUDA(cudaGetLastError());
    int st = LS_SUCCESS;
    double const n2 = host_sum<X>(ws.partial, vblocks, 2, 0, stream, &st);
    if (st) return st;
    double const nrm = std::sqrt(n2);
    if (!(nrm > 0.0)) return fail(LS_INVALID_ARGUMENT, "start vector is zero");
    { k_scale<X><<<vblocks, kBlock, 0, stream>>>(x, D, 1.0 / nrm); note_launches(1); }
    SED_TRY_CUDA(cudaGetLastError());
    if (out_norm) *out_norm = nrm;
    return LS_SUCCESS;
  }

  // y = H x with residual: returns E = <x,Hx>/<x,x> and ||Hx - E x||/||x||.
  int residual(X* x, double* E, double* r) {
    if (int st = operator_apply_device(op, dtype, 1, x, D, ws.y.ptr, D, stream, SED_FORM_AUTO)) return st;
    { k_dots<X><<<vblocks, kBlock, 0, stream>>>(x, ws.y.as<X>(), D, 0.0, 0, ws.partial.as<double>()); note_launches(1); }
    int st = LS_SUCCESS;
    std::vector<double> h(2 * (size_t)vblocks);
    SED_TRY_CUDA(cudaMemcpyAsync(h.data(), ws.partial.ptr, h.size() * 8, cudaMemcpyDeviceToHost, stream));
    SED_TRY_CUDA(cudaStreamSynchronize(stream));
    double xx = 0.0, xy = 0.0;
    for (unsigned i = 0; i < vblocks; ++i) {
      xx += h[2 * i];
      xy += h[2 * i + 1];
    }
    *E = xy / xx;
    { k_dots<X><<<vblocks, kBlock, 0, stream>>>(x, ws.y.as<X>(), D, *E, 1, ws.partial.as<double>()); note_launches(1); }
    double const rr = host_sum<X>(ws.partial, vblocks, 2, 0, stream, &st);
    if (st) return st;
    *r = std::sqrt(rr / xx);
    return LS_SUCCESS;
  }
};

// ------------------------------------------------- mixed precision ----
// FP32 Lanczos steps: vectors and their updates in FP32, reductions per warp
// in FP32 and per block in FP64.
__global__ void k_update32(float* __restrict__ V, uint64_t ld_v, uint64_t D, LzHeader const* h,
                           double const* __restrict__ alpha, double* __restrict__ beta,
                           double* __restrict__ partial, uint32_t* __restrict__ done) {
  __shared__ double red[kBlock / 32];
  if (h->stop) return;
  uint32_t const k = h->k;
  float* w = V + (uint64_t)(k + 1) * ld_v;
  float const* v = V + (uint64_t)k * ld_v;
  float const* vp = k ? V + (uint64_t)(k - 1) * ld_v : v;
  float const a = (float)alpha[k];
  float const b = k ? (float)beta[k - 1] : 0.0f;
  float part = 0.0f;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x) {
    float const wi = fmaf(-a, v[i], fmaf(-b, vp[i], w[i]));
    w[i] = wi;
    part = fmaf(wi, wi, part);
  }
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  double const tot = block_sum((threadIdx.x & 31) == 0 ? (double)part : 0.0, red);
  finish_sum(tot, partial, done, [&](double s) { beta[k] = sqrt(s); });
}

__global__ void k_scale_next32(float* __restrict__ V, uint64_t ld_v, uint64_t D, LzHeader* h,
                               double const* __restrict__ beta, uint32_t* __restrict__ done) {
  if (h->stop) return;
  uint32_t const k = h->k;
  double const b = beta[k];
  if (!(b > 0.0)) {
    advance_step(h, b, done);
    return;
  }
  float const inv = (float)(1.0 / b);
  float* w = V + (uint64_t)(k + 1) * ld_v;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x)
    w[i] *= inv;
  advance_step(h, b, done);
}

// out = s_0 psi + sum_{j=1}^{n-1} s_j V_j, accumulated in FP64.
__global__ void k_ritz_mixed(double const* __restrict__ psi, float const* __restrict__ V, uint64_t ld_v,
                             uint64_t D, double const* __restrict__ s, uint32_t n, double* __restrict__ out) {
  __shared__ double c[2048];
  for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) c[j] = s[j];
  __syncthreads();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x) {
    double acc = c[0] * psi[i];
    for (uint32_t j = 1; j < n; ++j) acc = fma(c[j], (double)V[(uint64_t)j * ld_v + i], acc);
    out[i] = acc;
  }
}

// v0 = (float) psi, v1 = (float) ((y - theta psi) / rn)
__global__ void k_start_cycle(double const* __restrict__ psi, double const* __restrict__ y, uint64_t D,
                              double theta, double inv_rn, float* __restrict__ v0, float* __restrict__ v1) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D;
       i += (uint64_t)gridDim.x * blockDim.x) {
    double const p = psi[i];
    v0[i] = (float)p;
    v1[i] = (float)((y[i] - theta * p) * inv_rn);
  }
}

uint32_t auto_basis(uint64_t D, size_t elem, uint32_t nev, uint32_t requested) {
  size_t free_b = 0;
  (void)device_free_bytes(&free_b);
  uint64_t const cap_mem = (uint64_t)(0.6 * (double)free_b) / std::max<uint64_t>(1, D * elem);
  uint64_t m = requested ? requested : 400;
  m = std::min<uint64_t>(m, cap_mem);
  m = std::min<uint64_t>(m, D + 1);
  m = std::min<uint64_t>(m, 2048);
  m = std::max<uint64_t>(m, std::min<uint64_t>(D + 1, nev + 2));
  return (uint32_t)m;
}

template <class X>
int solve(OperatorData& op, int out_dtype, sed_eigh_options const& o, double* evals, void* evecs,
          uint64_t ldv, double* rnorms, sed_eigh_info* info) {
  int const dtype = std::is_same<X, double>::value ? 1 : 3;
  auto t0 = std::chrono::steady_clock::now();
  BasisData& b = *op.basis;
  uint64_t const D = b.D;
  uint32_t const nev = o.nev;
  cudaStream_t stream = op.cuda_stream;
  double const tol = o.tol > 0 ? o.tol : 1e-8;
  uint64_t const max_iter = o.max_iter ? o.max_iter : 100000;
  // Stream form when it fits.
  auto ts = std::chrono::steady_clock::now();
  int const form = o.form == SED_FORM_AUTO ? op.form : (int)o.form;
  if (form != SED_FORM_ON_THE_FLY) {
    int st = operator_record_stream(op, stream);
    if (st && form == SED_FORM_STREAM) return st;
  }
  int const saved_form = op.form;
  op.form = form;
  struct FormGuard {
    OperatorData& o;
    int f;
    ~FormGuard() { o.form = f; }
  } form_guard{op, saved_form};
  double const setup = std::chrono::duration<double>(std::chrono::steady_clock::now() - ts).count();
  bool const reorth = nev > 1;
  uint32_t const m = auto_basis(D, sizeof(X), nev, o.max_basis);
  uint32_t const check = m < 64 ? 1u : 4u;
  Solver<X> S(op, dtype, stream);
  if (int st = S.init(m, check, reorth)) return st;
  // Start vector.
  if (o.start == SED_START_GIVEN && o.start_vectors) {
    size_t const es = sizeof(X);
    SED_TRY_CUDA(cudaMemcpyAsync(S.V(), o.start_vectors, D * es, cudaMemcpyDefault, stream));
  } else {
    { k_random<X><<<S.vblocks, kBlock, 0, stream>>>(S.V(), D, o.seed); note_launches(1); }
    SED_TRY_CUDA(cudaGetLastError());
  }
  if (int st = S.normalise_vec(S.V(), nullptr)) return st;
  if (int st = S.capture()) return st;
  uint64_t steps = 0, matvecs = 0, restarts = 0;
  std::vector<double> E(nev, 0.0), R(nev, 1e300);
  bool converged = false;
  Tridiagonal T(nev);
  while (!converged) {
    if (int st = S.cycle.start(stream, 0)) return st;
    if (int st = S.prescale()) return st;  // the start's and the residual matvecs used the workspace
    uint64_t const before = steps;
    if (int st = S.cycle.run(stream, T, 0.5 * tol, max_iter - std::min(steps, max_iter), [&](uint32_t taken) {
          if (o.progress) o.progress(o.progress_user, before + taken, T.theta.data(), T.est.data(), nev);
        }))
      return st;
    uint32_t const stop = S.cycle.stop;
    if (stop == kRunning) break;  // out of steps
    steps += S.cycle.steps;
    matvecs += S.cycle.steps;
    uint32_t const n = T.size();
    // Ritz vectors and their true residuals.
    bool all_ok = true;
    for (uint32_t j = 0; j < nev; ++j) {
      SED_TRY_CUDA(cudaMemcpyAsync(S.ws.s.ptr, T.vector(j).data(), n * 8, cudaMemcpyHostToDevice, stream));
      { k_ritz<X, X><<<S.vblocks, kBlock, 0, stream>>>(S.V(), D, D, S.ws.s.template as<double>(), n,
                                                     S.ws.ritz.template as<X>()); note_launches(1); }
      SED_TRY_CUDA(cudaGetLastError());
      if (int st = S.normalise_vec(S.ws.ritz.template as<X>(), nullptr)) return st;
      double e = 0.0, r = 0.0;
      if (int st = S.residual(S.ws.ritz.template as<X>(), &e, &r)) return st;
      ++matvecs;
      E[j] = e;
      R[j] = r;
      if (!(r <= tol)) all_ok = false;
      if (evecs)
        if (int st = S.store(S.ws.ritz.template as<X>(), out_dtype, static_cast<char*>(evecs) +
                             (size_t)j * ldv * elem_bytes(out_dtype))) return st;
    }
    if (all_ok || stop == kBreakdown || steps >= max_iter) {
      converged = all_ok || stop == kBreakdown;
      break;
    }
    // Restart from the (sum of the) Ritz vectors.
    ++restarts;
    if (nev == 1) {
      SED_TRY_CUDA(cudaMemcpyAsync(S.V(), S.ws.ritz.ptr, D * sizeof(X), cudaMemcpyDeviceToDevice, stream));
    } else {
      std::vector<double> all(n, 0.0);  // sum of all nev Ritz directions
      for (uint32_t j = 0; j < nev; ++j)
        for (uint32_t i = 0; i < n; ++i) all[i] += T.vector(j)[i];
      SED_TRY_CUDA(cudaMemcpyAsync(S.ws.s.ptr, all.data(), n * 8, cudaMemcpyHostToDevice, stream));
      { k_ritz<X, X><<<S.vblocks, kBlock, 0, stream>>>(S.V(), D, D, S.ws.s.template as<double>(), n,
                                                     S.ws.ritz.template as<X>()); note_launches(1); }
      SED_TRY_CUDA(cudaMemcpyAsync(S.V(), S.ws.ritz.ptr, D * sizeof(X), cudaMemcpyDeviceToDevice, stream));
    }
    if (int st = S.normalise_vec(S.V(), nullptr)) return st;
  }
  SED_TRY_CUDA(cudaStreamSynchronize(stream));
  for (uint32_t j = 0; j < nev; ++j) {
    if (evals) evals[j] = E[j];
    if (rnorms) rnorms[j] = R[j];
  }
  double const total = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  if (info) {
    info->iterations = steps;
    info->matvecs = matvecs;
    info->restarts = restarts;
    info->fp32_iterations = 0;
    info->seconds_total = total;
    info->seconds_setup = setup;
    info->seconds_solve = total - setup;
  }
  if (logging_enabled())
    log_line("sed_eigh: E0 = %.15g, residual %.3e, %llu steps, %llu restarts, %.3f s", E[0], R[0],
             (unsigned long long)steps, (unsigned long long)restarts, total);
  if (!converged) return fail(LS_NOT_CONVERGED, "residual " + std::to_string(R[0]) + " above tolerance after " +
                                                   std::to_string(steps) + " steps");
  return LS_SUCCESS;
}

// Mixed precision: FP64 anchor psi, FP32 Krylov cycles (see the file head).
int solve_mixed(OperatorData& op, int out_dtype, sed_eigh_options const& o, double* evals, void* evecs,
                uint64_t ldv, double* rnorms, sed_eigh_info* info) {
  auto t0 = std::chrono::steady_clock::now();
  uint64_t const D = op.basis->D;
  cudaStream_t stream = op.cuda_stream;
  double const tol = o.tol > 0 ? o.tol : 1e-8;
  uint64_t const max_iter = o.max_iter ? o.max_iter : 100000;
  auto ts = std::chrono::steady_clock::now();
  if (int st = operator_record_stream(op, stream)) return st;
  if (int st = operator_prepare_fp32(op, stream)) return st;
  double const setup = std::chrono::duration<double>(std::chrono::steady_clock::now() - ts).count();
  int const saved_form = op.form;
  op.form = SED_FORM_STREAM;
  struct FormGuard {
    OperatorData& o;
    int f;
    ~FormGuard() { o.form = f; }
  } form_guard{op, saved_form};
  uint32_t const m = std::max<uint32_t>(3, auto_basis(D, 4, 1, o.max_basis ? o.max_basis : 300));
  uint32_t const check = m < 64 ? 1u : 4u;
  unsigned const vb = grid_size(D, op.basis->device, 8);
  DeviceBuffer buf, V;
  DevicePart psi, y, state, sbuf, partial, done_b;
  struct KrylovGuard {
    DeviceBuffer& b;
    cudaStream_t s;
    ~KrylovGuard() {
      cudaStreamSynchronize(s);  // a replay may be in flight on an early exit
      krylov_give(b);
    }
  } krylov_guard{V, stream};
  if (int st = krylov_take((size_t)m * D * 4, V)) return st;
  uint64_t const nb = std::max<uint64_t>((D + kBlock - 1) / kBlock, vb) + 32;
  DeviceParts parts;
  parts.add(psi, D * 8);
  parts.add(y, D * 8);
  parts.add(state, state_bytes(m));
  parts.add(sbuf, (size_t)m * 8);
  parts.add(partial, nb * 16);
  parts.add(done_b, 16);
  if (int st = parts.allocate(buf)) return st;
  SED_TRY_CUDA(cudaMemsetAsync(done_b.ptr, 0, 16, stream));
  Cycle cycle;
  if (int st = cycle.init(state.as<LzHeader>(), m, check)) return st;
  Tridiagonal T(1);
  uint32_t* done = done_b.as<uint32_t>();
  LzHeader* h = cycle.hdr;
  float* Vf = V.as<float>();
  // FP64 start vector
  if (o.start == SED_START_GIVEN && o.start_vectors)
    SED_TRY_CUDA(cudaMemcpyAsync(psi.ptr, o.start_vectors, D * 8, cudaMemcpyDefault, stream));
  else
    { k_random<double><<<vb, kBlock, 0, stream>>>(psi.as<double>(), D, o.seed); note_launches(1); }
  auto sum2 = [&](int mode, double e, double& a, double& b) -> int {
    { k_dots<double><<<vb, kBlock, 0, stream>>>(psi.as<double>(), y.as<double>(), D, e, mode, partial.as<double>()); note_launches(1); }
    std::vector<double> hs(2 * (size_t)vb);
    SED_TRY_CUDA(cudaMemcpyAsync(hs.data(), partial.ptr, hs.size() * 8, cudaMemcpyDeviceToHost, stream));
    SED_TRY_CUDA(cudaStreamSynchronize(stream));
    a = b = 0.0;
    for (unsigned i = 0; i < vb; ++i) {
      a += hs[2 * i];
      b += hs[2 * i + 1];
    }
    return LS_SUCCESS;
  };
  // normalise psi: y <- psi so that mode 0 gives <psi,psi>
  SED_TRY_CUDA(cudaMemcpyAsync(y.ptr, psi.ptr, D * 8, cudaMemcpyDeviceToDevice, stream));
  double nn = 0, dummy = 0;
  if (int st = sum2(0, 0.0, nn, dummy)) return st;
  { k_scale<double><<<vb, kBlock, 0, stream>>>(psi.as<double>(), D, 1.0 / std::sqrt(nn)); note_launches(1); }
  // graph of `check` FP32 steps
  double *alpha = cycle.alpha(), *beta = cycle.beta();
  if (int st = cycle.capture(stream, [&]() -> int {
        Indirect ind;
        ind.k = &h->k;
        ind.stop = &h->stop;
        ind.ld = D;
        ind.partial = partial.as<double>();
        ind.done = done;
        ind.sum = alpha;
        if (int st = apply_with_alpha(ind, D, stream, [&](Indirect i) { return operator_apply_krylov32(op, Vf, i, stream); }))
          return st;
        k_update32<<<vb, kBlock, 0, stream>>>(Vf, D, D, h, alpha, beta, partial.as<double>(), done);
        k_scale_next32<<<vb, kBlock, 0, stream>>>(Vf, D, D, h, beta, done);
        SED_TRY_CUDA(cudaGetLastError());
        return LS_SUCCESS;
      }))
    return st;
  uint64_t steps32 = 0, matvecs = 0, cycles = 0;
  double E = 0.0, R = 1e300;
  bool converged = false;
  while (true) {
    // FP64: theta = <psi, H psi>, r = H psi - theta psi
    if (int st = operator_apply_device(op, 1, 1, psi.ptr, D, y.ptr, D, stream, SED_FORM_STREAM)) return st;
    ++matvecs;
    double pp = 0, py = 0;
    if (int st = sum2(0, 0.0, pp, py)) return st;
    E = py / pp;
    double rr = 0, unused = 0;
    if (int st = sum2(1, E, rr, unused)) return st;
    R = std::sqrt(rr / pp);
    if (o.progress) o.progress(o.progress_user, steps32 + matvecs, &E, &R, 1);
    if (R <= tol) {
      converged = true;
      break;
    }
    if (steps32 >= max_iter || cycles >= 64) break;
    // FP32 cycle from v0 = psi, v1 = r / ||r||
    double const rn = R * std::sqrt(pp);
    { k_start_cycle<<<vb, kBlock, 0, stream>>>(psi.as<double>(), y.as<double>(), D, E, 1.0 / rn, Vf, Vf + D); note_launches(1); }
    double const a0 = E, b0 = rn;
    SED_TRY_CUDA(cudaMemcpyAsync(alpha, &a0, 8, cudaMemcpyHostToDevice, stream));
    SED_TRY_CUDA(cudaMemcpyAsync(beta, &b0, 8, cudaMemcpyHostToDevice, stream));
    if (int st = cycle.start(stream, 1)) return st;
    if (int st = cycle.run(stream, T, std::max(0.5 * tol, 2e-6 * rn), max_iter - std::min<uint64_t>(steps32, max_iter),
                           [](uint32_t) {}))
      return st;
    steps32 += cycle.steps;
    ++cycles;
    if (cycle.stop == kRunning) break;  // out of steps
    uint32_t const n = T.size();
    SED_TRY_CUDA(cudaMemcpyAsync(sbuf.ptr, T.vector(0).data(), n * 8, cudaMemcpyHostToDevice, stream));
    { k_ritz_mixed<<<vb, kBlock, 0, stream>>>(psi.as<double>(), Vf, D, D, sbuf.as<double>(), n, y.as<double>()); note_launches(1); }
    SED_TRY_CUDA(cudaMemcpyAsync(psi.ptr, y.ptr, D * 8, cudaMemcpyDeviceToDevice, stream));
    double pn = 0, d2 = 0;
    if (int st = sum2(0, 0.0, pn, d2)) return st;  // y == psi here
    { k_scale<double><<<vb, kBlock, 0, stream>>>(psi.as<double>(), D, 1.0 / std::sqrt(pn)); note_launches(1); }
  }
  // output
  if (evecs) {
    int const own = 1;
    char* dst = static_cast<char*>(evecs);
    if (out_dtype == own) {
      SED_TRY_CUDA(cudaMemcpyAsync(dst, psi.ptr, D * 8, cudaMemcpyDefault, stream));
    } else {
      DeviceBuffer tmp;
      if (int st = tmp.allocate(D * (size_t)elem_bytes(out_dtype))) return st;
      switch (out_dtype) {
        case 0: { k_convert<double, float><<<vb, kBlock, 0, stream>>>(psi.as<double>(), D, tmp.as<float>()); note_launches(1); } break;
        case 2: { k_convert<double, float2><<<vb, kBlock, 0, stream>>>(psi.as<double>(), D, tmp.as<float2>()); note_launches(1); } break;
        default: { k_convert<double, double2><<<vb, kBlock, 0, stream>>>(psi.as<double>(), D, tmp.as<double2>()); note_launches(1); } break;
      }
      SED_TRY_CUDA(cudaMemcpyAsync(dst, tmp.ptr, D * (size_t)elem_bytes(out_dtype), cudaMemcpyDefault, stream));
    }
  }
  SED_TRY_CUDA(cudaStreamSynchronize(stream));
  if (evals) evals[0] = E;
  if (rnorms) rnorms[0] = R;
  double const total = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  if (info) {
    info->iterations = steps32 + matvecs;
    info->matvecs = steps32 + matvecs;
    info->restarts = cycles;
    info->fp32_iterations = steps32;
    info->seconds_total = total;
    info->seconds_setup = setup;
    info->seconds_solve = total - setup;
  }
  if (logging_enabled())
    log_line("sed_eigh (mixed): E0 = %.15g, residual %.3e, %llu FP32 steps, %llu FP64 matvecs, %llu cycles, %.3f s",
             E, R, (unsigned long long)steps32, (unsigned long long)matvecs, (unsigned long long)cycles, total);
  if (!converged)
    return fail(LS_NOT_CONVERGED, "mixed precision: residual " + std::to_string(R) + " above tolerance");
  return LS_SUCCESS;
}

}  // namespace
}  // namespace sed

using namespace sed;

extern "C" {

void sed_eigh_options_init(sed_eigh_options* o) {
  if (!o) return;
  std::memset(o, 0, sizeof(*o));
  o->struct_size = sizeof(sed_eigh_options);
  o->nev = 1;
  o->tol = 1e-8;
  o->block_size = 1;
  o->precision = SED_PRECISION_FP64;
  o->start = SED_START_RANDOM;
  o->form = SED_FORM_AUTO;
  o->seed = 1234;
}

int sed_eigh(ls_operator const* op, int dtype, sed_eigh_options const* opts, double* eigenvalues,
             void* eigenvectors, uint64_t ldv, double* residuals, sed_eigh_info* info) {
  if (!op) return fail(LS_INVALID_ARGUMENT, "sed_eigh: NULL operator");
  sed_eigh_options o;
  sed_eigh_options_init(&o);
  if (opts) {
    if (opts->struct_size != sizeof(sed_eigh_options))
      return fail(LS_INVALID_ARGUMENT, "sed_eigh: options struct_size mismatch");
    o = *opts;
  }
  if (o.nev == 0 || o.nev > kMaxNev) return fail(LS_INVALID_ARGUMENT, "nev must be in 1..16");
  if (dtype < 0 || dtype > 3) return fail(LS_INVALID_DATATYPE, "dtype must be 0..3");
  OperatorData& d = *op->d;
  std::lock_guard<std::mutex> lock(d.mu);
  if (!d.basis->built) return fail(LS_CACHE_NOT_BUILT, "basis has not been built (call ls_build)");
  if (!d.is_real && dtype < 2) return fail(LS_OPERATOR_IS_COMPLEX, "operator is complex; use dtype 2 or 3");
  uint64_t const D = d.basis->D;
  if (D == 0) return fail(LS_INVALID_ARGUMENT, "sed_eigh: the basis is empty");
  if (o.nev > D) return fail(LS_INVALID_ARGUMENT, "nev exceeds the dimension");
  if (eigenvectors && ldv < D) return fail(LS_INVALID_ARGUMENT, "ldv is smaller than the dimension");
  try {
    ScopedDevice dev(d.basis->device);
    if (int st = operator_ensure_ready(d)) return st;
    if (int st = wait_for_caller({o.start == SED_START_GIVEN ? o.start_vectors : nullptr, eigenvectors})) return st;
    if (int st = fix_wait(d)) return st;  // matvecs still queued on callers' streams share the workspace
    if (dtype >= 2 || !d.is_real) return solve<double2>(d, dtype, o, eigenvalues, eigenvectors, ldv, residuals, info);
    if (o.max_basis > 0 && o.max_basis <= 32 && o.block_size <= 1)
      return solve_thick(d, dtype, o, eigenvalues, eigenvectors, ldv, residuals, info);
    if (o.precision == SED_PRECISION_MIXED && o.nev == 1 && o.form != SED_FORM_ON_THE_FLY)
      return solve_mixed(d, dtype, o, eigenvalues, eigenvectors, ldv, residuals, info);
    return solve<double>(d, dtype, o, eigenvalues, eigenvectors, ldv, residuals, info);
  } catch (std::exception const& e) {
    return fail(LS_SYSTEM_ERROR, e.what());
  }
}

}  // extern "C"
