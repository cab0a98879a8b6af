// batch.cu — many Hamiltonians of uneven size solved in one persistent launch
// (sed_eigh_batched): the lowest nev <= 4 eigenpairs of every operator by
// block Lanczos with block size 4. Krylov blocks are held as double-floats
// (df.cuh), and the products of the block SpMV, the Gram-Schmidt sweeps,
// CholQR2 and the Ritz vectors run in that arithmetic on the FP32 pipe; the
// SpMV's row epilogue, the Rayleigh-Ritz solve, the Ritz vectors kept and their
// true residuals are FP64. Eigenvalues of 84 chains of 12 to 24 sites, four each
// and three seeds, err by 2.9e-15 (rms, relative; at most 1.0e-14) against dense
// or fully reorthogonalised FP64 solves; with FP64 copies of the blocks beside
// the double-floats and the second Gram-Schmidt update in double-float 2.9e-15
// (at most 1.3e-14).
//
// One cooperative kernel runs the whole solve for all problems. Its CTAs are
// split into groups (batch_layout: large problems get several CTAs, small
// ones share one-CTA groups and are solved one after another), and a group
// synchronises through a bounded barrier in global memory. Within a group
// the rows of the problem are split by SELL-32 slices, two runs to a CTA.
//
// Per problem, with Krylov blocks V_j stored row-interleaved ([D][4], so the
// SpMV gathers one 32-byte sector per element for all four columns):
//   V_0 = QR(start block)                                  (CholQR2)
//   W = H V_j ; C_i = V_i^T W, W -= V_i C_i for i <= j      (CGS2, two passes)
//   W = V_{j+1} B_j                                          (CholQR2)
//   T: diagonal blocks A_j = sym(C_j), sub-diagonal blocks B_j
// Every `rr_every` steps of a cycle that may converge, and at the end of each,
// the group's first CTA
// diagonalises T (cyclic Jacobi with parallel round-robin rotations in shared
// memory) and estimates the Ritz residuals ||B_j y_last||; the cycle ends when
// all nev estimates are below tol / 2 or the basis is full. Ritz vectors
// Psi = V Y are then formed, their true residuals ||H psi - theta psi|| are
// computed, and the problem is done when all are below tol; otherwise block
// Lanczos restarts from Psi.
//
// Cross-CTA data (partial sums, T, decisions, the gathered x of the SpMV) is
// read with ld.global.cg so that no stale L1 line is used after a barrier.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <mutex>
#include <numeric>
#include <tuple>
#include <vector>

#include "operator_impl.cuh"
#include "df.cuh"
#include "tc.cuh"

namespace sed {
namespace {

constexpr int kB = 4;               // block size
constexpr int kMaxBlocks = 16;      // stored Krylov blocks per cycle (n <= 64)
constexpr int kMaxN = kB * kMaxBlocks;
constexpr int kPart = 16 * (kMaxBlocks + 1);  // partial sums per CTA and slot
constexpr int kGsStages = 2;                   // shared-memory stages of the Gram-Schmidt row streams
constexpr uint64_t kGsWaitNs = 1000000000ull;  // default bound on a wait for one stage's copies (1 s)
constexpr uint64_t kBarrierNs = 20000000000ull;  // default: 20 s per barrier, far beyond any phase
// Part of a block step that more CTAs do not shorten, in rows of the mean
// work per row (the group layout's model). On 128 J1-J2 chains (N = 16..28)
// the launch takes 720 ms with 900 rows, 708 with 1400, 726 with 2200 and 734
// with 3500.
constexpr double kLayoutFixedRows = 1400.0;
constexpr size_t kStatsOff = 12 * 8;                // per-problem output record: out[12], stats[4], flag[4], prof[8]
constexpr size_t kProfOff = kStatsOff + 32;
constexpr size_t kOutBytes = kProfOff + 64;

struct ChainDesc {
  StreamView S;       // real operator, FP64 stream form
  uint64_t D, n_slices;
  double* V;          // [D][4]: the start block, then the Ritz vectors
  float* Vs;          // (m_blocks + 1) Krylov blocks of D double-float rows (Row4s)
  float* Xs;          // [D] Row4s: the block under Gram-Schmidt, in double-float
  float2* table_s;    // [n_codes]: the matrix-element table split into double-float (k_split_tables)
  double* W;          // [D][4]
  double* part;       // [2][ncta][kPart]
  double* W2;         // [D][4] second scratch block (thick restart)
  double* Tc;         // [kMaxBlocks][kMaxN * 4]: step j's projections C_i = V_i^T H V_j, i <= j
  double* Bblk;       // [kMaxBlocks][16] sub-diagonal blocks (upper triangular)
  double* Y;          // [kMaxN][8] Ritz vectors of T (row q, column i)
  double* out;        // theta[8], residual[4]
  uint32_t* stats;    // block steps, restarts, matvecs, status (0 running, 1 done, 2 not converged, 3 breakdown)
  uint32_t* flag;     // [4]: decision words written by the leader CTA
  uint64_t* prof;     // [8] nanoseconds per phase on the leader CTA: spmv, cgs2, qr, rayleigh-ritz, ritz+restart, residual
  uint32_t m_blocks;
  uint32_t nev;
  uint32_t packed;    // stream entries hold col | code << col_bits
  uint64_t seed;
};

struct GroupDesc {
  uint32_t cta0, ncta, first, count;  // CTAs [cta0, cta0 + ncta); chains order[first .. first + count)
  uint32_t* bar;                      // [2]: arrivals, generation
};

struct BatchArgs {
  ChainDesc const* chains;
  GroupDesc const* groups;
  uint32_t const* cta_group;
  uint32_t const* order;
  double tol;
  uint32_t max_steps;     // block steps per problem in total
  uint32_t rr_every;
  int* error;
  uint64_t wait_ns;        // bound on every barrier wait
  uint64_t copy_wait_ns;   // bound on every wait for a row-stream stage's copies
  uint32_t stage_bytes;    // dynamic shared memory for the row streams' stages
  uint32_t extra_arrivals; // arrivals a barrier waits for beyond its CTAs (0; see sed_debug_barrier_extra_arrivals)
};

// One row of a [D][4] block (32 bytes, one sector).
struct alignas(32) Row4 {
  double x, y, z, w;
};
__device__ __forceinline__ Row4 mk4(double a, double b, double c, double d) { return Row4{a, b, c, d}; }

__device__ __forceinline__ double ldcg(double const* p) { return __ldcg(p); }
__device__ __forceinline__ uint32_t ldcg(uint32_t const* p) { return __ldcg(p); }
__device__ __forceinline__ Row4 ldcg4(double const* p) {
  double2 const a = __ldcg(reinterpret_cast<double2 const*>(p));
  double2 const b = __ldcg(reinterpret_cast<double2 const*>(p) + 1);
  return mk4(a.x, a.y, b.x, b.y);
}

// Rows of split blocks for the double-float Gram-Schmidt products (df.cuh).
struct alignas(32) Row4s {
  float4 h, l;  // a [D][4] row: hi parts, then lo parts
};

__device__ __forceinline__ Row4s split_row(Row4 const& r) {
  Row4s o;
  df_split(r.x, o.h.x, o.l.x);
  df_split(r.y, o.h.y, o.l.y);
  df_split(r.z, o.h.z, o.l.z);
  df_split(r.w, o.h.w, o.l.w);
  return o;
}

// Bounded barrier of the `n` CTAs of a group; false if it timed out (then
// *error = 2) or another CTA has already reported an error, which ends the
// wait early. Every thread of the CTA must call it.
__device__ bool group_barrier(uint32_t* bar, uint32_t n, BatchArgs const& a) {
  __shared__ int ok_s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    uint32_t const need = n + a.extra_arrivals;
    if (need > 1) {
      volatile uint32_t* gen = bar + 1;
      uint32_t const g = *gen;
      __threadfence();
      if (atomicAdd(bar, 1u) == need - 1) {
        atomicExch(bar, 0u);
        __threadfence();
        atomicAdd(bar + 1, 1u);
      } else {
        uint64_t const t0 = tc::global_ns();
        while (*gen == g) {
          if (*(volatile int*)a.error) {
            ok = 0;
            break;
          }
          if (tc::global_ns() - t0 > a.wait_ns) {
            ok = 0;
            atomicExch(a.error, 2);
            break;
          }
          __nanosleep(64);
        }
      }
      __threadfence();
    }
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

// Sums K per-thread values over the CTA; thread k < K of the CTA gets total k
// in out[k] (shared). red: [warps][K] shared scratch.
template <int K>
__device__ __forceinline__ void cta_sum(double (&v)[K], double* red, double* out) {
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double x = v[k];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp * K + k] = x;
  }
  __syncthreads();
  if ((int)threadIdx.x < K) {
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += red[w * K + threadIdx.x];
    out[threadIdx.x] = s;
  }
  __syncthreads();
}

struct Ctx {
  ChainDesc const& c;
  uint32_t rank, ncta;
  uint32_t* bar;
  BatchArgs const* args;
  // Own slices and rows: two runs, [sa, sa + ns0) and [sb, ..), the rank-th of
  // 2 ncta equal pieces and the rank-th from the end. Rows lengthen from the
  // first representative to the last (22-site J1-J2 chain on 11 CTAs: 19.5
  // elements a row in the first eleventh, 29.6 in the last), so that one run
  // per CTA left the SpMV of the last CTA 16 % above the mean; two runs are even
  // in rows and in elements.
  uint32_t ns, ns0, n, n0;  // own slices and rows, of these in the first run
  uint64_t sa, sb, ra, rb;
  __device__ __forceinline__ uint64_t slice(uint32_t l) const { return l < ns0 ? sa + l : sb + (l - ns0); }
  __device__ __forceinline__ uint64_t row(uint32_t l) const { return l < n0 ? ra + l : rb + (l - n0); }
  uint32_t slot;        // partial-sum double buffer
  double* red;          // shared [warps][16]
  double* tmp;          // shared [kPart]
  double* dyn;          // the dynamic shared area (row-stream stages outside the Jacobi solve)
  uint64_t* gs_bar;     // shared [kGsStages] mbarriers of the row streams
  uint32_t* gs_phase;   // parity bit per mbarrier (same value in every thread)
};

// Publishes this CTA's K partial sums (in shared `local`), waits for the group
// and leaves the group totals in shared `total` (same order on every CTA).
__device__ bool group_sum(Ctx& x, double const* local, int K, double* total) {
  double* mine = x.c.part + ((size_t)x.slot * x.ncta + x.rank) * kPart;
  for (int k = threadIdx.x; k < K; k += blockDim.x) mine[k] = local[k];
  __threadfence();
  if (!group_barrier(x.bar, x.ncta, *x.args)) return false;
  double const* all = x.c.part + (size_t)x.slot * x.ncta * kPart;
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    double s = 0.0;
    for (uint32_t r = 0; r < x.ncta; ++r) s += ldcg(all + (size_t)r * kPart + k);
    total[k] = s;
  }
  x.slot ^= 1u;
  __syncthreads();
  return true;
}

// Cholesky of the 4x4 Gram matrix G (row-major) -> upper R with G = R^T R.
// Returns false on a pivot below eps * trace (rank deficiency).
__device__ bool chol4(double const* G, double* R) {
  double const tr = G[0] + G[5] + G[10] + G[15];
  for (int i = 0; i < 16; ++i) R[i] = 0.0;
  for (int j = 0; j < 4; ++j) {
    double d = G[j * 4 + j];
    for (int k = 0; k < j; ++k) d -= R[k * 4 + j] * R[k * 4 + j];
    if (!(d > 1e-24 * tr) || !(tr > 0.0)) return false;
    double const rjj = sqrt(d);
    R[j * 4 + j] = rjj;
    for (int i = j + 1; i < 4; ++i) {
      double s = G[j * 4 + i];
      for (int k = 0; k < j; ++k) s -= R[k * 4 + j] * R[k * 4 + i];
      R[j * 4 + i] = s / rjj;
    }
  }
  return true;
}

// In place X <- X R^{-1} on own rows (X = [D][4]); y R = x by forward
// substitution, dividing by the diagonal through its reciprocals (four FP64
// divisions per CTA instead of four per row: a division is a long sequence
// on GB300's narrow FP64 pipe).
__device__ void apply_rinv(Ctx& x, double* X, double const* R) {
  double const inv[4] = {1.0 / R[0], 1.0 / R[5], 1.0 / R[10], 1.0 / R[15]};
  for (uint32_t l = threadIdx.x; l < x.n; l += blockDim.x) {
    uint64_t const r = x.row(l);
    Row4 const v = *reinterpret_cast<Row4 const*>(X + r * 4);
    double const a[4] = {v.x, v.y, v.z, v.w};
    double y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      double s = a[j];
#pragma unroll
      for (int k = 0; k < j; ++k) s -= y[k] * R[k * 4 + j];
      y[j] = s * inv[j];
    }
    *reinterpret_cast<Row4*>(X + r * 4) = mk4(y[0], y[1], y[2], y[3]);
  }
}

// CholQR2 of the block X in place; Rtot (shared, 16) = R2 R1. false on
// breakdown or barrier failure (ok distinguishes them).
__device__ bool block_qr(Ctx& x, double* X, double* Rtot, bool& ok) {
  __shared__ double G[16], R[16], P[16];
  ok = true;
  for (int pass = 0; pass < 2; ++pass) {
    double g[10] = {};
    for (uint32_t l = threadIdx.x; l < x.n; l += blockDim.x) {
      uint64_t const r = x.row(l);
      Row4 const v = *reinterpret_cast<Row4 const*>(X + r * 4);
      double const a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = i; j < 4; ++j) {
          int const q = i * 4 - i * (i - 1) / 2 + (j - i);  // packed upper triangle
          g[q] = fma(a[i], a[j], g[q]);
        }
    }
    cta_sum<10>(g, x.red, x.tmp);
    if (!group_sum(x, x.tmp, 10, x.tmp + 16)) {
      ok = false;
      return false;
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < 4; ++i)
        for (int j = i; j < 4; ++j) {
          int const q = i * 4 - i * (i - 1) / 2 + (j - i);
          G[i * 4 + j] = G[j * 4 + i] = x.tmp[16 + q];
        }
    }
    __syncthreads();
    __shared__ int good;
    if (threadIdx.x == 0) good = chol4(G, R) ? 1 : 0;
    __syncthreads();
    if (!good) return false;
    apply_rinv(x, X, R);
    if (threadIdx.x == 0) {
      if (pass == 0) {
        for (int i = 0; i < 16; ++i) Rtot[i] = R[i];
      } else {  // Rtot = R2 * R1
        for (int i = 0; i < 4; ++i)
          for (int j = 0; j < 4; ++j) {
            double s = 0.0;
            for (int k = 0; k < 4; ++k) s += R[i * 4 + k] * Rtot[k * 4 + j];
            P[i * 4 + j] = s;
          }
        for (int i = 0; i < 16; ++i) Rtot[i] = P[i];
      }
    }
    __syncthreads();
  }
  return true;
}

// y R = v for one split row and R with its diagonal inverted, split (Rh, Rl):
// y_j = (v_j - sum_{k<j} y_k R_kj) / R_jj.
__device__ __forceinline__ Row4s df_rinv(Row4s const& v, float const* Rh, float const* Rl) {
  float yh[4] = {v.h.x, v.h.y, v.h.z, v.h.w}, yl[4] = {v.l.x, v.l.y, v.l.z, v.l.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
#pragma unroll
    for (int k = 0; k < j; ++k) {
      float ph, pl;
      df_mul(yh[k], yl[k], Rh[k * 4 + j], Rl[k * 4 + j], ph, pl);
      df_sub(yh[j], yl[j], ph, pl);
    }
    df_mul(yh[j], yl[j], Rh[j * 5], Rl[j * 5], yh[j], yl[j]);
  }
  Row4s o;
  o.h = make_float4(yh[0], yh[1], yh[2], yh[3]);
  o.l = make_float4(yl[0], yl[1], yl[2], yl[3]);
  return o;
}

// CholQR2 in double-float of the block in Xs (split), whose Gram matrix G
// (shared, 16, full) the last Gram-Schmidt sweep has left: one pass divides
// by the first factor and sums the second Gram matrix, one divides by the
// second and writes the split factor Vs_out. Rtot (shared, 16) = R2 R1; false
// on breakdown or barrier failure (ok distinguishes them).
__device__ bool block_qr_df(Ctx& x, double* G, Row4s* Vs_out, double* Rtot, bool& ok) {
  __shared__ double R[16], P[16];
  __shared__ float Rh[16], Rl[16];
  __shared__ int good;
  Row4s* Xs = reinterpret_cast<Row4s*>(x.c.Xs);
  ok = true;
  for (int pass = 0; pass < 2; ++pass) {
    if (threadIdx.x == 0) {
      good = chol4(G, R) ? 1 : 0;
      if (good) {
        // R's off-diagonal entries and the reciprocals of its diagonal, split
        for (int i = 0; i < 16; ++i) {
          double const v = (i % 5 == 0) ? 1.0 / R[i] : R[i];
          df_split(v, Rh[i], Rl[i]);
        }
        if (pass == 0) {
          for (int i = 0; i < 16; ++i) Rtot[i] = R[i];
        } else {  // Rtot = R2 * R1
          for (int i = 0; i < 4; ++i)
            for (int j = 0; j < 4; ++j) {
              double s = 0.0;
              for (int k = 0; k < 4; ++k) s += R[i * 4 + k] * Rtot[k * 4 + j];
              P[i * 4 + j] = s;
            }
          for (int i = 0; i < 16; ++i) Rtot[i] = P[i];
        }
      }
    }
    __syncthreads();
    if (!good) return false;
    if (pass == 1) break;
    float S[10] = {}, E[10] = {};
    for (uint32_t l = threadIdx.x; l < x.n; l += blockDim.x) {
      uint64_t const r = x.row(l);
      Row4s const v = df_rinv(Xs[r], Rh, Rl);
      Xs[r] = v;
      float const ah[4] = {v.h.x, v.h.y, v.h.z, v.h.w}, al[4] = {v.l.x, v.l.y, v.l.z, v.l.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = i; j < 4; ++j) {
          int const q = i * 4 - i * (i - 1) / 2 + (j - i);  // packed upper triangle
          df_mac(ah[i], al[i], ah[j], al[j], S[q], E[q]);
        }
    }
    double g[10];
#pragma unroll
    for (int q = 0; q < 10; ++q) g[q] = (double)S[q] + (double)E[q];
    cta_sum<10>(g, x.red, x.tmp);
    if (!group_sum(x, x.tmp, 10, x.tmp + 16)) {
      ok = false;
      return false;
    }
    if (threadIdx.x < 16) {
      int const i = min(threadIdx.x >> 2, threadIdx.x & 3), j = max(threadIdx.x >> 2, threadIdx.x & 3);
      G[threadIdx.x] = x.tmp[16 + i * 4 - i * (i - 1) / 2 + (j - i)];
    }
    __syncthreads();
  }
  for (uint32_t l = threadIdx.x; l < x.n; l += blockDim.x) {
    uint64_t const r = x.row(l);
    Vs_out[r] = df_rinv(Xs[r], Rh, Rl);
  }
  tc::fence_proxy_async_global();  // Vs_out is read by the row streams
  __syncthreads();
  return true;
}

constexpr int kBlockSpmvU = 4;  // slots whose gathers a lane issues together

// W = H X on own rows (X, W: [D][4]); gathers of X go through L2.
__device__ void block_spmv(Ctx& x, double const* X, double* W) {
  StreamView const& S = x.c.S;
  uint32_t const lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t const col_mask = S.col_bits < 32 ? ((1u << S.col_bits) - 1u) : 0xFFFFFFFFu;
  bool const packed = x.c.packed != 0;
  double const* table = static_cast<double const*>(S.table);
  for (uint32_t l = warp; l < x.ns; l += nw) {
    uint64_t const s = x.slice(l);
    uint64_t const base = S.slice_ptr[s];
    uint32_t const width = (uint32_t)((S.slice_ptr[s + 1] - base) >> 5);
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    uint32_t const* ent = S.entries + base + lane;
    // kBlockSpmvU slots per step: their entry loads (issued one step ahead),
    // then their gathers, then the FMAs in slot order (the same order as one
    // slot at a time), so several gathers are in flight per lane
    uint32_t v[kBlockSpmvU];
#pragma unroll
    for (int u = 0; u < kBlockSpmvU; ++u) v[u] = (uint32_t)u < width ? __ldcs(ent + (uint64_t)u * 32) : kNull;
    for (uint32_t e0 = 0; e0 < width; e0 += kBlockSpmvU) {
      uint32_t vn[kBlockSpmvU];
#pragma unroll
      for (int u = 0; u < kBlockSpmvU; ++u)
        vn[u] = e0 + kBlockSpmvU + u < width ? __ldcs(ent + (uint64_t)(e0 + kBlockSpmvU + u) * 32) : kNull;
      double t[kBlockSpmvU];
      Row4 xv[kBlockSpmvU];
#pragma unroll
      for (int u = 0; u < kBlockSpmvU; ++u) {
        if (v[u] != kNull) {
          uint32_t const col = v[u] & col_mask;
          uint32_t const code =
              packed ? (v[u] >> S.col_bits) : (uint32_t)__ldcs(S.codes + base + lane + (uint64_t)(e0 + u) * 32);
          t[u] = __ldg(table + code);
          xv[u] = ldcg4(X + (uint64_t)col * 4);
        } else {
          t[u] = 0.0;
          xv[u] = mk4(0.0, 0.0, 0.0, 0.0);
        }
      }
#pragma unroll
      for (int u = 0; u < kBlockSpmvU; ++u) {
        if (v[u] == kNull) continue;
        a0 = fma(t[u], xv[u].x, a0);
        a1 = fma(t[u], xv[u].y, a1);
        a2 = fma(t[u], xv[u].z, a2);
        a3 = fma(t[u], xv[u].w, a3);
      }
#pragma unroll
      for (int u = 0; u < kBlockSpmvU; ++u) v[u] = vn[u];
    }
    uint64_t const i = s * 32 + lane;
    if (i < x.c.D) {
      double const f = S.inv_sqrt_s[S.row_class[i]];
      double const dg = static_cast<double const*>(S.diag)[i];
      Row4 const xi = ldcg4(X + i * 4);
      *reinterpret_cast<Row4*>(W + i * 4) =
          mk4(fma(f, a0, dg * xi.x), fma(f, a1, dg * xi.y), fma(f, a2, dg * xi.z), fma(f, a3, dg * xi.w));
    }
  }
}

// ------------------------------------------- Gram-Schmidt row streams ---
// A sweep over the CTA's own rows reads a tile of rows of X and of the blocks
// concerned (split: Xs, Vs) into the dynamic shared area by bulk asynchronous
// copies (one thread issues them; an mbarrier per stage counts their bytes),
// the next tile's while this one is worked on. Waits are bounded
// (copy_wait_ns): a copy that does not arrive sets the launch's error flag;
// thread 0 then waits (bounded) for the CTA's copies still in flight and the
// solve returns.

// Waits for stage barrier q (every thread) and flips its parity. A warp's lanes
// give up together: the sweeps exchange values between them.
__device__ bool gs_wait(Ctx& x, uint32_t q) {
  bool const ok = tc::mbar_wait(&x.gs_bar[q], (*x.gs_phase >> q) & 1u, x.args->copy_wait_ns);
  *x.gs_phase ^= 1u << q;
  return __all_sync(0xffffffffu, ok);
}

// After a failed wait on barrier `failed` (its parity already flipped):
// records the error; thread 0 waits (bounded) for the copies still in
// flight on it and on the barriers in `pending` (bit mask, not yet waited).
__device__ bool gs_abort(Ctx& x, uint32_t failed, uint32_t pending) {
  if (threadIdx.x == 0) {
    atomicExch(x.args->error, 3);
    tc::mbar_wait(&x.gs_bar[failed], ((*x.gs_phase >> failed) & 1u) ^ 1u, x.args->copy_wait_ns);
    for (uint32_t q = 0; q < (uint32_t)kGsStages; ++q)
      if (pending & (1u << q)) tc::mbar_wait(&x.gs_bar[q], (*x.gs_phase >> q) & 1u, x.args->copy_wait_ns);
  }
  for (uint32_t q = 0; q < (uint32_t)kGsStages; ++q)
    if (pending & (1u << q)) *x.gs_phase ^= 1u << q;
  return false;
}

// (S, E) with E folded into S again: |E| <= ulp(S) / 2.
__device__ __forceinline__ void df_fold(float& S, float& E) {
  float const s = __fadd_rn(S, E);
  float const bb = __fsub_rn(s, S);
  E = __fadd_rn(__fsub_rn(S, __fsub_rn(s, bb)), __fsub_rn(E, bb));
  S = s;
}

// One sweep: X -= sum_{u0 <= i < nb} V_i C_i (u0 = nb: none), then with the
// new X the products V_i^T X for d0 <= i < nb (d0 = nb: none) into
// tmp[16 i ..] and, if `self`, X^T X into tmp[16 nb ..] (row-major 4 x 4, this
// CTA's rows). C in double-float in shared memory (ch, cl) by quarters of 2 x 2
// (coef_at).
//
// Update and products of a row tile share the tile, so that V is read once for
// both and X goes over memory once per sweep. One stream per block and product,
// which read X again for each, moved some 1340 bytes per row and step at nine
// blocks and another 390 in the QR; this moves 800 and 160. The sweeps are
// bound by issue: two CTAs of eight warps keep the FP32 pipe 60 % busy, waits
// for copies are 2 % of their time.
// `small`: the coefficients are below 2^-26 of X (cgs2), so that their products'
// high parts suffice and the update is 16 FMAs per row and block instead of 192
// operations.
// In the update four lanes share a row, a 2 x 2 quarter of C each; in the
// products sixteen lanes share one, a lane keeping one sum per block in
// registers over all tiles: no tile-by-tile reductions, and every thread has
// the same work whatever nb is. The error sums are folded every 7 rows, which
// keeps their rounding below that of the shorter per-thread sums they replace.
__device__ __forceinline__ uint32_t coef_at(uint32_t k) {  // entry k = 16 i + 4 s + t
  uint32_t const s = (k >> 2) & 3u, t = k & 3u;
  return (k & ~15u) | (s >> 1) << 3 | (t >> 1) << 2 | (s & 1u) << 1 | (t & 1u);
}

__device__ __forceinline__ bool gs_sweep(Ctx& x, uint32_t nb, uint32_t u0, uint32_t d0, bool self, bool small,
                                         float const* ch, float const* cl) {
  Row4s const* Vs = reinterpret_cast<Row4s const*>(x.c.Vs);
  Row4s* Xs = reinterpret_cast<Row4s*>(x.c.Xs);
  uint32_t const th = blockDim.x, b0 = min(u0, d0), nset = nb - b0 + 1, nd = nb - d0;
  // rows of a tile: two tiles of nset arrays fit, whole rounds of the update's lanes
  uint32_t const T = min(x.args->stage_bytes / (2 * nset * (uint32_t)sizeof(Row4s)), 512u) & ~3u;
  uint64_t const D = x.c.D;
  uint32_t const nt0 = (x.n0 + T - 1) / T, ntiles = nt0 + (x.n - x.n0 + T - 1) / T;
  Row4s* st = reinterpret_cast<Row4s*>(x.dyn);
  auto rows_of = [&](uint32_t k) { return k < nt0 ? min(T, x.n0 - k * T) : min(T, x.n - x.n0 - (k - nt0) * T); };
  auto first_of = [&](uint32_t k) { return k < nt0 ? x.ra + (uint64_t)k * T : x.rb + (uint64_t)(k - nt0) * T; };
  auto issue = [&](uint32_t k) {
    uint32_t const q = k & 1u, bytes = rows_of(k) * (uint32_t)sizeof(Row4s);
    uint64_t const row = first_of(k);
    Row4s* dst = st + (size_t)q * nset * T;
    if (threadIdx.x == 0) tc::mbar_expect_tx(&x.gs_bar[q], nset * bytes);
    for (uint32_t i = threadIdx.x >> 5; i < nset; i += th >> 5)
      tc::bulk_g2s(dst + i * T, i ? Vs + (uint64_t)(b0 + i - 1) * D + row : Xs + row, bytes, &x.gs_bar[q]);
  };
  float S[kMaxBlocks] = {}, E[kMaxBlocks] = {}, S2 = 0.0f, E2 = 0.0f;
  uint32_t const ut = threadIdx.x & 3u, us = ut >> 1, uu = ut & 1u;                // update: rows s, columns t of C
  uint32_t const pt = threadIdx.x & 3u, ps = (threadIdx.x >> 2) & 3u;              // products: columns of X and of V
  uint32_t unfolded = 0;
  tc::fence_proxy_async_smem();  // this thread's shared-memory accesses before the copies' writes
  __syncthreads();               // the stages' previous readers are done
  bool const issuer = (threadIdx.x & 31u) == 0;
  if (issuer)
    for (uint32_t k = 0; k < 2 && k < ntiles; ++k) issue(k);
  for (uint32_t k = 0; k < ntiles; ++k) {
    uint32_t const q = k & 1u, n = rows_of(k);
    bool const ok = gs_wait(x, q);
    Row4s* sx = st + (size_t)q * nset * T;
    uint64_t const row0 = first_of(k);
    if (u0 < nb) {
      if (ok) {
        float4 const* c4h = reinterpret_cast<float4 const*>(ch) + us * 2 + uu;
        float4 const* c4l = reinterpret_cast<float4 const*>(cl) + us * 2 + uu;
        uint32_t const mask = 0xFu << (threadIdx.x & 28u);
        uint32_t const col = 2 * uu + us;  // of the two columns, the one this lane finishes
        auto update = [&](uint32_t r, auto rows) {
          constexpr int R = decltype(rows)::value;  // rows r, r + th / 4
          float Su[R][2] = {}, Eu[R][2] = {};
          if (small) {
#pragma unroll 4
            for (uint32_t i = u0; i < nb; ++i) {
              float4 const h = c4h[4 * i];
              Row4s const* sv = sx + (i - b0 + 1) * T;
#pragma unroll
              for (int m = 0; m < R; ++m) {
                float2 const a = *reinterpret_cast<float2 const*>(reinterpret_cast<float const*>(sv + r + m * (th / 4)) + 2 * us);
                Su[m][0] = fmaf(a.x, h.x, fmaf(a.y, h.z, Su[m][0]));
                Su[m][1] = fmaf(a.x, h.y, fmaf(a.y, h.w, Su[m][1]));
              }
            }
          } else {
#pragma unroll 1
            for (uint32_t i = u0; i < nb; ++i) {
              float4 const h = c4h[4 * i], l = c4l[4 * i];
              Row4s const* sv = sx + (i - b0 + 1) * T;
#pragma unroll
              for (int m = 0; m < R; ++m) {
                float const* row = reinterpret_cast<float const*>(sv + r + m * (th / 4)) + 2 * us;
                float2 const ah = *reinterpret_cast<float2 const*>(row), al = *reinterpret_cast<float2 const*>(row + 4);
                df_mac(ah.x, al.x, h.x, l.x, Su[m][0], Eu[m][0]);
                df_mac(ah.x, al.x, h.y, l.y, Su[m][1], Eu[m][1]);
                df_mac(ah.y, al.y, h.z, l.z, Su[m][0], Eu[m][0]);
                df_mac(ah.y, al.y, h.w, l.w, Su[m][1], Eu[m][1]);
              }
            }
          }
#pragma unroll
          for (int m = 0; m < R; ++m) {
            // this lane's column: its own half of the sum over s and the partner's
            float const mine = us ? Su[m][1] : Su[m][0], give = us ? Su[m][0] : Su[m][1];
            float const mine_e = us ? Eu[m][1] : Eu[m][0], give_e = us ? Eu[m][0] : Eu[m][1];
            float const other = __shfl_xor_sync(mask, give, 2), other_e = __shfl_xor_sync(mask, give_e, 2);
            float const sum = __fadd_rn(mine, other);
            float const bb = __fsub_rn(sum, mine);
            float const err = __fadd_rn(__fsub_rn(mine, __fsub_rn(sum, bb)), __fsub_rn(other, bb));
            uint32_t const rr = r + m * (th / 4);
            float* px = reinterpret_cast<float*>(sx + rr) + col;
            float h = px[0], l = px[4];
            df_sub(h, l, sum, __fadd_rn(err, __fadd_rn(mine_e, other_e)));
            px[0] = h;
            px[4] = l;
            float* gx = reinterpret_cast<float*>(Xs + row0 + rr) + col;
            gx[0] = h;
            gx[4] = l;
          }
        };
        uint32_t r = threadIdx.x >> 2;
        for (; r + th / 4 < n; r += th / 2) update(r, std::integral_constant<int, 2>{});
        if (r < n) update(r, std::integral_constant<int, 1>{});
      }
      __syncthreads();
    }
    if (ok && (nd > 0 || self)) {
      auto products = [&](uint32_t r, auto rows) {
        constexpr int R = decltype(rows)::value;  // rows r, r + th / 16, ..
        float wh[R], wl[R];
#pragma unroll
        for (int m = 0; m < R; ++m) {
          float const* xr = reinterpret_cast<float const*>(sx + r + m * (th / 16));
          wh[m] = xr[pt];
          wl[m] = xr[4 + pt];
          if (self) df_mac(xr[ps], xr[4 + ps], wh[m], wl[m], S2, E2);
        }
        float const* vr = reinterpret_cast<float const*>(sx + (d0 - b0 + 1) * T + r) + ps;
#pragma unroll
        for (uint32_t i = 0; i < (uint32_t)kMaxBlocks; ++i) {
          if (i >= nd) break;
#pragma unroll
          for (int m = 0; m < R; ++m) df_mac(vr[m * (th / 2)], vr[m * (th / 2) + 4], wh[m], wl[m], S[i], E[i]);
          vr += T * 8;
        }
        unfolded += R;
        if (unfolded > 7 - R) {
          unfolded = 0;
#pragma unroll
          for (uint32_t i = 0; i < (uint32_t)kMaxBlocks; ++i) {
            if (i >= nd) break;
            df_fold(S[i], E[i]);
          }
          df_fold(S2, E2);
        }
      };
      uint32_t r = threadIdx.x >> 4;
      for (; r + th / 16 < n; r += th / 8) products(r, std::integral_constant<int, 2>{});
      if (r < n) products(r, std::integral_constant<int, 1>{});
    }
    tc::fence_proxy_async_smem();
    if (__syncthreads_or(!ok)) return gs_abort(x, q, (k + 1 < ntiles ? 1u << ((k + 1) & 1u) : 0u));
    if (issuer && k + 2 < ntiles) issue(k + 2);
  }
  // sums over the row groups: lanes 16 apart, then the warps (in the free stages)
  uint32_t const lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = th >> 5, K = 16 * (nd + (self ? 1 : 0));
  double* red = x.dyn;
  auto put = [&](uint32_t i, float Si, float Ei) {
    double v = (double)Si + (double)Ei;
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    if (lane < 16) red[warp * K + 16 * i + ps * 4 + pt] = v;
  };
#pragma unroll
  for (uint32_t i = 0; i < (uint32_t)kMaxBlocks; ++i)
    if (i < nd) put(i, S[i], E[i]);
  if (self) put(nd, S2, E2);
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < K; e += th) {
    double v = 0.0;
    for (uint32_t w = 0; w < nw; ++w) v += red[w * K + e];
    x.tmp[16 * d0 + e] = v;
  }
  tc::fence_proxy_async_global();  // the next sweep's copies read Xs
  __syncthreads();
  return true;
}

// Xs = H V_j (split) on own rows from the split copy of V_j (Vs block j,
// complete on every CTA): each element's product t x_c is formed and summed in
// double-float (df.cuh) with the split table, so the FP64 pipe only runs the
// row epilogue y = d x + a / sqrt(S_i), floats widened on the integer pipe. Same
// gathers (one 32-byte row per element) and slot scheme as block_spmv.
__device__ void block_spmv_df(Ctx& x, uint32_t j) {
  StreamView const& S = x.c.S;
  uint32_t const lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t const col_mask = S.col_bits < 32 ? ((1u << S.col_bits) - 1u) : 0xFFFFFFFFu;
  bool const packed = x.c.packed != 0;
  float2 const* table = x.c.table_s;
  Row4s const* Vj = reinterpret_cast<Row4s const*>(x.c.Vs) + (uint64_t)j * x.c.D;
  Row4s* Xs = reinterpret_cast<Row4s*>(x.c.Xs);
  for (uint32_t l = warp; l < x.ns; l += nw) {
    uint64_t const s = x.slice(l);
    uint64_t const base = S.slice_ptr[s];
    uint32_t const width = (uint32_t)((S.slice_ptr[s + 1] - base) >> 5);
    float Sa[4] = {}, Ea[4] = {};
    uint32_t const* ent = S.entries + base + lane;
    // the next step's entries are loaded while this step's gathers are in
    // flight (with 16 warps per SM, the entry load and the gather would
    // otherwise be two exposed latencies per step; two steps ahead measured
    // the same)
    uint32_t v[kBlockSpmvU];
#pragma unroll
    for (int u = 0; u < kBlockSpmvU; ++u) v[u] = (uint32_t)u < width ? __ldcs(ent + (uint64_t)u * 32) : kNull;
    for (uint32_t e0 = 0; e0 < width; e0 += kBlockSpmvU) {
      uint32_t vn[kBlockSpmvU];
#pragma unroll
      for (int u = 0; u < kBlockSpmvU; ++u)
        vn[u] = e0 + kBlockSpmvU + u < width ? __ldcs(ent + (uint64_t)(e0 + kBlockSpmvU + u) * 32) : kNull;
      float2 t[kBlockSpmvU];
      float4 gh[kBlockSpmvU], gl[kBlockSpmvU];
#pragma unroll
      for (int u = 0; u < kBlockSpmvU; ++u) {
        if (v[u] != kNull) {
          uint32_t const col = v[u] & col_mask;
          uint32_t const code =
              packed ? (v[u] >> S.col_bits) : (uint32_t)__ldcs(S.codes + base + lane + (uint64_t)(e0 + u) * 32);
          t[u] = __ldg(table + code);
          float4 const* row = reinterpret_cast<float4 const*>(Vj + col);
          gh[u] = __ldcg(row);
          gl[u] = __ldcg(row + 1);
        } else {
          t[u] = make_float2(0.0f, 0.0f);
          gh[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          gl[u] = gh[u];
        }
      }
#pragma unroll
      for (int u = 0; u < kBlockSpmvU; ++u) {
        df_mac(t[u].x, t[u].y, gh[u].x, gl[u].x, Sa[0], Ea[0]);
        df_mac(t[u].x, t[u].y, gh[u].y, gl[u].y, Sa[1], Ea[1]);
        df_mac(t[u].x, t[u].y, gh[u].z, gl[u].z, Sa[2], Ea[2]);
        df_mac(t[u].x, t[u].y, gh[u].w, gl[u].w, Sa[3], Ea[3]);
      }
#pragma unroll
      for (int u = 0; u < kBlockSpmvU; ++u) v[u] = vn[u];
    }
    uint64_t const i = s * 32 + lane;
    if (i < x.c.D) {
      double const f = S.inv_sqrt_s[S.row_class[i]];
      double const dg = static_cast<double const*>(S.diag)[i];
      float4 const* own = reinterpret_cast<float4 const*>(Vj + i);
      float4 const vh = __ldcg(own), vl = __ldcg(own + 1);
      auto row = [&](float S, float E, float h, float l) {
        return fma(f, widen(S) + widen(E), dg * (widen(h) + widen(l)));
      };
      auto split = [](double y, float& h, float& l) {
        h = __double2float_rn(y);
        l = __double2float_rn(y - widen(h));
      };
      Row4s o;
      split(row(Sa[0], Ea[0], vh.x, vl.x), o.h.x, o.l.x);
      split(row(Sa[1], Ea[1], vh.y, vl.y), o.h.y, o.l.y);
      split(row(Sa[2], Ea[2], vh.z, vl.z), o.h.z, o.l.z);
      split(row(Sa[3], Ea[3], vh.w, vl.w), o.h.w, o.l.w);
      Xs[i] = o;
    }
  }
  tc::fence_proxy_async_global();  // the row streams read Xs
  __syncthreads();
}

// X -= sum_{i<nb} V_i C_i (two passes of classical Gram-Schmidt) on the split
// rows in Xs, in three sweeps: first products; first update and second
// products; second update and the Gram matrix G (shared, 16) of the result. C
// (shared, nb * 16, row-major a*4+c per block, may be null) receives the summed
// coefficients. The second ones are rounding errors of the first pass, some
// 1e-14 of X; where every column of them is below 2^-26 of the column of X they
// are subtracted in single precision (an error of 2^-50 of X, under the split's
// 2^-48), and the Gram matrix summed beside them stands for the updated X (they
// change it by 2^-52): a sum over the group less; norms2 (shared; if `norms`) the squared column norms of X
// before the projection. The first pass runs against blocks first .. nb-1
// only (first > 0 where X = H V_{nb-1} is, in exact arithmetic, orthogonal
// to the older blocks); the second pass always runs against all nb blocks.
__device__ __forceinline__ bool cgs2(Ctx& x, uint32_t nb, double* C, bool norms, double* norms2, double* G,
                                     uint32_t first) {
  uint32_t const K = nb * 16;
  double* tot = x.tmp + kPart;
  // the coefficients in double-float, over this CTA's partial sums (no longer
  // needed once group_sum has returned)
  float* ch = reinterpret_cast<float*>(x.tmp);
  float* cl = ch + K;
  __shared__ bool small_s;
  bool small = false;
#pragma unroll 1
  for (int sweep = 0; sweep < 3; ++sweep) {
    uint32_t const u0 = sweep == 0 ? nb : sweep == 1 ? first : 0u, d0 = sweep == 0 ? first : sweep == 1 ? 0u : nb;
    bool const self = sweep == 0 ? norms : sweep == 1 || !small;
    if (!gs_sweep(x, nb, u0, d0, self, sweep == 2 && small, ch, cl)) return false;
    if (sweep == 2 && small) return true;
    uint32_t const from = 16 * d0;
    if (!group_sum(x, x.tmp + from, (int)(K - from) + (self ? 16 : 0), tot + from)) return false;
    if (sweep == 0 && norms && threadIdx.x < 4) norms2[threadIdx.x] = tot[K + 5 * threadIdx.x];
    if (sweep < 2) {
      if (C)
        for (uint32_t k = threadIdx.x; k < K; k += blockDim.x)
          C[k] = (sweep ? C[k] : 0.0) + (k >= from ? tot[k] : 0.0);
      for (uint32_t k = from + threadIdx.x; k < K; k += blockDim.x) df_split(tot[k], ch[coef_at(k)], cl[coef_at(k)]);
    }
    if (sweep > 0 && threadIdx.x < 16) G[threadIdx.x] = tot[K + threadIdx.x];
    if (sweep == 1 && threadIdx.x < 32) {
      uint32_t const t = threadIdx.x & 3u;
      double q = 0.0;
      for (uint32_t k = threadIdx.x; k < K; k += 32) q = fma(tot[k], tot[k], q);
      for (int o = 4; o < 32; o <<= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
      bool const all = __all_sync(0xffffffffu, q <= 0x1p-52 * tot[K + 5 * t]);
      if (threadIdx.x == 0) small_s = all;
    }
    __syncthreads();
    if (sweep == 1) small = small_s;
  }
  return true;
}

// dst = src split, own rows of one block.
__device__ void split_block(Ctx& x, Row4s* dst, double const* src) {
  for (uint32_t l = threadIdx.x; l < x.n; l += blockDim.x) {
    uint64_t const r = x.row(l);
    dst[r] = split_row(*reinterpret_cast<Row4 const*>(src + r * 4));
  }
  tc::fence_proxy_async_global();
  __syncthreads();
}

// Orthogonalises the new Krylov block in Xs: Gram-Schmidt against V_0 ..
// V_{nb-1} (C: the coefficients, see cgs2) and QR into Vs block nb, with
// deflation: a column whose norm fell below 1e-10 of its norm before the
// projection, or that is numerically dependent on the others, means the block
// Krylov space lost a direction there (typically a converged Ritz vector of the
// restart block). Such columns are replaced by random vectors, projected
// against the basis, and the block is factored by CholQR2. Rb gets R with the
// replaced columns zeroed (their coupling to H V_j is below the threshold).
// Returns false on barrier failure or if the replacement fails.
template <class Lap>
__device__ __forceinline__ bool lanczos_step(Ctx& x, uint32_t nb, double* C, double* Rb, uint32_t first, uint32_t step,
                                             bool& replaced, Lap&& lap) {
  __shared__ double R[16], G[16], norms2[4];
  Row4s* Xs = reinterpret_cast<Row4s*>(x.c.Xs);
  int total = 0;
#pragma unroll 1
  for (int attempt = 0;; ++attempt) {
    if (!cgs2(x, nb, attempt ? nullptr : C, attempt == 0, norms2, G, attempt ? 0u : first)) return false;
    int m = 0;
    for (int c = 0; c < 4; ++c)
      if (!(G[5 * c] > 1e-20 * norms2[c])) m |= 1 << c;
    total |= m;
    if (m == 0) break;
    if (attempt == 2) return false;
    for (uint32_t l = threadIdx.x; l < x.n; l += blockDim.x) {
      uint64_t const r = x.row(l);
      uint32_t cnt[4] = {(uint32_t)r, (uint32_t)(r >> 32), 0xDEF1u + step, (uint32_t)attempt};
      philox(cnt, (uint32_t)x.c.seed, (uint32_t)(x.c.seed >> 32));
      float* row = reinterpret_cast<float*>(Xs + r);
      for (int c = 0; c < 4; ++c)
        if (m & (1 << c)) df_split(2.0 * ((double)cnt[c] * (1.0 / 4294967296.0)) - 1.0, row[c], row[4 + c]);
    }
    tc::fence_proxy_async_global();
    __syncthreads();
    if (threadIdx.x < 4 && (m & (1 << threadIdx.x))) norms2[threadIdx.x] = (double)x.c.D;
    __syncthreads();
  }
  lap(1);
  bool ok;
  // dependent columns that are not small: a breakdown
  if (!block_qr_df(x, G, reinterpret_cast<Row4s*>(x.c.Vs) + (uint64_t)nb * x.c.D, R, ok)) return false;
  if (threadIdx.x < 16) {
    int const col = threadIdx.x & 3;
    Rb[threadIdx.x] = (total & (1 << col)) ? 0.0 : R[threadIdx.x];
  }
  __syncthreads();
  replaced = total != 0;
  return true;
}

// The Jacobi rotation of rows p and q, as three shears with h = tan(theta / 2)
// and s = sin(theta): (p, q) <- (c p - s q, s p + c q), c = 1 - h s, in three
// FMAs where the product form takes four FP64 instructions.
__device__ __forceinline__ void rotate(double h, double s, double& p, double& q) {
  p = fma(-h, q, p);
  q = fma(s, p, q);
  p = fma(-h, q, p);
}

// h of the rotation that annihilates apq, d = aqq - app: the root of smallest
// magnitude of apq (v^2 - u^2) + d v u = 0 with u = 1 - h^2, v = 2 h. In FP32
// from both numbers scaled by one power of two, then one Newton step in FP64
// (2^-45 of h; what it leaves of apq is below the solver's threshold one
// sweep later, as with a correctly rounded angle). Zero if apq is below 2^-126
// of d.
__device__ __forceinline__ double half_angle(double apq, double d) {
  unsigned const m = (unsigned)(__double_as_longlong(fmax(fabs(apq), fabs(d))) >> 52);
  double const scale = __longlong_as_double((long long)max(1, min(2046, 2046 - (int)m)) << 52);
  apq *= scale;
  d *= scale;
  float const a = (float)apq, e = (float)d;
  float t = 2.0f * fabsf(a) / (fabsf(e) + sqrtf(fmaf(e, e, 4.0f * a * a)));
  if (e != 0.0f && (e < 0.0f) != (a < 0.0f)) t = -t;
  float const h0 = t / (1.0f + sqrtf(fmaf(t, t, 1.0f)));
  double const h = h0, u = fma(-h, h, 1.0), v = h + h;
  double const g = fma(apq, (v - u) * (v + u), d * (v * u));
  float const uf = (float)u, vf = (float)v;
  float const slope = fmaf(a, 2.0f * vf * (2.0f + uf), e * fmaf(-vf, vf, 2.0f * uf));
  return h0 == 0.0f ? 0.0 : h - (double)((float)g / slope);
}

// Cyclic Jacobi on the symmetric n x n matrix A (shared, row-major with rows of
// n + 1, n a multiple of 4) with parallel round-robin rotations and a threshold: a rotation whose
// off-diagonal entry is at most 1e-16 of ||A||_F (invariant under the
// rotations) is skipped, and the sweeps end when one performs none (the
// eigenvalues then carry errors of order 1e-32 ||A||^2 / gap). Q (shared, rows
// of n) receives the eigenvectors as rows. Eigenvalues end on the diagonal of A.
//
// The FP64 pipe bounds it. A round rotates rows and columns in one go, a 2 x 2
// block of A per thread (a row pair and a column pair), blocks above the
// diagonal only and mirrored: half the operations of a pass over all rows and
// one over all columns, and one barrier less. With rows of
// n + 1, and the eigenvectors as rows, lanes fall into different banks. The
// next round's angles (warp 0) and this round's rotation of Q (the other
// warps) go together between two barriers: the angles were a chain of three
// FP64 divisions and square roots on one warp that all others waited for. A
// call with 46 chains of 12 to 20 sites 24.5 -> 17.6 ms, 16 of 18 to 26
// 60.4 -> 51.3, 128 of 16 to 28 681 -> 665. The three-shear rotations also
// round less than the product form did: eigenvalues of 64 x 64 matrices err by
// 2e-15 ||A|| where it was 1.2e-14, after the same number of sweeps.
__device__ void jacobi(double* A, double* Q, int n) {
  __shared__ double cs[2][kMaxN / 2][2];  // h and s, of this round and the next
  __shared__ int pp[2][kMaxN / 2][2];
  __shared__ double wsum[8];
  __shared__ double thr;
  __shared__ int rotated;
  double f = 0.0;
  int const ld = n + 1, half = n / 2;
  for (int k = threadIdx.x; k < n * n; k += blockDim.x) {
    int const r = k / n, c = k % n;
    Q[k] = r == c ? 1.0 : 0.0;
    f = fma(A[r * ld + c], A[r * ld + c], f);
  }
  // this thread's blocks (k1 <= k2) of the half (half + 1) / 2: rows k and
  // half - 1 - k of the triangle side by side, half + 1 blocks
  constexpr int kMine = 5;  // 528 blocks at n = 64 on 128 threads
  int mine[kMine];
#pragma unroll
  for (int m = 0; m < kMine; ++m) {
    int const e = (int)threadIdx.x + m * (int)blockDim.x, row = e / (half + 1), col = e % (half + 1);
    mine[m] = row >= half / 2 ? -1
              : col < half - row ? row << 8 | (row + col)
                                 : (half - 1 - row) << 8 | (half - 1 - row + col - (half - row));
  }
  uint32_t const inv_n = ((1u << 20) + (uint32_t)n - 1) / (uint32_t)n;  // e / n = e inv_n >> 20 for e < 2048
  for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = f;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += wsum[w];
    thr = 1e-16 * sqrt(t);
  }
  __syncthreads();
  bool any = false;  // warp 0: this lane has found an entry to rotate in this sweep
  auto angles = [&](int round, int to) {
    if ((int)threadIdx.x >= half) return;
    // round-robin pairing: player 0 fixed, the others rotate
    int const k = threadIdx.x;
    auto pos = [&](int q) {
      int const at = q - 1 + round;  // below 2 (n - 1)
      return q == 0 ? 0 : 1 + (at >= n - 1 ? at - (n - 1) : at);
    };
    int const p0 = pos(k), q0 = pos(n - 1 - k), p = min(p0, q0), q = max(p0, q0);
    double const apq = A[p * ld + q];
    double h = 0.0;
    if (fabs(apq) > thr) h = half_angle(apq, A[q * ld + q] - A[p * ld + p]);
    any = any || h != 0.0;
    cs[to][k][0] = h;
    cs[to][k][1] = h == 0.0 ? 0.0 : 2.0 * h / fma(h, h, 1.0);
    pp[to][k][0] = p;
    pp[to][k][1] = q;
  };
  int at = 0;
  if (threadIdx.x < 32) angles(0, at);
  __syncthreads();
  for (int sweep = 0; sweep < 40; ++sweep) {
    for (int round = 0; round < n - 1; ++round, at ^= 1) {
      // A <- J^T A J
#pragma unroll
      for (int m = 0; m < kMine; ++m) {
        if (mine[m] < 0) continue;
        int const k1 = mine[m] >> 8, k2 = mine[m] & 255;
        double const h1 = cs[at][k1][0], s1 = cs[at][k1][1], h2 = cs[at][k2][0], s2 = cs[at][k2][1];
        if (s1 == 0.0 && s2 == 0.0) continue;
        int const p1 = pp[at][k1][0], q1 = pp[at][k1][1], p2 = pp[at][k2][0], q2 = pp[at][k2][1];
        double app = A[p1 * ld + p2], apq = A[p1 * ld + q2], aqp = A[q1 * ld + p2], aqq = A[q1 * ld + q2];
        rotate(h1, s1, app, aqp);
        rotate(h1, s1, apq, aqq);
        rotate(h2, s2, app, apq);
        rotate(h2, s2, aqp, aqq);
        A[p1 * ld + p2] = app;
        A[p1 * ld + q2] = apq;
        A[q1 * ld + p2] = aqp;
        A[q1 * ld + q2] = aqq;
        if (k1 != k2) {
          A[p2 * ld + p1] = app;
          A[q2 * ld + p1] = apq;
          A[p2 * ld + q1] = aqp;
          A[q2 * ld + q1] = aqq;
        }
      }
      __syncthreads();
      if (threadIdx.x < 32) {
        bool const last = round == n - 2;
        if (last) {
          bool const r = __any_sync(0xffffffffu, any);
          if (threadIdx.x == 0) rotated = r;
          any = false;
        }
        angles(last ? 0 : round + 1, at ^ 1);
      } else {
        // Q <- J^T Q
        for (uint32_t e = threadIdx.x - 32; e < (uint32_t)(half * n); e += blockDim.x - 32) {
          uint32_t const k = e * inv_n >> 20, col = e - k * (uint32_t)n;
          double const s = cs[at][k][1];
          if (s == 0.0) continue;
          double* qp = Q + pp[at][k][0] * n + col;
          double* qq = Q + pp[at][k][1] * n + col;
          double vp = *qp, vq = *qq;
          rotate(cs[at][k][0], s, vp, vq);
          *qp = vp;
          *qq = vq;
        }
      }
      __syncthreads();
    }
    if (!rotated) break;  // written again behind the next sweep's first barrier
  }
}

// Rayleigh-Ritz of T (n = 4 (j + 1)) by the leader CTA. T is assembled from
// the projections of every step (T[block p][block q] = C_p of step q for
// p <= q), which also covers the arrowhead couplings after a thick restart.
// The lowest min(8, n) Ritz values go to c.out[0..8), their vectors to c.Y,
// the residual estimates ||B_j y_last|| of the lowest four to c.out[8..12).
// Returns the largest estimate over the nev wanted pairs.
__device__ double rayleigh_ritz(ChainDesc const& c, uint32_t j, bool have_B, double* A, double* Q) {
  int const n = 4 * (int)(j + 1);
  constexpr int kStride = kMaxN * 4;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    int const r = e / n, q = e % n;
    int const br = r / 4, bq = q / 4, a = r % 4, b = q % 4;
    double v;
    if (br == bq)
      v = 0.5 * (ldcg(c.Tc + bq * kStride + br * 16 + a * 4 + b) + ldcg(c.Tc + bq * kStride + br * 16 + b * 4 + a));
    else if (br < bq)
      v = ldcg(c.Tc + bq * kStride + br * 16 + a * 4 + b);
    else
      v = ldcg(c.Tc + br * kStride + bq * 16 + b * 4 + a);
    A[r * (n + 1) + q] = v;
  }
  __syncthreads();
  jacobi(A, Q, n);
  __shared__ int idx[8];
  __shared__ double worst, last_row[16];
  int const nk = n < 8 ? n : 8, t = (int)threadIdx.x;
  if (t < 8) idx[t] = t < n ? t : 0;
  __syncthreads();
  if (t < n) {
    // the nk smallest diagonal entries, ascending
    double const v = A[t * (n + 1) + t];
    int rank = 0;
    for (int q = 0; q < n; ++q) {
      double const o = A[q * (n + 1) + q];
      rank += o < v || (o == v && q < t);
    }
    if (rank < nk) idx[rank] = t;
  }
  __syncthreads();
  if (t < nk) c.out[t] = A[idx[t] * (n + 1) + idx[t]];
  if (t < 16) {  // entry t % 4 of B_j y_last of Ritz vector t / 4
    double s = 0.0;
    if (have_B)
      for (int b = 0; b < 4; ++b) s += ldcg(c.Bblk + j * 16 + t % 4 * 4 + b) * Q[idx[t / 4] * n + 4 * (int)j + b];
    last_row[t] = s;
  }
  __syncthreads();
  if (t == 0) {
    worst = 0.0;
    for (int i = 0; i < kB; ++i) {
      double r2 = 0.0;
      for (int a = 0; a < 4; ++a) r2 += last_row[4 * i + a] * last_row[4 * i + a];
      c.out[8 + i] = sqrt(r2);
      if (i < (int)c.nev) worst = fmax(worst, sqrt(r2));
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < n * 8; e += blockDim.x) {
    int const q = e / 8, i = e % 8;
    c.Y[q * 8 + i] = i < nk ? Q[idx[i] * n + q] : 0.0;
  }
  __syncthreads();
  return worst;
}

// Ritz vectors Psi = V Y over the basis blocks 0..j (own rows): the lowest
// four into W, the next four into W2 when `both`. The products run in
// double-float arithmetic on the split blocks Vs (every block 0..j is split
// by the time of a restart); Y is split once per call. Ys: shared scratch of
// at least 4 (j + 1) x 16 doubles.
__device__ void ritz_vectors(Ctx& x, uint32_t j, double* Ys, bool both) {
  int const n = 4 * (int)(j + 1);
  float* Yh = reinterpret_cast<float*>(Ys);
  float* Yl = Yh + n * 8;
  for (int e = threadIdx.x; e < n * 8; e += blockDim.x) df_split(ldcg(x.c.Y + e), Yh[e], Yl[e]);
  __syncthreads();
  uint64_t const D = x.c.D;
  Row4s const* Vs = reinterpret_cast<Row4s const*>(x.c.Vs);
  for (int half = 0; half < (both ? 2 : 1); ++half) {
    double* out = half ? x.c.W2 : x.c.W;
    for (uint32_t l = threadIdx.x; l < x.n; l += blockDim.x) {
      uint64_t const r = x.row(l);
      float S[4] = {}, E[4] = {};
      for (int b = 0; b <= (int)j; ++b) {
        Row4s const a = Vs[(uint64_t)b * D + r];
        float const ah[4] = {a.h.x, a.h.y, a.h.z, a.h.w}, al[4] = {a.l.x, a.l.y, a.l.z, a.l.w};
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          int const k = (4 * b + s) * 8 + 4 * half;
#pragma unroll
          for (int i = 0; i < 4; ++i) df_mac(ah[s], al[s], Yh[k + i], Yl[k + i], S[i], E[i]);
        }
      }
      *reinterpret_cast<Row4*>(out + r * 4) = mk4((double)S[0] + (double)E[0], (double)S[1] + (double)E[1],
                                                  (double)S[2] + (double)E[2], (double)S[3] + (double)E[3]);
    }
  }
  __syncthreads();
}

__device__ void copy_block(Ctx& x, double* dst, double const* src) {
  for (uint32_t l = threadIdx.x; l < x.n; l += blockDim.x) {
    uint64_t const r = x.row(l);
    *reinterpret_cast<Row4*>(dst + r * 4) = *reinterpret_cast<Row4 const*>(src + r * 4);
  }
  __syncthreads();
}

__device__ void random_block(Ctx& x) {
  for (uint32_t l = threadIdx.x; l < x.n; l += blockDim.x) {
    uint64_t const r = x.row(l);
    uint32_t c[4] = {(uint32_t)r, (uint32_t)(r >> 32), 0xB10Cu, 0u};
    philox(c, (uint32_t)x.c.seed, (uint32_t)(x.c.seed >> 32));
    double v[4];
    for (int k = 0; k < 4; ++k) v[k] = 2.0 * ((double)c[k] * (1.0 / 4294967296.0)) - 1.0;
    *reinterpret_cast<Row4*>(x.c.V + r * 4) = mk4(v[0], v[1], v[2], v[3]);
  }
  __syncthreads();
}

// Whole solve of one problem by the CTAs of its group. Cycles end when the
// basis is full or the Ritz estimates converge; the lowest eight Ritz vectors
// and the last Lanczos block then seed the next cycle (thick restart: T starts
// as diag(theta_1..8) and the next step's projections supply the arrowhead
// couplings), or, after a breakdown, the lowest four alone (explicit restart).
__device__ void solve_chain(ChainDesc const& c, uint32_t rank, uint32_t ncta, uint32_t* bar, BatchArgs const& a,
                            double* red, double* tmp, double* C, double* A, double* Q, uint64_t* gs_bar,
                            uint32_t* gs_phase) {
  Ctx x{c, rank, ncta, bar, &a, 0, 0, 0, 0, 0, 0, 0, 0, 0, red, tmp, A, gs_bar, gs_phase};
  auto piece = [&](uint32_t q) { return c.n_slices * q / (2 * ncta); };
  x.sa = piece(rank);
  x.sb = piece(2 * ncta - 1 - rank);
  x.ns0 = (uint32_t)(piece(rank + 1) - x.sa);
  x.ns = x.ns0 + (uint32_t)(piece(2 * ncta - rank) - x.sb);
  auto row_of = [&](uint64_t s) { return std::min<uint64_t>(c.D, s * 32); };
  x.ra = row_of(x.sa);
  x.rb = row_of(x.sb);
  x.n0 = (uint32_t)(row_of(x.sa + x.ns0) - x.ra);
  x.n = x.n0 + (uint32_t)(row_of(x.sb + (x.ns - x.ns0)) - x.rb);
  bool const leader = rank == 0;
  constexpr int kStride = kMaxN * 4;
  __shared__ double Rb[16];
  Row4s* Vs = reinterpret_cast<Row4s*>(c.Vs);
  uint32_t steps = 0, restarts = 0, matvecs = 0, status = 2;
  double const tol = a.tol;
  // phase timers, kept by thread 0 in shared memory (no registers held
  // across the phases)
  __shared__ unsigned long long acc[6], tmark;
  if (threadIdx.x == 0) {
    for (int q = 0; q < 6; ++q) acc[q] = 0;
    tmark = tc::global_ns();
  }
  auto lap = [&](int phase) {
    if (threadIdx.x == 0) {
      unsigned long long const now = tc::global_ns();
      acc[phase] += now - tmark;
      tmark = now;
    }
  };
  random_block(x);
  bool qr_ok;
  if (!block_qr(x, c.V, Rb, qr_ok)) {
    if (!qr_ok) return;
    status = 3;
  }
  uint32_t j0 = 0;
  // Whether a cycle may end before its basis is full: not while the last true
  // residual is above 1000 tol, since a whole cycle of ten block steps gains
  // a factor of 6 to 100 (the chains of 12 to 28 sites), and the solves of T
  // in between keep the group waiting for its first CTA. Same step counts and
  // eigenvalues; 46 chains of 12 to 20 sites 28.5 -> 24.0 ms a call, 128 of 16
  // to 28 696 -> 686.
  bool near = true;
  while (status != 3) {
    uint32_t j = j0;
    // block whose H-image needs full projections in both passes: the
    // continuation block of a restart (arrowhead couplings) or a block with
    // replaced (random) columns
    uint32_t full_from = j0;
    bool broke = false;
    for (;; ++j) {
      if (j == 0) split_block(x, Vs, c.V);  // later blocks come split from the QR of each step or the restart
      if (!group_barrier(bar, ncta, a)) return;  // V_j complete on every CTA before the gathers
      lap(4);
      block_spmv_df(x, j);
      ++matvecs;
      lap(0);
      // Gram-Schmidt and QR -> V_{j+1}, B_j (with deflation of lost directions)
      bool replaced = false;
      broke = !lanczos_step(x, j + 1, C, Rb, j > full_from ? j - 1 : 0u, steps + 1, replaced, lap);
      ++steps;
      if (replaced) full_from = j + 1;
      if (*(volatile int*)a.error) return;
      if (leader)
        for (int k = threadIdx.x; k < 16 * (int)(j + 1); k += blockDim.x) c.Tc[j * kStride + k] = C[k];
      if (leader)
        for (int k = threadIdx.x; k < 16; k += blockDim.x) c.Bblk[j * 16 + k] = broke ? 0.0 : Rb[k];
      lap(2);
      bool const full = j + 1 >= c.m_blocks || steps >= a.max_steps || broke;
      if (full || (near && (j + 1) % a.rr_every == 0)) {
        __threadfence();
        if (!group_barrier(bar, ncta, a)) return;  // T and B visible to the leader
        if (leader) {
          double const worst = rayleigh_ritz(c, j, !broke, A, Q);
          if (threadIdx.x == 0) {
            c.flag[0] = (worst <= 0.5 * tol) ? 1u : 0u;
            __threadfence();
          }
        }
        if (!group_barrier(bar, ncta, a)) return;
        lap(3);
        if (ldcg(c.flag) != 0u || full) break;
      }
    }
    bool const thick = !broke && j >= 1 && c.m_blocks >= 3;
    ritz_vectors(x, j, A, thick);  // A: the dynamic shared area, free outside the Jacobi solve
    if (!group_barrier(bar, ncta, a)) return;  // every CTA done reading the old basis
    if (thick) {  // Vs: the Ritz vectors, then the last Lanczos block
      if (j + 1 != 2)
        for (uint32_t l = threadIdx.x; l < x.n; l += blockDim.x) {
          uint64_t const r = x.row(l);
          Vs[2 * c.D + r] = Vs[(uint64_t)(j + 1) * c.D + r];
        }
      split_block(x, Vs, c.W);
      split_block(x, Vs + c.D, c.W2);
    }
    copy_block(x, c.V, c.W);
    if (!group_barrier(bar, ncta, a)) return;  // Psi rows visible to every CTA's SpMV gathers
    lap(4);
    // true residuals of the lowest four Ritz pairs
    block_spmv(x, c.V, c.W);
    ++matvecs;
    __syncthreads();
    double th[8];
    for (int i = 0; i < 8; ++i) th[i] = ldcg(c.out + i);
    {
      double p[4] = {};
      for (uint32_t l = threadIdx.x; l < x.n; l += blockDim.x) {
        uint64_t const r = x.row(l);
        Row4 const w = *reinterpret_cast<Row4 const*>(c.W + r * 4);
        Row4 const v = *reinterpret_cast<Row4 const*>(c.V + r * 4);
        double const d[4] = {w.x - th[0] * v.x, w.y - th[1] * v.y, w.z - th[2] * v.z, w.w - th[3] * v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = fma(d[i], d[i], p[i]);
      }
      cta_sum<4>(p, red, tmp);
      if (!group_sum(x, tmp, 4, tmp + 16)) return;
    }
    lap(5);
    bool all = true;
    near = true;
    for (uint32_t i = 0; i < c.nev; ++i) {
      all = all && sqrt(tmp[16 + i]) <= tol;
      near = near && sqrt(tmp[16 + i]) <= 1000.0 * tol;
    }
    __syncthreads();
    if (leader && threadIdx.x == 0)
      for (uint32_t i = 0; i < 4; ++i) c.out[8 + i] = sqrt(tmp[16 + i]);
    if (all) {
      status = 1;
      break;
    }
    if (steps >= a.max_steps) break;
    ++restarts;
    if (thick) {
      // T of the new cycle: diag(theta_1..8) on blocks 0 and 1
      if (leader) {
        for (int k = threadIdx.x; k < 2 * kStride; k += blockDim.x) c.Tc[k] = 0.0;
        __syncthreads();
        if (threadIdx.x < 8) {
          int const i = threadIdx.x, b = i / 4, a4 = i % 4;
          c.Tc[b * kStride + b * 16 + a4 * 4 + a4] = th[i];
        }
        __threadfence();
      }
      j0 = 2;
    } else {
      if (!block_qr(x, c.V, Rb, qr_ok)) {
        if (!qr_ok) return;
        status = 3;
        break;
      }
      j0 = 0;
    }
  }
  if (leader && threadIdx.x == 0) {
    c.stats[0] = steps;
    c.stats[1] = restarts;
    c.stats[2] = matvecs;
    c.stats[3] = status;
    for (int q = 0; q < 6; ++q) c.prof[q] = acc[q];
  }
}

__global__ void __launch_bounds__(256, 2) k_batch_lanczos(BatchArgs a) {
  __shared__ double red[8 * 16];
  __shared__ __align__(16) double tmp[2 * kPart];  // also read as float4 (split Gram-Schmidt coefficients)
  __shared__ double C[kPart];
  extern __shared__ __align__(128) double dyn[];  // A [kMaxN][kMaxN + 1], Q [kMaxN^2] (leader work); row-stream stages
  __shared__ uint64_t gs_bar[kGsStages];
  uint32_t gs_phase = 0;
  if (threadIdx.x == 0) {
    for (int q = 0; q < kGsStages; ++q) tc::mbar_init(&gs_bar[q], 1);
    tc::fence_mbar_init();
  }
  __syncthreads();
  uint32_t const gi = a.cta_group[blockIdx.x];
  GroupDesc const g = a.groups[gi];
  uint32_t const rank = blockIdx.x - g.cta0;
  for (uint32_t q = 0; q < g.count; ++q) {
    ChainDesc const& c = a.chains[a.order[g.first + q]];
    solve_chain(c, rank, g.ncta, g.bar, a, red, tmp, C, dyn, dyn + kMaxN * (kMaxN + 1), gs_bar, &gs_phase);
    if (*(volatile int*)a.error) return;
    if (!group_barrier(g.bar, g.ncta, a)) return;
  }
}

// chains[blockIdx.y].table_s = its FP64 matrix-element table split into
// double-float pairs.
__global__ void k_split_tables(ChainDesc const* __restrict__ chains) {
  ChainDesc const& c = chains[blockIdx.y];
  double const* t = static_cast<double const*>(c.S.table);
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < c.S.n_codes; k += gridDim.x * blockDim.x) {
    float h, l;
    df_split(t[k], h, l);
    c.table_s[k] = make_float2(h, l);
  }
}

// [D][4] block -> column-major D x nev with stride ld
__global__ void k_unpack_block(double const* __restrict__ V, uint64_t D, uint32_t nev, double* __restrict__ out,
                               uint64_t ld) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < D * nev; e += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t const i = e % D, c = e / D;
    out[c * ld + i] = V[i * 4 + c];
  }
}

// ------------------------------------------------------------ host side ---

// Groups of the persistent launch. A problem's block step on n CTAs is
// modelled as fixed + work / n: `fixed` is the part that more CTAs do not
// shorten (the leader's Rayleigh-Ritz solve, the group barriers), work the
// part that is split over the group's rows. The layout minimises the
// modelled makespan T on `grid` CTAs:
// - a problem with fixed + work > T gets a group of its own with
//   ceil(work / (T - fixed)) CTAs (at most max_ctas, its slice count);
// - the other problems are packed, first fit by decreasing work, into
//   one-CTA groups that solve them one after another within T;
// - T is the smallest bound (bisection) that needs no more than `grid` CTAs;
//   CTAs left over go one at a time to the multi-CTA group with the largest
//   modelled time.
struct BatchLayout {
  std::vector<GroupDesc> groups;
  std::vector<uint32_t> cta_group, order, group_of_chain;
};

BatchLayout batch_layout(std::vector<double> const& work, std::vector<uint32_t> const& max_ctas, double fixed,
                         unsigned grid) {
  size_t const count = work.size();
  std::vector<uint32_t> idx(count);
  std::iota(idx.begin(), idx.end(), 0u);
  std::stable_sort(idx.begin(), idx.end(), [&](uint32_t a, uint32_t b) { return work[a] > work[b]; });
  struct Try {
    std::vector<uint32_t> n;  // CTAs of a problem's own group, 0 when packed
    std::vector<std::vector<uint32_t>> bins;
    std::vector<double> load;
    unsigned ctas = 0;
  };
  auto attempt = [&](double T, Try& t) {
    t.n.assign(count, 0);
    t.bins.clear();
    t.load.clear();
    t.ctas = 0;
    for (uint32_t i : idx) {
      double const alone = fixed + work[i];
      if (alone <= T) {
        size_t b = 0;
        while (b < t.bins.size() && t.load[b] + alone > T) ++b;
        if (b == t.bins.size()) {
          t.bins.emplace_back();
          t.load.push_back(0.0);
          ++t.ctas;
        }
        t.bins[b].push_back(i);
        t.load[b] += alone;
      } else {
        if (T <= fixed) return false;
        double const need = std::ceil(work[i] / (T - fixed));
        if (need > (double)std::max<uint32_t>(1, max_ctas[i]) || need > (double)grid) return false;
        t.n[i] = (uint32_t)need;
        t.ctas += t.n[i];
      }
      if (t.ctas > grid) return false;
    }
    return true;
  };
  Try best;
  double hi = 0.0;
  for (double w : work) hi += fixed + w;
  hi = hi * 1.001 + 1.0;
  if (!attempt(hi, best)) {  // cannot happen: everything fits in one bin
    best.n.assign(count, 0);
    best.bins.assign(1, idx);
    best.ctas = 1;
  }
  double lo = 0.0;
  for (int it = 0; it < 64 && hi - lo > 1e-6 * hi; ++it) {
    double const mid = 0.5 * (lo + hi);
    Try t;
    if (attempt(mid, t)) {
      hi = mid;
      best = std::move(t);
    } else {
      lo = mid;
    }
  }
  // CTAs left over: to the slowest multi-CTA groups
  unsigned left = grid - std::min(grid, best.ctas);
  while (left > 0) {
    double worst = -1.0;
    uint32_t wi = UINT32_MAX;
    for (uint32_t i = 0; i < count; ++i)
      if (best.n[i] > 0 && best.n[i] < std::max<uint32_t>(1, max_ctas[i])) {
        double const t = fixed + work[i] / best.n[i];
        if (t > worst) {
          worst = t;
          wi = i;
        }
      }
    if (wi == UINT32_MAX) break;
    ++best.n[wi];
    --left;
  }
  BatchLayout L;
  L.group_of_chain.assign(count, 0);
  uint32_t cta = 0;
  for (uint32_t i : idx)
    if (best.n[i] > 0) {
      L.group_of_chain[i] = (uint32_t)L.groups.size();
      L.groups.push_back(GroupDesc{cta, best.n[i], (uint32_t)L.order.size(), 1, nullptr});
      L.order.push_back(i);
      cta += best.n[i];
    }
  for (auto const& bin : best.bins) {
    L.groups.push_back(GroupDesc{cta, 1, (uint32_t)L.order.size(), (uint32_t)bin.size(), nullptr});
    for (uint32_t i : bin) {
      L.group_of_chain[i] = (uint32_t)L.groups.size() - 1;
      L.order.push_back(i);
    }
    cta += 1;
  }
  for (uint32_t g = 0; g < L.groups.size(); ++g)
    for (uint32_t k = 0; k < L.groups[g].ncta; ++k) L.cta_group.push_back(g);
  return L;
}

struct Plan {
  unsigned threads = 256, ctas_per_sm = 1;
};

// Caller's fixed launch shape (sed_set_batched_launch); threads == 0: tune.
std::atomic<unsigned> g_force_threads{0}, g_force_per_sm{0};

std::mutex g_tune_mu;
std::map<std::tuple<int, unsigned, uint64_t>, Plan> g_tuned;

// Dynamic shared memory: the Rayleigh-Ritz solve's two matrices, or the row
// streams' stages. Not more: with 96 KB per CTA for wider stages the gathers in
// flight had too little of the 256 KB left as L1, and the SpMV took twice as
// long (870 -> 1385 ms for the 128-chain batch).
size_t dyn_smem() { return (size_t)kMaxN * (2 * kMaxN + 1) * sizeof(double); }

}  // namespace
}  // namespace sed

using namespace sed;

extern "C" {

int sed_eigh_batched(unsigned count, ls_operator* const ops[], sed_eigh_options const* opts, double* eigenvalues,
                     double* residuals, void* const eigenvectors[], uint64_t const ldv[], sed_batch_info* info) {
  auto t_start = std::chrono::steady_clock::now();
  if (count == 0) return LS_SUCCESS;
  if (!ops || !opts || !eigenvalues) return fail(LS_INVALID_ARGUMENT, "sed_eigh_batched: NULL argument");
  sed_eigh_options o{};
  sed_eigh_options_init(&o);
  std::memcpy(&o, opts, std::min<size_t>(sizeof(o), opts->struct_size ? opts->struct_size : sizeof(o)));
  uint32_t const nev = o.nev ? o.nev : 1;
  if (nev > (uint32_t)kB) return fail(LS_INVALID_ARGUMENT, "sed_eigh_batched: nev must be 1..4");
  if (o.block_size != 0 && o.block_size != 1 && o.block_size != (uint32_t)kB)
    return fail(LS_INVALID_ARGUMENT, "sed_eigh_batched: block_size must be 4");
  double const tol = o.tol > 0 ? o.tol : 1e-8;
  uint32_t const m_req = o.max_basis ? std::max<uint32_t>(2, o.max_basis / kB) : 12;
  int device = -1;
  if (int st = current_device(&device)) return st;
  std::vector<OperatorData*> od(count);
  for (unsigned i = 0; i < count; ++i) {
    if (!ops[i]) return fail(LS_INVALID_ARGUMENT, "sed_eigh_batched: NULL operator");
    od[i] = ops[i]->d.get();
    OperatorData& op = *od[i];
    if (!op.basis->built) return fail(LS_CACHE_NOT_BUILT, "basis has not been built (call ls_build)");
    if (op.basis->device != device) return fail(LS_INVALID_ARGUMENT, "sed_eigh_batched: operators on another device");
    if (!op.is_real) return fail(LS_OPERATOR_IS_COMPLEX, "sed_eigh_batched: operators must be real");
    if (op.basis->D < 2 * (uint64_t)kB) return fail(LS_INVALID_ARGUMENT, "sed_eigh_batched: dimension below 8");
    if (int st = operator_ensure_ready(op)) return st;
    if (!op.stream.ready)
      if (int st = operator_record_stream(op, op.cuda_stream)) return st;
  }
  for (unsigned i = 0; i < count; ++i) SED_TRY_CUDA(cudaStreamSynchronize(od[i]->cuda_stream));
  if (eigenvectors)
    for (unsigned i = 0; i < count; ++i)
      if (int st = wait_for_caller({eigenvectors[i]})) return st;
  auto t_setup = std::chrono::steady_clock::now();
  cudaStream_t stream = nullptr;
  SED_TRY_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
  struct StreamGuard {
    cudaStream_t s;
    ~StreamGuard() { cudaStreamDestroy(s); }
  } sguard{stream};

  int sms = 0, coop = 0;
  SED_TRY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  SED_TRY_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
  if (!coop) return fail(LS_CUDA_ERROR, "sed_eigh_batched: device lacks cooperative launch");
  SED_TRY_CUDA(cudaFuncSetAttribute(k_batch_lanczos, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn_smem()));
  // co-resident CTAs per SM for each block size (the cooperative launch
  // needs the whole grid resident)
  int occ128 = 0, occ256 = 0;
  SED_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ128, k_batch_lanczos, 128, dyn_smem()));
  SED_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ256, k_batch_lanczos, 256, dyn_smem()));
  int const max_per_sm = std::min(3, std::max(occ128, occ256));
  if (max_per_sm < 1) return fail(LS_CUDA_ERROR, "sed_eigh_batched: kernel does not fit on an SM");

  // work model per problem: streamed bytes of a block matvec plus the FP64
  // reorthogonalisation (rows x stored columns)
  std::vector<double> work(count);
  for (unsigned i = 0; i < count; ++i) {
    double const D = (double)od[i]->basis->D, E = (double)od[i]->stream.n_entries;
    work[i] = E * 4.0 + D * 40.0 + D * 16.0 * m_req * 6.0;
  }

  // Per-problem device arena
  std::vector<uint32_t> m_blocks(count);
  std::vector<size_t> off_V(count), off_Vs(count), off_Xs(count), off_Ts(count), off_W(count), off_W2(count), off_T(count), off_B(count), off_Y(count), off_out(count);
  size_t total = 0;
  auto take = [&](size_t bytes) {
    size_t const o = total;
    total += (bytes + 255) & ~size_t(255);
    return o;
  };
  for (unsigned i = 0; i < count; ++i) {
    uint64_t const D = od[i]->basis->D;
    uint32_t m = std::min<uint32_t>(std::min<uint32_t>(m_req, kMaxBlocks), (uint32_t)std::min<uint64_t>(kMaxBlocks, D / kB - 1));
    m = std::max<uint32_t>(m, 1);
    m_blocks[i] = m;
    off_V[i] = take((size_t)D * kB * 8);
    off_Vs[i] = take((size_t)(m + 1) * D * kB * 8);  // Row4s: 8 floats a row
    off_Xs[i] = take((size_t)D * kB * 8);
    off_Ts[i] = take((size_t)std::max<uint32_t>(1, od[i]->tables->n_codes) * sizeof(float2));
    off_W[i] = take((size_t)D * kB * 8);
    off_W2[i] = take((size_t)D * kB * 8);
    off_T[i] = take((size_t)kMaxBlocks * kMaxN * 4 * 8);
    off_B[i] = take((size_t)kMaxBlocks * 16 * 8);
    off_Y[i] = take((size_t)kMaxN * 8 * 8);
    off_out[i] = take(kOutBytes);
  }

  // Candidate launch shapes: 128 or 256 threads per CTA, 1 to 3 CTAs per SM
  // (as many as stay co-resident); the autotuner times each on a short trial
  // (two block steps of every problem) and keeps the fastest per (device,
  // count, size). A caller-fixed shape replaces the candidates.
  std::vector<Plan> cands;
  for (unsigned th : {256u, 128u}) {
    int const occ = th == 128 ? occ128 : occ256;
    for (unsigned per = 1; per <= (unsigned)std::min(occ, 3); ++per) cands.push_back(Plan{th, per});
  }
  if (unsigned const ft = g_force_threads.load()) {
    unsigned const fp = g_force_per_sm.load();
    int const occ = ft == 128 ? occ128 : occ256;
    if ((ft != 128 && ft != 256) || fp < 1 || (int)fp > std::min(occ, 3))
      return fail(LS_INVALID_ARGUMENT, "sed_eigh_batched: the fixed launch shape (" + std::to_string(ft) + " threads, " +
                                           std::to_string(fp) + " CTAs per SM) is not co-resident on this device");
    cands.assign(1, Plan{ft, fp});
  }
  uint64_t sumD = 0;
  for (unsigned i = 0; i < count; ++i) sumD += od[i]->basis->D;
  auto key = std::make_tuple(device, count, sumD);
  Plan plan = cands[0];
  bool tuned = cands.size() == 1;  // a fixed shape needs no trial runs
  if (!tuned) {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tuned.find(key);
    if (it != g_tuned.end()) {
      plan = it->second;
      tuned = true;
    }
  }

  // group layout for a given grid (batch_layout), the fixed part of a block
  // step expressed in rows of the batch's mean work per row
  using Layout = BatchLayout;
  std::vector<uint32_t> max_ctas(count);
  double sum_work = 0.0, sum_rows = 0.0;
  for (unsigned i = 0; i < count; ++i) {
    max_ctas[i] = (uint32_t)std::min<uint64_t>(od[i]->stream.n_slices, UINT32_MAX);
    sum_work += work[i];
    sum_rows += (double)od[i]->basis->D;
  }
  double const fixed = kLayoutFixedRows * sum_work / std::max(1.0, sum_rows);
  auto make_layout = [&](unsigned grid) { return batch_layout(work, max_ctas, fixed, grid); };

  unsigned max_per_cand = 1;
  for (Plan const& p : cands) max_per_cand = std::max(max_per_cand, p.ctas_per_sm);
  unsigned const max_grid = (unsigned)sms * max_per_cand;
  size_t const part_bytes = 2 * (size_t)max_grid * kPart * 8;
  std::vector<size_t> off_part(count);
  for (unsigned i = 0; i < count; ++i) off_part[i] = take(part_bytes);  // enough for any group size
  size_t const off_groups = take(sizeof(GroupDesc) * max_grid);
  size_t const off_ctag = take(4 * (size_t)max_grid);
  size_t const off_order = take(4 * (size_t)count);
  size_t const off_bars = take(8 * (size_t)max_grid);
  size_t const off_chains = take(sizeof(ChainDesc) * count);
  size_t const off_err = take(16);
  DeviceBuffer arena;
  if (int st = arena.allocate(total)) return st;
  char* base = arena.as<char>();

  std::vector<ChainDesc> chains(count);
  for (unsigned i = 0; i < count; ++i) {
    OperatorData& op = *od[i];
    ChainDesc& c = chains[i];
    c.S = stream_view(op);
    c.D = op.basis->D;
    c.n_slices = op.stream.n_slices;
    c.V = reinterpret_cast<double*>(base + off_V[i]);
    c.Vs = reinterpret_cast<float*>(base + off_Vs[i]);
    c.Xs = reinterpret_cast<float*>(base + off_Xs[i]);
    c.table_s = reinterpret_cast<float2*>(base + off_Ts[i]);
    c.W = reinterpret_cast<double*>(base + off_W[i]);
    c.part = reinterpret_cast<double*>(base + off_part[i]);
    c.W2 = reinterpret_cast<double*>(base + off_W2[i]);
    c.Tc = reinterpret_cast<double*>(base + off_T[i]);
    c.Bblk = reinterpret_cast<double*>(base + off_B[i]);
    c.Y = reinterpret_cast<double*>(base + off_Y[i]);
    c.out = reinterpret_cast<double*>(base + off_out[i]);
    c.stats = reinterpret_cast<uint32_t*>(base + off_out[i] + kStatsOff);
    c.flag = reinterpret_cast<uint32_t*>(base + off_out[i] + kStatsOff + 16);
    c.prof = reinterpret_cast<uint64_t*>(base + off_out[i] + kProfOff);
    c.m_blocks = m_blocks[i];
    c.nev = nev;
    c.packed = op.stream.packed ? 1u : 0u;
    c.seed = o.seed + 0x9E3779B97F4A7C15ull * (i + 1);
  }
  SED_TRY_CUDA(cudaMemcpyAsync(base + off_chains, chains.data(), sizeof(ChainDesc) * count, cudaMemcpyHostToDevice, stream));
  {
    uint32_t max_codes = 1;
    for (unsigned i = 0; i < count; ++i) max_codes = std::max(max_codes, od[i]->tables->n_codes);
    k_split_tables<<<dim3((max_codes + 255) / 256, count), 256, 0, stream>>>(
        reinterpret_cast<ChainDesc const*>(base + off_chains));
    note_launches(1);
  }

  uint32_t const max_steps_total = o.max_iter ? std::max<uint32_t>(1, o.max_iter / kB) : 2000;
  auto run = [&](Plan const& p, uint32_t max_steps, float* ms) -> int {
    unsigned const grid = (unsigned)sms * p.ctas_per_sm;
    Layout L = make_layout(grid);
    for (auto& g : L.groups) g.bar = reinterpret_cast<uint32_t*>(base + off_bars) + 2 * (&g - L.groups.data());
    unsigned const used = (unsigned)L.cta_group.size();
    SED_TRY_CUDA(cudaMemcpyAsync(base + off_groups, L.groups.data(), sizeof(GroupDesc) * L.groups.size(), cudaMemcpyHostToDevice, stream));
    SED_TRY_CUDA(cudaMemcpyAsync(base + off_ctag, L.cta_group.data(), 4 * (size_t)used, cudaMemcpyHostToDevice, stream));
    SED_TRY_CUDA(cudaMemcpyAsync(base + off_order, L.order.data(), 4 * (size_t)count, cudaMemcpyHostToDevice, stream));
    SED_TRY_CUDA(cudaMemsetAsync(base + off_bars, 0, 8 * (size_t)max_grid, stream));
    SED_TRY_CUDA(cudaMemsetAsync(base + off_err, 0, 16, stream));
    for (unsigned i = 0; i < count; ++i) SED_TRY_CUDA(cudaMemsetAsync(base + off_out[i], 0, kOutBytes, stream));
    BatchArgs a;
    a.chains = reinterpret_cast<ChainDesc const*>(base + off_chains);
    a.groups = reinterpret_cast<GroupDesc const*>(base + off_groups);
    a.cta_group = reinterpret_cast<uint32_t const*>(base + off_ctag);
    a.order = reinterpret_cast<uint32_t const*>(base + off_order);
    a.tol = tol;
    a.max_steps = max_steps;
    a.rr_every = 4;  // measured on the 128-chain workload: 772 ms against 797 ms every 2 steps, same step counts
    a.error = reinterpret_cast<int*>(base + off_err);
    a.wait_ns = device_wait_ns(kBarrierNs);
    a.copy_wait_ns = device_wait_ns(kGsWaitNs);
    a.stage_bytes = (uint32_t)dyn_smem();
    a.extra_arrivals = g_barrier_extra_arrivals.load();
    cudaEvent_t e0, e1;
    SED_TRY_CUDA(cudaEventCreate(&e0));
    SED_TRY_CUDA(cudaEventCreate(&e1));
    void* kargs[] = {&a};
    SED_TRY_CUDA(cudaEventRecord(e0, stream));
    cudaError_t le = cudaLaunchCooperativeKernel((void const*)k_batch_lanczos, dim3(used), dim3(p.threads), kargs,
                                                 dyn_smem(), stream);
    note_launches(1);
    SED_TRY_CUDA(cudaEventRecord(e1, stream));
    int err = 0;
    SED_TRY_CUDA(cudaMemcpyAsync(&err, base + off_err, 4, cudaMemcpyDeviceToHost, stream));
    cudaError_t se = cudaStreamSynchronize(stream);
    if (ms) cudaEventElapsedTime(ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    SED_TRY_CUDA(le);
    SED_TRY_CUDA(se);
    if (err) return fail(LS_DEVICE_TIMEOUT, err == 3 ? "sed_eigh_batched: a wait for a shared-memory copy timed out"
                                                    : "sed_eigh_batched: a group barrier timed out");
    return LS_SUCCESS;
  };

  if (!tuned && cands.size() > 1) {
    float best = 3e38f;
    for (Plan const& p : cands) {
      float ms = 0;
      if (int st = run(p, 2, &ms)) return st;
      if (ms < best) {
        best = ms;
        plan = p;
      }
    }
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tuned[key] = plan;
  }
  auto t_solve0 = std::chrono::steady_clock::now();
  float solve_ms = 0;
  if (int st = run(plan, max_steps_total, &solve_ms)) return st;

  // results
  std::vector<double> outs(12);
  std::vector<uint32_t> stats(4);
  bool all_ok = true;
  uint64_t max_steps = 0, max_restarts = 0, breakdowns = 0;
  std::string first_bad;
  for (unsigned i = 0; i < count; ++i) {
    SED_TRY_CUDA(cudaMemcpy(outs.data(), base + off_out[i], 96, cudaMemcpyDeviceToHost));
    SED_TRY_CUDA(cudaMemcpy(stats.data(), base + off_out[i] + kStatsOff, 16, cudaMemcpyDeviceToHost));
    for (uint32_t k = 0; k < nev; ++k) {
      eigenvalues[(size_t)i * nev + k] = outs[k];
      if (residuals) residuals[(size_t)i * nev + k] = outs[8 + k];
    }
    max_steps = std::max<uint64_t>(max_steps, stats[0]);
    max_restarts = std::max<uint64_t>(max_restarts, stats[1]);
    if (stats[3] != 1) {
      if (all_ok) {
        char buf[256];
        std::snprintf(buf, sizeof buf, " (first: problem %u, D = %llu, %u block steps, %u restarts, status %u, "
                      "residuals %.2e %.2e %.2e %.2e)", i, (unsigned long long)od[i]->basis->D, stats[0], stats[1],
                      stats[3], outs[8], outs[9], outs[10], outs[11]);
        first_bad = buf;
      }
      all_ok = false;
    }
    if (stats[3] == 3) ++breakdowns;
    if (eigenvectors && eigenvectors[i]) {
      uint64_t const D = od[i]->basis->D;
      uint64_t const ld = ldv ? ldv[i] : D;
      if (ld < D) return fail(LS_INVALID_ARGUMENT, "sed_eigh_batched: ldv below the dimension");
      DeviceBuffer tmpv;
      if (int st = tmpv.allocate((size_t)ld * nev * 8)) return st;
      { k_unpack_block<<<grid_size(D * nev, device), kBlock, 0, stream>>>(reinterpret_cast<double const*>(base + off_V[i]), D, nev, tmpv.as<double>(), ld); note_launches(1); }
      SED_TRY_CUDA(cudaMemcpyAsync(eigenvectors[i], tmpv.ptr, ((size_t)ld * (nev - 1) + D) * 8, cudaMemcpyDefault, stream));
      SED_TRY_CUDA(cudaStreamSynchronize(stream));
    }
  }
  if (logging_enabled()) {
    unsigned worst = 0;
    uint64_t worst_t = 0;
    std::vector<uint64_t> prof(8);
    Layout const L0 = make_layout((unsigned)sms * plan.ctas_per_sm);
    for (unsigned i = 0; i < count; ++i) {
      SED_TRY_CUDA(cudaMemcpy(prof.data(), base + off_out[i] + kProfOff, 64, cudaMemcpyDeviceToHost));
      SED_TRY_CUDA(cudaMemcpy(stats.data(), base + off_out[i] + kStatsOff, 16, cudaMemcpyDeviceToHost));
      uint64_t t = 0;
      for (int q = 0; q < 6; ++q) t += prof[q];
      GroupDesc const& g = L0.groups[L0.group_of_chain[i]];
      log_line("sed_eigh_batched: problem %u: D = %llu, group %u (%u CTAs, %u problems), %u block steps, %.2f ms "
               "(rayleigh-ritz %.2f ms)", i, (unsigned long long)od[i]->basis->D, L0.group_of_chain[i], g.ncta,
               g.count, stats[0], t * 1e-6, prof[3] * 1e-6);
      if (t > worst_t) {
        worst_t = t;
        worst = i;
      }
    }
    SED_TRY_CUDA(cudaMemcpy(prof.data(), base + off_out[worst] + kProfOff, 64, cudaMemcpyDeviceToHost));
    SED_TRY_CUDA(cudaMemcpy(stats.data(), base + off_out[worst] + kStatsOff, 16, cudaMemcpyDeviceToHost));
    unsigned const ncta = L0.groups[L0.group_of_chain[worst]].ncta;
    log_line("sed_eigh_batched: slowest problem %u (D = %llu, %u CTAs, %u block steps, %u restarts): spmv %.2f ms, "
             "cgs2 %.2f ms, qr %.2f ms, rayleigh-ritz %.2f ms, ritz/restart %.2f ms, residual %.2f ms",
             worst, (unsigned long long)od[worst]->basis->D, ncta, stats[0], stats[1], prof[0] * 1e-6,
             prof[1] * 1e-6, prof[2] * 1e-6, prof[3] * 1e-6, prof[4] * 1e-6, prof[5] * 1e-6);
  }
  auto t_end = std::chrono::steady_clock::now();
  if (info) {
    info->block_steps_max = max_steps;
    info->restarts_max = max_restarts;
    info->seconds_total = std::chrono::duration<double>(t_end - t_start).count();
    info->seconds_setup = std::chrono::duration<double>(t_setup - t_start).count();
    info->seconds_solve = std::chrono::duration<double>(t_end - t_solve0).count();
    info->kernel_ms = solve_ms;
    info->ctas_per_sm = plan.ctas_per_sm;
    info->threads_per_cta = plan.threads;
    info->grid = (uint32_t)(sms * plan.ctas_per_sm);
  }
  if (logging_enabled())
    log_line("sed_eigh_batched: %u problems, %.3f ms in one launch (%u CTAs/SM), max %llu block steps", count,
             solve_ms, plan.ctas_per_sm, (unsigned long long)max_steps);
  if (!all_ok)
    return fail(LS_NOT_CONVERGED, std::string(breakdowns ? "sed_eigh_batched: Krylov breakdown in some problems"
                                                         : "sed_eigh_batched: some problems did not converge") +
                                      first_bad);
  return LS_SUCCESS;
}

}  // extern "C"

extern "C" void sed_set_batched_launch(unsigned threads_per_cta, unsigned ctas_per_sm) {
  sed::g_force_threads.store(threads_per_cta ? threads_per_cta : 0u);
  sed::g_force_per_sm.store(threads_per_cta ? ctas_per_sm : 0u);
}

extern "C" unsigned sed_debug_batched_layout(unsigned count, double const* work, uint32_t const* max_ctas, double fixed,
                                             unsigned grid, uint32_t* group_of, uint32_t* ncta, uint32_t* nprob) {
  if (count == 0 || grid == 0 || !work || !max_ctas || !group_of || !ncta || !nprob || !(fixed >= 0.0)) return 0;
  std::vector<double> w(work, work + count);
  std::vector<uint32_t> m(max_ctas, max_ctas + count);
  for (double x : w)
    if (!(x >= 0.0)) return 0;
  sed::BatchLayout const L = sed::batch_layout(w, m, fixed, grid);
  if (L.groups.size() > grid) return 0;
  for (unsigned i = 0; i < count; ++i) group_of[i] = L.group_of_chain[i];
  for (size_t g = 0; g < L.groups.size(); ++g) {
    ncta[g] = L.groups[g].ncta;
    nprob[g] = L.groups[g].count;
  }
  return (unsigned)L.groups.size();
}
