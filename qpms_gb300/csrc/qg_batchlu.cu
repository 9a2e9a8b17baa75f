// Batched LU with partial pivoting of small row-major complex matrices, and
// the matching substitutions, for the mode problems of dispersion scans,
// serving batches and the finite plane-wave scatter (N <= 512).  The
// reference factorises each matrix with LAPACKE_zgetrf and solves with
// LAPACKE_zgetrs (scatsystem.c:2202-2273); the factors here have the same
// meaning (P M = L U, unit-lower L below the diagonal, U on and above, ipiv[i]
// the row exchanged with row i at step i, 0-based) on the row-major matrix
// as the reference stores it.
//
// getrf, N <= 64: one CTA per matrix with the matrix in shared memory
// (getrf_small_kernel).  Above: a cluster of C CTAs per matrix
// (getrf_cluster_kernel), right-looking by panels of PW columns held in
// registers; while CTA 0 brings the next panel up to date and factors it, the
// others update the remaining columns, one cluster barrier per panel.
// getrs: one warp per system with the factors in shared memory up to N = 64,
// one CTA per system by blocks of 32 unknowns above.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>

#include <atomic>

#include "qg_batchlu.h"
#include "qg_internal.h"
#include "qg_ktimer.h"

namespace qg {
namespace {

namespace cg = cooperative_groups;

// PW: panel columns.  CT: columns of an update tile (256 bytes of a row).
// PT: threads that factor a panel, each with kBatchLuMaxN / PT rows of it in
// registers; complex128 takes half the threads, because every warp of them
// forms the pivot's reciprocal and FP64 instructions cost 64 times FP32's.
template <typename T>
struct BL;
template <>
struct BL<float2> {
  typedef float R;
  static constexpr int PW = 16, CT = 32, PT = 256;
};
template <>
struct BL<double2> {
  typedef double R;
  static constexpr int PW = 8, CT = 16, PT = 128;
};

template <typename T>
__device__ __forceinline__ T cmk(typename BL<T>::R r, typename BL<T>::R i) {
  T z;
  z.x = r;
  z.y = i;
  return z;
}
__device__ __forceinline__ float fmar(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fmar(double a, double b, double c) { return fma(a, b, c); }
template <typename T>
__device__ __forceinline__ T cfma(T acc, T a, T b) {
  return cmk<T>(fmar(-a.y, b.y, fmar(a.x, b.x, acc.x)), fmar(a.y, b.x, fmar(a.x, b.y, acc.y)));
}
template <typename T>
__device__ __forceinline__ T cfms(T acc, T a, T b) {  // acc - a b
  return cmk<T>(fmar(a.y, b.y, fmar(-a.x, b.x, acc.x)), fmar(-a.y, b.x, fmar(-a.x, b.y, acc.y)));
}
template <typename T>
__device__ __forceinline__ T cmul(T a, T b) {
  return cmk<T>(fmar(-a.y, b.y, a.x * b.x), fmar(a.y, b.x, a.x * b.y));
}
// The largest exponent of b's parts, in units of 2^23 (FP32) or 2^20 (FP64).
__device__ __forceinline__ unsigned cexponent(float2 b) {
  return max(__float_as_uint(b.x) & 0x7fffffffu, __float_as_uint(b.y) & 0x7fffffffu);
}
__device__ __forceinline__ unsigned cexponent(double2 b) {
  return max((unsigned)__double2hiint(b.x) & 0x7fffffffu, (unsigned)__double2hiint(b.y) & 0x7fffffffu);
}
template <typename T>
__device__ __forceinline__ T crcp_plain(T b) {
  typedef typename BL<T>::R R;
  const R s = R(1) / fmar(b.x, b.x, b.y * b.y);
  return cmk<T>(b.x * s, -b.y * s);
}
template <typename T>
__device__ __noinline__ T crcp_scaled(T b, bool small) {
  typedef typename BL<T>::R R;
  const R up = R(sizeof(R) == 4 ? 0x1p75 : 0x1p600), f = small ? up : R(1) / up;
  const T r = crcp_plain(cmk<T>(b.x * f, b.y * f));
  return cmk<T>(r.x * f, r.y * f);
}
// 1 / b over the whole range of b: outside of 2^+-60 (FP32) or 2^+-500 (FP64), where
// |b|^2 may leave the type's range, b is scaled by a power of two.
template <typename T>
__device__ __forceinline__ T crcp(T b) {
  constexpr bool kF = sizeof(T) == 8;
  constexpr unsigned kOne = kF ? 127u << 23 : 1023u << 20, kSpan = kF ? 60u << 23 : 500u << 20;
  const unsigned x = cexponent(b);
  if (x - (kOne - kSpan) > 2 * kSpan) return crcp_scaled(b, x < kOne);  // rare
  return crcp_plain(b);
}

// a / b with r = crcp(b) at hand: a r corrected by the remainder, as good as a
// division; or a r alone for the complex128 multipliers, which are small against
// the pivot.  Errors of solves by the two factorisations and substitutions against
// divisions and tree sums, geometric mean over 200 to 400 matrices I - T S of
// clusters: complex64 0.93 to 1.01, complex128 0.97 to 1.00, at 12 to 512 unknowns
// (a r in place of every quotient and plain chains in the substitutions: up to
// 1.29 and 1.60).
template <typename T>
__device__ __forceinline__ T cquo_near(T a, T b, T r) {
  const T q = cmul(a, r);
  return cfma(q, cfms(a, q, b), r);
}
template <typename T>
__device__ __forceinline__ T cquo(T a, T b, T r) {
  return sizeof(T) == 16 ? cmul(a, r) : cquo_near(a, b, r);
}

// Pivot search over |Re| + |Im| (LAPACK's izamax measure), first of equals.
// A key orders candidates as unsigned integers, 0 for a NaN.  complex128: the bits
// of the measure plus one.  complex64: the measure with all its bits, as the FP32
// sum plus one and, below it, the sum's rounding error (TwoSum), which orders equal
// sums: the exact sums' order without FP64 instructions.  (32 LUs of 256 unknowns
// 278 us, with the FP32 sum alone, which takes the first of sums equal in 24 bits,
// 254 us; forming the low word only where the high words are equal, behind branches
// in the unrolled columns, 342 us.)
typedef unsigned long long PivKey;
__device__ __forceinline__ PivKey pivot_key(float2 z) {
  const float a = fabsf(z.x), b = fabsf(z.y), s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t));
  const int f = __float_as_int(e);
  unsigned low = f < 0 ? ~(unsigned)f : (unsigned)f | 0x80000000u;  // e's order
  if (isinf(s)) low = __float_as_uint(fmaf(0.5f, a, 0.5f * b));     // and of finite numbers past FP32's range
  return s >= 0 ? (PivKey)(__float_as_uint(s) + 1u) << 32 | low : 0ull;
}
__device__ __forceinline__ PivKey pivot_key(double2 z) {
  const double v = fabs(z.x) + fabs(z.y);
  return v >= 0 ? (PivKey)__double_as_longlong(v) + 1ull : 0ull;
}
__device__ __forceinline__ PivKey warp_max(PivKey k) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32));
  const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32) == hi ? (unsigned)k : 0u);
  return ((PivKey)hi << 32) | lo;
}

template <typename T>
__device__ __forceinline__ T shfl_c(T v, int lane) {
  return cmk<T>(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}

// ---------------- N <= 64: the matrix in shared memory ----------------
// Unblocked right-looking elimination, a rank-1 update per column: the FP64
// pipe (two FMAs per clock and SM) is the bound of the complex128 update
// whether its operands come from registers or shared memory, so nothing is
// gained from blocking here, and several CTAs share an SM to cover each
// other's pivot searches and barriers (three per column).
// Measured, complex128 (one CTA of 256 threads with panels of 16 columns through
// global memory before -> now): 4,096 matrices of N = 30 2,410 -> 455 us,
// 1,005 of N = 60 1,724 -> 863 us (0.29 and 0.58 GFLOP: 235 and 463 us at the
// FP64 pipes' 1.25 TFLOP/s).
constexpr int kSmallN = 64, kSmallThreads = 128;

template <typename T>
__global__ void __launch_bounds__(kSmallThreads) getrf_small_kernel(int N, T *A_all, int *piv_all, int *info_all) {
  extern __shared__ __align__(16) unsigned char sm[];
  T *S = reinterpret_cast<T *>(sm);
  const int LD = N + 1;
  __shared__ T lcol[kSmallN];
  __shared__ T s_rinv, s_piv, s_old;
  __shared__ int s_p;
  T *A = A_all + (size_t)blockIdx.x * N * N;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int t = tid, r = t / N, c = t - r * N; t < N * N; t += kSmallThreads) {
    S[r * LD + c] = A[t];
    c += kSmallThreads;
    while (c >= N) {
      c -= N;
      ++r;
    }
  }
  __syncthreads();
  int info = 0;
  for (int c = 0; c < N; ++c) {
    if (tid < 32) {
      PivKey k0 = 0, k1 = 0;
      const int r0 = c + lane, r1 = r0 + 32;
      if (r0 < N) k0 = pivot_key(S[r0 * LD + c]);
      if (r1 < N) k1 = pivot_key(S[r1 * LD + c]);
      const bool second = k1 > k0;
      const PivKey best = warp_max(second ? k1 : k0);
      unsigned r = INT_MAX;
      if (r0 < N && k0 == best)
        r = r0;
      else if (r1 < N && k1 == best)
        r = r1;
      const int p = (int)__reduce_min_sync(0xffffffffu, r);
      if (lane == 0) {
        const T d = S[p * LD + c];
        s_p = p;
        s_piv = d;
        s_old = S[c * LD + c];
        if (!(d.x == 0 && d.y == 0)) s_rinv = crcp(d);
        piv_all[(size_t)blockIdx.x * N + c] = p;
      }
    }
    __syncthreads();
    const int p = s_p;
    const T d = s_piv;
    const bool zero = (d.x == 0 && d.y == 0);
    if (zero && info == 0) info = c + 1;
    if (tid < 64) {  // column c: the pivot on the diagonal, multipliers below
      const int r = c + tid;
      if (r < N) {
        T v = r == c ? d : (r == p ? s_old : S[r * LD + c]);
        if (r > c) {
          if (!zero) v = cquo(v, d, s_rinv);
          lcol[r] = v;
        }
        S[r * LD + c] = v;
      }
    } else {  // exchange rows c and p in the other columns
      const int j = tid - 64;
      if (p != c && j < N && j != c) {
        const T a = S[c * LD + j];
        S[c * LD + j] = S[p * LD + j];
        S[p * LD + j] = a;
      }
    }
    __syncthreads();
    const int m = N - c - 1;
    if (!zero && m > 0) {
      const float im = 1.0f / m;
      for (int t = tid; t < m * m; t += kSmallThreads) {
        const int i = (int)((t + 0.5f) * im), j = t - i * m;  // exact: m * m <= 4096
        T *x = S + (c + 1 + i) * LD + c + 1 + j;
        *x = cfms(*x, lcol[c + 1 + i], S[c * LD + c + 1 + j]);
      }
    }
    __syncthreads();
  }
  for (int t = tid, r = t / N, c = t - r * N; t < N * N; t += kSmallThreads) {
    A[t] = S[r * LD + c];
    c += kSmallThreads;
    while (c >= N) {
      c -= N;
      ++r;
    }
  }
  if (tid == 0 && info_all) info_all[blockIdx.x] = info;
}

// ---------------- 64 < N <= 512: a cluster of CTAs per matrix ----------------
constexpr int kThreads = 256;

template <typename T>
struct ClusterSmem {
  static constexpr int PW = BL<T>::PW, CT = BL<T>::CT;
  static constexpr int LDP = PW + 16 / (int)sizeof(T);  // panel row stride: 16 bytes of padding
  static size_t bytes(int N) { return (2 * (size_t)N * LDP + (size_t)PW * CT) * sizeof(T); }
};

// The panel's row exchanges as one permutation of the rows it touches:
// row dst[e] receives row src[e].  The first pw entries are the panel's own
// rows, in order.
struct SwapList {
  int src[32], dst[32];
  int cnt;    // entries
  int moved;  // whether any row moves
};

// Called by warp 0.
__device__ __forceinline__ void build_swaps(SwapList &s, const int *piv, int k, int pw) {
  const int lane = threadIdx.x & 31;
  const int p0 = lane < pw ? piv[k + lane] : k + lane;
  const unsigned moved = __ballot_sync(0xffffffffu, p0 != k + lane);
  if (lane < pw) s.src[lane] = s.dst[lane] = k + lane;
  __syncwarp();
  int cnt = pw;
  for (unsigned left = moved; left; left &= left - 1) {  // uniform: the exchanges in order
    const int c = __ffs(left) - 1, p = __shfl_sync(0xffffffffu, p0, c);
    if (lane == 0) {
      int e = p - k;
      if (e >= pw) {
        for (e = pw; e < cnt && s.dst[e] != p; ++e) {
        }
        if (e == cnt) {
          s.src[e] = s.dst[e] = p;
          ++cnt;
        }
      }
      const int a = s.src[c];
      s.src[c] = s.src[e];
      s.src[e] = a;
    }
  }
  if (lane == 0) {
    s.cnt = cnt;
    s.moved = moved != 0;
  }
}

// Factors the panel of columns [k, k + pw): rows k..N-1 in registers (row
// k + tid + PT i in thread tid), one barrier per column.  Each warp offers its
// best row; the warp's winner and the owner of the diagonal row put these rows
// into one of two alternating slots, and after the barrier every thread picks
// the winner itself, exchanges and eliminates.  The panel comes from and goes
// back to Lp (a thread's row is strided in global memory: read and written
// from there it took as long as the elimination); the pivots (0-based rows of
// the matrix) go to piv.
template <typename T>
__device__ __forceinline__ void factor_panel(int N, int k, int pw, T *Lp, int *piv, int &info) {
  constexpr int PW = BL<T>::PW, PT = BL<T>::PT, RPT = kBatchLuMaxN / PT, NW = PT / 32;
  constexpr int LDP = ClusterSmem<T>::LDP;
  __shared__ T s_row[2][NW + 1][PW];
  __shared__ PivKey s_key[2][NW];
  __shared__ int s_r[2][NW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid >= PT) return;
  const int rows = N - k;
  T a[RPT][PW];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int r = tid + PT * i;
#pragma unroll
    for (int c = 0; c < PW; ++c) a[i][c] = (r < rows && c < pw) ? Lp[r * LDP + c] : cmk<T>(0, 0);
  }
#pragma unroll
  for (int c = 0; c < PW; ++c) {
    if (c < pw) {  // uniform
      const int buf = c & 1;
      PivKey key = 0;
      int br = INT_MAX;
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int r = tid + PT * i;
        if (r >= c && r < rows) {
          const PivKey q = pivot_key(a[i][c]);
          if (br == INT_MAX || q > key) {
            key = q;
            br = r;
          }
        }
      }
      const PivKey best = warp_max(key);
      const int rmin = (int)__reduce_min_sync(0xffffffffu, key == best ? (unsigned)br : (unsigned)INT_MAX);
      if (lane == 0) {
        s_key[buf][warp] = best;
        s_r[buf][warp] = rmin;
      }
      if (br == rmin && br != INT_MAX) {
#pragma unroll
        for (int i = 0; i < RPT; ++i)
          if (tid + PT * i == rmin)
#pragma unroll
            for (int j = 0; j < PW; ++j) s_row[buf][warp][j] = a[i][j];
      }
      if (tid == c) {
#pragma unroll
        for (int j = 0; j < PW; ++j) s_row[buf][NW][j] = a[0][j];
      }
      asm volatile("bar.sync 1, %0;" ::"n"(PT) : "memory");
      const int wl = min(lane, NW - 1);
      const PivKey wk = s_key[buf][wl], bk = warp_max(wk);
      const unsigned wr = wk == bk ? (unsigned)s_r[buf][wl] : (unsigned)INT_MAX;
      const int p = (int)__reduce_min_sync(0xffffffffu, wr);
      const int win = __ffs(__ballot_sync(0xffffffffu, wr == (unsigned)p)) - 1;
      T u[PW];
#pragma unroll
      for (int j = 0; j < PW; ++j) u[j] = s_row[buf][win][j];
      if (tid == 0) piv[k + c] = k + p;
      if (p != c) {
        if (tid == c) {
#pragma unroll
          for (int j = 0; j < PW; ++j) a[0][j] = u[j];
        }
#pragma unroll
        for (int i = 0; i < RPT; ++i)
          if (tid + PT * i == p)
#pragma unroll
            for (int j = 0; j < PW; ++j) a[i][j] = s_row[buf][NW][j];
      }
      const bool zero = (u[c].x == 0 && u[c].y == 0);
      if (zero) {
        if (info == 0) info = k + c + 1;
      } else {
        const T rinv = crcp(u[c]);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int r = tid + PT * i;
          if (PT * i < rows && r > c) {  // rows past the matrix hold zeros
            const T l = cquo(a[i][c], u[c], rinv);
            a[i][c] = l;
#pragma unroll
            for (int j = c + 1; j < PW; ++j) a[i][j] = cfms(a[i][j], l, u[j]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int r = tid + PT * i;
    if (r < rows) {
#pragma unroll
      for (int c = 0; c < PW; ++c) Lp[r * LDP + c] = a[i][c];
    }
  }
}

// The panel of columns [k, k + pw), rows k..N-1, between the matrix and shared memory.
template <typename T, bool STORE>
__device__ __forceinline__ void copy_panel(int N, int k, int pw, T *A, T *Lp) {
  constexpr int PW = BL<T>::PW, LDP = ClusterSmem<T>::LDP;
  const int c = threadIdx.x % PW;
  if (c >= pw) return;
#pragma unroll 4
  for (int r = threadIdx.x / PW; r < N - k; r += kThreads / PW) {
    if (STORE)
      A[(size_t)(k + r) * N + k + c] = Lp[r * LDP + c];
    else
      Lp[r * LDP + c] = A[(size_t)(k + r) * N + k + c];
  }
}

// Columns [c0, c0 + cw), cw <= CW, right of a full panel at k: row exchanges,
// U12 = L11^-1 A12 and A22 -= L21 U12.  Called by the whole CTA.  With `next`,
// A22's rows go there (the next panel, row stride LDP) and not to the matrix.
template <typename T, int CW>
__device__ __forceinline__ void update_tile(int N, int k, int c0, int cw, T *A, const T *Lp, T *Us,
                                            const SwapList &sw, T *next) {
  constexpr int PW = BL<T>::PW, LDP = ClusterSmem<T>::LDP;
  constexpr int PER = (2 * PW * CW + kThreads - 1) / kThreads;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  T v[PER];
  const int cnt = sw.cnt;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int e = (tid + kThreads * q) / CW, j = tid % CW;
    if (e < cnt && j < cw) v[q] = A[(size_t)sw.src[e] * N + c0 + j];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int e = (tid + kThreads * q) / CW, j = tid % CW;
    if (e < cnt && j < cw) {
      if (e < PW)
        Us[e * CW + j] = v[q];
      else
        A[(size_t)sw.dst[e] * N + c0 + j] = v[q];
    }
  }
  __syncthreads();
  // forward substitution with the unit lower L11: a lane per (row, column)
  for (int j0 = warp * (32 / PW); j0 < CW; j0 += (kThreads / 32) * (32 / PW)) {
    const int rr = lane % PW, cc = lane / PW, j = j0 + cc;
    T x = Us[rr * CW + j];
#pragma unroll
    for (int s = 0; s < PW - 1; ++s) {
      const T xs = shfl_c(x, cc * PW + s);
      if (rr > s) x = cfms(x, Lp[rr * LDP + s], xs);
    }
    Us[rr * CW + j] = x;
    if (j < cw) A[(size_t)(k + rr) * N + c0 + j] = x;
  }
  __syncthreads();
  {
    constexpr int RS = 32 / CW;  // rows of one warp step
    const int j = lane % CW, sub = lane / CW;
    T u[PW];
#pragma unroll
    for (int s = 0; s < PW; ++s) u[s] = Us[s * CW + j];
    if (j < cw) {
      constexpr int step = (kThreads / 32) * RS, UB = 4;  // UB rows in flight per thread
      for (int r = PW + warp * RS + sub; r < N - k; r += UB * step) {
        T acc[UB];
#pragma unroll
        for (int i = 0; i < UB; ++i)
          if (r + i * step < N - k) acc[i] = A[(size_t)(k + r + i * step) * N + c0 + j];
#pragma unroll
        for (int i = 0; i < UB; ++i) {
          if (r + i * step < N - k) {
            const T *l = Lp + (r + i * step) * LDP;
#pragma unroll
            for (int s = 0; s < PW; ++s) acc[i] = cfms(acc[i], l[s], u[s]);
            if (next)
              next[(r + i * step - PW) * LDP + j] = acc[i];
            else
              A[(size_t)(k + r + i * step) * N + c0 + j] = acc[i];
          }
        }
      }
    }
  }
  __syncthreads();
}

// Row exchanges of the columns [c0, c0 + cw) left of the panel.
template <typename T>
__device__ __forceinline__ void swap_tile(int N, int c0, int cw, T *A, const SwapList &sw) {
  constexpr int PW = BL<T>::PW, CW = BL<T>::CT;
  constexpr int PER = (2 * PW * CW + kThreads - 1) / kThreads;
  const int tid = threadIdx.x;
  T v[PER];
  const int cnt = sw.cnt;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int e = (tid + kThreads * q) / CW, j = tid % CW;
    if (e < cnt && j < cw) v[q] = A[(size_t)sw.src[e] * N + c0 + j];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int e = (tid + kThreads * q) / CW, j = tid % CW;
    if (e < cnt && j < cw) A[(size_t)sw.dst[e] * N + c0 + j] = v[q];
  }
  __syncthreads();
}

// C CTAs (one cluster) per matrix, C = 1 or >= 4.  Per panel: CTA 0 updates the
// next panel's columns and factors it (the serial chain), the other CTAs update
// the remaining tiles of CT columns and exchange rows on the left; with C = 1
// the one CTA does both.  All panel data pass through the matrix in global
// memory (L2); the cluster barrier orders them.  Every CTA runs the same
// number of barriers.
template <typename T>
__global__ void __launch_bounds__(kThreads) getrf_cluster_kernel(int N, int C, T *A_all, int *piv_all, int *info_all) {
  constexpr int PW = BL<T>::PW, CT = BL<T>::CT, LDP = ClusterSmem<T>::LDP;
  extern __shared__ __align__(16) unsigned char sm[];
  T *Lp = reinterpret_cast<T *>(sm);  // panel rows k..N-1, row stride LDP
  T *Ln = Lp + (size_t)N * LDP;       // CTA 0: the next panel
  T *Us = Ln + (size_t)N * LDP;       // U12 tile [PW][CT]
  __shared__ SwapList sw;
  const int m = blockIdx.x / C, cr = blockIdx.x - m * C;
  T *A = A_all + (size_t)m * N * N;
  int *piv = piv_all + (size_t)m * N;
  const int tid = threadIdx.x;
  cg::cluster_group cl = cg::this_cluster();
  int info = 0;
  if (cr == 0) {
    copy_panel<T, false>(N, 0, min(PW, N), A, Lp);
    __syncthreads();
    factor_panel(N, 0, min(PW, N), Lp, piv, info);
    __syncthreads();
    copy_panel<T, true>(N, 0, min(PW, N), A, Lp);
  }
  if (C > 1)
    cl.sync();
  else
    __syncthreads();
  for (int k = 0; k < N; k += PW) {
    const int pw = min(PW, N - k), k2 = k + pw, pn = min(PW, N - k2);
    if (tid < 32) build_swaps(sw, piv, k, pw);
    if (cr != 0 && pn > 0) copy_panel<T, false>(N, k, pw, A, Lp);
    __syncthreads();
    if (cr == 0 && pn > 0) update_tile<T, PW>(N, k, k2, pn, A, Lp, Us, sw, Ln);
    if (cr != 0 || C == 1) {
      const int first = C == 1 ? 0 : cr - 1, step = C == 1 ? 1 : C - 1;
      const int nt = pn > 0 ? (N - k2 - pn + CT - 1) / CT : 0;
      for (int t = first; t < nt; t += step) {
        const int c0 = k2 + pn + t * CT;
        update_tile<T, CT>(N, k, c0, min(CT, N - c0), A, Lp, Us, sw, (T *)nullptr);
      }
      if (sw.moved)
        for (int t = first; t * CT < k; t += step) swap_tile<T>(N, t * CT, min(CT, k - t * CT), A, sw);
    }
    if (cr == 0 && pn > 0) {
      T *t = Lp;
      Lp = Ln;
      Ln = t;
      factor_panel(N, k2, pn, Lp, piv, info);
      __syncthreads();
      copy_panel<T, true>(N, k2, pn, A, Lp);
    }
    if (C > 1)
      cl.sync();
    else
      __syncthreads();
  }
  if (cr == 0 && tid == 0 && info_all) info_all[m] = info;
}

// ---------------- substitutions, one right-hand side ----------------
// N <= 64: one warp per system, the factors staged in shared memory, lane l
// holding unknowns l and l + 32.
// b - sum x y, a term at a time, with no more roundings at the size of b than a
// sum over a tree: the products are summed apart from b, against which they are
// small in a mode problem, by K partial sums in turn, term q of K to sum q.
// get(q): the value after a term q; the other sums are added while term q is
// formed.  K: at 64 unknowns a general matrix's residual is 1.36 times that of
// divisions and tree sums with the products taken off b one by one, 1.28 with two
// sums, 1.13 with four, which cost 50 us of a scan of 4,096 matrices of 30.
template <typename T, int K>
struct PartSum {
  T b, a[K];
  __device__ __forceinline__ PartSum(T b_, T known) : b(b_) {
    a[0] = known;
#pragma unroll
    for (int i = 1; i < K; ++i) a[i] = cmk<T>(0, 0);
  }
  __device__ __forceinline__ void add(int q, T x, T y) { a[q] = cfma(a[q], x, y); }
  __device__ __forceinline__ T get(int q) const {
    T s[K];
#pragma unroll
    for (int i = 0; i < K - 1; ++i) s[i] = a[i < q ? i : i + 1];
#pragma unroll
    for (int n = K - 1; n > 1; n = (n + 1) / 2)
#pragma unroll
      for (int i = 0; i < n / 2; ++i) s[i] = cmk<T>(s[i].x + s[n - 1 - i].x, s[i].y + s[n - 1 - i].y);
    return cmk<T>(b.x - (a[q].x + s[0].x), b.y - (a[q].y + s[0].y));
  }
};
constexpr int kPart = 2;

// The same for the small substitutions: complex128 as above, complex64 with the
// roundings of the products and differences summed beside them (the error-free
// transformations of Knuth's TwoSum and of the product by FMA, as in Ogita, Rump
// and Oishi, Accurate Sum and Dot Product, 2005), since a lane's chain has up to 63
// terms.
template <typename T>
struct RowSum : PartSum<T, kPart> {
  __device__ __forceinline__ explicit RowSum(T b) : PartSum<T, kPart>(b, cmk<T>(0, 0)) {}
};
template <>
struct RowSum<float2> {
  float2 h, l;
  __device__ __forceinline__ explicit RowSum(float2 b) : h(b), l(make_float2(0, 0)) {}
  static __device__ __forceinline__ void term(float &h, float &l, float a, float b) {  // h + l -= a b
    const float p = __fmul_rn(a, b), e = __fmaf_rn(a, b, -p), s = __fsub_rn(h, p), z = __fsub_rn(s, h);
    l = __fadd_rn(l, __fsub_rn(__fsub_rn(__fsub_rn(h, __fsub_rn(s, z)), __fadd_rn(p, z)), e));
    h = s;
  }
  __device__ __forceinline__ void add(int, float2 a, float2 b) {
    term(h.x, l.x, a.x, b.x);
    term(h.x, l.x, -a.y, b.y);
    term(h.y, l.y, a.x, b.y);
    term(h.y, l.y, a.y, b.x);
  }
  __device__ __forceinline__ float2 get(int) const { return make_float2(h.x + l.x, h.y + l.y); }
};

template <typename T>
__global__ void __launch_bounds__(32) getrs_small_kernel(int N, const T *LU_all, const int *piv_all, T *b_all) {
  extern __shared__ __align__(16) unsigned char sm[];
  T *S = reinterpret_cast<T *>(sm);
  const int LD = N + 1, lane = threadIdx.x;
  T *xs = S + N * LD;  // [kSmallN]
  const T *A = LU_all + (size_t)blockIdx.x * N * N;
  const int *piv = piv_all + (size_t)blockIdx.x * N;
  T *b = b_all + (size_t)blockIdx.x * N;
  for (int t = lane, r = t / N, c = t - r * N; t < N * N; t += 32) {
    S[r * LD + c] = A[t];
    c += 32;
    while (c >= N) {
      c -= N;
      ++r;
    }
  }
  const int r0 = lane, r1 = lane + 32;
  if (r0 < N) xs[r0] = b[r0];
  if (r1 < N) xs[r1] = b[r1];
  const int p0 = r0 < N ? piv[r0] : 0, p1 = r1 < N ? piv[r1] : 0;
  __syncwarp();
  for (int i = 0; i < N; ++i) {
    const int p = __shfl_sync(0xffffffffu, i < 32 ? p0 : p1, i & 31);
    if (lane == 0 && p != i) {
      const T a = xs[i];
      xs[i] = xs[p];
      xs[p] = a;
    }
  }
  __syncwarp();
  const T z = cmk<T>(0, 0);
  RowSum<T> x0(r0 < N ? xs[r0] : z), x1(r1 < N ? xs[r1] : z);
  const int q0 = min(r0, N - 1), q1 = min(r1, N - 1);
  const T d0 = crcp(S[q0 * LD + q0]), d1 = N > 32 ? crcp(S[q1 * LD + q1]) : z;
  // terms j = j0 + q
  for (int j0 = 0; j0 < N; j0 += kPart)  // L y = P b, unit lower
#pragma unroll
    for (int q = 0; q < kPart; ++q) {
      const int j = j0 + q, last = (q + kPart - 1) % kPart;
      if (j < N) {
        const T y = shfl_c((j < 32 ? x0 : x1).get(last), j & 31);
        if (j < 31 && r0 > j) x0.add(q, S[q0 * LD + j], y);
        if (N > 32 && r1 > j) x1.add(q, S[q1 * LD + j], y);
      }
    }
  T u0 = x0.get(0), u1 = x1.get(0), w0 = z, w1 = z;
  x0 = RowSum<T>(u0);
  x1 = RowSum<T>(u1);
  const T g0 = S[q0 * LD + q0], g1 = S[q1 * LD + q1];
  for (int j0 = (N - 1) / kPart * kPart; j0 >= 0; j0 -= kPart)  // U x = y
#pragma unroll
    for (int q = kPart - 1; q >= 0; --q) {
      const int j = j0 + q, last = (q + 1) % kPart;
      if (j < N) {
        if (j < 32) {
          if (r0 == j) {
            w0 = x0.get(last);
            u0 = cquo(w0, g0, d0);
          }
        } else if (r1 == j) {
          w1 = x1.get(last);
          u1 = cquo(w1, g1, d1);
        }
        const T y = shfl_c(j < 32 ? u0 : u1, j & 31);
        if (r0 < j) x0.add(q, S[q0 * LD + j], y);
        if (j > 32 && r1 < j) x1.add(q, S[q1 * LD + j], y);
      }
    }
  if (sizeof(T) == 16) {  // the quotients' correction, off the chain (a scan of 4,096 matrices of 30: 3.07 -> 3.02 ms)
    u0 = cfma(u0, cfms(w0, u0, g0), d0);
    u1 = cfma(u1, cfms(w1, u1, g1), d1);
  }
  if (r0 < N) b[r0] = u0;
  if (r1 < N) b[r1] = u1;
}

// Above: one CTA per system, blocks of 32 unknowns.  Warp 0 solves a block's
// 32 x 32 triangle with a lane per row; meanwhile the other warps form the next
// block rows' products with the unknowns known before this block (coalesced
// along the rows) and stage the next triangle and the square beside it, so
// that between two triangles only the 32 new unknowns' products remain.
constexpr int kRsB = 32;

constexpr int kRsFar = 8, kRsThreads = 32 * (1 + kRsFar), kRsRows = kRsB / kRsFar;

template <typename T>
__global__ void __launch_bounds__(kRsThreads) getrs_block_kernel(int N, const T *LU_all, const int *piv_all, T *b_all) {
  typedef typename BL<T>::R R;
  __shared__ T x[kBatchLuMaxN], dinv[kBatchLuMaxN];
  __shared__ T tri[2][kRsB][kRsB + 1], near[kRsB][kRsB + 1], part[kRsB];
  __shared__ int sp[kBatchLuMaxN];
  const T *A = LU_all + (size_t)blockIdx.x * N * N;
  T *b = b_all + (size_t)blockIdx.x * N;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int moved = 0;
  for (int i = tid; i < N; i += kRsThreads) {
    x[i] = b[i];
    sp[i] = piv_all[(size_t)blockIdx.x * N + i];
    moved |= sp[i] != i;
    dinv[i] = crcp(A[(size_t)i * N + i]);
  }
  const int nb = (N + kRsB - 1) / kRsB;
  // stage q of 2 nb: the forward blocks in order, then the backward blocks
  auto block = [&](int q) { return (q < nb ? q : 2 * nb - 1 - q) * kRsB; };
  for (int t = tid; t < kRsB * kRsB; t += kRsThreads) {
    const int r = t / kRsB, c = t % kRsB;
    if (r < N && c < N) tri[0][r][c] = A[(size_t)r * N + c];
  }
  if (tid < kRsB) part[tid] = cmk<T>(0, 0);
  if (__syncthreads_or(moved)) {
    if (tid == 0)
      for (int i = 0; i < N; ++i) {
        const int p = sp[i];
        if (p != i) {
          const T a = x[i];
          x[i] = x[p];
          x[p] = a;
        }
      }
    __syncthreads();
  }
  for (int q = 0; q < 2 * nb; ++q) {
    const int i0 = block(q), bs = min(kRsB, N - i0);
    const bool more = q + 1 < 2 * nb, back = q + 1 >= nb;  // the next stage: is there one, is it backward
    const int n0 = more ? block(q + 1) : 0, ns = min(kRsB, N - n0);
    T acc[kRsRows];
    if (warp == 0) {
      const int r = min(lane, bs - 1);
      PartSum<T, kPart> v(x[i0 + r], part[r]);
      T u = cmk<T>(0, 0);
      const T(*tl)[kRsB + 1] = tri[q & 1];
      if (q < nb) {
        for (int j0 = 0; j0 < bs; j0 += kPart)
#pragma unroll
          for (int p = 0; p < kPart; ++p) {
            const int j = j0 + p;
            if (j < bs) {
              if (r == j) u = v.get((p + kPart - 1) % kPart);
              const T y = shfl_c(u, j);
              if (r > j) v.add(p, tl[r][j], y);
            }
          }
      } else {
        const T di = dinv[i0 + r];
        T w = u;
        for (int j0 = (bs - 1) / kPart * kPart; j0 >= 0; j0 -= kPart)
#pragma unroll
          for (int p = kPart - 1; p >= 0; --p) {
            const int j = j0 + p;
            if (j < bs) {
              if (r == j) {
                w = v.get((p + 1) % kPart);
                u = cmul(w, di);
              }
              const T y = shfl_c(u, j);
              if (r < j) v.add(p, tl[r][j], y);
            }
          }
        u = cfma(u, cfms(w, u, tl[r][r]), di);  // the quotient's correction, off the chain
      }
      if (lane < bs) x[i0 + lane] = u;
    } else if (more) {
      // the next triangle and the square beside it: lane = column, loads in flight together
      const int w0 = (warp - 1) * kRsRows;
      T vt[kRsRows], vn[kRsRows];
#pragma unroll
      for (int r = 0; r < kRsRows; ++r) {
        if (w0 + r < ns && lane < ns) vt[r] = A[(size_t)(n0 + w0 + r) * N + n0 + lane];
        if (w0 + r < ns && lane < bs) vn[r] = A[(size_t)(n0 + w0 + r) * N + i0 + lane];
      }
      // products with the unknowns of the stages before this one
      const int j0 = back ? i0 + bs : 0, j1 = back ? N : i0;
#pragma unroll
      for (int r = 0; r < kRsRows; ++r) acc[r] = cmk<T>(0, 0);
#pragma unroll 2
      for (int j = j0 + lane; j < j1; j += 32) {
        const T y = x[j];
#pragma unroll
        for (int r = 0; r < kRsRows; ++r) {
          const int i = n0 + min(w0 + r, ns - 1);
          acc[r] = cfma(acc[r], A[(size_t)i * N + j], y);
        }
      }
#pragma unroll
      for (int r = 0; r < kRsRows; ++r) {
        if (w0 + r < ns && lane < ns) tri[(q + 1) & 1][w0 + r][lane] = vt[r];
        if (w0 + r < ns && lane < bs) near[w0 + r][lane] = vn[r];
      }
    }
    __syncthreads();
    if (warp != 0 && more) {
      // the 32 new unknowns (none where the sweep turns round: the last forward
      // block is the first backward one)
      const int w0 = (warp - 1) * kRsRows;
      R v[8];
#pragma unroll
      for (int r = 0; r < kRsRows; ++r) {
        if (n0 != i0 && lane < bs && w0 + r < ns) acc[r] = cfma(acc[r], near[w0 + r][lane], x[i0 + lane]);
        v[2 * r] = acc[r].x;
        v[2 * r + 1] = acc[r].y;
      }
      const R sum = fold8(v, lane);
      if ((lane & 3) == 0) reinterpret_cast<R *>(part)[2 * w0 + (lane >> 2)] = sum;
    }
    __syncthreads();
  }
  for (int i = tid; i < N; i += kRsThreads) b[i] = x[i];
}

template <typename T>
void cluster_config(int C, int nm, int N, cudaStream_t st, cudaLaunchConfig_t *cfg, cudaLaunchAttribute *at) {
  *cfg = {};
  cfg->gridDim = dim3((unsigned)nm * C);
  cfg->blockDim = dim3(kThreads);
  cfg->dynamicSmemBytes = ClusterSmem<T>::bytes(N);
  cfg->stream = st;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = C;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg->attrs = at;
  cfg->numAttrs = 1;
}

// CTAs per matrix above N = 64.  The time of a batch, measured (us, GB300; diagonally
// dominant matrices, so without row exchanges):
//                            C = 1     4     6     8     9    16
//   complex128, N 512, 2     47300 15870 10080  7650  6815  4270  (FP64 pipes of C - 1 SMs)
//   complex128, N 390, 9     21710  7310  4770  3700  3300  4680  (two waves at 16)
//   complex128, N 200, 40     3310  2310  1740  2250  2190        (two, two, three and three waves)
//   complex64,  N 512, 2      2790   985   734   652   624   600  (the panels' serial chain)
//   complex64,  N 256, 32      570   278   533   786              (two and three waves)
// so the choice is the least waves x relative time, a wave being the clusters that the
// GPU holds at once (152, 36, 23, 15, 15, 7: a cluster lies within one group of SMs),
// among sizes whose CTAs all get a tile of the first update.  Relative times:
// complex128 as at N 512; complex64 between those of N 512 and N 256 (4 CTAs 0.35 and
// 0.49, 8 CTAs 0.23 and 0.46).  The counts are asked for once per device.
template <typename T>
int cluster_size(int nm, int N, int *C_out) {
  constexpr int kN = 6, kC[kN] = {1, 4, 6, 8, 9, 16}, kMaxDev = 64;
  constexpr double kCost[kN] = {1.0, sizeof(T) == 16 ? 0.34 : 0.45, sizeof(T) == 16 ? 0.22 : 0.35,
                                sizeof(T) == 16 ? 0.17 : 0.30, sizeof(T) == 16 ? 0.15 : 0.29,
                                sizeof(T) == 16 ? 0.10 : 0.25};
  static std::atomic<int> active[kMaxDev][kN];  // 0: not asked yet
  int dev = 0;
  QG_CUDA_TRY(cudaGetDevice(&dev));
  const int tiles = (N - 2 * BL<T>::PW + BL<T>::CT - 1) / BL<T>::CT;
  double best = 0;
  *C_out = 1;
  for (int i = 0; i < kN; ++i) {
    if (kC[i] > 1 && tiles < kC[i] - 1) break;
    int n = dev < kMaxDev ? active[dev][i].load() : 0;
    if (!n) {
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute at[1];
      cluster_config<T>(kC[i], 1, kBatchLuMaxN, 0, &cfg, at);
      QG_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, getrf_cluster_kernel<T>, &cfg));
      if (n < 1) n = -1;  // this size does not fit
      if (dev < kMaxDev) active[dev][i].store(n);
    }
    if (n < 1) continue;
    const double t = ((nm + n - 1) / n) * kCost[i];
    if (i == 0 || t < best) {
      best = t;
      *C_out = kC[i];
    }
  }
  return QPMS_SUCCESS;
}

template <typename T>
int cluster_launch(int nm, int N, T *A, int *piv, int *info, cudaStream_t st) {
  auto kern = getrf_cluster_kernel<T>;
  QG_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)ClusterSmem<T>::bytes(kBatchLuMaxN)));
  QG_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  int C = 1;
  const int e = cluster_size<T>(nm, N, &C);
  if (e) return e;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[1];
  cluster_config<T>(C, nm, N, st, &cfg, at);
  QG_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, N, C, A, piv, info));
  return QPMS_SUCCESS;
}

template <typename T>
int getrf_launch(int nm, int N, T *A, int *piv, int *info, cudaStream_t st) {
  if (N > kBatchLuMaxN) {
    set_error("batched LU: N = %d above %d", N, kBatchLuMaxN);
    return QPMS_EINVAL;
  }
  KtScope kt(KT_BATCHLU, st, nm * 8.0 * N * (double)N * N / 3.0);
  if (N <= kSmallN) {
    const size_t smem = (size_t)N * (N + 1) * sizeof(T);
    QG_CUDA_TRY(cudaFuncSetAttribute(getrf_small_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kSmallN * (kSmallN + 1) * (int)sizeof(T)));
    getrf_small_kernel<T><<<nm, kSmallThreads, smem, st>>>(N, A, piv, info);
    QG_CUDA_TRY(cudaGetLastError());
  } else {
    const int e = cluster_launch<T>(nm, N, A, piv, info, st);
    if (e) return e;
  }
  g_launches.fetch_add(1);
  return QPMS_SUCCESS;
}

template <typename T>
int getrs_launch(int nm, int N, const T *LU, const int *piv, T *b, cudaStream_t st) {
  if (N > kBatchLuMaxN) {
    set_error("batched LU: N = %d above %d", N, kBatchLuMaxN);
    return QPMS_EINVAL;
  }
  if (N <= kSmallN) {
    const size_t smem = ((size_t)N * (N + 1) + kSmallN) * sizeof(T);
    QG_CUDA_TRY(cudaFuncSetAttribute(getrs_small_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (kSmallN * (kSmallN + 1) + kSmallN) * (int)sizeof(T)));
    getrs_small_kernel<T><<<nm, 32, smem, st>>>(N, LU, piv, b);
  } else {
    getrs_block_kernel<T><<<nm, kRsThreads, 0, st>>>(N, LU, piv, b);
  }
  QG_CUDA_TRY(cudaGetLastError());
  g_launches.fetch_add(1);
  return QPMS_SUCCESS;
}

}  // namespace

int batch_getrf_c64(int nm, int N, void *A, int *piv, int *info, cudaStream_t st) {
  if (nm <= 0 || N <= 0) return QPMS_SUCCESS;
  return getrf_launch<float2>(nm, N, (float2 *)A, piv, info, st);
}
int batch_getrf_c128(int nm, int N, void *A, int *piv, int *info, cudaStream_t st) {
  if (nm <= 0 || N <= 0) return QPMS_SUCCESS;
  return getrf_launch<double2>(nm, N, (double2 *)A, piv, info, st);
}
int batch_getrs_c64(int nm, int N, const void *LU, const int *piv, void *b, cudaStream_t st) {
  if (nm <= 0 || N <= 0) return QPMS_SUCCESS;
  return getrs_launch<float2>(nm, N, (const float2 *)LU, piv, (float2 *)b, st);
}
int batch_getrs_c128(int nm, int N, const void *LU, const int *piv, void *b, cudaStream_t st) {
  if (nm <= 0 || N <= 0) return QPMS_SUCCESS;
  return getrs_launch<double2>(nm, N, (const double2 *)LU, piv, (double2 *)b, st);
}

}  // namespace qg

extern "C" int qpms_gpu_debug_batch_lu(int is_double, int nm, int N, void *A, int *piv, void *b) {
  using namespace qg;
  clear_error();
  if (nm <= 0 || N <= 0 || !A || !piv || !b) {
    set_error("batched LU: empty or NULL argument");
    return QPMS_EINVAL;
  }
  const size_t sz = is_double ? 16 : 8, na = (size_t)nm * N * N * sz, nb = (size_t)nm * N * sz, np = (size_t)nm * N * 4;
  char *d = nullptr;
  QG_CUDA_TRY(cudaMalloc(&d, na + nb + np));
  auto run = [&]() -> int {
    int *dp = (int *)(d + na + nb);
    QG_CUDA_TRY(cudaMemcpy(d, A, na, cudaMemcpyHostToDevice));
    QG_CUDA_TRY(cudaMemcpy(d + na, b, nb, cudaMemcpyHostToDevice));
    int e = is_double ? batch_getrf_c128(nm, N, d, dp, nullptr, 0) : batch_getrf_c64(nm, N, d, dp, nullptr, 0);
    if (e) return e;
    if ((e = is_double ? batch_getrs_c128(nm, N, d, dp, d + na, 0) : batch_getrs_c64(nm, N, d, dp, d + na, 0))) return e;
    QG_CUDA_TRY(cudaMemcpy(A, d, na, cudaMemcpyDeviceToHost));
    QG_CUDA_TRY(cudaMemcpy(b, d + na, nb, cudaMemcpyDeviceToHost));
    QG_CUDA_TRY(cudaMemcpy(piv, dp, np, cudaMemcpyDeviceToHost));
    return QPMS_SUCCESS;
  };
  const int e = run();
  cudaFree(d);
  return e;
}
