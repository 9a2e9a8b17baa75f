// Mode-problem assembly and the small-system solve pipeline on sm_103a.
//
// assemble_kernel writes the fecv x fecv blocks M_w[R, C] = delta_RC I - T_R
// S_w(R <- C) straight into the row-major complex128 matrix M_w (the
// reference's qpms_scatsysw_build_modeproblem_matrix_full,
// scatsystem.c:1283-1343, with the finite semantics S(R <- R) = 0).  S comes
// from the translation tables of the calculator: the per-pair factor table w
// (Hankel+ Bessel, Legendre, azimuthal phases) is built in shared memory, the
// elements of A and B are short FP64 dot products, one for each pair of
// elements that reciprocity makes equal up to sign, and each value lands in two
// blocks of the 2x2 (electric, magnetic) type structure
// (translations_inlines.h:213-240).  Diagonal T (Mie spheres) scales rows: a
// unit is then an unordered particle pair, because the opposite translation
// only changes signs, (-1)^(n + nu) for A and -(-1)^(n + nu) for B, and the
// dot products of a chunk's pairs form one list, so the lanes are full at every
// lMax.  A dense T is applied from shared memory, an ordered pair at a time.
// Bound: the FP64 pipe; the row scaling alone is four FMAs per element of M.
// 900 spheres at lMax 2 (14,400 unknowns, 3.3 GB): 2.9 ms, against 8.3 ms with
// a dot product per element and ordered pairs on CTAs of 256 threads.
#include <cuda_runtime.h>
#include <stdint.h>

#include "qg_internal.h"
#include "qg_ktimer.h"
#include "qg_specfunc.cuh"
#include "qg_assembly.h"

namespace qg {
namespace {

template <int LMAX>
struct AsmShape {
  static constexpr int L = 2 * LMAX + 1;
  static constexpr int S = (L + 1) * (L + 1);
  static constexpr int NL = (L + 1) * (L + 2) / 2;
  static constexpr int NE = LMAX * (LMAX + 2);
  static constexpr int NB = 2 * NE;  // block side
  // As in the translation kernel, small CTAs cover each other's set-up; V fills
  // the set-up's lanes where the pairs are cheap (us, one 14,400-unknown matrix
  // at lMax 2: V = 8 3,398, 16 3,013, 32 2,909; 14,400 at lMax 4: 2,404, 2,498,
  // 2,737).
  static constexpr int V = LMAX <= 2 ? 32 : (LMAX == 3 ? 16 : 8);
  static constexpr int kThreads = 128, kMinCtas = 5;
};

template <int LMAX>
constexpr size_t asm_smem_bytes(bool dense) {
  using Sh = AsmShape<LMAX>;
  return (size_t)Sh::V * Sh::S * 16 + (size_t)Sh::V * (Sh::L + 1) * 16 * 2 + (size_t)Sh::V * Sh::NL * 8 +
         (size_t)Sh::V * 32 + (dense ? (size_t)Sh::NB * Sh::NB * 16 : 0);
}

// degree n of the wave y = n(n+1) + m - 1
__device__ __forceinline__ int ydeg(int y) { return (int)sqrtf((float)y + 1.0f); }

struct __align__(16) PairInfo {
  double ct;
  int diag;   // R == C: identity block, no translation
  int valid;
  int w, R, C, pad;
};

template <int LMAX, bool DENSE>
__global__ void __launch_bounds__(AsmShape<LMAX>::kThreads, AsmShape<LMAX>::kMinCtas)
    assemble_kernel(AsmArgs a, TransDevTables T, int vc) {
  using Sh = AsmShape<LMAX>;
  constexpr int L = Sh::L, S = Sh::S, NL = Sh::NL, NE = Sh::NE, NB = Sh::NB, V = Sh::V;
  constexpr int kAThreads = Sh::kThreads;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  qg_c *w = reinterpret_cast<qg_c *>(smem_raw);
  qg_c *zb = w + V * S;
  qg_c *eph = zb + V * (L + 1);
  double *leg = reinterpret_cast<double *>(eph + V * (L + 1));
  PairInfo *info = reinterpret_cast<PairInfo *>(leg + V * NL);
  qg_c *sblk = reinterpret_cast<qg_c *>(info + V);  // [NB][NB] if DENSE

  const int tid = threadIdx.x;
  // a unit: the pair (R, C) of a frequency; unordered (C <= R) for a diagonal T
  const size_t np = (size_t)a.np, per = DENSE ? np * np : np * (np + 1) / 2, units = (size_t)a.nw * per;
  const size_t N = np * NB;
  const size_t nchunks = (units + vc - 1) / vc;  // vc <= V units per chunk
  for (size_t chunk = blockIdx.x; chunk < nchunks; chunk += gridDim.x) {
    const size_t base = chunk * vc;
    if (tid < vc) {
      const size_t u = base + tid;
      PairInfo inf;
      inf.valid = u < units;
      inf.diag = 1;
      inf.ct = 1.0;
      inf.w = inf.R = inf.C = 0;
      qg_c z[L + 1];
#pragma unroll
      for (int l = 0; l <= L; ++l) z[l] = cmk(0.0, 0.0);
      if (inf.valid) {
        const int wi = (int)(u / per);
        const size_t pr = u - (size_t)wi * per;
        inf.w = wi;
        if (DENSE) {
          inf.R = (int)(pr / np);
          inf.C = (int)(pr - (size_t)inf.R * np);
        } else {
          size_t r = (size_t)((sqrt(8.0 * (double)pr + 1.0) - 1.0) * 0.5);
          while ((r + 1) * (r + 2) / 2 <= pr) ++r;
          while (r * (r + 1) / 2 > pr) --r;
          inf.R = (int)r;
          inf.C = (int)(pr - r * (r + 1) / 2);
        }
        inf.diag = inf.R == inf.C;
        if (!inf.diag) {
          const double dx = a.pos[3 * inf.R] - a.pos[3 * inf.C];
          const double dy = a.pos[3 * inf.R + 1] - a.pos[3 * inf.C + 1];
          const double dz = a.pos[3 * inf.R + 2] - a.pos[3 * inf.C + 2];
          const double r = sqrt(dx * dx + dy * dy + dz * dz);
          // cart2sph (vectors.h:134-140), then kd.r *= k (translations.c:808-809); only
          // cos(theta) and e^{i phi} of the angles are needed (theta = pi/2, phi = 0 at r = 0)
          const double rho = sqrt(dx * dx + dy * dy);
          const qg_c k = a.k[wi];
          sph_bessel<L>(a.J, cmk(k.re * r, k.im * r), z);
          inf.ct = r > 0 ? dz / r : 0.0;
          const qg_c e1 = rho > 0 ? cmk(dx / rho, dy / rho) : cmk(1.0, 0.0);
          qg_c e = cmk(1.0, 0.0);
#pragma unroll
          for (int d = 0; d <= L; ++d) {
            eph[tid * (L + 1) + d] = e;
            e = cmul(e, e1);
          }
        }
      }
#pragma unroll
      for (int l = 0; l <= L; ++l) zb[tid * (L + 1) + l] = z[l];
      info[tid] = inf;
    }
    __syncthreads();
    for (int t = tid; t < vc * (L + 1); t += kAThreads) {
      const int v = t / (L + 1), m = t - v * (L + 1);
      if (!info[v].diag) legendre_column_rt(L, m, info[v].ct, leg + v * NL);
    }
    __syncthreads();
    for (int t = tid; t < vc * NL; t += kAThreads) {
      const int v = t / NL, i = t - v * NL;
      if (info[v].diag) continue;
      int p = (int)((sqrtf(8.0f * i + 1.0f) - 1.0f) * 0.5f);
      if ((p + 1) * (p + 2) / 2 <= i) ++p;
      if (p * (p + 1) / 2 > i) --p;
      const int ad = i - p * (p + 1) / 2;
      const qg_c uu = cscale(zb[v * (L + 1) + p], leg[v * NL + i]);
      const qg_c ph = eph[v * (L + 1) + ad];
      qg_c *wv = w + v * S + p * p + p;
      wv[ad] = cmul(uu, ph);
      if (ad) wv[-ad] = cmul(uu, cconj(ph));
    }
    __syncthreads();

    if (!DENSE) {
      // all elements of the chunk's pairs in one list, so that the lanes stay full
      // at small lMax (36 dot products of A and 36 of B at lMax 2)
      const int nAB = T.nA + T.nB;
      for (int t = tid; t < vc * nAB; t += kAThreads) {
        const int v = t / nAB, kk = t - v * nAB, which = kk >= T.nA, k = which ? kk - T.nA : kk;
        const PairInfo inf = info[v];
        if (!inf.valid || inf.diag) continue;
        const int nk = which ? T.nB : T.nA, c = which ? T.cntB[k] : T.cntA[k];
        const double *coef = (which ? T.coefB : T.coefA) + k;
        const uint16_t *slot = (which ? T.slotB : T.slotA) + k;
        const qg_c *wv = w + v * S;
        double sr = 0, si = 0;
        for (int q = 0; q < c; ++q) {
          const double cf = __ldg(coef + q * nk);
          const qg_c x = wv[__ldg(slot + q * nk)];
          sr = fma(cf, x.re, sr);
          si = fma(cf, x.im, si);
        }
        qg_c val = which ? cmk(xor_sign(si, kSignBit), sr) : cmk(sr, si);  // B multipliers are imaginary
        const uint32_t pr = __ldg((which ? T.pairB : T.pairA) + k);
        qg_c *M = a.M + (size_t)inf.w * N * N;
        const size_t row0 = (size_t)inf.R * NB, col0 = (size_t)inf.C * NB;
        const qg_c *TR = a.T + ((size_t)inf.w * a.ntm + a.tmid[inf.R]) * NB;
        const qg_c *TC = a.T + ((size_t)inf.w * a.ntm + a.tmid[inf.C]) * NB;
        const int ends = pair_second(pr) == pair_first(pr) ? 1 : 2;
        for (int h = 0; h < ends; ++h) {  // the two elements that share the dot product
          const int e = h ? pair_second(pr) : pair_first(pr);
          if (h && pair_negated(pr)) val = cmk(xor_sign(val.re, kSignBit), xor_sign(val.im, kSignBit));
          const int yi = e / NE, yj = e - yi * NE;
          // A: (E <- E) and (M <- M) blocks; B: (E <- M) and (M <- E) blocks
          const int r1 = yi, c1 = which ? NE + yj : yj;
          const int r2 = NE + yi, c2 = which ? yj : NE + yj;
          M[(row0 + r1) * N + col0 + c1] = cmul_neg(TR[r1], val);
          M[(row0 + r2) * N + col0 + c2] = cmul_neg(TR[r2], val);
          // (C, R): the opposite translation flips the waves of odd order,
          // S(C <- R) = (-1)^(n + nu) A, -(-1)^(n + nu) B
          const unsigned long long odd = ((ydeg(yi) + ydeg(yj) + which) & 1) ? kSignBit : 0ull;
          const qg_c u = cmk(xor_sign(val.re, odd), xor_sign(val.im, odd));
          M[(col0 + r1) * N + row0 + c1] = cmul_neg(TC[r1], u);
          M[(col0 + r2) * N + row0 + c2] = cmul_neg(TC[r2], u);
        }
      }
    }
    for (int v = 0; v < vc; ++v) {
      const PairInfo inf = info[v];
      if (!inf.valid) break;
      qg_c *M = a.M + (size_t)inf.w * N * N;
      const size_t row0 = (size_t)inf.R * NB, col0 = (size_t)inf.C * NB;
      if (inf.diag) {
        for (int t = tid; t < NB * NB; t += kAThreads) {
          const int i = t / NB, j = t - i * NB;
          M[(row0 + i) * N + col0 + j] = cmk(i == j ? 1.0 : 0.0, 0.0);
        }
        continue;
      }
      if (!DENSE) continue;
      const qg_c *wv = w + v * S;
      const qg_c *TR = a.T + ((size_t)inf.w * a.ntm + a.tmid[inf.R]) * NB * NB;
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        const uint8_t *cnt = which ? T.cntB : T.cntA;
        const double *coef = which ? T.coefB : T.coefA;
        const uint16_t *slot = which ? T.slotB : T.slotA;
        const uint32_t *pair = which ? T.pairB : T.pairA;
        const int nk = which ? T.nB : T.nA;
        for (int k = tid; k < nk; k += kAThreads) {
          const int c = cnt[k];
          double sr = 0, si = 0;
          for (int q = 0; q < c; ++q) {
            const double cf = __ldg(coef + q * nk + k);
            const qg_c x = wv[__ldg(slot + q * nk + k)];
            sr = fma(cf, x.re, sr);
            si = fma(cf, x.im, si);
          }
          qg_c val = which ? cmk(xor_sign(si, kSignBit), sr) : cmk(sr, si);
          const uint32_t pr = __ldg(pair + k);
          const int ends = pair_second(pr) == pair_first(pr) ? 1 : 2;
          for (int h = 0; h < ends; ++h) {
            const int e = h ? pair_second(pr) : pair_first(pr);
            if (h && pair_negated(pr)) val = cmk(xor_sign(val.re, kSignBit), xor_sign(val.im, kSignBit));
            const int yi = e / NE, yj = e - yi * NE;
            sblk[yi * NB + (which ? NE + yj : yj)] = val;
            sblk[(NE + yi) * NB + (which ? yj : NE + yj)] = val;
          }
        }
      }
      __syncthreads();
      for (int t = tid; t < NB * NB; t += kAThreads) {
        const int i = t / NB, j = t - i * NB;
        double sr = 0, si = 0;
        for (int q = 0; q < NB; ++q) {
          const qg_c tq = TR[i * NB + q], sq = sblk[q * NB + j];
          sr = fma(tq.re, sq.re, fma(-tq.im, sq.im, sr));
          si = fma(tq.re, sq.im, fma(tq.im, sq.re, si));
        }
        M[(row0 + i) * N + col0 + j] = cmk(-sr, -si);
      }
      __syncthreads();
    }
    __syncthreads();
  }
}

template <int LMAX>
int launch_asm(const AsmArgs &a, const TransDevTables &T, cudaStream_t st) {
  using Sh = AsmShape<LMAX>;
  int dev = 0, nsm = 0, per_sm = 0;
  QG_CUDA_TRY(cudaGetDevice(&dev));
  QG_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const size_t np = (size_t)a.np, units = (size_t)a.nw * (a.dense ? np * np : np * (np + 1) / 2);
  if (units == 0) return QPMS_SUCCESS;
  const double nrow = (double)a.np * 2 * LMAX * (LMAX + 2);
  KtScope kt(KT_ASSEMBLE, st, 16.0 * a.nw * nrow * nrow);
  const size_t smem = asm_smem_bytes<LMAX>(a.dense);
  auto run = [&](auto k) -> int {
    QG_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    QG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, Sh::kThreads, smem));
    const size_t resident = (size_t)nsm * std::max(per_sm, 1);
    // few pairs: fewer in a chunk, so that every resident CTA has one
    const int vc = (int)std::min<size_t>(Sh::V, (units + resident - 1) / resident);
    k<<<(unsigned)std::min(resident, (units + vc - 1) / vc), Sh::kThreads, smem, st>>>(a, T, vc);
    return QPMS_SUCCESS;
  };
  const int e = a.dense ? run(assemble_kernel<LMAX, true>) : run(assemble_kernel<LMAX, false>);
  if (e) return e;
  QG_CUDA_TRY(cudaGetLastError());
  g_launches.fetch_add(1);
  return QPMS_SUCCESS;
}

// ---------------- small pipeline kernels ----------------

// a[w][p*n + i] = coef[i] * exp(i kvec_w . r_p)
__global__ void incident_kernel(int nw, int np, int n, const qg_c *coef, size_t coef_stride, const double *kvec,
                                const double *pos, qg_c *a) {
  const size_t N = (size_t)np * n, tot = (size_t)nw * N;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < tot; t += (size_t)gridDim.x * blockDim.x) {
    const int w = (int)(t / N);
    const size_t r = t - (size_t)w * N;
    const int p = (int)(r / n), i = (int)(r - (size_t)p * n);
    const double ph = kvec[3 * w] * pos[3 * p] + kvec[3 * w + 1] * pos[3 * p + 1] + kvec[3 * w + 2] * pos[3 * p + 2];
    double s, c;
    sincos(ph, &s, &c);
    a[t] = cmul(coef[(size_t)w * coef_stride + i], cmk(c, s));
  }
}

// Incidence of the lattice scan, one thread per (frequency w, Bloch vector k):
// the plane wave of in-plane wavevector k and E along x made transverse (x at
// normal incidence), kvec its wavevector, coef its regular-wave coefficients
// (electric, then magnetic; vswf.c:445-467 with the dual harmonics, as
// planewave_coeffs of the host), all zero where the order is evanescent
// (|k| >= Re kappa_w), kk the medium wavenumber.  pi = m P / sin th comes from
// P / sin th's own recurrence and tau = dP/dth from neighbouring orders, so the
// polar axis needs no branch.  4,096 wavevectors took 4 ms on the host.
constexpr int kIncLMax = 6;
struct IncTables {
  double nf[(kIncLMax + 1) * (kIncLMax + 2) / 2];  // sqrt((2l+1)/(4 pi l(l+1)) (l-m)!/(l+m)!)
};

__global__ void __launch_bounds__(128) scan_incidence_kernel(int nw, int nk, int lMax, IncTables tb, const qg_c *kappa,
                                                             const double *beta, qg_c *coef, double *kvec, qg_c *kk) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nw * nk) return;
  const int w = t / nk, ik = t - w * nk, ne = lMax * (lMax + 2);
  const double kap = kappa[w].re, bx = beta[2 * ik], by = beta[2 * ik + 1], b2 = bx * bx + by * by;
  const bool prop = kap * kap > b2;
  const double kz = prop ? sqrt(kap * kap - b2) : 0.0, kn = sqrt(b2 + kz * kz);
  kk[t] = kappa[w];
  kvec[3 * t] = bx;
  kvec[3 * t + 1] = by;
  kvec[3 * t + 2] = kz;
  qg_c *el = coef + (size_t)t * 2 * ne, *mg = el + ne;
  if (!prop) {
    for (int y = 0; y < 2 * ne; ++y) el[y] = cmk(0, 0);
    return;
  }
  const double rho = sqrt(b2), ct = kz / kn, st = rho / kn, cf = rho > 0 ? bx / rho : 1.0, sf = rho > 0 ? by / rho : 0.0;
  const double ux = bx / kn;
  double E[3] = {1.0 - ux * bx / kn, -ux * by / kn, -ux * kz / kn};
  const double En = sqrt(E[0] * E[0] + E[1] * E[1] + E[2] * E[2]);
  const double Et = (E[0] * ct * cf + E[1] * ct * sf - E[2] * st) / En, Ep = (E[1] * cf - E[0] * sf) / En;
  // columns m - 1, m, m + 1 of P_l^m, and P_l^m / sin for m
  double Pm[kIncLMax + 2], P0[kIncLMax + 2], Pp[kIncLMax + 2], R[kIncLMax + 2];
  auto column = [&](int m, double first, double *out) {  // out[l], l = m .. lMax + 1, from its first entry
    double a = 0.0, b = first;
    for (int l = 0; l < m && l <= lMax + 1; ++l) out[l] = 0.0;
    for (int l = m; l <= lMax + 1; ++l) {
      out[l] = b;
      const double nx = ((2 * l + 1) * ct * b - (l + m) * a) / (l + 1 - m);
      a = b;
      b = nx;
    }
  };
  double pmm = 1.0;  // P_m^m
  column(0, 1.0, P0);
  column(1, -st, Pp);
  qg_c em = cmk(1.0, 0.0);  // e^{-i m phi}
  for (int m = 0; m <= lMax; ++m) {
    if (m > 0) {
      for (int l = 0; l <= lMax + 1; ++l) {
        Pm[l] = P0[l];
        P0[l] = Pp[l];
      }
      column(m, m == 1 ? -1.0 : -(2 * m - 1) * pmm, R);  // P / sin: its first entry is -(2m - 1) P_{m-1}^{m-1}
      pmm *= -(2 * m - 1) * st;
      column(m + 1, -(2 * m + 1) * st * pmm, Pp);
      em = cmul(em, cmk(cf, -sf));
    }
    for (int l = m > 1 ? m : 1; l <= lMax; ++l) {
      const double nf = 4 * 3.14159265358979323846 * tb.nf[l * (l + 1) / 2 + m];
      const double pi = m ? nf * m * R[l] : 0.0;
      const double tau = m ? -0.5 * nf * ((l + m) * (l - m + 1) * Pm[l] - Pp[l]) : nf * Pp[l];
      for (int sg = 0; sg < (m ? 2 : 1); ++sg) {
        // order -m: pi (-1)^(m+1), tau (-1)^m, conjugate phase
        const double f = (sg && (m & 1)) ? -1.0 : 1.0, pl = sg ? -f * pi : pi, tl = f * tau;
        const qg_c e = sg ? cconj(em) : em;
        qg_c a = cmul(cmk(-tl * Ep, -pl * Et), e), b = cmul(cmk(-tl * Et, pl * Ep), e);
        // a i^l (magnetic), b i^(l+1) (electric)
        for (int q = 0; q < (l & 3); ++q) a = cmk(-a.im, a.re);
        for (int q = 0; q < ((l + 1) & 3); ++q) b = cmk(-b.im, b.re);
        const int y = l * (l + 1) + (sg ? -m : m) - 1;
        mg[y] = a;
        el[y] = b;
      }
    }
  }
}

// b[w][p*n + i] = sum_j T_w,tm(p)[i][j] a[w][p*n + j]  (diag: T[i] a[i]); tper
// consecutive w share a T
__global__ void apply_t_kernel(int nw, int np, int n, int ntm, int dense, int tper, const int *tmid, const qg_c *T,
                               const qg_c *a, qg_c *b) {
  const size_t N = (size_t)np * n, tot = (size_t)nw * N;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < tot; t += (size_t)gridDim.x * blockDim.x) {
    const int w = (int)(t / N);
    const size_t r = t - (size_t)w * N;
    const int p = (int)(r / n), i = (int)(r - (size_t)p * n);
    const qg_c *Tp = T + ((size_t)(w / tper) * ntm + tmid[p]) * (dense ? (size_t)n * n : n);
    if (!dense) {
      b[t] = cmul(Tp[i], a[t]);
    } else {
      const qg_c *ap = a + (size_t)w * N + (size_t)p * n;
      qg_c s = cmk(0, 0);
      for (int j = 0; j < n; ++j) s = cadd(s, cmul(Tp[i * n + j], ap[j]));
      b[t] = s;
    }
  }
}

// r = b - M x for nw row-major N x N systems; one warp per row.  Also
// accumulates ||r||^2 and ||b||^2 per system (atomics on doubles).
__global__ void residual_kernel(int nw, size_t N, const qg_c *M, const qg_c *x, const qg_c *b, qg_c *r,
                                double *rn2, double *bn2) {
  const int lane = threadIdx.x & 31;
  const size_t warp = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5;
  const size_t nwarps = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t row = warp; row < (size_t)nw * N; row += nwarps) {
    const size_t w = row / N, i = row - w * N;
    const qg_c *Mi = M + w * N * N + i * N;
    const qg_c *xw = x + w * N;
    double sr = 0, si = 0;
    for (size_t j = lane; j < N; j += 32) {
      const qg_c m = Mi[j], xv = xw[j];
      sr = fma(m.re, xv.re, fma(-m.im, xv.im, sr));
      si = fma(m.re, xv.im, fma(m.im, xv.re, si));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, o);
      si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    if (lane == 0) {
      const qg_c bv = b[row];
      const qg_c rv = cmk(bv.re - sr, bv.im - si);
      r[row] = rv;
      atomicAdd(rn2 + w, cabs2(rv));
      atomicAdd(bn2 + w, cabs2(bv));
    }
  }
}

__global__ void c128_to_c64_kernel(size_t n, const qg_c *src, float2 *dst) {
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const qg_c v = src[t];
    dst[t] = make_float2((float)v.re, (float)v.im);
  }
}

// x += dx (complex64 correction), optionally x = dx when init
__global__ void add_c64_kernel(size_t n, const float2 *dx, qg_c *x, int init) {
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const float2 d = dx[t];
    if (init)
      x[t] = cmk(d.x, d.y);
    else
      x[t] = cmk(x[t].re + d.x, x[t].im + d.y);
  }
}

// sigma_w = -Re(a_w^H f_w) / Re(k_w)^2 ; one block per system
__global__ void sigma_ext_kernel(int nw, size_t N, const qg_c *a, const qg_c *f, const qg_c *k, double *sig) {
  __shared__ double red[32];
  const int w = blockIdx.x;
  if (w >= nw) return;
  double s = 0;
  for (size_t i = threadIdx.x; i < N; i += blockDim.x) {
    const qg_c av = a[(size_t)w * N + i], fv = f[(size_t)w * N + i];
    s += av.re * fv.re + av.im * fv.im;  // Re(conj(a) f)
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = (threadIdx.x < blockDim.x / 32) ? red[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) {
      const double kr = k[w].re;
      sig[w] = -s / (kr * kr);
    }
  }
}

// out-of-place transpose of nb square n x n complex128 matrices
__global__ void transpose_kernel(size_t n, int nb, const qg_c *src, qg_c *dst) {
  __shared__ qg_c tile[32][33];
  const int b = blockIdx.z;
  const size_t bx = blockIdx.x * 32, by = blockIdx.y * 32;
  const qg_c *s = src + (size_t)b * n * n;
  qg_c *d = dst + (size_t)b * n * n;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const size_t r = by + j, c = bx + threadIdx.x;
    if (r < n && c < n) tile[j][threadIdx.x] = s[r * n + c];
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const size_t r = bx + j, c = by + threadIdx.x;
    if (r < n && c < n) d[r * n + c] = tile[threadIdx.x][j];
  }
}

unsigned grid_for(size_t n, int threads) {
  size_t g = (n + threads - 1) / threads;
  if (g > 152 * 32) g = 152 * 32;
  if (g == 0) g = 1;
  return (unsigned)g;
}

}  // namespace

int launch_assemble(const AsmArgs &a, const TransDevTables &T, cudaStream_t st) {
  switch (T.lMax) {
#define QG_CASE(LM) \
  case LM: return launch_asm<LM>(a, T, st);
    QG_CASE(1) QG_CASE(2) QG_CASE(3) QG_CASE(4) QG_CASE(5) QG_CASE(6)
#undef QG_CASE
    default: set_error("assembly kernel: lMax %d not compiled (1..6)", T.lMax); return QPMS_EINVAL;
  }
}

int launch_incident(int nw, int np, int n, const qg_c *coef, const double *kvec, const double *pos, qg_c *a,
                    cudaStream_t st, size_t coef_stride) {
  incident_kernel<<<grid_for((size_t)nw * np * n, 256), 256, 0, st>>>(nw, np, n, coef, coef_stride, kvec, pos, a);
  QG_CUDA_TRY(cudaGetLastError());
  g_launches.fetch_add(1);
  return QPMS_SUCCESS;
}

int launch_scan_incidence(int nw, int nk, int lMax, const qg_c *kappa, const double *beta, qg_c *coef, double *kvec,
                          qg_c *kk, cudaStream_t st) {
  if (lMax < 1 || lMax > kIncLMax) {
    set_error("scan incidence: lMax %d", lMax);
    return QPMS_EINVAL;
  }
  IncTables tb;
  for (int l = 0; l <= kIncLMax; ++l)
    for (int m = 0; m <= l; ++m) {
      double f = l ? (2 * l + 1) / (4 * M_PI * l * (l + 1)) : 0.0;
      for (int x = l - m + 1; x <= l + m; ++x) f /= x;
      tb.nf[l * (l + 1) / 2 + m] = sqrt(f);
    }
  scan_incidence_kernel<<<(unsigned)(((size_t)nw * nk + 127) / 128), 128, 0, st>>>(nw, nk, lMax, tb, kappa, beta, coef,
                                                                                   kvec, kk);
  QG_CUDA_TRY(cudaGetLastError());
  g_launches.fetch_add(1);
  return QPMS_SUCCESS;
}

int launch_apply_t(int nw, int np, int n, int ntm, int dense, const int *tmid, const qg_c *T, const qg_c *a,
                   qg_c *b, cudaStream_t st, int tper) {
  apply_t_kernel<<<grid_for((size_t)nw * np * n, 256), 256, 0, st>>>(nw, np, n, ntm, dense, tper, tmid, T, a, b);
  QG_CUDA_TRY(cudaGetLastError());
  g_launches.fetch_add(1);
  return QPMS_SUCCESS;
}

int launch_residual(int nw, size_t N, const qg_c *M, const qg_c *x, const qg_c *b, qg_c *r, double *rn2,
                    double *bn2, cudaStream_t st) {
  QG_CUDA_TRY(cudaMemsetAsync(rn2, 0, sizeof(double) * nw, st));
  QG_CUDA_TRY(cudaMemsetAsync(bn2, 0, sizeof(double) * nw, st));
  residual_kernel<<<grid_for((size_t)nw * N * 32, 256), 256, 0, st>>>(nw, N, M, x, b, r, rn2, bn2);
  QG_CUDA_TRY(cudaGetLastError());
  g_launches.fetch_add(1);
  return QPMS_SUCCESS;
}

int launch_c128_to_c64(size_t n, const qg_c *src, void *dst, cudaStream_t st) {
  c128_to_c64_kernel<<<grid_for(n, 256), 256, 0, st>>>(n, src, (float2 *)dst);
  QG_CUDA_TRY(cudaGetLastError());
  g_launches.fetch_add(1);
  return QPMS_SUCCESS;
}

int launch_add_c64(size_t n, const void *dx, qg_c *x, int init, cudaStream_t st) {
  add_c64_kernel<<<grid_for(n, 256), 256, 0, st>>>(n, (const float2 *)dx, x, init);
  QG_CUDA_TRY(cudaGetLastError());
  g_launches.fetch_add(1);
  return QPMS_SUCCESS;
}

int launch_sigma_ext(int nw, size_t N, const qg_c *a, const qg_c *f, const qg_c *k, double *sig, cudaStream_t st) {
  sigma_ext_kernel<<<nw, 256, 0, st>>>(nw, N, a, f, k, sig);
  QG_CUDA_TRY(cudaGetLastError());
  g_launches.fetch_add(1);
  return QPMS_SUCCESS;
}

int launch_transpose(size_t n, int nb, const qg_c *src, qg_c *dst, cudaStream_t st) {
  dim3 grid((unsigned)((n + 31) / 32), (unsigned)((n + 31) / 32), (unsigned)nb), block(32, 8);
  transpose_kernel<<<grid, block, 0, st>>>(n, nb, src, dst);
  QG_CUDA_TRY(cudaGetLastError());
  g_launches.fetch_add(1);
  return QPMS_SUCCESS;
}

}  // namespace qg
