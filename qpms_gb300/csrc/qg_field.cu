// Scattered-field evaluation of a finite system,
//
//   E(r) = sum_p sum_{l,m} ( f_N[p](l,m) N_lm^{(J)}(k (r - r_p)) + f_M[p](l,m) M_lm^{(J)}(k (r - r_p)) ),
//
// in cartesian components: qpms_scatsys_scattered_E (scatsystem.c:2013-2039),
// i.e. per particle kr = k * cart2sph(where - pos) (vectors.h:134-140), the
// VSWFs of qpms_vswf_fill_csph (vswf.c:230-288) summed with the particle's
// coefficients (qpms_eval_vswf_csph, vswf.c:533-560) and turned to cartesian
// components by csphvec2ccart (vectors.h:272-303).  Default normalisation
// (qpms_types.h:167): Condon-Shortley phase, e^{i m phi}, factors 1.
//
// The sum over the waves of one particle is evaluated through its cartesian
// components.  M_lm = -r x grad(psi_lm) / sqrt(l(l+1)) and N = rot M / k, with
// psi_lm = z_l(kr) Y_lm: the angular momentum and gradient formulas for solid
// waves (e.g. Edmonds, Angular Momentum in Quantum Mechanics, 5.7-5.9) give
//   E_c = sum_{l' <= L+1, m'} C_c(l',m') psi_{l'm'}(k (r - r_p)),   c = x, y, z,
// where C is a fixed sparse linear map of f (three real coefficients per
// entry, FieldTables).  +-m' are paired into real harmonics
//   Q_lm(cos th) Re / Im (u_x + i u_y)^m,  u = (r - r_p) / |r - r_p|,
// Q_lm = P_l^m / sin^m th scaled to be monic, by Q_l = x Q_{l-1} - c Q_{l-2};
// no angle, no pole and no division by sin th appears.  Per pair that is a
// square root, a sine and cosine, two operations per recurrence step and six
// FMAs per real harmonic.
//
// Layout: one thread per evaluation point, all threads of a block walk the
// same particles.  A block maps the f of kTile particles to C in shared memory
// (about 2 % of the arithmetic) and its threads read C as broadcasts.  grid.y
// splits the particle list when the points alone do not fill the GPU; the
// partial sums [split][point][3] are then added in a fixed order by a second
// kernel, so the result does not depend on timing.
//
// Bound: the FP64 pipe (1/64 of the FP32 rate), so the FP64 instructions per
// pair count.  Through spherical components (radial, polar and azimuthal parts
// of N and M per (l, m), a complex product per coefficient) lMax 3 took 790 of
// them and 20.7 ms for 1.6e7 pairs (400 particles, 40,001 points); now 306 and
// 9.1 ms.  Six of them add a particle's field to the sum once all its waves are
// summed (8.9 ms without, with an error 1.03 to 1.06 times as large).
#include <math.h>
#include <string.h>

#include <mutex>
#include <vector>

#include "qg_internal.h"
#include "qg_specfunc.cuh"

namespace qg {
bool scatsys_is_own(const qpms_scatsys_t *ss);
int scatsys_lmax(const qpms_scatsys_t *ss);

namespace {

constexpr int kFieldLMax = 6;  // the systems' largest
constexpr int kFieldThreads = 128;
constexpr int kTile = 8;  // particles whose coefficients are staged together

// C_c(l', m') = -i al f_M(l', m' + d) + bm f_N(l' - 1, m' + d) + bp f_N(l' + 1, m' + d)
// for the components c = + (E_x + i E_y, d = -1), - (E_x - i E_y, d = 1) and z
// (d = 0), index l'(l'+1) + m'.  The scale of the monic harmonics and, for
// m' < 0, the sign of Y_{l',m'} against its conjugate are included.
template <int L>
struct FieldTables {
  double al[3][(L + 2) * (L + 2)], bm[3][(L + 2) * (L + 2)], bp[3][(L + 2) * (L + 2)];
};

template <int L>
struct FieldArgs {
  int npts, np, chunk, J;
  qg_c k, ik;  // wavenumber and its reciprocal
  const double *where;  // [npts][3]
  const double *pos;    // [np][3]
  const qg_c *cvf;      // [np][2 nelem]: electric block, then magnetic
  qg_c *out;            // [split][npts][3]
  FieldTables<L> tb;
};

template <int L>
const FieldTables<L> &field_tables() {
  static FieldTables<L> t;
  static std::once_flag once;
  std::call_once(once, [] {
    typedef long double ld;
    memset(&t, 0, sizeof t);
    auto fact = [](int n) {
      ld f = 1;
      for (int i = 2; i <= n; ++i) f *= i;
      return f;
    };
    // Y_lm = scale(l, m) Q_l|m| (u_x +- i u_y)^|m|
    auto scale = [&](int l, int m) {
      const int am = abs(m);
      const ld s = sqrtl((2 * l + 1) / (4 * 3.14159265358979323846264338327950288L) * fact(l - am) / fact(l + am)) *
                   fact(2 * l) / (powl(2, l) * fact(l) * fact(l - am));
      return (m > 0 && (am & 1)) ? -s : s;
    };
    // grad psi_lm / k: z component -a(l+1,m) psi_{l+1,m} + a(l,m) psi_{l-1,m}, x + iy component
    // g(l,m) psi_{l+1,m+1} + h(l,m) psi_{l-1,m+1}, x - iy component -g(l,-m) psi_{l+1,m-1} - h(l,-m) psi_{l-1,m-1}
    auto aa = [](int l, int m) { return abs(m) > l ? (ld)0 : sqrtl((ld)(l * l - m * m) / (4 * l * l - 1)); };
    auto g = [](int l, int m) { return sqrtl((ld)((l + m + 1) * (l + m + 2)) / ((2 * l + 1) * (2 * l + 3))); };
    auto h = [](int l, int m) { return sqrtl((ld)((l - m) * (l - m - 1)) / ((2 * l - 1) * (2 * l + 1))); };
    for (int l = 1; l <= L; ++l)
      for (int m = -l; m <= l; ++m) {
        const ld s = sqrtl((ld)l * (l + 1));
        const ld m0 = m / s, mp = sqrtl((ld)(l - m) * (l + m + 1)) / s, mm = sqrtl((ld)(l + m) * (l - m + 1)) / s;
        auto put = [&](double *row, int l2, int m2, ld v) {
          if (abs(m2) <= l2) row[l2 * (l2 + 1) + m2] = (double)(v * scale(l2, m2));
        };
        put(t.al[0], l, m + 1, mp);
        put(t.al[1], l, m - 1, mm);
        put(t.al[2], l, m, m0);
        put(t.bm[0], l + 1, m + 1, -mp * aa(l + 1, m + 1) - m0 * g(l, m));
        put(t.bm[1], l + 1, m - 1, mm * aa(l + 1, m - 1) - m0 * g(l, -m));
        put(t.bm[2], l + 1, m, (mp * g(l, -m - 1) + mm * g(l, m - 1)) / 2);
        put(t.bp[0], l - 1, m + 1, mp * aa(l, m + 1) - m0 * h(l, m));
        put(t.bp[1], l - 1, m - 1, -(mm * aa(l, m - 1) + m0 * h(l, -m)));
        put(t.bp[2], l - 1, m, (mp * h(l, -m - 1) + mm * h(l, m - 1)) / 2);
      }
  });
  return t;
}

// Cartesian components (x, y, z) of C(l, m) from one particle's f.
template <int L>
__device__ __forceinline__ void field_coef(const FieldTables<L> &t, const qg_c *f, int l, int m, qg_c C[3]) {
  constexpr int NE = L * (L + 2);
  const int i = l * (l + 1) + m;
  qg_c v[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int m2 = m + (c == 0 ? -1 : c == 1 ? 1 : 0), am = abs(m2);
    v[c] = cmk(0, 0);
    if (l >= 1 && l <= L && am <= l) {
      const qg_c x = f[NE + l * (l + 1) + m2 - 1];
      v[c] = cmk(t.al[c][i] * x.im, -t.al[c][i] * x.re);
    }
    if (l >= 2 && am <= l - 1) {
      const qg_c x = f[(l - 1) * l + m2 - 1];
      v[c] = cmk(fma(t.bm[c][i], x.re, v[c].re), fma(t.bm[c][i], x.im, v[c].im));
    }
    if (l <= L - 1 && am <= l + 1) {
      const qg_c x = f[(l + 1) * (l + 2) + m2 - 1];
      v[c] = cmk(fma(t.bp[c][i], x.re, v[c].re), fma(t.bp[c][i], x.im, v[c].im));
    }
  }
  C[0] = cscale(cadd(v[0], v[1]), 0.5);
  C[1] = cmk(0.5 * (v[0].im - v[1].im), -0.5 * (v[0].re - v[1].re));
  C[2] = v[2];
}

// KIND 0: outgoing waves, real wavenumber; 1: outgoing waves, complex
// wavenumber; 2: any Bessel kind.
template <int L, int KIND>
__global__ void __launch_bounds__(kFieldThreads) scattered_field_kernel(const FieldArgs<L> a) {
  constexpr int LP = L + 1;                           // highest order of the cartesian waves
  constexpr int NH = (LP + 1) * (LP + 1);             // real harmonics
  constexpr int NP = (LP + 1) * (LP + 2) / 2;         // (l, m >= 0)
  constexpr int NE = L * (L + 2);
  // [particle][harmonic][component]; harmonic l^2 is m = 0, l^2 + 2m - 1 and l^2 + 2m the cosine and sine of m
  __shared__ qg_c sC[kTile][NH][3];
  const int q0 = blockIdx.x * kFieldThreads + threadIdx.x;
  const int q = min(q0, a.npts - 1);
  const double wx = a.where[3 * (size_t)q], wy = a.where[3 * (size_t)q + 1], wz = a.where[3 * (size_t)q + 2];
  const int p0 = blockIdx.y * a.chunk;
  const int p1 = min(a.np, p0 + a.chunk);
  qg_c E[3] = {cmk(0, 0), cmk(0, 0), cmk(0, 0)};
  for (int pt = p0; pt < p1; pt += kTile) {
    const int nt = min(kTile, p1 - pt);
    __syncthreads();
    for (int t = threadIdx.x; t < nt * NP; t += kFieldThreads) {
      const int p = t / NP, i = t - p * NP;
      int l = (int)((sqrtf(8.0f * i + 1.0f) - 1.0f) * 0.5f);
      if ((l + 1) * (l + 2) / 2 <= i) ++l;
      if (l * (l + 1) / 2 > i) --l;
      const int m = i - l * (l + 1) / 2;
      const qg_c *f = a.cvf + (size_t)(pt + p) * 2 * NE;
      qg_c Cp[3], Cm[3];
      field_coef<L>(a.tb, f, l, m, Cp);
      if (m) field_coef<L>(a.tb, f, l, -m, Cm);
      for (int c = 0; c < 3; ++c) {
        if (m == 0) {
          sC[p][l * l][c] = Cp[c];
        } else {
          sC[p][l * l + 2 * m - 1][c] = cadd(Cp[c], Cm[c]);
          sC[p][l * l + 2 * m][c] = cmk(Cm[c].im - Cp[c].im, Cp[c].re - Cm[c].re);  // i (Cp - Cm)
        }
      }
    }
    __syncthreads();
    for (int p = 0; p < nt; ++p) {
      const double *pp = a.pos + 3 * (size_t)(pt + p);
      const double dx = wx - __ldg(pp), dy = wy - __ldg(pp + 1), dz = wz - __ldg(pp + 2);
      const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
      const double ir = r2 > 0 ? rsqrt(r2) : 0.0;  // at r = 0 only l = 0 is left of a regular wave
      // one Newton step: the phase k r carries r's error times k r
      const double rs = r2 * ir, r = fma(0.5 * ir, fma(-rs, rs, r2), rs);
      const double ux = dx * ir, uy = dy * ir, ct = dz * ir;
      qg_c z[LP + 1];
      if (KIND == 0) {  // h+_l(x), x real: e^{ix} once, forward recurrence
        const double ri = r2 > 0 ? ir * a.ik.re : __longlong_as_double(0x7ff8000000000000ULL);
        double sn, cs;
        sincos(a.k.re * r, &sn, &cs);
        z[0] = cmk(sn * ri, -cs * ri);
        z[1] = cmk(fma(z[0].re, ri, z[0].im), fma(z[0].im, ri, -z[0].re));
#pragma unroll
        for (int l = 1; l < LP; ++l) {
          const double f = (2 * l + 1) * ri;
          z[l + 1] = cmk(fma(f, z[l].re, -z[l - 1].re), fma(f, z[l].im, -z[l - 1].im));
        }
      } else if (KIND == 1) {
        const double nan = __longlong_as_double(0x7ff8000000000000ULL);
        const qg_c kr = cscale(a.k, r), ri = r2 > 0 ? cscale(a.ik, ir) : cmk(nan, nan);
        const qg_c ex = cexpi(kr);
        const qg_c h0 = cmul(cmk(ex.im, -ex.re), ri);
        const qg_c h1 = cadd(cmul(h0, ri), cmk(h0.im, -h0.re));  // h_1 = h_0 / x - i h_0
        sph_forward<LP>(ri, h0, h1, z);
      } else {
        sph_bessel<LP>(a.J, cscale(a.k, r), z);
      }
      double Q1[LP + 1], Q2[LP + 1], A[LP + 1], B[LP + 1];  // Q_{l-1,m}, Q_{l-2,m}; (u_x + i u_y)^m
      A[0] = 1.0;
      B[0] = 0.0;
      const qg_c(*C)[3] = sC[p];
      qg_c e[3];  // this particle's field: one rounding at the size of the sum per particle
#pragma unroll
      for (int l = 0; l <= LP; ++l) {
        if (l == 1) {
          A[1] = ux;
          B[1] = uy;
        } else if (l > 1) {
          A[l] = fma(A[l - 1], ux, -B[l - 1] * uy);
          B[l] = fma(A[l - 1], uy, B[l - 1] * ux);
        }
        qg_c S[3] = {cmk(0, 0), cmk(0, 0), cmk(0, 0)};
#pragma unroll
        for (int m = 0; m <= l; ++m) {
          double Q;
          if (m == l)
            Q = 1.0;
          else if (m == l - 1)
            Q = ct;
          else
            Q = fma(ct, Q1[m], -((l - 1) * (l - 1) - m * m) / (4.0 * (l - 1) * (l - 1) - 1) * Q2[m]);
          if (m < l) Q2[m] = Q1[m];
          Q1[m] = Q;
          const double R = m == l ? A[m] : (m == 0 ? Q : Q * A[m]);
          const int i = m == 0 ? l * l : l * l + 2 * m - 1;
#pragma unroll
          for (int c = 0; c < 3; ++c) S[c] = cmk(fma(R, C[i][c].re, S[c].re), fma(R, C[i][c].im, S[c].im));
          if (m) {
            const double I = m == l ? B[m] : Q * B[m];
#pragma unroll
            for (int c = 0; c < 3; ++c)
              S[c] = cmk(fma(I, C[i + 1][c].re, S[c].re), fma(I, C[i + 1][c].im, S[c].im));
          }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c)
          e[c] = l ? cmk(fma(-z[l].im, S[c].im, fma(z[l].re, S[c].re, e[c].re)),
                         fma(z[l].im, S[c].re, fma(z[l].re, S[c].im, e[c].im)))
                   : cmul(z[0], S[c]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) E[c] = cadd(E[c], e[c]);
    }
  }
  if (q0 >= a.npts) return;
  qg_c *o = a.out + ((size_t)blockIdx.y * a.npts + q) * 3;
#pragma unroll
  for (int c = 0; c < 3; ++c) o[c] = E[c];
}

// out[q][c] = sum over s of part[s][q][c], s in increasing order.
__global__ void field_reduce_kernel(const qg_c *__restrict__ part, int nsplit, size_t n, qg_c *__restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  qg_c s = part[i];
  for (int j = 1; j < nsplit; ++j) s = cadd(s, part[(size_t)j * n + i]);
  out[i] = s;
}

// What one evaluation needs beside the tables of its lMax.
struct FieldCall {
  int npts, np, J;
  qg_c k;
  const double *where, *pos;
  const qg_c *cvf;
  qg_c *out;
};

template <int L, int KIND>
int run_field(const FieldCall &f, cudaStream_t st) {
  FieldArgs<L> a;
  a.npts = f.npts;
  a.np = f.np;
  a.J = f.J;
  a.k = f.k;
  a.ik = crecip(f.k);
  a.where = f.where;
  a.pos = f.pos;
  a.cvf = f.cvf;
  a.tb = field_tables<L>();
  // Split the particles over grid.y so that the grid fills whole waves of
  // resident blocks (at least two waves), with >= 8 particles per split.
  int dev = 0, nsm = 152, per = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, scattered_field_kernel<L, KIND>, kFieldThreads, 0) !=
          cudaSuccess ||
      per < 1) {
    cudaGetLastError();
    per = 1;
  }
  const long bx = ((long)f.npts + kFieldThreads - 1) / kFieldThreads;
  const long wave = (long)nsm * per;
  const long maxsplit = std::max(1, std::min(a.np / 8, 65535));
  long nsplit = 1;
  double best = 2.0;
  for (long sp = 1; sp <= maxsplit; ++sp) {
    const long tot = bx * sp, waves = (tot + wave - 1) / wave;
    if (waves < 2 && sp < maxsplit) continue;
    const double idle = (double)(waves * wave - tot) / (double)(waves * wave);
    if (idle < best - 0.02) {  // a smaller split unless a larger one idles clearly less
      best = idle;
      nsplit = sp;
    }
    if (tot >= 16 * wave) break;
  }
  a.chunk = (int)((a.np + nsplit - 1) / nsplit);
  nsplit = (a.np + a.chunk - 1) / a.chunk;
  const dim3 grid((unsigned)bx, (unsigned)nsplit);
  if (nsplit == 1) {
    a.out = f.out;
    scattered_field_kernel<L, KIND><<<grid, kFieldThreads, 0, st>>>(a);
    g_launches.fetch_add(1);
    QG_CUDA_TRY(cudaGetLastError());
    return QPMS_SUCCESS;
  }
  qg_c *part = nullptr;
  const size_t n = 3 * (size_t)f.npts;
  QG_CUDA_TRY(cudaMallocAsync(reinterpret_cast<void **>(&part), (size_t)nsplit * n * sizeof(qg_c), st));
  a.out = part;
  scattered_field_kernel<L, KIND><<<grid, kFieldThreads, 0, st>>>(a);
  g_launches.fetch_add(1);
  cudaError_t le = cudaGetLastError();
  if (le == cudaSuccess) {
    field_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(part, (int)nsplit, n, f.out);
    g_launches.fetch_add(1);
    le = cudaGetLastError();
  }
  cudaFreeAsync(part, st);
  QG_CUDA_TRY(le);
  return QPMS_SUCCESS;
}

template <int L>
int run_field_L(const FieldCall &f, cudaStream_t st) {
  if (f.J != 3) return run_field<L, 2>(f, st);
  return f.k.im == 0.0 ? run_field<L, 0>(f, st) : run_field<L, 1>(f, st);
}

// Device positions of a system, uploaded once and kept with it.
struct PosCache {
  std::mutex mu;
  std::vector<std::pair<const qpms_scatsys_t *, std::pair<int, double *>>> v;  // ss -> (device, buffer)
};
PosCache &pos_cache() {
  static PosCache *c = new PosCache;
  return *c;
}

}  // namespace

// Forgets the device positions of a freed system.
void field_forget_system(const qpms_scatsys_t *ss) {
  PosCache &c = pos_cache();
  std::lock_guard<std::mutex> g(c.mu);
  for (size_t i = 0; i < c.v.size();) {
    if (c.v[i].first == ss) {
      int dev = 0;
      cudaGetDevice(&dev);
      cudaSetDevice(c.v[i].second.first);
      cudaFree(c.v[i].second.second);
      cudaSetDevice(dev);
      c.v.erase(c.v.begin() + i);
    } else {
      ++i;
    }
  }
}

namespace {
int device_positions(const qpms_scatsys_t *ss, const double **out) {
  int dev = 0;
  QG_CUDA_TRY(cudaGetDevice(&dev));
  PosCache &c = pos_cache();
  std::lock_guard<std::mutex> g(c.mu);
  for (auto &e : c.v)
    if (e.first == ss && e.second.first == dev) {
      *out = e.second.second;
      return QPMS_SUCCESS;
    }
  std::vector<double> h(3 * (size_t)ss->p_count);
  for (int i = 0; i < ss->p_count; ++i) {
    h[3 * i] = ss->p[i].pos.x;
    h[3 * i + 1] = ss->p[i].pos.y;
    h[3 * i + 2] = ss->p[i].pos.z;
  }
  double *d = nullptr;
  QG_CUDA_TRY(cudaMalloc(&d, h.size() * 8));
  QG_CUDA_TRY(cudaMemcpy(d, h.data(), h.size() * 8, cudaMemcpyHostToDevice));
  c.v.push_back({ss, {dev, d}});
  *out = d;
  return QPMS_SUCCESS;
}

int field_device(const qpms_scatsys_t *ss, int btyp, qg_c k, const qg_c *d_cvf, size_t npoints,
                 const double *d_where, qg_c *d_E, cudaStream_t st) {
  if (!ss || !d_cvf || !d_where || !d_E) { set_error("NULL argument"); return QPMS_EINVAL; }
  if (!scatsys_is_own(ss)) { set_error("system not created by this library"); return QPMS_EINVAL; }
  if (ss->lattice_dimension != 0) {
    set_error("scattered_E: finite systems only (the periodic field needs the lattice sums)");
    return QPMS_EINVAL;
  }
  if (btyp < 1 || btyp > 4) { set_error("scattered_E: Bessel kind %d", btyp); return QPMS_EINVAL; }
  if (npoints == 0) return QPMS_SUCCESS;
  if (npoints > (size_t)(1u << 30)) { set_error("scattered_E: too many points"); return QPMS_EINVAL; }
  const int lMax = scatsys_lmax(ss);
  if (lMax < 1 || lMax > kFieldLMax) { set_error("scattered_E: lMax %d", lMax); return QPMS_EINVAL; }
  const double *d_pos = nullptr;
  int e;
  if ((e = device_positions(ss, &d_pos))) return e;
  const FieldCall f = {(int)npoints, (int)ss->p_count, btyp, k, d_where, d_pos, d_cvf, d_E};
  switch (lMax) {
    case 1: return run_field_L<1>(f, st);
    case 2: return run_field_L<2>(f, st);
    case 3: return run_field_L<3>(f, st);
    case 4: return run_field_L<4>(f, st);
    case 5: return run_field_L<5>(f, st);
    default: return run_field_L<6>(f, st);
  }
}

}  // namespace
}  // namespace qg

using namespace qg;

extern "C" {

int qpms_gpu_scatsys_scattered_E_device(const qpms_scatsys_t *ss, qpms_bessel_t btyp, qpms_complex_t wavenumber,
                                        const qpms_complex_t *d_cvf, size_t npoints, const double *d_where_xyz,
                                        qpms_complex_t *d_E_xyz, void *stream) {
  clear_error();
  qg_c k;
  memcpy(&k, &wavenumber, sizeof k);
  return field_device(ss, btyp, k, reinterpret_cast<const qg_c *>(d_cvf), npoints, d_where_xyz,
                      reinterpret_cast<qg_c *>(d_E_xyz), reinterpret_cast<cudaStream_t>(stream));
}

int qpms_gpu_scatsys_scattered_E(const qpms_scatsys_t *ss, qpms_bessel_t btyp, qpms_complex_t wavenumber,
                                 const qpms_complex_t *cvf, size_t npoints, const double *where_xyz,
                                 qpms_complex_t *E_xyz) {
  clear_error();
  if (!ss || !cvf || !where_xyz || !E_xyz) { set_error("NULL argument"); return QPMS_EINVAL; }
  if (npoints == 0) return QPMS_SUCCESS;
  qg_c k;
  memcpy(&k, &wavenumber, sizeof k);
  const size_t nf = ss->fecv_size;
  cudaStream_t st = nullptr;
  QG_CUDA_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  char *buf = nullptr;
  const size_t bf = nf * 16, bw = (npoints * 24 + 15) / 16 * 16, be = npoints * 48;
  cudaError_t ce = cudaMallocAsync(reinterpret_cast<void **>(&buf), bf + bw + be, st);
  int e = QPMS_SUCCESS;
  if (ce == cudaSuccess) ce = cudaMemcpyAsync(buf, cvf, bf, cudaMemcpyHostToDevice, st);
  if (ce == cudaSuccess) ce = cudaMemcpyAsync(buf + bf, where_xyz, npoints * 24, cudaMemcpyHostToDevice, st);
  if (ce == cudaSuccess) {
    e = field_device(ss, btyp, k, reinterpret_cast<const qg_c *>(buf), npoints,
                     reinterpret_cast<const double *>(buf + bf), reinterpret_cast<qg_c *>(buf + bf + bw), st);
    if (e == QPMS_SUCCESS) ce = cudaMemcpyAsync(E_xyz, buf + bf + bw, be, cudaMemcpyDeviceToHost, st);
  }
  if (buf) cudaFreeAsync(buf, st);
  cudaError_t se = cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  if (e) return e;
  QG_CUDA_TRY(ce);
  QG_CUDA_TRY(se);
  return QPMS_SUCCESS;
}

// Single-point drop-ins (scatsystem.h:715-770).  A failure is reported as a
// NaN field and qpms_gpu_last_error(); the reference aborts instead.
ccart3_t qpms_scatsys_scattered_E(const qpms_scatsys_t *ss, qpms_bessel_t btyp, qpms_complex_t wavenumber,
                                  const qpms_complex_t *cvf, cart3_t where) {
  ccart3_t res;
  const double w[3] = {where.x, where.y, where.z};
  if (qpms_gpu_scatsys_scattered_E(ss, btyp, wavenumber, cvf, 1, w, &res.x)) {
    const double nan = NAN;
    qpms_complex_t c;
    memcpy(&c, &nan, sizeof nan);
    memcpy(reinterpret_cast<char *>(&c) + 8, &nan, sizeof nan);
    res.x = res.y = res.z = c;
  }
  return res;
}

ccart3_t qpms_scatsysw_scattered_E(const qpms_scatsys_at_omega_t *ssw, qpms_bessel_t btyp,
                                   const qpms_complex_t *cvf, cart3_t where) {
  return qpms_scatsys_scattered_E(ssw ? ssw->ss : nullptr, btyp, ssw ? ssw->wavenumber : qpms_complex_t{}, cvf,
                                  where);
}

// The reference's alternative route (translation to electric dipoles at the
// evaluation point, scatsystem.c:2048-2112) evaluates the same field; both
// names run the direct kernel.
ccart3_t qpms_scatsys_scattered_E__alt(const qpms_scatsys_t *ss, qpms_bessel_t btyp, qpms_complex_t wavenumber,
                                       const qpms_complex_t *cvf, cart3_t where) {
  return qpms_scatsys_scattered_E(ss, btyp, wavenumber, cvf, where);
}

ccart3_t qpms_scatsysw_scattered_E__alt(const qpms_scatsys_at_omega_t *ssw, qpms_bessel_t btyp,
                                        const qpms_complex_t *cvf, cart3_t where) {
  return qpms_scatsysw_scattered_E(ssw, btyp, cvf, where);
}

}  // extern "C"
