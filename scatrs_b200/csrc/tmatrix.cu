// The T-matrix of spheroids by the extended boundary condition method on the GPU
// (scatrs/src/tmatrix: kernel.rs for Q and P = RgQ of each azimuthal mode by Gauss-Legendre
// quadrature over the surface, solve.rs for T = -P Q^{-1} with residual refinement,
// kernel.rs:985-1010 for the orientation-averaged cross sections), batched over spheroids
// (geometries) and their modes (jobs) in four kernels:
//
//   tm_geom_kernel     one thread per (spheroid, node): r(theta), 1/r, the normal's
//                      theta-component, the weight factor, s r, and the radial functions
//                      j_n(r), y_n(r), j_n(s r) with their [z z_n]'/z, orders 0..N;
//   tm_angular_kernel  one thread per (mode, node): the normalized d, pi, tau, orders 0..N;
//   tm_series_kernel   one thread per (spheroid, node, order): the power series of y_n(r) and
//                      j_n(s r) with their partial sums (regular.rs);
//   tm_surface_kernel  one thread per (mode, i, k): the surface integrals
//                      J[a][b]_{ik} = sum_nodes w r^2 2 pi n . (A_i x B_k) of the regular
//                      and inner vector spherical wave functions, and the y-part of the outgoing
//                      ones in the cleanest of three exact forms per element of Q;
//   tm_solve_kernel    one block per (mode, parity class): Q^T and -P^T from J, an FP64 LU of Q^T
//                      with partial pivoting, the solve, and residual sweeps X += LU^{-1}
//                      (-P^T - Q^T X) with the residual in double-double; then the mode's
//                      -Re tr T and sum |T|^2.
//
// Everything before the factorization is double-double (dd.cuh): the EBCM's outgoing integrals
// cancel exactly in their singular (electrostatic) terms, by up to 1e16 and more at the sizes
// and aspect ratios of the spheroid workloads (research/tmatrix/README.md, findings 1-3), and
// any pointwise error of the sampled functions or the rule is amplified by that factor.
// The y-part's singular terms are removed as the reference removes them (regular.rs:1-24,
// kernel.rs:468-490): the terms of power <= 0 (or < 0) of each radial product's Laurent series
// integrate to zero over an element, so each element keeps the form without them whose
// magnitude sum is the smallest. Carrying the functions, the Gauss-Legendre rule and the sums
// in about 106 bits leaves the elements accurate to about 1e-32 times what cancellation
// remains; the residual refinement then removes the FP64 factorization's floor (Skeel(Q)
// 2^-53, finding 4), which is what the reference's refinement (solve.rs:249-385) does. The
// vector products of the integrands are the classical ones from the definition (Mishchenko,
// Travis & Lacis 2002, section 5.8; research/tmatrix/ebcm.py).
#include <cuda_runtime.h>

#include <cstdint>

#include "dd.cuh"
#include "kernels.h"

namespace sb {

using ddm::cdd;
using ddm::dd;
using ddm::mkc;
using ddm::mkdd;

namespace {

constexpr int kNodeD = 28;  // doubles per node
constexpr int kRadD = 20;   // doubles per (node, order): j, j', y, y' (dd), w, w', w/(s r) (cdd)
constexpr int kAngD = 6;    // doubles per (node, order): d, pi, tau (dd)
constexpr double kPiHi = 3.141592653589793, kPiLo = 1.2246467991473532e-16;

__device__ __forceinline__ dd ld(const double* p) { return dd{p[0], p[1]}; }
__device__ __forceinline__ void st(double* p, dd v) {
  p[0] = v.hi;
  p[1] = v.lo;
}
__device__ __forceinline__ cdd ldc(const double* p) { return cdd{dd{p[0], p[1]}, dd{p[2], p[3]}}; }
__device__ __forceinline__ void stc(double* p, cdd v) {
  p[0] = v.re.hi;
  p[1] = v.re.lo;
  p[2] = v.im.hi;
  p[3] = v.im.lo;
}

// The largest index i in [0, n) with first(i) <= t (first ascending, first(0) = 0).
template <class F>
__device__ __forceinline__ int owner(int n, int64_t t, F first) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (first(mid) <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

}  // namespace

__global__ void __launch_bounds__(128) tm_geom_kernel(TmArgs a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n_node_total) return;
  const int gi = owner(a.n_geoms, t, [&](int i) { return a.geoms[i].node0; });
  const TmGeom g = a.geoms[gi];
  const int q = (int)(t - g.node0), N = g.N;
  const double* rl = a.rule + 4 * (g.rule + q);
  const dd ct = ld(rl), wq = ld(rl + 2);
  const dd stt = ddm::dd_sqrt(mkdd(1.0) - ct * ct);
  // r(theta) and dr/dtheta of the spheroid with semi-axes a (equatorial) and c (ebcm.py:53-65).
  const dd A = mkdd(g.a), Cc = mkdd(g.c);
  const dd den = Cc * Cc * (stt * stt) + A * A * (ct * ct);
  const dd sden = ddm::dd_sqrt(den);
  const dd r = (A * Cc) / sden;
  const dd dr = -((A * Cc) * (Cc * Cc - A * A) * stt * ct) / (den * sden);
  const dd ir = mkdd(1.0) / r;
  double* ns = a.node + t * kNodeD;
  st(ns + 0, r);
  st(ns + 2, ir);
  const cdd s = mkc(g.s_re, g.s_im);
  const cdd sr = s * r;
  stc(ns + 8, sr);
  st(ns + 12, ct);
  st(ns + 14, stt);
  // The surface integrals' node constants: 2 w r^2 2 pi, that over r^2, nu, nu / r^2, r^2, r^4.
  const dd nu = -(dr * ir), ir2 = ir * ir, fac = (wq * (r * r) * dd{2.0 * kPiHi, 2.0 * kPiLo}) * 2.0;
  const dd r2 = r * r;
  st(ns + 16, fac);
  st(ns + 18, fac * ir2);
  st(ns + 20, nu);
  st(ns + 22, nu * ir2);
  st(ns + 24, r2);
  st(ns + 26, r2 * r2);
  double* f = a.rad + g.rad0 + (int64_t)q * (N + 1) * kRadD;
  // j_n(r): ratios rho_n = j_n / j_{n-1} = r / (2n + 1 - r rho_{n+1}) downward from far above
  // N (kept in the j slots), then values upward from j_0 = sin r / r, j_{-1} = cos r / r;
  // der_n = j_{n-1} - n j_n / r.
  dd sn, cs;
  ddm::dd_sincos(r, &sn, &cs);
  {
    const int start = N + 60 + (int)(2.0 * r.hi);
    dd rho = mkdd(0.0);
    for (int n = start; n >= 1; --n) {
      rho = r / (mkdd(2.0 * n + 1) - r * rho);
      if (n <= N) st(f + n * kRadD + 0, rho);
    }
    dd jm1 = cs * ir, j = sn * ir;
    for (int n = 0; n <= N; ++n) {
      if (n > 0) {
        const dd rn = ld(f + n * kRadD + 0);
        jm1 = j;
        j = rn * j;
      }
      st(f + n * kRadD + 0, j);
      st(f + n * kRadD + 2, jm1 - (j * ir) * (double)n);
    }
  }
  // y_n(r) upward from y_{-1} = sin r / r, y_0 = -cos r / r.
  {
    dd ym1 = sn * ir, y = -(cs * ir);
    for (int n = 0; n <= N; ++n) {
      if (n > 0) {
        const dd yn = (y * ir) * (double)(2 * n - 1) - ym1;
        ym1 = y;
        y = yn;
      }
      st(f + n * kRadD + 4, y);
      st(f + n * kRadD + 6, ym1 - (y * ir) * (double)n);
    }
  }
  // j_n(s r), its derivative term, and j_n(s r) / (s r).
  {
    const cdd isr = ddm::inv(sr);
    const double mag = fmax(fabs(sr.re.hi), fabs(sr.im.hi));
    const int start = N + 60 + (int)(2.0 * mag);
    cdd rho = mkc(0.0);
    for (int n = start; n >= 1; --n) {
      rho = sr * ddm::inv(mkc(2.0 * n + 1) - sr * rho);
      if (n <= N) stc(f + n * kRadD + 8, rho);
    }
    cdd sz, cz;
    ddm::c_sincos(sr, &sz, &cz);
    cdd jm1 = cz * isr, j = sz * isr;
    for (int n = 0; n <= N; ++n) {
      if (n > 0) {
        const cdd rn = ldc(f + n * kRadD + 8);
        jm1 = j;
        j = rn * j;
      }
      const cdd ji = j * isr;
      stc(f + n * kRadD + 8, j);
      stc(f + n * kRadD + 12, jm1 - ji * (double)n);
      stc(f + n * kRadD + 16, ji);
    }
  }
}

// Normalized d_{mn}(theta), pi = m d / sin, tau = dd/dtheta, n = 0..N, m >= 0 (ebcm.py:68-100).
__global__ void __launch_bounds__(128) tm_angular_kernel(TmArgs a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n_ang_total) return;
  const int ji = owner(a.n_jobs, t, [&](int i) { return a.jobs[i].ang_node0; });
  const TmJob jb = a.jobs[ji];
  const TmGeom g = a.geoms[jb.geom];
  const int q = (int)(t - jb.ang_node0), N = g.N, m = jb.m;
  const double* ns = a.node + (g.node0 + q) * kNodeD;
  const dd ct = ld(ns + 12), stt = ld(ns + 14);
  const dd ist = mkdd(1.0) / stt;
  double* f = a.ang + jb.ang0 + (int64_t)q * (N + 1) * kAngD;
  dd am = mkdd(1.0);
  for (int k = 1; k <= m; ++k) am = am * ddm::dd_sqrt(mkdd((double)(2 * k - 1)) / (double)(2 * k));
  dd sp = mkdd(1.0);
  for (int k = 0; k < m; ++k) sp = sp * stt;
  dd dprev = mkdd(0.0), dcur = mkdd(0.0);
  for (int n = 0; n <= N; ++n) {
    dd dn;
    if (n < m) dn = mkdd(0.0);
    else if (n == m) dn = am * sp;
    else if (n == m + 1) dn = ddm::dd_sqrt((double)(2 * m + 1)) * ct * dcur;
    else
      dn = ((ct * dcur) * (double)(2 * n - 1) -
            ddm::dd_sqrt((double)(n - 1) * (n - 1) - (double)m * m) * dprev) /
           ddm::dd_sqrt((double)n * n - (double)m * m);
    dd tau = mkdd(0.0), pi = mkdd(0.0);
    if (n >= (m > 1 ? m : 1)) {
      const dd prev = n - 1 >= m ? dcur : mkdd(0.0);
      tau = ((ct * dn) * (double)n - ddm::dd_sqrt((double)n * n - (double)m * m) * prev) * ist;
      pi = (dn * (double)m) * ist;
    }
    st(f + n * kAngD + 0, dn);
    st(f + n * kAngD + 2, pi);
    st(f + n * kAngD + 4, tau);
    dprev = dcur;
    dcur = dn;
  }
}

namespace {

constexpr int kMaxSeriesTerms = 4000;
// The plain form is kept only when its magnitude sum is below 2^-20 of the regularized forms':
// its integrand comes from the radial functions' recurrences, whose accumulated rounding its
// magnitude sum does not see, while the regularized forms within 2^20 of it still hold about 86
// bits against it. (At x = 25, aspect ratio 0.4 the unbiased choice left the mode-0 T-matrix's
// unitarity at 1e-3 to 1e-2, the biased one at 1e-5; at x = 21 and x = 25, aspect ratio 3,
// 5e-9 became 5e-11 and 1e-10 became 2e-12.)
constexpr double kPlainBias = 0x1p20;
constexpr double kSeriesTol = 0x1p-112;  // a term negligible against the largest at r_max

// The series table of one spheroid (tm_series_slot): j-slots of JS = 30 G + 17 doubles per
// (node h, order n), then the y-table, per (node h, kind c, index l <= G) five fields (the term
// hi, lo, the suffix sum hi, lo, the suffix magnitude sum), each over the orders 0..N.
__device__ __forceinline__ int64_t j_slot_size(int G) { return 30 * (int64_t)G + 17; }
struct JSlot {
  const double* p;
  int G;
  __device__ const double* jk(int c) const { return p + 2 + c * (10 * G + 5); }
};
struct YTab {  // the y-table of one (node, kind)
  const double* p;
  int n1;
  __device__ dd term(int l, int n) const {
    const double* q = p + (int64_t)l * 5 * n1 + n;
    return dd{q[0], q[n1]};
  }
  __device__ double hi(int l, int n) const { return p[(int64_t)l * 5 * n1 + n]; }
  __device__ dd sum(int l, int n) const {
    const double* q = p + ((int64_t)l * 5 + 2) * n1 + n;
    return dd{q[0], q[n1]};
  }
  __device__ double mag(int l, int n) const { return p[((int64_t)l * 5 + 4) * n1 + n]; }
};
__device__ __forceinline__ const double* y_table(const double* ser0, int n_theta, int N, int G,
                                                 int h, int c) {
  const int n1 = N + 1;
  return ser0 + (int64_t)n_theta * n1 * j_slot_size(G) + (int64_t)(h * 3 + c) * (G + 1) * 5 * n1;
}
// The forms table after the y-table: per (node h, column order k, product slot ts < 4) ten
// fields over the row orders 0..N: the form without the powers <= 0 (re hi, lo, im hi, lo), its
// magnitude sum, the form without the powers < 0 (the same five).
__device__ __forceinline__ double* forms_slot(const double* ser0, int n_theta, int N, int G, int h,
                                              int k, int ts) {
  const int64_t n1 = N + 1;
  return const_cast<double*>(ser0) + (int64_t)n_theta * n1 * (j_slot_size(G) + 15 * (int64_t)(G + 1)) +
         (((int64_t)h * n1 + k) * 4 + ts) * 10 * n1;
}

// 1 / y in double-double from one division and its exact remainder, so that a series' terms cost a
// product each instead of a double-double division.
__device__ __forceinline__ dd recip(double y) {
  const double q = 1.0 / y;
  return ddm::fast_two_sum(q, q * fma(-q, y, 1.0));
}

// The number of terms of a series with term ratios x^2 / den(l), l >= 1, until the terms at
// r_max are past their peak (after l_min) and below kSeriesTol of it (regular.rs:97-124, 140-150).
template <class Den>
__device__ int series_length(double x2max, int l_min, Den den) {
  double at = 1.0, peak = 1.0;
  for (int l = 1; l < kMaxSeriesTerms; ++l) {
    const double ratio = x2max / fabs(den(l));
    at *= ratio;
    peak = fmax(peak, at);
    if (l > l_min && ratio < 0.5 && at < kSeriesTol * peak) return l + 1;
  }
  return -1;
}

}  // namespace

// The power series of the radial factors at the nodes of one half of the surface (the
// integrands of the nonzero elements are even in cos theta), one thread per (spheroid, node,
// order n >= 1) (regular.rs:1-31, 155-211, in the unscaled functions of tm_geom_kernel):
//   y_n(r) = sum_l Y_l,      Y_l = a_l r^(2l - n - 1), a_0 = -(2n - 1)!!, a_l = -a_{l-1} / (2l (2l - 2n - 1));
//   j_n(s r) = sum_i t_i,    t_i = b_i (s r)^(n + 2i), b_0 = 1 / (2n + 1)!!, b_i = -b_{i-1} / (2i (2i + 2n + 1));
// with [r y]'/r = sum (2l - n) Y_l / r, y / r = sum Y_l / r, [z j]'/z = sum (n + 2i + 1) t_i / z and
// j / z = sum t_i / z (z = s r). Kept: the y terms l < G with their suffix sums (and the sums of
// their magnitudes) l <= G, the j prefix sums i < G and suffix sums i <= G, G = N/2 + 2, which
// is every index the surface kernel's forms reach. Each suffix sum is accumulated from the
// series' far end (its terms by the backward recurrence), so that it is accurate against its
// own terms.
__global__ void __launch_bounds__(128) tm_series_kernel(TmArgs a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n_ser_total) return;
  const int gi = owner(a.n_geoms, t, [&](int i) { return a.geoms[i].sth0; });
  const TmGeom g = a.geoms[gi];
  const int N = g.N, G = N / 2 + 2;
  const int64_t local = t - g.sth0;
  const int h = (int)(local / N), n = 1 + (int)(local % N);
  const int64_t JS = j_slot_size(G), n1 = N + 1;
  double* p = a.ser + g.ser0 + ((int64_t)h * n1 + n) * JS;
  double* yb[3];
  for (int c = 0; c < 3; ++c)
    yb[c] = const_cast<double*>(y_table(a.ser + g.ser0, g.n_theta, N, G, h, c)) + n;
  const double* ns = a.node + (g.node0 + g.n_theta + h) * kNodeD;
  const dd r = ld(ns), ir = ld(ns + 2);
  const cdd sr = ldc(ns + 8);
  const double xmax = fmax(g.a, g.c), smag2 = g.s_re * g.s_re + g.s_im * g.s_im;
  const int Ly = series_length(xmax * xmax, n, [&](int l) { return 2.0 * l * (2.0 * l - 2.0 * n - 1.0); });
  const int Lj = series_length(xmax * xmax * smag2, 0, [&](int i) { return 2.0 * i * (2.0 * i + 2.0 * n + 1.0); });
  if (Ly < 0 || Lj < 0) {
    atomicOr(a.err, 2u);
    return;
  }
  p[0] = Ly;
  p[1] = Lj;
  double* jb[3];
  for (int c = 0; c < 3; ++c) jb[c] = p + 2 + c * (10 * G + 5);
  // y: the first term, forward to the last, then back with the suffix sums.
  {
    const dd r2 = r * r, ir2 = ir * ir;
    dd v = -ir;
    for (int i = 1; i <= n; ++i) v = (v * (double)(2 * i - 1)) * ir;
    for (int l = 1; l < Ly; ++l) v = -(v * r2) * recip(2.0 * l * (2.0 * l - 2.0 * n - 1.0));
    dd sum[3] = {mkdd(0.0), mkdd(0.0), mkdd(0.0)};
    double mag[3] = {0.0, 0.0, 0.0};
    // The sums past a series shorter than the table (the forms read none further).
    if (Ly <= G)
      for (int c = 0; c < 3; ++c)
        for (int f = 0; f < 5; ++f) yb[c][((int64_t)Ly * 5 + f) * n1] = 0.0;
    for (int l = Ly - 1; l >= 0; --l) {
      const dd over = v * ir;
      const dd term[3] = {v, over * (double)(2 * l - n), over};
      for (int c = 0; c < 3; ++c) {
        sum[c] = sum[c] + term[c];
        mag[c] += fabs(term[c].hi);
        if (l <= G) {
          double* e = yb[c] + (int64_t)l * 5 * n1;
          if (l < G) {
            e[0] = term[c].hi;
            e[n1] = term[c].lo;
          }
          e[2 * n1] = sum[c].hi;
          e[3 * n1] = sum[c].lo;
          e[4 * n1] = mag[c];
        }
      }
      if (l > 0) v = -(v * (2.0 * l * (2.0 * l - 2.0 * n - 1.0))) * ir2;
    }
  }
  // j(s r): the first term, forward with the prefix sums, then back with the suffix sums.
  {
    const cdd sr2 = sr * sr, isr = ddm::inv(sr), isr2 = isr * isr;
    cdd v = mkc(1.0);
    for (int i = 1; i <= n; ++i) {
      v = (v * sr) * recip((double)(2 * i + 1));
    }
    cdd sum[3] = {mkc(0.0), mkc(0.0), mkc(0.0)};
    double mag[3] = {0.0, 0.0, 0.0};
    for (int i = 0; i < Lj; ++i) {
      if (i > 0) {
        v = -(v * sr2) * recip(2.0 * i * (2.0 * i + 2.0 * n + 1.0));
      }
      if (i < G) {
        const cdd over = v * isr;
        const cdd term[3] = {v, over * (double)(n + 2 * i + 1), over};
        for (int c = 0; c < 3; ++c) {
          sum[c] = sum[c] + term[c];
          mag[c] += fabs(term[c].re.hi) + fabs(term[c].im.hi);
          stc(jb[c] + 4 * i, sum[c]);
          jb[c][4 * G + i] = mag[c];
        }
      }
    }
    for (int c = 0; c < 3; ++c) {
      sum[c] = mkc(0.0);
      mag[c] = 0.0;
      if (Lj <= G) {
        stc(jb[c] + 5 * G + 4 * Lj, sum[c]);
        jb[c][9 * G + 4 + Lj] = 0.0;
      }
    }
    for (int i = Lj - 1; i >= 0; --i) {
      const cdd over = v * isr;
      const cdd term[3] = {v, over * (double)(n + 2 * i + 1), over};
      for (int c = 0; c < 3; ++c) {
        sum[c] = sum[c] + term[c];
        mag[c] += fabs(term[c].re.hi) + fabs(term[c].im.hi);
        if (i <= G) {
          stc(jb[c] + 5 * G + 4 * i, sum[c]);
          jb[c][9 * G + 4 + i] = mag[c];
        }
      }
      if (i > 0) v = -((v * isr2) * (2.0 * i * (2.0 * i + 2.0 * n + 1.0)));
    }
  }
}

namespace {

// R+ of one radial product R_t = r^e Y_t(r) J_t(s r) of the y-part at one node: R minus the
// terms of its Laurent series in r of power <= 0 (out[0]) and, with `below`, of power < 0 (out[1]),
// by the series of its higher powers or as R minus the lower ones, whichever adds less in magnitude
// (regular.rs:255-311). yk, jk: the kinds of the y_n and j_k factors (0 f, 1 [z f]'/z, 2 f/z);
// full = R_t at the node, xe = r^e. The magnitudes decide first, in FP64; only the chosen sum runs
// in double-double. The powers of a product are all even, so the two cuts differ by one term of
// each l's series (and by the last l).
__device__ __forceinline__ void reg_forms(const YTab& yt, int Ly, const JSlot& sk, int Lj, int yk,
                                          int jk, int e, int n, int k, bool below, dd xe, cdd full,
                                          cdd out[2], double out_abs[2]) {
  const double* jb = sk.jk(jk);
  const int G = sk.G;
  const int base0 = (-n - 1 - (yk > 0)) + (k - (jk > 0)) + e;
  // Terms l < l_end[c] reach power <= 0 (c = 0) or <= -2 (c = 1); i <= i0 - l - c.
  const int i0 = base0 <= 0 ? -base0 / 2 : -1;
  int l_end[2];
  l_end[0] = min(min(i0 + 1, Ly), G - 1);
  l_end[1] = min(min(max(i0, 0), Ly), G - 1);
  double neg_abs[2] = {0.0, 0.0}, pos_abs[2] = {0.0, 0.0};
#pragma unroll 4
  for (int l = 0; l < l_end[0]; ++l) {
    const double ya = fabs(yt.hi(l, n) * xe.hi);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (c == 1 && (!below || l >= l_end[1])) continue;
      const int i_max = i0 - l - c;
      neg_abs[c] += jb[4 * G + max(min(min(i_max, Lj - 1), G - 1), 0)] * ya;
      pos_abs[c] += jb[9 * G + 4 + min(min(i_max + 1, Lj), G)] * ya;
    }
  }
  bool take_pos[2];
  cdd sum[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (c == 1 && !below) continue;
    pos_abs[c] += jb[9 * G + 4] * yt.mag(l_end[c], n) * fabs(xe.hi);
    const double sub_abs = fabs(full.re.hi) + fabs(full.im.hi) + neg_abs[c];
    take_pos[c] = pos_abs[c] <= sub_abs;
    out_abs[c] = take_pos[c] ? pos_abs[c] : sub_abs;
    sum[c] = mkc(0.0);
  }
  for (int l = 0; l < l_end[0]; ++l) {
    const dd yv = yt.term(l, n) * xe;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (c == 1 && (!below || l >= l_end[1])) continue;
      const int i_max = i0 - l - c;
      const double* j = take_pos[c] ? jb + 5 * G + 4 * min(min(i_max + 1, Lj), G)
                                    : jb + 4 * max(min(min(i_max, Lj - 1), G - 1), 0);
      sum[c] = ddm::add_terms(sum[c], ldc(j) * yv);
    }
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (c == 1 && !below) continue;
    out[c] = take_pos[c]
                 ? ddm::add_terms(sum[c], ldc(jb + 5 * G) * (yt.sum(l_end[c], n) * xe))
                 : ddm::sub_terms(full, sum[c]);
  }
}

// The radial products of an (n, k) pair's nonzero elements, by the parity of n + k, as (y kind,
// j kind, e): even (MN, NM): R_1, R_4, R_6, R_2; odd (MM, NN): R_0, R_3, R_5, R_7.
__device__ __forceinline__ void product_kind(bool even, int ts, int* yk, int* jk, int* e) {
  *yk = (even ? 0x60 : 0x94) >> (2 * ts) & 3;
  *jk = (even ? 0x09 : 0x64) >> (2 * ts) & 3;
  *e = *yk == 2 || *jk == 2 ? 4 : 2;
}

}  // namespace

// The regularized forms of the radial products of the y-part, which do not depend on the
// azimuthal mode: one thread per (spheroid, node of the half surface, product of the pair's nonzero
// elements, row order n != column order k) (the reference computes them once per node before its
// mode loop, kernel.rs:327-342): the form without the powers <= 0 and (|n - k| >= 3) the one
// without those < 0, with their magnitude sums, into the forms table.
//
// Bound by the latency of the sums' loads (a third of the issue slots). The sums run over
// (n - k) / 2 terms, none below the diagonal: with a column's rows side by side and a thread's four
// products one after the other, a warp waited for its longest row with a third of its lanes at work
// and 2.6 warps a scheduler. By bands of diagonals the lanes of a warp run alike, and 4 rows of a
// column keep loads and stores in whole sectors (bands of 1, 2, 4, 8, 16: 80.4, 80.3, 78.6, 84.0,
// 95.3 ms); a product per thread halves the registers; four of the magnitudes' terms are loaded at
// once (78.6 -> 72.5). In all 134 -> 72.5 ms per pass of 288 spheroids to x = 21.
__global__ void __launch_bounds__(128) tm_forms_kernel(TmArgs a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n_forms_total) return;
  const int gi = owner(a.n_geoms, t, [&](int i) { return a.geoms[i].fth0; });
  const TmGeom g = a.geoms[gi];
  const int N = g.N, G = N / 2 + 2, nh = g.n_theta;
  // Node, product and pair: the pairs n > k by bands of kFormsBand diagonals, a column's rows of the
  // band side by side; then those with n < k, column by column.
  const int64_t local = t - g.fth0;
  const int per = forms_threads(N), upper = per - N * (N - 1) / 2;
  const int hs = (int)(local / per), h = hs >> 2, ts = hs & 3;
  int p = (int)(local % per), n, k;
  if (p < upper) {
    int band = 0, len = kFormsBand * (N - 1);
    for (; p >= len; len -= kFormsBand * kFormsBand, ++band) p -= len;
    k = 1 + p / kFormsBand;
    n = k + kFormsBand * band + 1 + p % kFormsBand;
    if (n > N) return;
  } else {
    p -= upper;
    int line = (int)((sqrtf(8.0f * p + 1.0f) - 1.0f) * 0.5f);
    while (line * (line + 1) / 2 > p) --line;
    while ((line + 1) * (line + 2) / 2 <= p) ++line;
    k = line + 2;
    n = 1 + p - line * (line + 1) / 2;
  }
  const int q = nh + h;
  const double* ser = a.ser + g.ser0;
  const int64_t JS = j_slot_size(G);
  const JSlot sk{ser + ((int64_t)h * (N + 1) + k) * JS, G};
  const int Ly = (int)ser[(int64_t)n * JS], Lj = (int)ser[(int64_t)k * JS + 1];
  const double* ns = a.node + (g.node0 + q) * kNodeD;
  const double* ri = a.rad + g.rad0 + ((int64_t)q * (N + 1) + n) * kRadD;
  const double* rk = a.rad + g.rad0 + ((int64_t)q * (N + 1) + k) * kRadD;
  const int n1 = N + 1;
  int yk, jk, e;
  product_kind(((n + k) & 1) == 0, ts, &yk, &jk, &e);
  const dd r = ld(ns), r2 = r * r, xe = e == 2 ? r2 : r2 * r2;
  dd yv = ld(ri + (yk == 1 ? 6 : 4));
  if (yk == 2) yv = yv * ld(ns + 2);
  const cdd full = ldc(rk + 8 + 4 * jk) * (yv * xe);
  double* fs = forms_slot(ser, nh, N, G, h, k, ts) + n;
  const bool below = abs(n - k) >= 3;
  const YTab yt{y_table(ser, nh, N, G, h, yk), N + 1};
  cdd v[2];
  double va[2];
  reg_forms(yt, Ly, sk, Lj, yk, jk, e, n, k, below, xe, full, v, va);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (c == 1 && !below) continue;
    double* f = fs + (int64_t)5 * c * n1;
    f[0] = v[c].re.hi;
    f[n1] = v[c].re.lo;
    f[2 * n1] = v[c].im.hi;
    f[3 * n1] = v[c].im.lo;
    f[4 * n1] = va[c];
  }
}

// The surface integrals of one (mode, i, k) (ebcm.py:103-186, pi -> -pi for the outgoing
// functions' phi-factor convention, g_i g_k taken out of the sum). With z = j_i(r) or
// i y_i(r), zeta = z or [r z]'/r, and the inner w, w' = [s r w]'/(s r), u = w/(s r) at s r, the
// triple products n . (A_i x B_k) are
//   MM = i z w (pi_i tau_k + tau_i pi_k)
//   MN = z w' (pi_i pi_k + tau_i tau_k) - nu k(k+1) z u tau_i d_k
//   NM = -z' w (tau_i tau_k + pi_i pi_k) + nu i(i+1) (z/r) w d_i tau_k
//   NN = i [z' w' (tau_i pi_k + pi_i tau_k) - nu (k(k+1) z' u pi_i d_k + i(i+1) (z/r) w' d_i pi_k)]
// where nu = -r'/r = nu' r^2, nu' = -beta sin cos (1/r^2 = alpha + beta cos^2). MN and NM are even
// in cos theta when i + k is even and odd otherwise, MM and NN the reverse: each (i, k) has two
// nonzero integrals, taken over the half cos theta > 0 of the rule and doubled; the other two
// are exactly zero.
//
// Out: J[0..3] = the regular (z = j) MM, MN, NM, NN; J[4 + 2 bi + bk] = the y-part (z = i y) of
// the element (bi, bk) of Q, -i s J_a - i J_b (tm_solve_kernel's pairs), in the cleanest of its
// three exact forms (kernel.rs:468-490): per type t the radial product R_t = r^e Y_t J_t has
// powers of r whose terms <= 0 integrate, over the element's four types together, to zero when
// i != k, and those < 0 when |i - k| >= 3 (the spheroid's 1/r^2 is a polynomial in cos theta);
// removing them removes the catastrophic cancellation of the plain integrals. The form whose
// magnitude sum is the smallest is kept: the magnitudes are summed first, in FP64, and only the
// chosen form runs in double-double.
//
// Bound by the latency of its loads, the forms table's above all (9 of 13 cycles per issue; L1 43 %,
// FP64 16 % busy). One form instead of three (and no state for the others) halves the operations:
// 196 -> 128 ms per pass of 288 spheroids to x = 21 (3 blocks per SM without spills: the same). Rows of both
// parities of i + k in a warp ran the two parities' code one after the other; one parity at a time:
// 128 -> 98 ms (the table's rows ordered by parity too: no faster, and its writer slower).
namespace {

// One (mode, i, k): its rows of the tables and the half surface's sums.
struct SurfacePair {
  const double* node;  // the first half node's record
  const double* ri;    // radial records of orders i and k at it, and their stride
  const double* rk;
  const double* ai;  // angular records
  const double* ak;
  const double* fs;  // forms of (k, row i)
  int64_t rad_stride, ang_stride, form_stride;
  int n1, nh, i, k;
  double cki, ckk;
  bool even;
};

// The magnitude sums of the two integrals in the three forms (plain, without the powers < 0,
// without those <= 0), with the double-double sums' weights rounded to FP64 (kernel.rs:418-442).
__device__ __forceinline__ void surface_magnitudes(const SurfacePair& P, double m0[3],
                                                   double m1[3]) {
  m0[0] = m0[1] = m0[2] = m1[0] = m1[1] = m1[2] = 0.0;
  const bool below = abs(P.i - P.k) >= 3;
  for (int h = 0; h < P.nh; ++h) {
    const double* ns = P.node + h * kNodeD;
    const double* ri = P.ri + h * P.rad_stride;
    const double* rk = P.rk + h * P.rad_stride;
    const double* ai = P.ai + h * P.ang_stride;
    const double* ak = P.ak + h * P.ang_stride;
    const double* fs = P.fs + h * P.form_stride;
    const double W = ns[18], nup = ns[22], r2 = ns[24], r4 = ns[26], ir = ns[2];
    const double yr = fabs(ri[4]), ydr = fabs(ri[6]), yo = yr * ir;
    const double w = fabs(rk[8]) + fabs(rk[10]), wd = fabs(rk[12]) + fabs(rk[14]),
                 u = fabs(rk[16]) + fabs(rk[18]);
    double c[4], full[4];  // |weight| and |plain product| of the four terms
    if (P.even) {
      const double A2 = fabs(fma(ai[2], ak[2], ai[4] * ak[4]) * W);
      c[0] = c[3] = A2;
      c[1] = fabs(ai[4] * ak[0] * nup * P.ckk * W);
      c[2] = fabs(ai[0] * ak[4] * nup * P.cki * W);
      full[0] = wd * yr * r2;
      full[1] = u * yr * r4;
      full[2] = w * yo * r4;
      full[3] = w * ydr * r2;
    } else {
      const double A1 = fabs(fma(ai[2], ak[4], ai[4] * ak[2]) * W);
      c[0] = c[1] = A1;
      c[2] = fabs(ai[2] * ak[0] * nup * P.ckk * W);
      c[3] = fabs(ai[0] * ak[2] * nup * P.cki * W);
      full[0] = w * yr * r2;
      full[1] = wd * ydr * r2;
      full[2] = u * ydr * r4;
      full[3] = wd * yo * r4;
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const double f2 = fs[(int64_t)(10 * t + 4) * P.n1];
      const double f1 = below ? fs[(int64_t)(10 * t + 9) * P.n1] : 0.0;
      // Terms 0 and 1 (even) or 0 (odd) are the first integral's.
      double* m = (P.even ? t < 2 : t < 1) ? m0 : m1;
      m[0] = fma(c[t], full[t], m[0]);
      m[1] = fma(c[t], f1, m[1]);
      m[2] = fma(c[t], f2, m[2]);
    }
  }
}

// The two integrals of the y-part in one form (0 plain, 1, 2) and, with kRegular, the regular
// ones.
template <bool kRegular>
__device__ __forceinline__ void surface_sums(const SurfacePair& P, int form, cdd& Y0, cdd& Y1,
                                             cdd& R0, cdd& R1) {
  Y0 = Y1 = mkc(0.0);
  if (kRegular) R0 = R1 = mkc(0.0);
  const int n1 = P.n1;
  for (int h = 0; h < P.nh; ++h) {
    const double* ns = P.node + h * kNodeD;
    const double* ri = P.ri + h * P.rad_stride;
    const double* rk = P.rk + h * P.rad_stride;
    const double* ai = P.ai + h * P.ang_stride;
    const double* ak = P.ak + h * P.ang_stride;
    const double* fs = P.fs + h * P.form_stride + (form == 1 ? (int64_t)5 * n1 : 0);
    const dd ir = ld(ns + 2), W = ld(ns + 18), nup = ld(ns + 22);
    const dd di = ld(ai), pii = ld(ai + 2), ti = ld(ai + 4);
    const dd dk = ld(ak), pik = ld(ak + 2), tk = ld(ak + 4);
    // One term: the form's value at the node times alpha W, times i where im.
    auto add = [&](cdd& sum, int t, dd alpha, bool im, cdd plain) {
      cdd v = plain;
      if (form != 0) {
        const double* f = fs + (int64_t)10 * t * n1;
        v = cdd{dd{f[0], f[n1]}, dd{f[2 * n1], f[3 * n1]}};
      }
      const cdd x = v * (alpha * W);
      sum = ddm::add_terms(sum, im ? ddm::times_i(x) : x);
    };
    auto product = [&](int at, dd y, dd xe) {  // the plain product; unused in the other forms
      return form == 0 ? ldc(rk + at) * (y * xe) : mkc(0.0);
    };
    dd yr{}, ydr{}, yo{}, r2{}, r4{};
    if (form == 0) {
      yr = ld(ri + 4);
      ydr = ld(ri + 6);
      yo = yr * ir;
      r2 = ld(ns + 24);
      r4 = ld(ns + 26);
    }
    if (P.even) {
      const dd A2 = ddm::add_terms(pii * pik, ti * tk), A3 = ti * dk, A4 = di * tk;
      if (kRegular) {
        // MN = j w' A2 - nu k(k+1) j u A3, NM = nu i(i+1) (j/r) w A4 - j' w A2.
        const cdd w = ldc(rk + 8), wd = ldc(rk + 12), u = ldc(rk + 16);
        const dd jr = ld(ri), jdr = ld(ri + 2), nu = ld(ns + 20), fac = ld(ns + 16);
        const cdd mn = ddm::sub_terms(wd * (jr * A2), u * ((jr * A3) * (nu * P.ckk)));
        const cdd nm = ddm::sub_terms(w * (((jr * ir) * A4) * (nu * P.cki)), w * (jdr * A2));
        R0 = ddm::add_terms(R0, mn * fac);
        R1 = ddm::add_terms(R1, nm * fac);
      }
      // MN = i A2 R_1 - i k(k+1) A3 nu' R_4, NM = i i(i+1) A4 nu' R_6 - i A2 R_2.
      add(Y0, 0, A2, true, product(12, yr, r2));
      add(Y0, 1, -((A3 * nup) * P.ckk), true, product(16, yr, r4));
      add(Y1, 2, (A4 * nup) * P.cki, true, product(8, yo, r4));
      add(Y1, 3, -A2, true, product(8, ydr, r2));
    } else {
      const dd A1 = ddm::add_terms(pii * tk, ti * pik), A5 = pii * dk, A6 = di * pik;
      if (kRegular) {
        // MM = i j w A1, NN = i [j' w' A1 - nu (k(k+1) j' u A5 + i(i+1) (j/r) w' A6)].
        const cdd w = ldc(rk + 8), wd = ldc(rk + 12), u = ldc(rk + 16);
        const dd jr = ld(ri), jdr = ld(ri + 2), nu = ld(ns + 20), fac = ld(ns + 16);
        const cdd mm = ddm::times_i(w * (jr * A1));
        const cdd nn = ddm::times_i(ddm::sub_terms(
            wd * (jdr * A1), ddm::add_terms(u * ((jdr * A5) * P.ckk),
                                            wd * (((jr * ir) * A6) * P.cki)) * nu));
        R0 = ddm::add_terms(R0, mm * fac);
        R1 = ddm::add_terms(R1, nn * fac);
      }
      // MM = -A1 R_0, NN = -A1 R_3 + k(k+1) A5 nu' R_5 + i(i+1) A6 nu' R_7.
      add(Y0, 0, -A1, false, product(8, yr, r2));
      add(Y1, 1, -A1, false, product(12, ydr, r2));
      add(Y1, 2, (A5 * nup) * P.ckk, false, product(16, ydr, r4));
      add(Y1, 3, (A6 * nup) * P.cki, false, product(12, yo, r4));
    }
  }
}

}  // namespace

__global__ void __launch_bounds__(128, 4) tm_surface_kernel(TmArgs a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n_pair_total) return;
  const int ji = owner(a.n_jobs, t, [&](int i) { return a.jobs[i].pair0; });
  const TmJob jb = a.jobs[ji];
  const TmGeom g = a.geoms[jb.geom];
  const int N = g.N, m = jb.m, n0 = m > 1 ? m : 1, K = jb.K;
  // The pairs of even i + k, then those of odd, rows fastest: a warp's threads run one parity's
  // code, mostly share the column order k and read the forms table's consecutive rows.
  const int half = (K + 1) >> 1, pr = (int)(t - jb.pair0), cls = pr >= half * K;
  const int col = pr / half - cls * K, row = 2 * (pr % half) + ((col + cls) & 1);
  if (row >= K) return;
  const int i = n0 + row, k = n0 + col;
  const int G = N / 2 + 2, nh = g.n_theta;
  SurfacePair P;
  P.node = a.node + (g.node0 + nh) * kNodeD;
  P.rad_stride = (int64_t)(N + 1) * kRadD;
  P.ri = a.rad + g.rad0 + nh * P.rad_stride + i * kRadD;
  P.rk = a.rad + g.rad0 + nh * P.rad_stride + k * kRadD;
  P.ang_stride = (int64_t)(N + 1) * kAngD;
  P.ai = a.ang + jb.ang0 + nh * P.ang_stride + i * kAngD;
  P.ak = a.ang + jb.ang0 + nh * P.ang_stride + k * kAngD;
  P.fs = forms_slot(a.ser + g.ser0, nh, N, G, 0, k, 0) + i;
  P.form_stride = (int64_t)(N + 1) * 40 * (N + 1);
  P.n1 = N + 1;
  P.nh = nh;
  P.i = i;
  P.k = k;
  P.cki = (double)i * (i + 1);
  P.ckk = (double)k * (k + 1);
  P.even = ((i + k) & 1) == 0;
  // The forms of the two elements of Q this (i, k) feeds: the cleanest, or the one asked for.
  const double sa = fabs(g.s_re) + fabs(g.s_im);
  int best[2] = {0, 0};
  if (a.form >= 0) {
    if (a.form == 2 && i != k) best[0] = best[1] = 2;
    if (a.form == 1 && abs(i - k) >= 3) best[0] = best[1] = 1;
  } else if (i != k) {
    double m0[3], m1[3];
    surface_magnitudes(P, m0, m1);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const double* first = e ? m1 : m0;
      const double* second = e ? m0 : m1;
      const double of2 = sa * first[2] + second[2];
      double mb = kPlainBias * (sa * first[0] + second[0]);
      if (of2 < mb) {
        best[e] = 2;
        mb = of2;
      }
      if (abs(i - k) >= 3 && sa * first[1] + second[1] < mb) best[e] = 1;
    }
  }
  // g_i g_k = sqrt((2i+1)(2k+1) / (16 pi^2 i(i+1) k(k+1))).
  const dd pi2 = dd{kPiHi, kPiLo} * dd{kPiHi, kPiLo};
  const dd gg = ddm::dd_sqrt((mkdd((double)(2 * i + 1) * (2 * k + 1)) / (pi2 * 16.0)) /
                             (P.cki * P.ckk));
  // With s on the first of their pair: even: (0, 0) = -i s MN - i NM, (1, 1) = -i s NM - i MN;
  // odd: (0, 1) = -i s MM - i NN, (1, 0) = -i s NN - i MM.
  const cdd s = mkc(g.s_re, g.s_im), mis = -ddm::times_i(s);
  auto element = [&](cdd first, cdd second) {
    return ddm::add_terms(mis * first, ddm::times_i(second) * -1.0) * gg;
  };
  double* o = a.J + 4 * jb.J0;
  const int64_t KK = (int64_t)K * K, e = (int64_t)(i - n0) * K + (k - n0);
  // The places J[0..3] of the regular integrals and J[4..7] of the elements; the others are zero
  // (and not read: the solve takes the two parity classes apart).
  const int c0 = P.even ? 1 : 0, c1 = P.even ? 2 : 3, e0 = P.even ? 4 : 5, e1 = P.even ? 7 : 6;
  cdd Y0, Y1, R0, R1;
  surface_sums<true>(P, best[0], Y0, Y1, R0, R1);
  stc(o + 4 * (c0 * KK + e), R0 * gg);
  stc(o + 4 * (c1 * KK + e), R1 * gg);
  stc(o + 4 * (e0 * KK + e), element(Y0, Y1));
  if (best[1] != best[0]) surface_sums<false>(P, best[1], Y0, Y1, R0, R1);
  stc(o + 4 * (e1 * KK + e), element(Y1, Y0));
}
namespace {

struct Cd {  // complex double
  double re, im;
};
__device__ __forceinline__ Cd cmul(Cd a, Cd b) {
  return Cd{fma(a.re, b.re, -(a.im * b.im)), fma(a.re, b.im, a.im * b.re)};
}
// a - b c.
__device__ __forceinline__ Cd cfms(Cd a, Cd b, Cd c) {
  return Cd{fma(b.im, c.im, fma(-b.re, c.re, a.re)), fma(-b.im, c.re, fma(-b.re, c.im, a.im))};
}
__device__ __forceinline__ Cd crecip(Cd b) {
  const double s = fmax(fabs(b.re), fabs(b.im));
  const Cd bs{b.re / s, b.im / s};
  const double d = (bs.re * bs.re + bs.im * bs.im) * s;
  return Cd{bs.re / d, -(bs.im / d)};
}

constexpr int kSolveThreads = 256, kSolveWarps = kSolveThreads / 32;

__device__ __forceinline__ double warp_max(double v) {
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// Y := U^-1 L^-1 Y (rows already permuted) on this warp's columns: 4 columns at a time, 8 lanes
// over the rows, right-looking, so that a step is one multiply-subtract per row and no warp waits
// for another.
__device__ __forceinline__ void solve_columns(const Cd* A, const Cd* dinv, Cd* Y, int K, int warp,
                                              int lane) {
  const int rl = lane >> 2, cl = lane & 3;
  for (int c0 = 4 * warp; c0 < K; c0 += 4 * kSolveWarps) {
    const int c = c0 + cl;
    const bool on = c < K;
    for (int k = 0; k + 1 < K; ++k) {
      if (on) {
        const Cd y = Y[(int64_t)k * K + c];
        for (int r = k + 1 + rl; r < K; r += 8) {
          const int64_t at = (int64_t)r * K + c;
          Y[at] = cfms(Y[at], A[(int64_t)r * K + k], y);
        }
      }
      __syncwarp();
    }
    for (int k = K - 1; k >= 0; --k) {
      Cd y{0.0, 0.0};
      if (on) {
        y = cmul(Y[(int64_t)k * K + c], dinv[k]);
        for (int r = rl; r < k; r += 8) {
          const int64_t at = (int64_t)r * K + c;
          Y[at] = cfms(Y[at], A[(int64_t)r * K + k], y);
        }
      }
      __syncwarp();
      if (on && rl == 0) Y[(int64_t)k * K + c] = y;
    }
    __syncwarp();
  }
}

}  // namespace

// One block per (mode, parity class). Q and P couple (element 0 or 1, order i) only with (element,
// order) of the same parity of element + order (the surface integrals of the others are exactly
// zero: the spheroid's mirror symmetry), so the 2K x 2K system is two of K unknowns: a quarter of
// the operations and half the storage of the whole. Workspace per class (doubles): Q^T and -P^T as
// complex double-double (4 K^2 each), X (2 K^2), and A and Y (2 K^2 each) where they do not fit
// shared memory. kWhere: 0 the factors A and the right-hand sides Y in shared memory, 1 the
// factors, 2 neither.
//
// Bound by the latency of a step's dependent reads: a factorization step is a pivot search that
// every warp does by itself (no exchange), one barrier, the rank-1 update, one barrier; the
// triangular solves need no block barrier (solve_columns). Against the undivided system in global
// memory with a column per thread (ten barriers a step): 366 -> 109 ms per pass of
// 288 spheroids to x = 21.
template <int kWhere>
__global__ void __launch_bounds__(kSolveThreads) tm_solve_kernel(TmArgs a, const int* list) {
  extern __shared__ __align__(16) unsigned char solve_raw[];
  __shared__ double red[3][kSolveWarps];
  const int job = list[blockIdx.x >> 1], p = blockIdx.x & 1;
  const TmJob jb = a.jobs[job];
  const TmGeom g = a.geoms[jb.geom];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int K = jb.K;
  const int64_t KK = (int64_t)K * K;
  const double* J = a.J + 4 * jb.J0;
  double* Qd = a.work + jb.W0 + p * 14 * KK;  // Q^T, dd complex
  double* Bd = Qd + 4 * KK;                   // -P^T, dd complex
  Cd* X = reinterpret_cast<Cd*>(Bd + 4 * KK);
  // Shared: the class's inverse pivots, a column of L, the row order; then A and Y.
  Cd* dinv = reinterpret_cast<Cd*>(solve_raw);
  Cd* lcol = dinv + K;
  int* perm = reinterpret_cast<int*>(lcol + K);   // factored row -> row
  int* place = perm + K;                          // row -> factored row
  Cd* sh = reinterpret_cast<Cd*>(place + K + (K & 1) * 2);
  Cd* A = kWhere < 2 ? sh : X + KK;
  Cd* Y = kWhere < 1 ? sh + KK : X + 2 * KK;
  // Unknown u of the class: element 0's orders of parity p, then element 1's of the other.
  const int n_a = (K + 1 - p) / 2;
  auto element = [&](int u) { return u >= n_a; };
  auto order = [&](int u) { return u < n_a ? 2 * u + p : 2 * (u - n_a) + 1 - p; };
  const cdd s = mkc(g.s_re, g.s_im);
  const cdd mis = -ddm::times_i(s), mi = mkc(0.0, -1.0);
  auto Jv = [&](int o, int q, int b, int64_t e) { return ldc(J + 4 * (((o * 2 + q) * 2 + b) * KK + e)); };
  // RgQ11 = -i s J12 - i J21, RgQ12 = -i s J11 - i J22, RgQ21 = -i s J22 - i J11,
  // RgQ22 = -i s J21 - i J12 (ebcm.py:189-195) of the regular J, and Q = RgQ + its y-part
  // (tm_surface_kernel); element (row, col) of Q goes to (col, row).
  for (int64_t idx = t; idx < KK; idx += kSolveThreads) {
    const int row = (int)(idx / K), col = (int)(idx % K);
    const int bi = element(row), bk = element(col);
    const int64_t e = (int64_t)order(row) * K + order(col);
    cdd q0;
    if (!bi && !bk) q0 = mis * Jv(0, 0, 1, e) + mi * Jv(0, 1, 0, e);
    else if (!bi && bk) q0 = mis * Jv(0, 0, 0, e) + mi * Jv(0, 1, 1, e);
    else if (bi && !bk) q0 = mis * Jv(0, 1, 1, e) + mi * Jv(0, 0, 0, e);
    else q0 = mis * Jv(0, 1, 0, e) + mi * Jv(0, 0, 1, e);
    const cdd q1 = q0 + Jv(1, bi, bk, e);
    const int64_t tr = (int64_t)col * K + row;
    stc(Qd + 4 * tr, q1);
    stc(Bd + 4 * tr, -q0);
    A[tr] = Cd{q1.re.hi + q1.re.lo, q1.im.hi + q1.im.lo};
  }
  __syncthreads();
  // Each equation scaled by the power of two that brings its largest coefficient to [1, 2):
  // the unscaled radial functions give the rows magnitudes over hundreds of decades, and
  // partial pivoting is only as good as the rows' balance. Exact, and the solution is unchanged.
  for (int r = warp; r < K; r += kSolveWarps) {
    double mx = 0.0;
    for (int c = lane; c < K; c += 32) {
      const Cd v = A[(int64_t)r * K + c];
      mx = fmax(mx, fmax(fabs(v.re), fabs(v.im)));
    }
    mx = warp_max(mx);
    if (lane == 0) perm[r] = r;
    if (!(mx > 0.0) || !isfinite(mx)) continue;
    const int e = -ilogb(mx);
    for (int c = lane; c < K; c += 32) {
      const int64_t idx = (int64_t)r * K + c;
      A[idx] = Cd{ldexp(A[idx].re, e), ldexp(A[idx].im, e)};
      for (int q = 0; q < 4; ++q) {
        Qd[4 * idx + q] = ldexp(Qd[4 * idx + q], e);
        Bd[4 * idx + q] = ldexp(Bd[4 * idx + q], e);
      }
    }
  }
  __syncthreads();
  // LU of A with partial pivoting (the largest modulus, the first row on ties).
  for (int kk = 0; kk < K; ++kk) {
    double best = -1.0;
    int at = kk;
    for (int r = kk + lane; r < K; r += 32) {
      const Cd v = A[(int64_t)r * K + kk];
      const double mag = v.re * v.re + v.im * v.im;
      if (mag > best) {
        best = mag;
        at = r;
      }
    }
    for (int off = 16; off > 0; off >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, off);
      const int oa = __shfl_xor_sync(0xffffffffu, at, off);
      if (ob > best || (ob == best && oa < at)) {
        best = ob;
        at = oa;
      }
    }
    if (!(best > 0.0)) {  // the same in every warp
      if (t == 0) atomicExch(a.err, 1u);
      return;
    }
    const Cd inv = crecip(A[(int64_t)at * K + kk]);
    // Column kk itself is rewritten after the barrier, so that a warp still searching reads it
    // whole.
    for (int r = kk + 1 + t; r < K; r += kSolveThreads)
      lcol[r] = cmul(A[(int64_t)(r == at ? kk : r) * K + kk], inv);
    const Cd pivot = A[(int64_t)at * K + kk];
    if (at != kk)
      for (int c = t; c < K; c += kSolveThreads)
        if (c != kk) {
          const Cd x = A[(int64_t)kk * K + c];
          A[(int64_t)kk * K + c] = A[(int64_t)at * K + c];
          A[(int64_t)at * K + c] = x;
        }
    __syncthreads();
    if (t == 0) {
      dinv[kk] = inv;
      A[(int64_t)kk * K + kk] = pivot;
      const int x = perm[kk];
      perm[kk] = perm[at];
      perm[at] = x;
    }
    for (int c = kk + lane; c < K; c += 32) {
      const Cd u = A[(int64_t)kk * K + c];
      for (int r = kk + 1 + warp; r < K; r += kSolveWarps) {
        const int64_t idx = (int64_t)r * K + c;
        A[idx] = c == kk ? lcol[r] : cfms(A[idx], lcol[r], u);
      }
    }
    __syncthreads();
  }
  for (int r = t; r < K; r += kSolveThreads) place[perm[r]] = r;
  __syncthreads();
  for (int64_t idx = t; idx < KK; idx += kSolveThreads) {
    const int r = (int)(idx / K), c = (int)(idx % K);
    const double* b = Bd + 4 * idx;
    Y[(int64_t)place[r] * K + c] = Cd{b[0] + b[1], b[2] + b[3]};
  }
  __syncthreads();
  solve_columns(A, dinv, Y, K, warp, lane);
  __syncthreads();
  for (int64_t idx = t; idx < KK; idx += kSolveThreads) X[idx] = Y[idx];
  __syncthreads();
  // Residual sweeps: R = -P^T - Q^T X, every product exact and the sums compensated (about
  // 2^-106 of |Q^T| |X|, as mixed-precision refinement needs), four rows at a time per thread.
  double rel = 0.0;
  for (int sweep = 0; sweep < a.max_sweeps; ++sweep) {
    for (int i0 = 4 * warp; i0 < K; i0 += 4 * kSolveWarps)
      for (int c = lane; c < K; c += 32) {
        double sr[4], si[4], er[4], ei[4];  // the sums and their errors
        const double* q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = min(i0 + i, K - 1);
          const double* b = Bd + 4 * ((int64_t)row * K + c);
          sr[i] = b[0];
          er[i] = b[1];
          si[i] = b[2];
          ei[i] = b[3];
          q[i] = Qd + 4 * (int64_t)row * K;
        }
        for (int j = 0; j < K; ++j) {
          const Cd x = X[(int64_t)j * K + c];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const double2 re = *reinterpret_cast<const double2*>(q[i] + 4 * j);
            const double2 im = *reinterpret_cast<const double2*>(q[i] + 4 * j + 2);
            auto sub = [](double& sum, double& err, double hi, double lo, double v) {
              const double h = hi * v;
              const dd w = ddm::two_sum(sum, -h);
              sum = w.hi;
              err += w.lo - fma(lo, v, fma(hi, v, -h));
            };
            sub(sr[i], er[i], re.x, re.y, x.re);
            sub(sr[i], er[i], im.x, im.y, -x.im);
            sub(si[i], ei[i], re.x, re.y, x.im);
            sub(si[i], ei[i], im.x, im.y, x.re);
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i0 + i < K)
            Y[(int64_t)place[i0 + i] * K + c] = Cd{sr[i] + er[i], si[i] + ei[i]};
      }
    __syncthreads();
    solve_columns(A, dinv, Y, K, warp, lane);
    __syncthreads();
    double xm = 0.0, rm = 0.0;
    for (int64_t idx = t; idx < KK; idx += kSolveThreads) {
      const Cd x = X[idx], d = Y[idx];
      xm = fmax(xm, fmax(fabs(x.re), fabs(x.im)));
      rm = fmax(rm, fmax(fabs(d.re), fabs(d.im)));
      X[idx] = Cd{x.re + d.re, x.im + d.im};
    }
    xm = warp_max(xm);
    rm = warp_max(rm);
    if (lane == 0) {
      red[0][warp] = xm;
      red[1][warp] = rm;
    }
    __syncthreads();
    for (int w = 0; w < kSolveWarps; ++w) {
      xm = fmax(xm, red[0][w]);
      rm = fmax(rm, red[1][w]);
    }
    __syncthreads();
    rel = xm > 0.0 ? rm / xm : 0.0;
    if (!(rel > 0x1p-54)) break;
  }
  // T[i][k] = X[k][i], zero between the classes.
  double ext = 0.0, sca = 0.0;
  double* T = a.T ? a.T + 2 * jb.T0 : nullptr;
  for (int64_t idx = t; idx < 2 * KK; idx += kSolveThreads) {
    const int u = (int)(idx / (2 * K)), col = (int)(idx % (2 * K));
    const int bk = col >= K, ko = col - bk * K;
    Cd v{0.0, 0.0};
    if (((ko + bk) & 1) == p) {
      const int w = bk ? n_a + ko / 2 : ko / 2;
      v = X[(int64_t)w * K + u];
      if (w == u) ext -= v.re;
      sca += v.re * v.re + v.im * v.im;
    }
    if (T) {
      const int64_t row = order(u) + (element(u) ? K : 0);
      T[2 * (row * 2 * K + col)] = v.re;
      T[2 * (row * 2 * K + col) + 1] = v.im;
    }
  }
  ext = warp_sum(ext);
  sca = warp_sum(sca);
  if (lane == 0) {
    red[0][warp] = ext;
    red[1][warp] = sca;
  }
  __syncthreads();
  if (t == 0) {
    for (int w = 1; w < kSolveWarps; ++w) {
      ext += red[0][w];
      sca += red[1][w];
    }
    double* o = a.sums + 3 * (2 * (int64_t)job + p);
    o[0] = ext;
    o[1] = sca;
    o[2] = rel;
  }
}

void launch_tm_tables(const TmArgs& a, cudaStream_t s) {
  if (a.n_jobs <= 0) return;
  tm_geom_kernel<<<(unsigned)((a.n_node_total + 127) / 128), 128, 0, s>>>(a);
  tm_angular_kernel<<<(unsigned)((a.n_ang_total + 127) / 128), 128, 0, s>>>(a);
  if (a.n_ser_total > 0)
    tm_series_kernel<<<(unsigned)((a.n_ser_total + 127) / 128), 128, 0, s>>>(a);
  if (a.n_forms_total > 0)
    tm_forms_kernel<<<(unsigned)((a.n_forms_total + 127) / 128), 128, 0, s>>>(a);
}
void launch_tm_surface(const TmArgs& a, cudaStream_t s) {
  if (a.n_jobs <= 0) return;
  tm_surface_kernel<<<(unsigned)((a.n_pair_total + 127) / 128), 128, 0, s>>>(a);
}
// The solves in groups of similar K, each with the shared memory its largest needs: both matrices
// up to 80 unknowns, the factors up to 112, neither beyond.
cudaError_t launch_tm_solve(const TmArgs& a, const TmSolveGroup* groups, int n_groups,
                            cudaStream_t s) {
  for (int k = 0; k < n_groups; ++k) {
    const TmSolveGroup& g = groups[k];
    if (g.n == 0) continue;
    const int where = tm_solve_where(g.max_k);
    const size_t head = (size_t)g.max_k * (2 * sizeof(Cd) + 2 * sizeof(int)) + 16;
    const size_t bytes = head + (size_t)(2 - where) * g.max_k * g.max_k * sizeof(Cd);
    auto f = where == 0 ? tm_solve_kernel<0> : where == 1 ? tm_solve_kernel<1> : tm_solve_kernel<2>;
    const cudaError_t e =
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    f<<<2 * g.n, kSolveThreads, bytes, s>>>(a, a.solve_list + g.first);
  }
  return cudaGetLastError();
}
}  // namespace sb
