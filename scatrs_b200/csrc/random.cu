// The orientation-averaged phase matrix of a spheroid from its T-matrix by the rank
// decomposition of T (scatrs/src/tmatrix/random.rs:85-335, after research/tmatrix/ranks.py),
// and its Greek coefficients (greek_raw, random.rs:283-292), batched over spheroids in five
// kernels:
//
//   ro_cg_kernel     the Clebsch-Gordan vectors of both tables, one thread per vector; they depend
//                    on the indices only, so a batch's spheroids share them (kept per context);
//   ro_rank_kernel   one block per (n <= n', two spheroids): the helicity blocks
//                    T^{p sigma}_mu(n, n') = (T11 + sigma T12 + p T21 + p sigma T22)/2 of every
//                    mode mu (T^{p sigma}_{-m} = T^{-p,-sigma}_m) and their rank components
//                    t^(s)(n, n') = sum_mu (-1)^(n'-mu) C^{s 0}_{n mu; n' -mu} T^{p sigma}_mu(n, n'),
//                    for (n, n') and (n', n), which have the same coefficients;
//   ro_w_kernel      one block per (spheroid, sigma, n, eight q, 128 ranks s):
//                    w_n = sum_n' inc_n' (-1)^(n'-sigma) C^{s q}_{n, q+sigma; n', -sigma}
//                    t^(s)(n, n') for both scattered helicities, times the cosine-independent part
//                    gamma_n (-i)^n of the far field;
//   ro_phi_kernel    one block per (spheroid, q, tile of 32 cosines): Phi_{sq} = sum_n w_n
//                    (pi_mn + p tau_mn) as FP64 MMAs (ranks x cosines, contraction over n), and
//                    the q-th share of <A_a A_b*> = sum_s Phi_a Phi_b* / (2s + 1) for the 16
//                    helicity pairs, whose four factors a thread holds together;
//   ro_f_kernel      one thread per (spheroid, cosine): the shares summed over q in order, and
//                    the Mueller form F11, F12, F22, F33, F34, F44 (S = U A U^{-1});
//   ro_greek_kernel  one thread per (spheroid, l): the six projections on the
//                    N + ceil((L+1)/2)-point Gauss rule (greek.rs:227-266).
//
// Clebsch-Gordan coefficients come from the three-term recursion of the 3j symbol in its first
// angular momentum (Schulten & Gordon, J. Math. Phys. 16, 1961 (1975)), run down from the
// largest J and up from the smallest, joined where the downward solution peaks, normalized by
// sum (2J + 1) f^2 = 1 and signed by the closed form at the largest J. All sums run in a fixed
// order, so the results are bitwise reproducible.
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.h"

namespace sb {

namespace {

constexpr double kPi = 3.14159265358979323846;

struct C2 {
  double re, im;
};
__device__ __forceinline__ C2 c_add(C2 a, C2 b) { return C2{a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ C2 c_mul(C2 a, C2 b) {
  return C2{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
__device__ __forceinline__ C2 c_scale(C2 a, double s) { return C2{a.re * s, a.im * s}; }
__device__ __forceinline__ C2 c_conj(C2 a) { return C2{a.re, -a.im}; }
__device__ __forceinline__ C2 ipow(int k) {  // i^k
  switch (((k % 4) + 4) % 4) {
    case 0: return C2{1, 0};
    case 1: return C2{0, 1};
    case 2: return C2{-1, 0};
    default: return C2{0, -1};
  }
}
__device__ __forceinline__ double sgn(int k) { return (k & 1) ? -1.0 : 1.0; }

// The recursion's coefficients for f(J) = (J ja jb; -M ma mb).
__device__ __forceinline__ double rec_a(int J, int ja, int jb, int M) {
  const double v = ((double)J * J - (double)(ja - jb) * (ja - jb)) *
                   ((double)(ja + jb + 1) * (ja + jb + 1) - (double)J * J) *
                   ((double)J * J - (double)M * M);
  return v > 0.0 ? sqrt(v) : 0.0;
}
__device__ __forceinline__ double rec_b(int J, int ja, int jb, int ma, int mb) {
  const int M = ma + mb;
  return -(2.0 * J + 1) * ((double)ja * (ja + 1) * (-M) - (double)jb * (jb + 1) * (-M) -
                           (double)J * (J + 1) * (mb - ma));
}

// C^{J, ma+mb}_{ja ma; jb mb} for J = J_min..ja+jb into v (in place: the downward solution, then
// the upward one below its peak); J_min = max(|ja - jb|, |ma + mb|). |ma| <= ja, |mb| <= jb.
__device__ void cg_vector(int ja, int ma, int jb, int mb, double* v) {
  const int M = ma + mb;
  const int jmin = max(abs(ja - jb), abs(M)), jmax = ja + jb;
  const int len = jmax - jmin + 1;
  // Downward from f(J_max) = 1.
  double next = 0.0, cur = 1.0, aj1 = rec_a(jmax + 1, ja, jb, M);
  int peak = len - 1;
  double pv = 1.0, at_peak = 1.0;
  v[len - 1] = 1.0;
  for (int J = jmax; J > jmin; --J) {
    const double aj = rec_a(J, ja, jb, M), den = (J + 1) * aj;
    const double prev =
        den == 0.0 ? 0.0 : -(J * aj1 * next + rec_b(J, ja, jb, ma, mb) * cur) / den;
    next = cur;
    cur = prev;
    aj1 = aj;
    v[J - 1 - jmin] = cur;
    if (fabs(cur) >= pv) {
      pv = fabs(cur);
      at_peak = cur;
      peak = J - 1 - jmin;
    }
  }
  if (peak > 0 && jmin > 0) {
    // Upward from f(J_min) = 1 to the peak, scaled to meet the downward solution there.
    double prev = 0.0, aj = rec_a(jmin, ja, jb, M);
    cur = 1.0;
    for (int p = 0; p < peak; ++p) {
      const int J = jmin + p;
      v[p] = cur;
      const double a1 = rec_a(J + 1, ja, jb, M), den = J * a1;
      const double up =
          den == 0.0 ? 0.0 : -(rec_b(J, ja, jb, ma, mb) * cur + (J + 1) * aj * prev) / den;
      prev = cur;
      cur = up;
      aj = a1;
    }
    // cur is the upward value at the peak; the downward one stays there.
    if (cur != 0.0) {
      const double sc = at_peak / cur;
      for (int p = 0; p < peak; ++p) v[p] *= sc;
    }
  }
  double norm = 0.0;
  for (int p = 0; p < len; ++p) norm += (2.0 * (jmin + p) + 1) * v[p] * v[p];
  double sc = 1.0 / sqrt(norm);
  const bool negative = ((ja - jb + M) % 2 + 2) % 2 == 1;
  if ((v[len - 1] < 0.0) != negative) sc = -sc;
  const double phase = negative ? -1.0 : 1.0;
  for (int p = 0; p < len; ++p) v[p] = phase * sqrt(2.0 * (jmin + p) + 1) * v[p] * sc;
}

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

// The rank table's vectors C^{s 0}_{n u; n' -u}, n <= n' <= N, 0 <= u <= n (s from n' - n, 2n + 1
// of them), and the far field's C^{s q}_{n m; n' -1}, q = m - 1, |m| <= n, n' <= N (from |n - n'|,
// zero below |q|; 2n + 1 places). Bound by each vector's serial recursion; made once per size.
__global__ void __launch_bounds__(128) ro_cg_kernel(RoCg cg, double* r, double* w) {
  const int N = cg.n, n = blockIdx.y + 1;
  const int64_t n_r = (int64_t)(N - n + 1) * (n + 1), n_w = (int64_t)(2 * n + 1) * N;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_r + n_w;
       t += (int64_t)gridDim.x * blockDim.x) {
    if (t < n_r) {
      const int np = n + (int)(t / (n + 1)), u = (int)(t % (n + 1));
      cg_vector(n, u, np, -u, r + cg.r_row(n, np, u));
    } else {
      const int m = (int)((t - n_r) / N) - n, np = 1 + (int)((t - n_r) % N);
      double* v = w + cg.w_row(n, m, np);
      const int skip = max(abs(m - 1) - abs(n - np), 0);
      for (int i = 0; i < min(skip, 2 * n + 1); ++i) v[i] = 0.0;
      if (abs(m - 1) <= n + np) cg_vector(n, m, np, -1, v + skip);
    }
  }
}

// Two spheroids of one (n, n') per block; thread i holds rank |n - n'| + i, its 16 sums per spheroid
// (four helicity pairs, complex, for (n, n') and for (n', n)). The coefficients are read once per
// two spheroids instead of being recomputed per spheroid (a thread per (spheroid, n, n') with its
// vectors in local memory): 107 -> 2.9 ms per pass of 288 spheroids to x = 21.
__global__ void __launch_bounds__(128) ro_rank_kernel(RoArgs a) {
  constexpr int kU = 16;
  __shared__ double h[2][kU][2][16];  // [spheroid][mode][parity of n + n' - s][the 16 factors]
  const int t = threadIdx.x;
  // blockIdx.x = n' (n' - 1) / 2 + n - 1.
  int np = (int)((sqrt(8.0 * blockIdx.x + 1.0) + 1.0) * 0.5);
  while (np * (np - 1) / 2 > (int)blockIdx.x) --np;
  while (np * (np + 1) / 2 <= (int)blockIdx.x) ++np;
  const int n = (int)blockIdx.x - np * (np - 1) / 2 + 1;
  const int s0 = 2 * blockIdx.y;
  bool live[2];
  RoSph sp[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    sp[e] = a.sph[min(s0 + e, a.n_sph - 1)];
    live[e] = s0 + e < a.n_sph && sp[e].N >= np;
  }
  if (!live[0] && !live[1]) return;
  const int len = 2 * n + 1;
  for (int i0 = 0; i0 < len; i0 += 128) {
    const int i = i0 + t;
    double acc[2][16];
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int k = 0; k < 16; ++k) acc[e][k] = 0.0;
    for (int u0 = 0; u0 <= n; u0 += kU) {
      __syncthreads();
      if (t < 2 * kU) {
        const int e = t / kU, u = u0 + t % kU;
        if (live[e] && u <= n) {
          const int nl = max(u, 1);
          const TmJob& jb = a.jobs[sp[e].job0 + u];
          const int K = jb.K;
          const C2* T = reinterpret_cast<const C2*>(a.T) + jb.T0;
          for (int o = 0; o < 2; ++o) {
            const int r = (o ? np : n) - nl, c = (o ? n : np) - nl;
            const C2 t11 = T[(int64_t)r * 2 * K + c], t12 = T[(int64_t)r * 2 * K + K + c];
            const C2 t21 = T[(int64_t)(K + r) * 2 * K + c],
                     t22 = T[(int64_t)(K + r) * 2 * K + K + c];
            const double ph = 0.5 * sgn((o ? n : np) - u);
            C2 hp[4];
            for (int k = 0; k < 4; ++k) {
              const double p = k & 2 ? -1.0 : 1.0, s = k & 1 ? -1.0 : 1.0;
              hp[k] = c_scale(
                  c_add(c_add(t11, c_scale(t12, s)), c_add(c_scale(t21, p), c_scale(t22, p * s))), ph);
            }
            // Mode -u adds T^{-p,-sigma}_u with (-1)^(n + n' - s).
            for (int par = 0; par < 2; ++par)
              for (int k = 0; k < 4; ++k) {
                const C2 v = u == 0 ? hp[k] : c_add(hp[k], c_scale(hp[3 - k], par ? -1.0 : 1.0));
                h[e][t % kU][par][8 * o + 2 * k] = v.re;
                h[e][t % kU][par][8 * o + 2 * k + 1] = v.im;
              }
          }
        }
      }
      __syncthreads();
      if (i < len) {
        const double* cgv = a.cg_r + a.cg.r_row(n, np, u0) + i;
        const int nu = min(kU, n + 1 - u0);
        for (int u = 0; u < nu; ++u) {
          const double c = cgv[(int64_t)u * len];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (!live[e]) continue;
            const double* f = h[e][u][i & 1];
#pragma unroll
            for (int k = 0; k < 16; ++k) acc[e][k] = fma(c, f[k], acc[e][k]);
          }
        }
      }
    }
    if (i >= len) continue;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (!live[e]) continue;
      const int n1 = sp[e].N + 1, S = 2 * sp[e].N + 1;
      C2* rank = reinterpret_cast<C2*>(a.rank + sp[e].rank0) + i;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        rank[((int64_t)(k * n1 + n) * n1 + np) * S] = C2{acc[e][2 * k], acc[e][2 * k + 1]};
        if (np != n)
          rank[((int64_t)(k * n1 + np) * n1 + n) * S] = C2{acc[e][8 + 2 * k], acc[e][9 + 2 * k]};
      }
    }
  }
}

// Thread t holds rank s = 128 blockIdx.z + t for eight q: the rank components are read once per
// eight q, the coefficients once per thread, both contiguous over s. Bound by
// L2 reads of the components; against a thread per (spheroid, q, sigma, n) that recomputed the
// coefficients: 97 -> 16 ms on the same pass.
__global__ void __launch_bounds__(128) ro_w_kernel(RoArgs a) {
  constexpr int kQ = 8;
  const RoSph sp = a.sph[blockIdx.y];
  const int N = sp.N, n1 = N + 1, S = 2 * N + 1, Q = 2 * N + 3, q_tiles = (a.max_n * 2 + 3 + kQ - 1) / kQ;
  const int qt = blockIdx.x % q_tiles, rest = blockIdx.x / q_tiles;
  const int sg = rest & 1, n = 1 + rest / 2, sigma = sg ? -1 : 1;
  const int s = 128 * blockIdx.z + threadIdx.x;
  if (n > N || qt * kQ >= Q || 128 * (int)blockIdx.z >= S) return;
  __shared__ C2 pre[kRoMaxN + 1];
  for (int np = 1 + threadIdx.x; np <= N; np += 128)
    pre[np] = c_scale(ipow(np - 1), 2.0 * sqrt(kPi * (2 * np + 1)) * sgn(np - sigma));
  __syncthreads();
  if (s >= S) return;
  C2 acc[kQ][2];
#pragma unroll
  for (int k = 0; k < kQ; ++k) acc[k][0] = acc[k][1] = C2{0.0, 0.0};
  // The coefficients of (q, sigma = 1) are the table's at m = q + 1; of (q, -1) those at -m, m =
  // q - 1, times (-1)^(n + n' - s).
  const double* cgq[kQ];
  bool on[kQ];
#pragma unroll
  for (int k = 0; k < kQ; ++k) {
    const int q = qt * kQ + k - N - 1, m = q + sigma;
    on[k] = qt * kQ + k < Q && abs(m) <= n;
    cgq[k] = a.cg_w + a.cg.w_row(n, on[k] ? sigma * m : 0, 1);
  }
  const C2* rank = reinterpret_cast<const C2*>(a.rank + sp.rank0);
  const C2* r0 = rank + ((int64_t)(sg * n1 + n) * n1) * S;
  const C2* r1 = rank + ((int64_t)((2 + sg) * n1 + n) * n1) * S;
  for (int np = max(1, abs(n - s)); np <= N; ++np) {
    const int i = s - abs(n - np);
    if (i < 0 || s > n + np) continue;
    const C2 p = pre[np];
    const C2 t0 = c_mul(p, r0[(int64_t)np * S + i]), t1 = c_mul(p, r1[(int64_t)np * S + i]);
    const double sign = sg && (i & 1) ? -1.0 : 1.0;
    const int64_t at = (int64_t)(np - 1) * (2 * n + 1) + i;
#pragma unroll
    for (int k = 0; k < kQ; ++k) {
      const double c = on[k] ? sign * cgq[k][at] : 0.0;
      acc[k][0].re = fma(c, t0.re, acc[k][0].re);
      acc[k][0].im = fma(c, t0.im, acc[k][0].im);
      acc[k][1].re = fma(c, t1.re, acc[k][1].re);
      acc[k][1].im = fma(c, t1.im, acc[k][1].im);
    }
  }
  // The far field's cosine-independent factor gamma_n (-i)^n (functions.rs:192-239).
  const C2 fn = c_scale(ipow(-n), sqrt((2.0 * n + 1) / (kPi * 4.0 * n * (n + 1))));
  C2* w = reinterpret_cast<C2*>(a.w + sp.w0);  // [q][sigma][p][n - 1][s]
#pragma unroll
  for (int k = 0; k < kQ; ++k) {
    const int qi = qt * kQ + k;
    if (qi >= Q) continue;
#pragma unroll
    for (int p = 0; p < 2; ++p)
      w[((int64_t)((qi * 2 + sg) * 2 + p) * N + n - 1) * S + s] = c_mul(acc[k][p], fn);
  }
}

namespace {
constexpr int kPhiStride = 36;  // doubles per order of the angular table: 32 cosines, conflict-free
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}
}  // namespace

// Eight warps: warp w takes cosines 8 (w & 3) .. + 7 of the tile and every second group of 8 ranks.
// A lane's D fragment holds the four helicity keys' Phi at one (rank, cosine) pair of columns, so
// the products need no exchange; they are summed over the ranks in registers, then over the 8
// lanes and the two warps of a cosine group. Bound by the serial angular recursion at a block's start
// and the FP64 tensor path; against one thread per (cosine, key) on scalar sums: 129 -> 20 ms on the
// same pass.
__global__ void __launch_bounds__(256) ro_phi_kernel(RoArgs a) {
  extern __shared__ double ro_pt[];  // [sigma][p][N rows, order n - 1][kPhiStride]: pi + p tau
  __shared__ double half[4][8][16];
  const int b = blockIdx.x, t = threadIdx.x;
  const int si = owner(a.n_sph, b, [&](int i) { return a.sph[i].t_phi; });
  const RoSph sp = a.sph[si];
  const int N = sp.N, S = 2 * N + 1, nq = sp.nq, tiles = (nq + 31) / 32;
  const int idx = b - (int)sp.t_phi, qi = idx / tiles, q = qi - N - 1, j0 = (idx % tiles) * 32;
  const int rows = (N + 3) & ~3;
  const int64_t plane = (int64_t)rows * kPhiStride;
  // The angular parts at the tile's cosines: normalized d_{|m| n}, pi and tau (functions.rs:
  // 192-239), m = q + sigma, zero where |m| > N or n < |m|. One thread per (sigma, cosine).
  if (t < 64) {
    const int sg = t >> 5, jl = t & 31, j = j0 + jl;
    double* pp = ro_pt + (int64_t)(sg * 2) * plane + jl;
    double* pm = pp + plane;
    for (int k = 0; k < rows; ++k) pp[k * kPhiStride] = pm[k * kPhiStride] = 0.0;
    const int m = q + (sg ? -1 : 1), am = abs(m);
    if (j < nq && am <= N) {
      const double ct = a.mu[sp.mu0 + j], st = sqrt(1.0 - ct * ct);
      double am_ = 1.0;
      for (int k = 1; k <= am; ++k) am_ *= sqrt((double)(2 * k - 1) / (2 * k));
      double sp_ = 1.0;
      for (int k = 0; k < am; ++k) sp_ *= st;
      const double flip = m < 0 ? sgn(am) : 1.0;
      double dprev = 0.0, dk = am_ * sp_;  // d_{am - 1} = 0, d_{am}
      double root = 0.0;                   // sqrt(k^2 - am^2)
      for (int k = am; k <= N; ++k) {
        const double root1 = sqrt((double)(k + 1) * (k + 1) - (double)am * am);
        const double rd = root * dprev;
        if (k >= 1) {
          const double tau = (k * ct * dk - rd) / st * flip;
          const double pi = am * dk / st;
          const double pv = m < 0 ? -(pi * flip) : pi;
          pp[(k - 1) * kPhiStride] = pv + tau;
          pm[(k - 1) * kPhiStride] = pv - tau;
        }
        const double dnext = k == am ? sqrt(2.0 * am + 1) * ct * dk
                                     : ((2 * k + 1) * ct * dk - rd) / root1;
        dprev = dk;
        dk = dnext;
        root = root1;
      }
    }
  }
  __syncthreads();
  const int warp = t >> 5, lane = t & 31, lq = lane & 3, g = lane >> 2, ct = warp & 3;
  const C2* w = reinterpret_cast<const C2*>(a.w + sp.w0) + (int64_t)qi * 4 * N * S;
  // Orders below |m| - 1 of the smaller |m| contribute nothing.
  const int k_lo = (max(min(abs(q + 1), abs(q - 1)), 1) - 1) & ~3;
  double prod[2][16];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int k = 0; k < 16; ++k) prod[j][k] = 0.0;
  for (int s0 = 8 * (warp >> 2); s0 < S; s0 += 16) {
    const int s = s0 + g;
    double re[4][2], im[4][2];
#pragma unroll
    for (int key = 0; key < 4; ++key) re[key][0] = re[key][1] = im[key][0] = im[key][1] = 0.0;
    for (int k0 = k_lo; k0 < N; k0 += 4) {
      const int k = k0 + lq;
      const bool valid = k < N && s < S;
      C2 av[4];
#pragma unroll
      for (int key = 0; key < 4; ++key) {
        // key = 2 p + sigma index (p, sigma = +1 first); w holds [sigma][p].
        const int plane_w = (key & 1) * 2 + (key >> 1);
        av[key] = valid ? w[((int64_t)plane_w * N + k) * S + s] : C2{0.0, 0.0};
      }
#pragma unroll
      for (int key = 0; key < 4; ++key) {
        const double bv =
            ro_pt[((key & 1) * 2 + (key >> 1)) * plane + (int64_t)k * kPhiStride + 8 * ct + g];
        dmma(re[key][0], re[key][1], av[key].re, bv);
        dmma(im[key][0], im[key][1], av[key].im, bv);
      }
    }
    const double inv = 1.0 / (2 * s + 1);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      int o = 4;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const double xr = re[x][j] * inv, xi = im[x][j] * inv;
        prod[j][x] += xr * re[x][j] + xi * im[x][j];
#pragma unroll
        for (int y = x + 1; y < 4; ++y) {
          prod[j][o] += xr * re[y][j] + xi * im[y][j];
          prod[j][o + 1] += xi * re[y][j] - xr * im[y][j];
          o += 2;
        }
      }
    }
  }
  // Over the eight lanes of a column (g), then over the two warps.
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int k = 0; k < 16; ++k)
#pragma unroll
      for (int off = 4; off < 32; off <<= 1)
        prod[j][k] += __shfl_xor_sync(0xffffffffu, prod[j][k], off);
  if (warp >= 4 && g == 0)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 16; ++k) half[ct][2 * lq + j][k] = prod[j][k];
  __syncthreads();
  if (warp < 4 && g == 0) {
    C2* part = reinterpret_cast<C2*>(a.part + sp.part0) + (int64_t)qi * 16 * nq;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int jc = j0 + 8 * ct + 2 * lq + j;
      if (jc >= nq) continue;
      double v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = prod[j][k] + half[ct][2 * lq + j][k];
      int o = 4;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        part[(int64_t)(5 * x) * nq + jc] = C2{v[x], 0.0};
#pragma unroll
        for (int y = x + 1; y < 4; ++y) {
          part[(int64_t)(4 * x + y) * nq + jc] = C2{v[o], v[o + 1]};
          part[(int64_t)(4 * y + x) * nq + jc] = C2{v[o], -v[o + 1]};
          o += 2;
        }
      }
    }
  }
}

__global__ void __launch_bounds__(128) ro_f_kernel(RoArgs a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n_f) return;
  const int si = owner(a.n_sph, t, [&](int i) { return a.sph[i].t_f; });
  const RoSph sp = a.sph[si];
  const int N = sp.N, nq = sp.nq, j = (int)(t - sp.t_f);
  const C2* part = reinterpret_cast<const C2*>(a.part + sp.part0);
  C2 prod[16];
  for (int k = 0; k < 16; ++k) prod[k] = C2{0, 0};
  for (int qi = 0; qi < 2 * N + 3; ++qi)
    for (int k = 0; k < 16; ++k) prod[k] = c_add(prod[k], part[((int64_t)qi * 16 + k) * nq + j]);
  // <S_ij S*_kl> = sum U_ia U^-1_bj conj(U_kc U^-1_dl) <A_ab A*_cd> (random.rs:295-335).
  const double r = sqrt(0.5);
  const C2 U[2][2] = {{C2{r, 0}, C2{r, 0}}, {C2{0, r}, C2{0, -r}}};
  const C2 Ui[2][2] = {{C2{r, 0}, C2{0, -r}}, {C2{r, 0}, C2{0, r}}};
  auto ss = [&](int i, int jj, int k, int l) {
    C2 acc{0, 0};
    for (int x = 0; x < 2; ++x)
      for (int b = 0; b < 2; ++b)
        for (int c = 0; c < 2; ++c)
          for (int e = 0; e < 2; ++e) {
            const C2 fct = c_mul(c_mul(U[i][x], Ui[b][jj]), c_conj(c_mul(U[k][c], Ui[e][l])));
            acc = c_add(acc, c_mul(fct, prod[((x * 2 + b) * 2 + c) * 2 + e]));
          }
    return acc;
  };
  const double s22 = ss(0, 0, 0, 0).re, s11 = ss(1, 1, 1, 1).re, s33 = ss(0, 1, 0, 1).re,
               s44 = ss(1, 0, 1, 0).re;
  const C2 s12 = ss(1, 1, 0, 0), s34 = ss(0, 1, 1, 0);
  double* f = a.f + sp.f0;
  f[0 * nq + j] = 0.5 * (s11 + s22 + s33 + s44);
  f[1 * nq + j] = 0.5 * (s22 - s11 + s44 - s33);
  f[2 * nq + j] = 0.5 * (s22 + s11 - s44 - s33);
  f[3 * nq + j] = s12.re + s34.re;
  f[4 * nq + j] = -s12.im - s34.im;
  f[5 * nq + j] = s12.re - s34.re;
}

__global__ void __launch_bounds__(128) ro_greek_kernel(RoArgs a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n_g) return;
  const int si = owner(a.n_sph, t, [&](int i) { return a.sph[i].t_g; });
  const RoSph sp = a.sph[si];
  const int nq = sp.nq, len = sp.L + 1, l = (int)(t - sp.t_g);
  const double* f = a.f + sp.f0;
  const double* D = a.proj[si];
  double a1 = 0, a4 = 0, pl = 0, mn = 0, b1 = 0, b2 = 0;
  for (int k = 0; k < nq; ++k) {
    const double d00 = D[((int64_t)0 * nq + k) * len + l], d22 = D[((int64_t)1 * nq + k) * len + l];
    const double d2m2 = D[((int64_t)2 * nq + k) * len + l], d02 = D[((int64_t)3 * nq + k) * len + l];
    a1 += f[k] * d00;
    b1 += f[nq + k] * d02;
    pl += (f[2 * nq + k] + f[3 * nq + k]) * d22;
    mn += (f[2 * nq + k] - f[3 * nq + k]) * d2m2;
    b2 += f[4 * nq + k] * d02;
    a4 += f[5 * nq + k] * d00;
  }
  double* g = a.greek + sp.g0;
  g[0 * len + l] = a1;
  g[1 * len + l] = 0.5 * (pl + mn);
  g[2 * len + l] = 0.5 * (pl - mn);
  g[3 * len + l] = a4;
  g[4 * len + l] = b1;
  g[5 * len + l] = b2;
}

void launch_cg(const RoCg& cg, double* r, double* w, cudaStream_t s) {
  ro_cg_kernel<<<dim3(64, cg.n), 128, 0, s>>>(cg, r, w);
}

cudaError_t launch_random(const RoArgs& a, cudaStream_t s) {
  if (a.n_sph <= 0) return cudaSuccess;
  auto grid = [](int64_t n) { return (unsigned)((n + 127) / 128); };
  ro_rank_kernel<<<dim3(a.max_n * (a.max_n + 1) / 2, (a.n_sph + 1) / 2), 128, 0, s>>>(a);
  // Each launch's own status: a later launch that succeeds can hide an earlier one's refusal.
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int q_tiles = (2 * a.max_n + 3 + 7) / 8;
  ro_w_kernel<<<dim3(2 * a.max_n * q_tiles, a.n_sph, (2 * a.max_n + 1 + 127) / 128), 128, 0, s>>>(a);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  // Shared memory: the angular parts of the four helicity keys at a tile of 32 cosines for the
  // batch's largest N.
  const size_t pt_bytes = (size_t)4 * ((a.max_n + 3) & ~3) * kPhiStride * sizeof(double);
  e = cudaFuncSetAttribute(ro_phi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)pt_bytes);
  if (e != cudaSuccess) return e;
  ro_phi_kernel<<<(unsigned)a.n_phi, 256, pt_bytes, s>>>(a);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  ro_f_kernel<<<grid(a.n_f), 128, 0, s>>>(a);
  ro_greek_kernel<<<grid(a.n_g), 128, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace sb
