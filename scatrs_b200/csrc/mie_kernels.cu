// K-a: the Mie recurrences of every size node, one thread per node, one warp per chunk of 32
// consecutive nodes of a (distribution, wavelength) unit. Compiled with -fmad=false (see
// mie_device.cuh). The coefficients leave in the layout the angle GEMM reads: for each chunk a
// row per order n (n = 1..N_c, N_c the chunk's largest number of terms, then zero rows to a multiple
// of 4) of 128 doubles,
// 4 per lane: u.re, u.im, v.re, v.im with (u, v) = (a_n, b_n) for odd n and (b_n, a_n) for even
// n (scatrs/src/ensemble/fast.rs:95-137), zero above the node's own N.
#include "kernels.h"
#include "layered_deriv.cuh"
#include "layered_fixed.cuh"
#include "mie_device.cuh"

namespace sb {

// Error word: the smallest (wavelength, distribution, radius) key of a node whose inputs fail,
// with its status in the low 2 bits.
__device__ __forceinline__ void record_error(unsigned long long* err, long long i_wl,
                                             long long d, long long j, long long n_dist,
                                             long long n_nodes, int status) {
  unsigned long long key = (unsigned long long)(((i_wl * n_dist + d) * n_nodes + j) << 2) |
                           (unsigned long long)status;
  atomicMin(err, key);
}

// Each chunk's largest number of terms (the band selector, engine.rs:961-978).
__global__ void plan_chunks_kernel(PlanArgs a) {
  int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (warp >= a.n_chunks) return;
  int64_t unit = warp / a.cpu;
  int c = warp % a.cpu;
  int64_t d = unit / a.n_wl, i = unit % a.n_wl;
  int j = c * 32 + lane;
  int64_t n = 0;
  if (j < a.n_nodes) {
    double r = a.radius[(a.per_unit ? unit : d) * a.n_nodes + j];
    if (r > 0.0) {
      double x = 2.0 * kPi * r / a.wl[i];
      n = default_n_max(x);
      if (n > (1 << 20)) n = 1 << 20;
    }
  }
  int nn = (int)n;
  for (int off = 16; off > 0; off >>= 1) {
    int o = __shfl_xor_sync(0xffffffffu, nn, off);
    nn = o > nn ? o : nn;
  }
  if (lane == 0) a.chunk_n[warp] = nn;
}

// NodeTableArgs: 16 threads per record. Bound by the records' copy from the host (256 B a panel
// against the 384 B of the three padded arrays it stands for, which a host thread would otherwise
// have to clear, fill and copy): 178,000 records take 19 us beside 0.86 ms of copies.
__global__ void node_table_kernel(NodeTableArgs a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t i = t >> 4;
  const int k = (int)(t & 15);
  if (i >= a.n_rec || k == 15) return;
  const double* rec = a.rec + i * node_record(a.n_theta);
  const int64_t at = __double_as_longlong(rec[0]) + k;
  const double h = rec[1], ur = rec[17 + k];
  if (h < 0.0) {
    if (k == 0) {
      a.radius[at] = rec[2];
      a.weight[at] = 1.0;
    }
    return;
  }
  const double wk = h * a.wk[k], wg = h * a.wg[k];
  a.radius[at] = rec[2 + k];
  a.weight[at] = wk * ur;
  a.wdiff[at] = wk * ur - wg * ur;
  for (int b = 0; b < a.n_theta; ++b) {
    const double dw = rec[32 + 15 * b + k];
    a.wtheta[3 * at + b] = wk * dw;
    a.wthdiff[3 * at + b] = wk * dw - wg * dw;
  }
}

// A chunk's side record (UnitArgs::side), from lane j's node: the factor sc = 4 pi r^2 / x^2 of its
// elements times the values' and the parameters' weights wb[0..P], then times the error weights wbd
// where there are any, and the largest number of terms n of each 8 nodes.
__device__ __forceinline__ void put_side(const MieFixedArgs& a, int chunk, int lane, double sc,
                                         const double* wb, const double* wbd, int P, int64_t n) {
  double* o = a.side + (int64_t)chunk * a.side_stride;
  for (int b = 0; b <= P; ++b) o[32 * b + lane] = wb[b] * sc;
  if (wbd)
    for (int b = 0; b <= P; ++b) o[32 * (1 + P + b) + lane] = wbd[b] * sc;
  int top = (int)n;
  for (int off = 1; off < 8; off <<= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, off));
  if ((lane & 7) == 0) o[a.side_stride - 4 + (lane >> 3)] = (double)top;
}

// The chunk's weighted sums of the 8 per-particle quantities, in a fixed tree order; on adaptive
// panels (qe weighted by w_K - w_G) then |Kronrod - Gauss| of each of the chunk's two panels (lanes
// 0-15, 16-31), added.
template <bool kAdaptive>
__device__ __forceinline__ void put_sums(const MieFixedArgs& a, int chunk, int lane,
                                         const double* q, const double* qe) {
  const int stride = kAdaptive ? 16 : 8;
  for (int k = 0; k < 8; ++k) {
    double v = q[k];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0) a.chunk_sums[(int64_t)chunk * stride + k] = v;
  }
  if constexpr (kAdaptive) {
    for (int k = 0; k < 8; ++k) {
      double v = qe[k];
      for (int off = 8; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      const double other = __shfl_sync(0xffffffffu, v, 16);
      if (lane == 0) a.chunk_sums[(int64_t)chunk * 16 + 8 + k] = fabs(v) + fabs(other);
    }
  }
}

// kL: 1 homogeneous, 2 to 4 layers with the state sized at compile time, 0 any number of layers.
template <int kL, bool kAdaptive>
__device__ __forceinline__ void mie_chunk(const MieFixedArgs& a, int chunk) {
  int lane = threadIdx.x & 31;
  int64_t unit = a.units[chunk / a.cpu];
  int c = chunk % a.cpu;
  int64_t d = unit / a.n_wl, i = unit % a.n_wl;
  int j = c * 32 + lane;
  int nc = a.chunk_n[chunk];
  int64_t row0 = a.chunk_row[chunk];
  // This lane's place in the coefficient row of order index k (kernels.h).
  auto Xk = [&](int64_t k) { return a.X + (row0 + k) * 128 + ((lane ^ (int)(k & 3)) << 2); };
  // Scratch: 2L - 1 complex ratio arrays (one for a sphere) of nc + 2 rows, and u_k(x).
  constexpr bool kLayered = kL != 1;
  const int n_arr = kLayered ? 2 * a.n_layers - 1 : 1;
  Scratch s;
  s.uz = a.uz + (row0 + 2 * (int64_t)chunk) * n_arr * 32 + lane;
  s.ux = a.ux + (row0 + 2 * (int64_t)chunk) * 32 + lane;
  s.stride = 32;
  double q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  double qe[kAdaptive ? 8 : 1] = {};  // adaptive: weighted by w_K - w_G
  double cm[4] = {0.0, 0.0, 0.0, 0.0};  // the largest |X| of this lane's four columns
  double sc = 0.0, wv = 0.0, wd = 0.0;
  int64_t n = 0;
  const int64_t node = (a.per_unit ? unit : d) * a.n_nodes + j;
  if (j < a.n_nodes && a.radius[node] > 0.0) {
    const double r = a.radius[node];
    const double w = a.weight[node];
    const double x = 2.0 * kPi * r / a.wl[i];
    n = default_n_max(x);
    auto emit = [&](int64_t k, cplx an, cplx bn) {
      const bool odd = (k & 1) != 0;
      const cplx u = odd ? an : bn, v = odd ? bn : an;
      *reinterpret_cast<double4*>(Xk(k - 1)) = make_double4(u.re, u.im, v.re, v.im);
      cm[0] = fmax(cm[0], fabs(u.re));
      cm[1] = fmax(cm[1], fabs(u.im));
      cm[2] = fmax(cm[2], fabs(v.re));
      cm[3] = fmax(cm[3], fabs(v.im));
    };
    ValueSums vs;
    double asum = 0.0;
    int st;
    if (!kLayered) {
      const double2 mv = a.m[unit];
      const cplx m = mk(mv.x, mv.y);
      st = check_node(x, m, n, a.allow_unvalidated != 0);
      if (st == 0 && n <= nc) {
        mie_prepare(x, m, n, s);
        asum = mie_finish(x, m, n, s, vs, emit);
      }
    } else {
      // A layered sphere: x_l = f_l x, the outer surface's x last (ensemble/particle.rs:186-195).
      const int L = kL > 1 ? kL : a.n_layers;
      double xs[kL > 1 ? kL : kMaxLayers];
      cplx ms[kL > 1 ? kL : kMaxLayers];
      bool lossless = true;
#pragma unroll
      for (int l = 0; l < L; ++l) {
        xs[l] = l < L - 1 ? a.fractions[d * (L - 1) + l] * x : x;
        const double2 mv = a.m_layers[(d * L + l) * a.n_wl + i];
        ms[l] = mk(mv.x, mv.y);
        lossless = lossless && mv.y == 0.0;
      }
      st = check_layered(xs, ms, L, n, a.allow_unvalidated != 0);
      if (st == 0 && n <= nc) {
        mie_prepare(x, ms[L - 1], n, s);
        const LayerArrays arr{s.uz, (int64_t)(nc + 2) * 32, 32};
        if constexpr (kL > 1) {
          lfix::LayeredT<kL, -1> lay;
          lay.arr.arr = arr;
          lay.prepare(n, xs, ms);
          asum = mie_finish(x, ms[L - 1], n, s, vs, emit, lay);
        } else {
          Layered lay;
          lay.layers = L;
          lay.x = xs;
          lay.m = ms;
          lay.arr = arr;
          lay.prepare(n);
          asum = mie_finish(x, ms[L - 1], n, s, vs, emit, lay);
        }
        // A lossless particle absorbs nothing (layered/kernel.rs:455-464).
        if (lossless) asum = 0.0;
      }
    }
    if (st != 0 || n > nc) {
      record_error(a.err, i, d, j, a.n_dist, a.n_nodes, st != 0 ? st : 1);
      n = 0;
    } else {
      const Eff e = efficiencies_from(x, asum, vs);
      // The per-particle quantities of pass 2 (engine.rs:1047-1057), weighted.
      const double area = kPi * r * r;
      const double qv[8] = {1.0,           area * e.q_ext, area * e.q_sca, area * e.q_sca * e.g,
                            area * e.q_abs, area * e.q_back, r * r,         r * r * r};
      for (int k = 0; k < 8; ++k) q[k] = w * qv[k];
      sc = 4.0 / (x * x) * (kPi * r * r);
      wv = w;
      if constexpr (kAdaptive) {
        wd = a.wdiff[node];
        for (int k = 0; k < 8; ++k) qe[k] = wd * qv[k];
      }
    }
  }
  put_side(a, chunk, lane, sc, &wv, kAdaptive ? &wd : nullptr, 0, n);
  // Orders above the node's own N are zero up to the chunk's, rounded up to the GEMM's 4.
  const int nc4 = (nc + 3) & ~3;
  for (int64_t k = n + 1; k <= nc4; ++k)
    *reinterpret_cast<double4*>(Xk(k - 1)) = make_double4(0.0, 0.0, 0.0, 0.0);
  if (a.colmax != nullptr)
    *reinterpret_cast<double4*>(a.colmax + (int64_t)chunk * 128 + lane * 4) =
        make_double4(cm[0], cm[1], cm[2], cm[3]);
  put_sums<kAdaptive>(a, chunk, lane, q, qe);
}

// One chunk of homogeneous spheres by the kSplitWarps warps of a block. The serial recurrences run side
// by side: warp 0 the downward u_k(mx), warp 1 the downward u_k(x) and the upward psi, chi (to order
// floor(x)) and xi ratios beyond, which leave each order's factors in its coefficient row (4 doubles a
// node) and a scratch row (1/xi). The orders are then independent: each warp takes a run of them and
// overwrites the rows with the coefficients, in the operations of mie_finish, and leaves each order's
// terms of the sums. Last, warp 0 adds the terms up over the orders, in the order of ValueSums and
// mie_finish, so that every result has the bits of a warp on its own (mie_chunk).
//
// Bound by the recurrences' latency (a complex reciprocal per order): on its own a warp takes about
// 2000 cycles per order, this block about 550.
constexpr int kSplitWarps = 8;
template <bool kAdaptive>
__device__ __forceinline__ void mie_split_chunk(const MieFixedArgs& a, int chunk, int64_t scratch) {
  constexpr int kW = kSplitWarps;
  __shared__ double part[4][kW][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t unit = a.units[chunk / a.cpu];
  const int c = chunk % a.cpu;
  const int64_t d = unit / a.n_wl, i = unit % a.n_wl;
  const int j = c * 32 + lane;
  const int nc = a.chunk_n[chunk], nc4 = (nc + 3) & ~3;
  const int64_t row0 = a.chunk_row[chunk];
  auto Xk = [&](int64_t k) { return a.X + (row0 + k) * 128 + ((lane ^ (int)(k & 3)) << 2); };
  // Scratch rows: u_k(mx) and u_k(x); 1/xi_k, later an order's terms of the sums (absorption, own and
  // pair terms of g, sca; back).
  Scratch s;
  s.uz = a.uz + (row0 + 2 * (int64_t)chunk) * 32 + lane;
  s.ux = a.ux + (row0 + 2 * (int64_t)chunk) * 32 + lane;
  s.stride = 32;
  double4* terms = a.split_rows + scratch * 64 + lane;
  const int64_t node = (a.per_unit ? unit : d) * a.n_nodes + j;
  const double r = j < a.n_nodes ? a.radius[node] : 0.0;
  const double2 mv = a.m[unit];
  const cplx m = mk(mv.x, mv.y);
  double x = 0.0;
  int64_t n = 0, n_s = 0;
  if (r > 0.0) {
    x = 2.0 * kPi * r / a.wl[i];
    n = default_n_max(x);
    int st = check_node(x, m, n, a.allow_unvalidated != 0);
    if (st == 0 && n > nc) st = 1;
    if (st != 0) {
      if (warp == 0) record_error(a.err, i, d, j, a.n_dist, a.n_nodes, st);
      n = 0;
    } else {
      n_s = upward_orders(x, n);
    }
  }
  const double inv_x = 1.0 / x;
  if (n > 0 && warp == 0) {
    mie_prepare_z(x, m, n, s);
  } else if (n > 0 && warp == 1) {
    mie_prepare_x(x, n, s);
    double sin_x, cos_x;
    sincos(x, &sin_x, &cos_x);
    double psi_prev = cos_x, psi = sin_x;
    double chi_prev = -sin_x, chi = cos_x;
    cplx t = rl(0.0), inv_xi = rl(0.0), rr = rl(0.0);
    if (n_s == 0) {
      cplx xi0 = mk(sin_x, -cos_x);
      t = rl(sin_x) * cinv(xi0);
      inv_xi = mk(sin_x, cos_x);
      rr = mk(0.0, 1.0);
    }
    for (int64_t k = 1; k <= n_s; ++k) {
      const double cc = (double)(2 * k - 1) * inv_x;
      const double psi_next = cc * psi - psi_prev;
      psi_prev = psi;
      psi = psi_next;
      const double chi_next = cc * chi - chi_prev;
      chi_prev = chi;
      chi = chi_next;
      *reinterpret_cast<double4*>(Xk(k - 1)) = make_double4(psi, chi, psi_prev, chi_prev);
    }
    if (n_s > 0) {
      const cplx xi = mk(psi, -chi);
      inv_xi = cinv(xi);
      t = rl(psi) * inv_xi;
      rr = mk(psi_prev, -chi_prev) * inv_xi;
    }
    for (int64_t k = n_s + 1; k <= n; ++k) {
      rr = cinv(rl((double)(2 * k - 1) * inv_x) - rr);
      t = scl(t * rr, s.get_x(k));
      inv_xi = inv_xi * rr;
      *reinterpret_cast<double4*>(Xk(k - 1)) = make_double4(rr.re, rr.im, t.re, t.im);
      terms[k * 64] = make_double4(inv_xi.re, inv_xi.im, 0.0, 0.0);
    }
  }
  __syncthreads();
  const int run = (nc + kW - 1) / kW;
  const int64_t k_lo = 1 + (int64_t)warp * run, k_hi = min((int64_t)(warp + 1) * run, (int64_t)nc);
  double cm[4] = {0.0, 0.0, 0.0, 0.0};
  cplx a_prev = rl(0.0), b_prev = rl(0.0);
  if (n > 0) {
    const cplx inv_z = cinv(scl(m, x)), inv_m = cinv(m), inv_m2 = inv_m * inv_m;
    const cplx c_a = -((m - rl(1.0)) * (m + rl(1.0)) * inv_m2);
    const int64_t last = min(k_hi, n);
    for (int64_t k = k_lo; k <= last; ++k) {
      const double4 f = *reinterpret_cast<const double4*>(Xk(k - 1));
      const double k_x = (double)k * inv_x;
      const cplx u_z1 = s.get_z(k + 1);
      const cplx dl = scl(inv_z, (double)(k + 1)) - u_z1;
      const cplx d_m = dl * inv_m, md = dl * m;
      const cplx big_a = d_m + rl(k_x), big_b = md + rl(k_x);
      cplx an, bn, inv_da, inv_db;
      if (k <= n_s) {
        const double psi = f.x, psi_prev = f.z;
        const cplx xi = mk(psi, -f.y), xi_prev = mk(psi_prev, -f.w);
        inv_da = cinv(big_a * xi - xi_prev);
        inv_db = cinv(big_b * xi - xi_prev);
        an = (scl(big_a, psi) - rl(psi_prev)) * inv_da;
        bn = (scl(big_b, psi) - rl(psi_prev)) * inv_db;
      } else {
        const cplx rr = mk(f.x, f.y), t = mk(f.z, f.w);
        const double4 iv = terms[k * 64];
        const cplx inv_xi = mk(iv.x, iv.y);
        const cplx u_x1 = rl(s.get_x(k + 1));
        const cplx num_a = scl(c_a, (double)(k + 1) * inv_x) + u_x1 - u_z1 * inv_m;
        const cplx num_b = u_x1 - m * u_z1;
        const cplx ia = cinv(big_a - rr), ib = cinv(big_b - rr);
        an = t * num_a * ia;
        bn = t * num_b * ib;
        inv_da = inv_xi * ia;
        inv_db = inv_xi * ib;
      }
      const bool odd = (k & 1) != 0;
      const cplx u = odd ? an : bn, v = odd ? bn : an;
      *reinterpret_cast<double4*>(Xk(k - 1)) = make_double4(u.re, u.im, v.re, v.im);
      cm[0] = fmax(cm[0], fabs(u.re));
      cm[1] = fmax(cm[1], fabs(u.im));
      cm[2] = fmax(cm[2], fabs(v.re));
      cm[3] = fmax(cm[3], fabs(v.im));
      const double kf = (double)k, w = (double)(2 * k + 1);
      // The terms of ValueSums::add, the pair term of orders k - 1 and k at order k (that of a run's
      // first order follows below).
      const double kp = kf - 1.0;
      const double pair = k > k_lo ? kp * (kp + 2.0) / (kp + 1.0) * (re_mul_conj(a_prev, an) +
                                                                     re_mul_conj(b_prev, bn))
                                   : 0.0;
      const cplx tb = scl(an - bn, w);
      terms[k * 64] = make_double4(w * (-(d_m.im * nsq(inv_da)) - md.im * nsq(inv_db)),
                                   w / (kf * (kf + 1.0)) * re_mul_conj(an, bn), pair,
                                   w * (nsq(an) + nsq(bn)));
      terms[k * 64 + 32] = odd ? make_double4(-tb.re, -tb.im, 0.0, 0.0)
                               : make_double4(tb.re, tb.im, 0.0, 0.0);
      a_prev = an;
      b_prev = bn;
    }
  }
  // Orders above the node's own N are zero up to the chunk's, rounded up to the GEMM's 4.
  const int64_t z_hi = warp == kW - 1 ? (int64_t)nc4 : k_hi;
  for (int64_t k = max(n + 1, min(k_lo, (int64_t)nc + 1)); k <= z_hi; ++k)
    *reinterpret_cast<double4*>(Xk(k - 1)) = make_double4(0.0, 0.0, 0.0, 0.0);
#pragma unroll
  for (int k = 0; k < 4; ++k) part[k][warp][lane] = cm[k];
  __syncthreads();
  if (warp != 0) return;
  // The pair terms at the runs' first orders.
  for (int w = 1; w < kW; ++w) {
    const int64_t k = 1 + (int64_t)w * run;
    if (k > n) break;
    const double4 p = *reinterpret_cast<const double4*>(Xk(k - 2));
    const double4 q = *reinterpret_cast<const double4*>(Xk(k - 1));
    // The rows hold (a, b) at odd and (b, a) at even orders.
    const cplx p0 = mk(p.x, p.y), p1 = mk(p.z, p.w), q0 = mk(q.x, q.y), q1 = mk(q.z, q.w);
    const bool odd = (k & 1) != 0;
    const double kp = (double)(k - 1);
    terms[k * 64].z = kp * (kp + 2.0) / (kp + 1.0) *
                      (re_mul_conj(odd ? p1 : p0, odd ? q0 : q1) +
                       re_mul_conj(odd ? p0 : p1, odd ? q1 : q0));
  }
  ValueSums vs;
  double asum = 0.0, own = 0.0;
#pragma unroll 4
  for (int64_t k = 1; k <= n; ++k) {
    const double4 p = terms[k * 64], q = terms[k * 64 + 32];
    if (k > 1) {
      vs.g += p.z;
      vs.g += own;
    }
    own = p.y;
    asum += p.x;
    vs.sca += p.w;
    vs.back = vs.back + mk(q.x, q.y);
  }
  if (n > 0) vs.g += own;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    cm[k] = part[k][0][lane];
    for (int w = 1; w < kW; ++w) cm[k] = fmax(cm[k], part[k][w][lane]);
  }
  double q[8] = {0, 0, 0, 0, 0, 0, 0, 0}, qe[kAdaptive ? 8 : 1] = {};
  double sc = 0.0, wv = 0.0, wd = 0.0;
  if (n > 0) {
    const Eff e = efficiencies_from(x, asum, vs);
    const double area = kPi * r * r;
    const double qv[8] = {1.0,           area * e.q_ext, area * e.q_sca, area * e.q_sca * e.g,
                          area * e.q_abs, area * e.q_back, r * r,         r * r * r};
    wv = a.weight[node];
    sc = 4.0 / (x * x) * area;
    for (int k = 0; k < 8; ++k) q[k] = wv * qv[k];
    if constexpr (kAdaptive) {
      wd = a.wdiff[node];
      for (int k = 0; k < 8; ++k) qe[k] = wd * qv[k];
    }
  }
  put_side(a, chunk, lane, sc, &wv, kAdaptive ? &wd : nullptr, 0, n);
  if (a.colmax != nullptr)
    *reinterpret_cast<double4*>(a.colmax + (int64_t)chunk * 128 + lane * 4) =
        make_double4(cm[0], cm[1], cm[2], cm[3]);
  put_sums<kAdaptive>(a, chunk, lane, q, qe);
}

// Homogeneous spheres with the derivatives along the distribution's parameters and m. The
// chunk's coefficient rows are two halves of 16 nodes, nc rows each (lanes 0-15, then 16-31);
// a row holds the 16 nodes' (u, v) in its first 64 doubles and their derivatives along m,
// (du/dm, dv/dm), in the last 64, so that one 128-column GEMM tile carries both. The chunk's
// sums are per block: values, then each parameter of the distribution (weights
// w_j (du/dtheta)(r_j) r_j), then Re m and Im m (engine.rs:1047-1109).
__device__ __forceinline__ void mie_chunk_deriv(const MieFixedArgs& a) {
  int wslot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (wslot >= a.n_chunks) return;
  int chunk = wslot;
  int64_t unit = a.units[chunk / a.cpu];
  int c = chunk % a.cpu;
  int64_t d = unit / a.n_wl, i = unit % a.n_wl;
  int j = c * 32 + lane;
  int nc = a.chunk_n[chunk];
  int64_t row0 = a.chunk_row[chunk];
  const int nc4 = (nc + 3) & ~3;  // rows of a half, rounded up to the GEMM's 4
  auto Xk = [&](int64_t k) {
    return a.X + (row0 + (int64_t)(lane >> 4) * nc4 + k) * 128 +
           (((lane & 15) ^ (int)(k & 3)) << 2);
  };
  Scratch s;
  s.uz = a.uz + (row0 + 2 * (int64_t)chunk) * 32 + lane;
  s.ux = a.ux + (row0 + 2 * (int64_t)chunk) * 32 + lane;
  s.stride = 32;
  const int P = a.n_theta;
  const int B = 3 + P;
  // The node's quantities, their derivatives along Re m and Im m, and the blocks' weights
  // (adaptive: and their error weights (w_K - w_G) ...).
  double qv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  double qd[2][8] = {{0, 0, 0, 0, 0, 0, 0, 0}, {0, 0, 0, 0, 0, 0, 0, 0}};
  double wb[4] = {0, 0, 0, 0}, wbd[4] = {0, 0, 0, 0};  // values, then each parameter
  double sc = 0.0;
  const bool adaptive = a.wdiff != nullptr;
  int64_t n = 0;
  const int64_t node = (a.per_unit ? unit : d) * a.n_nodes + j;
  if (j < a.n_nodes && a.radius[node] > 0.0) {
    const double r = a.radius[node];
    const double x = 2.0 * kPi * r / a.wl[i];
    n = default_n_max(x);
    ValueSums vs;
    DerivSums ds;
    MDeriv md;
    md.along_x = a.deriv_dir == 1;  // the x pass: derivatives along x at fixed m
    const double2 mv = a.m[unit];
    const cplx m = mk(mv.x, mv.y);
    const int st = check_node(x, m, n, a.allow_unvalidated != 0);
    double asum = 0.0;
    if (st == 0 && n <= nc) {
      mie_prepare(x, m, n, s);
      NoLayers none;
      auto emit = [&](int64_t k, cplx an, cplx bn, cplx dan, cplx dbn) {
        const bool odd = (k & 1) != 0;
        const cplx u = odd ? an : bn, v = odd ? bn : an;
        const cplx du = odd ? dan : dbn, dv = odd ? dbn : dan;
        double* x = Xk(k - 1);
        *reinterpret_cast<double4*>(x) = make_double4(u.re, u.im, v.re, v.im);
        *reinterpret_cast<double4*>(x + 64) =
            make_double4(du.re, du.im, dv.re, dv.im);
        ds.add(k, an, bn, dan, dbn);
      };
      asum = mie_finish(x, m, n, s, vs, emit, none, &md);
      ds.close(n);
    }
    if (st != 0 || n > nc) {
      record_error(a.err, i, d, j, a.n_dist, a.n_nodes, st != 0 ? st : 1);
      n = 0;
    } else {
      const Eff e = efficiencies_from(x, asum, vs);
      const double area = kPi * r * r;
      const double q0[8] = {1.0,           area * e.q_ext, area * e.q_sca, area * e.q_sca * e.g,
                            area * e.q_abs, area * e.q_back, r * r,         r * r * r};
      for (int k = 0; k < 8; ++k) qv[k] = q0[k];
      for (int p = 0; p < 2; ++p) {
        const Eff de = efficiency_derivs(x, vs, e, ds, p,
                                         p == 0 ? (md.along_x ? md.abs_x : md.abs_re) : md.abs_im);
        const double q1[8] = {0.0,
                              area * de.q_ext,
                              area * de.q_sca,
                              area * (de.q_sca * e.g + e.q_sca * de.g),
                              area * de.q_abs,
                              area * de.q_back,
                              0.0,
                              0.0};
        for (int k = 0; k < 8; ++k) qd[p][k] = q1[k];
      }
      sc = 4.0 / (x * x) * (kPi * r * r);
      wb[0] = a.weight[node];
      for (int p = 0; p < P; ++p) wb[1 + p] = a.wtheta[node * 3 + p];
      if (adaptive) {
        wbd[0] = a.wdiff[node];
        for (int p = 0; p < P; ++p) wbd[1 + p] = a.wthdiff[node * 3 + p];
      }
    }
  }
  put_side(a, chunk, lane, sc, wb, adaptive ? wbd : nullptr, P, n);
  for (int64_t k = n + 1; k <= nc4; ++k) {
    double* x = Xk(k - 1);
    *reinterpret_cast<double4*>(x) = make_double4(0.0, 0.0, 0.0, 0.0);
    *reinterpret_cast<double4*>(x + 64) = make_double4(0.0, 0.0, 0.0, 0.0);
  }
  // Per block: the values and each parameter weight the node's quantities, Re m and Im m
  // weight its derivatives with the values' weight. The chunk's sums in a fixed tree order;
  // adaptive: then |Kronrod - Gauss| of each of the chunk's two panels (lanes 0-15, 16-31),
  // added.
  const int stride = adaptive ? 2 * B : B;
  for (int b = 0; b < B; ++b) {
    const int wi = b <= P ? b : 0;
    for (int k = 0; k < 8; ++k) {
      const double qk = b <= P ? qv[k] : qd[b - 1 - P][k];
      double v = wb[wi] * qk;
      for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
      if (lane == 0) a.chunk_sums[((int64_t)chunk * stride + b) * 8 + k] = v;
      if (adaptive) {
        double e = wbd[wi] * qk;
        for (int off = 8; off > 0; off >>= 1) e += __shfl_xor_sync(0xffffffffu, e, off);
        const double other = __shfl_sync(0xffffffffu, e, 16);
        if (lane == 0)
          a.chunk_sums[((int64_t)chunk * stride + B + b) * 8 + k] = fabs(e) + fabs(other);
      }
    }
  }
}

// Homogeneous spheres, a chunk per warp. 16 warps per SM (128 registers): the recurrences are
// latency-bound, and they hide more of it than 12 (160 registers) did: 54.4 -> 49.7 ms per step of the
// batched workload (20 warps, 96 registers: 60.5 ms); adaptive panels 7.8 -> 5.1 ms on 16 lognormals x
// 256 wavelengths.
template <bool kAdaptive>
__global__ void __launch_bounds__(128, 4) mie_fixed_kernel(MieFixedArgs a) {
  const int chunk = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (chunk < a.n_chunks) mie_chunk<1, kAdaptive>(a, chunk);
}

// A chunk per block, the longest first, where a slab has too few chunks for their latency to hide
// (run_fixed): a warp's chunk of 750 orders takes 1.6 ms on its own. 96 units of droplets to 1800
// orders 1.93 -> 0.98 ms, 165 units to 170 orders 251 -> 126 us, 3 units 49 -> 21 us. Full slabs lose:
// the chunks take twice the SMs' time (64 x 512 units 24 -> 48 ms), and splitting only the longest
// beside the others gained nothing on 2048 units to 750 orders.
template <bool kAdaptive>
__global__ void __launch_bounds__(32 * kSplitWarps, 2) mie_split_kernel(MieFixedArgs a) {
  const MieSplit b = a.split_list[blockIdx.x];
  mie_split_chunk<kAdaptive>(a, b.chunk, b.row);
}

// Homogeneous spheres with derivatives.
__global__ void __launch_bounds__(128) mie_deriv_kernel(MieFixedArgs a) { mie_chunk_deriv(a); }

// Layered spheres with derivatives along one parameter direction (a.deriv_dir: 0..L-1 the
// complex derivative along layer l's index, then L..2L-2 along the fraction f_{l-L}): the same
// row layout and chunk sums as mie_chunk_deriv, the blocks "Re" and "Im" being the derivative
// along the direction and along i times it (meaningful for the index directions only).
// Scratch per chunk: 2 (2L - 1) arrays (the ratios and their derivatives) of nc + 2 rows.
// kL: 2 or 3 layers and the direction kDir known at compile time (layered_fixed.cuh); 0: any.
template <int kCap, int kL = 0, int kDir = 0>
__device__ __forceinline__ void layered_deriv_chunk(const MieFixedArgs& a) {
  int wslot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (wslot >= a.n_chunks) return;
  int chunk = wslot;
  int64_t unit = a.units[chunk / a.cpu];
  int c = chunk % a.cpu;
  int64_t d = unit / a.n_wl, i = unit % a.n_wl;
  int j = c * 32 + lane;
  int nc = a.chunk_n[chunk];
  int64_t row0 = a.chunk_row[chunk];
  const int nc4 = (nc + 3) & ~3;  // rows of a half, rounded up to the GEMM's 4
  auto Xk = [&](int64_t k) {
    return a.X + (row0 + (int64_t)(lane >> 4) * nc4 + k) * 128 +
           (((lane & 15) ^ (int)(k & 3)) << 2);
  };
  const int L = kL > 0 ? kL : a.n_layers, n_arr = 2 * L - 1;
  Scratch s;
  s.uz = a.uz + (row0 + 2 * (int64_t)chunk) * (2 * n_arr) * 32 + lane;
  s.ux = a.ux + (row0 + 2 * (int64_t)chunk) * 32 + lane;
  s.stride = 32;
  const int P = a.n_theta;
  const int B = 3 + P;
  // The node's quantities, their derivatives along the direction and along i times it, and
  // the blocks' weights (adaptive panels: and their error weights, as mie_chunk_deriv's).
  double qv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  double qd[2][8] = {{0, 0, 0, 0, 0, 0, 0, 0}, {0, 0, 0, 0, 0, 0, 0, 0}};
  double wb[4] = {0, 0, 0, 0}, wbd[4] = {0, 0, 0, 0};
  double sc = 0.0;
  const bool adaptive = a.wdiff != nullptr;
  int64_t n = 0;
  const int64_t node = (a.per_unit ? unit : d) * a.n_nodes + j;
  if (j < a.n_nodes && a.radius[node] > 0.0) {
    const double r = a.radius[node];
    const double x = 2.0 * kPi * r / a.wl[i];
    n = default_n_max(x);
    double xs[kCap];
    cplx ms[kCap];
    lder::DR xd[kCap];
    lder::DC md[kCap];
    bool lossless = true;
    const int dir = kL > 0 ? kDir : a.deriv_dir;
#pragma unroll
    for (int l = 0; l < L; ++l) {
      xs[l] = l < L - 1 ? a.fractions[d * (L - 1) + l] * x : x;
      const double2 mv = a.m_layers[(d * L + l) * a.n_wl + i];
      ms[l] = mk(mv.x, mv.y);
      lossless = lossless && mv.y == 0.0;
      xd[l] = lder::DR{xs[l], dir >= L && l == dir - L ? x : 0.0};
      md[l] = lder::DC{ms[l], rl(dir == l ? 1.0 : 0.0)};
    }
    const int st = check_layered(xs, ms, L, n, a.allow_unvalidated != 0);
    double asum = 0.0, abs_d[2] = {0.0, 0.0};
    ValueSums vs;
    DerivSums ds;
    if (st == 0 && n <= nc) {
      mie_prepare(x, ms[L - 1], n, s);  // u_k(x); array 0 is redone with its derivatives
      const LayerArrays arr{s.uz, (int64_t)(nc + 2) * 32, 32};
      auto emit = [&](int64_t k, cplx an, cplx bn, cplx dan, cplx dbn) {
        const bool odd = (k & 1) != 0;
        const cplx u = odd ? an : bn, v = odd ? bn : an;
        const cplx du = odd ? dan : dbn, dv = odd ? dbn : dan;
        double* x = Xk(k - 1);
        *reinterpret_cast<double4*>(x) = make_double4(u.re, u.im, v.re, v.im);
        *reinterpret_cast<double4*>(x + 64) =
            make_double4(du.re, du.im, dv.re, dv.im);
        ds.add(k, an, bn, dan, dbn);
      };
      if constexpr (kL > 0) {
        lfix::LayeredT<kL, kDir> lay;
        lay.arr.arr = arr;
        lay.prepare(n, xs, ms);
        asum = lfix::finish(x, ms[kL - 1], n, s, vs, emit, lay, abs_d);
      } else {
        lder::LayeredD<kCap> lay;
        lay.layers = L;
        lay.x = xd;
        lay.m = md;
        lay.arr.arr = arr;
        lay.arr.n_val = n_arr;
        lay.prepare(n, lder::DR{x, 0.0});
        asum = lder::layered_finish_d(x, md[L - 1], n, s, vs, emit, lay, abs_d);
      }
      ds.close(n);
      // A lossless particle absorbs nothing (layered/kernel.rs:455-464); its derivatives stand.
      if (lossless) asum = 0.0;
    }
    if (st != 0 || n > nc) {
      record_error(a.err, i, d, j, a.n_dist, a.n_nodes, st != 0 ? st : 1);
      n = 0;
    } else {
      const Eff e = efficiencies_from(x, asum, vs);
      const double area = kPi * r * r;
      const double q0[8] = {1.0,           area * e.q_ext, area * e.q_sca, area * e.q_sca * e.g,
                            area * e.q_abs, area * e.q_back, r * r,         r * r * r};
      for (int k = 0; k < 8; ++k) qv[k] = q0[k];
      for (int p = 0; p < 2; ++p) {
        const Eff de = efficiency_derivs(x, vs, e, ds, p, abs_d[p]);
        const double q1[8] = {0.0,
                              area * de.q_ext,
                              area * de.q_sca,
                              area * (de.q_sca * e.g + e.q_sca * de.g),
                              area * de.q_abs,
                              area * de.q_back,
                              0.0,
                              0.0};
        for (int k = 0; k < 8; ++k) qd[p][k] = q1[k];
      }
      sc = 4.0 / (x * x) * (kPi * r * r);
      wb[0] = a.weight[node];
      for (int p = 0; p < P; ++p) wb[1 + p] = a.wtheta[node * 3 + p];
      if (adaptive) {
        wbd[0] = a.wdiff[node];
        for (int p = 0; p < P; ++p) wbd[1 + p] = a.wthdiff[node * 3 + p];
      }
    }
  }
  put_side(a, chunk, lane, sc, wb, adaptive ? wbd : nullptr, P, n);
  for (int64_t k = n + 1; k <= nc4; ++k) {
    double* x = Xk(k - 1);
    *reinterpret_cast<double4*>(x) = make_double4(0.0, 0.0, 0.0, 0.0);
    *reinterpret_cast<double4*>(x + 64) = make_double4(0.0, 0.0, 0.0, 0.0);
  }
  // The chunk's sums per block (values and each parameter on the values' quantities, the
  // direction's blocks on the derivatives with the values' weight) in a fixed tree order;
  // adaptive: then |Kronrod - Gauss| of each of the chunk's two panels, added.
  const int stride = adaptive ? 2 * B : B;
  for (int b = 0; b < B; ++b) {
    const int wi = b <= P ? b : 0;
    for (int k = 0; k < 8; ++k) {
      const double qk = b <= P ? qv[k] : qd[b - 1 - P][k];
      double v = wb[wi] * qk;
      for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
      if (lane == 0) a.chunk_sums[((int64_t)chunk * stride + b) * 8 + k] = v;
      if (adaptive) {
        double e = wbd[wi] * qk;
        for (int off = 8; off > 0; off >>= 1) e += __shfl_xor_sync(0xffffffffu, e, off);
        const double other = __shfl_sync(0xffffffffu, e, 16);
        if (lane == 0)
          a.chunk_sums[((int64_t)chunk * stride + B + b) * 8 + k] = fabs(e) + fabs(other);
      }
    }
  }
}

// Up to 4 layers with the per-shell state sized for them; more through the general form.
__global__ void __launch_bounds__(128) mie_layered_deriv_kernel(MieFixedArgs a) {
  layered_deriv_chunk<4>(a);
}
__global__ void __launch_bounds__(128) mie_layered_deriv16_kernel(MieFixedArgs a) {
  layered_deriv_chunk<kMaxLayers>(a);
}

// 2 or 3 layers along one direction known at compile time.
template <int kL, int kDir>
__global__ void __launch_bounds__(128) mie_layered_deriv_fixed_kernel(MieFixedArgs a) {
  layered_deriv_chunk<kL, kL, kDir>(a);
}

// Layered spheres: 2 to 4 layers with their state in registers, more in local memory.
template <int kL, bool kAdaptive>
__global__ void __launch_bounds__(128, 3) mie_layered_kernel(MieFixedArgs a) {
  const int chunk = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (chunk < a.n_chunks) mie_chunk<kL, kAdaptive>(a, chunk);
}

// Independent spheres, one per thread (the batched Mie::compute): coefficients a_1..a_N then
// b_1..b_N per sphere, and the efficiencies.
__global__ void __launch_bounds__(128) mie_nodes_kernel(MieNodesArgs a) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n) return;
  double x = a.x[t];
  cplx m = mk(a.m[t].x, a.m[t].y);
  int64_t n = default_n_max(x);
  int st = check_node(x, m, n, a.allow_unvalidated != 0);
  if (st != 0) {
    unsigned long long key = ((unsigned long long)t << 2) | (unsigned long long)st;
    atomicMin(a.err, key);
    return;
  }
  if (a.n_terms) a.n_terms[t] = n;
  if (!a.coeffs) return;
  int64_t off = a.coeff_offset[t];
  Scratch s;
  s.uz = a.uz + off + 2 * t;
  s.ux = a.ux + off + 2 * t;
  s.stride = 1;
  mie_prepare(x, m, n, s);
  ValueSums vs;
  double2* out = reinterpret_cast<double2*>(a.coeffs) + 2 * off;
  double asum = mie_finish(x, m, n, s, vs, [&](int64_t k, cplx an, cplx bn) {
    out[k - 1] = make_double2(an.re, an.im);
    out[n + k - 1] = make_double2(bn.re, bn.im);
  });
  Eff e = efficiencies_from(x, asum, vs);
  if (a.eff) {
    a.eff[5 * t] = e.q_ext;
    a.eff[5 * t + 1] = e.q_sca;
    a.eff[5 * t + 2] = e.q_abs;
    a.eff[5 * t + 3] = e.q_back;
    a.eff[5 * t + 4] = e.g;
  }
}

// Pass 1 of the adaptive ensemble: one thread per node (engine.rs:369-449 quantities1 for
// spheres). Scratch rows scratch[t]..scratch[t+1]-1 hold u_k(mx) and u_k(x); a node whose
// number of terms does not fit them reports status 1 (the host sizes them from the same
// truncation rule with a margin).
__global__ void __launch_bounds__(128) pass1_kernel(Pass1Args a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n) return;
  const double r = a.radius[t];
  const int wi = a.wl_index[t];
  const double x = 2.0 * kPi * r / a.wl[wi];
  int64_t n = default_n_max(x);
  const int L = a.n_layers > 1 ? a.n_layers : 1;
  double xs[kMaxLayers];
  cplx ms[kMaxLayers];
  bool lossless = true;
  int st;
  if (L == 1) {
    ms[0] = mk(a.m[wi].x, a.m[wi].y);
    st = check_node(x, ms[0], n, a.allow_unvalidated != 0);
  } else {
    // x_l = f_l x, the outer surface's x last (ensemble/particle.rs:186-195).
    const int p = wi / a.n_wl, i = wi % a.n_wl;
    for (int l = 0; l < L; ++l) {
      xs[l] = l < L - 1 ? a.fractions[p * (L - 1) + l] * x : x;
      const double2 mv = a.m_layers[(p * L + l) * a.n_wl + i];
      ms[l] = mk(mv.x, mv.y);
      lossless = lossless && mv.y == 0.0;
    }
    st = check_layered(xs, ms, L, n, a.allow_unvalidated != 0);
  }
  const int64_t off = a.scratch[t], cap = a.scratch[t + 1] - off;
  if (st == 0 && n + 2 > cap) st = 1;
  a.status[t] = st;
  a.n_terms[t] = st == 0 ? n : 0;
  const int nq = a.deriv ? 16 : 6;
  double* q = a.q + nq * t;
  if (st != 0) {
    for (int k = 0; k < nq; ++k) q[k] = 0.0;
    return;
  }
  Scratch s;
  s.uz = a.uz + off * (2 * L - 1);
  s.ux = a.ux + off;
  s.stride = 1;
  mie_prepare(x, ms[L - 1], n, s);
  ValueSums vs;
  double asum;
  if (L == 1 && a.deriv) {
    // The derivatives of the pass-1 quantities along Re m and Im m (engine.rs:447-461).
    DerivSums ds;
    MDeriv md;
    NoLayers none;
    asum = mie_finish(
        x, ms[0], n, s, vs,
        [&](int64_t k, cplx an, cplx bn, cplx dan, cplx dbn) { ds.add(k, an, bn, dan, dbn); },
        none, &md);
    ds.close(n);
    const Eff e = efficiencies_from(x, asum, vs);
    const double area = kPi * r * r;
    for (int p = 0; p < 2; ++p) {
      const Eff d = efficiency_derivs(x, vs, e, ds, p, p == 0 ? md.abs_re : md.abs_im);
      double* o = q + 6 + 5 * p;
      o[0] = area * d.q_ext;
      o[1] = area * d.q_sca;
      o[2] = area * (d.q_sca * e.g + e.q_sca * d.g);
      o[3] = area * d.q_back;
      o[4] = area * d.q_abs;
    }
  } else if (L == 1) {
    asum = mie_finish(x, ms[0], n, s, vs, [](int64_t, cplx, cplx) {});
  } else {
    Layered lay;
    lay.layers = L;
    lay.x = xs;
    lay.m = ms;
    lay.arr.base = s.uz;
    lay.arr.astride = cap;
    lay.arr.stride = 1;
    lay.prepare(n);
    asum = mie_finish(x, ms[L - 1], n, s, vs, [](int64_t, cplx, cplx) {}, lay);
    // A lossless particle absorbs nothing (layered/kernel.rs:455-464).
    if (lossless) asum = 0.0;
  }
  const Eff e = efficiencies_from(x, asum, vs);
  const double area = kPi * r * r;
  q[0] = 1.0;
  q[1] = area * e.q_ext;
  q[2] = area * e.q_sca;
  q[3] = area * e.q_sca * e.g;
  q[4] = area * e.q_back;
  q[5] = area * e.q_abs;
}

// Pass 1 of a layered sphere's derivatives along one direction (engine.rs:447-461 with
// Solved::direction, particle.rs:206-219): one thread per node, the layered recursion in
// forward mode (layered_deriv.cuh) along a.deriv_dir; q[t] gets the node's 6 quantities and
// the derivatives of pi r^2 (Q_ext, Q_sca, Q_sca g, Q_back, Q_abs) along the direction, then
// along i times it (meaningful for an index direction only).
__global__ void __launch_bounds__(128) pass1_layered_deriv_kernel(Pass1Args a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n) return;
  const double r = a.radius[t];
  const int wi = a.wl_index[t];
  const double x = 2.0 * kPi * r / a.wl[wi];
  int64_t n = default_n_max(x);
  const int L = a.n_layers;
  double xs[kMaxLayers];
  cplx ms[kMaxLayers];
  bool lossless = true;
  const int p = wi / a.n_wl, i = wi % a.n_wl;
  for (int l = 0; l < L; ++l) {
    xs[l] = l < L - 1 ? a.fractions[p * (L - 1) + l] * x : x;
    const double2 mv = a.m_layers[(p * L + l) * a.n_wl + i];
    ms[l] = mk(mv.x, mv.y);
    lossless = lossless && mv.y == 0.0;
  }
  int st = check_layered(xs, ms, L, n, a.allow_unvalidated != 0);
  // The derivatives are validated up to x_L = 1000 (layered/domain.rs:39-70).
  if (st == 0 && a.allow_unvalidated == 0 && xs[L - 1] > 1e3) st = 3;
  const int64_t off = a.scratch[t], cap = a.scratch[t + 1] - off;
  if (st == 0 && n + 2 > cap) st = 1;
  a.status[t] = st;
  a.n_terms[t] = st == 0 ? n : 0;
  double* q = a.q + 16 * t;
  if (st != 0) {
    for (int k = 0; k < 16; ++k) q[k] = 0.0;
    return;
  }
  const int n_arr = 2 * L - 1, dir = a.deriv_dir;
  Scratch s;
  s.uz = a.uz + off * (2 * n_arr);
  s.ux = a.ux + off;
  s.stride = 1;
  lder::DR xd[kMaxLayers];
  lder::DC md[kMaxLayers];
  for (int l = 0; l < L; ++l) {
    xd[l] = lder::DR{xs[l], dir >= L && l == dir - L ? x : 0.0};
    md[l] = lder::DC{ms[l], rl(dir == l ? 1.0 : 0.0)};
  }
  mie_prepare(x, ms[L - 1], n, s);  // u_k(x); array 0 is redone with its derivatives
  lder::LayeredD<kMaxLayers> lay;
  lay.layers = L;
  lay.x = xd;
  lay.m = md;
  lay.arr.arr.base = s.uz;
  lay.arr.arr.astride = cap;
  lay.arr.arr.stride = 1;
  lay.arr.n_val = n_arr;
  lay.prepare(n, lder::DR{x, 0.0});
  ValueSums vs;
  DerivSums ds;
  double abs_d[2];
  double asum = lder::layered_finish_d(
      x, md[L - 1], n, s, vs,
      [&](int64_t k, cplx an, cplx bn, cplx dan, cplx dbn) { ds.add(k, an, bn, dan, dbn); }, lay,
      abs_d);
  ds.close(n);
  // A lossless particle absorbs nothing (layered/kernel.rs:455-464); its derivatives stand.
  if (lossless) asum = 0.0;
  const Eff e = efficiencies_from(x, asum, vs);
  const double area = kPi * r * r;
  q[0] = 1.0;
  q[1] = area * e.q_ext;
  q[2] = area * e.q_sca;
  q[3] = area * e.q_sca * e.g;
  q[4] = area * e.q_back;
  q[5] = area * e.q_abs;
  for (int c = 0; c < 2; ++c) {
    const Eff d = efficiency_derivs(x, vs, e, ds, c, abs_d[c]);
    double* o = q + 6 + 5 * c;
    o[0] = area * d.q_ext;
    o[1] = area * d.q_sca;
    o[2] = area * (d.q_sca * e.g + e.q_sca * d.g);
    o[3] = area * d.q_back;
    o[4] = area * d.q_abs;
  }
}

void launch_pass1_layered_deriv(const Pass1Args& a, cudaStream_t s) {
  const int threads = 128;
  const int64_t blocks = (a.n + threads - 1) / threads;
  if (blocks > 0) pass1_layered_deriv_kernel<<<(unsigned)blocks, threads, 0, s>>>(a);
}

void launch_pass1(const Pass1Args& a, cudaStream_t s) {
  const int threads = 128;
  const int64_t blocks = (a.n + threads - 1) / threads;
  if (blocks > 0) pass1_kernel<<<(unsigned)blocks, threads, 0, s>>>(a);
}

void launch_plan_chunks(const PlanArgs& a, cudaStream_t s) {
  int threads = 128;
  int blocks = (int)((a.n_chunks * 32 + threads - 1) / threads);
  plan_chunks_kernel<<<blocks, threads, 0, s>>>(a);
}

void launch_node_table(const NodeTableArgs& a, cudaStream_t s) {
  const int64_t blocks = (16 * a.n_rec + 127) / 128;
  if (blocks > 0) node_table_kernel<<<(unsigned)blocks, 128, 0, s>>>(a);
}

void launch_mie_fixed(const MieFixedArgs& a, cudaStream_t s) {
  int threads = 128;
  int blocks = (a.n_chunks * 32 + threads - 1) / threads;
  const auto run = [&](void (*f)(MieFixedArgs)) { f<<<blocks, threads, 0, s>>>(a); };
  if (a.deriv && a.n_layers > 4) {
    run(mie_layered_deriv16_kernel);
  } else if (a.deriv && a.n_layers == 2) {
    run(a.deriv_dir == 0   ? mie_layered_deriv_fixed_kernel<2, 0>
        : a.deriv_dir == 1 ? mie_layered_deriv_fixed_kernel<2, 1>
                           : mie_layered_deriv_fixed_kernel<2, 2>);
  } else if (a.deriv && a.n_layers == 3) {
    run(a.deriv_dir == 0   ? mie_layered_deriv_fixed_kernel<3, 0>
        : a.deriv_dir == 1 ? mie_layered_deriv_fixed_kernel<3, 1>
        : a.deriv_dir == 2 ? mie_layered_deriv_fixed_kernel<3, 2>
        : a.deriv_dir == 3 ? mie_layered_deriv_fixed_kernel<3, 3>
                           : mie_layered_deriv_fixed_kernel<3, 4>);
  } else if (a.deriv && a.n_layers > 1) {
    run(mie_layered_deriv_kernel);
  } else if (a.deriv) {
    run(mie_deriv_kernel);
  } else if (a.n_layers > 1) {
    const bool ad = a.wdiff != nullptr;
    if (a.n_layers == 2)
      run(ad ? mie_layered_kernel<2, true> : mie_layered_kernel<2, false>);
    else if (a.n_layers == 3)
      run(ad ? mie_layered_kernel<3, true> : mie_layered_kernel<3, false>);
    else if (a.n_layers == 4)
      run(ad ? mie_layered_kernel<4, true> : mie_layered_kernel<4, false>);
    else
      run(ad ? mie_layered_kernel<0, true> : mie_layered_kernel<0, false>);
  } else {
    run(a.wdiff ? mie_fixed_kernel<true> : mie_fixed_kernel<false>);
  }
}

void launch_mie_split(const MieFixedArgs& a, cudaStream_t s) {
  if (a.n_split <= 0) return;
  auto f = a.wdiff ? mie_split_kernel<true> : mie_split_kernel<false>;
  f<<<a.n_split, 32 * kSplitWarps, 0, s>>>(a);
}

void launch_mie_nodes(const MieNodesArgs& a, cudaStream_t s) {
  int threads = 128;
  int blocks = (int)((a.n + threads - 1) / threads);
  mie_nodes_kernel<<<blocks, threads, 0, s>>>(a);
}

}  // namespace sb
