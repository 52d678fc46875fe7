// The phase levels of the fixed grid: the small chunks' phase-matrix elements on a minimal set
// of Gauss nodes, and their interpolation onto the requested cosines.
//
// A chunk's elements (|S1|^2 + |S2|^2 and the others) with at most U orders are polynomials of
// degree <= 2 U in mu, so their values at 2 U + 1 nodes hold everything: the requested cosines'
// values by interpolation and the Greek coefficients by the same nodes' quadrature. Level t has
// U = 32 t - 1 orders and n_q = 64 t - 1 Gauss-Legendre nodes, h = 32 t of them >= 0 (t whole
// 32-row tiles, no padding rows). Where a level has fewer rows than the requested cosines and the
// projector band together, the angle GEMMs run on the level instead, and the unit's sums at its
// nodes (linear over the chunks) are interpolated once per unit (slot_project_kernel). For 360
// cosines and L = 64 a chunk of 48 orders runs 2 tiles of 32 rows instead of 8.
//
// Accuracy: the nodes are held in double-double (one Newton step from the double rule), the
// tables at them are rounded once from a double-double recurrence, and the interpolation is the
// barycentric form with the weights 1 / P_n'(x_k) of the same step. The Lagrange functions of
// Gauss nodes fall off away from a node, so the forward peak's rounding does not reach the backward
// directions: relative to its own value F11 there is 5e-15 off extended precision at x = 30, 3e-14
// at x = 300 (direct sums on tables from double recurrences: 6e-14, 3e-13). That needs the values at
// +mu and -mu kept apart: folded into even and odd parts, which halves the products, a backward
// element is the difference of two sums of the forward peak's size (5e-13, 7e-12). Compiled with
// -fmad=false (double-double).
#include "dd.cuh"
#include "kernels.h"

namespace sb {

using ddm::dd;
using ddm::mkdd;

// One thread per (level, half node): the node in double-double, its barycentric weight, and its
// rows of the G_E, G_O tables.
__global__ void __launch_bounds__(128) level_table_kernel(LevelTableArgs a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n_half) return;
  int lv = 0;
  while (lv + 1 < a.n_levels && a.half0[lv + 1] <= t) ++lv;
  const BandDesc B = a.bands[lv];
  const int i = t - a.half0[lv], n = B.n_q;
  dd x = mkdd(a.x0[t]);
  // P_n and P_{n-1} at the double node; one Newton step, and P_n' there to first order.
  dd p0 = mkdd(1.0), p1 = x;
  for (int k = 2; k <= n; ++k) {
    const dd p2 = ((x * p1) * (double)(2 * k - 1) - p0 * (double)(k - 1)) / (double)k;
    p0 = p1;
    p1 = p2;
  }
  const dd s = mkdd(1.0) - x * x;
  const dd dp = ((p0 - x * p1) * (double)n) / s;
  const dd step = p1 / dp;
  if (i == 0) {
    x = mkdd(0.0);  // the middle node of an odd rule
  } else {
    x = x - step;
  }
  const double dpn = dp.hi * (1.0 - 2.0 * x.hi / s.hi * step.hi);
  a.x_hi[t] = x.hi;
  a.x_lo[t] = x.lo;
  a.bary[t] = 1.0 / dpn;
  // pi_n, tau_n by their three-term recurrence, scaled by (2n + 1) / (n (n + 1)).
  double* tab = a.g + B.g_off;
  dd pi_prev = mkdd(0.0), pi = mkdd(1.0);
  for (int k = 1; k <= B.upper; ++k) {
    const double kf = (double)k, k1 = kf + 1.0;
    const dd mp = x * pi;
    const dd tau = mp * kf - pi_prev * k1;
    const dd wp = (pi * (double)(2 * k + 1)) / (kf * k1);
    const dd wt = (tau * (double)(2 * k + 1)) / (kf * k1);
    const double vp = wp.hi, vt = wt.hi;
    double* o = tab + table_at(i, k - 1, B.ld);
    o[0] = (k & 1) ? vp : vt;
    o[32] = (k & 1) ? vt : vp;
    const dd next = (mp * (double)(2 * k + 1) - pi_prev * k1) / kf;
    pi_prev = pi;
    pi = next;
  }
  // The row past the last order, which a rounded-up contraction meets with zero coefficients.
  double* o = tab + table_at(i, B.upper, B.ld);
  o[0] = o[32] = 0.0;
}

// One thread per (level, requested row): the row's interpolation weights l_k of the level's half
// nodes and l_{-k} of their mirrors (the middle node once). The row -c has the two exchanged, the
// middle node's weight being even in c.
__global__ void __launch_bounds__(128) level_matrix_kernel(LevelMatrixArgs a) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x, lv = blockIdx.y;
  if (r >= a.h_pad) return;
  const int h = a.bands[lv].h, k0 = a.half0[lv];
  const double* xh = a.x_hi + k0;
  const double* xl = a.x_lo + k0;
  const double* v = a.bary + k0;
  double* lp = a.lp + (int64_t)k0 * a.h_pad + r;
  double* lm = a.lm + (int64_t)k0 * a.h_pad + r;
  if (r >= a.h_u) {
    for (int k = 0; k < h; ++k) lp[(int64_t)k * a.h_pad] = lm[(int64_t)k * a.h_pad] = 0.0;
    return;
  }
  const double c = a.rows[r];
  // P_n' is even for the odd n_q, so node -k has node k's weight.
  double sum = 0.0;
  int hit = -1, hit_sign = 1;
  for (int k = 0; k < h; ++k) {
    const double dm = (c - xh[k]) - xl[k], dp = (c + xh[k]) + xl[k];
    if (dm == 0.0) hit = k;
    if (dp == 0.0 && k > 0) {
      hit = k;
      hit_sign = -1;
    }
    if (hit < 0) sum += k == 0 ? v[k] / dm : v[k] / dm + v[k] / dp;
  }
  const double is = hit < 0 ? 1.0 / sum : 0.0;
  for (int k = 0; k < h; ++k) {
    double p, m;
    if (hit >= 0) {
      p = k == hit && hit_sign > 0 ? 1.0 : 0.0;
      m = k == hit && hit_sign < 0 ? 1.0 : 0.0;
    } else {
      const double dm = (c - xh[k]) - xl[k], dp = (c + xh[k]) + xl[k];
      p = (v[k] / dm) * is;
      m = k == 0 ? 0.0 : (v[k] / dp) * is;
    }
    lp[(int64_t)k * a.h_pad] = p;
    lm[(int64_t)k * a.h_pad] = m;
  }
}

// The slots' sums (the fixed grid) onto the requested cosines and the Greek coefficients: two FP64
// GEMMs side by side per tile of 32 output rows and up to 16 slots of one table,
//   the requested cosines (levels): of the 4 elements at the half nodes (F+) and their mirrors (F-),
//     L+ F+ + L- F- at +c and L- F+ + L+ F- at -c;
//   alpha1, alpha4 and beta1, beta2: d00 [F11, F33] and d02 [F12, F34] over the n_q nodes;
//   alpha2, alpha3: d22 (F11 + F33) and d2-2 (F11 - F33); half their sum and difference.
// blockIdx.y runs over the row tiles in that order. Each output is one slot's (final_kernel adds a
// unit's slots in order), so the results do not depend on which slots share a tile.
//
// Bound by latency for a few units (a table's 4 to 100 stages of 8 nodes) and by the FP64 tensor
// path for many (57 % at 96 units x 4096 cosines). One tile per table, not one per unit over all its
// tables, keeps the stages few and the tiles many: 96 units x 4096 cosines 2.54 -> 0.94 ms, 165 units
// x 181 cosines with L = 50 299 -> 55 us (against one launch for the cosines over all of a unit's
// tables and one for the coefficients of 32 slots with a lane per slot); 0.64 ms and 53 us of them
// with the values at +mu and -mu folded, which is not accurate (above).
namespace {
constexpr int IK = 8;    // nodes per stage
constexpr int IG = kSlotGroup;
struct SlotSmem {
  double a[2][2][IK][36];  // [stage][matrix][node][row]
  double b[2][2][IK][68];  // [stage][matrix][node][column]
  int64_t off[IG];
  int reps[IG];
  int slot[IG];
};
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// kType 0: the requested cosines (64 columns: slot, element); 1: d00 and d02 (32 columns: slot,
// F11 or F33 and F12 or F34); 2: d22 and d2-2 (16 columns: slot).
template <int kType>
__device__ __forceinline__ void slot_tile(const SlotArgs& a, SlotSmem& sm, const BandDesc& B,
                                          int level, int count, int r0) {
  constexpr int kCols = kType == 0 ? 64 : (kType == 1 ? 32 : 16), kNt = kCols / 8;
  constexpr int kPer = kCols / 16;  // columns per slot
  const int t = threadIdx.x, w = t >> 5, lane = t & 31, q = lane & 3, g = lane >> 2;
  const int nq = B.n_q, K = kType == 0 ? B.h : nq;
  const int ld = kType == 0 ? a.h_pad : B.d_ld;
  const double* ma;
  const double* mb;
  if (kType == 0) {
    ma = a.lp + (int64_t)a.half0[level] * ld;
    mb = a.lm + (int64_t)a.half0[level] * ld;
  } else {
    const double* D = a.band_d + B.d_off;  // d00, d22, d2-2, d02
    ma = D + (int64_t)(kType == 1 ? 0 : 1) * nq * ld;
    mb = D + (int64_t)(kType == 1 ? 3 : 2) * nq * ld;
  }
  double cA[kNt][2], cB[kNt][2];
#pragma unroll
  for (int nt = 0; nt < kNt; ++nt) cA[nt][0] = cA[nt][1] = cB[nt][0] = cB[nt][1] = 0.0;
  const int n_nt = (count * kPer + 7) / 8;
  // This thread's share of a stage's columns: column col, kN nodes from kh.
  constexpr int kN = IK * kCols / 128;
  const int col = t % kCols, kh = (t / kCols) * kN;
  const int sl = col / kPer;
  const int64_t off = sl < count ? sm.off[sl] : -1;
  const int reps = sl < count ? sm.reps[sl] : 0;
  const int64_t rep_stride = 4 * (int64_t)nq * a.n_blk;
  double f0[kN], f1[kN];
  auto load_a = [&](int st, int k0) {
#pragma unroll
    for (int i = t; i < 2 * IK * 16; i += 128) {
      const int o = i / (IK * 16), kk = (i >> 4) % IK, c = i & 15;
      const bool valid = k0 + kk < K;
      const double* src = (o ? mb : ma) + (valid ? (int64_t)(k0 + kk) * ld + r0 + 2 * c : 0);
      const unsigned d = (unsigned)__cvta_generic_to_shared(&sm.a[st][o][kk][2 * c]);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src),
                   "r"(valid ? 16 : 0));
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  auto load_f = [&](int k0) {
#pragma unroll
    for (int j = 0; j < kN; ++j) f0[j] = f1[j] = 0.0;
    if (off < 0) return;
    const int e = col % kPer;
    for (int r = 0; r < reps; ++r) {
      const double* f = a.acc + off + r * rep_stride;
#pragma unroll
      for (int j = 0; j < kN; ++j) {
        const int k = k0 + kh + j;
        if (kType == 0) {
          // The element at the half node's +mu and -mu.
          f0[j] += f[(int64_t)e * nq + (B.h - 1) + k];
          f1[j] += f[(int64_t)e * nq + (B.h - 1) - k];
        } else if (k < K) {
          // F11 and F33 with d00, F12 and F34 with d02; F11 and F33.
          f0[j] += f[(int64_t)(kType == 1 ? 2 * e : 0) * nq + k];
          f1[j] += f[(int64_t)(kType == 1 ? 2 * e + 1 : 2) * nq + k];
        }
      }
    }
  };
  auto store_f = [&](int st) {
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      sm.b[st][0][kh + j][col] = kType == 2 ? f0[j] + f1[j] : f0[j];
      sm.b[st][1][kh + j][col] = kType == 2 ? f0[j] - f1[j] : f1[j];
    }
  };
  load_a(0, 0);
  load_f(0);
  store_f(0);
  int st = 0;
  for (int k0 = 0; k0 < K; k0 += IK, st ^= 1) {
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    const bool more = k0 + IK < K;
    if (more) {
      load_a(st ^ 1, k0 + IK);
      load_f(k0 + IK);
    }
#pragma unroll
    for (int k4 = 0; k4 < IK; k4 += 4) {
      const double va = sm.a[st][0][k4 + q][8 * w + g], vb = sm.a[st][1][k4 + q][8 * w + g];
#pragma unroll
      for (int nt = 0; nt < kNt; ++nt)
        if (nt < n_nt) {
          const double b0 = sm.b[st][0][k4 + q][8 * nt + g], b1 = sm.b[st][1][k4 + q][8 * nt + g];
          dmma(cA[nt][0], cA[nt][1], va, b0);
          dmma(cB[nt][0], cB[nt][1], vb, kType == 0 ? b0 : b1);
          if (kType == 0) {
            dmma(cA[nt][0], cA[nt][1], vb, b1);
            dmma(cB[nt][0], cB[nt][1], va, b1);
          }
        }
    }
    if (more) store_f(st ^ 1);
  }
  const int row = r0 + 8 * w + g;
  if (kType == 0) {
    if (row >= a.h_u) return;
    const int2 mp = a.user_map[row];
#pragma unroll
    for (int nt = 0; nt < kNt; ++nt) {
      const int s = 2 * nt + (q >> 1), e = 2 * (q & 1);
      if (s >= count) continue;
      double* out = a.slot_phase + (int64_t)sm.slot[s] * 4 * a.n_mu;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        out[(int64_t)(e + j) * a.n_mu + mp.x] = cA[nt][j];
        if (mp.y >= 0) out[(int64_t)(e + j) * a.n_mu + mp.y] = cB[nt][j];
      }
    }
  } else {
    const int glen = a.greek_order + 1;
    if (row > B.order) return;
#pragma unroll
    for (int nt = 0; nt < kNt; ++nt) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int c = 8 * nt + 2 * q + j, s = c / kPer;
        if (s >= count) continue;
        double* out = a.slot_greek + (int64_t)sm.slot[s] * 6 * glen + row;
        if (kType == 1) {
          out[(c & 1) ? 3 * glen : 0] = cA[nt][j];
          out[((c & 1) ? 5 : 4) * glen] = cB[nt][j];
        } else {
          out[glen] = 0.5 * (cA[nt][j] + cB[nt][j]);
          out[2 * glen] = 0.5 * (cA[nt][j] - cB[nt][j]);
        }
      }
    }
  }
}
}  // namespace

__global__ void __launch_bounds__(128, 4) slot_project_kernel(SlotArgs a) {
  extern __shared__ __align__(16) unsigned char slot_raw[];
  SlotSmem& sm = *reinterpret_cast<SlotSmem*>(slot_raw);
  const ProjItem it = a.items[blockIdx.x];
  const BandDesc B = a.bands[it.band];
  const bool level = it.band < a.n_levels;
  const int tu = level ? (a.h_u + 31) / 32 : 0, tg = a.greek_order >= 0 ? B.order / 32 + 1 : 0;
  if ((int)blockIdx.y >= tu + 2 * tg) return;
  if (threadIdx.x < it.count) {
    const int k = a.slot_index[it.first + threadIdx.x];
    const BandSlot s = a.slots[k];
    sm.slot[threadIdx.x] = k;
    sm.off[threadIdx.x] = s.off;
    sm.reps[threadIdx.x] = s.reps;
  }
  // A block per tile; beyond the grid's 65,535 rows (2^21 cosines) a block takes several.
  for (int tile = blockIdx.y; tile < tu + 2 * tg; tile += gridDim.y) {
    __syncthreads();
    if (tile < tu)
      slot_tile<0>(a, sm, B, it.band, it.count, 32 * tile);
    else if (tile < tu + tg)
      slot_tile<1>(a, sm, B, it.band, it.count, 32 * (tile - tu));
    else
      slot_tile<2>(a, sm, B, it.band, it.count, 32 * (tile - tu - tg));
  }
}

void launch_level_tables(const LevelTableArgs& a, cudaStream_t s) {
  if (a.n_half > 0) level_table_kernel<<<(a.n_half + 127) / 128, 128, 0, s>>>(a);
}

void launch_level_matrices(const LevelMatrixArgs& a, cudaStream_t s) {
  if (a.n_levels > 0 && a.h_u > 0)
    level_matrix_kernel<<<dim3((a.h_pad + 127) / 128, a.n_levels), 128, 0, s>>>(a);
}

cudaError_t launch_slot_project(const SlotArgs& a, int max_tiles, cudaStream_t s) {
  if (a.n_items <= 0 || max_tiles <= 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(
      slot_project_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SlotSmem));
  if (e != cudaSuccess) return e;
  slot_project_kernel<<<dim3((unsigned)a.n_items, (unsigned)(max_tiles < 65535 ? max_tiles : 65535)),
                        128, sizeof(SlotSmem), s>>>(a);
  return cudaGetLastError();
}

}  // namespace sb
