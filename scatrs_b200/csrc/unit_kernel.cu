// K-b, K-c and K-d: persistent CTAs work through shares of (distribution, wavelength) units, each in a
// fixed order, so the sums are deterministic.
//
// Per unit, per chunk of 32 nodes (ascending radius):
//   * K-b: S1, S2 of the chunk's 32 spheres at the table cosines as real FP64 GEMMs,
//     C_E = G_E X and C_O = G_O X (scatrs/src/ensemble/fast.rs:141-145), against the shared
//     pi/tau tables of the requested cosines and of the chunk's projector band;
//   * K-c: the phase-matrix elements at mu and at -mu (fast.rs:151-204), scaled per sphere and
//     weighted by w_j u(r_j) r_j, summed over the chunk into the unit's accumulators;
//   * K-d: the tables projected onto the Greek coefficients with (2l+1)/2 w_k d_l(mu_k)
//     (fast.rs:238-253, engine.rs:2310-2355): here for adaptive calls, on the fixed grid in
//     slot_project_kernel (phase_levels.cu).
// Then the averages and the outputs of engine.rs:2396-2497.
#include "kernels.h"
#include "mbar.cuh"

namespace sb {

namespace {

constexpr double kPi = 3.14159265358979323846264338327950288;
constexpr int KB = 8;     // orders per stage
constexpr int TR = 32;    // table rows per tile
constexpr int NT = 128;   // threads: 4 warps of 8 rows x 128 columns
constexpr int NS = 4;     // stages in flight (5: the same)
constexpr int RING = 8;   // job records: more than the stages, so none is overwritten in use

// One tile of one chunk (or half chunk, with derivatives) as every warp sees it.
struct Job {
  int end;    // no more work
  int rows4;  // orders, rounded up to the MMA's 4
  int r0, h;  // the tile's first table row; the table's rows
  int user;   // the requested cosines' table (outputs by user_map), else a band's or level's
  int len;    // outputs per element: n_mu or n_q
  int half;
  int64_t out;  // the sums' offset in acc
};

// kNw: weights per node (UnitArgs::side): values; then the parameters'; then the error weights.
template <int kNw>
struct UnitSmem {
  double a[NS][KB][kTableRow];  // [stage][order][G_E rows, G_O rows] (table_at)
  double xs[NS][KB][128];       // [stage][order][32 nodes x 4 columns]
  double side[RING][32 * kNw + 4];
  Job job[RING];
  unsigned long long full[NS], empty[NS];
  int abort;
  // The producer (warp 0): the item's next chunks with work for it, and its place among them.
  struct {
    int first_tile, tiles, t_user, rows4, h, n_q, ld;
    int64_t row, acc, ci;
    const double* g;
  } chunk[32];
  struct {
    int unit, group, n_groups, chunk0, n_chunks, c, tile, half, rows4, k0, next_item;
    int64_t user_acc;
    const double *g, *x, *side;
  } p;
};

// D (8x8) += A (8x4, row) B (4x8, col) in FP64 on the tensor cores (PTX mma.sync m8n8k4):
// lane l holds A[l/4][l%4], B[l%4][l/4] and D[l/4][2 (l%4) + {0, 1}].
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

__device__ __forceinline__ double swap_add(double v, int lane_bit) {
  return v + __shfl_xor_sync(0xffffffffu, v, lane_bit);
}

// The producer's next work item (its counter is taken one item ahead, so that only the item's chunks
// are waited for), then the records of its next 32 chunks: one lane per chunk, the chunks with rows
// for this item kept in order. Returns false when no item is left.
template <class Smem>
__device__ __forceinline__ bool next_chunks(const UnitArgs& a, Smem& sm) {
  auto& p = sm.p;
  const int lane = threadIdx.x & 31;
  for (;;) {
    int c0 = p.chunk0 + 32;
    __syncwarp();
    if (c0 >= a.cpu) {
      const int slot = p.next_item;
      if (slot >= a.n_items) return false;
      const WorkItem it = a.items[slot];
      __syncwarp();
      if (lane == 0) {
        p.next_item = atomicAdd(a.work_counter, 1);
        p.unit = it.unit;
        p.group = it.group;
        p.n_groups = it.n_groups;
        p.user_acc = a.unit_acc[it.unit];
      }
      c0 = 0;
      __syncwarp();
    }
    const int c = c0 + lane;
    bool on = c < a.cpu;
    const int64_t ci = (int64_t)p.unit * a.cpu + (on ? c : 0);
    const int nc = on ? a.chunk_n[ci] : 0;
    const int64_t row = a.chunk_row[ci], band_acc = a.chunk_acc[ci];
    // The int8 path's chunks are not this kernel's.
    on = on && nc > 0 && !(a.i8_above > 0 && nc > a.i8_above && nc <= kI8MaxTerms);
    int t_user = 0, tiles = 0, tile0 = 0;
    BandDesc B{};
    const double* g = nullptr;
    if (on) {
      const int b = chunk_band(nc, a.merge_max, a.n_levels, a.greek_order);
      t_user = nc <= a.merge_max ? 0 : (a.h_u + TR - 1) / TR;
      if (b >= 0) {
        B = a.bands[b];
        g = (b < a.n_levels ? a.level_g : a.band_g) + B.g_off;
      }
      tiles = t_user + (b >= 0 ? (B.h + TR - 1) / TR : 0);
      // This item's first tile; a level's tiles move on by one item per run of chunks.
      const int shift = nc <= a.merge_max ? (c / kRunChunks) % p.n_groups : 0;
      tile0 = p.group >= shift ? p.group - shift : p.group - shift + p.n_groups;
      on = tile0 < tiles;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, on);
    if (on) {
      auto& r = sm.chunk[__popc(mask & ((1u << lane) - 1))];
      r.first_tile = tile0;
      r.tiles = tiles;
      r.t_user = t_user;
      r.rows4 = (nc + 3) & ~3;
      r.h = B.h;
      r.n_q = B.n_q;
      r.ld = B.ld;
      r.row = row;
      r.acc = band_acc;
      r.ci = ci;
      r.g = g;
    }
    if (lane == 0) {
      p.chunk0 = c0;
      p.n_chunks = __popc(mask);
      p.c = 0;
    }
    __syncwarp();
    if (mask != 0) return true;
  }
}

// Moves the producer to its next job (warp 0): the halves of a tile, the tiles of a chunk, the
// chunks of a work item, the items in the order of the counter. Fills the job's record.
template <int kMode, class Smem>
__device__ __forceinline__ bool next_job(const UnitArgs& a, Smem& sm, int job) {
  constexpr int kHalves = (kMode == 1 || kMode == 3) ? 2 : 1;
  auto& p = sm.p;
  const int lane = threadIdx.x & 31;
  int c = p.c, half = p.half + 1, tile = p.tile;
  bool found = c < p.n_chunks;
  if (found && half >= kHalves) {
    half = 0;
    tile += p.n_groups;
    found = tile < sm.chunk[c].tiles;
  }
  if (!found) {
    if (++c >= p.n_chunks) {
      __syncwarp();
      if (!next_chunks(a, sm)) return false;
      c = 0;
    }
    half = 0;
    tile = sm.chunk[c].first_tile;
  }
  __syncwarp();
  if (lane == 0) {
    const auto& r = sm.chunk[c];
    const bool user = tile < r.t_user;
    const int tl = user ? tile : tile - r.t_user;
    p.c = c;
    p.half = half;
    p.tile = tile;
    p.rows4 = r.rows4;
    p.k0 = 0;
    p.g = (user ? a.g_u : r.g) + (int64_t)tl * (user ? a.ld_u : r.ld) * kTableRow;
    p.x = a.X + (r.row + (int64_t)half * r.rows4) * 128;
    p.side = a.side + r.ci * a.side_stride;
    Job& jb = sm.job[job % RING];
    jb.end = 0;
    jb.rows4 = r.rows4;
    jb.r0 = TR * tl;
    jb.h = user ? a.h_u : r.h;
    jb.user = user;
    jb.len = user ? a.n_mu : r.n_q;
    jb.half = half;
    jb.out = user ? p.user_acc : r.acc;
  }
  __syncwarp();
  return true;
}

// Where warp 0 is in producing (the same in its lanes): the next stage and job, the stages of the job
// still to issue, and whether the end has been issued.
struct Producer {
  int stage = 0, job = -1, left = 0;
  bool done = false;
};

// Warp 0 issues one stage: up to KB orders of the table's tile and of the chunk's coefficient rows,
// a bulk copy each, and with a job's first stage its weights. (A copy per row, 24 a stage, was
// bound by the copies' issue: 168 against 105 ms of the two-barrier cp.async form before, per pass
// of 64 x 512 units.) Stages run on across jobs, so the pipeline does not drain between tiles or
// chunks.
template <int kMode, class Smem>
__device__ __forceinline__ void issue_stage(const UnitArgs& a, Smem& sm, Producer& pr) {
  auto& p = sm.p;
  const int lane = threadIdx.x & 31, slot = pr.stage % NS;
  bool first = false;
  if (pr.left == 0) {
    ++pr.job;
    first = next_job<kMode>(a, sm, pr.job);
    if (!first) {
      if (lane == 0) {
        sm.job[pr.job % RING].end = 1;
        mbar_arrive(&sm.full[slot]);
      }
      pr.done = true;
      ++pr.stage;
      return;
    }
    pr.left = (p.rows4 + KB - 1) / KB;
  }
  if (lane == 0) {
    const int k0 = p.k0, rows = min(KB, p.rows4 - k0);
    const uint32_t side_bytes = first ? (uint32_t)a.side_stride * 8 : 0;
    mbar_expect_tx(&sm.full[slot], (uint32_t)rows * (128 + kTableRow) * 8 + side_bytes);
    bulk_load(sm.xs[slot], p.x + (int64_t)k0 * 128, rows * 1024, &sm.full[slot]);
    bulk_load(sm.a[slot], p.g + (int64_t)k0 * kTableRow, rows * kTableRow * 8, &sm.full[slot]);
    if (first) bulk_load(sm.side[pr.job % RING], p.side, side_bytes, &sm.full[slot]);
    p.k0 = k0 + KB;
  }
  --pr.left;
  ++pr.stage;
}

// Issues every stage whose buffer is free, up to NS ahead of stage `it`, and waits (bounded) only for
// the next one that warp 0 itself needs.
template <int kMode, class Smem>
__device__ __forceinline__ bool produce(const UnitArgs& a, Smem& sm, Producer& pr, int it) {
  while (!pr.done && pr.stage < it + NS) {
    if (pr.stage >= NS) {
      unsigned long long* e = &sm.empty[pr.stage % NS];
      const uint32_t parity = ((pr.stage / NS) - 1) & 1;
      const bool free = __shfl_sync(0xffffffffu, (int)mbar_done(e, parity), 0);
      if (!free) {
        if (pr.stage > it) return true;
        if (!mbar_wait(e, parity, sm, a.wait_err)) return false;
      }
    }
    issue_stage<kMode>(a, sm, pr);
  }
  return true;
}

// The sums over a job's nodes, for the lane's row (g) and column nodes 4 j + q of tile pairs j: the
// D fragments of tiles 2 j and 2 j + 1 hold (u.re, v.re) and (u.im, v.im) of one node in one
// thread, so that S1 = E_u +- O_v, S2 = E_v +- O_u (fast.rs:151-204) need no exchange.
struct Amp {
  double s1r, s1i, s2r, s2i;
};
__device__ __forceinline__ Amp amplitudes(const double (&cE)[16][2], const double (&cO)[16][2],
                                          int j, double sg) {
  return Amp{fma(sg, cO[2 * j][1], cE[2 * j][0]), fma(sg, cO[2 * j + 1][1], cE[2 * j + 1][0]),
             fma(sg, cO[2 * j][0], cE[2 * j][1]), fma(sg, cO[2 * j + 1][0], cE[2 * j + 1][1])};
}
// p += f (|S1|^2, |S2|^2, Re S2 S1*, Im S2 S1*) (scatrs/src/mie/phase.rs:54-59).
__device__ __forceinline__ void add_elements(double p[4], const Amp& s, double f) {
  const double t1r = f * s.s1r, t1i = f * s.s1i, t2r = f * s.s2r, t2i = f * s.s2i;
  p[0] = fma(t1r, s.s1r, fma(t1i, s.s1i, p[0]));
  p[1] = fma(t2r, s.s2r, fma(t2i, s.s2i, p[1]));
  p[2] = fma(t2r, s.s1r, fma(t2i, s.s1i, p[2]));
  p[3] = fma(t2i, s.s1r, fma(-t2r, s.s1i, p[3]));
}
// The four lanes of a row add up; lane q ends with element q (F11, F12, F33, F34) from the sums of
// (|S1|^2, |S2|^2) times c and the other two.
__device__ __forceinline__ double reduce_elements(const double p[4], double c) {
  const int q = threadIdx.x & 3;
  const bool hi = q & 2;
  double a0 = hi ? p[2] : p[0], a1 = hi ? p[3] : p[1];
  a0 += __shfl_xor_sync(0xffffffffu, hi ? p[0] : p[2], 2);
  a1 += __shfl_xor_sync(0xffffffffu, hi ? p[1] : p[3], 2);
  a0 = swap_add(a0, 1);
  a1 = swap_add(a1, 1);
  return hi ? (q & 1 ? a1 : a0) : c * (q & 1 ? a1 - a0 : a0 + a1);
}

// kMode 0: values; 1: with the derivative blocks; 2: adaptive panels (values and the sums of
// |Kronrod - Gauss| per panel); 3: adaptive panels with the derivative blocks (each block's sums,
// then its error sums: every 16-node half of a chunk is one panel).
template <int kMode, int kNw>
__device__ __forceinline__ void unit_body(const UnitArgs& a) {
  constexpr bool kDeriv = kMode == 1 || kMode == 3;
  using Smem = UnitSmem<kNw>;
  extern __shared__ __align__(16) unsigned char unit_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(unit_raw);
  const int t = threadIdx.x, w = t >> 5, lane = t & 31, q = lane & 3, g = lane >> 2;
  if (t == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], NT / 32);
    }
    sm.abort = 0;
    sm.p.chunk0 = a.cpu;  // no item yet
    sm.p.n_chunks = sm.p.c = sm.p.half = sm.p.tile = 0;
    sm.p.next_item = atomicAdd(a.work_counter, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  bool ok = true;
  Producer pr;
  if (w == 0) ok = produce<kMode>(a, sm, pr, 0);
  int it = 0;
  for (int job = 0; ok; ++job) {
    if (!mbar_wait(&sm.full[it % NS], (it / NS) & 1, sm, a.wait_err)) break;
    const Job jb = sm.job[job % RING];
    if (jb.end) break;
    const double* side = sm.side[job % RING];
    // The rows move round the warps from tile to tile (a row always with the same warp, which owns its
    // sums); a warp without rows only counts the stages.
    const int rg = (w + jb.r0 / TR) & 3, row0 = jb.r0 + 8 * rg;
    const bool active = row0 < jb.h;
    int gmax[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      gmax[i] = active ? (int)side[a.side_stride - 4 + (kDeriv ? 2 * jb.half + (i & 1) : i)] : 0;
    double cE[16][2], cO[16][2];
#pragma unroll
    for (int nt = 0; nt < 16; ++nt) cE[nt][0] = cE[nt][1] = cO[nt][0] = cO[nt][1] = 0.0;
    for (int k0 = 0; k0 < jb.rows4; k0 += KB, ++it) {
      if (k0 > 0 && !(ok = mbar_wait(&sm.full[it % NS], (it / NS) & 1, sm, a.wait_err))) break;
      const int st = it % NS;
#pragma unroll
      for (int k4 = 0; k4 < KB; k4 += 4) {
        if (k0 + k4 >= jb.rows4) break;
        const int kk = k4 + q;
        const int r = (8 * rg + g) ^ (4 * q);
        const double aE = sm.a[st][kk][r], aO = sm.a[st][kk][32 + r];
#pragma unroll
        for (int gr = 0; gr < 4; ++gr) {
          if (k0 + k4 < gmax[gr]) {
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
              const int j = 2 * gr + jj;
              const double2 b = *reinterpret_cast<const double2*>(
                  &sm.xs[st][kk][16 * j + 4 * ((g >> 1) ^ q) + 2 * (g & 1)]);
              dmma(cE[2 * j][0], cE[2 * j][1], aE, b.x);
              dmma(cE[2 * j + 1][0], cE[2 * j + 1][1], aE, b.y);
              dmma(cO[2 * j][0], cO[2 * j][1], aO, b.x);
              dmma(cO[2 * j + 1][0], cO[2 * j + 1][1], aO, b.y);
            }
          }
        }
      }
      warp_arrive(&sm.empty[st]);
      if (w == 0 && !(ok = produce<kMode>(a, sm, pr, it + 1))) break;
    }
    if (!ok) break;
    if (!active) continue;
    // Where this lane's sums go: row row0 + g at +mu and -mu.
    const int row = row0 + g;
    int at[2] = {-1, -1};
    if (row < jb.h) {
      if (jb.user) {
        const int2 mp = a.user_map[row];
        at[0] = mp.x;
        at[1] = mp.y;
      } else {
        at[0] = jb.len / 2 + row;
        at[1] = jb.len - 1 - at[0];
        if (at[1] == at[0]) at[1] = -1;
      }
    }
    double* out = a.acc + jb.out;
    if constexpr (kMode == 0) {
      double p[2][4] = {};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const double f = side[4 * j + q];
        add_elements(p[0], amplitudes(cE, cO, j, 1.0), f);
        add_elements(p[1], amplitudes(cE, cO, j, -1.0), f);
      }
      // Reductions without a reply: a thread's adds to one sum stay in its program order, and no
      // other thread adds to it while the kernel runs.
#pragma unroll
      for (int sd = 0; sd < 2; ++sd) {
        const double v = reduce_elements(p[sd], 0.5);
        if (at[sd] >= 0) atomicAdd(out + (int64_t)q * jb.len + at[sd], v);
      }
    } else if constexpr (kMode == 2) {
#pragma unroll 1
      for (int sd = 0; sd < 2; ++sd) {
        const double sg = sd ? -1.0 : 1.0;
        double p[4] = {}, e[2][4] = {};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const Amp s = amplitudes(cE, cO, j, sg);
          add_elements(p, s, side[4 * j + q]);
          add_elements(e[j >> 2], s, side[32 + 4 * j + q]);  // panel A: nodes 0-15, B: 16-31
        }
        const double v = reduce_elements(p, 0.5);
        const double ve = fabs(reduce_elements(e[0], 0.5)) + fabs(reduce_elements(e[1], 0.5));
        if (at[sd] >= 0) {
          double* o = out + (int64_t)q * jb.len + at[sd];
          atomicAdd(o, v);
          atomicAdd(o + (int64_t)4 * jb.len, ve);
        }
      }
    } else {
      // The half's 16 nodes: pairs 0-3 their (u, v) sums, pairs 4-7 those of (du/dm, dv/dm).
      // Blocks: values, the parameters (the elements by their weights), Re m and Im m (the element
      // derivatives along dS/dm and i dS/dm; phase.rs:62-73, 322-335), by the values' weight.
      const int n_blk = 3 + a.n_theta;
#pragma unroll 1
      for (int pass = 0; pass < (kMode == 3 ? 4 : 2); ++pass) {
        const int sd = pass & 1, err = pass >> 1;
        const double sg = sd ? -1.0 : 1.0;
        const double* wt = side + err * 32 * (1 + a.n_theta) + 16 * jb.half + q;
        double p[4][4] = {}, d[2][4] = {};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const Amp s = amplitudes(cE, cO, j, sg), ds = amplitudes(cE, cO, j + 4, sg);
          const double f = wt[4 * j];
          add_elements(p[0], s, f);
#pragma unroll
          for (int b = 1; b < 4; ++b)
            if (b <= a.n_theta) add_elements(p[b], s, wt[32 * b + 4 * j]);
          const double t1r = f * s.s1r, t1i = f * s.s1i, t2r = f * s.s2r, t2i = f * s.s2i;
          d[0][0] = fma(t1r, ds.s1r, fma(t1i, ds.s1i, d[0][0]));
          d[0][1] = fma(t2r, ds.s2r, fma(t2i, ds.s2i, d[0][1]));
          d[0][2] = fma(t1r, ds.s2r, fma(t1i, ds.s2i, fma(t2r, ds.s1r, fma(t2i, ds.s1i, d[0][2]))));
          d[0][3] = fma(t1r, ds.s2i, fma(-t1i, ds.s2r, fma(t2i, ds.s1r, fma(-t2r, ds.s1i, d[0][3]))));
          // Along i dS: (re, im) -> (-im, re).
          d[1][0] = fma(-t1r, ds.s1i, fma(t1i, ds.s1r, d[1][0]));
          d[1][1] = fma(-t2r, ds.s2i, fma(t2i, ds.s2r, d[1][1]));
          d[1][2] = fma(-t1r, ds.s2i, fma(t1i, ds.s2r, fma(-t2r, ds.s1i, fma(t2i, ds.s1r, d[1][2]))));
          d[1][3] = fma(t1r, ds.s2r, fma(t1i, ds.s2i, fma(-t2i, ds.s1i, fma(-t2r, ds.s1r, d[1][3]))));
        }
        auto emit = [&](int blk, const double (&v)[4], double c) {
          double x = reduce_elements(v, c);
          if (err) x = fabs(x);
          if (at[sd] >= 0)
            atomicAdd(out + ((int64_t)(err * n_blk + blk) * 4 + q) * jb.len + at[sd], x);
        };
        emit(0, p[0], 0.5);
#pragma unroll
        for (int b = 1; b < 4; ++b)
          if (b <= a.n_theta) emit(b, p[b], 0.5);
        emit(1 + a.n_theta, d[0], 1.0);
        emit(2 + a.n_theta, d[1], 1.0);
      }
    }
  }
  // A warp that gave up leaves stages in flight: they land before the CTA exits.
  if (*(volatile int*)&sm.abort && w == 0 && lane == 0)
    for (int s = pr.stage > NS ? pr.stage - NS : 0; s < pr.stage; ++s)
      mbar_wait_drain(&sm.full[s % NS], (s / NS) & 1, a.wait_err);
  __syncthreads();
}

}  // namespace

// K-b and K-c: persistent CTAs work through items (a unit and a share of its row tiles). A tile is 32
// table rows x the chunk's 128 coefficient columns: C_E = G_E X and C_O = G_O X on the FP64 MMA
// (mma.sync m8n8k4 f64; tcgen05 has no FP64 kind), each warp 8 rows x all columns, the MMAs of a
// group of 8 nodes stopping above its largest number of terms. Bulk copies into four stages of 8
// orders, issued by warp 0 and waited for on mbarriers, run on across tiles and chunks; the warps
// meet at no barrier, so a warp in its epilogue leaves the FP64 path to the others. Every output sum
// is owned by one thread of one work item and runs over the chunks in order, so the results do not
// depend on how a unit's tiles are split into items.
//
// Bound by the FP64 tensor path (71 to 76 % busy): the algorithmic operations of a pass of 64 x 512
// units of 512 nodes at 29 TFLOP/s, 0.82 of the DGEMM rate (100 ms; 105 with cp.async stages behind block barriers, which drained at every chunk).
// The derivative and adaptive forms ran on scalar FMAs with a 16-lane reduce-scatter per block of
// sums: 1.10 -> 0.69 ms (768 units, 5 blocks) and 10.5 -> 5.9 ms (1024 units).
__global__ void __launch_bounds__(NT, 3) unit_kernel(UnitArgs a) { unit_body<0, 1>(a); }

// With the derivative blocks: per chunk its two 16-node halves, values and derivative columns in
// one tile.
__global__ void __launch_bounds__(NT, 2) unit_deriv_kernel(UnitArgs a) { unit_body<1, 4>(a); }

// Adaptive panels: per tile the values' sums and the sums of |Kronrod - Gauss| per panel.
__global__ void __launch_bounds__(NT, 2) unit_adaptive_kernel(UnitArgs a) { unit_body<2, 2>(a); }

// Adaptive panels with the derivative blocks: per tile every block's sums and error sums.
__global__ void __launch_bounds__(NT, 2) unit_adaptive_deriv_kernel(UnitArgs a) {
  unit_body<3, 8>(a);
}

// K-d: the Greek coefficients of each band slot, (2l+1)/2 sum_k w_k F(mu_k) d_l(mu_k) with F
// the slot's averaged tables (fast.rs:238-253): a contraction over the band's n_q nodes shared
// by a tile of up to 32 slots. Lane s of each warp holds slot s; warp w the orders
// l0 + 9w + j (j < 9) of each block of 72 orders. The sums over k run in node order.
namespace {
constexpr int PQ = 32;   // nodes per stage
constexpr int PT = 256;  // threads
constexpr int PL = 72;   // orders per pass: 8 warps x 9
struct ProjSmem {
  double fs[4][PQ][33];  // F11, F12, F33, F34 per node and slot (padded against conflicts)
  double ds[4][PQ][PL];  // d00, d22, d2-2, d02 (scaled) per node and order
  double z[32], ez[32], tr[32];  // adaptive: Z, its error, the truncation term
  double dz[32], edz[32];        // adaptive derivatives: the slot's Z_p and its error
  int blk[32];                   // adaptive derivatives: the slot's block
  int64_t offs[32];
};
}  // namespace

// An adaptive call's table element o of slot s along its block b (engine.rs:1782-1836): the
// part's average (values) or its first-order error estimate (bounds), from the block's sums
// and error sums and the values' (a unit's slots per band: B value slots, then B error slots,
// 4 n_q doubles each). v = S_0/Z, e = (E_0 + |v| e_Z)/Z + t |v|; a parameter p:
// dv = (S_p - v Z_p)/Z, (E_p + |v| e_Zp + |dv| e_Z + e |Z_p|)/Z + t |dv|; along m: dv = S_m/Z,
// (E_m + |dv| e_Z)/Z + t |dv|.
__device__ __forceinline__ double ad_table(const ProjArgs& a, const ProjSmem& sm, int s,
                                           int64_t o, int q, bool bounds) {
  const int b = sm.blk[s], B = a.ad_blocks;
  const int64_t q4 = 4 * (int64_t)q;
  const double z = sm.z[s], ez = sm.ez[s], tr = sm.tr[s], dz = sm.dz[s], edz = sm.edz[s];
  if (!bounds) {
    const double v0 = a.acc[o - b * q4] / z;
    if (b == 0) return v0;
    if (b <= a.n_theta) return (a.acc[o] - v0 * dz) / z;
    return a.acc[o] / z;
  }
  const double v0 = a.acc[o - (B + b) * q4] / z, av0 = fabs(v0);
  const double e0 = (a.acc[o - b * q4] + av0 * ez) / z + tr * av0;
  if (b == 0) return e0;
  const double sb = a.acc[o - B * q4], eb = a.acc[o];
  if (b <= a.n_theta) {
    const double dv = (sb - v0 * dz) / z;
    return (eb + av0 * edz + fabs(dv) * ez + e0 * fabs(dz)) / z + tr * fabs(dv);
  }
  const double dv = sb / z;
  return (eb + fabs(dv) * ez) / z + tr * fabs(dv);
}

__global__ void __launch_bounds__(PT) proj_kernel(ProjArgs a) {
  extern __shared__ __align__(16) unsigned char proj_raw[];
  ProjSmem& sm = *reinterpret_cast<ProjSmem*>(proj_raw);
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int glen = a.greek_order + 1;
  for (int item = blockIdx.x; item < a.n_items; item += gridDim.x) {
    const ProjItem it = a.items[item];
    const BandDesc B = a.bands[it.band];
    const int q = B.n_q, len = B.order + 1;
    const bool bounds = it.kind == 1;
    if (t < 32) {
      int64_t off = -1;
      if (t < it.count) {
        const BandSlot bs = a.slots[a.slot_index[it.first + t]];
        const int stride = a.ad_blocks > 0 ? kNormStrideD : 8;
        const double* un = a.unit_norm + stride * (int64_t)a.units[bs.unit];
        sm.z[t] = un[0];
        sm.ez[t] = un[1];
        sm.tr[t] = un[2];
        if (a.ad_blocks > 0) {
          const int b = bs.pad, p = b - 1;
          sm.blk[t] = b;
          sm.dz[t] = (b >= 1 && b <= a.n_theta) ? un[8 + p] : 0.0;
          sm.edz[t] = (b >= 1 && b <= a.n_theta) ? un[11 + p] : 0.0;
        }
        off = bs.off;
      }
      sm.offs[t] = off;
    }
    __syncthreads();
    const double* D = a.band_d + B.d_off;
    for (int l0 = 0; l0 < len; l0 += PL) {
      double acc[9][6];
#pragma unroll
      for (int j = 0; j < 9; ++j)
#pragma unroll
        for (int e = 0; e < 6; ++e) acc[j][e] = 0.0;
      for (int k0 = 0; k0 < q; k0 += PQ) {
        const int kn = q - k0 < PQ ? q - k0 : PQ;
        // The averaged tables (S/Z) of the 32 slots at nodes k0..k0+kn-1; node fastest, so
        // each slot's run is one coalesced read.
        for (int idx = t; idx < 4 * 32 * PQ; idx += PT) {
          const int kk = idx % PQ, s = (idx / PQ) & 31, e = idx / (32 * PQ);
          double v = 0.0;
          const int64_t off = sm.offs[s];
          if (kk < kn && off >= 0) {
            const int64_t o = off + (int64_t)e * q + k0 + kk;
            if (a.ad_blocks > 0) {
              v = ad_table(a, sm, s, o, q, bounds);
            } else if (!bounds) {
              v = a.acc[o] / sm.z[s];
            } else {
              // The error sums of the slot after the values' (engine.rs:1782-1800).
              const double av = fabs(a.acc[o - 4 * (int64_t)q] / sm.z[s]);
              v = (a.acc[o] + av * sm.ez[s]) / sm.z[s] + sm.tr[s] * av;
            }
          }
          sm.fs[e][kk][s] = v;
        }
        for (int idx = t; idx < 4 * PQ * PL; idx += PT) {
          const int l = idx % PL, kk = (idx / PL) % PQ, m = idx / (PL * PQ);
          double v = 0.0;
          if (kk < kn && l0 + l < len) v = D[((int64_t)m * q + k0 + kk) * B.d_ld + l0 + l];
          sm.ds[m][kk][l] = bounds ? fabs(v) : v;
        }
        __syncthreads();
        for (int kk = 0; kk < kn; ++kk) {
          const double f11 = sm.fs[0][kk][lane], f12 = sm.fs[1][kk][lane];
          const double f33 = sm.fs[2][kk][lane], f34 = sm.fs[3][kk][lane];
          // Bounds: alpha2 and alpha3 share the half sum of the bounds of alpha2 +- alpha3
          // (fast.rs:256-271).
          const double fp = f11 + f33, fm = bounds ? fp : f11 - f33;
#pragma unroll
          for (int j = 0; j < 9; ++j) {
            const int l = 9 * w + j;
            const double d00 = sm.ds[0][kk][l], d22 = sm.ds[1][kk][l];
            const double d2m2 = sm.ds[2][kk][l], d02 = sm.ds[3][kk][l];
            acc[j][0] = fma(f11, d00, acc[j][0]);
            acc[j][1] = fma(f33, d00, acc[j][1]);
            acc[j][2] = fma(fp, d22, acc[j][2]);
            acc[j][3] = fma(fm, d2m2, acc[j][3]);
            acc[j][4] = fma(f12, d02, acc[j][4]);
            acc[j][5] = fma(f34, d02, acc[j][5]);
          }
        }
        __syncthreads();
      }
      if (lane < it.count) {
        double* out = a.slot_greek + (int64_t)a.slot_index[it.first + lane] * 6 * glen;
#pragma unroll
        for (int j = 0; j < 9; ++j) {
          const int l = l0 + 9 * w + j;
          if (l < len) {
            const double p = acc[j][2], mi = acc[j][3];
            out[l] = acc[j][0];
            out[glen + l] = (p + mi) * 0.5;
            out[2 * glen + l] = bounds ? (p + mi) * 0.5 : (p - mi) * 0.5;
            out[3 * glen + l] = acc[j][1];
            out[4 * glen + l] = acc[j][4];
            out[5 * glen + l] = acc[j][5];
          }
        }
      }
    }
    __syncthreads();
  }
}

// The outputs per unit: the averages S/Z (engine.rs:1782-1836), the Greek coefficients summed
// over the unit's band slots in increasing band order (engine.rs:2310-2355), and the assembly
// of engine.rs:2396-2497.
__global__ void __launch_bounds__(NT) final_kernel(FinalArgs a) {
  __shared__ double S[8];
  __shared__ double a0s;
  const int t = threadIdx.x;
  const int L = a.greek_order;
  const int glen = L >= 0 ? L + 1 : 0;
  const int64_t nu = a.n_units_total;
  for (int ul = blockIdx.x; ul < a.n_units; ul += gridDim.x) {
    const int64_t unit = a.units[ul];
    const int64_t d = unit / a.n_wl, i = unit % a.n_wl;
    if (t < 8) {
      double s = 0.0;
      for (int c = 0; c < a.cpu; ++c) s += a.chunk_sums[((int64_t)ul * a.cpu + c) * 8 + t];
      S[t] = s;
    }
    __syncthreads();
    const double z = S[0];
    const double* acc_user = a.acc + a.unit_acc[ul];
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = S[k] / z;
    const double ext = v[1], sca = v[2], scag = v[3], ab = v[4], back = v[5], r2 = v[6],
                 r3 = v[7];
    if (t == 0) {
      const bool bext = !(isfinite(ext) && ext != 0.0), bsca = !(isfinite(sca) && sca != 0.0);
      const bool bback = !(isfinite(back) && back != 0.0);
      if (bext || bsca || bback) {
        unsigned long long key = ((unsigned long long)(i * a.n_dist + d) << 2) |
                                 (unsigned long long)(bext ? 1 : (bsca ? 2 : 3));
        atomicMin(a.err + 1, key);
      }
      const double out[11] = {ext,         sca,        ab,  back,    sca / ext,
                              scag / sca, (4.0 * kPi) * (ext / back), 0.0, r3 / r2,
                              kPi * r2,   (4.0 * kPi / 3.0) * r3};
#pragma unroll
      for (int k = 0; k < 11; ++k) a.values[k * nu + unit] = out[k];
    }
    const int2 sl = a.slots ? a.unit_slots[ul] : make_int2(0, 0);
    if (a.phase) {
      int n_lev = 0;  // the unit's level slots, which come first
      while (n_lev < sl.y && a.slots[sl.x + n_lev].band < a.n_levels) ++n_lev;
      for (int j = t; j < a.n_mu; j += NT) {
        double f[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          double v = acc_user[e * a.n_mu + j];
          for (int k = 0; k < n_lev; ++k)
            v += a.slot_phase[((int64_t)(sl.x + k) * 4 + e) * a.n_mu + j];
          f[e] = v / z;
          if (a.normalized) f[e] = f[e] / sca;
        }
        const double o6[6] = {f[0], f[1], f[0], f[2], f[3], f[2]};
#pragma unroll
        for (int e = 0; e < 6; ++e) a.phase[((int64_t)e * nu + unit) * a.n_mu + j] = o6[e];
      }
    }
    if (glen > 0 && a.greek) {
      auto sum = [&](int idx) {
        const int e = idx / glen, l = idx % glen;
        double g = 0.0;
        for (int k = 0; k < sl.y; ++k) {
          const BandSlot bs = a.slots[sl.x + k];
          if (l <= bs.order)
            g += a.slot_greek[(int64_t)(sl.x + k) * 6 * glen + (int64_t)e * glen + l];
        }
        return g / z;
      };
      if (t == 0) a0s = sum(0);
      __syncthreads();
      const double a0 = a0s;
      for (int idx = t; idx < 6 * glen; idx += NT) {
        const int e = idx / glen, l = idx % glen;
        double g = sum(idx);
        if (a.normalized) g = idx == 0 ? 1.0 : g / a0;
        a.greek[((int64_t)e * nu + unit) * glen + l] = g;
      }
    }
    __syncthreads();
  }
}

// The outputs and their derivatives per unit. Blocks b of the sums S_b (b = 0 the values,
// 1..P_theta the distribution's parameters, then Re m and Im m): the averages v = S_0/Z, along a
// parameter (S_p - v Z_p)/Z, along m S_m/Z (engine.rs:1782-1836); the ratios and the
// normalizations with the quotient rule of ensemble/lin.rs; the Greek coefficients from each
// block's projected raw sums, averaged the same way (the projection is linear).
__global__ void __launch_bounds__(NT) final_deriv_kernel(FinalArgs a) {
  __shared__ double S[6][8];
  __shared__ double a0s[6];
  const int t = threadIdx.x;
  const int L = a.greek_order;
  const int glen = L >= 0 ? L + 1 : 0;
  const int64_t nu = a.n_units_total;
  const int P = a.n_theta + 2, B = 1 + P, nth = a.n_theta;
  for (int ul = blockIdx.x; ul < a.n_units; ul += gridDim.x) {
    const int64_t unit = a.units[ul];
    const int64_t d = unit / a.n_wl, i = unit % a.n_wl;
    if (t < 8 * B) {
      const int b = t / 8, k = t % 8;
      double s = 0.0;
      for (int c = 0; c < a.cpu; ++c)
        s += a.chunk_sums[(((int64_t)ul * a.cpu + c) * B + b) * 8 + k];
      S[b][k] = s;
    }
    __syncthreads();
    const double z = S[0][0];
    // An average and its derivatives from the raw sums s_b of one quantity.
    auto avg = [&](const double* sb, int stride, double* out) {
      const double v = sb[0] / z;
      out[0] = v;
      for (int p = 0; p < P; ++p) {
        const double sp = sb[(1 + p) * stride];
        out[1 + p] = p < nth ? (sp - v * S[1 + p][0]) / z : sp / z;
      }
    };
    // x / y with derivatives (lin.rs Lin::div).
    auto ldiv = [&](const double* x, const double* y, double* out) {
      const double v = x[0] / y[0];
      out[0] = v;
      for (int p = 0; p < P; ++p) out[1 + p] = (x[1 + p] - v * y[1 + p]) / y[0];
    };
    const double* acc_user = a.acc + a.unit_acc[ul];
    if (t == 0) {
      double v[8][6];
      for (int k = 0; k < 8; ++k) avg(&S[0][k], 8, v[k]);
      const double ext = v[1][0], sca = v[2][0], back = v[5][0];
      const bool bext = !(isfinite(ext) && ext != 0.0), bsca = !(isfinite(sca) && sca != 0.0);
      const bool bback = !(isfinite(back) && back != 0.0);
      if (bext || bsca || bback) {
        unsigned long long key = ((unsigned long long)(i * a.n_dist + d) << 2) |
                                 (unsigned long long)(bext ? 1 : (bsca ? 2 : 3));
        atomicMin(a.err + 1, key);
      }
      double out[11][6];
      for (int p = 0; p <= P; ++p) {
        out[0][p] = v[1][p];
        out[1][p] = v[2][p];
        out[2][p] = v[4][p];
        out[3][p] = v[5][p];
        out[7][p] = 0.0;
        out[9][p] = kPi * v[6][p];
        out[10][p] = (4.0 * kPi / 3.0) * v[7][p];
      }
      ldiv(v[2], v[1], out[4]);
      ldiv(v[3], v[2], out[5]);
      ldiv(v[1], v[5], out[6]);
      for (int p = 0; p <= P; ++p) out[6][p] *= 4.0 * kPi;
      ldiv(v[7], v[6], out[8]);
      for (int k = 0; k < 11; ++k) {
        a.values[k * nu + unit] = out[k][0];
        for (int p = 0; p < P; ++p) a.d_values[((int64_t)p * 11 + k) * nu + unit] = out[k][1 + p];
      }
    }
    double sca[6];
    {
      double v[6];
      avg(&S[0][2], 8, v);
      for (int p = 0; p <= P; ++p) sca[p] = v[p];
    }
    // The unit's slots are B consecutive entries (one per block) per table, the levels first.
    const int2 sl = a.slots ? a.unit_slots[ul] : make_int2(0, 0);
    if (a.phase) {
      int n_lev = 0;
      while (n_lev < sl.y && a.slots[sl.x + n_lev].band < a.n_levels) ++n_lev;
      const int64_t blk = 4 * (int64_t)a.n_mu;
      for (int j = t; j < a.n_mu; j += NT) {
        double f[4][6];
        for (int e = 0; e < 4; ++e) {
          double raw[6];
          for (int b = 0; b < B; ++b) raw[b] = acc_user[b * blk + (int64_t)e * a.n_mu + j];
          for (int k = 0; k < n_lev; k += B)
            for (int b = 0; b < B; ++b)
              raw[b] += a.slot_phase[((int64_t)(sl.x + k + b) * 4 + e) * a.n_mu + j];
          avg(raw, 1, f[e]);
          if (a.normalized) {
            double o[6];
            ldiv(f[e], sca, o);
            for (int p = 0; p <= P; ++p) f[e][p] = o[p];
          }
        }
        const int src[6] = {0, 1, 0, 2, 3, 2};
        for (int e = 0; e < 6; ++e) {
          a.phase[((int64_t)e * nu + unit) * a.n_mu + j] = f[src[e]][0];
          for (int p = 0; p < P; ++p)
            a.d_phase[(((int64_t)p * 6 + e) * nu + unit) * a.n_mu + j] = f[src[e]][1 + p];
        }
      }
    }
    if (glen > 0 && a.greek) {
      auto sum = [&](int b, int idx) {
        const int e = idx / glen, l = idx % glen;
        double g = 0.0;
        for (int k = b; k < sl.y; k += B) {
          const BandSlot bs = a.slots[sl.x + k];
          if (l <= bs.order)
            g += a.slot_greek[(int64_t)(sl.x + k) * 6 * glen + (int64_t)e * glen + l];
        }
        return g;
      };
      auto coeff = [&](int idx, double* out) {
        double raw[6];
        for (int b = 0; b < B; ++b) raw[b] = sum(b, idx);
        avg(raw, 1, out);
      };
      if (t == 0) coeff(0, a0s);
      __syncthreads();
      for (int idx = t; idx < 6 * glen; idx += NT) {
        const int e = idx / glen, l = idx % glen;
        double c[6];
        coeff(idx, c);
        if (a.normalized) {
          if (idx == 0) {
            c[0] = 1.0;
            for (int p = 0; p < P; ++p) c[1 + p] = 0.0;
          } else {
            double o[6];
            ldiv(c, a0s, o);
            for (int p = 0; p <= P; ++p) c[p] = o[p];
          }
        }
        a.greek[((int64_t)e * nu + unit) * glen + l] = c[0];
        for (int p = 0; p < P; ++p)
          a.d_greek[(((int64_t)p * 6 + e) * nu + unit) * glen + l] = c[1 + p];
      }
    }
    __syncthreads();
  }
}

// The outputs of adaptive panels per unit with their error estimates: averages from the
// Kronrod sums and the moments' Z, errors (e + |v| e_Z)/Z + truncation |v| (engine.rs:
// 1782-1836), <r^2>, <r^3> from the moments (a single radius keeps its own), the ratios and
// normalizations with the first-order bounds of ensemble/lin.rs (Lin::div, Lin::scale), and the
// Greek coefficients summed over the bands, values and bounds (engine.rs:2310-2355).
namespace {
struct LinE {
  double v, e;
};
__device__ __forceinline__ LinE ldiv(LinE a, LinE b) {
  const double v = a.v / b.v;
  return {v, (a.e + fabs(v) * b.e) / fabs(b.v)};
}
__device__ __forceinline__ LinE lscale(LinE a, double c) { return {c * a.v, fabs(c) * a.e}; }
}  // namespace

// Stage 1 of the adaptive outputs: each (part, wavelength) unit's averages with their error
// estimates into `avg` (per unit: the 8 scalars, the 4 n_mu cosine tables, the 6 (L + 1) Greek
// sums, each as values then errors). The Greek sums are projected per part and mixed after
// (the projection is linear and its bounds are linear in the errors).
__global__ void __launch_bounds__(NT) final_adaptive_kernel(FinalArgs a) {
  __shared__ double S[2][8];
  const int t = threadIdx.x;
  const int L = a.greek_order;
  const int glen = L >= 0 ? L + 1 : 0;
  const int64_t stride = 16 + 8 * (int64_t)a.n_mu + 12 * (int64_t)glen;
  for (int ul = blockIdx.x; ul < a.n_units; ul += gridDim.x) {
    const int64_t unit = a.units[ul];
    if (t < 16) {
      double s = 0.0;
      for (int c = 0; c < a.cpu; ++c) s += a.chunk_sums[((int64_t)ul * a.cpu + c) * 16 + t];
      S[t / 8][t % 8] = s;
    }
    __syncthreads();
    const double* un = a.unit_norm + 8 * unit;
    const double z = un[0], ez = un[1], tr = un[2];
    const bool point = un[3] != 0.0;
    auto avg = [&](double s, double e) {
      const double v = s / z;
      return LinE{v, (e + fabs(v) * ez) / z + tr * fabs(v)};
    };
    double* out = a.avg + stride * unit;
    if (t < 8) {
      LinE v = avg(S[0][t], S[1][t]);
      // <r^2>, <r^3> from the moment integration (a single radius keeps its own).
      if (!point && t >= 6) v = LinE{un[4 + 2 * (t - 6)], un[5 + 2 * (t - 6)]};
      out[t] = v.v;
      out[8 + t] = v.e;
    }
    const double* acc_user = a.acc + a.unit_acc[ul];
    for (int j = t; j < 4 * a.n_mu; j += NT) {
      const LinE f = avg(acc_user[j], acc_user[4 * a.n_mu + j]);
      out[16 + j] = f.v;
      out[16 + 4 * a.n_mu + j] = f.e;
    }
    if (glen > 0) {
      // The unit's slots: per band a values slot, then its bounds slot.
      const int2 sl = a.unit_slots[ul];
      double* og = out + 16 + 8 * (int64_t)a.n_mu;
      for (int idx = t; idx < 6 * glen; idx += NT) {
        const int e = idx / glen, l = idx % glen;
        double gv = 0.0, ge = 0.0;
        for (int k = 0; k + 1 < sl.y; k += 2) {
          const BandSlot bs = a.slots[sl.x + k];
          if (l <= bs.order) {
            gv += a.slot_greek[(int64_t)(sl.x + k) * 6 * glen + (int64_t)e * glen + l];
            ge += a.slot_greek[(int64_t)(sl.x + k + 1) * 6 * glen + (int64_t)e * glen + l];
          }
        }
        og[idx] = gv;
        og[6 * glen + idx] = ge;
      }
    }
    __syncthreads();
  }
}

// Stage 1 of an adaptive call with derivatives: each (part, wavelength) unit's averages along
// every block b < B (values, each distribution parameter, Re m, Im m) with their error
// estimates into `avg`, block after block: 8 scalars, 4 n_mu cosine values, 6 (L + 1) Greek
// coefficients, then the same for the errors (engine.rs:1782-1836 with the quotient rule of
// the parameter blocks). <r^2> and <r^3> and their parameter derivatives come from the moments
// (a single radius keeps its own; 0 along m). The Greek sums are already averaged per slot.
__global__ void __launch_bounds__(NT) final_adaptive_d_kernel(FinalArgs a) {
  __shared__ double S[12][8];
  const int t = threadIdx.x;
  const int L = a.greek_order;
  const int glen = L >= 0 ? L + 1 : 0;
  const int B = a.ad_blocks, nth = a.n_theta;
  const int64_t row = 8 + 4 * (int64_t)a.n_mu + 6 * (int64_t)glen;
  for (int ul = blockIdx.x; ul < a.n_units; ul += gridDim.x) {
    const int64_t unit = a.units[ul];
    if (t < 16 * B) {
      const int b = t / 8, k = t % 8;
      double s = 0.0;
      for (int c = 0; c < a.cpu; ++c)
        s += a.chunk_sums[(((int64_t)ul * a.cpu + c) * 2 * B + b) * 8 + k];
      S[b][k] = s;
    }
    __syncthreads();
    const double* un = a.unit_norm + kNormStrideD * unit;
    const double z = un[0], ez = un[1], tr = un[2];
    const bool point = un[3] != 0.0;
    // One element's average and error along block b from its sums (s0, e0: the values';
    // sb, eb: the block's).
    auto avg = [&](int b, double s0, double e0, double sb, double eb, double* v, double* e) {
      const double v0 = s0 / z, av0 = fabs(v0);
      const double er0 = (e0 + av0 * ez) / z + tr * av0;
      if (b == 0) {
        *v = v0;
        *e = er0;
      } else if (b <= nth) {
        const double dz = un[8 + b - 1], edz = un[11 + b - 1];
        const double dv = (sb - v0 * dz) / z;
        *v = dv;
        *e = (eb + av0 * edz + fabs(dv) * ez + er0 * fabs(dz)) / z + tr * fabs(dv);
      } else {
        const double dv = sb / z;
        *v = dv;
        *e = (eb + fabs(dv) * ez) / z + tr * fabs(dv);
      }
    };
    double* out = a.avg + 2 * B * row * unit;
    for (int idx = t; idx < 8 * B; idx += NT) {
      const int b = idx / 8, k = idx % 8;
      double v, e;
      avg(b, S[0][k], S[B][k], S[b][k], S[B + b][k], &v, &e);
      if (!point && k >= 6) {
        const int m = k - 6;
        if (b == 0) {
          v = un[4 + 2 * m];
          e = un[5 + 2 * m];
        } else if (b <= nth) {
          v = un[14 + 4 * (b - 1) + 2 * m];
          e = un[15 + 4 * (b - 1) + 2 * m];
        } else {
          v = 0.0;
          e = 0.0;
        }
      }
      out[2 * b * row + k] = v;
      out[(2 * b + 1) * row + k] = e;
    }
    const double* acc_user = a.acc + a.unit_acc[ul];
    const int64_t tl = 4 * (int64_t)a.n_mu;
    for (int64_t idx = t; idx < tl * B; idx += NT) {
      const int b = (int)(idx / tl);
      const int64_t j = idx % tl;
      double v, e;
      avg(b, acc_user[j], acc_user[B * tl + j], acc_user[b * tl + j], acc_user[(B + b) * tl + j],
          &v, &e);
      out[2 * b * row + 8 + j] = v;
      out[(2 * b + 1) * row + 8 + j] = e;
    }
    if (glen > 0) {
      // The unit's slots per band: B value slots, then B error slots.
      const int2 sl = a.unit_slots[ul];
      for (int64_t idx = t; idx < 6 * (int64_t)glen * B; idx += NT) {
        const int b = (int)(idx / (6 * glen));
        const int g = (int)(idx % (6 * glen)), e = g / glen, l = g % glen;
        double gv = 0.0, ge = 0.0;
        for (int k = 0; k + 2 * B <= sl.y; k += 2 * B) {
          const BandSlot bs = a.slots[sl.x + k];
          if (l <= bs.order) {
            gv += a.slot_greek[(int64_t)(sl.x + k + b) * 6 * glen + (int64_t)e * glen + l];
            ge += a.slot_greek[(int64_t)(sl.x + k + B + b) * 6 * glen + (int64_t)e * glen + l];
          }
        }
        out[2 * b * row + 8 + tl + g] = gv;
        out[(2 * b + 1) * row + 8 + tl + g] = ge;
      }
    }
    __syncthreads();
  }
}

// Stage 2: each output unit (o, wavelength i) mixes its parts' averages with their number
// fractions f (engine.rs:2121-2176: values and errors alike, in part order) and assembles the
// outputs: ratios, normalizations and bounds of ensemble/lin.rs, Greek normalized by the
// mixture's alpha1_0 (engine.rs:2396-2497).
__global__ void __launch_bounds__(NT) mix_assemble_kernel(MixArgs a) {
  __shared__ double V[16];
  __shared__ LinE a0s;
  const int t = threadIdx.x;
  const int glen = a.greek_order >= 0 ? a.greek_order + 1 : 0;
  const int64_t stride = 16 + 8 * (int64_t)a.n_mu + 12 * (int64_t)glen;
  const int64_t n_out = (int64_t)a.n_out * a.n_wl;
  auto mixed = [&](int64_t o, int64_t i, int64_t off) {
    double v = 0.0;
    for (int k = a.first[o]; k < a.first[o + 1]; ++k)
      v += a.fraction[k] * a.avg[stride * ((int64_t)a.part[k] * a.n_wl + i) + off];
    return v;
  };
  for (int64_t ou = blockIdx.x; ou < n_out; ou += gridDim.x) {
    const int64_t o = ou / a.n_wl, i = ou % a.n_wl;
    if (t < 16) V[t] = mixed(o, i, t);
    __syncthreads();
    auto lin = [&](int k) { return LinE{V[k], V[8 + k]}; };
    const LinE ext = lin(1), sca = lin(2), scag = lin(3), ab = lin(4), back = lin(5), r2 = lin(6),
               r3 = lin(7);
    if (t == 0) {
      const bool bext = !(isfinite(ext.v) && ext.v != 0.0);
      const bool bsca = !(isfinite(sca.v) && sca.v != 0.0);
      const bool bback = !(isfinite(back.v) && back.v != 0.0);
      if (bext || bsca || bback) {
        unsigned long long key = ((unsigned long long)(i * a.n_out + o) << 2) |
                                 (unsigned long long)(bext ? 1 : (bsca ? 2 : 3));
        atomicMin(a.err + 1, key);
      }
      const LinE out[11] = {ext,
                            sca,
                            ab,
                            back,
                            ldiv(sca, ext),
                            ldiv(scag, sca),
                            lscale(ldiv(ext, back), 4.0 * kPi),
                            LinE{0.0, 0.0},
                            ldiv(r3, r2),
                            lscale(r2, kPi),
                            lscale(r3, 4.0 * kPi / 3.0)};
      for (int k = 0; k < 11; ++k) {
        a.values[k * n_out + ou] = out[k].v;
        a.errors[k * n_out + ou] = out[k].e;
      }
    }
    if (a.phase) {
      for (int j = t; j < a.n_mu; j += NT) {
        LinE f[4];
        for (int e = 0; e < 4; ++e) {
          f[e] = LinE{mixed(o, i, 16 + e * a.n_mu + j),
                      mixed(o, i, 16 + (4 + e) * (int64_t)a.n_mu + j)};
          if (a.normalized) f[e] = ldiv(f[e], sca);
        }
        const int src[6] = {0, 1, 0, 2, 3, 2};
        for (int e = 0; e < 6; ++e) {
          a.phase[((int64_t)e * n_out + ou) * a.n_mu + j] = f[src[e]].v;
          a.phase_err[((int64_t)e * n_out + ou) * a.n_mu + j] = f[src[e]].e;
        }
      }
    }
    if (glen > 0 && a.greek) {
      const int64_t g0 = 16 + 8 * (int64_t)a.n_mu;
      if (t == 0) a0s = LinE{mixed(o, i, g0), mixed(o, i, g0 + 6 * glen)};
      __syncthreads();
      const LinE a0 = a0s;
      for (int idx = t; idx < 6 * glen; idx += NT) {
        const int e = idx / glen, l = idx % glen;
        LinE g{mixed(o, i, g0 + idx), mixed(o, i, g0 + 6 * glen + idx)};
        if (a.normalized) g = idx == 0 ? LinE{1.0, 0.0} : ldiv(g, a0);
        a.greek[((int64_t)e * n_out + ou) * glen + l] = g.v;
        a.greek_err[((int64_t)e * n_out + ou) * glen + l] = g.e;
      }
    }
    __syncthreads();
  }
}

void launch_mix(const MixArgs& a, cudaStream_t s) {
  const int64_t n = (int64_t)a.n_out * a.n_wl;
  const int grid = (int)(n < 4096 ? n : 4096);
  if (grid > 0) mix_assemble_kernel<<<grid, NT, 0, s>>>(a);
}

// The unit kernels' stage buffers are dynamic shared memory (above the 48 KB static limit);
// the attribute is per device: set it once on each.
static void configure_units() {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    const auto set = [](void (*f)(UnitArgs), size_t bytes) {
      cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    set(unit_kernel, sizeof(UnitSmem<1>));
    set(unit_deriv_kernel, sizeof(UnitSmem<4>));
    set(unit_adaptive_kernel, sizeof(UnitSmem<2>));
    set(unit_adaptive_deriv_kernel, sizeof(UnitSmem<8>));
    configured[dev] = true;
  }
}

int unit_kernel_blocks_per_sm(int mode) {
  configure_units();
  int n = 0;
  if (mode == 0)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, unit_kernel, NT, sizeof(UnitSmem<1>));
  else if (mode == 1)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, unit_deriv_kernel, NT, sizeof(UnitSmem<4>));
  else if (mode == 2)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, unit_adaptive_kernel, NT,
                                                  sizeof(UnitSmem<2>));
  else
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, unit_adaptive_deriv_kernel, NT,
                                                  sizeof(UnitSmem<8>));
  return n > 0 ? n : 1;
}

void launch_units(const UnitArgs& a, int grid, cudaStream_t s) {
  configure_units();
  if (a.deriv && a.adaptive)
    unit_adaptive_deriv_kernel<<<grid, NT, sizeof(UnitSmem<8>), s>>>(a);
  else if (a.deriv)
    unit_deriv_kernel<<<grid, NT, sizeof(UnitSmem<4>), s>>>(a);
  else if (a.adaptive)
    unit_adaptive_kernel<<<grid, NT, sizeof(UnitSmem<2>), s>>>(a);
  else
    unit_kernel<<<grid, NT, sizeof(UnitSmem<1>), s>>>(a);
}

void launch_proj(const ProjArgs& a, cudaStream_t s) {
  // The attribute is per device: set it once on each.
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaFuncSetAttribute(proj_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(ProjSmem));
    configured[dev] = true;
  }
  int grid = a.n_items < 8192 ? a.n_items : 8192;
  if (grid > 0) proj_kernel<<<grid, PT, sizeof(ProjSmem), s>>>(a);
}

void launch_final(const FinalArgs& a, cudaStream_t s) {
  int grid = a.n_units < 4096 ? a.n_units : 4096;
  if (a.ad_blocks > 0)
    final_adaptive_d_kernel<<<grid, NT, 0, s>>>(a);
  else if (a.d_values)
    final_deriv_kernel<<<grid, NT, 0, s>>>(a);
  else if (a.unit_norm)
    final_adaptive_kernel<<<grid, NT, 0, s>>>(a);
  else
    final_kernel<<<grid, NT, 0, s>>>(a);
}

}  // namespace sb
