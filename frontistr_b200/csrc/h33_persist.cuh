// h33_persist.cuh -- the whole CG + SSOR solve in one persistent launch.
//
// One iteration of hecmw_solve_CG with the SSOR preconditioner reads every block of A
// twice when it is written as z = M^-1 r followed by q = A p: once in the sweeps, once in
// the product.  With M = (D + L) D^-1 (D + U) built from A's own blocks (SIGMA_DIAG = 1)
// the product needs no second reading: the forward sweep leaves g = D y with
// (D + L) y = r, the backward sweep solves (D + U) z = g, so
//     A z = (D + U) z + L z = g + L z,
// and L z is one more pair of operands for the blocks that the NEXT forward sweep reads
// anyway.  That sweep in turn need not start from the new residual: y is linear in r, so
// it runs on the direction, (D + L) t = q, and g follows from g -= ALPHA D t as r follows
// from r -= ALPHA q.  With v = U z from the backward sweep (D + L) u = v gives
//     D t = h:  h = (g - L u) + BETA h_old,   q = (g + L z) + BETA q_old,
// so the order of an iteration is
//     backward:  v = U z,  z = D^-1 (g - v),            RHO = r.z
//     forward:   u = D^-1 (v - L u),  p, q, h as above,  C1 = p.q
//     update:    x += ALPHA p,  r -= ALPHA q,  g -= ALPHA h,  r.r
// The iterates are hecmw_solve_CG's in exact arithmetic (the same RHO, C1, ALPHA, BETA
// and tests on them); every true-residual refresh recomputes g from the new r by a plain
// forward sweep.
//
// Rounding: hecmw_solve_CG's q is the product with the very p that goes into x.  Here q
// follows z, so what p = z + BETA p loses to rounding would be missing from q for as long
// as the direction lives, and the gap between r and b - A x grew to 1.6-1.9 times
// hecmw_solve_CG's on slender boxes, 5 times on a chain with stiffness growing to 1e6 (64
// bits, CPU, geometric means over loads).  p's lost part is therefore kept beside it, in
// FP32 (pl: p to some 77 bits): 1.0-1.3 times, as wide as the scatter between loads.
// Keeping q's part as well changed nothing more; q from a product at every refresh alone
// left 1.5-1.8.
//
// What bounds it: the colours are a chain of 2 x NColor dependent steps.  As one launch
// per colour a step cost 5 to 10 us whatever its size (launch, ramp, tail); here one CTA
// per SM stays for the whole solve and a grid barrier (1.1 us bare, 1.6 us with the
// stores before it and the first load after it) separates the colours.  A small system
// runs as one cluster of 16 CTAs, whose hardware barrier takes 0.25 us.  What is left of
// a step is the latency of one slice per warp: a round of loads, 9 or 18 fused
// multiply-adds per block, the lane sums, the 3x3 solve.  Measured per iteration against
// the colour launches (us): 378 nodes 62 / 181, 19 thousand 109 / 305, 118 thousand
// 178 / 372, 275 thousand 285 / 501, 1.03 million 707 / 1125.
// Measured and dropped: the blocks through shared-memory rings filled by bulk copies
// (819 to 1000 us at 1.03 million nodes: 750 instructions a slice against 300, and a
// ring of 12 KB a warp holds little more than the slice in work); the next slice's
// blocks held in registers (spills); bulk prefetch of the next slice into L2 (821 us);
// 24 warps per CTA (80 registers, spills: 1129 us).
#pragma once

#include "h33_kernels.cuh"

namespace h33 {

// Warps per CTA, one CTA per SM.  With few rows a colour (K >= 8) 12 warps, whose 168
// registers hold a slice without spills (107 against 111 us an iteration at 19 thousand
// nodes); where every warp has several slices (K = 4) 16 of them (705 against 738 us at
// 1.03 million).
template <int K>
constexpr int persist_warps() {
  return K >= 8 ? 12 : 16;
}
constexpr int kPEnd = 0x7fffffff;            // end of a warp's list

// One sweep direction: the blocks and, for each warp of the grid, its slices in the
// order of the sweep: (first slot, slots, first row, step << 6 | rows), kPEnd in w ends it.
struct PersistSweep {
  const double *val;
  const int *col;
  const int4 *items;
  int stride;
};

// The fused sweeps' vectors in colour-position order.
struct SsorVecs {
  const double *alu;  // diagonal LU, entry e of position i at alu[e * n + i]
  int n;
  double *r, *g, *p, *q, *h;
  double2 *zu;        // per position z and v (backward sweep) or u (forward): 3 double2
  float *pl;          // what p's rounding dropped
};

struct PersistArgs {
  PersistSweep lo, up;
  SellView<double> A;
  SsorVecs v;
  const double *alu;        // block ILU: LU and nodes in the order of the forward levels
  const int *perm, *iperm;  // position -> node and back
  const double *alu_b;      // and of the backward levels, z in node order, the number of
  const int *perm_b;        // backward levels
  double *pz;
  int nback;
  const double *b;          // node order
  double *x, *r;            // node order: x in and out, r out
  double *px, *pr, *pp, *pq;  // position order (block ILU: node order)
  CgState *st;
  const CgParams *prm;
  double *parts;            // 3 x gridDim.x partial sums
  unsigned *bar;            // [0] arrivals at the grid barrier, [1] set when a wait gave up (the host reads it)
  int polls;                // of a grid barrier before it gives up
  int n, ncolor;
};

// The slices of every warp's list: slice t of a group goes to warp t mod nw of the grid.
static __global__ void persist_items_kernel(const int *__restrict__ gs, int ng, int reverse,
                                            const int *__restrict__ row0, const int *__restrict__ nrows,
                                            const int *__restrict__ slot0, const int *__restrict__ len, int nw,
                                            int stride, int4 *__restrict__ items) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nw) return;
  int4 *out = items + size_t(w) * stride;
  int k = 0;
  for (int c = 0; c < ng; c++) {
    const int g = reverse ? ng - 1 - c : c;
    for (int s = gs[g] + w; s < gs[g + 1]; s += nw) out[k++] = make_int4(slot0[s], len[s], row0[s], (c << 6) | nrows[s]);
  }
  for (; k < stride; k++) out[k] = make_int4(0, 0, 0, kPEnd);
}

static __global__ void invert_perm_kernel(const int *__restrict__ perm, int n, int *__restrict__ iperm) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) iperm[perm[i]] = i;
}

// ---- barriers and sums over the grid (or the cluster) ------------------------------
struct PersistShared {
  CgState st;
  double red[32];
  double val;
  int dead;
};

// A thread's way through the grid's barriers: the arrivals at the next one, and whether it
// has given up.  The CG keeps that in a register (read from shared memory it cost 30 ns a
// barrier, 1 % of the block ILU's levels); in the single application and the load cases,
// short of registers, reading it is 3 % the faster.
struct GridWay {
  unsigned target = 0;
  bool gone = false;
};

// One thread's arrival at the grid barrier and its wait until *bar has reached the target;
// after `polls` polls, or when another CTA has given up, it gives up (dead).  A CTA that
// has given up arrives nowhere any more, so none passes a barrier that a late one has not
// reached; the others see its mark in bar[1] and give up too.
__device__ __forceinline__ void grid_meet(unsigned *bar, GridWay &way, int polls, int &dead) {
  if (way.gone) return;
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
  unsigned v;
  int tries = 0;
  for (;;) {
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
    if (int(v - way.target) >= 0) break;
    if (++tries > polls || ((tries & 1023) == 0 && *((volatile unsigned *)(bar + 1)))) {
      way.gone = true;
      dead = 1;
      *((volatile unsigned *)(bar + 1)) = 1u;
      break;
    }
  }
}

// Every write made before it by any CTA is visible after it.  CLUSTER: the grid is one
// cluster and the barrier its hardware barrier; else a counter in global memory, its
// wait bounded.
template <bool CLUSTER>
__device__ __forceinline__ void persist_barrier(const PersistArgs &a, PersistShared &sh, GridWay &way) {
  if constexpr (CLUSTER) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    way.target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) grid_meet(a.bar, way, a.polls, sh.dead);
    __syncthreads();
  }
}

// Sum over the grid, the same value in every thread; includes a barrier.
template <bool CLUSTER>
__device__ __forceinline__ double persist_sum(const PersistArgs &a, PersistShared &sh, GridWay &way, double v,
                                              int slot) {
  v = block_sum(v, sh.red);
  double *parts = a.parts + slot * gridDim.x;
  if (threadIdx.x == 0) parts[blockIdx.x] = v;
  persist_barrier<CLUSTER>(a, sh, way);
  if (threadIdx.x < 32) {
    double s = 0.0;
    for (int i = threadIdx.x; i < int(gridDim.x); i += 32) s += __ldcg(parts + i);
    s = warp_sum(s);
    if (threadIdx.x == 0) sh.val = s;
  }
  __syncthreads();
  return sh.val;
}

// ---- one slice ----------------------------------------------------------------------
// Loads of what other CTAs wrote: coherent after a barrier, never the read-only path.
template <bool L2ONLY, class T>
__device__ __forceinline__ T ld_row(const T *p) {
  if constexpr (L2ONLY) return __ldcg(p);
  else return *p;
}

// A warp's slices one after another, as descriptors (first slot, slots, first row,
// step << 6 | rows) with kPEnd in w after the last: from its list,
struct ListCursor {
  const int4 *items;
  int steps;
  __device__ __forceinline__ int4 next() {
    const int4 it = __ldg(items);
    if (it.w != kPEnd) items++;
    return it;
  }
};
// or every nw-th slice of the groups [g0, g1) (in reverse), where the team that takes a
// system is not known beforehand.  desc has the slices' descriptors without their steps.
struct GroupCursor {
  const int4 *desc;
  const int *gs;
  int g0, steps, back, warp, nw, c, s, end;
  __device__ __forceinline__ void open() {
    const int g = back ? g0 + steps - 1 - c : g0 + c;
    s = __ldg(gs + g) + warp;
    end = __ldg(gs + g + 1);
  }
  __device__ __forceinline__ GroupCursor(const int4 *desc_, const int *gs_, int g0_, int g1_, bool back_, int warp_,
                                         int nw_)
      : desc(desc_), gs(gs_), g0(g0_), steps(g1_ - g0_), back(back_), warp(warp_), nw(nw_), c(0), s(0), end(0) {
    if (steps > 0) open();
  }
  __device__ __forceinline__ int4 next() {
    while (c < steps && s >= end)
      if (++c < steps) open();
    if (c >= steps) return make_int4(0, 0, 0, kPEnd);
    int4 it = __ldg(desc + s);
    it.w |= c << 6;
    s += nw;
    return it;
  }
};

// p = z + BETA (p + pl): p rounded, the new pl in `rest`.  The product is split exactly, the
// sum by the short form, which is exact for |BETA p| >= |z| and else misses a rounding of
// z, as q misses one of A z.  None of it may be contracted.
__device__ __forceinline__ double next_direction(double z, double beta, double p, float pl, float &rest) {
  const double bp = __dmul_rn(beta, p), s = __dadd_rn(bp, z);
  const double es = __dsub_rn(z, __dsub_rn(s, bp));
  const double lo = __dadd_rn(es, fma(beta, double(pl), fma(beta, p, -bp)));
  const double pn = __dadd_rn(s, lo);
  rest = float(__dsub_rn(lo, __dsub_rn(pn, s)));
  return pn;
}

// One sweep, MODE 0 backward, 1 forward on the direction, 2 forward from r (start and
// refresh): the colours in turn, a barrier between them.  K lanes per row; lane c < 3 of
// a row (MODE 1, K >= 8: of each half of its lanes) carries component c of its vectors.
// The columns of the slice whose turn is next are loaded before the barrier, so that
// what follows it is one round of loads: blocks, diagonal LU, own vectors, gathers.
template <int K, int MODE, bool CLUSTER, class Cursor, class Barrier>
__device__ __forceinline__ double ssor_sweep(const SsorVecs &a, const double *val, const int *cols, Cursor cur,
                                             Barrier barrier, double beta, bool first) {
  constexpr int U = 2;                          // slots taken together (4: more registers, no faster)
  constexpr bool HALVES = MODE == 1 && K >= 8;  // a row's upper lanes end with the sums over z, the lower over u
  const int lane = threadIdx.x & 31;
  const int sub = lane & (K - 1), roff = lane / K;
  const bool up = HALVES && (sub & (K / 2)) != 0;
  const int cc = HALVES ? sub & (K / 2 - 1) : sub, c0 = min(cc, 2);
  const size_t n = size_t(a.n);
  // In the first iteration BETA is 0 and p, q, h and pl hold zeros.  Over the grid with 8 and
  // 16 lanes not reading them then is 1 to 2 % of a solve the faster (less is in flight at
  // once), in a cluster or a team and with 4 lanes reading them always is, by as much.
  const bool fresh = first && K >= 8 && !CLUSTER;
  double dot = 0.0;
  int4 it = cur.next(), nx = cur.next();
  int col[U];
#pragma unroll
  for (int u = 0; u < U; u++) col[u] = u < it.y ? __ldg(cols + (it.x + u) * 32 + lane) : 0;
  for (int c = 0; c < cur.steps; c++) {
    if (c) barrier();
    while ((it.w >> 6) == c) {
      const bool act = roff < (it.w & 63);
      const int row = it.z + (act ? roff : 0), i3 = 3 * row;
      const double *lu = a.alu + row;
      const double a0 = __ldcs(lu), a1 = __ldcs(lu + n), a2 = __ldcs(lu + 2 * n);
      const double a3 = __ldcs(lu + 3 * n), a4 = __ldcs(lu + 4 * n), a5 = __ldcs(lu + 5 * n);
      const double a6 = __ldcs(lu + 6 * n), a7 = __ldcs(lu + 7 * n), a8 = __ldcs(lu + 8 * n);
      double o0, o1, o2;  // the row's own right-hand side: g, v or r
      double f0 = 0.0, f1 = 0.0, f2 = 0.0, f3 = 0.0, f4 = 0.0;
      float fl = 0.0f;
      const double *own = reinterpret_cast<const double *>(a.zu + 3 * size_t(row));
      if (MODE == 1) {
        o0 = __ldcg(own + 3), o1 = __ldcg(own + 4), o2 = __ldcg(own + 5);
        f0 = __ldcg(a.g + i3 + c0);
        if (HALVES) {
          if (!fresh) f1 = __ldcg((up ? a.q : a.h) + i3 + c0);
          if (up) {
            f2 = __ldcg(own + c0);
            if (!fresh) {
              f3 = __ldcg(a.p + i3 + c0);
              fl = __ldcg(a.pl + i3 + c0);
            }
          }
        } else {
          f2 = __ldcg(own + c0);
          if (!fresh) {
            f1 = __ldcg(a.h + i3 + c0);
            f3 = __ldcg(a.p + i3 + c0);
            f4 = __ldcg(a.q + i3 + c0);
            fl = __ldcg(a.pl + i3 + c0);
          }
        }
      } else {
        const double *src = (MODE == 0 ? a.g : a.r) + i3;
        o0 = __ldcg(src), o1 = __ldcg(src + 1), o2 = __ldcg(src + 2);
        if (MODE == 0) f0 = __ldcg(a.r + i3 + c0);
      }
      double l[3] = {0.0, 0.0, 0.0}, m[3] = {0.0, 0.0, 0.0};  // sums over u (z when MODE 0), and over z
      for (int s = 0; s < it.y; s += U) {
        const int nu = it.y - s;
        double2 ga[U], gb[U], gd[U];
        double v[U][9];
#pragma unroll
        for (int u = 0; u < U; u++) {
          ga[u] = gb[u] = gd[u] = make_double2(0.0, 0.0);
#pragma unroll
          for (int e = 0; e < 9; e++) v[u][e] = 0.0;
          if (u < nu) {
            const double2 *g = a.zu + 3 * size_t(col[u]);
            if (MODE != 2) ga[u] = ld_row<CLUSTER>(g);
            gb[u] = ld_row<CLUSTER>(g + 1);
            if (MODE != 0) gd[u] = ld_row<CLUSTER>(g + 2);
            const double *b = val + size_t(it.x + s + u) * 288 + lane;
#pragma unroll
            for (int e = 0; e < 9; e++) v[u][e] = __ldcs(b + 32 * e);
          }
        }
        // the columns after these: the slice's next slots, or the next slice's first
        const bool more = nu > U;
        const int slot = more ? it.x + s + U : nx.x, left = more ? nu - U : nx.y;
#pragma unroll
        for (int u = 0; u < U; u++)
          if (u < left) col[u] = __ldg(cols + (slot + u) * 32 + lane);
#pragma unroll
        for (int u = 0; u < U; u++)
          if (u < nu) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
              const double v0 = v[u][3 * i], v1 = v[u][3 * i + 1], v2 = v[u][3 * i + 2];
              if (MODE == 0) l[i] = fma(v2, gb[u].x, fma(v1, ga[u].y, fma(v0, ga[u].x, l[i])));
              else l[i] = fma(v2, gd[u].y, fma(v1, gd[u].x, fma(v0, gb[u].y, l[i])));
              if (MODE == 1) m[i] = fma(v2, gb[u].x, fma(v1, ga[u].y, fma(v0, ga[u].x, m[i])));
            }
          }
      }
      if (it.y == 0) {
#pragma unroll
        for (int u = 0; u < U; u++)
          if (u < nx.y) col[u] = __ldg(cols + (nx.x + u) * 32 + lane);
      }
      // the direction here, beside the lane sums: after them its chain would be the step's
      // tail
      float rest = 0.0f;
      double pn = 0.0;
      if (MODE == 1) pn = next_direction(f2, beta, f3, fl, rest);
      if (HALVES) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
          const double other = __shfl_xor_sync(0xffffffffu, up ? l[j] : m[j], K / 2);
          l[j] = (up ? m[j] : l[j]) + other;
        }
      }
#pragma unroll
      for (int o = HALVES ? K / 4 : K / 2; o > 0; o >>= 1) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
          l[j] += __shfl_xor_sync(0xffffffffu, l[j], o);
          if (MODE == 1 && !HALVES) m[j] += __shfl_xor_sync(0xffffffffu, m[j], o);
        }
      }
      const double e0 = o0 - l[0], e1 = o1 - l[1], e2 = o2 - l[2];
      double x1 = e0, x2 = e1, x3 = e2;  // D^-1 e by the reciprocal-pivot LU
      x2 = x2 - a3 * x1;
      x3 = x3 - a6 * x1 - a7 * x2;
      x3 = a8 * x3;
      x2 = a4 * (x2 - a5 * x3);
      x1 = a0 * (x1 - a2 * x3 - a1 * x2);
      if (act && cc < 3) {
        const int i = i3 + cc;
        const double xc = cc == 0 ? x1 : cc == 1 ? x2 : x3;
        const double lc = cc == 0 ? l[0] : cc == 1 ? l[1] : l[2];
        double *uo = reinterpret_cast<double *>(a.zu + 3 * size_t(row)) + 3 + cc;
        if (MODE == 0) {  // z = D^-1 (g - U z) and v = U z
          a.zu[3 * size_t(row) + cc] =
              cc == 0 ? make_double2(x1, x2) : cc == 1 ? make_double2(x3, l[0]) : make_double2(l[1], l[2]);
          dot += f0 * xc;
        } else if (MODE == 2) {
          *uo = xc;
          a.g[i] = cc == 0 ? e0 : cc == 1 ? e1 : e2;
        } else if (HALVES) {
          const double t = up ? f0 + lc : f0 - lc;  // g + L z, or g - L u
          const double tn = fresh ? t : t + beta * f1;
          (up ? a.q : a.h)[i] = tn;
          if (up) {
            a.p[i] = pn;
            a.pl[i] = rest;
            dot += pn * tn;
          } else {
            *uo = xc;
          }
        } else {
          const double mc = cc == 0 ? m[0] : cc == 1 ? m[1] : m[2];
          double qn = f0 + mc, hn = f0 - lc;
          if (!fresh) {
            qn = qn + beta * f4;
            hn = hn + beta * f1;
          }
          *uo = xc;
          a.p[i] = pn;
          a.pl[i] = rest;
          a.q[i] = qn;
          a.h[i] = hn;
          dot += pn * qn;
        }
      }
      it = nx;
      nx = cur.next();
    }
  }
  return dot;
}

template <int K, int MODE, bool CLUSTER>
__device__ __forceinline__ double persist_sweep(const PersistArgs &a, PersistShared &sh, GridWay &way, int w,
                                                double beta, bool first) {
  const PersistSweep S = MODE == 0 ? a.up : a.lo;
  return ssor_sweep<K, MODE, CLUSTER>(a.v, S.val, S.col, ListCursor{S.items + size_t(w) * S.stride, a.ncolor},
                                      [&] { persist_barrier<CLUSTER>(a, sh, way); }, beta, first);
}

// Descriptors of a layout's slices for GroupCursor.
static __global__ void slice_desc_kernel(const int *__restrict__ slot0, const int *__restrict__ len,
                                         const int *__restrict__ row0, const int *__restrict__ nrows, int n,
                                         int4 *__restrict__ desc) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    desc[i] = make_int4(slot0[i], len[i], row0[i], nrows[i]);
}

// r = b - A x from x in node order, r in position order (node order without iperm);
// |r|^2 or (BB) |b|^2.
template <bool BB>
__device__ __forceinline__ double persist_resid(const PersistArgs &a) {
  const int lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  double acc = 0.0;
  for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < a.A.nslices; s += nw) {
    const bool active = lane < a.A.nrows[s];
    const int row = a.A.row0[s] + lane;
    const int len = active ? a.A.rowlen[s * 32 + lane] : 0;
    double y0 = 0.0, y1 = 0.0, y2 = 0.0;
    row_gemv<double, double, 1, false, true>(a.A, s, lane, len, a.x, y0, y1, y2);
    if (active) {
      const double b0 = a.b[3 * row], b1 = a.b[3 * row + 1], b2 = a.b[3 * row + 2];
      y0 = b0 - y0;
      y1 = b1 - y1;
      y2 = b2 - y2;
      double *r = a.pr + 3 * (a.iperm ? a.iperm[row] : row);
      r[0] = y0;
      r[1] = y1;
      r[2] = y2;
      acc += BB ? b0 * b0 + b1 * b1 + b2 * b2 : y0 * y0 + y1 * y1 + y2 * y2;
    }
  }
  return acc;
}

// The CG's scalars at the start of a solve, one replica per CTA.
__device__ __forceinline__ void persist_begin(const PersistArgs &a, PersistShared &sh) {
  if (threadIdx.x == 0) {
    CgState &st = sh.st;
    st.rho = st.rho1 = st.alpha = st.beta = st.pq = st.rr = 0.0;
    st.bnrm2 = st.resid = st.rr_true = 0.0;
    st.tol = a.prm->tol;
    st.maxit = a.prm->maxit;
    st.iter = 1;
    st.done = st.error = st.n_indef = st.recompute = st.converged = st.zero_rhs = 0;
    st.guard = 0;
    st.inner = st.flexible = st.use_gnn = st.restart = st.fallback = 0;
    st.omega = st.c2 = 0.0;
    st.nrecompute = kIterRecomputeR;
    st.resid_mark = 1.0;
    st.gamma = 1.0f;
    st.reliable = st.ru_pending = st.ru_count = 0;
    st.ru_delta = a.prm->ru_delta;
    st.ru_mark = 1.0;
    const bool log = blockIdx.x == 0;  // every CTA takes the same decisions, one records them
    st.lanczos = log ? a.prm->lanczos : nullptr;
    st.lanczos_cap = a.prm->lanczos_cap;
    st.rhist = log ? a.prm->rhist : nullptr;
    st.rhist_cap = a.prm->rhist_cap;
    st.lanczos_n = st.rhist_n = 0;
    for (int i = 0; i < 8; i++) st.ticket[i] = 0u;
    sh.dead = 0;
  }
  __syncthreads();
}

// ||b||^2, and whether the loop runs at all.
__device__ __forceinline__ void persist_bnrm(PersistShared &sh, double bb) {
  if (threadIdx.x == 0) {
    CgState &st = sh.st;
    st.bnrm2 = bb;
    if (bb == 0.0) {
      st.zero_rhs = 1;
      st.done = 1;
    }
    if (st.maxit <= 0) st.done = 1;
  }
  __syncthreads();
}

// The residual recomputed from b - A x (every 50th iteration, or below the tolerance).
__device__ __forceinline__ void persist_true_resid(PersistShared &sh, double rr, bool refresh) {
  if (threadIdx.x == 0) {
    CgState &st = sh.st;
    st.rr = rr;
    st.resid = sqrt(rr / st.bnrm2);
    if (refresh) record_resid(&st);
    if (st.resid <= st.tol) {
      st.done = 1;
      st.converged = 1;
    }
  }
}

// The end of an iteration.
__device__ __forceinline__ void persist_ctl(PersistShared &sh) {
  if (threadIdx.x == 0) {
    loop_ctl(&sh.st, 0, 0);
    if (sh.dead) sh.st.done = 1;
  }
  __syncthreads();
}

// The state out, after the last use of the vectors.
__device__ __forceinline__ void persist_end(const PersistArgs &a, PersistShared &sh) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (sh.dead) {
      sh.st.error = HECMW33_ERR_TIMEOUT;
      sh.st.done = 1;
    }
    *a.st = sh.st;
  }
}

template <int K, bool CLUSTER>
__global__ void __launch_bounds__(32 * persist_warps<K>(), 1) cg_ssor_persist_kernel(const PersistArgs a) {
  __shared__ PersistShared sh;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int w = warp * gridDim.x + blockIdx.x;  // this warp's list: neighbouring slices on different SMs
  const int gt = blockIdx.x * blockDim.x + tid, nt = gridDim.x * blockDim.x;
  GridWay way;
  persist_begin(a, sh);
  // x in position order; z and u start at zero (padding blocks gather position 0), and what
  // the first iteration reads of p, q, h and pl
  for (int i = gt; i < a.n; i += nt) {
    const int node = a.perm[i];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      a.px[3 * i + c] = a.x[3 * node + c];
      a.v.zu[3 * size_t(i) + c] = make_double2(0.0, 0.0);
      a.v.p[3 * i + c] = a.v.q[3 * i + c] = a.v.h[3 * i + c] = 0.0;
      a.v.pl[3 * i + c] = 0.0f;
    }
  }
  CgState &st = sh.st;
  persist_bnrm(sh, persist_sum<CLUSTER>(a, sh, way, persist_resid<true>(a), 0));
  const int n3 = 3 * a.n, n2 = n3 / 2;
  bool restart = true;  // g from r
  while (!st.done) {
    if (restart) {
      persist_sweep<K, 2, CLUSTER>(a, sh, way, w, 0.0, false);
      persist_barrier<CLUSTER>(a, sh, way);
      restart = false;
    }
    if (tid == 0) st.guard++;
    const double rho = persist_sum<CLUSTER>(a, sh, way, persist_sweep<K, 0, CLUSTER>(a, sh, way, w, 0.0, false), 0);
    if (tid == 0) fin_rho(&st, rho);
    __syncthreads();
    if (st.done) break;
    const bool first = st.iter == 1;
    const double pq =
        persist_sum<CLUSTER>(a, sh, way, persist_sweep<K, 1, CLUSTER>(a, sh, way, w, st.beta, first), 1);
    if (tid == 0) fin_pq(&st, pq);
    __syncthreads();
    if (st.done) break;
    const bool refresh = (st.iter % st.nrecompute) == 0;
    {
      const double alpha = st.alpha;
      double rr = 0.0;
      double2 *x2 = reinterpret_cast<double2 *>(a.px), *r2 = reinterpret_cast<double2 *>(a.pr),
              *g2 = reinterpret_cast<double2 *>(a.v.g);
      const double2 *p2 = reinterpret_cast<const double2 *>(a.pp), *q2 = reinterpret_cast<const double2 *>(a.pq),
                    *h2 = reinterpret_cast<const double2 *>(a.v.h);
      for (int i = gt; i < n2; i += nt) {
        double2 x = __ldcg(x2 + i);
        const double2 p = __ldcg(p2 + i);
        x.x = alpha * p.x + x.x;
        x.y = alpha * p.y + x.y;
        x2[i] = x;
        if (!refresh) {
          double2 r = __ldcg(r2 + i), g = __ldcg(g2 + i);
          const double2 q = __ldcg(q2 + i), h = __ldcg(h2 + i);
          r.x = -alpha * q.x + r.x;
          r.y = -alpha * q.y + r.y;
          g.x = -alpha * h.x + g.x;
          g.y = -alpha * h.y + g.y;
          r2[i] = r;
          g2[i] = g;
          rr += r.x * r.x + r.y * r.y;
        }
      }
      if (gt == nt - 1 && (n3 & 1)) {
        const int i = n3 - 1;
        a.px[i] = alpha * __ldcg(a.pp + i) + __ldcg(a.px + i);
        if (!refresh) {
          const double r = -alpha * __ldcg(a.pq + i) + __ldcg(a.pr + i);
          a.pr[i] = r;
          a.v.g[i] = -alpha * __ldcg(a.v.h + i) + __ldcg(a.v.g + i);
          rr += r * r;
        }
      }
      if (refresh) persist_barrier<CLUSTER>(a, sh, way);
      else {
        rr = persist_sum<CLUSTER>(a, sh, way, rr, 2);
        if (tid == 0) fin_rr(&st, rr);
        __syncthreads();
      }
    }
    if (refresh || st.recompute) {
      for (int i = gt; i < a.n; i += nt) {
        const int node = a.perm[i];
#pragma unroll
        for (int c = 0; c < 3; c++) a.x[3 * node + c] = __ldcg(a.px + 3 * i + c);
      }
      persist_barrier<CLUSTER>(a, sh, way);
      persist_true_resid(sh, persist_sum<CLUSTER>(a, sh, way, persist_resid<false>(a), 2), refresh);
      restart = true;
    }
    persist_ctl(sh);
  }
  if (!sh.dead && !st.zero_rhs) {
    for (int i = gt; i < a.n; i += nt) {
      const int node = a.perm[i];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        a.x[3 * node + c] = __ldcg(a.px + 3 * i + c);
        a.r[3 * node + c] = __ldcg(a.pr + 3 * i + c);
      }
    }
  }
  persist_end(a, sh);
  if constexpr (CLUSTER) persist_barrier<true>(a, sh, way);
}

// ---- one application of the SSOR ---------------------------------------------------
// z = M^-1 r in one launch, for the methods whose loop is not one (BiCGSTAB, GMRES, ...):
// the colour kernels' arithmetic in their order (sweep_fwd_uni_kernel,
// sweep_bwd_uni_kernel), a grid barrier where they have a launch.  bar: arrivals, whether
// a wait gave up, CTAs that are done (the last sets the first and third back to zero).
struct ApplyArgs {
  SellView<double> lo, up;
  const int4 *lo_items, *up_items;
  int lo_stride, up_stride;
  const int *perm;
  const double *alu;
  int n, ncolor;
  const double *r;
  double *z, *zpos;
  const CgState *st;
  unsigned *bar;
  int polls;
};

template <int K>
__global__ void __launch_bounds__(32 * persist_warps<K>(), 1) ssor_apply_persist_kernel(const ApplyArgs a) {
  if (a.st && a.st->done) return;
  __shared__ int dead;
  const int lane = threadIdx.x & 31, roff = lane / K;
  const bool leader = (lane & (K - 1)) == 0;
  const int w = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  GridWay way;
  if (threadIdx.x == 0) dead = 0;
  const auto barrier = [&] {
    way.target += gridDim.x;
    way.gone = dead;
    __syncthreads();
    if (threadIdx.x == 0) grid_meet(a.bar, way, a.polls, dead);
    __syncthreads();
  };
  {
    ListCursor cur{a.lo_items + size_t(w) * a.lo_stride, a.ncolor};
    int4 it = cur.next();
    for (int c = 0; c < a.ncolor; c++) {
      if (c) barrier();
      while ((it.w >> 6) == c) {
        const int row = it.z + roff;
        const bool act = roff < (it.w & 63) && leader;
        double r0 = 0.0, r1 = 0.0, r2 = 0.0;
        if (act) {
          const int node = a.perm[row];
          r0 = a.r[3 * node];
          r1 = a.r[3 * node + 1];
          r2 = a.r[3 * node + 2];
        }
        double y0 = 0.0, y1 = 0.0, y2 = 0.0;
        slice_gemv_u<double, double, K, false, true>(a.lo, it.x, it.y, lane, a.zpos, y0, y1, y2);
        if (act) {
          double x1 = r0 - y0, x2 = r1 - y1, x3 = r2 - y2;
          lu_solve(a.alu, a.n, row, x1, x2, x3);
          a.zpos[3 * row] = x1;
          a.zpos[3 * row + 1] = x2;
          a.zpos[3 * row + 2] = x3;
        }
        it = cur.next();
      }
    }
  }
  ListCursor cur{a.up_items + size_t(w) * a.up_stride, a.ncolor};
  int4 it = cur.next();
  for (int c = 0; c < a.ncolor; c++) {
    barrier();
    while ((it.w >> 6) == c) {
      const int row = it.z + roff;
      const bool act = roff < (it.w & 63) && leader;
      int node = 0;
      double c0 = 0.0, c1 = 0.0, c2 = 0.0;
      if (act) {
        node = a.perm[row];
        c0 = __ldcg(a.zpos + 3 * row);
        c1 = __ldcg(a.zpos + 3 * row + 1);
        c2 = __ldcg(a.zpos + 3 * row + 2);
      }
      double x1 = 0.0, x2 = 0.0, x3 = 0.0;
      slice_gemv_u<double, double, K, true, true>(a.up, it.x, it.y, lane, a.zpos, x1, x2, x3);
      if (act) {
        lu_solve(a.alu, a.n, row, x1, x2, x3);
        const double z0 = c0 - x1, z1 = c1 - x2, z2 = c2 - x3;
        a.zpos[3 * row] = z0;
        a.zpos[3 * row + 1] = z1;
        a.zpos[3 * row + 2] = z2;
        a.z[3 * node] = z0;
        a.z[3 * node + 1] = z1;
        a.z[3 * node + 2] = z2;
      }
      it = cur.next();
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(a.bar + 2, 1u) == gridDim.x - 1) {
      a.bar[0] = 0u;
      a.bar[2] = 0u;
    }
  }
}

// ---- block ILU ----------------------------------------------------------------------
// The CG with a block ILU(p) preconditioner, whose levels take the place of the colours:
// its triangles are not A's, so q = A p is a pass of its own, and the vectors stay in
// node order.  A level of a lexicographically numbered box has a few hundred rows, so the
// solve is the latency of its two chains of levels: at 40^3 elements (281 + 281) an
// iteration took 4.5 ms as one launch per level and takes 1.68 ms here, 3 us a level of
// which the barrier with the stores before it and the first load after it are 1.65.
//
// One direction: forward z = LU^-1 (r - L z), backward z -= LU^-1 (U z) with RHO = r.z.
template <int K, bool BACK, bool CLUSTER>
__device__ __forceinline__ double persist_levels(const PersistArgs &a, PersistShared &sh, GridWay &way, int w) {
  constexpr int U = 2;
  const int lane = threadIdx.x & 31;
  const int sub = lane & (K - 1), roff = lane / K;
  const PersistSweep S = BACK ? a.up : a.lo;
  const double *alu = BACK ? a.alu_b : a.alu;
  const int *perm = BACK ? a.perm_b : a.perm;
  const int nstep = BACK ? a.nback : a.ncolor;
  const int4 *items = S.items + size_t(w) * S.stride;
  const size_t n = size_t(a.n);
  double dot = 0.0;
  int4 it = __ldg(items), nx = __ldg(items + 1);
  items += 2;
  int col[U];
#pragma unroll
  for (int u = 0; u < U; u++) col[u] = u < it.y ? __ldg(S.col + (it.x + u) * 32 + lane) : 0;
  int node = it.w == kPEnd ? 0 : __ldg(perm + it.z + (roff < (it.w & 63) ? roff : 0));
  for (int c = 0; c < nstep; c++) {
    if (c) persist_barrier<CLUSTER>(a, sh, way);
    while ((it.w >> 6) == c) {
      const bool act = roff < (it.w & 63);
      const int row = it.z + (act ? roff : 0), i3 = 3 * node;
      const double *lu = alu + row;
      const double a0 = __ldcs(lu), a1 = __ldcs(lu + n), a2 = __ldcs(lu + 2 * n);
      const double a3 = __ldcs(lu + 3 * n), a4 = __ldcs(lu + 4 * n), a5 = __ldcs(lu + 5 * n);
      const double a6 = __ldcs(lu + 6 * n), a7 = __ldcs(lu + 7 * n), a8 = __ldcs(lu + 8 * n);
      const double *own = (BACK ? a.pz : a.r) + i3;
      const double o0 = __ldcg(own), o1 = __ldcg(own + 1), o2 = __ldcg(own + 2);
      const double rc = BACK ? __ldcg(a.r + i3 + min(sub, 2)) : 0.0;
      double l[3] = {0.0, 0.0, 0.0};
      const int next = nx.w == kPEnd ? 0 : __ldg(perm + nx.z + (roff < (nx.w & 63) ? roff : 0));
      for (int s = 0; s < it.y; s += U) {
        const int nu = it.y - s;
        double x[U][3], v[U][9];
#pragma unroll
        for (int u = 0; u < U; u++) {
#pragma unroll
          for (int j = 0; j < 3; j++) x[u][j] = 0.0;
#pragma unroll
          for (int e = 0; e < 9; e++) v[u][e] = 0.0;
          if (u < nu) {
            const double *g = a.pz + 3 * size_t(col[u]);
#pragma unroll
            for (int j = 0; j < 3; j++) x[u][j] = ld_row<CLUSTER>(g + j);
            const double *b = S.val + size_t(it.x + s + u) * 288 + lane;
#pragma unroll
            for (int e = 0; e < 9; e++) v[u][e] = __ldcs(b + 32 * e);
          }
        }
        const bool more = nu > U;
        const int slot = more ? it.x + s + U : nx.x, left = more ? nu - U : nx.y;
#pragma unroll
        for (int u = 0; u < U; u++)
          if (u < left) col[u] = __ldg(S.col + (slot + u) * 32 + lane);
#pragma unroll
        for (int u = 0; u < U; u++)
          if (u < nu) {
#pragma unroll
            for (int i = 0; i < 3; i++)
              l[i] = fma(v[u][3 * i + 2], x[u][2], fma(v[u][3 * i + 1], x[u][1], fma(v[u][3 * i], x[u][0], l[i])));
          }
      }
      if (it.y == 0) {
#pragma unroll
        for (int u = 0; u < U; u++)
          if (u < nx.y) col[u] = __ldg(S.col + (nx.x + u) * 32 + lane);
      }
#pragma unroll
      for (int o = K / 2; o > 0; o >>= 1) {
#pragma unroll
        for (int j = 0; j < 3; j++) l[j] += __shfl_xor_sync(0xffffffffu, l[j], o);
      }
      double x1 = BACK ? l[0] : o0 - l[0], x2 = BACK ? l[1] : o1 - l[1], x3 = BACK ? l[2] : o2 - l[2];
      x2 = x2 - a3 * x1;
      x3 = x3 - a6 * x1 - a7 * x2;
      x3 = a8 * x3;
      x2 = a4 * (x2 - a5 * x3);
      x1 = a0 * (x1 - a2 * x3 - a1 * x2);
      if (act && sub < 3) {
        double zc = sub == 0 ? x1 : sub == 1 ? x2 : x3;
        if (BACK) {
          zc = (sub == 0 ? o0 : sub == 1 ? o1 : o2) - zc;
          dot += rc * zc;
        }
        a.pz[i3 + sub] = zc;
      }
      it = nx;
      node = next;
      nx = __ldg(items);
      if (nx.w != kPEnd) items++;
    }
  }
  return dot;
}

// q = A p over the grid with the partial of p.q.
__device__ __forceinline__ double persist_product(const PersistArgs &a) {
  const int lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  double acc = 0.0;
  for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < a.A.nslices; s += nw) {
    const bool active = lane < a.A.nrows[s];
    const int row = a.A.row0[s] + lane;
    const int len = active ? a.A.rowlen[s * 32 + lane] : 0;
    double y0 = 0.0, y1 = 0.0, y2 = 0.0;
    row_gemv<double, double, 1, false, true>(a.A, s, lane, len, a.pp, y0, y1, y2);
    if (active) {
      a.pq[3 * row] = y0;
      a.pq[3 * row + 1] = y1;
      a.pq[3 * row + 2] = y2;
      acc += __ldcg(a.pp + 3 * row) * y0 + __ldcg(a.pp + 3 * row + 1) * y1 + __ldcg(a.pp + 3 * row + 2) * y2;
    }
  }
  return acc;
}

template <int K, bool CLUSTER>
__global__ void __launch_bounds__(32 * persist_warps<K>(), 1) cg_ilu_persist_kernel(const PersistArgs a) {
  __shared__ PersistShared sh;
  const int tid = threadIdx.x;
  const int w = (tid >> 5) * gridDim.x + blockIdx.x;
  const int gt = blockIdx.x * blockDim.x + tid, nt = gridDim.x * blockDim.x;
  GridWay way;
  persist_begin(a, sh);
  const int n3 = 3 * a.n;
  for (int i = gt; i < n3; i += nt) a.pz[i] = 0.0;  // padding blocks gather node 0
  persist_bnrm(sh, persist_sum<CLUSTER>(a, sh, way, persist_resid<true>(a), 0));
  CgState &st = sh.st;
  while (!st.done) {
    if (tid == 0) st.guard++;
    persist_levels<K, false, CLUSTER>(a, sh, way, w);
    persist_barrier<CLUSTER>(a, sh, way);
    const double rho = persist_sum<CLUSTER>(a, sh, way, persist_levels<K, true, CLUSTER>(a, sh, way, w), 0);
    if (tid == 0) fin_rho(&st, rho);
    __syncthreads();
    if (st.done) break;
    const bool first = st.iter == 1;
    const double beta = st.beta;
    for (int i = gt; i < n3; i += nt) {
      const double z = __ldcg(a.pz + i);
      a.pp[i] = first ? z : z + beta * __ldcg(a.pp + i);
    }
    persist_barrier<CLUSTER>(a, sh, way);
    const double pq = persist_sum<CLUSTER>(a, sh, way, persist_product(a), 1);
    if (tid == 0) fin_pq(&st, pq);
    __syncthreads();
    if (st.done) break;
    const bool refresh = (st.iter % st.nrecompute) == 0;
    const double alpha = st.alpha;
    double rr = 0.0;
    for (int i = gt; i < n3; i += nt) {
      a.x[i] = alpha * __ldcg(a.pp + i) + __ldcg(a.x + i);
      if (!refresh) {
        const double r = -alpha * __ldcg(a.pq + i) + __ldcg(a.r + i);
        a.r[i] = r;
        rr += r * r;
      }
    }
    rr = persist_sum<CLUSTER>(a, sh, way, rr, 2);
    if (!refresh) {
      if (tid == 0) fin_rr(&st, rr);
      __syncthreads();
    }
    if (refresh || st.recompute)
      persist_true_resid(sh, persist_sum<CLUSTER>(a, sh, way, persist_resid<false>(a), 1), refresh);
    // r (and x) are complete at a barrier before the next sweep gathers or overwrites
    persist_ctl(sh);
  }
  persist_end(a, sh);
  if constexpr (CLUSTER) persist_barrier<true>(a, sh, way);
}

}  // namespace h33
