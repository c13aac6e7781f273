// h33_multi_persist.cuh -- the CG + SSOR of up to 16 load cases in one persistent launch:
// the fused iteration of h33_persist.cuh (no product: A z = g + L z out of the forward
// sweep that reads L anyway) with 16 vectors, a half-warp per block row and a lane per
// load case, as the kernels of h33_multi.cuh.
//
// What bounds it: the latency of a row's chain (columns and entries, the 384-byte
// gathers, the solve), two or three rows a half-warp and colour.  The colour launches
// handed a block's entries round by 19 shuffles, 26 blocks a row in the sweeps and 27 in
// the product; here they pass through shared memory (5 vector loads a block) and L's serve
// two products.  Measured per iteration with 16 load cases against the colour launches
// (us): 378 nodes 149 / 204, 19 thousand 287 / 352 (8 warps a CTA), 118 thousand 696 / 783,
// but 275 thousand 1521 / 1477 (with the row's vectors still loaded one by one), where 105 MB
// a vector stream through HBM and the launches' 24 warps an SM hide it better
// (run_multi_chunk's rule).  Measured and dropped: 20 or 24
// warps a CTA (spills: 753 to 840 at 118 thousand), the next row's blocks held in
// registers (922).
#pragma once

#include "h33_multi.cuh"
#include "h33_persist.cuh"

namespace h33 {

constexpr int kMrWarps = 16;  // most warps of a CTA
constexpr int kMrThreads = 32 * kMrWarps;
constexpr int kMrBlock = 5;  // double2 per staged block: nine entries and the column

struct MrPersistArgs {
  SellView<double> lo, up, A;  // A: 16 lanes per row, node order
  const int *rows, *lo_gs, *up_gs;  // colour g: rows [rows[g], rows[g+1]), from slice gs[g]
  const double *alu;
  const int *perm, *iperm;
  const double *b;             // node order, 48 doubles per node
  double *x;                   // node order
  double *px, *r, *g, *p, *q, *h, *z, *u;  // position order
  float *pl;                   // what p's rounding dropped, position order
  CgState *st;                 // kMaxRhs states out
  MultiCtl *ctl;
  const CgParams *prm;
  double *parts;               // 3 x gridDim.x x 16
  unsigned *bar;
  int polls;
  int n, ncolor, nrhs;
};

struct MrShared {
  CgState st[kMaxRhs];
  double red[2 * kMrWarps][kMaxRhs];
  double res[kMaxRhs];
  int again[kMaxRhs];  // load cases whose g has to be made from r
  int any, dead;
  double2 blk[2 * kMrWarps][16 * kMrBlock];  // last: as many as the CTA has half-warps
};

__device__ __forceinline__ void mr_persist_barrier(const MrPersistArgs &a, MrShared &sh, GridWay &way) {
  way.target += gridDim.x;
  way.gone = sh.dead;  // as in the single application
  __syncthreads();
  if (threadIdx.x == 0) grid_meet(a.bar, way, a.polls, sh.dead);
  __syncthreads();
}

// Sum over the grid for every load case, in sh.res; includes a barrier.
__device__ __forceinline__ void mr_persist_sum(const MrPersistArgs &a, MrShared &sh, GridWay &way, double v,
                                               int slot) {
  const int l = threadIdx.x & 15, hw = threadIdx.x >> 4, nh = blockDim.x >> 4;
  double *parts = a.parts + size_t(slot) * gridDim.x * kMaxRhs;
  sh.red[hw][l] = v;
  __syncthreads();
  if (threadIdx.x < kMaxRhs) {
    double s = 0.0;
    for (int k = 0; k < nh; k++) s += sh.red[k][threadIdx.x];
    parts[size_t(blockIdx.x) * kMaxRhs + threadIdx.x] = s;
  }
  mr_persist_barrier(a, sh, way);
  double s = 0.0;
  for (int i = hw; i < int(gridDim.x); i += nh) s += __ldcg(parts + size_t(i) * kMaxRhs + l);
  sh.red[hw][l] = s;
  __syncthreads();
  if (threadIdx.x < kMaxRhs) {
    double t = 0.0;
    for (int k = 0; k < nh; k++) t += sh.red[k][threadIdx.x];
    sh.res[threadIdx.x] = t;
  }
  __syncthreads();
}

// m += A(row, :) y and, with TWO, l += A(row, :) x for this lane's load case: the row 16
// blocks at a time, lane j of the half-warp staging block j's entries and column.  x and
// y are read coherently (they are written during the launch).
template <int K, bool TWO>
__device__ __forceinline__ void mr_persist_row(const SellView<double> &A, int s, int roff, int len, int lane,
                                               unsigned hmask, double2 *blk, const double *x, const double *y,
                                               double (&l)[3], double (&m)[3]) {
  const int slot0 = __ldg(A.slot0 + s);
  for (int k0 = 0; k0 < len; k0 += 16) {
    const int kn = min(16, len - k0);
    __syncwarp(hmask);
    if (lane < kn) {
      const int k = k0 + lane;
      const int sl = slot0 + k / K, lp = roff * K + (k & (K - 1));
      const int c = __ldg(A.col + sl * 32 + lp);
      const double *v = A.val + size_t(sl) * 288 + lp;
      double e[9];
#pragma unroll
      for (int i = 0; i < 9; i++) e[i] = __ldg(v + 32 * i);
      double2 *o = blk + lane * kMrBlock;
      o[0] = make_double2(e[0], e[1]);
      o[1] = make_double2(e[2], e[3]);
      o[2] = make_double2(e[4], e[5]);
      o[3] = make_double2(e[6], e[7]);
      o[4] = make_double2(e[8], __hiloint2double(0, c));
    }
    __syncwarp(hmask);
#pragma unroll(TWO ? 4 : 8)
    for (int kk = 0; kk < kn; kk++) {
      const double2 *o = blk + kk * kMrBlock;
      const double2 e4 = o[4];
      const size_t c = size_t(__double2loint(e4.y)) * kRhsStride + lane;
      const double y0 = y[c], y1 = y[c + 16], y2 = y[c + 32];
      double x0 = 0.0, x1 = 0.0, x2 = 0.0;
      if (TWO) x0 = x[c], x1 = x[c + 16], x2 = x[c + 32];
      const double2 e0 = o[0], e1 = o[1], e2 = o[2], e3 = o[3];
      m[0] = fma(e1.x, y2, fma(e0.y, y1, fma(e0.x, y0, m[0])));
      m[1] = fma(e2.y, y2, fma(e2.x, y1, fma(e1.y, y0, m[1])));
      m[2] = fma(e4.x, y2, fma(e3.y, y1, fma(e3.x, y0, m[2])));
      if (TWO) {
        l[0] = fma(e1.x, x2, fma(e0.y, x1, fma(e0.x, x0, l[0])));
        l[1] = fma(e2.y, x2, fma(e2.x, x1, fma(e1.y, x0, l[1])));
        l[2] = fma(e4.x, x2, fma(e3.y, x1, fma(e3.x, x0, l[2])));
      }
    }
  }
}

// One sweep: MODE 0 backward, 1 forward on the direction, 2 forward from r for the load
// cases of sh.again (start and refresh; the others keep g).
template <int K, int MODE>
__device__ __forceinline__ double mr_persist_sweep(const MrPersistArgs &a, MrShared &sh, GridWay &way) {
  constexpr int RPS = 32 / K;
  const int lane = threadIdx.x & 15, hwl = threadIdx.x >> 4;
  const int hw = hwl * gridDim.x + blockIdx.x, nhw = (blockDim.x >> 4) * gridDim.x;
  const unsigned hmask = (threadIdx.x & 16) ? 0xffff0000u : 0x0000ffffu;
  const SellView<double> &L = MODE == 0 ? a.up : a.lo;
  const int *gs = MODE == 0 ? a.up_gs : a.lo_gs;
  const bool live = !sh.st[lane].done, first = sh.st[lane].iter == 1, again = sh.again[lane] != 0;
  const double beta = sh.st[lane].beta;
  const size_t n = size_t(a.n);
  double dot = 0.0;
  for (int c = 0; c < a.ncolor; c++) {
    const int g = MODE == 0 ? a.ncolor - 1 - c : c;
    const int r0 = __ldg(a.rows + g), r1 = __ldg(a.rows + g + 1), s0 = __ldg(gs + g);
    int row = r0 + hw, s = s0 + (row - r0) / RPS, roff = (row - r0) % RPS;
    int len = row < r1 ? __ldg(L.rowlen + s * 32 + roff) : 0;
    if (c) mr_persist_barrier(a, sh, way);
    while (row < r1) {
      const double *lu = a.alu + row;
      const double a0 = __ldg(lu), a1 = __ldg(lu + n), a2 = __ldg(lu + 2 * n);
      const double a3 = __ldg(lu + 3 * n), a4 = __ldg(lu + 4 * n), a5 = __ldg(lu + 5 * n);
      const double a6 = __ldg(lu + 6 * n), a7 = __ldg(lu + 7 * n), a8 = __ldg(lu + 8 * n);
      const size_t o = size_t(row) * kRhsStride + lane;
      const double *own = (MODE == 0 ? a.g : MODE == 1 ? a.u : a.r) + o;  // g, v or r
      const double o0 = __ldcg(own), o1 = __ldcg(own + 16), o2 = __ldcg(own + 32);
      double lz[3] = {0.0, 0.0, 0.0}, lu_[3] = {0.0, 0.0, 0.0};
      mr_persist_row<K, MODE == 1>(L, s, roff, len, lane, hmask, sh.blk[hwl], a.z, MODE == 0 ? a.z : a.u, lz, lu_);
      const double e[3] = {o0 - lu_[0], o1 - lu_[1], o2 - lu_[2]};
      double x[3] = {e[0], e[1], e[2]};  // D^-1 e by the reciprocal-pivot LU
      x[1] = x[1] - a3 * x[0];
      x[2] = x[2] - a6 * x[0] - a7 * x[1];
      x[2] = a8 * x[2];
      x[1] = a4 * (x[1] - a5 * x[2]);
      x[0] = a0 * (x[0] - a2 * x[2] - a1 * x[1]);
      // the row's other vectors, their loads together (they took turns with the stores before:
      // 16 cases on 118 thousand nodes 252 ms a solve, 226 so)
      double f[3][5] = {};
      float fl[3] = {};
      if (MODE == 0 || (MODE == 1 && live)) {
#pragma unroll
        for (int i = 0; i < 3; i++) {
          const size_t k = o + 16 * i;
          f[i][0] = __ldcg((MODE == 0 ? a.r : a.g) + k);
          if (MODE == 1) {
            f[i][1] = __ldcg(a.z + k);
            if (!first) {
              f[i][2] = __ldcg(a.p + k);
              f[i][3] = __ldcg(a.q + k);
              f[i][4] = __ldcg(a.h + k);
              fl[i] = __ldcg(a.pl + k);
            }
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const size_t k = o + 16 * i;
        a.u[k] = MODE == 0 ? lu_[i] : x[i];
        if (MODE == 0) {  // z = D^-1 (g - U z) and v = U z
          a.z[k] = x[i];
          dot += f[i][0] * x[i];
        } else if (MODE == 2) {
          if (again) a.g[k] = e[i];
        } else if (live) {
          float rest;  // first: BETA and the old vectors are zero
          const double pn = next_direction(f[i][1], beta, f[i][2], fl[i], rest);
          const double qn = f[i][0] + lz[i] + beta * f[i][3], hn = f[i][0] - lu_[i] + beta * f[i][4];
          a.p[k] = pn;
          a.pl[k] = rest;
          a.q[k] = qn;
          a.h[k] = hn;
          dot += pn * qn;
        }
      }
      row += nhw;
      s = s0 + (row - r0) / RPS;
      roff = (row - r0) % RPS;
      len = row < r1 ? __ldg(L.rowlen + s * 32 + roff) : 0;
    }
  }
  return dot;
}

// r = b - A x (x in node order, r in position order) for the load cases with `mine`;
// |r|^2 or (BB) |b|^2 of this lane's load case.
template <bool BB>
__device__ __forceinline__ double mr_persist_resid(const MrPersistArgs &a, MrShared &sh, bool mine) {
  const int lane = threadIdx.x & 15, hwl = threadIdx.x >> 4;
  const int hw = hwl * gridDim.x + blockIdx.x, nhw = (blockDim.x >> 4) * gridDim.x;
  const unsigned hmask = (threadIdx.x & 16) ? 0xffff0000u : 0x0000ffffu;
  double acc = 0.0;
  for (int row = hw; row < a.n; row += nhw) {
    const int s = row / 2, roff = row & 1;  // 16 lanes per row: two rows a slice
    double y[3] = {0.0, 0.0, 0.0}, none[3] = {0.0, 0.0, 0.0};
    mr_persist_row<kMrLanes, false>(a.A, s, roff, __ldg(a.A.rowlen + s * 32 + roff), lane, hmask, sh.blk[hwl], a.x, a.x,
                                    none, y);
    const size_t o = size_t(row) * kRhsStride + lane, k = size_t(a.iperm[row]) * kRhsStride + lane;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double b = a.b[o + 16 * i], r = b - y[i];
      if (mine) a.r[k + 16 * i] = r;
      acc += BB ? b * b : r * r;
    }
  }
  return acc;
}

template <int K>
__global__ void __launch_bounds__(kMrThreads, 1) mr_cg_persist_kernel(const MrPersistArgs a) {
  extern __shared__ __align__(16) unsigned char mr_smem[];
  MrShared &sh = *reinterpret_cast<MrShared *>(mr_smem);
  const int tid = threadIdx.x, lane = tid & 15;
  const int hw = (tid >> 4) * gridDim.x + blockIdx.x, nhw = (blockDim.x >> 4) * gridDim.x;
  GridWay way;
  if (tid < kMaxRhs) {
    CgState s = {};
    s.tol = a.prm->tol;
    s.maxit = a.prm->maxit;
    s.iter = 1;
    s.nrecompute = kIterRecomputeR;
    s.resid_mark = 1.0;
    s.gamma = 1.0f;
    s.ru_mark = 1.0;
    sh.st[tid] = s;
    sh.again[tid] = 1;
  }
  if (tid == 0) sh.dead = 0;
  __syncthreads();
  // x in position order; z and u start at zero (padding blocks gather position 0)
  for (int i = hw; i < a.n; i += nhw) {
    const size_t o = size_t(i) * kRhsStride + lane, k = size_t(a.perm[i]) * kRhsStride + lane;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      a.px[o + 16 * c] = a.x[k + 16 * c];
      a.z[o + 16 * c] = 0.0;
      a.u[o + 16 * c] = 0.0;
    }
  }
  const auto nodes_x = [&] {
    for (int i = hw; i < a.n; i += nhw) {
      const size_t o = size_t(i) * kRhsStride + lane, k = size_t(a.perm[i]) * kRhsStride + lane;
#pragma unroll
      for (int c = 0; c < 3; c++) a.x[k + 16 * c] = __ldcg(a.px + o + 16 * c);
    }
  };
  const auto decide = [&] {  // whether a load case still iterates
    if (tid == 0) {
      int any = 0;
      for (int k = 0; k < kMaxRhs; k++) any |= !sh.st[k].done;
      sh.any = any && !sh.dead;
    }
    __syncthreads();
  };
  mr_persist_sum(a, sh, way, mr_persist_resid<true>(a, sh, true), 0);
  if (tid < kMaxRhs) {
    CgState &s = sh.st[tid];
    s.bnrm2 = sh.res[tid];
    if (tid >= a.nrhs) {
      s.done = 1;  // padding lane
    } else if (s.bnrm2 == 0.0) {
      s.zero_rhs = 1;
      s.done = 1;
    }
    if (s.maxit <= 0) s.done = 1;
  }
  __syncthreads();
  decide();
  int guard = 0;
  bool restart = true;
  while (sh.any) {
    guard++;
    if (restart) {
      mr_persist_sweep<K, 2>(a, sh, way);
      mr_persist_barrier(a, sh, way);
    }
    if (tid < kMaxRhs) {
      if (!sh.st[tid].done) sh.st[tid].guard++;
      sh.again[tid] = 0;
    }
    __syncthreads();
    mr_persist_sum(a, sh, way, mr_persist_sweep<K, 0>(a, sh, way), 0);
    if (tid < kMaxRhs && !sh.st[tid].done) fin_rho(&sh.st[tid], sh.res[tid]);
    __syncthreads();
    mr_persist_sum(a, sh, way, mr_persist_sweep<K, 1>(a, sh, way), 1);
    if (tid < kMaxRhs && !sh.st[tid].done) fin_pq(&sh.st[tid], sh.res[tid]);
    __syncthreads();
    {
      const CgState &s = sh.st[lane];
      const bool live = !s.done, refresh = (s.iter % kIterRecomputeR) == 0;
      const double alpha = s.alpha;
      double rr = 0.0;
      if (live)
        for (int i = hw; i < a.n; i += nhw) {
          const size_t o = size_t(i) * kRhsStride + lane;
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const size_t k = o + 16 * c;
            a.px[k] = alpha * __ldcg(a.p + k) + __ldcg(a.px + k);
            if (!refresh) {
              const double r = -alpha * __ldcg(a.q + k) + __ldcg(a.r + k);
              a.r[k] = r;
              a.g[k] = -alpha * __ldcg(a.h + k) + __ldcg(a.g + k);
              rr += r * r;
            }
          }
        }
      mr_persist_sum(a, sh, way, rr, 2);
    }
    if (tid < kMaxRhs) {
      CgState &s = sh.st[tid];
      if (!s.done && (s.iter % kIterRecomputeR) != 0) fin_rr(&s, sh.res[tid]);
      sh.again[tid] = !s.done && ((s.iter % kIterRecomputeR) == 0 || s.recompute);
    }
    const bool need = __syncthreads_or(tid < kMaxRhs && sh.again[tid]) != 0;
    restart = false;
    if (need) {  // a true residual is due for some load cases
      nodes_x();
      mr_persist_barrier(a, sh, way);
      mr_persist_sum(a, sh, way, mr_persist_resid<false>(a, sh, sh.again[lane] != 0), 1);
      if (tid < kMaxRhs && sh.again[tid]) {
        CgState &s = sh.st[tid];
        s.rr = sh.res[tid];
        s.resid = sqrt(s.rr / s.bnrm2);
        if (s.resid <= s.tol) {
          s.done = 1;
          s.converged = 1;
          sh.again[tid] = 0;
        }
      }
      restart = __syncthreads_or(tid < kMaxRhs && sh.again[tid]) != 0;
    }
    if (tid < kMaxRhs) loop_ctl(&sh.st[tid], 0, 0);
    __syncthreads();
    decide();
  }
  nodes_x();
  if (blockIdx.x == 0) {
    if (tid < kMaxRhs) a.st[tid] = sh.st[tid];
    if (tid == 0) {
      a.ctl->all_done = 1;
      a.ctl->guard = guard;
      a.ctl->nrhs = a.nrhs;
      a.ctl->fault = 0;  // a barrier that gave up: bar[1], read by the host
      for (int i = 0; i < 8; i++) a.ctl->ticket[i] = 0u;  // the kernels after this one count from zero
    }
  }
}

}  // namespace h33
