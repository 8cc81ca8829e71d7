// otm_direct.cuh -- the coarsest level's direct solve (replaces the host BiCGSTAB(ILUT) + nullspace
// projection of Grid_H::solveHostEquation, homogenization/grid.cpp:272-310).
//
// Once per update the dense FP64 inverse of A_c + (alpha/n) 1 1^T (SPD on the periodic nullspace,
// alpha the mean diagonal) is built by one cluster; each V-cycle applies it as a mat-vec.
//
// The inversion is an in-place block Gauss-Jordan elimination (SPD, no pivoting) in steps of kDirNB
// rows. The block rows are dealt round-robin to the cluster's CTAs, which keep them in shared memory
// (in global memory, L2-resident, when a CTA's share does not fit). Step K has a panel
// R = P A_K (P = A_KK^-1, with P itself in the columns K), made by the owner of block K; every other
// row i then takes A_i <- A_i - A_iK R (A_iK read first and set to zero), row block K becomes R.
// The owner of block K + 1 updates that block first and makes the next panel before it touches its
// other rows, and the other CTAs update theirs meanwhile: a step costs one cluster barrier, whose
// arrive and wait enclose those updates. Panels travel through global memory (two buffers): read
// from L2 by all CTAs at once, where copies out of the owner's shared memory would queue at its
// port. A warp's tile is 8 rows x 64 columns (16 FP64 accumulators a lane: per step of the inner
// product two column values and four broadcast pairs of row values feed 16 FMAs).
#pragma once

#include <cooperative_groups.h>

#include "otm_mg_kernels.cuh"

namespace otm {

constexpr int kDirNB = 16;        // rows per elimination step
constexpr int kDirThreads = 512;
constexpr int kDirWarps = kDirThreads / 32;
constexpr int kDirCl = 16;        // CTAs per cluster where that size can be scheduled, else 8

// Sizes of an inversion of n unknowns on a cluster of ncl CTAs.
struct DirPlan {
  int n, nb, npad;   // unknowns, block rows, nb * kDirNB (rows past n are the identity)
  int nloc;          // most block rows a CTA owns
  int smem_rows;     // the rows live in shared memory
  int ncl;
  size_t smem;       // dynamic shared memory per CTA (bytes)
  size_t work;       // global scratch (doubles): two panels, then the rows when not in shared memory
};

__host__ inline DirPlan dir_plan(int n, int ncl) {
  DirPlan p{};
  p.n = n;
  p.nb = (n + kDirNB - 1) / kDirNB;
  p.npad = p.nb * kDirNB;
  p.nloc = (p.nb + ncl - 1) / ncl;
  p.ncl = ncl;
  const size_t panel = size_t(kDirNB) * p.npad, lt = size_t(kDirNB) * p.nloc * kDirNB, pt = kDirNB * kDirNB;
  const size_t rows = size_t(p.nloc) * kDirNB * p.npad;
  p.smem_rows = (panel + lt + pt + rows) * sizeof(double) <= size_t(kMaxDynSmem);
  p.smem = (panel + lt + pt + (p.smem_rows ? rows : 0)) * sizeof(double);
  p.work = 2 * panel + (p.smem_rows ? 0 : rows * size_t(ncl));
  return p;
}

// acc[r][c] -= (kSub) or += sum_k Lt[k][r] R[k][j0 + lane + 32 c] over the kDirNB rows of R.
template <bool kSub>
__device__ __forceinline__ void dir_tile(const double* R, int npad, const double* Lt, int ls, int j, bool in0, bool in1,
                                         double (&acc)[8][2]) {
#pragma unroll 4
  for (int k = 0; k < kDirNB; k++) {
    const double b0 = in0 ? R[k * npad + j] : 0.0, b1 = in1 ? R[k * npad + j + 32] : 0.0;
    const double2* l2 = reinterpret_cast<const double2*>(Lt + k * ls);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const double2 l = l2[q];
      const double lx = kSub ? -l.x : l.x, ly = kSub ? -l.y : l.y;
      acc[2 * q][0] = fma(lx, b0, acc[2 * q][0]);
      acc[2 * q][1] = fma(lx, b1, acc[2 * q][1]);
      acc[2 * q + 1][0] = fma(ly, b0, acc[2 * q + 1][0]);
      acc[2 * q + 1][1] = fma(ly, b1, acc[2 * q + 1][1]);
    }
  }
}

// A_i -= L_i R for the kDirNB rows of one own block (rows: its first row, Lt: its columns of Lt).
// Tiles of 8 rows x 64 columns, dealt to the warps from warp w on.
__device__ __forceinline__ void dir_update_block(double* rows, const double* R, const double* Lt, int ls, int npad,
                                                 int w) {
  const int lane = threadIdx.x & 31, nct = (npad + 63) / 64;
  for (int t = w; t < 2 * nct; t += kDirWarps) {
    const int r0 = 8 * (t & 1), j = 64 * (t >> 1) + lane;
    const bool in0 = j < npad, in1 = j + 32 < npad;
    double* a = rows + r0 * npad + j;
    double acc[8][2];
#pragma unroll
    for (int r = 0; r < 8; r++) {
      acc[r][0] = in0 ? a[r * npad] : 0.0;
      acc[r][1] = in1 ? a[r * npad + 32] : 0.0;
    }
    dir_tile<true>(R, npad, Lt + r0, ls, j, in0, in1, acc);
#pragma unroll
    for (int r = 0; r < 8; r++) {
      if (in0) a[r * npad] = acc[r][0];
      if (in1) a[r * npad + 32] = acc[r][1];
    }
  }
}

// The panel of block kb (rows: its kDirNB rows, already updated by every earlier step) into `out`
// (global): P = A_KK^-1 by one warp, then P A_K, with P in the columns of block kb. All threads.
__device__ __forceinline__ void dir_make_panel(const double* rows, int kb, int npad, double* Pt, double* out,
                                               int* status) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0) {
    // lane holds 8 elements of row i of the diagonal block; Gauss-Jordan with shuffles
    const int i = lane & 15, h = lane >> 4;
    double a[8];
#pragma unroll
    for (int q = 0; q < 8; q++) a[q] = rows[i * npad + kb * kDirNB + h * 8 + q];
#pragma unroll
    for (int p = 0; p < kDirNB; p++) {
      const double pv = __shfl_sync(0xffffffffu, a[p & 7], p + 16 * (p >> 3));
      const double col = __shfl_sync(0xffffffffu, a[p & 7], i + 16 * (p >> 3));
      double rq[8];
#pragma unroll
      for (int q = 0; q < 8; q++) rq[q] = __shfl_sync(0xffffffffu, a[q], p + 16 * h);
      if (lane == 0 && !(pv > 0.0)) *status = 1;
      const double pinv = 1.0 / pv, cp = col * pinv;
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const bool at = h * 8 + q == p;
        if (i == p)
          a[q] = at ? pinv : a[q] * pinv;
        else
          a[q] = at ? -cp : a[q] - cp * rq[q];
      }
    }
#pragma unroll
    for (int q = 0; q < 8; q++) Pt[(h * 8 + q) * kDirNB + i] = a[q];
  }
  __syncthreads();
  const int nct = (npad + 63) / 64, k0 = kb * kDirNB;
  for (int t = warp; t < 2 * nct; t += kDirWarps) {
    const int r0 = 8 * (t & 1), j = 64 * (t >> 1) + lane;
    const bool in0 = j < npad, in1 = j + 32 < npad;
    double acc[8][2] = {};
    dir_tile<false>(rows, npad, Pt + r0, kDirNB, j, in0, in1, acc);
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int jc = j + 32 * c;
      if (jc >= npad) continue;
      const bool inK = jc >= k0 && jc < k0 + kDirNB;
#pragma unroll
      for (int r = 0; r < 8; r++) out[(r0 + r) * npad + jc] = inK ? Pt[(jc - k0) * kDirNB + r0 + r] : acc[r][c];
    }
  }
}

// Bound by the chain of steps (panel copy, update of the next block, 16 pivots, one barrier: about 8 us
// each), not by its 2 n^3 FP64 operations. update() + solve, in us, against one CTA that eliminated one
// pivot at a time (matrix in shared memory up to n = 160, else in L2):
//   n         64    125    216    315    343     729     990
//   before  1039   1527   5108  14097  18432  157614  382809
//   now     1029    889    965   1254   1225    2329    2508
template <bool kSmemRows>
__global__ void __launch_bounds__(kDirThreads) k_direct_inverse(Dims d, const float* __restrict__ st, double* Aout,
                                                                double* work, DirPlan pl, int* status) {
  extern __shared__ __align__(16) double dsm[];
  __shared__ double red[32];
  __shared__ double alpha_s;
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int rank = int(cluster.block_rank()), C = pl.ncl;
  const int n = pl.n, nb = pl.nb, npad = pl.npad, ls = pl.nloc * kDirNB;
  double* R = dsm;
  double* Lt = R + size_t(kDirNB) * npad;
  double* Pt = Lt + size_t(kDirNB) * ls;
  const size_t panel = size_t(kDirNB) * npad;
  double* rows = kSmemRows ? Pt + kDirNB * kDirNB : work + 2 * panel + size_t(rank) * ls * npad;
  const int nown = rank < nb ? (nb - rank + C - 1) / C : 0;  // own block rows: rank, rank + C, ...
  const int tid = threadIdx.x, warp = tid >> 5;
  auto vertex = [&](int lr) { return (rank + (lr / kDirNB) * C) * kDirNB + lr % kDirNB; };

  // assemble the own rows (one thread per row: small dimensions alias offsets onto one column)
  for (int i = tid; i < nown * kDirNB * npad; i += kDirThreads) rows[i] = 0.0;
  double tr[1] = {0.0};  // every axis has at least 2 vertices, so only offset 13 is on the diagonal
  for (int v = tid; v < n; v += kDirThreads) tr[0] += double(__ldg(st + size_t(13) * n + v));
  block_reduce_f64<1>(tr, red);
  if (tid == 0) alpha_s = tr[0] / double(n) / double(n);
  __syncthreads();
  const double alpha = alpha_s;
  for (int lr = tid; lr < nown * kDirNB; lr += kDirThreads) {
    const int v = vertex(lr);
    double* row = rows + size_t(lr) * npad;
    if (v >= n) {
      row[v] = 1.0;
      continue;
    }
    const int x = v % d.nx, y = (v / d.nx) % d.ny, z = v / (d.nx * d.ny);
    for (int o = 0; o < 27; o++) {
      const int jx = (x + o % 3 - 1 + d.nx) % d.nx, jy = (y + (o / 3) % 3 - 1 + d.ny) % d.ny,
                jz = (z + o / 9 - 1 + d.nz) % d.nz;
      row[jx + d.nx * (jy + d.ny * jz)] += double(__ldg(st + size_t(o) * n + v));
    }
  }
  __syncthreads();
  for (int i = tid; i < nown * kDirNB * npad; i += kDirThreads) {
    const int lr = i / npad, j = i - lr * npad;
    if (j < n && vertex(lr) < n) rows[i] += alpha;
  }
  __syncthreads();

  if (rank == 0) dir_make_panel(rows, 0, npad, Pt, work, status);
  cluster.sync();
  for (int kb = 0; kb < nb; kb++) {
    // the panel, and the own rows' columns of block kb (transposed; zeroed in place)
    const double2* src = reinterpret_cast<const double2*>(work + (kb & 1) * panel);
    for (int i = tid; i < int(panel / 2); i += kDirThreads) reinterpret_cast<double2*>(R)[i] = __ldcg(src + i);
    for (int i = tid; i < nown * kDirNB * kDirNB; i += kDirThreads) {
      const int lr = i / kDirNB, k = i % kDirNB;
      double* a = rows + size_t(lr) * npad + kb * kDirNB + k;
      Lt[k * ls + lr] = *a;
      *a = 0.0;
    }
    __syncthreads();
    // the next panel first, then (between the barrier's arrive and wait) the other rows
    const int next = kb + 1 < nb && (kb + 1) % C == rank ? (kb + 1) / C : -1;
    if (next >= 0) {
      double* nr = rows + size_t(next) * kDirNB * npad;
      dir_update_block(nr, R, Lt + next * kDirNB, ls, npad, warp);
      __syncthreads();
      dir_make_panel(nr, kb + 1, npad, Pt, work + ((kb + 1) & 1) * panel, status);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const int ntiles = 2 * ((npad + 63) / 64);
    int w = warp;  // the tiles of successive blocks continue over the warps
    for (int b = 0; b < nown; b++) {
      if (b == next) continue;
      double* br = rows + size_t(b) * kDirNB * npad;
      if (rank + b * C == kb) {
        for (int i = tid; i < int(panel); i += kDirThreads) br[i] = R[i];
      } else {
        dir_update_block(br, R, Lt + b * kDirNB, ls, npad, w);
        w = (w + kDirWarps - ntiles % kDirWarps) % kDirWarps;
      }
    }
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  for (int i = tid; i < nown * kDirNB * npad; i += kDirThreads) {
    const int lr = i / npad, j = i - lr * npad, v = vertex(lr);
    if (j < n && v < n) Aout[size_t(v) * n + j] = rows[i];
  }
}

// u = Ainv (f - mean f) for the 3 load cases: one warp per unknown (row of the symmetric inverse), the
// right-hand side and its means in every block's shared memory (3 n doubles).
constexpr int kDirSolveThreads = 256;
static __global__ void __launch_bounds__(kDirSolveThreads) k_coarsest_solve(int n, const double* __restrict__ Ainv,
                                                                            const float* __restrict__ f, float* u,
                                                                            const SolveScalars* sc) {
  pdl_wait();
  if (sc && solve_done(sc)) return;
  extern __shared__ double bsh[];
  __shared__ double mean[3];
  for (int i = threadIdx.x; i < 3 * n; i += blockDim.x) bsh[i] = __ldg(f + i);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < 3) {
    double s = 0.0;
    for (int i = lane; i < n; i += 32) s += bsh[warp * n + i];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) mean[warp] = s / n;
  }
  __syncthreads();
  const int i = blockIdx.x * (kDirSolveThreads / 32) + warp;
  if (i >= n) return;
  const double m0 = mean[0], m1 = mean[1], m2 = mean[2];
  double a0 = 0.0, a1 = 0.0, a2 = 0.0;
#pragma unroll 4
  for (int j = lane; j < n; j += 32) {
    const double m = __ldg(Ainv + size_t(i) * n + j);
    a0 += m * (bsh[j] - m0);
    a1 += m * (bsh[n + j] - m1);
    a2 += m * (bsh[2 * n + j] - m2);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    a0 += __shfl_xor_sync(0xffffffffu, a0, off);
    a1 += __shfl_xor_sync(0xffffffffu, a1, off);
    a2 += __shfl_xor_sync(0xffffffffu, a2, off);
  }
  if (lane == 0) {
    u[i] = float(a0);
    u[n + i] = float(a1);
    u[2 * n + i] = float(a2);
  }
}

}  // namespace otm
