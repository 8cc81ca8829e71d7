// otm_mma.cu -- method of moving asymptotes in FP64 on the device (Svanberg's MMA with the
// primal-dual interior-point subsolver), replacing MMAOptimizer / mmasubDevice
// (optimization/mmaOptimizer.cu:18-78, optimization/mmaOpt.cu:429-1062, mmaOpt.cpp:38-73).
//
// Every pass over the n design variables is one kernel that also reduces what the next step
// needs (sums with a fixed-order last-block finalisation, maxima). A Newton step is two passes:
// the step bounds of the direction, then the line-search trial, which recomputes the direction,
// writes the trial point to spare arrays and reduces both the residual there and the next Newton
// system (accepting the step swaps the arrays). The dual variables, the (m+1) x (m+1) KKT system
// (m <= 8, where the reference used Eigen on the host) and every decision of the interior-point
// iteration live on the device: the last block of a pass takes the step that the pass was for and
// says which pass comes next (MmaState), so the host only queues passes and looks once in a while
// whether the subproblem is solved. A pass queued for another step than the one that is due returns
// at once. When epsi falls, the residual and the Newton system at the same point follow from the
// sums of the pass before (they are polynomials in epsi), without another pass.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "opentm_b200_mma.h"
#include "otm_common.cuh"
#include "otm_mg_kernels.cuh"

namespace otm {

constexpr int kMmaMaxM = OTM_MMA_MAX_CONSTRAINTS;
constexpr double kEpsiMin = 1e-7, kRaa0 = 1e-5, kAlbefa = 0.1, kAsyInit = 0.5, kAsyIncr = 1.2, kAsyDecr = 0.7;

struct MVec {
  double v[kMmaMaxM];
};

// Work arrays of one subsolve, n (or m * n) doubles each. dx, dxsi, deta hold the line search's
// trial point, which trades places with xs, xsi, eta when it is accepted.
struct MmaWork {
  size_t n = 0;
  int m = 0;
  bool carved = false;  // the arrays lie in the owner's block
  double *alfa = nullptr, *beta = nullptr, *p0 = nullptr, *q0 = nullptr, *P = nullptr, *Q = nullptr;
  double *xs = nullptr, *xsi = nullptr, *eta = nullptr, *dx = nullptr, *dxsi = nullptr, *deta = nullptr;
  double* partials = nullptr;  // kMaxPartials * 96
  double* result = nullptr;    // kMmaSlots
  unsigned int* counter = nullptr;
  struct MmaState* state = nullptr;
  int* host = nullptr;         // pinned copy of the state's mode and error
};

constexpr int kMmaSlots = 128;  // >= 5 + 3 m + m^2 for m <= 8

// The pass that is due: the residual at the start point, the step bounds of a direction, a line-search
// trial, nothing any more.
enum MmaMode { kMmaInit = 0, kMmaDirmax = 1, kMmaTrial = 2, kMmaDone = 3 };
enum MmaError { kMmaOk = 0, kMmaSingular = 1, kMmaNanStep = 2 };

// Constants of a subproblem on the host side of a step (a0, a, c, d and the constraint values).
struct MmaProblem {
  double a0, a[kMmaMaxM], c[kMmaMaxM], d[kMmaMaxM], g[kMmaMaxM];
};

// The interior-point iteration on the device (subsolv, optimization/mmaOpt.cu:429-830): the dual and
// slack variables, their direction and line-search base, the sums of the last trial, and what is due.
struct MmaState {
  int mode, err;  // first: copied to the host together
  int parity;     // 1: the committed point is in the spare arrays
  int ittt, itto;
  MmaProblem pr;
  double n, b[kMmaMaxM];
  double y[kMmaMaxM], lam[kMmaMaxM], mu[kMmaMaxM], s[kMmaMaxM], z, zet, epsi;
  double dy[kMmaMaxM], dl[kMmaMaxM], dmu[kMmaMaxM], ds[kMmaMaxM], dz, dzet;
  double yo[kMmaMaxM], lo[kMmaMaxM], muo[kMmaMaxM], so[kMmaMaxM], zo, zeto;
  double steg, residunorm, residumax;
  // the last trial: sums and maxima over the variables (see k_mma_trial)
  double n2, tsum, gvec[kMmaMaxM], gd[kMmaMaxM], gs[kMmaMaxM], gg[kMmaMaxM * kMmaMaxM], mrex, mab, nab;
};

template <int NM>
__device__ __forceinline__ void block_reduce_max(double (&v)[NM], double* smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int i = 0; i < NM; i++)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[i] = fmax(v[i], __shfl_down_sync(0xffffffffu, v[i], off));
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < NM; i++) smem[warp * NM + i] = v[i];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < NM; i++) {
      double x = lane < nwarps ? smem[lane * NM + i] : -1e300;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) x = fmax(x, __shfl_down_sync(0xffffffffu, x, off));
      v[i] = x;
    }
  }
}

// Block partials of NS sums and NM maxima, then the last block writes result[0..NS+NM); true in the
// threads of that block, where the results can be read.
template <int NS, int NM>
__device__ __forceinline__ bool reduce_to_result(double (&s)[NS], double (&mx)[NM], double* partials,
                                                 double* result, unsigned int* counter) {
  __shared__ double smem[32 * (NS > NM ? NS : NM)];
  block_reduce_f64<NS>(s, smem);
  block_reduce_max<NM>(mx, smem);
  constexpr int W = NS + NM;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < NS; i++) partials[blockIdx.x * W + i] = s[i];
#pragma unroll
    for (int i = 0; i < NM; i++) partials[blockIdx.x * W + NS + i] = mx[i];
  }
  if (last_block(counter)) {
    // one warp per value: lanes stride over the blocks, then a shuffle reduction (fixed order)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = warp; i < W; i += int(blockDim.x >> 5)) {
      double acc = i < NS ? 0.0 : -1e300;
#pragma unroll 8
      for (int b = lane; b < int(gridDim.x); b += 32) {
        const double v = __ldcg(partials + b * W + i);  // L2: never a stale L1 line
        acc = i < NS ? acc + v : fmax(acc, v);
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double o = __shfl_xor_sync(0xffffffffu, acc, off);
        acc = i < NS ? acc + o : fmax(acc, o);
      }
      if (lane == 0) result[i] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) *counter = 0;
    return true;
  }
  return false;
}

// std::max's rule for NaN (the second argument is taken only if it is greater).
__device__ __forceinline__ double later_max(double a, double b) { return a < b ? b : a; }

// Dense N x N solve with partial pivoting (replaces Eigen ColPivHouseholderQR, mmaOpt.cpp:48-73).
template <int N>
__device__ bool dense_solve(double (&A)[N][N], double (&b)[N]) {
  for (int k = 0; k < N; k++) {
    int p = k;
    for (int i = k + 1; i < N; i++)
      if (fabs(A[i][k]) > fabs(A[p][k])) p = i;
    if (A[p][k] == 0.0) return false;
    if (p != k) {
      for (int j = 0; j < N; j++) {
        const double t = A[k][j];
        A[k][j] = A[p][j];
        A[p][j] = t;
      }
      const double t = b[k];
      b[k] = b[p];
      b[p] = t;
    }
    for (int i = k + 1; i < N; i++) {
      const double l = A[i][k] / A[k][k];
      for (int j = k; j < N; j++) A[i][j] -= l * A[k][j];
      b[i] -= l * b[k];
    }
  }
  for (int i = N - 1; i >= 0; i--) {
    double t = b[i];
    for (int j = i + 1; j < N; j++) t -= A[i][j] * b[j];
    b[i] = t / A[i][i];
  }
  return true;
}

// Residual norm and largest entry at the last trial's point with the current epsi: the variables' part
// from its sums, the duals' part here.
template <int M>
__device__ void mma_residual(MmaState& S, double* norm, double* mx) {
  const MmaProblem& P = S.pr;
  double n2 = S.n2, m = later_max(later_max(S.mrex, S.mab - S.epsi), S.nab + S.epsi), ad = 0.0;
  auto acc = [&](double r) {
    n2 += r * r;
    m = later_max(m, fabs(r));
  };
  for (int i = 0; i < M; i++) ad += P.a[i] * S.lam[i];
  for (int i = 0; i < M; i++) acc(P.c[i] + P.d[i] * S.y[i] - S.mu[i] - S.lam[i]);
  acc(P.a0 - S.zet - ad);
  for (int i = 0; i < M; i++) acc(S.gvec[i] - P.a[i] * S.z - S.y[i] + S.s[i] - S.b[i]);
  for (int i = 0; i < M; i++) acc(S.mu[i] * S.y[i] - S.epsi);
  acc(S.zet * S.z - S.epsi);
  for (int i = 0; i < M; i++) acc(S.lam[i] * S.s[i] - S.epsi);
  *norm = sqrt(n2);
  *mx = m;
}

// The sums of the last trial, from its result (see k_mma_trial).
template <int M>
__device__ void mma_take(MmaState& S, const double* r) {
  S.n2 = r[0];
  S.tsum = r[1];
  for (int i = 0; i < M; i++) {
    S.gvec[i] = r[2 + i];
    S.gd[i] = r[2 + M + i];
    S.gs[i] = r[2 + 2 * M + i];
    for (int k = 0; k < M; k++) S.gg[i * M + k] = r[2 + 3 * M + i * M + k];
  }
  const double* x = r + 2 + 3 * M + M * M;
  S.mrex = x[0];
  S.mab = x[1];
  S.nab = x[2];
}

// The trial point's duals for the step S.steg; the next pass is a trial there.
template <int M>
__device__ void mma_next_trial(MmaState& S) {
  S.itto++;
  for (int i = 0; i < M; i++) {
    S.y[i] = S.yo[i] + S.steg * S.dy[i];
    S.lam[i] = S.lo[i] + S.steg * S.dl[i];
    S.mu[i] = S.muo[i] + S.steg * S.dmu[i];
    S.s[i] = S.so[i] + S.steg * S.ds[i];
  }
  S.z = S.zo + S.steg * S.dz;
  S.zet = S.zeto + S.steg * S.dzet;
  S.mode = kMmaTrial;
}

// At a committed point: the next Newton direction of the duals, or the next epsi, or the end.
template <int M>
__device__ void mma_advance(MmaState& S) {
  const MmaProblem& P = S.pr;
  while (!(S.residumax > 0.9 * S.epsi && S.ittt < 200)) {
    const double e0 = S.epsi;
    S.epsi = 0.1 * e0;
    if (!(S.epsi > kEpsiMin)) {
      S.mode = kMmaDone;
      return;
    }
    // the same point with the smaller epsi: the entries a - epsi and b - epsi of the residual move by
    // de, and so does the epsi part of delx
    const double de = e0 - S.epsi;
    S.n2 += 2.0 * de * S.tsum + 2.0 * S.n * de * de;
    S.tsum += 2.0 * S.n * de;
    for (int i = 0; i < M; i++) S.gd[i] += de * S.gs[i];
    S.ittt = 0;
    mma_residual<M>(S, &S.residunorm, &S.residumax);
  }
  S.ittt++;
  double adl = 0.0;
  for (int i = 0; i < M; i++) adl += P.a[i] * S.lam[i];
  const double delz = P.a0 - adl - S.epsi / S.z;
  double AA[M + 1][M + 1], bb[M + 1], dely[M], diagy[M];
  for (int i = 0; i < M; i++) {
    dely[i] = P.c[i] + P.d[i] * S.y[i] - S.lam[i] - S.epsi / S.y[i];
    const double dellam = S.gvec[i] - P.a[i] * S.z - S.y[i] - S.b[i] + S.epsi / S.lam[i];
    diagy[i] = P.d[i] + S.mu[i] / S.y[i];
    bb[i] = dellam + dely[i] / diagy[i] - S.gd[i];
    for (int k = 0; k < M; k++) AA[i][k] = S.gg[i * M + k];
    AA[i][i] += S.s[i] / S.lam[i] + 1.0 / diagy[i];
    AA[i][M] = P.a[i];
    AA[M][i] = P.a[i];
  }
  AA[M][M] = -S.zet / S.z;
  bb[M] = delz;
  if (!dense_solve<M + 1>(AA, bb)) {
    S.err = kMmaSingular;
    S.mode = kMmaDone;
    return;
  }
  S.dz = bb[M];
  for (int i = 0; i < M; i++) {
    S.dl[i] = bb[i];
    S.dy[i] = -dely[i] / diagy[i] + bb[i] / diagy[i];
    S.dmu[i] = -S.mu[i] + S.epsi / S.y[i] - (S.mu[i] * S.dy[i]) / S.y[i];
    S.ds[i] = -S.s[i] + S.epsi / S.lam[i] - (S.s[i] * bb[i]) / S.lam[i];
    S.lo[i] = S.lam[i];
  }
  S.dzet = -S.zet + S.epsi / S.z - S.zet * S.dz / S.z;
  S.mode = kMmaDirmax;
}

// After the step-bound pass: the line search's first step.
template <int M>
__device__ void mma_after_dirmax(MmaState& S, const double* r) {
  double stm = later_max(r[1], r[2]);  // xsi, eta parts
  for (int i = 0; i < M; i++) {
    stm = later_max(stm, -1.01 * S.dy[i] / S.y[i]);
    stm = later_max(stm, -1.01 * S.dl[i] / S.lam[i]);
    stm = later_max(stm, -1.01 * S.dmu[i] / S.mu[i]);
    stm = later_max(stm, -1.01 * S.ds[i] / S.s[i]);
  }
  stm = later_max(stm, -1.01 * S.dz / S.z);
  stm = later_max(stm, -1.01 * S.dzet / S.zet);
  const double stmalbe = later_max(r[3], r[4]);
  S.steg = 1.0 / later_max(later_max(stmalbe, stm), 1.0);
  if (isnan(S.steg)) {
    S.err = kMmaNanStep;
    S.mode = kMmaDone;
    return;
  }
  for (int i = 0; i < M; i++) {
    S.yo[i] = S.y[i];
    S.muo[i] = S.mu[i];
    S.so[i] = S.s[i];
  }
  S.zo = S.z;
  S.zeto = S.zet;
  S.itto = 0;
  mma_next_trial<M>(S);
}

// After a trial (or the residual of the start point): accept it or halve the step.
template <int M>
__device__ void mma_after_trial(MmaState& S, const double* r) {
  mma_take<M>(S, r);
  double norm, mx;
  mma_residual<M>(S, &norm, &mx);
  if (S.mode == kMmaTrial) {
    S.steg /= 2;
    if (norm > S.residunorm && S.itto < 50) {
      mma_next_trial<M>(S);
      return;
    }
    S.parity ^= 1;  // the last point tried, as the reference commits after its line search
  }
  S.residunorm = norm;
  S.residumax = mx;
  mma_advance<M>(S);
}

// The last block's decision: step(S, sums) by one thread on a copy of the state in shared memory. It is a chain
// of some hundred dependent accesses at m = 4 and many more at m = 8; on the state in global memory three
// updates of 20,000 variables at m = 8 took 8.31 ms, more than with the decisions on the host (7.77), and take
// 7.59 now (m = 4 3.19 -> 3.06, m = 1 1.88 -> 1.73).
template <int NR, typename F>
__device__ __forceinline__ void mma_decide(MmaState* state, const double* result, F&& step) {
  __shared__ MmaState S;
  __shared__ double r[NR];
  static_assert(sizeof(MmaState) % sizeof(double) == 0, "copied as doubles");
  constexpr int kWords = int(sizeof(MmaState) / sizeof(double));
  double* dst = reinterpret_cast<double*>(&S);
  double* src = reinterpret_cast<double*>(state);
  for (int i = threadIdx.x; i < kWords; i += blockDim.x) dst[i] = src[i];
  for (int i = threadIdx.x; i < NR; i += blockDim.x) r[i] = result[i];
  __syncthreads();
  if (threadIdx.x == 0) step(S, r);
  __syncthreads();
  for (int i = threadIdx.x; i < kWords; i += blockDim.x) src[i] = dst[i];
}

// The start of a subproblem: constraint offsets sums[i] = sum_j P/ux + Q/xl from the set-up pass.
template <int M>
__device__ void mma_start(MmaState& S, const MmaProblem& pr, double n, const double* sums) {
  S.mode = kMmaInit;
  S.err = kMmaOk;
  S.parity = S.ittt = S.itto = 0;
  S.pr = pr;
  S.n = n;
  for (int i = 0; i < M; i++) {
    S.b[i] = sums[i] - pr.g[i];
    S.y[i] = S.lam[i] = S.s[i] = 1.0;
    S.mu[i] = later_max(0.5 * pr.c[i], 1.0);
    S.dl[i] = S.lo[i] = 0.0;
  }
  S.z = S.zet = S.epsi = 1.0;
  S.steg = 0.0;
}

// Asymptotes, move limits, approximation coefficients p0, q0, P, Q, the constraint offsets
// sum_j P/ux + Q/xl, and the subsolver's starting point (mmasub_ker, optimization/mmaOpt.cu:834-1019).
// The inputs are FP64 or FP32 (T); xvar_out, if given, receives x in FP64.
template <typename T>
struct MmaInputs {
  const T *x, *df0dx, *dgdx[kMmaMaxM];
  double* xvar_out;
};
template <int M, typename T>
__global__ void __launch_bounds__(256) k_mma_setup(size_t n, int itn, MmaInputs<T> in, const double* __restrict__ xmin,
                                                   const double* __restrict__ xmax, const double* __restrict__ xold1,
                                                   const double* __restrict__ xold2, double* low, double* upp,
                                                   double move, MmaProblem pr, MmaWork w) {
  double bs[M];
  double dummy[1] = {-1e300};
#pragma unroll
  for (int i = 0; i < M; i++) bs[i] = 0.0;
  for (size_t j = size_t(blockIdx.x) * blockDim.x + threadIdx.x; j < n; j += size_t(gridDim.x) * blockDim.x) {
    const double x = double(in.x[j]), dxr = xmax[j] - xmin[j], df = double(in.df0dx[j]);
    if (in.xvar_out) in.xvar_out[j] = x;
    double lo, up;
    if (itn <= 2) {
      lo = x - kAsyInit * dxr;
      up = x + kAsyInit * dxr;
    } else {
      const double zzz = (x - xold1[j]) * (xold1[j] - xold2[j]);
      const double f = zzz > 0 ? kAsyIncr : (zzz < 0 ? kAsyDecr : 1.0);
      lo = x - f * (xold1[j] - low[j]);
      up = x + f * (upp[j] - xold1[j]);
      lo = fmin(fmax(lo, x - 10.0 * dxr), x - 0.01 * dxr);
      up = fmax(fmin(up, x + 10.0 * dxr), x + 0.01 * dxr);
    }
    low[j] = lo;
    upp[j] = up;
    const double al = fmax(fmax(lo + kAlbefa * (x - lo), x - move * dxr), xmin[j]);
    const double be = fmin(fmin(up - kAlbefa * (up - x), x + move * dxr), xmax[j]);
    w.alfa[j] = al;
    w.beta[j] = be;
    const double xmamiinv = 1.0 / fmax(dxr, 1e-5);
    const double ux1 = up - x, xl1 = x - lo, ux2 = ux1 * ux1, xl2 = xl1 * xl1;
    const double dp = fmax(df, 0.0), dm = fmax(-df, 0.0);
    const double pq0 = 1e-3 * (dp + dm) + kRaa0 * xmamiinv;
    w.p0[j] = (dp + pq0) * ux2;
    w.q0[j] = (dm + pq0) * xl2;
#pragma unroll
    for (int i = 0; i < M; i++) {
      const double g = double(in.dgdx[i][j]);
      const double pp = fmax(g, 0.0), qq = fmax(-g, 0.0);
      const double pq = 1e-3 * (pp + qq) + kRaa0 * xmamiinv;
      const double Pij = (pp + pq) * ux2, Qij = (qq + pq) * xl2;
      w.P[i * n + j] = Pij;
      w.Q[i * n + j] = Qij;
      bs[i] += Pij / ux1 + Qij / xl1;
    }
    const double xs = 0.5 * (al + be);
    w.xs[j] = xs;
    w.xsi[j] = fmax(1.0 / (xs - al), 1.0);
    w.eta[j] = fmax(1.0 / (be - xs), 1.0);
  }
  if (reduce_to_result<M, 1>(bs, dummy, w.partials, w.result, w.counter) && threadIdx.x == 0)
    mma_start<M>(*w.state, pr, double(n), w.result);
}

// The per-variable data a subsolver pass reads: the point, its bounds and the approximation.
template <int M>
struct MmaElem {
  double x, xsi, eta, low, upp, al, be, p0, q0, P[M], Q[M];
};

// The committed point and the other one, by the state's parity.
struct MmaPoint {
  double *x, *xsi, *eta;
};
__device__ __forceinline__ MmaPoint mma_point(const MmaWork& w, bool spare) {
  return spare ? MmaPoint{w.dx, w.dxsi, w.deta} : MmaPoint{w.xs, w.xsi, w.eta};
}

template <int M>
__device__ __forceinline__ void load_elem(const MmaWork& w, const MmaPoint& pt, const double* __restrict__ low,
                                          const double* __restrict__ upp, size_t j, MmaElem<M>& e) {
  e.x = pt.x[j];
  e.xsi = pt.xsi[j];
  e.eta = pt.eta[j];
  e.low = low[j];
  e.upp = upp[j];
  e.al = w.alfa[j];
  e.be = w.beta[j];
  e.p0 = w.p0[j];
  e.q0 = w.q0[j];
#pragma unroll
  for (int i = 0; i < M; i++) {
    e.P[i] = w.P[i * w.n + j];
    e.Q[i] = w.Q[i * w.n + j];
  }
}

// Elements j and j + 1 (j even; n even and every array 16-byte aligned): one 16-byte load per
// array, twice the bytes in flight per instruction.
template <int M>
__device__ __forceinline__ void load_pair(const MmaWork& w, const MmaPoint& pt, const double* __restrict__ low,
                                          const double* __restrict__ upp, size_t j, MmaElem<M>& a, MmaElem<M>& b) {
  auto ld = [j](const double* p, double& u, double& v) {
    const double2 t = *reinterpret_cast<const double2*>(p + j);
    u = t.x;
    v = t.y;
  };
  ld(pt.x, a.x, b.x);
  ld(pt.xsi, a.xsi, b.xsi);
  ld(pt.eta, a.eta, b.eta);
  ld(low, a.low, b.low);
  ld(upp, a.upp, b.upp);
  ld(w.alfa, a.al, b.al);
  ld(w.beta, a.be, b.be);
  ld(w.p0, a.p0, b.p0);
  ld(w.q0, a.q0, b.q0);
#pragma unroll
  for (int i = 0; i < M; i++) {
    ld(w.P + i * w.n, a.P[i], b.P[i]);
    ld(w.Q + i * w.n, a.Q[i], b.Q[i]);
  }
}

// Newton direction of x, xsi, eta at e for multiplier lam and its step dlam (subsolv's dx, dxsi,
// deta, optimization/mmaOpt.cu:429-830), shared by the two passes below so both see the same
// values without storing them. The five distinct denominators are inverted once.
template <int M>
__device__ __forceinline__ void mma_dir(const MmaElem<M>& e, const MVec& lam, const MVec& dlam, double epsi,
                                        double* dx, double* dxsi, double* deta, double* rxa_out, double* rbx_out) {
  const double x = e.x;
  const double rux = 1.0 / (e.upp - x), rxl = 1.0 / (x - e.low);
  const double rux2 = rux * rux, rxl2 = rxl * rxl;
  const double rxa = 1.0 / (x - e.al), rbx = 1.0 / (e.be - x);
  double plam = e.p0, qlam = e.q0, gl = 0.0;
#pragma unroll
  for (int i = 0; i < M; i++) {
    plam += e.P[i] * lam.v[i];
    qlam += e.Q[i] * lam.v[i];
    gl += (e.P[i] * rux2 - e.Q[i] * rxl2) * dlam.v[i];
  }
  const double dpsidx = plam * rux2 - qlam * rxl2;
  const double delx = dpsidx - epsi * rxa + epsi * rbx;
  const double diagx = 2.0 * (plam * rux2 * rux + qlam * rxl2 * rxl) + e.xsi * rxa + e.eta * rbx;
  const double rd = 1.0 / diagx;
  *dx = -(delx + gl) * rd;
  *dxsi = -e.xsi + epsi * rxa - e.xsi * *dx * rxa;
  *deta = -e.eta + epsi * rbx + e.eta * *dx * rbx;
  *rxa_out = rxa;
  *rbx_out = rbx;
}

// The line search's step bounds: the largest ratios -1.01 dxsi/xsi, -1.01 deta/eta,
// -1.01 dx/(x - alfa), 1.01 dx/(beta - x), without storing the direction (the trial pass
// recomputes it). VW consecutive variables per loop step.
template <int M, int VW>
__global__ void __launch_bounds__(256) k_mma_dirmax(const double* __restrict__ low, const double* __restrict__ upp,
                                                    MmaWork w) {
  const MmaState& S = *w.state;
  if (S.mode != kMmaDirmax) return;  // another pass is due
  MVec lam, dlam;
#pragma unroll
  for (int i = 0; i < M; i++) {
    lam.v[i] = S.lo[i];
    dlam.v[i] = S.dl[i];
  }
  const double epsi = S.epsi;
  const MmaPoint pt = mma_point(w, S.parity != 0);
  double s[1] = {0.0};
  double mx[4] = {-1e300, -1e300, -1e300, -1e300};
  const size_t nq = w.n / VW;
  for (size_t q = size_t(blockIdx.x) * blockDim.x + threadIdx.x; q < nq; q += size_t(gridDim.x) * blockDim.x) {
    MmaElem<M> e[VW];
    if (VW == 2)
      load_pair<M>(w, pt, low, upp, 2 * q, e[0], e[VW - 1]);
    else
      load_elem<M>(w, pt, low, upp, q, e[0]);
#pragma unroll
    for (int v = 0; v < VW; v++) {
      double dx, dxsi, deta, rxa, rbx;
      mma_dir<M>(e[v], lam, dlam, epsi, &dx, &dxsi, &deta, &rxa, &rbx);
      mx[0] = fmax(mx[0], -1.01 * dxsi / e[v].xsi);
      mx[1] = fmax(mx[1], -1.01 * deta / e[v].eta);
      mx[2] = fmax(mx[2], -1.01 * dx * rxa);
      mx[3] = fmax(mx[3], 1.01 * dx * rbx);
    }
  }
  if (reduce_to_result<1, 4>(s, mx, w.partials, w.result, w.counter))
    mma_decide<5>(w.state, w.result, [](MmaState& T, const double* r) { mma_after_dirmax<M>(T, r); });
}

// One pass at the trial point x + steg dx (start point: steg = 0, nothing written): the relaxed KKT
// residual with the trial multiplier lam and, at the same point, the pieces of the next Newton system,
// so an accepted step needs no further pass. The trial point goes to the arrays that do not hold the
// committed one; accepting it flips the state's parity. VW consecutive variables per loop step.
// result = [residual sum of squares, sum (xsi (x - alfa) - epsi) + (eta (beta - x) - epsi),
//           gvec_i = sum P/ux + Q/xl (M), GG delx/diagx (M), GG (1/(x - alfa) - 1/(beta - x))/diagx (M),
//           GG diag(1/diagx) GG^T (M*M), max |dL/dx|, max and -min of xsi (x - alfa), eta (beta - x)].
template <int M, int VW>
__global__ void __launch_bounds__(256) k_mma_trial(const double* __restrict__ low, const double* __restrict__ upp,
                                                   MmaWork w) {
  const MmaState& S = *w.state;
  const bool moved = S.mode == kMmaTrial;
  if (!moved && S.mode != kMmaInit) return;  // another pass is due
  MVec lam, lam_dir, dlam;
#pragma unroll
  for (int i = 0; i < M; i++) {
    lam.v[i] = S.lam[i];
    lam_dir.v[i] = S.lo[i];
    dlam.v[i] = S.dl[i];
  }
  const double epsi = S.epsi, steg = S.steg;
  const MmaPoint pt = mma_point(w, S.parity != 0), out = mma_point(w, S.parity == 0);
  constexpr int NS = 2 + 3 * M + M * M;
  double s[NS];
  double mx[3] = {0.0, -1e300, -1e300};
#pragma unroll
  for (int i = 0; i < NS; i++) s[i] = 0.0;
  const size_t nq = w.n / VW;
  for (size_t q = size_t(blockIdx.x) * blockDim.x + threadIdx.x; q < nq; q += size_t(gridDim.x) * blockDim.x) {
    MmaElem<M> e[VW];
    if (VW == 2)
      load_pair<M>(w, pt, low, upp, 2 * q, e[0], e[VW - 1]);
    else
      load_elem<M>(w, pt, low, upp, q, e[0]);
#pragma unroll
    for (int v = 0; v < VW; v++) {
      if (moved) {
        double dx, dxsi, deta, r0, r1;
        mma_dir<M>(e[v], lam_dir, dlam, epsi, &dx, &dxsi, &deta, &r0, &r1);
        e[v].x = e[v].x + steg * dx;
        e[v].xsi = e[v].xsi + steg * dxsi;
        e[v].eta = e[v].eta + steg * deta;
      }
      const double x = e[v].x, xsi = e[v].xsi, eta = e[v].eta, al = e[v].al, be = e[v].be;
      // residual
      const double uxi = 1.0 / (e[v].upp - x), xli = 1.0 / (x - e[v].low);
      double plam = e[v].p0, qlam = e[v].q0;
#pragma unroll
      for (int i = 0; i < M; i++) {
        plam += e[v].P[i] * lam.v[i];
        qlam += e[v].Q[i] * lam.v[i];
        s[2 + i] += e[v].P[i] * uxi + e[v].Q[i] * xli;
      }
      const double rex = plam * uxi * uxi - qlam * xli * xli - xsi + eta;
      const double ca = xsi * (x - al), cb = eta * (be - x);
      const double rexsi = ca - epsi, reeta = cb - epsi;
      s[0] += rex * rex + rexsi * rexsi + reeta * reeta;
      s[1] += rexsi + reeta;
      mx[0] = fmax(mx[0], fabs(rex));
      mx[1] = fmax(mx[1], fmax(ca, cb));
      mx[2] = fmax(mx[2], -fmin(ca, cb));
      // Newton system pieces (its gvec is the residual's), with the reciprocals above and of
      // x - alfa, beta - x, diagx
      const double rux2 = uxi * uxi, rxl2 = xli * xli;
      const double rxa = 1.0 / (x - al), rbx = 1.0 / (be - x);
      double GG[M];
#pragma unroll
      for (int i = 0; i < M; i++) GG[i] = e[v].P[i] * rux2 - e[v].Q[i] * rxl2;
      const double dpsidx = plam * rux2 - qlam * rxl2;
      const double delx = dpsidx - epsi * rxa + epsi * rbx;
      const double diagx = 2.0 * (plam * rux2 * uxi + qlam * rxl2 * xli) + xsi * rxa + eta * rbx;
      const double id = 1.0 / diagx, dd = delx * id, de = (rxa - rbx) * id;
#pragma unroll
      for (int i = 0; i < M; i++) {
        s[2 + M + i] += GG[i] * dd;
        s[2 + 2 * M + i] += GG[i] * de;
#pragma unroll
        for (int k = 0; k < M; k++) s[2 + 3 * M + i * M + k] += GG[i] * GG[k] * id;
      }
    }
    if (moved) {
      if (VW == 2) {
        const size_t j = 2 * q;
        *reinterpret_cast<double2*>(out.x + j) = make_double2(e[0].x, e[VW - 1].x);
        *reinterpret_cast<double2*>(out.xsi + j) = make_double2(e[0].xsi, e[VW - 1].xsi);
        *reinterpret_cast<double2*>(out.eta + j) = make_double2(e[0].eta, e[VW - 1].eta);
      } else {
        out.x[q] = e[0].x;
        out.xsi[q] = e[0].xsi;
        out.eta[q] = e[0].eta;
      }
    }
  }
  if (reduce_to_result<NS, 3>(s, mx, w.partials, w.result, w.counter))
    mma_decide<NS + 3>(w.state, w.result, [](MmaState& T, const double* r) { mma_after_trial<M>(T, r); });
}

// The solution becomes x (also in FP32 to xf, if given), x and xold1 move one step back.
__global__ void k_mma_finish(size_t n, double* xvar, double* xold1, double* xold2, float* xf, MmaWork w) {
  const double* xs = mma_point(w, w.state->parity != 0).x;
  for (size_t j = size_t(blockIdx.x) * blockDim.x + threadIdx.x; j < n; j += size_t(gridDim.x) * blockDim.x) {
    const double x = xs[j];
    xold2[j] = xold1[j];
    xold1[j] = xvar[j];
    xvar[j] = x;
    if (xf) xf[j] = float(x);
  }
}

__global__ void k_cast_f2d(size_t n, const float* __restrict__ a, double* b) {
  for (size_t j = size_t(blockIdx.x) * blockDim.x + threadIdx.x; j < n; j += size_t(gridDim.x) * blockDim.x)
    b[j] = double(a[j]);
}

__global__ void k_fill(size_t n, double v, double* a) {
  for (size_t j = size_t(blockIdx.x) * blockDim.x + threadIdx.x; j < n; j += size_t(gridDim.x) * blockDim.x) a[j] = v;
}

// Device bytes of a subsolve's work arrays, every array 256-byte aligned.
static size_t mma_padded(size_t doubles) { return (doubles * sizeof(double) + 255) & ~size_t(255); }
static size_t mma_small_bytes() {
  return size_t(kMaxPartials) * kMmaSlots * sizeof(double) + kMmaSlots * sizeof(double) + 64 + sizeof(MmaState);
}
static size_t work_bytes(int m, size_t n) {
  return 10 * mma_padded(n) + 2 * mma_padded(size_t(m) * n) + mma_padded(mma_small_bytes() / sizeof(double) + 1);
}

// The work arrays carved out of `block` (work_bytes of it), or allocated one by one: from the scratch pool
// when async, else with cudaMalloc.
static otm_status work_alloc(MmaWork& w, int m, size_t n, cudaStream_t s, bool async, char* block = nullptr) {
  w.m = m;
  w.n = n;
  w.carved = block != nullptr;
  auto take = [&](void** p, size_t doubles) -> cudaError_t {
    if (block) {
      *p = block;
      block += mma_padded(doubles);
      return cudaSuccess;
    }
    const size_t bytes = doubles * sizeof(double);
    return async ? scratch_malloc(p, bytes, s) : cudaMalloc(p, bytes);
  };
  double** arr[] = {&w.alfa, &w.beta, &w.p0, &w.q0, &w.xs, &w.xsi, &w.eta, &w.dx, &w.dxsi, &w.deta};
  for (double** a : arr) OTM_CUDA(take((void**)a, n));
  for (double** a : {&w.P, &w.Q}) OTM_CUDA(take((void**)a, size_t(m) * n));
  OTM_CUDA(take((void**)&w.partials, mma_small_bytes() / sizeof(double) + 1));
  w.result = w.partials + size_t(kMaxPartials) * kMmaSlots;
  w.counter = (unsigned int*)(w.result + kMmaSlots);
  w.state = (MmaState*)(w.result + kMmaSlots + 8);
  OTM_CUDA(cudaMemsetAsync(w.counter, 0, 64, s));
  OTM_CUDA(cudaMallocHost((void**)&w.host, 2 * sizeof(int)));
  return OTM_OK;
}

static void work_free(MmaWork& w, cudaStream_t s, bool async) {
  double* arr[] = {w.alfa, w.beta, w.p0, w.q0, w.xs, w.xsi, w.eta, w.dx, w.dxsi, w.deta, w.P, w.Q, w.partials};
  for (double* a : arr)
    if (a && !w.carved) {
      if (async)
        cudaFreeAsync(a, s);
      else
        cudaFree(a);
    }
  if (w.host) cudaFreeHost(w.host);
  w = MmaWork{};
}

// Dispatch on the (compile-time) constraint count.
template <template <int> class K, typename... Args>
static void dispatch_m(int m, Args&&... args) {
  switch (m) {
    case 1: K<1>::run(args...); break;
    case 2: K<2>::run(args...); break;
    case 3: K<3>::run(args...); break;
    case 4: K<4>::run(args...); break;
    case 5: K<5>::run(args...); break;
    case 6: K<6>::run(args...); break;
    case 7: K<7>::run(args...); break;
    default: K<8>::run(args...); break;
  }
}

template <typename T>
struct Setup {
  template <int M>
  struct Launch {
    static void run(int nb, cudaStream_t s, size_t n, int itn, const MmaInputs<T>& in, const double* xmin,
                    const double* xmax, const double* xold1, const double* xold2, double* low, double* upp, double move,
                    const MmaProblem& pr, const MmaWork& w) {
      k_mma_setup<M, T><<<nb, 256, 0, s>>>(n, itn, in, xmin, xmax, xold1, xold2, low, upp, move, pr, w);
    }
  };
};

// The two passes of a Newton step; blocks_per_sm: how many of an instance's blocks are resident on an SM.
template <int M>
struct LaunchDirmax {
  static void run(int nb, bool pairs, cudaStream_t s, const double* low, const double* upp, const MmaWork& w) {
    if (pairs)
      k_mma_dirmax<M, 2><<<nb, 256, 0, s>>>(low, upp, w);
    else
      k_mma_dirmax<M, 1><<<nb, 256, 0, s>>>(low, upp, w);
  }
};
template <int M>
struct LaunchTrial {
  static void run(int nb, bool pairs, cudaStream_t s, const double* low, const double* upp, const MmaWork& w) {
    if (pairs)
      k_mma_trial<M, 2><<<nb, 256, 0, s>>>(low, upp, w);
    else
      k_mma_trial<M, 1><<<nb, 256, 0, s>>>(low, upp, w);
  }
};
template <int M>
struct ResidentBlocks {
  static void run(bool pairs, int* dirmax, int* trial, cudaError_t* e) {
    const void* d = pairs ? (const void*)k_mma_dirmax<M, 2> : (const void*)k_mma_dirmax<M, 1>;
    const void* t = pairs ? (const void*)k_mma_trial<M, 2> : (const void*)k_mma_trial<M, 1>;
    *e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(dirmax, d, 256, 0);
    if (*e == cudaSuccess) *e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(trial, t, 256, 0);
  }
};

// Newton steps (a step-bound pass and a trial) queued before the host first looks, and between later
// looks: a subproblem takes about 20 (measured on 128^3 and 384^3 design steps); a queued pair that
// finds nothing due costs about 3 us, a look about 15.
constexpr int kMmaFirstSteps = 16, kMmaMoreSteps = 4;

// One MMA step (mmasub_g, optimization/mmaOpt.cu:1021-1062): device arrays; a, c, d and the constraint
// values in pr.
template <typename T>
static otm_status mmasub_run(cudaStream_t s, int m, size_t n, int itn, const MmaInputs<T>& in, double* xvar,
                             const double* xmin, const double* xmax, double* xold1, double* xold2, double* low,
                             double* upp, const MmaProblem& pr, double move, float* xf, MmaWork& w) {
  const auto blocks = [](size_t work, int most) {
    return int(std::min<size_t>(size_t(most), std::max<size_t>(1, (work + 255) / 256)));
  };
  int dev = 0, sms = 0;
  OTM_CUDA(cudaGetDevice(&dev));
  OTM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int nb = blocks(n, std::min(4 * sms, kMaxPartials));
  uint64_t L = 0;
  dispatch_m<Setup<T>::template Launch>(m, nb, s, n, itn, in, xmin, xmax, xold1, xold2, low, upp, move, pr, w);
  L++;
  OTM_CHECK_LAUNCH("k_mma_setup");
  // pairs of variables per loop step when every array the passes read is 16-byte aligned at
  // every row (n even; the work arrays come from the allocator, low and upp from the caller)
  // (m <= 4: beyond that the pair of elements no longer fits the registers)
  const bool pairs = m <= 4 && n % 2 == 0 && (reinterpret_cast<uintptr_t>(low) % 16) == 0 &&
                     (reinterpret_cast<uintptr_t>(upp) % 16) == 0;
  const size_t groups = n / (pairs ? 2 : 1);
  // grids of the blocks that are resident at once, so that a block's reduction and the last block's sum over
  // all blocks are paid once per resident block (m = 1, n = 2.1 M: trial 51 us and step bounds 44 us, 76 and
  // 51 with 2048 blocks) and no second wave fills a part of the GPU: registers allow two and three blocks an SM
  // at m = 1, fewer from m = 2 on (three updates at n = 2.1 M with two and three blocks and with what fits:
  // m = 2 9.93 and 9.13 ms, m = 4 12.7 and 11.9, m = 8 30.5 and 28.9)
  int rd = 0, rt = 0;
  cudaError_t e = cudaSuccess;
  dispatch_m<ResidentBlocks>(m, pairs, &rd, &rt, &e);
  OTM_CUDA(e);
  const int nbt = blocks(groups, std::min(std::max(rt, 1) * sms, kMaxPartials)),
            nbd = blocks(groups, std::min(std::max(rd, 1) * sms, kMaxPartials));
  const double *lowc = low, *uppc = upp;
  dispatch_m<LaunchTrial>(m, nbt, pairs, s, lowc, uppc, w);
  L++;
  // the state machine ends: at most 200 Newton steps of at most 50 trials for each of 7 epsi
  for (int steps = kMmaFirstSteps;; steps = kMmaMoreSteps) {
    for (int i = 0; i < steps; i++) {
      dispatch_m<LaunchDirmax>(m, nbd, pairs, s, lowc, uppc, w);
      dispatch_m<LaunchTrial>(m, nbt, pairs, s, lowc, uppc, w);
      L += 2;
    }
    OTM_CHECK_LAUNCH("MMA passes");
    OTM_CUDA(cudaMemcpyAsync(w.host, w.state, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
    OTM_CUDA(cudaStreamSynchronize(s));
    if (w.host[0] == kMmaDone) break;
  }
  count_launches(L);
  if (w.host[1] != kMmaOk) {
    set_error(w.host[1] == kMmaSingular ? "singular MMA Newton system" : "NaN step in the MMA subproblem");
    return OTM_ERR_NAN;
  }
  k_mma_finish<<<nb, 256, 0, s>>>(n, xvar, xold1, xold2, xf, w);
  OTM_CHECK_LAUNCH("k_mma_finish");
  count_launches(1);
  return OTM_OK;
}

}  // namespace otm

using namespace otm;

struct otm_mma {
  int m = 0;
  size_t n = 0;
  double a0 = 1.0;
  std::vector<double> a, c, d;
  cudaStream_t stream = nullptr;
  double *xvar = nullptr, *xmin = nullptr, *xmax = nullptr, *xold1 = nullptr, *xold2 = nullptr;
  double *low = nullptr, *upp = nullptr;
  MmaWork w;
  char* block = nullptr;  // one allocation for all arrays, where it could be had
  ~otm_mma() {
    double* arr[] = {xvar, xmin, xmax, xold1, xold2, low, upp};
    for (double* p : arr)
      if (p && !block) cudaFree(p);
    work_free(w, nullptr, false);
    if (block) cudaFree(block);
  }
};

extern "C" {

otm_status otm_mma_create(int m, int n, double a0, double a, double c, double d, otm_mma** out) {
  if (!out || m < 1 || m > kMmaMaxM || n < 1) {
    set_error("need 1 <= m <= 8 constraints and n >= 1 variables");
    return OTM_ERR_INVALID_ARGUMENT;
  }
  *out = nullptr;
  otm_mma* o = new (std::nothrow) otm_mma();
  if (!o) return OTM_ERR_OUT_OF_MEMORY;
  o->m = m;
  o->n = size_t(n);
  o->a0 = a0;
  o->a.assign(m, a);
  o->c.assign(m, c);
  o->d.assign(m, d);
  auto fail = [&](otm_status st) {
    delete o;
    return st;
  };
  double** arr[] = {&o->xvar, &o->xmin, &o->xmax, &o->xold1, &o->xold2, &o->low, &o->upp};
  const size_t each = mma_padded(o->n);
  if (cudaMalloc((void**)&o->block, 7 * each + work_bytes(m, o->n)) != cudaSuccess) {
    cudaGetLastError();  // the arrays may still fit one by one
    o->block = nullptr;
  }
  char* at = o->block;
  for (double** p : arr) {
    if (at) {
      *p = (double*)at;
      at += each;
    } else {
      const cudaError_t e = cudaMalloc((void**)p, o->n * sizeof(double));
      if (e != cudaSuccess) return fail(cuda_fail(e, "cudaMalloc"));
    }
    cudaMemset(*p, 0, o->n * sizeof(double));
  }
  otm_status st = work_alloc(o->w, m, o->n, nullptr, false, at);
  if (st != OTM_OK) return fail(st);
  if (cudaDeviceSynchronize() != cudaSuccess) return fail(cuda_fail(cudaGetLastError(), "otm_mma_create"));
  *out = o;
  return OTM_OK;
}

otm_status otm_mma_destroy(otm_mma* mma) {
  if (!mma) return OTM_ERR_INVALID_ARGUMENT;
  cudaStreamSynchronize(mma->stream);
  delete mma;
  return OTM_OK;
}

otm_status otm_mma_set_stream(otm_mma* mma, void* stream) {
  if (!mma) return OTM_ERR_INVALID_ARGUMENT;
  mma->stream = (cudaStream_t)stream;
  return OTM_OK;
}

otm_status otm_mma_set_bound_scalar(otm_mma* mma, float xmin, float xmax) {
  if (!mma || !(xmax >= xmin)) return OTM_ERR_INVALID_ARGUMENT;
  const int nb = int(std::min<size_t>(kMaxPartials, (mma->n + 255) / 256));
  k_fill<<<nb, 256, 0, mma->stream>>>(mma->n, double(xmin), mma->xmin);
  k_fill<<<nb, 256, 0, mma->stream>>>(mma->n, double(xmax), mma->xmax);
  OTM_CHECK_LAUNCH("k_fill");
  count_launches(2);
  return OTM_OK;
}

otm_status otm_mma_set_bound(otm_mma* mma, const float* xmin_dev, const float* xmax_dev) {
  if (!mma || !xmin_dev || !xmax_dev) return OTM_ERR_INVALID_ARGUMENT;
  const int nb = int(std::min<size_t>(kMaxPartials, (mma->n + 255) / 256));
  k_cast_f2d<<<nb, 256, 0, mma->stream>>>(mma->n, xmin_dev, mma->xmin);
  k_cast_f2d<<<nb, 256, 0, mma->stream>>>(mma->n, xmax_dev, mma->xmax);
  OTM_CHECK_LAUNCH("k_cast_f2d");
  count_launches(2);
  return OTM_OK;
}

otm_status otm_mma_update(otm_mma* mma, int itn, float* x_dev, const float* dfdx_dev, const float* gval_host,
                          const float* const* dgdx_dev) {
  if (!mma || !x_dev || !dfdx_dev || !gval_host || !dgdx_dev) return OTM_ERR_INVALID_ARGUMENT;
  cudaStream_t s = mma->stream;
  const size_t n = mma->n;
  MmaInputs<float> in{};
  in.x = x_dev;
  in.df0dx = dfdx_dev;
  in.xvar_out = mma->xvar;
  MmaProblem pr{};
  pr.a0 = mma->a0;
  for (int i = 0; i < mma->m; i++) {
    if (!dgdx_dev[i]) return OTM_ERR_INVALID_ARGUMENT;
    in.dgdx[i] = dgdx_dev[i];
    pr.a[i] = mma->a[i];
    pr.c[i] = mma->c[i];
    pr.d[i] = mma->d[i];
    pr.g[i] = gval_host[i];
  }
  // f0val = 1 and move = 1 (optimization/mmaOptimizer.cu:69-70)
  return mmasub_run(s, mma->m, n, itn, in, mma->xvar, mma->xmin, mma->xmax, mma->xold1, mma->xold2, mma->low, mma->upp,
                    pr, 1.0, x_dev, mma->w);
}

otm_status otm_mmasub_device(int m, int n, int itn, double* xvar, double* xmin, double* xmax, double* xold1,
                             double* xold2, double f0val, double* df0dx, double* gval, otm_pitched_ptr dgdx,
                             double* low, double* upp, double a0, double* a, double* c, double* d, double move,
                             void* stream) {
  (void)f0val;  // unused by the reference as well
  if (m < 1 || m > kMmaMaxM || n < 1 || !xvar || !xmin || !xmax || !xold1 || !xold2 || !df0dx || !gval ||
      !dgdx.ptr || !low || !upp || !a || !c || !d || dgdx.pitch % sizeof(double) != 0 ||
      dgdx.pitch < size_t(n) * sizeof(double))
    return OTM_ERR_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  std::vector<double> hg(m), ha(m), hc(m), hd(m);
  OTM_CUDA(cudaMemcpyAsync(hg.data(), gval, m * sizeof(double), cudaMemcpyDeviceToHost, s));
  OTM_CUDA(cudaMemcpyAsync(ha.data(), a, m * sizeof(double), cudaMemcpyDeviceToHost, s));
  OTM_CUDA(cudaMemcpyAsync(hc.data(), c, m * sizeof(double), cudaMemcpyDeviceToHost, s));
  OTM_CUDA(cudaMemcpyAsync(hd.data(), d, m * sizeof(double), cudaMemcpyDeviceToHost, s));
  OTM_CUDA(cudaStreamSynchronize(s));
  MmaWork w;
  otm_status st = work_alloc(w, m, size_t(n), s, true);
  if (st == OTM_OK) {
    MmaInputs<double> in{};
    in.x = xvar;
    in.df0dx = df0dx;
    MmaProblem pr{};
    pr.a0 = a0;
    for (int i = 0; i < m; i++) {
      in.dgdx[i] = (const double*)dgdx.ptr + size_t(i) * (dgdx.pitch / sizeof(double));
      pr.a[i] = ha[i];
      pr.c[i] = hc[i];
      pr.d[i] = hd[i];
      pr.g[i] = hg[i];
    }
    st = mmasub_run(s, m, size_t(n), itn, in, xvar, xmin, xmax, xold1, xold2, low, upp, pr, move, (float*)nullptr, w);
  }
  work_free(w, s, true);
  return st;
}

}  // extern "C"
