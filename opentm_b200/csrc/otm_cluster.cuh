// otm_cluster.cuh -- the lower part of the V-cycle in one launch of one thread-block cluster.
//
// The levels with at most kClMaxNv unknowns, down to and including the coarsest direct solve,
// run in kCl CTAs of one cluster. Every level is split into slabs of z-planes, one slab per
// CTA; each CTA keeps u of its planes plus ghost copies of the two neighbouring planes, and f,
// r and the 27-point stencils of its planes (a first level too large for that keeps its stencils,
// right-hand side and residual in global memory, L2-resident), in its own shared memory. A CTA that writes
// an edge plane of u also stores the values into its neighbours' ghost copies (distributed
// shared memory), so colour passes and residuals read only local shared memory; restriction,
// prolongation and the coarsest gather read other CTAs' planes directly. The phases are
// separated by cluster barriers (barrier.cluster arrive/wait, release/acquire) instead of
// kernel boundaries, so the whole lower cycle costs one launch. A cluster barrier costs about
// as much as a small level's colour pass, so a sweep takes two: colours 0-3 update only the
// even planes and colours 4-7 only the odd ones, and within each half a vertex's changing
// neighbours lie in its own plane, held by its own CTA (CTA barriers between those passes). The arithmetic is that of the
// per-level kernels in otm_mg_kernels.cuh except for the summation order of the 27-point
// products; the coarsest solve is u = Ainv (f - mean f) as in k_coarsest_solve.
//
// The order of a vertex's 27 products is part of the results: a design run whose solves stop at a relative
// residual of 0.01 carries a last-bit change of one cycle into densities that differ by 1e-4 after ten
// steps. A colour pass sums the offsets 0..26 one after the other (three sums by plane, a shorter chain:
// 128^3 OC steps 0.7 % faster, 32^3 solves not), a residual as cl_resid_smem says.
#pragma once

#include <cooperative_groups.h>

#include <algorithm>
#include <climits>
#include <vector>

#include "otm_mg_kernels.cuh"

namespace otm {

constexpr int kCl = 16;            // CTAs per cluster (non-portable size, opted in at set-up): one
                                   // 32^3 colour pass at 16 CTAs loads half the stencils per SM of 8
constexpr int kClThreads = 512;    // 640: 2% slower on 32^3 and 40 x 56 x 72 solves, 4% faster on 96 x 128 x 64 V(1,1)
constexpr int kClMaxLevels = 8;
constexpr int kClMaxNv = 32768;    // unknowns of the first level handled by the cluster (32^3)
constexpr int kClSlots = 256;      // stencil stride of the levels with at most that many vertices per CTA
constexpr int kClMaxTab = 6144;    // plane-table entries over all levels (3 per plane)

struct ClLevel {
  Dims d;
  int cs;      // case stride of f and r in shared memory: (planes of the fullest slab) * nx * ny
  int uh;      // position of a row's odd sites in u: site x lies at (x odd ? uh : 0) + x / 2
  int urs;     // u row stride (at least nx, chosen with uh against shared-memory bank conflicts)
  int ups;     // u plane stride (ny * urs, padded)
  int ucs;     // u case stride: two more planes (ghost copies of the neighbouring slabs' edge planes)
  int u_off;   // float offsets in shared memory
  int f_off;   // < 0: right-hand side read from f_in (global; first level only, when not staged)
  int r_off;   // < 0: residual in rg (global, lexicographic, case-major)
  int ss;      // stencil stride: entry o of slot s at st_off + o * ss + s (kClSlots where the slots fit that)
  int st_off;  // < 0: stencils read from st (global, colour-blocked)
  int inv_off; // inverse diagonal per slot (with st_off >= 0)
  int tab_off; // plane tables of this level: nz ownership entries, then 2 nz ghost-push entries
  int lnx, lny;  // log2 of nx, ny rounded up (residual enumeration)
  int res8;    // the residual's 27 products in eight sums (levels of few vertices per CTA), else in one
  int zstart[kCl + 1];  // CTA c holds planes [zstart[c], zstart[c+1])
  const float* st;
  float* rg;
};

struct ClDesc {
  int nlev;  // levels in the cluster part; the last one is the coarsest
  int pre, post;
  int nc;          // unknowns of the coarsest level
  int gather_off;  // float offset of the coarsest right-hand-side gather buffer (3 nc floats)
  int tab_base;    // float offset of the plane tables (ints)
  int ntab;        // their entries (cl_tables), copied from tab_g at the start of a call
  const int* tab_g;
  ClLevel lv[kClMaxLevels];
  const float* f_in;  // right-hand side of the first level (global, case-major)
  float* u_out;       // its correction (global)
  const double* Ainv;
};

// Layout of u on a CTA that holds planes [z0, z1): local plane 0 is a copy of plane z0 - 1,
// planes 1..z1-z0 are its own, plane z1-z0+1 a copy of plane z1 (periodic). A CTA that writes
// an edge plane also writes the value into the copies held by its neighbours ("ghost push"),
// so every read of a colour pass or residual is a local shared-memory load.

// In-row position of site x of u: even and odd sites apart, so that the lanes of a colour pass, which
// take every other site of a row, read consecutive words.
__device__ __forceinline__ int cl_ux(const ClLevel& L, int x) { return ((x & 1) ? L.uh : 0) + (x >> 1); }

// On a level with its stencils in shared memory a CTA orders its vertices by colour ("slots": colours
// 0..3 of its even planes, then 4..7 of its odd planes, lexicographic inside a colour), and keeps the
// stencils, the inverse diagonal and the right-hand side in that order: the lanes of a pass read
// consecutive words.
struct ClSlots {
  int n[2], zf[2];  // vertices per colour and first plane, by plane parity
  int npl[2];       // own planes of the parity
  __device__ __forceinline__ ClSlots(const ClLevel& L, int rank) {
    const int z0 = L.zstart[rank], z1 = L.zstart[rank + 1], per = (L.d.nx >> 1) * (L.d.ny >> 1);
#pragma unroll
    for (int p = 0; p < 2; p++) {
      zf[p] = z0 + (((z0 & 1) != p) ? 1 : 0);
      npl[p] = zf[p] < z1 ? (z1 - zf[p] + 1) >> 1 : 0;
      n[p] = npl[p] * per;
    }
  }
  __device__ __forceinline__ int total() const { return 4 * (n[0] + n[1]); }
  __device__ __forceinline__ int base(int color) const {
    return (color >> 2) ? 4 * n[0] + (color & 3) * n[1] : color * n[0];
  }
  // slot of the own vertex (x, y, z)
  __device__ __forceinline__ int slot(const ClLevel& L, int x, int y, int z) const {
    const int hx = L.d.nx >> 1, hy = L.d.ny >> 1;
    return base((x & 1) + 2 * (y & 1) + 4 * (z & 1)) +
           ((((z - ((z & 1) ? zf[1] : zf[0])) >> 1) * hy + (y >> 1)) * hx + (x >> 1));
  }
};

// Plane z of r, or of f on the coarsest level (in-plane stride nx), at `off` of level L, wherever it
// lives in the cluster (case 0; case c is at + c * L.cs).
__device__ __forceinline__ const float* cl_plane(const ClLevel& L, const int* tab, float* const* rb, int off, int z) {
  const int e = tab[L.tab_off + z];
  return rb[e >> 16] + off + (e & 0xffff) * (L.d.nx * L.d.ny);
}

// Plane z of u (row stride urs; own planes start at local plane 1; case c at + c * L.ucs).
__device__ __forceinline__ const float* cl_uplane(const ClLevel& L, const int* tab, float* const* rb, int z) {
  const int e = tab[L.tab_off + z];
  return rb[e >> 16] + L.u_off + ((e & 0xffff) + 1) * L.ups;
}

// The ghost copies of plane z of u held by the neighbouring CTAs, at in-plane u index p of case
// 0 (null where plane z feeds fewer than two ghost copies). Taken before the stores of a vertex.
__device__ __forceinline__ void cl_ghosts(const ClLevel& L, const int* tab, float* const* rb, int z, int p,
                                          float*& g0, float*& g1) {
  const int* pt = tab + L.tab_off + L.d.nz + 2 * z;
  const int e0 = pt[0], e1 = pt[1];
  g0 = e0 >= 0 ? rb[e0 >> 16] + L.u_off + (e0 & 0xffff) * L.ups + p : nullptr;
  g1 = e1 >= 0 ? rb[e1 >> 16] + L.u_off + (e1 & 0xffff) * L.ups + p : nullptr;
}

// A read-only load that stays where it is written (the compiler otherwise moves loads next to their use
// to save registers, which makes a chain of L2 latencies of them).
__device__ __forceinline__ float ld_issue(const float* p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

// The colour passes (gs_coarse_body): a CTA updates its vertices of a colour and pushes updated edge-plane
// values to the ghosts. A colour of a CTA has at most kClThreads vertices (cl_plan_try), one lane each or
// one per load case.
// Stencils in shared memory: one colour pass of a half sweep (colours (cx, cy) of one plane parity) by
// one lane per vertex and load case. `V` is the lane's vertex block: what does not change over the four
// colours of the half sweep, so that a pass is its 26 products, one store and its pushes.
struct ClHalf {
  const float* st;  // stencils at the slot of colour (0, 0); colour q is q * n further
  float* up;        // u, local plane of z - 1, case of the lane
  float *g0, *g1;   // ghost copies of plane z, same case (null: none)
  int n;            // slots per colour
  int ss, ups;
  int row[4];       // offsets of the rows 2j - 1 .. 2j + 2
  int xp[4];        // in-row positions of the sites 2i - 1 .. 2i + 2
  float f[4], inv[4];  // right-hand side and inverse diagonal of the four colours
  bool on;
};

template <int q, int kSS>
__device__ __forceinline__ void cl_half_pass(const ClHalf& V) {
  constexpr int cx = q & 1, cy = q >> 1;
  const float* sp = V.st + q * V.n;
  const int ss = kSS ? kSS : V.ss;
  float st[27];
#pragma unroll
  for (int o = 0; o < 27; o++)
    if (o != 13) st[o] = sp[o * ss];
  float acc = 0.f;
#pragma unroll
  for (int o = 0; o < 27; o++)
    if (o != 13) acc += st[o] * V.up[(o / 9) * V.ups + V.row[cy + (o / 3) % 3] + V.xp[cx + o % 3]];
  const float v = (V.f[q] - acc) * V.inv[q];
  const int p = V.row[cy + 1] + V.xp[cx + 1];
  if (V.on) {
    V.up[V.ups + p] = v;
    if (V.g0) V.g0[p] = v;
    if (V.g1) V.g1[p] = v;
  }
}

// Colours 0..3 of the planes of parity pz (3..0 when kRev). A case's vertices are in warps of their own
// (the 27 products of a case need no other case's: 16^3 has 64 vertices of a colour on a CTA, two warps,
// which would each work through the three cases one after the other); the warps that hold a vertex
// synchronise among themselves between the colours. A pass used to be a chain of index arithmetic, table
// look-ups and conflicting reads, 2,100 cycles at 16^3 for a hundred instructions of work; the launch
// for 16^3 and below took 77 us (32^3 cell, warm) and takes 47 us.
template <bool kRev, int kSS>
__device__ __forceinline__ void cl_half_run(const ClHalf& V, int nthreads) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    switch (kRev ? 3 - k : k) {
      case 0: cl_half_pass<0, kSS>(V); break;
      case 1: cl_half_pass<1, kSS>(V); break;
      case 2: cl_half_pass<2, kSS>(V); break;
      default: cl_half_pass<3, kSS>(V); break;
    }
    if (k < 3) asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
  }
}

// As cl_half_pass by one lane per vertex with its three cases (more vertices of a colour than a third of
// the threads): fs, is: the right-hand side and the inverse diagonal at the slot of colour (0, 0).
template <int q>
__device__ __forceinline__ void cl_half_pass3(const ClHalf& V, const float* fs, const float* is, int cs, int ucs) {
  constexpr int cx = q & 1, cy = q >> 1;
  const float* sp = V.st + q * V.n;
  float acc[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int o = 0; o < 27; o++) {
    if (o == 13) continue;
    const float st = sp[o * V.ss];
    const float* u = V.up + (o / 9) * V.ups + V.row[cy + (o / 3) % 3] + V.xp[cx + o % 3];
#pragma unroll
    for (int c = 0; c < 3; c++) acc[c] += st * u[c * ucs];
  }
  const float inv = is[q * V.n];
  const int p = V.row[cy + 1] + V.xp[cx + 1];
  float v[3];
#pragma unroll
  for (int c = 0; c < 3; c++) v[c] = (fs[c * cs + q * V.n] - acc[c]) * inv;
  if (V.on) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      V.up[V.ups + p + c * ucs] = v[c];
      if (V.g0) V.g0[p + c * ucs] = v[c];
      if (V.g1) V.g1[p + c * ucs] = v[c];
    }
  }
}

template <bool kRev>
__device__ __forceinline__ void cl_half_sweep(const ClLevel& L, float* sm, const int* tab, float* const* rb, int rank,
                                              int pz) {
  const ClSlots sl(L, rank);
  const int zf = pz ? sl.zf[1] : sl.zf[0], n = pz ? sl.n[1] : sl.n[0];
  const int nx = L.d.nx, ny = L.d.ny, hx = nx >> 1, hy = ny >> 1, z0 = L.zstart[rank];
  const int cs = L.cs;
  const int nw = (n + 31) & ~31;  // whole warps per case
  const bool split = 3 * nw <= kClThreads;  // a lane per vertex and case, else per vertex
  const int nthreads = split ? 3 * nw : nw;
  if (int(threadIdx.x) >= nthreads) return;
  auto vertex = [&](int t, int c) {
    ClHalf V;
    V.on = t < n;
    if (!V.on) t = 0;
    const int row = t / hx, i = t - row * hx, pk = row / hy, j = row - pk * hy;
    const int z = zf + 2 * pk, s = (pz ? 4 * sl.n[0] : 0) + t;
    V.n = n;
    V.ss = L.ss;
    V.ups = L.ups;
    V.st = sm + L.st_off + s;
    V.up = sm + L.u_off + c * L.ucs + (z - z0) * L.ups;  // local planes z - z0 .. + 2 are z - 1, z, z + 1
#pragma unroll
    for (int k = 0; k < 4; k++) {
      V.row[k] = wrapm(2 * j - 1 + k, ny) * L.urs;
      V.xp[k] = cl_ux(L, wrapm(2 * i - 1 + k, nx));
      V.f[k] = sm[L.f_off + c * cs + s + k * n];
      V.inv[k] = sm[L.inv_off + s + k * n];
    }
    cl_ghosts(L, tab, rb, z, 0, V.g0, V.g1);
    if (V.g0) V.g0 += c * L.ucs;
    if (V.g1) V.g1 += c * L.ucs;
    return V;
  };
  if (split) {
    const int c = int(threadIdx.x) / nw;
    const ClHalf V = vertex(int(threadIdx.x) - c * nw, c);
    if (L.ss == kClSlots)
      cl_half_run<kRev, kClSlots>(V, nthreads);
    else
      cl_half_run<kRev, 0>(V, nthreads);
    return;
  }
  const ClHalf V = vertex(int(threadIdx.x), 0);
  const int at = (pz ? 4 * sl.n[0] : 0) + (V.on ? int(threadIdx.x) : 0), ucs = L.ucs;
  const float *fs = sm + L.f_off + at, *is = sm + L.inv_off + at;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    switch (kRev ? 3 - k : k) {
      case 0: cl_half_pass3<0>(V, fs, is, cs, ucs); break;
      case 1: cl_half_pass3<1>(V, fs, is, cs, ucs); break;
      case 2: cl_half_pass3<2>(V, fs, is, cs, ucs); break;
      default: cl_half_pass3<3>(V, fs, is, cs, ucs); break;
    }
    if (k < 3) asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
  }
}

// Stencils in global memory: colours 0..3 of the planes of parity pz (3..0 when kRev), one lane per vertex
// with its three cases, addresses and ghost targets found once for the four colours. A stencil value of the
// next colour is loaded into its register as soon as the current colour has used it, so a pass waits on
// shared memory and not on L2.
template <int q, int qn>
__device__ __forceinline__ void cl_half_pass_global(const ClHalf& V, int ucs, const float* sp, const float* f,
                                                    int nsub, int nv, int nx, float (&st)[27], float (&fv)[3]) {
  constexpr int cx = q & 1, cy = q >> 1;
  const float inv = 1.0f / st[13], f0 = fv[0], f1 = fv[1], f2 = fv[2];
  float acc[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int o = 0; o < 27; o++) {
    if (o != 13) {
      const float* u = V.up + (o / 9) * V.ups + V.row[cy + (o / 3) % 3] + V.xp[cx + o % 3];
#pragma unroll
      for (int c = 0; c < 3; c++) acc[c] += st[o] * u[c * ucs];
    }
    if (qn >= 0) st[o] = ld_issue(sp + (qn * nsub + o * nv));
  }
  if (qn >= 0)
#pragma unroll
    for (int c = 0; c < 3; c++) fv[c] = ld_issue(f + (c * nv + (qn >> 1) * nx + (qn & 1)));
  const int p = V.row[cy + 1] + V.xp[cx + 1];
  const float v[3] = {(f0 - acc[0]) * inv, (f1 - acc[1]) * inv, (f2 - acc[2]) * inv};
  if (V.on) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      V.up[V.ups + p + c * ucs] = v[c];
      if (V.g0) V.g0[p + c * ucs] = v[c];
      if (V.g1) V.g1[p + c * ucs] = v[c];
    }
  }
}

template <bool kRev>
__device__ __forceinline__ void cl_half_global(const ClLevel& L, const float* __restrict__ f_glob, float* sm,
                                               const int* tab, float* const* rb, int rank, int pz) {
  const ClSlots sl(L, rank);
  const int zf = pz ? sl.zf[1] : sl.zf[0], n = pz ? sl.n[1] : sl.n[0];
  const int nx = L.d.nx, ny = L.d.ny, hx = nx >> 1, hy = ny >> 1, z0 = L.zstart[rank];
  const int nthreads = (n + 31) & ~31;
  if (int(threadIdx.x) >= nthreads) return;
  ClHalf V;
  V.on = int(threadIdx.x) < n;
  const int t = V.on ? int(threadIdx.x) : 0;
  const int row = t / hx, i = t - row * hx, pk = row / hy, j = row - pk * hy, z = zf + 2 * pk;
  V.ups = L.ups;
  V.up = sm + L.u_off + (z - z0) * L.ups;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    V.row[k] = wrapm(2 * j - 1 + k, ny) * L.urs;
    V.xp[k] = cl_ux(L, wrapm(2 * i - 1 + k, nx));
  }
  cl_ghosts(L, tab, rb, z, 0, V.g0, V.g1);
  const int nv = int(L.d.nv()), nsub = nv >> 3;  // at most kClMaxNv
  const float* sp = L.st + (4 * pz * nsub + (zf >> 1) * hx * hy + t);
  const float* f = f_glob + ((z * ny + 2 * j) * nx + 2 * i);
  const int ucs = L.ucs;
  constexpr int q0 = kRev ? 3 : 0;
  float st[27], fv[3];
#pragma unroll
  for (int o = 0; o < 27; o++) st[o] = ld_issue(sp + (q0 * nsub + o * nv));
#pragma unroll
  for (int c = 0; c < 3; c++) fv[c] = ld_issue(f + (c * nv + (q0 >> 1) * nx + (q0 & 1)));
  cl_half_pass_global<(kRev ? 3 : 0), (kRev ? 2 : 1)>(V, ucs, sp, f, nsub, nv, nx, st, fv);
  asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
  cl_half_pass_global<(kRev ? 2 : 1), (kRev ? 1 : 2)>(V, ucs, sp, f, nsub, nv, nx, st, fv);
  asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
  cl_half_pass_global<(kRev ? 1 : 2), (kRev ? 0 : 3)>(V, ucs, sp, f, nsub, nv, nx, st, fv);
  asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
  cl_half_pass_global<(kRev ? 0 : 3), -1>(V, ucs, sp, f, nsub, nv, nx, st, fv);
}

// Half a sweep of a level: colours 0-3 update the even planes, 4-7 the odd ones, and a pass's changing
// neighbours are in its own plane, so the passes of a half need only the CTA's barriers; the cluster
// barrier after it makes the planes visible to the neighbouring CTAs.
template <bool kRev, typename Cluster>
__device__ __forceinline__ void cl_half(const ClLevel& L, const float* f_glob, float* sm, const int* tab,
                                        float* const* rb, int rank, int pz, Cluster& cluster) {
  if (L.st_off >= 0)
    cl_half_sweep<kRev>(L, sm, tab, rb, rank, pz);
  else
    cl_half_global<kRev>(L, f_glob, sm, tab, rb, rank, pz);
  cluster.sync();
}

// r = f - A u on this CTA's vertices (resid_coarse_body): stencils in global memory, one lane per vertex.
__device__ __forceinline__ void cl_resid_global(const ClLevel& L, const float* __restrict__ f_glob, float* sm,
                                                int rank) {
  const Dims d = L.d;
  const int nx = d.nx, ny = d.ny, plane = nx * ny;
  const int z0 = L.zstart[rank], z1 = L.zstart[rank + 1];
  const int lnx = L.lnx, lny = L.lny;
  const int n = (z1 - z0) << (lnx + lny);
  const int ucs = L.ucs, urs = L.urs, ups = L.ups;
  const size_t nv = d.nv();
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const int x = t & ((1 << lnx) - 1), y = (t >> lnx) & ((1 << lny) - 1), zl = t >> (lnx + lny), z = z0 + zl;
    if (x >= nx || y >= ny) continue;
    const int xo[3] = {cl_ux(L, wrapm(x - 1, nx)), cl_ux(L, x), cl_ux(L, wrapm(x + 1, nx))};
    const int yo[3] = {wrapm(y - 1, ny) * urs, y * urs, wrapm(y + 1, ny) * urs};
    const float* u = sm + L.u_off + zl * ups;
    const float* sp = L.st + cb_index(d, x, y, z);
    const size_t gi = size_t(z) * plane + y * nx + x;
    float st[27], fv[3], acc[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int o = 0; o < 27; o++) st[o] = ld_issue(sp + o * nv);
#pragma unroll
    for (int c = 0; c < 3; c++) fv[c] = ld_issue(f_glob + c * nv + gi);
#pragma unroll
    for (int o = 0; o < 27; o++) {
      const float* q = u + (o / 9) * ups + yo[(o / 3) % 3] + xo[o % 3];
#pragma unroll
      for (int c = 0; c < 3; c++) acc[c] += st[o] * q[c * ucs];
    }
#pragma unroll
    for (int c = 0; c < 3; c++) L.rg[c * nv + gi] = fv[c] - acc[c];
  }
}

// The same with the stencils in shared memory: one lane per vertex and load case, in slot order. kStride
// sums, of the offsets k, k + kStride, ..., added pairwise at half the distance each time.
template <int kStride>
__device__ __forceinline__ void cl_resid_smem(const ClLevel& L, float* sm, int rank) {
  const Dims d = L.d;
  const int nx = d.nx, ny = d.ny, hx = nx >> 1, hy = ny >> 1, z0 = L.zstart[rank];
  const ClSlots sl(L, rank);
  const int cs = L.cs, urs = L.urs, ups = L.ups, total = sl.total();
  for (int g = threadIdx.x; g < 3 * total; g += blockDim.x) {
    const int c = g >= 2 * total ? 2 : (g >= total ? 1 : 0), s = g - c * total;
    const int pz = s >= 4 * sl.n[0], q = s - (pz ? 4 * sl.n[0] : 0), n = pz ? sl.n[1] : sl.n[0];
    const int cxy = q >= 2 * n ? (q >= 3 * n ? 3 : 2) : (q >= n ? 1 : 0), t = q - cxy * n;
    const int row = t / hx, i = t - row * hx, pk = row / hy, j = row - pk * hy;
    const int x = 2 * i + (cxy & 1), y = 2 * j + (cxy >> 1), zl = (pz ? sl.zf[1] : sl.zf[0]) + 2 * pk - z0;
    const int xo[3] = {cl_ux(L, wrapm(x - 1, nx)), cl_ux(L, x), cl_ux(L, wrapm(x + 1, nx))};
    const int yo[3] = {wrapm(y - 1, ny) * urs, y * urs, wrapm(y + 1, ny) * urs};
    const float* u = sm + L.u_off + c * L.ucs + zl * ups;
    const float* sp = sm + L.st_off + s;
    float acc[kStride];
#pragma unroll
    for (int k = 0; k < kStride; k++) acc[k] = 0.f;
#pragma unroll
    for (int o = 0; o < 27; o++) acc[o % kStride] += sp[o * L.ss] * u[(o / 9) * ups + yo[(o / 3) % 3] + xo[o % 3]];
#pragma unroll
    for (int h = kStride >> 1; h > 0; h >>= 1)
#pragma unroll
      for (int k = 0; k < h; k++) acc[k] += acc[k + h];
    sm[L.r_off + c * cs + zl * nx * ny + y * nx + x] = sm[L.f_off + c * cs + s] - acc[0];
  }
}

__device__ __forceinline__ void cl_resid(const ClLevel& L, const float* f_glob, float* sm, int rank) {
  if (L.st_off < 0)
    cl_resid_global(L, f_glob, sm, rank);
  else if (L.res8)
    cl_resid_smem<8>(L, sm, rank);
  else
    cl_resid_smem<1>(L, sm, rank);
}

// u = 0 on this CTA's planes of a level, ghost copies included.
__device__ __forceinline__ void cl_zero_u(const ClLevel& L, float* sm, int rank) {
  const int n = (L.zstart[rank + 1] - L.zstart[rank] + 2) * L.ups;
  for (int idx = threadIdx.x; idx < 3 * n; idx += blockDim.x) {
    const int c = idx / n;
    sm[L.u_off + c * L.ucs + (idx - c * n)] = 0.f;
  }
}

// f_C = P^T r_F on this CTA's coarse vertices (restrict_body).
__device__ __forceinline__ void cl_restrict(const ClLevel& F, const ClLevel& C, float* sm, const int* tab,
                                            float* const* rb, int rank) {
  const Dims df = F.d, dc = C.d;
  const int pc = dc.nx * dc.ny, pf = df.nx * df.ny;
  const int Z0 = C.zstart[rank], Z1 = C.zstart[rank + 1];
  const ClSlots sl(C, rank);
  // one lane per coarse vertex and load case: 27 loads, most of them from other CTAs, in flight each
  const int n = (Z1 - Z0) * pc;
  for (int g = threadIdx.x; g < 3 * n; g += blockDim.x) {
    const int c = g / n, t = g - c * n;
    const int Zl = t / pc, rem = t - Zl * pc, Y = rem / dc.nx, X = rem - Y * dc.nx, Z = Z0 + Zl;
    const int xs[3] = {wrapm(2 * X - 1, df.nx), 2 * X, wrapm(2 * X + 1, df.nx)};
    const int ys[3] = {wrapm(2 * Y - 1, df.ny), 2 * Y, wrapm(2 * Y + 1, df.ny)};
    const int zs[3] = {wrapm(2 * Z - 1, df.nz), 2 * Z, wrapm(2 * Z + 1, df.nz)};
    const float* pr[3];
#pragma unroll
    for (int k = 0; k < 3; k++)
      pr[k] = F.r_off >= 0 ? cl_plane(F, tab, rb, F.r_off, zs[k]) + c * F.cs
                           : F.rg + size_t(c) * df.nv() + size_t(zs[k]) * pf;
    float acc = 0.f;
#pragma unroll
    for (int o = 0; o < 27; o++) {
      const int ox = o % 3 - 1, oy = (o / 3) % 3 - 1, oz = o / 9 - 1;
      const float w = (ox ? 0.5f : 1.f) * (oy ? 0.5f : 1.f) * (oz ? 0.5f : 1.f);
      const float* q = pr[oz + 1] + ys[oy + 1] * df.nx + xs[ox + 1];
      // a global residual was written by other CTAs of this launch: read it past L1
      acc += w * (F.r_off >= 0 ? *q : __ldcg(q));
    }
    sm[C.f_off + c * C.cs + (C.st_off >= 0 ? sl.slot(C, X, Y, Z) : t)] = acc;
  }
  cl_zero_u(C, sm, rank);
}

// u_C = Ainv (f_C - mean f_C) on this CTA's coarsest vertices (k_coarsest_solve): every CTA
// gathers the whole right-hand side, then one warp per own vertex forms the row product.
__device__ __forceinline__ void cl_coarsest(const ClDesc& cd, float* sm, const int* tab, float* const* rb,
                                            int rank, double* cmean) {
  const ClLevel& C = cd.lv[cd.nlev - 1];
  const int n = cd.nc, pc = C.d.nx * C.d.ny;
  float* g = sm + cd.gather_off;
  for (int idx = threadIdx.x; idx < 3 * n; idx += blockDim.x) {
    const int c = idx / n, v = idx - c * n, z = v / pc;
    g[idx] = cl_plane(C, tab, rb, C.f_off, z)[c * C.cs + (v - z * pc)];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < 3) {
    double s = 0.0;
    for (int i = lane; i < n; i += 32) s += double(g[warp * n + i]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) cmean[warp] = s / n;
  }
  __syncthreads();
  const int z0 = C.zstart[rank], z1 = C.zstart[rank + 1];
  const int nown = (z1 - z0) * pc;
  const double m0 = cmean[0], m1 = cmean[1], m2 = cmean[2];
  for (int t = warp; t < nown; t += int(blockDim.x >> 5)) {
    const int i = z0 * pc + t;  // lexicographic coarsest index
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
#pragma unroll 4
    for (int j = lane; j < n; j += 32) {
      const double m = __ldg(cd.Ainv + size_t(i) * n + j);  // symmetric: row i == column i
      a0 += m * (double(g[j]) - m0);
      a1 += m * (double(g[n + j]) - m1);
      a2 += m * (double(g[2 * n + j]) - m2);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      a0 += __shfl_xor_sync(0xffffffffu, a0, off);
      a1 += __shfl_xor_sync(0xffffffffu, a1, off);
      a2 += __shfl_xor_sync(0xffffffffu, a2, off);
    }
    if (lane == 0) {
      const int zl = t / pc, rem = t - zl * pc, y = rem / C.d.nx, x = rem - y * C.d.nx;
      float* u = sm + C.u_off + (zl + 1) * C.ups + y * C.urs + cl_ux(C, x);  // own planes start at local plane 1
      u[0] = float(a0);
      u[C.ucs] = float(a1);
      u[2 * C.ucs] = float(a2);
    }
  }
}

// u_F += P u_C on this CTA's fine vertices (prolong_body); edge-plane results pushed to ghosts.
__device__ __forceinline__ void cl_prolong(const ClLevel& F, const ClLevel& C, float* sm, const int* tab,
                                           float* const* rb, int rank) {
  const Dims df = F.d, dc = C.d;
  const int pf = df.nx * df.ny;
  const int z0 = F.zstart[rank], z1 = F.zstart[rank + 1];
  // one lane per fine vertex and load case
  const int n = (z1 - z0) * pf;
  for (int g = threadIdx.x; g < 3 * n; g += blockDim.x) {
    const int c = g >= 2 * n ? 2 : (g >= n ? 1 : 0), t = g - c * n;
    const int zl = t / pf, rem = t - zl * pf, y = rem / df.nx, x = rem - y * df.nx, z = z0 + zl;
    const int X0 = x >> 1, Y0 = y >> 1, Z0 = z >> 1;
    const int X1 = (x & 1) ? wrapm(X0 + 1, dc.nx) : X0;
    const int Y1 = (y & 1) ? wrapm(Y0 + 1, dc.ny) : Y0;
    const int Z1 = (z & 1) ? wrapm(Z0 + 1, dc.nz) : Z0;
    const float wx1 = (x & 1) ? 0.5f : 0.f, wy1 = (y & 1) ? 0.5f : 0.f, wz1 = (z & 1) ? 0.5f : 0.f;
    const float wx0 = 1.f - wx1, wy0 = 1.f - wy1, wz0 = 1.f - wz1;
    const float* u0 = cl_uplane(C, tab, rb, Z0) + c * C.ucs;
    const float* u1 = cl_uplane(C, tab, rb, Z1) + c * C.ucs;
    const int r0 = Y0 * C.urs, r1 = Y1 * C.urs;
    const int pu_idx = y * F.urs + cl_ux(F, x), p0 = cl_ux(C, X0), p1 = cl_ux(C, X1);
    // every load (coarse values, possibly in other CTAs, the old fine value and the ghost
    // targets) before the first store
    float* uf = sm + F.u_off + c * F.ucs + (zl + 1) * F.ups + pu_idx;
    const float a = wz0 * (wy0 * (wx0 * u0[r0 + p0] + wx1 * u0[r0 + p1]) +
                           wy1 * (wx0 * u0[r1 + p0] + wx1 * u0[r1 + p1])) +
                    wz1 * (wy0 * (wx0 * u1[r0 + p0] + wx1 * u1[r0 + p1]) +
                           wy1 * (wx0 * u1[r1 + p0] + wx1 * u1[r1 + p1]));
    float *g0, *g1;
    cl_ghosts(F, tab, rb, z, pu_idx, g0, g1);
    const float v = *uf + a;
    *uf = v;
    if (g0) g0[c * F.ucs] = v;
    if (g1) g1[c * F.ucs] = v;
  }
}

static __global__ void __cluster_dims__(kCl, 1, 1) __launch_bounds__(kClThreads)
    k_vcycle_cluster(ClDesc cdp, const SolveScalars* sc) {
  pdl_wait();
  // every CTA reads the same flag (written by earlier kernels), so the whole cluster leaves
  // together before any distributed shared memory access
  if (sc && solve_done(sc)) return;
  extern __shared__ __align__(16) float sm[];
  __shared__ float* rb[kCl];
  __shared__ double cmean[3];
  // the descriptor is indexed by level at run time: a shared copy keeps it out of local memory
  __shared__ ClDesc cd;
  {
    const int* src = reinterpret_cast<const int*>(&cdp);
    int* dst = reinterpret_cast<int*>(&cd);
    for (int i = threadIdx.x; i < int(sizeof(ClDesc) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int rank = int(cluster.block_rank());
  // other CTAs' shared memory through the cluster window, this CTA's own directly
  if (threadIdx.x < kCl) rb[threadIdx.x] = int(threadIdx.x) == rank ? sm : cluster.map_shared_rank(sm, int(threadIdx.x));
  int* tab = reinterpret_cast<int*>(sm + cd.tab_base);
  const int L = cd.nlev;
  // plane tables (built on the host by cl_tables): owner and local plane of every plane, and the
  // ghost copies every plane feeds
  for (int i = threadIdx.x; i < cd.ntab; i += blockDim.x) tab[i] = __ldg(cd.tab_g + i);
  // the coarsest inverse is read once, late in the cycle: bring it into L2 now
  l2_prefetch_share(cd.Ainv, size_t(cd.nc) * size_t(cd.nc) * sizeof(double));
  // first level: zero correction (ghosts included) and, where it is staged, its right-hand side;
  // stencils of the other smoothed levels. One thread per own vertex, all of its loads in flight
  // before its stores (a copy of one element per round trip made this a chain of L2 latencies).
  cl_zero_u(cd.lv[0], sm, rank);
  for (int l = 0; l < L - 1; l++) {
    const ClLevel& V = cd.lv[l];
    if (V.st_off < 0) continue;
    const ClSlots sl(V, rank);
    const int hx = V.d.nx >> 1, hy = V.d.ny >> 1, per = hx * hy, cs = V.cs;
    const size_t nv = V.d.nv();
    for (int s = threadIdx.x; s < sl.total(); s += blockDim.x) {
      const int pz = s >= 4 * sl.n[0], q = s - (pz ? 4 * sl.n[0] : 0), n = pz ? sl.n[1] : sl.n[0];
      const int cxy = q >= 2 * n ? (q >= 3 * n ? 3 : 2) : (q >= n ? 1 : 0), t = q - cxy * n;
      const int zf = pz ? sl.zf[1] : sl.zf[0];
      // a colour's vertices of the CTA's planes are consecutive in the global colour-blocked order too
      const float* src = V.st + size_t(cxy + 4 * pz) * (nv >> 3) + size_t(zf >> 1) * per + t;
      float a[27], f[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int o = 0; o < 27; o++) a[o] = __ldg(src + size_t(o) * nv);
      if (l == 0) {
        const int row = t / hx, i = t - row * hx, pk = row / hy, j = row - pk * hy;
        const size_t gi = (size_t(zf + 2 * pk) * V.d.ny + 2 * j + (cxy >> 1)) * V.d.nx + 2 * i + (cxy & 1);
#pragma unroll
        for (int c = 0; c < 3; c++) f[c] = __ldg(cd.f_in + c * nv + gi);
      }
      float* dst = sm + V.st_off + s;
#pragma unroll
      for (int o = 0; o < 27; o++) dst[o * V.ss] = a[o];
      sm[V.inv_off + s] = 1.0f / a[13];
      if (l == 0)
#pragma unroll
        for (int c = 0; c < 3; c++) sm[V.f_off + c * cs + s] = f[c];
    }
  }
  cluster.sync();
  for (int l = 0; l < L - 1; l++) {
    const ClLevel& F = cd.lv[l];
    for (int s = 0; s < 2 * cd.pre; s++) cl_half<false>(F, cd.f_in, sm, tab, rb, rank, s & 1, cluster);
    cl_resid(F, cd.f_in, sm, rank);
    cluster.sync();
    cl_restrict(F, cd.lv[l + 1], sm, tab, rb, rank);
    cluster.sync();
  }
  cl_coarsest(cd, sm, tab, rb, rank, cmean);
  cluster.sync();
  for (int l = L - 2; l >= 0; l--) {
    const ClLevel& F = cd.lv[l];
    cl_prolong(F, cd.lv[l + 1], sm, tab, rb, rank);
    cluster.sync();
    for (int s = 0; s < 2 * cd.post; s++) cl_half<true>(F, cd.f_in, sm, tab, rb, rank, 1 - (s & 1), cluster);
  }
  // no distributed access after the last barrier: write this CTA's planes of the correction
  {
    const ClLevel& T = cd.lv[0];
    const int pl = T.d.nx * T.d.ny, z0 = T.zstart[rank];
    const int n = (T.zstart[rank + 1] - z0) * pl;
    const size_t nv = T.d.nv();
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
      const size_t g = size_t(z0) * pl + t;
      const int zl = t / pl, rem = t - zl * pl, y = rem / T.d.nx, x = rem - y * T.d.nx;
#pragma unroll
      for (int c = 0; c < 3; c++) cd.u_out[c * nv + g] = sm[T.u_off + c * T.ucs + (zl + 1) * T.ups + y * T.urs + cl_ux(T, x)];
    }
  }
}

// Host-side layout of the cluster part for the level dimensions dims[0..n-1] (the last one is
// the coarsest). Returns the dynamic shared memory in bytes, or 0 when the levels do not fit
// one cluster (then the per-level kernels are used).
// Worst number of distinct shared-memory words per bank over the u reads of a warp: of a colour pass
// (lanes over (x/2, y/2, plane/2); row stride rs, plane stride ps), and of the
// residual's and the prolongation's natural order.
inline int cl_worst_bank(const int* addr, int n) {
  int in_bank[32][32], cnt[32] = {}, worst = 1;  // distinct words seen per bank
  for (int q = 0; q < n; q++) {
    const int b = addr[q] & 31;
    bool dup = false;
    for (int r = 0; r < cnt[b]; r++) dup = dup || in_bank[b][r] == addr[q];
    if (dup) continue;
    in_bank[b][cnt[b]++] = addr[q];
    worst = std::max(worst, cnt[b]);
  }
  return worst;
}
inline int cl_pass_conflicts(const Dims& d, int rs, int ps) {
  const int hx = d.nx / 2, hy = d.ny / 2;
  int addr[32];
  for (int t = 0; t < 32; t++) {
    const int row = t / hx, i = t % hx, k = row / hy, j = row % hy;
    addr[t] = i + 2 * j * rs + 2 * k * ps;
  }
  return cl_worst_bank(addr, 32);
}
inline int cl_row_conflicts(const Dims& d, int uh, int rs) {
  int addr[32];
  for (int t = 0; t < 32; t++) {
    const int x = t % d.nx, y = t / d.nx;
    addr[t] = ((x & 1) ? uh : 0) + (x >> 1) + y * rs;
  }
  return cl_worst_bank(addr, 32);
}

inline int cl_log2_ceil(int v) {
  int l = 0;
  while ((1 << l) < v) l++;
  return l;
}

// first_smem: the first level's stencils, right-hand side and residual also live in shared memory.
inline size_t cl_plan_try(const Dims* dims, int n, ClDesc* cd, bool first_smem) {
  if (n < 2 || n > kClMaxLevels) return 0;
  if (dims[0].nv() > size_t(kClMaxNv)) return 0;
  int off = 0, tab = 0;
  for (int l = 0; l < n; l++) {
    const Dims d = dims[l];
    ClLevel& V = cd->lv[l];
    V = ClLevel{};
    V.d = d;
    if (l < n - 1 && ((d.nx | d.ny | d.nz) & 1)) return 0;  // smoothed levels are colour-split
    if (d.nz > 0x7fff) return 0;
    int maxpl = 0;
    for (int c = 0; c <= kCl; c++) V.zstart[c] = int((long long)c * d.nz / kCl);
    for (int c = 0; c < kCl; c++) maxpl = std::max(maxpl, V.zstart[c + 1] - V.zstart[c]);
    const int plane = d.nx * d.ny;
    if (l < n - 1 && ((maxpl + 1) / 2) * (plane / 4) > kClThreads) return 0;  // a colour's lanes
    V.cs = maxpl * plane;
    V.lnx = cl_log2_ceil(d.nx);
    V.lny = cl_log2_ceil(d.ny);
    V.res8 = (maxpl << (V.lnx + V.lny)) <= kClThreads / 4;
    // u rows: the odd sites' place, row and plane strides with the fewest bank conflicts of a colour pass,
    // then of the natural order (the smallest such strides); plain on the coarsest level
    const bool smem_st = l < n - 1 && (l > 0 || first_smem);
    const int evens = (d.nx + 1) / 2;
    V.uh = evens;
    V.urs = d.nx;
    if (l < n - 1) {
      int best = INT_MAX;
      for (int rs = d.nx; rs <= d.nx + 16 && best > 9; rs++) {
        const int pass = 8 * cl_pass_conflicts(d, rs, rs * d.ny);
        for (int uh = evens; uh <= rs - d.nx / 2 && best > 9 && pass < best; uh++) {
          const int w = pass + cl_row_conflicts(d, uh, rs);
          if (w < best) {
            best = w;
            V.uh = uh;
            V.urs = rs;
          }
        }
      }
    }
    V.ups = V.urs * d.ny;
    if (l < n - 1 && plane / 4 < 32) {  // a warp spans planes
      int best = cl_pass_conflicts(d, V.urs, V.ups);
      for (int py = 1; py < 32 && best > 1; py++) {
        const int w = cl_pass_conflicts(d, V.urs, V.urs * d.ny + py);
        if (w < best) {
          best = w;
          V.ups = V.urs * d.ny + py;
        }
      }
    }
    V.ucs = (maxpl + 2) * V.ups;
    V.u_off = off;
    off += 3 * V.ucs;
    V.f_off = -1;  // the first level reads its right-hand side from global memory unless staged
    if (l > 0 || smem_st) {
      V.f_off = off;
      off += 3 * V.cs;
    }
    V.r_off = V.st_off = V.inv_off = -1;
    if (smem_st) {
      V.r_off = off;
      off += 3 * V.cs;
      V.ss = std::max(V.cs, V.cs <= kClSlots ? kClSlots : 0);
      V.st_off = off;
      off += 27 * V.ss;
      V.inv_off = off;
      off += V.cs;
    }
    V.tab_off = tab;
    tab += 3 * d.nz;
  }
  cd->nlev = n;
  cd->nc = int(dims[n - 1].nv());
  cd->gather_off = off;
  off += 3 * cd->nc;
  cd->tab_base = off;
  off += tab;
  if (tab > kClMaxTab) return 0;
  const size_t bytes = size_t(off) * sizeof(float);
  if (bytes > size_t(kMaxDynSmem)) return 0;
  return bytes;
}

// The plane tables of a plan, cd->ntab ints: per level (at tab_off) the owner CTA and local plane
// of every plane ((c << 16) | local), then for every plane the two ghost copies it feeds ((CTA <<
// 16) | local ghost plane, -1 for none): plane z is the lower ghost (local plane 0) of the CTA
// whose slab starts at z + 1 and the upper ghost (local plane slab + 1) of the CTA whose slab ends
// at z, periodically. Built once per plan on the host, copied into shared memory by every call.
inline void cl_tables(ClDesc* cd, std::vector<int>& tab) {
  int n = 0;
  for (int l = 0; l < cd->nlev; l++) n = std::max(n, cd->lv[l].tab_off + 3 * cd->lv[l].d.nz);
  tab.assign(size_t(n), 0);
  for (int l = 0; l < cd->nlev; l++) {
    const ClLevel& V = cd->lv[l];
    const int nz = V.d.nz;
    for (int z = 0; z < nz; z++) {
      int c = 0;
      while (c < kCl - 1 && z >= V.zstart[c + 1]) c++;
      tab[size_t(V.tab_off + z)] = (c << 16) | (z - V.zstart[c]);
      int k = 0;
      int* push = tab.data() + V.tab_off + nz + 2 * z;
      push[0] = push[1] = -1;
      for (int q = 0; q < kCl && k < 2; q++) {
        const int a = V.zstart[q], b = V.zstart[q + 1];
        if (b == a) continue;
        if ((a - 1 + nz) % nz == z) push[k++] = (q << 16) | 0;           // q's lower ghost
        if (k < 2 && b % nz == z) push[k++] = (q << 16) | (b - a + 1);   // q's upper ghost
      }
    }
  }
  cd->ntab = n;
}

// Host-side layout of the cluster part (see cl_plan_try): the first level's stencils in shared
// memory when everything fits, else in global memory.
inline size_t cl_plan(const Dims* dims, int n, ClDesc* cd) {
  const size_t b = cl_plan_try(dims, n, cd, true);
  return b ? b : cl_plan_try(dims, n, cd, false);
}

}  // namespace otm
