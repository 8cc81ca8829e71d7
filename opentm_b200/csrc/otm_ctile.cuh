// otm_ctile.cuh -- tile-staged Gauss-Seidel sweeps of the coarse (27-point stencil) levels.
//
// The coarse levels' smoothing (homogenization/grid.cu:707-809, eight colours per sweep) runs one
// launch per sweep instead of one launch per colour: every CTA stages the correction u (3 cases)
// of a tile of 16 x 8 x 8 vertices plus a one-site halo in shared memory, runs the eight colour
// passes of the sweep inside the tile with the halo held at the values it had when the sweep
// started, and writes the interior to a second buffer. As on the fine level, consecutive sweeps
// alternate between two tilings shifted by half a tile along every axis, so that the faces of one
// tiling lie inside the tiles of the other, and the post-smoothing sweeps run in the reverse colour
// order on the mirrored tilings (the V-cycle stays symmetric for PCG). The first sweep after the
// coarse-grid correction adds the trilinear prolongation of the next coarser level's correction
// while it stages the tile.
//
// One thread per vertex of the current colour (8 x 4 x 4 per tile): it reads the 27 stencil
// coefficients of its vertex from the level's colour-blocked stencil array in global memory (lanes
// of a warp read consecutive entries), the 26 neighbours from shared memory, and the right-hand side
// from global memory. The staged sites are float4 {u_case0, u_case1, u_case2, 0} with the even and
// the odd sites of a row stored apart and rows padded to 19 entries, so that the lanes of a warp,
// which update every other site of a row, read consecutive entries.
#pragma once

#include "otm_tile.cuh"

namespace otm {

constexpr int kCTX = 16, kCTY = 8, kCTZ = 8;                      // interior vertices of a coarse tile
constexpr int kCSX = kCTX + 2, kCSY = kCTY + 2, kCSZ = kCTZ + 2;  // staged sites
constexpr int kCSHalf = kCSX / 2;
constexpr int kCSRow = kCSX + 1;                                  // padded row pitch (float4)
constexpr int kCSPlane = kCSRow * kCSY;                           // 190
constexpr int kCSSites = kCSPlane * kCSZ;                         // 1900
constexpr int kCThreads = (kCTX / 2) * (kCTY / 2) * (kCTZ / 2);   // 128: one per vertex of a colour
constexpr int kCCX = kCTX / 2 + 2, kCCY = kCTY / 2 + 2, kCCZ = kCTZ / 2 + 2;  // coarser block (10 x 6 x 6)
constexpr int kCCSites = kCCX * kCCY * kCCZ;
constexpr size_t kCTileSmem = size_t(kCSSites) * sizeof(float4);                               // 30,400 B
constexpr size_t kCTileSmemProlong = kCTileSmem + size_t(kCCSites) * sizeof(float4);            // 36,160 B

// Whether a coarse level can be tiled.
__host__ __device__ inline bool ctile_fits(const Dims& d) {
  return d.nx % kCTX == 0 && d.ny % kCTY == 0 && d.nz % kCTZ == 0;
}
__host__ __device__ inline unsigned ctile_count(const Dims& d) {
  return unsigned(d.nx / kCTX) * unsigned(d.ny / kCTY) * unsigned(d.nz / kCTZ);
}

__device__ __forceinline__ int csite(int lx, int ly, int lz) {
  return lz * kCSPlane + ly * kCSRow + ((lx & 1) ? kCSHalf + (lx >> 1) : (lx >> 1));
}

// Origin of coarse tile b of tiling `shift` (unwrapped, as tile_origin).
__device__ __forceinline__ void ctile_origin(const Dims& d, unsigned b, int shift, int& x0, int& y0, int& z0) {
  const unsigned ntx = unsigned(d.nx / kCTX), nty = unsigned(d.ny / kCTY);
  const unsigned q = b / ntx;
  x0 = int(b - q * ntx) * kCTX + shift * (kCTX / 2);
  y0 = int(q % nty) * kCTY + shift * (kCTY / 2);
  z0 = int(q / nty) * kCTZ + shift * (kCTZ / 2);
}

// Trilinear prolongation at the fine site (ux, uy, uz) (unwrapped) from the staged coarser block
// (float4 per site, origin c0); the expression and weights of prolong_body.
__device__ __forceinline__ float3 cprolong_site(const float4* cb, int ux, int uy, int uz, int c0x, int c0y, int c0z) {
  const int ax0 = (ux >> 1) - c0x, ay0 = (uy >> 1) - c0y, az0 = (uz >> 1) - c0z;
  const int ax1 = ax0 + (ux & 1), ay1 = ay0 + (uy & 1), az1 = az0 + (uz & 1);
  const float wx1 = (ux & 1) ? 0.5f : 0.f, wy1 = (uy & 1) ? 0.5f : 0.f, wz1 = (uz & 1) ? 0.5f : 0.f;
  const float wx0 = 1.f - wx1, wy0 = 1.f - wy1, wz0 = 1.f - wz1;
  const float4* r00 = cb + (ay0 + kCCY * az0) * kCCX;
  const float4* r10 = cb + (ay1 + kCCY * az0) * kCCX;
  const float4* r01 = cb + (ay0 + kCCY * az1) * kCCX;
  const float4* r11 = cb + (ay1 + kCCY * az1) * kCCX;
  const float4 a00 = r00[ax0], b00 = r00[ax1], a10 = r10[ax0], b10 = r10[ax1];
  const float4 a01 = r01[ax0], b01 = r01[ax1], a11 = r11[ax0], b11 = r11[ax1];
  float3 o;
  o.x = wz0 * (wy0 * (wx0 * a00.x + wx1 * b00.x) + wy1 * (wx0 * a10.x + wx1 * b10.x)) +
        wz1 * (wy0 * (wx0 * a01.x + wx1 * b01.x) + wy1 * (wx0 * a11.x + wx1 * b11.x));
  o.y = wz0 * (wy0 * (wx0 * a00.y + wx1 * b00.y) + wy1 * (wx0 * a10.y + wx1 * b10.y)) +
        wz1 * (wy0 * (wx0 * a01.y + wx1 * b01.y) + wy1 * (wx0 * a11.y + wx1 * b11.y));
  o.z = wz0 * (wy0 * (wx0 * a00.z + wx1 * b00.z) + wy1 * (wx0 * a10.z + wx1 * b10.z)) +
        wz1 * (wy0 * (wx0 * a01.z + wx1 * b01.z) + wy1 * (wx0 * a11.z + wx1 * b11.z));
  return o;
}

// One colour pass over the tile: the thread's vertex of colour (CX, CY, CZ).
// The operands of this thread's vertex in colour pass (CX, CY, CZ) that do not depend on u: its
// 27 stencil values and its right-hand side. They are fetched one pass ahead (while the previous
// pass computes), so the passes wait on shared memory only, not on L2.
struct CPassOps {
  float s[27];
  float f[3];
};

template <int CX, int CY, int CZ>
__device__ __forceinline__ void ctile_fetch(const Dims& d, int x0, int y0, int z0, const float* __restrict__ st,
                                            const float* __restrict__ f, CPassOps& ops) {
  const int t = int(threadIdx.x);
  const int i = t & 7, j = (t >> 3) & 3, k = t >> 5;
  const int lx = 1 + 2 * i + CX, ly = 1 + 2 * j + CY, lz = 1 + 2 * k + CZ;
  const int X = wrapm(x0 + lx - 1, d.nx), Y = wrapm(y0 + ly - 1, d.ny), Z = wrapm(z0 + lz - 1, d.nz);
  const size_t nv = d.nv();
  const size_t v = size_t(X) + size_t(d.nx) * (size_t(Y) + size_t(d.ny) * Z);
  const size_t sb = cb_index(d, X, Y, Z);
#pragma unroll
  for (int o = 0; o < 27; o++) ops.s[o] = __ldg(st + size_t(o) * nv + sb);
#pragma unroll
  for (int c = 0; c < 3; c++) ops.f[c] = __ldg(f + c * nv + v);
}

// One colour pass (CX, CY, CZ) of the tile's interior from fetched operands: each thread updates
// one vertex (128 threads: 8 x 4 x 4 vertices of the colour in the 16 x 8 x 8 tile).
template <int CX, int CY, int CZ>
__device__ __forceinline__ void ctile_apply(float4* sm, const CPassOps& ops) {
  const int t = int(threadIdx.x);
  const int i = t & 7, j = (t >> 3) & 3, k = t >> 5;
  const int lx = 1 + 2 * i + CX, ly = 1 + 2 * j + CY, lz = 1 + 2 * k + CZ;
  float acc[3] = {ops.f[0], ops.f[1], ops.f[2]};
  const float4* b = sm + csite(lx, ly, lz);
  // neighbour offsets: the parity of lx is fixed by the pass, so left / right are compile-time
  constexpr int oL = (CX == 0) ? -kCSHalf : kCSHalf - 1;  // lx odd for CX = 0
  constexpr int oR = (CX == 0) ? -kCSHalf + 1 : kCSHalf;
#pragma unroll
  for (int o = 0; o < 27; o++) {
    if (o == 13) continue;
    const int ox = o % 3 - 1, oy = (o / 3) % 3 - 1, oz = o / 9 - 1;
    const int off = (ox < 0 ? oL : (ox > 0 ? oR : 0)) + oy * kCSRow + oz * kCSPlane;
    const float4 n = b[off];
    acc[0] -= ops.s[o] * n.x;
    acc[1] -= ops.s[o] * n.y;
    acc[2] -= ops.s[o] * n.z;
  }
  const float inv = 1.0f / ops.s[13];
  sm[csite(lx, ly, lz)] = make_float4(acc[0] * inv, acc[1] * inv, acc[2] * inv, 0.f);
}

// Colour pass A from its fetched operands, with the operands of the next pass B fetched first.
// No barrier here: the caller separates the passes.
template <int AX, int AY, int AZ, int BX, int BY, int BZ>
__device__ __forceinline__ void ctile_step(float4* sm, const Dims& d, int x0, int y0, int z0,
                                           const float* __restrict__ st, const float* __restrict__ f,
                                           const CPassOps& cur, CPassOps& next) {
  ctile_fetch<BX, BY, BZ>(d, x0, y0, z0, st, f, next);
  ctile_apply<AX, AY, AZ>(sm, cur);
}

// One Gauss-Seidel sweep of a coarse level on the tiles of tiling `shift`: stage u from zero, from
// u_in, or from u_in plus the prolongation of the coarser correction uc (kStart as TileStart), run
// the eight colour passes in the order 0..7 (7..0 when `reverse`), write the interior to u_out
// (which must not alias u_in). st: the level's 27-point stencils (colour-blocked), f: its
// right-hand side, all FP32, 3 cases.
template <int kStart>
__global__ void __launch_bounds__(kCThreads)
    k_ctile_sweep(Dims d, Dims dc, const float* __restrict__ st, const float* __restrict__ u_in,
                  const float* __restrict__ uc, float* __restrict__ u_out, const float* __restrict__ f, int shift,
                  int reverse, const SolveScalars* sc) {
  extern __shared__ float4 csm[];
  float4* cb = csm + kCSSites;
  pdl_wait();
  if (sc && solve_done(sc)) return;
  int x0, y0, z0;
  ctile_origin(d, blockIdx.x, shift, x0, y0, z0);
  const size_t nv = d.nv();
  const int t = int(threadIdx.x);
  // the first pass's stencils and right-hand side, in flight during the staging
  CPassOps first;
  if (!reverse)
    ctile_fetch<0, 0, 0>(d, x0, y0, z0, st, f, first);
  else
    ctile_fetch<1, 1, 1>(d, x0, y0, z0, st, f, first);
  const int c0x = x0 / 2 - 1, c0y = y0 / 2 - 1, c0z = z0 / 2 - 1;
  // staging: every thread first issues all its global loads (the coarser block, then the sites of
  // the staged box in natural order), then stores
  constexpr int kSI = (kCSX * kCSY * kCSZ + kCThreads - 1) / kCThreads;
  constexpr int kCI = (kCCSites + kCThreads - 1) / kCThreads;
  float cbv[kStart == kFromUProlong ? kCI : 1][3];
  if (kStart == kFromUProlong) {
    const size_t nvc = dc.nv();
#pragma unroll
    for (int it = 0; it < kCI; it++) {
      const int q = t + it * kCThreads;
      if (q < kCCSites) {
        const int ax = q % kCCX, ay = (q / kCCX) % kCCY, az = q / (kCCX * kCCY);
        const int X = wrapm(c0x + ax, dc.nx), Y = wrapm(c0y + ay, dc.ny), Z = wrapm(c0z + az, dc.nz);
        const size_t g = size_t(X) + size_t(dc.nx) * (size_t(Y) + size_t(dc.ny) * Z);
#pragma unroll
        for (int c = 0; c < 3; c++) cbv[it][c] = __ldg(uc + c * nvc + g);
      }
    }
  }
  float uv[kStart != kFromZero ? kSI : 1][3];
  if (kStart != kFromZero) {
#pragma unroll
    for (int it = 0; it < kSI; it++) {
      const int q = t + it * kCThreads;
      if (q < kCSX * kCSY * kCSZ) {
        const int lx = q % kCSX, ly = (q / kCSX) % kCSY, lz = q / (kCSX * kCSY);
        const size_t g = size_t(wrapm(x0 - 1 + lx, d.nx)) +
                         size_t(d.nx) * (size_t(wrapm(y0 - 1 + ly, d.ny)) + size_t(d.ny) * wrapm(z0 - 1 + lz, d.nz));
#pragma unroll
        for (int c = 0; c < 3; c++) uv[it][c] = __ldg(u_in + c * nv + g);
      }
    }
  }
  if (kStart == kFromUProlong) {
#pragma unroll
    for (int it = 0; it < kCI; it++) {
      const int q = t + it * kCThreads;
      if (q < kCCSites) cb[q] = make_float4(cbv[it][0], cbv[it][1], cbv[it][2], 0.f);
    }
    __syncthreads();
  }
#pragma unroll
  for (int it = 0; it < kSI; it++) {
    const int q = t + it * kCThreads;
    if (q < kCSX * kCSY * kCSZ) {
      const int lx = q % kCSX, ly = (q / kCSX) % kCSY, lz = q / (kCSX * kCSY);
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (kStart != kFromZero) {
        v.x = uv[it][0];
        v.y = uv[it][1];
        v.z = uv[it][2];
        if (kStart == kFromUProlong) {
          const float3 p = cprolong_site(cb, x0 - 1 + lx, y0 - 1 + ly, z0 - 1 + lz, c0x, c0y, c0z);
          v.x += p.x;
          v.y += p.y;
          v.z += p.z;
        }
      }
      csm[csite(lx, ly, lz)] = v;
    }
  }
  __syncthreads();
  CPassOps oa, ob;
  if (!reverse) {
    ctile_step<0, 0, 0, 1, 0, 0>(csm, d, x0, y0, z0, st, f, first, ob);
    __syncthreads();
    ctile_step<1, 0, 0, 0, 1, 0>(csm, d, x0, y0, z0, st, f, ob, oa);
    __syncthreads();
    ctile_step<0, 1, 0, 1, 1, 0>(csm, d, x0, y0, z0, st, f, oa, ob);
    __syncthreads();
    ctile_step<1, 1, 0, 0, 0, 1>(csm, d, x0, y0, z0, st, f, ob, oa);
    __syncthreads();
    ctile_step<0, 0, 1, 1, 0, 1>(csm, d, x0, y0, z0, st, f, oa, ob);
    __syncthreads();
    ctile_step<1, 0, 1, 0, 1, 1>(csm, d, x0, y0, z0, st, f, ob, oa);
    __syncthreads();
    ctile_step<0, 1, 1, 1, 1, 1>(csm, d, x0, y0, z0, st, f, oa, ob);
    __syncthreads();
    ctile_apply<1, 1, 1>(csm, ob);
  } else {
    ctile_step<1, 1, 1, 0, 1, 1>(csm, d, x0, y0, z0, st, f, first, ob);
    __syncthreads();
    ctile_step<0, 1, 1, 1, 0, 1>(csm, d, x0, y0, z0, st, f, ob, oa);
    __syncthreads();
    ctile_step<1, 0, 1, 0, 0, 1>(csm, d, x0, y0, z0, st, f, oa, ob);
    __syncthreads();
    ctile_step<0, 0, 1, 1, 1, 0>(csm, d, x0, y0, z0, st, f, ob, oa);
    __syncthreads();
    ctile_step<1, 1, 0, 0, 1, 0>(csm, d, x0, y0, z0, st, f, oa, ob);
    __syncthreads();
    ctile_step<0, 1, 0, 1, 0, 0>(csm, d, x0, y0, z0, st, f, ob, oa);
    __syncthreads();
    ctile_step<1, 0, 0, 0, 0, 0>(csm, d, x0, y0, z0, st, f, oa, ob);
    __syncthreads();
    ctile_apply<0, 0, 0>(csm, ob);
  }
  __syncthreads();
  for (int s = t; s < kCTX * kCTY * kCTZ; s += kCThreads) {
    const int lx = 1 + s % kCTX, ly = 1 + (s / kCTX) % kCTY, lz = 1 + s / (kCTX * kCTY);
    const float4 o = csm[csite(lx, ly, lz)];
    const size_t g = size_t(wrapm(x0 + lx - 1, d.nx)) +
                     size_t(d.nx) * (size_t(wrapm(y0 + ly - 1, d.ny)) + size_t(d.ny) * wrapm(z0 + lz - 1, d.nz));
    u_out[g] = o.x;
    u_out[nv + g] = o.y;
    u_out[2 * nv + g] = o.z;
  }
}

// ---- few tiles: stencils in shared memory, a lane per vertex and load case --------------------------
// With at most one tile per SM the sweep above is bound by the length of a warp's instruction chain (one
// warp per scheduler stages 14 sites and takes eight passes of three cases) and by eight L2 latencies. Here
// a CTA has 384 threads, one per vertex of a colour and load case; it first starts the copies of the
// stencils of all eight colours (108 KB, cp.async of 16 bytes: a row of 8 vertices of a colour is 32
// contiguous bytes of the colour-blocked array, in two halves because a shifted tile may wrap between
// them), one group per colour in the order of the passes, and the staging of u and the earlier passes run
// while they land. The sites are kept case by case with rows of 20 words, even and odd sites apart: the
// lanes of a pass (8 sites of 4 rows two apart) read 32 different banks. Arithmetic and order are those of
// k_ctile_sweep.
// The four sweeps of a 32^3 level (32 tiles; from zero, from u, prolonging, reverse): 64.6 -> 47.7 us. Its
// shared memory leaves one CTA per SM, so the line is at one tile per SM: a 64^3 level (256 tiles) takes
// 91 us this way, as two rounds of CTAs, and 64 with k_ctile_sweep.
constexpr int kCSmallThreads = 3 * kCThreads;
constexpr int kCSmallRow = 20, kCSmallPlane = kCSmallRow * kCSY, kCSmallCase = kCSmallPlane * kCSZ;  // 2000 floats
constexpr int kCSmallStencils = 8 * 27 * kCThreads;
constexpr size_t kCSmallSmem = size_t(kCSmallStencils + 3 * kCSmallCase) * sizeof(float);  // 134,592 B
constexpr size_t kCSmallSmemProlong = kCSmallSmem + size_t(3 * kCCSites) * sizeof(float);
constexpr unsigned kCSmallTiles = 148;

__device__ __forceinline__ int cspos(int lx, int ly, int lz) {
  return lz * kCSmallPlane + ly * kCSmallRow + ((lx & 1) ? kCSHalf + (lx >> 1) : (lx >> 1));
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

// Pass number P of the sweep: the lane's vertex (i, j, k) of the pass's colour, case plane u of the sites,
// stencils at st (27 x 128 per colour), its right-hand side f. Waits for its colour's copies.
template <int P, bool kReverse>
__device__ __forceinline__ void ctile_small_pass(float* u, const float* st, float f, int i, int j, int k) {
  constexpr int C = kReverse ? 7 - P : P, CX = C & 1, CY = (C >> 1) & 1, CZ = C >> 2;
  constexpr int oL = (CX == 0) ? -kCSHalf : kCSHalf - 1, oR = (CX == 0) ? -kCSHalf + 1 : kCSHalf;
  asm volatile("cp.async.wait_group %0;" ::"n"(7 - P) : "memory");
  __syncthreads();  // the copies of every thread, and the previous pass
  const float* sp = st + C * 27 * kCThreads + i + 8 * j + 32 * k;
  float* b = u + cspos(1 + 2 * i + CX, 1 + 2 * j + CY, 1 + 2 * k + CZ);
  float acc = f;
#pragma unroll
  for (int o = 0; o < 27; o++) {
    if (o == 13) continue;
    const int ox = o % 3 - 1, oy = (o / 3) % 3 - 1, oz = o / 9 - 1;
    acc -= sp[o * kCThreads] * b[(ox < 0 ? oL : (ox > 0 ? oR : 0)) + oy * kCSmallRow + oz * kCSmallPlane];
  }
  *b = acc * (1.0f / sp[13 * kCThreads]);
}

template <int kStart, bool kReverse>
__global__ void __launch_bounds__(kCSmallThreads, 1)
    k_ctile_sweep_small(Dims d, Dims dc, const float* __restrict__ st, const float* __restrict__ u_in,
                        const float* __restrict__ uc, float* __restrict__ u_out, const float* __restrict__ f, int shift,
                        const SolveScalars* sc) {
  extern __shared__ float4 csm_small[];
  float* st_sm = reinterpret_cast<float*>(csm_small);
  float* sites = st_sm + kCSmallStencils;
  float* cb = sites + 3 * kCSmallCase;
  const int t = int(threadIdx.x), warp = t >> 5, lane = t & 31;
  int x0, y0, z0;
  ctile_origin(d, blockIdx.x, shift, x0, y0, z0);
  const size_t nv = d.nv(), nsub = nv >> 3;
  pdl_wait();
  if (sc && solve_done(sc)) return;
  {
    // lane: row r = j + 4 k of a colour's 8 x 4 x 4 vertices and half h of the row; the 12 warps take the
    // (pass, offset) pairs q = 27 p + o in turn
    const int h = lane & 1, r = lane >> 1;
    const int hx = d.nx >> 1, hy = d.ny >> 1, hz = d.nz >> 1;
    const int X = wrapm(x0 / 2 + 4 * h, hx), Y = wrapm(y0 / 2 + (r & 3), hy), Z = wrapm(z0 / 2 + (r >> 2), hz);
    const float* src = st + (size_t(X) + size_t(hx) * (size_t(Y) + size_t(hy) * Z));
    float* dst = st_sm + r * 8 + h * 4;
    int q = warp;
#pragma unroll
    for (int p = 0; p < 8; p++) {
      const int c = kReverse ? 7 - p : p;
#pragma unroll
      for (int e = 0; e < 3; e++)
        if (q < 27 * (p + 1)) {
          const int o = q - 27 * p;
          cp_async16(dst + (c * 27 + o) * kCThreads, src + size_t(o) * nv + c * nsub);
          q += kCSmallThreads / 32;
        }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
  }
  // this lane's vertex (i, j, k) of a colour and its case; its right-hand side of every colour
  const int i = lane & 7, j = lane >> 3, k = warp & 3, cs = warp >> 2;
  float fr[8];
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const int X = wrapm(x0 + 2 * i + (c & 1), d.nx), Y = wrapm(y0 + 2 * j + ((c >> 1) & 1), d.ny),
              Z = wrapm(z0 + 2 * k + (c >> 2), d.nz);
    fr[c] = __ldg(f + cs * nv + size_t(X) + size_t(d.nx) * (size_t(Y) + size_t(d.ny) * Z));
  }
  // staging: all loads first, then the prolongation and the stores
  constexpr int kSites = kCSX * kCSY * kCSZ, kItems = 3 * kSites, kSI = (kItems + kCSmallThreads - 1) / kCSmallThreads;
  constexpr int kCI = (3 * kCCSites + kCSmallThreads - 1) / kCSmallThreads;
  const int c0x = x0 / 2 - 1, c0y = y0 / 2 - 1, c0z = z0 / 2 - 1;
  float uv[kSI];
  if (kStart == kFromUProlong) {
    const size_t nvc = dc.nv();
    float cv[kCI];
#pragma unroll
    for (int it = 0; it < kCI; it++) {
      const int q = t + it * kCSmallThreads, c = q / kCCSites, s = q - c * kCCSites;
      const int ax = s % kCCX, ay = (s / kCCX) % kCCY, az = s / (kCCX * kCCY);
      const int X = wrapm(c0x + ax, dc.nx), Y = wrapm(c0y + ay, dc.ny), Z = wrapm(c0z + az, dc.nz);
      if (q < 3 * kCCSites) cv[it] = __ldg(uc + c * nvc + size_t(X) + size_t(dc.nx) * (size_t(Y) + size_t(dc.ny) * Z));
    }
#pragma unroll
    for (int it = 0; it < kCI; it++) {
      const int q = t + it * kCSmallThreads;
      if (q < 3 * kCCSites) cb[q] = cv[it];
    }
  }
#pragma unroll
  for (int it = 0; it < kSI; it++) {
    const int q = t + it * kCSmallThreads, c = q / kSites, s = q - c * kSites;
    const int lx = s % kCSX, ly = (s / kCSX) % kCSY, lz = s / (kCSX * kCSY);
    const size_t g = size_t(wrapm(x0 - 1 + lx, d.nx)) +
                     size_t(d.nx) * (size_t(wrapm(y0 - 1 + ly, d.ny)) + size_t(d.ny) * wrapm(z0 - 1 + lz, d.nz));
    uv[it] = kStart != kFromZero && q < kItems ? __ldg(u_in + c * nv + g) : 0.f;
  }
  if (kStart == kFromUProlong) __syncthreads();  // the coarser block
#pragma unroll
  for (int it = 0; it < kSI; it++) {
    const int q = t + it * kCSmallThreads, c = q / kSites, s = q - c * kSites;
    if (q >= kItems) continue;
    const int lx = s % kCSX, ly = (s / kCSX) % kCSY, lz = s / (kCSX * kCSY);
    float v = uv[it];
    if (kStart == kFromUProlong) {
      // the expression and weights of cprolong_site, one case
      const int ux = x0 - 1 + lx, uy = y0 - 1 + ly, uz = z0 - 1 + lz;
      const int ax0 = (ux >> 1) - c0x, ay0 = (uy >> 1) - c0y, az0 = (uz >> 1) - c0z;
      const int ax1 = ax0 + (ux & 1), ay1 = ay0 + (uy & 1), az1 = az0 + (uz & 1);
      const float wx1 = (ux & 1) ? 0.5f : 0.f, wy1 = (uy & 1) ? 0.5f : 0.f, wz1 = (uz & 1) ? 0.5f : 0.f;
      const float wx0 = 1.f - wx1, wy0 = 1.f - wy1, wz0 = 1.f - wz1;
      const float* b = cb + c * kCCSites;
      const float* r00 = b + (ay0 + kCCY * az0) * kCCX;
      const float* r10 = b + (ay1 + kCCY * az0) * kCCX;
      const float* r01 = b + (ay0 + kCCY * az1) * kCCX;
      const float* r11 = b + (ay1 + kCCY * az1) * kCCX;
      v += wz0 * (wy0 * (wx0 * r00[ax0] + wx1 * r00[ax1]) + wy1 * (wx0 * r10[ax0] + wx1 * r10[ax1])) +
           wz1 * (wy0 * (wx0 * r01[ax0] + wx1 * r01[ax1]) + wy1 * (wx0 * r11[ax0] + wx1 * r11[ax1]));
    }
    sites[c * kCSmallCase + cspos(lx, ly, lz)] = v;
  }
  float* u = sites + cs * kCSmallCase;
  ctile_small_pass<0, kReverse>(u, st_sm, fr[kReverse ? 7 : 0], i, j, k);
  ctile_small_pass<1, kReverse>(u, st_sm, fr[kReverse ? 6 : 1], i, j, k);
  ctile_small_pass<2, kReverse>(u, st_sm, fr[kReverse ? 5 : 2], i, j, k);
  ctile_small_pass<3, kReverse>(u, st_sm, fr[kReverse ? 4 : 3], i, j, k);
  ctile_small_pass<4, kReverse>(u, st_sm, fr[kReverse ? 3 : 4], i, j, k);
  ctile_small_pass<5, kReverse>(u, st_sm, fr[kReverse ? 2 : 5], i, j, k);
  ctile_small_pass<6, kReverse>(u, st_sm, fr[kReverse ? 1 : 6], i, j, k);
  ctile_small_pass<7, kReverse>(u, st_sm, fr[kReverse ? 0 : 7], i, j, k);
  __syncthreads();
#pragma unroll
  for (int it = 0; it < kCTX * kCTY * kCTZ / kCThreads; it++) {
    const int s = (t - cs * kCThreads) + it * kCThreads;  // the lane's case
    const int lx = 1 + s % kCTX, ly = 1 + (s / kCTX) % kCTY, lz = 1 + s / (kCTX * kCTY);
    u_out[cs * nv + size_t(wrapm(x0 + lx - 1, d.nx)) +
          size_t(d.nx) * (size_t(wrapm(y0 + ly - 1, d.ny)) + size_t(d.ny) * wrapm(z0 + lz - 1, d.nz))] =
        u[cspos(lx, ly, lz)];
  }
}

}  // namespace otm
