// otm_tile.cuh -- tile-staged fine-level smoother and residual (sm_100a).
//
// The fine level's Gauss-Seidel smoothing runs one launch per sweep instead of one launch per
// colour pair: every CTA stages a tile of 16 x 16 x 8 vertices plus a one-site halo in shared
// memory, as one float4 per site {u_case0, u_case1, u_case2, k_e} (k_e the conductivity of the
// element whose lower corner is the site), runs the four colour-pair passes of the sweep inside
// the tile with the halo held at the values it had when the sweep started, and writes the tile's
// interior to a second buffer (so that no tile reads a halo another tile has already overwritten).
// Inside a tile this is the colour-ordered Gauss-Seidel sweep of the reference smoother
// (homogenization/grid.cu:318-471, colours in the order 0,4,1,5,2,6,3,7, the pairs (cx,cy,0) /
// (cx,cy,1) updated together because the cube element couples no vertices one edge apart); across
// tile faces it is block Jacobi. Block Jacobi alone leaves the error that is constant inside each
// tile and alternates in sign from tile to tile nearly undamped, so consecutive sweeps alternate
// between two tilings, the second shifted by half a tile along every axis: the faces of one
// tiling lie inside the tiles of the other. The first sweep after the coarse-grid correction adds the
// trilinear prolongation P u_c while it stages the tile. Pre-smoothing runs forward with the
// tilings 0, 1, 0, ..., post-smoothing in the reverse pair order with the tilings mirrored, so the
// V-cycle stays symmetric (the post leg is the transpose of the pre leg), as PCG needs.
//
// Shared-memory layout of the sites: site (lx, ly, lz), lx, ly in [0, 18), lz in [0, 10), lies at
// lz * 342 + ly * 19 + (lx odd ? 9 + lx / 2 : lx / 2): within a row the even and the odd sites are
// stored apart, so that the 8 lanes that update every other site of a row read 8 consecutive
// float4, and rows are padded to 19 float4 so that the rows two apart, which the other lanes of a
// warp read, start in other banks.
//
// A thread owns a block of 2 x 2 x 4 vertices and keeps its values and conductivities in registers; in
// the pass of colour pair (cx, cy) it updates the 4 vertices of one of its four columns, streaming the
// 6 planes around them: of the 8 neighbour columns 3 are its own, so a plane costs 5 shared-memory
// loads (8 in the two planes above and below the block). Every plane is read once and added to the
// three vertices it couples to (the one above, the one in the plane, the one below). The right-hand
// side is read from global memory into registers, two columns at a time, ahead of their passes, and
// the results are written to global memory from registers. The sweep is bound by latency at 12 warps per
// SM and by the shared-memory pipe; the registers take it from 54 site loads and 12 right-hand-side
// loads per thread and pass to 37 site loads (7.9 -> 3.5 M shared-memory wavefronts per launch at 128^3)
// and free the shared memory of a third CTA per SM.
#pragma once

#include "otm_mg_kernels.cuh"

namespace otm {

constexpr int kTX = 16, kTY = 16, kTZ = 8;                    // interior vertices of a tile
constexpr int kSX = kTX + 2, kSY = kTY + 2, kSZ = kTZ + 2;    // staged sites (one halo site each side)
constexpr int kSHalf = kSX / 2;                               // sites of one parity in a row
constexpr int kSRow = kSX + 1;                                // row pitch in float4 (padded)
constexpr int kSPlane = kSRow * kSY;                          // 342
constexpr int kSSites = kSPlane * kSZ;                        // 3420
constexpr int kSmoothThreads = 128;                           // 8 x 8 pair columns x 2 segments
constexpr int kResidThreads = 256;                            // one thread per column
constexpr int kSeg = 4;                                       // vertices per thread and pass
constexpr int kCX = kTX / 2 + 2, kCY = kTY / 2 + 2, kCZ = kTZ / 2 + 2;  // staged coarse sites
constexpr int kCSites = kCX * kCY * kCZ;                      // 600
static_assert((kTX / 2) * (kTY / 2) * (kTZ / kSeg) == kSmoothThreads, "one thread per column segment");
static_assert(kTX * kTY == kResidThreads, "one thread per column");

// Dynamic shared memory: [sites][coarse block (prolonging sweep)].
constexpr size_t kTileSmem = size_t(kSSites) * sizeof(float4);                        // 54,720 B
constexpr size_t kTileSmemProlong = kTileSmem + size_t(kCSites) * sizeof(float4);      // 64,320 B

// Whether a level's dimensions can be tiled.
__host__ __device__ inline bool tile_fits(const Dims& d) {
  return d.nx % kTX == 0 && d.ny % kTY == 0 && d.nz % kTZ == 0;
}
__host__ __device__ inline unsigned tile_count(const Dims& d) {
  return unsigned(d.nx / kTX) * unsigned(d.ny / kTY) * unsigned(d.nz / kTZ);
}

__device__ __forceinline__ int tsite(int lx, int ly, int lz) {
  return lz * kSPlane + ly * kSRow + ((lx & 1) ? kSHalf + (lx >> 1) : (lx >> 1));
}
__device__ __forceinline__ int rsite(int lx, int ly, int lz) { return lz * kSPlane + ly * kSRow + lx; }

// Origin (x0, y0, z0) of tile b of tiling `shift` (0: tiles at multiples of the tile size; 1:
// shifted by half a tile along every axis, so the last tile of a row wraps around the periodic
// cell). Tiles are ordered x fastest so that neighbouring CTAs share halos. The origin is not
// wrapped: global indices of the tile's sites are.
__device__ __forceinline__ void tile_origin(const Dims& d, unsigned b, int shift, int& x0, int& y0, int& z0) {
  const unsigned ntx = unsigned(d.nx / kTX), nty = unsigned(d.ny / kTY);
  const unsigned q = b / ntx;
  x0 = int(b - q * ntx) * kTX + shift * (kTX / 2);
  y0 = int(q % nty) * kTY + shift * (kTY / 2);
  z0 = int(q / nty) * kTZ + shift * (kTZ / 2);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- vector loads and stores of consecutive values in the storage types --------------------
__device__ __forceinline__ void ld4(const float* p, float (&v)[4]) {
  const float4 q = __ldg(reinterpret_cast<const float4*>(p));
  v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
}
__device__ __forceinline__ void ld4(const __nv_bfloat16* p, float (&v)[4]) {
  const uint2 q = __ldg(reinterpret_cast<const uint2*>(p));
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&q.x);
  const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&q.y);
  v[0] = __low2float(a), v[1] = __high2float(a), v[2] = __low2float(b), v[3] = __high2float(b);
}
__device__ __forceinline__ void ld4(const __half* p, float (&v)[4]) {
  const uint2 q = __ldg(reinterpret_cast<const uint2*>(p));
  const __half2 a = *reinterpret_cast<const __half2*>(&q.x);
  const __half2 b = *reinterpret_cast<const __half2*>(&q.y);
  v[0] = __low2float(a), v[1] = __high2float(a), v[2] = __low2float(b), v[3] = __high2float(b);
}

// 2 consecutive values (8 bytes in FP32, 4 bytes in 16-bit storage)
__device__ __forceinline__ void st2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void st2(__nv_bfloat16* p, float a, float b) {
  *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
}
__device__ __forceinline__ void st2(__half* p, float a, float b) {
  *reinterpret_cast<__half2*>(p) = __floats2half2_rn(a, b);
}

// ---- coefficients ------------------------------------------------------------------------------
// Coefficients of the 8 neighbour columns of a vertex for one element plane, from the 4
// conductivities K[b] (b = bx + 2 by: the element whose lower corner is (x - 1 + bx, y - 1 + by)
// in that plane). Neighbour n: 0 (-1,-1) 1 (0,-1) 2 (+1,-1) 3 (-1,0) 4 (+1,0) 5 (-1,+1) 6 (0,+1)
// 7 (+1,+1). Corners couple through one element of the plane (c3, three axes apart), the four
// edge neighbours through two (c2, two axes apart): A(v, v+o) = c[|o|_0] * sum of the
// conductivities of the elements holding both vertices.
struct PlaneCoef {
  float w[8];
  __device__ __forceinline__ void make(const float (&K)[4], const FineOp& op) {
    w[0] = op.c3 * K[0];
    w[1] = op.c2 * (K[0] + K[1]);
    w[2] = op.c3 * K[1];
    w[3] = op.c2 * (K[0] + K[2]);
    w[4] = op.c2 * (K[1] + K[3]);
    w[5] = op.c3 * K[2];
    w[6] = op.c2 * (K[2] + K[3]);
    w[7] = op.c3 * K[3];
  }
};

// acc -= sum_n w[n] * nb[n] (3 cases)
__device__ __forceinline__ void sub_plane(float (&acc)[3], const PlaneCoef& c, const float4 (&nb)[8]) {
#pragma unroll
  for (int n = 0; n < 8; n++) {
    acc[0] -= c.w[n] * nb[n].x;
    acc[1] -= c.w[n] * nb[n].y;
    acc[2] -= c.w[n] * nb[n].z;
  }
}

// in-plane corners of the vertex in the plane: c2 * (K_below + K_above) per corner
__device__ __forceinline__ void sub_inplane(float (&acc)[3], const float (&Kb)[4], const float (&Ka)[4],
                                            const FineOp& op, const float4 (&nb)[8]) {
  const int cn[4] = {0, 2, 5, 7};
#pragma unroll
  for (int b = 0; b < 4; b++) {
    const float w = op.c2 * (Kb[b] + Ka[b]);
    acc[0] -= w * nb[cn[b]].x;
    acc[1] -= w * nb[cn[b]].y;
    acc[2] -= w * nb[cn[b]].z;
  }
}

// The block of vertices a thread owns: column PX + 2 PY, plane q.
struct TileBlock {
  float u[4][kSeg][3];
  float k[4][kSeg];
};

// The right-hand side of the two columns of row PY of the own block (both PX), from global memory.
struct TileRhs {
  float2 v[kSeg][3];
};

// One colour-pair pass (PX, PY): the thread updates the vertices of its column (PX, PY), planes
// lz0 .. lz0 + 3 (lz0 = 1 + 4 seg), reading planes lz0 - 1 .. lz0 + 4. fs: the per-case scale of the
// right-hand side. kLast: no pass follows, so the values stay in registers.
template <int PX, int PY, bool kLast>
__device__ __forceinline__ void tile_pass(float4* sm, TileBlock& own, const TileRhs& rhs, const FineOp& op,
                                          const float (&fs)[3], int lx, int ly, int lz0) {
  constexpr int kCol = PX + 2 * PY;
  // positions of the left / right neighbour columns relative to the own site: the parity of lx
  // is fixed by the pass, so they are compile-time offsets in the parity-split row
  constexpr int oL = PX ? kSHalf - 1 : -kSHalf, oR = PX ? kSHalf : -kSHalf + 1;
  constexpr int dxn[8] = {-1, 0, 1, -1, 1, -1, 0, 1}, dyn[8] = {-1, -1, -1, 0, 0, 1, 1, 1};
  const float4* col = sm + tsite(lx + PX, ly + PY, lz0 - 1);
  float Kp[4] = {0.f, 0.f, 0.f, 0.f};  // conductivities of the previous plane
  PlaneCoef Cp;                        // coefficients of the previous plane
  float accA[3] = {0.f, 0.f, 0.f}, accB[3] = {0.f, 0.f, 0.f}, accC[3] = {0.f, 0.f, 0.f};  // P-1, P, P+1
  float dA = 0.f, dB = 0.f;  // their conductivity sums so far
#pragma unroll
  for (int s = 0; s < kSeg + 2; s++) {  // plane P = lz0 - 1 + s
    const float4* b = col + s * kSPlane;
    float4 nb[8];
#pragma unroll
    for (int n = 0; n < 8; n++) {
      const int cx = PX + dxn[n], cy = PY + dyn[n];
      if (s >= 1 && s <= kSeg && cx >= 0 && cx <= 1 && cy >= 0 && cy <= 1) {
        const int c = cx + 2 * cy;
        nb[n] = make_float4(own.u[c][s - 1][0], own.u[c][s - 1][1], own.u[c][s - 1][2], own.k[c][s - 1]);
      } else {
        nb[n] = b[(dxn[n] < 0 ? oL : (dxn[n] > 0 ? oR : 0)) + dyn[n] * kSRow];
      }
    }
    float kown = 0.f;
    if (s >= 1 && s <= kSeg)
      kown = own.k[kCol][s - 1];
    else if (s == 0)
      kown = reinterpret_cast<const float*>(b)[3];
    const float K[4] = {nb[0].w, nb[1].w, nb[3].w, kown};
    const float sK = (K[0] + K[1]) + (K[2] + K[3]);
    PlaneCoef C;
    if (s <= kSeg) C.make(K, op);
    // vertex P + 1 (segment index s): its lower element plane is P
    float dC = 0.f;
    if (s < kSeg) {
#pragma unroll
      for (int c = 0; c < 3; c++) accC[c] = (PX ? rhs.v[s][c].y : rhs.v[s][c].x) * fs[c];
      sub_plane(accC, C, nb);
      dC = sK;
    }
    // vertex P (index s - 1): in-plane corners, elements of planes P - 1 and P
    if (s >= 1 && s <= kSeg) {
      sub_inplane(accB, Kp, K, op, nb);
      dB += sK;
    }
    // vertex P - 1 (index s - 2): its upper element plane is P - 1; complete now
    if (s >= 2) {
      sub_plane(accA, Cp, nb);
      const float inv = 1.0f / (op.c0 * dA);
#pragma unroll
      for (int c = 0; c < 3; c++) own.u[kCol][s - 2][c] = accA[c] * inv;
      if (!kLast)
        sm[tsite(lx + PX, ly + PY, lz0 + s - 2)] =
            make_float4(own.u[kCol][s - 2][0], own.u[kCol][s - 2][1], own.u[kCol][s - 2][2], own.k[kCol][s - 2]);
    }
    // rotate: P becomes P - 1, P + 1 becomes P
#pragma unroll
    for (int c = 0; c < 3; c++) {
      accA[c] = accB[c];
      accB[c] = accC[c];
    }
    dA = dB;
    dB = dC;
#pragma unroll
    for (int q = 0; q < 4; q++) Kp[q] = K[q];
    Cp = C;
  }
}

// Trilinear prolongation of the staged coarse block (float4 per coarse site, cases in x, y, z) at
// the fine site with unwrapped coordinates (ux, uy, uz); c0x/c0y/c0z are the coarse coordinates
// of the block's first site. The expression and weights are those of prolong_body.
__device__ __forceinline__ float3 prolong_site(const float4* cb, int ux, int uy, int uz, int c0x, int c0y, int c0z) {
  const int ax0 = (ux >> 1) - c0x, ay0 = (uy >> 1) - c0y, az0 = (uz >> 1) - c0z;
  const int ax1 = ax0 + (ux & 1), ay1 = ay0 + (uy & 1), az1 = az0 + (uz & 1);
  const float wx1 = (ux & 1) ? 0.5f : 0.f, wy1 = (uy & 1) ? 0.5f : 0.f, wz1 = (uz & 1) ? 0.5f : 0.f;
  const float wx0 = 1.f - wx1, wy0 = 1.f - wy1, wz0 = 1.f - wz1;
  const float4* r00 = cb + (ay0 + kCY * az0) * kCX;
  const float4* r10 = cb + (ay1 + kCY * az0) * kCX;
  const float4* r01 = cb + (ay0 + kCY * az1) * kCX;
  const float4* r11 = cb + (ay1 + kCY * az1) * kCX;
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

// The prolongation at the 4 fine sites xs .. xs + 3 of a row (xs even, unwrapped), reading the 3
// coarse columns under them once per coarse row instead of 8 coarse sites per fine site. The
// trilinear weights are separable: each coarse column is first interpolated over (y, z), then the
// even sites take their column's value and the odd ones the mean of two columns (the weights of
// prolong_site, summed in another order).
__device__ __forceinline__ void prolong_quad(const float4* cb, int xs, int uy, int uz, int c0x, int c0y, int c0z,
                                             float3 (&o)[4]) {
  const int ax = (xs >> 1) - c0x;  // coarse columns ax, ax + 1, ax + 2
  const int ay0 = (uy >> 1) - c0y, az0 = (uz >> 1) - c0z;
  const int ay1 = ay0 + (uy & 1), az1 = az0 + (uz & 1);
  const float wy1 = (uy & 1) ? 0.5f : 0.f, wz1 = (uz & 1) ? 0.5f : 0.f;
  const float wy0 = 1.f - wy1, wz0 = 1.f - wz1;
  const float4* rows[4] = {cb + (ay0 + kCY * az0) * kCX + ax, cb + (ay1 + kCY * az0) * kCX + ax,
                           cb + (ay0 + kCY * az1) * kCX + ax, cb + (ay1 + kCY * az1) * kCX + ax};
  float3 col[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float4 v0 = rows[0][a], v1 = rows[1][a], v2 = rows[2][a], v3 = rows[3][a];
    col[a].x = wz0 * (wy0 * v0.x + wy1 * v1.x) + wz1 * (wy0 * v2.x + wy1 * v3.x);
    col[a].y = wz0 * (wy0 * v0.y + wy1 * v1.y) + wz1 * (wy0 * v2.y + wy1 * v3.y);
    col[a].z = wz0 * (wy0 * v0.z + wy1 * v1.z) + wz1 * (wy0 * v2.z + wy1 * v3.z);
  }
  o[0] = col[0];
  o[1] = make_float3(0.5f * (col[0].x + col[1].x), 0.5f * (col[0].y + col[1].y), 0.5f * (col[0].z + col[1].z));
  o[2] = col[1];
  o[3] = make_float3(0.5f * (col[1].x + col[2].x), 0.5f * (col[1].y + col[2].y), 0.5f * (col[1].z + col[2].z));
}

// Stages the tile's sites {u_case0, u_case1, u_case2, k_e} in shared memory (parity-split order
// when kSplit, natural order otherwise). With kWithU the values are u (and, when uc is given, plus
// the trilinear prolongation of the coarse correction uc, whose block under the tile is staged in
// cb first); without it they start at 0. Every thread first issues all its global loads (4 values
// of a row at a time for the interior, single values for the two halo columns and the coarse
// block) and only then stores, so a CTA waits for one round of memory latency, not one per site.
template <bool kWithU, int NT, bool kSplit, typename KT, typename VT>
__device__ __forceinline__ void stage_tile(const Dims& d, const Dims& dc, int x0, int y0, int z0,
                                           const KT* __restrict__ ks, const VT* __restrict__ u,
                                           const float* __restrict__ uc, float4* sm, float4* cb) {
  constexpr int kQuads = kSY * kSZ * (kTX / 4), kQI = (kQuads + NT - 1) / NT;
  constexpr int kHalo = kSY * kSZ * 2, kHI = (kHalo + NT - 1) / NT;
  constexpr int kCI = (kCSites + NT - 1) / NT;
  const int t = int(threadIdx.x);
  const size_t nv = d.nv();
  const int c0x = x0 / 2 - 1, c0y = y0 / 2 - 1, c0z = z0 / 2 - 1;
  const bool prolong = kWithU && uc != nullptr;
  // 1. all loads
  float cbv[kCI][3];
  if (prolong) {
    const size_t nvc = dc.nv();
#pragma unroll
    for (int it = 0; it < kCI; it++) {
      const int s = t + it * NT;
      if (s < kCSites) {
        const int ax = s % kCX, ay = (s / kCX) % kCY, az = s / (kCX * kCY);
        const int X = wrapm(c0x + ax, dc.nx), Y = wrapm(c0y + ay, dc.ny), Z = wrapm(c0z + az, dc.nz);
        const size_t g = size_t(X) + size_t(dc.nx) * (size_t(Y) + size_t(dc.ny) * Z);
#pragma unroll
        for (int c = 0; c < 3; c++) cbv[it][c] = __ldg(uc + c * nvc + g);
      }
    }
  }
  float kq[kQI][4], uq[kWithU ? kQI : 1][3][4];
#pragma unroll
  for (int it = 0; it < kQI; it++) {
    const int w = t + it * NT;
    if (w < kQuads) {
      const int q = w & 3, row = w >> 2;
      const int ly = row % kSY, lz = row / kSY;
      const size_t g = size_t(wrapm(x0 + 4 * q, d.nx)) +
                       size_t(d.nx) * (size_t(wrapm(y0 - 1 + ly, d.ny)) + size_t(d.ny) * wrapm(z0 - 1 + lz, d.nz));
      ld4(ks + g, kq[it]);
      if (kWithU)
#pragma unroll
        for (int c = 0; c < 3; c++) ld4(u + c * nv + g, uq[it][c]);
    }
  }
  float kh[kHI], uh[kWithU ? kHI : 1][3];
#pragma unroll
  for (int it = 0; it < kHI; it++) {
    const int w = t + it * NT;
    if (w < kHalo) {
      const int side = w & 1, row = w >> 1;
      const int ly = row % kSY, lz = row / kSY;
      const int lx = side ? kSX - 1 : 0;
      const size_t g = size_t(wrapm(x0 - 1 + lx, d.nx)) +
                       size_t(d.nx) * (size_t(wrapm(y0 - 1 + ly, d.ny)) + size_t(d.ny) * wrapm(z0 - 1 + lz, d.nz));
      kh[it] = ld(ks + g);
      if (kWithU)
#pragma unroll
        for (int c = 0; c < 3; c++) uh[it][c] = ld(u + c * nv + g);
    }
  }
  // 2. the coarse block, needed by every thread's prolongation
  if (prolong) {
#pragma unroll
    for (int it = 0; it < kCI; it++) {
      const int s = t + it * NT;
      if (s < kCSites) cb[s] = make_float4(cbv[it][0], cbv[it][1], cbv[it][2], 0.f);
    }
    __syncthreads();
  }
  // 3. the sites
#pragma unroll
  for (int it = 0; it < kQI; it++) {
    const int w = t + it * NT;
    if (w < kQuads) {
      const int q = w & 3, row = w >> 2;
      const int ly = row % kSY, lz = row / kSY;
      float3 p[4] = {};
      if (prolong) prolong_quad(cb, x0 + 4 * q, y0 - 1 + ly, z0 - 1 + lz, c0x, c0y, c0z, p);
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int lx = 1 + 4 * q + e;
        float4 v = make_float4(0.f, 0.f, 0.f, kq[it][e]);
        if (kWithU) {
          v.x = uq[it][0][e];
          v.y = uq[it][1][e];
          v.z = uq[it][2][e];
          if (prolong) {
            v.x += p[e].x;
            v.y += p[e].y;
            v.z += p[e].z;
          }
        }
        sm[kSplit ? tsite(lx, ly, lz) : rsite(lx, ly, lz)] = v;
      }
    }
  }
#pragma unroll
  for (int it = 0; it < kHI; it++) {
    const int w = t + it * NT;
    if (w < kHalo) {
      const int side = w & 1, row = w >> 1;
      const int ly = row % kSY, lz = row / kSY;
      const int lx = side ? kSX - 1 : 0;
      float4 v = make_float4(0.f, 0.f, 0.f, kh[it]);
      if (kWithU) {
        v.x = uh[it][0];
        v.y = uh[it][1];
        v.z = uh[it][2];
        if (prolong) {
          const float3 p = prolong_site(cb, x0 - 1 + lx, y0 - 1 + ly, z0 - 1 + lz, c0x, c0y, c0z);
          v.x += p.x;
          v.y += p.y;
          v.z += p.z;
        }
      }
      sm[kSplit ? tsite(lx, ly, lz) : rsite(lx, ly, lz)] = v;
    }
  }
}

// Start of a sweep: from zero (the first pre-smoothing sweep), from u_in, or from u_in plus the
// trilinear prolongation of the coarse correction (the first post-smoothing sweep).
enum TileStart { kFromZero = 0, kFromU = 1, kFromUProlong = 2 };

// The right-hand side of row PY of the own block (its two columns), from global memory.
template <int PY>
__device__ __forceinline__ void tile_rhs(const Dims& d, const float* __restrict__ f, int X, const int (&Y)[2],
                                         const int (&Z)[kSeg], TileRhs& rhs) {
  const size_t nv = d.nv();
#pragma unroll
  for (int q = 0; q < kSeg; q++) {
    const float* p = f + size_t(X) + size_t(d.nx) * (size_t(Y[PY]) + size_t(d.ny) * Z[q]);
#pragma unroll
    for (int c = 0; c < 3; c++) rhs.v[q][c] = __ldg(reinterpret_cast<const float2*>(p + c * nv));
  }
}

// One Gauss-Seidel sweep of the fine level on the tiles of tiling `shift` (see above): the tile is
// staged from the start values (kStart), the four colour-pair passes run in the order 0,1,2,3, or
// 3,2,1,0 when kReverse, and the interior goes to u_out, which must not alias u_in. ks: fine
// conductivity (storage KT); f: the right-hand side (FP32, 3 cases, scaled per case by fscale when
// given); u_in / u_out in storage VT; uc: the coarse correction (FP32, kFromUProlong,
// homogenization/grid.cu:881-940); arithmetic and shared memory FP32.
// Per launch at 128^3 (from zero, from u, prolonging): 33.8 / 38.3 / 64.3 us; with the right-hand side
// and the own block read from shared memory in every pass, 2 CTAs per SM: 45.7 / 55.2 / 82.1 us. At
// two CTAs per SM (no spills, 190-226 registers) the 128^3 and 256^3 solves are 2% slower than at three.
template <int kStart, bool kReverse, typename KT, typename VT>
__global__ void __launch_bounds__(kSmoothThreads, 3)
    k_tile_sweep(Dims d, Dims dc, const KT* __restrict__ ks, FineOp op, const VT* __restrict__ u_in,
                 const float* __restrict__ uc, VT* __restrict__ u_out, const float* __restrict__ f,
                 const double* fscale, int shift, const SolveScalars* sc) {
  extern __shared__ float4 sweep_sm[];
  float4* sm = sweep_sm;
  float4* cb = sweep_sm + kSSites;
  const int t = int(threadIdx.x);
  int x0, y0, z0;
  tile_origin(d, blockIdx.x, shift, x0, y0, z0);
  // the own block: 2 x 2 columns from (lx, ly), planes lz0 .. lz0 + 3
  const int lx = 2 * (t & 7) + 1, ly = 2 * ((t >> 3) & 7) + 1, lz0 = 1 + kSeg * (t >> 6);
  const int X = wrapm(x0 + lx - 1, d.nx);
  int Y[2], Z[kSeg];
#pragma unroll
  for (int e = 0; e < 2; e++) Y[e] = wrapm(y0 + ly - 1 + e, d.ny);
#pragma unroll
  for (int q = 0; q < kSeg; q++) Z[q] = wrapm(z0 + lz0 - 1 + q, d.nz);
  pdl_wait();
  if (sc && solve_done(sc)) return;
  TileRhs rhs;
  tile_rhs<kReverse ? 1 : 0>(d, f, X, Y, Z, rhs);
  float fs[3] = {1.f, 1.f, 1.f};
  if (fscale)
#pragma unroll
    for (int c = 0; c < 3; c++) fs[c] = float(fscale[c]);
  stage_tile<kStart != kFromZero, kSmoothThreads, true>(d, dc, x0, y0, z0, ks, u_in,
                                                        kStart == kFromUProlong ? uc : nullptr, sm, cb);
  __syncthreads();
  TileBlock own;
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int q = 0; q < kSeg; q++) {
      const float4 v = sm[tsite(lx + (c & 1), ly + (c >> 1), lz0 + q)];
      own.u[c][q][0] = v.x;
      own.u[c][q][1] = v.y;
      own.u[c][q][2] = v.z;
      own.k[c][q] = v.w;
    }
  // two passes on one row of columns, the other row's right-hand side fetched before the second
  TileRhs rhs2;
  constexpr int PA = kReverse ? 1 : 0, PB = 1 - PA;
  tile_pass<PA, PA, false>(sm, own, rhs, op, fs, lx, ly, lz0);
  __syncthreads();
  tile_rhs<PB>(d, f, X, Y, Z, rhs2);
  tile_pass<PB, PA, false>(sm, own, rhs, op, fs, lx, ly, lz0);
  __syncthreads();
  tile_pass<PA, PB, false>(sm, own, rhs2, op, fs, lx, ly, lz0);
  __syncthreads();
  tile_pass<PB, PB, true>(sm, own, rhs2, op, fs, lx, ly, lz0);
  const size_t nv = d.nv();
#pragma unroll
  for (int q = 0; q < kSeg; q++)
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const size_t g = size_t(X) + size_t(d.nx) * (size_t(Y[e]) + size_t(d.ny) * Z[q]);
#pragma unroll
      for (int c = 0; c < 3; c++) st2(u_out + c * nv + g, own.u[2 * e][q][c], own.u[2 * e + 1][q][c]);
    }
}

// r = f - A u on the fine level for every vertex of a tile (tiling 0), from a staged tile with its
// halo (natural site order here: lanes take consecutive sites of a row). A thread owns one column
// of the tile and streams its 10 planes; the right-hand side is read one plane ahead. Bound by latency at
// 24 warps per SM: 38.2 us at 128^3 (cold caches) against 40.0 with the right-hand side staged too, which
// left two CTAs per SM; the 256^3 solve 0.8% faster.
template <typename KT, typename VT>
__global__ void __launch_bounds__(kResidThreads, 3)
    k_tile_resid(Dims d, const KT* __restrict__ ks, FineOp op, const VT* __restrict__ u, const float* __restrict__ f,
                 VT* __restrict__ r, const double* fscale, const SolveScalars* sc) {
  extern __shared__ float4 resid_sm[];
  float4* sm = resid_sm;
  pdl_wait();
  if (sc && solve_done(sc)) return;
  int x0, y0, z0;
  tile_origin(d, blockIdx.x, 0, x0, y0, z0);
  const size_t nv = d.nv();
  float fs[3] = {1.f, 1.f, 1.f};
  if (fscale)
#pragma unroll
    for (int c = 0; c < 3; c++) fs[c] = float(fscale[c]);
  const int lx = 1 + (int(threadIdx.x) & 15), ly = 1 + (int(threadIdx.x) >> 4);
  const size_t pl = size_t(d.nx) * d.ny;
  const size_t col = size_t(x0 + lx - 1) + size_t(d.nx) * size_t(y0 + ly - 1) + size_t(z0) * pl;
  float fn[3];  // right-hand side of vertex P + 1
#pragma unroll
  for (int c = 0; c < 3; c++) fn[c] = __ldg(f + c * nv + col);
  stage_tile<true, kResidThreads, false>(d, d, x0, y0, z0, ks, u, (const float*)nullptr, sm, (float4*)nullptr);
  __syncthreads();
  float Kp[4] = {0.f, 0.f, 0.f, 0.f};
  PlaneCoef Cp;
  float accA[3] = {0.f, 0.f, 0.f}, accB[3] = {0.f, 0.f, 0.f}, accC[3] = {0.f, 0.f, 0.f};
  float dA = 0.f, dB = 0.f;
  float uA[3] = {0.f, 0.f, 0.f}, uB[3] = {0.f, 0.f, 0.f};  // own values of the vertices P - 1, P
#pragma unroll 1
  for (int P = 0; P < kSZ; P++) {
    const float4* b = sm + rsite(lx, ly, P);
    float4 nb[8];
    nb[0] = b[-kSRow - 1];
    nb[1] = b[-kSRow];
    nb[2] = b[-kSRow + 1];
    nb[3] = b[-1];
    nb[4] = b[1];
    nb[5] = b[kSRow - 1];
    nb[6] = b[kSRow];
    nb[7] = b[kSRow + 1];
    const float4 own = b[0];
    const float K[4] = {nb[0].w, nb[1].w, nb[3].w, own.w};
    const float sK = (K[0] + K[1]) + (K[2] + K[3]);
    PlaneCoef C;
    C.make(K, op);
    float dC = 0.f;
    // vertex P + 1 (interior planes 1..8): lower element plane P
    if (P + 1 <= kTZ) {
#pragma unroll
      for (int c = 0; c < 3; c++) accC[c] = fn[c] * fs[c];
      if (P + 2 <= kTZ)
#pragma unroll
        for (int c = 0; c < 3; c++) fn[c] = __ldg(f + c * nv + col + size_t(P + 1) * pl);
      sub_plane(accC, C, nb);
      dC = sK;
    }
    // vertex P: in-plane corners and its own value
    if (P >= 1 && P <= kTZ) {
      sub_inplane(accB, Kp, K, op, nb);
      dB += sK;
      uB[0] = own.x;
      uB[1] = own.y;
      uB[2] = own.z;
    }
    // vertex P - 1: upper element plane P - 1, then r = f - offdiag - diag u
    if (P >= 2) {
      sub_plane(accA, Cp, nb);
      const float diag = op.c0 * dA;
      const size_t g = col + size_t(P - 2) * pl;
      st(r + g, accA[0] - diag * uA[0]);
      st(r + nv + g, accA[1] - diag * uA[1]);
      st(r + 2 * nv + g, accA[2] - diag * uA[2]);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      accA[c] = accB[c];
      accB[c] = accC[c];
      uA[c] = uB[c];
    }
    dA = dB;
    dB = dC;
#pragma unroll
    for (int q = 0; q < 4; q++) Kp[q] = K[q];
    Cp = C;
  }
}

// The PCG direction update and operator product of k_update_p_apply_dot on tiles (FP32, cube
// elements): p = (z - zbar) + beta p, q = A z + beta q (A p = A z + beta A p_old, A annihilating
// constants), and the p . q partial sums of the tile, reduced by the last CTA into alpha = rho /
// (p . q). z is staged like u in k_tile_resid (tiling 0, one thread per column streaming its 10
// planes) so its 20 neighbours come from shared memory; beta == 0 (the first iteration) ignores
// the old p and q. part: 3 doubles per tile. At 80 registers three CTAs stay on an SM: 40.5 us at 128^3
// (cold caches) against 47.0 with two; the 256^3 solve 3.2% faster.
static __global__ void __launch_bounds__(kResidThreads, 3)
    k_tile_apply_dot(Dims d, const float* __restrict__ ks, FineOp op, const float* __restrict__ z,
                     float* __restrict__ p, float* __restrict__ q, double* part, SolveScalars* sc) {
  extern __shared__ float4 apply_sm[];
  float4* sm = apply_sm;
  pdl_wait();
  if (solve_done(sc)) return;
  int x0, y0, z0;
  tile_origin(d, blockIdx.x, 0, x0, y0, z0);
  const size_t nv = d.nv();
  float be[3], zb[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    be[c] = float(sc->beta[c]);
    zb[c] = float(sc->zmean[c]);
  }
  stage_tile<true, kResidThreads, false>(d, d, x0, y0, z0, ks, z, (const float*)nullptr, sm, (float4*)nullptr);
  __syncthreads();
  const int lx = 1 + (int(threadIdx.x) & 15), ly = 1 + (int(threadIdx.x) >> 4);
  const size_t col = size_t(x0 + lx - 1) + size_t(d.nx) * size_t(y0 + ly - 1);
  const size_t pl = size_t(d.nx) * d.ny;
  float Kp[4] = {0.f, 0.f, 0.f, 0.f};
  PlaneCoef Cp;
  // minus the off-diagonal sums of the vertices P - 1, P, P + 1
  float accA[3] = {0.f, 0.f, 0.f}, accB[3] = {0.f, 0.f, 0.f}, accC[3] = {0.f, 0.f, 0.f};
  float dA = 0.f, dB = 0.f;
  float uA[3] = {0.f, 0.f, 0.f}, uB[3] = {0.f, 0.f, 0.f};  // z of the vertices P - 1, P
  double v[3] = {0, 0, 0};
#pragma unroll 1
  for (int P = 0; P < kSZ; P++) {
    const float4* b = sm + rsite(lx, ly, P);
    float4 nb[8];
    nb[0] = b[-kSRow - 1];
    nb[1] = b[-kSRow];
    nb[2] = b[-kSRow + 1];
    nb[3] = b[-1];
    nb[4] = b[1];
    nb[5] = b[kSRow - 1];
    nb[6] = b[kSRow];
    nb[7] = b[kSRow + 1];
    const float4 own = b[0];
    const float K[4] = {nb[0].w, nb[1].w, nb[3].w, own.w};
    const float sK = (K[0] + K[1]) + (K[2] + K[3]);
    PlaneCoef C;
    C.make(K, op);
    float dC = 0.f;
    if (P + 1 <= kTZ) {  // vertex P + 1: lower element plane P
#pragma unroll
      for (int c = 0; c < 3; c++) accC[c] = 0.f;
      sub_plane(accC, C, nb);
      dC = sK;
    }
    if (P >= 1 && P <= kTZ) {  // vertex P: in-plane corners and its own value
      sub_inplane(accB, Kp, K, op, nb);
      dB += sK;
      uB[0] = own.x;
      uB[1] = own.y;
      uB[2] = own.z;
    }
    if (P >= 2) {  // vertex P - 1: upper element plane P - 1, then the update
      sub_plane(accA, Cp, nb);
      const float diag = op.c0 * dA;
      const size_t g = col + size_t(z0 + P - 2) * pl;
      float po[3], qo[3];  // all loads of the vertex before its stores
#pragma unroll
      for (int c = 0; c < 3; c++) {
        po[c] = be[c] != 0.f ? p[c * nv + g] : 0.f;
        qo[c] = be[c] != 0.f ? q[c * nv + g] : 0.f;
      }
#pragma unroll
      for (int c = 0; c < 3; c++) {
        float pc = uA[c] - zb[c], qc = diag * uA[c] - accA[c];  // accA = -(off-diagonal sum)
        if (be[c] != 0.f) {
          pc += be[c] * po[c];
          qc += be[c] * qo[c];
        }
        p[c * nv + g] = pc;
        q[c * nv + g] = qc;
        v[c] += double(pc) * qc;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      accA[c] = accB[c];
      accB[c] = accC[c];
      uA[c] = uB[c];
    }
    dA = dB;
    dB = dC;
#pragma unroll
    for (int q4 = 0; q4 < 4; q4++) Kp[q4] = K[q4];
    Cp = C;
  }
  double* red = reinterpret_cast<double*>(sm);  // the tile is no longer read
  __syncthreads();
  block_reduce_f64<3>(v, red);
  if (threadIdx.x == 0)
#pragma unroll
    for (int i = 0; i < 3; i++) part[size_t(blockIdx.x) * 3 + i] = v[i];
  if (last_block(&sc->counter[T_PQ])) {
    double t[3];
    reduce_partials<3>(part, int(gridDim.x), t, red);
    if (threadIdx.x == 0) {
      for (int c = 0; c < 3; c++) sc->alpha[c] = t[c] != 0.0 ? sc->rz[c] / t[c] : 0.0;
      sc->counter[T_PQ] = 0;
    }
  }
}

}  // namespace otm
