// otm_filter.cu -- density filter (radial convolution with in-bounds renormalisation), the
// fused SIMP density chain and their adjoints (AutoDiff/TensorExpression.h:993-1185,
// AutoDiff/TensorExpression.cuh:281-385).
//
// The normalised weights travel as a kernel parameter (constant bank, broadcast to the
// warp), so no device allocation or global state is used.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "otm_common.cuh"

namespace otm {

constexpr int kMaxHalf = 6;
constexpr int kMaxTaps = (2 * kMaxHalf + 1) * (2 * kMaxHalf + 1) * (2 * kMaxHalf + 1);

struct ConvWeights {
  int half;  // h = int(radius + 0.5)
  int taps;  // (2h+1)^3
  float w[kMaxTaps];  // w(off) / sum_cube w, off enumerated x fastest from -h
};

// Radial weight functions WeightFunc<Spline4> / WeightFunc<Linear>
// (AutoDiff/TensorExpression.h:1054-1077), evaluated in FP32 as in the reference.
static float radial_weight(int type, float r, int ox, int oy, int oz) {
  const float q2 = float(ox * ox + oy * oy + oz * oz) / (r * r);
  const float q = std::sqrt(q2);
  if (!(q2 < 1.f)) return 0.f;
  if (type == OTM_WEIGHT_SPLINE4) return 1.f - 6.f * q2 + 8.f * q2 * q - 3.f * q2 * q2;
  return 1.f - q;
}

static otm_status make_weights(int type, float radius, ConvWeights* cw) {
  if (type != OTM_WEIGHT_SPLINE4 && type != OTM_WEIGHT_LINEAR) {
    set_error("unknown filter weight type");
    return OTM_ERR_INVALID_ARGUMENT;
  }
  if (!(radius > 0.f)) {
    set_error("filter radius must be positive");
    return OTM_ERR_INVALID_ARGUMENT;
  }
  const int h = int(radius + 0.5f);  // convker_t halfdomain = r + 0.5 truncated (TensorExpression.h:1079-1093)
  if (h > kMaxHalf) {
    set_error("filter radius too large (half width must be <= 6)");
    return OTM_ERR_UNSUPPORTED;
  }
  cw->half = h;
  cw->taps = (2 * h + 1) * (2 * h + 1) * (2 * h + 1);
  float wsum = 0.f;
  for (int i = 0; i < cw->taps; i++) {
    const int ox = i % (2 * h + 1) - h, oy = i / (2 * h + 1) % (2 * h + 1) - h, oz = i / ((2 * h + 1) * (2 * h + 1)) - h;
    cw->w[i] = radial_weight(type, radius, ox, oy, oz);
    wsum += cw->w[i];
  }
  for (int i = 0; i < cw->taps; i++) cw->w[i] /= wsum;  // normalize = true
  return OTM_OK;
}

// Convolution streaming along z: a 128-thread block produces the outputs of a tile of 32 x 4 kNY
// (x, y) columns for a chunk of z planes, kNY rows of outputs per thread and plane. Each input plane of
// the chunk (and H planes either side) is staged once in shared memory, with periodic wrap or zeros
// outside, the next one being fetched into registers meanwhile; a thread reads the (kNY + 2H) x (2H + 1)
// window around its outputs once per plane and adds every value to the 2H + 1 outputs along z that it
// is a tap of (rolling accumulators): 9 reads per output at radius 2 with one row, 10 at radius 3 with
// four, where a read per tap takes 27 and 93. The weight depends on the squared distance only, and with the
// loops unrolled its place in the parameter bank is a constant, so a tap is one FMA. The radii in common
// use (1.5 to 2, 2.5 to 3, 3.5 to 3.6, 3.75 to 4) have their set of taps compiled in; the other radii of a half
// width H share the taps within H - 1/2, and those from there to H + 1/2 are predicated on the radius. (With a
// branch per tap, and from half width 5 on with weights looked up by a run-time index and four rows a thread,
// these radii took up to four times the time of a kernel that reads every tap's value for itself: 128^3,
// radius 4.4, 5 and 6: 194, 333 and 845 us against 140, 189 and 297; now 92, 127 and 187.) An output's taps
// are summed in the reference's order (x fastest, z slowest; the adjoint streams z downwards for that).
//   MODE 0: forward            out = sum w src / sum_valid w
//   MODE 1: forward + SIMP     also k = (k0 - kmin) out^p + kmin and dk = dk/dout
//   MODE 2: adjoint            out = sum_off w g(i - off) / ws(i - off)
//   MODE 3: adjoint chain      as 2 with g = g_k * dk
//   MODE 4: forward + SIMP + conductivity import: as 1, with k written as the solver's raw
//           conductivity and ks = 1e-9 + k^pp beside it (k_import's arithmetic), a negative,
//           NaN or Inf k flagged in *bad
//   MODE 5: OC sensitivity     out = sum w src / (sum w * rho), rho (ws_in) pitched like out
constexpr int kTX = 32, kTYT = 4, kConvThreads = kTX * kTYT;

// A radial filter: weight by squared distance, zero from smax on.
template <int H>
struct Radial {
  float w[3 * H * H + 1];
  int smax;
};

template <int H>
static void make_radial(const ConvWeights& cw, Radial<H>* r) {
  constexpr int W1 = 2 * H + 1;
  for (float& w : r->w) w = 0.f;
  r->smax = 0;
  for (int k = 0; k <= H; k++)
    for (int oy = -H; oy <= H; oy++)
      for (int ox = -H; ox <= H; ox++) {
        const int s = ox * ox + oy * oy + k * k;
        r->w[s] = cw.w[(ox + H) + W1 * ((oy + H) + W1 * (k + H))];
        if (r->w[s] != 0.f && s >= r->smax) r->smax = s + 1;
      }
}

// Zero padding: the valid weight of a voxel is the sum of its in-bounds taps in the reference's order (x
// fastest, z slowest), one after the other. A column's taps are in bounds for offsets xlo..xhi, ylo..yhi in
// its planes; along z a voxel may be cut above (its sum is an intermediate value of the whole column's) or
// below (its sum starts at a later plane). up[m]: planes -H..m; low[g]: planes -g..H, g < H, with kLow
// (from half width 5 on only those the block needs, g0 <= g < g1, and up only where it reaches plane H).
// Taps past the filter's reach add a weight of zero. (Summed plane by plane first,
// the weights of boundary voxels differed in the last bits from those of the reference's order, and with them
// every density of a zero-padded design run.)
template <int H, int kS, bool kLow>
__device__ __forceinline__ void valid_weights(const Radial<H>& rw, int xlo, int xhi, int ylo, int yhi, int g0, int g1,
                                              float (&up)[H + 1], float (&low)[H + 1]) {
  constexpr int kReach = kS > 0 ? kS : H * H + H + 1;
  float a = 0.f;
#pragma unroll
  for (int g = 0; g <= H; g++) low[g] = 0.f;
  auto row = [&](int ez, int ey) {
    float w[2 * H + 1];
    auto beyond = [&](int ex) { return H <= 4 && ex * ex + ey * ey + ez * ez >= kReach; };  // of every radius
#pragma unroll
    for (int ex = -H; ex <= H; ex++)
      if (!beyond(ex)) w[ex + H] = ex >= xlo && ex <= xhi ? rw.w[ex * ex + ey * ey + ez * ez] : 0.f;
    if (H <= 4 || !kLow || g1 >= H)
#pragma unroll
      for (int ex = -H; ex <= H; ex++)
        if (!beyond(ex)) a += w[ex + H];
    if (kLow)
#pragma unroll
      for (int g = 0; g < H; g++)
        if (ez >= -g && (H <= 4 || (g >= g0 && g < g1)))
#pragma unroll
          for (int ex = -H; ex <= H; ex++)
            if (!beyond(ex)) low[g] += w[ex + H];
  };
#pragma unroll(H <= 4 ? 2 * H + 1 : 1)
  for (int ez = -H; ez <= H; ez++) {
    if (H <= 4) {
#pragma unroll
      for (int ey = -H; ey <= H; ey++)
        if (ey >= ylo && ey <= yhi && ey * ey + ez * ez < rw.smax) row(ez, ey);  // the same for all lanes of a warp
    } else {
      int ry = H;  // rows of the plane within the filter's reach
      while (ry >= 0 && ry * ry + ez * ez >= rw.smax) ry--;
#pragma unroll 4
      for (int ey = max(ylo, -ry); ey <= min(yhi, ry); ey++) row(ez, ey);
    }
#pragma unroll
    for (int m = 0; m <= H; m++)
      if (ez == m) up[m] = a;
  }
}

// kS: the filter's smax where it is known at compile time (then the taps are straight-line code), else 0.
template <int H, int kS, int kNY, int MODE>
__global__ void __launch_bounds__(kConvThreads) k_conv_stream(Dims d, const float* __restrict__ src, size_t src_pitch,
                                                              const float* __restrict__ dk_in,
                                                              const float* __restrict__ ws_in,
                                                              float* __restrict__ dst, size_t dst_pitch,
                                                              float* __restrict__ ws_out, int periodic, int zchunk,
                                                              const __grid_constant__ Radial<H> rw, float wsum_all,
                                                              float p, float k0, float kmin, float* __restrict__ kout,
                                                              float* __restrict__ dkout, float* __restrict__ ksout,
                                                              float pp, int* bad) {
  constexpr int kTY = kTYT * kNY;
  constexpr int SX = kTX + 2 * H, SY = kTY + 2 * H, SN = SX * SY, NL = (SN + kConvThreads - 1) / kConvThreads;
  constexpr bool kFwd = MODE < 2 || MODE >= 4, kValid = kFwd && MODE != 5;
  constexpr int W1 = 2 * H + 1;
  // squared distances below kSure are taps of every radius of this half width (at least H - 1/2), those from
  // kReach on of none
  constexpr int kSure = kS > 0 ? kS : (H == 0 ? 1 : H * H - H + 1), kReach = kS > 0 ? kS : H * H + H + 1;
  __shared__ float buf[2][SN];
  // zero padding: valid weights of a column's voxels m = 0..H - 1 planes from its upper end, of those farther
  // from both ends (H) and of plane g (H + 1 + g); of plane g (g) where there are at most 2H planes
  __shared__ float wcol[kValid ? 2 * H + 1 : 1][kTY][kTX];
  const int tid = threadIdx.x + kTX * threadIdx.y;
  // blocks in one dimension, x tiles fastest: a launch's y and z extents end at 65,535
  const unsigned tx = unsigned(d.nx + kTX - 1) / kTX, ty = unsigned(d.ny + kTY - 1) / kTY, bq = blockIdx.x / tx;
  const int x0 = int(blockIdx.x - bq * tx) * kTX, y0 = int(bq % ty) * kTY, z0 = int(bq / ty) * zchunk;
  const int z1 = min(z0 + zchunk, d.nz), planes = z1 - z0 + 2 * H;
  const int ox = x0 + int(threadIdx.x), oyr = int(threadIdx.y) * kNY, oy0 = y0 + oyr;  // own outputs
  const int xlo = max(-H, -ox), xhi = min(H, d.nx - 1 - ox);  // own taps in bounds along x
  if (kValid && !periodic) {
    const bool cut_z = z0 < H || z1 > d.nz - H;
#pragma unroll 1
    for (int j = 0; j < kNY; j++) {
      const int ylo = max(-H, -(oy0 + j)), yhi = min(H, d.ny - 1 - (oy0 + j));
      const bool cut = cut_z || ylo > -H || yhi < H || xlo > -H || xhi < H;
      if (!__any_sync(0xffffffffu, cut)) continue;
      if (d.nz <= 2 * H) {
        for (int g = 0; g < d.nz; g++) {
          float a = 0.f;
          for (int ez = -min(g, H); ez <= min(H, d.nz - 1 - g); ez++)
            for (int ey = ylo; ey <= yhi; ey++)
              for (int ex = xlo; ex <= xhi; ex++) a += rw.w[ex * ex + ey * ey + ez * ez];
          wcol[kValid ? g : 0][oyr + j][threadIdx.x] = a;
        }
        continue;
      }
      float up[H + 1], low[H + 1];
      if (z0 < H)
        valid_weights<H, kS, true>(rw, xlo, xhi, ylo, yhi, z0, min(z1, H), up, low);
      else
        valid_weights<H, kS, false>(rw, xlo, xhi, ylo, yhi, 0, 0, up, low);
#pragma unroll
      for (int m = 0; m <= H; m++) wcol[m][oyr + j][threadIdx.x] = up[m];
      if (z0 < H)
#pragma unroll
        for (int g = 0; g < H; g++) wcol[kValid ? H + 1 + g : 0][oyr + j][threadIdx.x] = low[g];
    }
  }
  // this thread's staged positions (the same in every plane): offsets in a plane of src and of the
  // unpitched dk and ws
  size_t off[NL], offw[kFwd ? 1 : NL];
  bool ok[NL];
#pragma unroll
  for (int i = 0; i < NL; i++) {
    const int s = tid + i * kConvThreads;
    int x = x0 + s % SX - H, y = y0 + s / SX - H;
    const bool in = x >= 0 && x < d.nx && y >= 0 && y < d.ny;
    if (!in) {
      x = ((x % d.nx) + d.nx) % d.nx;
      y = ((y % d.ny) + d.ny) % d.ny;
    }
    off[i] = size_t(y) * src_pitch + x;
    if (!kFwd) offw[kFwd ? 0 : i] = size_t(y) * d.nx + x;
    ok[i] = s < SN && (in || periodic);
  }
  // plane `pl` of the chunk, counted in streaming order: the loads into registers first (none waits for
  // another), the arithmetic when the plane is staged
  float v[NL], vk[MODE == 3 ? NL : 1], vw[kFwd ? 1 : NL];
  auto fetch = [&](int pl) {
    int gz = kFwd ? z0 - H + pl : z1 - 1 + H - pl;
    const bool inz = gz >= 0 && gz < d.nz;
    if (!inz) gz = ((gz % d.nz) + d.nz) % d.nz;
    const float* ps = src + size_t(gz) * d.ny * src_pitch;
    const size_t pw = size_t(gz) * d.ny * d.nx;
    const bool any = inz || periodic;
#pragma unroll
    for (int i = 0; i < NL; i++) {
      const bool take = ok[i] && any;
      v[i] = take ? __ldg(ps + off[i]) : 0.f;
      if (MODE == 3) vk[MODE == 3 ? i : 0] = take ? __ldg(dk_in + pw + offw[kFwd ? 0 : i]) : 0.f;
      if (!kFwd) vw[kFwd ? 0 : i] = take ? __ldg(ws_in + pw + offw[kFwd ? 0 : i]) : 1.f;
    }
  };
  auto stage = [&](float* b) {
#pragma unroll
    for (int i = 0; i < NL; i++) {
      float t = v[i];
      if (MODE == 3) t *= vk[MODE == 3 ? i : 0];
      if (!kFwd) t /= vw[kFwd ? 0 : i];
      if (tid + i * kConvThreads < SN) b[tid + i * kConvThreads] = t;
    }
  };
  fetch(0);
  stage(buf[0]);
  __syncthreads();
  const int base = (oyr + H) * SX + int(threadIdx.x) + H;
  float acc[W1][kNY];  // acc[a]: the output H - a planes behind the current input plane
#pragma unroll
  for (int a = 0; a < W1; a++)
#pragma unroll
    for (int j = 0; j < kNY; j++) acc[a][j] = 0.f;
  for (int pl = 0; pl < planes; pl++) {
    if (pl + 1 < planes) fetch(pl + 1);
    const float* b = buf[pl & 1] + base;
    // row by row of the window, every value read once; an output meets its taps (oy, ox) in the
    // reference's order (the adjoint's offsets are negated, so it takes the rows downwards)
#pragma unroll
    for (int i = 0; i < kNY + 2 * H; i++) {
      const int r = kFwd ? i - H : kNY - 1 + H - i;
#pragma unroll
      for (int ex = -H; ex <= H; ex++) {
        if (ex * ex >= kReach) continue;
        const float t = b[r * SX + (kFwd ? ex : -ex)];
#pragma unroll
        for (int j = 0; j < kNY; j++) {
          const int ey = kFwd ? r - j : j - r;
          if (ey < -H || ey > H) continue;
#pragma unroll
          for (int k = 0; k <= H; k++) {
            const int q = ex * ex + ey * ey + k * k;
            if (q >= kReach) continue;
            if (q < kSure || q < rw.smax) {
              acc[H - k][j] += rw.w[q] * t;
              if (k > 0) acc[H + k][j] += rw.w[q] * t;
            }
          }
        }
      }
    }
    if (pl >= 2 * H) {
      const int gz = kFwd ? z0 + pl - 2 * H : z1 - 1 - (pl - 2 * H);
#pragma unroll
      for (int j = 0; j < kNY; j++) {
        const int oy = oy0 + j;
        if (ox >= d.nx || oy >= d.ny) continue;
        const float sumv = acc[0][j];
        const size_t row = size_t(oy) + size_t(d.ny) * gz;
        const size_t e = row * d.nx + ox;
        if (!kFwd) {
          dst[row * dst_pitch + ox] = sumv;
        } else if (MODE == 5) {
          const size_t q = row * dst_pitch + ox;
          dst[q] = sumv / (wsum_all * __ldg(ws_in + q));
        } else {
          float ws = wsum_all;
          if (!periodic && (ox < H || ox >= d.nx - H || oy < H || oy >= d.ny - H || gz < H || gz >= d.nz - H)) {
            const int m = d.nz <= 2 * H ? gz : (gz < H ? H + 1 + gz : min(d.nz - 1 - gz, H));
            ws = wcol[kValid ? m : 0][oyr + j][threadIdx.x];
          }
          const float out = sumv / ws;
          if (dst) dst[row * dst_pitch + ox] = out;
          if (ws_out) ws_out[e] = ws;
          if (MODE == 1 || MODE == 4) {
            const float pw = (p == 3.f) ? out * out * out : powf(out, p);
            const float k = (k0 - kmin) * pw + kmin;
            kout[e] = k;
            const float dpw = (p == 3.f) ? 3.f * out * out : p * powf(out, p - 1.f);
            dkout[e] = (k0 - kmin) * dpw;
            if (MODE == 4) {
              if (!(k >= 0.f) || !isfinite(k)) atomicOr(bad, 1);
              ksout[e] = kRhoPenalMin + (pp == 1.f ? k : powf(k, pp));
            }
          }
        }
      }
    }
#pragma unroll
    for (int a = 0; a < 2 * H; a++)
#pragma unroll
      for (int j = 0; j < kNY; j++) acc[a][j] = acc[a + 1][j];
#pragma unroll
    for (int j = 0; j < kNY; j++) acc[2 * H][j] = 0.f;
    if (pl + 1 < planes) stage(buf[(pl + 1) & 1]);  // last read one plane ago, before the barrier below
    __syncthreads();
  }
}

// Blocks of a launch with ny rows per thread and z chunks of zc planes.
constexpr long long kConvSms = 148;
static long long conv_blocks(const Dims& d, int ny, int zc) {
  return (long long)((d.nx + kTX - 1) / kTX) * ((d.ny + kTYT * ny - 1) / (kTYT * ny)) * ((d.nz + zc - 1) / zc);
}
// The z chunk: a block works through its planes and 2 H more, and the blocks of an SM share it once there are
// more than kShare, so the chunk with the least planes x max(kShare, blocks per SM). Within 3 % of the best
// of 2 to 64 planes on average over 16^3 to 256^3 and radii 1.2 to 6. The longest chunk that leaves eight
// blocks per SM, as it was, costs 25 % more at radius 6 (96^3: 249 against 140 us) and 2 to 4 % at radius 1.2
// to 2.2.
template <int H>
static int conv_zchunk(const Dims& d, int ny) {
  constexpr long long kShare = H <= 2 ? 4 : 3;
  int best = 32;
  long long least = LLONG_MAX;
  for (int zc = 32; zc >= 4; zc /= 2) {
    const long long per_sm = (conv_blocks(d, ny, zc) + kConvSms - 1) / kConvSms;
    const long long cost = (std::min(zc, d.nz) + 2 * H) * std::max(kShare, per_sm);
    if (cost < least) {
      least = cost;
      best = zc;
    }
  }
  return best;
}

template <int H, int MODE>
static otm_status launch_stream(const Dims& d, const float* src, size_t src_pitch, const float* dk_in, const float* ws_in,
                                float* dst, size_t dst_pitch, float* ws_out, int periodic, const ConvWeights& cw,
                                float wsum_all, float p, float k0, float kmin, float* kout, float* dkout, float* ksout,
                                float pp, int* bad, cudaStream_t s) {
  Radial<H> rw;
  make_radial<H>(cw, &rw);
  auto run = [&](auto ny_tag) {
    constexpr int kNY = decltype(ny_tag)::value;
    const int zchunk = conv_zchunk<H>(d, kNY);
    const unsigned grid = unsigned(conv_blocks(d, kNY, zchunk));
    auto launch = [&](auto kern) {
      kern<<<grid, dim3(kTX, kTYT), 0, s>>>(d, src, src_pitch, dk_in, ws_in, dst, dst_pitch, ws_out, periodic, zchunk,
                                            rw, wsum_all, p, k0, kmin, kout, dkout, ksout, pp, bad);
    };
    if (H == 2 && rw.smax == 3)
      launch(k_conv_stream<H, (H == 2 ? 3 : 0), kNY, MODE>);
    else if (H == 2 && rw.smax == 4)
      launch(k_conv_stream<H, (H == 2 ? 4 : 0), kNY, MODE>);
    else if (H == 3 && rw.smax == 7)
      launch(k_conv_stream<H, (H == 3 ? 7 : 0), kNY, MODE>);
    else if (H == 3 && rw.smax == 9)
      launch(k_conv_stream<H, (H == 3 ? 9 : 0), kNY, MODE>);
    else if (H == 4 && rw.smax == 13)
      launch(k_conv_stream<H, (H == 4 ? 13 : 0), kNY, MODE>);
    else if (H == 4 && rw.smax == 15)
      launch(k_conv_stream<H, (H == 4 ? 15 : 0), kNY, MODE>);
    else
      launch(k_conv_stream<H, 0, kNY, MODE>);
  };
  // rows per thread: 4 where shared-memory reads bound a single row (half widths 3 and 4: about one read per
  // three multiply-adds; five and more from half width 5 on) and the cell fills the GPU with the fewer
  // threads, else 1
  constexpr int kFew = 1, kMany = H == 3 || H == 4 ? 4 : 1;
  if (kFew != kMany && conv_blocks(d, kMany, 16) < 8 * kConvSms)
    run(std::integral_constant<int, kFew>{});
  else
    run(std::integral_constant<int, kMany>{});
  OTM_CHECK_LAUNCH("k_conv_stream");
  count_launches(1);
  return OTM_OK;
}

template <int MODE>
static otm_status conv_dispatch(const Dims& d, const float* src, size_t src_pitch, const float* dk_in,
                                const float* ws_in, float* dst, size_t dst_pitch, float* ws_out, int periodic,
                                const ConvWeights& cw, float p, float k0, float kmin, float* kout, float* dkout,
                                cudaStream_t s, float* ksout = nullptr, float pp = 1.f, int* bad = nullptr) {
  // sum of the normalised weights in the reference's tap order (the in-bounds weight of a
  // periodic filter)
  float wsum_all = 0.f;
  for (int t = 0; t < cw.taps; t++) wsum_all += cw.w[t];
  switch (cw.half) {
#define OTM_H(HH) \
  case HH:        \
    return launch_stream<HH, MODE>(d, src, src_pitch, dk_in, ws_in, dst, dst_pitch, ws_out, periodic, cw, wsum_all, \
                                  p, k0, kmin, kout, dkout, ksout, pp, bad, s);
    OTM_H(0) OTM_H(1) OTM_H(2) OTM_H(3) OTM_H(4) OTM_H(5) OTM_H(6)
#undef OTM_H
  }
  set_error("unsupported filter half width");
  return OTM_ERR_UNSUPPORTED;
}

// The density chain's forward pass writing straight into a homogenization handle's conductivity
// buffers (otm_homo_update_density): rho_f, dk and wsum as otm_density_forward, k as kraw and
// ks = 1e-9 + k^pp, invalid values flagged in *bad.
otm_status density_forward_import(const Dims& d, const float* rho, int rho_pitchT, float* rho_f, float* dk,
                                  float* wsum, int weight_type, float radius, int periodic, float p, float k0,
                                  float kmin, float* kraw, float* ks, float pp, int* bad, cudaStream_t s) {
  if (!rho || !dk || !wsum) return OTM_ERR_INVALID_ARGUMENT;
  if (rho_pitchT <= 0) rho_pitchT = d.nx;
  if (rho_pitchT < d.nx) return OTM_ERR_INVALID_ARGUMENT;
  ConvWeights cw;
  OTM_TRY(make_weights(weight_type, radius, &cw));
  return conv_dispatch<4>(d, rho, rho_pitchT, nullptr, nullptr, rho_f, d.nx, wsum, periodic, cw, p, k0, kmin, kraw,
                          dk, s, ks, pp, bad);
}

__global__ void __launch_bounds__(256) k_product(Dims d, const float* __restrict__ sens, const float* __restrict__ rho,
                                                 size_t pitch, float* __restrict__ out) {
  const size_t v = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= d.nv()) return;
  const size_t row = v / d.nx, q = row * pitch + (v - row * d.nx);
  out[v] = sens[q] * rho[q];
}

// OCOptimizer::filterSens (optimization/OCOptimizer.cu:76-152): s_e <- sum w s_n rho_n / (sum w * rho_e)
// over the periodic Linear neighbourhood, in place. The products s rho go to tmp (d.nv() floats)
// first, so that the convolution can write s. At 128^3, radius 2: products 9.5 us and convolution 25 us,
// against 1457 us with every tap read and wrapped from global memory by each voxel and a copy back.
otm_status oc_filter_run(const Dims& d, float* sens, const float* rho, size_t pitch, float* tmp, float radius,
                         cudaStream_t s) {
  ConvWeights cw;
  OTM_TRY(make_weights(OTM_WEIGHT_LINEAR, radius, &cw));
  k_product<<<unsigned(ceil_div(d.nv(), 256)), 256, 0, s>>>(d, sens, rho, pitch, tmp);
  OTM_CHECK_LAUNCH("k_product");
  count_launches(1);
  return conv_dispatch<5>(d, tmp, d.nx, nullptr, rho, sens, pitch, nullptr, 1, cw, 1.f, 1.f, 0.f, nullptr, nullptr, s);
}

static otm_status check_reso(const int reso[3]) {
  if (!reso || reso[0] < 1 || reso[1] < 1 || reso[2] < 1) {
    set_error("invalid resolution");
    return OTM_ERR_INVALID_ARGUMENT;
  }
  return OTM_OK;
}

}  // namespace otm

using namespace otm;

extern "C" {

otm_status otm_filter_forward(const int reso[3], const float* src, int src_pitchT, float* dst, int dst_pitchT,
                              float* wsum, int weight_type, float radius, int periodic, void* stream) {
  OTM_TRY(check_reso(reso));
  if (!src || !dst) return OTM_ERR_INVALID_ARGUMENT;
  const Dims d{reso[0], reso[1], reso[2]};
  if (src_pitchT <= 0) src_pitchT = d.nx;
  if (dst_pitchT <= 0) dst_pitchT = d.nx;
  if (src_pitchT < d.nx || dst_pitchT < d.nx) return OTM_ERR_INVALID_ARGUMENT;
  ConvWeights cw;
  OTM_TRY(make_weights(weight_type, radius, &cw));
  return conv_dispatch<0>(d, src, src_pitchT, nullptr, nullptr, dst, dst_pitchT, wsum, periodic, cw, 1.f, 1.f, 0.f,
                         nullptr, nullptr, (cudaStream_t)stream);
}

otm_status otm_filter_backward(const int reso[3], const float* g_dst, int g_dst_pitchT, const float* wsum,
                               float* g_src, int g_src_pitchT, int weight_type, float radius, int periodic,
                               void* stream) {
  OTM_TRY(check_reso(reso));
  if (!g_dst || !wsum || !g_src) return OTM_ERR_INVALID_ARGUMENT;
  const Dims d{reso[0], reso[1], reso[2]};
  if (g_dst_pitchT <= 0) g_dst_pitchT = d.nx;
  if (g_src_pitchT <= 0) g_src_pitchT = d.nx;
  if (g_dst_pitchT < d.nx || g_src_pitchT < d.nx) return OTM_ERR_INVALID_ARGUMENT;
  ConvWeights cw;
  OTM_TRY(make_weights(weight_type, radius, &cw));
  return conv_dispatch<2>(d, g_dst, g_dst_pitchT, nullptr, wsum, g_src, g_src_pitchT, nullptr, periodic, cw, 1.f,
                         1.f, 0.f, nullptr, nullptr, (cudaStream_t)stream);
}

otm_status otm_density_forward(const int reso[3], const float* rho, int rho_pitchT, float* rho_f, float* k,
                               float* dk, float* wsum, int weight_type, float radius, int periodic, float p,
                               float k0, float kmin, void* stream) {
  OTM_TRY(check_reso(reso));
  if (!rho || !k || !dk || !wsum) return OTM_ERR_INVALID_ARGUMENT;
  const Dims d{reso[0], reso[1], reso[2]};
  if (rho_pitchT <= 0) rho_pitchT = d.nx;
  if (rho_pitchT < d.nx) return OTM_ERR_INVALID_ARGUMENT;
  ConvWeights cw;
  OTM_TRY(make_weights(weight_type, radius, &cw));
  return conv_dispatch<1>(d, rho, rho_pitchT, nullptr, nullptr, rho_f, d.nx, wsum, periodic, cw, p, k0, kmin, k, dk,
                         (cudaStream_t)stream);
}

otm_status otm_density_backward(const int reso[3], const float* g_k, const float* dk, const float* wsum,
                                float* g_rho, int g_rho_pitchT, int weight_type, float radius, int periodic,
                                void* stream) {
  OTM_TRY(check_reso(reso));
  if (!g_k || !dk || !wsum || !g_rho) return OTM_ERR_INVALID_ARGUMENT;
  const Dims d{reso[0], reso[1], reso[2]};
  if (g_rho_pitchT <= 0) g_rho_pitchT = d.nx;
  if (g_rho_pitchT < d.nx) return OTM_ERR_INVALID_ARGUMENT;
  ConvWeights cw;
  OTM_TRY(make_weights(weight_type, radius, &cw));
  return conv_dispatch<3>(d, g_k, d.nx, dk, wsum, g_rho, g_rho_pitchT, nullptr, periodic, cw, 1.f, 1.f, 0.f, nullptr,
                         nullptr, (cudaStream_t)stream);
}

}  // extern "C"
