// CPU check of a handle's device memory: otm::Homo::build on a CUDA runtime that only counts, linked with the
// library's own objects. A handle of its own takes one device allocation, a handle of the server none that
// the size it is admitted with does not cover. Host code only; prints "ok".
#include <cstdio>

#include "opentm_b200_server.h"
#include "otm_homo_impl.h"

// counting_runtime.cpp
extern int mallocs;
extern size_t malloc_bytes, pool_bytes;

static int fails = 0;

static void check_handle(int nx, int ny, int nz, int sweeps, int precision) {
  otm_config c;
  otm_config_init(&c);
  c.reso[0] = nx, c.reso[1] = ny, c.reso[2] = nz;
  c.pre_smooth = c.post_smooth = sweeps;
  c.precision = precision;
  mallocs = 0;
  malloc_bytes = 0;
  otm::Homo h;
  const otm_status st = h.build(c);
  if (st != OTM_OK || mallocs != 1 || h.arena_left != 0 || h.bytes_allocated > malloc_bytes) {
    std::printf("%dx%dx%d V(%d,%d) precision %d: status %d, %d allocations, %zu bytes left of %zu\n", nx, ny, nz, sweeps,
                sweeps, precision, int(st), mallocs, h.arena_left, malloc_bytes);
    fails++;
  }
}

static void check_server(int nx, int ny, int nz) {
  const int reso[3] = {nx, ny, nz};
  otm_config c;
  otm_config_init(&c);
  for (int i = 0; i < 3; i++) c.reso[i] = reso[i];
  c.pre_smooth = c.post_smooth = 2;  // the server's default
  pool_bytes = 0;
  otm::Homo h;
  const otm_status st = h.build(c, nullptr, reinterpret_cast<cudaMemPool_t>(size_t(16)), true);
  const size_t counted = otm_server_request_bytes(reso);
  const size_t field = size_t(nx) * ny * nz * sizeof(float);  // imported while the request is set up
  // at most the padding of some forty buffers and the plane tables above what is taken
  if (st != OTM_OK || counted < pool_bytes + field || counted > pool_bytes + field + pool_bytes / 50 + 65536) {
    std::printf("request of %dx%dx%d: takes %zu bytes, counted as %zu\n", nx, ny, nz, pool_bytes + field, counted);
    fails++;
  }
}

int main() {
  const int cells[][3] = {{8, 8, 8},    {9, 9, 9},    {18, 18, 18}, {20, 22, 18},  {32, 32, 32},   {36, 36, 36},
                          {40, 56, 72}, {64, 64, 64}, {96, 64, 48}, {96, 128, 64}, {128, 128, 128}, {256, 256, 256}};
  for (const auto& d : cells)
    for (int sweeps = 1; sweeps <= 2; sweeps++)
      for (int precision : {int(OTM_PRECISION_FP32), int(OTM_PRECISION_MIXED_BF16)})
        if (precision == OTM_PRECISION_FP32 || (d[0] >= 16 && d[0] % 4 == 0))
          check_handle(d[0], d[1], d[2], sweeps, precision);
  for (const auto& d : cells) check_server(d[0], d[1], d[2]);
  if (fails) {
    std::printf("%d failures\n", fails);
    return 1;
  }
  std::printf("ok\n");
  return 0;
}
