// CPU check of a handle's device memory: otm::Homo::build on a CUDA runtime that only counts, linked with the
// library's own objects. A handle of its own takes one device allocation. Host code only; prints "ok".
#include <cstdio>

#include "otm_homo_impl.h"

// counting_runtime.cpp
extern int mallocs;
extern size_t malloc_bytes;

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

int main() {
  const int cells[][3] = {{8, 8, 8},    {9, 9, 9},    {18, 18, 18}, {20, 22, 18},  {32, 32, 32},   {36, 36, 36},
                          {40, 56, 72}, {64, 64, 64}, {96, 64, 48}, {96, 128, 64}, {128, 128, 128}, {256, 256, 256}};
  for (const auto& d : cells)
    for (int sweeps = 1; sweeps <= 2; sweeps++)
      for (int precision : {int(OTM_PRECISION_FP32), int(OTM_PRECISION_MIXED_BF16)})
        if (precision == OTM_PRECISION_FP32 || (d[0] >= 16 && d[0] % 4 == 0))
          check_handle(d[0], d[1], d[2], sweeps, precision);
  if (fails) {
    std::printf("%d failures\n", fails);
    return 1;
  }
  std::printf("ok\n");
  return 0;
}
