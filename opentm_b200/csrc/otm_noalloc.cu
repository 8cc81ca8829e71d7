// otm_noalloc.cu -- the OC sensitivity filter without any device allocation.
//
// For callers that cannot allocate GPU memory while they run (their allocator already owns the
// device's memory, or a cudaMalloc/cudaFree with its possible device-wide synchronisation is
// not allowed in their loop). The filter's products s rho live in `g_noalloc_scratch`, a
// file-scope device array of OTM_NOALLOC_MAX_CELLS floats that every GPU loading the library
// holds until the process exits. In host code that symbol is only a host-side stand-in, never
// a device address: its device address is looked up once per device with
// cudaGetSymbolAddress while that device is current, and that pointer is what the kernels
// get. Calls share the array, so calls whose GPU work overlaps race on it.
#include <cuda_runtime.h>

#include <mutex>

#include "opentm_b200_noalloc.h"
#include "otm_common.cuh"

namespace otm {

static __device__ __align__(256) float g_noalloc_scratch[OTM_NOALLOC_MAX_CELLS];

constexpr int kNaMaxDevices = 64;
static float* g_scratch_ptr[kNaMaxDevices] = {};
static std::mutex g_scratch_mu;

// Device address of the scratch array on the current device (looked up on first use).
static otm_status scratch_address(float** out) {
  int dev = 0;
  OTM_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNaMaxDevices) {
    set_error("device ordinal out of range for the allocation-free filter");
    return OTM_ERR_UNSUPPORTED;
  }
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
    g_scratch_ptr[dev] = static_cast<float*>(p);
  }
  *out = g_scratch_ptr[dev];
  return OTM_OK;
}

constexpr int kNaMaxHalf = 6;

}  // namespace otm

using namespace otm;

extern "C" otm_status otm_oc_filter_sens_noalloc(float* sens, const float* rho, size_t pitchT, const int reso[3],
                                                 float radius, void* stream) {
  if (!sens || !rho || !reso || reso[0] < 1 || reso[1] < 1 || reso[2] < 1) return OTM_ERR_INVALID_ARGUMENT;
  const Dims d{reso[0], reso[1], reso[2]};
  if (d.nv() > size_t(OTM_NOALLOC_MAX_CELLS)) {
    set_error("the allocation-free filter accepts at most OTM_NOALLOC_MAX_CELLS (2^21 = 128^3) voxels");
    return OTM_ERR_UNSUPPORTED;
  }
  if (pitchT == 0) pitchT = size_t(d.nx);
  if (pitchT < size_t(d.nx)) return OTM_ERR_INVALID_ARGUMENT;
  const int h = int(radius + 0.5f);
  if (!(radius > 0.f) || h > kNaMaxHalf) {
    set_error("filter radius must be in (0, 6.5)");
    return OTM_ERR_INVALID_ARGUMENT;
  }
  float* scratch = nullptr;
  OTM_TRY(scratch_address(&scratch));
  return oc_filter_run(d, sens, rho, pitchT, scratch, radius, (cudaStream_t)stream);
}
