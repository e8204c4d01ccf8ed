// Host-side check of weight_tensor_map where the driver does not do its part at once.  The runtime calls it makes and the
// encoder are replaced by the ones below: the first lookup finds nothing, the second an encoder that wants a context until the
// device is set, later a rejected map.  Exit status 0: the failed lookup is not kept, the device is set once and the
// driver's status comes back.
#include <cstdio>
#include <cuda.h>
#include <cuda_runtime.h>

static int lookups = 0, sets = 0, encodes = 0;
static CUresult answer = CUDA_SUCCESS;

static CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                       CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  ++encodes;
  return sets == 0 ? CUDA_ERROR_INVALID_CONTEXT : answer;
}
static cudaError_t entry_point(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* found) {
  *fn = ++lookups == 1 ? nullptr : reinterpret_cast<void*>(encode);
  *found = lookups == 1 ? cudaDriverEntryPointSymbolNotFound : cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
static cudaError_t get_device(int* dev) { *dev = 3; return cudaSuccess; }
static cudaError_t set_device(int dev) { sets += dev == 3; return cudaSuccess; }

#define cudaGetDriverEntryPoint entry_point
#define cudaGetDevice get_device
#define cudaSetDevice set_device
#include "../../fgms_b200/csrc/umma.cuh"

int main() {
  CUtensorMap map;
  int rc[4];
  for (int i = 0; i < 4; ++i) {
    if (i == 2) answer = CUDA_ERROR_INVALID_VALUE;
    if (i == 3) answer = CUDA_SUCCESS;
    rc[i] = fgms::weight_tensor_map(&map, nullptr, 27, 64, 64, true, true);
  }
  std::printf("status %d %d %d %d, %d lookups, device set %d times, %d encodes\n", rc[0], rc[1], rc[2], rc[3], lookups, sets, encodes);
  return rc[0] == -1000 - CUDA_ERROR_NOT_FOUND && rc[1] == 0 && rc[2] == -1000 - CUDA_ERROR_INVALID_VALUE && rc[3] == 0 && lookups == 2 && sets == 1 &&
         encodes == 4 ? 0 : 1;
}
