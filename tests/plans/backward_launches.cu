// What fgms_b200_bwd launches, seen from the host: the runtime calls that the library makes to ask about the device and to
// launch are the ones below, which write down every grid.  Two tensor-core passes share the SMs; where a pointer sends one of them
// to the CUDA cores, the other one has all of them, and where SMs are to stay free neither pass is let go beside the other.
// Exit status 0 if all of that holds.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>
#include <cuda.h>
#include <cuda_runtime.h>
#include "../../include/fgms_b200.h"
#include "../../fgms_b200/csrc/common.cuh"

namespace {
constexpr int SMS = 148;
struct Launch { bool dgrad, beside, alone; int grid; };
std::vector<Launch> launches;
constexpr size_t OUT_GRAD = 1u << 30;  // where the output gradient lies
const char* base = reinterpret_cast<const char*>(1 << 20);

CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) { return CUDA_SUCCESS; }

void note(void** args, int grid) {
  // both parameter blocks begin with the rows they gather: the output gradient in the input gradient's, the features in the other's
  const char* rows;
  std::memcpy(&rows, args[0], sizeof(rows));
  Launch l = {rows >= base + OUT_GRAD && rows < base + OUT_GRAD + 64, false, false, grid};
  if (l.dgrad) {
    const auto* p = static_cast<const fgms::GmsParams*>(args[0]);
    l.beside = p->beside != 0, l.alone = p->alone != 0;
  } else {
    l.alone = static_cast<const fgms::WgradParams*>(args[0])->alone != 0;
  }
  launches.push_back(l);
}
}  // namespace

// under the library's names for them; the runtime's headers define some of these names in a .cu file themselves
#define STANDS_IN_FOR(name) __asm__(#name)
extern "C" {
cudaError_t get_device(int* dev) STANDS_IN_FOR(cudaGetDevice);
cudaError_t get_properties(cudaDeviceProp* p, int) STANDS_IN_FOR(cudaGetDeviceProperties_v2);
cudaError_t set_attribute(const void*, cudaFuncAttribute, int) STANDS_IN_FOR(cudaFuncSetAttribute);
cudaError_t occupancy(int* n, const void*, int, size_t, unsigned) STANDS_IN_FOR(cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags);
cudaError_t plain_occupancy(int* n, const void*, int, size_t) STANDS_IN_FOR(cudaOccupancyMaxActiveBlocksPerMultiprocessor);
cudaError_t last_error() STANDS_IN_FOR(cudaGetLastError);
cudaError_t entry_point(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* found) STANDS_IN_FOR(cudaGetDriverEntryPoint);
cudaError_t launch_ex(const cudaLaunchConfig_t* c, const void*, void** args) STANDS_IN_FOR(cudaLaunchKernelExC);
cudaError_t launch(const void*, dim3 grid, dim3, void** args, size_t, cudaStream_t) STANDS_IN_FOR(cudaLaunchKernel);

cudaError_t get_device(int* dev) { *dev = 0; return cudaSuccess; }
cudaError_t get_properties(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof(*p));
  p->multiProcessorCount = SMS;
  p->sharedMemPerBlockOptin = 232448;
  return cudaSuccess;
}
cudaError_t set_attribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t occupancy(int* n, const void*, int, size_t, unsigned) { *n = 1; return cudaSuccess; }
cudaError_t plain_occupancy(int* n, const void*, int, size_t) { *n = 1; return cudaSuccess; }
cudaError_t last_error() { return cudaSuccess; }
cudaError_t entry_point(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* found) {
  *fn = reinterpret_cast<void*>(encode);
  *found = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t launch_ex(const cudaLaunchConfig_t* c, const void*, void** args) { note(args, (int)c->gridDim.x); return cudaSuccess; }
cudaError_t launch(const void*, dim3 grid, dim3, void** args, size_t, cudaStream_t) { note(args, (int)grid.x); return cudaSuccess; }
}

// pointer `off` (0: none; 1 .. 5: output gradient, features, weights, input gradient, weight gradient) begins 4 bytes further on
static bool backward(int off, int c_in, int c_out, int pairs, bool f16) {
  launches.clear();
  auto at = [&](size_t where, int which) { return const_cast<char*>(base + where + (off == which ? 4 : 0)); };
  const int32_t* maps = reinterpret_cast<const int32_t*>(base + (6u << 28));
  const int rc = fgms_b200_bwd(at(OUT_GRAD, 1), at(0, 2), at(2u << 28, 3), at(3u << 28, 4), at((3ull << 28) + (1u << 27), 5), maps, nullptr, maps + 64,
                               maps + 64 + pairs, pairs, 30000, 30000, c_in, c_in, c_out, 27, 0, f16 ? FGMS_DTYPE_F16 : FGMS_DTYPE_F32,
                               f16 ? FGMS_MATH_F16 : FGMS_MATH_TF32, 0, nullptr, 0, nullptr);
  if (rc != 0) std::printf("status %d: %s\n", rc, fgms_b200_last_error());
  return rc == 0;
}

int main() {
  int bad = 0;
  auto expect = [&](bool ok, const std::string& what) {
    if (ok) return;
    ++bad;
    std::printf("%s:", what.c_str());
    for (const Launch& l : launches) std::printf(" %s %d%s", l.dgrad ? "input gradient" : "weight gradient", l.grid, l.beside ? " beside" : "");
    std::printf("\n");
  };
  struct { int c_in, c_out, pairs; bool f16; } shapes[] = {{64, 64, 930000, true}, {128, 128, 303000, true}, {48, 80, 300000, false}};
  for (const auto& s : shapes) {
    const std::string name = std::string(s.f16 ? "fp16 " : "tf32 ") + std::to_string(s.c_in) + " -> " + std::to_string(s.c_out);
    for (int off = 0; off <= 5; ++off) {
      if (s.f16 && (off == 1 || off == 2 || off == 5)) continue;  // refused: the single-launch weight gradient wants aligned tensors
      if (!backward(off, s.c_in, s.c_out, s.pairs, s.f16)) { ++bad; continue; }
      bool two = launches.size() == 2 && launches[0].dgrad != launches[1].dgrad;
      expect(two, name + ", two launches");
      if (!two) continue;
      if (off == 0) {
        expect(launches[0].grid + launches[1].grid <= SMS && launches[1].beside, name + ", a share each");
      } else {
        for (const Launch& l : launches)
          expect(l.grid >= SMS, name + ", pointer " + std::to_string(off) + " not aligned");
      }
    }
    fgms_b200_set_reserved_sms(16);
    if (backward(0, s.c_in, s.c_out, s.pairs, s.f16))
      for (const Launch& l : launches) expect(l.grid <= SMS - 16 && !l.beside && l.alone, name + ", 16 SMs to stay free");
    fgms_b200_set_reserved_sms(0);
  }
  std::printf("%d violations\n", bad);
  return bad ? 1 : 0;
}
