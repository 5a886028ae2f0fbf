// Launches of the step's host code on pretended devices, for tests that run
// without a GPU: the CUDA runtime calls of libjgs2.so that a launch makes are
// answered here (an executable's symbols come before a library's).  Kernels
// are recorded, not run, and a launch is refused as a device would refuse it
// when its dynamic shared memory was not allowed for that kernel on the current
// device.  Usage: fake_cudart < script; every line of the script is
//   device N | sms N | solve count K jacobi cloth contacts listed shift
//   | sweep K cloth | convergence vertices cloth | prologue vertices cloth
// and every launch answers with one line: status, kernel, device, grid, block,
// dynamic shared memory.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <iostream>
#include <map>
#include <set>
#include <sstream>
#include <string>
#include <utility>
#include <vector>

#include "jgs2_kernels.cuh"

namespace {
int device = 0, sms = 148;
constexpr size_t kOptIn = 232448, kPerSm = 233472, kDefault = 48 * 1024;
std::map<const void*, std::string>& names() {
  static std::map<const void*, std::string> m;
  return m;
}
std::map<std::pair<int, const void*>, size_t> allowed;
struct Config {
  dim3 grid, block;
  size_t shared;
  cudaStream_t stream;
};
std::vector<Config> pending;

cudaError_t record(const void* fn, dim3 grid, dim3 block, size_t shared) {
  const auto it = allowed.find({device, fn});
  const bool ok = shared <= (it == allowed.end() ? kDefault : it->second);
  std::printf("%s %s %d %u %u %zu\n", ok ? "ok" : "refused", names()[fn].c_str(), device, grid.x, block.x, shared);
  return ok ? cudaSuccess : cudaErrorInvalidValue;
}
}  // namespace

extern "C" {
void** __cudaRegisterFatBinary(void*) {
  static void* handle = nullptr;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, cudaStream_t stream) {
  pending.push_back({grid, block, shared, stream});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, void* stream) {
  const Config c = pending.back();
  pending.pop_back();
  *grid = c.grid;
  *block = c.block;
  *shared = c.shared;
  *static_cast<cudaStream_t*>(stream) = c.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 grid, dim3 block, void**, size_t shared, cudaStream_t) {
  return record(fn, grid, block, shared);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void**) {
  return record(fn, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
cudaError_t cudaGetDevice(int* out) {
  *out = device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* out, cudaDeviceAttr a, int) {
  switch (a) {
    case cudaDevAttrMaxSharedMemoryPerBlockOptin: *out = static_cast<int>(kOptIn); return cudaSuccess;
    case cudaDevAttrMaxSharedMemoryPerMultiprocessor: *out = static_cast<int>(kPerSm); return cudaSuccess;
    case cudaDevAttrReservedSharedMemoryPerBlock: *out = 1024; return cudaSuccess;
    case cudaDevAttrMultiProcessorCount: *out = sms; return cudaSuccess;
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute a, int value) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize || value < 0 || size_t(value) > kOptIn)
    return cudaErrorInvalidValue;
  allowed[{device, fn}] = static_cast<size_t>(value);
  return cudaSuccess;
}
// A kernel whose shared memory is not allowed has no resident block.
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* blocks, const void* fn, int, size_t shared) {
  const auto it = allowed.find({device, fn});
  *blocks = shared <= (it == allowed.end() ? kDefault : it->second) ? 1 : 0;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
}

int main() {
  std::string line;
  while (std::getline(std::cin, line)) {
    std::istringstream in(line);
    std::string what;
    in >> what;
    jgs2::Buffers b;
    std::memset(&b, 0, sizeof(b));
    // Never read through: the launches only look at whether they are there.
    static uint4 some[1];
    if (what == "device") {
      in >> device;
    } else if (what == "sms") {
      in >> sms;
    } else if (what == "solve") {
      uint32_t count = 0, K = 0, jacobi = 0, cloth = 0, contacts = 0, listed = 0, shift = 0;
      in >> count >> K >> jacobi >> cloth >> contacts >> listed >> shift;
      static uint32_t list[1];
      if (cloth) b.clothRange = some;
      if (contacts) b.contactIdx = some;
      b.contactCount = contacts;
      b.vertexTotal = count;
      b.solveShift = shift;
      jgs2::launchSolve(b, nullptr, nullptr, nullptr, listed ? list : nullptr, count, K, jacobi != 0, nullptr);
    } else if (what == "sweep") {
      uint32_t K = 0, cloth = 0;
      in >> K >> cloth;
      if (cloth) b.clothRange = some;
      uint32_t barrier[16] = {};
      const int n = jgs2::launchColoredSweep(b, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 2, 60, K, 30, 40,
                                             true, barrier, 1u << 10, nullptr);
      if (n < 0) std::printf("declined\n");
    } else if (what == "convergence" || what == "prologue") {
      uint32_t V = 0, cloth = 0;
      in >> V >> cloth;
      if (cloth) b.clothRange = some;
      b.vertexTotal = V;
      b.convBlocks = (V + jgs2::kConvChunk - 1) / jgs2::kConvChunk;
      if (what == "convergence") jgs2::launchConvergence(b, nullptr, nullptr, nullptr, true, nullptr);
      else jgs2::launchPrologue(b, nullptr, nullptr);
    }
  }
  return 0;
}
