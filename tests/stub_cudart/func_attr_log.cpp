// Test infrastructure only: the stand-in CUDA runtime (stub_cudart.cpp) with the
// dynamic shared-memory limits of kernels recorded. The limit is a property of the
// function, shared by every thread of the process.
#include <cuda_runtime_api.h>

#define cudaFuncSetAttribute stub_ignored_func_set_attribute
#include "stub_cudart.cpp"
#undef cudaFuncSetAttribute

#include <set>

namespace {
std::map<const void *, std::set<int>> &smem_limits() {
  static std::map<const void *, std::set<int>> m;
  return m;
}
}  // namespace

cudaError_t cudaFuncSetAttribute(const void *fn, cudaFuncAttribute attr, int value) {
  std::lock_guard<std::mutex> lock(g_mu);
  if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) smem_limits()[fn].insert(value);
  return cudaSuccess;
}

extern "C" {
// Kernels whose limit was set, and the most values that one of them was given.
int stub_cudart_limited_kernels() { return (int)smem_limits().size(); }
int stub_cudart_limits_of_one_kernel() {
  size_t most = 0;
  for (const auto &x : smem_limits()) most = x.second.size() > most ? x.second.size() : most;
  return (int)most;
}
}
