// Fakes of the runtime's calls for host checks of allocations that fail: the
// g_fail-th allocation gives an error, the others a few bytes and a record of
// the size asked for; copies and launches do nothing.
#pragma once
#include <cstdio>
#include <cstdlib>
#include <map>

#include <cuda_runtime.h>

static int g_calls = 0, g_fail = -1;  // allocations so far, the one that fails
static std::map<const void*, size_t> g_live;

template <typename T>
static cudaError_t fake_malloc(T** p, size_t n) {
  if (g_calls++ == g_fail) return cudaErrorMemoryAllocation;
  *p = (T*)malloc(16);
  g_live[(void*)*p] = n;
  return cudaSuccess;
}
static cudaError_t fake_free(void* p) {
  g_live.erase(p);
  free(p);
  return cudaSuccess;
}
static size_t live_size(const void* p) { return p && g_live.count(p) ? g_live[p] : 0; }

static int check(bool ok, const char* what, int k) {
  if (!ok) printf("allocation %d: %s\n", k, what);
  return ok ? 0 : 1;
}

#define cudaMalloc(p, n) fake_malloc(p, n)
#define cudaFree(p) fake_free(p)
#define cudaMemcpy(...) cudaSuccess
#define cudaMemsetAsync(...) cudaSuccess
#define cudaStreamSynchronize(...) cudaSuccess
#define cudaFuncSetAttribute(...) cudaSuccess
#define cudaLaunchKernelEx(...) cudaSuccess
#define cudaGetLastError() cudaSuccess
