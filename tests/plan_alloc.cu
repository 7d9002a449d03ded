// Host check of pme_setup with allocations that fail: csrc/k_pme.cu compiled
// with fakes of the runtime's allocation and copy calls, no device needed.
// For every allocation of a plan in turn: a call in which it fails says so,
// and the plan is not taken for complete by the next call, which lays it out
// anew; a plan of another grid that was there before does not stay half used.
#include <cstdio>
#include <cstdlib>
#include <map>

#include <cuda_runtime.h>

static int g_calls = 0, g_fail = -1;  // allocations so far, the one that fails
static std::map<void*, size_t> g_live;

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
#define cudaMalloc(p, n) fake_malloc(p, n)
#define cudaFree(p) fake_free(p)
#define cudaMemcpy(...) cudaSuccess
#define cudaFuncSetAttribute(...) cudaSuccess
#include "k_pme.cu"

int ctx_fail(orac_gpu_ctx*, int code, const char*, ...) { return code; }

static int check(bool ok, const char* what, int k) {
  if (!ok) printf("allocation %d: %s\n", k, what);
  return ok ? 0 : 1;
}

// every buffer there, of the grid's size
static bool whole(const PmePlan& P, int n1, int n2, int n3, bool saves) {
  const size_t ng = (size_t)n1 * n2 * n3, nc = (size_t)(n1 / 2 + 1) * n2 * n3;
  auto size = [](const void* p) { return p && g_live.count((void*)p) ? g_live[(void*)p] : (size_t)0; };
  return size(P.qfix) == 8 * ng && size(P.rgrid) == 4 * ng && size(P.cgrid) == 8 * nc &&
         (!saves || size(P.cgsave) == 8 * nc) && size(P.tw1) == sizeof(float2) * n1 &&
         size(P.tw2) == sizeof(float2) * n2 && size(P.tw3) == sizeof(float2) * n3 && size(P.bsp1) == 4u * n1 &&
         size(P.bsp2) == 4u * n2 && size(P.bsp3) == 4u * n3;
}

int main() {
  int bad = 0;
  for (int saves = 0; saves < 2; saves++) {
    int total = 0;
    for (int k = 0; k <= total; k++) {
      orac_gpu_ctx* ctx = new orac_gpu_ctx();
      g_fail = -1;
      bad += check(pme_setup(ctx, 16, 16, 16, 4) == ORAC_OK, "the first plan", k);
      if (saves) {
        bad += check(dev_alloc(ctx, &ctx->pme.cgsave, 9 * 16 * 16) == ORAC_OK, "the kept grid", k);
        ctx->pme.saves = true;
      }
      g_calls = 0;
      g_fail = k;
      const int rc = pme_setup(ctx, 20, 24, 18, 4);
      if (k == 0) {  // count them once: this one failed, so lay it out again
        g_fail = -1;
        g_calls = 0;
        bad += check(rc != ORAC_OK, "a failure passed over", k);
        bad += check(pme_setup(ctx, 20, 24, 18, 4) == ORAC_OK, "after a failure", k);
        total = g_calls - 1;
        bad += check(total >= 8, "fewer allocations than buffers", k);
      } else {
        bad += check(rc != ORAC_OK, "a failure passed over", k);
        bad += check(!ctx->pme.ready, "a half-built plan counts as complete", k);
        g_fail = -1;
        bad += check(pme_setup(ctx, 20, 24, 18, 4) == ORAC_OK, "after a failure", k);
      }
      bad += check(whole(ctx->pme, 20, 24, 18, saves), "buffers of the grid", k);
      bad += check(pme_setup(ctx, 20, 24, 18, 4) == ORAC_OK && whole(ctx->pme, 20, 24, 18, saves), "a second call", k);
      delete ctx;
    }
  }
  printf(bad ? "%d failed\n" : "ok\n", bad);
  return bad ? 1 : 0;
}
