// The lists' growth with allocations that fail: the H list and the two that
// nest in its rows take the new capacity together or not at all, so a later
// build grows them again before any kernel writes.
#include "alloc_fakes.h"
static long long g_total = 0;  // what a build finds
#define cudaMemcpyAsync(dst, ...) (*(long long*)(dst) = g_total, cudaSuccess)
#include "k_list.cu"

int ctx_fail(orac_gpu_ctx*, int code, const char*, ...) { return code; }

static bool whole(const orac_gpu_ctx* c, long long least) {
  for (const GList& L : c->lists)
    if (L.cap < least || live_size(L.j) != 4u * L.cap || live_size(L.mask) != 8u * L.cap) return false;
  return true;
}

int main() {
  int bad = 0;
  for (int k = 0; k < 6; k++) {
    orac_gpu_ctx* ctx = new orac_gpu_ctx();
    ctx->G = 8;
    g_fail = -1;
    g_total = 100;
    bad += check(list_build_allpairs(ctx, 9.0, &ctx->lists[0]) == ORAC_OK && whole(ctx, 100), "the first build", k);
    g_total = 50000;
    g_calls = 0;
    g_fail = k;
    bad += check(list_build_allpairs(ctx, 9.0, &ctx->lists[0]) != ORAC_OK, "a failure passed over", k);
    bad += check(!ctx->lists[0].valid, "a list without room counts as built", k);
    g_fail = -1;
    for (long long n : {100ll, 50000ll}) {
      g_total = n;
      bad += check(list_build_allpairs(ctx, 9.0, &ctx->lists[0]) == ORAC_OK, "after a failure", k);
      bad += check(whole(ctx, n) && ctx->lists[0].valid, "room in the three lists", k);
    }
    delete ctx;
  }
  printf(bad ? "%d failed\n" : "ok\n", bad);
  return bad ? 1 : 0;
}
