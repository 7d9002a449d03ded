// pme_setup with allocations that fail: for every allocation of a plan in turn,
// a call in which it fails says so, and the plan is not taken for complete by
// the next call, which lays it out anew; a plan of another grid that was there
// before does not stay half used, nor is its kept grid lost.
#include "alloc_fakes.h"
#include "k_pme.cu"

int ctx_fail(orac_gpu_ctx*, int code, const char*, ...) { return code; }

// every buffer there, of the grid's size
static bool whole(const PmePlan& P, int n1, int n2, int n3, bool saves) {
  const size_t ng = (size_t)n1 * n2 * n3, nc = (size_t)(n1 / 2 + 1) * n2 * n3;
  return live_size(P.qfix) == 8 * ng && live_size(P.rgrid) == 4 * ng && live_size(P.cgrid) == 8 * nc &&
         (!saves || live_size(P.cgsave) == 8 * nc) && live_size(P.tw1) == sizeof(float2) * n1 &&
         live_size(P.tw2) == sizeof(float2) * n2 && live_size(P.tw3) == sizeof(float2) * n3 &&
         live_size(P.bsp1) == 4u * n1 && live_size(P.bsp2) == 4u * n2 && live_size(P.bsp3) == 4u * n3;
}

int main() {
  int bad = 0;
  for (int saves = 0; saves < 2; saves++) {
    const int total = 9 + saves;  // three twiddle tables, three moduli, three grids, the kept one
    for (int k = 0; k < total; k++) {
      orac_gpu_ctx* ctx = new orac_gpu_ctx();
      PmePlan& P = ctx->pme;
      g_fail = -1;
      bad += check(pme_setup(ctx, 16, 16, 16, 4) == ORAC_OK, "the first plan", k);
      if (saves) {
        bad += check(dev_alloc(ctx, &P.cgsave, 9 * 16 * 16) == ORAC_OK, "the kept grid", k);
        P.saves = true;
      }
      g_calls = 0;
      g_fail = k;
      bad += check(pme_setup(ctx, 20, 24, 18, 4) != ORAC_OK, "a failure passed over", k);
      bad += check(!P.ready, "a half-built plan counts as complete", k);
      g_calls = 0;
      g_fail = -1;
      bad += check(pme_setup(ctx, 20, 24, 18, 4) == ORAC_OK && P.ready, "after a failure", k);
      bad += check(whole(P, 20, 24, 18, saves), "buffers of the grid", k);
      bad += check(g_calls == total, "the number of allocations", k);
      bad += check(pme_setup(ctx, 20, 24, 18, 4) == ORAC_OK && g_calls == total, "a second call", k);
      delete ctx;
    }
  }
  printf(bad ? "%d failed\n" : "ok\n", bad);
  return bad ? 1 : 0;
}
