// rsd_smem against a fake runtime: which (device, kernel) pairs were granted
// dynamic shared memory, and what a refused call leaves behind.
#include <math.h>

#include <set>
#include <string>
#include <utility>

#include "rsd_internal.cuh"

static int g_device = 0, g_calls = 0, g_refuse = 0;
static std::set<std::pair<int, const void*>> g_granted;

extern "C" cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int bytes) {
  g_calls++;
  if (g_refuse || a != cudaFuncAttributeMaxDynamicSharedMemorySize || bytes <= 0) return cudaErrorInvalidValue;
  g_granted.insert({g_device, f});
  return cudaSuccess;
}
int rsd_cuda_check(rsd_ctx*, cudaError_t e, const char*) { return e == cudaSuccess ? RSD_OK : RSD_ECUDA; }
int rsd_fail(rsd_ctx*, int code, const char*, ...) { return code; }

static void kernel_a(int) {}
static void kernel_b(float*, int) {}

// 0, or the number of the step that went wrong
extern "C" int smem_check() {
  rsd_ctx c[2];
  c[1].device = 1;
  for (int round = 0; round < 2; round++)
    for (int d = 0; d < 2; d++) {
      g_device = d;
      if (rsd_smem(&c[d], kernel_a, 64 << 10) != RSD_OK || rsd_smem(&c[d], kernel_b, 64 << 10) != RSD_OK) return 1;
      if (!g_granted.count({d, (const void*)kernel_a}) || !g_granted.count({d, (const void*)kernel_b})) return 2;
    }
  if (g_calls != 4) return 3;  // once per context and kernel
  rsd_ctx e;
  g_refuse = 1;
  if (rsd_smem(&e, kernel_a, 64 << 10) == RSD_OK) return 4;
  g_refuse = 0;
  if (rsd_smem(&e, kernel_a, 64 << 10) != RSD_OK || g_calls != 6) return 5;  // a refusal is not remembered as a grant
  return 0;
}
