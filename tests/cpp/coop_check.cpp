// rsd_coop_launch against a fake runtime that holds `room` CTAs.
#include "coop.cuh"

static cudaError_t g_last = cudaSuccess;
extern "C" cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}

// the grid taken from `grid` on with `room` CTAs to be had, or -1; *launched: whether it ran,
// *left: the error left behind; other != 0: the launch fails with that instead
extern "C" int coop_check(int grid, int room, int other, int* launched, int* left) {
  *launched = 0;
  g_last = cudaSuccess;
  const cudaError_t e = rsd_coop_launch(&grid, [&](int g) {
    const cudaError_t r = other ? (cudaError_t)other : (g > room ? cudaErrorCooperativeLaunchTooLarge : cudaSuccess);
    g_last = r;
    *launched += r == cudaSuccess;
    return r;
  });
  *left = (int)g_last;
  return e == cudaSuccess ? grid : -(int)e;
}
