// Cooperative launches with as many CTAs as the process may have resident.
#pragma once
#include <cuda_runtime.h>

// Calls launch(grid) and, as long as the grid is refused as too large to be
// resident at once, again with half of it: a process given part of the GPU's
// SMs (a limited share, a partition) holds fewer CTAs than the device has SMs.
// grid ends as the one taken.
template <typename F>
cudaError_t rsd_coop_launch(int* grid, F launch) {
  for (;;) {
    const cudaError_t e = launch(*grid);
    if (e != cudaErrorCooperativeLaunchTooLarge || *grid <= 1) return e;
    cudaGetLastError();
    *grid /= 2;
  }
}
