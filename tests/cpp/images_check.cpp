// Host build of the column bases.
#include "images.cuh"

extern "C" void images_check(const double* R, const double* A, int nx, int ny, float* pf, float* ps) {
  dsf Rs[3], As[9];
  float Rf[3], Af[9];
  for (int k = 0; k < 3; k++) Rf[k] = (Rs[k] = dsf_from(R[k])).hi;
  for (int k = 0; k < 9; k++) Af[k] = (As[k] = dsf_from(A[k])).hi;
  column_base_f(Rf, Af, nx, ny, pf);
  column_base_s(Rs, As, nx, ny, ps);
}
