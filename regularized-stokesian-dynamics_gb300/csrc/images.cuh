// Column bases p = R + nx a1 + ny a2 of a pair's images p + nz a3 in FP32; a1, a2,
// a3 are the columns of A.  Also compiles as host C++ (see dsf.cuh).
#pragma once
#include "dsf.cuh"

// from R and A rounded to FP32: the sequence that sorts the images into near and
// far ones, the same for both sets
DSF_FN void column_base_f(const float* R, const float* A, int nx, int ny, float* p) {
  for (int k = 0; k < 3; k++) p[k] = DSF_FMA(A[3 + k], (float)ny, DSF_FMA(A[k], (float)nx, R[k]));
}

// from double-single R and A, rounded once
DSF_FN void column_base_s(const dsf* R, const dsf* A, int nx, int ny, float* p) {
  for (int k = 0; k < 3; k++) p[k] = (R[k] + nx * A[k] + ny * A[3 + k]).hi;
}
