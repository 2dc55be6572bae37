// Kernel 1: Ewald-summed periodic grand mobility (PER_GRPERY_INV_FRI,
// src/per_GRPY_YZD.f90:13-200, with PER_ROTNE_PRAGER_SELF/IJ of
// src/Ewald_summation.f90:19-423).
//
// Layout: the grand mobility M (11N x 11N, column-major, leading dimension
// ldm) in the reference's order: rows/cols 3a..3a+2 translation of particle
// a, 3N+3a.. rotation, 6N+5a.. stresslet (Y2 basis).
//
// Work split:
//   ewald_weights     per reciprocal vector k (half space k > 0): the weights
//                     of the pair sums, in the layout [weight][vector]
//   ewald_trig        per (particle, k): cos(k.x_a), sin(k.x_a), so that
//                     cos(k.R_ab) = c_a c_b + s_a s_b needs no sincos per pair
//   ewald_pair64      FP64 form, a group of lanes per pair a < b: real-space
//                     and reciprocal sums and the epilogue, both 11x11 blocks
//                     of the pair written once
//   ewald_pair_*      mixed form, a thread per pair (below)
//   ewald_self_sums, ewald_self*  the diagonal blocks (images n != 0, k != 0
//                     and the analytic terms of PER_ROTNE_PRAGER_SELF 179-188)
// The closed forms come from ewald_gen.cuh (generated by gen_ewald.py).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "ewald_gen.cuh"
#include "overlap.cuh"
#include "dsf.cuh"
#include "f32x2.cuh"
#include "images.cuh"
#include "pdl.cuh"
#include "rsd_internal.cuh"

namespace {

constexpr int KW = 3 + RSD_NMOM_KCOS + RSD_NMOM_KSIN;  // doubles per k entry

__host__ __device__ inline void half_space_index(int h, int NI, int* nx, int* ny, int* nz) {
  const int w = 2 * NI + 1;
  const int q = (w * w * w - 1) / 2 + 1 + h;  // entries after the origin
  *nx = q / (w * w) - NI;
  *ny = (q / w) % w - NI;
  *nz = q % w - NI;
}

// outputs (gen_ewald.py's order) that the sin sums feed: TR and G
__host__ __device__ constexpr bool kblock_is_sin(int q) { return (q >= 12 && q < 15) || (q >= 30 && q < 45); }

// S(k) of F_Jk (Ewald_summation.f90:1067-1071): F_Jk = S (delta k^2 - k k)
template <typename T>
__device__ inline T kernel_S(T k2, T lam) {
  const T l2 = lam * lam;
  return T(8.0 * RSD_PI) * (T(1) + k2 / (T(4) * l2) + k2 * k2 / (T(8) * l2 * l2)) * exp(-k2 / (T(4) * l2)) / (k2 * k2);
}

// Weights of the listed half-space vectors (kv: 3 doubles each), W[q * Kh + h]:
// with equal radii (EQ) the 60 block weights -- the epilogue of the moment
// weights for the common radius a, scaled like the block (ewald_kblock_list);
// otherwise the 80 moment weights (cos, then sin).  blockIdx.y = 0 forms the
// cos part, 1 the sin part: one warp issues an FP64 instruction every 64
// cycles here, so a thread's instruction count is the kernel's time.
template <bool EQ>
__global__ void ewald_weights(rsd_lat_dev L, int Kh, const double* __restrict__ kv, double a, double inv_pimu,
                              double* __restrict__ W) {
  pdl_enter();
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= Kh) return;
  const double k0 = kv[3 * h], k1 = kv[3 * h + 1], k2v = kv[3 * h + 2];
  const double S = kernel_S<double>(k0 * k0 + k1 * k1 + k2v * k2v, L.lam);
  const double f = 2.0 / L.LV, na = f * inv_pimu / (6.0 * a), na3 = na / (a * a);  // EQ: half space counted twice
  double w[RSD_NMOM_KCOS], v[60];
  if (blockIdx.y == 0) {
    rsd_kcos_weights<double>(k0, k1, k2v, S, L.lam, w);
    if (EQ) {
      rsd_kcos_epilogue<double>(w, a, a, L.phix, v);
#pragma unroll
      for (int q = 0; q < 60; q++) {
        const bool a3 = (q >= 6 && q < 12) || (q >= 15 && q < 30) || q >= 45;
        if (!kblock_is_sin(q)) W[(size_t)q * Kh + h] = v[q] * (a3 ? na3 : na);
      }
    } else {
#pragma unroll
      for (int m = 0; m < RSD_NMOM_KCOS; m++) W[(size_t)m * Kh + h] = w[m];
    }
  } else {
    rsd_ksin_weights<double>(k0, k1, k2v, S, L.lam, w);
    if (EQ) {
      rsd_ksin_epilogue<double>(w, a, a, L.phix, v);
#pragma unroll
      for (int q = 0; q < 60; q++)
        if (kblock_is_sin(q)) W[(size_t)q * Kh + h] = v[q] * na;  // TR and G
    } else {
#pragma unroll
      for (int m = 0; m < RSD_NMOM_KSIN; m++) W[(size_t)(RSD_NMOM_KCOS + m) * Kh + h] = w[m];
    }
  }
}

// cs[a * Kh + h] = (cos, sin)(k_h . x_a)
__global__ void ewald_trig(int nn, int Kh, const double* __restrict__ kv, const double* __restrict__ pos,
                           double2* __restrict__ cs) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)nn * Kh) return;
  const int a = (int)(t / Kh), h = (int)(t % Kh);
  double s, c;
  sincos(kv[3 * h] * pos[3 * a] + kv[3 * h + 1] * pos[3 * a + 1] + kv[3 * h + 2] * pos[3 * a + 2], &s, &c);
  cs[t] = make_double2(c, s);
}

// Weights and trig tables restricted to a list of half-space indices, in
// precision T (the mixed form splits the reciprocal sum by shell).
template <typename T>
__global__ void ewald_ktable_list(rsd_lat_dev L, int count, const int* __restrict__ hlist, T* __restrict__ tab) {
  pdl_enter();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= count) return;
  int nx, ny, nz;
  half_space_index(hlist[q], L.NI, &nx, &ny, &nz);
  double k[3];
  for (int j = 0; j < 3; j++)
    k[j] = 2.0 * RSD_PI * (nx * L.LI[0 + 3 * j] + ny * L.LI[1 + 3 * j] + nz * L.LI[2 + 3 * j]);
  const double k2 = k[0] * k[0] + k[1] * k[1] + k[2] * k[2];
  const double S = kernel_S<double>(k2, L.lam);
  double wc[RSD_NMOM_KCOS], ws[RSD_NMOM_KSIN];
  rsd_kcos_weights<double>(k[0], k[1], k[2], S, L.lam, wc);
  rsd_ksin_weights<double>(k[0], k[1], k[2], S, L.lam, ws);
  T* e = tab + (size_t)q * KW;
  e[0] = (T)k[0];
  e[1] = (T)k[1];
  e[2] = (T)k[2];
  for (int m = 0; m < RSD_NMOM_KCOS; m++) e[3 + m] = (T)wc[m];
  for (int m = 0; m < RSD_NMOM_KSIN; m++) e[3 + RSD_NMOM_KCOS + m] = (T)ws[m];
}

__device__ __forceinline__ void put_trig(float2* p, double c, double sn) { *p = make_float2((float)c, (float)sn); }
__device__ __forceinline__ void put_trig(float4* p, double c, double sn) {
  const dsf dc = dsf_from(c), ds = dsf_from(sn);
  *p = make_float4(dc.hi, dc.lo, ds.hi, ds.lo);
}

template <typename T2>
__global__ void ewald_trig_list(int nn, rsd_lat_dev L, const int* __restrict__ hlist, const double* __restrict__ pos,
                                T2* __restrict__ cs) {
  pdl_enter();
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  const int q = blockIdx.y;
  if (a >= nn) return;
  int nx, ny, nz;
  half_space_index(hlist[q], L.NI, &nx, &ny, &nz);
  double k[3];
  for (int j = 0; j < 3; j++)
    k[j] = 2.0 * RSD_PI * (nx * L.LI[0 + 3 * j] + ny * L.LI[1 + 3 * j] + nz * L.LI[2 + 3 * j]);
  const double kr = k[0] * pos[3 * a] + k[1] * pos[3 * a + 1] + k[2] * pos[3 * a + 2];
  double sn, c;
  sincos(kr, &sn, &c);
  put_trig(cs + (size_t)q * nn + a, c, sn);
}

// Scatter of the pair block (a,b), a < b, and its mirror (b,a) with
// b -> -b, g -> -g (per_GRPY_YZD.f90:123-151,160-188).  v holds the 60
// unique values (order of gen_ewald.py) already scaled; add != 0 adds.
// Destinations of the pair blocks.  DenseSink: the FP64 grand mobility
// (column-major, ld).  PlaneSink: the mixed form's grand mobility as two
// FP32 planes, M = hi + lo with |lo| <= ulp(hi)/2 (~48 bits, the precision
// the mixed assembly computes in), read by the FP32 factorisation (hi) and
// by the double-single residual products of the refinement (both).
// put<K> stores (add = 0) or read-modify-writes (add = 1) K entries; all K
// loads are issued before the first store, so a thread waits for one memory
// round trip per group rather than one per entry (the offsets of a group are
// distinct).
struct DenseSink {
  double* M;
  int64_t ld;
  template <int K>
  __device__ __forceinline__ void put(const int64_t* o, const double* x, int add) const {
    if (add) {
      double v[K];
#pragma unroll
      for (int i = 0; i < K; i++) v[i] = M[o[i]];
#pragma unroll
      for (int i = 0; i < K; i++) M[o[i]] = v[i] + x[i];
    } else {
#pragma unroll
      for (int i = 0; i < K; i++) M[o[i]] = x[i];
    }
  }
};

struct PlaneSink {
  float* hi;
  float* lo;
  int64_t ld;
  template <int K>
  __device__ __forceinline__ void put(const int64_t* o, const dsf* x, int add) const {
    if (add) {
      float h[K], l[K];
#pragma unroll
      for (int i = 0; i < K; i++) {
        h[i] = hi[o[i]];
        l[i] = lo[o[i]];
      }
#pragma unroll
      for (int i = 0; i < K; i++) {
        const dsf v = dsf(h[i], l[i]) + x[i];
        hi[o[i]] = v.hi;
        lo[o[i]] = v.lo;
      }
    } else {
#pragma unroll
      for (int i = 0; i < K; i++) {
        hi[o[i]] = x[i].hi;
        lo[o[i]] = x[i].lo;
      }
    }
  }
};

// Writes the pair blocks (a, b) and (b, a), a != b, of the grand mobility
// from the 60 values of a pair (TT 0-5, RR 6-11, TR 12-14, QQ 15-29, G
// 30-44, H 45-59), in 14 groups of at most 25 entries.  V: double
// (DenseSink) or dsf (PlaneSink).
template <typename V, typename S>
__device__ inline void store_pair_t(const S& sk, int N, int a, int b, const V* v, int add) {
  auto at = [&](int r, int c) { return (int64_t)r + (int64_t)c * sk.ld; };
  constexpr int sym[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
  // TT and RR, both orders
#pragma unroll
  for (int blk = 0; blk < 2; blk++) {
    const int o = blk ? 3 * N : 0;
    int64_t p[18];
    V x[18];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const V t = v[6 * blk + sym[i][j]];
        p[6 * i + 2 * j] = at(o + 3 * a + i, o + 3 * b + j);
        p[6 * i + 2 * j + 1] = at(o + 3 * b + i, o + 3 * a + j);
        x[6 * i + 2 * j] = x[6 * i + 2 * j + 1] = t;
      }
    sk.template put<18>(p, x, add);
  }
  // TR: translation of one particle against rotation of the other, both
  // placements (upper and lower triangle) of each
#pragma unroll
  for (int side = 0; side < 2; side++) {
    const int t = side ? b : a, r = side ? a : b;
    int64_t p[18];
    V x[18];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        V tr = V(0);
        if (i < j) tr = v[12 + (i == 0 ? j - 1 : 2)];
        if (i > j) tr = -v[12 + (j == 0 ? i - 1 : 2)];
        if (side) tr = -tr;
        p[6 * i + 2 * j] = at(3 * t + i, 3 * N + 3 * r + j);
        p[6 * i + 2 * j + 1] = at(3 * N + 3 * r + j, 3 * t + i);
        x[6 * i + 2 * j] = x[6 * i + 2 * j + 1] = tr;
      }
    sk.template put<18>(p, x, add);
  }
  // G (translation-stresslet, odd under a <-> b) and H (rotation-stresslet)
#pragma unroll
  for (int grp = 0; grp < 8; grp++) {
    const int side = grp >> 2, h = (grp >> 1) & 1, lower = grp & 1;
    const int u = side ? b : a, sp = side ? a : b;  // velocity row particle, stresslet column particle
    const int ro = h ? 3 * N : 0;
    int64_t p[15];
    V x[15];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int m = 0; m < 5; m++) {
        V g = v[(h ? 45 : 30) + 5 * i + m];
        if (side && !h) g = -g;
        p[5 * i + m] = lower ? at(6 * N + 5 * sp + m, ro + 3 * u + i) : at(ro + 3 * u + i, 6 * N + 5 * sp + m);
        x[5 * i + m] = g;
      }
    sk.template put<15>(p, x, add);
  }
  // QQ, both orders
#pragma unroll
  for (int side = 0; side < 2; side++) {
    const int r = side ? b : a, c = side ? a : b;
    int64_t p[25];
    V x[25];
#pragma unroll
    for (int xi = 0; xi < 5; xi++)
#pragma unroll
      for (int y = 0; y < 5; y++) {
        const int lo = xi < y ? xi : y, hi = xi < y ? y : xi;
        p[5 * xi + y] = at(6 * N + 5 * r + xi, 6 * N + 5 * c + y);
        x[5 * xi + y] = v[15 + lo * 5 - lo * (lo - 1) / 2 + (hi - lo)];
      }
    sk.template put<25>(p, x, add);
  }
}

// Mixed form: only the entries whose row belongs to particle a (a < b) of
// each pair block are written (121 of 242: the pair's rows of the grand
// matrix, all coalesced along a); the consumers read the other half at the
// mirrored position.  Values as in store_pair_t.
__device__ inline void store_pair_rows_a(const PlaneSink& sk, int N, int a, int b, const dsf* v, int add) {
  auto at = [&](int r, int c) { return (int64_t)r + (int64_t)c * sk.ld; };
  constexpr int sym[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
  {  // TT and RR
    int64_t p[18];
    dsf x[18];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        p[3 * i + j] = at(3 * a + i, 3 * b + j);
        x[3 * i + j] = v[sym[i][j]];
        p[9 + 3 * i + j] = at(3 * N + 3 * a + i, 3 * N + 3 * b + j);
        x[9 + 3 * i + j] = v[6 + sym[i][j]];
      }
    sk.template put<18>(p, x, add);
  }
  {  // TR: a's translation rows against b's rotation, a's rotation rows against b's translation
    int64_t p[18];
    dsf x[18];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        dsf tr = dsf(0);
        if (i < j) tr = v[12 + (i == 0 ? j - 1 : 2)];
        if (i > j) tr = -v[12 + (j == 0 ? i - 1 : 2)];
        p[3 * i + j] = at(3 * a + i, 3 * N + 3 * b + j);
        x[3 * i + j] = tr;
        p[9 + 3 * i + j] = at(3 * N + 3 * a + j, 3 * b + i);
        x[9 + 3 * i + j] = -tr;
      }
    sk.template put<18>(p, x, add);
  }
#pragma unroll
  for (int grp = 0; grp < 4; grp++) {  // G and H: a's velocity rows, then a's stresslet rows
    const int h = grp & 1, srow = grp >> 1;
    const int ro = h ? 3 * N : 0;
    int64_t p[15];
    dsf x[15];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int m = 0; m < 5; m++) {
        dsf g = v[(h ? 45 : 30) + 5 * i + m];
        if (srow && !h) g = -g;
        p[5 * i + m] = srow ? at(6 * N + 5 * a + m, ro + 3 * b + i) : at(ro + 3 * a + i, 6 * N + 5 * b + m);
        x[5 * i + m] = g;
      }
    sk.template put<15>(p, x, add);
  }
  {  // QQ
    int64_t p[25];
    dsf x[25];
#pragma unroll
    for (int xi = 0; xi < 5; xi++)
#pragma unroll
      for (int y = 0; y < 5; y++) {
        const int lo = xi < y ? xi : y, hi = xi < y ? y : xi;
        p[5 * xi + y] = at(6 * N + 5 * a + xi, 6 * N + 5 * b + y);
        x[5 * xi + y] = v[15 + lo * 5 - lo * (lo - 1) / 2 + (hi - lo)];
      }
    sk.template put<25>(p, x, add);
  }
}

// A pair block computed in FP64 into either destination.
__device__ __forceinline__ void store_pair_d(const DenseSink& sk, int N, int a, int b, const double* o, int add) {
  store_pair_t<double>(sk, N, a, b, o, add);
}
__device__ __forceinline__ void store_pair_d(const PlaneSink& sk, int N, int a, int b, const double* o, int add) {
  dsf v[60];
#pragma unroll
  for (int q = 0; q < 60; q++) v[q] = dsf_from(o[q]);
  store_pair_rows_a(sk, N, a, b, v, add);
}

// scale by nondim (1/(6 a_i) for TT, TR, G; 1/(6 a_i^3) for RR, QQ, H) and
// by 1/(pi mu_f)
__device__ inline void scale_block(double* v, double ai, double inv_pimu) {
  const double na = inv_pimu / (6.0 * ai), na3 = inv_pimu / (6.0 * ai * ai * ai);
  for (int q = 0; q < 60; q++) {
    const bool a3 = (q >= 6 && q < 12) || (q >= 15 && q < 30) || q >= 45;
    v[q] *= a3 ? na3 : na;
  }
}

__device__ inline bool pair_of(int nn, int* a, int* b) {
  *a = blockIdx.x * blockDim.x + threadIdx.x;
  *b = blockIdx.y * blockDim.y + threadIdx.y;
  return *a < nn && *b < nn && *a < *b;
}

template <typename T>
struct Vec2;
template <>
struct Vec2<float> {
  using type = float4;  // four weights per shared-memory load
  static constexpr int W = 4;
};

// Reciprocal-space pair sums: per half-space vector, cos and sin of k.(x_a -
// x_b) from the per-particle trig table, times the vector's 80 moment
// weights.  The weights are staged in shared memory 16 vectors at a time and
// read as 16-byte vectors (the same address for every thread of a warp).
template <typename T, typename T2, typename S>
__global__ void __launch_bounds__(128) ewald_pair_k(int nn, rsd_lat_dev L, int Kh, const T* __restrict__ tab,
                                                    const T2* __restrict__ cs, const double* __restrict__ radii,
                                                    double inv_pimu, S sk, int add) {
  pdl_enter();
  constexpr int KWT = 3 + RSD_NMOM_KCOS + RSD_NMOM_KSIN;
  constexpr int NW = RSD_NMOM_KCOS + RSD_NMOM_KSIN;  // 80
  constexpr int KC = 16;
  using V = typename Vec2<T>::type;
  constexpr int VW = Vec2<T>::W;
  static_assert(NW % VW == 0, "weights per vector");
  __shared__ __align__(16) T sw[KC * NW];
  __shared__ T2 sca[KC][32], scb[KC][4];  // trig values of the CTA's 32 + 4 particles (block 32 x 4)
  // blocks entirely on or below the diagonal (a >= b everywhere) have no work
  if ((int)(blockIdx.x * blockDim.x) >= (int)(blockIdx.y * blockDim.y + blockDim.y - 1)) return;
  int a, b;
  const bool valid = pair_of(nn, &a, &b);
  const int tid = threadIdx.y * blockDim.x + threadIdx.x, nthr = blockDim.x * blockDim.y;
  const int a0 = blockIdx.x * blockDim.x, b0 = blockIdx.y * blockDim.y;
  T ac[RSD_NMOM_KCOS], as[RSD_NMOM_KSIN];
#pragma unroll
  for (int m = 0; m < RSD_NMOM_KCOS; m++) ac[m] = T(0);
#pragma unroll
  for (int m = 0; m < RSD_NMOM_KSIN; m++) as[m] = T(0);
  for (int h0 = 0; h0 < Kh; h0 += KC) {
    const int kc = min(KC, Kh - h0);
    __syncthreads();
    for (int e = tid; e < kc * NW; e += nthr) sw[e] = tab[(size_t)(h0 + e / NW) * KWT + 3 + e % NW];
    for (int e = tid; e < kc * 36; e += nthr) {
      const int hh = e / 36, q = e % 36, part = q < 32 ? a0 + q : b0 + q - 32;
      if (part < nn) {
        const T2 v = cs[(size_t)(h0 + hh) * nn + part];
        if (q < 32)
          sca[hh][q] = v;
        else
          scb[hh][q - 32] = v;
      }
    }
    __syncthreads();
    if (!valid) continue;
    for (int hh = 0; hh < kc; hh++) {
      const T2 ua = sca[hh][threadIdx.x], ub = scb[hh][threadIdx.y];
      const T c = ua.x * ub.x + ua.y * ub.y;  // cos(k.(x_a - x_b))
      const T sn = ua.y * ub.x - ua.x * ub.y;  // sin(k.(x_a - x_b))
      const V* e = reinterpret_cast<const V*>(sw + hh * NW);
#pragma unroll
      for (int m4 = 0; m4 < NW / VW; m4++) {
        const V w = e[m4];
        const T* wq = reinterpret_cast<const T*>(&w);
#pragma unroll
        for (int q = 0; q < VW; q++) {
          const int m = m4 * VW + q;
          if (m < RSD_NMOM_KCOS)
            ac[m] = fma(wq[q], c, ac[m]);
          else
            as[m - RSD_NMOM_KCOS] = fma(wq[q], sn, as[m - RSD_NMOM_KCOS]);
        }
      }
    }
  }
  if (!valid) return;
  const T ai = (T)radii[a], aj = (T)radii[b], phix = (T)L.phix;
  T v[60], w[60];
  rsd_kcos_epilogue<T>(ac, ai, aj, phix, v);
  rsd_ksin_epilogue<T>(as, ai, aj, phix, w);
  double o[60];
  const double f = 2.0 / L.LV;  // half space counted twice
#pragma unroll
  for (int q = 0; q < 60; q++) o[q] = ((double)v[q] + (double)w[q]) * f;
  scale_block(o, radii[a], inv_pimu);
  store_pair_d(sk, nn, a, b, o, add);
}

// Reciprocal-space pair sums of the FP64 shells of the mixed form (unequal
// radii) in double-single: the trig table holds (cos, sin) as float pairs
// (float4 per vector and particle), the moment weights are split into float
// pairs as they are staged in shared memory, two moments go through each
// packed instruction (dsacc's multiply-add as in ewald_pair_kblock; N = 300
// 440 -> 365 us), and the epilogue runs in FP64.
template <typename S>
__global__ void __launch_bounds__(128) ewald_pair_k_ds(int nn, rsd_lat_dev L, int Kh, const double* __restrict__ tab,
                                                       const float4* __restrict__ cs, const double* __restrict__ radii,
                                                       double inv_pimu, S sk, int add) {
  pdl_enter();
  constexpr int KWT = 3 + RSD_NMOM_KCOS + RSD_NMOM_KSIN;
  constexpr int NW = RSD_NMOM_KCOS + RSD_NMOM_KSIN;
  static_assert(NW % 4 == 0, "16-byte rows");
  constexpr int KC = 16;
  __shared__ __align__(16) float sw[KC][2][NW];  // heads, tails
  __shared__ float4 sca[KC][32], scb[KC][4];  // trig values of the CTA's 32 + 4 particles (block 32 x 4)
  if ((int)(blockIdx.x * blockDim.x) >= (int)(blockIdx.y * blockDim.y + blockDim.y - 1)) return;
  int a, b;
  const bool valid = pair_of(nn, &a, &b);
  const int tid = threadIdx.y * blockDim.x + threadIdx.x, nthr = blockDim.x * blockDim.y;
  const int a0 = blockIdx.x * blockDim.x, b0 = blockIdx.y * blockDim.y;
  uint64_t hi[NW / 2], lo[NW / 2];
#pragma unroll
  for (int p = 0; p < NW / 2; p++) hi[p] = lo[p] = 0;
  for (int h0 = 0; h0 < Kh; h0 += KC) {
    const int kc = min(KC, Kh - h0);
    __syncthreads();
    for (int e = tid; e < kc * NW; e += nthr) {
      const dsf w = dsf_from(tab[(size_t)(h0 + e / NW) * KWT + 3 + e % NW]);
      sw[e / NW][0][e % NW] = w.hi;
      sw[e / NW][1][e % NW] = w.lo;
    }
    for (int e = tid; e < kc * 36; e += nthr) {
      const int hh = e / 36, q = e % 36, part = q < 32 ? a0 + q : b0 + q - 32;
      if (part < nn) {
        const float4 v = cs[(size_t)(h0 + hh) * nn + part];
        if (q < 32)
          sca[hh][q] = v;
        else
          scb[hh][q - 32] = v;
      }
    }
    __syncthreads();
    if (!valid) continue;
    for (int hh = 0; hh < kc; hh++) {
      const float4 ua = sca[hh][threadIdx.x], ub = scb[hh][threadIdx.y];
      const dsf ca(ua.x, ua.y), sa(ua.z, ua.w), cb(ub.x, ub.y), sb(ub.z, ub.w);
      const dsf c = ca * cb + sa * sb;   // cos(k.(x_a - x_b))
      const dsf sn = sa * cb - ca * sb;  // sin(k.(x_a - x_b))
      // cos, sin, or one of each where the moments turn from the one to the other
      const uint64_t ch[3] = {f2_pack(c.hi, c.hi), f2_pack(sn.hi, sn.hi), f2_pack(c.hi, sn.hi)};
      const uint64_t nh[3] = {f2_pack(-c.hi, -c.hi), f2_pack(-sn.hi, -sn.hi), f2_pack(-c.hi, -sn.hi)};
      const uint64_t nl[3] = {f2_pack(-c.lo, -c.lo), f2_pack(-sn.lo, -sn.lo), f2_pack(-c.lo, -sn.lo)};
      const ulonglong2* eh = reinterpret_cast<const ulonglong2*>(sw[hh][0]);
      const ulonglong2* el = reinterpret_cast<const ulonglong2*>(sw[hh][1]);
#pragma unroll
      for (int g = 0; g < NW / 4; g++) {
        const ulonglong2 wh = eh[g], wl = el[g];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const int p = 2 * g + u, k = 2 * p + 1 < RSD_NMOM_KCOS ? 0 : (2 * p >= RSD_NMOM_KCOS ? 1 : 2);
          const uint64_t xh = u ? wh.y : wh.x, xl = u ? wl.y : wl.x;
          const uint64_t pr = f2_mul(xh, ch[k]);
          const uint64_t ne = f2_fma(xh, nl[k], f2_fma(xl, nh[k], f2_fma(xh, nh[k], pr)));  // minus the product's error
          const uint64_t s = f2_add(hi[p], pr), bb = f2_sub(s, hi[p]);
          const uint64_t e = f2_add(f2_sub(hi[p], f2_sub(s, bb)), f2_sub(pr, bb));
          lo[p] = f2_add(lo[p], f2_sub(e, ne));
          hi[p] = s;
        }
      }
    }
#pragma unroll
    for (int p = 0; p < NW / 2; p++) {  // at most 16 steps between renormalisations
      const uint64_t s = f2_add(hi[p], lo[p]);
      lo[p] = f2_sub(lo[p], f2_sub(s, hi[p]));
      hi[p] = s;
    }
  }
  if (!valid) return;
  double acd[RSD_NMOM_KCOS], asd[RSD_NMOM_KSIN];
#pragma unroll
  for (int p = 0; p < NW / 2; p++) {
    float h[2], l[2];
    f2_unpack(hi[p], h[0], h[1]);
    f2_unpack(lo[p], l[0], l[1]);
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int m = 2 * p + u;
      const double d = (double)h[u] + (double)l[u];
      if (m < RSD_NMOM_KCOS)
        acd[m] = d;
      else
        asd[m - RSD_NMOM_KCOS] = d;
    }
  }
  double v[60], w[60];
  rsd_kcos_epilogue<double>(acd, radii[a], radii[b], L.phix, v);
  rsd_ksin_epilogue<double>(asd, radii[a], radii[b], L.phix, w);
  double o[60];
  const double f = 2.0 / L.LV;  // half space counted twice
#pragma unroll
  for (int q = 0; q < 60; q++) o[q] = (v[q] + w[q]) * f;
  scale_block(o, radii[a], inv_pimu);
  store_pair_d(sk, nn, a, b, o, add);
}

// ---------------------------------------------------- equal radii, k space
// With one radius for every particle, the reciprocal-space epilogue (linear
// in the moments) can be applied per vector instead of per pair: each of
// the 60 block entries is then sum_k W_q(k) cos(k.R) (41 entries: TT, RR,
// QQ, H) or sum_k W_q(k) sin(k.R) (the 18 TR and G entries), with the block
// weights W_q(k) = epilogue(moment weights of k) formed once per vector in
// FP64.  A pair then costs 60 multiply-adds per vector instead of 80, and
// its FP32 rounding is no longer amplified by the epilogue's cancellation
// between moments.
constexpr int KBW = 64;  // weights per vector (60 used, padded for 16-byte rows)

// Block weights of the listed vectors: the first K64 as a row of hi parts and
// a row of lo parts (2 KBW floats a vector), the K32 others in FP32 (KBW
// floats).  blockIdx.y = 0 forms the cos outputs, 1 the sin ones: a warp
// issues an FP64 instruction every 64 cycles, so the kernel's time is one
// thread's instruction count.
__global__ void ewald_kblock_lists(rsd_lat_dev L, int K64, int K32, const int* __restrict__ hlist, double a,
                                   double inv_pimu, float* __restrict__ W64, float* __restrict__ W32) {
  pdl_enter();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= K64 + K32) return;
  int nx, ny, nz;
  half_space_index(hlist[q], L.NI, &nx, &ny, &nz);
  double k[3];
  for (int j = 0; j < 3; j++)
    k[j] = 2.0 * RSD_PI * (nx * L.LI[0 + 3 * j] + ny * L.LI[1 + 3 * j] + nz * L.LI[2 + 3 * j]);
  const double k2 = k[0] * k[0] + k[1] * k[1] + k[2] * k[2];
  const double S = kernel_S<double>(k2, L.lam);
  // half space counted twice, and the non-dimensionalisation of scale_block
  const double f = 2.0 / L.LV, na = f * inv_pimu / (6.0 * a), na3 = na / (a * a);
  auto put = [&](int i, double v) {
    if (q < K64) {
      const dsf d = dsf_from(v);
      W64[(size_t)q * 2 * KBW + i] = d.hi;
      W64[(size_t)q * 2 * KBW + KBW + i] = d.lo;
    } else {
      W32[(size_t)(q - K64) * KBW + i] = (float)v;
    }
  };
  double w[RSD_NMOM_KCOS], v[60];
  if (blockIdx.y == 0) {
    rsd_kcos_weights<double>(k[0], k[1], k[2], S, L.lam, w);
    rsd_kcos_epilogue<double>(w, a, a, L.phix, v);
#pragma unroll
    for (int i = 0; i < 60; i++) {
      const bool a3 = (i >= 6 && i < 12) || (i >= 15 && i < 30) || i >= 45;
      if (!kblock_is_sin(i)) put(i, v[i] * (a3 ? na3 : na));
    }
    for (int i = 60; i < KBW; i++) put(i, 0.0);
  } else {
    rsd_ksin_weights<double>(k[0], k[1], k[2], S, L.lam, w);
    rsd_ksin_epilogue<double>(w, a, a, L.phix, v);
#pragma unroll
    for (int i = 0; i < 60; i++)
      if (kblock_is_sin(i)) put(i, v[i] * na);  // TR and G
  }
}

// Stages 16 vectors' weights (floats per vector: NW) and the trig values of
// the CTA's 32 + 4 particles in shared memory.
template <int NW, typename TT>
__device__ __forceinline__ void kblock_stage(int nn, int h0, int kc, const float* __restrict__ W,
                                             const TT* __restrict__ cs, float* sw, TT* sca, TT* scb) {
  const int tid = threadIdx.y * blockDim.x + threadIdx.x, nthr = blockDim.x * blockDim.y;
  const int a0 = blockIdx.x * blockDim.x, b0 = blockIdx.y * blockDim.y;
  const float4* src = reinterpret_cast<const float4*>(W + (size_t)h0 * NW);
  for (int e = tid; e < kc * NW / 4; e += nthr) reinterpret_cast<float4*>(sw)[e] = src[e];
  for (int e = tid; e < kc * 36; e += nthr) {
    const int hh = e / 36, q = e % 36, part = q < 32 ? a0 + q : b0 + q - 32;
    if (part < nn) {
      const TT v = cs[(size_t)(h0 + hh) * nn + part];
      if (q < 32)
        sca[hh * 32 + q] = v;
      else
        scb[hh * 4 + q - 32] = v;
    }
  }
}

// Reciprocal-space pair blocks with per-vector block weights (equal radii),
// the sums sum_k W_q(k) {cos, sin}(k.(x_a - x_b)) in packed pairs of outputs
// (30 pairs; a pair takes cos, sin or, at two seams, one of each):
//   - the K32 FP32 vectors first, a chunk of 16 summed in FP32 and folded into
//     a double-single total (hi + lo, Knuth's two-sum): a plain FP32 sum over
//     all K32 vectors has a rounding error ~ sqrt(K32) times that of its
//     terms, which grows with lambda^3;
//   - then the K64 double-single ones on top, as dsacc's multiply-add (dsf.cuh)
//     with the products taken against -cos, -sin, so that no sign is flipped.
// The blocks are written (add = 0) or added (add = 1) once.  Bound by FP32
// issue at 8 warps per SM (accumulators in registers); the packed form halves
// the instructions: N = 2048 10.4 -> 8.1 ms, N = 512 0.74 -> 0.56 ms.
// SLICED: slice blockIdx.z of each list is summed, into part (see
// ewald_join_slices).
template <bool SLICED>
__global__ void __launch_bounds__(128) ewald_pair_kblock(int nn, int K32, const float* __restrict__ W32,
                                                         const float2* __restrict__ c32, int K64,
                                                         const float* __restrict__ W64, const float4* __restrict__ c64,
                                                         PlaneSink sk, int add, float2* __restrict__ part) {
  pdl_enter();
  constexpr int KC = 16;
  if (SLICED) {
    // whole chunks of the FP32 vectors, so that their FP32 sums are those of one slice
    const int z = blockIdx.z, S = gridDim.z, nc = (K32 + KC - 1) / KC, f = KC * (nc * z / S), g = K64 * z / S;
    K32 = min(K32, KC * (nc * (z + 1) / S)) - f;
    W32 += (size_t)f * KBW;
    c32 += (size_t)f * nn;
    K64 = K64 * (z + 1) / S - g;
    W64 += (size_t)g * 2 * KBW;
    c64 += (size_t)g * nn;
  }
  __shared__ __align__(16) float sw[KC * 2 * KBW];  // the FP32 phase uses the first half
  __shared__ __align__(16) float4 sca[KC * 32], scb[KC * 4];
  if ((int)(blockIdx.x * blockDim.x) >= (int)(blockIdx.y * blockDim.y + blockDim.y - 1)) return;
  int a, b;
  const bool valid = pair_of(nn, &a, &b);
  uint64_t hi[30], lo[30];
#pragma unroll
  for (int p = 0; p < 30; p++) hi[p] = lo[p] = 0;
  {
    uint64_t f[30];
#pragma unroll
    for (int p = 0; p < 30; p++) f[p] = 0;
    float2 *ta = reinterpret_cast<float2*>(sca), *tb = reinterpret_cast<float2*>(scb);
    for (int h0 = 0; h0 < K32; h0 += KC) {
      const int kc = min(KC, K32 - h0);
      __syncthreads();
      kblock_stage<KBW>(nn, h0, kc, W32, c32, sw, ta, tb);
      __syncthreads();
      if (!valid) continue;
      for (int hh = 0; hh < kc; hh++) {
        const float2 ua = ta[hh * 32 + threadIdx.x], ub = tb[hh * 4 + threadIdx.y];
        const float c = ua.x * ub.x + ua.y * ub.y;   // cos(k.(x_a - x_b))
        const float sn = ua.y * ub.x - ua.x * ub.y;  // sin(k.(x_a - x_b))
        const uint64_t cc = f2_pack(c, c), ss = f2_pack(sn, sn), sc = f2_pack(sn, c);
        const ulonglong2* e = reinterpret_cast<const ulonglong2*>(sw + hh * KBW);
#pragma unroll
        for (int g = 0; g < 15; g++) {
          const ulonglong2 w = e[g];
#pragma unroll
          for (int u = 0; u < 2; u++) {
            const int q = 4 * g + 2 * u;
            f[2 * g + u] = f2_fma(u ? w.y : w.x, !kblock_is_sin(q) ? cc : (kblock_is_sin(q + 1) ? ss : sc), f[2 * g + u]);
          }
        }
      }
#pragma unroll
      for (int p = 0; p < 30; p++) {
        const uint64_t s = f2_add(hi[p], f[p]), bb = f2_sub(s, hi[p]);
        lo[p] = f2_add(lo[p], f2_add(f2_sub(hi[p], f2_sub(s, bb)), f2_sub(f[p], bb)));
        hi[p] = s;
        f[p] = 0;
      }
    }
  }
  for (int h0 = 0; h0 < K64; h0 += KC) {
    const int kc = min(KC, K64 - h0);
    __syncthreads();
    kblock_stage<2 * KBW>(nn, h0, kc, W64, c64, sw, sca, scb);
    __syncthreads();
    if (!valid) continue;
    for (int hh = 0; hh < kc; hh++) {
      const float4 ua = sca[hh * 32 + threadIdx.x], ub = scb[hh * 4 + threadIdx.y];
      const dsf ca(ua.x, ua.y), sa(ua.z, ua.w), cb(ub.x, ub.y), sb(ub.z, ub.w);
      const dsf c = ca * cb + sa * sb, sn = sa * cb - ca * sb;
      const uint64_t ch[3] = {f2_pack(c.hi, c.hi), f2_pack(sn.hi, sn.hi), f2_pack(sn.hi, c.hi)};
      const uint64_t nh[3] = {f2_pack(-c.hi, -c.hi), f2_pack(-sn.hi, -sn.hi), f2_pack(-sn.hi, -c.hi)};
      const uint64_t nl[3] = {f2_pack(-c.lo, -c.lo), f2_pack(-sn.lo, -sn.lo), f2_pack(-sn.lo, -c.lo)};
      const ulonglong2* eh = reinterpret_cast<const ulonglong2*>(sw + hh * 2 * KBW);
      const ulonglong2* el = reinterpret_cast<const ulonglong2*>(sw + hh * 2 * KBW + KBW);
#pragma unroll
      for (int g = 0; g < 15; g++) {
        const ulonglong2 wh = eh[g], wl = el[g];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const int q = 4 * g + 2 * u, p = 2 * g + u;
          const int k = !kblock_is_sin(q) ? 0 : (kblock_is_sin(q + 1) ? 1 : 2);
          const uint64_t xh = u ? wh.y : wh.x, xl = u ? wl.y : wl.x;
          const uint64_t pr = f2_mul(xh, ch[k]);
          const uint64_t ne = f2_fma(xh, nl[k], f2_fma(xl, nh[k], f2_fma(xh, nh[k], pr)));  // minus the product's error
          const uint64_t s = f2_add(hi[p], pr), bb = f2_sub(s, hi[p]);
          const uint64_t e = f2_add(f2_sub(hi[p], f2_sub(s, bb)), f2_sub(pr, bb));
          lo[p] = f2_add(lo[p], f2_sub(e, ne));
          hi[p] = s;
        }
      }
    }
#pragma unroll
    for (int p = 0; p < 30; p++) {  // at most 16 steps between renormalisations
      const uint64_t s = f2_add(hi[p], lo[p]);
      lo[p] = f2_sub(lo[p], f2_sub(s, hi[p]));
      hi[p] = s;
    }
  }
  if (!valid) return;
  dsf o[60];
#pragma unroll
  for (int p = 0; p < 30; p++) {
    const uint64_t s = f2_add(hi[p], lo[p]), l = f2_sub(lo[p], f2_sub(s, hi[p]));
    f2_unpack(s, o[2 * p].hi, o[2 * p + 1].hi);
    f2_unpack(l, o[2 * p].lo, o[2 * p + 1].lo);
  }
  if (SLICED) {
    const int64_t np = (int64_t)nn * (nn - 1) / 2;
    part += (int64_t)blockIdx.z * 60 * np + (int64_t)b * (b - 1) / 2 + a;
#pragma unroll
    for (int q = 0; q < 60; q++) part[q * np] = make_float2(o[q].hi, o[q].lo);
  } else {
    store_pair_rows_a(sk, nn, a, b, o, add);
  }
}

__device__ __forceinline__ float image_r2f(float p0, float p1, float p2, float a0, float a1, float a2, int nz,
                                           float* x0, float* x1, float* x2) {
  const float z = (float)nz;
  *x0 = __fmaf_rn(a0, z, p0);
  *x1 = __fmaf_rn(a1, z, p1);
  *x2 = __fmaf_rn(a2, z, p2);
  return __fmaf_rn(*x2, *x2, __fmaf_rn(*x1, *x1, __fmul_rn(*x0, *x0)));
}

// ------------------------------------------ real space, mixed
// Far images (lambda r from the context's mixed_rcut up to mixed_rmax, beyond
// which the terms change a block by less than ~1e-12 of its largest entry) in
// FP32, near ones in double-single: the radial functions of erfc(lambda r)
// feed moments that the epilogue combines with 2-3 orders of cancellation, so
// FP32 is kept for images whose terms are below ~1e-6 of a block (a few 1e-11
// of a block after the epilogue), and ~48 bits keep a block within ~1e-12 of
// FP64.  An image within a rounding of the boundary may fall on either side;
// both are accurate there.
//
// Equal radii: one kernel for both real-space image sets of a pair, all in FP32 and
// double-single arithmetic (the FP64 pipe of GB300 runs at ~1/60 of the
// FP32 rate, so no FP64 is left in the image loops or the epilogue):
//   - images are classified in FP32: column base p = R + nx a1 + ny a2 and
//     image p + nz a3 (fused multiply-adds in a fixed order), near when its
//     squared distance is below rc^2, far up to rmax^2, so every image lands
//     in exactly one set;
//   - each set is processed from a per-thread list of image indices in
//     shared memory (REAL_CAP at a time), so the lanes of a warp run their
//     own images together instead of idling through each other's;
//   - far images: FP32 moments; near images: double-single coordinates
//     R + nx a1 + ny a2 + nz a3, r, erfc, exp and moments (dsacc);
//   - the epilogues apply the coefficient table of the common radius
//     (rsd_real_epi_coef_scaled, formed once in FP64), output by output, and
//     the pair blocks are added to M's planes once.
constexpr int REAL_CAP = 32;
constexpr int REAL_THREADS = 128;
struct RealEqShared {
  dsf_tables T;
  dsf cr[RSD_REAL_EPI_NC];
  float cf[RSD_REAL_EPI_NC];
  int list[REAL_CAP][REAL_THREADS];
  float oh[60][REAL_THREADS];  // the pair block: far part, then hi of the sum
  float ol[60][REAL_THREADS];  // lo of the sum
};
constexpr int SMEM_REAL_EQ = (int)sizeof(RealEqShared);

__device__ __forceinline__ int pack_image(int nx, int ny, int nz, int NR) {
  return (nx + NR) | ((ny + NR) << 8) | ((nz + NR) << 16);
}

// Lists the next images of the set (near: r2 < rc2; far: rc2 <= r2 < rmax2)
// from the resumable position (col, nz) into list[.][t], at most REAL_CAP;
// takes every step-th column; returns the count.
template <bool NEAR>
__device__ __forceinline__ int list_images(int (*list)[REAL_THREADS], int t, const float* Rf, const float* A, int NR,
                                           int& col, int& nz, int step, float rc2, float rmax2) {
  const int w = 2 * NR + 1, ncol = w * w;
  int cnt = 0, nx = 0, ny = 0;
  float p[3];
  bool base = false;
  while (col < ncol && cnt < REAL_CAP) {
    if (!base) {
      nx = col / w - NR;
      ny = col % w - NR;
      column_base_f(Rf, A, nx, ny, p);
      base = true;
    }
    float y0, y1, y2;
    const float r2 = image_r2f(p[0], p[1], p[2], A[6], A[7], A[8], nz, &y0, &y1, &y2);
    if (NEAR ? (r2 < rc2) : (r2 >= rc2 && r2 < rmax2)) list[cnt++][t] = pack_image(nx, ny, nz, NR);
    if (++nz > NR) {
      nz = -NR;
      col += step;
      base = false;
    }
  }
  return cnt;
}

// The near images' moments of part P (of NP, rsd_mom_part): one pass over
// the near set of the columns col, col + step, ..., into acc (normalised).
template <int NP, int P>
__device__ __forceinline__ void near_moments(const dsf_tables& T, int (*list)[REAL_THREADS], int t, const float* Rf,
                                             const float* A, const dsf* Rs, const dsf* As, int NR, float rc2,
                                             dsf lam_s, dsf cd_s, int col, int step, dsacc* acc) {
#pragma unroll
  for (int m = 0; m < RSD_NMOM_REAL; m++) acc[m] = dsacc(0);
  int nz = -NR;
  do {
    const int cnt = list_images<true>(list, t, Rf, A, NR, col, nz, step, rc2, 0.f);
    for (int q = 0; q < cnt; q++) {
      const int e = list[q][t];
      const int ix = (e & 255) - NR, iy = ((e >> 8) & 255) - NR, iz = (e >> 16) - NR;
      const dsf x0 = Rs[0] + ix * As[0] + iy * As[3] + iz * As[6];
      const dsf x1 = Rs[1] + ix * As[1] + iy * As[4] + iz * As[7];
      const dsf x2 = Rs[2] + ix * As[2] + iy * As[5] + iz * As[8];
      const dsf r = dsf_sqrt(x0 * x0 + x1 * x1 + x2 * x2);
      const dsf ir = dsf_rcp(r);
      dsf E0, G;
      dsf_erfc_gauss(lam_s * r, T, &E0, &G);
      rsd_real_image<dsf, dsacc, NP, P>(x0, x1, x2, r, ir, E0, cd_s * G, lam_s, acc);
      if ((q & 3) == 3) {  // keep the accumulators' lo parts small
#pragma unroll
        for (int m = 0; m < RSD_NMOM_REAL; m++) dsacc_norm(acc[m]);
      }
    }
#pragma unroll
    for (int m = 0; m < RSD_NMOM_REAL; m++) dsacc_norm(acc[m]);
  } while (col < (2 * NR + 1) * (2 * NR + 1));
}

// The same for the far images, in FP32 (EXACT: from column_base_s).
template <bool EXACT = false>
__device__ __forceinline__ void far_moments(int (*list)[REAL_THREADS], int t, const float* Rf, const float* A,
                                            const dsf* Rs, const dsf* As, int NR, float rc2, float rmax2, float lamf,
                                            float cdf, int col, int step, float* acc) {
  const float lam2f = lamf * lamf;
#pragma unroll
  for (int m = 0; m < RSD_NMOM_REAL; m++) acc[m] = 0.f;
  int nz = -NR;
  do {
    const int cnt = list_images<false>(list, t, Rf, A, NR, col, nz, step, rc2, rmax2);
    for (int q = 0; q < cnt; q++) {
      const int e = list[q][t];
      const int ix = (e & 255) - NR, iy = ((e >> 8) & 255) - NR, iz = (e >> 16) - NR;
      float p[3], x0, x1, x2;
      if (EXACT) {
        column_base_s(Rs, As, ix, iy, p);
      } else {
        column_base_f(Rf, A, ix, iy, p);
      }
      const float r2 = image_r2f(p[0], p[1], p[2], A[6], A[7], A[8], iz, &x0, &x1, &x2);
      const float r = sqrtf(r2), ir = 1.f / r;
      rsd_real_image<float>(x0, x1, x2, r, ir, erfcf(lamf * r), cdf * expf(-r2 * lam2f), lamf, acc);
    }
  } while (col < (2 * NR + 1) * (2 * NR + 1));
}

// Part P's share of every output, added into the pair block held in shared
// memory (oh + ol).
template <int NP, int P>
__device__ __forceinline__ void near_part(RealEqShared& sh, int t, const float* Rf, const float* A, const dsf* Rs,
                                          const dsf* As, int NR, float rc2, dsf lam_s, dsf cd_s) {
  dsacc acc[RSD_NMOM_REAL];
  near_moments<NP, P>(sh.T, sh.list, t, Rf, A, Rs, As, NR, rc2, lam_s, cd_s, 0, 1, acc);
  dsf accn[RSD_NMOM_REAL];
#pragma unroll
  for (int m = 0; m < RSD_NMOM_REAL; m++) accn[m] = dsf(acc[m].hi, acc[m].lo);
#pragma unroll
  for (int q = 0; q < 60; q++) {
    dsacc o = rsd_real_epi_row<dsf, dsf, dsacc, NP, P>(q, accn, sh.cr);
    o += dsf(sh.oh[q][t], sh.ol[q][t]);
    dsacc_norm(o);
    sh.oh[q][t] = o.hi;
    sh.ol[q][t] = o.lo;
  }
}

template <int NP, int P>
__device__ __forceinline__ void near_parts(RealEqShared& sh, int t, const float* Rf, const float* A, const dsf* Rs,
                                           const dsf* As, int NR, float rc2, dsf lam_s, dsf cd_s) {
  if constexpr (P < NP) {
    near_part<NP, P>(sh, t, Rf, A, Rs, As, NR, rc2, lam_s, cd_s);
    near_parts<NP, P + 1>(sh, t, Rf, A, Rs, As, NR, rc2, lam_s, cd_s);
  }
}

// The lattice and the minimum image of pair (a, b): the shift found in FP32,
// applied in double-single.
struct RealPair {
  float A[9], Rf[3];
  dsf As[9], Rs[3];
};
__device__ __forceinline__ void real_pair(const rsd_lat_dev& L, const double* __restrict__ pos, int a, int b,
                                          RealPair& g) {
  float LIf[9];
#pragma unroll
  for (int k = 0; k < 9; k++) {
    g.As[k] = dsf_from(L.LR[k]);
    g.A[k] = g.As[k].hi;
    LIf[k] = (float)L.LI[k];
  }
  const double R[3] = {pos[3 * a] - pos[3 * b], pos[3 * a + 1] - pos[3 * b + 1], pos[3 * a + 2] - pos[3 * b + 2]};
  const float R0[3] = {(float)R[0], (float)R[1], (float)R[2]};
  int k[3];
  rsd_skew_shift_f32(g.A, LIf, R0, k);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    g.Rs[i] = dsf_from(R[i]) - (k[0] * g.As[i] + k[1] * g.As[3 + i] + k[2] * g.As[6 + i]);
    g.Rf[i] = g.Rs[i].hi;
  }
}

// Unequal radii: both image sets as above, one FP64 epilogue on their sum (a
// pair's radii enter only there).  N = 300: ~510 us; in two kernels over the
// image cube, with FP64 column bases and minimum images and an epilogue each,
// 958.
struct RealMixShared {
  dsf_tables T;
  int list[REAL_CAP][REAL_THREADS];
  float far[RSD_NMOM_REAL][REAL_THREADS];
};
__global__ void __launch_bounds__(REAL_THREADS, 2) ewald_pair_real_mix(int nn, rsd_lat_dev L,
                                                                      const double* __restrict__ pos,
                                                                      const double* __restrict__ radii,
                                                                      double inv_pimu, float rc2, float rmax2,
                                                                      PlaneSink sk) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smraw_real[];
  RealMixShared& sh = *reinterpret_cast<RealMixShared*>(smraw_real);
  // blocks entirely on or below the diagonal (a >= b everywhere) have no work
  if ((int)(blockIdx.x * blockDim.x) >= (int)(blockIdx.y * blockDim.y + blockDim.y - 1)) return;
  const int t = threadIdx.y * blockDim.x + threadIdx.x;
  dsf_tables_fill(sh.T, t, REAL_THREADS);
  __syncthreads();
  int a, b;
  if (!pair_of(nn, &a, &b)) return;
  RealPair g;
  real_pair(L, pos, a, b, g);
  {
    float acc[RSD_NMOM_REAL];
    far_moments<true>(sh.list, t, g.Rf, g.A, g.Rs, g.As, L.NR, rc2, rmax2, (float)L.lam,
                      (float)(2.0 * RSD_PIP5 * L.lam), 0, 1, acc);
#pragma unroll
    for (int m = 0; m < RSD_NMOM_REAL; m++) sh.far[m][t] = acc[m];
  }
  double accd[RSD_NMOM_REAL];
  {
    dsacc acc[RSD_NMOM_REAL];
    near_moments<1, 0>(sh.T, sh.list, t, g.Rf, g.A, g.Rs, g.As, L.NR, rc2, dsf_from(L.lam),
                       dsf_from(2.0 * RSD_PIP5 * L.lam), 0, 1, acc);
#pragma unroll
    for (int m = 0; m < RSD_NMOM_REAL; m++) accd[m] = dsacc_to(acc[m]) + (double)sh.far[m][t];
  }
  double v[60];
  rsd_real_epilogue<double>(accd, radii[a], radii[b], L.phix, v);
  scale_block(v, radii[a], inv_pimu);
  store_pair_d(sk, nn, a, b, v, 1);
}

// NP: passes over the near images, each summing one part of the moments
// (fewer live accumulators and a shorter loop body per pass, at the cost of
// evaluating r, erfc and exp once per pass); MINB: CTAs per SM to fit.
template <int NP, int MINB>
__global__ void __launch_bounds__(REAL_THREADS, MINB) ewald_pair_real_eq(int nn, rsd_lat_dev L,
                                                                        const double* __restrict__ pos,
                                                                        const dsf* __restrict__ cr_g,
                                                                        const float* __restrict__ cf_g, float rc2,
                                                                        float rmax2, PlaneSink sk) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smraw_real[];
  RealEqShared& sh = *reinterpret_cast<RealEqShared*>(smraw_real);
  // blocks entirely on or below the diagonal (a >= b everywhere) have no work
  if ((int)(blockIdx.x * blockDim.x) >= (int)(blockIdx.y * blockDim.y + blockDim.y - 1)) return;
  const int t = threadIdx.y * blockDim.x + threadIdx.x;
  dsf_tables_fill(sh.T, t, REAL_THREADS);
  for (int k = t; k < RSD_REAL_EPI_NC; k += REAL_THREADS) {
    sh.cr[k] = cr_g[k];
    sh.cf[k] = cf_g[k];
  }
  __syncthreads();
  int a, b;
  if (!pair_of(nn, &a, &b)) return;
  RealPair g;
  real_pair(L, pos, a, b, g);
  const int NR = L.NR;
  {
    float acc[RSD_NMOM_REAL];
    far_moments(sh.list, t, g.Rf, g.A, g.Rs, g.As, NR, rc2, rmax2, (float)L.lam, (float)(2.0 * RSD_PIP5 * L.lam), 0, 1, acc);
#pragma unroll
    for (int q = 0; q < 60; q++) {
      sh.oh[q][t] = rsd_real_epi_row<float, float, float>(q, acc, sh.cf);
      sh.ol[q][t] = 0.f;
    }
  }
  // near images, double-single, in NP passes
  near_parts<NP, 0>(sh, t, g.Rf, g.A, g.Rs, g.As, NR, rc2, dsf_from(L.lam), dsf_from(2.0 * RSD_PIP5 * L.lam));
  dsf v[60];
#pragma unroll
  for (int q = 0; q < 60; q++) v[q] = dsf(sh.oh[q][t], sh.ol[q][t]);
  store_pair_rows_a(sk, nn, a, b, v, 1);
}


// ----------------------------------------------------------- FP64 pair sums
// GB300's FP64 pipe (2 multiply-adds per SM and cycle) bounds the FP64
// assembly: an image costs ~400 FP64 instructions, a reciprocal vector ~66
// (equal radii) or ~86, everything else (loads included) hides behind them.
// So the work per pair is what counts, and it is cut to what FP64 can
// represent: the Ewald sum does not depend on its splitting parameter, which
// is moved to EWALD64_SCALE times the reference's, and terms beyond lambda r =
// EWALD64_XC or k^2 / (4 lambda^2) = EWALD64_YC are left out.  Against long
// double sums over larger cubes the largest entry of a pair block moves by
// <= 3e-17 by that (2e-16 at two spheres in a box of 3.5 radii), with FP64
// rounding of a block at 1e-17 to 1e-16 either way.  A pair then takes ~77
// images and ~357 vectors instead of 343 to 1331 and 171 to 665.  Measured,
// pair sums in all, a thread per pair over the whole cubes before: N = 1000
// at zero strain 122.7 -> 47.4 ms (0.63e12 FP64 instructions/s, the pipe's
// rate), N = 512 at skew 0.5 76.3 -> 12.5 ms, N = 125 9.8 -> 0.91 ms, N = 64
// 9.8 -> 0.29 ms.
//
// A group of G lanes takes a pair: the group lists the images inside the
// sphere (an FP32 test; images within rounding of the surface may fall
// either way), its lanes take them and then the vectors in turn, and the
// moments are added up by halving exchanges, each lane left with 1/G of them.
// The lanes of a warp stay on images of the same pairs, so none idles
// through another's, and a small system still fills the GPU.  The epilogue
// is spread over the outputs (equal radii) or taken by one thread per pair.
constexpr double EWALD64_SCALE = 1.45, EWALD64_XC = 6.8, EWALD64_YC = 46.0;
constexpr int P64_THREADS = 128, P64_CAP = 128;

// Halving exchange over the lanes of a group: N values per lane in, the sums
// of `n` of them from `off` on out (the rest is with the other lanes).
template <int H, int N, int G>
__device__ __forceinline__ void group_halve(double (&v)[G], int gl, int& off, int& n) {
  if constexpr (H > 0) {
    constexpr int HN = (N + 1) / 2;
    const bool up = (gl & H) != 0;
#pragma unroll
    for (int i = 0; i < HN; i++) {
      const double lo = v[i], hi = i + HN < N ? v[i + HN] : 0.0;
      v[i] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, H);
    }
    if (up) {
      off += HN;
      n -= HN;
    } else {
      n = min(n, HN);
    }
    group_halve<H / 2, HN, G>(v, gl, off, n);
  }
}

template <int L, int N>
__device__ __forceinline__ void group_sum(double (&v)[N], int gl, double* dst) {
  int off = 0, n = N;
  group_halve<L / 2, N, N>(v, gl, off, n);
  constexpr int LEFT = (N + L - 1) / L + 1;
#pragma unroll
  for (int i = 0; i < LEFT; i++)
    if (i < n) dst[off + i] = v[i];
}

// Entry (r, c) of the 11 x 11 block (a, b), a < b, from the pair's 60 values.
template <typename T>
__device__ __forceinline__ T pair_block_entry(const T* v, int r, int c) {
  const int rs = r < 3 ? 0 : (r < 6 ? 1 : 2), cs = c < 3 ? 0 : (c < 6 ? 1 : 2);
  const int i = rs == 2 ? r - 6 : r - 3 * rs, j = cs == 2 ? c - 6 : c - 3 * cs;
  if (rs == cs && rs < 2) {  // TT, RR: symmetric 3 x 3 as 00 01 02 11 12 22
    const int lo = min(i, j), hi = max(i, j);
    return v[6 * rs + (lo == 0 ? hi : lo + hi + 1)];
  }
  if (rs == 2 && cs == 2) {
    const int lo = min(i, j), hi = max(i, j);
    return v[15 + lo * 5 - lo * (lo - 1) / 2 + (hi - lo)];
  }
  if (rs < 2 && cs < 2) {  // TR: antisymmetric, odd under a <-> b
    const int t = rs == 0 ? i : j, q = rs == 0 ? j : i;
    if (t == q) return T(0);
    const T x = v[12 + min(t, q) + max(t, q) - 1];
    return (t < q) == (rs == 0) ? x : -x;
  }
  if (rs < 2) return v[(rs ? 45 : 30) + 5 * i + j];   // G, H
  const T x = v[(cs ? 45 : 30) + 5 * j + i];
  return cs == 0 ? -x : x;                             // G is odd under a <-> b
}

// grand-matrix index of component k (0..10) of particle p
__device__ __forceinline__ int64_t grand_row(int N, int p, int k) {
  return k < 3 ? 3 * p + k : (k < 6 ? 3 * N + 3 * p + k - 3 : 6 * N + 5 * p + k - 6);
}

// ------------------------------------- equal radii, mixed, a small system
// Fewer pairs than the GPU holds threads leave the two kernels above waiting
// on one thread's chain (N = 32: 8 CTAs, 116 and 160 us).  The vectors of a
// pair and its images are then dealt out over S slices (blockIdx.z: a range of
// the vectors, every S-th column of images), the two kernels run side by side
// and write partial sums - the block's 60 values, the 97 moments near
// (double-single) and far (FP32) - at [slice][value][pair], pair (a, b) at
// b (b - 1) / 2 + a; the last kernel adds them up in double-single and writes
// the blocks.  N = 32: 285 -> 90 us from the trig tables to the blocks, N = 173
// 470 -> 250.  The FP32 vectors are cut at whole chunks, so that a step's
// outputs move by ~1e-13 only (cut anywhere: 5e-10, their FP32 rounding).
struct RealSliceShared {
  dsf_tables T;
  int list[REAL_CAP][REAL_THREADS];
};

__global__ void __launch_bounds__(REAL_THREADS, 2) ewald_real_slices(int nn, rsd_lat_dev L,
                                                                    const double* __restrict__ pos, float rc2,
                                                                    float rmax2, float2* __restrict__ near,
                                                                    float* __restrict__ far) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smraw_real[];
  RealSliceShared& sh = *reinterpret_cast<RealSliceShared*>(smraw_real);
  if ((int)(blockIdx.x * blockDim.x) >= (int)(blockIdx.y * blockDim.y + blockDim.y - 1)) return;
  const int t = threadIdx.y * blockDim.x + threadIdx.x, z = blockIdx.z, S = gridDim.z;
  dsf_tables_fill(sh.T, t, REAL_THREADS);
  __syncthreads();
  int a, b;
  if (!pair_of(nn, &a, &b)) return;
  RealPair g;
  real_pair(L, pos, a, b, g);
  const int64_t np = (int64_t)nn * (nn - 1) / 2, o = (int64_t)z * RSD_NMOM_REAL * np + (int64_t)b * (b - 1) / 2 + a;
  {
    float acc[RSD_NMOM_REAL];
    far_moments(sh.list, t, g.Rf, g.A, g.Rs, g.As, L.NR, rc2, rmax2, (float)L.lam, (float)(2.0 * RSD_PIP5 * L.lam), z, S,
                acc);
#pragma unroll
    for (int m = 0; m < RSD_NMOM_REAL; m++) far[o + m * np] = acc[m];
  }
  dsacc acc[RSD_NMOM_REAL];
  near_moments<1, 0>(sh.T, sh.list, t, g.Rf, g.A, g.Rs, g.As, L.NR, rc2, dsf_from(L.lam),
                     dsf_from(2.0 * RSD_PIP5 * L.lam), z, S, acc);
#pragma unroll
  for (int m = 0; m < RSD_NMOM_REAL; m++) near[o + m * np] = make_float2(acc[m].hi, acc[m].lo);
}

constexpr int JOIN_PAIRS = 16;
__global__ void __launch_bounds__(256) ewald_join_slices(int nn, int S, const float2* __restrict__ kpart,
                                                         const float2* __restrict__ near,
                                                         const float* __restrict__ far, const dsf* __restrict__ cr,
                                                         const unsigned short* __restrict__ etab, PlaneSink sk) {
  pdl_enter();
  __shared__ dsf mom[RSD_NMOM_REAL][JOIN_PAIRS], v[JOIN_PAIRS][61], c[RSD_REAL_EPI_NC];
  __shared__ unsigned short tab[61 + RSD_REAL_EPI_NC];
  __shared__ int2 ab[JOIN_PAIRS];
  const int t = threadIdx.x;
  const int64_t np = (int64_t)nn * (nn - 1) / 2, p0 = (int64_t)blockIdx.x * JOIN_PAIRS;
  const int cnt = (int)min((int64_t)JOIN_PAIRS, np - p0);
  for (int k = t; k < RSD_REAL_EPI_NC; k += 256) c[k] = cr[k];
  for (int k = t; k < 61 + RSD_REAL_EPI_NC; k += 256) tab[k] = etab[k];
  if (t < cnt) {
    int b = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)(p0 + t))) * 0.5f);
    while ((int64_t)b * (b - 1) / 2 > p0 + t) b--;
    while ((int64_t)b * (b + 1) / 2 <= p0 + t) b++;
    ab[t] = make_int2((int)(p0 + t - (int64_t)b * (b - 1) / 2), b);
  }
  for (int e = t; e < RSD_NMOM_REAL * JOIN_PAIRS; e += 256) {
    const int m = e / JOIN_PAIRS, i = e % JOIN_PAIRS;
    dsf s(0);
    if (i < cnt)
      for (int z = 0; z < S; z++) {
        const int64_t o = ((int64_t)z * RSD_NMOM_REAL + m) * np + p0 + i;
        const float2 x = near[o];
        s = s + dsf(x.x, x.y) + dsf(far[o], 0.f);
      }
    mom[m][i] = s;
  }
  __syncthreads();
  for (int e = t; e < 60 * JOIN_PAIRS; e += 256) {
    const int q = e / JOIN_PAIRS, i = e % JOIN_PAIRS;
    dsf s(0);
    if (i < cnt)
      for (int z = 0; z < S; z++) {
        const float2 x = kpart[((int64_t)z * 60 + q) * np + p0 + i];
        s = s + dsf(x.x, x.y);
      }
    for (int k = tab[q]; k < tab[q + 1]; k++) s = fma(c[k], mom[tab[61 + k]][i], s);
    v[i][q] = s;
  }
  __syncthreads();
  for (int e = t; e < 121 * JOIN_PAIRS; e += 256) {
    const int i = e % JOIN_PAIRS, rc = e / JOIN_PAIRS, r = rc % 11, col = rc / 11;
    if (i >= cnt) continue;
    const dsf x = pair_block_entry(v[i], r, col);
    const int64_t o = grand_row(nn, ab[i].x, r) + grand_row(nn, ab[i].y, col) * sk.ld;
    sk.hi[o] = x.hi;
    sk.lo[o] = x.lo;
  }
}

// cube: every listed image counts, around the exact minimum image of
// rsd_skew_correction (a sum whose cube the reference cuts visibly).
template <int G, bool EQ>
__global__ void __launch_bounds__(P64_THREADS) ewald_pair64(int nn, int64_t npair, rsd_lat_dev L, int cube, int nimg,
                                                            const double* __restrict__ img,
                                                            const float4* __restrict__ imgf, float rc2, int Kh,
                                                            const double* __restrict__ W,
                                                            const double2* __restrict__ cs,
                                                            const double* __restrict__ pos,
                                                            const double* __restrict__ radii, double inv_pimu,
                                                            const double* __restrict__ coef,
                                                            const unsigned short* __restrict__ etab, DenseSink sk) {
  pdl_enter();
  constexpr int PP = P64_THREADS / G, NK = EQ ? 60 : RSD_NMOM_KCOS + RSD_NMOM_KSIN, NR = RSD_NMOM_REAL;
  __shared__ double mom[PP][NR + NK];
  __shared__ int list[PP][P64_CAP];
  __shared__ double sc[EQ ? RSD_REAL_EPI_NC : 1];
  __shared__ unsigned short st[EQ ? RSD_REAL_EPI_NC : 1], so[EQ ? 61 : 1];
  const int t = threadIdx.x, g = t / G, gl = t % G, seg = (t & 31) / G * G;
  if (EQ) {
    for (int k = t; k < RSD_REAL_EPI_NC; k += P64_THREADS) {
      sc[k] = coef[k];
      st[k] = etab[61 + k];
    }
    for (int q = t; q < 61; q += P64_THREADS) so[q] = etab[q];
  }
  // pair p = b (b - 1) / 2 + a; the groups past the end repeat the last pair
  const int64_t p0 = (int64_t)blockIdx.x * PP;
  auto pair_ab = [&](int64_t p, int* pa, int* pb) {
    int b = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)p)) * 0.5f);
    while ((int64_t)b * (b - 1) / 2 > p) b--;
    while ((int64_t)(b + 1) * b / 2 <= p) b++;
    *pb = b;
    *pa = (int)(p - (int64_t)b * (b - 1) / 2);
  };
  int a, b;
  pair_ab(min(p0 + g, npair - 1), &a, &b);
  double R[3] = {pos[3 * a] - pos[3 * b], pos[3 * a + 1] - pos[3 * b + 1], pos[3 * a + 2] - pos[3 * b + 2]};
  if (cube) {
    double dmin;
    rsd_skew_correction(L.LR, L.LI, R, &dmin);
  } else {
    float A[9], LIf[9];
    for (int k = 0; k < 9; k++) {
      A[k] = (float)L.LR[k];
      LIf[k] = (float)L.LI[k];
    }
    const float R0[3] = {(float)R[0], (float)R[1], (float)R[2]};
    int k[3];
    rsd_skew_shift_f32(A, LIf, R0, k);
    if (max(abs(k[0]), max(abs(k[1]), abs(k[2]))) < 2000) {  // FP32 holds the fraction to 1e-3 of a cell
      for (int i = 0; i < 3; i++) R[i] -= k[0] * L.LR[i] + k[1] * L.LR[3 + i] + k[2] * L.LR[6 + i];
    } else {
      double dmin;
      rsd_skew_correction(L.LR, L.LI, R, &dmin);
    }
  }
  {
    const float Rf[3] = {(float)R[0], (float)R[1], (float)R[2]};
    const double lam = L.lam, lam2 = lam * lam, cd = 2.0 * RSD_PIP5 * lam;
    double acc[NR];
#pragma unroll
    for (int m = 0; m < NR; m++) acc[m] = 0.0;
    int cnt = 0;
    auto flush = [&](bool last) {
      const int nb = last ? (cnt + G - 1) / G : cnt / G;
      const int mb = __reduce_max_sync(0xffffffffu, nb);
      __syncwarp();
      for (int q = 0; q < mb; q++) {
        const int e = q * G + gl;
        if (q < nb && e < cnt) {
          const double* x = img + 3 * (size_t)list[g][e];
          const double x0 = R[0] + x[0], x1 = R[1] + x[1], x2 = R[2] + x[2];
          const double r2 = x0 * x0 + x1 * x1 + x2 * x2, r = sqrt(r2);
          rsd_real_image<double>(x0, x1, x2, r, 1.0 / r, erfc(lam * r), cd * exp(-r2 * lam2), lam, acc);
        }
      }
      if (!last) {  // the images of the last, partly filled round start the next list
        const int rem = cnt - nb * G;
        const int v = gl < rem ? list[g][nb * G + gl] : 0;
        __syncwarp();
        if (gl < rem) list[g][gl] = v;
        cnt = rem;
      }
      __syncwarp();
    };
    for (int c0 = 0; c0 < nimg; c0 += G) {
      const int i = c0 + gl;
      bool in = false;
      if (i < nimg) {
        const float4 x = imgf[i];
        const float x0 = Rf[0] + x.x, x1 = Rf[1] + x.y, x2 = Rf[2] + x.z;
        in = x0 * x0 + x1 * x1 + x2 * x2 < rc2;
      }
      unsigned m = __ballot_sync(0xffffffffu, in) >> seg;
      if (G < 32) m &= (1u << (G & 31)) - 1u;
      if (in) list[g][cnt + __popc(m & ((1u << gl) - 1u))] = i;
      cnt += __popc(m);
      if (__any_sync(0xffffffffu, cnt > P64_CAP - G)) flush(false);
    }
    flush(true);
    group_sum<G, NR>(acc, gl, mom[g]);
  }
  {
    double acc[NK];
#pragma unroll
    for (int m = 0; m < NK; m++) acc[m] = 0.0;
    const double2 *ca = cs + (size_t)a * Kh, *cb = cs + (size_t)b * Kh;
    for (int h = gl; h < Kh; h += G) {
      const double2 ua = ca[h], ub = cb[h];
      const double c = ua.x * ub.x + ua.y * ub.y;   // cos(k.(x_a - x_b))
      const double sn = ua.y * ub.x - ua.x * ub.y;  // sin(k.(x_a - x_b))
#pragma unroll
      for (int m = 0; m < NK; m++)
        acc[m] = ::fma(W[(size_t)m * Kh + h], (EQ ? kblock_is_sin(m) : m >= RSD_NMOM_KCOS) ? sn : c, acc[m]);
    }
    __syncwarp();
    group_sum<G, NK>(acc, gl, mom[g] + NR);
  }
  __syncthreads();
  const int np = (int)min((int64_t)PP, npair - p0);
  if (EQ) {
    for (int e = t; e < np * 60; e += P64_THREADS) {
      double* m = mom[e / 60];
      const int q = e % 60;
      double v = m[NR + q];
      for (int k = so[q]; k < so[q + 1]; k++) v = ::fma(sc[k], m[st[k]], v);
      m[NR + q] = v;
    }
  } else if (t < np) {
    pair_ab(p0 + t, &a, &b);
    const double ai = radii[a], aj = radii[b], f = 2.0 / L.LV;  // half space counted twice
    double* m = mom[t];
    double v[60], w[60], o[60];
    rsd_real_epilogue<double>(m, ai, aj, L.phix, o);
    rsd_kcos_epilogue<double>(m + NR, ai, aj, L.phix, v);
    rsd_ksin_epilogue<double>(m + NR + RSD_NMOM_KCOS, ai, aj, L.phix, w);
#pragma unroll
    for (int q = 0; q < 60; q++) o[q] += (v[q] + w[q]) * f;
    scale_block(o, ai, inv_pimu);
#pragma unroll
    for (int q = 0; q < 60; q++) m[NR + q] = o[q];
  }
  __syncthreads();
  for (int e = t; e < np * 121; e += P64_THREADS) {
    const int pr = e % np, en = e / np, r = en % 11, c = en / 11;
    pair_ab(p0 + pr, &a, &b);
    const double v = pair_block_entry(mom[pr] + NR, r, c);
    const int64_t i = grand_row(nn, a, r), j = grand_row(nn, b, c);
    sk.M[i + j * sk.ld] = v;
    sk.M[j + i * sk.ld] = v;
  }
}

// Self sums.  The real-space images n != 0 of a particle and the cos weights
// of the half space do not depend on the particle (only the epilogue does,
// through its radius), so one CTA sums them once in FP64.  EQ: out[0..59] =
// the whole diagonal block of the common radius ai, scaled; otherwise the
// moments, out[0..96] real and out[97..145] kcos.
constexpr int SELF_NMOM = RSD_NMOM_REAL + RSD_NMOM_KCOS;
constexpr int SELF_THREADS = 256;

// analytic self terms (Ewald_summation.f90:179-188) of output q
__device__ __forceinline__ double self_analytic(int q, double ai, double lam, double phix) {
  const double sp = sqrt(RSD_PI), a3 = ai * ai * ai, l3 = lam * lam * lam;
  if (q == 0 || q == 3 || q == 5) return 1.0 - 6.0 * lam / sp * ai + 40.0 / 3.0 / sp * l3 * a3 * phix;
  if (q == 6 || q == 9 || q == 11) return 0.75 - 10.0 / sp * a3 * l3;
  if (q == 15 || q == 20 || q == 24 || q == 27 || q == 29)  // QQ diagonal in the upper-triangle order
    return 0.9 - l3 * a3 / 25.0 / sp * (50.0 - 126.0 * lam * lam * ai * ai) * 6.0;
  return 0.0;
}

template <bool EQ>
__global__ void __launch_bounds__(SELF_THREADS) ewald_self_sums(rsd_lat_dev L, int nimg,
                                                                const double* __restrict__ img,
                                                                const float4* __restrict__ imgf, float rc2, int Kh,
                                                                const double* __restrict__ W, double ai,
                                                                double inv_pimu, const double* __restrict__ coef,
                                                                const unsigned short* __restrict__ etab,
                                                                double* __restrict__ out) {
  pdl_enter();
  constexpr int NW = SELF_THREADS / 32, NR = RSD_NMOM_REAL, NQ = EQ ? 60 : RSD_NMOM_KCOS;
  __shared__ double part[NW][NR], mom[NR], ks[NQ];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  {
    const double lam = L.lam, lam2 = lam * lam, cd = 2.0 * RSD_PIP5 * lam;
    double acc[NR];
#pragma unroll
    for (int m = 0; m < NR; m++) acc[m] = 0.0;
    for (int i = t; i < nimg; i += SELF_THREADS) {  // shortest first; n = 0 is left out (PER_ROTNE_PRAGER_SELF 61)
      const float4 f = imgf[i];
      const float r2f = f.x * f.x + f.y * f.y + f.z * f.z;
      if (!(r2f > 0.f && r2f < rc2)) continue;
      const double x0 = img[3 * i], x1 = img[3 * i + 1], x2 = img[3 * i + 2];
      const double r2 = x0 * x0 + x1 * x1 + x2 * x2, r = sqrt(r2);
      rsd_real_image<double>(x0, x1, x2, r, 1.0 / r, erfc(lam * r), cd * exp(-r2 * lam2), lam, acc);
    }
    __syncwarp();
    group_sum<32, NR>(acc, lane, part[warp]);
  }
  for (int q = warp; q < NQ; q += NW) {  // sin sums vanish: k and -k cancel
    double v = 0.0;
    if (!EQ || !kblock_is_sin(q))
      for (int h = lane; h < Kh; h += 32) v += W[(size_t)q * Kh + h];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) ks[q] = v;
  }
  __syncthreads();
  if (t < NR) {
    double v = 0.0;
    for (int w = 0; w < NW; w++) v += part[w][t];
    mom[t] = v;
  }
  __syncthreads();
  if (EQ) {
    if (t < 60) {
      const bool a3 = (t >= 6 && t < 12) || (t >= 15 && t < 30) || t >= 45;
      double v = self_analytic(t, ai, L.lam, L.phix) * inv_pimu / (6.0 * (a3 ? ai * ai * ai : ai)) + ks[t];
      for (int k = etab[t]; k < etab[t + 1]; k++) v = ::fma(coef[k], mom[etab[61 + k]], v);
      out[t] = v;
    }
  } else {
    if (t < NR) out[t] = mom[t];
    if (t < RSD_NMOM_KCOS) out[NR + t] = ks[t];
  }
}

// Diagonal blocks from the self sums (ewald_self_sums<false>) and the
// particle's radius.
__device__ __forceinline__ void sink_put(const DenseSink& sk, int64_t o, double x) { sk.M[o] = x; }
__device__ __forceinline__ void sink_put(const PlaneSink& sk, int64_t o, double x) {
  const dsf d = dsf_from(x);
  sk.hi[o] = d.hi;
  sk.lo[o] = d.lo;
}

template <typename S>
__global__ void __launch_bounds__(64) ewald_self(int nn, rsd_lat_dev L, const double* __restrict__ mom,
                                                 const double* __restrict__ radii, double inv_pimu, S sk) {
  pdl_enter();
  const int64_t ldm = sk.ld;
  auto M = [&](int64_t o, double x) { sink_put(sk, o, x); };
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= nn) return;
  const double ai = radii[a], lam = L.lam;
  double v[60], w[60];
  {
    double acc[RSD_NMOM_REAL];
    for (int m = 0; m < RSD_NMOM_REAL; m++) acc[m] = mom[m];
    rsd_real_epilogue<double>(acc, ai, ai, L.phix, v);
  }
  {
    double ac[RSD_NMOM_KCOS];
    for (int m = 0; m < RSD_NMOM_KCOS; m++) ac[m] = mom[RSD_NMOM_REAL + m];
    rsd_kcos_epilogue<double>(ac, ai, ai, L.phix, w);
  }
  // analytic self terms (Ewald_summation.f90:179-188)
  const double sp = sqrt(RSD_PI), a3 = ai * ai * ai, l3 = lam * lam * lam;
  const double ttsr = 1.0 - 6.0 * lam / sp * ai + 40.0 / 3.0 / sp * l3 * a3 * L.phix;
  const double rrsr = 0.75 - 10.0 / sp * a3 * l3;
  const double qqsr = 0.9 - l3 * a3 / 25.0 / sp * (50.0 - 126.0 * lam * lam * ai * ai) * 6.0;
  for (int q = 0; q < 60; q++) v[q] += w[q] * (2.0 / L.LV);
  v[0] += ttsr;
  v[3] += ttsr;
  v[5] += ttsr;
  v[6] += rrsr;
  v[9] += rrsr;
  v[11] += rrsr;
  const int dq[5] = {15, 20, 24, 27, 29};  // QQ diagonal in the upper-triangle order
  for (int x = 0; x < 5; x++) v[dq[x]] += qqsr;
  scale_block(v, ai, inv_pimu);
  // diagonal block: TT, RR, QQ; TR, G, H are zero (per_GRPY_YZD.f90:63-66)
  const int N = nn;
  const int sym[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      M((3 * a + i) + (int64_t)(3 * a + j) * ldm, v[sym[i][j]]);
      M((3 * N + 3 * a + i) + (int64_t)(3 * N + 3 * a + j) * ldm, v[6 + sym[i][j]]);
      M((3 * a + i) + (int64_t)(3 * N + 3 * a + j) * ldm, 0.0);
      M((3 * N + 3 * a + j) + (int64_t)(3 * a + i) * ldm, 0.0);
    }
  for (int i = 0; i < 3; i++)
    for (int m = 0; m < 5; m++) {
      M((3 * a + i) + (int64_t)(6 * N + 5 * a + m) * ldm, 0.0);
      M((3 * N + 3 * a + i) + (int64_t)(6 * N + 5 * a + m) * ldm, 0.0);
      M((6 * N + 5 * a + m) + (int64_t)(3 * a + i) * ldm, 0.0);
      M((6 * N + 5 * a + m) + (int64_t)(3 * N + 3 * a + i) * ldm, 0.0);
    }
  int q = 15;
  double qq[5][5];
  for (int x = 0; x < 5; x++)
    for (int y = x; y < 5; y++) qq[x][y] = qq[y][x] = v[q++];
  for (int x = 0; x < 5; x++)
    for (int y = 0; y < 5; y++) M((6 * N + 5 * a + x) + (int64_t)(6 * N + 5 * a + y) * ldm, qq[x][y]);
}

// Diagonal blocks of equal spheres: the one block of ewald_self_sums<true>
// written for every particle (TT, RR, QQ; TR, G, H are zero,
// per_GRPY_YZD.f90:63-66), a thread per entry.
template <typename S>
__global__ void ewald_self_eq(int nn, const double* __restrict__ v, S sk) {
  pdl_enter();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 121 * nn) return;
  const int a = t % nn, r = t / nn % 11, c = t / nn / 11;
  const bool same = (r < 3) == (c < 3) && (r < 6) == (c < 6);
  sink_put(sk, grand_row(nn, a, r) + grand_row(nn, a, c) * sk.ld, same ? pair_block_entry(v, r, c) : 0.0);
}

__global__ void overlap_count(int nn, rsd_lat_dev L, const double* __restrict__ pos, const double* __restrict__ radii,
                              int* __restrict__ count) {
  pdl_enter();
  int a, b;
  if (!pair_of(nn, &a, &b)) return;
  double R[3] = {pos[3 * a] - pos[3 * b], pos[3 * a + 1] - pos[3 * b + 1], pos[3 * a + 2] - pos[3 * b + 2]};
  double d;
  rsd_skew_correction(L.LR, L.LI, R, &d);
  if (d <= radii[a] + radii[b]) atomicAdd(count, 1);
}

// Overlapping pairs (minimum image with r <= a_i + a_j, the test of
// per_GRPY_YZD.f90:98) into a list of at most cap pairs; count ends at the
// number found.
__global__ void overlap_list(int nn, rsd_lat_dev L, const double* __restrict__ pos, const double* __restrict__ radii,
                             int cap, int2* __restrict__ list, int* __restrict__ count) {
  pdl_enter();
  int a, b;
  if (!pair_of(nn, &a, &b)) return;
  double R[3] = {pos[3 * a] - pos[3 * b], pos[3 * a + 1] - pos[3 * b + 1], pos[3 * a + 2] - pos[3 * b + 2]};
  double d;
  rsd_skew_correction(L.LR, L.LI, R, &d);
  if (d <= radii[a] + radii[b]) {
    const int k = atomicAdd(count, 1);
    if (k < cap) list[k] = make_int2(a, b);
  }
}

// Overlap correction (correction_method 1 or 2) of the listed pairs, one thread
// per pair, added to the assembled blocks at the minimum image: the blocks
// of different pairs are disjoint, so the sum does not depend on the order
// of the list.
template <typename S>
__global__ void __launch_bounds__(64) overlap_correct(int method, int npair, const int2* __restrict__ list, int nn,
                                                       rsd_lat_dev L, const double* __restrict__ pos,
                                                       const double* __restrict__ radii, double inv_pimu, S sk) {
  pdl_enter();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= npair) return;
  const int a = list[q].x, b = list[q].y;
  double R[3] = {pos[3 * a] - pos[3 * b], pos[3 * a + 1] - pos[3 * b + 1], pos[3 * a + 2] - pos[3 * b + 2]};
  double d;
  rsd_skew_correction(L.LR, L.LI, R, &d);
  double v[60];
  rsd_overlap_correction60(method, R, radii[a], radii[b], v);
  for (int k = 0; k < 60; k++) v[k] *= inv_pimu;
  store_pair_d(sk, nn, a, b, v, 1);
}

}  // namespace

int rsd_overlap_correct(rsd_ctx* ctx, int method, int precision, int nn, const double* d_pos, const double* d_radii,
                        const rsd_lattice* lat, double mu_f, int npair, double* d_M, int64_t ldm) {
  if (npair <= 0) return RSD_OK;
  const rsd_lat_dev L = rsd_lat_pack(lat);
  int* cnt = (int*)rsd_scratch(ctx, "overlap_count", sizeof(int));
  int2* list = (int2*)rsd_scratch(ctx, "overlap_list", sizeof(int2) * (size_t)npair);
  if (!cnt || !list) return RSD_ENOMEM;
  RSD_CUDA(ctx, cudaMemsetAsync(cnt, 0, sizeof(int), ctx->stream));
  dim3 blk(32, 4), grd((nn + 31) / 32, (nn + 3) / 4);
  pdl_launch(overlap_list, grd, blk, 0, ctx->stream, nn, L, d_pos, d_radii, npair, list, cnt);
  const double inv_pimu = 1.0 / (RSD_PI * mu_f);
  const unsigned nblk = (unsigned)((npair + 63) / 64);
  if (precision == RSD_PREC_MIXED) {
    float* hi = reinterpret_cast<float*>(d_M);
    const PlaneSink psk{hi, hi + (size_t)ldm * (11LL * nn), ldm};
    pdl_launch(overlap_correct<PlaneSink>, nblk, 64, 0, ctx->stream, method, npair, list, nn, L, d_pos, d_radii, inv_pimu,
                                                             psk);
  } else {
    const DenseSink dsk{d_M, ldm};
    pdl_launch(overlap_correct<DenseSink>, nblk, 64, 0, ctx->stream, method, npair, list, nn, L, d_pos, d_radii, inv_pimu,
                                                             dsk);
  }
  RSD_CUDA(ctx, cudaGetLastError());
  return RSD_OK;
}

int rsd_count_overlaps(rsd_ctx* ctx, int nn, const double* d_pos, const double* d_radii, const rsd_lattice* lat,
                       int* count) {
  rsd_lat_dev L = rsd_lat_pack(lat);
  int* d = (int*)rsd_scratch(ctx, "overlap_count", sizeof(int));
  if (!d) return RSD_ENOMEM;
  RSD_CUDA(ctx, cudaMemsetAsync(d, 0, sizeof(int), ctx->stream));
  dim3 blk(32, 4), grd((nn + 31) / 32, (nn + 3) / 4);
  pdl_launch(overlap_count, grd, blk, 0, ctx->stream, nn, L, d_pos, d_radii, d);
  RSD_CUDA(ctx, cudaGetLastError());
  RSD_CUDA(ctx, cudaMemcpyAsync(count, d, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  RSD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return RSD_OK;
}

// The Ewald sum does not depend on its splitting parameter lambda (checked
// with the oracle: moving lambda by 1.25-2x changes pair blocks by ~3e-15
// when the image cubes hold the sums).  The mixed form moves it by the
// context's mixed_lambda_scale, which trades double-single real-space
// images for cheaper reciprocal vectors, and sizes the cubes to hold its
// truncation spheres: lambda |x| < mixed_rmax, k^2 / (4 lambda^2) <
// mixed_kexp.  With fractional coordinates of the minimum image within
// [-1/2, 1/2], |n_i| <= r_max |b_i| + 1/2 in real space and |n_i| <= k_max
// |a_i| / (2 pi) in reciprocal space (a_i the lattice vectors, b_i their
// reciprocal vectors).  Scale 1 keeps the reference's lambda and cubes.
static rsd_lat_dev mixed_lattice(const rsd_ctx* ctx, rsd_lat_dev L) {
  const double f = ctx->mixed_lambda_scale;
  if (f == 1.0) return L;
  L.lam *= f;
  double amax = 0.0, bmax = 0.0;
  for (int i = 0; i < 3; i++) {
    double a2 = 0.0, b2 = 0.0;
    for (int j = 0; j < 3; j++) {
      a2 += L.LR[j + 3 * i] * L.LR[j + 3 * i];  // column i of LR
      b2 += L.LI[i + 3 * j] * L.LI[i + 3 * j];  // row i of LI
    }
    amax = fmax(amax, sqrt(a2));
    bmax = fmax(bmax, sqrt(b2));
  }
  const double rmax = ctx->mixed_rmax / L.lam, kmax = 2.0 * L.lam * sqrt(ctx->mixed_kexp);
  L.NR = max(L.NR, (int)ceil(rmax * bmax + 0.5));
  L.NI = max(L.NI, (int)ceil(kmax * amax / (2.0 * RSD_PI)));
  return L;
}

namespace {
template <int NP, int MINB>
int launch_real_eq_t(rsd_ctx* ctx, dim3 grd, dim3 blk, int nn, const rsd_lat_dev& L, const double* d_pos,
                     const dsf* cr, const float* cf, float rc2, float rmax2, const PlaneSink& psk) {
  RSD_TRY(rsd_smem(ctx, ewald_pair_real_eq<NP, MINB>, SMEM_REAL_EQ));
  pdl_launch(ewald_pair_real_eq<NP, MINB>, grd, blk, SMEM_REAL_EQ, ctx->stream, nn, L, d_pos, cr, cf, rc2, rmax2, psk);
  return RSD_OK;
}

constexpr int EWALD_SLICES = 16;
struct slice_parts {
  float2 *k, *near;
  float* far;
};
int slice_buffers(rsd_ctx* ctx, int S, int nn, slice_parts* o) {
  const size_t np = (size_t)nn * (nn - 1) / 2, nm = (size_t)S * RSD_NMOM_REAL * np;
  o->k = (float2*)rsd_scratch(ctx, "ewald_slices_k", sizeof(float2) * S * 60 * np);
  o->near = (float2*)rsd_scratch(ctx, "ewald_slices_near", sizeof(float2) * nm);
  o->far = (float*)rsd_scratch(ctx, "ewald_slices_far", sizeof(float) * nm);
  return o->k && o->near && o->far ? RSD_OK : RSD_ENOMEM;
}

// The images' slices on stream s (the side stream), ctx->ev_panel behind them.
int real_slices(rsd_ctx* ctx, cudaStream_t s, int S, dim3 grd, dim3 blk, int nn, const rsd_lat_dev& L,
                const double* d_pos, float rc2, float rmax2) {
  slice_parts p;
  RSD_TRY(slice_buffers(ctx, S, nn, &p));
  RSD_TRY(rsd_smem(ctx, ewald_real_slices, (int)sizeof(RealSliceShared)));
  grd.z = S;
  pdl_launch(ewald_real_slices, grd, blk, sizeof(RealSliceShared), s, nn, L, d_pos, rc2, rmax2, p.near, p.far);
  RSD_CUDA(ctx, cudaEventRecord(ctx->ev_panel, s));
  return RSD_OK;
}

// The vectors' slices, then the blocks from all of them.
int join_slices(rsd_ctx* ctx, int S, dim3 grd, dim3 blk, int nn, int K32, const float* w32, const float2* c32, int K64,
                const float* w64, const float4* c64, const dsf* cr, const unsigned short* etab, const PlaneSink& psk) {
  cudaStream_t s = ctx->stream;
  slice_parts p;
  RSD_TRY(slice_buffers(ctx, S, nn, &p));
  grd.z = S;
  pdl_launch(ewald_pair_kblock<true>, grd, blk, 0, s, nn, K32, w32, c32, K64, w64, c64, psk, 0, p.k);
  RSD_CUDA(ctx, cudaStreamWaitEvent(s, ctx->ev_panel, 0));
  const int64_t np = (int64_t)nn * (nn - 1) / 2;
  pdl_launch(ewald_join_slices, (unsigned)((np + JOIN_PAIRS - 1) / JOIN_PAIRS), 256, 0, s, nn, S, p.k, p.near, p.far,
             cr, etab, psk);
  return RSD_OK;
}

int launch_real_eq(rsd_ctx* ctx, int passes, dim3 grd, dim3 blk, int nn, const rsd_lat_dev& L, const double* d_pos,
                   const dsf* cr, const float* cf, float rc2, float rmax2, const PlaneSink& psk) {
  switch (passes) {
    case 1: return launch_real_eq_t<1, 2>(ctx, grd, blk, nn, L, d_pos, cr, cf, rc2, rmax2, psk);
    case 2: return launch_real_eq_t<2, 2>(ctx, grd, blk, nn, L, d_pos, cr, cf, rc2, rmax2, psk);
    case 3: return launch_real_eq_t<3, 2>(ctx, grd, blk, nn, L, d_pos, cr, cf, rc2, rmax2, psk);
    default: return launch_real_eq_t<4, 2>(ctx, grd, blk, nn, L, d_pos, cr, cf, rc2, rmax2, psk);
  }
}
}  // namespace

namespace {
// Lattice vectors and reciprocal vectors of a sum, made on the host.
struct ewald_lists {
  std::vector<double> img;  // lattice vectors LR n, shortest first (3 each)
  std::vector<double> kv;   // half-space reciprocal vectors (3 each)
  double rc2 = 0.0;         // images beyond rc2 are left out (infinite: none)
};

// The images within EWALD64_XC / lam of a point of the cell around the
// origin (self_only: of the origin), and the half-space vectors below
// EWALD64_YC.
ewald_lists ewald_sphere_lists(const rsd_lat_dev& L, double lam, bool self_only) {
  ewald_lists o;
  const double rc = EWALD64_XC / lam, kmax = 2.0 * lam * sqrt(EWALD64_YC);
  o.rc2 = rc * rc;
  double dmax = 0.0;  // a minimum image is no longer than half the longest diagonal of the cell
  for (int m = 0; m < 4 && !self_only; m++) {
    double d2 = 0.0;
    for (int j = 0; j < 3; j++) {
      const double x = L.LR[j] + (m & 1 ? -L.LR[3 + j] : L.LR[3 + j]) + (m & 2 ? -L.LR[6 + j] : L.LR[6 + j]);
      d2 += x * x;
    }
    dmax = fmax(dmax, 0.5 * sqrt(d2));
  }
  const double lim = rc + 1.001 * dmax;
  int nr[3], ni[3];
  for (int i = 0; i < 3; i++) {
    double a2 = 0.0, b2 = 0.0;
    for (int j = 0; j < 3; j++) {
      a2 += L.LR[j + 3 * i] * L.LR[j + 3 * i];
      b2 += L.LI[i + 3 * j] * L.LI[i + 3 * j];
    }
    nr[i] = (int)(lim * sqrt(b2)) + 1;
    ni[i] = (int)(kmax * sqrt(a2) / (2.0 * RSD_PI)) + 1;
  }
  std::vector<std::pair<double, int>> key;
  std::vector<double> x;
  for (int nx = -nr[0]; nx <= nr[0]; nx++)
    for (int ny = -nr[1]; ny <= nr[1]; ny++)
      for (int nz = -nr[2]; nz <= nr[2]; nz++) {
        double v[3], r2 = 0.0;
        for (int j = 0; j < 3; j++) {
          v[j] = L.LR[j] * nx + L.LR[3 + j] * ny + L.LR[6 + j] * nz;
          r2 += v[j] * v[j];
        }
        if (r2 >= lim * lim) continue;
        key.emplace_back(r2, (int)key.size());
        x.insert(x.end(), v, v + 3);
      }
  std::sort(key.begin(), key.end());
  for (const auto& q : key) o.img.insert(o.img.end(), x.begin() + 3 * q.second, x.begin() + 3 * q.second + 3);
  for (int nx = 0; nx <= ni[0]; nx++)
    for (int ny = -ni[1]; ny <= ni[1]; ny++)
      for (int nz = -ni[2]; nz <= ni[2]; nz++) {
        if (nx == 0 && (ny < 0 || (ny == 0 && nz <= 0))) continue;
        double k[3], k2 = 0.0;
        for (int j = 0; j < 3; j++) {
          k[j] = 2.0 * RSD_PI * (nx * L.LI[3 * j] + ny * L.LI[1 + 3 * j] + nz * L.LI[2 + 3 * j]);
          k2 += k[j] * k[j];
        }
        if (k2 < kmax * kmax) o.kv.insert(o.kv.end(), k, k + 3);
      }
  return o;
}

// The reference's cubes, whole.
ewald_lists ewald_cube_lists(const rsd_lat_dev& L) {
  ewald_lists o;
  o.rc2 = INFINITY;
  for (int nx = -L.NR; nx <= L.NR; nx++)
    for (int ny = -L.NR; ny <= L.NR; ny++)
      for (int nz = -L.NR; nz <= L.NR; nz++)
        for (int j = 0; j < 3; j++) o.img.push_back(L.LR[j] * nx + L.LR[3 + j] * ny + L.LR[6 + j] * nz);
  const int w = 2 * L.NI + 1, Kh = (w * w * w - 1) / 2;
  for (int h = 0; h < Kh; h++) {
    int nx, ny, nz;
    half_space_index(h, L.NI, &nx, &ny, &nz);
    for (int j = 0; j < 3; j++)
      o.kv.push_back(2.0 * RSD_PI * (nx * L.LI[3 * j] + ny * L.LI[1 + 3 * j] + nz * L.LI[2 + 3 * j]));
  }
  return o;
}

// Whether the reference's cubes reach as far as FP64 shows: the nearest image
// they leave out is at lambda r >= 6, the first vector at k^2 / (4 lambda^2)
// >= 40 (terms below ~1e-13 of a block).  True for EWS_ERR up to 1e-9 or so
// in a cell of any skew; a looser EWS_ERR cuts the sum where it shows, and
// its result is then the reference's cut sum.
bool cubes_converged(const rsd_lat_dev& L) {
  for (int i = 0; i < 3; i++) {
    double a2 = 0.0, b2 = 0.0;
    for (int j = 0; j < 3; j++) {
      a2 += L.LR[j + 3 * i] * L.LR[j + 3 * i];
      b2 += L.LI[i + 3 * j] * L.LI[i + 3 * j];
    }
    const double k = 2.0 * RSD_PI * (L.NI + 1) / sqrt(a2);
    if (L.lam * (L.NR + 0.5) < 6.0 * sqrt(b2) || k * k < 40.0 * 4.0 * L.lam * L.lam) return false;
  }
  return true;
}

struct ewald_dev_lists {
  int nimg = 0, Kh = 0;
  float rc2 = 0.f;
  const double *img = nullptr, *kv = nullptr, *coef = nullptr;
  const float4* imgf = nullptr;
  const unsigned short* etab = nullptr;  // rsd_real_epi_off (61), rsd_real_epi_mom
};

// One copy brings the lists and, for equal radii, the coefficients of the
// real-space epilogue to the device.
int upload_lists(rsd_ctx* ctx, cudaStream_t s, const ewald_lists& H, bool equal, double a, const rsd_lat_dev& L, double inv_pimu,
                 ewald_dev_lists* D) {
  const size_t ni = H.img.size() / 3, nk = H.kv.size() / 3;
  const size_t nt = 5 * ni + 3 * nk + RSD_REAL_EPI_NC;  // float4 = two doubles
  const size_t nd = nt + (61 + RSD_REAL_EPI_NC + 3) / 4;
  std::vector<double> h(nd, 0.0);
  float* f = reinterpret_cast<float*>(h.data());
  for (size_t i = 0; i < ni; i++)
    for (int j = 0; j < 3; j++) f[4 * i + j] = (float)H.img[3 * i + j];
  std::copy(H.img.begin(), H.img.end(), h.begin() + 2 * ni);
  std::copy(H.kv.begin(), H.kv.end(), h.begin() + 5 * ni);
  if (equal) {
    const double s1 = inv_pimu / (6.0 * a);
    rsd_real_epi_coef_scaled<double>(a, a, L.phix, s1, s1 / (a * a), h.data() + 5 * ni + 3 * nk);
    unsigned short* e = reinterpret_cast<unsigned short*>(h.data() + nt);
    for (int q = 0; q < 61; q++) e[q] = (unsigned short)rsd_real_epi_off(q);
    for (int k = 0; k < RSD_REAL_EPI_NC; k++) e[61 + k] = (unsigned short)rsd_real_epi_mom(k);
  }
  double* d = (double*)rsd_scratch(ctx, "ewald_lists", sizeof(double) * nd);
  if (!d) return RSD_ENOMEM;
  RSD_CUDA(ctx, cudaMemcpyAsync(d, h.data(), sizeof(double) * nd, cudaMemcpyHostToDevice, s));
  D->nimg = (int)ni;
  D->Kh = (int)nk;
  D->rc2 = (float)H.rc2;
  D->imgf = reinterpret_cast<const float4*>(d);
  D->img = d + 2 * ni;
  D->kv = d + 5 * ni;
  D->coef = d + 5 * ni + 3 * nk;
  D->etab = reinterpret_cast<const unsigned short*>(d + nt);
  return RSD_OK;
}

// The weights of D's vectors on stream ws, then the diagonal blocks on the
// side stream, beside the pair kernels: latency-bound kernels of one CTA (~65
// us).  Forked by the caller when ws is the side stream, else here.
template <typename S>
int assemble_self(rsd_ctx* ctx, int nn, const double* d_radii, double a0, bool equal, const rsd_lat_dev& L,
                  double inv_pimu, const ewald_dev_lists& D, cudaStream_t ws, rsd_fork& beside, const S& sk) {
  cudaStream_t s = beside.side;
  double* W = (double*)rsd_scratch(ctx, "ewald_weights", sizeof(double) * (size_t)D.Kh * 80);
  double* self = (double*)rsd_scratch(ctx, "ewald_self_sums", sizeof(double) * SELF_NMOM);
  if (!W || !self) return RSD_ENOMEM;
  const dim3 wg((unsigned)((D.Kh + 31) / 32), 2);
  if (equal) {
    pdl_launch(ewald_weights<true>, wg, 32, 0, ws, L, D.Kh, D.kv, a0, inv_pimu, W);
    if (ws != s) RSD_TRY(beside.fork());
    pdl_launch(ewald_self_sums<true>, 1, SELF_THREADS, 0, s, L, D.nimg, D.img, D.imgf, D.rc2, D.Kh, W, a0, inv_pimu, D.coef,
                                                     D.etab, self);
    pdl_launch(ewald_self_eq<S>, (121 * nn + 255) / 256, 256, 0, s, nn, self, sk);
  } else {
    pdl_launch(ewald_weights<false>, wg, 32, 0, ws, L, D.Kh, D.kv, a0, inv_pimu, W);
    if (ws != s) RSD_TRY(beside.fork());
    pdl_launch(ewald_self_sums<false>, 1, SELF_THREADS, 0, s, L, D.nimg, D.img, D.imgf, D.rc2, D.Kh, W, a0, inv_pimu, D.coef,
                                                      D.etab, self);
    pdl_launch(ewald_self<S>, (nn + 63) / 64, 64, 0, s, nn, L, self, d_radii, inv_pimu, sk);
  }
  RSD_CUDA(ctx, cudaGetLastError());
  return RSD_OK;
}

// FP64 form.  Lanes per pair, counted by what the exchanges cost: 8 keep the lanes' shares of ~77 images even and
// the exchanges at 87 additions per pair; below P64_WIDE pairs (N = 128)
// there are fewer groups of 8 than the FP64 pipes want warps, and 32 lanes
// take a pair.
constexpr int64_t P64_WIDE = 8192;
int assemble_fp64(rsd_ctx* ctx, int nn, const double* d_pos, const double* d_radii, double a0, bool equal,
                  rsd_lat_dev L, double inv_pimu, const DenseSink& sk) {
  cudaStream_t s = ctx->stream;
  const bool cube = !cubes_converged(L);
  if (!cube) L.lam *= EWALD64_SCALE;
  ewald_dev_lists D;
  RSD_TRY(upload_lists(ctx, s, cube ? ewald_cube_lists(L) : ewald_sphere_lists(L, L.lam, false), equal, a0, L,
                       inv_pimu, &D));
  RSD_TRY(rsd_side_stream(ctx));
  rsd_fork beside{ctx, ctx->side, ctx->ev_la[0], ctx->ev_la[1]};
  RSD_TRY(assemble_self(ctx, nn, d_radii, a0, equal, L, inv_pimu, D, s, beside, sk));
  if (nn < 2) return beside.join();
  double2* cs = (double2*)rsd_scratch(ctx, "ewald_trig", sizeof(double2) * (size_t)D.Kh * nn);
  const double* W = (const double*)rsd_scratch(ctx, "ewald_weights", sizeof(double) * (size_t)D.Kh * 80);
  if (!cs || !W) return RSD_ENOMEM;
  pdl_launch(ewald_trig, (unsigned)(((int64_t)nn * D.Kh + 127) / 128), 128, 0, s, nn, D.Kh, D.kv, d_pos, cs);
  const int64_t npair = (int64_t)nn * (nn - 1) / 2;
  auto go = [&](auto lanes, auto eq) {
    constexpr int G = decltype(lanes)::value;
    constexpr int PP = P64_THREADS / G;
    pdl_launch(ewald_pair64<G, decltype(eq)::value>, (unsigned)((npair + PP - 1) / PP), P64_THREADS, 0, s, 
        nn, npair, L, cube, D.nimg, D.img, D.imgf, D.rc2, D.Kh, W, cs, d_pos, d_radii, inv_pimu, D.coef, D.etab, sk);
  };
  using wide = std::integral_constant<int, 32>;
  using narrow = std::integral_constant<int, 8>;
  if (npair < P64_WIDE) {
    equal ? go(wide{}, std::true_type{}) : go(wide{}, std::false_type{});
  } else {
    equal ? go(narrow{}, std::true_type{}) : go(narrow{}, std::false_type{});
  }
  RSD_CUDA(ctx, cudaGetLastError());
  return beside.join();
}
}  // namespace

int rsd_ewald_assemble(rsd_ctx* ctx, int nn, const double* d_pos, const double* d_radii, const rsd_lattice* lat,
                       double mu_f, int precision, const double* h_radii, double* d_M, int64_t ldm, bool exported) {
  if (nn < 1 || ldm < 11LL * nn) return rsd_fail(ctx, RSD_EARG, "bad size nn=%d ldm=%lld", nn, (long long)ldm);
  rsd_lat_dev L = rsd_lat_pack(lat);
  if (precision == RSD_PREC_MIXED) L = mixed_lattice(ctx, L);
  if (L.NR > 40 || L.NI > 40) return rsd_fail(ctx, RSD_EARG, "image cubes too large (NR=%d NI=%d)", L.NR, L.NI);
  const double inv_pimu = 1.0 / (RSD_PI * mu_f);
  cudaStream_t s = ctx->stream;
  bool equal = true;
  for (int i = 1; i < nn && equal; i++) equal = h_radii[i] == h_radii[0];
  if (precision != RSD_PREC_MIXED)
    return assemble_fp64(ctx, nn, d_pos, d_radii, h_radii[0], equal, L, inv_pimu, DenseSink{d_M, ldm});
  // M as FP32 planes hi + lo (PlaneSink), in the buffer of the FP64 matrix
  const PlaneSink psk{reinterpret_cast<float*>(d_M), reinterpret_cast<float*>(d_M) + (size_t)ldm * (11LL * nn), ldm};
  RSD_TRY(rsd_side_stream(ctx));
  rsd_fork beside{ctx, ctx->side, ctx->ev_la[0], ctx->ev_la[1]};
  RSD_TRY(beside.fork());
  if (nn > 1) {
    dim3 blk(32, 4), grd((nn + 31) / 32, (nn + 3) / 4);
    {
      // Double-single: real images with lambda r < mixed_rcut (default 4.5)
      // and reciprocal vectors with k^2/(4 lambda^2) <= 3 pi mixed_kshell^2
      // (default 1); FP32 for the rest.  The FP32 error of a block follows
      // the largest FP32 term: at the defaults (with lambda x 1.75) a step's
      // velocities move by ~3e-11 and its stresslets by ~2e-10 relative.
      // Truncation: real images with lambda r >= mixed_rmax and reciprocal
      // vectors with k^2 / (4 lambda^2) >= mixed_kexp are dropped (each
      // changes a block by less than ~1e-12 of its largest entry at the
      // defaults 6.0 and 10 pi; the FP64 form keeps the whole cube).
      const double rc = ctx->mixed_rcut / L.lam, rc2 = rc * rc;
      const double rm = ctx->mixed_rmax / L.lam, rmax2 = rm * rm;
      const int ks = ctx->mixed_kshell;
      // double-single reciprocal vectors: k^2 / (4 lambda^2) <= 3 pi ks^2
      // (at the reference's lambda on a cubic cell, ks = 1 is the shell
      // max|n_i| <= 1); FP32 for the others below the truncation
      const double k2ds = 4.0 * L.lam * L.lam * 3.0 * RSD_PI * ks * ks;
      const double k2max = 4.0 * L.lam * L.lam * ctx->mixed_kexp;
      const int w = 2 * L.NI + 1, Kh = (w * w * w - 1) / 2;
      std::vector<int> h64, h32;
      for (int h = 0; h < Kh; h++) {
        int nx, ny, nz;
        half_space_index(h, L.NI, &nx, &ny, &nz);
        double k2 = 0.0;
        for (int j = 0; j < 3; j++) {
          const double kj = 2.0 * RSD_PI * (nx * L.LI[3 * j] + ny * L.LI[1 + 3 * j] + nz * L.LI[2 + 3 * j]);
          k2 += kj * kj;
        }
        if (k2 <= k2ds * (1.0 + 1e-12))
          h64.push_back(h);
        else if (k2 < k2max)
          h32.push_back(h);
      }
      const int K64 = (int)h64.size(), K32 = (int)h32.size();
      // one copy: the vector indices and, for equal radii, the coefficients of
      // the real-space epilogue (double-single, FP32)
      const size_t nidx = (h64.size() + h32.size() + 3) / 4 * 4;
      std::vector<int> up(nidx + 3 * RSD_REAL_EPI_NC + (61 + RSD_REAL_EPI_NC + 1) / 2, 0);
      std::copy(h64.begin(), h64.end(), up.begin());
      std::copy(h32.begin(), h32.end(), up.begin() + h64.size());
      if (equal) {
        double c[RSD_REAL_EPI_NC];
        const double s1 = inv_pimu / (6.0 * h_radii[0]);
        rsd_real_epi_coef_scaled<double>(h_radii[0], h_radii[0], L.phix, s1, s1 / (h_radii[0] * h_radii[0]), c);
        dsf* hr = reinterpret_cast<dsf*>(up.data() + nidx);
        float* hf = reinterpret_cast<float*>(hr + RSD_REAL_EPI_NC);
        for (int k = 0; k < RSD_REAL_EPI_NC; k++) {
          const float h = (float)c[k];
          hr[k].hi = hf[k] = h;
          hr[k].lo = (float)(c[k] - (double)h);
        }
        unsigned short* e = reinterpret_cast<unsigned short*>(hf + RSD_REAL_EPI_NC);
        for (int q = 0; q < 61; q++) e[q] = (unsigned short)rsd_real_epi_off(q);
        for (int k = 0; k < RSD_REAL_EPI_NC; k++) e[61 + k] = (unsigned short)rsd_real_epi_mom(k);
      }
      // Slices of a small system: so many that their CTAs (those above the
      // diagonal) come to two per SM, what the kernels' registers allow.  Sums in
      // several passes are asked for by the caller, and taken unsliced.
      int ctas = 0;
      for (unsigned y = 0; y < grd.y; y++) ctas += std::min((4 * (int)y + 3 + 31) / 32, (int)grd.x);
      const int S = std::min(EWALD_SLICES, 2 * ctx->sm_count / ctas);
      const bool sliced = equal && !exported && S >= 2 && ctx->mixed_real_passes == 1;
      if (sliced) RSD_TRY(real_slices(ctx, beside.side, S, grd, blk, nn, L, d_pos, (float)rc2, (float)rmax2));
      int* dh = (int*)rsd_scratch(ctx, "ewald_hlist", sizeof(int) * up.size());
      double* t64 = equal ? nullptr : (double*)rsd_scratch(ctx, "ewald_ktab64", sizeof(double) * (size_t)(K64 > 0 ? K64 : 1) * KW);
      float* t32 = equal ? nullptr : (float*)rsd_scratch(ctx, "ewald_ktab32", sizeof(float) * (size_t)(K32 > 0 ? K32 : 1) * KW);
      float4* c64 = (float4*)rsd_scratch(ctx, "ewald_trig64", sizeof(float4) * (size_t)(K64 > 0 ? K64 : 1) * nn);
      float2* c32 = (float2*)rsd_scratch(ctx, "ewald_trig32", sizeof(float2) * (size_t)(K32 > 0 ? K32 : 1) * nn);
      if (!dh || (!equal && (!t64 || !t32)) || !c64 || !c32) return RSD_ENOMEM;
      RSD_CUDA(ctx, cudaMemcpyAsync(dh, up.data(), sizeof(int) * up.size(), cudaMemcpyHostToDevice, s));
      const dsf* cr = reinterpret_cast<const dsf*>(dh + nidx);
      const float* cf = reinterpret_cast<const float*>(cr + RSD_REAL_EPI_NC);
      if (K64) {
        pdl_launch(ewald_trig_list<float4>, dim3((nn + 127) / 128, K64), 128, 0, s, nn, L, dh, d_pos, c64);
      }
      if (K32) {
        pdl_launch(ewald_trig_list<float2>, dim3((nn + 127) / 128, K32), 128, 0, s, nn, L, dh + K64, d_pos, c32);
      }
      if (equal) {
        float* w64 = (float*)rsd_scratch(ctx, "ewald_kblock64", sizeof(float) * (size_t)(K64 > 0 ? K64 : 1) * 2 * KBW);
        float* w32 = (float*)rsd_scratch(ctx, "ewald_kblock32", sizeof(float) * (size_t)(K32 > 0 ? K32 : 1) * KBW);
        if (!w64 || !w32) return RSD_ENOMEM;
        if (K64 + K32) {
          pdl_launch(ewald_kblock_lists, dim3((K64 + K32 + 31) / 32, 2), 32, 0, s, L, K64, K32, dh, h_radii[0], inv_pimu, w64, w32);
        }
        if (sliced) {
          RSD_TRY(join_slices(ctx, S, grd, blk, nn, K32, w32, c32, K64, w64, c64, cr,
                              reinterpret_cast<const unsigned short*>(cf + RSD_REAL_EPI_NC), psk));
        } else {
          pdl_launch(ewald_pair_kblock<false>, grd, blk, 0, s, nn, K32, w32, c32, K64, w64, c64, psk, 0, nullptr);
        }
      } else {
        if (K64) {
          pdl_launch(ewald_ktable_list<double>, (K64 + 127) / 128, 128, 0, s, L, K64, dh, t64);
        }
        if (K32) {
          pdl_launch(ewald_ktable_list<float>, (K32 + 127) / 128, 128, 0, s, L, K32, dh + K64, t32);
        }
        pdl_launch(ewald_pair_k_ds<PlaneSink>, grd, blk, 0, s, nn, L, K64, t64, c64, d_radii, inv_pimu, psk, 0);
        pdl_launch(ewald_pair_k<float, float2, PlaneSink>, grd, blk, 0, s, nn, L, K32, t32, c32, d_radii, inv_pimu, psk, 1);
      }
      if (sliced) {
      } else if (equal) {
        RSD_TRY(launch_real_eq(ctx, ctx->mixed_real_passes, grd, blk, nn, L, d_pos, cr, cf, (float)rc2, (float)rmax2, psk));
      } else {
        RSD_TRY(rsd_smem(ctx, ewald_pair_real_mix, (int)sizeof(RealMixShared)));
        pdl_launch(ewald_pair_real_mix, grd, blk, sizeof(RealMixShared), s, nn, L, d_pos, d_radii, inv_pimu, (float)rc2,
                   (float)rmax2, psk);
      }
    }
  }
  // last: the host makes their lists while the pair kernels run
  ewald_dev_lists D;
  RSD_TRY(upload_lists(ctx, beside.side, ewald_sphere_lists(L, L.lam, /*self_only=*/true), equal, h_radii[0], L,
                       inv_pimu, &D));
  RSD_TRY(assemble_self(ctx, nn, d_radii, h_radii[0], equal, L, inv_pimu, D, beside.side, beside, psk));
  RSD_CUDA(ctx, cudaGetLastError());
  return beside.join();
}
