// Kernel 2: two-body lubrication resistance R_lub - R_2B (lubmxcalc,
// src/hydro_lub.f90:22-308, with lubcalc 310-398 and lubtabcalc 400-525).
//
// Pipeline (all FP64, deterministic order):
//   lub_near      one warp per particle a: near partners b > a (s <= 4 in
//                 the minimum image), ballot-compacted -> count[a]
//   lub_scan      exclusive scan of the counts (one block)
//   lub_near      the same sweep writes the pair list, sorted by (a, b)
//   lub_pairs     one thread per near pair: the 19 resistance scalars and
//                 the projected two-body blocks (139 values per pair)
//   lub_cross     one thread per (pair, entry): the (a,b) and (b,a) blocks
//   lub_self      one thread per (particle, entry): the sum of the particle's
//                 own blocks over its pairs, in pair order
// The output is the grand layout L = [rfu rfe; rfe^T rse] (11N x 11N),
// scaled by 6 pi mu_f like hydro_lub.f90:304-306, either written over a
// zeroed matrix or added into one (arrangResist, src/matrices.f90:218-228).
#include <cuda_runtime.h>

#include "pdl.cuh"
#include "rsd_internal.cuh"

namespace {

constexpr int PB = 139;  // doubles per pair block
// offsets inside a pair block
constexpr int O_A11 = 0, O_A12 = 9, O_B11 = 18, O_B12 = 27, O_C11 = 36, O_C12 = 45;
constexpr int O_G11 = 54, O_G12 = 69, O_H11 = 84, O_H12 = 99, O_M = 114;

struct lub_dev_tab {
  const double *abc, *gh, *m;
  int nabc, ngh, nm;
};

__device__ void lubcalc_dev(const lub_dev_tab& t, double r, double* o) {
  if (r < 2.1) {
    const double xi = r - 2.0, invxi = 1.0 / xi, loginvxi = log(invxi), xiloginvxi = xi * loginvxi;
    o[0] = -1.23041 + 0.25 * invxi + 1.8918 * xi + 9.0 * loginvxi / 40.0 + 3.0 * xiloginvxi / 112.0;
    o[1] = -o[0] + 0.00312 - 0.0011 * xi;
    o[2] = -0.39394 + 0.95665 * xi + loginvxi / 6.0;
    o[3] = -o[2] + 0.004636 - 0.007049 * xi;
    o[4] = 0.408286 - 0.84055 * xi - loginvxi / 6.0 - xiloginvxi / 12.0;
    o[5] = -0.405978 + 0.833042 * xi + loginvxi / 6.0 + xiloginvxi / 12.0;
    o[6] = 0.0479 + 0.12494 * xi - xiloginvxi / 6.0;
    o[7] = -o[6] + 0.016869 + 0.049536 * xi;
    o[8] = -0.605434 + 0.939139 * xi + 4.0 * loginvxi / 15.0 + 94.0 * xiloginvxi / 375.0;
    o[9] = loginvxi / 15.0 + 62.0 * xiloginvxi / 375.0 - 0.219032 + 0.332843 * xi;
    o[10] = -1.16897 + 1.47882 * xi + invxi / 4.0 + 9.0 * loginvxi / 40.0 + 39.0 * xiloginvxi / 280.0;
    o[11] = -o[10] + 0.01 - 0.00167 * xi;
    o[12] = -0.2041 + 0.44226 * xi + loginvxi / 12.0 + xiloginvxi / 24.0;
    o[13] = -o[12] + 0.012265 - 0.02757 * xi;
    o[14] = -0.143777 + 0.264207 * xi + loginvxi / 30.0 + 137.0 * xiloginvxi / 1500.0;
    o[15] = -0.298166 + 0.534123 * xi + 2.0 * loginvxi / 15.0 + 113.0 * xiloginvxi / 1500.0;
    o[16] = invxi / 6.0 + 3.0 * loginvxi / 20.0 + 47.0 * xiloginvxi / 280.0 - 0.740815 + 0.706802 * xi;
    o[17] = -0.193518 + 0.553883 * xi + loginvxi / 12.0 - 29.0 * xiloginvxi / 500.0;
    o[18] = 0.00645755 - 0.021142 * xi;
    return;
  }
#pragma unroll
  for (int q = 0; q < 19; q++) o[q] = 0.0;
  for (int i = 0; i < t.nabc - 1; i++) {
    const double* a = t.abc + 11 * i;
    const double* b = a + 11;
    if (a[0] <= r && b[0] > r) {
      const double f = (r - a[0]) / (b[0] - a[0]);
#pragma unroll
      for (int q = 0; q < 10; q++) o[q] = a[q + 1] + f * (b[q + 1] - a[q + 1]);
      break;
    }
  }
  for (int i = 0; i < t.ngh - 1; i++) {
    const double* a = t.gh + 7 * i;
    const double* b = a + 7;
    if (a[0] <= r && b[0] > r) {
      const double f = (r - a[0]) / (b[0] - a[0]);
#pragma unroll
      for (int q = 0; q < 6; q++) o[10 + q] = a[q + 1] + f * (b[q + 1] - a[q + 1]);
      break;
    }
  }
  for (int i = 0; i < t.nm - 1; i++) {
    const double* a = t.m + 4 * i;
    const double* b = a + 4;
    if (a[0] <= r && b[0] > r) {
      const double f = (r - a[0]) / (b[0] - a[0]);
#pragma unroll
      for (int q = 0; q < 3; q++) o[16 + q] = (a[q + 1] + f * (b[q + 1] - a[q + 1])) / 2.0;
      break;
    }
  }
}

// FP32 screen of a pair: false where it is clearly beyond the cut-off s = 4
__device__ __forceinline__ bool maybe_near(const float* LR, const float* LI, int is_period, const float R[3], float asum) {
  if (is_period) return rsd_maybe_within_f32(LR, LI, R, 2.0f * asum);
  const float lim = 2.0f * asum * 1.001f + 1e-3f;
  return !(R[0] * R[0] + R[1] * R[1] + R[2] * R[2] > lim * lim);
}

__device__ inline bool near_pair(const rsd_lat_dev& L, int is_period, const double* pos, const double* radii, int a,
                                 int b) {
  double R[3] = {pos[3 * a] - pos[3 * b], pos[3 * a + 1] - pos[3 * b + 1], pos[3 * a + 2] - pos[3 * b + 2]};
  double r = sqrt(R[0] * R[0] + R[1] * R[1] + R[2] * R[2]);
  if (is_period) rsd_skew_correction(L.LR, L.LI, R, &r);
  const double s = r / (0.5 * (radii[a] + radii[b]));
  return !(s > 4.0);
}

// The near partners b > a of a particle, ascending, one warp per particle:
// lanes screen 32 partners at a time in FP32 and the survivors are collected,
// so that the FP64 test (a warp issues an FP64 instruction every 64 cycles)
// runs over full warps of them.  LIST: the pairs are written from off[a] on;
// otherwise they are counted.
constexpr int LUB_WARPS = 8, LUB_CAND = 64;
template <bool LIST>
__global__ void lub_near(int nn, int nb, int is_period, rsd_lat_dev L, const double* __restrict__ pos,
                         const double* __restrict__ radii, int* __restrict__ count, const int* __restrict__ off,
                         int2* __restrict__ pairs) {
  pdl_enter();
  __shared__ int cand[LUB_WARPS][LUB_CAND];
  const int warp = threadIdx.x / 32, a = blockIdx.x * LUB_WARPS + warp, lane = threadIdx.x & 31;
  if (a >= nn) return;
  float LR[9], LI[9];
#pragma unroll
  for (int k = 0; k < 9; k++) {
    LR[k] = (float)L.LR[k];
    LI[k] = (float)L.LI[k];
  }
  const double x0 = pos[3 * a], x1 = pos[3 * a + 1], x2 = pos[3 * a + 2];
  const float ra = (float)radii[a];
  const unsigned below = (1u << lane) - 1;
  int found = 0, nc = 0;
  auto flush = [&](int n) {  // tests the first n <= 32 candidates and drops them
    __syncwarp();
    const int b = lane < n ? cand[warp][lane] : -1;
    const bool nr = b >= 0 && near_pair(L, is_period, pos, radii, a, b);
    const unsigned m = __ballot_sync(0xffffffffu, nr);
    if (LIST && nr) pairs[off[a] + found + __popc(m & below)] = make_int2(a, b);
    found += __popc(m);
    const int rest = lane + n < nc ? cand[warp][lane + n] : 0;
    __syncwarp();
    cand[warp][lane] = rest;
    nc -= n;
    __syncwarp();
  };
  if (a < nn - nb)
    for (int b0 = a + 1; b0 < nn; b0 += 32) {
      const int b = b0 + lane;
      bool c = false;
      if (b < nn) {
        const float R[3] = {(float)(x0 - pos[3 * b]), (float)(x1 - pos[3 * b + 1]), (float)(x2 - pos[3 * b + 2])};
        c = maybe_near(LR, LI, is_period, R, ra + (float)radii[b]);
      }
      const unsigned m = __ballot_sync(0xffffffffu, c);
      if (c) cand[warp][nc + __popc(m & below)] = b;
      nc += __popc(m);
      if (nc >= 32) flush(32);
    }
  if (nc > 0) flush(nc);
  if (!LIST && lane == 0) count[a] = found;
}

// exclusive scan of count[0..n) into off[0..n], one block of 1024 threads
__global__ void lub_scan(int n, const int* __restrict__ count, int* __restrict__ off) {
  pdl_enter();
  __shared__ int part[1024];
  const int t = threadIdx.x;
  const int per = (n + 1023) / 1024;
  const int lo = t * per, hi = min(n, lo + per);
  int s = 0;
  for (int i = lo; i < hi; i++) s += count[i];
  part[t] = s;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    int v = t >= d ? part[t - d] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  int base = t ? part[t - 1] : 0;
  for (int i = lo; i < hi; i++) {
    off[i] = base;
    base += count[i];
  }
  if (t == 1023) off[n] = part[1023];
}

// The two-body blocks of a pair (hydro_lub.f90:95-160 with rtd_front and
// DD_transY2, tensors.f90:966-1023), in closed form.  With v_m = Y_m e and q_m
// = e.v_m (Y_m the symmetric traceless basis, Y_m : Y_n = delta_mn) the tensor
// sums of the reference contract to
//   G(m, c) = x q_m e_c + y (2 v_mc - 2 q_m e_c)
//   H(m, c) = 2 y (e x v_m)_c
//   M(m, n) = 3/2 x q_m q_n + 2 y (v_m.v_n - q_m q_n) + z (delta_mn - 2 v_m.v_n + q_m q_n / 2)
// about 600 FP64 instructions a pair where the sums take 9700.  A warp issues
// one every 64 cycles, so this is the kernel's time: 300 -> 72 us (N = 512).
__device__ inline void pair_tensors(const double* o, const double e[3], double* B) {
  const double x11a = o[0], x12a = o[1], y11a = o[2], y12a = o[3], y11b = o[4], y12b = o[5], x11c = o[6],
               x12c = o[7], y11c = o[8], y12c = o[9], x11g = o[10], x12g = o[11], y11g = o[12], y12g = o[13],
               y11h = o[14], y12h = o[15], xm = o[16], ym = o[17], zm = o[18];
#pragma unroll
  for (int j = 0; j < 3; j++)
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double ee = e[i] * e[j], t = (i == j ? 1.0 : 0.0) - ee;
      // eps_ijk e_k
      const double pe = i == j ? 0.0 : ((j - i + 3) % 3 == 1 ? e[3 - i - j] : -e[3 - i - j]);
      B[O_A11 + i + 3 * j] = x11a * ee + y11a * t;
      B[O_A12 + i + 3 * j] = x12a * ee + y12a * t;
      B[O_B11 + i + 3 * j] = y11b * pe;
      B[O_B12 + i + 3 * j] = y12b * pe;
      B[O_C11 + i + 3 * j] = x11c * ee + y11c * t;
      B[O_C12 + i + 3 * j] = x12c * ee + y12c * t;
    }
  const double s2 = 0.70710678118654752440, s6 = 0.40824829046386301637;  // 1/sqrt 2, 1/sqrt 6
  const double v[5][3] = {{s2 * e[1], s2 * e[0], 0.0},
                          {0.0, -s2 * e[2], -s2 * e[1]},
                          {-s6 * e[0], -s6 * e[1], 2.0 * s6 * e[2]},
                          {-s2 * e[2], 0.0, -s2 * e[0]},
                          {s2 * e[0], -s2 * e[1], 0.0}};
  double q[5];
#pragma unroll
  for (int m = 0; m < 5; m++) q[m] = e[0] * v[m][0] + e[1] * v[m][1] + e[2] * v[m][2];
#pragma unroll
  for (int m = 0; m < 5; m++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double qe = q[m] * e[c], w = 2.0 * (v[m][c] - qe);
      const double h = 2.0 * (e[(c + 1) % 3] * v[m][(c + 2) % 3] - e[(c + 2) % 3] * v[m][(c + 1) % 3]);
      B[O_G11 + m + 5 * c] = x11g * qe + y11g * w;
      B[O_G12 + m + 5 * c] = x12g * qe + y12g * w;
      B[O_H11 + m + 5 * c] = y11h * h;
      B[O_H12 + m + 5 * c] = y12h * h;
    }
#pragma unroll
  for (int m = 0; m < 5; m++)
#pragma unroll
    for (int n = m; n < 5; n++) {
      const double qq = q[m] * q[n], vv = v[m][0] * v[n][0] + v[m][1] * v[n][1] + v[m][2] * v[n][2];
      const double t = 1.5 * xm * qq + 2.0 * ym * (vv - qq) + zm * ((m == n ? 1.0 : 0.0) - 2.0 * vv + 0.5 * qq);
      B[O_M + m + 5 * n] = t;
      B[O_M + n + 5 * m] = t;
    }
}

__global__ void __launch_bounds__(32) lub_pairs(int npair, lub_dev_tab tab, int is_period, rsd_lat_dev L,
                                                const double* __restrict__ pos, const double* __restrict__ radii,
                                                const int2* __restrict__ pairs, double* __restrict__ blk,
                                                int* __restrict__ contacts) {
  pdl_enter();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npair) return;
  const int a = pairs[p].x, b = pairs[p].y;
  double R[3] = {pos[3 * a] - pos[3 * b], pos[3 * a + 1] - pos[3 * b + 1], pos[3 * a + 2] - pos[3 * b + 2]};
  double r = sqrt(R[0] * R[0] + R[1] * R[1] + R[2] * R[2]);
  if (is_period) rsd_skew_correction(L.LR, L.LI, R, &r);
  double s = r / (0.5 * (radii[a] + radii[b]));
  if (s <= 2.0) {  // hydro_lub.f90:85-92: report and mirror
    atomicAdd(contacts, 1);
    s = 4.00001 - s;
  }
  double o[19];
  lubcalc_dev(tab, s, o);
  const double e[3] = {R[0] / r, R[1] / r, R[2] / r};
  pair_tensors(o, e, blk + (size_t)p * PB);
}

__device__ inline void lput(double* L, int64_t ld, int r, int c, double v, int acc) {
  double* p = L + (int64_t)r + (int64_t)c * ld;
  *p = acc ? *p + v : v;
}

// grand-layout index of component k (0..10) of particle part
__device__ inline int gidx(int N, int part, int k) {
  return k < 3 ? 3 * part + k : (k < 6 ? 3 * N + 3 * part + k - 3 : 6 * N + 5 * part + k - 6);
}

// Entry (r, c) of the (a,b) particle block (ab = true) or of the (b,a)
// block (ab = false) of pair block B, r and c in 0..10.
__device__ inline double pair_entry(const double* B, int r, int c, bool ab) {
  if (r < 3 && c < 3) return ab ? B[O_A12 + r + 3 * c] : B[O_A12 + c + 3 * r];  // TT, (b,a) mirrored
  if (r >= 3 && r < 6 && c >= 3 && c < 6)                                          // RR
    return ab ? B[O_C12 + (r - 3) + 3 * (c - 3)] : B[O_C12 + (c - 3) + 3 * (r - 3)];
  if (r >= 3 && r < 6 && c < 3) return (ab ? 1.0 : -1.0) * B[O_B12 + (r - 3) + 3 * c];   // RT: b12, b21 = -b12
  if (r < 3 && c >= 3 && c < 6) return (ab ? -1.0 : 1.0) * B[O_B12 + (c - 3) + 3 * r];   // TR = RT^T
  if (r >= 6 && c < 3) return (ab ? 1.0 : -1.0) * B[O_G12 + (r - 6) + 5 * c];            // G: g12, -g12
  if (r < 3 && c >= 6) return (ab ? -1.0 : 1.0) * B[O_G12 + (c - 6) + 5 * r];            // rfe = QP^T
  if (r >= 6 && c >= 3 && c < 6) return B[O_H12 + (r - 6) + 5 * (c - 3)];               // H: h12 both ways
  if (r >= 3 && r < 6 && c >= 6) return B[O_H12 + (c - 6) + 5 * (r - 3)];
  return B[O_M + (r - 6) + 5 * (c - 6)];                                                 // QQ: mmx both ways
}

// Entry (r, c) of a particle's own block contributed by pair block B;
// sgn = +1 when the particle is the pair's first, -1 when its second.
__device__ inline double self_entry(const double* B, int r, int c, double sgn) {
  if (r < 3 && c < 3) return B[O_A11 + r + 3 * c];
  if (r >= 3 && r < 6 && c >= 3 && c < 6) return B[O_C11 + (r - 3) + 3 * (c - 3)];
  if (r >= 3 && r < 6 && c < 3) return sgn * B[O_B11 + (r - 3) + 3 * c];
  if (r < 3 && c >= 3 && c < 6) return sgn * B[O_B11 + (c - 3) + 3 * r];
  if (r >= 6 && c < 3) return sgn * B[O_G11 + (r - 6) + 5 * c];
  if (r < 3 && c >= 6) return sgn * B[O_G11 + (c - 6) + 5 * r];
  if (r >= 6 && c >= 3 && c < 6) return B[O_H11 + (r - 6) + 5 * (c - 3)];
  if (r >= 3 && r < 6 && c >= 6) return B[O_H11 + (c - 6) + 5 * (r - 3)];
  return B[O_M + (r - 6) + 5 * (c - 6)];
}

// 121 entries of the (a,b) block and 121 of the (b,a) block per pair
__global__ void lub_cross(int npair, int N, const int2* __restrict__ pairs, const double* __restrict__ blk,
                          double scale, double* __restrict__ L, int64_t ld, int acc) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)npair * 121) return;
  const int p = (int)(t / 121), e = (int)(t % 121);
  const int a = pairs[p].x, b = pairs[p].y;
  const double* B = blk + (size_t)p * PB;
  const int r = e % 11, c = e / 11;  // position inside an 11x11 particle block
  lput(L, ld, gidx(N, a, r), gidx(N, b, c), pair_entry(B, r, c, true) * scale, acc);
  lput(L, ld, gidx(N, b, r), gidx(N, a, c), pair_entry(B, r, c, false) * scale, acc);
}

// Second-particle lists: for each particle u, the pairs (a,u) with a < u,
// in pair order (which is a-ascending, the order lubmxcalc adds them in).
__global__ void lub_second_count(int npair, const int2* __restrict__ pairs, int* __restrict__ cnt2) {
  pdl_enter();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < npair) atomicAdd(&cnt2[pairs[p].y], 1);
}

__global__ void lub_second_fill(int npair, const int2* __restrict__ pairs, const int* __restrict__ off2,
                                int* __restrict__ cur, int* __restrict__ list2) {
  pdl_enter();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npair) return;
  const int b = pairs[p].y;
  list2[off2[b] + atomicAdd(&cur[b], 1)] = p;
}

// list2 in pair order: an entry's place is the number of smaller ones in its
// particle's list, a thread per entry
__global__ void lub_second_rank(int npair, const int2* __restrict__ pairs, const int* __restrict__ off2,
                                const int* __restrict__ raw, int* __restrict__ list2) {
  pdl_enter();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npair) return;
  const int u = pairs[p].y, lo = off2[u], hi = off2[u + 1];
  int k = lo;
  for (int q = lo; q < hi; q++) k += raw[q] < p;
  list2[k] = p;
}

// self block of particle u: its pairs as second particle, then as first,
// in the order lubmxcalc visits them.  Written into L (grand layout) or,
// when L is null, into self[u * 121 + r + 11 c].
__global__ void lub_self(int N, const int* __restrict__ off, const int* __restrict__ off2,
                         const int* __restrict__ list2, const double* __restrict__ blk, double scale,
                         double* __restrict__ L, int64_t ld, int acc, double* __restrict__ self) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)N * 121) return;
  const int u = (int)(t / 121), e = (int)(t % 121);
  const int r = e % 11, c = e / 11;
  double v = 0.0;
  for (int q = off2[u]; q < off2[u + 1]; q++) v += self_entry(blk + (size_t)list2[q] * PB, r, c, -1.0);
  for (int q = off[u]; q < off[u + 1]; q++) v += self_entry(blk + (size_t)q * PB, r, c, 1.0);
  if (L)
    lput(L, ld, gidx(N, u, r), gidx(N, u, c), v * scale, acc);
  else
    self[t] = v * scale;
}

// Position and sign of entry (r, c) in a pair block: pair_entry as a table
// lookup, for the block of the pair's first particle (ab) or its second.
__device__ inline void pair_pos(int r, int c, bool ab, int* off, double* sgn) {
  const int R = r < 3 ? 0 : (r < 6 ? 1 : 2), C = c < 3 ? 0 : (c < 6 ? 1 : 2);
  const int i = R == 2 ? r - 6 : r - 3 * R, j = C == 2 ? c - 6 : c - 3 * C;
  *sgn = 1.0;
  if (R == C && R < 2) {
    *off = (R ? O_C12 : O_A12) + (ab ? i + 3 * j : j + 3 * i);
  } else if (R == 2 && C == 2) {
    *off = O_M + i + 5 * j;
  } else if (R < 2 && C < 2) {
    *off = O_B12 + (R ? i + 3 * j : j + 3 * i);
    *sgn = (R == 1) == ab ? 1.0 : -1.0;
  } else {
    const int p = R == 2 ? C : R;  // the velocity section: 0 G, 1 H
    *off = (p ? O_H12 : O_G12) + (R == 2 ? i + 5 * j : j + 5 * i);
    if (p == 0) *sgn = (R == 2) == ab ? 1.0 : -1.0;
  }
}

// y = L w for the sparse operator: the particle's self block, then its pairs
// as first and as second particle.  One CTA per (particle, right-hand side),
// a thread per entry (r, c) of its 11 x 11 blocks: the position in the pair
// block is fixed per thread, a neighbour costs one multiply-add of each, and
// the 11 columns are added at the end in a fixed order.  Bound by the FP64
// pipe and the latency of the neighbour loop.  ABS: the sum of the terms' sizes,
// |L| |w| (blocks of several pairs taken whole).
template <bool ABS>
__global__ void __launch_bounds__(128) lub_spmv_w(int N, const int* __restrict__ off, const int* __restrict__ off2,
                                                  const int* __restrict__ list2, const int2* __restrict__ pairs,
                                                  const double* __restrict__ blk, const double* __restrict__ self,
                                                  double scale, const double* __restrict__ w, int64_t ldw,
                                                  double* __restrict__ y, int64_t ldy) {
  pdl_enter();
  __shared__ double sv[121], pv[121];
  const int u = blockIdx.x, t = threadIdx.x, r = t % 11, c = t / 11;
  const double* wc = w + blockIdx.y * ldw;
  if (t < 121) {
    int oa, ob;
    double sa, sb;
    pair_pos(r, c, true, &oa, &sa);
    pair_pos(r, c, false, &ob, &sb);
    auto term = [](double x) { return ABS ? fabs(x) : x; };
    if (ABS) sa = sb = 1.0;
    const int wbase = c < 3 ? c : (c < 6 ? 3 * N + c - 3 : 6 * N + c - 6), wstep = c < 6 ? 3 : 5;
    sv[t] = term(self[(size_t)u * 121 + t] * wc[wbase + wstep * u]);
    double va = 0.0, vb = 0.0;
    const int p1 = off[u + 1], q1 = off2[u + 1];
#pragma unroll 4
    for (int p = off[u]; p < p1; p++) va = fma(term(blk[(size_t)p * PB + oa]), term(wc[wbase + wstep * pairs[p].y]), va);
#pragma unroll 4
    for (int q = off2[u]; q < q1; q++) {
      const int p = list2[q];
      vb = fma(term(blk[(size_t)p * PB + ob]), term(wc[wbase + wstep * pairs[p].x]), vb);
    }
    pv[t] = sa * va + sb * vb;
  }
  __syncthreads();
  if (t < 11) {
    double vs = 0.0, vp = 0.0;
#pragma unroll
    for (int k = 0; k < 11; k++) {
      vs += sv[t + 11 * k];
      vp += pv[t + 11 * k];
    }
    y[gidx(N, u, t) + blockIdx.y * ldy] = vs + vp * scale;
  }
}

// A (ld lda) += the force/torque-velocity part L_PP of the sparse
// operator: pair blocks (each entry of A is touched by at most one pair or
// self block, so no two threads add to the same entry)
template <typename T>
__global__ void lub_pp_pairs(int npair, int N, const int2* __restrict__ pairs, const double* __restrict__ blk,
                             double scale, T* __restrict__ A, int64_t lda) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)npair * 36) return;
  const int p = (int)(t / 36), e = (int)(t % 36);
  const int r = e % 6, c = e / 6;
  const int a = pairs[p].x, b = pairs[p].y;
  const double* B = blk + (size_t)p * PB;
  A[gidx(N, a, r) + gidx(N, b, c) * lda] += (T)(pair_entry(B, r, c, true) * scale);
  A[gidx(N, b, r) + gidx(N, a, c) * lda] += (T)(pair_entry(B, r, c, false) * scale);
}

template <typename T>
__global__ void lub_pp_self(int N, const double* __restrict__ self, T* __restrict__ A, int64_t lda) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)N * 36) return;
  const int u = (int)(t / 36), e = (int)(t % 36);
  const int r = e % 6, c = e / 6;
  A[gidx(N, u, r) + gidx(N, u, c) * lda] += (T)self[(size_t)u * 121 + r + 11 * c];
}

__global__ void zero_matrix(int64_t rows, int64_t cols, double* __restrict__ A, int64_t ld) {
  pdl_enter();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= rows * cols) return;
  A[(t % rows) + (t / rows) * ld] = 0.0;
}

}  // namespace

static double* lubtab_device(rsd_ctx* ctx, const rsd_lubtab* tab) {
  rsd_lubtab* t = const_cast<rsd_lubtab*>(tab);
  auto it = t->dev.find(ctx->device);
  if (it != t->dev.end()) return it->second;
  double* d = nullptr;
  const size_t n = 64 * 11 + 64 * 7 + 64 * 4;
  if (cudaMalloc(&d, n * sizeof(double)) != cudaSuccess) return nullptr;
  cudaMemcpy(d, t->abc, 64 * 11 * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(d + 64 * 11, t->gh, 64 * 7 * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(d + 64 * 18, t->m, 64 * 4 * sizeof(double), cudaMemcpyHostToDevice);
  t->dev[ctx->device] = d;
  return d;
}

constexpr int LUB_NPAIR = 26;  // the mirror word that takes the pair count

// The pair stage shared by the dense and the sparse assembly: near-pair
// list, pair blocks (unscaled), second-particle lists and contact count.
// The host waits for the pair count in between, so that a caller with other
// work to launch calls rsd_lub_begin first.
int rsd_lub_begin(rsd_ctx* ctx, cudaStream_t s, int nn, int nb, int is_period, const double* d_pos,
                  const double* d_radii, const rsd_lattice* lat) {
  int* cnt = (int*)rsd_scratch(ctx, "lub_count", sizeof(int) * (nn + 1));
  int* off = (int*)rsd_scratch(ctx, "lub_off", sizeof(int) * (nn + 1));
  if (!cnt || !off) return RSD_ENOMEM;
  pdl_launch(lub_near<false>, (nn + LUB_WARPS - 1) / LUB_WARPS, 32 * LUB_WARPS, 0, s, nn, nb, is_period, rsd_lat_pack(lat),
                                                                              d_pos, d_radii, cnt, nullptr, nullptr);
  pdl_launch(lub_scan, 1, 1024, 0, s, nn, cnt, off);
  RSD_CUDA(ctx, cudaMemcpyAsync(ctx->h_info + LUB_NPAIR, off + nn, sizeof(int), cudaMemcpyDeviceToHost, s));
  return RSD_OK;
}

static int lub_pair_stage(rsd_ctx* ctx, cudaStream_t s, const rsd_lubtab* tab, int nn, int nb, int is_period,
                          const double* d_pos, const double* d_radii, const rsd_lattice* lat, rsd_lub_sparse* sp) {
  double* dt = lubtab_device(ctx, tab);
  if (!dt) return rsd_fail(ctx, RSD_ENOMEM, "lub table upload failed");
  lub_dev_tab T{dt, dt + 64 * 11, dt + 64 * 18, tab->nabc, tab->ngh, tab->nm};
  rsd_lat_dev Ld = rsd_lat_pack(lat);
  const int* off = (const int*)rsd_scratch(ctx, "lub_off", sizeof(int) * (nn + 1));
  if (!off) return RSD_ENOMEM;
  const unsigned ng = (unsigned)((nn + LUB_WARPS - 1) / LUB_WARPS);
  RSD_CUDA(ctx, cudaStreamSynchronize(s));
  const int npair = ctx->h_info[LUB_NPAIR];
  int* dcon = ctx->d_info + RSD_INFO_CONTACTS;
  int2* pairs = (int2*)rsd_scratch(ctx, "lub_pairs", sizeof(int2) * (size_t)(npair > 0 ? npair : 1));
  double* blk = (double*)rsd_scratch(ctx, "lub_blocks", sizeof(double) * PB * (size_t)(npair > 0 ? npair : 1));
  int* cnt2 = (int*)rsd_scratch(ctx, "lub_count2", sizeof(int) * (nn + 1));
  int* off2 = (int*)rsd_scratch(ctx, "lub_off2", sizeof(int) * (nn + 1));
  int* cur = (int*)rsd_scratch(ctx, "lub_cur", sizeof(int) * (nn + 1));
  int* list2 = (int*)rsd_scratch(ctx, "lub_list2", sizeof(int) * 2 * (size_t)(npair > 0 ? npair : 1));
  int* raw2 = list2 ? list2 + npair : nullptr;
  if (!pairs || !blk || !cnt2 || !off2 || !cur || !list2) return RSD_ENOMEM;
  RSD_CUDA(ctx, cudaMemsetAsync(dcon, 0, sizeof(int), s));
  RSD_CUDA(ctx, cudaMemsetAsync(cnt2, 0, sizeof(int) * (nn + 1), s));
  RSD_CUDA(ctx, cudaMemsetAsync(cur, 0, sizeof(int) * (nn + 1), s));
  if (npair > 0) {
    pdl_launch(lub_near<true>, ng, 32 * LUB_WARPS, 0, s, nn, nb, is_period, Ld, d_pos, d_radii, nullptr, off, pairs);
    pdl_launch(lub_pairs, (npair + 31) / 32, 32, 0, s, npair, T, is_period, Ld, d_pos, d_radii, pairs, blk, dcon);
    pdl_launch(lub_second_count, (npair + 255) / 256, 256, 0, s, npair, pairs, cnt2);
    pdl_launch(lub_scan, 1, 1024, 0, s, nn, cnt2, off2);
    pdl_launch(lub_second_fill, (npair + 255) / 256, 256, 0, s, npair, pairs, off2, cur, raw2);
    pdl_launch(lub_second_rank, (npair + 255) / 256, 256, 0, s, npair, pairs, off2, raw2, list2);
  } else {
    RSD_CUDA(ctx, cudaMemsetAsync(off2, 0, sizeof(int) * (nn + 1), s));
  }
  RSD_CUDA(ctx, cudaMemcpyAsync(ctx->h_info + RSD_INFO_CONTACTS, dcon, sizeof(int), cudaMemcpyDeviceToHost, s));
  sp->nn = nn;
  sp->npair = npair;
  sp->pairs = pairs;
  sp->blk = blk;
  sp->off = off;
  sp->off2 = off2;
  sp->list2 = list2;
  return RSD_OK;
}

int rsd_lub_assemble(rsd_ctx* ctx, const rsd_lubtab* tab, int nn, int nb, int is_period, const double* d_pos,
                     const double* d_radii, const rsd_lattice* lat, double mu_f, double* d_L, int64_t ldl,
                     int accumulate, int* n_contact) {
  if (!tab) return rsd_fail(ctx, RSD_EARG, "no lubrication tables");
  if (nn < 1 || ldl < 11LL * nn) return rsd_fail(ctx, RSD_EARG, "bad size nn=%d ldl=%lld", nn, (long long)ldl);
  cudaStream_t s = ctx->stream;
  if (!accumulate) {
    const int64_t tot = 121LL * nn * nn;
    pdl_launch(zero_matrix, (unsigned)((tot + 255) / 256), 256, 0, s, 11LL * nn, 11LL * nn, d_L, ldl);
  }
  rsd_lub_sparse sp;
  RSD_TRY(rsd_lub_begin(ctx, s, nn, nb, is_period, d_pos, d_radii, lat));
  RSD_TRY(lub_pair_stage(ctx, s, tab, nn, nb, is_period, d_pos, d_radii, lat, &sp));
  const double scale = 6.0 * (RSD_PI * mu_f);
  if (sp.npair > 0) {
    const int64_t tc = 121LL * sp.npair;
    pdl_launch(lub_cross, (unsigned)((tc + 255) / 256), 256, 0, s, sp.npair, nn, sp.pairs, sp.blk, scale, d_L, ldl, 1);
    const int64_t ts = 121LL * nn;
    pdl_launch(lub_self, (unsigned)((ts + 255) / 256), 256, 0, s, nn, sp.off, sp.off2, sp.list2, sp.blk, scale, d_L, ldl, 1,
                                                            nullptr);
  }
  RSD_CUDA(ctx, cudaGetLastError());
  if (n_contact) {
    RSD_CUDA(ctx, cudaStreamSynchronize(s));
    *n_contact = ctx->h_info[RSD_INFO_CONTACTS];
  }
  return RSD_OK;
}

// Sparse form for the mixed-precision refinement: the same pair blocks and
// the per-particle self blocks (scaled), no dense 11N x 11N matrix.
int rsd_lub_build_sparse(rsd_ctx* ctx, cudaStream_t s, const rsd_lubtab* tab, int nn, int nb, int is_period,
                         const double* d_pos, const double* d_radii, const rsd_lattice* lat, double mu_f,
                         rsd_lub_sparse* sp) {
  if (!tab) return rsd_fail(ctx, RSD_EARG, "no lubrication tables");
  if (nn < 1) return rsd_fail(ctx, RSD_EARG, "bad size nn=%d", nn);
  double* self = (double*)rsd_scratch(ctx, "lub_self_blocks", sizeof(double) * 121 * (size_t)nn);
  if (!self) return RSD_ENOMEM;
  RSD_TRY(lub_pair_stage(ctx, s, tab, nn, nb, is_period, d_pos, d_radii, lat, sp));
  sp->scale = 6.0 * (RSD_PI * mu_f);
  sp->self = self;
  const int64_t ts = 121LL * nn;
  pdl_launch(lub_self, (unsigned)((ts + 255) / 256), 256, 0, s, nn, sp->off, sp->off2, sp->list2, sp->blk, sp->scale,
                                                          nullptr, 0, 0, self);
  RSD_CUDA(ctx, cudaGetLastError());
  return RSD_OK;
}

// y (11N x nr, grand layout, ld ldy) = L w
int rsd_lub_spmv(rsd_ctx* ctx, const rsd_lub_sparse* sp, int nr, const double* w, int64_t ldw, double* y,
                 int64_t ldy) {
  pdl_launch(lub_spmv_w<false>, dim3(sp->nn, nr), 128, 0, ctx->stream, sp->nn, sp->off, sp->off2, sp->list2, sp->pairs,
             sp->blk, sp->self, sp->scale, w, ldw, y, ldy);
  RSD_CUDA(ctx, cudaGetLastError());
  return RSD_OK;
}

// y (11N) = |L| |w|
int rsd_lub_absmv(rsd_ctx* ctx, const rsd_lub_sparse* sp, const double* w, double* y) {
  const int64_t n = 11LL * sp->nn;
  pdl_launch(lub_spmv_w<true>, dim3(sp->nn, 1), 128, 0, ctx->stream, sp->nn, sp->off, sp->off2, sp->list2, sp->pairs,
             sp->blk, sp->self, sp->scale, w, n, y, n);
  RSD_CUDA(ctx, cudaGetLastError());
  return RSD_OK;
}

// A (6N x 6N, ld lda) += L_PP
template <typename T>
static int lub_add_pp(rsd_ctx* ctx, const rsd_lub_sparse* sp, T* A, int64_t lda) {
  cudaStream_t s = ctx->stream;
  if (sp->npair > 0) {
    const int64_t tp = 36LL * sp->npair;
    pdl_launch(lub_pp_pairs<T>, (unsigned)((tp + 255) / 256), 256, 0, s, sp->npair, sp->nn, sp->pairs, sp->blk, sp->scale, A,
                                                                 lda);
  }
  const int64_t ts = 36LL * sp->nn;
  pdl_launch(lub_pp_self<T>, (unsigned)((ts + 255) / 256), 256, 0, s, sp->nn, sp->self, A, lda);
  RSD_CUDA(ctx, cudaGetLastError());
  return RSD_OK;
}
int rsd_lub_add_pp_f32(rsd_ctx* ctx, const rsd_lub_sparse* sp, float* A, int64_t lda) {
  return lub_add_pp<float>(ctx, sp, A, lda);
}
int rsd_lub_add_pp_f64(rsd_ctx* ctx, const rsd_lub_sparse* sp, double* A, int64_t lda) {
  return lub_add_pp<double>(ctx, sp, A, lda);
}
