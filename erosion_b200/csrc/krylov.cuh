// One Arnoldi step of GMRES on the device: classical Gram-Schmidt applied twice
// and the normalisation, five launches that take the column count k from device
// memory (*kp), so that a captured graph serves every iteration up to the
// column bound it was captured for.
//
//   k_cgs_dot            part = V^T w, by blocks of rows and groups of columns
//   k_dot_reduce_dk      h1 = their sums
//   k_cgs_update_dot     w -= V h1, and part = V^T w from the same reading of V
//   k_dot_reduce_dk      h2
//   k_cgs_update_norm    w -= V h2, and parts of |w|^2 (k_cgs_vh_norm for long w)
//   k_cgs_finish         V[k] = w/|w| (and the buffers the next step reads), the
//                        column h1 + h2, |w|^2 to the host
//
// Bound by reading V (8 k n bytes three times, where a launch per product and
// update read it four times) for long vectors and by latency for short ones:
// the splits over rows and columns keep a warp's chain of loads short.  n =
// 4638, k = 180: 17 us for the step, with one launch per operation 52 us; n =
// 55,596, k = 240: 65 us (102 us).
#pragma once
#include "kernels.cuh"

namespace {

constexpr int CGS_MAX = 1024;      // columns up to which these kernels run
constexpr int CGS_ROWS = 32;       // rows of a chunk of k_cgs_update_*

__global__ void __launch_bounds__(256)
k_cgs_dot(const double* __restrict__ V, long long ldv, const int* __restrict__ kp, const double* __restrict__ w,
          long long n, int R, double* __restrict__ part) {
  extern __shared__ double swv[];
  const int k = *kp, per = ((k + (int)gridDim.y - 1) / (int)gridDim.y + 3) & ~3;
  const int c0 = blockIdx.y * per, kc = min(k - c0, per);
  if (kc <= 0) return;
  dot_cols_cta(V + (long long)c0 * ldv, ldv, kc, w, n, R, part + (size_t)c0 * gridDim.x, swv);
}

// One row per lane; warp q takes columns q, q + 8, ...  tile (k x 33) keeps the
// chunk's block of V for the second product, in which thread t owns columns t,
// t + 256, ...
__global__ void __launch_bounds__(256)
k_cgs_update_dot(const double* __restrict__ V, long long ldv, const int* __restrict__ kp, const double* __restrict__ h,
                 double* __restrict__ w, long long n, double* __restrict__ part) {
  extern __shared__ double tile[];
  __shared__ double red[8][32], wsm[32];
  const int k = *kp, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* hs = tile + (size_t)k * 33;
  for (int j = threadIdx.x; j < k; j += 256) hs[j] = h[j];
  double acc[CGS_MAX / 256];
#pragma unroll
  for (int q = 0; q < CGS_MAX / 256; ++q) acc[q] = 0.0;
  __syncthreads();
  for (long long r0 = (long long)blockIdx.x * CGS_ROWS; r0 < n; r0 += (long long)gridDim.x * CGS_ROWS) {
    const bool in = r0 + lane < n;
    const double* __restrict__ v = V + r0 + lane;
    double s = 0.0;
#pragma unroll 8
    for (int j = wid; j < k; j += 8) {
      const double x = in ? __ldg(v + (long long)j * ldv) : 0.0;
      tile[j * 33 + lane] = x;
      s = fma(x, hs[j], s);
    }
    red[wid][lane] = s;
    __syncthreads();
    if (wid == 0) {
      double t = red[0][lane];
#pragma unroll
      for (int q = 1; q < 8; ++q) t += red[q][lane];
      const double x = in ? w[r0 + lane] - t : 0.0;
      if (in) w[r0 + lane] = x;
      wsm[lane] = x;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < CGS_MAX / 256; ++q) {
      const int c = threadIdx.x + 256 * q;
      if (c < k) {
        double a = acc[q];
#pragma unroll 8
        for (int l = 0; l < 32; ++l) a = fma(tile[c * 33 + l], wsm[l], a);
        acc[q] = a;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < CGS_MAX / 256; ++q) {
    const int c = threadIdx.x + 256 * q;
    if (c < k) part[(size_t)c * gridDim.x + blockIdx.x] = acc[q];
  }
}

__global__ void __launch_bounds__(256)
k_cgs_update_norm(const double* __restrict__ V, long long ldv, const int* __restrict__ kp,
                  const double* __restrict__ h, double* __restrict__ w, long long n, double* __restrict__ npart) {
  __shared__ double red[8][32], hs[CGS_MAX];
  const int k = *kp, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int j = threadIdx.x; j < k; j += 256) hs[j] = h[j];
  __syncthreads();
  double nn = 0.0;
  for (long long r0 = (long long)blockIdx.x * CGS_ROWS; r0 < n; r0 += (long long)gridDim.x * CGS_ROWS) {
    const bool in = r0 + lane < n;
    const double* __restrict__ v = V + r0 + lane;
    double s = 0.0;
#pragma unroll 8
    for (int j = wid; j < k; j += 8) s = fma(in ? __ldg(v + (long long)j * ldv) : 0.0, hs[j], s);
    red[wid][lane] = s;
    __syncthreads();
    if (wid == 0 && in) {
      double t = red[0][lane];
#pragma unroll
      for (int q = 1; q < 8; ++q) t += red[q][lane];
      const double x = w[r0 + lane] - t;
      w[r0 + lane] = x;
      nn = fma(x, x, nn);
    }
    __syncthreads();
  }
  if (wid == 0) {
    nn = warp_sum(nn);
    if (lane == 0) npart[blockIdx.x] = nn;
  }
}

// The same update with a row per thread (k_vh_dk), for long vectors.
__global__ void __launch_bounds__(256)
k_cgs_vh_norm(const double* __restrict__ V, long long ldv, const int* __restrict__ kp, const double* __restrict__ h,
              double* __restrict__ w, long long n, double* __restrict__ npart) {
  __shared__ double sh[CGS_MAX], red[32];
  const int k = *kp;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  for (int t = threadIdx.x; t < k; t += 256) sh[t] = h[t];
  __syncthreads();
  double x = 0.0;
  if (i < n) {
    const double* __restrict__ vp = V + i;
    double a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    int j = 0;
    for (; j + 7 < k; j += 8)   // eight independent loads in flight
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] = fma(__ldg(vp + (long long)(j + q) * ldv), sh[j + q], a[q]);
    for (; j < k; ++j) a[0] = fma(__ldg(vp + (long long)j * ldv), sh[j], a[0]);
    x = w[i] - (((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7])));
    w[i] = x;
  }
  const double s = block_sum<256>(x * x, red);
  if (threadIdx.x == 0) npart[blockIdx.x] = s;
}

// Every CTA sums the parts of |w|^2 in the same order.  z (may be nullptr): the
// preconditioned vector of this step, kept as column k - 1 of Z.  host: two
// pinned slots of `slot` doubles, written in turn: the column, then |w|^2.
__global__ void __launch_bounds__(256)
k_cgs_finish(double* __restrict__ V, double* __restrict__ Z, long long ldv, const int* __restrict__ kp,
             const double* __restrict__ h1, const double* __restrict__ h2, const double* __restrict__ npart, int np,
             const double* __restrict__ w, const double* __restrict__ z, double* __restrict__ cur, long long n,
             double* __restrict__ host, int slot) {
  __shared__ double sh[32];
  double s = 0.0;
  for (int b = threadIdx.x; b < np; b += 256) s += npart[b];
  s = block_sum<256>(s, sh);
  const int k = *kp;
  const double a = s > 0.0 ? 1.0 / sqrt(s) : 0.0;
  double* __restrict__ v = V + (long long)k * ldv;
  double* __restrict__ zc = Z + (long long)(k - 1) * ldv;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
    const double x = w[i] * a;
    v[i] = x;
    cur[i] = x;
    if (z) zc[i] = z[i];
  }
  if (blockIdx.x == 0) {
    double* o = host + (size_t)(k & 1) * slot;
    for (int j = threadIdx.x; j < k; j += 256) o[j] = h1[j] + h2[j];
    if (threadIdx.x == 0) o[k] = s;
  }
}

}  // namespace
