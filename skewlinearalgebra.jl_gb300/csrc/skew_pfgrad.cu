// Gradients 1/2 A^{-T} = Q (-1/2 T^{-1}) Q^T of log|Pf(A)| for the larger matrices of a
// batch, from the reduction's reflectors and subdiagonal, on the tensor cores.
//
// The fused kernel (skew_batch.cu) applies the reflectors to -1/2 T^{-1} from both sides, 5/6 n^3
// FMAs on the FP64 pipe in blocks of 8 reflectors.  Here, all matrices at a time:
//   Q = H_0 .. H_{n-3} applied to the identity in panels of 128 (skew_back.cuh);
//   Y = Q (-1/2 T^{-1}), two bidiagonal recurrences per row of Q (O(n^2));
//   G = Y Q^T, the lower triangle of tiles (skew_oz.cuh), mirrored with the sign, so G is
//   exactly skew as before.
// 4096 matrices of n = 16 .. 256 (those above n = 96 here): the gradient's share of the
// call 34.8 -> 21.1 ms.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "skew_internal.h"
#include "skew_back.cuh"
#include "skew_common.cuh"

namespace skew {

// Workspace of one matrix (doubles): reflectors, later Y (n^2) | Q (n^2) | the
// back-transformation's | Y's row exponents (n ints).
static __host__ __device__ size_t pg_back_doubles(int n) { return n > 2 ? back_ws_doubles<false>(n, n - 2, n, 1) : 0; }
size_t pfgrad_ws_doubles(int n) { return 2 * (size_t)n * n + pg_back_doubles(n) + (size_t)(n + 1) / 2; }

struct PgItem {
  int b, n;
  double *R, *Q, *back;
  int* ey;
};
// matrix t of the launch; false if it has no gradient (its G becomes NaN)
__device__ __forceinline__ bool pg_item(const PfGrad& P, int t, PgItem& I) {
  I.b = P.order[t];
  I.n = P.n[I.b];
  const size_t nn = (size_t)I.n * I.n;
  I.R = P.refl[I.b];
  I.Q = I.R + nn;
  I.back = I.Q + nn;
  I.ey = (int*)(I.back + pg_back_doubles(I.n));
  return P.status[I.b] == SKEW_OK;
}

struct PgBack {
  PfGrad P;
  __device__ bool get(int t, BackTask<false>& T) const {
    PgItem I;
    if (!pg_item(P, t, I) || I.n < 3) return false;
    T.A = I.R;
    T.lda = I.n;
    T.tau = P.tau + P.off[I.b];
    T.n = I.n;
    T.nref = I.n - 2;
    T.X[0] = T.X[1] = I.Q;
    T.ldx = I.n;
    T.nc[0] = I.n;
    T.nc[1] = 0;
    T.identity = 1;
    T.status = P.status + I.b;
    back_ws_set(T, I.back, I.n, 1);
    return true;
  }
};

__global__ void pg_identity_kernel(PfGrad P) {  // grid (chunks, count)
  PgItem I;
  if (!pg_item(P, blockIdx.y, I)) return;
  const int tot = I.n * I.n;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += gridDim.x * blockDim.x)
    I.Q[q] = (q % (I.n + 1) == 0) ? 1.0 : 0.0;
}

// Y = Q M, M = -1/2 T^{-1}: with d_c = ev[2c], r_c = ev[2c-1] / ev[2c],
//   M[2a+1, 2b] = -M[2b, 2a+1] = (1/2 / d_b) r_{b+1} .. r_a  (a >= b), zero elsewhere below,
//   y[2b] = (1/2 / d_b) s_b,  s_b = q[2b+1] + r_{b+1} s_{b+1};
//   y[2a+1] = -u_a,           u_a = r_a u_{a-1} + q[2a] (1/2 / d_a).
// One thread per row of Q, grid (rows / 128, count); Y over the reflectors.
__global__ void __launch_bounds__(128) pg_solve_kernel(PfGrad P) {
  extern __shared__ double pgs[];  // r (n / 2), 1/2 / d (n / 2)
  PgItem I;
  if (!pg_item(P, blockIdx.y, I) || (int)blockIdx.x * 128 >= I.n) return;
  const int n = I.n, h = n / 2;
  const double* ev = P.ev + P.off[I.b];
  double* r = pgs;
  double* w = pgs + h;
  for (int c = threadIdx.x; c < h; c += 128) {
    r[c] = (c > 0) ? ev[2 * c - 1] / ev[2 * c] : 0.0;
    w[c] = 0.5 / ev[2 * c];
  }
  __syncthreads();
  const int i = blockIdx.x * 128 + threadIdx.x;
  if (i >= n) return;
  const double* q = I.Q + i;
  double* y = I.R + i;
  int e = 1;
  double u = 0.0;
#pragma unroll 4
  for (int a = 0; a < h; a++) {
    u = fma(r[a], u, q[(size_t)n * (2 * a)] * w[a]);
    const double v = neg(u);
    y[(size_t)n * (2 * a + 1)] = v;
    e = max(e, oz_exponent(v));
  }
  double s = 0.0;
#pragma unroll 4
  for (int b = h - 1; b >= 0; b--) {
    s = fma((b + 1 < h) ? r[b + 1] : 0.0, s, q[(size_t)n * (2 * b + 1)]);
    const double v = w[b] * s;
    y[(size_t)n * (2 * b)] = v;
    e = max(e, oz_exponent(v));
  }
  I.ey[i] = e;
}

struct PgTile {
  const double *Y, *Q;
  const int* ey;
  double* G;
  int n;
  int* status;
  __device__ int rows() const { return n; }
  __device__ int cols() const { return n; }
  __device__ int ksteps() const { return (n + OZ_K - 1) / OZ_K; }
  __device__ bool contiguousA() const { return false; }
  __device__ bool contiguousB() const { return false; }
  __device__ int expA(int i) const { return ey[i]; }
  __device__ int expB(int) const { return 1023; }  // rows of Q: |q| <= 1 up to rounding
  template <int NV>
  __device__ __forceinline__ void load(const double* M, int i, int k, double (&v)[NV]) const {
#pragma unroll
    for (int u = 0; u < NV; u++) v[u] = (k + u < n) ? M[i + (size_t)n * (k + u)] : 0.0;
  }
  __device__ void loadA(int i, int s, int k, double (&v)[8]) const { load<8>(Y, i, s * OZ_K + k, v); }
  __device__ void loadB(int j, int s, int k, double (&v)[4]) const { load<4>(Q, j, s * OZ_K + k, v); }
  __device__ void store(int i, int j, double x) const {
    if (i < j) return;
    G[i + (size_t)n * j] = (i == j) ? 0.0 : x;
    if (i != j) G[j + (size_t)n * i] = neg(x);
  }
  __device__ void timeout() const { *status = SKEW_TIMEOUT; }
};

// G = Y Q^T; a matrix without a gradient (a zero Pfaffian) gets NaN.  grid (tiles, count)
__global__ void __launch_bounds__(OZ_NT, 1) pg_product_kernel(PfGrad P) {
  extern __shared__ __align__(1024) unsigned char oz_buf[];
  PgItem I;
  const bool ok = pg_item(P, blockIdx.y, I);
  const int n = I.n, mt = (n + OZ_M - 1) / OZ_M, nt = (n + OZ_N - 1) / OZ_N;
  if ((int)blockIdx.x >= mt * nt) return;
  double* G = P.grad[I.b];
  if (!ok) {
    for (int q = blockIdx.x * OZ_NT + threadIdx.x; q < n * n; q += mt * nt * OZ_NT) G[q] = nan("");
    return;
  }
  const int i0 = (int)(blockIdx.x % mt) * OZ_M, j0 = (int)(blockIdx.x / mt) * OZ_N;
  if (i0 + OZ_M <= j0) return;  // above the diagonal
  PgTile T{I.R, I.Q, I.ey, G, n, P.status + I.b};
  oz_tile(T, i0, j0, oz_buf);
}

cudaError_t launch_pfgrad(const PfGrad& P, int count, int nmax, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  static std::atomic<uint64_t> raised{0};
  cudaError_t e = raise_smem_limit_once((const void*)pg_product_kernel, raised);
  if (e != cudaSuccess) return e;
  const int tiles = ((nmax + OZ_M - 1) / OZ_M) * ((nmax + OZ_N - 1) / OZ_N);
  for (int b0 = 0; b0 < count; b0 += BACK_SLICE) {
    const int m = std::min(count - b0, BACK_SLICE);
    PfGrad Q = P;
    Q.order += b0;
    pg_identity_kernel<<<dim3(std::max(1, nmax * nmax / 2048), m), 256, 0, st>>>(Q);
    if ((e = back_transform_oz<false>(PgBack{Q}, m, nmax, nmax - 2, nmax, 1, st))) return e;
    pg_solve_kernel<<<dim3((nmax + 127) / 128, m), 128, sizeof(double) * nmax, st>>>(Q);
    pg_product_kernel<<<dim3(tiles, m), OZ_NT, OZ_SMEM, st>>>(Q);
    if ((e = cudaGetLastError())) return e;
  }
  return cudaSuccess;
}

}  // namespace skew
