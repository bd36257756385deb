// X <- Q X with Q = H_0 H_1 ... from stored Householder reflectors, for one large matrix
// or many, real or complex, with every product on the tensor cores (skew_oz.cuh).
//
// The reflectors are taken in panels of BK<CX>::PB: Q_p = I - V T V^H (compact WY, forward,
// columnwise).  Once per call, for all panels and matrices at a time:
//   G = V^H V, T from G (back_tfac_kernel), VT = V T;
// then from the last panel to the first, all matrices at a time:
//   W = V^H X (split along the rows when few tiles would leave SMs idle), X <- X - VT W.
// A complex product runs as a real one on [[Re, -Im], [Im, Re]] of its left operand; the
// right operand and the result are interleaved complex columns, real columns of twice
// the rows.
//
// Scaling (biased exponents): |v| <= 1 and |v_l| <= sqrt(2) (tau between 1 and 2, Re tau
// >= 1 for complex), and the columns of X have unit norm, so entries of V, X and W = V^H X
// are below 2 (1023) throughout; a column that comes larger takes 2^12 more, one that is
// not finite stays NaN.  VT and T are measured.
#pragma once
#include <algorithm>
#include <atomic>

#include "skew_common.cuh"
#include "skew_internal.h"
#include "skew_oz.cuh"

namespace skew {

template <bool CX>
struct BK {
  static constexpr int PB = CX ? 64 : 128;  // reflectors per panel: 128 rows of W fill a tile
  static constexpr int R = CX ? 2 : 1;      // doubles per entry
};

constexpr int BACK_SLICE = 65535;  // matrices per launch: the largest grid in y and z

// One matrix.  nref reflectors: column c of A below the diagonal, v[c + 1] = 1, zero above.
template <bool CX>
struct BackTask {
  const double* A;
  int64_t lda;
  const double* tau;
  int n, nref;
  double* X[2];  // two groups of columns, nc[0] and nc[1] of them
  int64_t ldx;
  int nc[2];
  double *t, *vt, *w;     // T: panels of ldt x ldt; VT: R n x nref; W: R ldt x columns (x splits)
  int *et, *evt, *ex;     // exponents: T's columns, VT's rows per panel, X's columns
  int identity;           // X starts as the identity: a panel from column c0 leaves columns 0 .. c0 alone
  int* status;            // SKEW_TIMEOUT if a bounded wait gave up (or null)
  int skip_cta = -1;      // >= 0: this CTA of each X <- X - VT W counts as given up (a test of the status)
  __host__ __device__ int ldt() const { return nref < BK<CX>::PB ? nref : BK<CX>::PB; }
  __host__ __device__ int panels() const { return (nref + BK<CX>::PB - 1) / BK<CX>::PB; }
  __device__ int cols() const { return nc[0] + nc[1]; }
  __device__ double* column(int j) const {
    return j < nc[0] ? X[0] + BK<CX>::R * ldx * j : X[1] + BK<CX>::R * ldx * (j - nc[0]);
  }
};

// Doubles of workspace behind t, vt, w, et, evt, ex for a matrix of size n.
template <bool CX>
__host__ __device__ inline size_t back_ws_doubles(int n, int nref, int cols, int splits) {
  const size_t ldt = nref < BK<CX>::PB ? nref : BK<CX>::PB, np = (nref + BK<CX>::PB - 1) / BK<CX>::PB;
  const size_t R = BK<CX>::R;
  const size_t ints = (size_t)nref + R * n * np + cols;
  return np * R * ldt * ldt + R * (size_t)n * nref + R * ldt * cols * (splits > 1 ? splits + 1 : 1) + (ints + 1) / 2 + 2;
}
template <bool CX>
__host__ __device__ inline void back_ws_set(BackTask<CX>& B, double* ws, int cols, int splits) {
  const size_t R = BK<CX>::R, ldt = B.ldt(), np = B.panels();
  B.t = ws;
  B.vt = B.t + np * R * ldt * ldt;
  B.w = B.vt + R * (size_t)B.n * B.nref;
  B.et = (int*)(B.w + R * ldt * cols * (splits > 1 ? splits + 1 : 1));
  B.evt = B.et + B.nref;
  B.ex = B.evt + R * B.n * np;
}

// A row of V^H (CONJT: reflector l, along the rows of A) or of V (a row of A, along the
// reflectors) of panel p as the left operand.
template <bool CX, bool CONJT>
struct BackV {
  const double* A;
  const double* tau;
  int64_t lda;
  int c0, nb, n;
  __device__ __forceinline__ void entry(int row, int l, double& re, double& im) const {
    const int c = c0 + l;
    re = im = 0.0;
    if (row >= n || l >= nb || row <= c) return;
    if (CX) {
      if (tau[2 * c] == 0.0 && tau[2 * c + 1] == 0.0) return;
      if (row == c + 1) {
        re = 1.0;
      } else {
        const double2 z = *reinterpret_cast<const double2*>(A + 2 * (row + (int64_t)c * lda));  // 16-byte aligned
        re = z.x;
        im = z.y;
      }
    } else {
      if (tau[c] == 0.0) return;
      re = (row == c + 1) ? 1.0 : A[row + (int64_t)c * lda];
    }
  }
  __device__ __forceinline__ void load(int i, int k, double (&v)[8]) const {
    if (!CX) {
      double im;
#pragma unroll
      for (int u = 0; u < 8; u++)
        if (CONJT)
          entry(c0 + 1 + k + u, i, v[u], im);
        else
          entry(c0 + 1 + i, k + u, v[u], im);
    } else {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        double re, im;
        if (CONJT)
          entry(c0 + 1 + k / 2 + u, i >> 1, re, im);
        else
          entry(c0 + 1 + (i >> 1), k / 2 + u, re, im);
        if (CONJT) im = -im;
        v[2 * u] = (i & 1) ? im : re;
        v[2 * u + 1] = (i & 1) ? re : -im;
      }
    }
  }
};

template <int NV>
__device__ __forceinline__ void back_load_column(const double* p, int k, int len, double (&v)[NV]) {
#pragma unroll
  for (int u = 0; u < NV; u++) v[u] = (k + u < len) ? p[k + u] : 0.0;
}

// G = V^H V of one panel
template <bool CX>
struct BackGram {
  BackTask<CX> B;
  BackV<CX, true> V;
  int p;
  __device__ int rows() const { return BK<CX>::R * V.nb; }
  __device__ int cols() const { return V.nb; }
  __device__ int ksteps() const { return (BK<CX>::R * (B.n - V.c0 - 1) + OZ_K - 1) / OZ_K; }
  __device__ bool contiguousA() const { return true; }
  __device__ bool contiguousB() const { return true; }
  __device__ int expA(int) const { return 1023; }
  __device__ int expB(int) const { return 1023; }
  __device__ void loadA(int i, int s, int k, double (&v)[8]) const { V.load(i, s * OZ_K + k, v); }
  __device__ void loadB(int j, int s, int k, double (&v)[4]) const {
    const int k0 = s * OZ_K + k;
    if (CX) {
#pragma unroll
      for (int u = 0; u < 2; u++) V.entry(V.c0 + 1 + k0 / 2 + u, j, v[2 * u], v[2 * u + 1]);
    } else {
      double im;
#pragma unroll
      for (int u = 0; u < 4; u++) V.entry(V.c0 + 1 + k0 + u, j, v[u], im);
    }
  }
  __device__ void store(int i, int j, double x) const {
    const size_t ldt = B.ldt();
    B.t[BK<CX>::R * ldt * (p * ldt + j) + i] = x;
  }
  __device__ void timeout() const { if (B.status) *B.status = SKEW_TIMEOUT; }
};

// VT = V T of one panel
template <bool CX>
struct BackVT {
  BackTask<CX> B;
  BackV<CX, false> V;
  int p;
  __device__ int rows() const { return BK<CX>::R * (B.n - V.c0 - 1); }
  __device__ int cols() const { return V.nb; }
  __device__ int ksteps() const { return (BK<CX>::R * V.nb + OZ_K - 1) / OZ_K; }
  __device__ bool contiguousA() const { return false; }
  __device__ bool contiguousB() const { return true; }
  __device__ int expA(int) const { return 1023; }
  __device__ int expB(int j) const { return B.et[V.c0 + j]; }
  __device__ void loadA(int i, int s, int k, double (&v)[8]) const { V.load(i, s * OZ_K + k, v); }
  __device__ void loadB(int j, int s, int k, double (&v)[4]) const {
    const size_t ldt = B.ldt();
    back_load_column<4>(B.t + BK<CX>::R * ldt * (p * ldt + j), s * OZ_K + k, BK<CX>::R * V.nb, v);
  }
  __device__ void store(int i, int j, double x) const {
    B.vt[(size_t)BK<CX>::R * B.n * (V.c0 + j) + i] = x;
  }
  __device__ void timeout() const { if (B.status) *B.status = SKEW_TIMEOUT; }
};

// W = V^H X (rows of the split: buffers [s0, s1) of K)
template <bool CX>
struct BackW {
  BackTask<CX> B;
  BackV<CX, true> V;
  int s0, s1;
  double* w;
  __device__ int rows() const { return BK<CX>::R * V.nb; }
  __device__ int cols() const { return B.cols(); }
  __device__ int ksteps() const { return s1 - s0; }
  __device__ bool contiguousA() const { return true; }
  __device__ bool contiguousB() const { return true; }
  __device__ int expA(int) const { return 1023; }
  __device__ int expB(int j) const { return B.ex[j]; }
  __device__ void loadA(int i, int s, int k, double (&v)[8]) const { V.load(i, (s0 + s) * OZ_K + k, v); }
  __device__ void loadB(int j, int s, int k, double (&v)[4]) const {
    back_load_column<4>(B.column(j) + BK<CX>::R * (V.c0 + 1), (s0 + s) * OZ_K + k, BK<CX>::R * (B.n - V.c0 - 1), v);
  }
  __device__ void store(int i, int j, double x) const { w[BK<CX>::R * (size_t)B.ldt() * j + i] = x; }
  __device__ void timeout() const { if (B.status) *B.status = SKEW_TIMEOUT; }
};

// X <- X - VT W
template <bool CX>
struct BackX {
  BackTask<CX> B;
  int p, c0, nb;
  __device__ int rows() const { return BK<CX>::R * (B.n - c0 - 1); }
  __device__ int cols() const { return B.cols(); }
  __device__ int ksteps() const { return (BK<CX>::R * nb + OZ_K - 1) / OZ_K; }
  __device__ bool contiguousA() const { return false; }
  __device__ bool contiguousB() const { return true; }
  __device__ int expA(int i) const { return B.evt[BK<CX>::R * (size_t)B.n * p + i]; }
  __device__ int expB(int j) const { return B.ex[j]; }
  __device__ void loadA(int i, int s, int k, double (&v)[8]) const {
    const size_t ld = BK<CX>::R * (size_t)B.n;
    const int k0 = s * OZ_K + k;
    const double* q = B.vt + ld * c0;
    if (CX) {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int l = k0 / 2 + u;
        double2 z = make_double2(0.0, 0.0);
        if (l < nb) z = make_double2(q[ld * l + (i & ~1)], q[ld * l + (i | 1)]);
        v[2 * u] = (i & 1) ? z.y : z.x;
        v[2 * u + 1] = (i & 1) ? z.x : -z.y;
      }
    } else {
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = (k0 + u < nb) ? q[ld * (k0 + u) + i] : 0.0;
    }
  }
  __device__ void loadB(int j, int s, int k, double (&v)[4]) const {
    back_load_column<4>(B.w + BK<CX>::R * (size_t)B.ldt() * j, s * OZ_K + k, BK<CX>::R * nb, v);
  }
  __device__ void store(int i, int j, double x) const {
    double* q = B.column(j) + BK<CX>::R * (c0 + 1) + i;
    *q -= x;
  }
  __device__ void timeout() const { if (B.status) *B.status = SKEW_TIMEOUT; }
};

// Src: bool get(int b, BackTask<CX>&) const: matrix b, false if there is nothing to do.
// A launch takes the matrices b0, b0 + 1, ...: as many as a grid's y or z may count.
template <bool CX, class Src>
__global__ void __launch_bounds__(256) back_ex_kernel(Src S, int b0) {  // grid (columns / 8, count)
  BackTask<CX> B;
  if (!S.get(b0 + blockIdx.y, B)) return;
  const int j = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (j >= B.cols()) return;
  const double* x = B.column(j);
  int e = 1;
  for (int i = threadIdx.x & 31; i < BK<CX>::R * B.n; i += 32) e = max(e, oz_exponent(x[i]));
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0) B.ex[j] = e <= 1023 ? 1023 : (e == 2047 ? 2047 : min(e + 12, 2046));
}

template <bool CX, class Src>
__global__ void __launch_bounds__(OZ_NT, 1) back_gram_kernel(Src S, int b0) {  // grid (column tiles, panels, count)
  extern __shared__ __align__(1024) unsigned char oz_buf[];
  BackGram<CX> P;
  if (!S.get(b0 + blockIdx.z, P.B)) return;
  P.p = blockIdx.y;
  const int c0 = P.p * BK<CX>::PB, nb = min(BK<CX>::PB, P.B.nref - c0);
  if ((int)blockIdx.x * OZ_N >= nb) return;
  P.V = BackV<CX, true>{P.B.A, P.B.tau, P.B.lda, c0, nb, P.B.n};
  oz_tile(P, 0, blockIdx.x * OZ_N, oz_buf);
}

// T(i, i) = tau_i, T(0:i, i) = -tau_i T(0:i, 0:i) G(0:i, i), in place of G: one CTA per
// panel, grid (panels, count).  Thread j + PB q takes every fourth (eighth) term of row j.
template <bool CX, class Src>
__global__ void __launch_bounds__(512) back_tfac_kernel(Src S, int b0) {
  constexpr int PB = BK<CX>::PB, R = BK<CX>::R, Q = 512 / PB;
  extern __shared__ __align__(16) double tf[];  // T (PB x (PB + 1) entries), partial sums (512 entries)
  BackTask<CX> B;
  if (!S.get(b0 + blockIdx.y, B)) return;
  const int c0 = blockIdx.x * PB, nb = min(PB, B.nref - c0);
  if (nb <= 0) return;
  const int ldt = B.ldt(), j = threadIdx.x % PB, q = threadIdx.x / PB;
  double* G = B.t + (size_t)R * ldt * ldt * blockIdx.x;
  double* red = tf + R * PB * (PB + 1);
  for (int i = 0; i < nb; i++) {
    double sr = 0.0, si = 0.0;
    if (j < i)
      for (int l = j + q; l < i; l += Q) {
        if (CX) {
          const double tr = tf[2 * (j * (PB + 1) + l)], ti = tf[2 * (j * (PB + 1) + l) + 1];
          const double gr = G[2 * (l + i * ldt)], gi = G[2 * (l + i * ldt) + 1];
          sr = fma(tr, gr, fma(-ti, gi, sr));
          si = fma(tr, gi, fma(ti, gr, si));
        } else {
          sr = fma(tf[j * (PB + 1) + l], G[l + i * ldt], sr);
        }
      }
    red[R * threadIdx.x] = sr;
    if (CX) red[R * threadIdx.x + 1] = si;
    __syncthreads();
    if (q == 0 && j < nb) {
      double ar = 0.0, ai = 0.0;
      const double tr = B.tau[R * (c0 + i)], ti = CX ? B.tau[R * (c0 + i) + 1] : 0.0;
      if (j < i) {
#pragma unroll
        for (int u = 0; u < Q; u++) {
          sr = (u == 0) ? red[R * j] : sr + red[R * (j + PB * u)];
          if (CX) si = (u == 0) ? red[R * j + 1] : si + red[R * (j + PB * u) + 1];
        }
        ar = -(tr * sr - ti * si);
        ai = -(tr * si + ti * sr);
      } else if (j == i) {
        ar = tr;
        ai = ti;
      }
      tf[R * (j * (PB + 1) + i)] = ar;
      if (CX) tf[R * (j * (PB + 1) + i) + 1] = ai;
    }
    __syncthreads();
  }
  for (int i = q; i < nb; i += Q)
    if (j < nb) {
      G[R * (j + i * ldt)] = tf[R * (j * (PB + 1) + i)];
      if (CX) G[R * (j + i * ldt) + 1] = tf[R * (j * (PB + 1) + i) + 1];
    }
  for (int i = threadIdx.x >> 5; i < nb; i += 16) {
    int e = 1;
    for (int k = threadIdx.x & 31; k < nb; k += 32)
#pragma unroll
      for (int c = 0; c < R; c++) e = max(e, oz_exponent(tf[R * (k * (PB + 1) + i) + c]));
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) B.et[c0 + i] = e;
  }
}

template <bool CX, class Src>
__global__ void __launch_bounds__(OZ_NT, 1) back_vt_kernel(Src S, int b0, int rt) {  // grid (row tiles x column tiles, panels, count)
  extern __shared__ __align__(1024) unsigned char oz_buf[];
  BackVT<CX> P;
  if (!S.get(b0 + blockIdx.z, P.B)) return;
  P.p = blockIdx.y;
  const int c0 = P.p * BK<CX>::PB, nb = min(BK<CX>::PB, P.B.nref - c0);
  const int i0 = (int)(blockIdx.x % rt) * OZ_M, j0 = (int)(blockIdx.x / rt) * OZ_N;
  if (nb <= 0 || j0 >= nb || i0 >= BK<CX>::R * (P.B.n - c0 - 1)) return;
  P.V = BackV<CX, false>{P.B.A, P.B.tau, P.B.lda, c0, nb, P.B.n};
  oz_tile(P, i0, j0, oz_buf);
}

template <bool CX, class Src>
__global__ void __launch_bounds__(256) back_evt_kernel(Src S, int b0) {  // grid (rows / 256, panels, count)
  constexpr int R = BK<CX>::R;
  BackTask<CX> B;
  if (!S.get(b0 + blockIdx.z, B)) return;
  const int p = blockIdx.y, c0 = p * BK<CX>::PB, nb = min(BK<CX>::PB, B.nref - c0);
  const int i = blockIdx.x * 256 + threadIdx.x;  // row of the real matrix
  if (nb <= 0 || i >= R * (B.n - c0 - 1)) return;
  const double* q = B.vt + (size_t)R * B.n * c0;
  int e = 1;
  for (int l = 0; l < nb; l++)
#pragma unroll
    for (int c = 0; c < R; c++) e = max(e, oz_exponent(q[(size_t)R * B.n * l + (CX ? (i & ~1) + c : i)]));
  B.evt[(size_t)R * B.n * p + i] = e;
}

// step: panels from the last one, each matrix its own; grid (column tiles, splits, count)
template <bool CX, class Src>
__global__ void __launch_bounds__(OZ_NT, 1) back_w_kernel(Src S, int b0, int step) {
  extern __shared__ __align__(1024) unsigned char oz_buf[];
  BackW<CX> P;
  if (!S.get(b0 + blockIdx.z, P.B)) return;
  const int p = P.B.panels() - 1 - step;
  if (p < 0 || (int)blockIdx.x * OZ_N >= P.B.cols()) return;
  const int c0 = p * BK<CX>::PB, nb = min(BK<CX>::PB, P.B.nref - c0);
  if (P.B.identity && (int)blockIdx.x * OZ_N + OZ_N - 1 <= c0) return;
  P.V = BackV<CX, true>{P.B.A, P.B.tau, P.B.lda, c0, nb, P.B.n};
  const int all = (BK<CX>::R * (P.B.n - c0 - 1) + OZ_K - 1) / OZ_K;
  const int chunks = (all + 3) / 4, per = (chunks + gridDim.y - 1) / gridDim.y * 4;  // whole exact sums
  P.s0 = min(all, (int)blockIdx.y * per);
  P.s1 = min(all, P.s0 + per);
  P.w = P.B.w + (gridDim.y > 1 ? blockIdx.y + 1 : 0) * (BK<CX>::R * (size_t)P.B.ldt() * P.B.cols());
  oz_tile(P, 0, blockIdx.x * OZ_N, oz_buf);
}

template <bool CX, class Src>
__global__ void back_join_kernel(Src S, int b0, int splits) {  // the splits' sums of W; grid (chunks, count)
  BackTask<CX> B;
  if (!S.get(b0 + blockIdx.y, B)) return;
  const size_t len = BK<CX>::R * (size_t)B.ldt() * B.cols();
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < len; q += (size_t)gridDim.x * blockDim.x) {
    double s = B.w[len + q];
    for (int u = 2; u <= splits; u++) s += B.w[u * len + q];
    B.w[q] = s;
  }
}

template <bool CX, class Src>
__global__ void __launch_bounds__(OZ_NT, 1) back_x_kernel(Src S, int b0, int step, int rt) {  // grid (row x column tiles, count)
  extern __shared__ __align__(1024) unsigned char oz_buf[];
  BackX<CX> P;
  if (!S.get(b0 + blockIdx.y, P.B)) return;
  P.p = P.B.panels() - 1 - step;
  if (P.p < 0) return;
  P.c0 = P.p * BK<CX>::PB;
  P.nb = min(BK<CX>::PB, P.B.nref - P.c0);
  const int i0 = (int)(blockIdx.x % rt) * OZ_M, j0 = (int)(blockIdx.x / rt) * OZ_N;
  if (i0 >= P.rows() || j0 >= P.cols() || (P.B.identity && j0 + OZ_N - 1 <= P.c0)) return;
  if ((int)blockIdx.x == P.B.skip_cta) {
    if (threadIdx.x == 0) P.timeout();
    return;
  }
  oz_tile(P, i0, j0, oz_buf);
}

// Splits of W's sums so that a single matrix's column tiles fill the SMs.
inline int back_splits(int cols, int count, int sms) {
  const int tiles = (cols + OZ_N - 1) / OZ_N * count;
  int s = 1;
  while (s < 8 && tiles * s * 2 <= sms + sms / 4) s *= 2;
  return s;
}

// nmax, nref_max, cols_max: the largest of the matrices
template <bool CX, class Src>
inline cudaError_t back_transform_oz(const Src& S, int count, int nmax, int nref_max, int cols_max, int splits,
                                     cudaStream_t st) {
  constexpr int PB = BK<CX>::PB, R = BK<CX>::R;
  const int np = (nref_max + PB - 1) / PB;
  if (count <= 0 || np <= 0 || cols_max <= 0) return cudaSuccess;
  static std::atomic<uint64_t> raised[5];
  cudaError_t e;
  if ((e = raise_smem_limit_once((const void*)back_gram_kernel<CX, Src>, raised[0])) ||
      (e = raise_smem_limit_once((const void*)back_tfac_kernel<CX, Src>, raised[1])) ||
      (e = raise_smem_limit_once((const void*)back_vt_kernel<CX, Src>, raised[2])) ||
      (e = raise_smem_limit_once((const void*)back_w_kernel<CX, Src>, raised[3])) ||
      (e = raise_smem_limit_once((const void*)back_x_kernel<CX, Src>, raised[4])))
    return e;
  const int ct = (cols_max + OZ_N - 1) / OZ_N, rt = (R * nmax + OZ_M - 1) / OZ_M, pt = PB / OZ_N;
  const size_t tf = sizeof(double) * R * (PB * (PB + 1) + 512);
  for (int b0 = 0; b0 < count; b0 += BACK_SLICE) {
    const int m = std::min(count - b0, BACK_SLICE);
    back_ex_kernel<CX, Src><<<dim3((cols_max + 7) / 8, m), 256, 0, st>>>(S, b0);
    back_gram_kernel<CX, Src><<<dim3(pt, np, m), OZ_NT, OZ_SMEM, st>>>(S, b0);
    back_tfac_kernel<CX, Src><<<dim3(np, m), 512, tf, st>>>(S, b0);
    back_vt_kernel<CX, Src><<<dim3(rt * pt, np, m), OZ_NT, OZ_SMEM, st>>>(S, b0, rt);
    back_evt_kernel<CX, Src><<<dim3((R * nmax + 255) / 256, np, m), 256, 0, st>>>(S, b0);
    if ((e = cudaGetLastError())) return e;
    for (int q = 0; q < np; q++) {
      back_w_kernel<CX, Src><<<dim3(ct, splits, m), OZ_NT, OZ_SMEM, st>>>(S, b0, q);
      if (splits > 1) back_join_kernel<CX, Src><<<dim3(64, m), 256, 0, st>>>(S, b0, splits);
      back_x_kernel<CX, Src><<<dim3(rt * ct, m), OZ_NT, OZ_SMEM, st>>>(S, b0, q, rt);
      if ((e = cudaGetLastError())) return e;
    }
  }
  return cudaSuccess;
}

}  // namespace skew
