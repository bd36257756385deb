// ComplexF64 skew-Hermitian Householder tridiagonalisation (the complex branches
// of hessenberg.jl: householder! :26-44 with complex alpha, skewhess! :70-90,
// skewlatrd! :92-131 with the alpha correction of :123-126, the trailing update
// of skewblockedhess! :158-166).
//
// For column c with x = A[c+1:n, c] (alpha = x[1]):
//   beta = -sign(Re alpha) hypot(|alpha|, |x[2:]|) (real), tau = 1 - alpha/beta,
//   v = [1; x[2:] / (alpha - beta)]; zero column -> tau = 0, v = 0, beta = 0.
//   The last step (a 1 x 1 column) is a phase that makes the last subdiagonal real.
// With p = A22 v, W = tau p and a = tau (W^H v) / 2, w = W + a v, the update
//   A22 += v w^H - w v^H
// equals H^H A22 H for H = I - tau v v^H (the term a v restores the v v^H part
// that v^H A22 v, purely imaginary, contributes).  The lower triangle is updated,
// the upper one mirrored as -conj, and the diagonal only receives the purely
// imaginary part 2i Im(v_j conj(w_j)), as the blocked reference's
// Omega - Omega^H does.  On exit A holds the reflectors below the subdiagonal
// (v[1] = 1 on the subdiagonal), ev the real subdiagonal, dvim = imag(diag(A)).
//
// Two forms: zhess_cta_kernel, one CTA per matrix (batched, or the tail of a
// large reduction); and per-column multi-CTA kernels for large n (reflector,
// matvec partials over (row block, column chunk) tiles, combination, and the
// rank-2 update on 32 x 32 tiles of the lower triangle with a transposed mirror).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "skew_internal.h"
#include "skew_back.cuh"
#include "skew_common.cuh"
#include "skew_complex.cuh"
#include "skew_funcs.cuh"

namespace skew {

namespace cg = cooperative_groups;

constexpr int ZNT = 256;
constexpr int ZNW = ZNT / 32;

// ---------------------------------------------------------------------------
// reflector from (alpha, amax, ss) with |x[2:]| = amax * sqrt(ss)
// ---------------------------------------------------------------------------
struct ZRefl {
  zc tau, scale;
  double beta;
};

__device__ ZRefl zrefl(zc alpha, double xnorm) {
  ZRefl R;
  if (xnorm == 0.0 && alpha.re == 0.0 && alpha.im == 0.0) {
    R.tau = zc{0.0, 0.0};
    R.scale = zc{0.0, 0.0};
    R.beta = 0.0;
    return R;
  }
  const double h = hypot(hypot(alpha.re, alpha.im), xnorm);
  const double beta = (alpha.re > 0.0) ? neg(h) : h;
  R.beta = beta;
  R.tau = zc{1.0 - alpha.re / beta, neg(alpha.im / beta)};
  R.scale = zinv(zc{alpha.re - beta, alpha.im});
  return R;
}

// ---------------------------------------------------------------------------
// one cluster of CTAs per matrix
// ---------------------------------------------------------------------------
__device__ __forceinline__ double block_max(double x, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = x;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < ZNW; i++) s = fmax(s, red[i]);
  __syncthreads();
  return s;
}

// One cluster of CS CTAs per matrix, P.count matrices.  Bound by the FP64 pipe (8/3 n^3 complex
// multiply-adds' worth of FMAs per matrix), so the cluster is as wide as fills the SMs: the
// CTAs share the rows of A22 v (interleaved blocks of 32 rows, a block's columns split over
// the warps that have no block) and the entries of the update, exchange W through
// distributed shared memory and each form the reflector themselves.  The matrix lies in
// global memory (L2); what another CTA wrote is read with L2-only loads.
// 64 x n = 256: 20.4 -> 13.3 ms (clusters of 4; one CTA per matrix before).
template <int CS>
__global__ void __launch_bounds__(ZNT) zhess_cta_kernel(ZHessParams P) {
  extern __shared__ __align__(16) double zsm[];  // x, then v (n complex) | w (n complex)
  const int n = P.n;
  zc* vs = reinterpret_cast<zc*>(zsm);
  zc* ws = vs + n;
  __shared__ double red[ZNW];
  __shared__ zc part[ZNT];
  __shared__ ZRefl s_R;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = CS > 1 ? (int)cl.block_rank() : 0;
  const int b = blockIdx.x / CS;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  auto sync = [&]() {
    if (CS > 1)
      cl.sync();
    else
      __syncthreads();
  };
  auto ld2 = [](const zc* p) {
    const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
    return zc{v.x, v.y};
  };
  const int64_t ld = P.ld;
  zc* W = reinterpret_cast<zc*>(P.W) + (int64_t)b * P.stride;
  zc* tau = reinterpret_cast<zc*>(P.tau) + (int64_t)b * n;
  double* ev = P.ev + (int64_t)b * n;
  if (CS > 1) cl.sync();  // all CTAs run before the first write into another's shared memory
  for (int c = 0; c + 1 < n; c++) {
    const int m = n - c - 1;
    zc* x = W + (c + 1) + (int64_t)c * ld;
    double amax = 0.0;
    for (int i = tid; i < m; i += ZNT) {
      const zc v = ld2(x + i);
      vs[i] = v;
      if (i > 0) amax = fmax(amax, fmax(fabs(v.re), fabs(v.im)));
    }
    amax = block_max(amax, red);
    double ss = 0.0;
    if (amax > 0.0) {
      const double inv = 1.0 / amax;
      for (int i = tid; i < m; i += ZNT)
        if (i > 0) {
          const double a = vs[i].re * inv, bb = vs[i].im * inv;
          ss = fma(a, a, fma(bb, bb, ss));
        }
    }
    ss = block_sum<ZNW>(ss, red);
    if (tid == 0) {
      s_R = zrefl(vs[0], amax * sqrt(ss));
      if (rank == 0) {
        ev[c] = s_R.beta;
        tau[c] = s_R.tau;
      }
    }
    __syncthreads();
    const ZRefl R = s_R;
    const bool zero = (R.tau.re == 0.0 && R.tau.im == 0.0);
    for (int i = tid; i < m; i += ZNT)
      vs[i] = zero ? zc{0.0, 0.0} : (i == 0 ? zc{1.0, 0.0} : zmul(vs[i], R.scale));
    if (zero) {  // H = I: nothing to update
      sync();    // every CTA has read x
      for (int i = rank * ZNT + tid; i < m; i += ZNT * CS) x[i] = zc{0.0, 0.0};
      continue;
    }
    __syncthreads();
    zc* A22 = W + (c + 1) + (int64_t)(c + 1) * ld;
    // W = tau A22 v: this CTA's row blocks rank, rank + CS, ...; eight loads in flight per thread
    {
      const int nb = (m + 31) / 32, mine = (nb - rank + CS - 1) / CS;
      const int segs = mine > 0 ? max(1, ZNW / mine) : 1;
      for (int q0 = 0; q0 < mine; q0 += ZNW) {
        const int blocks = min(mine - q0, ZNW);
        const int q = w % blocks, seg = w / blocks;
        const int i = ((q0 + q) * CS + rank) * 32 + lane;
        zc p{0.0, 0.0};
        if (seg < segs && i < m) {
          const int j1 = m * (seg + 1) / segs;
          int j = m * seg / segs;
          zc a0{0.0, 0.0}, a1{0.0, 0.0}, a2{0.0, 0.0}, a3{0.0, 0.0};
          const zc* row = A22 + i;
          for (; j + 7 < j1; j += 8) {
            zc y[8];
#pragma unroll
            for (int u = 0; u < 8; u++) y[u] = ld2(row + (int64_t)(j + u) * ld);
            a0 = zfma(y[0], vs[j], a0);
            a1 = zfma(y[1], vs[j + 1], a1);
            a2 = zfma(y[2], vs[j + 2], a2);
            a3 = zfma(y[3], vs[j + 3], a3);
            a0 = zfma(y[4], vs[j + 4], a0);
            a1 = zfma(y[5], vs[j + 5], a1);
            a2 = zfma(y[6], vs[j + 6], a2);
            a3 = zfma(y[7], vs[j + 7], a3);
          }
          for (; j < j1; j++) a0 = zfma(ld2(row + (int64_t)j * ld), vs[j], a0);
          p = zadd(zadd(a0, a1), zadd(a2, a3));
        }
        part[tid] = p;
        __syncthreads();
        if (w < blocks && i < m) {  // seg 0 joins the block's segments
          for (int g = 1; g < segs; g++) p = zadd(p, part[(g * blocks + w) * 32 + lane]);
          p = zmul(R.tau, p);
          if (CS > 1) {
#pragma unroll
            for (int r = 0; r < CS; r++) cl.map_shared_rank(ws, r)[i] = p;
          } else {
            ws[i] = p;
          }
        }
        __syncthreads();
      }
    }
    sync();
    for (int i = rank * ZNT + tid; i < m; i += ZNT * CS) x[i] = vs[i];
    // a = tau (W^H v) / 2
    double dr = 0.0, di = 0.0;
    for (int i = tid; i < m; i += ZNT) {
      const zc d = zcmul(ws[i], vs[i]);  // conj(W_i) v_i
      dr += d.re;
      di += d.im;
    }
    dr = block_sum<ZNW>(dr, red);
    di = block_sum<ZNW>(di, red);
    const zc a = zmul(R.tau, zc{0.5 * dr, 0.5 * di});
    for (int i = tid; i < m; i += ZNT) ws[i] = zfma(a, vs[i], ws[i]);
    __syncthreads();
    // A22 += v w^H - w v^H on the lower triangle (diagonal included), mirrored.
    // The triangle is walked column by column as one list of m (m + 1) / 2 entries
    // (no division per entry); four entries per thread and iteration, loads first.
    {
      int j = 0, r = rank * ZNT + tid;  // entry (j + r, j): column j has m - j entries
      while (j < m && r >= m - j) {
        r -= m - j;
        j++;
      }
      while (j < m) {
        int jj[4], ii[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          jj[u] = j;
          ii[u] = j + r;
          if (j < m) {
            r += ZNT * CS;
            while (j < m && r >= m - j) {
              r -= m - j;
              j++;
            }
          }
        }
        zc y[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (jj[u] < m) y[u] = ld2(A22 + ii[u] + (int64_t)jj[u] * ld);
#pragma unroll
        for (int u = 0; u < 4; u++) {
          if (jj[u] >= m) continue;
          const int i = ii[u], jc = jj[u];
          const zc vi = vs[i], wi = ws[i];
          if (i == jc) {
            y[u].im += 2.0 * (vi.im * wi.re - vi.re * wi.im);  // 2 Im(v conj(w))
            A22[i + (int64_t)i * ld] = y[u];
          } else {
            const zc vj = vs[jc], wj = ws[jc];
            const zc uu = zsub(zadd(y[u], zmulc(vi, wj)), zmulc(wi, vj));  // + v_i conj(w_j) - w_i conj(v_j)
            A22[i + (int64_t)jc * ld] = uu;
            A22[jc + (int64_t)i * ld] = zc{neg(uu.re), uu.im};  // -conj(u)
          }
        }
      }
    }
    sync();
  }
  if (P.dvim) {
    double* dv = P.dvim + (int64_t)b * n;
    for (int k = rank * ZNT + tid; k < n; k += ZNT * CS) dv[k] = ld2(W + k + (int64_t)k * ld).im;
  }
  if (CS > 1) cl.sync();  // no CTA leaves while another may still write its shared memory
}

template <int CS>
static cudaError_t launch_zhess_t(const ZHessParams& P, cudaStream_t st) {
  static std::atomic<uint64_t> raised{0};
  cudaError_t e = raise_smem_limit_once((const void*)zhess_cta_kernel<CS>, raised);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(P.count * CS));
  cfg.blockDim = dim3(ZNT);
  cfg.dynamicSmemBytes = sizeof(double) * 4 * (size_t)std::max(P.n, 1);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, zhess_cta_kernel<CS>, P);
}

// CTAs per matrix: up to two CTAs per SM in all, and a block of 32 rows for each.
cudaError_t launch_zhess_cta(const ZHessParams& P, cudaStream_t st) {
  if (P.count <= 0) return cudaSuccess;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int cs = 1;
  while (cs < 8 && (long long)P.count * cs * 2 <= 2 * sms && P.n >= 64 * cs) cs *= 2;
  if (cs == 1) return launch_zhess_t<1>(P, st);
  if (cs == 2) return launch_zhess_t<2>(P, st);
  if (cs == 4) return launch_zhess_t<4>(P, st);
  return launch_zhess_t<8>(P, st);
}

// ---------------------------------------------------------------------------
// multi-CTA per-column reduction of one large matrix
// ---------------------------------------------------------------------------
constexpr int ZR_NT = 1024;  // reflector / combine CTA
constexpr int ZMV_ROWS = 256, ZMV_CH = 256;
constexpr int ZU_T = 32;

struct ZColWs {
  zc* v;       // m
  zc* w;       // m
  zc* part;    // nchunk x n
  ZRefl* R;    // 1
};

__global__ void __launch_bounds__(ZR_NT) zcol_refl_kernel(zc* A, int64_t lda, int n, int c, zc* tau, double* ev,
                                                          ZColWs ws) {
  __shared__ double red[ZR_NT / 32];
  __shared__ ZRefl s_R;
  const int m = n - c - 1;
  zc* x = A + (c + 1) + (int64_t)c * lda;
  double amax = 0.0;
  for (int i = 1 + threadIdx.x; i < m; i += ZR_NT) amax = fmax(amax, fmax(fabs(x[i].re), fabs(x[i].im)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = 0.0;
  for (int i = 0; i < ZR_NT / 32; i++) amax = fmax(amax, red[i]);
  __syncthreads();
  double ss = 0.0;
  if (amax > 0.0) {
    const double inv = 1.0 / amax;
    for (int i = 1 + threadIdx.x; i < m; i += ZR_NT) {
      const double a = x[i].re * inv, bb = x[i].im * inv;
      ss = fma(a, a, fma(bb, bb, ss));
    }
  }
  ss = block_sum<ZR_NT / 32>(ss, red);
  if (threadIdx.x == 0) {
    s_R = zrefl(x[0], amax * sqrt(ss));
    ev[c] = s_R.beta;
    tau[c] = s_R.tau;
    *ws.R = s_R;
  }
  __syncthreads();
  const ZRefl R = s_R;
  const bool zero = (R.tau.re == 0.0 && R.tau.im == 0.0);
  for (int i = threadIdx.x; i < m; i += ZR_NT) {
    const zc v = zero ? zc{0.0, 0.0} : (i == 0 ? zc{1.0, 0.0} : zmul(x[i], R.scale));
    x[i] = v;
    ws.v[i] = v;
  }
}

// partial p over a (row block, column chunk) tile: part[chunk][i] = sum_j A22[i,j] v_j
__global__ void __launch_bounds__(ZMV_ROWS) zcol_matvec_kernel(const zc* __restrict__ A, int64_t lda, int n, int c,
                                                               ZColWs ws) {
  __shared__ zc sv[ZMV_CH];
  const int m = n - c - 1;
  const int i = blockIdx.x * ZMV_ROWS + threadIdx.x;
  const int j0 = blockIdx.y * ZMV_CH, j1 = min(j0 + ZMV_CH, m);
  for (int j = j0 + threadIdx.x; j < j1; j += ZMV_ROWS) sv[j - j0] = ws.v[j];
  __syncthreads();
  if (i >= m) return;
  const zc* A22 = A + (c + 1) + (int64_t)(c + 1) * lda;
  zc a0{0.0, 0.0}, a1{0.0, 0.0}, a2{0.0, 0.0}, a3{0.0, 0.0};
  int j = j0;
  for (; j + 3 < j1; j += 4) {
    a0 = zfma(A22[i + (int64_t)j * lda], sv[j - j0], a0);
    a1 = zfma(A22[i + (int64_t)(j + 1) * lda], sv[j + 1 - j0], a1);
    a2 = zfma(A22[i + (int64_t)(j + 2) * lda], sv[j + 2 - j0], a2);
    a3 = zfma(A22[i + (int64_t)(j + 3) * lda], sv[j + 3 - j0], a3);
  }
  for (; j < j1; j++) a0 = zfma(A22[i + (int64_t)j * lda], sv[j - j0], a0);
  ws.part[(int64_t)blockIdx.y * n + i] = zadd(zadd(a0, a1), zadd(a2, a3));
}

// p = sum of partials (fixed order), W = tau p, a = tau (W^H v)/2, w = W + a v
__global__ void __launch_bounds__(ZR_NT) zcol_combine_kernel(int n, int c, int nchunk, ZColWs ws) {
  __shared__ double red[ZR_NT / 32];
  const int m = n - c - 1;
  const ZRefl R = *ws.R;
  double dr = 0.0, di = 0.0;
  for (int i = threadIdx.x; i < m; i += ZR_NT) {
    zc p{0.0, 0.0};
    for (int k = 0; k < nchunk; k++) p = zadd(p, ws.part[(int64_t)k * n + i]);
    const zc W = zmul(R.tau, p);
    ws.w[i] = W;
    const zc d = zcmul(W, ws.v[i]);
    dr += d.re;
    di += d.im;
  }
  dr = block_sum<ZR_NT / 32>(dr, red);
  di = block_sum<ZR_NT / 32>(di, red);
  const zc a = zmul(R.tau, zc{0.5 * dr, 0.5 * di});
  for (int i = threadIdx.x; i < m; i += ZR_NT) ws.w[i] = zfma(a, ws.v[i], ws.w[i]);
}

// A22 += v w^H - w v^H on lower 32 x 32 tiles (ti >= tj), upper tile mirrored
__global__ void __launch_bounds__(ZU_T * 8) zcol_update_kernel(zc* A, int64_t lda, int n, int c, ZColWs ws) {
  __shared__ zc tile[ZU_T][ZU_T + 1];
  __shared__ zc svi[ZU_T], swi[ZU_T], svj[ZU_T], swj[ZU_T];
  const int m = n - c - 1;
  // linear block index -> (ti, tj), tj <= ti
  const long long q = blockIdx.x;
  int ti = (int)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
  while ((long long)ti * (ti + 1) / 2 > q) ti--;
  while ((long long)(ti + 1) * (ti + 2) / 2 <= q) ti++;
  const int tj = (int)(q - (long long)ti * (ti + 1) / 2);
  const int i0 = ti * ZU_T, j0 = tj * ZU_T;
  zc* A22 = A + (c + 1) + (int64_t)(c + 1) * lda;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  if (threadIdx.x < ZU_T) {
    const int i = i0 + threadIdx.x, j = j0 + threadIdx.x;
    svi[threadIdx.x] = (i < m) ? ws.v[i] : zc{0.0, 0.0};
    swi[threadIdx.x] = (i < m) ? ws.w[i] : zc{0.0, 0.0};
    svj[threadIdx.x] = (j < m) ? ws.v[j] : zc{0.0, 0.0};
    swj[threadIdx.x] = (j < m) ? ws.w[j] : zc{0.0, 0.0};
  }
  __syncthreads();
  for (int jj = ty; jj < ZU_T; jj += 8) {
    const int i = i0 + tx, j = j0 + jj;
    zc u{0.0, 0.0};
    if (i < m && j < m && i >= j) {
      zc* p = A22 + i + (int64_t)j * lda;
      const zc vi = svi[tx], wi = swi[tx], vj = svj[jj], wj = swj[jj];
      if (i == j) {
        u = *p;
        u.im += 2.0 * (vi.im * wi.re - vi.re * wi.im);
      } else {
        u = zsub(zadd(*p, zmulc(vi, wj)), zmulc(wi, vj));
      }
      *p = u;
    }
    tile[jj][tx] = u;
  }
  if (ti == tj) {
    __syncthreads();
    // diagonal tile: mirror the strictly lower part into the upper part
    for (int jj = ty; jj < ZU_T; jj += 8) {
      const int i = i0 + jj, j = j0 + tx;  // element (i, j) of the upper part: row i < column j
      if (i < m && j < m && i < j) A22[i + (int64_t)j * lda] = zc{neg(tile[jj][tx].re), tile[jj][tx].im};
    }
    return;
  }
  __syncthreads();
  // off-diagonal tile: A22[j, i] = -conj(A22[i, j]) (rows j0.., columns i0..), coalesced along j
  for (int ii = ty; ii < ZU_T; ii += 8) {
    const int j = j0 + tx, i = i0 + ii;
    if (i < m && j < m) A22[j + (int64_t)i * lda] = zc{neg(tile[tx][ii].re), tile[tx][ii].im};
  }
}

__global__ void zdiag_im_kernel(const zc* __restrict__ A, int64_t lda, int n, double* dvim) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) dvim[k] = A[k + (int64_t)k * lda].im;
}

cudaError_t launch_zdiag_im(const double* A, int64_t lda, int n, double* dvim, cudaStream_t st) {
  if (!dvim || n <= 0) return cudaSuccess;
  zdiag_im_kernel<<<(n + 255) / 256, 256, 0, st>>>(reinterpret_cast<const zc*>(A), lda, n, dvim);
  return cudaGetLastError();
}

constexpr int ZTAIL = 96;  // trailing columns left to the one-CTA kernel

size_t zhess_large_ws_doubles(int n) {
  const int nchunk = (n + ZMV_CH - 1) / ZMV_CH;
  return (2 * (2 * (size_t)n) + 2 * (size_t)nchunk * n + 8 + 31) & ~(size_t)31;
}

cudaError_t zhess_large(double* Ad, int64_t lda, int n, double* taud, double* ev, double* dvim, double* wsd,
                        cudaStream_t st) {
  zc* A = reinterpret_cast<zc*>(Ad);
  zc* tau = reinterpret_cast<zc*>(taud);
  ZColWs ws;
  ws.v = reinterpret_cast<zc*>(wsd);
  ws.w = ws.v + n;
  ws.part = ws.w + n;
  const int nchunk_max = (n + ZMV_CH - 1) / ZMV_CH;
  ws.R = reinterpret_cast<ZRefl*>(ws.part + (size_t)nchunk_max * n);
  cudaError_t e;
  const int cend = n - 1 - ZTAIL;  // columns [0, cend) here, the rest by the one-CTA kernel
  for (int c = 0; c < cend; c++) {
    const int m = n - c - 1;
    zcol_refl_kernel<<<1, ZR_NT, 0, st>>>(A, lda, n, c, tau, ev, ws);
    const int nrb = (m + ZMV_ROWS - 1) / ZMV_ROWS, nch = (m + ZMV_CH - 1) / ZMV_CH;
    zcol_matvec_kernel<<<dim3(nrb, nch), ZMV_ROWS, 0, st>>>(A, lda, n, c, ws);
    zcol_combine_kernel<<<1, ZR_NT, 0, st>>>(n, c, nch, ws);
    const long long nt = (m + ZU_T - 1) / ZU_T;
    zcol_update_kernel<<<(unsigned)(nt * (nt + 1) / 2), ZU_T * 8, 0, st>>>(A, lda, n, c, ws);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  // tail: the trailing (n - c0) x (n - c0) block with the one-CTA kernel (in place, ld = lda)
  const int c0 = cend > 0 ? cend : 0;
  ZHessParams P;
  P.W = reinterpret_cast<double*>(A + c0 + (int64_t)c0 * lda);
  P.stride = 0;
  P.ld = lda;
  P.n = n - c0;
  P.count = 1;
  P.tau = reinterpret_cast<double*>(tau + c0);
  P.ev = ev + c0;
  P.dvim = nullptr;
  e = launch_zhess_cta(P, st);
  if (e != cudaSuccess) return e;
  zdiag_im_kernel<<<(n + 255) / 256, 256, 0, st>>>(A, lda, n, dvim);
  return cudaGetLastError();
}


// ===========================================================================
// Complex eigenproblem.  The reference solves eigen(Hermitian(i A)) by LAPACK
// (eigen.jl:101-106; eigvals :18-27: values -mu, mu ascending, so the imaginary
// parts come out descending).  Here: A = Q T Q^H from the reduction above, then
// i T = D S D^H with S real symmetric tridiagonal (diagonal -dvim, off-diagonal
// |ev|) and D = diag(d), d_1 = 1, d_{k+1} = d_k i sign(ev_k) (the phase scaling
// of to_symtridiagonal, tridiag.jl:558-583); S = Y diag(mu) Y^T by bisection and
// twisted-factorisation eigenvectors; the eigenvectors of A are Q D Y.
// ===========================================================================

// S's diagonal and off-diagonal, the phases, Gershgorin bound and pivmin:
// bp[0] = lower bound, bp[1] = pivmin, bp[2] = upper bound.
__global__ void __launch_bounds__(1024) zprep_kernel(const double* __restrict__ ev, const double* __restrict__ dvim,
                                                    int n, double* __restrict__ dg, double* __restrict__ off,
                                                    zc* __restrict__ ph, double* __restrict__ bp) {
  const size_t mb = blockIdx.x;  // problem of a batch: arrays n (bp: 8) apart
  ev += mb * n;
  dvim += mb * n;
  dg += mb * n;
  off += mb * n;
  ph += mb * n;
  bp += mb * 8;
  __shared__ double red[3][32];
  double lo = INFINITY, hi = -INFINITY, e2 = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double d = neg(dvim[i]);
    const double l = (i > 0) ? fabs(ev[i - 1]) : 0.0, r = (i + 1 < n) ? fabs(ev[i]) : 0.0;
    dg[i] = d;
    if (i + 1 < n) {
      off[i] = r;
      e2 = fmax(e2, r * r);
    }
    lo = fmin(lo, d - l - r);
    hi = fmax(hi, d + l + r);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    e2 = fmax(e2, __shfl_xor_sync(0xffffffffu, e2, o));
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = lo;
    red[1][threadIdx.x >> 5] = hi;
    red[2][threadIdx.x >> 5] = e2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
      lo = fmin(lo, red[0][w]);
      hi = fmax(hi, red[1][w]);
      e2 = fmax(e2, red[2][w]);
    }
    const double span = fmax(fabs(lo), fabs(hi));
    bp[0] = lo - 1e-14 * span - 1e-300;
    bp[1] = 2.2250738585072014e-308 * fmax(1.0, e2);
    bp[2] = hi + 1e-14 * span + 1e-300;
    // phases: d_{k+1} = d_k * (i sign(ev_k)), i^k times the sign product
    int quarter = 0;  // d_k = i^quarter
    ph[0] = zc{1.0, 0.0};
    for (int k = 0; k + 1 < n; k++) {
      quarter = (quarter + ((ev[k] < 0.0) ? 3 : 1)) & 3;
      const double re = (quarter == 0) ? 1.0 : ((quarter == 2) ? -1.0 : 0.0);
      const double im = (quarter == 1) ? 1.0 : ((quarter == 3) ? -1.0 : 0.0);
      ph[k + 1] = zc{re, im};
    }
  }
}

// SkewHermTridiagonal{ComplexF64} input (complex subdiagonal ev, imaginary diagonal
// dvim or none): to_symtridiagonal (tridiag.jl:558-583) gives S = SymTridiagonal(-dvim,
// |ev|) and the phases d_1 = 1, d_{k+1} = d_k (i ev_k) / |ev_k|; bnd = {lo, pivmin, hi}.
__global__ void __launch_bounds__(1024) zprep_tri_kernel(const zc* __restrict__ ev, const double* __restrict__ dvim,
                                                        int n, double* __restrict__ dg, double* __restrict__ off,
                                                        zc* __restrict__ ph, double* __restrict__ bp) {
  __shared__ double red[3][32];
  double lo = INFINITY, hi = -INFINITY, e2 = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double d = dvim ? neg(dvim[i]) : 0.0;
    const double l = (i > 0) ? hypot(ev[i - 1].re, ev[i - 1].im) : 0.0;
    const double r = (i + 1 < n) ? hypot(ev[i].re, ev[i].im) : 0.0;
    dg[i] = d;
    if (i + 1 < n) {
      off[i] = r;
      e2 = fmax(e2, r * r);
    }
    lo = fmin(lo, d - l - r);
    hi = fmax(hi, d + l + r);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    e2 = fmax(e2, __shfl_xor_sync(0xffffffffu, e2, o));
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = lo;
    red[1][threadIdx.x >> 5] = hi;
    red[2][threadIdx.x >> 5] = e2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
      lo = fmin(lo, red[0][w]);
      hi = fmax(hi, red[1][w]);
      e2 = fmax(e2, red[2][w]);
    }
    const double span = fmax(fabs(lo), fabs(hi));
    bp[0] = lo - 1e-14 * span - 1e-300;
    bp[1] = 2.2250738585072014e-308 * fmax(1.0, e2);
    bp[2] = hi + 1e-14 * span + 1e-300;
    zc d{1.0, 0.0};
    ph[0] = d;
    for (int k = 0; k + 1 < n; k++) {
      const double a = hypot(ev[k].re, ev[k].im);
      if (a > 0.0) d = zmul(d, zc{neg(ev[k].im) / a, ev[k].re / a});  // (i ev_k) / |ev_k|
      ph[k + 1] = d;
    }
  }
}

cudaError_t zsymtri_prep(const double* ev, const double* dvim, int n, double* dg, double* off, double* ph,
                         double* bnd, cudaStream_t st) {
  zprep_kernel<<<1, 1024, 0, st>>>(ev, dvim, n, dg, off, reinterpret_cast<zc*>(ph), bnd);
  return cudaGetLastError();
}

// mu_k = k-th smallest eigenvalue of S by a group of p lanes (multisection,
// absolute tolerance eps * max|Gershgorin bound|); vals_im[k] = -mu_k.  Problem
// blockIdx.y; the scaled diagonal and squares are staged for the CTA up to
// n = STURM_STAGE.
__global__ void zbisect_kernel(const double* __restrict__ dg, const double* __restrict__ off, int n,
                               const double* __restrict__ bp, double* __restrict__ mu, double* __restrict__ vals_im,
                               int p) {
  extern __shared__ double sq[];
  const int k0 = (blockIdx.x * blockDim.x + threadIdx.x) / p;
  const int gl = (threadIdx.x & 31) % p;
  const bool active = k0 < n;
  const int k = active ? k0 : 0;
  const size_t mb = blockIdx.y;
  dg += mb * n;
  off += mb * n;
  bp += mb * 8;
  const double lo = bp[0], hi = bp[2], scale = sturm_scale(fmax(fabs(lo), fabs(hi)));
  double* sd = sq + n;
  const bool staged = n <= STURM_STAGE;
  if (staged) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const double v = (i + 1 < n) ? off[i] * scale : 0.0;
      sq[i] = v * v;
      sd[i] = dg[i] * scale;
    }
    __syncthreads();
  }
  auto count = [&](double y) {
    const double x = y * scale;
    if (staged) return sturm_products(n, [&](int i) { return sd[i] - x; }, [&](int i) { return sq[i]; });
    return sturm_products(n, [&](int i) { return fma(dg[i], scale, neg(x)); }, [&](int i) {
      const double v = off[i] * scale;
      return v * v;
    });
  };
  const double x = group_rootsect(lo, hi, k, 2.220446049250313e-16 * fmax(fabs(lo), fabs(hi)), p, active, count);
  if (active && gl == 0) {
    if (mu) mu[mb * n + k] = x;
    vals_im[mb * n + k] = neg(x);
  }
}

static cudaError_t launch_zbisect(const double* dg, const double* off, int n, int batch, const double* bp, double* mu,
                                  double* vals_im, cudaStream_t st) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int p = multisect_lanes(n * batch, sms);
  const unsigned ctas = (unsigned)(((long long)n * p + 127) / 128);
  const size_t smem = n <= STURM_STAGE ? 2 * n * sizeof(double) : 0;
  zbisect_kernel<<<dim3(ctas, batch), 128, smem, st>>>(dg, off, n, bp, mu, vals_im, p);
  return cudaGetLastError();
}

// V(:, k) = D Y(:, k)
__global__ void zassemble_kernel(const double* __restrict__ Y, const zc* __restrict__ ph, int n, zc* __restrict__ V,
                                 int64_t ldv) {
  const size_t mb = blockIdx.z;  // problem mb: Y, V n^2 (V: ldv n) apart, ph n apart
  Y += mb * n * n;
  ph += mb * n;
  V += mb * (size_t)ldv * n;
  const int k = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double y = Y[i + (int64_t)k * n];
    V[i + (int64_t)k * ldv] = zc{ph[i].re * y, ph[i].im * y};
  }
}

// ---------------------------------------------------------------------------
// X <- Q X (skew_back.cuh): problem b at A + lda n b, tau + n b, X + ldx n b (complex)
// ---------------------------------------------------------------------------
struct ZBack {
  BackTask<true> B;  // problem 0
  size_t stride;     // doubles of workspace per problem
  __device__ bool get(int b, BackTask<true>& T) const {
    T = B;
    T.A += 2 * (size_t)b * B.lda * B.n;
    T.tau += 2 * (size_t)b * B.n;
    T.X[0] += 2 * (size_t)b * B.ldx * B.n;
    const size_t o = b * stride;
    T.t += o;
    T.vt += o;
    T.w += o;
    T.et += 2 * o;
    T.evt += 2 * o;
    T.ex += 2 * o;
    if (T.status) T.status += b;
    return true;
  }
};

// workspace segments are rounded to 32 doubles so that every complex array is 16-byte aligned
static inline size_t seg(size_t d) { return (d + 31) & ~(size_t)31; }

// The back-transformation's workspace lies in that of the vectors, which are done with it,
// where it fits (3 n KP doubles per problem; splits of W are chosen to fit).
static size_t zback_extra_doubles(int n, int batch) {
  const size_t per = seg(n > 1 ? back_ws_doubles<true>(n, n - 1, n, 1) : 0);
  return per <= large_eigen_ws_doubles(n) ? 0 : seg((size_t)batch * per);
}

size_t zeigen_ws_doubles(int n, int batch) {
  const size_t B = (size_t)(batch > 0 ? batch : 1);
  return 3 * seg(B * n)                      // dg, off, mu
         + seg(2 * B * n)                    // phases
         + seg(8 * B)                        // bp
         + seg(B * n * n)                    // Y
         + zback_extra_doubles(n, (int)B)
         + B * large_eigen_ws_doubles(n) + 64;
}

// Eigen-decomposition of `batch` reduced matrices of size n (A: the reflectors,
// lda*n apart; tau, ev, dvim, vals_im n apart): vals_im (descending) and, if
// V != null, the eigenvectors V (ldv*n apart).
cudaError_t zeigen_from_tridiag(const double* Ad, int64_t lda, int n, const double* taud, const double* ev,
                                const double* dvim, double* vals_im, double* Vd, int64_t ldv, double* ws, int batch,
                                int* status, int skip_cta, cudaStream_t st) {
  const size_t B = (size_t)batch;
  double* dg = ws;
  double* off = dg + seg(B * n);
  double* mu = off + seg(B * n);
  zc* ph = reinterpret_cast<zc*>(mu + seg(B * n));
  double* bp = mu + seg(B * n) + seg(2 * B * n);
  double* Y = bp + seg(8 * B);
  double* extra = Y + seg(B * n * n);
  const size_t nextra = zback_extra_doubles(n, batch);
  double* tws = extra + nextra;
  zprep_kernel<<<batch, 1024, 0, st>>>(ev, dvim, n, dg, off, ph, bp);
  cudaError_t e = launch_zbisect(dg, off, n, batch, bp, mu, vals_im, st);
  if (e != cudaSuccess || !Vd) return e;
  e = symtri_vectors(dg, off, n, mu, bp, Y, tws, batch, st);
  if (e != cudaSuccess) return e;
  zc* V = reinterpret_cast<zc*>(Vd);
  zassemble_kernel<<<dim3((n + 255) / 256, n, batch), 256, 0, st>>>(Y, ph, n, V, ldv);
  e = cudaGetLastError();
  if (e != cudaSuccess || n < 2) return e;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  ZBack S;
  S.B.A = Ad;
  S.B.lda = lda;
  S.B.tau = taud;
  S.B.n = n;
  S.B.nref = n - 1;
  S.B.X[0] = S.B.X[1] = Vd;
  S.B.ldx = ldv;
  S.B.nc[0] = n;
  S.B.nc[1] = 0;
  S.B.identity = 0;
  S.B.status = status;
  S.B.skip_cta = skip_cta;
  int splits = 1;
  if (nextra) {
    S.stride = seg(back_ws_doubles<true>(n, n - 1, n, 1));
  } else {
    S.stride = large_eigen_ws_doubles(n);
    splits = back_splits(n, batch, sms);
    while (splits > 1 && back_ws_doubles<true>(n, n - 1, n, splits) > S.stride) splits /= 2;
  }
  back_ws_set(S.B, nextra ? extra : tws, n, splits);
  return back_transform_oz<true>(S, batch, n, n - 1, n, splits, st);
}

// ---------------------------------------------------------------------------
// complex products for exp and its adjoint: C = op(A) op(B), op in {N, H}, on the tensor
// cores (skew_oz.cuh) as the real product of [[Re, -Im], [Im, Re]] of op(A) with op(B)'s
// interleaved columns.  The four products of 64 matrices of n = 256: 27.5 -> 1.9 ms; one
// at n = 1501: 22.4 -> 1.4 ms.
// ---------------------------------------------------------------------------
struct ZGemm {
  const double* A;
  const double* B;
  double* C;
  int64_t lda, ldb, ldc;
  int n, ha, hb;
  int *ea, *eb;  // largest exponents of op(A)'s rows and op(B)'s columns, n per problem
  int* status;   // SKEW_TIMEOUT per problem (or null)
};

// grid (vectors / 8, 2, batch): one warp per vector
__global__ void __launch_bounds__(256) zexps_kernel(ZGemm P) {
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5), n = P.n;
  if (i >= n) return;
  const size_t mb = blockIdx.z;
  const bool side = blockIdx.y != 0;
  const int64_t ld = side ? P.ldb : P.lda;
  const bool column = side ? !P.hb : (P.ha != 0);  // the vector is a column of the stored matrix
  const double* M = (side ? P.B : P.A) + 2 * mb * (size_t)ld * n;
  int e = 1;
  for (int k = threadIdx.x & 31; k < n; k += 32) {
    const double2 z = *reinterpret_cast<const double2*>(M + 2 * (column ? k + i * ld : i + k * ld));
    e = max(e, max(oz_exponent(z.x), oz_exponent(z.y)));
  }
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0) (side ? P.eb : P.ea)[mb * n + i] = e;
}

struct ZGemmTile : ZGemm {
  __device__ int rows() const { return 2 * n; }
  __device__ int cols() const { return n; }
  __device__ int ksteps() const { return (2 * n + OZ_K - 1) / OZ_K; }
  __device__ bool contiguousA() const { return ha; }
  __device__ bool contiguousB() const { return !hb; }
  __device__ int expA(int i) const { return ea[i >> 1]; }
  __device__ int expB(int j) const { return eb[j]; }
  __device__ void loadA(int i, int s, int k, double (&v)[8]) const {
    const int k0 = (s * OZ_K + k) / 2, r = i >> 1;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      double2 z = make_double2(0.0, 0.0);
      if (k0 + u < n) z = *reinterpret_cast<const double2*>(A + 2 * (ha ? k0 + u + r * lda : r + (k0 + u) * lda));
      const double im = ha ? neg(z.y) : z.y;
      v[2 * u] = (i & 1) ? im : z.x;
      v[2 * u + 1] = (i & 1) ? z.x : neg(im);
    }
  }
  __device__ void loadB(int j, int s, int k, double (&v)[4]) const {
    const int k0 = (s * OZ_K + k) / 2;
#pragma unroll
    for (int u = 0; u < 2; u++) {
      double2 z = make_double2(0.0, 0.0);
      if (k0 + u < n) z = *reinterpret_cast<const double2*>(B + 2 * (hb ? j + (k0 + u) * ldb : k0 + u + j * ldb));
      v[2 * u] = z.x;
      v[2 * u + 1] = hb ? neg(z.y) : z.y;
    }
  }
  __device__ void store(int i, int j, double x) const { C[i + 2 * j * ldc] = x; }
  __device__ void timeout() const {
    if (status) *status = SKEW_TIMEOUT;
  }
};

__global__ void __launch_bounds__(OZ_NT, 1) zgemm_kernel(ZGemm P, int rt) {  // grid (row x column tiles, batch)
  extern __shared__ __align__(1024) unsigned char oz_buf[];
  const size_t mb = blockIdx.y;  // problem mb: each operand ld*n apart
  ZGemmTile T;
  static_cast<ZGemm&>(T) = P;
  T.A += 2 * mb * (size_t)P.lda * P.n;
  T.B += 2 * mb * (size_t)P.ldb * P.n;
  T.C += 2 * mb * (size_t)P.ldc * P.n;
  T.ea += mb * P.n;
  T.eb += mb * P.n;
  if (T.status) T.status += mb;
  oz_tile(T, (int)(blockIdx.x % rt) * OZ_M, (int)(blockIdx.x / rt) * OZ_N, oz_buf);
}

static cudaError_t zgemm(int n, const zc* A, int64_t lda, int ha, const zc* B, int64_t ldb, int hb, zc* C, int64_t ldc,
                         int* exps, int batch, int* status, cudaStream_t st) {
  static std::atomic<uint64_t> raised{0};
  cudaError_t e = raise_smem_limit_once((const void*)zgemm_kernel, raised);
  if (e != cudaSuccess) return e;
  ZGemm P{reinterpret_cast<const double*>(A), reinterpret_cast<const double*>(B), reinterpret_cast<double*>(C),
          lda, ldb, ldc, n, ha, hb, exps, exps + (size_t)batch * n, status};
  const int rt = (2 * n + OZ_M - 1) / OZ_M, ct = (n + OZ_N - 1) / OZ_N;
  zexps_kernel<<<dim3((n + 7) / 8, 2, batch), 256, 0, st>>>(P);
  zgemm_kernel<<<dim3(rt * ct, batch), OZ_NT, OZ_SMEM, st>>>(P, rt);
  return cudaGetLastError();
}

// mode 0: P(:, k) = V(:, k) f(i mu_k)   (F = P V^H for the function `func`)
// mode 1: M(j, k) <- conj(Phi(j, k)) M(j, k), Phi(j,k) = e^{i(mu_j+mu_k)/2} sinc((mu_j-mu_k)/2)
__global__ void zscale_kernel(int mode, int func, int n, const double* __restrict__ mu, const zc* __restrict__ V,
                              int64_t ldv, zc* __restrict__ M, int64_t ldm, int* __restrict__ status) {
  const size_t mb = blockIdx.z;  // problem mb: mu n, V ldv*n, M ldm*n apart
  mu += mb * n;
  V += mb * (size_t)ldv * n;
  M += mb * (size_t)ldm * n;
  const int k = blockIdx.y;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    if (mode == 0) {
      double fa, fb;
      bool sing = false;
      skew_scalar_func(func, mu[k], &fa, &fb, &sing);
      if (sing && j == 0 && status) status[mb] = SKEW_SINGULAR;
      M[j + (int64_t)k * ldm] = zmul(V[j + (int64_t)k * ldv], zc{fa, fb});
    } else {
      const double a = mu[j], bb = mu[k];
      const double d = 0.5 * (a - bb);
      const double sc = (fabs(d) < 1e-8) ? fma(neg(d) * d, 1.0 / 6.0, 1.0) : sin(d) / d;
      double s, c;
      sincos(0.5 * (a + bb), &s, &c);
      M[j + (int64_t)k * ldm] = zmul(M[j + (int64_t)k * ldm], zc{c * sc, neg(s) * sc});
    }
  }
}

// O <- (O + s O^H) / 2 in place (s = +1 Hermitian part, -1 skew-Hermitian part)
__global__ void zsymmetrize_kernel(int n, zc* __restrict__ O, int64_t ldo, int s) {
  O += (size_t)blockIdx.z * ldo * n;
  const int64_t tot = (int64_t)n * n;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < tot; q += (int64_t)gridDim.x * blockDim.x) {
    const int j = (int)(q / n), i = (int)(q - (int64_t)j * n);
    if (i < j) continue;
    zc* pij = O + i + (int64_t)j * ldo;
    if (i == j) {  // Hermitian: real diagonal; skew-Hermitian: imaginary diagonal
      if (s > 0)
        pij->im = 0.0;
      else
        pij->re = 0.0;
      continue;
    }
    zc* pji = O + j + (int64_t)i * ldo;
    const zc x = *pij, y = *pji;
    const zc u = zc{0.5 * (x.re + s * y.re), 0.5 * (x.im - s * y.im)};  // (x + s conj(y)) / 2
    *pij = u;
    *pji = zc{s * u.re, neg(s * u.im)};  // s conj(u)
  }
}

cudaError_t zfunc_from_eigen(int mode, int func, int n, const double* vals_im, const double* Vd, int64_t ldv,
                             const double* Cd, int64_t ldc, double* Od, int64_t ldo, double* ws, int batch,
                             int* status, cudaStream_t st) {
  const zc* V = reinterpret_cast<const zc*>(Vd);
  zc* O = reinterpret_cast<zc*>(Od);
  zc* T1 = reinterpret_cast<zc*>(ws);
  zc* T2 = T1 + (size_t)batch * n * n;
  int* exps = reinterpret_cast<int*>(T2 + (size_t)batch * n * n);
  auto gemm = [&](const zc* A, int64_t lda, int ha, const zc* B, int64_t ldb, int hb, zc* C, int64_t ldc) {
    return zgemm(n, A, lda, ha, B, ldb, hb, C, ldc, exps, batch, status, st);
  };
  cudaError_t e;
  const dim3 gs((n + 255) / 256, n, batch);
  if (mode == 0) {  // F = V diag(f(i mu)) V^H, then its (skew-)Hermitian part
    zscale_kernel<<<gs, 256, 0, st>>>(0, func, n, vals_im, V, ldv, T1, n, status);
    if ((e = gemm(T1, n, 0, V, ldv, 1, O, ldo))) return e;
    const int sym = skew_func_symmetry(func);
    if (sym != 0) {
      const int64_t tot = (int64_t)n * n;
      zsymmetrize_kernel<<<dim3((unsigned)std::min<int64_t>((tot + 255) / 256, 1024), 1, batch), 256, 0, st>>>(
          n, O, ldo, sym);
    }
  } else {  // G = V (conj(Phi) o (V^H C V)) V^H
    const zc* C = reinterpret_cast<const zc*>(Cd);
    if ((e = gemm(V, ldv, 1, C, ldc, 0, T1, n)) ||  // V^H C
        (e = gemm(T1, n, 0, V, ldv, 0, T2, n)))     // (V^H C) V
      return e;
    zscale_kernel<<<gs, 256, 0, st>>>(1, 0, n, vals_im, V, ldv, T2, n, nullptr);
    if ((e = gemm(V, ldv, 0, T2, n, 0, T1, n)) ||   // V M
        (e = gemm(T1, n, 0, V, ldv, 1, O, ldo)))    // (V M) V^H
      return e;
  }
  return cudaGetLastError();
}

size_t zfunc_ws_doubles(int n, int batch) { return (size_t)batch * n * (4 * (size_t)n + 1) + 32; }

// eigen of a SkewHermTridiagonal{ComplexF64}: vals_im (descending) and, if V != null,
// V = D Y (no reflectors); ws: zeigen_ws_doubles(n, 1)
cudaError_t zeigen_tridiag(const double* evd, const double* dvim, int n, double* vals_im, double* Vd, int64_t ldv,
                           double* ws, cudaStream_t st) {
  double* dg = ws;
  double* off = dg + seg(n);
  double* mu = off + seg(n);
  zc* ph = reinterpret_cast<zc*>(mu + seg(n));
  double* bp = mu + seg(n) + seg(2 * (size_t)n);
  double* Y = bp + seg(8);
  double* tws = Y + seg((size_t)n * n) + zback_extra_doubles(n, 1);
  zprep_tri_kernel<<<1, 1024, 0, st>>>(reinterpret_cast<const zc*>(evd), dvim, n, dg, off, ph, bp);
  cudaError_t e = launch_zbisect(dg, off, n, 1, bp, mu, vals_im, st);
  if (e != cudaSuccess || !Vd) return e;
  e = symtri_vectors(dg, off, n, mu, bp, Y, tws, 1, st);
  if (e != cudaSuccess) return e;
  zassemble_kernel<<<dim3((n + 255) / 256, n, 1), 256, 0, st>>>(Y, ph, n, reinterpret_cast<zc*>(Vd), ldv);
  return cudaGetLastError();
}

}  // namespace skew
