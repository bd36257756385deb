// Blocked ComplexF64 skew-Hermitian tridiagonalisation of one large matrix: the complex
// skewlatrd! panel (hessenberg.jl:92-131, with the alpha correction of :123-126) in one
// cooperative launch per panel, then the trailing update of skewblockedhess!
// (:158-166), A22 += V W^H - W V^H on the lower triangle, mirrored as -conj, on the
// tensor cores.
//
// Per panel column c (panel step i, panel start p):
//   -  every CTA forms reflector c from the same norm partials in the same order (warp 0)
//      and stages the column.
//   A  Each warp takes a static share of the items: the panel dots u1 = W^H x and
//      u2 = V^H x over ZDOT rows, and (32-row, column-chunk) tiles of A22 x whose partial
//      sums go to ypart; each CTA also writes its share of x^H (A22 x).
//   B  every CTA sums the partials in a fixed order and forms the alpha correction without
//      a further reduction: with y = A22 v + V u1 - W u2,
//        v^H y = v^H (A22 v) + u2^H u1 - u1^H u2,   alpha = |tau|^2 conj(v^H y) / 2,
//      which equals tau (W^H v) / 2 for W = tau y (the reference's
//      tau * dot(W, v) / 2).  Row blocks then form W[:, i] = tau y + alpha v, store
//      v into column c, apply the deferred rank-2(i+1) update to column c+1 and
//      write the norm partials of its rows below the subdiagonal.
// Two grid barriers per column, each a monotonic arrival counter polled with acquire loads
// and a bounded number of polls (error flag, every CTA returns, the call reports
// SKEW_TIMEOUT).  Data written by other CTAs during the launch is read through L2 (__ldcg).
//
// What bounds it: a chain of about 21 us per column, of which A22 x needs 5 us on average
// at n = 1501 (its 4 m^2 FMAs on the FP64 pipe, 2 per clock and SM; the matrix stays in
// L2).  The rest is latency: two barriers 4 us, the reflector (a square root and a
// division) 3, the sums before alpha 3, the rows 2 to 3.  An FP64 instruction holds its
// quarter of the SM for 64 cycles however few of its lanes count, so what is left of the
// FP64 work in the serial parts is spread over lanes and quarters.  n = 1501, whole
// reduction: 63 ms -> 34 ms (per column 44 us -> 21; trailing updates 16 ms on the FP64
// pipe -> 1.8 ms).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "skew_common.cuh"
#include "skew_complex.cuh"
#include "skew_internal.h"
#include "skew_oz.cuh"

namespace skew {

namespace {

constexpr int ZP_NT = 256;
constexpr int ZP_NW = ZP_NT / 32;
constexpr int ZBNB = 32;   // largest panel width
constexpr int ZDOT = 256;  // rows per panel dot item
constexpr int ZP_MAXCK = 128;  // column chunks of a matvec
constexpr int ZTAILP = 128;  // trailing columns left to the one-CTA kernel
constexpr long long ZP_POLL = 1LL << 24;  // default polls before a grid barrier gives up
constexpr int ZP_MAXCTAS = 2048;

struct ZRef {
  zc tau, scale;
  double beta;
};

// Reflector of (alpha, |x[2:]|), hessenberg.jl:26-44 complex branch (as zrefl).
__device__ ZRef zp_refl(zc alpha, double xnorm) {
  ZRef R;
  if (xnorm == 0.0 && alpha.re == 0.0 && alpha.im == 0.0) {
    R.tau = zc{0.0, 0.0};
    R.scale = zc{0.0, 0.0};
    R.beta = 0.0;
    return R;
  }
  const double h = hypot(hypot(alpha.re, alpha.im), xnorm);
  const double beta = (alpha.re > 0.0) ? neg(h) : h;
  const double rb = 1.0 / beta;
  R.beta = beta;
  R.tau = zc{1.0 - alpha.re * rb, neg(alpha.im * rb)};
  R.scale = zinv(zc{alpha.re - beta, alpha.im});
  return R;
}

__device__ __forceinline__ zc ldz(const zc* p) {
  const double2 v = __ldcg((const double2*)p);
  return zc{v.x, v.y};
}
__device__ __forceinline__ void stz(zc* p, zc x) { __stcg((double2*)p, make_double2(x.re, x.im)); }
__device__ __forceinline__ bool zzero(zc z) { return z.re == 0.0 && z.im == 0.0; }

__device__ __forceinline__ double zp_block_max(double x, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < ZP_NW; i++) s = fmax(s, red[i]);
  __syncthreads();
  return s;
}

}  // namespace

struct ZPersistParams {
  zc* A;
  int64_t lda;
  int n, p, nbp;   // this launch's panel: reflector columns [p, p + nbp), nbp <= ZBNB
  unsigned round;  // grid barriers of the panels before
  zc* tau;
  double* ev;
  zc* W;           // n x ZBNB, column j at W + j * n
  zc* ypart;       // column chunks x n
  zc* dpart;       // one per CTA
  zc* u;           // per ZDOT rows: ZBNB of W^H v, ZBNB of V^H v
  double* sspart;  // norm partials, one per CTA
  int *ea, *ew;    // largest exponents of the panel's rows of V and W
  unsigned* sync;  // [0] barrier arrivals, [1] a wait gave up, [2] largest exponent of W
  int items_per_warp;    // matvec tiles per warp and column (chunk count)
  long long poll_limit;  // polls before a grid barrier gives up
  int skip_cta;          // >= 0: this CTA never arrives (a test of the timeout path)
};

namespace {

// Grid barrier; pre() is run by thread 0 between the CTA's own barrier and its arrival.
template <class Pre>
__device__ bool zp_gsync(const ZPersistParams& P, unsigned& round, Pre pre) {
  __shared__ int s_ok;
  __syncthreads();
  round++;
  if (threadIdx.x == 0) {
    const unsigned target = round * gridDim.x;
    int ok = 1;
    unsigned* cnt = P.sync;
    volatile unsigned* err = P.sync + 1;
    long long it = 0;
    if ((int)blockIdx.x == P.skip_cta) {
      // no arrival: the others give up after poll_limit polls; wait (bounded) for that
      while (!*err && ++it <= P.poll_limit) __nanosleep(32);
      ok = 0;
    } else {
      pre();
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(cnt) : "memory");
      for (;;) {
        unsigned cur;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(cnt) : "memory");
        if ((int)(cur - target) >= 0) break;
        if ((++it & 63) == 0) {
          if (*err) {
            ok = 0;
            break;
          }
          if (it > P.poll_limit) {
            atomicExch(P.sync + 1, 1u);
            ok = 0;
            break;
          }
          __nanosleep(32);
        }
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Reflector of column c from its entries, by the whole CTA (identical in every CTA).
__device__ ZRef zp_refl_from_column(const ZPersistParams& P, int c, double* red) {
  const int n = P.n;
  const zc* col = P.A + (int64_t)c * P.lda;
  double part = 0.0;
  for (int r = c + 2 + threadIdx.x; r < n; r += ZP_NT) {
    const zc x = ldz(col + r);
    part = fma(x.re, x.re, fma(x.im, x.im, part));
  }
  const double ss = block_sum<ZP_NW>(part, red);
  double xn = sqrt(ss);
  if (ss_needs_scaling(ss)) {
    double mx = 0.0;
    for (int r = c + 2 + threadIdx.x; r < n; r += ZP_NT) {
      const zc x = ldz(col + r);
      mx = fmax(mx, fmax(fabs(x.re), fabs(x.im)));
    }
    mx = zp_block_max(mx, red);
    double qq = 0.0;
    if (mx > 0.0) {
      const double inv = 1.0 / mx;
      for (int r = c + 2 + threadIdx.x; r < n; r += ZP_NT) {
        const zc x = ldz(col + r);
        const double a = x.re * inv, b = x.im * inv;
        qq = fma(a, a, fma(b, b, qq));
      }
    }
    qq = block_sum<ZP_NW>(qq, red);
    xn = mx * sqrt(qq);
  }
  // one thread forms the reflector (a warp-wide FP64 instruction costs the same
  // with one lane as with 32), the others read it from shared memory
  __shared__ ZRef s_R;
  if (threadIdx.x == 0) s_R = zp_refl(ldz(col + c + 1), xn);
  __syncthreads();
  const ZRef R = s_R;
  __syncthreads();
  return R;
}

// Reflector from alpha and ss = |x[2:]|^2 in the safe range, by a full warp: lanes 0 and 1
// divide at once.  |alpha - beta|^2 lies between h^2 and 4 h^2.
__device__ ZRef zp_refl_warp(zc alpha, double ss) {
  ZRef R;
  const double t = fma(alpha.re, alpha.re, fma(alpha.im, alpha.im, ss));
  if (ss == 0.0 || !(t < 1e290)) return zp_refl(alpha, sqrt(ss));
  const double h = sqrt(t);
  R.beta = (alpha.re > 0.0) ? neg(h) : h;
  const double dr = alpha.re - R.beta, d2 = fma(dr, dr, alpha.im * alpha.im);
  const double q = 1.0 / ((threadIdx.x & 31) == 0 ? R.beta : d2);
  const double rb = __shfl_sync(0xffffffffu, q, 0), rd = __shfl_sync(0xffffffffu, q, 1);
  R.tau = zc{1.0 - alpha.re * rb, neg(alpha.im * rb)};
  R.scale = zc{dr * rd, neg(alpha.im * rd)};
  return R;
}

static_assert(ZP_NW == 8 && ZBNB == 32, "the warps' shares of the head, a lane per panel column");
struct ZpShared {
  zc u[2 * ZBNB], Wrow[ZBNB], Arow[ZBNB];
  double red[2 * ZP_NW], dot[2], y1[2], alpha[2], yt[2];
};

// The vector of a column: v = x s with x staged in shared memory, its entries scaled by a
// power of two to at most 1 (an integer operation; multiplying by s would cost 4 FP64
// operations per entry in every CTA); v[c + 1] is 1 (0: no reflector).
struct ZpVec {
  zc s;
  double one;
};

// Phase B head: u1, u2 and x^H (A22 x) from their partials in a fixed order, row c + 1 of V,
// W and y; from these alpha and y[c + 1].  An FP64 instruction holds its quarter of the SM
// for 64 cycles whatever its lanes, so components go to different lanes and warps.
__device__ __forceinline__ void zp_head(const ZPersistParams& P, int c, int i, int nck, const ZRef& R, const ZpVec& V,
                                        ZpShared& H) {
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int n = P.n, r0 = c + 1, nd = (n - r0 + ZDOT - 1) / ZDOT;
  double cs = 0.0, ct = 0.0;
  if (w < 4) {  // component tid & 1 of dot tid / 2
    double x = 0.0;
    if (((tid >> 1) & (ZBNB - 1)) < i)
      for (int q = 0; q < nd; q += 8) {
        double t[8];
#pragma unroll
        for (int z = 0; z < 8; z++)
          t[z] = (q + z < nd) ? __ldcg(reinterpret_cast<const double*>(P.u + (size_t)(q + z) * 2 * ZBNB) + tid) : 0.0;
#pragma unroll
        for (int z = 0; z < 8; z++)
          if (q + z < nd) x += t[z];
      }
    const double o = __shfl_xor_sync(0xffffffffu, x, 1);
    reinterpret_cast<double*>(H.u)[tid] = fma(V.s.re, x, ((tid & 1) ? V.s.im : neg(V.s.im)) * o);
    if (w == 0 || w == 3) {
      ct = 0.5 * fma(R.tau.re, R.tau.re, R.tau.im * R.tau.im);
      cs = ct * fma(V.s.re, V.s.re, V.s.im * V.s.im);
    }
  } else if (w < 6) {
    if (lane < i) {
      if (w == 4)
        H.Wrow[lane] = ldz(P.W + (size_t)lane * n + r0);
      else
        H.Arow[lane] = ldz(P.A + r0 + (int64_t)(P.p + lane) * P.lda);
    }
    double x = 0.0;
    for (int q = lane; q < (int)gridDim.x; q += 160) {
      double t[5];
#pragma unroll
      for (int z = 0; z < 5; z++)
        t[z] = (q + 32 * z < (int)gridDim.x) ? __ldcg(reinterpret_cast<const double*>(P.dpart + q + 32 * z) + (w & 1)) : 0.0;
#pragma unroll
      for (int z = 0; z < 5; z++) x += t[z];
    }
    x = warp_sum(x);
    if (lane == 0) H.dot[w & 1] = x;
  } else {
    double x = 0.0;
    for (int q = lane; q < nck; q += 32)
      x += __ldcg(reinterpret_cast<const double*>(P.ypart + (size_t)q * n + r0) + (w & 1));
    x = warp_sum(x);
    if (lane == 0) H.y1[w & 1] = x;
  }
  __syncthreads();
  // v^H y = v^H (A22 v) + u2^H u1 - u1^H u2 (the last two: 2i Im(u2^H u1)),
  // alpha = |tau|^2 conj(v^H y) / 2;  y_{c+1} = (A22 v)_{c+1} + sum_j (V[c+1, j] u1_j - W[c+1, j] u2_j)
  if (w < 3) {
    double x = 0.0;
    if (lane < i) {
      const zc u1 = H.u[lane], u2 = H.u[ZBNB + lane];
      if (w == 0) {
        x = fma(u2.re, u1.im, neg(u2.im * u1.re));
      } else {
        const zc a = H.Arow[lane], b = H.Wrow[lane];
        x = (w == 1) ? fma(a.re, u1.re, fma(neg(a.im), u1.im, fma(neg(b.re), u2.re, b.im * u2.im)))
                     : fma(a.re, u1.im, fma(a.im, u1.re, fma(neg(b.re), u2.im, neg(b.im * u2.re))));
      }
    }
    x = warp_sum(x);
    if (lane == 0) {
      if (w == 0)
        H.alpha[1] = neg(fma(cs, H.dot[1], 2.0 * ct * x));
      else if (w == 1)
        H.yt[0] = fma(V.s.re, H.y1[0], fma(neg(V.s.im), H.y1[1], x));
      else
        H.yt[1] = fma(V.s.re, H.y1[1], fma(V.s.im, H.y1[0], x));
    }
  } else if (w == 3 && lane == 0) {
    H.alpha[0] = cs * H.dot[0];
  }
  __syncthreads();
}

// Sum over groups of TPR neighbouring lanes: re in the even, im in the odd lanes.
template <int TPR>
__device__ __forceinline__ double zp_group_sum(zc v) {
  const bool odd = threadIdx.x & 1;
  double x = odd ? v.im : v.re;
  x += __shfl_xor_sync(0xffffffffu, odd ? v.re : v.im, 1);
#pragma unroll
  for (int o = 2; o < TPR; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Phase B: rows, TPR threads per row; row blocks go to the warps like the items of phase
// A, so that TPR chosen for one block per quarter SM spreads the FP64 work evenly.
// Everything a thread reads for its first row is requested before the head, whose chain of
// sums hides the reads.
template <int TPR>
__device__ void zp_rows(const ZPersistParams& P, int c, int i, int nck, bool last, const ZRef& R, const ZpVec& V,
                        const zc* vs, ZpShared& H, double& ssp) {
  constexpr int RPW = 32 / TPR, NJ = ZBNB / TPR;
  const int n = P.n, lane = threadIdx.x & 31, g = lane % TPR, odd = lane & 1;
  const int64_t lda = P.lda;
  const int nrb = (n - c - 1 + RPW - 1) / RPW;
  const int rb0 = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  zc aj[NJ], wj[NJ], y;  // panel terms j = g + TPR t, this thread's share of A22 x
  double old = 0.0;      // its component of A[row, c + 1]
  auto load = [&](int rb) {
    const int row = c + 1 + rb * RPW + lane / TPR;
    const bool valid = rb < nrb && row < n;
#pragma unroll
    for (int t = 0; t < NJ; t++) {
      const int j = g + TPR * t;
      aj[t] = zc{0.0, 0.0};
      wj[t] = zc{0.0, 0.0};
      if (valid && j < i) {
        aj[t] = ldz(P.A + row + (int64_t)(P.p + j) * lda);
        wj[t] = ldz(P.W + (size_t)j * n + row);
      }
    }
    y = zc{0.0, 0.0};
    if (valid) {
      if (!last && g < 2) old = __ldcg(reinterpret_cast<const double*>(P.A + row + (int64_t)(c + 1) * lda) + odd);
      for (int q = g; q < nck; q += 4 * TPR) {
        zc x[4];
#pragma unroll
        for (int z = 0; z < 4; z++)
          x[z] = (q + z * TPR < nck) ? ldz(P.ypart + (size_t)(q + z * TPR) * n + row) : zc{0.0, 0.0};
#pragma unroll
        for (int z = 0; z < 4; z++)
          if (q + z * TPR < nck) y = zadd(y, x[z]);
      }
    }
  };
  load(rb0);
  zp_head(P, c, i, nck, R, V, H);
  ssp = 0.0;
  const zc alpha{H.alpha[0], H.alpha[1]}, yt{H.yt[0], H.yt[1]};
  const zc Wi = zfma(R.tau, yt, alpha);  // W[c + 1, i]
  for (int rb = rb0; rb < nrb; rb += gridDim.x * ZP_NW) {
    if (rb != rb0) load(rb);
    const int row = c + 1 + rb * RPW + lane / TPR;
    const bool valid = row < n;
    zc acc = zmul(y, V.s);
#pragma unroll
    for (int t = 0; t < NJ; t++) {
      if (TPR * t < i) {
        const int j = g + TPR * t;  // beyond i: aj, wj are zero
        const zc u1 = (j < i) ? H.u[j] : zc{0.0, 0.0}, u2 = (j < i) ? H.u[ZBNB + j] : zc{0.0, 0.0};
        acc.re = fma(aj[t].re, u1.re, fma(neg(aj[t].im), u1.im, fma(neg(wj[t].re), u2.re, fma(wj[t].im, u2.im, acc.re))));
        acc.im = fma(aj[t].re, u1.im, fma(aj[t].im, u1.re, fma(neg(wj[t].re), u2.im, fma(neg(wj[t].im), u2.re, acc.im))));
      }
    }
    const double yo = zp_group_sum<TPR>(acc), yx = __shfl_xor_sync(0xffffffffu, yo, 1);
    const zc x = valid ? vs[row] : zc{0.0, 0.0};
    double vo = fma(V.s.re, odd ? x.im : x.re, odd ? V.s.im * x.re : neg(V.s.im * x.im));
    if (row == c + 1) vo = odd ? 0.0 : V.one;
    const double vx = __shfl_xor_sync(0xffffffffu, vo, 1);
    // W = tau y + alpha v
    double wo = fma(alpha.re, vo, fma(odd ? alpha.im : neg(alpha.im), vx,
                                      fma(R.tau.re, yo, (odd ? R.tau.im : neg(R.tau.im)) * yx)));
    if (row == c + 1) wo = odd ? Wi.im : Wi.re;
    if (valid && g < 2) {
      __stcg(reinterpret_cast<double*>(P.W + (size_t)i * n + row) + odd, wo);
      __stcg(reinterpret_cast<double*>(P.A + row + (int64_t)c * lda) + odd, vo);
    }
    if (last) continue;
    // deferred update of column c+1 (rows c+1.., the diagonal included):
    // A[row, c+1] += sum_{j <= i} V[row, j] conj(W[c+1, j]) - W[row, j] conj(V[c+1, j])
    zc uu{0.0, 0.0};
#pragma unroll
    for (int t = 0; t < NJ; t++) {
      if (TPR * t < i) {
        const int j = g + TPR * t;
        const zc a = (j < i) ? H.Arow[j] : zc{0.0, 0.0}, b = (j < i) ? H.Wrow[j] : zc{0.0, 0.0};
        uu.re = fma(aj[t].re, b.re, fma(aj[t].im, b.im, fma(neg(wj[t].re), a.re, fma(neg(wj[t].im), a.im, uu.re))));
        uu.im = fma(aj[t].im, b.re, fma(neg(aj[t].re), b.im, fma(neg(wj[t].im), a.re, fma(wj[t].re, a.im, uu.im))));
      }
    }
    double uo = zp_group_sum<TPR>(uu);
    uo = fma(vo, Wi.re, fma(vx, odd ? neg(Wi.im) : Wi.im, fma(neg(wo), V.one, uo)));
    if (row == c + 1 && !odd) uo = 0.0;  // the diagonal receives the imaginary part only
    if (valid && g < 2) {
      const double a = old + uo;
      __stcg(reinterpret_cast<double*>(P.A + row + (int64_t)(c + 1) * lda) + odd, a);
      if (row >= c + 3) ssp = fma(a, a, ssp);
    }
  }
}

}  // namespace

// Columns per matvec item of 32 rows, by a full warp: of the multiples of the eight reads in
// flight, the one that makes the busiest quarter SM's share smallest, an item's first read
// counted as 16 columns.
__device__ __forceinline__ int zp_chunk(int m, int nrt, int items) {
  const int quarters = 4 * gridDim.x;
  const int chunk = 8 * ((threadIdx.x & 7) + 1), nck = (m + chunk - 1) / chunk;
  const int t = ((nrt * nck + quarters - 1) / quarters) * (chunk + 16);
  const bool ok = nck <= ZP_MAXCK || chunk == 64;
  const int best = (int)__reduce_min_sync(0xffffffffu, ok ? (unsigned)t * 128u + chunk : 0xffffffffu) & 127;
  const int most = (2 * items * quarters + nrt - 1) / nrt;  // items per warp
  return max(best, max((m + most - 1) / most, (m + ZP_MAXCK - 1) / ZP_MAXCK));
}

__global__ void __launch_bounds__(ZP_NT, 1) zpersist_kernel(ZPersistParams P) {
  extern __shared__ __align__(16) double zpsm_raw[];
  zc* vs = reinterpret_cast<zc*>(zpsm_raw);  // v
  __shared__ ZpShared H;
  __shared__ ZRef s_R;
  __shared__ int s_scal, s_chunk;
  const int n = P.n, p = P.p;
  const int64_t lda = P.lda;
  zc* A = P.A;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int nwarps = gridDim.x * ZP_NW;
  const bool lead = blockIdx.x == 0 && tid == 0;
  unsigned round = P.round;
  if (*(volatile unsigned*)(P.sync + 1)) return;  // an earlier panel's wait gave up
  if (lead) P.sync[2] = 0;

  int nss = 0;
  for (int i = 0; i < P.nbp; i++) {
    const int c = p + i, m = n - c - 1, nrt = (m + 31) >> 5;
    // reflector c, identically in every CTA, by warp 0 while the others stage the column
    if (w == 0) {
      if (i > 0) {
        const zc x = ldz(A + (c + 1) + (int64_t)c * lda);
        double ss = 0.0;
        for (int t = lane; t < nss; t += 32) ss += __ldcg(P.sspart + t);
        ss = warp_sum(ss);
        const bool scal = ss_needs_scaling(ss);
        if (lane == 0) s_scal = scal;
        if (!scal) {
          const ZRef R = zp_refl_warp(x, ss);
          if (lane == 0) s_R = R;
        }
      } else if (lane == 0) {
        s_scal = 1;
      }
    } else {
      for (int j = c + tid - 31; j < n; j += ZP_NT - 32) vs[j] = ldz(A + j + (int64_t)c * lda);
      if (w == 1) s_chunk = zp_chunk(m, nrt, P.items_per_warp);
    }
    __syncthreads();
    ZRef R;
    if (s_scal)
      R = zp_refl_from_column(P, c, H.red);
    else
      R = s_R;
    if (lead) {
      P.ev[c] = R.beta;
      P.tau[c] = R.tau;
    }
    const bool zero = zzero(R.tau);
    const int k = zero ? 0 : ((__double2hiint(R.beta) >> 20) & 0x7ff) - 1023;
    const ZpVec V{zero ? zc{0.0, 0.0} : zc{oz_ldexp(R.scale.re, k), oz_ldexp(R.scale.im, k)}, zero ? 0.0 : 1.0};
    for (int j = c + 1 + tid; j < n; j += ZP_NT) {
      const zc x = vs[j];
      if (j > c + 1)
        vs[j] = zero ? zc{0.0, 0.0} : zc{oz_ldexp(x.re, -k), oz_ldexp(x.im, -k)};
      else  // alpha - beta = 1 / scale
        vs[j] = zero ? zc{0.0, 0.0} : zc{oz_ldexp(x.re - R.beta, -k), oz_ldexp(x.im, -k)};
    }
    __syncthreads();
    // ---- A: a static share of the items per warp.  Warps are numbered CTA-minor
    // (consecutive items on different SMs); matvec tile q goes to warp q mod nwarps, panel
    // dot d to warp nwarps - 1 - d mod nwarps.  The CTAs' shares of v^H (A22 v) are summed
    // in a fixed order (deterministic).
    const int chunk = s_chunk;
    const int nck = (m + chunk - 1) / chunk;
    const int nmv = nrt * nck;
    const int gw = w * gridDim.x + blockIdx.x;
    // u1_j = W[:, j]^H v, u2_j = V[:, j]^H v over ZDOT rows from c + 1: eight loads at once
    for (int d = nwarps - 1 - gw; d < i * ((m + ZDOT - 1) / ZDOT); d += nwarps) {
      const int q = d / i, j = d - q * i;
      const int r0 = c + 1 + q * ZDOT + lane;
      const zc* wc = P.W + (size_t)j * n;
      const zc* ac = A + (int64_t)(p + j) * lda;
      zc x[ZDOT / 32], z[ZDOT / 32];
#pragma unroll
      for (int t = 0; t < ZDOT / 32; t++) {
        const int r = r0 + 32 * t;
        x[t] = (r < n) ? ldz(wc + r) : zc{0.0, 0.0};
        z[t] = (r < n) ? ldz(ac + r) : zc{0.0, 0.0};
      }
      zc u1{0.0, 0.0}, u2{0.0, 0.0};
#pragma unroll
      for (int t = 0; t < ZDOT / 32; t++) {
        const int r = r0 + 32 * t;
        const zc v = (r < n) ? vs[r] : zc{0.0, 0.0};
        u1 = zfma(zconj(x[t]), v, u1);
        u2 = zfma(zconj(z[t]), v, u2);
      }
      u1.re = warp_sum(u1.re);
      u1.im = warp_sum(u1.im);
      u2.re = warp_sum(u2.re);
      u2.im = warp_sum(u2.im);
      if (lane == 0) {
        stz(P.u + (size_t)q * 2 * ZBNB + j, u1);
        stz(P.u + (size_t)q * 2 * ZBNB + ZBNB + j, u2);
      }
    }
    zc dl{0.0, 0.0};  // this lane's share of v^H (A22 v)
    for (int qq = gw; qq < nmv; qq += nwarps) {  // partial y = A22 v over (32 rows, column chunk)
      const int rt = qq / nck, ck = qq - rt * nck;
      const int r = c + 1 + rt * 32 + lane;
      const int cb = c + 1 + ck * chunk, ce = min(n, cb + chunk);
      if (r < n) {
        const zc* row = A + r;
        zc a0{0.0, 0.0}, a1{0.0, 0.0}, a2{0.0, 0.0}, a3{0.0, 0.0};
        int j = cb;
        zc x[8], z[8];  // eight reads in flight behind the eight in use
        auto get = [&](zc (&t)[8], int j0) {
#pragma unroll
          for (int u = 0; u < 8; u++) t[u] = ldz(row + (int64_t)(j0 + u) * lda);
        };
        auto add = [&](const zc (&t)[8], int j0) {
          a0 = zfma(t[0], vs[j0], a0);
          a1 = zfma(t[1], vs[j0 + 1], a1);
          a2 = zfma(t[2], vs[j0 + 2], a2);
          a3 = zfma(t[3], vs[j0 + 3], a3);
          a0 = zfma(t[4], vs[j0 + 4], a0);
          a1 = zfma(t[5], vs[j0 + 5], a1);
          a2 = zfma(t[6], vs[j0 + 6], a2);
          a3 = zfma(t[7], vs[j0 + 7], a3);
        };
        if (j + 8 <= ce) get(x, j);
        while (j + 8 <= ce) {
          if (j + 16 <= ce) get(z, j + 8);
          add(x, j);
          j += 8;
          if (j + 8 > ce) break;
          if (j + 16 <= ce) get(x, j + 8);
          add(z, j);
          j += 8;
        }
        for (; j < ce; j++) a0 = zfma(ldz(row + (int64_t)j * lda), vs[j], a0);
        const zc acc = zadd(zadd(a0, a1), zadd(a2, a3));
        stz(P.ypart + (size_t)ck * n + r, acc);
        dl = zadd(dl, zcmul(vs[r], acc));  // conj(v_r) y_r
      }
    }
    {
      const double dr = warp_sum(dl.re), di = warp_sum(dl.im);
      if (lane == 0) {
        H.red[w] = dr;
        H.red[ZP_NW + w] = di;
      }
    }
    auto tree = [](const double* x) { return ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7])); };
    if (!zp_gsync(P, round, [&]() { stz(P.dpart + blockIdx.x, zc{tree(H.red), tree(H.red + ZP_NW)}); })) return;

    // ---- B: rows, as many threads per row as leaves one row block per quarter SM
    const bool last = (i == P.nbp - 1);
    const int quarters = 4 * gridDim.x;
    double ssp;
    if (m <= quarters)
      zp_rows<32>(P, c, i, nck, last, R, V, vs, H, ssp);
    else if (m <= 2 * quarters)
      zp_rows<16>(P, c, i, nck, last, R, V, vs, H, ssp);
    else if (m <= 4 * quarters)
      zp_rows<8>(P, c, i, nck, last, R, V, vs, H, ssp);
    else
      zp_rows<4>(P, c, i, nck, last, R, V, vs, H, ssp);
    if (last) break;
    nss = gridDim.x;
    ssp = warp_sum(ssp);
    if (lane == 0) H.red[w] = ssp;
    if (!zp_gsync(P, round, [&]() { __stcg(P.sspart + blockIdx.x, tree(H.red)); })) return;
  }
}

// ---------------------------------------------------------------------------
// Trailing update: A22 += V W^H - W V^H
// ---------------------------------------------------------------------------
// Largest exponents of the panel's rows of V and of W, and of all of W (grid: rows / 8).
__global__ void __launch_bounds__(256) zp_exps_kernel(ZPersistParams P) {
  const int r = P.p + P.nbp + blockIdx.x * 8 + (threadIdx.x & 7), l = threadIdx.x >> 3;  // 32 columns at once
  __shared__ int sa[32][8], sw[32][8];
  int a = 1, b = 1;
  if (r < P.n && l < P.nbp) {
    const zc v = P.A[r + (int64_t)(P.p + l) * P.lda], x = P.W[(size_t)l * P.n + r];
    a = max(oz_exponent(v.re), oz_exponent(v.im));
    b = max(oz_exponent(x.re), oz_exponent(x.im));
  }
  sa[l][threadIdx.x & 7] = a;
  sw[l][threadIdx.x & 7] = b;
  __syncthreads();
  if (threadIdx.x < 8) {
    for (int t = 1; t < 32; t++) {
      a = max(a, sa[t][threadIdx.x]);
      b = max(b, sw[t][threadIdx.x]);
    }
    if (r < P.n) {
      P.ea[r] = a;
      P.ew[r] = b;
    }
    b = __reduce_max_sync(0xffu, b);
    if (threadIdx.x == 0) atomicMax(P.sync + 2, (unsigned)b);
  }
}

// Real rows 2 r, 2 r + 1 of the result (re, im of row r: neighbours in memory), 2^-k (V W^H -
// W V^H) as four buffers of at most 32 terms, W scaled by 2^-k to the size of V, so that the
// products stay in range for any A:
//   re: vr wr' + vi wi' + wr (-vr') + wi (-vi'),   im: vi wr' + (-vr) wi' + wi (-vr') + (-wr) (-vi').
struct ZpUpdate {
  ZPersistParams P;
  int q, k;
  __device__ int rows() const { return 2 * (P.n - q); }
  __device__ int cols() const { return P.n - q; }
  __device__ int ksteps() const { return 4; }
  __device__ bool contiguousA() const { return false; }
  __device__ bool contiguousB() const { return false; }
  __device__ int exponent(int r) const {
    const int a = P.ea[q + r], b = P.ew[q + r];
    if (a == 2047 || b == 2047) return 2047;
    return min(2046, max(max(a, b - k), 1));
  }
  __device__ int expA(int i) const { return exponent(i >> 1); }
  __device__ int expB(int j) const { return exponent(j); }
  template <int NV>
  __device__ __forceinline__ void load(int r, int part, int l0, bool vside, bool minus, double (&v)[NV]) const {
    const double* src = reinterpret_cast<const double*>(vside ? P.A + q + r + (int64_t)(P.p + l0) * P.lda
                                                              : P.W + (size_t)l0 * P.n + q + r) + part;
    const int64_t ld = 2 * (vside ? P.lda : (int64_t)P.n);
#pragma unroll
    for (int u = 0; u < NV; u++) {
      double x = (l0 + u < P.nbp) ? src[u * ld] : 0.0;
      if (!vside) x = oz_ldexp(x, -k);
      v[u] = minus ? neg(x) : x;
    }
  }
  __device__ void loadA(int i, int s, int l, double (&v)[8]) const {
    load<8>(i >> 1, (i ^ s) & 1, l, s < 2, (i & s & 1) != 0, v);
  }
  __device__ void loadB(int j, int s, int l, double (&v)[4]) const { load<4>(j, s & 1, l, s >= 2, s >= 2, v); }
  __device__ void store(int i, int j, double x) const {
    const int r = i >> 1, part = i & 1;
    if (r < j || (r == j && part == 0)) return;  // the diagonal receives the imaginary part only
    double* a = reinterpret_cast<double*>(P.A + q + r + (int64_t)(q + j) * P.lda) + part;
    const double y = *a + oz_ldexp(x, k);
    *a = y;
    if (r > j) reinterpret_cast<double*>(P.A + q + j + (int64_t)(q + r) * P.lda)[part] = part ? y : neg(y);
  }
  __device__ void timeout() const { P.sync[1] = 1u; }
};

__global__ void __launch_bounds__(OZ_NT, 1) zp_update_kernel(ZPersistParams P, int q) {  // grid: lower 64 x 64 tiles
  extern __shared__ __align__(1024) unsigned char oz_buf[];
  const int t = blockIdx.x;
  int ti = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
  while ((ti + 1) * (ti + 2) / 2 <= t) ti++;
  while (ti * (ti + 1) / 2 > t) ti--;
  const int tj = t - ti * (ti + 1) / 2;
  const int k = max(-1000, min(1000, (int)P.sync[2] - 1023));
  const ZpUpdate U{P, q, k};
  oz_tile(U, ti * OZ_M, tj * OZ_N, oz_buf);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static int zp_maxck(int n) { return std::min(ZP_MAXCK, (n + 7) / 8); }

size_t zhess_persist_ws_doubles(int n) {
  const size_t nn = (size_t)n;
  const size_t maxck = (size_t)zp_maxck(n);
  return 2 * nn * ZBNB                           // W
         + 2 * maxck * nn                        // ypart
         + 2 * ZP_MAXCTAS                        // dpart
         + 4 * ZBNB * ((nn + ZDOT - 1) / ZDOT)   // u
         + ZP_MAXCTAS                            // sspart
         + nn                                    // ea, ew
         + 8;                                    // sync words
}

__global__ void zp_merge_err_kernel(const unsigned* sync, int* info) {
  if (sync[1] && info) *info = SKEW_TIMEOUT;
}

// Reduces columns [0, n - 1 - ZTAILP) in panels and the rest with the one-CTA kernel.
// cudaErrorNotSupported when the device cannot co-schedule the grid or n is outside the
// staged range (the caller then uses the per-column path).
cudaError_t zhess_persistent(double* Ad, int64_t lda, int n, double* taud, double* ev, double* dvim, double* wsd,
                             int sms, int* info, const Tuning& tune, cudaStream_t st) {
  const size_t smem = (size_t)n * sizeof(zc);
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  cudaFuncAttributes fa;
  e = cudaFuncGetAttributes(&fa, zpersist_kernel);
  if (e != cudaSuccess) return e;
  if (smem + fa.sharedSizeBytes > (size_t)optin || n <= ZTAILP + 2) return cudaErrorNotSupported;
  e = cudaFuncSetAttribute(zpersist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  static std::atomic<uint64_t> raised{0};
  if ((e = raise_smem_limit_once((const void*)zp_update_kernel, raised))) return e;
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, zpersist_kernel, ZP_NT, smem);
  if (e != cudaSuccess) return e;
  if (occ < 1) return cudaErrorNotSupported;
  int grid = sms;
  if (tune.zpersist_ctas > 0) grid = std::max(1, std::min(sms * occ, tune.zpersist_ctas));
  grid = std::min(grid, ZP_MAXCTAS);
  zc* A = reinterpret_cast<zc*>(Ad);
  zc* tau = reinterpret_cast<zc*>(taud);
  ZPersistParams P;
  P.A = A;
  P.lda = lda;
  P.n = n;
  P.tau = tau;
  P.ev = ev;
  const size_t nn = (size_t)n, maxck = (size_t)zp_maxck(n);
  double* wp = wsd;
  P.W = reinterpret_cast<zc*>(wp);
  wp += 2 * nn * ZBNB;
  P.ypart = reinterpret_cast<zc*>(wp);
  wp += 2 * maxck * nn;
  P.dpart = reinterpret_cast<zc*>(wp);
  wp += 2 * ZP_MAXCTAS;
  P.u = reinterpret_cast<zc*>(wp);
  wp += 4 * ZBNB * ((nn + ZDOT - 1) / ZDOT);
  P.sspart = wp;
  wp += ZP_MAXCTAS;
  P.ea = reinterpret_cast<int*>(wp);
  P.ew = P.ea + n;
  wp += nn;
  P.sync = reinterpret_cast<unsigned*>(wp);
  P.items_per_warp = std::max(1, std::min(8, tune.zpersist_items));
  P.poll_limit = tune.wait_polls > 0 ? tune.wait_polls : ZP_POLL;
  P.skip_cta = tune.wait_skip_cta;
  e = cudaMemsetAsync(wp, 0, 4 * sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  const int nb = std::max(4, std::min(ZBNB, tune.zpersist_nb)), pend = n - 1 - ZTAILP;
  P.round = 0;
  for (int p = 0; p < pend; p += nb) {
    P.p = p;
    P.nbp = std::min(nb, pend - p);
    void* args[] = {&P};
    e = cudaLaunchCooperativeKernel((const void*)zpersist_kernel, dim3(grid), dim3(ZP_NT), args, smem, st);
    if (e != cudaSuccess) return p == 0 ? e : cudaErrorUnknown;
    P.round += 2 * P.nbp - 1;
    const int q = p + P.nbp, mt = (n - q + OZ_N - 1) / OZ_N;
    zp_exps_kernel<<<(n - q + 7) / 8, 256, 0, st>>>(P);
    zp_update_kernel<<<mt * (mt + 1) / 2, OZ_NT, OZ_SMEM, st>>>(P, q);
    if ((e = cudaGetLastError())) return e;
  }
  // tail: the trailing block with the one-CTA kernel, in place
  ZHessParams T;
  T.W = reinterpret_cast<double*>(A + pend + (int64_t)pend * lda);
  T.stride = 0;
  T.ld = lda;
  T.n = n - pend;
  T.count = 1;
  T.tau = reinterpret_cast<double*>(tau + pend);
  T.ev = ev + pend;
  T.dvim = nullptr;
  e = launch_zhess_cta(T, st);
  if (e != cudaSuccess) return e;
  e = launch_zdiag_im(Ad, lda, n, dvim, st);
  if (e != cudaSuccess) return e;
  zp_merge_err_kernel<<<1, 1, 0, st>>>(P.sync, info);
  return cudaGetLastError();
}

}  // namespace skew
