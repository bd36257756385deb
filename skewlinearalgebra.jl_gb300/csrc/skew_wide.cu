// Blocked Householder tridiagonalisation of one real skew matrix with n > 640 (the
// skewblockedhess! / skewlatrd! structure of hessenberg.jl:92-173), with the two O(n^3)
// parts off the FP64 pipe.
//
// The latrd product y = A22 v and the trailing update are 2/3 n^3 flops each; on the FP64
// pipe (2 FMAs per clock and SM) they took 0.45 and 0.30 of the 0.93 s at n = 8192.
//   * A22 of a panel is copied once per panel into 64 x 64 tiles of its lower triangle in
//     fixed point: 56 bits relative to the tile's largest entry, as two 28-bit integers
//     (8 bytes an entry, a tile in one piece).  A tile gives both A v and, transposed, its
//     mirror image's share; a multiply-add of two 56-bit numbers is three IMAD.WIDE, of
//     which an SM does 64 per clock, so the product is bound by reading half the matrix.
//   * The trailing update V W^T - W V^T runs on the tensor cores (skew_oz.cuh).
// Per panel of nb columns: fxp_pack_kernel, fxp_panel_kernel (one cooperative launch, two
// grid barriers per column), fxp_exps_kernel, fxp_update_kernel.  The last columns go to the
// one-CTA kernel of skew_batch.cu.  Sums of the tiles are formed in a fixed order.
//
// Whole reduction: n = 2048 51.0 -> 35.4 ms, 8192 929 -> 335 (panels 284, update 43,
// packing 5).
//
// Eigenvalues in the QR's deflation order (n <= 1024) keep the kernels of skew_blocked.cu
// and skew_cluster.cu: the order depends on the last bits of the tridiagonal.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "skew_internal.h"
#include "skew_common.cuh"
#include "skew_oz.cuh"

namespace skew {

constexpr int FXP_T = 64;                     // tile edge
constexpr int FXP_TILE = FXP_T * FXP_T;       // entries (int2) of a tile
constexpr int FXP_NT = 256, FXP_NW = FXP_NT / 32;
constexpr int FXP_NB = 64;                    // widest panel
constexpr int FXP_TAIL = 128;                 // columns left to the one-CTA kernel
constexpr int FXP_SLOTS = 3;                  // quarter tiles in flight per warp
constexpr int FXP_QUARTER = FXP_TILE / 4 * 8; // bytes
constexpr int FXP_DOT_ROWS = 256;             // rows and columns of a panel dot item: 8 x 4 FMAs per lane
constexpr int FXP_DOT_COLS = 4;
constexpr int FXP_CTAS = 1024;                // largest grid of the panel kernel
// shared memory: quarter tiles, x of a tile's rows and columns per warp, barriers
constexpr int FXP_SMEM = FXP_NW * (FXP_SLOTS * FXP_QUARTER + 2 * FXP_T * 8 + FXP_SLOTS * 8);
constexpr long long FXP_POLLS = 1LL << 24;    // default polls of a grid barrier: seconds

// (h, l) with x = 2^(e - 1078) (h 2^28 + l), rounded; |h| <= 2^28, -2^27 <= l < 2^27
__device__ __forceinline__ int2 fxp_split(double x, int e) {
  const long long v = (long long)(oz_fixed(x, e) - OZ_BIAS) + (1LL << 27);
  return make_int2((int)(v >> 28), (int)(v & ((1 << 28) - 1)) - (1 << 27));
}

// Position of entry (r, c) of a tile: quarters of 16 columns; lane 4 (r / 8) + (c % 16) / 4
// holds 8 x 4 entries, stored pairwise so that the 32 lanes' 16-byte loads are contiguous.
__device__ __forceinline__ int fxp_pos(int r, int c) {
  const int q = c >> 4, lane = 4 * (r >> 3) + ((c & 15) >> 2), step = 2 * (r & 7) + ((c & 3) >> 1);
  return ((q * 16 + step) * 32 + lane) * 2 + (c & 1);
}

struct FxpWs {
  int2* pack;       // lower tiles, column by column of tiles
  int* etile;       // their largest exponents
  double* W;        // n x FXP_NB
  double* rowpart;  // tile columns x n: shares of A22 v from tiles right of (and on) the diagonal
  double* colpart;  // slots x n: shares of the mirrored tiles
  double* upart;    // row chunks x 2 FXP_NB
  double* sspart;   // one per CTA
  int *ev, *ew;     // largest exponents of the panel's rows of V and W
  unsigned* sync;   // [0] barrier arrivals, [1] error, [2] W's largest exponent
};

static int fxp_tiles(int n) { return (n - 1 + FXP_T - 1) / FXP_T; }
static size_t fxp_even(size_t d) { return (d + 1) & ~(size_t)1; }  // 16-byte alignment

static size_t fxp_carve(FxpWs* w, double* base, int n) {
  const size_t T = fxp_tiles(n), nt = T * (T + 1) / 2;
  double* p = base;
  auto take = [&](size_t d) {
    double* r = p;
    p += fxp_even(d);
    return r;
  };
  FxpWs x;
  x.pack = (int2*)take(nt * FXP_TILE);
  x.etile = (int*)take((nt + 1) / 2);
  x.W = take((size_t)n * FXP_NB);
  x.rowpart = take(T * n);
  x.colpart = take((T + 2) * n);
  x.upart = take(((size_t)n / FXP_DOT_ROWS + 1) * 2 * FXP_NB);
  x.sspart = take(FXP_CTAS);
  x.ev = (int*)take((size_t)n / 2 + 1);
  x.ew = (int*)take((size_t)n / 2 + 1);
  x.sync = (unsigned*)take(4);
  if (w) *w = x;
  return p - base;
}
size_t wide_ws_doubles(int n) { return n > kWideMin ? fxp_carve(nullptr, nullptr, n) + 2 : 0; }

// ---------------------------------------------------------------------------
// A22 (rows and columns from s0) into tiles; one CTA per lower tile
// ---------------------------------------------------------------------------
// index of tile (ti, tj), ti >= tj, of T x T lower tiles, column by column
__host__ __device__ __forceinline__ int fxp_first(int T, int tj) { return tj * T - tj * (tj - 1) / 2; }

__device__ __forceinline__ void fxp_tile_at(int T, int t, int* ti, int* tj) {
  int j = (int)(T + 0.5f - sqrtf((T + 0.5f) * (T + 0.5f) - 2.0f * t));  // corrected below
  j = max(0, min(T - 1, j));
  while (j > 0 && fxp_first(T, j) > t) j--;
  while (j + 1 < T && fxp_first(T, j + 1) <= t) j++;
  *tj = j;
  *ti = j + (t - fxp_first(T, j));
}

__global__ void __launch_bounds__(256) fxp_pack_kernel(const double* __restrict__ A, int64_t lda, int n, int s0, int T,
                                                       int2* __restrict__ pack, int* __restrict__ etile) {
  __shared__ int2 out[FXP_TILE];
  __shared__ int red[8];
  int ti, tj;
  fxp_tile_at(T, blockIdx.x, &ti, &tj);
  const int r0 = s0 + ti * FXP_T, c0 = s0 + tj * FXP_T;
  const int rr = threadIdx.x & 63, cg = threadIdx.x >> 6;  // a row, every fourth column
  const int row = r0 + rr;
  double v[16];
  int e = 1;
#pragma unroll
  for (int u = 0; u < 16; u++) {
    const int col = c0 + cg + 4 * u;
    v[u] = (row < n && col < row) ? A[row + (int64_t)col * lda] : 0.0;  // col < row < n: strictly below the diagonal
    e = max(e, oz_exponent(v[u]));
  }
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; q++) e = max(e, red[q]);
#pragma unroll
  for (int u = 0; u < 16; u++) out[fxp_pos(rr, cg + 4 * u)] = fxp_split(v[u], e);
  __syncthreads();
  int4* dst = reinterpret_cast<int4*>(pack + (size_t)blockIdx.x * FXP_TILE);
  const int4* src = reinterpret_cast<const int4*>(out);
#pragma unroll
  for (int q = 0; q < FXP_TILE / 2 / 256; q++) dst[threadIdx.x + 256 * q] = src[threadIdx.x + 256 * q];
  if (threadIdx.x == 0) etile[blockIdx.x] = e;
}

// ---------------------------------------------------------------------------
// One panel: columns p .. p + nbp - 1
// ---------------------------------------------------------------------------
struct FxpPanel {
  double* A;
  int64_t lda;
  int n, p, nbp;
  int T, per;  // tiles per edge of A22 from row p + 1; tiles per warp
  double* tau;
  double* evals;
  FxpWs w;
  long long poll_limit;
  int skip_cta;
};

// Grid barrier on a monotonic arrival counter; false if it gave up or an error was set
// before it.  pre() is run by thread 0 between the CTA's own barrier and its arrival.
template <class Pre>
__device__ bool fxp_barrier(const FxpPanel& P, unsigned& round, Pre pre) {
  __shared__ int s_ok;
  __syncthreads();
  round++;
  if (threadIdx.x == 0) {
    const unsigned target = round * gridDim.x;
    int ok = 1;
    unsigned* cnt = P.w.sync;
    volatile unsigned* err = P.w.sync + 1;
    if ((int)blockIdx.x == P.skip_cta) {  // never arrives: the others' waits run out
      long long it = 0;
      while (!*err && ++it <= P.poll_limit) __nanosleep(100);
      ok = 0;
    } else {
      pre();
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(cnt) : "memory");
      const unsigned before = *err;  // looked at after the wait, which hides the read
      long long it = 0;
      for (;;) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(cnt) : "memory");
        if ((int)(v - target) >= 0) break;
        if ((++it & 15) == 0 && *err) {
          ok = 0;
          break;
        }
        if (it > P.poll_limit) {
          atomicExch(P.w.sync + 1, 1u);
          ok = 0;
          break;
        }
      }
      ok = ok && !before;
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

struct FxpRefl {
  double beta, tau, scale;
};

// Reflector of column c from its entries, by the whole CTA.
__device__ FxpRefl fxp_reflector(const FxpPanel& P, int c, double* red) {
  const double* col = P.A + (int64_t)c * P.lda;
  double part = 0.0;
  for (int r = c + 2 + threadIdx.x; r < P.n; r += FXP_NT) {
    const double x = __ldcg(col + r);
    part = fma(x, x, part);
  }
  const double ss = block_sum<FXP_NW>(part, red);
  double xn = -1.0;
  if (ss_needs_scaling(ss)) {
    double mx = 0.0;
    for (int r = c + 2 + threadIdx.x; r < P.n; r += FXP_NT) mx = fmax(mx, fabs(__ldcg(col + r)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    __shared__ double rm[FXP_NW];
    if ((threadIdx.x & 31) == 0) rm[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = 0.0;
    for (int q = 0; q < FXP_NW; q++) mx = fmax(mx, rm[q]);
    double qq = 0.0;
    if (mx > 0.0)
      for (int r = c + 2 + threadIdx.x; r < P.n; r += FXP_NT) {
        const double x = __ldcg(col + r) / mx;
        qq = fma(x, x, qq);
      }
    qq = block_sum<FXP_NW>(qq, red);
    xn = mx * sqrt(qq);
  }
  __shared__ FxpRefl s_R;
  if (threadIdx.x == 0) {
    const Reflector R = make_reflector(__ldcg(col + c + 1), ss, xn);
    s_R = FxpRefl{R.beta, R.tau, R.scale};
  }
  __syncthreads();
  const FxpRefl R = s_R;
  __syncthreads();
  return R;
}

// A warp's tiles: a run of per tiles in the column-by-column order, in quarters through
// FXP_SLOTS buffers filled by bulk copies.  The copies of the next column's first quarters
// are issued before the grid barriers.
struct FxpStream {
  const char* src;   // the run
  uint32_t buf, bar; // shared addresses of this warp's buffers and barriers
  int quarters;      // of the run
  unsigned issued;   // quarters requested so far, over all columns
  __device__ __forceinline__ void request(int q) {  // lane 0: quarter q of the run into the next slot
    const uint32_t s = issued % FXP_SLOTS, b = bar + 8 * s;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(FXP_QUARTER) : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            buf + s * FXP_QUARTER),
        "l"(src + (size_t)q * FXP_QUARTER), "r"(FXP_QUARTER), "r"(b)
        : "memory");
  }
};

// x of the 64 rows from r0, two per lane: zero up to row c + 1 and past n
__device__ __forceinline__ double2 fxp_entries(const double* col, int n, int c, int r0) {
  const int r = r0 + 2 * (threadIdx.x & 31);
  return make_double2((r > c + 1 && r < n) ? __ldcg(col + r) : 0.0,
                      (r + 1 > c + 1 && r + 1 < n) ? __ldcg(col + r + 1) : 0.0);
}
// in fixed point into xs; returns the largest exponent
__device__ __forceinline__ int fxp_vector(double2 x, int2* xs) {
  const int lane = threadIdx.x & 31;
  const int e = __reduce_max_sync(0xffffffffu, max(oz_exponent(x.x), oz_exponent(x.y)));
  __syncwarp();
  xs[2 * lane] = fxp_split(x.x, e);
  xs[2 * lane + 1] = fxp_split(x.y, e);
  __syncwarp();
  return e;
}

__device__ __forceinline__ long long fxp_shfl_xor(long long v, int o) {
  return (long long)__shfl_xor_sync(0xffffffffu, (unsigned long long)v, o);
}

// S 2^(ea + ex - 2100 + k), NaN where an exponent says that its entries are not finite
__device__ __forceinline__ double fxp_double(long long s, int ea, int ex, int k) {
  if (ea == 2047 || ex == 2047) return __longlong_as_double(0x7ff8000000000000LL);
  return oz_double(s, ea + ex - 2100 + k);
}

// rowpart and colpart of this warp's tiles: (A22 x) 2^k for x = column c below row c + 1.
__device__ __forceinline__ bool fxp_matvec(const FxpPanel& P, FxpStream& S, int c, int t0, int t1, int k, bool more,
                                           const int2* buf, int2* xrow, int2* xcol) {
  const int lane = threadIdx.x & 31, a = lane >> 2, b = lane & 3;
  const int n = P.n, s0 = P.p + 1;
  const double* col = P.A + (int64_t)c * P.lda;
  if (t0 >= t1) return true;
  int ti, tj;
  fxp_tile_at(P.T, t0, &ti, &tj);
  double2 xc = fxp_entries(col, n, c, s0 + tj * FXP_T), xr = fxp_entries(col, n, c, s0 + ti * FXP_T);
  int ecol = fxp_vector(xc, xcol);
  double cacc[2] = {0.0, 0.0};  // mirrored sums of two columns
  const unsigned first = S.issued - min(S.quarters, FXP_SLOTS);  // quarter 0 of this column
  int q = 0;
  for (int t = t0; t < t1; t++) {
    const int et = P.w.etile[t];
    const int erow = fxp_vector(xr, xrow);
    if (t + 1 < t1) {  // the next tile's rows (and columns, where it starts a column of tiles)
      const bool turn = ti + 1 == P.T;
      xr = fxp_entries(col, n, c, s0 + (turn ? tj + 1 : ti + 1) * FXP_T);
      if (turn) xc = xr;  // a column of tiles starts on the diagonal
    }
    int rx[8], ry[8];
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const int2 v = xrow[8 * a + r];
      rx[r] = v.x;
      ry[r] = v.y;
    }
    long long rh[8], rm[8], cs[16];
#pragma unroll
    for (int r = 0; r < 8; r++) {
      rh[r] = 0;
      rm[r] = 0;
    }
#pragma unroll
    for (int qd = 0; qd < 4; qd++, q++) {
      const unsigned at = first + q;
      const bool got = oz_wait(S.bar + 8 * (at % FXP_SLOTS), (at / FXP_SLOTS) & 1);
      const int4* src = reinterpret_cast<const int4*>(buf) + (at % FXP_SLOTS) * (FXP_TILE / 4 / 2) + lane;
      int cx[4], cy[4];
      long long ch[4], cm[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int2 v = xcol[16 * qd + 4 * b + j];
        cx[j] = v.x;
        cy[j] = v.y;
        ch[j] = 0;
        cm[j] = 0;
      }
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const int4 u = src[(2 * r) * 32], v = src[(2 * r + 1) * 32];
        const int h[4] = {u.x, u.z, v.x, v.z}, l[4] = {u.y, u.w, v.y, v.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
          rh[r] += (long long)h[j] * cx[j];
          rm[r] += (long long)h[j] * cy[j];
          rm[r] += (long long)l[j] * cx[j];
          ch[j] += (long long)h[j] * rx[r];
          cm[j] += (long long)h[j] * ry[r];
          cm[j] += (long long)l[j] * rx[r];
        }
      }
      __syncwarp();
      if (!__all_sync(0xffffffffu, got)) return false;  // the whole warp, if one lane's wait gave up
      const bool want = q + FXP_SLOTS < S.quarters || more;  // the next column starts over
      if (want) {
        if (lane == 0) S.request((q + FXP_SLOTS) % S.quarters);
        S.issued++;
      }
#pragma unroll
      for (int j = 0; j < 4; j++) cs[4 * qd + j] = ch[j] + ((cm[j] + (1 << 27)) >> 28);
    }
    // the mirrored tile: sums over the 64 rows (8 lanes), halving the columns a lane keeps
    {
      const bool u16 = lane & 16, u8 = lane & 8, u4 = lane & 4;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const long long got = fxp_shfl_xor(u16 ? cs[j] : cs[j + 8], 16);
        cs[j] = (u16 ? cs[j + 8] : cs[j]) + got;
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const long long got = fxp_shfl_xor(u8 ? cs[j] : cs[j + 4], 8);
        cs[j] = (u8 ? cs[j + 4] : cs[j]) + got;
      }
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const long long got = fxp_shfl_xor(u4 ? cs[j] : cs[j + 2], 4);
        cs[j] = (u4 ? cs[j + 2] : cs[j]) + got;
      }
      cacc[0] += fxp_double(cs[0], et, erow, k);  // index 8 u16 + 4 u8 + 2 u4 of 16: quarter 2 u16 + u8,
      cacc[1] += fxp_double(cs[1], et, erow, k);  // column 4 b + 2 u4 (+ 1) of it
    }
    // rows: sums over the 64 columns, two rows per lane
#pragma unroll
    for (int r = 0; r < 8; r++) rh[r] += (rm[r] + (1 << 27)) >> 28;
    const bool u1 = lane & 1, u2 = lane & 2;
    long long s4[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const long long got = fxp_shfl_xor(u1 ? rh[r] : rh[r + 4], 1);
      s4[r] = (u1 ? rh[r + 4] : rh[r]) + got;
    }
    long long s2[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const long long got = fxp_shfl_xor(u2 ? s4[r] : s4[r + 2], 2);
      s2[r] = (u2 ? s4[r + 2] : s4[r]) + got;
    }
    const int row = s0 + ti * FXP_T + 8 * a + (u1 ? 4 : 0) + (u2 ? 2 : 0);
    double* out = P.w.rowpart + (size_t)tj * n;
    if (row < n) out[row] = fxp_double(s2[0], et, ecol, k);
    if (row + 1 < n) out[row + 1] = fxp_double(s2[1], et, ecol, k);
    ti++;
    if (ti == P.T || t + 1 == t1) {  // the column of tiles ends: its share of the mirrored sums
      const int slot = blockIdx.x * FXP_NW + (threadIdx.x >> 5) - fxp_first(P.T, tj) / P.per;
      const int cc = s0 + tj * FXP_T + 16 * ((lane >> 3) & 3) + 4 * b + ((lane & 4) ? 2 : 0);
      if (cc < n) P.w.colpart[(size_t)slot * n + cc] = cacc[0];
      if (cc + 1 < n) P.w.colpart[(size_t)slot * n + cc + 1] = cacc[1];
      cacc[0] = cacc[1] = 0.0;
      if (ti == P.T) {
        tj++;
        ti = tj;
        if (t + 1 < t1) ecol = fxp_vector(xc, xcol);
      }
    }
  }
  return true;
}

// Panel dots: item (chunk of rows, group of the 2 i columns W_0 .. W_{i-1}, A_p .. A_{c-1})
// against v = x scale with v[c + 1] = 1.
__device__ __forceinline__ void fxp_dots(const FxpPanel& P, int c, int i, int item, int groups, double scale,
                                         bool zero) {
  constexpr int NR = FXP_DOT_ROWS / 32;
  const int lane = threadIdx.x & 31, n = P.n;
  const int chunk = item / groups, g = item - chunk * groups;
  const double* col = P.A + (int64_t)c * P.lda;
  const int r0 = c + 1 + chunk * FXP_DOT_ROWS + lane;
  double a[FXP_DOT_COLS][NR];
#pragma unroll
  for (int j = 0; j < FXP_DOT_COLS; j++) {
    const int d = g * FXP_DOT_COLS + j;
    const double* q = d < i ? P.w.W + (size_t)d * n : P.A + (int64_t)(P.p + d - i) * P.lda;
#pragma unroll
    for (int u = 0; u < NR; u++) a[j][u] = (d < 2 * i && r0 + 32 * u < n) ? __ldcg(q + r0 + 32 * u) : 0.0;
  }
  double s[FXP_DOT_COLS] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int u = 0; u < NR; u++) {
    const int r = r0 + 32 * u;
    const double v = (r < n && !zero) ? (r == c + 1 ? 1.0 : __ldcg(col + r) * scale) : 0.0;
#pragma unroll
    for (int j = 0; j < FXP_DOT_COLS; j++) s[j] = fma(a[j][u], v, s[j]);
  }
  // sums over the lanes, transposed: lanes 8 j .. 8 j + 7 end with column j's
  static_assert(FXP_DOT_COLS == 4, "two halving steps");
#pragma unroll
  for (int o = 16, w = 2; w >= 1; o >>= 1, w >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < w; j++) {
      const double send = up ? s[j] : s[j + w];
      const double keep = up ? s[j + w] : s[j];
      s[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (int o = 4; o >= 1; o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
  const int d = g * FXP_DOT_COLS + (lane >> 3);
  if (!(lane & 7) && d < 2 * i) P.w.upart[(size_t)chunk * 2 * FXP_NB + (d < i ? d : FXP_NB + d - i)] = s[0];
}

// y of one row 2^k (partial sums of the tiles), TPR threads per row: thread g's share, eight
// reads at a time
template <int TPR>
__device__ __forceinline__ double fxp_row_sum(const FxpPanel& P, int row, int g) {
  const int n = P.n, tr = (row - P.p - 1) / FXP_T;
  const int f = fxp_first(P.T, tr), slots = (f + P.T - tr - 1) / P.per - f / P.per + 1;
  double y[2] = {0.0, 0.0};
  for (int q = g; q <= tr; q += 8 * TPR) {
    double t[8];
#pragma unroll
    for (int z = 0; z < 8; z++) t[z] = (q + z * TPR <= tr) ? __ldcg(P.w.rowpart + (size_t)(q + z * TPR) * n + row) : 0.0;
#pragma unroll
    for (int z = 0; z < 8; z++)
      if (q + z * TPR <= tr) y[z & 1] += t[z];
  }
  for (int q = g; q < slots; q += 4 * TPR) {
    double t[4];
#pragma unroll
    for (int z = 0; z < 4; z++) t[z] = (q + z * TPR < slots) ? __ldcg(P.w.colpart + (size_t)(q + z * TPR) * n + row) : 0.0;
#pragma unroll
    for (int z = 0; z < 4; z++)
      if (q + z * TPR < slots) y[1] -= t[z];
  }
  return y[0] + y[1];
}

// What the rows of a step share: sums of the panel dots (u1, u2) and row c + 1 of W and A.
struct FxpShared {
  double su[2 * FXP_NB];
  double Wrow[FXP_NB + 1], Arow[FXP_NB + 1];
  double red[FXP_NW];
};

// What a thread reads for it: two threads per dot, even and odd chunks; the last warp, which
// has the fewest rows, also row c + 1.
struct FxpHead {
  double up[8], w[2], a[2];
};
__device__ __forceinline__ void fxp_head_load(const FxpPanel& P, int c, int i, int chunks, FxpHead& L) {
  const int tid = threadIdx.x, lane = tid & 31, n = P.n, r0 = c + 1;
  const int d = tid >> 1, h = tid & 1;
  const bool in = (d & (FXP_NB - 1)) < i;
#pragma unroll
  for (int z = 0; z < 8; z++)
    L.up[z] = (in && h + 2 * z < chunks) ? __ldcg(P.w.upart + (size_t)(h + 2 * z) * 2 * FXP_NB + d) : 0.0;
#pragma unroll
  for (int t = 0; t < 2; t++) {
    const int j = lane + 32 * t;
    L.w[t] = L.a[t] = 0.0;
    if (tid >= FXP_NT - 32 && j < i) {
      L.w[t] = __ldcg(P.w.W + (size_t)j * n + r0);
      L.a[t] = __ldcg(P.A + r0 + (int64_t)(P.p + j) * P.lda);
    }
  }
}

// Fills it, by the whole CTA.  m2 = scale 2^-k.
__device__ __forceinline__ void fxp_step_shared(const FxpPanel& P, int c, int i, int chunks, const FxpRefl& R,
                                                double m2, const FxpHead& L, FxpShared& H) {
  const int tid = threadIdx.x, lane = tid & 31, r0 = c + 1;
  const int d = tid >> 1, h = tid & 1;
  double s0 = 0.0, s1 = 0.0;
  if ((d & (FXP_NB - 1)) < i) {
#pragma unroll
    for (int z = 0; z < 8; z++)
      if (h + 2 * z < chunks) (z & 1 ? s1 : s0) += L.up[z];
    for (int q = h + 16; q < chunks; q += 16) {
      double t[8];
#pragma unroll
      for (int z = 0; z < 8; z++)
        t[z] = (q + 2 * z < chunks) ? __ldcg(P.w.upart + (size_t)(q + 2 * z) * 2 * FXP_NB + d) : 0.0;
#pragma unroll
      for (int z = 0; z < 8; z++)
        if (q + 2 * z < chunks) (z & 1 ? s1 : s0) += t[z];
    }
    s0 += s1;
  }
  s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
  if (!h) H.su[d] = s0;
  const bool head = tid >= FXP_NT - 32;
  double acc = head ? fxp_row_sum<32>(P, r0, lane) : 0.0;
  __syncthreads();
  if (head) {  // row c + 1 of W, which every row's column update needs
    acc *= m2;
#pragma unroll
    for (int t = 0; t < 2; t++) {
      const int j = lane + 32 * t;
      if (j < i) {
        acc = fma(L.a[t], H.su[j], fma(-L.w[t], H.su[FXP_NB + j], acc));
        H.Wrow[j] = L.w[t];
        H.Arow[j] = L.a[t];
      }
    }
    acc = warp_sum(acc);
    if (lane == 0) {
      H.Wrow[i] = (R.tau == 0.0) ? 0.0 : R.tau * acc;
      H.Arow[i] = (R.tau == 0.0) ? 0.0 : 1.0;
    }
  }
  __syncthreads();
}

// Rows of the panel step: W[:, i], v into column c, the deferred update of column c + 1 and
// the sum of squares of its rows below the subdiagonal (ssp: this thread's share).  Row blocks
// go to the warps CTA-minor, so that TPR chosen for one block per quarter SM spreads the FP64
// work evenly.  A block's loads go out before the shared sums are formed.
template <int TPR>
__device__ void fxp_rows(const FxpPanel& P, int c, int i, int chunks, bool last, const FxpRefl& R, double m2,
                         FxpShared& H, double& ssp) {
  constexpr int RPW = 32 / TPR, NJ = FXP_NB / TPR;
  double* A = P.A;
  const int64_t lda = P.lda;
  const int lane = threadIdx.x & 31, n = P.n, p = P.p, g = lane % TPR;
  const int nrb = (n - c - 1 + RPW - 1) / RPW;
  const int rb0 = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  double aj[NJ], wj[NJ], vr, y, next;  // next: column c + 1 as it was at the panel's start
  auto load = [&](int rb) {
    const int row = c + 1 + rb * RPW + lane / TPR;
    const bool valid = rb < nrb && row < n;
#pragma unroll
    for (int t = 0; t < NJ; t++) {
      const int j = g + TPR * t;
      aj[t] = 0.0;
      wj[t] = 0.0;
      if (valid && j < i) {
        aj[t] = __ldcg(A + row + (int64_t)(p + j) * lda);
        wj[t] = __ldcg(P.w.W + (size_t)j * n + row);
      }
    }
    vr = y = next = 0.0;
    if (valid) {
      next = (row >= c + 2) ? __ldcg(A + row + (int64_t)(c + 1) * lda) : 0.0;
      vr = (R.tau == 0.0 || row == c + 1) ? 0.0 : __ldcg(A + row + (int64_t)c * lda);
      y = fxp_row_sum<TPR>(P, row, g);
    }
  };
  FxpHead L;
  fxp_head_load(P, c, i, chunks, L);
  load(rb0);
  fxp_step_shared(P, c, i, chunks, R, m2, L, H);
  ssp = 0.0;
  for (int rb = rb0; rb < nrb; rb += gridDim.x * FXP_NW) {
    if (rb != rb0) load(rb);
    const int row = c + 1 + rb * RPW + lane / TPR;
    const bool valid = row < n;
    double acc = y * m2, acc1 = (g == 0) ? next : 0.0;  // v[c + 1] = 1
#pragma unroll
    for (int t = 0; t < NJ; t++) {
      const int j = g + TPR * t;
      if (j < i) {
        acc = fma(aj[t], H.su[j], acc);
        acc1 = fma(-wj[t], H.su[FXP_NB + j], acc1);
      }
    }
    acc += acc1;
#pragma unroll
    for (int o = 1; o < TPR; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    double wri = (R.tau == 0.0) ? 0.0 : R.tau * acc;
    if (row == c + 1) wri = H.Wrow[i];
    vr = (R.tau == 0.0) ? 0.0 : (row == c + 1 ? 1.0 : vr * R.scale);
    if (valid && g == 0) {
      P.w.W[(size_t)i * n + row] = wri;
      A[row + (int64_t)c * lda] = vr;
    }
    if (last) continue;
    double uu = 0.0, uu1 = 0.0;
#pragma unroll
    for (int t = 0; t < NJ; t++) {
      const int j = g + TPR * t;
      if (j < i) {
        uu = fma(aj[t], H.Wrow[j], uu);
        uu1 = fma(-wj[t], H.Arow[j], uu1);
      }
    }
    if (i % TPR == g) uu = fma(vr, H.Wrow[i], fma(-wri, H.Arow[i], uu));
    uu += uu1;
#pragma unroll
    for (int o = 1; o < TPR; o <<= 1) uu += __shfl_xor_sync(0xffffffffu, uu, o);
    if (valid && row >= c + 2 && g == 0) {
      const double anew = next + uu;
      A[row + (int64_t)(c + 1) * lda] = anew;
      if (row >= c + 3) ssp = fma(anew, anew, ssp);
    }
  }
}

// n = 8192, first panel, per column: the product 44 us (268 MB, 6.1 TB/s; 115 us on the
// FP64 pipe from the full square), rows 15, the two barriers' waits 12, the next reflector 3; at
// m = 3072, where the tiles stay in L2, 7, 8, 8 and 3.  Loads in batches before the sums that
// wait for them and row blocks dealt to the warps of all CTAs took rows and the wait behind
// them from 24 to 18 us (from 14 to 11 at m = 3072).  At small m the product is the latency of
// one tile (7 us): its 768 IMADs per warp take 3, the rest is reading x, shuffles, conversions.
__global__ void __launch_bounds__(FXP_NT, 1) fxp_panel_kernel(FxpPanel P) {
  extern __shared__ __align__(128) unsigned char fsm[];
  __shared__ double red[FXP_NW];
  __shared__ FxpShared H;
  __shared__ int s_scal;
  __shared__ FxpRefl s_R;
  const int n = P.n, p = P.p;
  const int64_t lda = P.lda;
  double* A = P.A;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int nwarps = gridDim.x * FXP_NW, gw = blockIdx.x * FXP_NW + w;
  const int ntiles = P.T * (P.T + 1) / 2;
  const int t0 = min(ntiles, gw * P.per), t1 = min(ntiles, t0 + P.per);
  int2* buf = reinterpret_cast<int2*>(fsm + (size_t)w * FXP_SLOTS * FXP_QUARTER);
  int2* xrow = reinterpret_cast<int2*>(fsm + (size_t)FXP_NW * FXP_SLOTS * FXP_QUARTER) + w * 2 * FXP_T;
  int2* xcol = xrow + FXP_T;
  uint64_t* bars = reinterpret_cast<uint64_t*>(fsm + (size_t)FXP_NW * (FXP_SLOTS * FXP_QUARTER + 2 * FXP_T * 8)) +
                   w * FXP_SLOTS;
  FxpStream S;
  S.src = reinterpret_cast<const char*>(P.w.pack + (size_t)t0 * FXP_TILE);
  S.buf = oz_smem(buf);
  S.bar = oz_smem(bars);
  S.quarters = 4 * (t1 - t0);
  S.issued = 0;
  if (lane == 0) {
    for (int q = 0; q < FXP_SLOTS; q++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(S.bar + 8 * q) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  for (int q = 0; q < min(S.quarters, FXP_SLOTS); q++) {
    if (lane == 0) S.request(q);
    S.issued++;
  }
  unsigned round = 0;
  FxpRefl R = fxp_reflector(P, p, red);
  if (blockIdx.x == 0 && tid == 0) {
    P.evals[p] = R.beta;
    P.tau[p] = R.tau;
  }
  for (int i = 0; i < P.nbp; i++) {
    const int c = p + i, m = n - c - 1;
    const bool last = (i == P.nbp - 1);
    // ---- A: shares of A22 x 2^k and the panel dots; k brings x to about v's size
    const int k = (R.tau == 0.0) ? 0 : ((__double2hiint(R.scale) >> 20) & 0x7ff) - 1023;
    if (!fxp_matvec(P, S, c, t0, t1, k, !last, buf, xrow, xcol) && lane == 0) atomicExch(P.w.sync + 1, 1u);
    const int groups = (2 * i + FXP_DOT_COLS - 1) / FXP_DOT_COLS;
    const int chunks = (m + FXP_DOT_ROWS - 1) / FXP_DOT_ROWS;
    for (int item = nwarps - 1 - gw; item < groups * chunks; item += nwarps)
      fxp_dots(P, c, i, item, groups, R.scale, R.tau == 0.0);
    if (!fxp_barrier(P, round, []() {})) break;
    // ---- B: rows, as many threads per row as leaves one row block per quarter SM
    const double m2 = (R.tau == 0.0) ? 0.0 : oz_ldexp(R.scale, -k);
    const int quarters = 4 * gridDim.x;
    double ssp;
    if (m <= quarters)
      fxp_rows<32>(P, c, i, chunks, last, R, m2, H, ssp);
    else if (m <= 2 * quarters)
      fxp_rows<16>(P, c, i, chunks, last, R, m2, H, ssp);
    else if (m <= 4 * quarters)
      fxp_rows<8>(P, c, i, chunks, last, R, m2, H, ssp);
    else
      fxp_rows<4>(P, c, i, chunks, last, R, m2, H, ssp);
    if (last) break;
    ssp = warp_sum(ssp);
    if (lane == 0) H.red[w] = ssp;
    static_assert(FXP_NW == 8, "a tree of eight sums");
    if (!fxp_barrier(P, round, [&]() {
          const double* x = H.red;
          P.w.sspart[blockIdx.x] = ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
        }))
      break;
    // reflector c + 1, identically in every CTA, formed by one lane
    const int c1 = c + 1;
    if (w == 0) {
      const double alpha = __ldcg(A + (c1 + 1) + (int64_t)c1 * lda);
      double ss = 0.0;
      for (int t = lane; t < (int)gridDim.x; t += 32) ss += __ldcg(P.w.sspart + t);
      ss = warp_sum(ss);
      if (lane == 0) {
        s_scal = ss_needs_scaling(ss) ? 1 : 0;
        if (!s_scal) {
          const Reflector Rf = make_reflector(alpha, ss, -1.0);
          s_R = FxpRefl{Rf.beta, Rf.tau, Rf.scale};
        }
      }
    }
    __syncthreads();
    if (s_scal)
      R = fxp_reflector(P, c1, red);
    else
      R = s_R;
    __syncthreads();
    if (blockIdx.x == 0 && tid == 0) {
      P.evals[c1] = R.beta;
      P.tau[c1] = R.tau;
    }
  }
  // no CTA leaves with a copy of its own in flight (a barrier that gave up: the next column's)
  for (int q = 0; q < min(S.quarters, FXP_SLOTS); q++) {
    const unsigned at = S.issued - 1 - q;
    oz_wait(S.bar + 8 * (at % FXP_SLOTS), (at / FXP_SLOTS) & 1);
  }
}

// ---------------------------------------------------------------------------
// Trailing update: A22 += V W^T - W V^T, lower triangle
// ---------------------------------------------------------------------------
// Largest exponents of the panel's rows of V and of W, and of all of W (grid: rows / 256).
__global__ void __launch_bounds__(256) fxp_exps_kernel(const double* __restrict__ A, int64_t lda, int n, int p, int nbp,
                                                       FxpWs w) {
  const int q = p + nbp, r = q + blockIdx.x * 256 + threadIdx.x;
  int a = 1, b = 1;
  if (r < n) {
    for (int l = 0; l < nbp; l++) {
      a = max(a, oz_exponent(A[r + (int64_t)(p + l) * lda]));
      b = max(b, oz_exponent(w.W[(size_t)l * n + r]));
    }
    w.ev[r] = a;
    w.ew[r] = b;
  }
  b = __reduce_max_sync(0xffffffffu, b);
  if ((threadIdx.x & 31) == 0) atomicMax(w.sync + 2, (unsigned)b);
}

// C = [V | W 2^-k] [W 2^-k | -V]^T = 2^-k (V W^T - W V^T), 2^k the size of W: both factors
// near 1, so C stays in range for any A (V scaled to W instead would square A's scale).
struct FxpUpdate {
  double* A;
  int64_t lda;
  int n, p, nbp, q, half;  // half: entries of K per side, a multiple of the buffer
  FxpWs w;
  int k;
  __device__ int rows() const { return n - q; }
  __device__ int cols() const { return n - q; }
  __device__ int ksteps() const { return 2 * half / OZ_K; }
  __device__ bool contiguousA() const { return false; }
  __device__ bool contiguousB() const { return false; }
  __device__ int exponent(int r) const {
    const int a = w.ev[q + r], b = w.ew[q + r];
    if (a == 2047 || b == 2047) return 2047;
    return min(2046, max(max(a, b - k), 1));
  }
  __device__ int expA(int i) const { return exponent(i); }
  __device__ int expB(int j) const { return exponent(j); }
  template <int NV>
  __device__ __forceinline__ void load(int r, int kk, bool left, double (&v)[NV]) const {
    const bool low = kk < half;
    const int l0 = low ? kk : kk - half;
    const bool vside = (low == left);
#pragma unroll
    for (int u = 0; u < NV; u++) {
      double x = 0.0;
      if (l0 + u < nbp) x = vside ? A[q + r + (int64_t)(p + l0 + u) * lda] : w.W[(size_t)(l0 + u) * n + q + r];
      if (!vside) x = oz_ldexp(x, -k);
      v[u] = (vside && !left) ? neg(x) : x;
    }
  }
  __device__ void loadA(int i, int s, int kk, double (&v)[8]) const { load<8>(i, s * OZ_K + kk, true, v); }
  __device__ void loadB(int j, int s, int kk, double (&v)[4]) const { load<4>(j, s * OZ_K + kk, false, v); }
  __device__ void store(int i, int j, double x) const {
    if (i > j) A[q + i + (int64_t)(q + j) * lda] += oz_ldexp(x, k);
  }
  __device__ void timeout() const { w.sync[1] = 1u; }
};

__global__ void __launch_bounds__(OZ_NT, 1) fxp_update_kernel(FxpUpdate U) {  // grid: row tiles x column tiles
  extern __shared__ __align__(1024) unsigned char oz_buf[];
  const int i0 = blockIdx.x * OZ_M, j0 = blockIdx.y * OZ_N;
  if (i0 + OZ_M - 1 <= j0) return;  // above the diagonal
  U.k = max(-1000, min(1000, (int)U.w.sync[2] - 1023));
  oz_tile(U, i0, j0, oz_buf);
}

// A[c, r] = -A[r, c] in the last block from row q, zero diagonal untouched (the one-CTA kernel reads both triangles)
__global__ void fxp_mirror_kernel(double* A, int64_t lda, int n, int q) {
  const int m = n - q;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < m * m; t += gridDim.x * blockDim.x) {
    const int r = t % m, c = t / m;
    if (r > c) A[q + c + (int64_t)(q + r) * lda] = neg(A[q + r + (int64_t)(q + c) * lda]);
  }
}

__global__ void fxp_status_kernel(const unsigned* sync, int* info) {
  if (sync[1] && info) *info = SKEW_TIMEOUT;
}

// A reduced in place into tau, ev.  cudaErrorNotSupported where the panel kernel cannot run.
cudaError_t wide_hessenberg(double* A, int64_t lda, int n, double* tau, double* ev, int* info, double* wsbase, int sms,
                            const Tuning& T, cudaStream_t st) {
  if (n <= kWideMin || T.persist_nb > FXP_NB) return cudaErrorNotSupported;
  FxpWs w;
  fxp_carve(&w, (double*)(((uintptr_t)wsbase + 15) & ~(uintptr_t)15), n);
  cudaError_t e = cudaFuncSetAttribute(fxp_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FXP_SMEM);
  if (e != cudaSuccess) return cudaErrorNotSupported;
  static std::atomic<uint64_t> raised{0};
  if ((e = raise_smem_limit_once((const void*)fxp_update_kernel, raised))) return e;
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fxp_panel_kernel, FXP_NT, FXP_SMEM);
  if (e != cudaSuccess) return e;
  if (occ < 1) return cudaErrorNotSupported;
  int grid = std::min(sms, FXP_CTAS), tail = FXP_TAIL;
  if (T.persist_ctas > 0) grid = std::max(1, std::min(grid, T.persist_ctas));
  if (T.persist_tail > 0) tail = std::max(32, std::min(FXP_TAIL, T.persist_tail));
  const int nb = std::max(8, std::min(FXP_NB, T.persist_nb));
  const int pend = n - tail;
  if ((e = cudaMemsetAsync(w.sync, 0, 4 * sizeof(unsigned), st))) return e;
  for (int p = 0; p < pend; p += nb) {
    FxpPanel P;
    P.A = A;
    P.lda = lda;
    P.n = n;
    P.p = p;
    P.nbp = std::min(nb, pend - p);
    P.T = (n - p - 1 + FXP_T - 1) / FXP_T;
    const int ntiles = P.T * (P.T + 1) / 2;
    P.per = (ntiles + grid * FXP_NW - 1) / (grid * FXP_NW);
    P.tau = tau;
    P.evals = ev;
    P.w = w;
    P.poll_limit = T.wait_polls > 0 ? T.wait_polls : FXP_POLLS;
    P.skip_cta = T.wait_skip_cta;
    if (p > 0 && (e = cudaMemsetAsync(w.sync, 0, sizeof(unsigned), st))) return e;
    if ((e = cudaMemsetAsync(w.sync + 2, 0, sizeof(unsigned), st))) return e;
    fxp_pack_kernel<<<ntiles, 256, 0, st>>>(A, lda, n, p + 1, P.T, w.pack, w.etile);
    void* args[] = {&P};
    e = cudaLaunchCooperativeKernel((const void*)fxp_panel_kernel, dim3(grid), dim3(FXP_NT), args, FXP_SMEM, st);
    if (e != cudaSuccess) return p == 0 ? e : cudaErrorUnknown;
    const int q = p + P.nbp, m = n - q;
    fxp_exps_kernel<<<(m + 255) / 256, 256, 0, st>>>(A, lda, n, p, P.nbp, w);
    FxpUpdate U;
    U.A = A;
    U.lda = lda;
    U.n = n;
    U.p = p;
    U.nbp = P.nbp;
    U.q = q;
    U.half = (P.nbp + OZ_K - 1) / OZ_K * OZ_K;
    U.w = w;
    U.k = 0;
    fxp_update_kernel<<<dim3((m + OZ_M - 1) / OZ_M, (m + OZ_N - 1) / OZ_N), OZ_NT, OZ_SMEM, st>>>(U);
    if ((e = cudaGetLastError())) return e;
  }
  fxp_mirror_kernel<<<16, 256, 0, st>>>(A, lda, n, pend);
  SingleParams S;
  S.A = A + pend + (int64_t)pend * lda;
  S.lda = lda;
  S.n = n - pend;
  S.G = nullptr;
  S.ldg = 0;
  S.logpf = nullptr;
  S.sign = nullptr;
  S.ev = ev + pend;
  S.tau = tau + pend;
  S.info = info;
  S.check = 0;
  S.want_pf = 0;
  e = launch_single(S, st);
  if (e != cudaSuccess) return e;
  fxp_status_kernel<<<1, 1, 0, st>>>(w.sync, info);
  return cudaGetLastError();
}

}  // namespace skew
