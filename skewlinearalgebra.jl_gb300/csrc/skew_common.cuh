// Shared device helpers for libskewgpu (sm_103a, FP64).
//
// Cost model this code is written against (measured on GB300): the FP64 pipe of
// an SM sub-partition retires one warp-wide DFMA every 64 cycles (1.19 TFLOP/s
// per GPU), whatever the number of active lanes; a double divide or square
// root costs about ten DFMAs.  So: every FP64 instruction should carry 32
// useful lanes, scalar FP64 work stays off the critical path where it can, and
// integer index arithmetic, loads and shuffles are close to free.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/skewgpu.h"

namespace skew {

constexpr int WARP = 32;

// Negation by flipping the sign bit on the integer pipe (keeps the FP64 pipe free).
__device__ __forceinline__ double neg(double x) {
  return __hiloint2double(__double2hiint(x) ^ 0x80000000, __double2loint(x));
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Block-wide sum for a block of NW warps; red must hold NW doubles. All threads
// get the result.  Contains two __syncthreads().
template <int NW>
__device__ __forceinline__ double block_sum(double x, double* red) {
  x = warp_sum(x);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = x;
  __syncthreads();
  double s = 0;
#pragma unroll
  for (int i = 0; i < NW; i++) s += red[i];
  __syncthreads();
  return s;
}

// Householder reflector parameters following hessenberg.jl:26-44 (householder!):
// beta = -sign(alpha) * hypot(alpha, |x|), tau = 1 - alpha/beta, v = [1; x/(alpha-beta)].
// ss = |x|^2 (sum of squares of the part below alpha); xnorm_scaled >= 0 is |x|
// computed with scaling, supplied by the caller only when ss over/underflowed
// (then hypot is used, as the reference does).  One division is shared by tau
// and the scale: with d = alpha - beta and r = 1/(beta*d), 1/beta = d*r and
// 1/d = beta*r.
struct Reflector {
  double tau, beta, scale;
};
__device__ __forceinline__ bool ss_needs_scaling(double ss) { return !(ss < 1e290) || (ss > 0.0 && ss < 1e-290); }

__device__ __forceinline__ Reflector make_reflector(double alpha, double ss, double xnorm_scaled) {
  Reflector R;
  if (ss == 0.0 && alpha == 0.0) {  // :38-41
    R.tau = 0.0;
    R.beta = 0.0;
    R.scale = 0.0;
    return R;
  }
  double h;
  if (xnorm_scaled < 0.0 && fabs(alpha) < 1e145) {
    h = sqrt(fma(alpha, alpha, ss));
  } else {
    h = hypot(alpha, xnorm_scaled < 0.0 ? sqrt(ss) : xnorm_scaled);
  }
  const double beta = alpha > 0.0 ? neg(h) : h;  // :33
  const double d = alpha - beta;                 // never cancels: beta has the opposite sign
  if (fabs(h) < 1e150 && fabs(h) > 1e-150) {
    const double r = 1.0 / (beta * d);
    R.tau = neg(d * (d * r));  // 1 - alpha/beta = -d/beta
    R.scale = beta * r;        // 1/(alpha - beta)
  } else {
    R.tau = 1.0 - alpha / beta;
    R.scale = 1.0 / d;
  }
  R.beta = beta;
  return R;
}

// Sum over the 32 lanes of 32 per-lane values at once (butterfly transpose):
// on return lane L holds sum_lanes v[L].  31 adds instead of 32 x 5.
__device__ __forceinline__ double warp_transpose_sum32(double (&v)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    const bool up = lane & s;
#pragma unroll
    for (int i = 0; i < s; i++) {
      const double send = up ? v[i] : v[i + s];
      const double keep = up ? v[i + s] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
    }
  }
  return v[0];
}

// Reduce per-thread partial values part[0..npair) (npair <= 32) over the block
// into out[0..npair); scratch holds NW*32 doubles.
template <int NT>
__device__ void block_reduce_pairs(double (&part)[32], int npair, double* scratch, double* out) {
  constexpr int NW = NT / 32;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double mine = warp_transpose_sum32(part);  // lane L holds the warp's sum for slot L
  scratch[w * 32 + lane] = mine;
  __syncthreads();
  if ((int)threadIdx.x < npair) {
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < NW; q++) acc += scratch[q * 32 + threadIdx.x];
    out[threadIdx.x] = acc;
  }
  __syncthreads();
}

// Pair (l1 < l2) of 8 columns -> slot; 28 slots.
__device__ __forceinline__ int pair_slot(int l1, int l2) { return l1 * 8 - (l1 * (l1 + 1)) / 2 + (l2 - l1 - 1); }

// Bounded spin on a device flag: returns false if `limit` polls pass first.
__device__ __forceinline__ bool spin_until_geq(const volatile unsigned* flag, unsigned target, long long limit) {
  for (long long it = 0; it < limit; it++) {
    if (*flag >= target) return true;
    __nanosleep(64);
  }
  return false;
}

}  // namespace skew

namespace skew {

// Multisection for the target-th smallest eigenvalue (0-based) of a symmetric
// tridiagonal, given count(x) = number of eigenvalues smaller than x (Sturm).
// Groups of p lanes (p a power of two, p <= 32) share one eigenvalue: each step
// the p lanes count at p interior points of [lo, hi] and the group keeps the
// sub-interval [x_{j-1}, x_j] where x_j is the first point whose count exceeds
// the target, so the bracket count(lo) <= target < count(hi) holds by
// construction.  The interval shrinks (p+1)-fold per step until it is below
// max(2 eps max(|lo|, |hi|), abstol).  All 32 lanes of the warp must call this
// (active = false for a group with nothing to find).  Returns the midpoint.
template <class Count>
__device__ double group_multisect(double lo, double hi, int target, double abstol, int p, bool active, Count count) {
  const int lane = threadIdx.x & 31;
  const int g = lane / p, gl = lane - g * p;
  const unsigned gmask = (p == 32) ? 0xffffffffu : (((1u << p) - 1u) << (g * p));
  const double inv = 1.0 / (double)(p + 1);
  bool run = active;
  for (int it = 0; it < 256; it++) {
    const double w = hi - lo;
    if (run && !(w > fmax(2.220446049250313e-16 * fmax(fabs(lo), fabs(hi)), abstol))) run = false;
    if (!__any_sync(0xffffffffu, run)) break;
    const double x = lo + w * ((double)(gl + 1) * inv);
    const bool below = run ? (count(x) <= target) : true;
    const unsigned bits = __ballot_sync(0xffffffffu, below) & gmask;
    if (run) {
      const unsigned above = ~bits & gmask;  // points whose count exceeds the target
      const int j = above ? (__ffs(above) - 1 - g * p) : p;  // first such point (p: none)
      const double nlo = (j == 0) ? lo : lo + w * ((double)j * inv);
      const double nhi = (j == p) ? hi : lo + w * ((double)(j + 1) * inv);
      lo = nlo;
      hi = nhi;
    }
  }
  return 0.5 * (lo + hi);
}

// Sturm count by the characteristic polynomials of the leading blocks of T - x I,
//   p_0 = 1, p_1 = d_1 - x, p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}:
// the eigenvalues below x are the sign changes.  Bound by the FP64 pipe (one warp
// instruction per 64 cycles of a sub-partition, whatever its active lanes): two
// instructions per row from the squares e2 = e^2 (three with a diagonal), where the
// pivot form q_i = d_i - x - e^2 / q_{i-1} takes a division and about twelve.  The
// multisection of 512 problems of n = 32 .. 512: 86.4 -> 23.4 ms; n = 2048: 16.9 -> 4.3 ms
// (3.4 with group_rootsect's fewer steps).
// Each step's rounding is a relative change of its (d_i - x) and e^2, so with a zero
// diagonal tiny eigenvalues keep their relative accuracy, as with the pivots.  A zero
// p_i stands for a pivot a hair below zero and is counted, as the pivot form's -pivmin
// (a split e = 0 then starts over from it).  The pair (p_{i-1}, p_i) is brought back to
// the middle of the exponent range whenever both lie outside 2^-256 .. 2^256; d, e2 and
// x come scaled to a spectrum within [-1, 1], so one step cannot leave the range.
// d(i), e2(i): entry i of the scaled diagonal (dx(i) = d_i - x) and of the squares.
struct SturmVal {
  int c;     // eigenvalues below x
  double m;  // p_n(x) = m 2^k
  int k;
};
template <class DX, class E2>
__device__ __forceinline__ SturmVal sturm_products(int n, DX dx, E2 e2) {
  // p == 0: the other sign than the entry before it (high word hb), 2^-400 of its size
  auto settle = [](double& p, int& h, int hb) {
    if (((h << 1) | __double2loint(p)) == 0) {
      h = ((hb & 0x80000000) ^ 0x80000000) | max((hb & 0x7ff00000) - (400 << 20), 0x00100000);
      p = __hiloint2double(h, 0);
    }
  };
  double p0 = 1.0, p1 = dx(0);
  int h1 = __double2hiint(p1);
  settle(p1, h1, 0x3ff00000);
  int c = (unsigned)h1 >> 31, k = 0;
  for (int i = 1; i < n; i++) {
    double p2 = fma(dx(i), p1, neg(e2(i - 1) * p0));
    int h2 = __double2hiint(p2);
    settle(p2, h2, h1);
    c += (unsigned)(h2 ^ h1) >> 31;
    const int top = max(h2 & 0x7fffffff, h1 & 0x7fffffff);
    if ((unsigned)(top - 0x2ff00000) > 0x20000000u) {  // the pair lies outside 2^-256 .. 2^256
      const double f = (top < 0x3ff00000) ? 0x1p+500 : 0x1p-500;
      k += (top < 0x3ff00000) ? -500 : 500;
      p1 *= f;
      p2 *= f;
      const int s2 = h2 & 0x80000000;
      h2 = __double2hiint(p2);
      if (((h2 << 1) | __double2loint(p2)) == 0) {  // underflow keeps its sign
        h2 = s2 | 0x00100000;
        p2 = __hiloint2double(h2, 0);
      }
    }
    p0 = p1;
    p1 = p2;
    h1 = h2;
  }
  return SturmVal{c, p1, k};
}

// |a / b| of two values m 2^k
__device__ __forceinline__ double sturm_ratio(double am, int ak, double bm, int bk) {
  const int d = max(-1000, min(1000, ak - bk));
  return fabs(am / bm) * __hiloint2double((1023 + d) << 20, 0);
}

// group_multisect where the count comes with the value of the characteristic polynomial:
// once one eigenvalue is left between two counted points, the secant through the
// polynomial's values there says where it lies.  The points are then
//   p = 1: the secant's root, and after it twice as far from the new end as the next secant's
//          root, so that the other end follows;
//   p > 1: pairs around the secant's root at distances of 2^-s of the interval (p = 2, 4: s
//          doubles while it succeeds).
// The counts alone decide which points become the new interval, so it keeps the bracket
// count(lo) <= target < count(hi) of group_multisect and ends at the same width.  Guesses that
// brought less than even division (another eigenvalue close outside) are followed by even
// steps, more after each failure; so is the end, within four final widths.
// Bound by the FP64 pipe and its latency: two FMAs per row and step, so the steps count: 19 to
// 24 instead of 53 with one lane per eigenvalue, 11 to 13 instead of 23 with 4, 8 to 10 instead
// of 13 with 16, 8 instead of 11 with 32.
template <class Eval>
__device__ double group_rootsect(double lo, double hi, int target, double abstol, int p, bool active, Eval eval) {
  const int lane = threadIdx.x & 31;
  const int g = lane / p, gl = lane - g * p;
  const unsigned gmask = (p == 32) ? 0xffffffffu : (((1u << p) - 1u) << (g * p));
  const double inv = 1.0 / (double)(p + 1);
  const double enough = (p == 1) ? 0.25 : inv;  // of the interval a guess (p = 1: two) may leave
  const int gap = (p == 8) ? 5 : (p == 16 ? 4 : 3);
  const int pair = (gl < p / 2) ? gl : p - 1 - gl;
  SturmVal vl{-1, 0.0, 0}, vh{-1, 0.0, 0};  // at lo and hi, once counted there
  int wait = 0, fails = 0, s = 3;
  int moved = 0;  // p = 1: the end that the first guess of two moved (1: hi, 2: lo)
  double wref = 0.0;
  bool run = active;
  for (int it = 0; it < 256; it++) {
    const double w = hi - lo;
    const double tol = fmax(2.220446049250313e-16 * fmax(fabs(lo), fabs(hi)), abstol);
    if (run && !(w > tol)) run = false;
    if (!__any_sync(0xffffffffu, run)) break;
    bool guess = vl.c >= 0 && vh.c == vl.c + 1 && w > 4.0 * tol;
    if (!guess) moved = 0;
    if (guess && moved == 0) {
      if (wait > 0) {
        wait--;
        guess = false;
      } else if (wref > 0.0 && w > wref * enough) {
        wait = min(2 * fails, 8);
        fails++;
        s = 3;
        wref = 0.0;
        guess = false;
      } else {
        if (wref > 0.0) {
          fails = 0;
          s = min(2 * s, 24);
        }
        wref = w;
      }
    }
    double x = lo + w * ((double)(gl + 1) * inv);
    if (run && guess) {
      double root = lo + w / (1.0 + sturm_ratio(vh.m, vh.k, vl.m, vl.k));
      if (p == 1) {
        if (moved == 2) root += fmax(root - lo, 0.25 * tol);
        if (moved == 1) root -= fmax(hi - root, 0.25 * tol);
        x = fmin(fmax(root, lo + 0.5 * tol), hi - 0.5 * tol);
      } else {
        const int e = (p <= 4) ? s * (pair + 1) : 2 + gap * pair;  // at most 48
        const double o = fmax(w * __hiloint2double((1023 - e) << 20, 0), 0.45 * tol);
        x = (gl < p / 2) ? fmax(lo, root - o) : fmin(hi, root + o);
      }
    }
    SturmVal v{0, 0.0, 0};
    if (run) v = eval(x);
    const bool below = run ? (v.c <= target) : true;
    const unsigned bits = __ballot_sync(0xffffffffu, below) & gmask;
    const unsigned above = ~bits & gmask;  // points whose count exceeds the target
    const int j = above ? (__ffs(above) - 1 - g * p) : p;  // first such point (p: none)
    const int sl = g * p + max(j - 1, 0), sh = g * p + min(j, p - 1);
    const double xl = __shfl_sync(0xffffffffu, x, sl), xh = __shfl_sync(0xffffffffu, x, sh);
    const SturmVal nl{__shfl_sync(0xffffffffu, v.c, sl), __shfl_sync(0xffffffffu, v.m, sl),
                      __shfl_sync(0xffffffffu, v.k, sl)};
    const SturmVal nh{__shfl_sync(0xffffffffu, v.c, sh), __shfl_sync(0xffffffffu, v.m, sh),
                      __shfl_sync(0xffffffffu, v.k, sh)};
    if (run) {
      if (p == 1) moved = (guess && moved == 0) ? j + 1 : 0;
      if (j > 0) {
        lo = xl;
        vl = nl;
      }
      if (j < p) {
        hi = xh;
        vh = nh;
      }
    }
  }
  return 0.5 * (lo + hi);
}

// The power of two that brings a spectrum within [-bound, bound] into [-1, 1].
__device__ __forceinline__ double sturm_scale(double bound) {
  const int k = ((__double2hiint(bound) >> 20) & 0x7ff) - 1022;  // bound < 2^k
  const int b = min(max(1023 - k, 1), 2046);
  return __hiloint2double(b << 20, 0);
}

// rows whose scaled squares (and diagonal) a CTA stages in its 48 KB of shared memory;
// above this they are formed on the fly (one more FP64 instruction per row)
constexpr int STURM_STAGE = 3072;

// lanes per eigenvalue for m eigenvalues on a GPU with `sms` SMs: enough groups
// to give every SM sub-partition a warp, at most a warp per eigenvalue
__host__ __device__ inline int multisect_lanes(int m, int sms) {
  const long long want = (long long)sms * 4 * 32 / (m > 0 ? m : 1);
  int p = 1;
  while (p < 32 && 2LL * p <= want) p *= 2;
  return p;
}

}  // namespace skew
