// The implicit-QR iteration of the skew tridiagonal eigenproblem (skewtrieigvals!,
// skeweigen.jl:73-156, and the iteration of skewtrieigen_divided!, :158-193, 322-383), four
// lanes per matrix.
//
// The iteration is one chain of dependent Givens rotations, and an FP64 instruction
// occupies its sub-partition's pipe for 64 cycles whatever its active lanes, so a step costs
// its number of FP64 instructions.  One lane per matrix took about 50 of them: the hypot
// and two divisions of the rotation, eight products and three sums.  With four lanes the
// divisions run side by side, and so do the products and sums:
//   lane 0: c a + s bulge -> ev[i-2]   lane 1: c b - s g -> ev[i-1]
//   lane 2: s b + c g -> ev[i]         lane 3: c z -> ev[i+1], s z -> the next bulge
// two products and one sum in all.  Every product, sum and quotient is rounded separately,
// as in the reference's Float64 code: the deflation decisions depend on the last bits.
// Comparisons with constants are made on the bit patterns.  The subdiagonal lies in shared
// memory.  The loop takes one rotation per turn for each of a warp's eight matrices, a
// matrix at the end of its sweep deflating and starting the next one in the same turn, so
// they do not wait for one another's sweeps.
// n = 512, one matrix: 218.2 -> 175.0 ms; 4096 matrices of n = 16 .. 256: 59.9 -> 48.5 ms;
// with the rotations logged, 256 matrices of n = 15 .. 200: 36.9 -> 30.0 ms.  Of a step's
// 2 650 cycles hypot takes 1 100 and a division 560; a lane with nothing left to do must keep
// off their special cases (with 0 / 0 in the idle lanes one matrix took 250 ms).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "skew_common.cuh"

namespace skew {

constexpr int CH_G = 4;          // lanes per matrix
constexpr int CH_M = 32 / CH_G;  // matrices per warp (and CTA)

// |x| < 2^-52 m (m = 1 or 10) for the tolerances eps and 10 eps; false for a NaN
__device__ __forceinline__ bool ch_below(double x, double tol) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffLL) < __double_as_longlong(tol);
}
__device__ __forceinline__ bool ch_at_most(double x, double tol) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffLL) <= __double_as_longlong(tol);
}
__device__ __forceinline__ bool ch_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }

// State of one matrix, equal in its four lanes but for q1, q2 (this lane's factors).
// LOG: the rotations go to log after a header (start, n) per sweep, and a split found in
// mid-sweep restarts the shifted rotation from there (implicitstep_vec!); else it ends the
// sweep (implicitstep_novec).  merged: without the mem deflation of skeweigen.jl:355.
template <bool LOG>
struct Chain {
  double* ev;    // shared memory
  double* vals;  // global
  double* log;
  int64_t len, cap;
  int n, start, i, m, iter, max_iter, count_static, merged, status, fb_n;
  bool run;
  double mem, shift, q1, q2, nb, bulge;  // nb: ev[i-2] as the previous step left it

  __device__ __forceinline__ void begin(double* ev_, int N, double* vals_, int cap_iter, int merged_, double* log_,
                                        int64_t cap_) {
    ev = ev_;
    vals = vals_;
    log = log_;
    cap = cap_;
    len = 0;
    n = N;
    start = 1;
    iter = 0;
    max_iter = cap_iter > 0 ? cap_iter : 30 * n;
    count_static = 0;
    merged = merged_;
    status = SKEW_OK;
    fb_n = 0;
    mem = 1.0;
    run = true;
    sweep();
  }

  __device__ __forceinline__ void finish(int st) {
    status = st;
    run = false;
  }

  // Start of a sweep over the active size n, or the end of the iteration.
  __device__ __forceinline__ void sweep() {
    const int g = threadIdx.x & (CH_G - 1);
    if (!(n > 2 && iter < max_iter)) {
      if (n == 2 && g == 0) {
        vals[0] = ev[0];
        vals[1] = neg(ev[0]);
      }
      if (n == 1 && g == 0) vals[0] = 0.0;
      finish(n > 2 ? SKEW_NO_CONVERGENCE : SKEW_OK);
      return;
    }
    m = n - 1;
    if (LOG) {
      if (len + 2 + 2 * (int64_t)(m - start) > cap) {
        finish(SKEW_NO_CONVERGENCE);
        return;
      }
      if (g == 0) {
        log[len] = (double)start;
        log[len + 1] = (double)m;
      }
      len += 2;
    }
    i = start;
    shift = __dmul_rn(ev[m - 1], ev[m - 1]);
    const double b = ev[start - 1], gg = ev[start], z = (start < m - 1) ? ev[start + 1] : 0.0;
    nb = 0.0;
    bulge = 0.0;
    q1 = (g == 0) ? 0.0 : (g == 3 ? z : b);
    q2 = (g == 0) ? 0.0 : (g == 3 ? z : gg);
  }

  // Deflation after a sweep (skeweigen.jl:121-146, 346-383).
  __device__ __forceinline__ void deflate() {
    const bool w = (threadIdx.x & (CH_G - 1)) == 0;
    const double tol = 10.0 * 2.220446049250313e-16;
    while (n > 2 && ch_at_most(ev[n - 2], tol)) {
      if (w) vals[n - 1] = 0.0;
      n -= 1;
    }
    while (n > 2 && fabs(ev[n - 3]) <= tol * fabs(ev[n - 2])) {
      if (w) {
        vals[n - 2] = ev[n - 2];
        vals[n - 1] = neg(ev[n - 2]);
      }
      n -= 2;
    }
    if (LOG && !merged && n > 2 && ch_below(ev[n - 2] - mem, tol)) {
      if (w) {
        vals[n - 2] = ev[n - 2];
        vals[n - 1] = neg(ev[n - 2]);
      }
      n -= 2;
    }
    if (start > n - 2) start = 1;
    if (n > 1 && fabs(mem - ev[n - 2]) < 0.0001 * fabs(ev[n - 2])) {
      count_static += 1;
      if (count_static > 4) {  // stagnation: symmetric tridiagonal fallback (:134-137)
        fb_n = n;
        finish(SKEW_FALLBACK_USED);
        return;
      }
    } else {
      count_static = 0;
    }
    mem = (n > 1 ? ev[n - 2] : 0.0);
    iter += 1;
    sweep();
  }

  // One rotation; all 32 lanes of the warp together.
  __device__ __forceinline__ void step() {
    const int g = threadIdx.x & (CH_G - 1);
    const unsigned full = 0xffffffffu;
    double x = run ? nb : 1.0, y = run ? bulge : 1.0;  // a finished matrix stays off the special cases' slow paths
    // ev[i+1] of the next step, untouched in this sweep (lane 3 only)
    const double zn = (g == 3 && run && i + 2 <= m - 1) ? ev[i + 2] : 0.0;
    if (run && i == start) {  // the shifted rotation, from a = 0
      const double b = ev[start - 1], gg = ev[start];
      x = __dadd_rn(__dsub_rn(neg(__dmul_rn(0.0, 0.0)), __dmul_rn(b, b)), shift);
      y = __dadd_rn(neg(__dmul_rn(0.0, bulge)), __dmul_rn(b, gg));
      if (g == 0) q1 = 0.0;
    }
    const double nm = hypot(x, y);
    const double q = __ddiv_rn((g & 1) ? y : x, nm);  // even lanes c, odd lanes s
    double c = __shfl_sync(full, q, 0, CH_G), s = __shfl_sync(full, q, 1, CH_G);
    if (ch_zero(nm)) {
      c = 1.0;
      s = 0.0;
    }
    const double u = __dmul_rn((g == 2) ? s : c, q1);
    const double v = __dmul_rn((g == 2) ? c : s, q2);
    const double r = __dadd_rn(u, (g == 1) ? neg(v) : v);
    const double nb1 = __shfl_sync(full, r, 1, CH_G), bl1 = __shfl_sync(full, v, 3, CH_G);
    const double ng1 = __shfl_sync(full, r, 2, CH_G), nz1 = __shfl_sync(full, u, 3, CH_G);
    if (run) {
      if (LOG && g < 2) log[len + g] = (g == 0) ? c : s;
      if (LOG) len += 2;
      const bool inner = i < m - 1;
      // every lane stores its entry: ev[i-2], ev[i-1], ev[i], ev[i+1]
      if (g == 3 ? inner : (g > 0 || i > 1)) ev[i - 2 + g] = (g == 3) ? u : r;
      nb = nb1;
      bulge = bl1;
      q1 = (g == 0) ? nb1 : (g == 3 ? zn : ng1);
      q2 = (g == 0) ? bl1 : (g == 3 ? zn : nz1);
      if (inner && ch_below(bl1, LOG ? 10.0 * 2.220446049250313e-16 : 2.220446049250313e-16) &&
          ch_below(nb1, LOG ? 10.0 * 2.220446049250313e-16 : 2.220446049250313e-16)) {
        start = i + 1;
        if (!LOG) i = m;  // the sweep ends
      }
      i++;
    }
    __syncwarp();
    if (run && i > m - 1) deflate();
    __syncwarp();
  }
};

}  // namespace skew
