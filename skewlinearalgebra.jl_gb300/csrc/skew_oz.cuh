// Products of FP64 matrices on the tensor cores, at FP64 accuracy.
//
// The FP64 pipe of a GB300 SM retires 2 FMAs per clock, its fifth-generation tensor
// core about 3 900 fp16 multiply-adds.  A row of A (a column of B) is scaled by the
// power of two that brings its largest entry below 1, rounded to 56 bits and cut into
// seven signed base-256 digits (after Ozaki, Ogita, Oishi and Rump's error-free
// splitting):
//   x = 2^(e - 1078) sum_i d_i 256^(6 - i),  |d_0| <= 256, -128 <= d_i < 128,
// e the vector's largest biased exponent.  Digits are exact in fp16.  The products of
// digits i and j with i + j = g are summed over 128 entries in one FP32 accumulator of
// group g: at most 2^24 up to g = 5, so those sums are exact (g = 6 could exceed it by an
// eighth if every digit were extreme: one unit of 2^-64).  Groups 0 .. 7 are kept (34 of
// the 49 digit products); the rest is below 2^-60 of the largest product.  After each 128
// entries the eight sums are joined in a 96-bit integer (2^-64 of the largest product),
// whatever the length of the sum.  Measured against products summed in 113 bits (entries
// N(0, 1), K = 16, 128, 512, 2048): 4.9e-17 to 5.2e-17 of the result, the rounding of the
// result itself; FMAs 1.4e-16, 3.8e-16, 7.5e-16, 1.5e-15.  That is relative to the largest
// entries: one below 1/8 of its vector's largest keeps fewer than 53 bits, so where large
// entries meet zeros, a small result beside them is less accurate than by FMAs (block-diagonal
// times a cotangent graded by 1e-6: its small block to 1.9e-11 instead of 2.4e-16).  A vector with an infinity or a
// NaN (e = 2047) makes its results NaN.
//
// One CTA of 17 warps computes a 128 x 64 tile; its eight groups fill the SM's 512
// columns of tensor memory, so one CTA runs per SM.  Per 32 entries of K the threads
// read A and B, cut them and store the digits in shared memory (K-major core matrices of
// 8 rows x 16 bytes, two buffers) while the tensor core works on the buffer before; the
// digits of B lie next to each other, so one instruction multiplies digit i of A by up to
// four digits of B and adds to the four groups i + j at once: the tile of A is read 11
// instead of 34 times per 16 entries.  2048^3: 0.76 ms (22.5 TFLOP/s; the MMAs alone take
// 0.37, cutting and loading 0.53, joining the sums 0.15, in part one after the other),
// 8192 x 8192 x 128: 0.98 ms; FMAs at the FP64 peak take 13.7 ms for
// either.  With 256 instead of 512 threads on
// the digits and the MMAs issued from a loop it took 1.06 ms.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace skew {

constexpr int OZ_M = 128, OZ_N = 64, OZ_K = 32;  // tile, entries of K per buffer
constexpr int OZ_NT = 544;  // 512 that cut digits and join sums, one warp that issues the MMAs
constexpr int OZ_S = 7;       // digits
constexpr int OZ_CHUNK = 128;  // entries of K per exact FP32 sum
// Bytes between the core matrices of neighbouring groups of 8 entries of K: a digit of A's
// 128 rows, all digits of B's 64 columns, padded so that neighbouring lanes holding
// neighbouring groups store to different banks.
constexpr int OZ_A_LBO = OZ_M * 16 + 32, OZ_B_LBO = OZ_S * OZ_N * 16 + 64;
constexpr int OZ_A_DIGIT = OZ_A_LBO * (OZ_K / 8), OZ_B_DIGIT = OZ_N * 16;
constexpr int OZ_A_BYTES = OZ_S * OZ_A_DIGIT, OZ_B_BYTES = OZ_B_LBO * (OZ_K / 8);
constexpr int OZ_STAGE = OZ_A_BYTES + OZ_B_BYTES;  // 87 168
constexpr int OZ_SMEM = 2 * OZ_STAGE + 1024;       // + exponents (768), barriers
constexpr int OZ_POLLS = 1 << 22;

// Biased exponent of x for the scaling maximum (zero and subnormal count as 1).
__device__ __forceinline__ int oz_exponent(double x) { return max((__double2hiint(x) >> 20) & 0x7ff, 1); }

// 56-bit integer of x (|x| at most of the biased exponent e, rounded) with the bias that
// makes bits 48 .. 57 digit 0 + 512 and the six bytes below digits 1 .. 6 + 128.  The
// threads' integer instructions (64 lanes per clock and SM) bound the cutting, so the
// usual case avoids the two instructions that a subnormal needs.
constexpr unsigned long long OZ_BIAS = 0x0200808080808080ull;
static __device__ __noinline__ unsigned long long oz_fixed_tiny(double x, int e) {  // e < 64: subnormals count
  const int hi = __double2hiint(x);
  const int ex = (hi >> 20) & 0x7ff;
  unsigned long long m = ((unsigned long long)(unsigned)((hi & 0xfffff) | (ex ? 0x100000 : 0)) << 32) |
                         (unsigned)__double2loint(x);
  m = (((m << 4) >> (e - max(ex, 1))) + 1) >> 1;
  return (hi < 0) ? OZ_BIAS - m : OZ_BIAS + m;
}
__device__ __forceinline__ unsigned long long oz_fixed(double x, int e) {
  if (e < 64) return oz_fixed_tiny(x, e);
  const int hi = __double2hiint(x);
  const int sh = min(e - ((hi >> 20) & 0x7ff), 60);  // x = m 2^(ex - 1075); m 2^3 has 56 bits; 0 shifts out
  const unsigned long long m = ((unsigned long long)(unsigned)((hi & 0xfffff) | 0x100000) << 32) |
                               (unsigned)__double2loint(x);
  const long long sg = (long long)(hi >> 31);
  return (((((m << 4) >> sh) + 1) >> 1) ^ sg) + (OZ_BIAS - sg);
}

// v 2^e, rounded to nearest, on the integer pipe (a conversion and a scaling take three
// FP64 instructions of 64 cycles); results outside the normal range take the FP64 form.
static __device__ __noinline__ double oz_double_edge(long long v, int e) { return scalbn((double)v, e); }
__device__ __forceinline__ double oz_double(long long v, int e) {
  if (v == 0) return 0.0;
  const unsigned long long a = (v < 0) ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int lz = __clzll((long long)a);
  const int ex = 1086 - lz + e;  // biased exponent of 2^(63 - lz) 2^e
  if (ex < 1 || ex > 2045) return oz_double_edge(v, e);
  const unsigned long long m = a << lz;
  const unsigned long long bits = ((unsigned long long)(ex - 1) << 52) + (m >> 11) + ((m >> 10) & 1);
  return __longlong_as_double((long long)(bits | ((unsigned long long)(v < 0) << 63)));
}

// x 2^k: the exponent field where x is finite and stays normal, else by multiplication (out
// of line: as a select it would put FP64 instructions on every entry)
static __device__ __noinline__ double oz_ldexp_edge(double x, int k) { return scalbn(x, k); }
__device__ __forceinline__ double oz_ldexp(double x, int k) {
  const int h = __double2hiint(x), e = (h >> 20) & 0x7ff;
  if ((unsigned)(e - 1) < 2046u && (unsigned)(e + k - 1) < 2045u) return __hiloint2double(h + (k << 20), __double2loint(x));
  return x == 0.0 ? x : oz_ldexp_edge(x, k);
}

__device__ __forceinline__ uint32_t oz_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t oz_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3ffff) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
         (1ull << 46);
}

__device__ __forceinline__ void oz_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t n, uint32_t acc) {
  // fp16 x fp16 -> fp32, both K-major, M = 128
  const uint32_t idesc = (1u << 4) | ((n >> 3) << 17) | ((OZ_M >> 4) << 24);
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

// Bounded wait for a phase of an mbarrier.  A lane may give up where its neighbours did not:
// they vote before the next warp-wide instruction.
__device__ __forceinline__ bool oz_wait(uint32_t bar, uint32_t parity) {
  for (int t = 0; t < OZ_POLLS; t++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// All MMAs of one buffer (OZ_K entries of K).  FRESH: the first buffer of an exact sum.
template <bool FRESH>
__device__ __forceinline__ void oz_issue(uint32_t tmem, uint32_t sa, uint32_t sb) {
  const uint64_t da = oz_desc(sa, OZ_A_LBO, 128), db = oz_desc(sb, OZ_B_LBO, 128);  // offsets add in 16-byte units
#pragma unroll
  for (int q = 0; q < OZ_K / 16; q++)
#pragma unroll
    for (int i = 0; i < OZ_S; i++) {
      const int nj = OZ_S < OZ_S + 1 - i ? OZ_S : OZ_S + 1 - i;  // digits j = 0 .. nj - 1 of B: groups i .. i + nj - 1 <= 7
      const bool first = FRESH && q == 0;
#pragma unroll
      for (int j = 0; j < OZ_S; j++) {
        // runs of up to four digits; group 7's first product (i = 1, j = 6) starts it, the groups beside it go on
        const bool alone = first && i == 1 && j == 6;
        if (j < nj && (j == 0 || j == 4 || alone)) {
          const int end = (first && i == 1 && j < 6) ? 6 : nj;
          const int w = end - j < 4 ? end - j : 4;
          oz_mma(tmem + (i + j) * OZ_N, da + ((q * 2 * OZ_A_LBO + i * OZ_A_DIGIT) >> 4),
                 db + ((q * 2 * OZ_B_LBO + j * OZ_B_DIGIT) >> 4), w * OZ_N, !(first && (i == 0 || alone)));
        }
      }
    }
}

// One tile: rows i0 .. i0 + 127 of op(A) times columns j0 .. j0 + 63 of op(B).
// P: rows(), cols() (sizes of the result), ksteps() (buffers of OZ_K entries),
//    contiguousA(), contiguousB(): whether neighbours in K are neighbours in memory,
//    expA(i), expB(j): largest exponents of a row of A, a column of B (in range),
//    loadA(i, s, k, v[8]), loadB(j, s, k, v[4]): entries k .. k + 7 (k + 3) of buffer s of a
//    row / column in range (zeros past the end of K),
//    store(i, j, x): result entry in range,
//    timeout(): a wait gave up; nothing more of the tile is stored.
template <class Prob>
__device__ __forceinline__ void oz_tile(const Prob& P, int i0, int j0, unsigned char* smem) {
  int* eA = reinterpret_cast<int*>(smem + 2 * OZ_STAGE);
  int* eB = eA + OZ_M;
  uint64_t* bars = reinterpret_cast<uint64_t*>(eB + OZ_N);
  uint32_t* tptr = reinterpret_cast<uint32_t*>(bars + 2);
  const int tid = threadIdx.x, warp = tid >> 5;
  const bool worker = warp < 16;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(oz_smem(tptr)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(oz_smem(bars)) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(oz_smem(bars + 1)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < OZ_M) eA[tid] = (i0 + tid < P.rows()) ? P.expA(i0 + tid) : 1;
  if (tid >= OZ_M && tid < OZ_M + OZ_N) eB[tid - OZ_M] = (j0 + tid - OZ_M < P.cols()) ? P.expB(j0 + tid - OZ_M) : 1;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tptr);

  const int steps = P.ksteps();
  // this thread's entries: 8 ka .. 8 ka + 7 of row ra of A, 4 kb .. 4 kb + 3 of column rb of B;
  // neighbouring lanes go along the contiguous direction
  const bool ca = P.contiguousA(), cb = P.contiguousB();
  const int ra = ca ? (tid >> 2) & 127 : tid & 127, ka = ca ? tid & 3 : (tid >> 7) & 3;
  const int rb = cb ? (tid >> 3) & 63 : tid & 63, kb = cb ? tid & 7 : (tid >> 6) & 7;
  const bool inA = worker && i0 + ra < P.rows(), inB = worker && j0 + rb < P.cols();
  double va[8], vb[4];
#pragma unroll
  for (int u = 0; u < 8; u++) va[u] = 0.0;
#pragma unroll
  for (int u = 0; u < 4; u++) vb[u] = 0.0;
  auto fetch = [&](int s) {
    if (inA) P.loadA(i0 + ra, s, 8 * ka, va);
    if (inB) P.loadB(j0 + rb, s, 4 * kb, vb);
  };
  // digits of two neighbouring entries of K, one fp16 pair per digit
  auto cut = [](double x0, double x1, int e, uint32_t (&d)[OZ_S]) {
    const unsigned long long y0 = oz_fixed(x0, e), y1 = oz_fixed(x1, e);
    const uint32_t l0 = (uint32_t)y0, h0 = (uint32_t)(y0 >> 32), l1 = (uint32_t)y1, h1 = (uint32_t)(y1 >> 32);
    auto pack = [](uint32_t x, uint32_t mask, uint32_t mid) {  // fp16 1024 + field, less the middle: exact
      const uint32_t w = (x & mask) | 0x64006400u;
      const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&w), *reinterpret_cast<const __half2*>(&mid));
      return *reinterpret_cast<const uint32_t*>(&r);
    };
    constexpr uint32_t MID = 0x64806480u, MID0 = 0x66006600u;  // 1152, 1536
    d[0] = pack(__byte_perm(h0, h1, 0x7632), 0x03ff03ffu, MID0);
    d[1] = pack(__byte_perm(h0, h1, 0x0501), 0x00ff00ffu, MID);
    d[2] = pack(__byte_perm(h0, h1, 0x0400), 0x00ff00ffu, MID);
    d[3] = pack(__byte_perm(l0, l1, 0x0703), 0x00ff00ffu, MID);
    d[4] = pack(__byte_perm(l0, l1, 0x0602), 0x00ff00ffu, MID);
    d[5] = pack(__byte_perm(l0, l1, 0x0501), 0x00ff00ffu, MID);
    d[6] = pack(__byte_perm(l0, l1, 0x0400), 0x00ff00ffu, MID);
  };

  // columns 16 (warp / 4) + c of row 32 (warp % 4) + lane: sum 2^80 + frac 2^48
  long long sum[16];
  uint32_t frac[16];
#pragma unroll
  for (int c = 0; c < 16; c++) {
    sum[c] = 0;
    frac[c] = 0;
  }
  const uint32_t tlane = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * 16;
  auto drain = [&]() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int c0 = 0; c0 < 16; c0 += 4) {
      uint32_t r[8][4];
#pragma unroll
      for (int g = 0; g < 8; g++)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[g][0]), "=r"(r[g][1]), "=r"(r[g][2]), "=r"(r[g][3])
                     : "r"(tlane + g * OZ_N + c0));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int c = 0; c < 4; c++) {
        int v[8];
#pragma unroll
        for (int g = 0; g < 8; g++) v[g] = __float2int_rn(__uint_as_float(r[g][c]));
        long long hi = (long long)v[1] * 256 + v[2];
        hi += (long long)v[0] * 65536;
        long long lo = (long long)v[6] * 256 + v[7];
        lo += (long long)v[5] * 65536;
        lo += (long long)v[4] * (1 << 24);
        lo += (long long)v[3] << 32;
        const long long t = ((lo + 128) >> 8) + frac[c0 + c];
        frac[c0 + c] = (uint32_t)t;
        sum[c0 + c] += hi + (t >> 32);
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  };

  bool ok = true;
  int uses[2] = {0, 0};
  fetch(0);
  for (int s = 0; s < steps && ok; s++) {
    const int w = s & 1;
    unsigned char* sa = smem + w * OZ_STAGE;
    unsigned char* sb = sa + OZ_A_BYTES;
    // the buffer's previous MMAs have read it
    const bool fresh = (s % (OZ_CHUNK / OZ_K)) == 0;
    if (worker) {
      if (uses[w] > 0) ok = oz_wait(oz_smem(bars + w), (uses[w] - 1) & 1);
      {  // A: one 16-byte row of a core matrix per digit
        uint32_t d[4][OZ_S];
        const int e = eA[ra];
#pragma unroll
        for (int u = 0; u < 4; u++) cut(va[2 * u], va[2 * u + 1], e, d[u]);
        unsigned char* dst = sa + ka * OZ_A_LBO + ra * 16;
#pragma unroll
        for (int i = 0; i < OZ_S; i++)
          *reinterpret_cast<uint4*>(dst + i * OZ_A_DIGIT) = make_uint4(d[0][i], d[1][i], d[2][i], d[3][i]);
      }
      {  // B: half a row
        uint32_t d[2][OZ_S];
        const int e = eB[rb];
#pragma unroll
        for (int u = 0; u < 2; u++) cut(vb[2 * u], vb[2 * u + 1], e, d[u]);
        unsigned char* dst = sb + (kb >> 1) * OZ_B_LBO + rb * 16 + (kb & 1) * 8;
#pragma unroll
        for (int i = 0; i < OZ_S; i++)
          *reinterpret_cast<uint2*>(dst + i * OZ_B_DIGIT) = make_uint2(d[0][i], d[1][i]);
      }
      if (s + 1 < steps) fetch(s + 1);
      if (fresh && s > 0) {  // the previous sum is complete: join it before its accumulators start over
        ok = __all_sync(0xffffffffu, ok && oz_wait(oz_smem(bars + (w ^ 1)), (uses[w ^ 1] - 1) & 1));
        if (ok) drain();
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    ok = __syncthreads_and(ok);
    if (!ok) break;
    if (tid == 512) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (fresh)
        oz_issue<true>(tmem, oz_smem(sa), oz_smem(sb));
      else
        oz_issue<false>(tmem, oz_smem(sa), oz_smem(sb));
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       oz_smem(bars + w))
                   : "memory");
    }
    uses[w]++;
  }
  if (ok && steps > 0 && worker) {
    const int w = (steps - 1) & 1;
    ok = __all_sync(0xffffffffu, oz_wait(oz_smem(bars + w), (uses[w] - 1) & 1));
    if (ok) drain();
  }
  if (!__syncthreads_and(ok)) {  // a wait gave up: what was issued ends before its memory is given back
    ok = false;
    for (int w = 0; w < 2; w++)
      if (uses[w] > 0) oz_wait(oz_smem(bars + w), (uses[w] - 1) & 1);
    __syncthreads();
  }
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  if (!ok) {
    if (tid == 0) P.timeout();
    return;
  }
  if (!worker) return;
  const int row = (warp & 3) * 32 + (tid & 31);
  if (i0 + row >= P.rows()) return;
  const int ea = eA[row];
#pragma unroll
  for (int c = 0; c < 16; c++) {
    const int col = (warp >> 2) * 16 + c;
    if (j0 + col < P.cols()) {
      const int eb = eB[col];
      // the leading 64 bits of the sum; value = sum 2^80 2^(ea - 1078 + eb - 1078)
      const int up = min(__clzll(sum[c] < 0 ? ~sum[c] : sum[c]) - 1, 32);
      const long long v = (sum[c] << up) + (long long)(((unsigned long long)frac[c] << up) >> 32);
      const double x = (ea == 2047 || eb == 2047) ? __longlong_as_double(0x7ff8000000000000LL)
                                                  : oz_double(v, ea + eb - 2156 + 80 - up);
      P.store(i0 + row, j0 + col, x);
    }
  }
}

}  // namespace skew
