// sep_ozaki_split.cuh -- the digit split of sep_ozaki.cuh as device functions,
// for the kernels that write an operand's digit planes.
#pragma once

#include <cstdint>

#include "sep_ozaki.cuh"

namespace sep {
namespace oz {

// biased FP64 exponent field of x (0 for zero and denormals)
__device__ __forceinline__ int exp_field(double x) {
  return (int)((__double_as_longlong(x) >> 52) & 0x7FF);
}

// scale exponent of a row whose largest exponent field is ex: |x| < 2^e
__host__ __device__ constexpr int scale_of(int ex_max) { return ex_max - 1022; }

// x 2^(B-e) rounded to an integer, B = 55 bits in 7 digits (|X| <= 2^55) or 62 in
// 8 (|X| <= 2^62); integer operations only
template <int S> __device__ __forceinline__ long long fixed_point(double x, int e) {
  static_assert(S == kSlices || S == kBatchSlices, "bits of the fixed point");
  constexpr int bits_of_x = S == kSlices ? 55 : 62;
  const long long bits = __double_as_longlong(x);
  const int ex = (int)((bits >> 52) & 0x7FF);
  long long X = 0;
  if (ex != 0) {
    const long long m = (bits & 0xFFFFFFFFFFFFFLL) | (1LL << 52);
    const int sh = 1075 - bits_of_x + e - ex;  // X = m 2^-sh, sh >= 53 - 1 - bits_of_x
    if (sh <= 0)
      X = m << (-sh);
    else if (sh < 62)
      X = (m + (1LL << (sh - 1))) >> sh;
    if (bits < 0) X = -X;
  }
  return X;
}

// X split into S balanced base-256 digits, most significant first
template <int S> __device__ __forceinline__ void digits(long long X, int (&d)[S]) {
#pragma unroll
  for (int s = 0; s < S - 1; ++s) {
    const int w = 8 * (S - 1 - s);
    const long long q = (X + (1LL << (w - 1))) >> w;
    d[s] = (int)q;
    X -= q << w;
  }
  d[S - 1] = (int)X;
}

__device__ __forceinline__ uint32_t bf16_pair(int lo, int hi) {
  return (__float_as_uint((float)lo) >> 16) | (__float_as_uint((float)hi) & 0xFFFF0000u);
}

// element offset of (row block rb, K chunk kc, slice s) + position (rr, kk) in it
template <int S = kSlices>
__device__ __forceinline__ long long plane_off(int s, long long kc, long long rb, long long nkc,
                                               long long nrb, int rr, int kk) {
  (void)nrb;
  return (rb * nkc + kc) * block_elems(S) + ((s * 16 + (rr >> 3)) * 2 + (kk >> 3)) * 64 +
         (rr & 7) * 8 + (kk & 7);
}

// eight consecutive K values of one row -> S 16-byte stores
template <int S = kSlices>
__device__ __forceinline__ void store_digits8(const double (&x)[8], int e, uint16_t* planes,
                                              long long kc, long long rb, long long nkc,
                                              long long nrb, int rr, int k0) {
  int d[8][S];
#pragma unroll
  for (int i = 0; i < 8; ++i) digits<S>(fixed_point<S>(x[i], e), d[i]);
#pragma unroll
  for (int s = 0; s < S; ++s) {
    uint4 v;
    v.x = bf16_pair(d[0][s], d[1][s]);
    v.y = bf16_pair(d[2][s], d[3][s]);
    v.z = bf16_pair(d[4][s], d[5][s]);
    v.w = bf16_pair(d[6][s], d[7][s]);
    *reinterpret_cast<uint4*>(planes + plane_off<S>(s, kc, rb, nkc, nrb, rr, k0)) = v;
  }
}

// v 2^k without overflow of the intermediate power (k = ea + eb - 38)
__device__ __forceinline__ double pow2i(int k) {
  return (k < -1022) ? 0.0 : __longlong_as_double((long long)(k + 1023) << 52);
}
__device__ __forceinline__ double scale2(double v, int k) {
  const int k1 = k / 2;
  return v * pow2i(k1) * pow2i(k - k1);
}

// h 2^32 + l rounded to the nearest double (ties to even), by integer operations
__device__ __forceinline__ double round_sum(long long h, long long l) {
  h += l >> 32;
  uint32_t lo = (uint32_t)l;  // the value is h 2^32 + lo
  const bool neg = h < 0;
  if (neg) {
    h = -h - (lo != 0u);
    lo = 0u - lo;
  }
  unsigned long long m;  // the leading 64 bits; lost: some bit below them is set
  int top;               // exponent of the leading bit
  bool lost = false;
  if (h != 0) {
    const int z = __clzll(h);  // >= 1
    m = ((unsigned long long)h << z) | (((unsigned long long)lo << 32) >> (64 - z));
    lost = z < 32 && (lo << z) != 0u;
    top = 95 - z;
  } else {
    if (lo == 0u) return 0.0;
    const int z = __clz((int)lo);
    m = (unsigned long long)lo << (32 + z);
    top = 31 - z;
  }
  const unsigned rest = (unsigned)m & 0x7FFu;
  unsigned long long r = m >> 11;  // 53 bits
  r += rest > 0x400u || (rest == 0x400u && (lost || (r & 1)));
  // r's leading bit adds one to the exponent field
  const unsigned long long bits = ((unsigned long long)(top + 1022) << 52) + r;
  return __longlong_as_double((long long)(bits | (neg ? 1ULL << 63 : 0ULL)));
}

// d 2^e: the scale is added to the exponent field while the result stays normal
__device__ __forceinline__ double scaled(double d, int e) {
  const long long bits = __double_as_longlong(d);
  const int ex = (int)((bits >> 52) & 0x7FF);
  if (ex == 0) return d;  // a sum of integers: zero
  if (ex + e > 0 && ex + e < 0x7FF) return __longlong_as_double(bits + ((long long)e << 52));
  return scale2(d, e);
}

}  // namespace oz
}  // namespace sep
