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
__device__ __forceinline__ int scale_of(int ex_max) { return ex_max - 1022; }

// x 2^(55-e) rounded to an integer (|X| <= 2^55), split into kSlices balanced
// base-256 digits, most significant first; integer operations only
__device__ __forceinline__ void split7(double x, int e, int (&d)[kSlices]) {
  const long long bits = __double_as_longlong(x);
  const int ex = (int)((bits >> 52) & 0x7FF);
  long long X = 0;
  if (ex != 0) {
    const long long m = (bits & 0xFFFFFFFFFFFFFLL) | (1LL << 52);
    const int sh = 1020 + e - ex;  // X = m 2^-sh, sh >= -2
    if (sh <= 0)
      X = m << (-sh);
    else if (sh < 62)
      X = (m + (1LL << (sh - 1))) >> sh;
    if (bits < 0) X = -X;
  }
#pragma unroll
  for (int s = 0; s < kSlices - 1; ++s) {
    const int w = 8 * (kSlices - 1 - s);
    const long long q = (X + (1LL << (w - 1))) >> w;
    d[s] = (int)q;
    X -= q << w;
  }
  d[kSlices - 1] = (int)X;
}

__device__ __forceinline__ uint32_t bf16_pair(int lo, int hi) {
  return (__float_as_uint((float)lo) >> 16) | (__float_as_uint((float)hi) & 0xFFFF0000u);
}

// element offset of (row block rb, K chunk kc, slice s) + position (rr, kk) in it
__device__ __forceinline__ long long plane_off(int s, long long kc, long long rb, long long nkc,
                                               long long nrb, int rr, int kk) {
  (void)nrb;
  return (rb * nkc + kc) * kBlockElems + ((s * 16 + (rr >> 3)) * 2 + (kk >> 3)) * 64 +
         (rr & 7) * 8 + (kk & 7);
}

// eight consecutive K values of one row -> kSlices 16-byte stores
__device__ __forceinline__ void store_digits8(const double (&x)[8], int e, uint16_t* planes,
                                              long long kc, long long rb, long long nkc,
                                              long long nrb, int rr, int k0) {
  int d[8][kSlices];
#pragma unroll
  for (int i = 0; i < 8; ++i) split7(x[i], e, d[i]);
#pragma unroll
  for (int s = 0; s < kSlices; ++s) {
    uint4 v;
    v.x = bf16_pair(d[0][s], d[1][s]);
    v.y = bf16_pair(d[2][s], d[3][s]);
    v.z = bf16_pair(d[4][s], d[5][s]);
    v.w = bf16_pair(d[6][s], d[7][s]);
    *reinterpret_cast<uint4*>(planes + plane_off(s, kc, rb, nkc, nrb, rr, k0)) = v;
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

// the value of a batched product's integer sum (gemm_nt_batched), e = the two
// rows' scale exponents - 38 - batch_shift: one FP64 conversion, the scale added
// to the exponent field while the result stays normal
__device__ __forceinline__ double sum_value(long long v, int e) {
  const double d = (double)v;
  const long long bits = __double_as_longlong(d);
  const int ex = (int)((bits >> 52) & 0x7FF) + e;
  if (v == 0) return 0.0;
  if (ex > 0 && ex < 0x7FF) return __longlong_as_double(bits + ((long long)e << 52));
  return scale2(d, e);
}

}  // namespace oz
}  // namespace sep
