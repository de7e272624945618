// sep_spinor.cu -- the non-local spin-orbit operator of the spinor filter
// (the reference's spinors/filterSpinors/), |psinl> = Vso |psi>, on the GPU.
//
// Spinors are 2 ngrid complex values, the spin-up grid then the spin-down
// grid (filterSpinors/hamiltonian.c:38-44).  Each atom acts on the grid
// points of its neighbour list (nlc_st entries, filterSpinors/fd.h:55-60;
// nl[a] used of nnlc per atom); the atoms' contributions add up.
//
// Gaussian form (filterSpinors/hamiltonian.c:81-190): for each point j1 of an
// atom, six sums over the atom's points j2 of
//   K(j1, j2) conj(Y_m(j2)) psi_s(j2),
//   K = (Vr1 + Vr2)/2 exp(-((r1 - r2) sigma_1)^2) / ((r2_1 + r2_2)/2),
// combined with tmp Y_m(j1), tmp = 0.5 dv / sqrt(2 pi sigma^2).  One CTA per
// atom; the j2 points are staged through shared memory in tiles of 256 with
// conj(Y) psi already formed, so each pair costs one exp and 12 FMAs.  K
// depends on the operator alone: a context that applies it many times keeps
// K(j1, j2) of every atom (k_vso_kernel), and the sums are matrix products on
// the tensor cores (k_vso_x_slice, k_vso_combine) or, for short lists and rows
// that the digits do not cover, 12 FMAs
// per pair (k_vso_stored); there each list point's contribution is stored and
// a grid point sums its own in list order (k_vso_gather).
// Kleinman-Bylander form (filterSpinors/hamiltonian.c:193-401): twelve
// projections per atom (block reduction), scaled by Elkb dv, then spread back
// over the atom's points with the reference's coefficients, term by term.
// Contributions of overlapping atoms are added with atomicAdd in the
// Kleinman-Bylander form and where K is formed in place.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <string>

#include "../../include/sep_gb300.h"
#include "sep_ozaki_split.cuh"
#include "sep_spinor.cuh"

namespace sep {
void set_error(const std::string& msg);
}

namespace {

constexpr int kT = 256;
constexpr double kTwoPi = 6.28318530717958647692;  // filterSpinors/fd.h TWOPI

int fail(int status, const std::string& msg) {
  sep::set_error(msg);
  return status;
}

#define SK(...)                                                                      \
  do {                                                                               \
    cudaError_t _e = (__VA_ARGS__);                                                  \
    if (_e != cudaSuccess) {                                                         \
      char _b[320];                                                                  \
      snprintf(_b, sizeof _b, "CUDA error %d (%s) at sep_spinor.cu:%d", (int)_e,     \
               cudaGetErrorString(_e), __LINE__);                                    \
      return fail(_e == cudaErrorMemoryAllocation ? SEP_ERR_NOMEM : SEP_ERR_CUDA, _b); \
    }                                                                                \
  } while (0)

struct C2 {
  double re, im;
};
__device__ __forceinline__ C2 ld2(const double* p) { return {p[0], p[1]}; }
// conj(y) psi, as the reference forms it (hamiltonian.c:139-140)
__device__ __forceinline__ C2 conj_mul(C2 y, C2 p) {
  return {y.re * p.re + y.im * p.im, y.re * p.im - y.im * p.re};
}
__device__ __forceinline__ C2 mul(C2 a, C2 b) {
  return {a.re * b.re - a.im * b.im, a.im * b.re + a.re * b.im};
}
__device__ __forceinline__ C2 scale(double s, C2 a) { return {s * a.re, s * a.im}; }
__device__ __forceinline__ C2 add(C2 a, C2 b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ C2 sub(C2 a, C2 b) { return {a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ void atomic_add(double* p, C2 v) {
  atomicAdd(p, v.re);
  atomicAdd(p + 1, v.im);
}

// Vso psi at one point from its six sums (hamiltonian.c:167-186)
__device__ __forceinline__ void vso_gauss_point(const sep_nlc& e, double tmp, const C2 (&acc)[6],
                                                C2& up, C2& dn) {
  const double sqrttwo = sqrt(2.0);
  const C2 t11 = scale(tmp, ld2(e.y11)), t10 = scale(tmp, ld2(e.y10)),
           t1_1 = scale(tmp, ld2(e.y1_1));
  up = add(sub(mul(t11, acc[0]), mul(t1_1, acc[2])),
           scale(sqrttwo, add(mul(t10, acc[3]), mul(t1_1, acc[4]))));
  dn = add(sub(scale(-1.0, mul(t11, acc[3])), mul(t1_1, acc[5])),
           scale(sqrttwo, add(mul(t10, acc[2]), mul(t11, acc[1]))));
}

// sums index: 0 y11 up, 1 y10 up, 2 y1_1 up, 3 y11 dn, 4 y10 dn, 5 y1_1 dn
// grid: x = atom, y = spinor of the batch (spinors 4 ngrid doubles apart)
__global__ void __launch_bounds__(kT) k_vso_gauss(const double* __restrict__ psi, long ngrid,
                                                  long nnlc, const sep_nlc* __restrict__ nlc,
                                                  const long* __restrict__ nl, double tmp,
                                                  double sigma_1, double* __restrict__ out) {
  __shared__ double sr[kT], sr2[kT], svr[kT];
  __shared__ C2 sx[6][kT];
  const long a = blockIdx.x;
  psi += (size_t)blockIdx.y * 4 * (size_t)ngrid;
  out += (size_t)blockIdx.y * 4 * (size_t)ngrid;
  const long n = nl[a];
  const sep_nlc* base = nlc + a * nnlc;
  const int tid = threadIdx.x;
  for (long j1b = 0; j1b < n; j1b += kT) {
    const long j1 = j1b + tid;
    const bool act = j1 < n;
    double r1 = 0.0, r21 = 1.0, vr1 = 0.0;
    if (act) {
      r1 = base[j1].r;
      r21 = base[j1].r2;
      vr1 = base[j1].Vr;
    }
    C2 acc[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) acc[m] = {0.0, 0.0};
    for (long t0 = 0; t0 < n; t0 += kT) {
      __syncthreads();
      const long j2 = t0 + tid;
      if (j2 < n) {
        const sep_nlc& e = base[j2];
        const C2 up = ld2(psi + 2 * e.jxyz), dn = ld2(psi + 2 * (ngrid + e.jxyz));
        const C2 y11 = ld2(e.y11), y10 = ld2(e.y10), y1_1 = ld2(e.y1_1);
        sr[tid] = e.r;
        sr2[tid] = e.r2;
        svr[tid] = e.Vr;
        sx[0][tid] = conj_mul(y11, up);
        sx[1][tid] = conj_mul(y10, up);
        sx[2][tid] = conj_mul(y1_1, up);
        sx[3][tid] = conj_mul(y11, dn);
        sx[4][tid] = conj_mul(y10, dn);
        sx[5][tid] = conj_mul(y1_1, dn);
      }
      __syncthreads();
      if (act) {
        const int cnt = (int)((n - t0) < kT ? (n - t0) : kT);
        for (int jj = 0; jj < cnt; ++jj) {
          const double d = (r1 - sr[jj]) * sigma_1;
          const double k = 0.5 * (vr1 + svr[jj]) * exp(-(d * d)) / (0.5 * (r21 + sr2[jj]));
#pragma unroll
          for (int m = 0; m < 6; ++m) {
            acc[m].re += k * sx[m][jj].re;
            acc[m].im += k * sx[m][jj].im;
          }
        }
      }
    }
    if (act) {
      C2 up, dn;
      vso_gauss_point(base[j1], tmp, acc, up, dn);
      atomic_add(out + 2 * base[j1].jxyz, up);
      atomic_add(out + 2 * (ngrid + base[j1].jxyz), dn);
    }
  }
}

// K(j1, j2) of every atom, km[(a nmax + j2) ld + j1], by the expression of
// k_vso_gauss: once per operator
__global__ void __launch_bounds__(kT) k_vso_kernel(long nnlc, const sep_nlc* __restrict__ nlc,
                                                   const long* __restrict__ nl, double sigma_1,
                                                   long nmax, long ld, double* __restrict__ km) {
  const long a = blockIdx.x, n = nl[a];
  const sep_nlc* base = nlc + a * nnlc;
  const long j1 = (long)blockIdx.y * kT + threadIdx.x;
  if (j1 >= n) return;
  const double r1 = base[j1].r, r21 = base[j1].r2, vr1 = base[j1].Vr;
  double* col = km + (size_t)a * nmax * ld + j1;
  for (long j2 = 0; j2 < n; ++j2) {
    const double d = (r1 - base[j2].r) * sigma_1;
    col[(size_t)j2 * ld] =
        0.5 * (vr1 + base[j2].Vr) * exp(-(d * d)) / (0.5 * (r21 + base[j2].r2));
  }
}

// The six sums of point j1 of a list of n points (act: there is one), with K read
// back: FP64 FMAs over tiles of kTS points, which the block's kTS threads share.
constexpr int kTS = 64;
__device__ __forceinline__ void vso_stored_sums(const double* __restrict__ psi, long ngrid,
                                                const sep_nlc* __restrict__ base, long n,
                                                const double* __restrict__ kc, long ld, bool act,
                                                C2 (&sx)[kTS][6], C2 (&acc)[6]) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int m = 0; m < 6; ++m) acc[m] = {0.0, 0.0};
  for (long t0 = 0; t0 < n; t0 += kTS) {
    __syncthreads();
    const long j2 = t0 + tid;
    if (j2 < n) {
      const sep_nlc& e = base[j2];
      const C2 up = ld2(psi + 2 * e.jxyz), dn = ld2(psi + 2 * (ngrid + e.jxyz));
      const C2 y11 = ld2(e.y11), y10 = ld2(e.y10), y1_1 = ld2(e.y1_1);
      sx[tid][0] = conj_mul(y11, up);
      sx[tid][1] = conj_mul(y10, up);
      sx[tid][2] = conj_mul(y1_1, up);
      sx[tid][3] = conj_mul(y11, dn);
      sx[tid][4] = conj_mul(y10, dn);
      sx[tid][5] = conj_mul(y1_1, dn);
    }
    __syncthreads();
    if (act) {
      const int cnt = (int)((n - t0) < kTS ? (n - t0) : kTS);
#pragma unroll 4
      for (int jj = 0; jj < cnt; ++jj) {
        const double k = kc[(size_t)(t0 + jj) * ld];
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          acc[m].re += k * sx[jj][m].re;
          acc[m].im += k * sx[jj][m].im;
        }
      }
    }
  }
}

// The Gaussian form with K read back: block (atom, 64 points j1, spinor).  For
// operators whose lists are too short for the tensor cores (VsoTensor::pays), and
// where those are switched off or K has a value that is not finite.
// Bound by the FP64 pipe: 12 FMAs per pair and spinor, where forming K costs
// about 45 more FP64 operations.  Two warps a block, so that the points of an
// atom spread over several SMs (one block per atom and spinor left most of
// them with one or two blocks).  64 atoms x 340 points,
// 4 spinors: 0.73 ms (12 FMAs per pair at the pipe's rate: 0.57 ms), 2.83 ms
// forming K in place; K itself 0.79 ms once.
__global__ void __launch_bounds__(kTS)
    k_vso_stored(const double* __restrict__ psi, long ngrid, long nnlc,
                 const sep_nlc* __restrict__ nlc, const long* __restrict__ nl,
                 const double* __restrict__ km, long nmax, long ld, double tmp,
                 double2* __restrict__ contrib) {
  __shared__ C2 sx[kTS][6];
  const long a = blockIdx.x, n = nl[a];
  if ((long)blockIdx.y * kTS >= n) return;
  psi += (size_t)blockIdx.z * 4 * (size_t)ngrid;
  contrib += (size_t)blockIdx.z * 2 * (size_t)gridDim.x * (size_t)nmax;
  const sep_nlc* base = nlc + a * nnlc;
  const long j1 = (long)blockIdx.y * kTS + threadIdx.x;
  const bool act = j1 < n;
  C2 acc[6];
  vso_stored_sums(psi, ngrid, base, n, km + (size_t)a * nmax * ld + j1, ld, act, sx, acc);
  if (act) {
    C2 up, dn;
    vso_gauss_point(base[j1], tmp, acc, up, dn);
    double2* o = contrib + 2 * ((size_t)a * nmax + j1);
    o[0] = make_double2(up.re, up.im);
    o[1] = make_double2(dn.re, dn.im);
  }
}

// ---- the sums on the tensor cores -----------------------------------------
// Per atom the sums are a matrix product, (K: n x n) times (conj(Y) psi: n x
// 12 per spinor, the real and imaginary parts of the six products), done for
// all atoms at once by the batched contraction of sep_ozaki.cu: K's digit
// planes are kept with the operator, the products' are written per apply.
// Accuracy: a term's error is below 2^-60 of the product of the largest K of its
// row and the largest of its product over the list, so a row's sums are no worse
// than by FP64 FMAs unless every one of its terms lies far below that product:
// K grows towards the atom, so that is where psi falls towards it by orders of
// magnitude.  vso_row_covered finds such rows, and they take the FP64 sums.
// 64 atoms x 340 points, 4 spinors, with cold caches: digits of the products 26 us,
// contraction 74 (two waves of tiles, K's digits read once: 138 MB),
// contributions 17, gather 11, where the FMAs take 736 us.
// scale exponent of every row of every K (mpad rows per atom); *bad: some
// value is not finite
__global__ void k_vso_k_expo(const long* __restrict__ nl, const double* __restrict__ km,
                             long nmax, long ld, long mpad, int* __restrict__ expo,
                             int* __restrict__ bad) {
  const long a = blockIdx.x / mpad, j1 = blockIdx.x % mpad, n = nl[a];
  int mx = 0;
  if (j1 < n)  // K is symmetric
    for (long j2 = threadIdx.x; j2 < n; j2 += 32)
      mx = max(mx, sep::oz::exp_field(km[((size_t)a * nmax + j1) * ld + j2]));
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (threadIdx.x == 0) {
    expo[blockIdx.x] = j1 < n ? sep::oz::scale_of(mx) : 0;
    if (mx == 0x7ff) *bad = 1;
  }
}

// the four largest values of every row of every K: columns and exponent fields
__global__ void __launch_bounds__(kTS)
    k_vso_k_top(const long* __restrict__ nl, const double* __restrict__ km, long nmax, long ld,
                long mpad, int4* __restrict__ top, ushort4* __restrict__ top_exp) {
  const long a = blockIdx.x, n = nl[a], j1 = (long)blockIdx.y * kTS + threadIdx.x;
  if (j1 >= n) return;
  const double* col = km + (size_t)a * nmax * ld + j1;
  unsigned long long v[4] = {};  // the bits of |K| order as |K| does
  int at[4] = {};
  for (long j2 = 0; j2 < n; ++j2) {
    unsigned long long x = (unsigned long long)__double_as_longlong(col[(size_t)j2 * ld]) << 1 >> 1;
    int c = (int)j2;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (x > v[q]) {
        const unsigned long long y = v[q];
        const int d = at[q];
        v[q] = x;
        at[q] = c;
        x = y;
        c = d;
      }
  }
  top[a * mpad + j1] = make_int4(at[0], at[1], at[2], at[3]);
  top_exp[a * mpad + j1] =
      make_ushort4((unsigned short)(v[0] >> 52), (unsigned short)(v[1] >> 52),
                   (unsigned short)(v[2] >> 52), (unsigned short)(v[3] >> 52));
}

// digit planes of every K: block (16 values of j2, 128 rows)
constexpr int kSliceT = sep::oz::kBlockRows * sep::oz::kChunkK / 8;
__global__ void __launch_bounds__(kSliceT)
    k_vso_k_slice(const long* __restrict__ nl, const double* __restrict__ km, long nmax, long ld,
                  long mb, const int* __restrict__ expo, uint16_t* __restrict__ planes,
                  long nkc) {
  const long kc = blockIdx.x, rb = blockIdx.y, a = rb / mb, n = nl[a];
  const int rr = threadIdx.x / 2, k0 = threadIdx.x % 2 * 8;
  const long j1 = rb % mb * sep::oz::kBlockRows + rr, j2 = kc * sep::oz::kChunkK + k0;
  double x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
    x[i] = j1 < n && j2 + i < n ? km[((size_t)a * nmax + j1) * ld + j2 + i] : 0.0;
  sep::oz::store_digits8<sep::oz::kBatchSlices>(x, expo[rb * sep::oz::kBlockRows + rr], planes, kc,
                                                rb, nkc, 0, rr, k0);
}

// product m of a list point, in the order of the sums above
__device__ __forceinline__ C2 vso_product(const double* __restrict__ psi, long ngrid,
                                          const sep_nlc& e, int m) {
  const C2 p = ld2(psi + 2 * (m < 3 ? e.jxyz : ngrid + e.jxyz));
  const int q = m % 3;
  return conj_mul(ld2(q == 0 ? e.y11 : q == 1 ? e.y10 : e.y1_1), p);
}

// exponents and digit planes of the products: block (atom, spinor) writes the
// 12 rows 12 s .. of the atom's nb row blocks, zero from the list's end to the
// last chunk's, and the exponent field of every product (xe, `most` spinors per
// atom).  A thread takes one product of eight points; where that covers
// the list (up to 672 points) they stay in registers between the exponents and
// the digits, beyond it they are formed again.
constexpr int kSliceX = 512;
__global__ void __launch_bounds__(kSliceX)
    k_vso_x_slice(const double* __restrict__ psi, long ngrid, long nnlc,
                  const sep_nlc* __restrict__ nlc, const long* __restrict__ nl, long nb, long nkc,
                  long most, int* __restrict__ expo, uint16_t* __restrict__ xe,
                  uint16_t* __restrict__ planes) {
  __shared__ int top[12];
  const long a = blockIdx.x, n = nl[a];
  const int row0 = 12 * blockIdx.y, nt = blockDim.x;
  psi += (size_t)blockIdx.y * 4 * (size_t)ngrid;
  xe += ((size_t)a * most + blockIdx.y) * (size_t)nkc * sep::oz::kChunkK * 8;
  const sep_nlc* base = nlc + a * nnlc;
  if (threadIdx.x < 12) top[threadIdx.x] = 0;
  __syncthreads();
  const int groups = (int)nkc * (sep::oz::kChunkK / 8), items = 6 * groups;
  double x[8], y[8];
  auto form = [&](int t) {
    const int m = t / groups;
    const long j0 = 8 * (t - m * groups);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      C2 v = {0.0, 0.0};
      if (j0 + i < n) v = vso_product(psi, ngrid, base[j0 + i], m);
      x[i] = v.re;
      y[i] = v.im;
    }
    return m;
  };
  for (int t = threadIdx.x; t < items; t += nt) {
    const int m = form(t);
    int ex = 0, ey = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int fx = sep::oz::exp_field(x[i]), fy = sep::oz::exp_field(y[i]);
      ex = max(ex, fx);
      ey = max(ey, fy);
      xe[(8 * (t - m * groups) + i) * 8 + m] = (uint16_t)max(fx, fy);
    }
    atomicMax(&top[2 * m], ex);
    atomicMax(&top[2 * m + 1], ey);
  }
  __syncthreads();
  if (threadIdx.x < 12)
    expo[a * nb * sep::oz::kBlockRows + row0 + threadIdx.x] = sep::oz::scale_of(top[threadIdx.x]);
  for (int t = threadIdx.x; t < items; t += nt) {
    if (items > nt) form(t);
    const int m = t / groups, g = t - m * groups;
    const int r = row0 + 2 * m;  // even: both rows are in one block
    const long rb = a * nb + r / sep::oz::kBlockRows;
    const int rr = r % sep::oz::kBlockRows;
    constexpr int kS = sep::oz::kBatchSlices;
    sep::oz::store_digits8<kS>(x, sep::oz::scale_of(top[2 * m]), planes, g / 2, rb, nkc, 0, rr,
                               g % 2 * 8);
    sep::oz::store_digits8<kS>(y, sep::oz::scale_of(top[2 * m + 1]), planes, g / 2, rb, nkc, 0,
                               rr + 1, g % 2 * 8);
  }
}

// whether the digits hold the terms of a row (K's scale exponent ea) well enough:
// for either component (products 0-2, 3-5; eb: their scale exponents) one of the
// terms of the row's four largest K is at least 2^-kCover of the bound 2^(ea +
// eb) that the digits' error is measured by, or the component is zero.
// Error of Vso psi against extended precision, relative to the sum of the
// absolute values added up, root mean square over a list of 590 points (FP64
// FMAs): normally distributed psi 6e-18 (1.8e-17), constant 4e-18 (2.6e-17), psi
// falling by nine decades away from the atom 6e-17 (8e-17), by three towards it
// 4.9e-18 (6.9e-18, some rows not covered), by nine towards it the FP64 sums for
// every row.  With kCover 8 a point of the fourth erred by 1.6 times the FP64
// sums' worst; without the test a list near a grid point errs by 1e-9.
constexpr int kCover = 6;
__device__ __forceinline__ bool vso_row_covered(const uint16_t* __restrict__ xe, int4 at, ushort4 k,
                                                int ea, const int* __restrict__ eb) {
  constexpr int zero = sep::oz::scale_of(0);
  if (ea == zero) return true;
  const int col[4] = {at.x, at.y, at.z, at.w};
  const int kf[4] = {k.x, k.y, k.z, k.w};
  int best[2] = {-4096, -4096};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 f = *reinterpret_cast<const uint4*>(xe + (size_t)col[q] * 8);
    const int x[2] = {(int)max(max(f.x & 0xFFFFu, f.x >> 16), f.y & 0xFFFFu),
                      (int)max(max(f.y >> 16, f.z & 0xFFFFu), f.z >> 16)};
#pragma unroll
    for (int c = 0; c < 2; ++c)
      if (x[c] > 0 && kf[q] > 0) best[c] = max(best[c], x[c] + kf[q] - 2044);
  }
  bool ok = true;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    int e = eb[6 * c];
#pragma unroll
    for (int m = 1; m < 6; ++m) e = max(e, eb[6 * c + m]);
    ok = ok && (e == zero || best[c] >= ea + e - kCover);
  }
  return ok;
}

// contributions from the sums: block (atom, 64 points j, spinor s); sums[(a mpad
// + j) ldc + 12 s + 2 m] (re, im), scaled by the exponents of K's row and of the
// product's.  Products with an infinite or NaN value have no digits: an (atom,
// spinor) that holds one takes the FP64 sums, which pass it on, and so do the
// rows whose terms the digits do not cover.
__global__ void __launch_bounds__(kTS)
    k_vso_combine(const double* __restrict__ sums, const int* __restrict__ ea,
                  const int* __restrict__ eb, long xpad, const int4* __restrict__ top,
                  const ushort4* __restrict__ top_exp, const uint16_t* __restrict__ xe,
                  long xe_spinor, long most, long ldc, long mpad, const double* __restrict__ psi,
                  long ngrid, long nnlc, const sep_nlc* __restrict__ nlc,
                  const long* __restrict__ nl, const double* __restrict__ km, long nmax, long ld,
                  double tmp, double2* __restrict__ contrib) {
  __shared__ C2 sx[kTS][6];
  const long a = blockIdx.x, n = nl[a];
  if ((long)blockIdx.y * kTS >= n) return;
  const sep_nlc* base = nlc + a * nnlc;
  const long j = (long)blockIdx.y * kTS + threadIdx.x;
  const bool act = j < n;
  eb += a * xpad + 12 * blockIdx.z;
  xe += ((size_t)a * most + blockIdx.z) * (size_t)xe_spinor;
  bool ok = true;
#pragma unroll
  for (int m = 0; m < 12; ++m) ok = ok && eb[m] != sep::oz::scale_of(0x7ff);
  const long r = a * mpad + j;
  if (ok && act) ok = vso_row_covered(xe, top[r], top_exp[r], ea[r], eb);
  C2 acc[6];
  if (__syncthreads_or(!ok))
    vso_stored_sums(psi + (size_t)blockIdx.z * 4 * (size_t)ngrid, ngrid, base, n,
                    km + (size_t)a * nmax * ld + j, ld, act, sx, acc);
  if (!act) return;
  if (ok) {
    const double* row = sums + (size_t)r * ldc + 12 * blockIdx.z;
    const int e = ea[r] - sep::oz::kBatchUnit;
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const double2 v = *reinterpret_cast<const double2*>(row + 2 * m);
      acc[m] = {sep::oz::scaled(v.x, e + eb[2 * m]), sep::oz::scaled(v.y, e + eb[2 * m + 1])};
    }
  }
  C2 up, dn;
  vso_gauss_point(base[j], tmp, acc, up, dn);
  double2* o = contrib + 2 * (((size_t)blockIdx.z * gridDim.x + a) * nmax + j);
  o[0] = make_double2(up.re, up.im);
  o[1] = make_double2(dn.re, dn.im);
}

// Vso psi of every grid point from the list points' contributions: point g
// sums the entries idx[off[g]] .. idx[off[g + 1] - 1] (a nmax + j, ascending),
// so the result does not depend on the order in which blocks finish.  Added
// atomically it did: three overlapping atoms change the last bit, and the
// subspace steps keep directions down to 1e-10 of the largest, which turned
// it into 1e-6 of the Ritz values of the states that are not converged.  It
// writes every point (zero where no list reaches), so no memset goes before;
// bound by that store.
__global__ void __launch_bounds__(kT)
    k_vso_gather(const double2* __restrict__ contrib, const int* __restrict__ off,
                 const int* __restrict__ idx, long ngrid, long entries,
                 double2* __restrict__ out) {
  const long g = (long)blockIdx.x * kT + threadIdx.x;
  if (g >= ngrid) return;
  contrib += (size_t)blockIdx.y * 2 * (size_t)entries;
  out += (size_t)blockIdx.y * 2 * (size_t)ngrid;
  double2 up = make_double2(0.0, 0.0), dn = up;
  const int end = off[g + 1];
  for (int t = off[g]; t < end; ++t) {
    const double2 u = contrib[2 * (size_t)idx[t]], d = contrib[2 * (size_t)idx[t] + 1];
    up.x += u.x;
    up.y += u.y;
    dn.x += d.x;
    dn.y += d.y;
  }
  out[g] = up;
  out[ngrid + g] = dn;
}

// projections p[g][m][s] (g: 0 G1, 1 G_2; m: 0 y10, 1 y11, 2 y1_1; s: 0 up, 1 dn)
__global__ void __launch_bounds__(kT) k_vso_kb(const double* __restrict__ psi, long ngrid,
                                               long nnlc, const sep_nlc* __restrict__ nlc,
                                               const long* __restrict__ nl,
                                               const double* __restrict__ elkb, long natom,
                                               double dv, double* __restrict__ out) {
  __shared__ double red[kT / 32][24];
  __shared__ double proj[24];
  const long a = blockIdx.x;
  psi += (size_t)blockIdx.y * 4 * (size_t)ngrid;
  out += (size_t)blockIdx.y * 4 * (size_t)ngrid;
  const long n = nl[a];
  const sep_nlc* base = nlc + a * nnlc;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double p[24];
#pragma unroll
  for (int i = 0; i < 24; ++i) p[i] = 0.0;
  for (long j = tid; j < n; j += kT) {
    const sep_nlc& e = base[j];
    const C2 s[2] = {ld2(psi + 2 * e.jxyz), ld2(psi + 2 * (ngrid + e.jxyz))};
    const C2 y[3] = {ld2(e.y10), ld2(e.y11), ld2(e.y1_1)};
    const double g[2] = {e.Vs0G1, e.Vs0G_2};
#pragma unroll
    for (int gi = 0; gi < 2; ++gi)
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int si = 0; si < 2; ++si) {
          const C2 v = conj_mul(y[m], s[si]);
          const int i = ((gi * 3 + m) * 2 + si) * 2;
          p[i] += g[gi] * v.re;
          p[i + 1] += g[gi] * v.im;
        }
  }
#pragma unroll
  for (int i = 0; i < 24; ++i) {
    double x = p[i];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp][i] = x;
  }
  __syncthreads();
  if (tid < 24) {
    double x = 0.0;
    for (int w = 0; w < kT / 32; ++w) x += red[w][tid];
    const double el = (tid < 12 ? elkb[a] : elkb[a + natom]) * dv;  // hamiltonian.c:284-285
    proj[tid] = x * el;
  }
  __syncthreads();
  auto P = [&](int gi, int m, int si) {
    const int i = ((gi * 3 + m) * 2 + si) * 2;
    return C2{proj[i], proj[i + 1]};
  };
  const double s6 = sqrt(2.0) / 6.0, s3 = sqrt(2.0) / 3.0;
  const double o6 = 1.0 / 6.0, o3 = 1.0 / 3.0, t3 = 2.0 / 3.0;
  for (long j = tid; j < n; j += kT) {
    const sep_nlc& e = base[j];
    const C2 y10 = ld2(e.y10), y11 = ld2(e.y11), y1_1 = ld2(e.y1_1);
    const double g1 = e.Vs0G1, g2 = e.Vs0G_2;
    // hamiltonian.c:318-353, in its order: G_2 terms, then G1 terms
    C2 up = scale(o6 * g2, mul(P(1, 2, 0), y1_1));
    up = add(up, scale(o3 * g2, mul(P(1, 0, 0), y10)));
    up = add(up, scale(0.5 * g2, mul(P(1, 1, 0), y11)));
    up = add(up, scale(s6 * g2, mul(P(1, 0, 1), y1_1)));
    up = add(up, scale(s6 * g2, mul(P(1, 1, 1), y10)));
    up = add(up, scale(-t3 * g1, mul(P(0, 2, 0), y1_1)));
    up = add(up, scale(-o3 * g1, mul(P(0, 0, 0), y10)));
    up = add(up, scale(s3 * g1, mul(P(0, 0, 1), y1_1)));
    up = add(up, scale(s3 * g1, mul(P(0, 1, 1), y10)));
    // hamiltonian.c:358-395
    C2 dn = scale(o6 * g2, mul(P(1, 1, 1), y11));
    dn = add(dn, scale(o3 * g2, mul(P(1, 0, 1), y10)));
    dn = add(dn, scale(-0.5 * g2, mul(P(1, 2, 1), y1_1)));
    dn = add(dn, scale(s6 * g2, mul(P(1, 2, 0), y10)));
    dn = add(dn, scale(s6 * g2, mul(P(1, 0, 0), y11)));
    dn = add(dn, scale(s3 * g1, mul(P(0, 2, 0), y10)));
    dn = add(dn, scale(s3 * g1, mul(P(0, 0, 0), y10)));
    dn = add(dn, scale(-o3 * g1, mul(P(0, 0, 1), y10)));
    dn = add(dn, scale(-t3 * g1, mul(P(0, 1, 1), y11)));
    atomic_add(out + 2 * e.jxyz, up);
    atomic_add(out + 2 * (ngrid + e.jxyz), dn);
  }
}

}  // namespace

namespace sep {
// K of every atom for spinor_vso_kept: natom x nmax x ld doubles, nmax the
// largest list, ld >= nmax
cudaError_t spinor_vso_kernel(long natom, long nnlc, const sep_nlc* nlc, const long* nl,
                              double sigma, long nmax, long ld, double* km, cudaStream_t st) {
  const long tiles = (nmax + kT - 1) / kT;
  if (natom == 0 || nmax == 0) return cudaSuccess;
  if (tiles > 65535) return cudaErrorInvalidValue;
  k_vso_kernel<<<dim3((unsigned)natom, (unsigned)tiles), kT, 0, st>>>(
      nnlc, nlc, nl, sqrt(0.5) / sigma, nmax, ld, km);  // init.c:97
  return cudaGetLastError();
}

bool VsoTensor::fits(long natom, long nmax) {
  const double mb = (double)((nmax + oz::kBlockRows - 1) / oz::kBlockRows);
  return natom > 0 && nmax > 0 && (double)natom * mb <= 65535.0;
}

// Below 64 points both take about as long (8 atoms, 4 spinors: 39 and 40 us at 64).
// From there on, in us for 4 spinors, fitted to 64 and 1000 atoms with longest
// lists of 67 to 356 points, of which all to one in fifty lists were long and the
// rest had 10 points: the FMAs wait for the longest list and then take the pairs
// (64 atoms x 346 points 743, one such list among 64 175, 20 of them among 1000
// 587); the contraction takes every list as long as the longest (129, 113, 913).
// The rule misses the faster of the two by a tenth at most there.
bool VsoTensor::pays(long natom, long nmax, double pairs) {
  const double na = (double)natom;
  const double mb = (double)((nmax + oz::kBlockRows - 1) / oz::kBlockRows);
  const double nkc = (double)((nmax + oz::kChunkK - 1) / oz::kChunkK);
  return nmax >= 64 &&
         0.5 * (double)nmax + 8.8e-5 * pairs > 25.0 + 0.12 * na + 0.0095 * na * mb * nkc;
}

long VsoTensor::spinors() const { return nb * oz::kBlockRows / 12; }

size_t VsoTensor::carve(void* base, long natom_, long nmax_) {
  natom = natom_;
  nmax = nmax_;
  mb = (nmax + oz::kBlockRows - 1) / oz::kBlockRows;
  nkc = (nmax + oz::kChunkK - 1) / oz::kChunkK;
  // 128 columns of products at a time per block of B: as many blocks as stay
  // below half a gigabyte, at most 4 (42 spinors)
  constexpr int elems = oz::block_elems(oz::kBatchSlices);
  const double per = (double)natom * ((double)nkc * elems * 2 + mb * 128.0 * 1024.0);
  nb = (long)std::max(1.0, std::min(4.0, 536870912.0 / per));
  char* p = static_cast<char*>(base);
  auto take = [&](size_t bytes) {
    char* q = p;
    p += (bytes + 255) & ~(size_t)255;
    return q;
  };
  const size_t blk = sizeof(uint16_t) * (size_t)nkc * elems;
  ka = reinterpret_cast<uint16_t*>(take(blk * natom * mb));
  xb = reinterpret_cast<uint16_t*>(take(blk * natom * nb));
  ea = reinterpret_cast<int*>(take(sizeof(int) * natom * mb * oz::kBlockRows));
  eb = reinterpret_cast<int*>(take(sizeof(int) * natom * nb * oz::kBlockRows));
  top = reinterpret_cast<int4*>(take(sizeof(int4) * natom * mb * oz::kBlockRows));
  top_exp = reinterpret_cast<ushort4*>(take(sizeof(ushort4) * natom * mb * oz::kBlockRows));
  xe = reinterpret_cast<uint16_t*>(
      take(sizeof(uint16_t) * 8 * (size_t)natom * spinors() * nkc * oz::kChunkK));
  sums = reinterpret_cast<double*>(
      take(sizeof(double) * (size_t)(natom * mb * oz::kBlockRows) * nb * oz::kBlockRows));
  err = reinterpret_cast<int*>(take(2 * sizeof(int)));
  return (size_t)(p - static_cast<char*>(base));
}

cudaError_t spinor_vso_planes(const VsoTensor& v, const long* nl, const double* km, long ld,
                              int* bad, cudaStream_t st) {
  const long mpad = v.mb * oz::kBlockRows;
  cudaError_t e = cudaMemsetAsync(v.err, 0, 2 * sizeof(int), st);
  if (e != cudaSuccess) return e;
  k_vso_k_expo<<<(unsigned)(v.natom * mpad), 32, 0, st>>>(nl, km, v.nmax, ld, mpad, v.ea,
                                                          v.err + 1);
  k_vso_k_top<<<dim3((unsigned)v.natom, (unsigned)((v.nmax + kTS - 1) / kTS)), kTS, 0, st>>>(
      nl, km, v.nmax, ld, mpad, v.top, v.top_exp);
  k_vso_k_slice<<<dim3((unsigned)v.nkc, (unsigned)(v.natom * v.mb)), kSliceT, 0, st>>>(
      nl, km, v.nmax, ld, v.mb, v.ea, v.ka, v.nkc);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  e = cudaMemcpyAsync(bad, v.err + 1, sizeof(int), cudaMemcpyDeviceToHost, st);
  return e != cudaSuccess ? e : cudaStreamSynchronize(st);
}

cudaError_t spinor_vso_kept(const double* psi, long ngrid, long nsp, long natom, long nnlc,
                            const sep_nlc* nlc, const long* nl, double sigma, double dv,
                            const double* km, long nmax, long ld, const VsoTensor* tensor,
                            const int* off, const int* idx, double* contrib, double* psinl,
                            cudaStream_t st) {
  const double tmp = 0.5 / sqrt(kTwoPi * (sigma * sigma)) * dv;  // hamiltonian.c:89
  double2* cb = reinterpret_cast<double2*>(contrib);
  if (tensor) {
    const VsoTensor& v = *tensor;
    const long most = v.spinors();
    for (long s0 = 0; s0 < nsp; s0 += most) {
      const long k = std::min(most, nsp - s0), nb = (12 * k + oz::kBlockRows - 1) / oz::kBlockRows;
      const int items = (int)(6 * v.nkc * (oz::kChunkK / 8));
      k_vso_x_slice<<<dim3((unsigned)natom, (unsigned)k), std::min(kSliceX, (items + 31) / 32 * 32),
                      0, st>>>(
          psi + (size_t)s0 * 4 * ngrid, ngrid, nnlc, nlc, nl, nb, v.nkc, most, v.eb, v.xe,
          v.xb);
      oz::Planes A, B;
      A.d = v.ka;
      A.expo = v.ea;
      B.d = v.xb;
      B.expo = v.eb;
      A.k = B.k = nmax;
      A.nkc = B.nkc = v.nkc;
      A.nrb = natom * v.mb;
      B.nrb = natom * nb;
      const cudaError_t e =
          oz::gemm_nt_batched(A, B, (int)natom, 12 * k, v.sums, 12 * k, v.err, st);
      if (e != cudaSuccess) return e;
      k_vso_combine<<<dim3((unsigned)natom, (unsigned)((nmax + kTS - 1) / kTS), (unsigned)k), kTS, 0,
                      st>>>(v.sums, v.ea, v.eb, nb * oz::kBlockRows, v.top, v.top_exp, v.xe,
                            v.nkc * oz::kChunkK * 8, most, 12 * k, v.mb * oz::kBlockRows,
                            psi + (size_t)s0 * 4 * ngrid, ngrid, nnlc, nlc, nl, km, nmax, ld, tmp,
                            cb + (size_t)s0 * 2 * (size_t)(natom * nmax));
    }
  } else {
    const dim3 g((unsigned)natom, (unsigned)((nmax + kTS - 1) / kTS), (unsigned)nsp);
    k_vso_stored<<<g, kTS, 0, st>>>(psi, ngrid, nnlc, nlc, nl, km, nmax, ld, tmp, cb);
  }
  const dim3 gg((unsigned)((ngrid + kT - 1) / kT), (unsigned)nsp);
  k_vso_gather<<<gg, kT, 0, st>>>(cb, off, idx, ngrid, natom * nmax,
                                  reinterpret_cast<double2*>(psinl));
  return cudaGetLastError();
}
// Vso on nsp spinors (4 ngrid doubles apart) into psinl (zeroed first), on st,
// K formed in place; the arguments are already checked.  nsp <= 65535.
cudaError_t spinor_vso_launch(const double* psi, long ngrid, long nsp, long natom, long nnlc,
                              const sep_nlc* nlc, const long* nl, double sigma, double dv,
                              int flagkb, const double* elkb, double* psinl, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(psinl, 0, sizeof(double) * 4 * (size_t)ngrid * nsp, st);
  if (e != cudaSuccess || natom == 0) return e;
  const dim3 grid((unsigned)natom, (unsigned)nsp);
  if (flagkb) {
    k_vso_kb<<<grid, kT, 0, st>>>(psi, ngrid, nnlc, nlc, nl, elkb, natom, dv, psinl);
  } else {
    const double tmp = 0.5 / sqrt(kTwoPi * (sigma * sigma)) * dv;  // hamiltonian.c:89
    const double sigma_1 = sqrt(0.5) / sigma;  // init.c:97
    k_vso_gauss<<<grid, kT, 0, st>>>(psi, ngrid, nnlc, nlc, nl, tmp, sigma_1, psinl);
  }
  return cudaGetLastError();
}
}  // namespace sep

extern "C" {

int sep_spinor_vso_dev(const double* psi, long ngrid, long natom, long nnlc, const sep_nlc* nlc,
                       const long* nl, double sigma, double dv, int flagkb, const double* elkb,
                       double* psinl, void* cuda_stream) {
  if (!psi || !psinl || !nlc || !nl || ngrid < 1 || natom < 0 || nnlc < 0 ||
      (flagkb && !elkb) || (!flagkb && !(sigma > 0.0)))
    return fail(SEP_ERR_ARG, "sep_spinor_vso: bad arguments");
  cudaStream_t st = (cudaStream_t)cuda_stream;
  SK(sep::spinor_vso_launch(psi, ngrid, 1, natom, nnlc, nlc, nl, sigma, dv, flagkb, elkb,
                            psinl, st));
  return SEP_OK;
}

int sep_spinor_vso(const double* psi, long ngrid, long natom, long nnlc, const sep_nlc* nlc,
                   const long* nl, double sigma, double dv, int flagkb, const double* elkb,
                   double* psinl) {
  if (!psi || !psinl || !nlc || !nl || ngrid < 1 || natom < 0 || nnlc < 0 || (flagkb && !elkb))
    return fail(SEP_ERR_ARG, "sep_spinor_vso: bad arguments");
  for (long a = 0; a < natom; ++a)
    if (nl[a] < 0 || nl[a] > nnlc) return fail(SEP_ERR_ARG, "sep_spinor_vso: nl[a] > nnlc");
  for (long a = 0; a < natom; ++a)
    for (long j = 0; j < nl[a]; ++j) {
      const long g = nlc[a * nnlc + j].jxyz;
      if (g < 0 || g >= ngrid) return fail(SEP_ERR_ARG, "sep_spinor_vso: jxyz outside the grid");
    }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) {
    cudaGetLastError();
    return fail(SEP_ERR_NO_DEVICE, "sep_spinor_vso: no CUDA device");
  }
  double *d_psi = nullptr, *d_out = nullptr, *d_el = nullptr;
  sep_nlc* d_nlc = nullptr;
  long* d_nl = nullptr;
  cudaStream_t st = nullptr;
  int r = SEP_OK;
  auto done = [&](int status) {
    if (st) cudaStreamSynchronize(st);
    cudaFree(d_psi);
    cudaFree(d_out);
    cudaFree(d_el);
    cudaFree(d_nlc);
    cudaFree(d_nl);
    if (st) cudaStreamDestroy(st);
    return status;
  };
  const size_t nbytes = sizeof(double) * 4 * ngrid;
  const size_t lbytes = sizeof(sep_nlc) * (size_t)(natom * nnlc > 0 ? natom * nnlc : 1);
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess ||
      cudaMalloc(&d_psi, nbytes) != cudaSuccess || cudaMalloc(&d_out, nbytes) != cudaSuccess ||
      cudaMalloc(&d_nlc, lbytes) != cudaSuccess ||
      cudaMalloc(&d_nl, sizeof(long) * (natom > 0 ? natom : 1)) != cudaSuccess ||
      cudaMalloc(&d_el, sizeof(double) * (natom > 0 ? 2 * natom : 1)) != cudaSuccess)
    return done(fail(SEP_ERR_NOMEM, "sep_spinor_vso: device allocation failed"));
  if (cudaMemcpyAsync(d_psi, psi, nbytes, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      (natom > 0 && cudaMemcpyAsync(d_nlc, nlc, sizeof(sep_nlc) * natom * nnlc,
                                    cudaMemcpyHostToDevice, st) != cudaSuccess) ||
      (natom > 0 && cudaMemcpyAsync(d_nl, nl, sizeof(long) * natom, cudaMemcpyHostToDevice,
                                    st) != cudaSuccess) ||
      (flagkb && natom > 0 && cudaMemcpyAsync(d_el, elkb, sizeof(double) * 2 * natom,
                                              cudaMemcpyHostToDevice, st) != cudaSuccess))
    return done(fail(SEP_ERR_CUDA, "sep_spinor_vso: upload failed"));
  r = sep_spinor_vso_dev(d_psi, ngrid, natom, nnlc, d_nlc, d_nl, sigma, dv, flagkb, d_el, d_out,
                         st);
  if (r != SEP_OK) return done(r);
  if (cudaMemcpyAsync(psinl, d_out, nbytes, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return done(fail(SEP_ERR_CUDA, "sep_spinor_vso: download failed"));
  return done(SEP_OK);
}

}  // extern "C"
