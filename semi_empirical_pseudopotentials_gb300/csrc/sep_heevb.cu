// sep_heevb.cu -- the lowest eigenpairs of many small Hermitian matrices at
// once (the bulk fit's per-k-point problems, pseudopotFitting/diag.c:12-48,
// where the reference calls zheev for every k-point and keeps the lowest
// bands, fit.c:86-88).
//
// Per matrix (n <= 512, column-major, both triangles stored):
//  1. k_hetrd (a cluster of blocks per matrix): Householder reduction to real
//     symmetric tridiagonal form with LAPACK zhetd2's conventions (lower
//     triangle; H_j = I - tau_j v_j v_j^H with v_j(j+1) = 1 and a real beta_j,
//     so T = Q^H A Q has a real diagonal d and off-diagonal e).  Per step: the reflector of the next
//     column, p = tau A22 v, w = p - (tau/2)(p^H v) v and the rank-2 update
//     A22 -= v w^H + w v^H of the lower triangle.  Warps take columns (lanes
//     on consecutive rows: coalesced); for p each column adds A_ik v_k to
//     its rows' per-lane sums (scatter) and sum_{i>k} conj(A_ik) v_i to p_k
//     (gather), and the sums of warps and blocks are added in a fixed order,
//     so the result does not depend on timing.  The reflectors stay below the
//     subdiagonal for the back-transformation.
//  2. k_stebz: the lowest nw eigenvalues of T by multisection on Sturm counts
//     (16 or four threads per eigenvalue; the counts by the division-free continuant
//     recursion with exact power-of-two rescaling).
//  3. k_stein: their eigenvectors by inverse iteration (LAPACK dstein's
//     scheme): Gaussian elimination with partial pivoting of T - lambda I,
//     eigenvalues closer than 1e-3 ||T||_1 form a group whose vectors are
//     orthogonalised against each other (modified Gram-Schmidt), eigenvalues
//     inside a group closer than 10 eps |lambda| are moved apart by that much;
//     a warp per group.
//  4. k_unmtr: x = H_0 H_1 ... H_{n-2} z for each vector (a warp per vector,
//     the vector in shared memory).
// On GB300 every FP64 operation goes through the FP64 pipe (about 2 FMAs per
// clock per SM); the reduction costs 8 n^3 / 3 FMAs per matrix, 35 ms on one
// SM at n = 377.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <vector>

#include "sep_heevb.cuh"

namespace sep {
namespace hb {
namespace {

namespace cg = cooperative_groups;
using Z = double2;
constexpr int kWarps = 16;
constexpr int kThreads = 32 * kWarps;

__device__ __forceinline__ Z zmk(double a, double b) {
  Z r;
  r.x = a;
  r.y = b;
  return r;
}
__device__ __forceinline__ Z zadd(Z a, Z b) { return zmk(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ Z zmul(Z a, Z b) { return zmk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// acc + a * b
__device__ __forceinline__ Z zfma(Z a, Z b, Z acc) {
  return zmk(fma(a.x, b.x, fma(-a.y, b.y, acc.x)), fma(a.x, b.y, fma(a.y, b.x, acc.y)));
}
// acc + conj(a) * b
__device__ __forceinline__ Z zfmac(Z a, Z b, Z acc) {
  return zmk(fma(a.x, b.x, fma(a.y, b.y, acc.x)), fma(a.x, b.y, fma(-a.y, b.x, acc.y)));
}
// acc - a * conj(b), four FMAs
__device__ __forceinline__ Z zfnmsc(Z a, Z b, Z acc) {
  return zmk(fma(-a.x, b.x, fma(-a.y, b.y, acc.x)), fma(-a.y, b.x, fma(a.x, b.y, acc.y)));
}
// acc - a * b, four FMAs
__device__ __forceinline__ Z zfnms(Z a, Z b, Z acc) {
  return zmk(fma(-a.x, b.x, fma(a.y, b.y, acc.x)), fma(-a.x, b.y, fma(-a.y, b.x, acc.y)));
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sums over the warp of two values per lane: a's in lanes 0-15, b's in 16-31
__device__ __forceinline__ double warp_sum2(double a, double b, int lane) {
  const bool up = lane & 16;
  double c = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  return c;
}

// sums over the warp of 8 values per lane, with 9 additions a lane instead of
// 40 (on this part an FP64 warp instruction holds its sub-partition for 64
// clocks): value q's total ends in the lanes with lane / 4 == q
__device__ __forceinline__ double warp_sum8(const double (&x)[8], int lane) {
  double a[4], b[2];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const bool up = lane & 16;
    a[q] = (up ? x[4 + q] : x[q]) + __shfl_xor_sync(0xffffffffu, up ? x[q] : x[4 + q], 16);
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const bool up = lane & 8;
    b[q] = (up ? a[2 + q] : a[q]) + __shfl_xor_sync(0xffffffffu, up ? a[q] : a[2 + q], 8);
  }
  const bool up = lane & 4;
  double c = (up ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, up ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  return c + __shfl_xor_sync(0xffffffffu, c, 1);
}

// ---------------------------------------------------------------------------
// 1. tridiagonal reduction: a cluster of G blocks per matrix.  Column k always
//    belongs to warp k % (G kWarps) of the cluster, so a block reads and
//    writes its own columns only, and the column that becomes the next
//    reflector is the one thing every block reads (from L2).  Each block holds
//    v, w and its part of A22 v in shared memory; the parts are added over
//    distributed shared memory in block order, so every block has the same p.
//    Two cluster barriers per step.  A warp takes kCols columns at a time:
//    their products go into the rows' sums with one shared read and write, and
//    their gather sums are reduced together (warp_sum8).  Bound by the FP64
//    pipe (16 FMAs per element of the trailing triangle and step) and, for
//    large G or small n, by the chain of each step (about 16 us).  42 matrices of
//    377: 19.6 ms with clusters of 3, 55 ms with one block per matrix.
//    shared memory: v, w, gather sums, this block's part (4 n complex) and the
//    warps' scatter sums (kWarps x n complex)
constexpr int kCols = 4;

__global__ void __launch_bounds__(kThreads, 1)
    k_hetrd(Z* Aall, int n, int G, double* __restrict__ dall,
            double* __restrict__ eall, Z* __restrict__ tauall) {
  extern __shared__ __align__(16) unsigned char hb_smem[];
  const cg::cluster_group cluster = cg::this_cluster();
  Z* v = reinterpret_cast<Z*>(hb_smem);
  Z* w = v + n;
  Z* gs = w + n;                 // gather part of p per own column
  Z* part = gs + n;              // this block's part of A22 v
  Z* pw = part + n;              // scatter parts: kWarps x n
  static_assert(kWarps == 16, "red: a warp reads it with one value per lane");
  __shared__ double red[2 * kWarps];
  __shared__ double sh_q[4];  // tau, 1 / (alpha - beta)
  __shared__ int sh_skip;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = blockIdx.x % G, m = blockIdx.x / G;
  const int stride = G * kWarps, own = rank * kWarps + warp;
  Z* A = Aall + (size_t)m * n * n;
  double* d = dall + (size_t)m * n;
  double* e = eall + (size_t)m * n;
  Z* tau = tauall + (size_t)m * n;

  for (int j = 0; j < n - 1; ++j) {
    const int r0 = j + 1;
    // ---- reflector of column j (rows r0 .. n-1), warp 0 of every block
    if (warp == 0) {
      double part2 = 0.0;
      for (int i = r0 + 1 + lane; i < n; i += 32) {
        const Z x = __ldcg(&A[(size_t)j * n + i]);
        part2 = fma(x.x, x.x, fma(x.y, x.y, part2));
      }
      const double xn2 = warp_sum(part2);
      const Z al = __ldcg(&A[(size_t)j * n + r0]);
      const bool skip = xn2 == 0.0 && al.y == 0.0;  // already reduced: H_j = I
      double beta = al.x, q = 0.0;
      if (!skip) {
        beta = -copysign(sqrt(al.x * al.x + al.y * al.y + xn2), al.x);
        const double dx = al.x - beta, dy = al.y, dd = dx * dx + dy * dy;
        // the four quotients in four lanes: one division's instructions
        const double num = lane == 0 ? -dx : lane == 2 ? dx : -dy;
        q = num / (lane < 2 ? beta : dd);
      }
      if (lane < 4) {
        sh_q[lane] = q;
        if (lane == 0) sh_skip = skip;
        if (rank == 0) {
          if (lane < 2) reinterpret_cast<double*>(tau + j)[lane] = q;
          if (lane == 2) d[j] = __ldcg(&A[(size_t)j * n + j]).x;
          if (lane == 3) e[j] = beta;
        }
      }
    }
    __syncthreads();
    if (sh_skip) {  // the same in every block; the barrier keeps sh_skip until every thread has read it
      __syncthreads();
      continue;
    }
    const Z tj = zmk(sh_q[0], sh_q[1]), sc = zmk(sh_q[2], sh_q[3]);
    for (int i = r0 + tid; i < n; i += kThreads)
      v[i] = i > r0 ? zmul(__ldcg(&A[(size_t)j * n + i]), sc) : zmk(1.0, 0.0);
    Z* mine = pw + (size_t)warp * n;
    for (int i = r0 + lane; i < n; i += 32) mine[i] = zmk(0.0, 0.0);
    __syncthreads();
    const int kfirst = r0 + ((own - r0) % stride + stride) % stride;
    // ---- this block's part of A22 v: warps on columns k, lanes on rows i >= k
    // in groups of 32 that end at the last row
    for (int k = kfirst; k < n; k += kCols * stride) {
      Z vk[kCols];
      double g[2 * kCols];
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        vk[c] = k + c * stride < n ? v[k + c * stride] : zmk(0.0, 0.0);
        g[2 * c] = g[2 * c + 1] = 0.0;
      }
      for (int i0 = n - (n - k + 31) / 32 * 32; i0 < n; i0 += 32) {
        const int i = i0 + lane;
        const bool in = i >= k;
        const Z vi = in ? v[i] : zmk(0.0, 0.0);
        Z s = in ? mine[i] : zmk(0.0, 0.0);
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          const int kc = k + c * stride;
          if (kc < n && i0 + 31 >= kc) {  // uniform: some row of the group lies in column kc
            const Z a = i >= kc ? A[(size_t)kc * n + i] : zmk(0.0, 0.0);
            s = zfma(a, vk[c], s);
            const Z b = i > kc ? a : zmk(0.0, 0.0);
            const Z q = zfmac(b, vi, zmk(g[2 * c], g[2 * c + 1]));
            g[2 * c] = q.x;
            g[2 * c + 1] = q.y;
          }
        }
        if (in) mine[i] = s;
      }
      const double t = warp_sum8(g, lane);
      const int kc = k + (lane >> 3) * stride;
      if ((lane & 3) == 0 && kc < n) reinterpret_cast<double*>(gs)[2 * kc + ((lane >> 2) & 1)] = t;
    }
    __syncthreads();
    for (int i = r0 + tid; i < n; i += kThreads) {
      Z s = i % stride / kWarps == rank ? gs[i] : zmk(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < kWarps; ++q) s = zadd(s, pw[(size_t)q * n + i]);
      part[i] = s;
    }
    cluster.sync();  // every part is written, every block has read column j
    // ---- p = tau A22 v, p^H v, w = p - (tau / 2) (p^H v) v, in every block
    double px = 0.0, py = 0.0;
    for (int i = r0 + tid; i < n; i += kThreads) {
      Z s = *cluster.map_shared_rank(&part[i], 0);
      for (int q = 1; q < G; ++q) s = zadd(s, *cluster.map_shared_rank(&part[i], q));
      const Z pi = zmul(tj, s);
      w[i] = pi;
      const Z c = zfmac(pi, v[i], zmk(0.0, 0.0));  // conj(p_i) v_i
      px += c.x;
      py += c.y;
      if (j % stride / kWarps == rank && i > r0)
        A[(size_t)j * n + i] = v[i];  // kept for the back-transformation
    }
    const double ps = warp_sum2(px, py, lane);
    if ((lane & 15) == 0) red[lane + warp] = ps;  // 16 sums of px, 16 of py
    __syncthreads();
    double pt = red[lane];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) pt += __shfl_xor_sync(0xffffffffu, pt, o);
    const double dx = __shfl_sync(0xffffffffu, pt, 0), dy = __shfl_sync(0xffffffffu, pt, 16);
    // w = p + alpha v, alpha = -tau (p^H v) / 2
    const Z alpha = zmul(zmk(-0.5 * tj.x, -0.5 * tj.y), zmk(dx, dy));
    for (int i = r0 + tid; i < n; i += kThreads) w[i] = zfma(alpha, v[i], w[i]);
    __syncthreads();
    // ---- A22 -= v w^H + w v^H, lower triangle of the own columns
    for (int k = kfirst; k < n; k += kCols * stride) {
      Z vk[kCols], wk[kCols];
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const int kc = min(k + c * stride, n - 1);
        vk[c] = v[kc];
        wk[c] = w[kc];
      }
      for (int i0 = n - (n - k + 31) / 32 * 32; i0 < n; i0 += 32) {
        const int i = i0 + lane;
        const bool in = i >= k;
        const Z vi = in ? v[i] : zmk(0.0, 0.0), wi = in ? w[i] : zmk(0.0, 0.0);
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          const int kc = k + c * stride;
          if (kc < n && i0 + 31 >= kc) {
            Z* p = &A[(size_t)kc * n + i];
            Z a = i >= kc ? *p : zmk(0.0, 0.0);
            a = zfnmsc(vi, wk[c], a);
            a = zfnmsc(wi, vk[c], a);
            if (i == kc) a.y = 0.0;  // the diagonal stays real
            if (i >= kc) *p = a;
          }
        }
      }
    }
    cluster.sync();  // column j + 1 is final, the parts have been read
  }
  if (tid == 0 && rank == 0) {
    d[n - 1] = __ldcg(&A[(size_t)(n - 1) * n + n - 1]).x;
    e[n - 1] = 0.0;
  }
}

// ---------------------------------------------------------------------------
// Sturm count: eigenvalues of T below x = sign changes in the leading
// principal minors p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2} (p_{-1} = 1),
// two FP64 operations per step and no division.  When the larger of the two
// current minors leaves [2^-400, 2^400], both are multiplied by the same
// exact power of two (integer work on the exponent fields) that brings the
// larger near 1; a smaller one that would underflow becomes 0.  A minor that
// is exactly zero counts as having the sign opposite to its predecessor (as
// LAPACK's dlaebz, whose zero pivots count as negative).
__device__ __forceinline__ int expo_field(double v) {
  return (int)((__double_as_longlong(v) >> 52) & 0x7ff);
}
__device__ __forceinline__ double scale_pow2(double v, int k) {  // v 2^k
  const int ex = expo_field(v);
  if (ex == 0) return v;                 // zero
  if (ex + k <= 0) return copysign(0.0, v);  // underflow
  return __longlong_as_double(__double_as_longlong(v) + ((long long)k << 52));
}
__device__ int sturm_count(const double* d, const double* e2, int n, double x) {
  double pm = 1.0, p = d[0] - x;
  int c = 0;
  bool sprev = false;  // p_{-1} = 1 is positive
  for (int i = 0;; ++i) {
    // sign and zero tests on the bits (integer work, not the FP64 pipe)
    const long long pb = __double_as_longlong(p);
    const bool sn = (pb < 0 && (pb << 1) != 0) || ((pb << 1) == 0 && !sprev);
    c += (sn != sprev);
    sprev = sn;
    if (i == n - 1) break;
    const double q = fma(d[i + 1] - x, p, -e2[i] * pm);
    pm = p;
    p = q;
    const int emx = max(expo_field(p), expo_field(pm));
    if (emx > 1023 + 400 || emx < 1023 - 400) {
      const int k = 1023 - emx;
      p = scale_pow2(p, k);
      pm = scale_pow2(pm, k);
    }
  }
  return c;
}

// 2. lowest nw eigenvalues, S threads each; w[nw .. n-1] = NaN.  Every round
//    the S threads count at the points that cut the interval into S + 1 parts,
//    so an eigenvalue takes log2(S + 1) times fewer rounds of n dependent steps
//    than bisection.  Bound by that chain as long as no sub-partition holds
//    many warps; a block is one warp, so a matrix spreads over several SMs.
//    42 matrices of 377, 32 eigenvalues: 1.24 ms with S = 16; 2.13 ms with S = 4
//    and one block per matrix, 4.9 ms by bisection.
template <int S>
__global__ void __launch_bounds__(32)
    k_stebz(const double* __restrict__ dall, const double* __restrict__ eall, int n, int nw,
            double* __restrict__ wall, double* __restrict__ tnorm) {
  extern __shared__ double sb[];
  double* d = sb;
  double* e2 = sb + n;
  __shared__ double sh_lo, sh_hi, sh_piv;
  const double* dg = dall + (size_t)blockIdx.x * n;
  const double* eg = eall + (size_t)blockIdx.x * n;
  double* w = wall + (size_t)blockIdx.x * n;
  for (int i = threadIdx.x; i < n; i += 32) {
    d[i] = dg[i];
    e2[i] = (i < n - 1) ? eg[i] * eg[i] : 0.0;
  }
  __syncthreads();
  {  // Gershgorin interval, |T|_1 and the largest e^2
    double lo = d[0], hi = d[0], emax = 0.0, onenrm = 0.0;
    for (int i = threadIdx.x; i < n; i += 32) {
      const double r = (i > 0 ? fabs(eg[i - 1]) : 0.0) + (i < n - 1 ? fabs(eg[i]) : 0.0);
      lo = fmin(lo, d[i] - r);
      hi = fmax(hi, d[i] + r);
      onenrm = fmax(onenrm, fabs(d[i]) + r);
      emax = fmax(emax, e2[i]);
    }
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      onenrm = fmax(onenrm, __shfl_xor_sync(0xffffffffu, onenrm, o));
      emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
    }
    if (threadIdx.x == 0) {
      const double span = fmax(hi - lo, DBL_MIN);
      sh_lo = lo - 2.1 * DBL_EPSILON * span - 1e-300;
      sh_hi = hi + 2.1 * DBL_EPSILON * span + 1e-300;
      sh_piv = DBL_MIN * fmax(1.0, emax);
      if (blockIdx.y == 0) tnorm[blockIdx.x] = onenrm;
    }
  }
  __syncthreads();
  for (int t = nw + threadIdx.x; t < n && blockIdx.y == 0; t += 32)
    w[t] = __longlong_as_double(0x7ff8000000000000LL);  // NaN: not computed
  const int t = blockIdx.y * (32 / S) + threadIdx.x / S, q = threadIdx.x % S;
  double lo = sh_lo, hi = sh_hi;
  bool done = t >= nw;
  for (int it = 0; it < 200; ++it) {
    // this thread's point; the interval is done when it is as short as the
    // eigenvalue's precision or no point lies inside it (towards the end some
    // round to an end, whose count is known)
    const double x = lo + (hi - lo) * ((q + 1) * (1.0 / (S + 1)));
    const bool inside = x > lo && x < hi;
    const int base = threadIdx.x & ~(S - 1);
    const unsigned in = __ballot_sync(0xffffffffu, inside);
    done = done || hi - lo <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + sh_piv ||
           ((in >> base) & ((1u << S) - 1u)) == 0;
    if (__all_sync(0xffffffffu, done)) break;
    // eigenvalue t lies below x
    const bool above = !done && (inside ? sturm_count(d, e2, n, x) > t : x >= hi);
    const unsigned ab = (__ballot_sync(0xffffffffu, above) >> base) & ((1u << S) - 1u);
    const int first = ab ? __ffs(ab) - 1 : S;  // the lowest point above eigenvalue t
    const double xl = __shfl_sync(0xffffffffu, x, base + max(first - 1, 0));
    const double xh = __shfl_sync(0xffffffffu, x, base + min(first, S - 1));
    if (!done) {
      if (first > 0) lo = xl;
      if (first < S) hi = xh;
    }
  }
  if (t < nw && q == 0) w[t] = 0.5 * (lo + hi);
}

// ---------------------------------------------------------------------------
// 3. eigenvectors of T by inverse iteration: block (matrix, i) is one warp
//    that makes the vectors of the group whose first eigenvalue is i, if one
//    begins there.  T - lambda I, its LU and the iterate are in shared memory
//    (5 n doubles and n flags).  Lane 0 runs the three recurrences; sums,
//    norms, scaling, reciprocal pivots and Gram-Schmidt take all lanes.  Bound
//    by the recurrences' chains, about 24 dependent FP64 operations per row
//    and vector (12 of them the elimination's division), which is why the groups
//    spread over all SMs' sub-partitions, where an FP64 instruction of one lane
//    holds its pipe as long as one of 32.  42 matrices of 377, 32 vectors each:
//    1.95 ms; 5.6 ms with a thread per group in one block per matrix, every
//    row through global scratch and a division per pivot and iteration.
__device__ double lcg_uniform(unsigned long long s) {  // (-1, 1)
  return (double)(s >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// (value, index) of the largest value over the warp, the lowest index of equal ones
__device__ __forceinline__ void warp_largest(unsigned long long& v, int& i) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v2 = __shfl_xor_sync(0xffffffffu, v, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, i, o);
    if (v2 > v || (v2 == v && i2 < i)) {
      v = v2;
      i = i2;
    }
  }
}

size_t stein_smem(int n) { return (size_t)n * (5 * sizeof(double) + 1); }

__global__ void __launch_bounds__(32)
    k_stein(const double* __restrict__ dall, const double* __restrict__ eall,
            const double* __restrict__ wall, const double* __restrict__ tnorm, int n, int nw,
            double* zall, int* __restrict__ info) {
  extern __shared__ double st[];
  double* u0 = st;          // T's diagonal, then U's reciprocal diagonal
  double* lm = st + n;      // T's off-diagonal, then the multipliers
  double* u1 = st + 2 * n;  // U's first superdiagonal
  double* u2 = st + 3 * n;  // U's second superdiagonal
  double* x = st + 4 * n;
  char* piv = reinterpret_cast<char*>(st + 5 * n);
  const int m = blockIdx.x, first = blockIdx.y, lane = threadIdx.x;
  const double* w = wall + (size_t)m * n;
  const double onenrm = tnorm[m];
  const double ortol = 1e-3 * onenrm;
  if (first > 0 && !(w[first] - w[first - 1] > ortol)) return;
  const double* d = dall + (size_t)m * n;
  const double* e = eall + (size_t)m * n;
  double* Zm = zall + (size_t)m * n * nw;
  const double eps = DBL_EPSILON;
  const double dtpcrt = sqrt(0.1 / n);
  const double tol = fmax(eps * onenrm, DBL_MIN);
  // the generator's step of 32 places, s <- a32 s + c32
  constexpr unsigned long long kA = 6364136223846793005ULL, kC = 1442695040888963407ULL;
  unsigned long long a32 = 1, c32 = 0;
#pragma unroll
  for (int q = 0; q < 32; ++q) {
    c32 = c32 * kA + kC;
    a32 *= kA;
  }
  double xjm = 0.0;
  for (int jj = first; jj < nw && (jj == first || !(w[jj] - w[jj - 1] > ortol)); ++jj) {
    double xj = w[jj];
    if (jj > first) {
      const double pertol = 10.0 * fabs(eps * xj);
      if (xj - xjm < pertol) xj = xjm + pertol;
    }
    xjm = xj;
    __syncwarp();
    unsigned long long seed = 0x9E3779B97F4A7C15ULL * (unsigned long long)(m * 4096 + jj + 1);
    for (int q = 0; q <= lane; ++q) seed = seed * kA + kC;
    for (int i = lane; i < n; i += 32) {
      u0[i] = d[i];
      lm[i] = i < n - 1 ? e[i] : 0.0;
      x[i] = lcg_uniform(seed);
      seed = seed * a32 + c32;
    }
    __syncwarp();
    // T - xj I = P L U (partial pivoting): row k holds (u0, u1, u2)
    if (lane == 0) {
      double a = u0[0] - xj, c = lm[0], b = c;  // b: subdiagonal (k + 1, k)
      for (int k = 0; k < n - 1; ++k) {
        const double an = u0[k + 1] - xj;  // next row's diagonal
        const double cn = lm[k + 1];       // 0 in the last row
        const bool keep = fabs(a) >= fabs(b);
        const double num = keep ? b : a, den = keep ? a : b;
        const double l = den != 0.0 ? num / den : 0.0;
        u0[k] = den;
        u1[k] = keep ? c : an;
        u2[k] = keep ? 0.0 : cn;
        lm[k] = l;
        piv[k] = !keep;
        a = keep ? fma(-l, c, an) : fma(-l, an, c);
        c = keep ? cn : -l * cn;
        b = cn;
      }
      u0[n - 1] = a;
      u1[n - 1] = u2[n - 1] = 0.0;
    }
    __syncwarp();
    // small pivots are perturbed (dlagts with a tolerance)
    const double last = fmax(fabs(u0[n - 1]), tol);
    __syncwarp();
    for (int k = lane; k < n; k += 32) {
      double u = u0[k];
      if (fabs(u) < tol) u = u < 0.0 ? -tol : tol;
      u0[k] = 1.0 / u;
    }
    int nrmchk = 0;
    for (int its = 0; its < 5; ++its) {
      double asum = 0.0;
      for (int i = lane; i < n; i += 32) asum += fabs(x[i]);
      asum = warp_sum(asum);
      const double scl = n * onenrm * fmax(eps, last) / fmax(asum, DBL_MIN);
      for (int i = lane; i < n; i += 32) x[i] *= scl;
      __syncwarp();
      // solve P L U y = x: forward with the row interchanges, then U; the next
      // row's operands are read before this row's result is stored
      if (lane == 0) {
        double xk = x[0], xn = x[1], l = lm[0];
        bool p = piv[0];
        for (int k = 0; k < n - 1; ++k) {
          const int k1 = min(k + 1, n - 2), k2 = min(k + 2, n - 1);
          const double xn2 = x[k2], l2 = lm[k1];
          const bool p2 = piv[k1];
          const double keep = p ? xn : xk, other = p ? xk : xn;
          x[k] = keep;
          xk = fma(-l, keep, other);
          xn = xn2;
          l = l2;
          p = p2;
        }
        double s = xk, y1 = 0.0, y2 = 0.0;
        double r = u0[n - 1], v1 = 0.0, v2 = 0.0;
        for (int k = n - 1; k >= 0; --k) {
          const int kp = max(k - 1, 0);
          const double sn = x[kp], rn = u0[kp], v1n = u1[kp], v2n = u2[kp];
          const double y = fma(-v1, y1, fma(-v2, y2, s)) * r;
          x[k] = y;
          y2 = y1;
          y1 = y;
          s = sn;
          r = rn;
          v1 = v1n;
          v2 = v2n;
        }
      }
      __syncwarp();
      // orthogonalise against the group's earlier vectors
      for (int q = first; q < jj; ++q) {
        const double* zq = Zm + (size_t)q * n;
        double dot = 0.0;
        for (int i = lane; i < n; i += 32) dot += zq[i] * x[i];
        dot = warp_sum(dot);
        for (int i = lane; i < n; i += 32) x[i] -= dot * zq[i];
      }
      unsigned long long big = 0;
      int at = 0;
      for (int i = lane; i < n; i += 32) {
        // the bits of |x| order as |x| does
        const unsigned long long v = (unsigned long long)__double_as_longlong(x[i]) << 1 >> 1;
        big = v > big ? v : big;
      }
      warp_largest(big, at);
      if (!(__longlong_as_double((long long)big) >= dtpcrt)) continue;
      if (++nrmchk < 3) continue;
      break;
    }
    if (nrmchk == 0 && lane == 0) atomicAdd(info + m, 1);  // no growth: not accepted by dstein
    double s2 = 0.0;
    unsigned long long big = 0;
    int jmax = n;
    for (int i = lane; i < n; i += 32) {
      s2 += x[i] * x[i];
      const unsigned long long v = (unsigned long long)__double_as_longlong(x[i]) << 1 >> 1;
      if (v > big || jmax == n) {
        big = v;
        jmax = i;
      }
    }
    s2 = warp_sum(s2);
    warp_largest(big, jmax);
    __syncwarp();  // x[jmax] was last written by another lane; shuffles order no memory
    double scl = 1.0 / sqrt(s2);
    if (x[jmax] < 0.0) scl = -scl;
    double* zj = Zm + (size_t)jj * n;
    for (int i = lane; i < n; i += 32) zj[i] = x[i] * scl;
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// 4. X = Q Z: warps on vectors, the vector in shared memory, lanes on the rows
//    of each reflector.  Blocks of 4 vectors: bound by the FP64 pipe (8 FMAs
//    per row and reflector) once a crystal's vectors cover every SM, which one
//    block per matrix did not (42 matrices of 377, 32 vectors each: 2.5 ms, 7.3 ms
//    with one block of 16 warps per matrix)
constexpr int kUnWarps = 4;

__global__ void __launch_bounds__(32 * kUnWarps)
    k_unmtr(const Z* __restrict__ Aall, const Z* __restrict__ tauall,
            const double* __restrict__ zall, int n, int nw, Z* __restrict__ xall) {
  extern __shared__ __align__(16) unsigned char hb_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m = blockIdx.x, c = blockIdx.y * kUnWarps + warp;
  if (c >= nw) return;
  const Z* A = Aall + (size_t)m * n * n;
  const Z* tau = tauall + (size_t)m * n;
  Z* x = reinterpret_cast<Z*>(hb_smem) + (size_t)warp * n;
  const double* z = zall + ((size_t)m * nw + c) * n;
  for (int i = lane; i < n; i += 32) x[i] = zmk(z[i], 0.0);
  __syncwarp();
  for (int j = n - 2; j >= 0; --j) {
    const Z tj = tau[j];
    if (tj.x == 0.0 && tj.y == 0.0) continue;
    const Z* col = A + (size_t)j * n;
    Z s = zmk(0.0, 0.0);  // v^H x
    for (int i = j + 1 + lane; i < n; i += 32)
      s = zfmac(i == j + 1 ? zmk(1.0, 0.0) : col[i], x[i], s);
    const double st = warp_sum2(s.x, s.y, lane);
    s = zmk(__shfl_sync(0xffffffffu, st, 0), __shfl_sync(0xffffffffu, st, 16));
    const Z f = zmul(tj, s);
    for (int i = j + 1 + lane; i < n; i += 32) {
      const Z vi = (i == j + 1) ? zmk(1.0, 0.0) : col[i];
      x[i] = zfnms(f, vi, x[i]);
    }
    __syncwarp();
  }
  Z* xo = xall + ((size_t)m * nw + c) * n;
  for (int i = lane; i < n; i += 32) xo[i] = x[i];
}

// the vectors into the first nw columns of each matrix
__global__ void k_put_vectors(const Z* __restrict__ xall, int n, int nw, long nmat,
                              Z* __restrict__ Aall) {
  const long per = (long)n * nw;
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < nmat * per;
       t += (long)gridDim.x * blockDim.x) {
    const long m = t / per, r = t - m * per;
    Aall[m * (long)n * n + r] = xall[t];
  }
}

size_t hetrd_smem(int n) { return (size_t)(4 + kWarps) * n * sizeof(Z); }

// Blocks per matrix: the cluster size G of the least estimated time, the
// number of rounds that nmat clusters need (the clusters of G that the device
// holds at once, one block per SM) times the time of one, which falls as
// 1 / G + 64 / n (measured, 42 or 20 matrices, whole band solve without
// vectors: n = 377 G = 1 48.5 ms, 2 28.4, 3 21.9, 6 15.6, and 42 clusters of 4
// need a second round: 35.1; n = 219 12.5, 8.2, 6.9, 5.7; n = 73 1.63, 1.43,
// 1.37, 1.30).
cudaError_t cluster_size(cudaLaunchConfig_t cfg, int n, int nmat, int* size) {
  double best = 0.0;
  *size = 1;
  for (int g = 1; g <= 8; ++g) {
    int active = 0;
    cfg.gridDim = dim3((unsigned)g);
    cfg.attrs[0].val.clusterDim.x = (unsigned)g;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&active, k_hetrd, &cfg);
    if (e != cudaSuccess) return e;
    if (active < 1) continue;
    const double t = (double)((nmat + active - 1) / active) * (1.0 / g + 64.0 / n);
    if (g == 1 || t < best) {
      best = t;
      *size = g;
    }
  }
  return cudaSuccess;
}

cudaError_t launch_hetrd(Z* A, int n, int nmat, const Work& wk, cudaStream_t s) {
  // the limit is set to what the largest n needs, the same value from every
  // thread: calls for different n may run at once from several host threads
  cudaError_t e = cudaFuncSetAttribute(k_hetrd, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)hetrd_smem(512));
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = hetrd_smem(n);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int g = 1;
  if ((e = cluster_size(cfg, n, nmat, &g)) != cudaSuccess) return e;
  at[0].val.clusterDim.x = (unsigned)g;
  cfg.gridDim = dim3((unsigned)(nmat * g));
  return cudaLaunchKernelEx(&cfg, k_hetrd, A, n, g, wk.d, wk.e, wk.tau);
}

cudaError_t run_all(Z* A, int n, int nmat, int nw, bool vectors, double* w, const Work& wk,
                    cudaStream_t s) {
  cudaError_t e = launch_hetrd(A, n, nmat, wk, s);
  if (e != cudaSuccess) return e;
  const auto stebz = [&](auto kernel, int sect) {
    const dim3 grid((unsigned)nmat, (unsigned)((sect * nw + 31) / 32));
    kernel<<<grid, 32, 2 * n * sizeof(double), s>>>(wk.d, wk.e, n, nw, w, wk.tnorm);
  };
  // 16 points per round while that gives a sub-partition no more than two
  // warps: a round then takes about as long as with four points, and 13 rounds
  // do for 23.  Beyond it the FP64 pipe is full and the fewer counts of four
  // points (4 x 23 per eigenvalue, not 16 x 13) are the faster.
  if ((long)nmat * nw * 16 <= 2L * 4 * 152 * 32)
    stebz(k_stebz<16>, 16);
  else
    stebz(k_stebz<4>, 4);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (!vectors) return cudaSuccess;
  if ((e = cudaMemsetAsync(wk.info, 0, sizeof(int) * nmat, s)) != cudaSuccess) return e;
  k_stein<<<dim3((unsigned)nmat, (unsigned)nw), 32, stein_smem(n), s>>>(wk.d, wk.e, w, wk.tnorm,
                                                                        n, nw, wk.z, wk.info);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  k_unmtr<<<dim3((unsigned)nmat, (unsigned)((nw + kUnWarps - 1) / kUnWarps)), 32 * kUnWarps,
            (size_t)kUnWarps * n * sizeof(Z), s>>>(A, wk.tau, wk.z, n, nw, wk.x);
  const long tot = (long)nmat * n * nw;
  k_put_vectors<<<(unsigned)std::min<long>((tot + 255) / 256, 152L * 16), 256, 0, s>>>(
      wk.x, n, nw, nmat, A);
  return cudaGetLastError();
}

}  // namespace

size_t work_bytes(int n, int nmat, int nw) {
  const size_t nm = (size_t)nmat;
  return nm * n * sizeof(double) * 2       // d, e
         + nm * n * sizeof(Z)              // tau
         + nm * sizeof(double)             // |T|_1
         + nm * sizeof(int) + 64           // info
         + nm * n * nw * sizeof(double)    // tridiagonal eigenvectors
         + nm * n * nw * sizeof(Z)         // eigenvectors of A
         + 8 * 256;
}

Work carve(void* base, int n, int nmat, int nw) {
  Work wk;
  char* p = static_cast<char*>(base);
  auto take = [&](size_t bytes) {
    char* q = p;
    p += (bytes + 255) & ~(size_t)255;
    return q;
  };
  const size_t nm = (size_t)nmat;
  wk.d = reinterpret_cast<double*>(take(nm * n * sizeof(double)));
  wk.e = reinterpret_cast<double*>(take(nm * n * sizeof(double)));
  wk.tau = reinterpret_cast<Z*>(take(nm * n * sizeof(Z)));
  wk.tnorm = reinterpret_cast<double*>(take(nm * sizeof(double)));
  wk.info = reinterpret_cast<int*>(take(nm * sizeof(int)));
  wk.z = reinterpret_cast<double*>(take(nm * n * nw * sizeof(double)));
  wk.x = reinterpret_cast<Z*>(take(nm * n * nw * sizeof(Z)));
  return wk;
}

bool supported(int n, int nw) { return n >= 2 && n <= 512 && nw >= 1 && nw <= kMaxWanted && nw <= n; }

cudaError_t lowest(Z* A, int n, int nmat, int nw, bool vectors, double* w, void* work,
                   cudaStream_t s) {
  if (!supported(n, nw) || nmat < 1) return cudaErrorInvalidValue;
  const Work wk = carve(work, n, nmat, nw);
  return run_all(A, n, nmat, nw, vectors, w, wk, s);
}

cudaError_t failed_vectors(const void* work, int n, int nmat, int nw, int* host_count,
                           cudaStream_t s) {
  const Work wk = carve(const_cast<void*>(work), n, nmat, nw);
  std::vector<int> h((size_t)nmat);
  cudaError_t e = cudaMemcpyAsync(h.data(), wk.info, sizeof(int) * nmat, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  int c = 0;
  for (int v : h) c += v;
  *host_count = c;
  return e;
}

}  // namespace hb
}  // namespace sep
