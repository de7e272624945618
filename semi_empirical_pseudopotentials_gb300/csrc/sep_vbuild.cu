// sep_vbuild.cu -- local potential on the grid and its backward.
//
// Forward (filter/init.c:157-182, filter/interpolate.c:11-23, with the
// per-atom factor of filterStrainCube/interpolate.c:11-25):
//   potl[g] = sum_a v_{t(a)}(|r_g - R_a|),  v = a r + b on the table segment
//   i = (long)(r / dr), zero when i > n - 2.
// The reference loops over every atom for every point.  Here each block owns
// a brick of grid points, keeps (in atom order) only the atoms whose table
// range reaches the brick, and sums those; the dropped atoms contribute
// exactly zero, so the per-point sum is the reference's, term for term.  What
// the pairs of a segment, or of a brick and an atom, have in common is formed
// once, by the same operations.
// Products and sums are issued with explicit round-to-nearest intrinsics so
// the compiler cannot contract them into FMAs: the result is bit-identical to
// the reference's C loop.
//
// Backward: dL/dtab_v[t][i] (and dL/dscale[a]) from dL/dpotl, through the
// linear interpolation weights v = s ((1 - w) p_i + w p_{i+1}),
// w = (r - r_i) / (r_{i+1} - r_i).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <type_traits>
#include <vector>

#include "../../include/sep_gb300.h"
#include "sep_ctx.cuh"

namespace sep {
int cuda_fail(cudaError_t e, const char* what, int line);
int arg_fail(const char* msg);
}  // namespace sep

using namespace sep;

#define CK(...)                                                  \
  do {                                                            \
    cudaError_t _e = (__VA_ARGS__);                                      \
    if (_e != cudaSuccess) return cuda_fail(_e, #__VA_ARGS__, __LINE__); \
  } while (0)

namespace {

constexpr int BX = 8, BY = 8;  // points per brick in x and y; in z 2 PZ
constexpr int kNT = 128;       // threads per block, PZ z points each
constexpr int kListCap = 512;          // atoms kept per round
constexpr int kTile = 64;              // atoms whose squares are in shared memory at once

struct VArgs {
  const double* xyz;     // natom x 3
  const int* types;
  const double* scale;   // or null
  const double* tab_r;   // ntype x stride
  const double* tab_v;
  const long* tab_n;
  const double* rcut;    // ntype: (n - 1) * dr, beyond which the table gives 0
  double2* seg;          // ntype x stride, made by k_segments
  long long natom;
  long long stride;
  const double* vx;      // axis coordinates (running sums, filter/init.c:157-159)
  const double* vy;
  const double* vz;
  int nx, ny, nz;
};

// What a pair needs of table segment i, once per call: the line (a, b) of the
// forward (filter/interpolate.c:11-23), or (r_i, 1 / (r_{i+1} - r_i)) of the
// backward
__global__ void k_segments(VArgs v, long ntype, int backward) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < ntype * v.stride;
       q += (long long)gridDim.x * blockDim.x) {
    const long t = (long)(q / v.stride), i = (long)(q - t * v.stride);
    if (i > v.tab_n[t] - 2) continue;
    const double* tr = v.tab_r + t * v.stride;
    const double* tv = v.tab_v + t * v.stride;
    if (backward) {
      v.seg[q] = make_double2(tr[i], 1.0 / (tr[i + 1] - tr[i]));
    } else {
      const double a = __dadd_rn(tv[i + 1], -tv[i]) / __dadd_rn(tr[i + 1], -tr[i]);
      v.seg[q] = make_double2(a, __dadd_rn(tv[i], -__dmul_rn(tr[i], a)));
    }
  }
}

// (long)(r / dr) of the reference, -1 beyond segment n - 2, from q = r / dr in
// FP32 (sqrtf of r^2: within 3e-7 relative) unless that leaves the integer
// open: then the division itself.
__device__ __forceinline__ long segment(float q, double r, double dr, long n) {
  const float i = truncf(q), f = q - i, e = 4e-7f * q + 1e-30f;
  if (f > e && f < 1.0f - e) return (long)i > n - 2 ? -1 : (long)i;
  const long k = (long)(r / dr);
  return k > n - 2 ? -1 : k;
}

// distance from point p to the interval [lo, hi] along one axis
__device__ __forceinline__ double gap(double p, double lo, double hi) {
  return p < lo ? lo - p : (p > hi ? p - hi : 0.0);
}

// in-order compaction of the atoms of one kNT-atom chunk that can reach the brick
__device__ int collect(const VArgs& a, long long a0, double bx0, double bx1, double by0,
                       double by1, double bz0, double bz1, int* list, int base) {
  __shared__ int warp_tot[kNT / 32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const long long ai = a0 + tid;
  bool keep = false;
  if (ai < a.natom) {
    const double px = a.xyz[3 * ai], py = a.xyz[3 * ai + 1], pz = a.xyz[3 * ai + 2];
    const double gx = gap(px, bx0, bx1), gy = gap(py, by0, by1), gz = gap(pz, bz0, bz1);
    const double rc = a.rcut[a.types[ai]] * (1.0 + 1e-12) + 1e-12;
    keep = gx * gx + gy * gy + gz * gz <= rc * rc;
  }
  const unsigned m = __ballot_sync(0xffffffffu, keep);
  const int before = __popc(m & ((1u << lane) - 1u));
  if (lane == 0) warp_tot[w] = __popc(m);
  __syncthreads();
  int off = 0, tot = 0;
  for (int k = 0; k < kNT / 32; ++k) {
    if (k < w) off += warp_tot[k];
    tot += warp_tot[k];
  }
  if (keep) list[base + off + before] = (int)ai;
  __syncthreads();
  return tot;
}

// Calls body(u, d, atom, type, segment) in atom order for the PZ points u of
// this thread (x, y, z0 + u of the brick) and every atom whose table reaches
// them; d = |r_g - R_a| with the reference's roundings.  (x - X)^2, (y - Y)^2
// and (z - Z)^2 take 18 to 24 values per atom and brick, which the block forms once,
// so a pair costs one addition and the square root; a third of the pairs of a
// brick lie beyond the table, which FP32 decides where all of a warp do.
template <int PZ, typename F> __device__ __forceinline__ void each_pair(const VArgs& a, F body) {
  constexpr int BZ = kNT / (BX * BY) * PZ;
  __shared__ int list[kListCap];
  __shared__ double sq[kTile][BX + BY + BZ];
  __shared__ int atom_type[kTile];
  __shared__ double tab_dr[kTile];
  __shared__ float tab_inv[kTile], tab_end[kTile];
  const int tid = threadIdx.x;
  const int x = tid % BX, y = tid / BX % BY, z0 = tid / (BX * BY) * PZ;
  const int jx0 = blockIdx.x * BX, jy0 = blockIdx.y * BY, jz0 = blockIdx.z * BZ;
  const int ex = min(jx0 + BX, a.nx) - 1, ey = min(jy0 + BY, a.ny) - 1,
            ez = min(jz0 + BZ, a.nz) - 1;
  const double bx0 = a.vx[jx0], bx1 = a.vx[ex], by0 = a.vy[jy0], by1 = a.vy[ey],
               bz0 = a.vz[jz0], bz1 = a.vz[ez];
  long long a0 = 0;
  while (a0 < a.natom) {
    int cnt = 0;
    // fill the list with up to kListCap kept atoms, in atom order
    while (a0 < a.natom && cnt <= kListCap - kNT) {
      cnt += collect(a, a0, bx0, bx1, by0, by1, bz0, bz1, list, cnt);
      a0 += kNT;
    }
    for (int c0 = 0; c0 < cnt; c0 += kTile) {
      const int m = min(kTile, cnt - c0);
      for (int q = tid; q < m * (BX + BY + BZ); q += kNT) {
        const int k = q / (BX + BY + BZ), p = q - k * (BX + BY + BZ);
        const long long ia = list[c0 + k];
        const double at = p < BX        ? a.vx[min(jx0 + p, ex)]
                          : p < BX + BY ? a.vy[min(jy0 + p - BX, ey)]
                                        : a.vz[min(jz0 + p - BX - BY, ez)];
        const double df = __dadd_rn(at, -a.xyz[3 * ia + (p < BX ? 0 : (p < BX + BY ? 1 : 2))]);
        sq[k][p] = __dmul_rn(df, df);
        if (p == 0) {
          const int t = a.types[ia];
          const double* tr = a.tab_r + t * a.stride;
          const double dr = __dadd_rn(tr[1], -tr[0]);
          atom_type[k] = t;
          tab_dr[k] = dr;
          tab_inv[k] = 1.0f / (float)dr;
          tab_end[k] = (float)a.tab_n[t] * 1.00001f + 1.0f;
        }
      }
      __syncthreads();
      for (int k = 0; k < m; ++k) {
        const int t = atom_type[k];
        const double dr = tab_dr[k];
        const float inv = tab_inv[k], fn = tab_end[k];
        const long n = a.tab_n[t];
        const double xy = __dadd_rn(sq[k][x], sq[k][BX + y]);
#pragma unroll
        for (int u = 0; u < PZ; ++u) {
          const double d2 = __dadd_rn(xy, sq[k][BX + BY + z0 + u]);
          const float q = sqrtf((float)d2) * inv;
          if (q > fn && q < 1e30f) continue;  // past n - 1 by more than the rounding
          const double d = sqrt(d2);
          const long i = segment(q, d, dr, n);
          if (i >= 0) body(u, d, list[c0 + k], t, i);
        }
      }
      __syncthreads();
    }
  }
}

// this thread's points inside the grid: offset of point u, or -1
template <int PZ> __device__ __forceinline__ long long point_of(const VArgs& a, int u) {
  constexpr int BZ = kNT / (BX * BY) * PZ;
  const int tid = threadIdx.x;
  const int jx = blockIdx.x * BX + tid % BX, jy = blockIdx.y * BY + tid / BX % BY,
            jz = blockIdx.z * BZ + tid / (BX * BY) * PZ + u;
  return jx < a.nx && jy < a.ny && jz < a.nz
             ? (long long)a.nx * ((long long)a.ny * jz + jy) + jx
             : -1;
}

// Bound by the FP64 pipe: a pair's sum, square root and line (about 16
// operations; with the two divisions of the segment's line and of r / dr in
// each pair, and a thread per point, about 45).  2260 atoms on 128^3, 310 M
// pairs within the tables: 11.9 ms, 30.1 ms before.
template <int PZ>
__global__ void __launch_bounds__(kNT) k_vbuild(VArgs a, double* __restrict__ potl) {
  double sum[PZ] = {};
  each_pair<PZ>(a, [&](int u, double d, int ia, int t, long i) {
    double2 l;
    if (a.scale) {  // filterStrainCube/interpolate.c:11-25
      const double* tr = a.tab_r + t * a.stride;
      const double* tv = a.tab_v + t * a.stride;
      const double s = a.scale[ia];
      l.x = __dmul_rn(s, __dadd_rn(tv[i + 1], -tv[i])) / __dadd_rn(tr[i + 1], -tr[i]);
      l.y = __dadd_rn(__dmul_rn(s, tv[i]), -__dmul_rn(tr[i], l.x));
    } else {
      l = a.seg[t * a.stride + i];
    }
    sum[u] = __dadd_rn(sum[u], __dadd_rn(__dmul_rn(l.x, d), l.y));
  });
#pragma unroll
  for (int u = 0; u < PZ; ++u) {
    const long long g = point_of<PZ>(a, u);
    if (g >= 0) potl[g] = sum[u];
  }
}

// Bound by the FP64 pipe and by the two shared-memory additions of a pair.
// The same case: 15.7 ms, 30.3 ms before.
template <int PZ>
__global__ void __launch_bounds__(kNT)
k_vbuild_bwd(VArgs a, const double* __restrict__ dpotl, int nbins_smem,
             double* __restrict__ dtab, double* __restrict__ dscale) {
  extern __shared__ double hist[];  // ntype * stride when it fits
  const bool use_smem = nbins_smem > 0;
  for (int i = threadIdx.x; i < nbins_smem; i += blockDim.x) hist[i] = 0.0;
  __syncthreads();
  double gval[PZ];
#pragma unroll
  for (int u = 0; u < PZ; ++u) {
    const long long g = point_of<PZ>(a, u);
    gval[u] = g >= 0 ? dpotl[g] : 0.0;
  }
  each_pair<PZ>(a, [&](int u, double d, int ia, int t, long i) {
    if (gval[u] == 0.0) return;
    const long long b = (long long)t * a.stride + i;
    const double2 l = a.seg[b];
    const double w = (d - l.x) * l.y;
    const double g = a.scale ? gval[u] * a.scale[ia] : gval[u];
    const double g1 = g * w, g0 = g - g1;
    if (use_smem) {
      atomicAdd(&hist[b], g0);
      atomicAdd(&hist[b + 1], g1);
    } else {
      atomicAdd(&dtab[b], g0);
      atomicAdd(&dtab[b + 1], g1);
    }
    if (dscale) {
      const double* tv = a.tab_v + t * a.stride;
      atomicAdd(&dscale[ia], gval[u] * ((1.0 - w) * tv[i] + w * tv[i + 1]));
    }
  });
  __syncthreads();
  for (int i = threadIdx.x; i < nbins_smem; i += blockDim.x)
    if (hist[i] != 0.0) atomicAdd(&dtab[i], hist[i]);
}

// Points per thread, by the 8 x 8 x 8 bricks of the grid.  Small grids have too few
// of them to fill the chip, and a thread's four points add one after another; the
// lists and squares of a brick cost more with smaller ones.  400 atoms, forward /
// backward call in us with 1, 2 and 4 points (a thread per point in 8 x 8 x 4
// bricks, squares and divisions per pair: 14^3 1237 / 1291, 32^3 1258 / 1300):
// 14^3 386 / 622, 656 / 1013, 1165 / 1868; 36^3 (125 bricks) 810 / 1142, 1000 / 1411,
// 1210 / 1955; 48^3 (216) 1550 / 2150, 1472 / 2005, 1855 / 2631; 96^3 (1728) 5344 /
// 6106, 5255 / 5786, 5701 / 6159; 128^3 (4096) 7627 / 7543, 7351 / 6935, 7271 / 6984.
int points_per_thread(const sep_ctx* c) {
  const auto parts = [](long n) { return (n + 7) / 8; };
  const long bricks = parts(c->nx) * parts(c->ny) * parts(c->nz);
  return bricks < 152 ? 1 : bricks < 2048 ? 2 : 4;
}

// launches f(points per thread, grid of bricks)
template <typename F> void with_bricks(const sep_ctx* c, F f) {
  const auto grid = [&](int pz) {
    const int bz = kNT / (BX * BY) * pz;
    return dim3((unsigned)((c->nx + BX - 1) / BX), (unsigned)((c->ny + BY - 1) / BY),
                (unsigned)((c->nz + bz - 1) / bz));
  };
  switch (points_per_thread(c)) {
    case 1: f(std::integral_constant<int, 1>{}, grid(1)); break;
    case 2: f(std::integral_constant<int, 2>{}, grid(2)); break;
    default: f(std::integral_constant<int, 4>{}, grid(4)); break;
  }
}

struct VHost {
  std::vector<double> vx, vy, vz, rcut;
};

int prepare(sep_ctx* c, long natom, const double* xyz, const int* types, const double* scale,
            long ntype, const double* tab_r, const double* tab_v, const long* tab_n,
            long stride, const double mins[3], bool backward, VHost& h, VArgs& a, DevBuf& buf) {
  if (natom < 1 || ntype < 1 || stride < 2 || !xyz || !types || !tab_r || !tab_v || !tab_n ||
      !mins)
    return arg_fail("sep_vbuild: bad argument");
  for (long a_ = 0; a_ < natom; ++a_)
    if (types[a_] < 0 || types[a_] >= ntype) return arg_fail("sep_vbuild: atom type out of range");
  for (long t = 0; t < ntype; ++t)
    if (tab_n[t] < 0 || tab_n[t] > stride) return arg_fail("sep_vbuild: table length > stride");
  h.vx = host::axis_coords(c->nx, mins[0], c->dx);
  h.vy = host::axis_coords(c->ny, mins[1], c->dy);
  h.vz = host::axis_coords(c->nz, mins[2], c->dz);
  h.rcut.assign(ntype, 0.0);
  for (long t = 0; t < ntype; ++t) {
    const long n = tab_n[t];
    if (n >= 2) {
      // i = (long)(r/dr) <= n - 2 needs r < (n - 1) dr
      const double dr = tab_r[t * stride + 1] - tab_r[t * stride];
      h.rcut[t] = (double)(n - 1) * dr;
    }
  }
  const size_t sz_xyz = 3 * (size_t)natom, sz_tab = (size_t)ntype * stride;
  const size_t doubles = sz_xyz + (scale ? natom : 0) + 4 * sz_tab + ntype + c->nx + c->ny +
                         c->nz + 16;
  const size_t bytes = doubles * sizeof(double) + (size_t)natom * sizeof(int) +
                       (size_t)ntype * sizeof(long) + 256;
  CK(buf.ensure(bytes));
  char* p = static_cast<char*>(buf.p);
  auto put = [&](const void* src, size_t nb) {
    void* dst = p;
    cudaMemcpyAsync(dst, src, nb, cudaMemcpyHostToDevice, c->stream);
    p += (nb + 15) / 16 * 16;
    return dst;
  };
  a.xyz = (const double*)put(xyz, sizeof(double) * sz_xyz);
  a.scale = scale ? (const double*)put(scale, sizeof(double) * natom) : nullptr;
  a.tab_r = (const double*)put(tab_r, sizeof(double) * sz_tab);
  a.tab_v = (const double*)put(tab_v, sizeof(double) * sz_tab);
  a.rcut = (const double*)put(h.rcut.data(), sizeof(double) * ntype);
  a.vx = (const double*)put(h.vx.data(), sizeof(double) * c->nx);
  a.vy = (const double*)put(h.vy.data(), sizeof(double) * c->ny);
  a.vz = (const double*)put(h.vz.data(), sizeof(double) * c->nz);
  a.types = (const int*)put(types, sizeof(int) * natom);
  a.tab_n = (const long*)put(tab_n, sizeof(long) * ntype);
  a.seg = reinterpret_cast<double2*>(p);
  a.natom = natom;
  a.stride = stride;
  a.nx = (int)c->nx;
  a.ny = (int)c->ny;
  a.nz = (int)c->nz;
  CK(cudaGetLastError());
  k_segments<<<(unsigned)std::min<size_t>((sz_tab + 255) / 256, 1024), 256, 0, c->stream>>>(
      a, ntype, backward ? 1 : 0);
  CK(cudaGetLastError());
  return kOk;
}

}  // namespace

extern "C" {

int sep_vbuild(sep_ctx* c, long natom, const double* xyz, const int* types, const double* scale,
               long ntype, const double* tab_r, const double* tab_v, const long* tab_n,
               long tab_stride, const double mins[3], double* potl, int install) {
  if (!c) return arg_fail("sep_vbuild: null context");
  CK(cudaSetDevice(c->device));
  DevBuf in;
  VHost h;
  VArgs a;
  int r = prepare(c, natom, xyz, types, scale, ntype, tab_r, tab_v, tab_n, tab_stride, mins,
                  false, h, a, in);
  if (r != kOk) {
    in.release();
    return r;
  }
  double* d_pot = nullptr;
  cudaError_t e = cudaMalloc(&d_pot, sizeof(double) * c->n);
  if (e != cudaSuccess) {
    in.release();
    return cuda_fail(e, "cudaMalloc potl", __LINE__);
  }
  with_bricks(c, [&](auto pz, dim3 g) {
    k_vbuild<decltype(pz)::value><<<g, kNT, 0, c->stream>>>(a, d_pot);
  });
  e = cudaGetLastError();
  if (e == cudaSuccess && potl)
    e = cudaMemcpyAsync(potl, d_pot, sizeof(double) * c->n, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  int rr = (e == cudaSuccess) ? kOk : cuda_fail(e, "vbuild", __LINE__);
  if (rr == kOk && install) rr = sep_ctx_set_potential_dev(c, d_pot);
  cudaStreamSynchronize(c->stream);
  cudaFree(d_pot);
  in.release();
  return rr;
}

int sep_vbuild_backward(sep_ctx* c, long natom, const double* xyz, const int* types,
                        const double* scale, long ntype, const double* tab_r,
                        const double* tab_v, const long* tab_n, long tab_stride,
                        const double mins[3], const double* dpotl, double* dtab_v,
                        double* dscale) {
  if (!c || !dpotl || !dtab_v) return arg_fail("sep_vbuild_backward: null argument");
  CK(cudaSetDevice(c->device));
  DevBuf in;
  VHost h;
  VArgs a;
  int r = prepare(c, natom, xyz, types, scale, ntype, tab_r, tab_v, tab_n, tab_stride, mins,
                  true, h, a, in);
  if (r != kOk) {
    in.release();
    return r;
  }
  const size_t nb = (size_t)ntype * tab_stride;
  double *d_g = nullptr, *d_tab = nullptr, *d_sc = nullptr;
  cudaError_t e = cudaMalloc(&d_g, sizeof(double) * c->n);
  if (e == cudaSuccess) e = cudaMalloc(&d_tab, sizeof(double) * nb);
  if (e == cudaSuccess && dscale) e = cudaMalloc(&d_sc, sizeof(double) * natom);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_g, dpotl, sizeof(double) * c->n, cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_tab, 0, sizeof(double) * nb, c->stream);
  if (e == cudaSuccess && d_sc) e = cudaMemsetAsync(d_sc, 0, sizeof(double) * natom, c->stream);
  if (e == cudaSuccess) {
    // bins in shared memory as far as a block's 48 KB go beside the 16 KB of
    // each_pair; beyond it global atomics are the faster (2260 atoms on 128^3, whole
    // calls: 2 x 2049 to 2 x 2304 bins 42 to 40 ms, 46 with 36 KB of shared bins)
    const int smem_bins = (nb * sizeof(double) <= 32 * 1024) ? (int)nb : 0;
    with_bricks(c, [&](auto pz, dim3 g) {
      k_vbuild_bwd<decltype(pz)::value>
          <<<g, kNT, smem_bins * sizeof(double), c->stream>>>(a, d_g, smem_bins, d_tab, d_sc);
    });
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(dtab_v, d_tab, sizeof(double) * nb, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess && dscale)
    e = cudaMemcpyAsync(dscale, d_sc, sizeof(double) * natom, cudaMemcpyDeviceToHost,
                        c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  cudaFree(d_g);
  cudaFree(d_tab);
  if (d_sc) cudaFree(d_sc);
  in.release();
  return (e == cudaSuccess) ? kOk : cuda_fail(e, "vbuild backward", __LINE__);
}

}  // extern "C"
