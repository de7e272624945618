// sep_xy_impl.cuh -- launches of the fused xy plane pass (complex64) for the
// lengths nx of one translation unit (SEP_XY_GROUP, SEP_XY_NX).
#pragma once

#include "sep_engine.cuh"
#include "sep_xypass.cuh"

namespace sep {

namespace {

template <int LX, int LY>
cudaError_t launch_xy(int mode, const PassArgs<float>& a, int B, cudaStream_t s) {
  using T = XyTune<LX, LY>;
  using S = XyShape<LX, LY, T::nt>;
  if (a.nz > 65535 || B < 1) return cudaErrorInvalidValue;
  // planes up to 64^2 take one block each (several per SM); larger planes:
  // min_blocks blocks per SM walk the planes
  const long long planes = (long long)B * a.nz;
  if (planes > 0x7fffffffLL) return cudaErrorInvalidValue;
  const long long walkers = (long long)sm_count() * T::min_blocks;
  const int grid = (T::area <= 4096 || planes < walkers) ? (int)planes : (int)walkers;
  xy_plane_pass<LX, LY><<<grid, T::nt, S::smem_bytes, s>>>(a, B, mode);
  return cudaGetLastError();
}

template <int LX, int LY> cudaError_t prepare_xy() {
  return cudaFuncSetAttribute(xy_plane_pass<LX, LY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)XyShape<LX, LY, XyTune<LX, LY>::nt>::smem_bytes);
}

#define SEP_XY_NY(X, LX)                                                                      \
  X(LX, 14) X(LX, 16) X(LX, 18) X(LX, 20) X(LX, 24) X(LX, 32) X(LX, 36) X(LX, 40) X(LX, 48)   \
  X(LX, 56) X(LX, 64) X(LX, 72) X(LX, 80) X(LX, 96) X(LX, 112) X(LX, 128)

template <int LX> cudaError_t launch_nx(int mode, const PassArgs<float>& a, int B, cudaStream_t s) {
#define SEP_XY_RUN(LX_, LY_)      \
  if constexpr (plane_pair(LX_, LY_)) \
    if (a.ny == LY_) return launch_xy<LX_, LY_>(mode, a, B, s);
  SEP_XY_NY(SEP_XY_RUN, LX)
#undef SEP_XY_RUN
  return cudaErrorInvalidValue;
}

template <int LX> cudaError_t prepare_nx(int ny) {
#define SEP_XY_PREP(LX_, LY_)     \
  if constexpr (plane_pair(LX_, LY_)) \
    if (ny == LY_) return prepare_xy<LX_, LY_>();
  SEP_XY_NY(SEP_XY_PREP, LX)
#undef SEP_XY_PREP
  return cudaErrorInvalidValue;
}

}  // namespace

#define SEP_XY_CAT_(a, b) a##b
#define SEP_XY_CAT(a, b) SEP_XY_CAT_(a, b)

cudaError_t SEP_XY_CAT(xy_launch_, SEP_XY_GROUP)(int mode, const PassArgs<float>& a, int B,
                                                 cudaStream_t s) {
#define SEP_XY_L(LX_) \
  if (a.nx == LX_) return launch_nx<LX_>(mode, a, B, s);
  SEP_XY_NX(SEP_XY_L)
#undef SEP_XY_L
  return cudaErrorInvalidValue;
}

cudaError_t SEP_XY_CAT(xy_prepare_, SEP_XY_GROUP)(int nx, int ny) {
#define SEP_XY_P(LX_) \
  if (nx == LX_) return prepare_nx<LX_>(ny);
  SEP_XY_NX(SEP_XY_P)
#undef SEP_XY_P
  return cudaErrorInvalidValue;
}

}  // namespace sep
