// sep_xy_f32.cu -- dispatch of the fused complex64 Newton step's two passes:
// plane form (sep_xypass.cuh, launched by sep_xy_f32_g*.cu) and sub-plane form
// (sep_sp_f32.cu).
#include "sep_engine.cuh"
#include "sep_xypass.cuh"

namespace sep {

namespace {
// 2: sub-plane form, 1: plane form, 0: none
int xy_form(int nx, int ny, int nz) {
  if (nx == ny && nz == nx && subplane_length(nx)) return 2;
  return plane_pair(nx, ny) ? 1 : 0;
}

int split_n1(int L) {
#define SEP_XY_N1(LL) \
  if (L == LL) return Split<LL>::n1;
  SEP_XY_N1(14) SEP_XY_N1(16) SEP_XY_N1(18) SEP_XY_N1(20) SEP_XY_N1(24) SEP_XY_N1(32)
  SEP_XY_N1(36) SEP_XY_N1(40) SEP_XY_N1(48) SEP_XY_N1(56) SEP_XY_N1(64) SEP_XY_N1(72)
  SEP_XY_N1(80) SEP_XY_N1(96) SEP_XY_N1(112) SEP_XY_N1(128) SEP_XY_N1(160) SEP_XY_N1(192)
  SEP_XY_N1(256)
#undef SEP_XY_N1
  return 0;
}
}  // namespace

int xy_split_x(int nx, int ny, int nz) { return xy_form(nx, ny, nz) ? split_n1(nx) : 0; }

// y: R x (L / R) in the sub-plane form, the line passes' N1 otherwise
int xy_split_y(int nx, int ny, int nz) {
  const int f = xy_form(nx, ny, nz);
  return f == 2 ? subplane_rows(ny) : (f == 1 ? split_n1(ny) : 0);
}

bool xy_supported(const GridDev<float>& g) {
  return g.kxr && g.kyr && xy_form(g.nx, g.ny, g.nz) > 0;
}

cudaError_t xy_prepare(const GridDev<float>& g) {
  if (xy_form(g.nx, g.ny, g.nz) == 2) return subplane_prepare(g.nx);
  if (g.nx <= 40) return xy_prepare_g0(g.nx, g.ny);
  if (g.nx <= 64) return xy_prepare_g1(g.nx, g.ny);
  if (g.nx <= 80) return xy_prepare_g2(g.nx, g.ny);
  return xy_prepare_g3(g.nx, g.ny);
}

cudaError_t run_xy_pass(int mode, const GridDev<float>& g, const PassIO<float>& io, int B,
                        cudaStream_t s) {
  PassArgs<float> a{};
  a.data = io.data;
  a.src = io.src;
  a.psi_in = io.psi_in;
  a.psi_out = io.psi_out;
  a.coefs = io.coefs;
  a.step = io.step;
  a.pot = g.pot;
  a.tw = g.tw[0];
  a.tw_y = g.tw[1];
  a.alpha = io.alpha;
  a.beta = io.beta;
  a.nx = g.nx;
  a.ny = g.ny;
  a.nz = g.nz;
  const int form = xy_form(g.nx, g.ny, g.nz);
  if (form == 2) return subplane_launch(mode, a, B, s);
  if (form != 1) return cudaErrorInvalidValue;
  if (g.nx <= 40) return xy_launch_g0(mode, a, B, s);
  if (g.nx <= 64) return xy_launch_g1(mode, a, B, s);
  if (g.nx <= 80) return xy_launch_g2(mode, a, B, s);
  return xy_launch_g3(mode, a, B, s);
}

// the z pass of the fused step: the z line pass with x and y looked up in
// position order, or (sub-plane form) the zy pass
cudaError_t run_xy_zpass(const GridDev<float>& g, const PassIO<float>& io, int B,
                         cudaStream_t s) {
  const int form = xy_form(g.nx, g.ny, g.nz);
  if (form == 2) return zy_launch(g, io.data, B, s);
  if (form != 1) return cudaErrorInvalidValue;
  GridDev<float> gz = g;
  gz.kx = g.kxr;
  gz.ky = g.kyr;
  return run_pass<float>(2, kFwdKInv, gz, io, B, s);
}

}  // namespace sep
