// sep_xy_f32_g3.cu -- the fused xy plane pass for nx in {96, 112, 128}.
#define SEP_XY_GROUP g3
#define SEP_XY_NX(X) X(96) X(112) X(128)
#include "sep_xy_impl.cuh"
