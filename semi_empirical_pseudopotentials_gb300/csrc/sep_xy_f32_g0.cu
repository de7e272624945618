// sep_xy_f32_g0.cu -- the fused xy plane pass for nx in {14, 16, 18, 20, 24, 36, 32, 40}.
#define SEP_XY_GROUP g0
#define SEP_XY_NX(X) X(14) X(16) X(18) X(20) X(24) X(36) X(32) X(40)
#include "sep_xy_impl.cuh"
