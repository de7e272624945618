// sep_xy_f32_g1.cu -- the fused xy plane pass for nx in {48, 56, 64}.
#define SEP_XY_GROUP g1
#define SEP_XY_NX(X) X(48) X(56) X(64)
#include "sep_xy_impl.cuh"
