// sep_xy_f32_g2.cu -- the fused xy plane pass for nx in {72, 80}.
#define SEP_XY_GROUP g2
#define SEP_XY_NX(X) X(72) X(80)
#include "sep_xy_impl.cuh"
