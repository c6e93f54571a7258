// The kernels of linear_attn_tc.cu for decays by head and silu of q, k and v (vy_linear_attn): an object per build of the kernels whose warps share registers out
#define VY_LA_FIXED
#include "linear_attn_tc.cu"
