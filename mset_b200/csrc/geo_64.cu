// 64 x 64 windows: up to 6 positions per SM, and the sequential sessions' one-CTA shape
#include "mset_kernels_impl.cuh"
MSET_DEFINE_GEO_SEQ(64, 64, 8, 256, 2)
