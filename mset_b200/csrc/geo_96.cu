// kernels for 96 x 96 windows: up to one position per SM, and the sequential sessions' one-CTA shape
#include "mset_kernels_impl.cuh"
MSET_DEFINE_GEO_SEQ(96, 96, 16, 384, 1)
