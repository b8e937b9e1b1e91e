// kernels for 96 x 96 windows: two CTAs per SM
#include "mset_kernels_impl.cuh"
MSET_DEFINE_GEO(96a, 96, 16, 384, 2)
