// 64 x 64 windows: many positions per SM
#include "mset_kernels_impl.cuh"
MSET_DEFINE_GEO(64p, 64, 8, 128, 4)
