// kernels for 48 x 48 windows: many positions per SM
#include "mset_kernels_impl.cuh"
MSET_DEFINE_GEO(48a, 48, 16, 192, 4)
