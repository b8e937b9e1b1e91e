// kernels for 128 x 128 windows in the sequential sessions' layout
#include "mset_kernels_impl.cuh"
MSET_DEFINE_GEO_SEQ_ONLY(128, 128, 16, 512, 1)
