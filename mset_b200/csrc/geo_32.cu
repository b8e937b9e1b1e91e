// kernels for 32 x 32 windows, and the sequential sessions' shape without scratch
#include "mset_kernels_impl.cuh"
MSET_DEFINE_GEO_SEQ(32, 32, 8, 128, 4)
