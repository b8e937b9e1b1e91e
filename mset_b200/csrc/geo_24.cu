// kernels for 24 x 24 windows, and the sequential sessions' shape without scratch
#include "mset_kernels_impl.cuh"
MSET_DEFINE_GEO_SEQ(24, 24, 8, 192, 4)
