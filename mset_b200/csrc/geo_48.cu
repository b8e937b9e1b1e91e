// kernels for 48 x 48 windows: few positions per SM, and the sequential sessions' one-CTA shape
#include "mset_kernels_impl.cuh"
MSET_DEFINE_GEO_SEQ(48, 48, 16, 192, 2)
