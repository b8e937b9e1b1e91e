// the sequential modes of 24 x 24 windows
#include "seq_kernel.cuh"
MSET_DEFINE_SEQ(24, 8, 1)
