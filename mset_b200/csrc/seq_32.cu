// the sequential modes of 32 x 32 windows
#include "seq_kernel.cuh"
MSET_DEFINE_SEQ(32, 8, 1)
