// the sequential modes of 128 x 128 windows
#include "seq_kernel.cuh"
MSET_DEFINE_SEQ(128, 16, 8)
