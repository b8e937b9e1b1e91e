// the sequential modes of 96 x 96 windows
#include "seq_kernel.cuh"
MSET_DEFINE_SEQ(96, 16, 16)
