// the sequential modes of 256 x 256 windows
#include "seq_kernel.cuh"
MSET_DEFINE_SEQ(256, 16, 16)
