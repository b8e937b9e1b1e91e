// the sequential modes of 64 x 64 windows
#include "seq_kernel.cuh"
MSET_DEFINE_SEQ(64, 8, 8)
