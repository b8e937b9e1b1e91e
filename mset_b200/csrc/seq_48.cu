// the sequential modes of 48 x 48 windows
#include "seq_kernel.cuh"
MSET_DEFINE_SEQ(48, 16, 8)
