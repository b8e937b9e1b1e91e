// the sequential modes of 160 x 160 windows
#include "seq_kernel.cuh"
MSET_DEFINE_SEQ(160, 16, 16)
