// The step's kernels for one storage type and group (IW_INST): 1, 2 the x and y
// transforms (FP32, FP64), 3, 4 the z-column kernels and the solves.
#include "iw_lib.cu"
