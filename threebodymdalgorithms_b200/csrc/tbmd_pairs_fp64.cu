// The kernels of the FP64 pair-tensor product, a module of their own.
#define TBMD_PAIRS_MODULE 2
#include "tbmd_pairs.cu"
