// The kernels of the mixed pair-tensor adjoint, a module of their own.
#define TBMD_PAIRS_MODULE 1
#include "tbmd_pairs.cu"
