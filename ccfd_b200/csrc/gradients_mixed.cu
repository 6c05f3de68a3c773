// Mixed-precision (FP32) gradient kernels (see stage_impl.cuh).
#define CCFD_GRAD_T float
#define CCFD_GRAD_SUFFIX fp32
#include "gradients.inc"
