// FP64 gradient kernels (see stage_impl.cuh).
#define CCFD_GRAD_T double
#define CCFD_GRAD_SUFFIX fp64
#include "gradients.inc"
