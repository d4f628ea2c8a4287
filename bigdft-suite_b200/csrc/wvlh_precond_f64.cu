// FP64 kernels and launcher of the preconditioner (wvlh_fused_impl.cuh).
#define WVLH_FUSED_F64
#define WVLH_FUSED_PRECOND
#include "wvlh_fused_impl.cuh"
