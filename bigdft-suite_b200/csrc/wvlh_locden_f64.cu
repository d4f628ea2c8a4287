// FP64 kernels and launcher of the density (wvlh_fused_impl.cuh).
#define WVLH_FUSED_F64
#define WVLH_FUSED_LOCDEN
#define WVLH_FUSED_COMMON
#include "wvlh_fused_impl.cuh"
