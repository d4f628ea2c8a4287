// FP32 kernels and launcher of the density (wvlh_fused_impl.cuh).
#define WVLH_FUSED_F32
#define WVLH_FUSED_LOCDEN
#include "wvlh_fused_impl.cuh"
