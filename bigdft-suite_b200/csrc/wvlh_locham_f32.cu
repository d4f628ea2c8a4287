// FP32 kernels and launcher of the local Hamiltonian (wvlh_fused_impl.cuh).
#define WVLH_FUSED_F32
#define WVLH_FUSED_LOCHAM
#include "wvlh_fused_impl.cuh"
