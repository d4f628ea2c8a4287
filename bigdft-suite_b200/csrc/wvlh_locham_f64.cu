// FP64 kernels and launcher of the local Hamiltonian (wvlh_fused_impl.cuh).
#define WVLH_FUSED_F64
#define WVLH_FUSED_LOCHAM
#include "wvlh_fused_impl.cuh"
