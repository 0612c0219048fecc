// FP32 kernels of planes_sq.cuh, the longer lengths
#include "planes_sq.cuh"

Q3B_SQ_INSTANTIATE(f32_large, float, Q3B_SQ_LARGE)
