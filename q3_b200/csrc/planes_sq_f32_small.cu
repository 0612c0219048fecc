// FP32 kernels of planes_sq.cuh, the shorter lengths
#include "planes_sq.cuh"

Q3B_SQ_INSTANTIATE(f32_small, float, Q3B_SQ_SMALL)
