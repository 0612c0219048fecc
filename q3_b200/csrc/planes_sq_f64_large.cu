// FP64 kernels of planes_sq.cuh, the longer lengths
#include "planes_sq.cuh"

Q3B_SQ_INSTANTIATE(f64_large, double, Q3B_SQ_LARGE)
Q3B_SQ_DENSITY_INSTANTIATE(f64_large, Q3B_SQ_LARGE)
