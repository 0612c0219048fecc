// FP64 kernels of planes_sq.cuh, the shorter lengths
#include "planes_sq.cuh"

Q3B_SQ_INSTANTIATE(f64_small, double, Q3B_SQ_SMALL)
Q3B_SQ_DENSITY_INSTANTIATE(f64_small, Q3B_SQ_SMALL)
