// k_axis_f64.cu -- the double form of the kernels of k_axis.cuh.
#include "k_axis.cuh"

cudaError_t launch_axis_f64(const LineParams &p, cudaStream_t s) { return axis::launch<double>(p, s); }
