// bw_group_f64.cu -- group launches: 64-bit path: 32-bit coefficients in double-precision arithmetic.
#include "bw_group.cuh"

template cudaError_t bw_enqueue_group_of<ArD<0>, false>(const bw_group_launch&, cudaStream_t);
