// bw_group_p32.cu -- group launches: 32-bit path, 16-bit coefficients.
#include "bw_group.cuh"

template cudaError_t bw_enqueue_group_of<Ar32, true>(const bw_group_launch&, cudaStream_t);
