// Instances of the tensor-core decode kernel for 3-bit codes.
#include "mz_decode_mma.cuh"

bool mz_mma_kernel_b3(int D, int G, int nt, MzMmaKernel* k) { return mzm::pick_instance<3>(D, G, nt, k); }
