// Instances of the tensor-core decode kernel for 1-bit codes.
#include "mz_decode_mma.cuh"

bool mz_mma_kernel_b1(int D, int G, int nt, MzMmaKernel* k) { return mzm::pick_instance<1>(D, G, nt, k); }
