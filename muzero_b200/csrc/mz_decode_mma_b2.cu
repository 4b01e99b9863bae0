// Instances of the tensor-core decode kernel for 2-bit codes.
#include "mz_decode_mma.cuh"

bool mz_mma_kernel_b2(int D, int G, int nt, MzMmaKernel* k) { return mzm::pick_instance<2>(D, G, nt, k); }
