// Instances of the tensor-core decode kernel for 4-bit codes.
#include "mz_decode_mma.cuh"

bool mz_mma_kernel_b4(int D, int G, int nt, MzMmaKernel* k) { return mzm::pick_instance<4>(D, G, nt, k); }
