// Instances of the tensor-core decode kernel for 8-bit codes.
#include "mz_decode_mma.cuh"

bool mz_mma_kernel_b8(int D, int G, int nt, MzMmaKernel* k) { return mzm::pick_instance<8>(D, G, nt, k); }
