// Instances of the tensor-core decode kernel for codes of 5 to 7 bits.
#include "mz_decode_mma.cuh"

bool mz_mma_kernel_wide(int D, int G, int nt, MzMmaKernel* k) { return mzm::pick_instance<0>(D, G, nt, k); }
