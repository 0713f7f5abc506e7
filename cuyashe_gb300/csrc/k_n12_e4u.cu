// Kernel instantiations for N = 4096 with 2^4 coefficients per thread: three product
// blocks per SM (80 registers), the keyswitch with the whole register file.
#include "kernels.cuh"

namespace cy {
void fill_n12_e4u(KernelSet& ks) { fill_kernel_set<12, 4, true, 3, 1>(ks); }
}  // namespace cy
