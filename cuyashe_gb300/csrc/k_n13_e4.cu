// Kernel instantiations for N = 8192 with 2^4 coefficients per thread.
#include "kernels.cuh"

namespace cy {
void fill_n13_e4(KernelSet& ks) { fill_kernel_set<13, 4, true, 0, 0, 2, 2>(ks); }
}  // namespace cy
