// Products with a kept operand (k_mul_key), N = 8192 and 16384.
#include "kernels.cuh"

namespace cy {

const KeyKernel* key_kernel2(int logn, int l64) { return logn == 13 ? key_row<13, 2>(l64) : key_row<14, 1>(l64); }

}  // namespace cy
