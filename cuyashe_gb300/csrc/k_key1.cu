// Products with a kept operand (k_mul_key), N = 1024 .. 4096.
#include "kernels.cuh"

namespace cy {

const KeyKernel* key_kernel2(int logn, int l64);

// 64 registers, 80 at N = 4096 (three blocks per SM), as the products that measured fastest
const KeyKernel* key_kernel(int logn, int l64) {
    if (l64 < 0 || l64 > 6) return nullptr;
    switch (logn) {
        case 10: return key_row<10, 16>(l64);
        case 11: return key_row<11, 8>(l64);
        case 12: return key_row<12, 3>(l64);
        case 13:
        case 14: return key_kernel2(logn, l64);
        default: return nullptr;
    }
}

}  // namespace cy
