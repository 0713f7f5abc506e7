// Products with a kept operand (k_mul_key), N = 1024 .. 4096.
#include "kernels.cuh"

namespace cy {

#define CY_KEY(LOGN, L64, MINB) \
    {(void*)k_mul_key<LOGN, 4, L64, MINB>, NttPlan<LOGN, 4>::G, region_bytes<NttPlan<LOGN, 4>, 2>()}
#define CY_KEY_ROW(LOGN, MINB)                                                                              \
    {CY_KEY(LOGN, 0, MINB), CY_KEY(LOGN, 1, MINB), CY_KEY(LOGN, 2, MINB), CY_KEY(LOGN, 3, MINB), CY_KEY(LOGN, 4, MINB), \
     CY_KEY(LOGN, 5, MINB), CY_KEY(LOGN, 6, MINB)}

const KeyKernel* key_kernel2(int logn, int l64);

// 16 coefficients per thread; 64 registers, 80 at N = 4096 (three blocks per SM), as the
// products that measured fastest
const KeyKernel* key_kernel(int logn, int l64) {
    static const KeyKernel table[3][7] = {CY_KEY_ROW(10, 16), CY_KEY_ROW(11, 8), CY_KEY_ROW(12, 3)};
    if (logn < 10 || logn > 14 || l64 < 0 || l64 > 6) return nullptr;
    return logn <= 12 ? &table[logn - 10][l64] : key_kernel2(logn, l64);
}

}  // namespace cy
