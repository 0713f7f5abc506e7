// Products with a kept operand (k_mul_key), N = 8192 and 16384.
#include "kernels.cuh"

namespace cy {

#define CY_KEY(LOGN, L64, MINB) \
    {(void*)k_mul_key<LOGN, 4, L64, MINB>, NttPlan<LOGN, 4>::G, region_bytes<NttPlan<LOGN, 4>, 2>()}
#define CY_KEY_ROW(LOGN, MINB)                                                                              \
    {CY_KEY(LOGN, 0, MINB), CY_KEY(LOGN, 1, MINB), CY_KEY(LOGN, 2, MINB), CY_KEY(LOGN, 3, MINB), CY_KEY(LOGN, 4, MINB), \
     CY_KEY(LOGN, 5, MINB), CY_KEY(LOGN, 6, MINB)}

const KeyKernel* key_kernel2(int logn, int l64) {
    static const KeyKernel table[2][7] = {CY_KEY_ROW(13, 2), CY_KEY_ROW(14, 1)};
    return &table[logn - 13][l64];
}

}  // namespace cy
