// Epilogues for any prime count, q of 10 to 12 words (k_epi_c with K = 0).
#include "kernels.cuh"

namespace cy {

#define CY_EPI_ANY(L, MODE)                                                               \
    {(void*)k_epi_c<L, MODE, 0>, sizeof(EpiConst<L, KMAX>), fill_epi_const<L, KMAX>, \
     MODE == EPI_MODQ ? (void*)k_epi_c<L, EPI_MODQ, 0, true> : nullptr}
#define CY_EPI_ROW(L) {CY_EPI_ANY(L, EPI_MODQ), CY_EPI_ANY(L, EPI_YASHE), CY_EPI_ANY(L, EPI_DECRYPT)}

const EpiConstKernel* epi_any3(int l32, int mode) {
    static const EpiConstKernel table[][3] = {CY_EPI_ROW(10), CY_EPI_ROW(11), CY_EPI_ROW(12)};
    return &table[l32 - 10][mode];
}

}  // namespace cy
