// Epilogues with their constants as a kernel parameter (k_epi_c): for any prime count,
// for every number of words of q, in k_epi_any1.cu .. k_epi_any3.cu, and here those
// compiled for the prime counts of the common parameter sets: 4-word q (N = 4096, 127-bit
// q: tensor 9, keyswitch 6, product 9 primes), 2-word q (62-bit, N = 2048: 5 / 4), 6-word q
// (190-bit, N = 8192: 14 / 8) and 12-word q (380-bit, N = 16384: 26 / 15).
#include "kernels.cuh"

namespace cy {

namespace {
struct EpiEntry {
    int l32, k, mode;
    EpiConstKernel s;
};
}  // namespace

#define CY_EPI_K(L, K, MODE) {L, K, MODE, {(void*)k_epi_c<L, MODE, K>, sizeof(EpiConst<L, K>), fill_epi_const<L, K>, nullptr}}
// with the kernel for any X, for cy_icrt at 127-bit q: 500 polynomials of N = 4096 27.6 us, 39 without
// the prime count, 52 with the constants in shared memory (k_epi)
#define CY_EPI_KX(L, K)                                                                                     \
    {L, K, EPI_MODQ,                                                                                        \
     {(void*)k_epi_c<L, EPI_MODQ, K>, sizeof(EpiConst<L, K>), fill_epi_const<L, K>, (void*)k_epi_c<L, EPI_MODQ, K, true>}}

static const EpiEntry kEpiSpecial[] = {
    CY_EPI_K(4, 9, EPI_YASHE),   CY_EPI_K(4, 6, EPI_MODQ),  CY_EPI_KX(4, 9),
    CY_EPI_K(2, 5, EPI_YASHE),   CY_EPI_K(2, 4, EPI_MODQ),  CY_EPI_K(6, 14, EPI_YASHE),
    CY_EPI_K(6, 8, EPI_MODQ),    CY_EPI_K(12, 26, EPI_YASHE), CY_EPI_K(12, 15, EPI_MODQ),
};

const EpiConstKernel* epi_any1(int l32, int mode);  // 1 .. 5 words
const EpiConstKernel* epi_any2(int l32, int mode);  // 6 .. 9
const EpiConstKernel* epi_any3(int l32, int mode);  // 10 .. 12

const EpiConstKernel* epi_const_any(int l32, int mode) {
    if (l32 < 1 || l32 > L32MAX || mode < 0 || mode > 2) return nullptr;
    return l32 <= 5 ? epi_any1(l32, mode) : l32 <= 9 ? epi_any2(l32, mode) : epi_any3(l32, mode);
}

const EpiConstKernel* epi_const(int l32, int k, int mode) {
    for (const EpiEntry& e : kEpiSpecial)
        if (e.l32 == l32 && e.k == k && e.mode == mode) return &e.s;
    return k >= 1 && k <= KMAX ? epi_const_any(l32, mode) : nullptr;
}

}  // namespace cy
