// common.h -- definitions shared by the host set-up code and the CUDA kernels.
#pragma once

#include <stdint.h>
#include <vector_types.h>

namespace cy {

constexpr int KMAX = 40;          // primes per CRT basis
constexpr int L32MAX = 12;        // 32-bit words of q (384 bits)
constexpr int LOGN_MAX = 14;      // N <= 16384
constexpr int NMAX = 1 << LOGN_MAX;
constexpr int TABLE_PRIMES = 64;  // word-sized NTT primes with device twiddle tables
constexpr int PRIME_TWO_ADIC = 16;  // every table prime is 1 mod 2^16
// Length with a 64-coefficients-per-thread schedule (two passes of six stages).
constexpr int ROWS_LOGN = 12;
constexpr int ROWS_N = 1 << ROWS_LOGN;
constexpr int ROWS_G = ROWS_N >> 6;       // threads per transform

// Index of position `pos` in a kept transform of length n (evaluation keys, kept operands):
// the 16-byte pieces of 16 consecutive positions are n / 4 words apart, so that threads with
// 16 (or 8) consecutive positions each load consecutive pieces (a 16-byte load of a warp that
// steps 64 bytes per lane takes four times the L1 cycles).
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int key_index(int pos, int n) {
    return n < 64 ? pos : ((pos >> 2) & 3) * (n >> 2) + (pos >> 4) * 4 + (pos & 3);
}

// What the epilogue of a product kernel computes from the recombined integer X
// (|X| < M/4, M the basis product):
//   MODQ     X mod q                                  -> [N][L] limbs
//   YASHE    round(t*X/q) mod q                       -> [N][L] limbs
//   DECRYPT  round(t*(X mod q)/q) mod t               -> [N] uint64
enum EpiMode { EPI_MODQ = 0, EPI_YASHE = 1, EPI_DECRYPT = 2 };

// Coefficients per thread of the ICRT epilogue kernel for q of l32 words (the
// constants of a prime are read once for all of them); the launch grid is
// ceil(coefficients / (threads * this)).
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int epi_coefs_per_thread(int l32) { return l32 <= 6 ? 2 : 1; }

// Twiddle tables of the first prime; those of prime i follow i tables on. `lanes`: the last
// (forward) or first (inverse) pass's twiddles laid out by lane, for plans with 2^e
// coefficients per thread, e = 4 .. 6 (rows_index; null where no schedule reads them). In the
// natural order a thread with 16 coefficients reads 64 consecutive bytes of a stage, and a warp's
// 16-byte loads step 64 bytes per lane: 16 L1 cycles each instead of four. Measured, natural ->
// lane order: 512 x 14 transforms of length 8192 146 -> 142 us forward, 151 -> 141 inverse; 512
// keyswitches at N = 8192, 190-bit q, 742 -> 717 us; 64 at N = 16384, 380-bit q, 779 -> 756 us.
struct TwiddleTables {
    const uint2* psi;
    const uint2* ipsi;
    const uint2* psi_lanes[3];
    const uint2* ipsi_lanes[3];
};
// The plans of at least 1024 with 16 coefficients per thread, and those with 32 or 64. (With 8 a
// run is 32 bytes: 96 HE multiplies at N = 2048, 62-bit q, 21.15 us with a table, 21.15 without.)
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr bool has_lane_table(int logn, int loge) {
    return logn >= 10 && (loge == 4 || (loge == 5 && logn == LOGN_MAX) || (loge == 6 && logn == ROWS_LOGN));
}
// Entry of a lane-ordered table (G threads per transform) of stage l, twiddle h (< 2^l) and lane
// tau: stage l starts at G (2^l - 1); for l >= 1 the pairs (h, h+1) are 16-byte records
// [h/2][tau].
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int rows_index(int G, int l, int h, int tau) {
    return l == 0 ? tau : G * ((1 << l) - 1) + (h >> 1) * 2 * G + 2 * tau + (h & 1);
}

// Constants of one CRT basis for one ring (N, q). Lives in device memory; the
// kernels read the per-prime fields of their own prime and the epilogue copies
// what it needs into shared memory.
//
// Notation: p_i the basis primes, M = prod p_i, Mhat_i = M/p_i, s = 32*l32 -
// bits(q) the normalising shift so that q' = q << s has its top bit set.
struct BasisDev {
    int n, logn, k, l32, l64, mode, shift, qbits;
    uint32_t t;        // plaintext modulus (YASHE / DECRYPT)
    uint32_t centered; // inputs are taken as symmetric representatives (YASHE)
    uint64_t mu;       // floor(2^(32*l32+37) / q')
    uint64_t mu45;     // floor(2^(32*l32+44) / q')
    uint32_t qn[L32MAX];       // q'
    uint32_t qhalf[L32MAX];    // (q-1)/2
    uint32_t qhalf_n[L32MAX];  // ((q-1)/2) << s
    uint32_t B0[L32MAX];       // MODQ: ((-M) mod q) << s        YASHE: ((-I_M) mod q) << s
    uint32_t B1[L32MAX];       //                                YASHE: (q - R_M) << s
    uint32_t p[KMAX];
    uint32_t p2[KMAX], np[KMAX], np2[KMAX];  // 2p, -p, -2p (mod 2^32), read apart from p (arith.cuh, Mod)
    uint32_t pinv[KMAX];       // p^-1 mod 2^32
    uint32_t ycon[KMAX];       // residue -> [X * Mhat_i^-1]_{p_i} factor (N^-1, Montgomery factors folded)
    uint32_t ycon_sh[KMAX];    // Shoup companion of ycon
    uint32_t flo[KMAX], fhi[KMAX];  // floor(2^64/p_i) split in words (estimate of X'/M)
    uint32_t qmont[KMAX];      // q 2^-32 mod p_i (centering)
    uint32_t crt[KMAX][L32MAX + 1];    // 2^(32 j) mod p_i
    uint32_t A0[KMAX][L32MAX];  // MODQ: (Mhat_i mod q) << s     YASHE: (I_i mod q) << s, t*Mhat_i = I_i q + R_i
    uint32_t A1[KMAX][L32MAX];  //                                YASHE: R_i << s
    uint32_t frac[KMAX][2];     // YASHE: floor(R_i 2^64 / q) (lo, hi words)
    uint32_t frac_m[2];         // YASHE: floor((q - R_M) 2^64 / q)
    const uint2* psi[KMAX];     // forward twiddles (w, floor(w 2^32/p)), bit-reversed powers of psi
    const uint2* ipsi[KMAX];    // inverse twiddles
    TwiddleTables tw;           // (the mixed batches' lane-ordered tables)
};

// What the product, keyswitch and transform kernels read of a basis, passed by value
// as their first parameter: a block reads the constants of its one prime from the
// constant bank with a uniform index, so they are uniform operands (no register file
// ports, no registers) and no dependent loads from memory precede the first coefficient.
// A butterfly whose p, 2p, -p, -2p are registers takes 10.0 cycles of a scheduler, with
// uniform operands 8.9 (the fma-heavy pipe alone needs 8.0; 8 warps per scheduler). In
// the kernels: 512 products at N = 4096, 127-bit q, 192 -> 179 us; 4096 HE multiplies
// 3.13 -> 3.02 ms; one HE multiply 30.7 -> 28.7 us; 509 x 14 inverse transforms of length 8192
// 221 -> 213 us.
struct PrimeParam {
    uint32_t p, p2, np, np2;  // p, 2p, -p, -2p (mod 2^32), each read on its own (arith.cuh, Mod)
    uint32_t pinv;            // p^-1 mod 2^32
    uint32_t cadd;            // 2p - (q 2^-32 mod p): added where q is subtracted (centring)
    uint32_t crt[L32MAX];     // 2^(32 j) mod p
};
struct ProdParams {
    PrimeParam pr[KMAX];
    uint32_t qhalf[L32MAX];  // (q-1)/2
    int k, l64;
    // Kept out of PrimeParam: an address formed from a pointer read with the block's index drags
    // that index, and with it every constant, out of the uniform registers.
    TwiddleTables tw;
};

// The same for the standalone transforms (700 bytes instead of 3 KB to copy per launch).
struct NttParams {
    struct {
        uint32_t p, p2, np, np2;
    } pr[KMAX];
    int k;
    TwiddleTables tw;
};

// One job of a mixed batch (different N and q per job) for the persistent
// kernel k_mixed: a polynomial product (mode MODQ, no keyswitch) or a YASHE
// multiply (tensor with the rounding epilogue, then optionally the keyswitch).
struct MixedJob {
    const BasisDev* B;   // product / tensor basis
    const BasisDev* B2;  // keyswitch basis (YASHE with relinearisation), else null
    const uint64_t* a;
    const uint64_t* b;
    uint64_t* c;
    uint32_t* resid;     // [max(k, k2)][N] residues of this job in the batch scratch
    const void* epi;     // EpiConst of B and of B2 (constants of the epilogues)
    const void* epi2;
    const uint32_t* evk; // keyswitch key [ell][k2][N] (NTT domain, times 2^32)
    int logn, k, l32, l64;
    int mode;            // EPI_MODQ (product) or EPI_YASHE (tensor rounding)
    int centered;        // inputs taken as symmetric representatives (YASHE)
    int k2, ell;         // keyswitch primes and digits (k2 = 0: none)
    int n_epi;           // epilogue units of the job (each phase)
    int need0;           // NTT units' primes the first epilogue waits for (k unless a test starves it)
};

// A unit of work claimed by one block: kind 0 runs the forward/pointwise/inverse
// transforms of `count` consecutive primes of a job starting at `first`; kind 1
// the job's first epilogue over coefficients [first, first + count) once all
// its kind-0 primes are done; kind 2 the keyswitch transforms of `count` primes
// once every kind-1 unit of the job is done; kind 3 the keyswitch's mod-q
// epilogue once every kind-2 prime is done.
struct MixedUnit {
    int job, kind, first, count;
};

}  // namespace cy
