// kernels.cuh -- CUDA kernels of the multiply path (templates; instantiated in
// the k_*.cu translation units).
//
//   k_mul        per (job, prime): CRT split of a and b -> forward NTTs ->
//                pointwise Montgomery product -> inverse NTT -> residues.
//                Replaces callCRT (src/cuda_bn.cu:970-1002) and the NTT branch of
//                callPolynomialMul (src/cuda_functions.cu:658-738).
//   k_keyswitch  per (job, prime): base-2^32 digits of c -> forward NTTs ->
//                sum_d D_d * evk_d in the NTT domain -> inverse NTT -> residues.
//                Replaces Ciphertext::keyswitch (src/ciphertext.cpp:81-107).
//   k_epi        per coefficient: ICRT of the k residues to the exact integer,
//                then mod q, round(t/q .) or decryption. Replaces cuPreICRT /
//                cuICRT / cuModN (src/cuda_bn.cu:759-968), Polynomial::reduce's
//                mod q (src/cuda_functions.cu:1076) and the host rounding loop
//                of Ciphertext::operator* (src/ciphertext.cpp:55-63).
//   k_ntt, k_crt standalone transforms (callNTT, callCRT).
#pragma once

#include <stdint.h>

#include "arith.cuh"
#include "common.h"
#include "dispatch.h"
#include "ntt_core.cuh"

namespace cy {

// Bytes of the exchange buffer of NOPS operands.
template <class PL, int NOPS>
__host__ __device__ constexpr size_t region_bytes() {
    return (size_t)NOPS * PL::SMW * 4;
}

// The modulus of prime i with its derived constants, each read on its own.
__device__ __forceinline__ Mod load_mod(const BasisDev* __restrict__ B, int i) {
    Mod m;
    m.p = B->p[i];
    m.p2 = B->p2[i];
    m.np = B->np[i];
    m.np2 = B->np2[i];
    return m;
}

// The tables of prime i.
__device__ __forceinline__ const uint2* table_of(const uint2* base, int i) { return base + (size_t)i * NMAX; }
template <class PL>
__device__ __forceinline__ auto lanes_of(const uint2* const (&tab)[3], int i) {
    if constexpr (has_lane_table(PL::LOGN, PL::LOGE)) return tab[PL::LOGE - 4] + (size_t)i * (PL::N - PL::G);
    else return NoLanes();
}
template <class Param>  // PrimeParam, or a prime of NttParams
__device__ __forceinline__ Mod load_mod(const Param& q) {
    return Mod{q.p, q.p2, q.np, q.np2};
}

// a + b reduced from [0, 4p) to [0, 2p) (a, b in [0, 2p)): one add, one add-then-min
__device__ __forceinline__ uint32_t mac_red(uint32_t a, uint32_t b, const Mod& m) {
    return __viaddmin_u32(a, b, a + b + m.np2);
}

// Per-prime constants a product kernel keeps in registers.
struct PrimeCtx {
    uint32_t p, pinv, cadd;  // p, p^-1 mod 2^32, 2p - (q 2^-32 mod p)
    Mod m;
};

__device__ __forceinline__ PrimeCtx load_prime_ctx(const BasisDev* __restrict__ B, int i) {
    PrimeCtx c;
    c.m = load_mod(B, i);
    c.p = c.m.p;
    c.pinv = B->pinv[i];
    c.cadd = c.m.p2 - B->qmont[i];
    return c;
}

__device__ __forceinline__ PrimeCtx load_prime_ctx(const PrimeParam& q) {
    return PrimeCtx{q.p, q.pinv, q.cadd, load_mod(q)};
}

// x 2^-32 mod p in (0, 4p) (valid forward-NTT input) from T = x + a multiple of p,
// T < 4p 2^32: T and m p (m = T p^-1 mod 2^32) have equal low words, so the
// difference of the high words is exact. REDUCE: T's high word may reach 2p and is
// brought below it first. neg: all ones where q is to be subtracted from x, else 0.
template <bool REDUCE>
__device__ __forceinline__ uint32_t crt_finish(uint64_t T, uint32_t neg, const PrimeCtx& c) {
    uint32_t hi = (uint32_t)(T >> 32);
    if (REDUCE) hi = __viaddmin_u32(hi, c.m.np2, hi);
    const uint32_t h = __umulhi((uint32_t)T * c.pinv, c.p);
    return hi - h + (c.p ^ (neg & (c.p ^ c.cadd)));  // (-p, 2p) + p, or + 2p - (q 2^-32 mod p)
}

// T with its high word (below 4p) brought below 2p: the same residue, and two more
// products of a word and a residue fit.
__device__ __forceinline__ uint64_t lazy_high(uint64_t T, const Mod& m) {
    const uint32_t hi = (uint32_t)(T >> 32);
    return (uint64_t)__viaddmin_u32(hi, m.np2, hi) << 32 | (uint32_t)T;
}

// Residue (times 2^-32) in (0, 4p) of coefficient `pos` of a polynomial stored as
// [N][l64] limbs. `crt` holds 2^(32 j) mod p for j < 2*l64 <= L32MAX.
// With CENTER, values above (q-1)/2 stand for x - q.
template <bool CENTER>
__device__ __forceinline__ uint32_t crt_coef(const uint64_t* __restrict__ src, int pos, int l64,
                                             const uint32_t* crt, const uint32_t* qhalf, const PrimeCtx& c) {
    const uint64_t* s = src + (size_t)pos * l64;
    uint64_t T = 0;
    bool gt = false;
    for (int j = 0; j < l64; j++) {
        const uint64_t limb = ld_dep(s + j);
        const uint32_t lo = (uint32_t)limb, hi = (uint32_t)(limb >> 32);
        T = lazy_high(T, c.m) + (uint64_t)lo * crt[2 * j] + (uint64_t)hi * crt[2 * j + 1];
        if (CENTER) {
            const uint64_t h = (uint64_t)qhalf[2 * j + 1] << 32 | qhalf[2 * j];
            gt = limb > h || (limb == h && gt);
        }
    }
    return crt_finish<true>(T, gt ? ~0u : 0u, c);
}

// The limbs of one coefficient as 32-bit words (16-byte loads when L64 is even).
template <int L64>
__device__ __forceinline__ void load_words(const uint64_t* __restrict__ p, uint32_t (&w)[2 * L64]) {
    if constexpr (L64 % 2 == 0) {
#pragma unroll
        for (int i = 0; i < L64 / 2; i++) {
            const uint4 v = ld_dep(reinterpret_cast<const uint4*>(p) + i);
            w[4 * i] = v.x;
            w[4 * i + 1] = v.y;
            w[4 * i + 2] = v.z;
            w[4 * i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < L64; i++) {
            const uint2 v = ld_dep(reinterpret_cast<const uint2*>(p) + i);
            w[2 * i] = v.x;
            w[2 * i + 1] = v.y;
        }
    }
}

// All ones when x (words w) is above (q-1)/2 (words qh), else 0: (q-1)/2 - x borrows
// exactly then, so one subtract-with-borrow chain and its final borrow spread to a
// mask (no compares, no selects, no branches).
template <int W>
__device__ __forceinline__ uint32_t above_half(const uint32_t (&w)[W], const uint32_t (&qh)[W]) {
    static_assert(W % 2 == 0 && W >= 2 && W <= 12, "an even number of words");
    // 64-bit words: each asm statement must hold the whole chain (the carry flag does
    // not outlive it), so one statement per width
    auto v = [&](int i) { return (uint64_t)w[2 * i + 1] << 32 | w[2 * i]; };
    auto h = [&](int i) { return (uint64_t)qh[2 * i + 1] << 32 | qh[2 * i]; };
    uint32_t mask;
    if constexpr (W == 2) {
        asm("{\n\t.reg .u64 d;\n\tsub.cc.u64 d, %1, %2;\n\tsubc.u32 %0, 0, 0;\n\t}"
            : "=r"(mask) : "l"(h(0)), "l"(v(0)));
    } else if constexpr (W == 4) {
        asm("{\n\t.reg .u64 d;\n\tsub.cc.u64 d, %1, %2;\n\tsubc.cc.u64 d, %3, %4;\n\tsubc.u32 %0, 0, 0;\n\t}"
            : "=r"(mask) : "l"(h(0)), "l"(v(0)), "l"(h(1)), "l"(v(1)));
    } else if constexpr (W == 6) {
        asm("{\n\t.reg .u64 d;\n\tsub.cc.u64 d, %1, %2;\n\tsubc.cc.u64 d, %3, %4;\n\tsubc.cc.u64 d, %5, %6;\n\t"
            "subc.u32 %0, 0, 0;\n\t}"
            : "=r"(mask) : "l"(h(0)), "l"(v(0)), "l"(h(1)), "l"(v(1)), "l"(h(2)), "l"(v(2)));
    } else if constexpr (W == 8) {
        asm("{\n\t.reg .u64 d;\n\tsub.cc.u64 d, %1, %2;\n\tsubc.cc.u64 d, %3, %4;\n\tsubc.cc.u64 d, %5, %6;\n\t"
            "subc.cc.u64 d, %7, %8;\n\tsubc.u32 %0, 0, 0;\n\t}"
            : "=r"(mask)
            : "l"(h(0)), "l"(v(0)), "l"(h(1)), "l"(v(1)), "l"(h(2)), "l"(v(2)), "l"(h(3)), "l"(v(3)));
    } else if constexpr (W == 10) {
        asm("{\n\t.reg .u64 d;\n\tsub.cc.u64 d, %1, %2;\n\tsubc.cc.u64 d, %3, %4;\n\tsubc.cc.u64 d, %5, %6;\n\t"
            "subc.cc.u64 d, %7, %8;\n\tsubc.cc.u64 d, %9, %10;\n\tsubc.u32 %0, 0, 0;\n\t}"
            : "=r"(mask)
            : "l"(h(0)), "l"(v(0)), "l"(h(1)), "l"(v(1)), "l"(h(2)), "l"(v(2)), "l"(h(3)), "l"(v(3)), "l"(h(4)),
              "l"(v(4)));
    } else {
        asm("{\n\t.reg .u64 d;\n\tsub.cc.u64 d, %1, %2;\n\tsubc.cc.u64 d, %3, %4;\n\tsubc.cc.u64 d, %5, %6;\n\t"
            "subc.cc.u64 d, %7, %8;\n\tsubc.cc.u64 d, %9, %10;\n\tsubc.cc.u64 d, %11, %12;\n\t"
            "subc.u32 %0, 0, 0;\n\t}"
            : "=r"(mask)
            : "l"(h(0)), "l"(v(0)), "l"(h(1)), "l"(v(1)), "l"(h(2)), "l"(v(2)), "l"(h(3)), "l"(v(3)), "l"(h(4)),
              "l"(v(4)), "l"(h(5)), "l"(v(5)));
    }
    return mask;
}

// Residue (times 2^-32) in (0, 4p) of the coefficient whose 32-bit words are w
// (compile-time count W); cc[j] = 2^(32 j) mod p. With CENTER, values above (q-1)/2
// (words qh) stand for x - q. The factor 2^-32 is folded into the ICRT constants,
// so that word 0 needs no product and one Montgomery step (a multiply, a mul.hi)
// ends the sum. The fma-heavy pipe bounds these kernels (mul.hi and wide products take
// four of its cycles per warp, other multiplies two): the sum of W products and two
// Shoup reductions per four words that this replaces took 32 of them at W = 4 against
// 48 for the coefficient's forward transform, this takes 18. 512 tensor products at
// N = 4096, 127-bit q: 224 -> 194 us; at N = 8192, 190-bit q: 1044 -> 791 us.
template <int W, bool CENTER>
__device__ __forceinline__ uint32_t crt_words(const uint32_t (&w)[W], const uint32_t (&cc)[W],
                                              const uint32_t (&qh)[W], const PrimeCtx& c) {
    uint64_t T = w[0];
#pragma unroll
    for (int j = 1; j < W; j++) {
        if (j >= 4 && j % 2 == 0) T = lazy_high(T, c.m);  // below 2p 2^32, two products more
        T += (uint64_t)w[j] * cc[j];
    }
    return crt_finish<(W > 3)>(T, CENTER ? above_half<W>(w, qh) : 0u, c);
}

// --------------------------------------------------------------------------
// k_mul: one block per (job, prime); G = N/E threads. Jobs are the fast grid
// dimension: the blocks resident at a time then share few primes, so their twiddle
// tables stay in L1 and L2 (512 HE multiplies at N = 8192, 190-bit q: 2.16 -> 2.05 ms;
// within 1% either way at N <= 4096).
// --------------------------------------------------------------------------
// L64 > 0: coefficients have exactly L64 limbs (specialised load and CRT
// split); L64 == 0: the limb count is read from the basis at run time.
// Blocks per SM the product kernel is compiled for: 48 resident warps with 8
// coefficients per thread, 32 with 16 (more registers per thread).
template <int LOGN, int LOGE>
constexpr int mul_min_blocks() {
    constexpr int G = NttPlan<LOGN, LOGE>::G;
    constexpr int target = (LOGE <= 3 ? 1536 : 1024) / G;
    return target < 1 ? 1 : (target > 16 ? 16 : target);
}
template <int LOGN, int LOGE>
__host__ __device__ constexpr int ks_min_blocks() {
    constexpr int G = NttPlan<LOGN, LOGE>::G;
    constexpr int target = 1024 / G;
    return target < 1 ? 1 : (target > 16 ? 16 : target);
}

template <int LOGN, int LOGE>
constexpr int ntt_min_blocks() {
    constexpr int G = NttPlan<LOGN, LOGE>::G;
    constexpr int target = (LOGE <= 4 ? 1024 : 512) / G;
    return target < 1 ? 1 : (target > 16 ? 16 : target);
}

// MINB > 0 overrides the blocks per SM the kernel is compiled for (a schedule
// with a larger register budget per thread).
template <int LOGN, int LOGE, int L64, bool CENTER, int MINB = 0>
__global__ void __launch_bounds__(NttPlan<LOGN, LOGE>::G, (MINB > 0 ? MINB : mul_min_blocks<LOGN, LOGE>()))
    k_mul(const __grid_constant__ ProdParams M, const uint64_t* __restrict__ A, long long a_stride,
          const uint64_t* __restrict__ Bv, long long b_stride, uint32_t* __restrict__ resid) {
    using PL = NttPlan<LOGN, LOGE>;
    constexpr int E = PL::E;
    extern __shared__ __align__(16) uint32_t smem[];  // exchange buffer, 2 operands x SMW
    const int tau = threadIdx.x;
    const int prime = blockIdx.y;
    const int job = blockIdx.x;
    const int k = M.k;
    const PrimeParam& Q = M.pr[prime];
    const PrimeCtx c = load_prime_ctx(Q);
    const uint2* __restrict__ psi = table_of(M.tw.psi, prime);
    const uint2* __restrict__ ipsi = table_of(M.tw.ipsi, prime);

    const uint64_t* a = A + (size_t)job * a_stride;
    const uint64_t* b = Bv + (size_t)job * b_stride;
    dep_wait(a, b);
    uint32_t x[2][E];
    if constexpr (L64 > 0) {
        constexpr int W = 2 * L64;
        uint32_t cc[W], qh[W];
#pragma unroll
        for (int j = 0; j < W; j++) {
            cc[j] = Q.crt[j];
            qh[j] = M.qhalf[j];
        }
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int pos = slot_pos<PL, 0>(tau, e);
            uint32_t wa[W], wb[W];
            load_words<L64>(a + (size_t)pos * L64, wa);
            load_words<L64>(b + (size_t)pos * L64, wb);
            x[0][e] = crt_words<W, CENTER>(wa, cc, qh, c);
            x[1][e] = crt_words<W, CENTER>(wb, cc, qh, c);
        }
    } else {
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int pos = slot_pos<PL, 0>(tau, e);
            x[0][e] = crt_coef<CENTER>(a, pos, M.l64, Q.crt, M.qhalf, c);
            x[1][e] = crt_coef<CENTER>(b, pos, M.l64, Q.crt, M.qhalf, c);
        }
    }
    // 64 coefficients per thread at N = 4096: both transforms loop over one copy of
    // the pass code (the unrolled three transforms overflow the instruction cache)
    constexpr bool LOOP64 = LOGN == 12 && LOGE == 6;
    if constexpr (LOOP64) ntt64_forward<PL, 2>(x, psi, lanes_of<PL>(M.tw.psi_lanes, prime), c.m, tau, smem);
    else ntt_forward<PL, 2>(x, psi, c.m, tau, smem, false, CtaSync(), 1, lanes_of<PL>(M.tw.psi_lanes, prime));
    uint32_t z[1][E];
#pragma unroll
    for (int e = 0; e < E; e++) z[0][e] = mont(red_2p(x[0][e], c.m), red_2p(x[1][e], c.m), c.pinv, c.m);
    if constexpr (LOOP64) ntt64_inverse<PL, 1>(z, ipsi, lanes_of<PL>(M.tw.ipsi_lanes, prime), c.m, tau, smem, nullptr);
    else ntt_inverse<PL, 1>(z, ipsi, c.m, tau, smem, CtaSync(), 1, lanes_of<PL>(M.tw.ipsi_lanes, prime));
    dep_launch();
    uint32_t* out = resid + ((size_t)job * k + prime) * PL::N;
#pragma unroll
    for (int e = 0; e < E; e++) out[slot_pos<PL, 0>(tau, e)] = z[0][e];
}

// --------------------------------------------------------------------------
// k_keyswitch: one block per (job, prime). Digits are the 32-bit words of the
// coefficients of c in [0, q) (w = 2^32), processed ND at a time.
// evk: [ell][k][N] values times 2^32 mod p in the forward-NTT output order (key_index).
// --------------------------------------------------------------------------
// The E key values (key_index order in a row of N) of the consecutive positions pos0 ...
template <int N, int E>
__device__ __forceinline__ void load_evk(const uint32_t* __restrict__ row, int pos0, uint32_t (&v)[E]) {
    if constexpr (E % 4 == 0) {
#pragma unroll
        for (int h = 0; h < E / 4; h++) {
            const uint4 W = __ldg(reinterpret_cast<const uint4*>(row + key_index(pos0 + 4 * h, N)));
            v[4 * h] = W.x;
            v[4 * h + 1] = W.y;
            v[4 * h + 2] = W.z;
            v[4 * h + 3] = W.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = __ldg(row + key_index(pos0 + e, N));
    }
}
// first of thread tau's consecutive positions after the last forward pass
template <class PL>
__device__ __forceinline__ int last_pos(int tau) {
    constexpr int LAST = PL::NPASS - 1;
    static_assert(PL::LOGD(LAST) == 0 && PL::R(LAST) == PL::LOGE, "contiguous last-pass positions");
    return group_base<PL, LAST>(tau, 0);
}

// Sum of up to four products of a digit in [0, 4p) and a key value below p (T < 4p 2^32)
// -> T 2^-32 mod p in [0, 2p). MANY: more than two products since T was below 2^32.
template <bool MANY>
__device__ __forceinline__ uint32_t mac_finish(uint64_t T, uint32_t pinv, const Mod& m) {
    uint32_t hi = (uint32_t)(T >> 32);
    if (MANY) hi = __viaddmin_u32(hi, m.np2, hi);
    return red_2p(hi - __umulhi((uint32_t)T * pinv, m.p) + m.p, m);  // (0, 3p) -> [0, 2p)
}

// The products with the key are summed in 64 bits (one wide multiply-add each) and
// reduced once per coefficient by a Montgomery step; a Shoup product per digit and
// coefficient took three multiplies and twice the key bytes.
// ONE: all digits in one pass (kernels of one or two limbs), no sums kept across
// transforms. Otherwise the 64-bit sums stay in registers where there is room; with more
// than 16 coefficients per thread, or 16 in 64 registers (ACC32), each pass's sums are
// reduced and added to 32-bit ones (three more cycles of the fma-heavy pipe per digit and
// coefficient, but fewer spills: 64 keyswitches at N = 16384, 380-bit q, 1059 -> 821 us; 512 at N =
// 8192, 190-bit q, 948 -> 765 us).
template <int L64, int ND>
__host__ __device__ constexpr bool ks_one_pass() {
    return (L64 == 1 && ND >= 2) || (L64 == 2 && ND >= 4);
}

template <int LOGN, int LOGE, int L64, int ND, int MINB = 0>
__global__ void __launch_bounds__(NttPlan<LOGN, LOGE>::G, (MINB > 0 ? MINB : ks_min_blocks<LOGN, LOGE>()))
    k_keyswitch(const __grid_constant__ ProdParams M, const uint64_t* __restrict__ C, const uint32_t* __restrict__ evk,
                int ell, uint32_t* __restrict__ resid, int cs, int ls) {
    using PL = NttPlan<LOGN, LOGE>;
    constexpr int E = PL::E;
    constexpr int LAST = PL::NPASS - 1;
    constexpr bool ONE = ks_one_pass<L64, ND>();
    constexpr int REGS = 65536 / (PL::G * (MINB > 0 ? MINB : ks_min_blocks<LOGN, LOGE>()));
    constexpr bool ACC32 = !ONE && (LOGE > 4 || (LOGE == 4 && REGS <= 64));
    extern __shared__ __align__(16) uint32_t smem[];  // exchange buffer, ND operands x SMW
    const int tau = threadIdx.x;
    const int prime = blockIdx.y;
    const int job = blockIdx.x;
    const PrimeParam& Q = M.pr[prime];
    const int k = M.k, l64 = L64 > 0 ? L64 : M.l64;
    const Mod m = load_mod(Q);
    const uint32_t p = m.p, pinv = Q.pinv;
    const uint2* __restrict__ psi = table_of(M.tw.psi, prime);
    const uint2* __restrict__ ipsi = table_of(M.tw.ipsi, prime);
    const uint64_t* cj = C + (size_t)job * PL::N * l64;
    // limb w of coefficient pos at cj[pos * cs + w * ls]: (cs, ls) = (limbs, 1) for
    // [N][limb], (1, N) for limb-major (the HE multiply's intermediate: a warp's
    // loads of one limb are then contiguous). Kernel parameters, so that they stay
    // in the constant bank.

    dep_wait(cj);
    uint64_t T[E];           // sums of products
    uint32_t acc[1][E];      // reduced sums: the inverse transform's input
#pragma unroll
    for (int e = 0; e < E; e++) {
        T[e] = 0;
        acc[0][e] = 0;
    }
    for (int d0 = 0; d0 < (ONE ? 1 : ell); d0 += ND) {
        uint32_t x[ND][E];
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int pos = slot_pos<PL, 0>(tau, e);
            if constexpr (L64 > 0 && ND % 2 == 0) {
                // digits d0 .. d0+ND-1 are limbs d0/2 .. d0/2+ND/2-1 of the coefficient;
                // digits past the last word of q are zero (coefficients are < q)
                const uint64_t* src = cj + (size_t)pos * cs + (size_t)(d0 >> 1) * ls;
                uint32_t w[ND];
                bool both = false;  // two limbs side by side: one 16-byte load
                if constexpr (ND == 4 && L64 % 2 == 0) {
                    if (ls == 1) {
                        const uint4 v = ld_dep(reinterpret_cast<const uint4*>(src));
                        w[0] = v.x;
                        w[1] = v.y;
                        w[ND - 2] = v.z;
                        w[ND - 1] = v.w;
                        both = true;
                    }
                }
                if (!both) {
#pragma unroll
                    for (int o = 0; o < ND; o += 2) {
                        const uint2 v = ld_dep(reinterpret_cast<const uint2*>(src + (o >> 1) * ls));
                        w[o] = v.x;
                        w[o + 1] = v.y;
                    }
                }
#pragma unroll
                for (int o = 0; o < ND; o++) x[o][e] = red_2p(w[o], m);  // digit < 2^32 < 6p -> [0, 4p)
            } else {
#pragma unroll
                for (int o = 0; o < ND; o++) {
                    const int d = d0 + o;
                    uint32_t w = 0;
                    if (d < ell) {
                        const uint64_t limb = ld_dep(cj + (size_t)pos * cs + (size_t)(d >> 1) * ls);
                        w = (uint32_t)(limb >> (32 * (d & 1)));
                    }
                    x[o][e] = red_2p(w, m);  // digit < 2^32 < 6p -> [0, 4p)
                }
            }
        }
        if constexpr (LOGN == 12 && LOGE == 6) {  // one copy of the pass code (see k_mul)
            ntt64_forward<PL, ND>(x, psi, lanes_of<PL>(M.tw.psi_lanes, prime), m, tau, smem, d0 > 0);
        } else {
            ntt_forward<PL, ND>(x, psi, m, tau, smem, d0 > 0, CtaSync(), 1, lanes_of<PL>(M.tw.psi_lanes, prime));
        }
        if constexpr (E == 64) {
            // the key's copy laid out by lane (after the [ell][k][N] table): values u .. u+3
            // of lane tau are the 16-byte record [u/4][tau]
            static_assert(ND == 1, "one digit per pass with 64 coefficients per thread");
            const uint4* g4 = reinterpret_cast<const uint4*>(evk + ((size_t)(ell + d0) * k + prime) * PL::N) + tau;
#pragma unroll
            for (int h = 0; h < E / 4; h++) {
                const uint4 W = __ldg(g4 + h * PL::G);
                const uint32_t v[4] = {W.x, W.y, W.z, W.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {  // one product: (x v 2^-32) in (0, 2p)
                    const uint64_t t = (uint64_t)x[0][4 * h + j] * v[j];
                    const uint32_t r = (uint32_t)(t >> 32) - __umulhi((uint32_t)t * pinv, p) + p;
                    acc[0][4 * h + j] = mac_red(acc[0][4 * h + j], r, m);
                }
            }
        } else {
            if constexpr (ACC32) {
#pragma unroll
                for (int e = 0; e < E; e++) T[e] = 0;
            }
#pragma unroll
            for (int o = 0; o < ND; o++) {
                const int d = d0 + o;
                if (!ONE && !ACC32 && o % 2 == 0) {  // two products fit on top of a high word below 2p
#pragma unroll
                    for (int e = 0; e < E; e++) T[e] = lazy_high(T[e], m);
                }
                if (d < ell) {
                    uint32_t v[E];
                    load_evk<PL::N, E>(evk + ((size_t)d * k + prime) * PL::N, last_pos<PL>(tau), v);
#pragma unroll
                    for (int e = 0; e < E; e++) T[e] += (uint64_t)x[o][e] * v[e];
                }
            }
            if constexpr (ACC32) {
#pragma unroll
                for (int e = 0; e < E; e++) acc[0][e] = mac_red(acc[0][e], mac_finish<(ND > 2)>(T[e], pinv, m), m);
            }
        }
    }
    if constexpr (!ACC32 && E < 64) {
#pragma unroll
        for (int e = 0; e < E; e++) acc[0][e] = mac_finish<!(ONE && ND <= 2)>(T[e], pinv, m);
    }
    if constexpr (LOGN == 12 && LOGE == 6) ntt64_inverse<PL, 1>(acc, ipsi, lanes_of<PL>(M.tw.ipsi_lanes, prime), m, tau, smem, nullptr);
    else ntt_inverse<PL, 1>(acc, ipsi, m, tau, smem, CtaSync(), 1, lanes_of<PL>(M.tw.ipsi_lanes, prime));
    dep_launch();
    uint32_t* out = resid + ((size_t)job * k + prime) * PL::N;
#pragma unroll
    for (int e = 0; e < E; e++) out[slot_pos<PL, 0>(tau, e)] = acc[0][e];
}

// --------------------------------------------------------------------------
// k_mul_key: products of a batch with one polynomial whose transform is kept (a scheme's
// keys: encryption's h, decryption's f and f^2). key: [k][N] transforms times 2^-32
// (key_index). One split, one forward and one inverse transform per product and
// prime instead of two, two and one; a block takes two jobs (shared twiddles and key values;
// with an odd count the last block repeats its job and stores it once).
// 512 products with a kept operand (256 encryptions and their decryptions) at N = 4096, 127-bit
// q: 123 us (k_mul: 152).
// L64 = 0: the other operand is small (encryption's s), a signed 32-bit word per coefficient at
// the start of its job's row, its residues s or s + p; key: transforms times 2^32. 256
// encryptions and their decryptions at N = 4096, 127-bit q: 140 us with s as limbs mod q in the
// product basis (nine primes), 126 with words in the keyswitch basis (six).
// --------------------------------------------------------------------------
template <int LOGN, int LOGE, int L64, int MINB>
__global__ void __launch_bounds__(NttPlan<LOGN, LOGE>::G, MINB)
    k_mul_key(const __grid_constant__ ProdParams M, const uint32_t* __restrict__ key, const uint64_t* __restrict__ Bv,
              long long b_stride, uint32_t* __restrict__ resid, int njobs) {
    using PL = NttPlan<LOGN, LOGE>;
    constexpr int E = PL::E, W = 2 * (L64 ? L64 : 1);
    extern __shared__ __align__(16) uint32_t smem[];  // exchange buffer, 2 operands x SMW
    const int tau = threadIdx.x;
    const int prime = blockIdx.y;
    const int job0 = 2 * blockIdx.x;
    const int job1 = job0 + 1 < njobs ? job0 + 1 : job0;
    const PrimeParam& Q = M.pr[prime];
    const PrimeCtx c = load_prime_ctx(Q);
    const uint64_t* b0 = Bv + (size_t)job0 * b_stride;
    const uint64_t* b1 = Bv + (size_t)job1 * b_stride;
    dep_wait(b0, b1);
    uint32_t x[2][E];
    uint32_t cc[W], qh[W];
#pragma unroll
    for (int j = 0; j < W; j++) {
        cc[j] = Q.crt[j];
        qh[j] = 0;
    }
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int pos = slot_pos<PL, 0>(tau, e);
        if constexpr (L64 == 0) {
            const int s0 = (int)ld_dep_cg(reinterpret_cast<const uint32_t*>(b0) + pos);
            const int s1 = (int)ld_dep_cg(reinterpret_cast<const uint32_t*>(b1) + pos);
            x[0][e] = s0 < 0 ? s0 + c.m.p : s0;
            x[1][e] = s1 < 0 ? s1 + c.m.p : s1;
        } else {
            uint32_t w[W];
            load_words<L64>(b0 + (size_t)pos * L64, w);
            x[0][e] = crt_words<W, false>(w, cc, qh, c);
            load_words<L64>(b1 + (size_t)pos * L64, w);
            x[1][e] = crt_words<W, false>(w, cc, qh, c);
        }
    }
    ntt_forward<PL, 2>(x, table_of(M.tw.psi, prime), c.m, tau, smem, false, CtaSync(), 1, lanes_of<PL>(M.tw.psi_lanes, prime));
    uint32_t v[E];
    load_evk<PL::N, E>(key + (size_t)prime * PL::N, last_pos<PL>(tau), v);
#pragma unroll
    for (int o = 0; o < 2; o++)
#pragma unroll
        for (int e = 0; e < E; e++) x[o][e] = mont(x[o][e], v[e], c.pinv, c.m);  // [0, 4p) times [0, p) -> (0, 2p)
    ntt_inverse<PL, 2>(x, table_of(M.tw.ipsi, prime), c.m, tau, smem, CtaSync(), 1, lanes_of<PL>(M.tw.ipsi_lanes, prime));
    dep_launch();
    uint32_t* out = resid + ((size_t)job0 * M.k + prime) * PL::N;
#pragma unroll
    for (int e = 0; e < E; e++) out[slot_pos<PL, 0>(tau, e)] = x[0][e];
    if (job1 == job0) return;
    out += (size_t)M.k * PL::N;
#pragma unroll
    for (int e = 0; e < E; e++) out[slot_pos<PL, 0>(tau, e)] = x[1][e];
}

// --------------------------------------------------------------------------
// k_ntt: in-place transform of residue vectors [batch][k][N], values in [0, p).
// Forward output in bit-reversed order; inverse includes N^-1. A block runs the
// transforms of two jobs for one prime side by side (shared twiddle loads and
// barriers); with an odd job count the last block repeats its job and stores it
// once.
// --------------------------------------------------------------------------
template <int LOGN, int LOGE, bool INV>
__global__ void __launch_bounds__(NttPlan<LOGN, LOGE>::G, (ntt_min_blocks<LOGN, LOGE>()))
    k_ntt(const __grid_constant__ NttParams M, uint32_t* __restrict__ res, const uint32_t* __restrict__ ninv,
          int njobs) {
    using PL = NttPlan<LOGN, LOGE>;
    constexpr int E = PL::E;
    constexpr int LAST = PL::NPASS - 1;
    extern __shared__ __align__(16) uint32_t smem[];
    const int tau = threadIdx.x;
    const int prime = blockIdx.x;
    const int job0 = 2 * blockIdx.y;
    const bool two = job0 + 1 < njobs;
    const int k = M.k;
    const Mod m = load_mod(M.pr[prime]);
    const uint32_t p = m.p;
    uint32_t* v[2] = {res + ((size_t)job0 * k + prime) * PL::N, res + ((size_t)(two ? job0 + 1 : job0) * k + prime) * PL::N};
    uint32_t x[2][E];
    // after the last pass a thread's E positions are contiguous (16-byte accesses); with
    // whole warps and 16-byte pieces in the buffer they change places inside the warp first, so that
    // a warp's access covers 512 consecutive bytes (2048 x 9 forward transforms of length 4096: 162
    // -> 140 us; 512 x 14 of length 8192: 161 -> 146 forward, 159 -> 151 us inverse)
    constexpr bool VEC = PL::LOGD(LAST) == 0 && PL::R(LAST) == PL::LOGE && E % 4 == 0;
    constexpr bool COAL = VEC && lanes_ok<PL>();
    if (!INV) {
#pragma unroll
        for (int o = 0; o < 2; o++)
#pragma unroll
            for (int e = 0; e < E; e++) x[o][e] = v[o][slot_pos<PL, 0>(tau, e)];
        ntt_forward<PL, 2>(x, table_of(M.tw.psi, prime), m, tau, smem, false, CtaSync(), 1, lanes_of<PL>(M.tw.psi_lanes, prime));
        if constexpr (COAL) rows_to_lanes<PL, 2>(x, smem, tau);
#pragma unroll
        for (int o = 0; o < 2; o++) {
            if (o == 1 && !two) break;
            if constexpr (COAL) {
#pragma unroll
                for (int e = 0; e < E; e += 4)
                    *reinterpret_cast<uint4*>(v[o] + lane_pos<PL>(tau, e)) =
                        make_uint4(red(red_2p(x[o][e], m), p), red(red_2p(x[o][e + 1], m), p),
                                   red(red_2p(x[o][e + 2], m), p), red(red_2p(x[o][e + 3], m), p));
            } else if constexpr (VEC) {
                uint4* d4 = reinterpret_cast<uint4*>(v[o] + group_base<PL, LAST>(tau, 0));
#pragma unroll
                for (int h = 0; h < E / 4; h++)
                    d4[h] = make_uint4(red(red(x[o][4 * h], 2 * p), p), red(red(x[o][4 * h + 1], 2 * p), p),
                                       red(red(x[o][4 * h + 2], 2 * p), p), red(red(x[o][4 * h + 3], 2 * p), p));
            } else {
#pragma unroll
                for (int e = 0; e < E; e++) v[o][slot_pos<PL, LAST>(tau, e)] = red(red(x[o][e], 2 * p), p);
            }
        }
    } else {
        const uint32_t w = ninv[4 * prime], ws = ninv[4 * prime + 1];
#pragma unroll
        for (int o = 0; o < 2; o++) {
            if constexpr (COAL) {
#pragma unroll
                for (int e = 0; e < E; e += 4) {
                    const uint4 q4 = *reinterpret_cast<const uint4*>(v[o] + lane_pos<PL>(tau, e));
                    x[o][e] = q4.x;
                    x[o][e + 1] = q4.y;
                    x[o][e + 2] = q4.z;
                    x[o][e + 3] = q4.w;
                }
            } else if constexpr (VEC) {
                const uint4* s4 = reinterpret_cast<const uint4*>(v[o] + group_base<PL, LAST>(tau, 0));
#pragma unroll
                for (int h = 0; h < E / 4; h++) {
                    const uint4 q4 = s4[h];
                    x[o][4 * h] = q4.x;
                    x[o][4 * h + 1] = q4.y;
                    x[o][4 * h + 2] = q4.z;
                    x[o][4 * h + 3] = q4.w;
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; e++) x[o][e] = v[o][slot_pos<PL, LAST>(tau, e)];
            }
        }
        if constexpr (COAL) lanes_to_rows<PL, 2>(x, smem, tau);
        ntt_inverse<PL, 2>(x, table_of(M.tw.ipsi, prime), m, tau, smem, CtaSync(), 1, lanes_of<PL>(M.tw.ipsi_lanes, prime));
#pragma unroll
        for (int o = 0; o < 2; o++) {
            if (o == 1 && !two) break;
#pragma unroll
            for (int e = 0; e < E; e++) v[o][slot_pos<PL, 0>(tau, e)] = red(shoup(x[o][e], w, ws, p), p);
        }
    }
}

// --------------------------------------------------------------------------
// k_ntt1: the same transform, one residue vector per block, for schedules whose
// threads hold many coefficients (E = 64: 64 threads, two register passes of six
// stages and one exchange, a transpose through shared memory). Grid (jobs,
// primes): consecutive blocks share a prime, so the blocks resident on an SM
// read the same twiddle table (L1 hits).
// MINB > 0: blocks per SM the kernel is compiled for.
// COAL (two passes of six stages): the row side of the transform (forward
// output, inverse input) goes through the exchange region once more, so that
// every global access of a warp covers 128 consecutive bytes instead of 32
// rows 256 bytes apart.
// TPB: transforms per block (TPB groups of G threads, one exchange region each,
// block-wide barriers). Several transforms in step keep the warps of an SM on
// nearby instructions (the unrolled transform is larger than the instruction
// cache). Jobs past the last are computed on the last job and not stored.
// --------------------------------------------------------------------------
// LOOP (N = 4096, E = 64): the two passes run as a loop over one copy of the pass
// code (ntt_core.cuh, ntt64_forward / ntt64_inverse).
template <int LOGN, int LOGE, bool INV, int MINB = 0, bool COAL = false, int TPB = 1, bool LOOP = false>
__global__ void __launch_bounds__(NttPlan<LOGN, LOGE>::G * TPB, (MINB > 0 ? MINB : 1))
    k_ntt1(const __grid_constant__ NttParams M, uint32_t* __restrict__ res, const uint32_t* __restrict__ ninv,
           int njobs) {
    using PL = NttPlan<LOGN, LOGE>;
    constexpr int E = PL::E;
    constexpr int LAST = PL::NPASS - 1;
    static_assert(!COAL || (PL::NPASS == 2 && LOGE == 6 && LOGN == 12), "row-side staging: N = 4096, E = 64");
    extern __shared__ __align__(16) uint32_t smem_all[];
    const int sub = TPB > 1 ? (int)threadIdx.x / PL::G : 0;
    const int tau = TPB > 1 ? (int)threadIdx.x % PL::G : (int)threadIdx.x;
    uint32_t* smem = smem_all + sub * PL::SMW;
    const int job_raw = blockIdx.x * TPB + sub;
    const bool store = job_raw < njobs;
    const int job = store ? job_raw : njobs - 1;
    const int prime = blockIdx.y;
    const int k = M.k;
    const Mod m = load_mod(M.pr[prime]);
    const uint32_t p = m.p;
    uint32_t* v = res + ((size_t)job * k + prime) * PL::N;
    uint32_t x[1][E];
    constexpr bool VEC = PL::LOGD(LAST) == 0 && PL::R(LAST) == PL::LOGE && E % 4 == 0;
    if (!INV) {
#pragma unroll
        for (int e = 0; e < E; e++) x[0][e] = COAL ? __ldcs(v + slot_pos<PL, 0>(tau, e)) : v[slot_pos<PL, 0>(tau, e)];
        if constexpr (LOOP) ntt64_forward<PL, 1>(x, table_of(M.tw.psi, prime), lanes_of<PL>(M.tw.psi_lanes, prime), m, tau, smem);
        else ntt_forward<PL, 1>(x, table_of(M.tw.psi, prime), m, tau, smem, false, CtaSync(), 1, lanes_of<PL>(M.tw.psi_lanes, prime));
        if constexpr (COAL) {
            // row tau (positions 64 tau + u) into the padded buffer (word 65 tau + u: the words
            // this thread read last), then column tau (positions tau + 64 m, word 65 m + tau)
            // to global memory
#pragma unroll
            for (int u = 0; u < E; u++) smem[65 * tau + u] = red(red(x[0][u], 2 * p), p);
            __syncthreads();
            if (store) {
#pragma unroll
                for (int m = 0; m < E; m++) __stcs(v + tau + 64 * m, smem[tau + 65 * m]);
            }
        } else if constexpr (VEC) {
            if (store) {
                uint4* d4 = reinterpret_cast<uint4*>(v + group_base<PL, LAST>(tau, 0));
#pragma unroll
                for (int h = 0; h < E / 4; h++)
                    d4[h] = make_uint4(red(red(x[0][4 * h], 2 * p), p), red(red(x[0][4 * h + 1], 2 * p), p),
                                       red(red(x[0][4 * h + 2], 2 * p), p), red(red(x[0][4 * h + 3], 2 * p), p));
            }
        } else if (store) {
#pragma unroll
            for (int e = 0; e < E; e++) v[slot_pos<PL, LAST>(tau, e)] = red(red(x[0][e], 2 * p), p);
        }
    } else {
        if constexpr (COAL) {
            // columns in (coalesced), rows out of the padded buffer; the inverse's exchange then
            // writes back the words each thread read
#pragma unroll
            for (int m = 0; m < E; m++) smem[tau + 65 * m] = __ldcs(v + tau + 64 * m);
            __syncthreads();
#pragma unroll
            for (int u = 0; u < E; u++) x[0][u] = smem[65 * tau + u];
        } else if constexpr (VEC) {
            const uint4* s4 = reinterpret_cast<const uint4*>(v + group_base<PL, LAST>(tau, 0));
#pragma unroll
            for (int h = 0; h < E / 4; h++) {
                const uint4 q4 = s4[h];
                x[0][4 * h] = q4.x;
                x[0][4 * h + 1] = q4.y;
                x[0][4 * h + 2] = q4.z;
                x[0][4 * h + 3] = q4.w;
            }
        } else {
#pragma unroll
            for (int e = 0; e < E; e++) x[0][e] = v[slot_pos<PL, LAST>(tau, e)];
        }
        // N^-1 is applied inside the last stage (outputs in [0, p))
        if constexpr (LOOP)
            ntt64_inverse<PL, 1>(x, table_of(M.tw.ipsi, prime), lanes_of<PL>(M.tw.ipsi_lanes, prime), m, tau, smem, ninv + 4 * prime);
        else
            ntt_inverse<PL, 1>(x, table_of(M.tw.ipsi, prime), m, tau, smem, CtaSync(), 1, lanes_of<PL>(M.tw.ipsi_lanes, prime),
                               ninv + 4 * prime);
        if (store) {
#pragma unroll
            for (int e = 0; e < E; e++) {
                if constexpr (COAL) __stcs(v + slot_pos<PL, 0>(tau, e), x[0][e]);
                else v[slot_pos<PL, 0>(tau, e)] = x[0][e];
            }
        }
    }
}

// --------------------------------------------------------------------------
// k_epi: ICRT + mod q / round(t/q) / decrypt. One thread per coefficient.
// L = 32-bit words of q.
// --------------------------------------------------------------------------
template <int L>
struct Cols {
    uint64_t c[L + 2];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int w = 0; w < L + 2; w++) c[w] = 0;
    }
    __device__ __forceinline__ void mac(uint32_t y, const uint32_t* a) {
#pragma unroll
        for (int w = 0; w < L; w++) c[w] += (uint64_t)y * a[w];
    }
    __device__ __forceinline__ void add(const uint32_t* a) {
#pragma unroll
        for (int w = 0; w < L; w++) c[w] += a[w];
    }
    // carry-propagate so that c[w] < 2^32 for w <= L
    __device__ __forceinline__ void norm() {
#pragma unroll
        for (int w = 0; w < L + 1; w++) {
            c[w + 1] += c[w] >> 32;
            c[w] &= 0xFFFFFFFFULL;
        }
    }
};

// Barrett division of a normalised column value x (< 2^(32L+37)) by q' (top bit
// of word L-1 set): returns the quotient, writes the remainder (< q') to r.
template <int L>
__device__ __forceinline__ uint64_t barrett(const Cols<L>& x, const uint32_t* qn, uint64_t mu, uint32_t (&r)[L]) {
    const uint64_t x1 = (x.c[L + 1] << 33) | (x.c[L] << 1) | (x.c[L - 1] >> 31);  // floor(x / 2^(32L-1)) < 2^38
    const uint64_t hi = __umul64hi(x1, mu), lo = x1 * mu;
    uint64_t Q = (hi << 26) | (lo >> 38);  // Q-2 <= Q <= Q_true
    const uint32_t Ql = (uint32_t)Q, Qh = (uint32_t)(Q >> 32);
    uint32_t P[L + 2];
    uint64_t carry = 0;
#pragma unroll
    for (int w = 0; w < L; w++) {
        const uint64_t t = (uint64_t)Ql * qn[w] + carry;
        P[w] = (uint32_t)t;
        carry = t >> 32;
    }
    P[L] = (uint32_t)carry;
    carry = 0;
#pragma unroll
    for (int w = 0; w < L; w++) {
        const uint64_t t = (uint64_t)Qh * qn[w] + P[w + 1] + carry;
        P[w + 1] = (uint32_t)t;
        carry = t >> 32;
    }
    P[L + 1] = (uint32_t)carry;
    uint32_t rr[L + 1];
    int64_t br = 0;
#pragma unroll
    for (int w = 0; w <= L; w++) {
        const int64_t d = (int64_t)x.c[w] - (int64_t)P[w] - br;
        rr[w] = (uint32_t)d;
        br = d < 0;
    }
#pragma unroll
    for (int it = 0; it < 2; it++) {
        uint32_t t[L + 1];
        int64_t b2 = 0;
#pragma unroll
        for (int w = 0; w < L; w++) {
            const int64_t d = (int64_t)rr[w] - (int64_t)qn[w] - b2;
            t[w] = (uint32_t)d;
            b2 = d < 0;
        }
        const int64_t d = (int64_t)rr[L] - b2;
        t[L] = (uint32_t)d;
        b2 = d < 0;
        if (!b2) {
#pragma unroll
            for (int w = 0; w <= L; w++) rr[w] = t[w];
            Q++;
        }
    }
#pragma unroll
    for (int w = 0; w < L; w++) r[w] = rr[w];
    return Q;
}

// Epilogue constants in shared memory. The per-prime rows are padded to a
// multiple of three primes with zero factors (ycon = 0, zero rows), so that a
// padded prime contributes exactly nothing and the prime loop runs whole
// groups of three without guards.
constexpr int KPAD = KMAX + 2;

// Scalars of one prime, read with two 16-byte shared loads.
struct __align__(16) EpiPrime {
    uint32_t p, ycon, ycon_sh, fhi, flo;
    uint32_t F0, F1;  // YASHE: R_i / q in units of 2^-64 (lo, hi)
    uint32_t pad;
};
struct EpiShared {
    EpiPrime pr[KPAD];
    __align__(16) uint32_t A0[KPAD * L32MAX];
    __align__(16) uint32_t A1[KPAD * L32MAX];
    uint32_t B0[L32MAX], B1[L32MAX], qn[L32MAX], qhalf_n[L32MAX];
    uint32_t FM[2];  // YASHE: (q - R_M) / q in units of 2^-64
};

// Copy the epilogue constants of basis B into shared memory (threads tid, tid +
// nthreads, ... of the caller's group), with the zero padding up to 3*ceil(k/3).
template <int L, int MODE>
__device__ __forceinline__ void epi_stage(EpiShared& S, const BasisDev* __restrict__ B, int tid, int nthreads) {
    const int k = B->k, kp = 3 * ((k + 2) / 3);
    for (int i = tid; i < kp; i += nthreads) {
        EpiPrime e{1u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
        if (i < k) {
            e.p = B->p[i];
            e.ycon = B->ycon[i];
            e.ycon_sh = B->ycon_sh[i];
            e.fhi = B->fhi[i];
            e.flo = B->flo[i];
            if (MODE == EPI_YASHE) {
                e.F0 = B->frac[i][0];
                e.F1 = B->frac[i][1];
            }
        }
        S.pr[i] = e;
    }
    for (int i = tid; i < kp * L; i += nthreads) {
        const bool in = i < k * L;
        S.A0[i] = in ? B->A0[i / L][i % L] : 0u;
        if (MODE == EPI_YASHE) S.A1[i] = in ? B->A1[i / L][i % L] : 0u;
    }
    if (MODE == EPI_YASHE && tid < 2) S.FM[tid] = B->frac_m[tid];
    for (int i = tid; i < L; i += nthreads) {
        S.B0[i] = B->B0[i];
        S.B1[i] = B->B1[i];
        S.qn[i] = B->qn[i];
        S.qhalf_n[i] = B->qhalf_n[i];
    }
}

// Row of L words of shared memory (16- or 8-byte loads when L allows).
template <int L>
__device__ __forceinline__ void load_row(const uint32_t* src, uint32_t (&a)[L]) {
    if constexpr (L % 4 == 0) {
#pragma unroll
        for (int w = 0; w < L; w += 4) {
            const uint4 v = *reinterpret_cast<const uint4*>(src + w);
            a[w] = v.x;
            a[w + 1] = v.y;
            a[w + 2] = v.z;
            a[w + 3] = v.w;
        }
    } else if constexpr (L % 2 == 0) {
#pragma unroll
        for (int w = 0; w < L; w += 2) {
            const uint2 v = *reinterpret_cast<const uint2*>(src + w);
            a[w] = v.x;
            a[w + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int w = 0; w < L; w++) a[w] = src[w];
    }
}

// YASHE rounding, exact: Q = floor((S' + (q-1)/2) / q) with S' = sum y_i R_i +
// v (q - R_M), from the residues again (the rare case that the fixed-point
// estimate cannot decide).
template <int L>
__device__ __noinline__ uint64_t yashe_round_exact(const EpiShared& S, const BasisDev* __restrict__ B,
                                                   const uint32_t* __restrict__ r0, size_t stride, uint32_t v) {
    const int k = B->k;
    Cols<L> c1;
    c1.zero();
    for (int i = 0; i < k; i++) {
        const EpiPrime P = S.pr[i];
        const uint32_t y = red(shoup(__ldcg(r0 + (size_t)i * stride), P.ycon, P.ycon_sh, P.p), P.p);
        c1.mac(y, &S.A1[i * L]);
        if (i % 3 == 2) c1.norm();
    }
    c1.norm();
    c1.mac(v, S.B1);
    c1.add(S.qhalf_n);
    c1.norm();
    uint32_t rdummy[L];
    return barrett<L>(c1, S.qn, B->mu, rdummy);
}

// Epilogue of C coefficients: r0[c] points at the residue of coefficient c for
// prime 0, residues of the next primes follow `stride` words apart. Writes the
// limbs of dst[c] (MODQ, YASHE) or one word (DECRYPT) where store[c] is set.
// The constants of a prime are read once for all C coefficients.
//
// YASHE rounding: Q = round(S'/q) is first estimated in 64-bit fixed point,
// Z = sum y_i F_i + v F_M + 2^63 (F = floor(R 2^64 / q)), which undershoots the
// true value by less than (k+1) 2^30 2^-64 < 2^-28. floor(Z / 2^64) is exact
// unless the fraction of Z is within 2^-28 of the next integer; those
// coefficients (about one in 2^28), and all of them when frac_limit is 0, take
// the exact multiword path.
// lstride: distance in words between the limbs of an output coefficient (1, or
// N for the limb-major layout)
template <int L, int MODE, int C>
__device__ __forceinline__ void epi_coefs(const EpiShared& S, const BasisDev* __restrict__ B,
                                          const uint32_t* const (&r0)[C], size_t stride, uint64_t* const (&dst)[C],
                                          const bool (&store)[C], uint64_t frac_limit, size_t lstride = 1) {
    const int k = B->k, shift = B->shift, l64 = B->l64;
    const int groups = (k + 2) / 3;
    const uint64_t mu = B->mu;
    Cols<L> c0[C];
    Cols<2> fz[C];  // YASHE: Z in 32-bit columns
    uint64_t vacc[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
        c0[c].zero();
        fz[c].zero();
        vacc[c] = 0;
    }
    // One prime's contribution to every coefficient: y = [X Mhat_i^-1]_{p_i}, the
    // fixed-point estimate of y/p_i for v, y times the row of constants into the
    // columns and (YASHE) y F_i into Z.
    auto absorb = [&](int i, const uint32_t (&r)[C]) {
        const EpiPrime P = S.pr[i];
        uint32_t a[L];
        load_row<L>(&S.A0[i * L], a);
        const uint32_t F[2] = {P.F0, P.F1};
#pragma unroll
        for (int c = 0; c < C; c++) {
            const uint32_t y = red(shoup(r[c], P.ycon, P.ycon_sh, P.p), P.p);
            vacc[c] += (uint64_t)y * P.fhi + __umulhi(y, P.flo);  // sum y_i/p_i in 2^-32 units
            c0[c].mac(y, a);
            if (MODE == EPI_YASHE) fz[c].mac(y, F);
        }
    };
    // Residues come from L2: the loads of the next two groups of three primes are
    // in flight while a group is absorbed. Loads past the last prime re-read its
    // residue (a valid address); its padded factors make the contribution zero.
    auto load3 = [&](int g, uint32_t (&d)[3][C]) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const size_t off = (size_t)min(3 * g + j, k - 1) * stride;
#pragma unroll
            for (int c = 0; c < C; c++) d[j][c] = __ldcg(r0[c] + off);
        }
    };
    uint32_t g0[3][C], g1[3][C], g2[3][C];
    load3(0, g0);
    load3(min(1, groups - 1), g1);
    for (int g = 0; g < groups; g++) {
        load3(min(g + 2, groups - 1), g2);
#pragma unroll
        for (int j = 0; j < 3; j++) absorb(3 * g + j, g0[j]);
#pragma unroll
        for (int c = 0; c < C; c++) {
            c0[c].norm();  // columns take three products of < 2^62 between carry passes
            if (MODE == EPI_YASHE) fz[c].norm();
        }
#pragma unroll
        for (int j = 0; j < 3; j++)
#pragma unroll
            for (int c = 0; c < C; c++) {
                g0[j][c] = g1[j][c];
                g1[j][c] = g2[j][c];
            }
    }
#pragma unroll
    for (int c = 0; c < C; c++) {
        const uint32_t v = (uint32_t)((vacc[c] + 0x80000000ULL) >> 32);  // X = sum y_i Mhat_i - v M
        Cols<L>& x = c0[c];
        x.norm();
        x.mac(v, S.B0);
        if (MODE == EPI_YASHE) {
            Cols<2>& z = fz[c];
            z.mac(v, S.FM);
            z.c[1] += 0x80000000u;  // + 1/2
            z.norm();
            const uint64_t frac = z.c[0] | (z.c[1] << 32);
            uint64_t Q2 = z.c[2] | (z.c[3] << 32);  // round(S/q) + v, S = sum y_i R_i - v R_M
            if (frac >= frac_limit) Q2 = yashe_round_exact<L>(S, B, r0[c], stride, v);
            // x += Q2 << shift
            const uint64_t lo = Q2 << shift;
            const uint64_t hi = shift ? (Q2 >> (64 - shift)) : 0;
            x.c[0] += (uint32_t)lo;
            x.c[1] += (uint32_t)(lo >> 32);
            x.c[2] += hi;
        }
        x.norm();
        uint32_t r[L];
        barrett<L>(x, S.qn, mu, r);  // r = (result mod q) << shift
        if (!store[c]) continue;
        if constexpr (MODE == EPI_DECRYPT) {
            Cols<L> c2;
            c2.zero();
            c2.mac(B->t, r);
            c2.add(S.qhalf_n);
            c2.norm();
            uint32_t rd[L];
            uint64_t Q = barrett<L>(c2, S.qn, mu, rd);  // round(t x / q) in [0, t]
            if (Q >= B->t) Q -= B->t;
            dst[c][0] = Q;
        } else {
            uint32_t o[L];
#pragma unroll
            for (int w = 0; w < L; w++) {
                const uint32_t nx = (w + 1 < L) ? r[w + 1] : 0u;
                o[w] = __funnelshift_r(r[w], nx, shift);
            }
#pragma unroll
            for (int j = 0; j < (L + 1) / 2; j++) {
                const uint64_t lo32 = o[2 * j];
                const uint64_t hi32 = (2 * j + 1 < L) ? o[2 * j + 1] : 0u;
                if (j < l64) dst[c][j * lstride] = lo32 | (hi32 << 32);
            }
        }
    }
}

// lm: outputs limb-major ([job][limb][N]) instead of [job][N][limb] (modes
// MODQ and YASHE; the HE multiply's intermediate before its keyswitch)
template <int L, int MODE>
__global__ void __launch_bounds__(256) k_epi(const BasisDev* __restrict__ B, const uint32_t* __restrict__ resid,
                                             void* __restrict__ out, int njobs, unsigned long long frac_limit,
                                             int lm) {
    constexpr int C = epi_coefs_per_thread(L);  // coefficients per thread
    __shared__ EpiShared S;
    epi_stage<L, MODE>(S, B, threadIdx.x, blockDim.x);
    __syncthreads();
    const int logn = B->logn, k = B->k, l64 = B->l64;
    const int n = 1 << logn;
    const long long total = (long long)njobs << logn;
    const long long base = (long long)blockIdx.x * blockDim.x * C + threadIdx.x;
    if (base >= total) return;
    const uint32_t* r0[C];
    uint64_t* dst[C];
    bool store[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
        long long idx = base + (long long)c * blockDim.x;  // coalesced across the warp for every c
        store[c] = idx < total;
        if (!store[c]) idx = base;  // computed and not written
        const long long job = idx >> logn;
        const int coef = (int)(idx & (n - 1));
        r0[c] = resid + (size_t)job * k * n + coef;
        dst[c] = reinterpret_cast<uint64_t*>(out) +
                 (MODE == EPI_DECRYPT ? (size_t)job * n + coef
                                      : (size_t)job * n * l64 + (lm ? (size_t)coef : (size_t)coef * l64));
    }
    epi_coefs<L, MODE, C>(S, B, r0, (size_t)n, dst, store, frac_limit, lm ? (size_t)n : 1);
}

// --------------------------------------------------------------------------
// k_epi_c: the epilogue with its constants in the constant bank. The constants of a
// basis travel by value as a kernel parameter, so each is a uniform operand of the
// instruction that uses it: no shared-memory staging, no barrier, no address
// arithmetic per thread. K > 0: the prime count at compile time (straight-line code);
// K = 0: any count, in groups of four (a carry pass each: four products of a residue
// and a word plus a normalised word stay below 2^64) with the next group's residues in
// flight, and a rest of up to three.
//
// The kernel is bound by the fma-heavy pipe (a wide or high product takes four of its
// cycles, a low one two), so what a prime costs there was cut: v = round(sum y_i / p_i)
// is summed in 26-bit fixed point from 13-bit factors (one shift and one low product
// instead of a wide and a high one): each term is low by at most 2^-13 + 2^-13, the sum
// of 40 by less than 0.01, and |X| < M/4 leaves 0.25. ANYX (cy_icrt: residues of any X in
// (-M/2, M/2)): k_epi's 64-bit sum. Barrett's quotient is formed from 32-bit pieces
// of 45-bit operands and is at most one low, so one conditional subtraction ends it.
// --------------------------------------------------------------------------
template <int L>
struct __align__(16) EpiPrimeC {
    uint32_t fhi, np, ycon, ycon_sh;  // floor(2^64 / p) in words fhi, flo (ANYX)
    uint32_t g, F0, F1, flo;          // floor(2^43 / p); R_i / q in units of 2^-64 (YASHE)
    uint32_t A0[L];
};
template <int L, int KS>
struct EpiConst {
    EpiPrimeC<L> pr[KS];
    uint32_t B0[L], qn[L], qhalf_n[L];
    uint32_t FM[2];
    uint32_t mu_lo, mu_hi;  // floor(2^(32 L + 44) / q')
    uint32_t t;
    int shift, logn, k;
};

// The exact YASHE rounding of yashe_round_exact with the constants read from
// the basis in global memory (the rare path of k_epi_c).
template <int L>
__device__ __noinline__ uint64_t yashe_round_exact_g(const BasisDev* __restrict__ B, const uint32_t* __restrict__ r0,
                                                     size_t stride, uint32_t v) {
    const int k = B->k;
    Cols<L> c1;
    c1.zero();
    for (int i = 0; i < k; i++) {
        const uint32_t p = B->p[i];
        const uint32_t y = red(shoup(ld_dep_cg(r0 + (size_t)i * stride), B->ycon[i], B->ycon_sh[i], p), p);
        c1.mac(y, B->A1[i]);
        if (i % 3 == 2) c1.norm();
    }
    c1.norm();
    c1.mac(v, B->B1);
    c1.add(B->qhalf_n);
    c1.norm();
    uint32_t rdummy[L];
    return barrett<L>(c1, B->qn, B->mu, rdummy);
}

// Carry chains over 32-bit words (consecutive volatile statements: the compiler emits
// no other instruction that touches the carry flag in between).
__device__ __forceinline__ uint32_t sub_cc(uint32_t a, uint32_t b) {
    uint32_t r;
    asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t subc_cc(uint32_t a, uint32_t b) {
    uint32_t r;
    asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t sub_borrow() {  // all ones if the chain borrowed
    uint32_t r;
    asm volatile("subc.u32 %0, 0, 0;" : "=r"(r));
    return r;
}

// x (normalised columns, below 2^(32 L + 37)) modulo q' (top bit of word L-1 set):
// returns the quotient, writes the remainder to r. With x1 = floor(x / 2^(32 L - 8))
// and mu = floor(2^(32 L + 44) / q') below 2^46, Q = floor(x1 mu / 2^52) is the
// quotient or one less (the two roundings cost less than 2^-6 together).
template <int L>
__device__ __forceinline__ uint64_t barrett_c(const Cols<L>& x, const uint32_t (&qn)[L], uint32_t mu_lo,
                                              uint32_t mu_hi, uint32_t (&r)[L]) {
    const uint32_t t1 = (uint32_t)x.c[L], t0 = (uint32_t)x.c[L - 1];
    const uint32_t xl = __funnelshift_l(t0, t1, 8);
    const uint32_t xh = __funnelshift_l(t1, (uint32_t)x.c[L + 1], 8);
    const uint64_t S = (uint64_t)xh * mu_lo + (uint64_t)xl * mu_hi + __umulhi(xl, mu_lo);
    uint64_t Q = (S >> 20) + ((uint64_t)(xh * mu_hi) << 12);
    const uint32_t Ql = (uint32_t)Q, Qh = (uint32_t)(Q >> 32);
    uint32_t P[L + 1];
    uint64_t carry = 0;
#pragma unroll
    for (int w = 0; w < L; w++) {
        const uint64_t lo = (uint64_t)Ql * qn[w] + (uint32_t)carry;
        P[w] = (uint32_t)lo;
        carry = (uint64_t)Qh * qn[w] + ((lo >> 32) + (carry >> 32));
    }
    P[L] = (uint32_t)carry;
    uint32_t rr[L + 1], t[L + 1];
    rr[0] = sub_cc((uint32_t)x.c[0], P[0]);
#pragma unroll
    for (int w = 1; w <= L; w++) rr[w] = subc_cc((uint32_t)x.c[w], P[w]);
    t[0] = sub_cc(rr[0], qn[0]);
#pragma unroll
    for (int w = 1; w < L; w++) t[w] = subc_cc(rr[w], qn[w]);
    t[L] = subc_cc(rr[L], 0u);
    const bool keep = sub_borrow() != 0;
#pragma unroll
    for (int w = 0; w < L; w++) r[w] = keep ? rr[w] : t[w];
    return keep ? Q : Q + 1;
}

// x in [0, 2m) -> [0, m) with nm = -m
__device__ __forceinline__ uint32_t red_neg(uint32_t x, uint32_t nm) { return __viaddmin_u32(x, nm, x); }

// One coefficient: residues r0[i n] of primes i < k, result to out (word j at out[j
// lstride], or one word for DECRYPT). P: the basis's constants (a kernel parameter, or a
// copy in shared memory).
// DEP: called by k_epi_c (dependent launches).
template <int L, int MODE, int K, bool DEP, bool ANYX = false, class Const>
__device__ __forceinline__ void epi_c_one(const Const& P, const BasisDev* __restrict__ B,
                                          const uint32_t* __restrict__ r0, int n, uint64_t* __restrict__ out,
                                          size_t lstride, unsigned long long frac_limit) {
    constexpr int L64 = (L + 1) / 2;
    const int shift = P.shift;
    const int k = K ? K : P.k;

    Cols<L> x;   // sum y_i A0_i
    Cols<2> z;   // YASHE: Z = sum y_i F_i in 32-bit columns
    std::conditional_t<ANYX, uint64_t, uint32_t> vs = ANYX ? 0x80000000u : 0x2000000u;  // sum y_i / p_i + 1/2 in units of 2^-32 or 2^-26
    x.zero();
    z.zero();
    auto absorb = [&](const EpiPrimeC<L>& E, uint32_t res) {
        const uint32_t y = red_neg(__umulhi(res, E.ycon_sh) * E.np + res * E.ycon, E.np);
        if constexpr (ANYX) vs += (uint64_t)y * E.fhi + __umulhi(y, E.flo);
        else vs += (y >> 17) * E.g;
#pragma unroll
        for (int w = 0; w < L; w++) x.c[w] += (uint64_t)y * E.A0[w];
        if (MODE == EPI_YASHE) {
            z.c[0] += (uint64_t)y * E.F0;
            z.c[1] += (uint64_t)y * E.F1;
        }
    };
    if constexpr (K > 0) {
        uint32_t r[K];
#pragma unroll
        for (int i = 0; i < K; i++) r[i] = ld_dep_cg(r0 + (size_t)i * n);
#pragma unroll
        for (int i = 0; i < K; i++) {
            absorb(P.pr[i], r[i]);
            if (i % 4 == 3 && i + 1 < K) {
                x.norm();
                if (MODE == EPI_YASHE) z.norm();
            }
        }
    } else {
        const int rest = k & 3, whole = k - rest;
        uint32_t cur[4], nxt[4];
        auto load = [&](int i, uint32_t(&d)[4]) {  // past the last prime: its residue again, not used
#pragma unroll
            for (int j = 0; j < 4; j++) d[j] = ld_dep_cg(r0 + (size_t)min(i + j, k - 1) * n);
        };
        load(0, cur);
#pragma unroll 1
        for (int i = 0; i < whole; i += 4) {
            load(i + 4, nxt);
#pragma unroll
            for (int j = 0; j < 4; j++) absorb(P.pr[i + j], cur[j]);
            x.norm();
            if (MODE == EPI_YASHE) z.norm();
#pragma unroll
            for (int j = 0; j < 4; j++) cur[j] = nxt[j];
        }
#pragma unroll
        for (int j = 0; j < 3; j++)
            if (j < rest) absorb(P.pr[whole + j], cur[j]);
    }
    // every table prime is at least 2^18 below 2^30: four products leave 2^50 for what follows
    const uint32_t v = (uint32_t)(vs >> (ANYX ? 32 : 26));  // X = sum y_i Mhat_i - v M
#pragma unroll
    for (int w = 0; w < L; w++) x.c[w] += (uint64_t)v * P.B0[w];
    if (MODE == EPI_YASHE) {
        z.c[0] += (uint64_t)v * P.FM[0];
        z.c[1] += (uint64_t)v * P.FM[1] + 0x80000000u;  // + 1/2
        z.norm();
        const uint64_t frac = z.c[0] | (z.c[1] << 32);
        uint64_t Q2 = z.c[2] | (z.c[3] << 32);  // round(S/q) + v, S = sum y_i R_i - v R_M
        if (frac >= frac_limit) Q2 = yashe_round_exact_g<L>(B, r0, (size_t)n, v);
        // x += Q2 << shift
        const uint64_t lo = Q2 << shift;
        const uint64_t hi = shift ? (Q2 >> (64 - shift)) : 0;
        x.c[0] += (uint32_t)lo;
        x.c[1] += (uint32_t)(lo >> 32);
        x.c[2] += hi;
    }
    x.norm();
    uint32_t qn[L], rm[L];
#pragma unroll
    for (int w = 0; w < L; w++) qn[w] = P.qn[w];
    barrett_c<L>(x, qn, P.mu_lo, P.mu_hi, rm);  // rm = (result mod q) << shift
    if (DEP) dep_launch();
    if constexpr (MODE == EPI_DECRYPT) {
        Cols<L> c2;
#pragma unroll
        for (int w = 0; w < L; w++) c2.c[w] = (uint64_t)P.t * rm[w] + P.qhalf_n[w];
        c2.c[L] = c2.c[L + 1] = 0;
        c2.norm();
        uint32_t rd[L];
        uint64_t Q = barrett_c<L>(c2, qn, P.mu_lo, P.mu_hi, rd);  // round(t x / q) in [0, t]
        if (Q >= P.t) Q -= P.t;
        out[0] = Q;
    } else {
        uint64_t o[L64];
#pragma unroll
        for (int j = 0; j < L64; j++) {
            auto word = [&](int w) { return w < L ? __funnelshift_r(rm[w], w + 1 < L ? rm[w + 1] : 0u, shift) : 0u; };
            o[j] = (uint64_t)word(2 * j + 1) << 32 | word(2 * j);
        }
        if constexpr (L64 % 2 == 0) {
            if (lstride == 1) {
                ulonglong2* d2 = reinterpret_cast<ulonglong2*>(out);
#pragma unroll
                for (int j = 0; j < L64 / 2; j++) d2[j] = make_ulonglong2(o[2 * j], o[2 * j + 1]);
                return;
            }
        }
#pragma unroll
        for (int j = 0; j < L64; j++) out[j * lstride] = o[j];
    }
}

template <int L, int MODE, int K, bool ANYX = false>
__global__ void __launch_bounds__(256) k_epi_c(const __grid_constant__ EpiConst<L, (K ? K : KMAX)> P,
                                               const BasisDev* __restrict__ B, const uint32_t* __restrict__ resid,
                                               void* __restrict__ out, int njobs, unsigned long long frac_limit,
                                               int lm) {
    constexpr int L64 = (L + 1) / 2;
    const int logn = P.logn;
    const int n = 1 << logn;
    const int k = K ? K : P.k;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)njobs << logn) return;
    const long long job = idx >> logn;
    const int coef = (int)(idx & (n - 1));
    const uint32_t* r0 = resid + (size_t)job * k * n + coef;
    dep_wait(r0);
    uint64_t* dst = reinterpret_cast<uint64_t*>(out) +
                    (MODE == EPI_DECRYPT ? (size_t)idx : (size_t)job * n * L64 + (lm ? (size_t)coef : (size_t)coef * L64));
    epi_c_one<L, MODE, K, true, ANYX>(P, B, r0, n, dst, lm ? (size_t)n : 1, frac_limit);
}

// Constants of a basis for k_epi_c (K = 0 or KS = K primes).
template <int L, int KS>
void fill_epi_const(const BasisDev& h, void* param) {
    static_assert(sizeof(EpiConst<L, KS>) <= 4096, "fits a kernel parameter");
    EpiConst<L, KS>& c = *static_cast<EpiConst<L, KS>*>(param);
    for (int i = 0; i < h.k; i++) {
        EpiPrimeC<L>& e = c.pr[i];
        e.fhi = h.fhi[i];
        e.flo = h.flo[i];
        e.np = 0u - h.p[i];
        e.ycon = h.ycon[i];
        e.ycon_sh = h.ycon_sh[i];
        e.g = (uint32_t)((1ull << 43) / h.p[i]);
        e.F0 = h.frac[i][0];
        e.F1 = h.frac[i][1];
        for (int w = 0; w < L; w++) e.A0[w] = h.A0[i][w];
    }
    for (int w = 0; w < L; w++) {
        c.B0[w] = h.B0[w];
        c.qn[w] = h.qn[w];
        c.qhalf_n[w] = h.qhalf_n[w];
    }
    c.FM[0] = h.frac_m[0];
    c.FM[1] = h.frac_m[1];
    c.mu_lo = (uint32_t)h.mu45;
    c.mu_hi = (uint32_t)(h.mu45 >> 32);
    c.t = h.t;
    c.shift = h.shift;
    c.logn = h.logn;
    c.k = h.k;
}

}  // namespace cy

namespace cy {

// The kernels of k_mul_key for N = 2^LOGN by limb count (0: the small operand), 16 coefficients per
// thread, compiled for MINB blocks per SM.
template <int LOGN, int MINB, int L64>
KeyKernel key_entry() {
    return {(void*)k_mul_key<LOGN, 4, L64, MINB>, NttPlan<LOGN, 4>::G, region_bytes<NttPlan<LOGN, 4>, 2>()};
}
template <int LOGN, int MINB>
const KeyKernel* key_row(int l64) {
    static const KeyKernel row[7] = {key_entry<LOGN, MINB, 0>(), key_entry<LOGN, MINB, 1>(), key_entry<LOGN, MINB, 2>(),
                                     key_entry<LOGN, MINB, 3>(), key_entry<LOGN, MINB, 4>(), key_entry<LOGN, MINB, 5>(),
                                     key_entry<LOGN, MINB, 6>()};
    return &row[l64];
}

template <int LOGN, int LOGE, int L64, int MB_MUL, int MB_KS, int ND_LO, int ND_HI>
void fill_l64(KernelSet& ks) {
    ks.mul[L64][0] = (void*)k_mul<LOGN, LOGE, L64, false, MB_MUL>;
    ks.mul[L64][1] = (void*)k_mul<LOGN, LOGE, L64, true, MB_MUL>;
    ks.ks[L64][0] = (void*)k_keyswitch<LOGN, LOGE, L64, ND_LO, MB_KS>;
    // odd limb counts have 1 or 2 digits more than a multiple of four, so none takes ND_HI at a time
    if constexpr (L64 % 2 == 0) ks.ks[L64][1] = (void*)k_keyswitch<LOGN, LOGE, L64, ND_HI, MB_KS>;
}

// SPECIALISE: instantiate the kernels for each limb count of SPEC_MASK (all six by default:
// 512 products of four limbs at N = 4096 376 us against 531 with the generic
// kernels); limb counts left out use the generic kernels.
// MB_MUL / MB_KS > 0: blocks per SM the product / keyswitch kernels are
// compiled for (0: the defaults above).
// ND_LO: digits per pass of the keyswitch kernel used when four do not fit (2, or 1
// for fewer registers); ND_HI: digits per pass of the one used when the digit
// count is a multiple of four and it fits (4, or 2 for fewer registers).
// SPEC_MASK: the limb counts (bit L64) that get specialised kernels when
// SPECIALISE is set.
template <int LOGN, int LOGE, bool SPECIALISE, int MB_MUL = 0, int MB_KS = 0, int ND_LO = 2, int ND_HI = 4,
          unsigned SPEC_MASK = 0x7Eu>
void fill_kernel_set(KernelSet& ks) {
    using PL = NttPlan<LOGN, LOGE>;
    ks.logn = LOGN;
    ks.loge = LOGE;
    ks.threads = PL::G;
    ks.mul_id = LOGE * 100 + (MB_MUL > 0 ? MB_MUL : mul_min_blocks<LOGN, LOGE>());
    ks.ks_id = (LOGE * 100 + (MB_KS > 0 ? MB_KS : ks_min_blocks<LOGN, LOGE>())) * 100 + ND_LO * 10 + ND_HI;
    ks.ntt_id = LOGE;
    if constexpr (!SPECIALISE || SPEC_MASK != 0x7Eu) fill_l64<LOGN, LOGE, 0, MB_MUL, MB_KS, ND_LO, ND_HI>(ks);
    if constexpr (SPECIALISE && (SPEC_MASK & 2u)) fill_l64<LOGN, LOGE, 1, MB_MUL, MB_KS, ND_LO, ND_HI>(ks);
    if constexpr (SPECIALISE && (SPEC_MASK & 4u)) fill_l64<LOGN, LOGE, 2, MB_MUL, MB_KS, ND_LO, ND_HI>(ks);
    if constexpr (SPECIALISE && (SPEC_MASK & 8u)) fill_l64<LOGN, LOGE, 3, MB_MUL, MB_KS, ND_LO, ND_HI>(ks);
    if constexpr (SPECIALISE && (SPEC_MASK & 16u)) fill_l64<LOGN, LOGE, 4, MB_MUL, MB_KS, ND_LO, ND_HI>(ks);
    if constexpr (SPECIALISE && (SPEC_MASK & 32u)) fill_l64<LOGN, LOGE, 5, MB_MUL, MB_KS, ND_LO, ND_HI>(ks);
    if constexpr (SPECIALISE && (SPEC_MASK & 64u)) fill_l64<LOGN, LOGE, 6, MB_MUL, MB_KS, ND_LO, ND_HI>(ks);
    if constexpr (LOGE >= 6) {  // one transform per block (k_ntt1), coalesced row side at N = 4096
        // N = 4096: coalesced row side, the two passes as a loop over one copy of the
        // pass code, 96 registers (10 blocks per SM), measured best in both directions
        constexpr bool COAL = LOGN == 12 && LOGE == 6;
        ks.ntt[0] = (void*)k_ntt1<LOGN, LOGE, false, 10, COAL, 1, COAL>;
        ks.ntt[1] = (void*)k_ntt1<LOGN, LOGE, true, 10, COAL, 1, COAL>;
        ks.ntt_jobs_per_block = 1;
    } else {
        ks.ntt[0] = (void*)k_ntt<LOGN, LOGE, false>;
        ks.ntt[1] = (void*)k_ntt<LOGN, LOGE, true>;
    }
    ks.smem_mul = region_bytes<PL, 2>();
    ks.smem_ks[0] = region_bytes<PL, ND_LO>();
    ks.smem_ks[1] = region_bytes<PL, ND_HI>();
    ks.smem_ntt = LOGE >= 6 ? region_bytes<PL, 1>() : region_bytes<PL, 2>();
}

}  // namespace cy
