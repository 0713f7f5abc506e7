// k_mixed: one persistent launch for a batch of polynomial products and YASHE
// multiplies of different rings (N from 1024 to 8192, q up to 192 bits): the
// fused CRT -> NTT -> pointwise -> INTT -> ICRT -> mod q (or YASHE rounding)
// path, then for relinearised YASHE jobs the keyswitch (digits -> NTT -> MAC
// with the resident evaluation key -> INTT -> ICRT -> mod q), over a work list.
//
// Blocks claim units from an atomic counter, in list order: every job's
// transform units (largest transforms first), then the first epilogues, then
// the keyswitch transforms, then the keyswitch epilogues. A unit of N = 8192
// fills a block; units of N = 4096, 2048 and 1024 run 2, 4 or 8 primes side by
// side, each on its own named barrier. A block that claims a unit whose inputs
// come from earlier units of its job waits until their count is complete. Those
// units were claimed earlier by blocks that are running, and the earliest
// unfinished unit waits for nothing, so every wait ends; no cooperative launch is
// needed. The spin is still bounded: on expiry the block records an error word
// and skips the unit instead of hanging.
//
// Two schedules (the autotuner picks per batch), both with 16 coefficients per thread in
// 512-thread blocks and the same primes in a unit at every N, so one work list serves both:
// two blocks per SM at 64 registers, where one's barriers, waits and epilogues overlap the
// other's transforms, or one at 128, where a unit ends sooner. Before, with 8 coefficients per
// thread in one 1024-thread block, a staged epilogue and a copy of the transforms per limb
// count and centring: 192 relinearised multiplies of N = 2048, 4096 and 8192 365 us, now 299; 12 of
// them 98 us, now 68.
#include "kernels.cuh"

namespace cy {

// Spin limit (iterations of a 256 ns back-off) a launch uses unless its plan
// sets a shorter one: about seconds, far beyond any unit's run time.
constexpr unsigned kMixedSpinDefault = 1u << 24;

template <int LOGN>
using MixedNtt = NttPlan<LOGN, 4>;
constexpr int kMixedThreads = 512;
constexpr int kMixedPrimes = 16;  // primes of a basis, at most (N <= 8192, q of up to 192 bits: 14)

// CRT split of a thread's coefficients of both operands (L64 limbs each); values above
// (q-1)/2 stand for x - q where `centered` is all ones.
template <class PL, int L64>
__device__ __forceinline__ void mixed_split(uint32_t (&x)[2][PL::E], const MixedJob& J, const BasisDev* __restrict__ B,
                                            int prime, int tau, uint32_t centered, const PrimeCtx& c) {
    constexpr int W = 2 * L64;
    uint32_t cc[W], qh[W];
#pragma unroll
    for (int w = 0; w < W; w++) {
        cc[w] = B->crt[prime][w];
        qh[w] = B->qhalf[w] | ~centered;  // all ones: no value is above
    }
#pragma unroll
    for (int e = 0; e < PL::E; e++) {
        const int pos = slot_pos<PL, 0>(tau, e);
        uint32_t wa[W], wb[W];
        load_words<L64>(J.a + (size_t)pos * L64, wa);
        load_words<L64>(J.b + (size_t)pos * L64, wb);
        x[0][e] = crt_words<W, true>(wa, cc, qh, c);
        x[1][e] = crt_words<W, true>(wb, cc, qh, c);
    }
}

// The limb count (1..3) and the centring are run-time choices around the CRT split only:
// one copy of the transforms per N (the blocks of an SM run different units).
template <int LOGN>
__device__ __forceinline__ void mixed_ntt_unit(const MixedJob& J, const MixedUnit& U, uint32_t* smem,
                                               uint32_t* __restrict__ done) {
    using PL = MixedNtt<LOGN>;
    constexpr int E = PL::E, G = PL::G;
    constexpr int SUBW = 2 * PL::SMW;  // exchange buffer of two operands per sub-group
    const int sub = threadIdx.x / G, tau = threadIdx.x % G;
    if (sub >= U.count) return;  // fewer primes than sub-groups in this unit
    const int prime = U.first + sub;
    const GroupSync bar{1 + sub, G};
    uint32_t* sm = smem + sub * SUBW;
    const BasisDev* __restrict__ B = J.B;
    const PrimeCtx c = load_prime_ctx(B, prime);
    const Mod& m = c.m;
    const uint32_t centered = J.centered ? ~0u : 0u;
    uint32_t x[2][E];
    if (J.l64 == 1) mixed_split<PL, 1>(x, J, B, prime, tau, centered, c);
    else if (J.l64 == 2) mixed_split<PL, 2>(x, J, B, prime, tau, centered, c);
    else mixed_split<PL, 3>(x, J, B, prime, tau, centered, c);
    ntt_forward<PL, 2, GroupSync>(x, B->psi[prime], m, tau, sm, false, bar, 1, lanes_of<PL>(B->tw.psi_lanes, prime));
    uint32_t z[1][E];
#pragma unroll
    for (int e = 0; e < E; e++) z[0][e] = mont(red_2p(x[0][e], c.m), red_2p(x[1][e], c.m), c.pinv, c.m);
    ntt_inverse<PL, 1, GroupSync>(z, B->ipsi[prime], m, tau, sm, bar, 1, lanes_of<PL>(B->tw.ipsi_lanes, prime));
    uint32_t* out = J.resid + (size_t)prime * PL::N;
#pragma unroll
    for (int e = 0; e < E; e++) out[slot_pos<PL, 0>(tau, e)] = z[0][e];
    __threadfence();  // residues visible device-wide before the count says so
    bar.sync();
    if (tau == 0) atomicAdd(&done[4 * U.job], 1u);
}

// Keyswitch transforms of `count` primes of the keyswitch basis: digits of c
// (written by this launch's first epilogues, so read through L2), two digits
// per pass, multiply-accumulate with the evaluation key in the NTT domain.
// ACC32: as in k_keyswitch (the 64-register schedule).
template <int LOGN, bool ACC32>
__device__ __forceinline__ void mixed_ks_unit(const MixedJob& J, const MixedUnit& U, uint32_t* smem,
                                              uint32_t* __restrict__ done) {
    using PL = MixedNtt<LOGN>;
    constexpr int E = PL::E, G = PL::G;
    constexpr int SUBW = 2 * PL::SMW;
    const int sub = threadIdx.x / G, tau = threadIdx.x % G;
    if (sub >= U.count) return;
    const int prime = U.first + sub;
    const GroupSync bar{1 + sub, G};
    uint32_t* sm = smem + sub * SUBW;
    const BasisDev* __restrict__ B = J.B2;
    const Mod m = load_mod(B, prime);
    const uint32_t pinv = B->pinv[prime];
    const int k2 = J.k2, ell = J.ell;
    uint64_t T[E];  // sums of products with the key (see k_keyswitch)
    uint32_t acc[1][E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        T[e] = 0;
        acc[0][e] = 0;
    }
    for (int d0 = 0; d0 < ell; d0 += 2) {
        uint32_t x[2][E];
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int pos = slot_pos<PL, 0>(tau, e);
#pragma unroll
            for (int o = 0; o < 2; o++) {
                const int d = d0 + o;
                uint32_t w = 0;
                if (d < ell) {  // c is limb-major here ([limb][N]): a warp's loads are contiguous
                    const uint64_t limb = __ldcg(reinterpret_cast<const unsigned long long*>(J.c) +
                                                 (size_t)(d >> 1) * PL::N + pos);
                    w = (uint32_t)(limb >> (32 * (d & 1)));
                }
                x[o][e] = __viaddmin_u32(w, m.np2, w);  // digit < 2^32 < 6p -> [0, 4p)
            }
        }
        ntt_forward<PL, 2, GroupSync>(x, B->psi[prime], m, tau, sm, d0 > 0, bar, 1,
                                      lanes_of<PL>(B->tw.psi_lanes, prime));
#pragma unroll
        for (int e = 0; e < E; e++) T[e] = ACC32 ? 0 : lazy_high(T[e], m);
#pragma unroll
        for (int o = 0; o < 2; o++) {
            const int d = d0 + o;
            if (d < ell) {
                uint32_t v[E];
                load_evk<PL::N, E>(J.evk + ((size_t)d * k2 + prime) * PL::N, last_pos<PL>(tau), v);
#pragma unroll
                for (int e = 0; e < E; e++) T[e] += (uint64_t)x[o][e] * v[e];
            }
        }
        if (ACC32) {
#pragma unroll
            for (int e = 0; e < E; e++) acc[0][e] = mac_red(acc[0][e], mac_finish<false>(T[e], pinv, m), m);
        }
    }
    if (!ACC32) {
#pragma unroll
        for (int e = 0; e < E; e++) acc[0][e] = mac_finish<true>(T[e], pinv, m);
    }
    ntt_inverse<PL, 1, GroupSync>(acc, B->ipsi[prime], m, tau, sm, bar, 1, lanes_of<PL>(B->tw.ipsi_lanes, prime));
    uint32_t* out = J.resid + (size_t)prime * PL::N;
#pragma unroll
    for (int e = 0; e < E; e++) out[slot_pos<PL, 0>(tau, e)] = acc[0][e];
    __threadfence();
    bar.sync();
    if (tau == 0) atomicAdd(&done[4 * U.job + 2], 1u);
}

// An epilogue unit: the basis's constants (blob: EpiConst<L, KMAX>) copied to shared
// memory, then one coefficient per thread and step.
template <int L, int MODE>
__device__ __forceinline__ void mixed_epi_coefs(const MixedJob& J, const BasisDev* __restrict__ B,
                                                const void* __restrict__ blob, int k, const MixedUnit& U, void* S,
                                                unsigned long long frac_limit) {
    using Const = EpiConst<L, kMixedPrimes>;
    using Blob = EpiConst<L, KMAX>;
    constexpr int TAIL = (sizeof(Blob) - KMAX * sizeof(EpiPrimeC<L>)) / 4;
    static_assert(TAIL == (sizeof(Const) - kMixedPrimes * sizeof(EpiPrimeC<L>)) / 4, "the same fields after the primes");
    Const& P = *static_cast<Const*>(S);
    const Blob& G = *static_cast<const Blob*>(blob);
    for (int i = threadIdx.x; i < k * (int)(sizeof(EpiPrimeC<L>) / 16); i += kMixedThreads)
        reinterpret_cast<uint4*>(P.pr)[i] = __ldg(reinterpret_cast<const uint4*>(G.pr) + i);
    for (int i = threadIdx.x; i < TAIL; i += kMixedThreads)
        reinterpret_cast<uint32_t*>(P.pr + kMixedPrimes)[i] = __ldg(reinterpret_cast<const uint32_t*>(G.pr + KMAX) + i);
    __syncthreads();
    const int n = 1 << J.logn;
    // a job with a keyswitch gets its first epilogue's output limb-major (the
    // keyswitch units' digit loads), and the keyswitch's epilogue writes over it
    const bool lm = U.kind == 1 && J.k2 > 0;
    const uint32_t* resid = J.resid;
    asm volatile("" : "+l"(resid) : : "memory");  // the residues' loads stay behind the wait for their units
    for (int c = U.first + threadIdx.x; c < U.first + U.count; c += kMixedThreads)
        epi_c_one<L, MODE, 0, false>(P, B, resid + c, n, J.c + (lm ? (size_t)c : (size_t)c * J.l64), lm ? (size_t)n : 1,
                                     frac_limit);
}

template <int MODE>
__device__ __forceinline__ void mixed_epi(const MixedJob& J, const BasisDev* __restrict__ B, const void* __restrict__ blob,
                                          int k, const MixedUnit& U, void* S, unsigned long long frac_limit) {
    switch (J.l32) {
        case 1: mixed_epi_coefs<1, MODE>(J, B, blob, k, U, S, frac_limit); break;
        case 2: mixed_epi_coefs<2, MODE>(J, B, blob, k, U, S, frac_limit); break;
        case 3: mixed_epi_coefs<3, MODE>(J, B, blob, k, U, S, frac_limit); break;
        case 4: mixed_epi_coefs<4, MODE>(J, B, blob, k, U, S, frac_limit); break;
        case 5: mixed_epi_coefs<5, MODE>(J, B, blob, k, U, S, frac_limit); break;
        case 6: mixed_epi_coefs<6, MODE>(J, B, blob, k, U, S, frac_limit); break;
        default: break;
    }
}

__device__ __forceinline__ uint32_t load_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// ctl[0]: unit counter; ctl[1]: set when a wait expired; ctl[2]: units skipped.
template <int BLOCKS>
__global__ void __launch_bounds__(kMixedThreads, BLOCKS)
    k_mixed(const MixedJob* __restrict__ jobs, const MixedUnit* __restrict__ units, int n_units,
            uint32_t* __restrict__ done, uint32_t* __restrict__ ctl, unsigned spin_limit,
            unsigned long long frac_limit) {
    extern __shared__ __align__(16) uint32_t smem[];
    __shared__ __align__(16) unsigned char S[sizeof(EpiConst<6, kMixedPrimes>)];  // the widest
    __shared__ int s_unit, s_ok;
    for (;;) {
        if (threadIdx.x == 0) s_unit = (int)atomicAdd(&ctl[0], 1u);
        __syncthreads();
        const int u = s_unit;
        if (u >= n_units) break;
        const MixedUnit U = units[u];
        const MixedJob J = jobs[U.job];
        if (U.kind != 0) {
            // inputs of this unit: every earlier-phase unit of its job
            const uint32_t need = U.kind == 1 ? (uint32_t)J.need0 : U.kind == 2 ? (uint32_t)J.n_epi : (uint32_t)J.k2;
            const uint32_t* cnt = &done[4 * U.job + (U.kind - 1)];
            if (threadIdx.x == 0) {
                unsigned spins = 0;
                while (load_acquire(cnt) < need && spins < spin_limit) {
                    __nanosleep(256);
                    spins++;
                }
                s_ok = load_acquire(cnt) >= need;
                if (!s_ok) {
                    atomicExch(&ctl[1], 1u);
                    atomicAdd(&ctl[2], 1u);
                }
            }
            __syncthreads();
            if (s_ok) __threadfence();
        }
        if (U.kind == 0) {
            switch (J.logn) {
                case 10: mixed_ntt_unit<10>(J, U, smem, done); break;
                case 11: mixed_ntt_unit<11>(J, U, smem, done); break;
                case 12: mixed_ntt_unit<12>(J, U, smem, done); break;
                case 13: mixed_ntt_unit<13>(J, U, smem, done); break;
                default: break;
            }
        } else if (U.kind == 2) {
            if (s_ok) {
                switch (J.logn) {
                    case 10: mixed_ks_unit<10, (BLOCKS > 1)>(J, U, smem, done); break;
                    case 11: mixed_ks_unit<11, (BLOCKS > 1)>(J, U, smem, done); break;
                    case 12: mixed_ks_unit<12, (BLOCKS > 1)>(J, U, smem, done); break;
                    case 13: mixed_ks_unit<13, (BLOCKS > 1)>(J, U, smem, done); break;
                    default: break;
                }
            }
        } else if (s_ok) {  // kinds 1 and 3: epilogues
            if (U.kind == 1 && J.mode == EPI_YASHE) mixed_epi<EPI_YASHE>(J, J.B, J.epi, J.k, U, S, frac_limit);
            else if (U.kind == 1) mixed_epi<EPI_MODQ>(J, J.B, J.epi, J.k, U, S, frac_limit);
            else mixed_epi<EPI_MODQ>(J, J.B2, J.epi2, J.k2, U, S, frac_limit);
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) atomicAdd(&done[4 * U.job + (U.kind == 1 ? 1 : 3)], 1u);
        }
        __syncthreads();  // shared memory and s_unit are reused by the next unit
    }
}

// Dynamic shared memory: exchange buffers of two operands of the widest unit (N = 8192).
constexpr size_t kMixedSmem = (size_t)2 * MixedNtt<13>::SMW * sizeof(uint32_t);
template <int LOGN>
constexpr bool mixed_fits() {
    constexpr int subs = kMixedThreads / MixedNtt<LOGN>::G;
    return subs >= 1 && subs * 2 * MixedNtt<LOGN>::SMW * sizeof(uint32_t) <= kMixedSmem;
}
static_assert(mixed_fits<10>() && mixed_fits<11>() && mixed_fits<12>() && mixed_fits<13>(), "every unit fits");

// schedule 0: two blocks per SM (64 registers); 1: one (128 registers)
int mixed_schedules() { return 2; }
void* mixed_kernel(int sched) { return sched == 1 ? (void*)k_mixed<1> : (void*)k_mixed<2>; }
size_t mixed_smem_bytes(int) { return kMixedSmem; }
int mixed_threads(int) { return kMixedThreads; }
unsigned mixed_spin_default() { return kMixedSpinDefault; }

}  // namespace cy
