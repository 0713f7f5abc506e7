// ntt_core.cuh -- negacyclic NTT of length N = 2^LOGN held in registers.
//
// The reference runs one radix-2 Stockham stage per kernel launch, through
// global memory, with one block per residue (NTT / NTTIteration,
// src/cuda_functions.cu:404-458; 3*log2(n) launches per product). Here a thread
// block of G = N/E threads owns one length-N transform: every thread keeps E
// coefficients in registers, the log2(N) stages are grouped into passes of at
// most LOGE stages that run entirely in registers, and consecutive passes swap
// data through a shared-memory buffer, in place (one barrier per swap, between
// the threads that share a sub-transform). Several operands (NOPS) of the same prime share the
// twiddle loads and interleave for instruction-level parallelism.
//
// Transform (merged negacyclic twist): forward Cooley-Tukey on natural-order
// input with twiddles psi^bitrev(m+i), output in bit-reversed order; inverse
// Gentleman-Sande on bit-reversed input with psi^-bitrev(m+i), natural-order
// output, without the N^-1 factor (folded into the ICRT constants). So
// INTT(NTT(a) . NTT(b)) = N * a*b mod (x^N + 1, p): the fold by x^N + 1 that the
// reference does on the host (src/cuda_functions.cu:1061-1072) is implicit.
//
// Index map of a pass that covers stages s0 .. s0+R-1 (stage s pairs j and
// j + N/2^(s+1)): with d = N >> (s0 + R), a butterfly group is the 2^R
// positions g*2^R*d + r + u*d (u < 2^R); thread tau owns groups
// gamma = tau + v*G (v < E/2^R) with g = gamma / d, r = gamma % d. The
// twiddle of stage s0+l for element u is tw[2^(s0+l) + g*2^l + (u >> (R-l))].
#pragma once
#include <type_traits>

#include <stdint.h>

#include "arith.cuh"

namespace cy {

template <int LOGN_, int LOGE_>
struct NttPlan {
    static constexpr int LOGN = LOGN_;
    static constexpr int LOGE = LOGE_;
    static constexpr int N = 1 << LOGN;
    static constexpr int E = 1 << LOGE;
    static constexpr int G = N >> LOGE;  // threads per transform
    static constexpr int NPASS = (LOGN + LOGE - 1) / LOGE;
    static constexpr int R0 = LOGN - (NPASS - 1) * LOGE;  // the first pass takes the remainder
    // words per operand buffer: N, and one more per 2^LOGE with 32 or 64 coefficients (XMap)
    static constexpr int SMW = LOGE >= 5 ? N + (N >> LOGE) : N;
    __host__ __device__ static constexpr int R(int pass) { return pass == 0 ? R0 : LOGE; }
    __host__ __device__ static constexpr int S0(int pass) { return pass == 0 ? 0 : R0 + (pass - 1) * LOGE; }
    __host__ __device__ static constexpr int LOGD(int pass) { return LOGN - S0(pass) - R(pass); }
};

// Barrier of the threads that own one transform: the whole block, or a named
// barrier (ids 1..15) shared by `count` threads when a block runs several
// independent transforms side by side.
struct CtaSync {
    __device__ __forceinline__ void sync() const { __syncthreads(); }
};
struct GroupSync {
    int id, count;
    __device__ __forceinline__ void sync() const {
        asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
    }
};

// Shared-memory layout of the exchanges of a plan with E = 2^R coefficients per
// thread. For one register slot of a pass whose butterflies span 2^D positions
// (D = LOGD) a warp touches 32 consecutive positions when D >= 5, else 32/2^D runs of
// 2^D positions 2^(D+R) apart; D is 0, R, 2R, .. . One layout for all of them, free of bank
// conflicts, so that every exchange of a plan is in place:
//   * R = 3, 4: an XOR of bits 2 .. 4 with bits of the row (pos >> 5), which permutes the
//     16-byte pieces of each 32-word row. It is linear over XOR, so the address of slot u of
//     a group is the group's address XOR a constant, and only the low 5 bits of that need an
//     instruction. The pass with D = 0 (a thread's positions are consecutive) moves 16 bytes
//     at a time, 8 lanes on distinct pieces of a row's 8;
//   * R >= 5: one padding word after every 2^R (an address stays base + constant): lanes
//     32 or 64 positions apart fall on distinct banks, runs of 32 stay together.
// Every pass, slot and warp of every plan was checked for conflicts on the host.
template <int R>
struct XMap {
    static constexpr bool SWZ = R == 3 || R == 4;
    __host__ __device__ static constexpr int map(int pos) {
        const int x = pos >> 5;
        if (R == 3) return pos ^ ((x & 7) << 2);
        if (R == 4) return pos ^ (((x & 3) | (((x >> 3) & 1) << 2)) << 2);
        return pos + (pos >> (R >= 6 ? 6 : 5));
    }
    // address of the position g | k from base = map(g), for k with no bit in common with g
    __device__ __forceinline__ static int at(int base, int k) {
        const int c = map(k);
        return SWZ ? (base ^ (c & 31)) + (c & ~31) : base + c;
    }
};

// position of the first element of group v of thread tau in pass PASS
template <class PL, int PASS>
__device__ __forceinline__ int group_base(int tau, int v) {
    constexpr int R = PL::R(PASS), LOGD = PL::LOGD(PASS);
    const int gam = tau + (v << (PL::LOGN - PL::LOGE));
    const int g = gam >> LOGD;
    const int r = gam & ((1 << LOGD) - 1);
    return (g << (LOGD + R)) | r;
}

// position of slot e (= v*2^R + u) of thread tau in pass PASS
template <class PL, int PASS>
__device__ __forceinline__ int slot_pos(int tau, int e) {
    constexpr int R = PL::R(PASS), LOGD = PL::LOGD(PASS);
    return group_base<PL, PASS>(tau, e >> R) + ((e & ((1 << R) - 1)) << LOGD);
}

// Twiddle h of a stage with 2^l twiddles per group. For l >= 1 the group
// starts at an even index of a 16-byte aligned table, so twiddles h and h+1 come
// from one 16-byte load (issued at even h; the compiler keeps the odd half).
__device__ __forceinline__ uint2 load_twiddle(const uint2* __restrict__ twl, int h, int l) {
    if (l == 0) return __ldg(twl);
    const uint4 W2 = __ldg(reinterpret_cast<const uint4*>(twl + (h & ~1)));
    return (h & 1) ? make_uint2(W2.z, W2.w) : make_uint2(W2.x, W2.y);
}

// The last forward (first inverse) pass, in which thread tau owns the E consecutive
// positions of row tau, needs twiddles tw[2^(S0+l) + tau 2^l + h] (h < 2^l): 2^l consecutive
// entries per thread. It reads a copy of the table laid out by lane (rows_index), so that a
// warp's loads are consecutive, where there is one.
struct NoLanes {};  // in place of that table
template <class PL, int PASS, class LT>
__host__ __device__ constexpr bool rows_pass() {
    return std::is_same<LT, const uint2*>::value && PASS == PL::NPASS - 1 && PL::NPASS > 1;
}
template <bool ROWS, class LT>
__device__ __forceinline__ auto lanes_if(LT twr) {
    if constexpr (ROWS) return twr;
    else return NoLanes();
}
// first entry of stage l (a pass's group g, or lane tau of a lane-ordered table)
template <class PL>
__device__ __forceinline__ const uint2* stage_twiddles(const uint2*, const uint2* __restrict__ twr, int l, int, int tau) {
    return twr + rows_index(PL::G, l, 0, tau);
}
template <class PL>
__device__ __forceinline__ const uint2* stage_twiddles(const uint2* __restrict__ tws, NoLanes, int l, int g, int) {
    return tws + (g << l);  // 16-byte aligned for l >= 1
}
__device__ __forceinline__ uint2 load_twiddle_rows(const uint2* __restrict__ twl, int h, int l, int G) {
    if (l == 0) return __ldg(twl);
    const uint4 W2 = __ldg(reinterpret_cast<const uint4*>(twl + (h >> 1) * 2 * G));
    return (h & 1) ? make_uint2(W2.z, W2.w) : make_uint2(W2.x, W2.y);
}

// tm: twiddle-offset multiplier. A transform of length N is stages 0.. of one of
// length 2N restricted to half h of it when its stage-s twiddles start at
// (2 + h) * 2^s instead of 2^s (tm = 2 + h); tm = 1 for a whole transform.
// twr: the lane-ordered table of this prime and length, or NoLanes.
template <class PL, int PASS, int NOPS, class LT = NoLanes>
__device__ __forceinline__ void fwd_pass(uint32_t (&x)[NOPS][PL::E], const uint2* __restrict__ tw, const Mod& m,
                                         int tau, int tm = 1, LT twr = LT()) {
    constexpr int R = PL::R(PASS), S0 = PL::S0(PASS), LOGD = PL::LOGD(PASS);
    constexpr int GS = 1 << R;
    constexpr int NV = PL::E >> R;
    constexpr bool ROWS = rows_pass<PL, PASS, LT>();
    const auto lanes = lanes_if<ROWS>(twr);
#pragma unroll
    for (int v = 0; v < NV; v++) {
        const int gam = tau + (v << (PL::LOGN - PL::LOGE));
        const int g = (S0 == 0) ? 0 : (gam >> LOGD);
#pragma unroll
        for (int l = 0; l < R; l++) {
            const int half = 1 << (R - 1 - l);
            const uint2* twl = stage_twiddles<PL>(tw + (tm << (S0 + l)), lanes, l, g, tau);
            // one flat loop of 2^(R-1) butterflies per stage (a trip count that does
            // not depend on l, so that every loop unrolls fully for R = 6 too):
            // butterfly b is j = b mod half of twiddle group h = b / half
            uint2 W = make_uint2(0u, 0u);
#pragma unroll
            for (int b = 0; b < GS / 2; b++) {
                const int h = b >> (R - 1 - l), j = b & (half - 1);
                if (j == 0) W = ROWS ? load_twiddle_rows(twl, h, l, PL::G) : load_twiddle(twl, h, l);
                const int u = (h << (R - l)) + j;
#pragma unroll
                for (int o = 0; o < NOPS; o++) ct_bfly(x[o][v * GS + u], x[o][v * GS + u + half], W.x, W.y, m);
            }
        }
    }
}

// scale (inverse, pass 0, optional): {N^-1, Shoup, N^-1 w1, Shoup} with w1 the
// twiddle of the last stage; that stage then writes (X + Y) N^-1 and
// (X - Y) w1 N^-1 in [0, p), so no separate scaling pass is needed.
template <class PL, int PASS, int NOPS, class LT = NoLanes>
__device__ __forceinline__ void inv_pass(uint32_t (&x)[NOPS][PL::E], const uint2* __restrict__ tw, const Mod& m,
                                         int tau, int tm = 1, LT twr = LT(),
                                         const uint32_t* __restrict__ scale = nullptr) {
    constexpr int R = PL::R(PASS), S0 = PL::S0(PASS), LOGD = PL::LOGD(PASS);
    constexpr int GS = 1 << R;
    constexpr int NV = PL::E >> R;
    constexpr bool ROWS = rows_pass<PL, PASS, LT>();
    const auto lanes = lanes_if<ROWS>(twr);
#pragma unroll
    for (int v = 0; v < NV; v++) {
        const int gam = tau + (v << (PL::LOGN - PL::LOGE));
        const int g = (S0 == 0) ? 0 : (gam >> LOGD);
#pragma unroll
        for (int l = R - 1; l >= 0; l--) {
            const int half = 1 << (R - 1 - l);
            const uint2* twl = stage_twiddles<PL>(tw + (tm << (S0 + l)), lanes, l, g, tau);
            uint2 W = make_uint2(0u, 0u);
            if (PASS == 0 && l == 0 && scale != nullptr) {  // last stage, N^-1 folded in (S0 = 0, g = 0)
                const uint32_t n0 = __ldg(scale), n0s = __ldg(scale + 1), n1 = __ldg(scale + 2),
                               n1s = __ldg(scale + 3);
#pragma unroll
                for (int b = 0; b < GS / 2; b++) {
                    const int u = b;  // l = 0: half = 2^(R-1), one twiddle group
#pragma unroll
                    for (int o = 0; o < NOPS; o++) {
                        uint32_t& X = x[o][v * GS + u];
                        uint32_t& Y = x[o][v * GS + u + half];
                        const uint32_t s = shoup_m(X + Y, n0, n0s, m);         // [0, 2p)
                        const uint32_t d = shoup_m(X - Y + m.p2, n1, n1s, m);  // [0, 2p)
                        X = __viaddmin_u32(s, m.np, s);
                        Y = __viaddmin_u32(d, m.np, d);
                    }
                }
                continue;
            }
#pragma unroll
            for (int b = 0; b < GS / 2; b++) {  // as in fwd_pass
                const int h = b >> (R - 1 - l), j = b & (half - 1);
                if (j == 0) W = ROWS ? load_twiddle_rows(twl, h, l, PL::G) : load_twiddle(twl, h, l);
                const int u = (h << (R - l)) + j;
#pragma unroll
                for (int o = 0; o < NOPS; o++) gs_bfly(x[o][v * GS + u], x[o][v * GS + u + half], W.x, W.y, m);
            }
        }
    }
}

// Registers laid out for pass PA -> registers laid out for pass PB (a neighbour), through
// shared memory `sm` (NOPS buffers of SMW words). In place: every exchange of a plan uses
// one layout, so a thread writes exactly the words it read in the exchange before, and one
// barrier, between the writes and the reads, is enough. Only the first forward exchange
// into a buffer whose words other threads may still be reading (the transform before)
// needs one ahead of its writes (`sync_before`). When the passes' sub-transforms (the N >> S0
// positions that the earlier pass's butterflies stay within) belong to one warp, the
// barrier is the warp's.
// Two alternating regions (fewer blocks per SM), or two barriers per exchange, took its place
// before. With 16 coefficients per thread, 512 products at N = 4096, 127-bit q: 164 -> 150 us, 512
// keyswitches 171 -> 154 us; 512 x 14 transforms of length 8192: 220 -> 158 us forward, 212 ->
// 161 us inverse.
template <class PL, int PA, int PB, int NOPS, class Sync = CtaSync>
__device__ __forceinline__ void exchange(uint32_t (&x)[NOPS][PL::E], uint32_t* sm, int tau, bool sync_before,
                                         Sync bar = Sync()) {
    constexpr int RA = PL::R(PA), LA = PL::LOGD(PA), NVA = PL::E >> RA;
    constexpr int RB = PL::R(PB), LB = PL::LOGD(PB), NVB = PL::E >> RB;
    constexpr int PLO = PA < PB ? PA : PB;
    // threads that share a sub-transform of pass PLO (whole warps hold whole groups)
    constexpr bool WARP = PL::G >= 32 && ((PL::N >> PL::S0(PLO)) >> PL::LOGE) <= 32;
    using X = XMap<PL::LOGE>;
    // consecutive positions: 16-byte accesses
    constexpr bool VECA = X::SWZ && LA == 0 && NVA == 1, VECB = X::SWZ && LB == 0 && NVB == 1;
    if (sync_before) bar.sync();
#pragma unroll
    for (int v = 0; v < NVA; v++) {
        const int base = X::map(group_base<PL, PA>(tau, v));  // bits of u << LA are zero in it
        if constexpr (VECA) {
#pragma unroll
            for (int u = 0; u < PL::E; u += 4) {
                const int a = X::at(base, u);
#pragma unroll
                for (int o = 0; o < NOPS; o++)
                    *reinterpret_cast<uint4*>(sm + o * PL::SMW + a) =
                        make_uint4(x[o][u], x[o][u + 1], x[o][u + 2], x[o][u + 3]);
            }
        } else {
#pragma unroll
            for (int u = 0; u < (1 << RA); u++) {
                const int a = X::at(base, u << LA);
#pragma unroll
                for (int o = 0; o < NOPS; o++) sm[o * PL::SMW + a] = x[o][(v << RA) + u];
            }
        }
    }
    if constexpr (WARP) __syncwarp();
    else bar.sync();
#pragma unroll
    for (int v = 0; v < NVB; v++) {
        const int base = X::map(group_base<PL, PB>(tau, v));
        if constexpr (VECB) {
#pragma unroll
            for (int u = 0; u < PL::E; u += 4) {
                const int a = X::at(base, u);
#pragma unroll
                for (int o = 0; o < NOPS; o++) {
                    const uint4 q = *reinterpret_cast<const uint4*>(sm + o * PL::SMW + a);
                    x[o][u] = q.x;
                    x[o][u + 1] = q.y;
                    x[o][u + 2] = q.z;
                    x[o][u + 3] = q.w;
                }
            }
        } else {
#pragma unroll
            for (int u = 0; u < (1 << RB); u++) {
                const int a = X::at(base, u << LB);
#pragma unroll
                for (int o = 0; o < NOPS; o++) x[o][(v << RB) + u] = sm[o * PL::SMW + a];
            }
        }
    }
}

// The last pass's layout (thread tau has the E positions from E tau on) against one in which
// four consecutive registers of a warp's lanes are 128 consecutive positions: register e (a
// multiple of 4) of lane L is position E 32 (tau / 32) + 32 e + 4 L, so that a warp's 16-byte global
// accesses are consecutive. Inside a warp's own words of `sm`; rows_to_lanes follows a forward
// transform, lanes_to_rows precedes an inverse one.
template <class PL>
__host__ __device__ constexpr bool lanes_ok() {
    return XMap<PL::LOGE>::SWZ && PL::G >= 32;
}
template <class PL>
__device__ __forceinline__ int lane_pos(int tau, int e) {
    return ((tau >> 5) << (5 + PL::LOGE)) + 32 * e + 4 * (tau & 31);
}
template <class PL, int NOPS>
__device__ __forceinline__ void rows_to_lanes(uint32_t (&x)[NOPS][PL::E], uint32_t* sm, int tau) {
    using X = XMap<PL::LOGE>;
    const int base = X::map(tau << PL::LOGE);
#pragma unroll
    for (int u = 0; u < PL::E; u += 4)
#pragma unroll
        for (int o = 0; o < NOPS; o++)
            *reinterpret_cast<uint4*>(sm + o * PL::SMW + X::at(base, u)) =
                make_uint4(x[o][u], x[o][u + 1], x[o][u + 2], x[o][u + 3]);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < PL::E; e += 4) {
        const int a = X::map(lane_pos<PL>(tau, e));
#pragma unroll
        for (int o = 0; o < NOPS; o++) {
            const uint4 q = *reinterpret_cast<const uint4*>(sm + o * PL::SMW + a);
            x[o][e] = q.x;
            x[o][e + 1] = q.y;
            x[o][e + 2] = q.z;
            x[o][e + 3] = q.w;
        }
    }
}
template <class PL, int NOPS>
__device__ __forceinline__ void lanes_to_rows(uint32_t (&x)[NOPS][PL::E], uint32_t* sm, int tau) {
    using X = XMap<PL::LOGE>;
#pragma unroll
    for (int e = 0; e < PL::E; e += 4) {
        const int a = X::map(lane_pos<PL>(tau, e));
#pragma unroll
        for (int o = 0; o < NOPS; o++)
            *reinterpret_cast<uint4*>(sm + o * PL::SMW + a) = make_uint4(x[o][e], x[o][e + 1], x[o][e + 2], x[o][e + 3]);
    }
    __syncwarp();
    const int base = X::map(tau << PL::LOGE);
#pragma unroll
    for (int u = 0; u < PL::E; u += 4) {
        const int a = X::at(base, u);
#pragma unroll
        for (int o = 0; o < NOPS; o++) {
            const uint4 q = *reinterpret_cast<const uint4*>(sm + o * PL::SMW + a);
            x[o][u] = q.x;
            x[o][u + 1] = q.y;
            x[o][u + 2] = q.z;
            x[o][u + 3] = q.w;
        }
    }
}

// Forward passes PASS .. NPASS-1 (sync_before: as in exchange, for the first one).
template <class PL, int PASS, int NOPS, class Sync = CtaSync, class LT = NoLanes>
struct FwdFrom {
    __device__ __forceinline__ static void run(uint32_t (&x)[NOPS][PL::E], const uint2* __restrict__ tw,
                                               const Mod& m, int tau, uint32_t* sm, bool sync_before,
                                               Sync bar = Sync(), int tm = 1, LT twr = LT()) {
        if constexpr (PASS < PL::NPASS) {
            exchange<PL, PASS - 1, PASS, NOPS, Sync>(x, sm, tau, sync_before, bar);
            fwd_pass<PL, PASS, NOPS>(x, tw, m, tau, tm, twr);
            FwdFrom<PL, PASS + 1, NOPS, Sync, LT>::run(x, tw, m, tau, sm, false, bar, tm, twr);
        }
    }
};

// Inverse passes PASS .. 0 where pass PASS+1 was the previous one.
template <class PL, int PASS, int NOPS, class Sync = CtaSync, class LT = NoLanes>
struct InvFrom {
    __device__ __forceinline__ static void run(uint32_t (&x)[NOPS][PL::E], const uint2* __restrict__ tw,
                                               const Mod& m, int tau, uint32_t* sm, Sync bar = Sync(), int tm = 1,
                                               LT twr = LT(),
                                               const uint32_t* __restrict__ scale = nullptr) {
        if constexpr (PASS >= 0) {
            exchange<PL, PASS + 1, PASS, NOPS, Sync>(x, sm, tau, false, bar);
            inv_pass<PL, PASS, NOPS>(x, tw, m, tau, tm, twr, scale);
            InvFrom<PL, PASS - 1, NOPS, Sync, LT>::run(x, tw, m, tau, sm, bar, tm, twr, scale);
        }
    }
};

// Full forward transform: registers in pass-0 layout (natural order) ->
// registers in last-pass layout (bit-reversed order). sync_before: other threads may still
// be reading `sm` (a transform before this one in the same block).
template <class PL, int NOPS, class Sync = CtaSync, class LT = NoLanes>
__device__ __forceinline__ void ntt_forward(uint32_t (&x)[NOPS][PL::E], const uint2* __restrict__ tw, const Mod& m,
                                            int tau, uint32_t* sm, bool sync_before = false, Sync bar = Sync(),
                                            int tm = 1, LT twr = LT()) {
    fwd_pass<PL, 0, NOPS>(x, tw, m, tau, tm, twr);
    FwdFrom<PL, 1, NOPS, Sync, LT>::run(x, tw, m, tau, sm, sync_before, bar, tm, twr);
}

// Full inverse transform: registers in last-pass layout -> pass-0 layout. `sm` may hold a
// forward transform of this block (each thread then writes the words it read last).
template <class PL, int NOPS, class Sync = CtaSync, class LT = NoLanes>
__device__ __forceinline__ void ntt_inverse(uint32_t (&x)[NOPS][PL::E], const uint2* __restrict__ tw, const Mod& m,
                                            int tau, uint32_t* sm, Sync bar = Sync(), int tm = 1,
                                            LT twr = LT(),
                                            const uint32_t* __restrict__ scale = nullptr) {
    inv_pass<PL, PL::NPASS - 1, NOPS>(x, tw, m, tau, tm, twr, scale);
    InvFrom<PL, PL::NPASS - 2, NOPS, Sync, LT>::run(x, tw, m, tau, sm, bar, tm, twr, scale);
}

// ---------------------------------------------------------------------------
// Two-pass transforms of 64 coefficients per thread (N = 4096) with ONE copy of
// the pass code: both passes pair the same register slots at every stage (slot
// u with u + 2^(5-l)); only their twiddles differ (the first pass's are the same
// for every thread, the row pass's come from the lane-ordered table). The passes
// therefore run as two iterations of a loop that is not unrolled, with the
// twiddle pointers of the iteration in registers: half the instructions of the
// unrolled transform in the instruction cache.
// twp[l]: twiddle 0 of stage l (pairs (h, h+1) start there for l >= 1);
// tws: distance in uint2 between consecutive pairs (2, or 2G in the rows table).
template <int NOPS>
__device__ __forceinline__ uint2 tw_dyn(const uint2* __restrict__ base, int h, int l, int tws) {
    if (l == 0) return __ldg(base);
    const uint4 W2 = __ldg(reinterpret_cast<const uint4*>(base + (h >> 1) * tws));
    return (h & 1) ? make_uint2(W2.z, W2.w) : make_uint2(W2.x, W2.y);
}

template <int NOPS>
__device__ __forceinline__ void fwd_pass64(uint32_t (&x)[NOPS][64], const uint2* const (&twp)[6], int tws,
                                           const Mod& m) {
#pragma unroll
    for (int l = 0; l < 6; l++) {
        const int half = 1 << (5 - l);
        uint2 W = make_uint2(0u, 0u);
#pragma unroll
        for (int b = 0; b < 32; b++) {
            const int h = b >> (5 - l), j = b & (half - 1);
            if (j == 0) W = tw_dyn<NOPS>(twp[l], h, l, tws);
            const int u = (h << (6 - l)) + j;
#pragma unroll
            for (int o = 0; o < NOPS; o++) ct_bfly(x[o][u], x[o][u + half], W.x, W.y, m);
        }
    }
}

template <int NOPS>
__device__ __forceinline__ void inv_pass64(uint32_t (&x)[NOPS][64], const uint2* const (&twp)[6], int tws,
                                           const Mod& m, const uint32_t* __restrict__ scale) {
#pragma unroll
    for (int l = 5; l >= 0; l--) {
        const int half = 1 << (5 - l);
        if (l == 0 && scale != nullptr) {  // the transform's last stage with N^-1 folded in
            const uint32_t n0 = __ldg(scale), n0s = __ldg(scale + 1), n1 = __ldg(scale + 2), n1s = __ldg(scale + 3);
#pragma unroll
            for (int u = 0; u < 32; u++)
#pragma unroll
                for (int o = 0; o < NOPS; o++) {
                    uint32_t& X = x[o][u];
                    uint32_t& Y = x[o][u + 32];
                    const uint32_t sv = shoup_m(X + Y, n0, n0s, m);
                    const uint32_t dv = shoup_m(X - Y + m.p2, n1, n1s, m);
                    X = __viaddmin_u32(sv, m.np, sv);
                    Y = __viaddmin_u32(dv, m.np, dv);
                }
            continue;
        }
        uint2 W = make_uint2(0u, 0u);
#pragma unroll
        for (int b = 0; b < 32; b++) {
            const int h = b >> (5 - l), j = b & (half - 1);
            if (j == 0) W = tw_dyn<NOPS>(twp[l], h, l, tws);
            const int u = (h << (6 - l)) + j;
#pragma unroll
            for (int o = 0; o < NOPS; o++) gs_bfly(x[o][u], x[o][u + half], W.x, W.y, m);
        }
    }
}

// twiddle pointers of pass `pass` (0: column pass, shared by all threads; 1: row
// pass, lane-ordered table) of a transform of 4096 with 64 threads
__device__ __forceinline__ void pass64_twiddles(int pass, const uint2* __restrict__ tw, const uint2* __restrict__ twr,
                                                int tau, const uint2* (&twp)[6], int& tws) {
#pragma unroll
    for (int l = 0; l < 6; l++)
        twp[l] = pass == 0 ? tw + (1 << l) : twr + rows_index(64, l, 0, tau);
    tws = pass == 0 ? 2 : 128;
}

// Forward transform, registers in column layout (positions tau + 64 u) ->
// row layout (64 tau + u); exchange region `sm` (one, SMW = 4160 words per operand).
template <class PL, int NOPS>
__device__ __forceinline__ void ntt64_forward(uint32_t (&x)[NOPS][64], const uint2* __restrict__ tw,
                                              const uint2* __restrict__ twr, const Mod& m, int tau, uint32_t* sm,
                                              bool sync_before = false) {
    static_assert(PL::LOGN == 12 && PL::LOGE == 6, "two passes of six stages");
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
        const uint2* twp[6];
        int tws;
        pass64_twiddles(pass, tw, twr, tau, twp, tws);
        fwd_pass64<NOPS>(x, twp, tws, m);
        if (pass == 0) exchange<PL, 0, 1, NOPS>(x, sm, tau, sync_before);
    }
}

// Inverse transform, row layout -> column layout; scale as in inv_pass (or null).
template <class PL, int NOPS>
__device__ __forceinline__ void ntt64_inverse(uint32_t (&x)[NOPS][64], const uint2* __restrict__ tw,
                                              const uint2* __restrict__ twr, const Mod& m, int tau, uint32_t* sm,
                                              const uint32_t* __restrict__ scale) {
    static_assert(PL::LOGN == 12 && PL::LOGE == 6, "two passes of six stages");
#pragma unroll 1
    for (int it = 0; it < 2; it++) {
        const int pass = 1 - it;
        const uint2* twp[6];
        int tws;
        pass64_twiddles(pass, tw, twr, tau, twp, tws);
        inv_pass64<NOPS>(x, twp, tws, m, pass == 0 ? scale : nullptr);
        if (pass == 1) exchange<PL, 1, 0, NOPS>(x, sm, tau, false);
    }
}

}  // namespace cy
