// encrypt.cu -- YASHE encryption on the GPU with on-device sampling.
//
// Replaces Yashe::encrypt (src/yashe.cpp:104-142) and its samplers
// (src/distribution.cpp:4-60, src/cuda_distribution.cu:11-35, which draw
// uniform values with cuRAND where the scheme asks for an error distribution):
//   ct = [h*s + e + Delta*m]_q,  Delta = floor(q/t),  s, e ~ D_sigma (discrete
//   Gaussian on [-B, B], B = ceil(6 sigma)).
//
// Randomness is counter-based, so that every coefficient is drawn
// independently on its own thread and the draws can be reproduced exactly on
// the CPU: draw number c of a call with seed S is the c-th output of splitmix64
// seeded with S, i.e. mix(S + (c+1) * 0x9E3779B97F4A7C15). Coefficient i of s
// (of e) for ciphertext b uses counter (2b) * N + i ((2b+1) * N + i). A draw
// u is mapped to x = j - B with j the first index of the CDT table with
// u < T[j] (T: 64-bit cumulative thresholds, see gaussian_cdt).
//
// Three steps on the caller's stream: a sampling kernel writes s (as limbs mod q, or
// as signed words) into the output, the product kernels compute h*s in place (a chunk's product
// kernel reads its inputs before its epilogue writes), and k_enc_finish adds e
// and Delta*m and reduces mod q.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "host.h"
#include "kernels.cuh"

namespace cy {

cy_status run_product_api(const Basis& B, bool centered, const uint64_t* a, long long a_stride, const uint64_t* b,
                          long long b_stride, void* out, long long out_stride, int batch, Workspace& ws,
                          cudaStream_t st, int variant = -1, const uint32_t* key = nullptr, bool small = false);
int trace_begin(const char* name, int logn, cudaStream_t st);
void trace_end(int idx, cudaStream_t st);

constexpr int kCdtMax = 512;  // thresholds (sigma up to 42)

// Host: the 64-bit CDT thresholds of D_sigma on [-B, B], B = ceil(6 sigma):
// w_j = exp(-x^2 / (2 sigma^2)) for x = j - B, acc_j = sum_{i<=j} w_i / total,
// T_j = floor(acc_j * 2^64) (2^64 - 1 for the last entry and when acc_j >= 1).
std::vector<uint64_t> gaussian_cdt(double sigma) {
    const int bound = (int)std::ceil(6.0 * sigma);
    std::vector<double> w(2 * bound + 1);
    double total = 0.0;
    for (int j = 0; j <= 2 * bound; j++) {
        const int x = j - bound;
        w[j] = std::exp(-(double)(x * x) / (2.0 * sigma * sigma));
        total += w[j];
    }
    std::vector<uint64_t> T(w.size());
    double acc = 0.0;
    for (size_t j = 0; j < w.size(); j++) {
        acc += w[j] / total;
        T[j] = acc >= 1.0 ? ~0ULL : (uint64_t)(acc * 18446744073709551616.0);
    }
    T.back() = ~0ULL;
    return T;
}

struct EncConsts {
    uint64_t q[6];
    uint64_t delta[6];  // floor(q / t)
    uint64_t seed;
    uint32_t t;
    int l64, logn, bound, ncdt;
};

__device__ __forceinline__ uint64_t counter_draw(uint64_t seed, uint64_t ctr) {
    uint64_t z = seed + (ctr + 1) * 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

// first j with u < T[j] (the last threshold is 2^64 - 1, so j <= ncdt - 1)
__device__ __forceinline__ int cdt_sample(const uint64_t* T, int ncdt, int bound, uint64_t u) {
    int lo = 0, hi = ncdt - 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (T[mid] <= u) lo = mid + 1;
        else hi = mid;
    }
    return lo - bound;
}

__device__ __forceinline__ void load_cdt(uint64_t* sT, const uint64_t* __restrict__ T, int ncdt) {
    for (int i = threadIdx.x; i < ncdt; i += blockDim.x) sT[i] = T[i];
    __syncthreads();
}

// The limbs of one coefficient (16-byte accesses when their number is even).
template <int L>
__device__ __forceinline__ void load_limbs(const uint64_t* __restrict__ p, uint64_t (&x)[L]) {
    if constexpr (L % 2 == 0) {
#pragma unroll
        for (int w = 0; w < L; w += 2) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p + w);
            x[w] = v.x;
            x[w + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int w = 0; w < L; w++) x[w] = p[w];
    }
}
template <int L>
__device__ __forceinline__ void store_limbs(uint64_t* __restrict__ p, const uint64_t* x) {
    if constexpr (L % 2 == 0) {
#pragma unroll
        for (int w = 0; w < L; w += 2) *reinterpret_cast<ulonglong2*>(p + w) = make_ulonglong2(x[w], x[w + 1]);
    } else {
#pragma unroll
        for (int w = 0; w < L; w++) p[w] = x[w];
    }
}

// [s]_q of a small signed s
template <int L>
__device__ __forceinline__ void store_signed(const EncConsts& C, long long s, uint64_t* __restrict__ dst) {
    uint64_t x[L];
    uint64_t borrow = s < 0 ? (uint64_t)(-s) : 0;  // q - |s|, or 0 + s
#pragma unroll
    for (int w = 0; w < L; w++) {
        const uint64_t qw = s < 0 ? C.q[w] : (w == 0 ? (uint64_t)s : 0);
        x[w] = qw - borrow;
        borrow = qw < borrow;
    }
    store_limbs<L>(dst, x);
}

// x (below 4q) -> x mod q, written to dst
template <int L>
__device__ __forceinline__ void reduce_small_multiple(uint64_t (&x)[L + 1], const uint64_t* q, uint64_t* __restrict__ dst) {
#pragma unroll
    for (int it = 0; it < 3; it++) {
        uint64_t t[L + 1];
        uint64_t borrow = 0;
#pragma unroll
        for (int w = 0; w <= L; w++) {
            const uint64_t qw = w < L ? q[w] : 0;
            const uint64_t d = x[w] - qw;
            t[w] = d - borrow;
            borrow = (x[w] < qw) | (d < borrow);
        }
        if (borrow) break;  // x < q
#pragma unroll
        for (int w = 0; w <= L; w++) x[w] = t[w];
    }
    store_limbs<L>(dst, x);
}

// x = c + Delta (m mod t), below Delta t + q
template <int L>
__device__ __forceinline__ void add_scaled(const EncConsts& C, uint64_t m, const uint64_t* __restrict__ c,
                                           uint64_t (&x)[L + 1]) {
    const uint64_t mv = m < C.t ? m : m % C.t;
    uint64_t cv[L];
    load_limbs<L>(c, cv);
    uint64_t carry = 0;
#pragma unroll
    for (int w = 0; w < L; w++) {
        const uint64_t lo = C.delta[w] * mv, hi = __umul64hi(C.delta[w], mv);  // hi < 2^32
        const uint64_t s = lo + cv[w];
        x[w] = s + carry;
        carry = hi + (s < lo) + (x[w] < s);
    }
    x[L] = carry;
}

// These kernels move each limb once and are bound by that; with the limb count at run time
// (loops, 128-bit arithmetic, 8-byte strided accesses) 256 ciphertexts at N = 4096, 127-bit q,
// took 28 us to sample and 54 us to finish, now 13 and 18.

// s -> out as limbs of [s]_q
template <int L>
__global__ void k_enc_sample(const __grid_constant__ EncConsts C, const uint64_t* __restrict__ T,
                             uint64_t* __restrict__ out, int batch) {
    __shared__ uint64_t sT[kCdtMax];
    load_cdt(sT, T, C.ncdt);
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= ((long long)batch << C.logn)) return;
    const long long b = idx >> C.logn, i = idx & ((1LL << C.logn) - 1);
    const int s = cdt_sample(sT, C.ncdt, C.bound, counter_draw(C.seed, ((uint64_t)(2 * b) << C.logn) + i));
    store_signed<L>(C, s, out + idx * L);
}

// s -> the first words of each ciphertext's row, one signed word per coefficient
__global__ void k_enc_sample_small(const __grid_constant__ EncConsts C, const uint64_t* __restrict__ T,
                                   uint64_t* __restrict__ out, int batch) {
    __shared__ uint64_t sT[kCdtMax];
    load_cdt(sT, T, C.ncdt);
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= ((long long)batch << C.logn)) return;
    const long long b = idx >> C.logn, i = idx & ((1LL << C.logn) - 1);
    reinterpret_cast<int*>(out + ((b * C.l64) << C.logn))[i] =
        cdt_sample(sT, C.ncdt, C.bound, counter_draw(C.seed, ((uint64_t)(2 * b) << C.logn) + i));
}

// ct = [hs + e + Delta*(m mod t)]_q in place (hs in [0, q), e in [-B, B])
template <int L>
__global__ void k_enc_finish(const __grid_constant__ EncConsts C, const uint64_t* __restrict__ T,
                             const uint64_t* __restrict__ m, uint64_t* __restrict__ ct, int batch) {
    __shared__ uint64_t sT[kCdtMax];
    load_cdt(sT, T, C.ncdt);
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= ((long long)batch << C.logn)) return;
    const long long b = idx >> C.logn, i = idx & ((1LL << C.logn) - 1);
    const int e = cdt_sample(sT, C.ncdt, C.bound, counter_draw(C.seed, ((uint64_t)(2 * b + 1) << C.logn) + i));
    uint64_t* c = ct + idx * L;
    uint64_t x[L + 1];
    add_scaled<L>(C, m[idx], c, x);
    // + e, or + (q - |e|): the sum stays in [0, 3q + B]
    uint64_t carry = (uint64_t)(e < 0 ? -e : e), borrow = 0;
    if (e < 0) {
        borrow = carry;
        carry = 0;
    }
#pragma unroll
    for (int w = 0; w <= L; w++) {
        const uint64_t qw = (e < 0 && w < L) ? C.q[w] : 0;
        const uint64_t s = x[w] + qw, s2 = s + carry;
        carry = (s < x[w]) | (s2 < s);
        x[w] = s2 - borrow;
        borrow = s2 < borrow;
    }
    reduce_small_multiple<L>(x, C.q, c);
}

// out = [c + Delta*(m mod t)]_q (plaintext addition)
template <int L>
__global__ void k_add_plain(const __grid_constant__ EncConsts C, const uint64_t* __restrict__ m,
                            const uint64_t* __restrict__ cin, uint64_t* __restrict__ out, int batch) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= ((long long)batch << C.logn)) return;
    uint64_t x[L + 1];
    add_scaled<L>(C, m[idx], cin + idx * L, x);
    reduce_small_multiple<L>(x, C.q, out + idx * L);
}

// out = [m_c]_q with m_c the representative of m mod t in (-t/2, t/2]
template <int L>
__global__ void k_lift_plain(const __grid_constant__ EncConsts C, const uint64_t* __restrict__ m,
                             uint64_t* __restrict__ out, int batch) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= ((long long)batch << C.logn)) return;
    const uint64_t mv = m[idx];
    const long long v = (long long)(mv < C.t ? mv : mv % C.t);
    store_signed<L>(C, v <= (long long)(C.t / 2) ? v : v - (long long)C.t, out + idx * L);
}

// the kernel of a template above for l64 limbs
#define CY_ENC_TABLE(NAME)                                                                                         \
    static void* NAME##_for(int l64) {                                                                             \
        static void* table[7] = {nullptr,          (void*)NAME<1>, (void*)NAME<2>, (void*)NAME<3>, (void*)NAME<4>, \
                                 (void*)NAME<5>, (void*)NAME<6>};                                                  \
        return l64 >= 1 && l64 <= 6 ? table[l64] : nullptr;                                                        \
    }
CY_ENC_TABLE(k_enc_sample)
CY_ENC_TABLE(k_enc_finish)
CY_ENC_TABLE(k_add_plain)
CY_ENC_TABLE(k_lift_plain)

static cy_status launch_enc(void* func, const char* name, const EncConsts& C, long long total, cudaStream_t st,
                            void** args) {
    const int tr = trace_begin(name, C.logn, st);
    const cudaError_t e = cudaLaunchKernel(func, dim3((unsigned)((total + 255) / 256)), dim3(256), args, 0, st);
    trace_end(tr, st);
    return e == cudaSuccess ? CY_OK : cuda_error(e, name);
}

}  // namespace cy

using namespace cy;

namespace {

cy_status plain_consts(cy_yashe* y, EncConsts& C) {
    cy_ring* r = y->ring;
    int cur = -1;
    CY_CUDA(cudaGetDevice(&cur));
    if (cur != r->device) return set_error(CY_ERR_INVALID_ARGUMENT, "handle belongs to another CUDA device");
    if (r->l64 > 6) return set_error(CY_ERR_UNSUPPORTED, "plaintext operations support q of up to 384 bits");
    C = EncConsts{};
    r->q.to_limbs64(C.q, r->l64);
    (r->q / BigUInt(y->t)).to_limbs64(C.delta, r->l64);
    C.t = (uint32_t)y->t;
    C.l64 = r->l64;
    C.logn = r->logn;
    return CY_OK;
}

cy_status plain_args(cy_yashe* y, const void* a, const void* b, const void* out, int batch) {
    if (!y) return set_error(CY_ERR_INVALID_ARGUMENT, "yashe handle is NULL");
    if (batch < 0 || (batch > 0 && (!a || !b || !out))) return set_error(CY_ERR_INVALID_ARGUMENT, "bad argument");
    for (const void* p : {a, out})
        if (((uintptr_t)p & 15) != 0) return set_error(CY_ERR_INVALID_ARGUMENT, "buffer not 16-byte aligned");
    return CY_OK;
}

}  // namespace

extern "C" cy_status cy_yashe_add_plain(cy_yashe* y, const uint64_t* d_c, const uint64_t* d_m, uint64_t* d_out,
                                        int batch, cy_stream_t stream) {
    CY_TRY(plain_args(y, d_c, d_m, d_out, batch));
    if (batch == 0) return CY_OK;
    EncConsts C;
    CY_TRY(plain_consts(y, C));
    const long long total = (long long)batch << C.logn;
    cudaStream_t st = (cudaStream_t)stream;
    void* args[] = {(void*)&C, (void*)&d_m, (void*)&d_c, (void*)&d_out, (void*)&batch};
    return launch_enc(k_add_plain_for(C.l64), "add_plain", C, total, st, args);
}

extern "C" cy_status cy_yashe_mul_plain(cy_yashe* y, const uint64_t* d_c, const uint64_t* d_m, uint64_t* d_out,
                                        int batch, cy_stream_t stream) {
    CY_TRY(plain_args(y, d_c, d_m, d_out, batch));
    if (batch == 0) return CY_OK;
    if (d_out == d_c) return set_error(CY_ERR_INVALID_ARGUMENT, "out must not alias the ciphertext");
    EncConsts C;
    CY_TRY(plain_consts(y, C));
    cy_ring* r = y->ring;
    std::lock_guard<std::mutex> lock(r->mu);
    const long long total = (long long)batch << C.logn;
    cudaStream_t st = (cudaStream_t)stream;
    void* args[] = {(void*)&C, (void*)&d_m, (void*)&d_out, (void*)&batch};
    CY_TRY(launch_enc(k_lift_plain_for(C.l64), "lift_plain", C, total, st, args));
    const long long stride = (long long)r->n * r->l64;
    return run_product_api(r->mul, false, d_c, stride, d_out, stride, d_out, stride, batch, r->own_ws.ws, st);
}

extern "C" cy_status cy_gaussian_cdt(double sigma, uint64_t* out, int max_entries, int* n_entries) {
    if (!(sigma > 0.0) || !n_entries || max_entries < 0 || (max_entries > 0 && !out))
        return set_error(CY_ERR_INVALID_ARGUMENT, "bad argument");
    const std::vector<uint64_t> T = gaussian_cdt(sigma);
    *n_entries = (int)T.size();
    if ((int)T.size() > max_entries) return set_error(CY_ERR_INVALID_ARGUMENT, "table does not fit");
    std::copy(T.begin(), T.end(), out);
    return CY_OK;
}

extern "C" cy_status cy_yashe_encrypt(cy_yashe* y, const uint64_t* d_m, uint64_t* d_ct, int batch, uint64_t seed,
                                      cy_stream_t stream) {
    if (!y) return set_error(CY_ERR_INVALID_ARGUMENT, "yashe handle is NULL");
    if (batch < 0 || (batch > 0 && (!d_m || !d_ct))) return set_error(CY_ERR_INVALID_ARGUMENT, "bad argument");
    if (!y->has_keys || !y->d_h) return set_error(CY_ERR_NO_KEYS, "no keys installed");
    if (batch == 0) return CY_OK;
    if (((uintptr_t)d_ct & 15) != 0) return set_error(CY_ERR_INVALID_ARGUMENT, "ciphertext buffer not 16-byte aligned");
    cy_ring* r = y->ring;
    int cur = -1;
    CY_CUDA(cudaGetDevice(&cur));
    if (cur != r->device) return set_error(CY_ERR_INVALID_ARGUMENT, "handle belongs to another CUDA device");
    if (r->l64 > 6) return set_error(CY_ERR_UNSUPPORTED, "GPU encryption supports q of up to 384 bits");
    cudaStream_t st = (cudaStream_t)stream;
    std::lock_guard<std::mutex> lock(r->mu);
    if (!y->d_cdt) {
        const std::vector<uint64_t> T = gaussian_cdt(y->sigma);
        if ((int)T.size() > kCdtMax) return set_error(CY_ERR_UNSUPPORTED, "sigma too large for the sampler table");
        CY_CUDA(cudaMalloc(&y->d_cdt, T.size() * sizeof(uint64_t)));
        CY_CUDA(cudaMemcpy(y->d_cdt, T.data(), T.size() * sizeof(uint64_t), cudaMemcpyHostToDevice));
        y->n_cdt = (int)T.size();
    }
    EncConsts C{};
    r->q.to_limbs64(C.q, r->l64);
    (r->q / BigUInt(y->t)).to_limbs64(C.delta, r->l64);
    C.seed = seed;
    C.t = (uint32_t)y->t;
    C.l64 = r->l64;
    C.logn = r->logn;
    C.bound = (y->n_cdt - 1) / 2;
    C.ncdt = y->n_cdt;
    const long long total = (long long)batch << r->logn;
    void* sargs[] = {(void*)&C, (void*)&y->d_cdt, (void*)&d_ct, (void*)&batch};
    const long long stride = (long long)r->n * r->l64;
    // The product with s runs in the keyswitch basis, which is wide enough for it and has fewer
    // primes than the product's (six instead of nine at 127-bit q); N < 1024 takes the ordinary one.
    const bool small = y->d_h_key != nullptr;
    CY_TRY(launch_enc(small ? (void*)k_enc_sample_small : k_enc_sample_for(C.l64), "enc_sample", C, total, st, sargs));
    CY_TRY(run_product_api(small ? y->relin : r->mul, false, y->d_h, 0, d_ct, stride, d_ct, stride, batch, r->own_ws.ws, st,
                           -1, y->d_h_key, small));
    void* fargs[] = {(void*)&C, (void*)&y->d_cdt, (void*)&d_m, (void*)&d_ct, (void*)&batch};
    return launch_enc(k_enc_finish_for(C.l64), "enc_finish", C, total, st, fargs);
}
