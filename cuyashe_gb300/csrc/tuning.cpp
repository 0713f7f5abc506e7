// tuning.cpp -- choice of NTT schedule per (device, N, limb count, operation).
//
// Every transform length has one or more compiled schedules (kernel variants:
// 8 to 64 coefficients per thread, hence 512 to 64 threads per transform and
// 4 to 2 register passes at N = 4096). The autotuner runs each schedule of an
// operation on a synthetic batch of the caller's ring, checks that its output is
// bit-identical to the default schedule's, times it with CUDA events and keeps
// the fastest, for calls of the same regime (the default rule depends on the call's size). Choices live
// in a process-wide table and can be exported and
// imported as text ("n4096.l2.mul=1@8;n4096.l2.ks=0;...": 0 for the default, @8 for calls whose default is
// schedule 8) so that a serving process tunes once. The reference has a single fixed launch shape per kernel
// (e.g. src/cuda_functions.cu:447-458) and commented-out block-size notes
// (src/cuda_bn.cu:983-988, 1014-1019).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <sstream>
#include <string>
#include <tuple>
#include <vector>

#include "host.h"

namespace cy {

cy_status run_product_api(const Basis& B, bool centered, const uint64_t* a, long long a_stride, const uint64_t* b,
                          long long b_stride, void* out, long long out_stride, int batch, Workspace& ws,
                          cudaStream_t st, int variant, const uint32_t* key = nullptr, bool small = false);
cy_status run_keyswitch_api(const Basis& B, const uint64_t* c, const uint32_t* evk, int ell, uint64_t* out, int batch,
                            Workspace& ws, cudaStream_t st, int variant, int chunk_k, int lm);
size_t evk_words(const Basis& relin, int ell);
cy_status prepare_evk(const Basis& relin, const uint64_t* d_h, const uint64_t* d_limbs, int ell, uint32_t* d_res,
                      uint32_t* d_evk);

cy_status run_ntt_api(const Basis& B, uint32_t* res, int batch, bool inverse, cudaStream_t st, int variant);
cy_status run_yashe_mul(const Basis& tensor, const Basis& relin, const uint32_t* evk, int ell, const uint64_t* c1,
                        const uint64_t* c2, uint64_t* out, int batch, bool do_relin, Workspace& ws, cudaStream_t st,
                        int ks_variant);

static const char* kOpNames[TUNE_OPS] = {"mul", "mulc", "ks", "ntt"};

static std::mutex g_mu;
// (device, logn, l64, op, rule) -> schedule number. A choice that was measured holds where the default
// rule takes the same kernel set `rule` as at the measured size: another regime (a single call after a batch
// was tuned) keeps its default. With 16384 x 380 bits tuned on a batch, a single product takes 27 us, 40 with
// the batch's schedule. rule = -1: for all sizes (an import that names no rule).
static std::map<std::tuple<int, int, int, int, int>, int> g_choice;

// SMs of the current device (the GB300's 152 if it cannot be queried).
static int sm_count() {
    static std::atomic<int> known[64];
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
    sms = known[dev].load(std::memory_order_relaxed);
    if (sms > 0) return sms;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) sms = 152;
    known[dev].store(sms, std::memory_order_relaxed);
    return sms;
}

// The schedule of a call that the autotuner has not chosen one for: `blocks` transforms'
// blocks per launch (jobs times primes). Two regimes: up to one block per SM the time is one
// block's latency (more threads per transform, or a pair of blocks); above, throughput. The
// lines, measured with every schedule at q of 60 to 380 bits: [jobs, bits of q] us per call with the
// schedule taken : with the other one.
//   N = 1024   8 coefficients per thread (keyswitch [512, 380] 213 : 505 with 16, [512, 62] 17.1 : 17.8), but
//              16 for products from two blocks per SM on ([2048, 127] 132 : 146, [512, 380] 157 : 203, [64,
//              127] 8.3 : 8.8; at the line [34, 127] 7.5 : 7.0) and transforms from four on ([2048, 127] 33 :
//              38; below it [64, 127] 4.4 : 4.7)
//   N = 2048   products 16 per thread ([512, 250] 179 : 214; [1, 250] 9.0 : 8.8), transforms 8 below four
//              blocks per SM ([8, 127] 4.9 : 5.9), 16 from there on ([2048, 127] 66 : 83); keyswitch 8
//              ([512, 250] 225 : 445)
//   N = 4096   16 per thread, products and transforms at three blocks per SM ([2048, 127] 566 : 622 and 138 :
//              171 with 8; between two and four blocks per SM four fit better, [64, 127] 24.8 : 22.6).
//              Keyswitch: two blocks of 128 registers ([2048, 127] 560 : 605 with 8); up to one block per SM
//              8 per thread with the full register file (three limbs [1, 190] 12.9 : 14.7, five [1, 320] 20.5
//              : 24.4; even digit counts are within 3% either way, [1, 127] 10.5 : 10.2)
//   N = 8192   16 per thread at 64 registers ([512, 190] 585 : 711 with 8), keyswitches of two
//              limbs or more 128 registers ([37, 190] 54.7 : 58.0; [64, 380] 300 : 353)
//   N = 16384  a pair of blocks per transform while that is one block per SM at most ([1, 380] product 26 :
//              37, [15, 62] 19.5 : 23.8; above it [16, 62] 24.0 : 35.7; keyswitch [5, 380] 73 : 106, above it
//              [8, 250] 73 : 96). Above: keyswitch 32 per thread ([64, 62] 46 : 50, [256, 380] 2690 : 2800);
//              products of five limbs or more too ([64, 300] 369 : 380, [256, 380] 1686 : 1822), those of
//              fewer 16 ([64, 250] 236 : 246), and centred ones always ([64, 300] 359 : 374, [64, 380] 420 :
//              463; inside the multiply of 256 pairs 4052 : 4177); all else 16
int default_variant(int logn, int l64, int op, long long blocks) {
    const int sms = sm_count();
    const bool small = blocks <= sms;
    const bool product = op == TUNE_MUL || op == TUNE_MULC;
    switch (logn) {
        case 10: return (product && blocks >= 2 * sms) || (op == TUNE_NTT && blocks >= 4 * sms) ? 1 : 0;
        case 11: return product || (op == TUNE_NTT && blocks >= 4 * sms) ? 1 : 0;
        case 12: return op == TUNE_KS ? (small ? 2 : 3) : 8;
        case 13: return op == TUNE_KS && l64 > 1 ? 2 : 0;
        case 14:
            if (op != TUNE_NTT && 2 * blocks <= sms) return 3;
            return op == TUNE_KS || (op == TUNE_MUL && l64 >= 5) ? 1 : 0;
        default: return 0;
    }
}

// The kernel set of schedule `number`: 0 is the default rule for a call of `blocks`, and a negative
// number the autotuner's (or an imported) choice, the default where there is none.
int tuned_variant(int logn, int l64, int op, long long blocks, int number) {
    const int rule = default_variant(logn, l64, op, blocks);
    int dev = 0;
    if (number < 0 && cudaGetDevice(&dev) == cudaSuccess) {
        std::lock_guard<std::mutex> lock(g_mu);
        auto it = g_choice.find(std::make_tuple(dev, logn, l64, op, rule));
        if (it == g_choice.end()) it = g_choice.find(std::make_tuple(dev, logn, l64, op, -1));
        if (it != g_choice.end()) number = it->second;
    }
    return number > 0 ? number : rule;
}

// A schedule number that always runs kernel set v.
static int number_of(int logn, int v) {
    if (v > 0) return v;
    switch (logn) {  // set 0's second number (k_misc.cu)
        case 10: return 2;
        case 11: return 2;
        case 12: return 5;
        case 13: return 3;
        case 14: return 4;
        default: return 0;
    }
}

static void set_choice(int dev, int logn, int l64, int op, int rule, int number) {
    std::lock_guard<std::mutex> lock(g_mu);
    if (rule < 0) {  // for all sizes: nothing else stands
        auto it = g_choice.lower_bound(std::make_tuple(dev, logn, l64, op, -1));
        while (it != g_choice.end() && it->first < std::make_tuple(dev, logn, l64, op + 1, -1)) it = g_choice.erase(it);
    }
    g_choice[std::make_tuple(dev, logn, l64, op, rule)] = number;
}

// values < q: random words below the top bit of q
static std::vector<uint64_t> random_polys(int count, int n, int l64, int qbits, uint64_t seed) {
    std::vector<uint64_t> v((size_t)count * n * l64);
    uint64_t s = seed;
    for (auto& x : v) {
        s += 0x9E3779B97F4A7C15ULL;
        uint64_t z = s;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
        x = z ^ (z >> 31);
    }
    const int top = (qbits - 2) % 64 + 1;  // bits kept in the top limb: value < 2^(qbits-1) <= q
    const int toplimb = (qbits - 2) / 64;
    for (size_t i = 0; i < v.size(); i += l64) {
        for (int j = toplimb + 1; j < l64; j++) v[i + j] = 0;
        if (top < 64) v[i + toplimb] &= (1ull << top) - 1;
    }
    return v;
}

struct DevBuf {
    void* p = nullptr;
    ~DevBuf() {
        if (p) cudaFree(p);
    }
};

// Whether two kernel sets run an operation alike.
static bool same_kernels(const KernelSet& a, const KernelSet& b, int op) {
    if (op == TUNE_NTT) return a.ntt_id == b.ntt_id && a.intt_tma == b.intt_tma;
    return op == TUNE_KS ? a.ks_id == b.ks_id : a.mul_id == b.mul_id;
}

// Whether schedule number v runs kernels of its own: not those of the default or of an earlier number.
static bool distinct(int logn, int op, int rule, int v) {
    const KernelSet& ks = kernel_variant(logn, v);
    if (v > 0 && same_kernels(ks, kernel_variant(logn, rule), op)) return false;
    for (int u = 1; u < v; u++)
        if (same_kernels(ks, kernel_variant(logn, u), op)) return false;
    return true;
}

// Time each schedule of one operation at `blocks` transforms per launch; `run(v, out)` launches it on `st`.
template <class Run>
static cy_status tune_op(int logn, int l64, int op, long long blocks, size_t out_bytes, cudaStream_t st, Run run) {
    const int nv = variant_count(logn);
    int dev = 0;
    CY_CUDA(cudaGetDevice(&dev));
    const int rule = default_variant(logn, l64, op, blocks);
    if (nv <= 1) {
        set_choice(dev, logn, l64, op, rule, 0);
        return CY_OK;
    }
    DevBuf ref, cur, flag;
    CY_CUDA(cudaMalloc(&ref.p, out_bytes));
    CY_CUDA(cudaMalloc(&cur.p, out_bytes));
    CY_CUDA(cudaMalloc(&flag.p, sizeof(int)));
    cudaEvent_t e0, e1;
    CY_CUDA(cudaEventCreate(&e0));
    CY_CUDA(cudaEventCreate(&e1));
    float best = 0;
    int best_v = 0;
    cy_status st_all = CY_OK;
    for (int v = 0; v < nv && st_all == CY_OK; v++) {
        if (!distinct(logn, op, rule, v)) continue;
        void* out = v == 0 ? ref.p : cur.p;
        st_all = run(v, out);  // warm-up and the output to check
        if (st_all != CY_OK && v > 0) {
            // a schedule this device cannot launch (e.g. a block-pair cluster that
            // does not fit) is skipped; launch errors are not sticky
            cudaGetLastError();
            if (cudaStreamSynchronize(st) != cudaSuccess) break;
            st_all = CY_OK;
            continue;
        }
        if (st_all != CY_OK) break;
        if (cudaStreamSynchronize(st) != cudaSuccess) {
            st_all = set_error(CY_ERR_CUDA, "autotune warm-up failed");
            break;
        }
        if (v > 0) {  // compared on the device: large batches cost no host copies
            bool differ = false;
            st_all = words_differ(ref.p, cur.p, out_bytes, (int*)flag.p, st, &differ);
            if (st_all == CY_OK && differ)
                st_all = set_error(CY_ERR_INTERNAL, "autotune: a schedule disagrees with the default");
            if (st_all != CY_OK) break;
        }
        const int reps = 3;
        cudaEventRecord(e0, st);
        for (int r = 0; r < reps && st_all == CY_OK; r++) st_all = run(v, out);
        cudaEventRecord(e1, st);
        cudaEventSynchronize(e1);
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        if (v == 0 || ms < best) {
            best = ms;
            best_v = v;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st_all != CY_OK) return st_all;
    set_choice(dev, logn, l64, op, rule, best_v);
    return CY_OK;
}

static cy_status tune_product(const Basis& B, bool centered, int batch, cudaStream_t st) {
    const int n = B.h.n, l64 = B.h.l64;
    const size_t bytes = sizeof(uint64_t) * (size_t)batch * n * l64;
    std::vector<uint64_t> ha = random_polys(batch, n, l64, B.h.qbits, 1), hb = random_polys(batch, n, l64, B.h.qbits, 2);
    DevBuf a, b;
    CY_CUDA(cudaMalloc(&a.p, bytes));
    CY_CUDA(cudaMalloc(&b.p, bytes));
    CY_CUDA(cudaMemcpy(a.p, ha.data(), bytes, cudaMemcpyHostToDevice));
    CY_CUDA(cudaMemcpy(b.p, hb.data(), bytes, cudaMemcpyHostToDevice));
    Workspace ws;
    CY_CUDA(cudaGetDevice(&ws.device));
    const long long stride = (long long)n * l64;
    const long long ostride = B.h.mode == EPI_DECRYPT ? n : stride;
    const size_t obytes = sizeof(uint64_t) * (size_t)batch * ostride;
    const long long blocks = (long long)std::min(batch, chunk_jobs(n, B.h.k)) * B.h.k;
    return tune_op(B.h.logn, l64, centered ? TUNE_MULC : TUNE_MUL, blocks, obytes, st,
                   [&](int v, void* out) {
                       return run_product_api(B, centered, (const uint64_t*)a.p, stride, (const uint64_t*)b.p, stride,
                                              out, ostride, batch, ws, st, v);
                   });
}

// The keyswitch schedule is chosen inside the HE multiply it serves: each schedule
// runs the whole relinearised multiply of `batch` pairs (its chunks cut to whole
// waves of that schedule, its keyswitch overlapping the tensor products of the
// neighbouring chunks), with the tensor schedule already chosen. Timing the
// keyswitch alone kept a schedule 3% slower in the multiply.
static cy_status tune_keyswitch(const cy_yashe* y, const uint32_t* evk, int batch, cudaStream_t st) {
    const int n = y->ring->n, l64 = y->ring->l64;
    const size_t bytes = sizeof(uint64_t) * (size_t)batch * n * l64;
    std::vector<uint64_t> h1 = random_polys(batch, n, l64, y->ring->qbits, 3);
    std::vector<uint64_t> h2 = random_polys(batch, n, l64, y->ring->qbits, 5);
    DevBuf c1, c2;
    CY_CUDA(cudaMalloc(&c1.p, bytes));
    CY_CUDA(cudaMalloc(&c2.p, bytes));
    CY_CUDA(cudaMemcpy(c1.p, h1.data(), bytes, cudaMemcpyHostToDevice));
    CY_CUDA(cudaMemcpy(c2.p, h2.data(), bytes, cudaMemcpyHostToDevice));
    Workspace ws;
    CY_CUDA(cudaGetDevice(&ws.device));
    const long long blocks =
        (long long)std::min(batch, chunk_jobs(n, std::max(y->tensor.h.k, y->relin.h.k))) * y->relin.h.k;
    return tune_op(y->relin.h.logn, l64, TUNE_KS, blocks, bytes, st,
                   [&](int v, void* out) {
                       return run_yashe_mul(y->tensor, y->relin, evk, y->ell, (const uint64_t*)c1.p,
                                            (const uint64_t*)c2.p, (uint64_t*)out, batch, true, ws, st, v);
                   });
}

// The standalone transforms (cy_ntt) of `batch` residue vectors, inverse then
// forward (schedules may differ in either direction); each run transforms a
// fresh copy of the same input and must give it back.
static cy_status tune_ntt(const Basis& B, int batch, cudaStream_t st) {
    const size_t words = (size_t)batch * B.h.k * B.h.n;
    std::vector<uint32_t> h(words);
    uint64_t s = 5;
    for (size_t i = 0; i < words; i++) {
        s = s * 6364136223846793005ULL + 1442695040888963407ULL;
        h[i] = (uint32_t)((s >> 33) % B.h.p[(i / B.h.n) % B.h.k]);
    }
    DevBuf src;
    CY_CUDA(cudaMalloc(&src.p, words * sizeof(uint32_t)));
    CY_CUDA(cudaMemcpy(src.p, h.data(), words * sizeof(uint32_t), cudaMemcpyHostToDevice));
    return tune_op(B.h.logn, B.h.l64, TUNE_NTT, (long long)batch * B.h.k, words * sizeof(uint32_t), st,
                   [&](int v, void* out) {
                       cudaError_t e = cudaMemcpyAsync(out, src.p, words * sizeof(uint32_t),
                                                       cudaMemcpyDeviceToDevice, st);
                       if (e != cudaSuccess) return cuda_error(e, "autotune copy");
                       CY_TRY(run_ntt_api(B, (uint32_t*)out, batch, true, st, v));
                       return run_ntt_api(B, (uint32_t*)out, batch, false, st, v);
                   });
}

}  // namespace cy

using namespace cy;

extern "C" {

cy_status cy_ring_autotune(cy_ring* r, int batch, cy_stream_t stream) {
    if (!r || batch < 1) return set_error(CY_ERR_INVALID_ARGUMENT, "bad argument");
    std::lock_guard<std::mutex> lock(r->mu);
    CY_TRY(tune_product(r->mul, false, batch, (cudaStream_t)stream));
    return tune_ntt(r->plain, batch, (cudaStream_t)stream);
}

cy_status cy_yashe_autotune(cy_yashe* y, int batch, cy_stream_t stream) {
    if (!y || batch < 1) return set_error(CY_ERR_INVALID_ARGUMENT, "bad argument");
    cy_ring* r = y->ring;
    std::lock_guard<std::mutex> lock(r->mu);
    cudaStream_t st = (cudaStream_t)stream;
    CY_TRY(tune_product(r->mul, false, batch, st));
    CY_TRY(tune_product(y->tensor, true, batch, st));
    const uint32_t* evk = y->d_evk;
    DevBuf tmp, limbs, res;
    if (!y->has_keys) {  // an evaluation key of random values has the same cost
        std::vector<uint64_t> h = random_polys(y->ell, r->n, r->l64, r->qbits, 4);
        CY_CUDA(cudaMalloc(&limbs.p, h.size() * sizeof(uint64_t)));
        CY_CUDA(cudaMalloc(&res.p, (size_t)y->ell * y->relin.h.k * r->n * sizeof(uint32_t)));
        CY_CUDA(cudaMalloc(&tmp.p, evk_words(y->relin, y->ell) * sizeof(uint32_t)));
        CY_CUDA(cudaMemcpy(limbs.p, h.data(), h.size() * sizeof(uint64_t), cudaMemcpyHostToDevice));
        CY_TRY(prepare_evk(y->relin, nullptr, (const uint64_t*)limbs.p, y->ell, (uint32_t*)res.p, (uint32_t*)tmp.p));
        CY_CUDA(cudaDeviceSynchronize());
        evk = static_cast<const uint32_t*>(tmp.p);
    }
    return tune_keyswitch(y, evk, batch, st);
}

cy_status cy_tuning_export(char* buf, size_t len, size_t* needed) {
    int dev = 0;
    CY_CUDA(cudaGetDevice(&dev));
    std::ostringstream os;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        for (const auto& kv : g_choice) {
            if (std::get<0>(kv.first) != dev) continue;
            os << "n" << (1 << std::get<1>(kv.first)) << ".l" << std::get<2>(kv.first) << "."
               << kOpNames[std::get<3>(kv.first)] << "=" << kv.second;
            if (std::get<4>(kv.first) >= 0) os << "@" << number_of(std::get<1>(kv.first), std::get<4>(kv.first));
            os << ";";
        }
    }
    const std::string s = os.str();
    if (needed) *needed = s.size() + 1;
    if (buf && len > 0) {
        std::strncpy(buf, s.c_str(), len - 1);
        buf[len - 1] = 0;
        if (len < s.size() + 1) return set_error(CY_ERR_INVALID_ARGUMENT, "buffer too small");
    }
    return CY_OK;
}

cy_status cy_tuning_schedule(int n, int q_limbs, const char* op, long long blocks, int* schedule) {
    if (!op || !schedule || blocks < 0) return set_error(CY_ERR_INVALID_ARGUMENT, "bad argument");
    int logn = 0;
    while (logn < LOGN_MAX && (1 << logn) < n) logn++;
    int o = -1;
    for (int i = 0; i < TUNE_OPS; i++)
        if (std::strcmp(op, kOpNames[i]) == 0) o = i;
    if ((1 << logn) != n || logn < 1 || o < 0 || q_limbs < 1 || q_limbs > 6)
        return set_error(CY_ERR_INVALID_ARGUMENT, "no such operation");
    int dev = 0;
    CY_CUDA(cudaGetDevice(&dev));
    *schedule = number_of(logn, tuned_variant(logn, q_limbs, o, blocks, -1));
    return CY_OK;
}

cy_status cy_tuning_import(const char* spec) {
    if (!spec) return set_error(CY_ERR_INVALID_ARGUMENT, "NULL spec");
    int dev = 0;
    CY_CUDA(cudaGetDevice(&dev));
    std::string s(spec);
    size_t pos = 0;
    while (pos < s.size()) {
        size_t end = s.find(';', pos);
        if (end == std::string::npos) end = s.size();
        const std::string item = s.substr(pos, end - pos);
        pos = end + 1;
        if (item.empty()) continue;
        int n = 0, l64 = 0, v = 0, where = 0;
        char op[8] = {0};
        const int fields = std::sscanf(item.c_str(), "n%d.l%d.%7[a-z]=%d@%d", &n, &l64, op, &v, &where);
        if (fields < 4)
            return set_error(CY_ERR_INVALID_ARGUMENT, "bad tuning item: " + item);
        int logn = 0;
        while ((1 << logn) < n) logn++;
        int o = -1;
        for (int i = 0; i < TUNE_OPS; i++)
            if (std::strcmp(op, kOpNames[i]) == 0) o = i;
        if ((1 << logn) != n || logn < 1 || logn > LOGN_MAX || o < 0 || v < 0 || v >= variant_count(logn) ||
            l64 < 1 || l64 > 6 || where < 0 || where >= variant_count(logn))
            return set_error(CY_ERR_INVALID_ARGUMENT, "bad tuning item: " + item);
        const int rule = fields < 5 ? -1 : where == number_of(logn, 0) ? 0 : where;
        set_choice(dev, logn, l64, o, rule, v);
    }
    return CY_OK;
}

}  // extern "C"
