// dispatch.h -- table of kernel instantiations per transform length.
#pragma once

#include <stddef.h>

#include "common.h"

namespace cy {

// [l64][...]: index 0 holds the generic kernels (limb count read at run time),
// index L64 the kernels specialised for coefficients of L64 limbs (or null).
struct KernelSet {
    int logn = 0, loge = 0, threads = 0;
    void* mul[7][2] = {};  // [l64][centered]
    void* ks[7][2] = {};   // [l64][keyswitch with ND_LO (2 or 1) / ND_HI (4 or 2) digits per pass]
    void* ntt[2] = {nullptr, nullptr};  // forward / inverse
    size_t smem_mul = 0, smem_ks[2] = {0, 0}, smem_ntt = 0;
    int blocks_per_prime = 1;  // product / keyswitch blocks per (prime, job): 2 for block pairs
    int ntt_jobs_per_block = 2;  // k_ntt: two jobs per block, grid (primes, jobs/2); k_ntt1: one, grid (jobs, primes)
    // equal for sets that run an operation with the same code (compiled with each set, so that the
    // pointers differ): coefficients per thread, blocks per SM, digits per pass
    int mul_id = 0, ks_id = 0, ntt_id = 0;
    bool intt_tma = false;  // N = 4096: the standalone inverse NTT takes its input tile by TMA (k_intt_tma)
    void* mul_for(int l64, bool centered) const { return mul[mul[l64][0] ? l64 : 0][centered ? 1 : 0]; }
    void* ks_for(int l64, int nd4) const { return ks[ks[l64][0] ? l64 : 0][nd4]; }
};

// Kernel sets for transforms of length 2^logn (1 <= logn <= LOGN_MAX). Each
// length has one or more schedules ("variants": coefficients per thread, hence
// threads per transform and passes). Set v is schedule number v for v > 0, and number 0 is the
// default rule (tuning.cpp), so set 0 has a second number.
int variant_count(int logn);
const KernelSet& kernel_variant(int logn, int v);

// Products with a kept operand (k_mul_key) for N = 2^logn >= 1024 and l64 limbs (0: the other
// operand is small).
struct KeyKernel {
    void* func;
    int threads;
    size_t smem;
};
const KeyKernel* key_kernel(int logn, int l64);

// Tuned operations (keys of the autotuner's table).
enum TuneOp { TUNE_MUL = 0, TUNE_MULC = 1, TUNE_KS = 2, TUNE_NTT = 3, TUNE_OPS = 4 };

// ICRT epilogue for `l32` words of q and epilogue mode (EpiMode) with its constants
// in shared memory (for comparison: cy_set_epilogue_generic).
void* epi_kernel(int l32, int mode);

// Epilogue with the constants of its basis as the first parameter, by value
// (k_epi_c): the kernel, that parameter's size and the function that writes it. The
// common parameter sets have one compiled for their prime count.
struct EpiConstKernel {
    void* func;
    size_t param_bytes;
    void (*fill)(const BasisDev& h, void* param);
    void* any_x;  // the kernel for residues of any X (cy_icrt; null where the one for any prime count serves)
};
const EpiConstKernel* epi_const(int l32, int k, int mode);
const EpiConstKernel* epi_const_any(int l32, int mode);  // for any prime count

}  // namespace cy
