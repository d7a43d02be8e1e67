// Launchers of the thread-per-state kernels (pjg_wave.cuh), two of their forms,
// and the species thermo kernel.
#include <cuda_runtime.h>

#include "pjg_eval.cuh"
#include "pjg_math.cuh"
#include "pjg_wave.cuh"

using namespace pjg;

PJG_WAVE_INSTANCE(KIND_RATES, PJG_RATES_MINB)
PJG_WAVE_INSTANCE(KIND_VJP, PJG_VJP_MINB)

thread_local cudaError_t pjg_launch_err = cudaSuccess;
const char* pjg_launch_error_string() { return cudaGetErrorString(pjg_launch_err); }

namespace {

constexpr int kChemBlock = 128;

// Species thermo of the chem_utils kernel type (rate_subs.py write_chem_utils
// :3391-3444, polyfit_kernel_gen :3281-3388): at the guarded temperature,
// cp (cv), h (u) and the Gibbs function b of every species.  Entry (s, k) of
// each output at out[s * out_ss + k * out_sk].
__global__ void __launch_bounds__(kChemBlock) chem_utils_kernel(const double* __restrict__ sp, int ns,
                                                               int64_t n, int conp,
                                                               const double* __restrict__ phi,
                                                               int64_t phi_ss, double* cp, double* h,
                                                               double* b, int64_t out_ss,
                                                               int64_t out_sk)
{
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const double Tc = fmin(10000.0, fmax(100.0, phi[s * phi_ss]));
    const double logT = log(Tc), Tinv = 1.0 / Tc;
    for (int k = 0; k < ns; ++k) {
        const Thermo t = thermo<false>(sp + (int64_t)k * PJG_SP_DOUBLES, Tc, logT, Tinv, conp);
        const int64_t o = s * out_ss + (int64_t)k * out_sk;
        cp[o] = t.cp;
        h[o] = t.h;
        b[o] = t.b;
    }
}

}  // namespace

int pjg_launch_chem_utils(const double* sp, int ns, int64_t n, int conp, const double* phi,
                          int64_t phi_ss, double* cp, double* h, double* b, int64_t out_ss,
                          int64_t out_sk, void* stream)
{
    if (n <= 0) return 0;
    chem_utils_kernel<<<(unsigned)((n + kChemBlock - 1) / kChemBlock), kChemBlock, 0, (cudaStream_t)stream>>>(
        sp, ns, n, conp, phi, phi_ss, cp, h, b, out_ss, out_sk);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

namespace {

const void* wave_of(int kind, bool large)
{
    return kind == KIND_JAC ? (large ? wave_fn<KIND_JAC, kLargeBlocks>() : wave_fn<KIND_JAC, PJG_JAC_MINB>())
           : kind == KIND_VJP ? wave_fn<KIND_VJP, PJG_VJP_MINB>() : wave_fn<KIND_RATES, PJG_RATES_MINB>();
}

}  // namespace

int pjg_wave_blocks_per_sm(int kind, bool large)
{
    int b = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, wave_of(kind, large), PJG_BLOCK, 0);
    return e == cudaSuccess && b > 0 ? b : 1;
}

int pjg_launch_wave(const EvalArgs& a, int kind, int sms, bool large, void* stream)
{
    if (a.n <= 0) return 0;
    const cudaStream_t st = (cudaStream_t)stream;
    const unsigned grid = (unsigned)((a.n + PJG_BLOCK - 1) / PJG_BLOCK);
    if (kind == KIND_VJP) wave_launch<KIND_VJP, PJG_VJP_MINB>(a, grid, st);
    else if (kind == KIND_RATES) wave_launch<KIND_RATES, PJG_RATES_MINB>(a, grid, st);
    else if (grid <= (unsigned)(kFewBlocks * sms)) wave_launch<KIND_JAC, kFewBlocks>(a, grid, st);
    else if (large && (grid <= (unsigned)(kLargeBlocks * sms) || grid > (unsigned)(PJG_JAC_MINB * sms)))
        wave_launch<KIND_JAC, kLargeBlocks>(a, grid, st);
    else wave_launch<KIND_JAC, PJG_JAC_MINB>(a, grid, st);
    pjg_launch_err = cudaGetLastError();
    return pjg_launch_err == cudaSuccess ? 0 : -2;
}
