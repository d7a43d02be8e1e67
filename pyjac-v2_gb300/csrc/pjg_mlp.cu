// BF16 tensor-core (tcgen05) GEMM kernels for the learned species-rate
// surrogate: an MLP whose layers are Y = act(X W^T + b) with BF16 weights and
// activations and FP32 accumulation in tensor memory.
//
// Two kernels cover forward, input-gradient (dgrad) and weight-gradient
// (wgrad) passes; both multiply K-major operands staged in shared memory in the
// no-swizzle core-matrix layout (8 rows x 16 bytes per core matrix), with one
// elected thread issuing tcgen05.mma and completion signalled through an
// mbarrier:
//
// * umma_rows_kernel: C[M x N] = A[M x K] . B[N x K]^T for a tall A (M = states)
//   and a small resident B (weights, N, K <= 256).  Persistent over 128-row tiles
//   of A; the epilogue reads the accumulator with tcgen05.ld and fuses bias,
//   SiLU, SiLU' (for dgrad), BF16 conversion, a transposed copy (the K-major
//   operand of the next wgrad) and column sums (bias gradients).
// * umma_wgrad_kernel: C[Mo x No] += A[Mo x Kb] . B[No x Kb]^T with the long
//   reduction over states split across CTAs; FP32 partial results are added to
//   the output with atomics.
//
// Waits on mbarriers are bounded; on timeout the kernel records an error
// (pjg_mlp_status) and finishes without hanging.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "pjg_umma.cuh"

namespace {

__device__ int g_umma_err = 0;

using bf16 = __nv_bfloat16;

struct RowsArgs {
    const bf16* A;
    int64_t lda;
    const bf16* B;
    int64_t ldb;
    int64_t M;
    int N, K;
    const float* bias;
    int act;           // 1: SiLU
    const bf16* zp;    // dgrad: multiply by SiLU'(zp)
    int64_t ldzp;
    int zvec;          // zp's rows start on 16-byte boundaries
    bf16* Y;
    int64_t ldy;
    bf16* YT;          // transposed copy YT[n * ldyt + m]
    int64_t ldyt;
    int ytvec;         // pairs of YT's columns start on 4-byte boundaries
    bf16* Z;           // pre-activation copy
    int64_t ldz;
    float* Y32;        // FP32 output
    int64_t ldy32;
    float* colsum;     // += column sums of the output
    int NT;            // columns of one CTA (N, or its half)
    int stages;        // tiles of A in shared memory
};

// logistic sigmoid with the fast division intrinsic (2 ulp in FP32; results are
// rounded to BF16), shared by every kernel so that training and inference
// evaluate SiLU identically
// sigmoid(x) = (1 + tanh(x / 2)) / 2 with the hardware tanh (tanh.approx.f32,
// relative error about 2^-11, below the BF16 rounding the activations take):
// one special-function operation instead of an exponential and a reciprocal,
// which bound the epilogues (16 special-function results per clock per SM)
__device__ __forceinline__ float tanh_approx(float x)
{
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float sigmoidf_(float x) { return fmaf(0.5f, tanh_approx(0.5f * x), 0.5f); }

// One CTA keeps a slice of NT columns of B in shared memory (all of them, or a
// half where that lets two tiles of A fit beside it) and walks the 128-row
// tiles of A.  Two stages: while the tensor core multiplies tile i, the 16 warps
// read tile i - 1's accumulator (two TMEM buffers) and write its outputs, and
// tile i + 1 is copied into the stage that tile i - 1 left.  Bound by the
// outputs' bytes; with one stage, four warps and element-wise reads of zp (2
// bytes per lane and row) it was bound by latency.  49,152 rows, K = N = 256, on
// GB300: forward with Y, Z, Y^T 87 -> 38 us (48 with 8 warps and a row per
// lane), input gradient with Y, Y^T and column sums 268 -> 48 us (53).  L2 and
// L1 run at 30 to 40 % of their rates; what is left is latency between barriers.
constexpr int kRowsThreads = 512, kRowsParts = kRowsThreads / 128;

// Lane p of a quad holds r[0..3]; afterwards r[q] is what lane q held in r[p].
// The epilogues read and write a row's 64 bytes with the four lanes of a quad
// (8 rows per instruction, whole sectors) instead of one lane (32 rows).
__device__ __forceinline__ void quad_transpose(uint4 (&r)[4], int lane)
{
    auto swap = [&](uint4& lo, uint4& hi, bool up, int h) {
        const uint4 send = up ? lo : hi;
        uint4 recv;
        recv.x = __shfl_xor_sync(0xffffffffu, send.x, h);
        recv.y = __shfl_xor_sync(0xffffffffu, send.y, h);
        recv.z = __shfl_xor_sync(0xffffffffu, send.z, h);
        recv.w = __shfl_xor_sync(0xffffffffu, send.w, h);
        if (up) lo = recv;
        else hi = recv;
    };
    swap(r[0], r[2], lane & 2, 2);
    swap(r[1], r[3], lane & 2, 2);
    swap(r[0], r[1], lane & 1, 1);
    swap(r[2], r[3], lane & 1, 1);
}

// rows m0 .. m0 + 31 (one per lane, 64 bytes of each in r) to base + row * ld bytes
__device__ __forceinline__ void store_rows64(uint8_t* base, int64_t ld, int64_t m0, int64_t M, uint4 (&r)[4], int lane)
{
    quad_transpose(r, lane);
    const int64_t row = m0 + (lane & ~3);
    uint8_t* d = base + row * ld + (lane & 3) * 16;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (row + q < M) *reinterpret_cast<uint4*>(d + q * ld) = r[q];
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b)
{
    const uint32_t lo = __bfloat16_as_ushort(__float2bfloat16(a));
    const uint32_t hi = __bfloat16_as_ushort(__float2bfloat16(b));
    return lo | (hi << 16);
}

template <bool ZP>
__global__ void __launch_bounds__(kRowsThreads, 1) umma_rows_kernel(const RowsArgs g)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar[2];
    __shared__ uint32_t tmem_s;
    __shared__ __align__(16) float sbias[256];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kc = g.K >> 3;  // 16-byte chunks per row
    const int NT = g.NT, halves = g.N / NT, n0 = (int)(blockIdx.x % halves) * NT;
    uint8_t* sB = smem;
    uint8_t* sA = smem + (size_t)NT * g.K * 2;
    const uint32_t stage_bytes = 128u * g.K * 2, stages = g.stages;
    uint32_t ncols = 64;  // two accumulators
    while (ncols < 2u * NT) ncols *= 2;
    const uint32_t acc = ncols / 2;
    if (warp == 0) {
        umma::tmem_alloc(&tmem_s, ncols);
        umma::tmem_relinquish();
    }
    if (tid == 0) {
        umma::mbar_init(&mbar[0], 1);
        umma::mbar_init(&mbar[1], 1);
    }
    if (g.bias)
        for (int j = tid; j < NT; j += kRowsThreads) sbias[j] = g.bias[n0 + j];
    const int lr = tid / kc, lc = tid % kc, dr = kRowsThreads / kc, dc = kRowsThreads % kc;
    for (int idx = tid; idx < NT * kc; idx += kRowsThreads) {
        const int n = idx / kc, c = idx - n * kc;
        umma::cp_async16(sB + ((size_t)(n >> 3) * kc + c) * 128 + (n & 7) * 16,
                         g.B + (int64_t)(n0 + n) * g.ldb + c * 8, 16);
    }
    auto load_a = [&](int64_t t, uint32_t stage) {
        const int64_t row0 = t * 128;
        uint8_t* dst = sA + stage * stage_bytes;
        for (int r = lr, c = lc; r < 128;) {
            const int64_t grow = row0 + r;
            const bool ok = grow < g.M;
            umma::cp_async16(dst + ((size_t)(r >> 3) * kc + c) * 128 + (r & 7) * 16,
                             g.A + (ok ? grow : 0) * g.lda + c * 8, ok ? 16u : 0u);
            r += dr;
            c += dc;
            if (c >= kc) {
                c -= kc;
                ++r;
            }
        }
    };
    const int64_t ntiles = (g.M + 127) / 128, step = gridDim.x / halves, t0 = blockIdx.x / halves;
    if (t0 < ntiles) load_a(t0, 0);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = tmem_s;
    const uint32_t idesc = umma::idesc_bf16(128, NT);
    const uint32_t sAu = umma::smem_u32(sA), sBu = umma::smem_u32(sB);
    const uint32_t sbo = (uint32_t)kc * 128;
    const int quarter = warp & 3, part = warp >> 2;  // TMEM lanes 32 * quarter.., every kRowsParts-th 32 columns
    const int m = quarter * 32 + lane;
    float csum[8 / kRowsParts] = {};  // column sums: lane's column of this warp's chunks

    auto epilogue = [&](int64_t t, uint32_t buf) {
        const int64_t grow = t * 128 + m;
        const bool ok = grow < g.M;
        const uint32_t trow = tmem + buf * acc + ((uint32_t)(quarter * 32) << 16);
        const int64_t m0 = t * 128 + quarter * 32;
#pragma unroll
        for (int ci = 0; ci < 8 / kRowsParts; ++ci) {
            const int c0 = 32 * (part + ci * kRowsParts);
            if (c0 >= NT) break;
            const int n = n0 + c0;  // first column of this chunk
            uint4 zq[4];
            if (ZP) {
                if (g.zvec) {
                    const int64_t row = m0 + (lane & ~3);
                    const bf16* src = g.zp + row * g.ldzp + n + (lane & 3) * 8;
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        zq[q] = row + q < g.M ? *reinterpret_cast<const uint4*>(src + q * g.ldzp) : make_uint4(0, 0, 0, 0);
                    quad_transpose(zq, lane);
                } else {
                    const bf16* src = g.zp + (ok ? grow : 0) * g.ldzp + n;
                    bf16* d = reinterpret_cast<bf16*>(zq);
#pragma unroll
                    for (int j = 0; j < 32; ++j) d[j] = src[j];
                }
            }
            float v[32];
            umma::tmem_ld32(trow + (uint32_t)c0, v);
            uint4 yq[4];
            uint32_t* yw = reinterpret_cast<uint32_t*>(yq);
            if (g.bias) {
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 b = *reinterpret_cast<const float4*>(sbias + c0 + j);
                    v[j] += b.x;
                    v[j + 1] += b.y;
                    v[j + 2] += b.z;
                    v[j + 3] += b.w;
                }
            }
            if (g.Z) {
#pragma unroll
                for (int j = 0; j < 16; ++j) yw[j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
                store_rows64(reinterpret_cast<uint8_t*>(g.Z + n), g.ldz * 2, m0, g.M, yq, lane);
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                float x = v[j];
                if (ZP) {
                    const float z = ok ? __bfloat162float(reinterpret_cast<const bf16*>(zq)[j]) : 0.0f;
                    const float sg = sigmoidf_(z);
                    x *= sg * (1.0f + z * (1.0f - sg));
                }
                v[j] = g.act ? x * sigmoidf_(x) : x;
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) yw[j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
            if (g.YT) {
                // two rows of one column per lane: the even lane takes column 2k, the odd one 2k + 1
                const int odd = lane & 1;
                const int64_t row = grow - odd;
                bf16* yt = g.YT + (int64_t)(n + odd) * g.ldyt + row;
#pragma unroll
                for (int k = 0; k < 16; ++k, yt += 2 * g.ldyt) {
                    const uint32_t other = __shfl_xor_sync(0xffffffffu, yw[k], 1);
                    const uint32_t two = odd ? __byte_perm(other, yw[k], 0x7632) : __byte_perm(yw[k], other, 0x5410);
                    if (g.ytvec && row + 1 < g.M) {
                        *reinterpret_cast<uint32_t*>(yt) = two;
                    } else {
                        if (row < g.M) yt[0] = __ushort_as_bfloat16((unsigned short)two);
                        if (row + 1 < g.M) yt[1] = __ushort_as_bfloat16((unsigned short)(two >> 16));
                    }
                }
            }
            if (g.Y) store_rows64(reinterpret_cast<uint8_t*>(g.Y + n), g.ldy * 2, m0, g.M, yq, lane);
            if (g.Y32) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) yw[j] = __float_as_uint(v[16 * h + j]);
                    store_rows64(reinterpret_cast<uint8_t*>(g.Y32 + n + 16 * h), g.ldy32 * 4, m0, g.M, yq, lane);
                }
            }
            if (g.colsum) {
                // 32 columns over 32 lanes in 31 exchanges: each step folds the
                // halves of the columns onto the halves of the lanes; lane l ends
                // with the sum of column l
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (!ok) v[j] = 0.0f;
#pragma unroll
                for (int h = 16; h > 0; h >>= 1) {
                    const bool up = lane & h;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (j >= h) break;
                        const float send = up ? v[j] : v[j + h], keep = up ? v[j + h] : v[j];
                        v[j] = keep + __shfl_xor_sync(0xffffffffu, send, h);
                    }
                }
                csum[ci] += v[0];
            }
        }
    };

    bool timeout = false;
    int64_t i = 0;
    for (int64_t t = t0; t < ntiles; t += step, ++i) {
        const uint32_t buf = (uint32_t)i & 1u, stage = stages == 2 ? buf : 0u;
        umma::cp_async_wait_all();
        umma::fence_proxy_async();
        umma::fence_before();
        __syncthreads();
        if (tid == 0) {
            umma::fence_after();
            for (int ks = 0; ks < (g.K >> 4); ++ks) {
                const uint64_t ad = umma::sdesc(sAu + stage * stage_bytes + ks * 256, 128, sbo);
                const uint64_t bd = umma::sdesc(sBu + ks * 256, 128, sbo);
                umma::mma_bf16(tmem + buf * acc, ad, bd, idesc, ks > 0 ? 1u : 0u);
            }
            umma::mma_commit(&mbar[buf]);
        }
        if (stages == 2) {
            // tile i - 1 is multiplied (waited for below): its stage takes tile i + 1
            if (t + step < ntiles) load_a(t + step, buf ^ 1u);
            if (i > 0) epilogue(t - step, buf ^ 1u);
            if (!umma::mbar_wait(&mbar[buf], (uint32_t)(i >> 1) & 1u)) timeout = true;
            umma::fence_after();
        } else {
            if (!umma::mbar_wait(&mbar[buf], (uint32_t)(i >> 1) & 1u)) timeout = true;
            umma::fence_after();
            if (t + step < ntiles) load_a(t + step, 0);
            epilogue(t, buf);
        }
    }
    if (stages == 2 && i > 0) epilogue(t0 + (i - 1) * step, (uint32_t)(i - 1) & 1u);
    if (timeout && lane == 0) atomicExch(&g_umma_err, 1);
    if (g.colsum) {
#pragma unroll
        for (int ci = 0; ci < 8 / kRowsParts; ++ci) {
            const int c0 = 32 * (part + ci * kRowsParts);
            if (c0 < NT && i > 0) atomicAdd(g.colsum + n0 + c0 + lane, csum[ci]);
        }
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    if (warp == 0) umma::tmem_dealloc(tmem, ncols);
}

struct WgradArgs {
    const bf16* A;   // [Mo x Kb], Kb contiguous
    int64_t lda;
    const bf16* B;   // [No x Kb]
    int64_t ldb;
    int Mo, No;
    int64_t Kb, kchunk;
    float* C;        // [Mo x No] += A B^T
    int64_t ldc;
    int vec;         // C and ldc allow 16-byte reductions
};

constexpr int WK = 64;  // reduction block staged per step

// The reduction blocks pass through a ring of kWStages shared-memory stages:
// the copies of the next ones run while the tensor core multiplies.  The FP32
// partial result is added to C four columns per reduction.  256 x 256 over
// 49,152 states on GB300: 69 us with one stage and one column per reduction,
// 26 us here
// (31 without the quad transpose before the reductions).
constexpr int kWThreads = 256, kWStages = 4;

__global__ void __launch_bounds__(kWThreads, 1) umma_wgrad_kernel(const WgradArgs g)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar[kWStages];
    __shared__ uint32_t tmem_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int kc = WK / 8;
    const uint32_t a_bytes = 128u * WK * 2, stage_bytes = (128u + (uint32_t)g.No) * WK * 2;
    const uint32_t ncols = g.No <= 32 ? 32u : (g.No <= 64 ? 64u : (g.No <= 128 ? 128u : 256u));
    if (warp == 0) {
        umma::tmem_alloc(&tmem_s, ncols);
        umma::tmem_relinquish();
    }
    if (tid == 0)
        for (int q = 0; q < kWStages; ++q) umma::mbar_init(&mbar[q], 1);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = tmem_s;
    const uint32_t idesc = umma::idesc_bf16(128, g.No);
    const uint32_t su = umma::smem_u32(smem);
    const int mrow0 = blockIdx.x * 128;
    const int64_t k0 = (int64_t)blockIdx.y * g.kchunk;
    const int64_t k1 = k0 + g.kchunk < g.Kb ? k0 + g.kchunk : g.Kb;
    const int steps = k1 > k0 ? (int)((k1 - k0) / WK) : 0;
    auto load = [&](int s) {
        if (s < steps) {
            uint8_t* sA = smem + (size_t)(s % kWStages) * stage_bytes;
            uint8_t* sB = sA + a_bytes;
            const int64_t kb = k0 + (int64_t)s * WK;
            for (int idx = tid; idx < 128 * kc; idx += kWThreads) {
                const int r = idx / kc, c = idx - r * kc;
                const bool ok = mrow0 + r < g.Mo;
                umma::cp_async16(sA + ((size_t)(r >> 3) * kc + c) * 128 + (r & 7) * 16,
                                 g.A + (int64_t)(ok ? mrow0 + r : 0) * g.lda + kb + c * 8, ok ? 16u : 0u);
            }
            for (int idx = tid; idx < g.No * kc; idx += kWThreads) {
                const int n = idx / kc, c = idx - n * kc;
                umma::cp_async16(sB + ((size_t)(n >> 3) * kc + c) * 128 + (n & 7) * 16,
                                 g.B + (int64_t)n * g.ldb + kb + c * 8, 16u);
            }
        }
        umma::cp_async_commit();
    };
    for (int s = 0; s < kWStages - 1; ++s) load(s);
    bool timeout = false;
    for (int s = 0; s < steps; ++s) {
        umma::cp_async_wait<kWStages - 2>();
        umma::fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
            umma::fence_after();
            const uint32_t sAu = su + (uint32_t)(s % kWStages) * stage_bytes, sBu = sAu + a_bytes;
#pragma unroll
            for (int ks = 0; ks < WK / 16; ++ks) {
                const uint64_t ad = umma::sdesc(sAu + ks * 256, 128, kc * 128);
                const uint64_t bd = umma::sdesc(sBu + ks * 256, 128, kc * 128);
                umma::mma_bf16(tmem, ad, bd, idesc, (s == 0 && ks == 0) ? 0u : 1u);
            }
            umma::mma_commit(&mbar[s % kWStages]);
        }
        // the stage of step s - 1, once multiplied, takes step s + kWStages - 1
        if (s > 0 && !umma::mbar_wait(&mbar[(s - 1) % kWStages], (uint32_t)((s - 1) / kWStages) & 1u)) timeout = true;
        load(s + kWStages - 1);
    }
    if (steps > 0) {
        if (!umma::mbar_wait(&mbar[(steps - 1) % kWStages], (uint32_t)((steps - 1) / kWStages) & 1u)) timeout = true;
        umma::fence_after();
        const int quarter = warp & 3;
        const int m = mrow0 + quarter * 32 + lane;
        for (int c0 = 32 * (warp >> 2); c0 < g.No; c0 += 64) {
            float v[32];
            umma::tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, v);
            if (g.vec) {
                // the quad transpose of the layer kernels: 64 bytes of a row per quad
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint4 r[4];
                    uint32_t* w = reinterpret_cast<uint32_t*>(r);
#pragma unroll
                    for (int j = 0; j < 16; ++j) w[j] = __float_as_uint(v[16 * h + j]);
                    quad_transpose(r, lane);
                    const int row = m & ~3;
                    float* c = g.C + (int64_t)row * g.ldc + c0 + 16 * h + 4 * (lane & 3);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (row + q < g.Mo)
                            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                                         :: "l"(__cvta_generic_to_global(c + q * g.ldc)),
                                            "f"(__uint_as_float(r[q].x)), "f"(__uint_as_float(r[q].y)),
                                            "f"(__uint_as_float(r[q].z)), "f"(__uint_as_float(r[q].w)) : "memory");
                }
            } else if (m < g.Mo) {
                float* c = g.C + (int64_t)m * g.ldc + c0;
                for (int j = 0; j < 32; ++j) atomicAdd(c + j, v[j]);
            }
        }
    }
    if (timeout && lane == 0) atomicExch(&g_umma_err, 1);
    umma::cp_async_wait_all();
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    if (warp == 0) umma::tmem_dealloc(tmem, ncols);
}


// dY [M x 64] FP32 to what the backward pass starts from, in one pass: BF16,
// BF16 transposed and column sums (the last bias's gradient).  A block takes
// 64 x 64 tiles; bound by dY's bytes.  49,152 rows on GB300: 45 us as a sum, a
// cast and a transposed copy; a training pass 567 -> 498 us with this kernel and
// one zeroed buffer for the gradients.
constexpr int HEAD_THREADS = 256;

__global__ void __launch_bounds__(HEAD_THREADS) head_grad_kernel(const float* __restrict__ dY, int64_t ldy, int64_t M,
                                                                 bf16* __restrict__ Z, int64_t ldz,
                                                                 bf16* __restrict__ ZT, int64_t ldzt, int ztvec,
                                                                 float* __restrict__ colsum)
{
    __shared__ __align__(16) bf16 t[64][72];  // [column][row], rows padded to spread the banks
    __shared__ float part[16][64];
    const int cg = threadIdx.x & 15, r0 = threadIdx.x >> 4;  // columns 4 cg.., rows r0, r0 + 16, ..
    float s[4] = {};
    for (int64_t row0 = (int64_t)blockIdx.x * 64; row0 < M; row0 += (int64_t)gridDim.x * 64) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = r0 + 16 * k;
            const int64_t row = row0 + r;
            float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (row < M) y = *reinterpret_cast<const float4*>(dY + row * ldy + 4 * cg);
            s[0] += y.x;
            s[1] += y.y;
            s[2] += y.z;
            s[3] += y.w;
            const uint2 w = make_uint2(pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
            if (row < M) *reinterpret_cast<uint2*>(Z + row * ldz + 4 * cg) = w;
            t[4 * cg][r] = __ushort_as_bfloat16((unsigned short)w.x);
            t[4 * cg + 1][r] = __ushort_as_bfloat16((unsigned short)(w.x >> 16));
            t[4 * cg + 2][r] = __ushort_as_bfloat16((unsigned short)w.y);
            t[4 * cg + 3][r] = __ushort_as_bfloat16((unsigned short)(w.y >> 16));
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int e = threadIdx.x + k * HEAD_THREADS, c = e >> 3, r = 8 * (e & 7);
            bf16* d = ZT + c * ldzt + row0 + r;
            if (ztvec && row0 + r + 8 <= M) {
                *reinterpret_cast<uint4*>(d) = *reinterpret_cast<const uint4*>(&t[c][r]);
            } else {
                for (int j = 0; j < 8; ++j)
                    if (row0 + r + j < M) d[j] = t[c][r + j];
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) part[r0][4 * cg + j] = s[j];
    __syncthreads();
    if (threadIdx.x < 64) {
        float a = 0.0f;
        for (int r = 0; r < 16; ++r) a += part[r][threadIdx.x];
        atomicAdd(colsum + threadIdx.x, a);
    }
}

// ---------------------------------------------------------------------------
// Fused forward pass of the whole network, 64 -> 256 -> 256 -> 256 -> 256 -> 64
// (SiLU on the hidden layers), for inference.  A persistent CTA takes 128-row
// tiles two at a time; a tile's activations stay in shared memory from layer to
// layer (the epilogue of layer l writes the BF16 A operand of layer l + 1), so
// only the features are read from and the FP32 outputs written to global memory.
// The two tiles take turns: while one warp multiplies one (tcgen05, half of
// TMEM each), 16 warps (four per TMEM lane quarter, each a quarter of the
// columns) read the other's accumulator from TMEM and apply bias and SiLU.  The
// weights stream from L2 through a ring of 16 KB slots, a slice of K = 32 of all
// 256 columns each (K = 64 of the last layer's 64), one tensor copy per slice:
// the packed weights are rows of core matrices to the tensor map, 8 columns each.
// Bound by the hardware tanh (half the rate of the other special functions:
// 452 us of 1,048,576 rows on GB300).  1022 us with one tile at a time, whose
// layers multiplied, then applied SiLU; 1088 us with two tiles while one warp
// copied and multiplied (its own instructions per slice cost more than the
// slice); 745 us with a warp for each; 606 us with the biases in shared memory.
struct FusedArgs {
    CUtensorMap W[5];    // packed weights: 256x64, 256x256 (x3), 64x256
    const bf16* X;       // [M x 64] features
    int64_t ldx, M;
    const float* b[5];
    float* Y;            // [M x 64] outputs
    int64_t ldy;
};

constexpr uint32_t FUSED_SLOT = 16 * 1024;
constexpr uint32_t FUSED_ACT = 64 * 1024;                 // activation tile
constexpr int FUSED_SLOTS = 5;
constexpr size_t FUSED_SMEM = 2 * (size_t)FUSED_ACT + FUSED_SLOTS * (size_t)FUSED_SLOT;

// SiLU of the fused inference epilogue, the same expression as the layer kernels'
__device__ __forceinline__ float silu_fast(float x) { return x * sigmoidf_(x); }

constexpr int FUSED_EPI = 512, FUSED_THREADS = FUSED_EPI + 64;  // 16 warps: four per TMEM lane quarter, each a quarter of the columns

template <int N>
struct IntC {
    static constexpr int value = N;
};

// bounded wait that also ends when another warp gave up
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t phase, volatile int* stop)
{
    bool ok = false;
    for (uint32_t it = 0; it < (1u << 26); ++it) {
        ok = umma::mbar_try_wait(bar, phase);
        if (ok || ((it & 1023u) == 1023u && *stop)) break;
    }
    if (!ok) *stop = 1;
    return ok;
}

__global__ void __launch_bounds__(FUSED_THREADS, 1) mlp_fused_kernel(const __grid_constant__ FusedArgs g)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[FUSED_SLOTS], empty[FUSED_SLOTS];  // a slot's slice has arrived, is multiplied
    __shared__ uint64_t ready[2], accum[2], drain;              // a tile's operand is written, is multiplied
    __shared__ uint32_t tmem_s;
    __shared__ int s_abort;
    __shared__ __align__(16) float sbias[4 * 256 + 64];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < 4 * 256 + 64; i += FUSED_THREADS)
        sbias[i] = i < 1024 ? g.b[i >> 8][i & 255] : g.b[4][i - 1024];
    if (warp == 0) {
        umma::tmem_alloc(&tmem_s, 512);
        umma::tmem_relinquish();
    }
    if (tid == 0) {
        for (int q = 0; q < FUSED_SLOTS; ++q) {
            umma::mbar_init(&full[q], 1);
            umma::mbar_init(&empty[q], 1);
        }
        for (int q = 0; q < 2; ++q) {
            umma::mbar_init(&ready[q], FUSED_EPI / 32);
            umma::mbar_init(&accum[q], 1);
        }
        umma::mbar_init(&drain, 1);
        s_abort = 0;
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = tmem_s;
    const int64_t ntiles = (g.M + 127) / 128;
    const int mine = (int)((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x);  // grid <= ntiles
    auto row_of = [&](int i) { return ((int64_t)blockIdx.x + (int64_t)i * gridDim.x) * 128; };
    bool ok = true;
    uint32_t phases = 0u;  // a bit per tile: of ready (the multiplying warp) or accum (the epilogue)

    if (warp == FUSED_EPI / 32) {
        // multiplies; one thread, with descriptors that only add to a word, because
        // each instruction before an MMA delays it
        if (lane == 0) {
            const uint32_t a0 = umma::smem_u32(smem) >> 4, w0 = a0 + (2 * FUSED_ACT >> 4);
            const uint32_t lbo = (128u >> 4) << 16;
            auto desc = [&](uint32_t lo, uint32_t sbo) {
                return ((uint64_t)((1u << 14) | (sbo >> 4)) << 32) | (lo | lbo);
            };
            int slot = 0;
            uint32_t sphase = 0u;
            auto step = [&](int b, int nch, auto nks_c, uint32_t asbo, uint32_t bsbo, uint32_t id) {
                constexpr int nks = decltype(nks_c)::value;
                ok = wait_or_abort(&ready[b], phases >> b & 1u, &s_abort);
                phases ^= 1u << b;
                uint64_t ad = desc(a0 + b * (FUSED_ACT >> 4), asbo);
                uint32_t acc = 0u;
                for (int c = 0; c < nch && ok; ++c, ad += nks * 16) {
                    ok = wait_or_abort(&full[slot], sphase, &s_abort);
                    if (!ok) break;
                    umma::fence_after();
                    const uint64_t bd = desc(w0 + slot * (FUSED_SLOT >> 4), bsbo);
#pragma unroll
                    for (int ks = 0; ks < nks; ++ks) {
                        umma::mma_bf16(tmem + 256u * b, ad + ks * 16, bd + ks * 16, id, acc);
                        acc = 1u;
                    }
                    umma::mma_commit(&empty[slot]);
                    if (++slot == FUSED_SLOTS) {
                        slot = 0;
                        sphase ^= 1u;
                    }
                }
                if (ok) umma::mma_commit(&accum[b]);
            };
            for (int p = 0; 2 * p < mine && ok; ++p) {
                const int nb = 2 * p + 1 < mine ? 2 : 1;
                for (int b = 0; b < nb && ok; ++b)
                    step(b, 2, IntC<2>{}, 8 * 128, 512, umma::idesc_bf16(128, 256));
                for (int l = 1; l < 4; ++l)
                    for (int b = 0; b < nb && ok; ++b)
                        step(b, 8, IntC<2>{}, 32 * 128, 512, umma::idesc_bf16(128, 256));
                for (int b = 0; b < nb && ok; ++b)
                    step(b, 4, IntC<4>{}, 32 * 128, 1024, umma::idesc_bf16(128, 64));
            }
            // no MMA may still be reading or writing this CTA's memory when it exits
            umma::mma_commit(&drain);
            umma::mbar_wait(&drain, 0u);
            if (!ok) atomicExch(&g_umma_err, 1);
        }
        __syncwarp();
    } else if (warp == FUSED_EPI / 32 + 1) {
        // copies the slices, layer by layer and a pair's tiles in turn
        if (lane == 0) {
            int slot = 0, n = 0;
            uint32_t ephase = 1u, fphase = 0u;  // a slot's first use waits for nothing
            for (int p = 0; 2 * p < mine && ok; ++p)
                for (int l = 0; l < 5; ++l)
                    for (int b = 0; b < 2 && 2 * p + b < mine && ok; ++b) {
                        const int nch = l == 0 ? 2 : (l < 4 ? 8 : 4), width = l < 4 ? 128 : 256;
                        for (int c = 0; c < nch && ok; ++c) {
                            if (n >= FUSED_SLOTS) ok = wait_or_abort(&empty[slot], ephase, &s_abort);
                            if (!ok) break;
                            umma::mbar_expect_tx(&full[slot], l < 4 ? FUSED_SLOT : FUSED_SLOT / 2);
                            umma::tensor_g2s_2d(smem + 2 * FUSED_ACT + slot * FUSED_SLOT, &g.W[l], c * width, 0, &full[slot]);
                            ++n;
                            if (++slot == FUSED_SLOTS) {
                                slot = 0;
                                ephase ^= 1u;
                                fphase ^= 1u;
                            }
                        }
                    }
            // nor may a copy: the last use of every slot has arrived
            for (int q = 0; q < FUSED_SLOTS && q < n; ++q) {
                if (slot-- == 0) {
                    slot = FUSED_SLOTS - 1;
                    fphase ^= 1u;
                }
                umma::mbar_wait(&full[slot], fphase);
            }
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3, part = warp >> 2;  // TMEM lanes 32 * quarter.., column quarter
        const int m = quarter * 32 + lane;
        // this thread's two 16-byte pieces of a tile's features (8 per row), and
        // their places in the A operand of layer 0
        uint4 f[2];
        auto load_x = [&](int i) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int idx = tid + q * FUSED_EPI;
                const int64_t row = row_of(i) + (idx >> 3);
                f[q] = row < g.M ? *reinterpret_cast<const uint4*>(g.X + row * g.ldx + (idx & 7) * 8)
                                 : make_uint4(0, 0, 0, 0);
            }
        };
        auto put_x = [&](int b) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int idx = tid + q * FUSED_EPI, r = idx >> 3, c = idx & 7;
                *reinterpret_cast<uint4*>(smem + b * FUSED_ACT + ((r >> 3) * 8 + c) * 128 + (r & 7) * 16) = f[q];
            }
        };
        auto publish = [&](int b) {  // this warp's share of a tile's operand is written, its accumulator read
            umma::fence_before();
            umma::fence_proxy_async();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&ready[b]);
        };
        for (int b = 0; b < 2 && b < mine; ++b) {
            load_x(b);
            put_x(b);
            publish(b);
        }
        for (int p = 0; 2 * p < mine && ok; ++p)
            for (int l = 0; l < 5 && ok; ++l)
                for (int b = 0; b < 2 && 2 * p + b < mine && ok; ++b) {
                    const bool more = 2 * (p + 1) + b < mine;
                    if (l == 4 && more) load_x(2 * (p + 1) + b);
                    ok = __all_sync(0xffffffffu, wait_or_abort(&accum[b], phases >> b & 1u, &s_abort));
                    if (!ok) break;
                    phases ^= 1u << b;
                    umma::fence_after();
                    const uint32_t trow = tmem + 256u * b + ((uint32_t)(quarter * 32) << 16);
                    if (l < 4) {
                        const float* bias = sbias + 256 * l;
                        uint8_t* dst = smem + b * FUSED_ACT + ((m >> 3) * 32) * 128 + (m & 7) * 16;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int c0 = 64 * part + 32 * h;
                            float v[32];
                            umma::tmem_ld32(trow + (uint32_t)c0, v);
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                alignas(16) float bb[8];
                                *reinterpret_cast<float4*>(bb) = *reinterpret_cast<const float4*>(bias + c0 + 8 * q);
                                *reinterpret_cast<float4*>(bb + 4) = *reinterpret_cast<const float4*>(bias + c0 + 8 * q + 4);
                                uint32_t w[4];
#pragma unroll
                                for (int e = 0; e < 4; ++e)
                                    w[e] = pack_bf16x2(silu_fast(v[8 * q + 2 * e] + bb[2 * e]),
                                                       silu_fast(v[8 * q + 2 * e + 1] + bb[2 * e + 1]));
                                *reinterpret_cast<uint4*>(dst + ((c0 >> 3) + q) * 128) = make_uint4(w[0], w[1], w[2], w[3]);
                            }
                        }
                        publish(b);
                    } else {
                        const int c0 = 16 * part;
                        float v[16];
                        umma::tmem_ld16(trow + (uint32_t)c0, v);
                        if (more) put_x(b);
                        publish(b);
                        uint4 r[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const float4 bb = *reinterpret_cast<const float4*>(sbias + 1024 + c0 + 4 * q);
                            r[q] = make_uint4(__float_as_uint(v[4 * q] + bb.x), __float_as_uint(v[4 * q + 1] + bb.y),
                                              __float_as_uint(v[4 * q + 2] + bb.z), __float_as_uint(v[4 * q + 3] + bb.w));
                        }
                        store_rows64(reinterpret_cast<uint8_t*>(g.Y + c0), g.ldy * 4,
                                     row_of(2 * p + b) + quarter * 32, g.M, r, lane);
                    }
                }
        if (!ok && lane == 0) atomicExch(&g_umma_err, 1);
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------
// Surrogate input and output stages (thread per state, C-order states).
//
// Features: X[s] = BF16 of ((T - 1500) / 400, (ln P - mu_P) / sd_P,
// (log10 max(c_k, floor) - mu_k) / sd_k for the ns - 1 species, 0 ...) with
// c_k = max(n_k, 0) / V; logarithms in FP32 (the features are BF16).
__global__ void surr_features_kernel(int64_t n, int nn, const double* __restrict__ phi,
                                     const double* __restrict__ param, const double* __restrict__ st,
                                     bf16* X, float floor_c)
{
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const double* p = phi + s * nn;
    const float inv_v = (float)(1.0 / p[1]);  // one FP64 division per state; the rest is FP32
    // st: lnP_mu, lnP_sd, lc_mu[nn - 2], lc_sd[nn - 2]
    alignas(16) bf16 f[64];
    f[0] = __float2bfloat16((float)(p[0] - 1500.0) * 0.0025f);
    f[1] = __float2bfloat16((float)((log(param[s]) - st[0]) / st[1]));
    const int nsp = nn - 2;
    for (int k = 0; k < nsp; ++k) {
        const float c = fmaxf((float)p[2 + k], 0.0f) * inv_v;
        const float lc = log10f(fmaxf(c, floor_c));
        f[2 + k] = __float2bfloat16(__fdividef(lc - (float)st[2 + k], (float)st[2 + nsp + k]));
    }
    for (int k = nn; k < 64; ++k) f[k] = __float2bfloat16(0.0f);
    uint4* d = reinterpret_cast<uint4*>(X + s * 64);
    const uint4* src = reinterpret_cast<const uint4*>(f);
#pragma unroll
    for (int q = 0; q < 8; ++q) d[q] = src[q];
}

// Outputs: y_j = sinh(Y[s][j] z_sd_j + z_mu_j) s_j (FP32 transcendental, FP64
// result) for the 53 rates {dT/dt, dn_k/dt}; dphi = (Tdot, extra-variable rate
// recomputed as the FP64 path does, the ndot_k); lerr[s] = Y[s][err_col].
__global__ void surr_outputs_kernel(int64_t n, int nn, const float* __restrict__ Y,
                                    const double* __restrict__ phi,
                                    const double* __restrict__ param,
                                    const double* __restrict__ st, int err_col,
                                    double* __restrict__ dphi, float* __restrict__ lerr)
{
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int nout = nn - 1;                       // Tdot + (nn - 2) species rates
    const double* zmu = st;
    const double* zsd = st + nout;
    const double* sc = st + 2 * nout;
    const double* omw = st + 3 * nout;             // 1 - W_k / W_ns, nn - 2 values
    const float* y = Y + s * 64;
    const double* p = phi + s * nn;
    double* o = dphi + s * nn;
    const double T = fmin(10000.0, fmax(100.0, p[0]));
    const double V = fmax(p[1], 1e-30);
    const double P = param[s];
    double dE = 0.0;  // sum_k (1 - W_k / W_ns) ndot_k; divided by V once below
    for (int j = 0; j < nout; ++j) {
        const float z = fmaf(y[j], (float)zsd[j], (float)zmu[j]);
        const double v = (double)sinhf(z) * sc[j];
        if (j == 0) {
            o[0] = v;
        } else {
            o[1 + j] = v;
            dE = fma(v, omw[j - 1], dE);
        }
    }
    o[1] = V * o[0] / T + dE * T * 8314.4621 / P;
    lerr[s] = y[err_col];
}

int sm_count()
{
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
    }
    return n;
}

constexpr size_t kRowsSmemMax = (227 << 10) - 2048;  // less the kernel's static shared memory
// cuTensorMapEncodeTiled of the loaded driver (the library does not link libcuda)
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled tensor_map_encoder()
{
    static const EncodeTiled fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiled>(p);
    }();
    return fn;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

}  // namespace

// launchers (declared in pjg_mlp.cuh-free form: used only by pjg_capi.cu)
int mlp_launch_rows(const void* A, int64_t lda, const void* B, int64_t ldb, int64_t M, int N, int K,
                 const float* bias, int act, const void* zp, int64_t ldzp, void* Y, int64_t ldy,
                 void* YT, int64_t ldyt, void* Z, int64_t ldz, float* Y32, int64_t ldy32,
                 float* colsum, void* stream)
{
    if (M <= 0) return 0;
    if (N < 32 || N > 256 || N % 32 || K < 16 || K > 256 || K % 16 || !A || !B) return -1;
    if (lda % 8 || ldb % 8 || !aligned16(A) || !aligned16(B)) return -1;
    if ((Y && (ldy % 8 || !aligned16(Y))) || (Z && (ldz % 8 || !aligned16(Z))) ||
        (Y32 && (ldy32 % 4 || !aligned16(Y32))))
        return -1;
    RowsArgs g;
    g.A = (const bf16*)A; g.lda = lda; g.B = (const bf16*)B; g.ldb = ldb;
    g.M = M; g.N = N; g.K = K; g.bias = bias; g.act = act;
    g.zp = (const bf16*)zp; g.ldzp = ldzp;
    g.Y = (bf16*)Y; g.ldy = ldy; g.YT = (bf16*)YT; g.ldyt = ldyt; g.Z = (bf16*)Z; g.ldz = ldz;
    g.Y32 = Y32; g.ldy32 = ldy32; g.colsum = colsum;
    g.ytvec = YT && ldyt % 2 == 0 && ((uintptr_t)YT & 3) == 0;
    g.zvec = zp && ldzp % 8 == 0 && aligned16(zp);
    // half of the columns per CTA where that lets a second tile of A fit (A is
    // then read twice, from L2), as for N = K = 256; an output that overlaps A
    // keeps whole rows in one CTA, which reads a tile before it writes it
    g.NT = N;
    g.stages = 2;
    auto smem_of = [&](int nt, int st) { return ((size_t)nt + 128 * st) * K * 2; };
    auto meets_a = [&](const void* p, int64_t ld, int bytes) {
        const uintptr_t a0 = (uintptr_t)A, a1 = a0 + ((M - 1) * lda + K) * 2;
        const uintptr_t p0 = (uintptr_t)p, p1 = p0 + ((M - 1) * ld + N) * bytes;
        return p && p0 < a1 && a0 < p1;
    };
    if (smem_of(N, 2) > kRowsSmemMax) {
        const bool split = N % 64 == 0 && smem_of(N / 2, 2) <= kRowsSmemMax &&
                           !meets_a(Y, ldy, 2) && !meets_a(Z, ldz, 2) && !meets_a(Y32, ldy32, 4);
        if (split) g.NT = N / 2;
        else g.stages = 1;
    }
    const size_t smem = smem_of(g.NT, g.stages);
    auto kern = zp ? umma_rows_kernel<true> : umma_rows_kernel<false>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int64_t ntiles = (M + 127) / 128;
    const int halves = N / g.NT, per = sm_count() > halves ? sm_count() / halves : 1;
    const int grid = (int)(ntiles < per ? ntiles : per) * halves;
    kern<<<grid, kRowsThreads, smem, (cudaStream_t)stream>>>(g);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int mlp_launch_wgrad(const void* A, int64_t lda, const void* B, int64_t ldb, int Mo, int No, int64_t Kb,
                  float* C, int64_t ldc, void* stream)
{
    if (Kb <= 0) return 0;
    if (No < 32 || No > 256 || No % 32 || Mo <= 0 || Kb % WK || !A || !B || !C) return -1;
    if (lda % 8 || ldb % 8 || !aligned16(A) || !aligned16(B)) return -1;
    WgradArgs g;
    g.A = (const bf16*)A; g.lda = lda; g.B = (const bf16*)B; g.ldb = ldb;
    g.Mo = Mo; g.No = No; g.Kb = Kb; g.C = C; g.ldc = ldc;
    const int mt = (Mo + 127) / 128;
    int splits = (sm_count() + mt - 1) / mt;
    int64_t chunk = (Kb + splits - 1) / splits;
    chunk = (chunk + WK - 1) / WK * WK;
    splits = (int)((Kb + chunk - 1) / chunk);
    g.kchunk = chunk;
    g.vec = ldc % 4 == 0 && aligned16(C);
    const size_t smem = (size_t)kWStages * (128 + No) * WK * 2;
    cudaFuncSetAttribute(umma_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    umma_wgrad_kernel<<<dim3(mt, splits), kWThreads, smem, (cudaStream_t)stream>>>(g);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int mlp_launch_head(const float* dY, int64_t ldy, int64_t M, void* Z, int64_t ldz, void* ZT, int64_t ldzt,
                    float* colsum, void* stream)
{
    if (M <= 0) return 0;
    if (!dY || !Z || !ZT || !colsum || ldy % 4 || ldz % 4 || !aligned16(dY) || ((uintptr_t)Z & 7)) return -1;
    const int64_t ntiles = (M + 63) / 64;
    const int grid = (int)(ntiles < 4 * sm_count() ? ntiles : 4 * sm_count());
    head_grad_kernel<<<grid, HEAD_THREADS, 0, (cudaStream_t)stream>>>(dY, ldy, M, (bf16*)Z, ldz, (bf16*)ZT, ldzt,
                                                                      ldzt % 8 == 0 && aligned16(ZT), colsum);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int mlp_launch_fused(const void* X, int64_t ldx, int64_t M, const void* const* W,
                     const float* const* b, float* Y, int64_t ldy, void* stream)
{
    if (M <= 0) return 0;
    if (!X || !Y || ldx % 8 || ldy % 4 || ldx < 64 || ldy < 64 || !aligned16(X) || !aligned16(Y))
        return -1;
    const auto encode = tensor_map_encoder();
    if (!encode) return -2;
    FusedArgs g;
    g.X = (const bf16*)X;
    g.ldx = ldx;
    g.M = M;
    for (int l = 0; l < 5; ++l) {
        if (!W[l] || !b[l] || !aligned16(W[l])) return -1;
        g.b[l] = b[l];
        // rows of 8 columns' core matrices, as 32-bit words; a slice is K = 32 (the last layer: 64) of every row
        const cuuint64_t dims[2] = {(cuuint64_t)(l ? 1024 : 256), (cuuint64_t)(l < 4 ? 32 : 8)};
        const cuuint64_t pitch[1] = {dims[0] * 4};
        const cuuint32_t box[2] = {l < 4 ? 128u : 256u, (cuuint32_t)dims[1]}, ones[2] = {1, 1};
        if (encode(&g.W[l], CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(W[l]), dims, pitch, box, ones,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return -2;
    }
    g.Y = Y;
    g.ldy = ldy;
    cudaFuncSetAttribute(mlp_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FUSED_SMEM);
    const int64_t ntiles = (M + 127) / 128;
    const int grid = (int)(ntiles < sm_count() ? ntiles : sm_count());
    mlp_fused_kernel<<<grid, FUSED_THREADS, FUSED_SMEM, (cudaStream_t)stream>>>(g);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int surr_launch_features(int64_t n, int nn, const double* phi, const double* param,
                         const double* st, void* X, float floor_c, void* stream)
{
    if (n <= 0) return 0;
    if (nn > 64 || nn < 3 || !aligned16(X)) return -1;
    surr_features_kernel<<<(unsigned)((n + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
        n, nn, phi, param, st, (bf16*)X, floor_c);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int surr_launch_outputs(int64_t n, int nn, const float* Y, const double* phi, const double* param,
                        const double* st, int err_col, double* dphi, float* lerr, void* stream)
{
    if (n <= 0) return 0;
    if (nn > 65 || nn < 3 || err_col < 0 || err_col >= 64) return -1;
    surr_outputs_kernel<<<(unsigned)((n + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
        n, nn, Y, phi, param, st, err_col, dphi, lerr);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int mlp_error_flag(int clear)
{
    int h = 0;
    cudaMemcpyFromSymbol(&h, g_umma_err, sizeof(int));
    if (clear) {
        const int z = 0;
        cudaMemcpyToSymbol(g_umma_err, &z, sizeof(int));
    }
    return h;
}
