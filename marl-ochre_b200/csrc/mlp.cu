// Inference kernels of the reaction surrogate (a tcgen05 GEMM per layer, and the
// whole network in one persistent kernel), the feature statistics and the
// initial weights.  Training is in mlp_train.cu.
//
// GEMM form: C[M][N] = A[M][K] * B[N][K]^T with A and B BF16, both K-major
// (row-major with K contiguous), FP32 accumulation in tensor memory.  One CTA
// owns a 128-row tile of C and BN columns; K advances in 64-element chunks
// (one 128-byte swizzle atom of BF16).  All 128 threads copy a chunk of A and
// B from global memory straight into the 128B-swizzled K-major layout
// (cp.async, 16 bytes a copy) while the tensor core works on the previous
// chunk; one elected thread issues the four K=16 tcgen05.mma of a chunk and a
// tcgen05.commit onto the stage's mbarrier.  The epilogue reads the
// accumulator with tcgen05.ld (warp w owns TMEM lanes 32w..32w+31, i.e. rows
// of the tile) and applies one of:
//   BIAS_GELU_FAST  h = gelu(acc + b) with the hardware tanh: BF16 out
//   BIAS_OUT        y = (acc + b) * scale + shift: FP32 out, row- or column-major
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "kernel_setup.h"
#include "mlp.h"
#include "mlp_umma.cuh"

namespace marl {
namespace mlp {

constexpr int kGemmThreads = 128;

template <int BN, int EPI>
__global__ void __launch_bounds__(kGemmThreads) k_gemm(const __grid_constant__ GemmArgs a) {
    static_assert(BN % 16 == 0 && BN >= 16 && BN <= 256, "UMMA N for M=128");
    constexpr uint32_t kTmemCols = BN <= 32 ? 32 : (BN <= 64 ? 64 : (BN <= 128 ? 128 : 256));
    constexpr uint32_t kStageA = kBM * 128;
    constexpr uint32_t kStageB = BN * 128;
    constexpr uint32_t kStage = kStageA + kStageB;
    extern __shared__ uint8_t gsm_raw[];
    __shared__ uint64_t bars[2];
    __shared__ uint32_t tmem_slot;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(gsm_raw) + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment
    const int m0 = blockIdx.x * kBM;
    const int n0 = blockIdx.y * BN;
    const int nch = a.K / kBK;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    constexpr uint32_t idesc = idesc_bf16(kBM, BN);

    bool ok = true;
    for (int c = 0; c < nch; ++c) {
        const int s = c & 1;
        if (c >= 2) ok = wait_commit(&bars[s], ((c - 2) >> 1) & 1, a.err) && ok;
        const uint32_t sa = base + s * kStage, sb = sa + kStageA;
        const int k0 = c * kBK;
        // A: 128 rows x 8 pieces of 16 bytes; rows beyond M are zero-filled.
#pragma unroll
        for (int i = 0; i < (kBM * 8) / kGemmThreads; ++i) {
            const int p = tid + i * kGemmThreads, r = p >> 3, q = p & 7;
            const int m = m0 + r;
            const bool in = m < a.M;
            const __nv_bfloat16* src = a.A + (size_t)(in ? m : 0) * a.lda + k0 + q * 8;
            cp_async16_zfill(sa + r * 128 + ((q ^ (r & 7)) << 4), src, in ? 16u : 0u);
        }
#pragma unroll
        for (int i = 0; i < (BN * 8 + kGemmThreads - 1) / kGemmThreads; ++i) {
            const int p = tid + i * kGemmThreads;
            if (p < BN * 8) {
                const int r = p >> 3, q = p & 7;
                const __nv_bfloat16* src = a.B + (size_t)(n0 + r) * a.ldb + k0 + q * 8;
                cp_async16_zfill(sb + r * 128 + ((q ^ (r & 7)) << 4), src, 16u);
            }
        }
        cp_async_commit_wait_all();
        fence_proxy_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk)
                umma_bf16(tmem, sw128_desc(sa + kk * 32), sw128_desc(sb + kk * 32), idesc, (c > 0 || kk > 0) ? 1u : 0u);
            umma_commit(&bars[s]);
        }
    }
    if (nch > 0) ok = wait_commit(&bars[(nch - 1) & 1], ((nch - 1) >> 1) & 1, a.err) && ok;
    tc_fence_after();

    const int row = m0 + warp * 32 + lane;
    const bool row_ok = row < a.M && ok && nch > 0;
    const uint32_t t_lane = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
    for (int cb = 0; cb < BN; cb += 16) {
        float v[16];
        tmem_ld16(t_lane + cb, v);
        const int n = n0 + cb;
        if constexpr (EPI == EPI_BIAS_GELU_FAST) {
            float h[16];
#pragma unroll
            for (int i = 0; i < 16; i += 2)
                gelu_fast2(pair_f32(v[i], v[i + 1]), pair_f32(a.bias[n + i], a.bias[n + i + 1]), h[i], h[i + 1]);
            if (row_ok) {
                uint4* o = reinterpret_cast<uint4*>(a.out_bf + (size_t)row * a.ldo + n);
                o[0] = make_uint4(pack_bf16(h[0], h[1]), pack_bf16(h[2], h[3]), pack_bf16(h[4], h[5]),
                                  pack_bf16(h[6], h[7]));
                o[1] = make_uint4(pack_bf16(h[8], h[9]), pack_bf16(h[10], h[11]), pack_bf16(h[12], h[13]),
                                  pack_bf16(h[14], h[15]));
            }
        } else if constexpr (EPI == EPI_BIAS_OUT) {
            if (row_ok) {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float y = v[i] + a.bias[n + i];
                    if (a.scale) y = y * a.scale[n + i] + a.shift[n + i];
                    if (a.out_col_major)
                        a.out_f[(size_t)(n + i) * a.ldf + row] = y;
                    else
                        a.out_f[(size_t)row * a.ldf + n + i] = y;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

template <int BN, int EPI>
static cudaError_t launch_one(const GemmArgs& a, cudaStream_t s) {
    constexpr int smem = 2 * (kBM * 128 + BN * 128) + 1024;
    static std::atomic<int> setup[kSetupDevices];
    cudaError_t e = set_smem_once(setup, k_gemm<BN, EPI>, smem);
    if (e != cudaSuccess) return e;
    dim3 grid((a.M + kBM - 1) / kBM, a.N / BN);
    k_gemm<BN, EPI><<<grid, kGemmThreads, smem, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_gemm(const GemmArgs& a, int bn, int epi, cudaStream_t s) {
    if (a.M <= 0 || a.K <= 0 || a.K % kBK || a.N % bn || a.lda % 8 || a.ldb % 8) return cudaErrorInvalidValue;
    if (bn == 256 && epi == EPI_BIAS_GELU_FAST) return launch_one<256, EPI_BIAS_GELU_FAST>(a, s);
    if (bn == 16 && epi == EPI_BIAS_OUT) return launch_one<16, EPI_BIAS_OUT>(a, s);
    return cudaErrorInvalidValue;
}

// ------------------------------------------------------- fused inference --
// The whole forward pass in one persistent kernel: one CTA per SM (16 warps)
// walks 128-row tiles.  All weights stay in shared memory for the kernel's
// life (W1 256 x 128, W2 256 x 256, W3 16 x 256: 200 KB, 128B-swizzled).  The
// activations never leave the SM: a tile's inputs and hidden layers live in
// tensor memory as BF16 and feed the next MMA as its A operand straight from
// tensor memory (the TS form of tcgen05.mma; A is row-per-lane, two BF16 per
// 32-bit column, lower k in the low half).  Tensor-memory columns: 0-255 the
// FP32 accumulator of layers 1 and 2, 256-383 the first hidden layer (BF16),
// 384-447 the inputs (BF16), 448-463 the accumulator of layer 3; the second
// hidden layer overwrites the accumulator it comes from, each warp its own 64
// columns (once it has read them all).
//
// What bounds it: 512 hardware tanh a row, 34 us for 300,000 rows on the MUFU
// pipes, against 26 us of tensor-core time.  Each hidden layer is two MMAs of
// 128 columns with a commit each, and two groups of eight warps: while a group
// takes the activations of the first half, the tensor core works on the
// second.  Warp w owns TMEM lanes 32 (w % 4).. (tile rows) and 64 columns, read
// in two 32-column loads that are both in flight before the first is used.  The
// next tile's inputs are read from global memory into registers during
// epilogue 1 and stored to tensor memory while layer 2 runs; its layer 1 is
// issued before the output of this tile is written.
// 300,000 rows: 144 us with one 256-column MMA a layer, 8 warps and scalar
// activation arithmetic.
constexpr int kFusedThreads = 512;
constexpr uint32_t kFW1 = kHid * kInPad * 2;   // 64 KB
constexpr uint32_t kFW2 = kHid * kHid * 2;     // 128 KB
constexpr uint32_t kFW3 = kOut * kHid * 2;     // 8 KB
constexpr uint32_t kFusedSmem = kFW1 + kFW2 + kFW3 + 1024;
constexpr uint32_t kTAcc = 0, kTH = 256, kTX = 384, kTAcc3 = 448;

// Copies rows [0, R) x K (K a multiple of 64) of a row-major BF16 matrix
// into 128B-swizzled K-major atoms of R rows each.
__device__ __forceinline__ void load_sw128(uint32_t dst, const __nv_bfloat16* src, int ld, int R, int K, int tid,
                                           int nthreads) {
    const int pieces = (K / 64) * R * 8;
    for (int p = tid; p < pieces; p += nthreads) {
        const int a = p / (R * 8), rem = p % (R * 8), r = rem >> 3, q = rem & 7;
        cp_async16_zfill(dst + a * R * 128 + r * 128 + ((q ^ (r & 7)) << 4), src + (size_t)r * ld + a * 64 + q * 8,
                         16u);
    }
}

__device__ __forceinline__ void umma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Row `row` of the inputs, K quarter `part` (32 BF16 = 16 TMEM columns), read
// into registers; zeros beyond M.
__device__ __forceinline__ void load_x_part(const __nv_bfloat16* x, int M, int row, int part, uint32_t (&r)[16]) {
    if (row < M) {
        const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)row * kInPad + part * 32);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 v = __ldg(src + i);
            r[4 * i] = v.x, r[4 * i + 1] = v.y, r[4 * i + 2] = v.z, r[4 * i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = 0u;
    }
}

// Epilogue of a hidden layer: 64 columns of the accumulator from `from` ->
// gelu(acc + bias) -> 32 columns of BF16 pairs at `to` (which may be the same
// columns: all are read first).  `bias` is in shared memory, 16-byte aligned.
__device__ __forceinline__ void hidden_epilogue(uint32_t from, uint32_t to, const float* bias) {
    uint32_t r[2][32];
    tmem_ld32_issue(from, r[0]);
    tmem_ld32_issue(from + 32, r[1]);
    tmem_ld_wait();
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 bb = reinterpret_cast<const float4*>(bias)[8 * b + i];
            const uint32_t* v = &r[b][4 * i];
            float h0, h1, h2, h3;
            gelu_fast2(pair_f32(__uint_as_float(v[0]), __uint_as_float(v[1])), pair_f32(bb.x, bb.y), h0, h1);
            gelu_fast2(pair_f32(__uint_as_float(v[2]), __uint_as_float(v[3])), pair_f32(bb.z, bb.w), h2, h3);
            w[2 * i] = pack_bf16(h0, h1);
            w[2 * i + 1] = pack_bf16(h2, h3);
        }
        tmem_st16(to + 16 * b, w);
    }
}

__global__ void __launch_bounds__(kFusedThreads, 1) k_mlp_fused(FusedArgs a) {
    extern __shared__ uint8_t fsm_raw[];
    __shared__ uint64_t bars[5];  // layer 1 halves, layer 2 halves, layer 3
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) float sb1[kHid], sb2[kHid], sb3[kOut], sscale[kOut], sshift[kOut];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(fsm_raw) + 1023u) & ~1023u;
    const uint32_t sW1 = base, sW2 = sW1 + kFW1, sW3 = sW2 + kFW2;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < 5; ++i) mbar_init(&bars[i], 1);
        fence_mbar_init();
    }
    load_sw128(sW1, a.w1, kInPad, kHid, kInPad, tid, kFusedThreads);
    load_sw128(sW2, a.w2, kHid, kHid, kHid, tid, kFusedThreads);
    load_sw128(sW3, a.w3, kHid, kOut, kHid, tid, kFusedThreads);
    for (int i = tid; i < kHid; i += kFusedThreads) sb1[i] = a.b1[i], sb2[i] = a.b2[i];
    if (tid < kOut) sb3[tid] = a.b3[tid], sscale[tid] = a.scale[tid], sshift[tid] = a.shift[tid];
    const int quarter = warp & 3, part = warp >> 2;  // tile rows; columns 64 part .. 64 part + 63
    const int half = part >> 1;
    const int ntiles = (a.M + kBM - 1) / kBM;
    int tile = blockIdx.x;
    uint32_t xr[16];
    load_x_part(a.x, a.M, tile * kBM + quarter * 32 + lane, part, xr);
    cp_async_commit_wait_all();
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t t_lane = tmem + ((uint32_t)(quarter * 32) << 16);
    constexpr uint32_t idesc = idesc_bf16(kBM, kHid / 2);
    // One half of a hidden layer: columns [128 h, +128) of the accumulator.
    auto layer1 = [&](int h) {
#pragma unroll
        for (int k = 0; k < kInPad / 16; ++k)
            umma_bf16_ts(tmem + kTAcc + h * 128, tmem + kTX + k * 8,
                         sw128_desc(sW1 + (k >> 2) * kHid * 128 + h * 128 * 128 + (k & 3) * 32), idesc, k > 0 ? 1u : 0u);
        umma_commit(&bars[h]);
    };
    auto layer2 = [&](int h) {
#pragma unroll
        for (int k = 0; k < kHid / 16; ++k)
            umma_bf16_ts(tmem + kTAcc + h * 128, tmem + kTH + k * 8,
                         sw128_desc(sW2 + (k >> 2) * kHid * 128 + h * 128 * 128 + (k & 3) * 32), idesc, k > 0 ? 1u : 0u);
        umma_commit(&bars[2 + h]);
    };
    bool ok = true;
    uint32_t it = 0;
    tmem_st16(t_lane + kTX + part * 16, xr);
    tmem_st_wait();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
        tc_fence_after();
        layer1(0);
        layer1(1);
    }

    for (; tile < ntiles; tile += gridDim.x, ++it) {
        const int m0 = tile * kBM, next = tile + gridDim.x;
        ok = wait_commit(&bars[half], it & 1, a.err) && ok;
        tc_fence_after();
        if (next < ntiles) load_x_part(a.x, a.M, next * kBM + quarter * 32 + lane, part, xr);  // in flight
        hidden_epilogue(t_lane + kTAcc + part * 64, t_lane + kTH + part * 32, sb1 + part * 64);
        tmem_st_wait();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            layer2(0);
            layer2(1);
        }
        // The next tile's inputs go to tensor memory while layer 2 runs (both
        // halves of layer 1 are done with them: every warp has seen its own).
        if (next < ntiles) tmem_st16(t_lane + kTX + part * 16, xr);
        ok = wait_commit(&bars[2 + half], it & 1, a.err) && ok;
        tc_fence_after();
        hidden_epilogue(t_lane + kTAcc + part * 64, t_lane + kTAcc + part * 64, sb2 + part * 64);
        tmem_st_wait();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < kHid / 16; ++k)
                umma_bf16_ts(tmem + kTAcc3, tmem + kTAcc + (k >> 2) * 64 + (k & 3) * 8,
                             sw128_desc(sW3 + (k >> 2) * kOut * 128 + (k & 3) * 32), idesc_bf16(kBM, kOut),
                             k > 0 ? 1u : 0u);
            umma_commit(&bars[4]);
        }
        ok = wait_commit(&bars[4], it & 1, a.err) && ok;
        tc_fence_after();
        // Layer 3 is done with the hidden layer in the accumulator's columns, and
        // the next tile's inputs were stored before the barrier above.
        if (tid == 0 && next < ntiles) {
            layer1(0);
            layer1(1);
        }
        if (part == 3) {  // not the warp that issues
            float v[16];
            tmem_ld16(t_lane + kTAcc3, v);
            const int row = m0 + quarter * 32 + lane;
            if (row < a.M && ok) {
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    a.y[(size_t)i * a.ldy + row] = (v[i] + sb3[i]) * sscale[i] + sshift[i];
            }
        }
        // The accumulator of layer 3 is read before the barriers of the next
        // tile, and so before it is written again.
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

cudaError_t launch_mlp_fused(const FusedArgs& a, int num_sms, cudaStream_t s) {
    if (a.M <= 0) return cudaSuccess;
    static std::atomic<int> setup[kSetupDevices];
    cudaError_t e = set_smem_once(setup, k_mlp_fused, kFusedSmem);
    if (e != cudaSuccess) return e;
    const int ntiles = (a.M + kBM - 1) / kBM;
    k_mlp_fused<<<ntiles < num_sms ? ntiles : num_sms, kFusedThreads, kFusedSmem, s>>>(a);
    return cudaGetLastError();
}

// --------------------------------------------------- standardisation ----
// Sums and sums of squares (FP64) of the transformed features and the
// targets over raw rows [0, n): acc[0..109) sums, acc[109..218) squares.
__global__ void k_raw_stats(const float* __restrict__ raw, uint32_t n, double* __restrict__ acc) {
    constexpr int kCols = kIn + kOut;
    __shared__ double s[2 * kCols];
    for (int i = threadIdx.x; i < 2 * kCols; i += blockDim.x) s[i] = 0.0;
    __syncthreads();
    const int col = threadIdx.x % 128;
    if (col < kCols) {
        double sum = 0.0, sq = 0.0;
        for (uint32_t r = blockIdx.x * (blockDim.x / 128) + threadIdx.x / 128; r < n;
             r += gridDim.x * (blockDim.x / 128)) {
            float v = raw[(size_t)r * MARL_SURR_RAW_STRIDE + col];
            if (col < kIn) v = feature_transform(col, v);
            sum += v;
            sq += (double)v * v;
        }
        atomicAdd(&s[col], sum);
        atomicAdd(&s[kCols + col], sq);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * kCols; i += blockDim.x) atomicAdd(&acc[i], s[i]);
}

cudaError_t launch_raw_stats(const float* raw, uint32_t n, double* acc, cudaStream_t s) {
    k_raw_stats<<<296, 512, 0, s>>>(raw, n, acc);
    return cudaGetLastError();
}

// Standardised BF16 inputs [n][128] and FP32 targets [n][16] from raw rows.
// norm: in_mean[93], in_std[93], out_mean[16], out_std[16].
__global__ void k_standardise(const float* __restrict__ raw, uint32_t n, const float* __restrict__ norm,
                              __nv_bfloat16* __restrict__ X, float* __restrict__ T) {
    const uint32_t r = blockIdx.x;
    if (r >= n) return;
    const int i = threadIdx.x;  // 0..127
    const float* row = raw + (size_t)r * MARL_SURR_RAW_STRIDE;
    float v = 0.0f;
    if (i < kIn) v = (feature_transform(i, row[i]) - norm[i]) / norm[kIn + i];
    X[(size_t)r * kInPad + i] = __float2bfloat16_rn(v);
    if (i < kOut) T[(size_t)r * kOut + i] = (row[kIn + i] - norm[2 * kIn + i]) / norm[2 * kIn + kOut + i];
}

cudaError_t launch_standardise(const float* raw, uint32_t n, const float* norm, __nv_bfloat16* X, float* T,
                               cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_standardise<<<n, kInPad, 0, s>>>(raw, n, norm, X, T);
    return cudaGetLastError();
}

// Normwise relative error of x_T + prediction against x_T + plain deltas, per
// row, accumulated: err_out[r], and acc = {accepted count, sum err, max err
// bits, squared error of standardised outputs}.
__global__ void k_eval_rows(const float* __restrict__ raw, const float* __restrict__ pred, uint32_t ldp, uint32_t n,
                            const float* __restrict__ norm, float tol, float c_max, float* __restrict__ err_out,
                            double* __restrict__ acc, uint32_t* __restrict__ max_bits) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const float* row = raw + (size_t)r * MARL_SURR_RAW_STRIDE;
    float num = 0.0f, den = 0.0f, se = 0.0f;
    for (int k = 0; k < kOut; ++k) {
        const float xt = row[k];
        const float plain = xt + row[kIn + k];
        const float d = pred[(size_t)k * ldp + r];
        const float mlp = fminf(fmaxf(xt + d, 0.0f), c_max);
        num = fmaxf(num, fabsf(mlp - plain));
        den = fmaxf(den, fabsf(plain));
        const float e = (d - row[kIn + k]) / norm[2 * kIn + kOut + k];
        se += e * e;
    }
    const float err = num / fmaxf(den, 1e-6f);
    if (err_out) err_out[r] = err;
    atomicAdd(&acc[0], err <= tol ? 1.0 : 0.0);
    atomicAdd(&acc[1], (double)err);
    atomicAdd(&acc[2], (double)se);
    atomicMax(max_bits, __float_as_uint(err));
}

cudaError_t launch_eval_rows(const float* raw, const float* pred, uint32_t ldp, uint32_t n, const float* norm,
                             float tol, float c_max, float* err_out, double* acc, uint32_t* max_bits,
                             cudaStream_t s) {
    k_eval_rows<<<(n + 255) / 256, 256, 0, s>>>(raw, pred, ldp, n, norm, tol, c_max, err_out, acc, max_bits);
    return cudaGetLastError();
}

// Initial weights: uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) from a counter
// hash; W1 columns 93..127 and all biases zero.
__global__ void k_init_weights(float* __restrict__ p, uint64_t seed) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < kParams; i += gridDim.x * blockDim.x) {
        const double u = (double)(mix64(seed ^ mix64(i)) >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
        float v = 0.0f;
        if (i < kOffB1) {
            v = (i % kInPad) < kIn ? (float)(u / sqrt((double)kIn)) : 0.0f;
        } else if (i >= kOffW2 && i < kOffB2) {
            v = (float)(u / sqrt((double)kHid));
        } else if (i >= kOffW3 && i < kOffB3) {
            v = (float)(u / sqrt((double)kHid));
        }
        p[i] = v;
    }
}

cudaError_t launch_init_weights(float* p, uint64_t seed, cudaStream_t s) {
    k_init_weights<<<256, 256, 0, s>>>(p, seed);
    return cudaGetLastError();
}

}  // namespace mlp
}  // namespace marl
