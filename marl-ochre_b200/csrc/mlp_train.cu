// Training step of the reaction surrogate on the fifth-generation tensor cores:
// six kernels (forward 1, forward 2, output layer with the loss, two input
// gradients, all weight gradients) and Adam.
//
//   h1 = gelu(x W1^T + b1)      rows of x drawn from the prepared pairs
//   h2 = gelu(h1 W2^T + b2)
//   y  = h2 W3^T + b3;  dy = 2 (y - t) / (16 B);  loss, db3
//   dz2 = (dy W3) * gelu'(z2);  db2
//   dz1 = (dz2 W2) * gelu'(z1);  db1
//   dW2 = dz2^T h1, dW1 = dz1^T x, dW3 = dy^T h2   (split over the batch)
//
// Every sum over the batch leaves its kernel as partial sums (a split's weight
// tile, a row tile's bias and loss sums), which the last kernel adds in a
// fixed order: a run repeats bit for bit, and no gradient buffer has to be
// zeroed or accumulated into by atomics.
//
// What bounds a step is latency: 4.6 GFLOP at a batch of 8192 are 3 us of the
// tensor cores.  So each kernel spreads over as many SMs as the shape gives
// (128 x 128 tiles: 128 blocks a layer, 8 x 16 blocks for the weight
// gradients), has all its operand chunks in flight at once, and starts under
// the tail of the one before it (programmatic dependent launch).  No operand is
// transposed in memory: where a matrix is contracted over its rows, the tensor
// core reads it as it lies (operands contiguous in M or N, the descriptor's
// MN-major form).  The forward epilogues store gelu' from the tanh they have
// already taken, so the backward ones take none.  The batch is never copied:
// its rows are drawn by the loads that use them.
// A step at a batch of 8192 takes 62 us (46 at 1024); it took 347 (295) as 14
// kernels with transposed copies, shared-memory atomics in the loss (75 us) and
// 60-us input-gradient epilogues.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "kernel_setup.h"
#include "mlp.h"
#include "mlp_umma.cuh"

namespace marl {
namespace mlp {

constexpr int kTrThreads = 256;
constexpr int kTrN = 128;                  // columns of a block's tile
constexpr uint32_t kTile = kBM * 128;      // a staged 128 x 64 (or 64 x 128) BF16 operand: 16 KB
constexpr uint32_t kMnBlock = kBK * 128;   // 64 k-rows of 64 elements: the stride between MN-major blocks
constexpr int kTrStages = 4;

template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// Chunk of 64 k of `rows` rows (row r at src + at(r) * ld), K-major.
template <class At>
__device__ __forceinline__ void stage_k(uint32_t dst, const __nv_bfloat16* src, int ld, int rows, int k0, int pieces,
                                        At at) {
    for (int p = threadIdx.x; p < rows * pieces; p += kTrThreads) {
        const int r = p / pieces, q = p % pieces;
        cp_async16_zfill(dst + r * 128 + ((q ^ (r & 7)) << 4), src + (size_t)at(r) * ld + k0 + q * 8, 16u);
    }
}

// Rows at(0..krows-1) of a row-major matrix as k, columns n0 .. n0 + 8 pieces - 1
// as the operand's M or N: MN-major, blocks of 64 columns.
template <class At>
__device__ __forceinline__ void stage_mn(uint32_t dst, const __nv_bfloat16* src, int ld, int krows, int n0, int pieces,
                                         At at) {
    for (int p = threadIdx.x; p < krows * pieces; p += kTrThreads) {
        const int r = p / pieces, q = p % pieces;
        cp_async16_zfill(dst + (q >> 3) * kMnBlock + r * 128 + (((q & 7) ^ (r & 7)) << 4),
                         src + (size_t)at(r) * ld + n0 + q * 8, 16u);
    }
}

struct TrSetup {
    uint32_t tmem, base;
};

// Tensor memory (kTrN columns), `bars` barriers, 1024-byte aligned staging.
__device__ __forceinline__ TrSetup tr_setup(uint8_t* raw, uint64_t* bars, int n_bars, uint32_t* slot) {
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                     "r"((uint32_t)kTrN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < n_bars; ++i) mbar_init(&bars[i], 1);
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    return TrSetup{*slot, (smem_u32(raw) + 1023u) & ~1023u};
}

__device__ __forceinline__ void tr_teardown(uint32_t tmem) {
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kTrN)
                     : "memory");
}

// Sums of v[0..15] over the warp's 32 lanes: 16 exchanges that halve what a lane
// still carries.  Lanes with bit 0 clear return column (lane >> 1)'s sum.
__device__ __forceinline__ float column_sums16(float (&v)[16], int lane) {
#pragma unroll
    for (int half = 8, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
        const bool up = lane & bit;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float give = up ? v[i] : v[i + half];
            const float keep = up ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, give, bit);
        }
    }
    return v[0] + __shfl_xor_sync(0xFFFFFFFFu, v[0], 1);
}

__device__ __forceinline__ void store_bf16x16(__nv_bfloat16* dst, const float (&h)[16]) {
    uint4* o = reinterpret_cast<uint4*>(dst);
    o[0] = make_uint4(pack_bf16(h[0], h[1]), pack_bf16(h[2], h[3]), pack_bf16(h[4], h[5]), pack_bf16(h[6], h[7]));
    o[1] = make_uint4(pack_bf16(h[8], h[9]), pack_bf16(h[10], h[11]), pack_bf16(h[12], h[13]),
                      pack_bf16(h[14], h[15]));
}

// Batch row r's prepared row.
__device__ __forceinline__ uint32_t drawn_row(const TrainArgs& a, uint32_t r) {
    return a.n_rows ? (uint32_t)(mix64(a.seed ^ mix64(a.step * 0x100000001B3ull + r)) % a.n_rows) : r;
}

enum TrRows : int { TR_FORWARD1, TR_FORWARD2, TR_LOSS, TR_BACK2, TR_BACK1 };

// One layer over the batch's rows: a block owns 128 rows and N columns, with all
// K (16, 128 or 256) staged at once, a commit group per chunk.  Eight warps:
// warp w reads tensor-memory lanes 32 (w % 4).. (tile rows) and the column half
// w / 4.
template <int KIND>
__global__ void __launch_bounds__(kTrThreads) k_train_rows(const __grid_constant__ TrainArgs a) {
    constexpr bool kFwd = KIND == TR_FORWARD1 || KIND == TR_FORWARD2;
    constexpr bool kBack = KIND == TR_BACK1 || KIND == TR_BACK2;
    constexpr int N = KIND == TR_LOSS ? kOut : kTrN;
    constexpr int K = KIND == TR_FORWARD1 ? kInPad : (KIND == TR_BACK2 ? kOut : kHid);
    constexpr int kChunks = K < kBK ? 1 : K / kBK;
    constexpr int kSteps = (K < kBK ? K : kBK) / 16;  // MMAs a chunk
    extern __shared__ uint8_t raw[];
    __shared__ uint64_t bar;
    __shared__ uint32_t slot;
    __shared__ uint32_t s_idx[kBM];
    __shared__ float s_col[4][kTrN], s_bias[kTrN], s_loss[4];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * N;
    const TrSetup t = tr_setup(raw, &bar, 1, &slot);
    constexpr uint32_t kStage = 2 * kTile;
    auto sa = [&](int c) { return t.base + c * kStage; };
    auto sb = [&](int c) { return t.base + c * kStage + kTile; };
    auto self = [](int r) { return r; };

    // Weights and biases were written by Adam before the kernel in front of
    // this one began (each waits for its predecessor before it lets the next
    // start), so they are staged ahead of the wait; forward 1 follows Adam
    // itself.
    auto stage_b = [&](int c) {
        if constexpr (KIND == TR_FORWARD1)
            stage_k(sb(c), a.w1 + (size_t)n0 * kInPad, kInPad, N, c * kBK, 8, self);
        else if constexpr (KIND == TR_FORWARD2)
            stage_k(sb(c), a.w2 + (size_t)n0 * kHid, kHid, N, c * kBK, 8, self);
        else if constexpr (KIND == TR_LOSS)
            stage_k(sb(c), a.w3, kHid, N, c * kBK, 8, self);
        else if constexpr (KIND == TR_BACK2)
            stage_mn(sb(c), a.w3, kHid, kOut, n0, 16, self);
        else
            stage_mn(sb(c), a.w2 + (size_t)c * kBK * kHid, kHid, kBK, n0, 16, self);
    };
    auto stage_a = [&](int c) {
        if constexpr (KIND == TR_FORWARD1)
            stage_k(sa(c), a.X, kInPad, kBM, c * kBK, 8, [&](int r) { return s_idx[r]; });
        else if constexpr (KIND == TR_BACK2)
            stage_k(sa(c), a.dy + (size_t)m0 * kOut, kOut, kBM, 0, 2, self);
        else
            stage_k(sa(c), (KIND == TR_FORWARD2 ? a.h1 : (KIND == TR_LOSS ? a.h2 : a.dz2)) + (size_t)m0 * kHid, kHid,
                    kBM, c * kBK, 8, self);
    };
    const float* bias = a.p + (KIND == TR_FORWARD1 ? kOffB1 : (KIND == TR_FORWARD2 ? kOffB2 : kOffB3));
    if constexpr (KIND == TR_FORWARD1) {
        if (tid < kBM) s_idx[tid] = drawn_row(a, (uint32_t)(m0 + tid));
        griddep_wait();
        griddep_launch_dependents();
        if (tid < kBM && blockIdx.y == 0) a.idx[m0 + tid] = s_idx[tid];
        __syncthreads();
    } else {
#pragma unroll
        for (int c = 0; c < kChunks; ++c) stage_b(c);
        griddep_wait();
        griddep_launch_dependents();
    }
    if constexpr (!kBack)
        if (tid < N) s_bias[tid] = bias[n0 + tid];
    float* const part = a.row_part + (size_t)blockIdx.x * kTrRowSums;
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
        if constexpr (KIND == TR_FORWARD1) stage_b(c);
        stage_a(c);
        cp_async_commit_group();
    }
    constexpr uint32_t idesc = idesc_bf16(kBM, N) | (kBack ? kIdescBMn : 0u);
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
        if (c == 0) cp_async_wait<kChunks - 1>();
        if (c == 1) cp_async_wait<(kChunks > 2 ? kChunks - 2 : 0)>();
        if (c == 2) cp_async_wait<(kChunks > 3 ? kChunks - 3 : 0)>();
        if (c == 3) cp_async_wait<0>();
        fence_proxy_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < kSteps; ++kk)
                umma_bf16(t.tmem, sw128_desc(sa(c) + kk * 32),
                          kBack ? sw128_desc_mn(sb(c) + kk * 2048, kMnBlock) : sw128_desc(sb(c) + kk * 32), idesc,
                          (c > 0 || kk > 0) ? 1u : 0u);
            if (c == kChunks - 1) umma_commit(&bar);
        }
    }
    const bool ok = wait_commit(&bar, 0, a.err);
    tc_fence_after();

    const int quarter = warp & 3, half = warp >> 2;
    const int row = m0 + quarter * 32 + lane;
    const uint32_t t_lane = t.tmem + ((uint32_t)(quarter * 32) << 16);
    if constexpr (KIND == TR_LOSS) {
        if (half == 0) {
            float v[16], g[16];
            tmem_ld16(t_lane, v);
            const float4* tp = reinterpret_cast<const float4*>(a.T + (size_t)(a.n_rows ? a.idx[row] : row) * kOut);
            float4* yp = reinterpret_cast<float4*>(a.y + (size_t)row * kOut);
            const float sc = 2.0f / ((float)a.B * 16.0f);
            float loss = 0.0f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 tt = tp[q];
                const float y0 = v[4 * q] + s_bias[4 * q], y1 = v[4 * q + 1] + s_bias[4 * q + 1],
                            y2 = v[4 * q + 2] + s_bias[4 * q + 2], y3 = v[4 * q + 3] + s_bias[4 * q + 3];
                const float e0 = y0 - tt.x, e1 = y1 - tt.y, e2 = y2 - tt.z, e3 = y3 - tt.w;
                loss += e0 * e0 + e1 * e1 + e2 * e2 + e3 * e3;
                g[4 * q] = ok ? e0 * sc : 0.0f, g[4 * q + 1] = ok ? e1 * sc : 0.0f;
                g[4 * q + 2] = ok ? e2 * sc : 0.0f, g[4 * q + 3] = ok ? e3 * sc : 0.0f;
                yp[q] = make_float4(y0, y1, y2, y3);
            }
            store_bf16x16(a.dy + (size_t)row * kOut, g);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xFFFFFFFFu, loss, o);
            const float sum = column_sums16(g, lane);
            if (!(lane & 1)) s_col[quarter][lane >> 1] = sum;
            if (lane == 0) s_loss[quarter] = loss;
        }
        __syncthreads();
        if (tid < kOut) part[2 * kHid + tid] = (s_col[0][tid] + s_col[1][tid]) + (s_col[2][tid] + s_col[3][tid]);
        if (tid == kOut) part[2 * kHid + kOut] = (s_loss[0] + s_loss[1]) + (s_loss[2] + s_loss[3]);
    } else {
        __nv_bfloat16* out = KIND == TR_FORWARD1 ? a.h1 : (KIND == TR_FORWARD2 ? a.h2 : (KIND == TR_BACK2 ? a.dz2 : a.dz1));
        float* d = (KIND == TR_FORWARD1 || KIND == TR_BACK1) ? a.d1 : a.d2;
#pragma unroll 1
        for (int cb = half * (N / 2); cb < (half + 1) * (N / 2); cb += 16) {
            float v[16], h[16];
            const size_t at = (size_t)row * kHid + n0 + cb;
            float4* dp = reinterpret_cast<float4*>(d + at);
            if constexpr (kFwd) {
                tmem_ld16(t_lane + cb, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) h[i] = gelu_and_grad(v[i] + s_bias[cb + i], v[i]);
#pragma unroll
                for (int q = 0; q < 4; ++q) dp[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                store_bf16x16(out + at, h);
            } else {
                float4 dg[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) dg[q] = dp[q];
                tmem_ld16(t_lane + cb, v);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    h[4 * q] = ok ? v[4 * q] * dg[q].x : 0.0f, h[4 * q + 1] = ok ? v[4 * q + 1] * dg[q].y : 0.0f;
                    h[4 * q + 2] = ok ? v[4 * q + 2] * dg[q].z : 0.0f, h[4 * q + 3] = ok ? v[4 * q + 3] * dg[q].w : 0.0f;
                }
                store_bf16x16(out + at, h);
                const float sum = column_sums16(h, lane);
                if (!(lane & 1)) s_col[quarter][cb + (lane >> 1)] = sum;
            }
        }
        if constexpr (kBack) {
            __syncthreads();
            if (tid < N)
                part[(KIND == TR_BACK2 ? kHid : 0) + n0 + tid] =
                    (s_col[0][tid] + s_col[1][tid]) + (s_col[2][tid] + s_col[3][tid]);
        }
    }
    tr_teardown(t.tmem);
}

// The weight gradients: block (job, split) sums split_rows rows of the batch
// (chunks of 64 as K; 512 rows up to a batch of 16,384: 128 blocks at 8192) for
// a 128-row tile of a gradient.  Jobs 0-3: dW2's 128 x 128
// quarters; 4, 5: dW1's halves; 6, 7: dW3 transposed ([256][16]), by halves.
// Chunks stream through four stages.
constexpr int kTrJobs = 8;
constexpr uint32_t kTrSmem = kTrStages * 2 * kTile + 1024;

__global__ void __launch_bounds__(kTrThreads) k_train_weights(const __grid_constant__ TrainArgs a) {
    extern __shared__ uint8_t raw[];
    __shared__ uint64_t bars[kTrStages];
    __shared__ uint32_t slot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int job = blockIdx.x;
    const TrSetup t = tr_setup(raw, bars, kTrStages, &slot);
    griddep_wait();
    griddep_launch_dependents();
    const int per = (int)(a.split_rows / kBK), c0 = (int)blockIdx.y * per, c1 = min(c0 + per, (int)(a.B / kBK));
    float* const sums = a.weight_part + (size_t)blockIdx.y * kParams;
    const int mt = job < 4 ? job >> 1 : job & 1;
    const bool last_layer = job >= 6, first_layer = job == 4 || job == 5;
    const __nv_bfloat16* A = (first_layer ? a.dz1 : (last_layer ? a.h2 : a.dz2)) + mt * kBM;
    auto stage = [&](int c) {
        const uint32_t sa = t.base + (uint32_t)((c - c0) & (kTrStages - 1)) * 2 * kTile, sb = sa + kTile;
        const int r0 = c * kBK;
        auto rows = [&](int r) { return r0 + r; };
        stage_mn(sa, A, kHid, kBK, 0, 16, rows);
        if (last_layer)
            stage_mn(sb, a.dy, kOut, kBK, 0, 2, rows);
        else if (first_layer)
            stage_mn(sb, a.X, kInPad, kBK, 0, 16, [&](int r) { return a.n_rows ? a.idx[r0 + r] : (uint32_t)(r0 + r); });
        else
            stage_mn(sb, a.h1, kHid, kBK, (job & 1) * kTrN, 16, rows);
    };
    const uint32_t idesc = (last_layer ? idesc_bf16(kBM, kOut) : idesc_bf16(kBM, kTrN)) | kIdescAMn | kIdescBMn;
    bool ok = true;
    // Three chunks ahead; a commit group per chunk, empty ones past the end.
    for (int c = c0; c < c0 + kTrStages - 1; ++c) {
        if (c < c1) stage(c);
        cp_async_commit_group();
    }
    for (int c = c0; c < c1; ++c) {
        const int s = (c - c0) & (kTrStages - 1);
        cp_async_wait<kTrStages - 2>();
        fence_proxy_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const uint32_t sa = t.base + (uint32_t)s * 2 * kTile, sb = sa + kTile;
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk)
                umma_bf16(t.tmem, sw128_desc_mn(sa + kk * 2048, kMnBlock), sw128_desc_mn(sb + kk * 2048, kMnBlock), idesc,
                          (c > c0 || kk > 0) ? 1u : 0u);
            umma_commit(&bars[s]);
        }
        // The stage that chunk c + 3 goes to was chunk c - 1's.
        const int next = c + kTrStages - 1;
        if (next < c1) {
            if (c > c0) ok = wait_commit(&bars[(s + kTrStages - 1) & (kTrStages - 1)], ((c - 1 - c0) / kTrStages) & 1, a.err) && ok;
            stage(next);
        }
        cp_async_commit_group();
    }
    if (c1 > c0) {
        const int l = c1 - 1 - c0;
        ok = wait_commit(&bars[l & (kTrStages - 1)], (l / kTrStages) & 1, a.err) && ok;
        tc_fence_after();
        const int quarter = warp & 3, half = warp >> 2;
        const int m = mt * kBM + quarter * 32 + lane;
        const uint32_t t_lane = t.tmem + ((uint32_t)(quarter * 32) << 16);
        if (last_layer) {
            if (half == 0) {
                float v[16];
                tmem_ld16(t_lane, v);
#pragma unroll
                for (int i = 0; i < kOut; ++i) sums[kOffW3 + (size_t)i * kHid + m] = ok ? v[i] : 0.0f;
            }
        } else {
            float* out = sums + (first_layer ? kOffW1 + (size_t)m * kInPad
                                             : kOffW2 + (size_t)m * kHid + (job & 1) * kTrN);
#pragma unroll 1
            for (int cb = half * (kTrN / 2); cb < (half + 1) * (kTrN / 2); cb += 16) {
                float v[16];
                tmem_ld16(t_lane + cb, v);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    reinterpret_cast<float4*>(out + cb)[q] =
                        ok ? make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3])
                           : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
    }
    tr_teardown(t.tmem);
}
static_assert(kOffW1 % 4 == 0 && kOffW2 % 4 == 0 && kParams % 4 == 0, "four-wide stores");

template <int KIND>
static cudaError_t launch_rows(const TrainArgs& a, cudaStream_t s) {
    constexpr int chunks = KIND == TR_FORWARD1 ? kInPad / kBK : (KIND == TR_BACK2 ? 1 : kHid / kBK);
    constexpr int smem = chunks * 2 * kTile + 1024;
    static std::atomic<int> setup[kSetupDevices];
    cudaError_t e = set_smem_once(setup, k_train_rows<KIND>, smem);
    if (e != cudaSuccess) return e;
    return launch_dependent(k_train_rows<KIND>, dim3(a.B / kBM, KIND == TR_LOSS ? 1 : kHid / kTrN), dim3(kTrThreads),
                            smem, s, a);
}

cudaError_t launch_forward_backward(const TrainArgs& a, cudaStream_t s) {
    if (a.B == 0 || a.B % kBM) return cudaErrorInvalidValue;
    cudaError_t e = launch_rows<TR_FORWARD1>(a, s);
    if (e == cudaSuccess) e = launch_rows<TR_FORWARD2>(a, s);
    if (e == cudaSuccess) e = launch_rows<TR_LOSS>(a, s);
    if (e == cudaSuccess) e = launch_rows<TR_BACK2>(a, s);
    if (e == cudaSuccess) e = launch_rows<TR_BACK1>(a, s);
    if (e != cudaSuccess) return e;
    static std::atomic<int> setup[kSetupDevices];
    if ((e = set_smem_once(setup, k_train_weights, kTrSmem)) != cudaSuccess) return e;
    const unsigned splits = train_splits(a.B, a.split_rows);
    return launch_dependent(k_train_weights, dim3(kTrJobs, splits), dim3(kTrThreads), kTrSmem, s, a);
}

// ------------------------------------------------- gradients and Adam ----
// The BF16 copies of the parameters that the tensor cores read.
__device__ __forceinline__ void put_bf16(uint32_t i, float v, __nv_bfloat16* w1, __nv_bfloat16* w2, __nv_bfloat16* w3) {
    const __nv_bfloat16 b = __float2bfloat16_rn(v);
    if (i < kOffB1)
        w1[i] = b;
    else if (i >= kOffW2 && i < kOffB2)
        w2[i - kOffW2] = b;
    else if (i >= kOffW3 && i < kOffB3)
        w3[i - kOffW3] = b;
}

// Adds the partial sums of gradient i (thread i for a weight, a warp for each of
// the 528 biases and the loss) in a fixed order and, with ADAM, updates the FP32
// master parameter and its BF16 copy; without, writes the gradient.
struct AdamArgs {
    float *p, *m, *v;
    float lr, b1, b2, eps, bc1, bc2;
    __nv_bfloat16 *w1, *w2, *w3;
};
constexpr int kSumThreads = 256;
constexpr int kSumBlocksW = (kParams + kSumThreads - 1) / kSumThreads;
constexpr int kSumBlocksB = (kTrRowSums + kSumThreads / 32 - 1) / (kSumThreads / 32);

template <bool ADAM>
__global__ void __launch_bounds__(kSumThreads) k_train_update(const __grid_constant__ TrainArgs a, AdamArgs o,
                                                              uint32_t splits) {
    uint32_t i;
    bool owner = true;
    griddep_wait();
    griddep_launch_dependents();
    float sum = 0.0f;
    if (blockIdx.x < (unsigned)kSumBlocksW) {
        i = blockIdx.x * kSumThreads + threadIdx.x;
        const bool weight = i < kOffB1 || (i >= kOffW2 && i < kOffB2) || (i >= kOffW3 && i < kOffB3);
        if (!weight) return;
        const float* part = a.weight_part + i;
        uint32_t q = 0;
        for (; q + 8 <= splits; q += 8) {  // eight in flight, added as a tree
            float t[8];
#pragma unroll
            for (int d = 0; d < 8; ++d) t[d] = part[(size_t)(q + d) * kParams];
            sum += ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
        }
        for (; q < splits; ++q) sum += part[(size_t)q * kParams];
    } else {
        const uint32_t b = (blockIdx.x - kSumBlocksW) * (kSumThreads / 32) + (threadIdx.x >> 5);
        if (b >= (uint32_t)kTrRowSums) return;
        const uint32_t tiles = a.B / kBM;
        for (uint32_t q = threadIdx.x & 31; q < tiles; q += 32) sum += a.row_part[(size_t)q * kTrRowSums + b];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
        owner = (threadIdx.x & 31) == 0;
        if (b == kTrRowSums - 1) {
            if (owner) *a.loss_sum = sum;
            return;
        }
        i = b < (uint32_t)kHid ? kOffB1 + b : (b < 2u * kHid ? kOffB2 + b - kHid : kOffB3 + b - 2 * kHid);
    }
    if (!owner) return;
    const float gi = sum;
    if constexpr (ADAM) {
        const float mi = o.b1 * o.m[i] + (1.0f - o.b1) * gi;
        const float vi = o.b2 * o.v[i] + (1.0f - o.b2) * gi * gi;
        o.m[i] = mi;
        o.v[i] = vi;
        const float pi = o.p[i] - o.lr * (mi / o.bc1) / (sqrtf(vi / o.bc2) + o.eps);
        o.p[i] = pi;
        put_bf16(i, pi, o.w1, o.w2, o.w3);
    } else {
        a.g[i] = gi;
    }
}

__global__ void k_weights_bf16(const float* __restrict__ p, __nv_bfloat16* __restrict__ w1,
                               __nv_bfloat16* __restrict__ w2, __nv_bfloat16* __restrict__ w3) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < kParams; i += gridDim.x * blockDim.x)
        put_bf16(i, p[i], w1, w2, w3);
}

cudaError_t launch_train_update(const TrainArgs& a, float* p, float* m, float* v, float lr, float b1, float b2,
                                float eps, uint64_t t, __nv_bfloat16* w1, __nv_bfloat16* w2, __nv_bfloat16* w3,
                                cudaStream_t s) {
    const float bc1 = 1.0f - (float)pow((double)b1, (double)t);
    const float bc2 = 1.0f - (float)pow((double)b2, (double)t);
    return launch_dependent(k_train_update<true>, dim3(kSumBlocksW + kSumBlocksB), dim3(kSumThreads), 0, s, a,
                            AdamArgs{p, m, v, lr, b1, b2, eps, bc1, bc2, w1, w2, w3}, train_splits(a.B, a.split_rows));
}

cudaError_t launch_train_gradients(const TrainArgs& a, cudaStream_t s) {
    return launch_dependent(k_train_update<false>, dim3(kSumBlocksW + kSumBlocksB), dim3(kSumThreads), 0, s, a,
                            AdamArgs{}, train_splits(a.B, a.split_rows));
}

cudaError_t launch_weights_bf16(const float* p, __nv_bfloat16* w1, __nv_bfloat16* w2, __nv_bfloat16* w3,
                                cudaStream_t s) {
    k_weights_bf16<<<256, 256, 0, s>>>(p, w1, w2, w3);
    return cudaGetLastError();
}

}  // namespace mlp
}  // namespace marl
