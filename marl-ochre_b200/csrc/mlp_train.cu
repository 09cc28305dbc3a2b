// Training step of the reaction surrogate on the fifth-generation tensor cores, in
// three kernels: everything that goes row by row (three layers, loss, input
// gradients), all weight gradients, and Adam.
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
// tensor cores.  So each kernel spreads over as many SMs as the shape gives (128
// blocks at 8192 for the rows, 8 x 16 for the weight gradients), has its operand
// chunks in flight at once, and starts under the tail of the one before it
// (programmatic dependent launch).  No operand is transposed in memory: where a
// matrix is contracted over its rows, the tensor core reads it as it lies
// (operands contiguous in M or N, the descriptor's MN-major form).  The forward
// epilogues take gelu' from the tanh they have already taken, so the backward
// ones take none.  The batch is never copied: its rows are drawn by the loads that
// use them.
// In calls of 50 steps a step takes 32 us at a batch of 8192 (30 at 512, 200 at
// 65,536; in calls of 200 31, 29, 199).  With X and the
// moments read after the wait for the kernel before it took 34 (31, 201), with weights
// gathered 16 bytes a thread and a wait of the block pair before each overwrite it
// took 37 (34, 220), with rows instead of tile images 54 (50, 335), with a kernel
// per layer and direction 71 (55, 372), as 14 kernels with transposed copies and
// shared-memory atomics in the loss 347 at 8192.
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
constexpr uint32_t kImage = kTile;         // a tile's image in memory
constexpr uint32_t kMnBlock = kBK * 128;   // 64 k-rows of 64 elements: the stride between MN-major blocks
constexpr int kTrStages = 4;

template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// Chunk of 64 k of `rows` rows (row r at src + at(r) * ld), K-major.
template <int THREADS, class At>
__device__ __forceinline__ void stage_k(uint32_t dst, const __nv_bfloat16* src, int ld, int rows, int k0, int pieces,
                                        At at) {
    for (int p = threadIdx.x; p < rows * pieces; p += THREADS) {
        const int r = p / pieces, q = p % pieces;
        cp_async16_zfill(dst + r * 128 + ((q ^ (r & 7)) << 4), src + (size_t)at(r) * ld + k0 + q * 8, 16u);
    }
}

struct TrSetup {
    uint32_t tmem, base;
};

// Tensor memory (COLS columns), `bars` barriers, 1024-byte aligned staging.
template <uint32_t COLS>
__device__ __forceinline__ TrSetup tr_setup(uint8_t* raw, uint64_t* bars, int n_bars, uint32_t* slot) {
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                     "r"(COLS)
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

template <uint32_t COLS>
__device__ __forceinline__ void tr_teardown(uint32_t tmem) {
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS)
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

// Batch row r's prepared row.
__device__ __forceinline__ uint32_t drawn_row(const TrainArgs& a, uint32_t r) {
    return a.n_rows ? (uint32_t)(mix64(a.seed ^ mix64(a.step * 0x100000001B3ull + r)) % a.n_rows) : r;
}

// Everything of a step that goes row by row: three layers forward, the loss, two
// backward.  A cluster of two blocks owns 128 rows; each block computes 128 of a
// layer's 256 columns, so that 8192 rows are 128 blocks, and writes what the next
// layer reads (H1, then H2, then dZ2) into both blocks' shared memory.  The
// weights it needs are fetched once, in the order of their use, and gelu' of layers 1 and 2 stays
// in tensor memory.  What the weight gradients need leaves as images of the
// shared-memory tiles (128 rows of 64 columns, swizzled, 16 KB), one bulk copy
// each: k_train_weights loads halves of them (64 rows) the same way, and they are
// its operands as they are.  Stored row by row, 16 bytes a thread, they took 12
// wavefronts of 32 rows a thread and 6k cycles of an epilogue.
//
// 16 warps: warp w reads tensor-memory lanes 32 (w % 4).. (tile rows) and columns
// 32 (w / 4).. of its block's 128.
constexpr int kRowThreads = 512;
constexpr uint32_t kRowTmem = 512;              // columns 0-127 and 128-255: an accumulator each; 256-383: gelu' of layer 1
// Shared memory, each four chunks of 64 k.  What is written next goes where both
// blocks have finished by the exchange before it, so nothing else has to be waited for.
constexpr uint32_t kRowP = 0;                   // X and W1, then H2, then dZ1
constexpr uint32_t kRowQ = 4 * kTile;           // H1, then dZ2
constexpr uint32_t kRowW2 = 8 * kTile;          // W2's own rows (K-major), then its own columns (MN-major)
constexpr uint32_t kRowW3 = 12 * kTile;         // four chunks [16][64]: K-major forward, MN-major backward
constexpr uint32_t kRowW3Chunk = kOut * 128;
constexpr uint32_t kRowDy = kRowW3 + 4 * kRowW3Chunk;
constexpr uint32_t kRowSmem = kRowDy + kTile + 1024;

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_map(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_store(uint32_t addr, uint4 v) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}
// Asynchronous copies of whole tile images; sizes and addresses are multiples of 16.
__device__ __forceinline__ void image_store(void* dst, uint32_t src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void image_stores_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void image_stores_done() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void image_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// After an expired wait: waits (bounded) for the phase `parity` of a barrier that
// image_load()s arrive on, so that no copy lands in shared memory that another block
// may hold by then.
__device__ __forceinline__ void image_loads_drain(uint64_t* bar, uint32_t parity) { mbar_wait_bounded(bar, parity); }
// Generic writes (either block's shared memory) before asynchronous reads.
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kRowThreads, 1)
    k_train_rows(const __grid_constant__ TrainArgs a) {
    extern __shared__ uint8_t raw[];
    __shared__ uint64_t bars[5];
    __shared__ uint32_t slot;
    __shared__ uint32_t s_idx[kBM];
    __shared__ float s_col[2][4][kTrN], s_col3[4][kOut], s_b1[kTrN], s_b2[kTrN], s_b3[kOut], s_loss[4];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = blockIdx.x & 1u;
    const uint32_t tile = blockIdx.x >> 1;
    const int m0 = (int)tile * kBM, n0 = (int)rank * kTrN;
    const TrSetup t = tr_setup<kRowTmem>(raw, bars, 5, &slot);
    uint64_t &bar = bars[0], *const w_bar = bars + 1;  // products done; W1, W2's rows, W3, W2's columns have landed
    const uint32_t P = t.base + kRowP, Q = t.base + kRowQ, w2 = t.base + kRowW2, w3 = t.base + kRowW3,
                   dy = t.base + kRowDy, peer = cluster_map(t.base, rank ^ 1u) - t.base;
    cluster_arrive();  // this block has started: its shared memory may be written
    if (tid < kBM) s_idx[tid] = drawn_row(a, (uint32_t)(m0 + tid));
    __syncthreads();
    // X is gathered, a commit group per chunk, before the wait: no kernel that may
    // still be running writes it (whoever does ends with a synchronisation, or is a
    // copy, which this kernel does not overtake).
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        stage_k<kRowThreads>(P + c * kTile, a.X, kInPad, kBM, c * kBK, 8, [&](int r) { return s_idx[r]; });
        cp_async_commit_group();
    }
    griddep_wait();  // Adam's weights
    griddep_launch_dependents();
    if (tid == 0) {
        mbar_arrive_expect_tx(&w_bar[0], 2 * kTile);
        image_load(P + 2 * kTile, a.wi + rank * 2 * kImage, 2 * kTile, &w_bar[0]);
    }
    if (tid == 0) {
        mbar_arrive_expect_tx(&w_bar[1], 4 * kTile);
        image_load(w2, a.wi + (4 + rank * 4) * kImage, 4 * kTile, &w_bar[1]);
        mbar_arrive_expect_tx(&w_bar[2], 4 * kRowW3Chunk);
        image_load(w3, a.wi + 12 * kImage, 4 * kRowW3Chunk, &w_bar[2]);
    }
    if (tid < kTrN) s_b1[tid] = a.p[kOffB1 + n0 + tid], s_b2[tid] = a.p[kOffB2 + n0 + tid];
    if (tid < kOut) s_b3[tid] = a.p[kOffB3 + tid];

    const uint32_t d0 = t.tmem, d1 = t.tmem + kTrN, g1 = t.tmem + 2 * kTrN;  // the accumulators, gelu'
    const uint32_t idesc = idesc_bf16(kBM, kTrN), idesc_back = idesc | kIdescBMn;
    // Layer 1: X (128 k) by W1's own rows.
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        if (c == 0) cp_async_wait<1>();
        else cp_async_wait<0>();
        fence_proxy_async_smem();
        __syncthreads();
        if (tid == 0) {
            if (c == 0) wait_commit(&w_bar[0], 0, a.err);
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                umma_bf16(d0, sw128_desc(P + c * kTile + kk * 32), sw128_desc(P + (2 + c) * kTile + kk * 32), idesc,
                          (c > 0 || kk > 0) ? 1u : 0u);
            if (c == 1) umma_commit(&bar);
            if (c == (int)rank) image_store(a.xt + ((size_t)tile * 2 + c) * kImage, P + c * kTile, kTile);
        }
    }
    bool ok = wait_commit(&bar, 0, a.err);
    tc_fence_after();
    cluster_wait();

    const int quarter = warp & 3, c_lo = (warp >> 2) * 32;
    const int rl = quarter * 32 + lane;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    // 16 columns (from column `col` of 256) of this thread's row into the operand at
    // `to`, here and, where the next product needs all 256, in the other block.
    auto put = [&](uint32_t to, int col, const float (&h)[16], bool both) {
        to += (uint32_t)(col >> 6) * kTile + (uint32_t)rl * 128;
        const uint32_t q = (uint32_t)(col & 63) >> 3;
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i) {
            const uint4 v = make_uint4(pack_bf16(h[8 * i], h[8 * i + 1]), pack_bf16(h[8 * i + 2], h[8 * i + 3]),
                                       pack_bf16(h[8 * i + 4], h[8 * i + 5]), pack_bf16(h[8 * i + 6], h[8 * i + 7]));
            const uint32_t at = to + (((q + i) ^ ((uint32_t)rl & 7u)) << 4);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                         : "memory");
            if (both) cluster_store(at + peer, v);
        }
    };
    // This block's half of an operand to memory.
    auto store_half = [&](uint8_t* images, uint32_t from) {
        if (tid == 0) image_store(images + ((size_t)tile * 4 + 2 * rank) * kImage, from + 2 * rank * kTile, 2 * kTile);
    };
    // Before it, what both blocks have written, sent and had multiplied; after it, what uses that.
    auto exchange = [&]() {
        if (tid == 0) image_stores_read();
        fence_proxy_async_all();
        tc_fence_before();
        cluster_arrive();
        cluster_wait();
    };
    // D = A (256 k) by B's chunks.
    auto mma = [&](uint32_t d, uint32_t A, uint32_t idesc_n, uint64_t* landed, auto bdesc) {
        if (tid == 0) {
            wait_commit(landed, 0, a.err);
            fence_proxy_async_all();
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < 16; ++k)
                umma_bf16(d, sw128_desc(A + (k >> 2) * kTile + (k & 3) * 32), bdesc(k >> 2, k & 3), idesc_n, k > 0 ? 1u : 0u);
            umma_commit(&bar);
        }
    };
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int cb = c_lo + 16 * i;
        float v[16], h[16];
        tmem_ld16(d0 + lanes + cb, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) h[j] = gelu_and_grad(v[j] + s_b1[cb + j], v[j]);
        uint32_t g[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) g[j] = __float_as_uint(v[j]);
        tmem_st16(g1 + lanes + cb, g);
        put(Q, n0 + cb, h, true);
    }
    tmem_st_wait();
    exchange();
    // Layer 2: H1 by W2's own rows.
    mma(d1, Q, idesc, &w_bar[1], [&](int c, int kk) { return sw128_desc(w2 + c * kTile + kk * 32); });
    store_half(a.h1, Q);
    ok = wait_commit(&bar, 1, a.err) && ok;
    tc_fence_after();
    if (tid == 0) {  // W2's own columns, chunk c: its rows 64 c.., a half of two row images
        mbar_arrive_expect_tx(&w_bar[3], 4 * kTile);
#pragma unroll 1
        for (uint32_t c = 0; c < 4; ++c)
#pragma unroll
            for (uint32_t b = 0; b < 2; ++b)
                image_load(w2 + c * kTile + b * kMnBlock,
                           a.wi + (4 + (c >> 1) * 4 + 2 * rank + b) * kImage + (c & 1) * kMnBlock, kMnBlock, &w_bar[3]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int cb = c_lo + 16 * i;
        float v[16], h[16];
        uint32_t g[16];
        tmem_ld16(d1 + lanes + cb, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            float grad;
            h[j] = gelu_and_grad(v[j] + s_b2[cb + j], grad);
            g[j] = __float_as_uint(grad);
        }
        tmem_st16(d1 + lanes + cb, g);
        put(P, n0 + cb, h, true);
    }
    tmem_st_wait();
    exchange();
    // Layer 3 and the loss, in both blocks alike; the first one writes them.
    mma(d0, P, idesc_bf16(kBM, kOut), &w_bar[2], [&](int c, int kk) { return sw128_desc(w3 + c * kRowW3Chunk + kk * 32); });
    store_half(a.h2, P);
    float4 target[4];
    if (warp < 4) {
#pragma unroll
        for (int q = 0; q < 4; ++q) target[q] = reinterpret_cast<const float4*>(a.T + (size_t)s_idx[rl] * kOut)[q];
    }
    ok = wait_commit(&bar, 0, a.err) && ok;
    tc_fence_after();
    if (warp < 4) {
        float v[16], g[16];
        tmem_ld16(d0 + lanes, v);
        float4* yp = reinterpret_cast<float4*>(a.y + (size_t)(m0 + rl) * kOut);
        const float sc = 2.0f / ((float)a.B * 16.0f);
        float loss = 0.0f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 tt = target[q];
            const float y0 = v[4 * q] + s_b3[4 * q], y1 = v[4 * q + 1] + s_b3[4 * q + 1],
                        y2 = v[4 * q + 2] + s_b3[4 * q + 2], y3 = v[4 * q + 3] + s_b3[4 * q + 3];
            const float e0 = y0 - tt.x, e1 = y1 - tt.y, e2 = y2 - tt.z, e3 = y3 - tt.w;
            loss += e0 * e0 + e1 * e1 + e2 * e2 + e3 * e3;
            g[4 * q] = ok ? e0 * sc : 0.0f, g[4 * q + 1] = ok ? e1 * sc : 0.0f;
            g[4 * q + 2] = ok ? e2 * sc : 0.0f, g[4 * q + 3] = ok ? e3 * sc : 0.0f;
            if (rank == 0) yp[q] = make_float4(y0, y1, y2, y3);
        }
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dy + (uint32_t)rl * 128 +
                                                                          ((i ^ ((uint32_t)rl & 7u)) << 4)),
                         "r"(pack_bf16(g[8 * i], g[8 * i + 1])), "r"(pack_bf16(g[8 * i + 2], g[8 * i + 3])),
                         "r"(pack_bf16(g[8 * i + 4], g[8 * i + 5])), "r"(pack_bf16(g[8 * i + 6], g[8 * i + 7]))
                         : "memory");
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xFFFFFFFFu, loss, o);
        const float sum = column_sums16(g, lane);
        if (!(lane & 1)) s_col3[quarter][lane >> 1] = sum;
        if (lane == 0) s_loss[quarter] = loss;
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    float* const part = a.row_part + (size_t)(blockIdx.x >> 1) * kTrRowSums;
    // dH2's own columns: dY (16 k) by W3.
    if (tid == 0) {
        tc_fence_after();
        umma_bf16(d0, sw128_desc(dy), sw128_desc_mn(w3 + 2 * rank * kRowW3Chunk, kRowW3Chunk), idesc_back, 0u);
        umma_commit(&bar);
        if (rank == 0) image_store(a.dy + (size_t)tile * kImage, dy, kTile);
    }
    if (rank == 0 && tid < kOut)
        part[2 * kHid + tid] = (s_col3[0][tid] + s_col3[1][tid]) + (s_col3[2][tid] + s_col3[3][tid]);
    if (rank == 0 && tid == kOut) part[2 * kHid + kOut] = (s_loss[0] + s_loss[1]) + (s_loss[2] + s_loss[3]);
    ok = wait_commit(&bar, 1, a.err) && ok;
    tc_fence_after();
    // dZ = dH gelu'.
    auto back = [&](uint32_t d, uint32_t g, int cb, float (&h)[16]) {
        float v[16], dg[16];
        tmem_ld16(g + lanes + cb, dg);
        tmem_ld16(d + lanes + cb, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) h[j] = ok ? v[j] * dg[j] : 0.0f;
    };
    auto sums = [&](int which, int cb, float (&h)[16]) {
        const float sum = column_sums16(h, lane);
        if (!(lane & 1)) s_col[which][quarter][cb + (lane >> 1)] = sum;
    };
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int cb = c_lo + 16 * i;
        float h[16];
        back(d0, d1, cb, h);
        put(Q, n0 + cb, h, true);
        sums(0, cb, h);
    }
    exchange();
    // dH1's own columns: dZ2 by W2's columns.
    mma(d1, Q, idesc_back, &w_bar[3], [&](int c, int kk) { return sw128_desc_mn(w2 + c * kTile + kk * 2048, kMnBlock); });
    store_half(a.dz2, Q);
    if (tid < kTrN)
        part[kHid + n0 + tid] = (s_col[0][0][tid] + s_col[0][1][tid]) + (s_col[0][2][tid] + s_col[0][3][tid]);
    ok = wait_commit(&bar, 0, a.err) && ok;
    tc_fence_after();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int cb = c_lo + 16 * i;
        float h[16];
        back(d1, g1, cb, h);
        put(P, n0 + cb, h, false);
        sums(1, cb, h);
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (tid < kTrN) part[n0 + tid] = (s_col[1][0][tid] + s_col[1][1][tid]) + (s_col[1][2][tid] + s_col[1][3][tid]);
    store_half(a.dz1, P);
    if (tid == 0) image_stores_done();
    if (warp == kRowThreads / 32 - 1 && lane < 4) image_loads_drain(&w_bar[lane], 0);  // landed long ago, or a wait expired
    tr_teardown<kRowTmem>(t.tmem);
}

// The weight gradients: block (job, split) sums split_rows rows of the batch
// (chunks of 64 as K; 512 rows up to a batch of 16,384: 128 blocks at 8192) for
// a 128-row tile of a gradient.  Jobs 0-3: dW2's 128 x 128
// quarters; 4, 5: dW1's halves; 6, 7: dW3 transposed ([256][16]), by halves.
// One thread streams the chunks through four stages and issues the products.
//
// A partial sum is kept as the epilogue's threads have it: tiles of 16,384, in them
// [column / 4][row][column % 4] (neighbouring lanes are neighbouring rows); dW3
// after the six of them, in its own order.
constexpr int kTrJobs = 8;
constexpr uint32_t kTrSmem = kTrStages * 2 * kTile + 1024;
constexpr uint32_t kTrTileSums = kBM * kTrN, kTrW3Sums = 6 * kTrTileSums;
constexpr uint32_t kTrSums = kTrW3Sums + kOut * kHid;
static_assert(kTrSums <= kParams, "a split's sums");

__global__ void __launch_bounds__(kTrThreads) k_train_weights(const __grid_constant__ TrainArgs a) {
    extern __shared__ uint8_t raw[];
    __shared__ uint64_t bars[2 * kTrStages + 1];  // a chunk has landed; has been used; all have been used
    __shared__ uint32_t slot;
    __shared__ int s_ok;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int job = blockIdx.x;
    const TrSetup t = tr_setup<kTrN>(raw, bars, 2 * kTrStages + 1, &slot);
    griddep_wait();
    griddep_launch_dependents();
    const int per = (int)(a.split_rows / kBK), c0 = (int)blockIdx.y * per, n = min(per, (int)(a.B / kBK) - c0);
    float* const sums = a.weight_part + (size_t)blockIdx.y * kParams;
    const int mt = job < 4 ? job >> 1 : job & 1;
    const bool last_layer = job >= 6, first_layer = job == 4 || job == 5;
    if (tid == 0) {
        const uint8_t* A = first_layer ? a.dz1 : (last_layer ? a.h2 : a.dz2);
        auto load = [&](int i) {  // chunk i of the split: half an image of each of an operand's 64-column blocks
            const int s = i & (kTrStages - 1), c = c0 + i;
            const uint32_t sa = t.base + (uint32_t)s * 2 * kTile, sb = sa + kTile;
            const size_t image = (size_t)(c >> 1), half = (size_t)(c & 1) * kMnBlock;
            mbar_arrive_expect_tx(&bars[s], 2 * kMnBlock + (last_layer ? kMnBlock : 2 * kMnBlock));
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                image_load(sa + b * kMnBlock, A + (image * 4 + 2 * mt + b) * kImage + half, kMnBlock, &bars[s]);
                if (last_layer) {
                    if (b == 0) image_load(sb, a.dy + image * kImage + half, kMnBlock, &bars[s]);
                } else if (first_layer) {
                    image_load(sb + b * kMnBlock, a.xt + (image * 2 + b) * kImage + half, kMnBlock, &bars[s]);
                } else {
                    image_load(sb + b * kMnBlock, a.h1 + (image * 4 + 2 * (job & 1) + b) * kImage + half, kMnBlock, &bars[s]);
                }
            }
        };
        const uint32_t idesc = (last_layer ? idesc_bf16(kBM, kOut) : idesc_bf16(kBM, kTrN)) | kIdescAMn | kIdescBMn;
        bool ok = true;
        for (int i = 0; i < min(n, kTrStages); ++i) load(i);
        for (int i = 0; i < n; ++i) {
            const int s = i & (kTrStages - 1);
            ok = wait_commit(&bars[s], (i / kTrStages) & 1, a.err) && ok;
            tc_fence_after();
            const uint32_t sa = t.base + (uint32_t)s * 2 * kTile, sb = sa + kTile;
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk)
                umma_bf16(t.tmem, sw128_desc_mn(sa + kk * 2048, kMnBlock), sw128_desc_mn(sb + kk * 2048, kMnBlock), idesc,
                          (i > 0 || kk > 0) ? 1u : 0u);
            umma_commit(&bars[kTrStages + s]);
            // The stage of the chunk before this one, now that this one's products queue behind its.
            const int next = i - 1 + kTrStages, before = (i - 1) & (kTrStages - 1);
            if (i > 0 && next < n) {
                ok = wait_commit(&bars[kTrStages + before], ((i - 1) / kTrStages) & 1, a.err) && ok;
                load(next);
            }
        }
        if (!ok)
#pragma unroll 1
            for (int i = max(0, n - kTrStages); i < n; ++i)
                image_loads_drain(&bars[i & (kTrStages - 1)], (i / kTrStages) & 1);
        s_ok = ok;
        umma_commit(&bars[2 * kTrStages]);
    }
    __syncthreads();
    const bool ok = wait_commit(&bars[2 * kTrStages], 0, a.err) && s_ok;
    tc_fence_after();
    const int quarter = warp & 3, half = warp >> 2, ml = quarter * 32 + lane;
    const uint32_t t_lane = t.tmem + ((uint32_t)(quarter * 32) << 16);
    if (last_layer) {
        if (half == 0) {
            float v[16];
            tmem_ld16(t_lane, v);
#pragma unroll
            for (int i = 0; i < kOut; ++i) sums[kTrW3Sums + (size_t)i * kHid + mt * kBM + ml] = ok ? v[i] : 0.0f;
        }
    } else {
        float4* out = reinterpret_cast<float4*>(sums + (size_t)job * kTrTileSums);
#pragma unroll 1
        for (int cb = half * (kTrN / 2); cb < (half + 1) * (kTrN / 2); cb += 16) {
            float v[16];
            tmem_ld16(t_lane + cb, v);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                out[(cb / 4 + q) * kBM + ml] = ok ? make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3])
                                                  : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    tr_teardown<kTrN>(t.tmem);
}
static_assert(kParams % 4 == 0, "four-wide stores");

cudaError_t launch_forward_backward(const TrainArgs& a, cudaStream_t s) {
    if (a.B == 0 || a.B % kBM) return cudaErrorInvalidValue;
    static std::atomic<int> setup_rows[kSetupDevices];
    cudaError_t e = set_smem_once(setup_rows, k_train_rows, kRowSmem);
    if (e == cudaSuccess)
        e = launch_dependent(k_train_rows, dim3(2 * (a.B / kBM)), dim3(kRowThreads), kRowSmem, s, a);
    if (e != cudaSuccess) return e;
    static std::atomic<int> setup[kSetupDevices];
    if ((e = set_smem_once(setup, k_train_weights, kTrSmem)) != cudaSuccess) return e;
    const unsigned splits = train_splits(a.B, a.split_rows);
    return launch_dependent(k_train_weights, dim3(kTrJobs, splits), dim3(kTrThreads), kTrSmem, s, a);
}

// ------------------------------------------------- gradients and Adam ----
// The BF16 copies of the parameters that the tensor cores read: row-major for
// inference, as tile images (row n, column k) for training: W1's four (rows 128,
// columns 64 each), W2's eight, W3's columns in four of 16 rows.
__device__ __forceinline__ uint32_t image_at(uint32_t n, uint32_t k) {
    return n * 128 + ((((k & 63u) >> 3) ^ (n & 7u)) << 4) + (k & 7u) * 2;
}
__device__ __forceinline__ void put_bf16(uint32_t i, float v, const Bf16Weights& w) {
    const __nv_bfloat16 b = __float2bfloat16_rn(v);
    uint32_t at;
    if (i < kOffB1) {
        const uint32_t n = i / kInPad, k = i % kInPad;
        w.w1[i] = b;
        at = ((n >> 7) * 2 + (k >> 6)) * kImage + image_at(n & 127u, k);
    } else if (i >= kOffW2 && i < kOffB2) {
        const uint32_t j = i - kOffW2, n = j / kHid, k = j % kHid;
        w.w2[j] = b;
        at = (4 + (n >> 7) * 4 + (k >> 6)) * kImage + image_at(n & 127u, k);
    } else if (i >= kOffW3 && i < kOffB3) {
        const uint32_t j = i - kOffW3, n = j / kHid, k = j % kHid;
        w.w3[j] = b;
        at = 12 * kImage + (k >> 6) * kRowW3Chunk + image_at(n, k);
    } else {
        return;
    }
    *reinterpret_cast<__nv_bfloat16*>(w.images + at) = b;
}
static_assert(12 * kImage + 4 * kRowW3Chunk == kWeightImageBytes, "the weights' images");

// Adds the partial sums of gradient i (thread i for a weight, a warp for each of
// the 528 biases and the loss) in a fixed order and, with ADAM, updates the FP32
// master parameter and its BF16 copy; without, writes the gradient.
struct AdamArgs {
    float *p, *m, *v;
    float lr, b1, b2, eps, bc1, bc2;
    Bf16Weights w;
};
constexpr int kSumThreads = 256;
constexpr int kSumBlocksW = kTrSums / kSumThreads;
static_assert(kTrSums % kSumThreads == 0, "a thread per weight");
constexpr int kSumBlocksB = (kTrRowSums + kSumThreads / 32 - 1) / (kSumThreads / 32);

template <bool ADAM>
__global__ void __launch_bounds__(kSumThreads) k_train_update(const __grid_constant__ TrainArgs a, AdamArgs o,
                                                              uint32_t splits) {
    uint32_t i;
    bool owner = true;
    float sum = 0.0f, m0 = 0.0f, v0 = 0.0f, p0 = 0.0f;
    // Read ahead of the wait: the step before, which wrote them, was over before this
    // step's row kernel went past its own.  After the wait a step takes 31.4 us at a
    // batch of 8192 instead of 30.9.
    if constexpr (ADAM) reads_before_wait();
    auto moments = [&]() {
        if constexpr (ADAM) m0 = __ldcg(o.m + i), v0 = __ldcg(o.v + i), p0 = __ldcg(o.p + i);
    };
    if (blockIdx.x < (unsigned)kSumBlocksW) {
        const uint32_t j = blockIdx.x * kSumThreads + threadIdx.x;
        const uint32_t tile = j / kTrTileSums, row = (j >> 2) & (kBM - 1), col = ((j >> 9) & 31u) * 4 + (j & 3u);
        if (j >= kTrW3Sums)
            i = kOffW3 + (j - kTrW3Sums);
        else if (tile < 4)
            i = kOffW2 + ((tile >> 1) * kBM + row) * kHid + (tile & 1) * kTrN + col;
        else
            i = kOffW1 + ((tile - 4) * kBM + row) * kInPad + col;
        moments();
        griddep_wait();
        griddep_launch_dependents();
        const float* part = a.weight_part + j;
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
        if (b >= (uint32_t)kTrRowSums) {
            griddep_wait();
            return;
        }
        i = b < (uint32_t)kHid ? kOffB1 + b : (b < 2u * kHid ? kOffB2 + b - kHid : kOffB3 + b - 2 * kHid);
        if (b < kTrRowSums - 1) moments();
        griddep_wait();
        griddep_launch_dependents();
        const uint32_t tiles = a.B / kBM;
        for (uint32_t q = threadIdx.x & 31; q < tiles; q += 32) sum += a.row_part[(size_t)q * kTrRowSums + b];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
        owner = (threadIdx.x & 31) == 0;
        if (b == kTrRowSums - 1) {
            if (owner) *a.loss_sum = sum;
            return;
        }
    }
    if (!owner) return;
    const float gi = sum;
    if constexpr (ADAM) {
        // Which product is fused is written out, as in gelu_and_grad().
        const float mi = __fmaf_rn(1.0f - o.b1, gi, __fmul_rn(o.b1, m0));
        const float vi = __fmaf_rn(__fmul_rn(1.0f - o.b2, gi), gi, __fmul_rn(o.b2, v0));
        o.m[i] = mi;
        o.v[i] = vi;
        const float pi = p0 - o.lr * (mi / o.bc1) / (sqrtf(vi / o.bc2) + o.eps);
        o.p[i] = pi;
        put_bf16(i, pi, o.w);
    } else {
        a.g[i] = gi;
    }
}

__global__ void k_weights_bf16(const float* __restrict__ p, Bf16Weights w) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < kParams; i += gridDim.x * blockDim.x)
        put_bf16(i, p[i], w);
}

cudaError_t launch_train_update(const TrainArgs& a, float* p, float* m, float* v, float lr, float b1, float b2,
                                float eps, uint64_t t, const Bf16Weights& w, cudaStream_t s) {
    const float bc1 = 1.0f - (float)pow((double)b1, (double)t);
    const float bc2 = 1.0f - (float)pow((double)b2, (double)t);
    return launch_dependent(k_train_update<true>, dim3(kSumBlocksW + kSumBlocksB), dim3(kSumThreads), 0, s, a,
                            AdamArgs{p, m, v, lr, b1, b2, eps, bc1, bc2, w}, train_splits(a.B, a.split_rows));
}

cudaError_t launch_train_gradients(const TrainArgs& a, cudaStream_t s) {
    return launch_dependent(k_train_update<false>, dim3(kSumBlocksW + kSumBlocksB), dim3(kSumThreads), 0, s, a,
                            AdamArgs{}, train_splits(a.B, a.split_rows));
}

cudaError_t launch_weights_bf16(const float* p, const Bf16Weights& w, cudaStream_t s) {
    k_weights_bf16<<<256, 256, 0, s>>>(p, w);
    return cudaGetLastError();
}

}  // namespace mlp
}  // namespace marl
