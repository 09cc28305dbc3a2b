// Host-side interface of the surrogate's tensor-core kernels (mlp.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/marl_cuda.h"

namespace marl {
namespace mlp {

constexpr int kIn = MARL_SURR_FEATURES;  // 93 features
constexpr int kInPad = 128;              // first-layer K, zero-padded
constexpr int kHid = 256;
constexpr int kOut = 16;

// Flat parameter layout (FP32 master copy, gradients, Adam moments).
constexpr uint32_t kOffW1 = 0;
constexpr uint32_t kOffB1 = kOffW1 + kHid * kInPad;
constexpr uint32_t kOffW2 = kOffB1 + kHid;
constexpr uint32_t kOffB2 = kOffW2 + kHid * kHid;
constexpr uint32_t kOffW3 = kOffB2 + kHid;
constexpr uint32_t kOffB3 = kOffW3 + kOut * kHid;
constexpr uint32_t kParams = kOffB3 + kOut;
static_assert(kParams == MARL_SURR_PARAMS, "parameter layout");

#ifdef __CUDACC__
// Feature transform before standardisation: log(|v| + 1e-3) for k_m, v_max
// and k_cat (features 29 + 4r + {0, 1, 2}), identity otherwise.
__device__ __forceinline__ float feature_transform(int f, float v) {
    if (f >= 29 && ((f - 29) & 3) != 3) return logf(fabsf(v) + 1e-3f);
    return v;
}
#endif

enum Epi : int { EPI_BIAS_OUT, EPI_BIAS_GELU_FAST };

struct GemmArgs {
    const __nv_bfloat16* A = nullptr;  // [M][lda], K contiguous
    int lda = 0;
    const __nv_bfloat16* B = nullptr;  // [N][ldb], K contiguous
    int ldb = 0;
    int M = 0, N = 0, K = 0;
    const float* bias = nullptr;       // [N]
    const float* scale = nullptr;      // [N] optional (EPI_BIAS_OUT)
    const float* shift = nullptr;      // [N] with scale
    __nv_bfloat16* out_bf = nullptr;   // [M][ldo]
    int ldo = 0;
    float* out_f = nullptr;            // FP32 output (EPI_BIAS_OUT)
    int ldf = 0;
    int out_col_major = 0;             // out_f as [N][ldf]
    uint32_t* err = nullptr;           // kErr* bits on a wait timeout
};

// Arguments of the fused inference kernel: standardised BF16 inputs x
// [M][128], BF16 weights, FP32 biases, de-standardisation, and the output
// y [16][ldy] (species-major).
struct FusedArgs {
    const __nv_bfloat16* x = nullptr;
    int M = 0;
    const __nv_bfloat16 *w1 = nullptr, *w2 = nullptr, *w3 = nullptr;
    const float *b1 = nullptr, *b2 = nullptr, *b3 = nullptr;
    const float *scale = nullptr, *shift = nullptr;
    float* y = nullptr;
    uint32_t ldy = 0;
    uint32_t* err = nullptr;
};
cudaError_t launch_mlp_fused(const FusedArgs& a, int num_sms, cudaStream_t s);

// (bn, epi): (256, EPI_BIAS_GELU_FAST) or (16, EPI_BIAS_OUT).
cudaError_t launch_gemm(const GemmArgs& a, int bn, int epi, cudaStream_t s);

// The BF16 copies of the weights: row-major, and all of them as tile images.
struct Bf16Weights {
    __nv_bfloat16 *w1 = nullptr, *w2 = nullptr, *w3 = nullptr;
    uint8_t* images = nullptr;  // kWeightImageBytes
};
constexpr uint32_t kWeightImageBytes = 2 * (kHid * kInPad + kHid * kHid + kOut * kHid);

// One training step's buffers (B rows, a multiple of 128; see mlp_train.cu).
struct TrainArgs {
    uint32_t B = 0;
    const __nv_bfloat16* X = nullptr;  // standardised rows [.][128]
    const float* T = nullptr;          // their targets [.][16]
    uint32_t n_rows = 0;               // batch row r is a hashed draw from [0, n_rows); 0: row r itself
    uint64_t seed = 0, step = 0;       // of the draws
    const uint8_t* wi = nullptr;       // the BF16 weights' tile images
    const float* p = nullptr;          // FP32 parameters (the biases are read)
    // Images of 128-row, 64-column shared-memory tiles (16 KB, BF16): two to a row
    // tile of X, four of h1, h2, dz2 and dz1, one (16 columns used) of dy.
    uint8_t *xt = nullptr, *h1 = nullptr, *h2 = nullptr, *dy = nullptr, *dz2 = nullptr, *dz1 = nullptr;
    float* y = nullptr;                // [B][16]
    uint32_t split_rows = 0;           // rows of a weight-gradient partial sum (train_split_rows)
    float* weight_part = nullptr;      // [splits][kParams]: the weights' partial sums
    float* row_part = nullptr;         // [B / 128][kTrRowSums]: db1, db2, db3 and loss partial sums
    float* g = nullptr;                // gradients (launch_train_gradients)
    float* loss_sum = nullptr;
    uint32_t* err = nullptr;
};
constexpr int kTrRowSums = 2 * kHid + kOut + 1;
// Rows per partial sum of the weight gradients: 512, more where that would be
// more than 32 sums.
inline uint32_t train_split_rows(uint32_t B) { return 512u * ((B + 512u * 32u - 1u) / (512u * 32u)); }
inline uint32_t train_splits(uint32_t B, uint32_t split_rows) { return (B + split_rows - 1) / split_rows; }
cudaError_t launch_forward_backward(const TrainArgs& a, cudaStream_t s);
// The gradients from the partial sums into a.g, or Adam's step with them (on the
// FP32 parameters and their BF16 copies); both set *a.loss_sum.
cudaError_t launch_train_gradients(const TrainArgs& a, cudaStream_t s);
cudaError_t launch_train_update(const TrainArgs& a, float* p, float* m, float* v, float lr, float b1, float b2,
                                float eps, uint64_t t, const Bf16Weights& w, cudaStream_t s);
cudaError_t launch_weights_bf16(const float* p, const Bf16Weights& w, cudaStream_t s);
cudaError_t launch_raw_stats(const float* raw, uint32_t n, double* acc, cudaStream_t s);
cudaError_t launch_standardise(const float* raw, uint32_t n, const float* norm, __nv_bfloat16* X, float* T,
                               cudaStream_t s);
cudaError_t launch_eval_rows(const float* raw, const float* pred, uint32_t ldp, uint32_t n, const float* norm,
                             float tol, float c_max, float* err_out, double* acc, uint32_t* max_bits,
                             cudaStream_t s);
cudaError_t launch_init_weights(float* p, uint64_t seed, cudaStream_t s);

}  // namespace mlp
}  // namespace marl
