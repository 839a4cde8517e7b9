// Router helper for the expert-routed product: softmax over the experts, top-k by probability,
// renormalise.  Semantics of hf2q's softmax_topk_renorm_cpu
// (src/inference/models/qwen35/gpu_ffn.rs:1879-1924), which its GPU path reaches through
// dispatch_moe_softmax_topk (gpu_ffn.rs:2551): descending probability, equal probabilities keep
// the lower expert index first (the reference sorts stably), weights = p / sum(selected p), with
// the same 1e-20 guards.  One warp per token; probabilities live in shared memory.
// Sigmoid scores without renormalisation take the same selection.
#include <math_constants.h>

#include "common.cuh"
#include "kernels.h"

namespace hf2q {

namespace {
constexpr int WARPS = 4;

template <bool SIGMOID>
__global__ void __launch_bounds__(WARPS * 32) topk_kernel(const float* logits, uint32_t ld,
                                                                  uint32_t* __restrict__ ids,
                                                                  float* __restrict__ weights,
                                                                  uint32_t n_tokens, uint32_t n_experts,
                                                                  uint32_t top_k) {
    extern __shared__ float probs_all[];
    pdl_trigger();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t t = blockIdx.x * WARPS + warp;
    if (t >= n_tokens) return;
    float* probs = probs_all + static_cast<size_t>(warp) * n_experts;
    const float* row = logits + static_cast<size_t>(t) * ld;

    if constexpr (SIGMOID) {
        for (uint32_t e = lane; e < n_experts; e += 32) probs[e] = 1.0f / (1.0f + expf(-row[e]));
    } else {
        float mx = -CUDART_INF_F;
        for (uint32_t e = lane; e < n_experts; e += 32) mx = fmaxf(mx, row[e]);
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float denom = 0.f;
        for (uint32_t e = lane; e < n_experts; e += 32) {
            const float v = expf(row[e] - mx);
            probs[e] = v;
            denom += v;
        }
        for (int o = 16; o > 0; o >>= 1) denom += __shfl_xor_sync(0xffffffffu, denom, o);
        const float inv_d = denom > 1e-20f ? 1.0f / denom : 1.0f;
        for (uint32_t e = lane; e < n_experts; e += 32) probs[e] *= inv_d;
    }
    __syncwarp();

    // Selection is total: a NaN probability (a NaN logit, or a row whose logits are all -inf) ranks
    // below every number and among NaNs the lower index wins, so every round finds a candidate
    // (top_k <= n_experts) and no index is ever out of range.  Taken entries are marked -2 in
    // shared memory; the ranking key of a NaN is -1, so the two cannot be confused.  The reported
    // weight is the probability itself (a NaN stays a NaN, as IEEE arithmetic gives the reference).
    float sum_sel = 0.f;
    float my_w = 0.f;          // lane s keeps the s-th selected probability (top_k <= 32 per pass)
    uint32_t my_id = 0;
    for (uint32_t s = 0; s < top_k; ++s) {
        float best = -1.5f;    // keys are >= -1; taken entries (-2) never qualify
        uint32_t bi = 0xffffffffu;
        for (uint32_t e = lane; e < n_experts; e += 32) {
            const float v = probs[e];
            const float key = v != v ? -1.0f : v;
            if (key > best) { best = key; bi = e; }  // strided scan keeps the lowest index on ties
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        float val = 0.f;
        if (bi < n_experts) {                        // always true for top_k <= n_experts; guards the store
            val = probs[bi];
            __syncwarp();
            if (lane == 0) probs[bi] = -2.0f;
        } else {
            bi = 0;
        }
        __syncwarp();
        sum_sel += val;
        if ((s & 31u) == static_cast<uint32_t>(lane)) { my_w = val; my_id = bi; }
        if ((s & 31u) == 31u || s + 1 == top_k) {
            // flush this pass of up to 32 selections; weights are scaled after the loop
            const uint32_t base = s & ~31u;
            if (base + lane <= s) {
                ids[static_cast<size_t>(t) * top_k + base + lane] = my_id;
                weights[static_cast<size_t>(t) * top_k + base + lane] = my_w;
            }
        }
    }
    if constexpr (SIGMOID) return;
    __syncwarp();
    const float inv_sum = sum_sel > 1e-20f ? 1.0f / sum_sel : 1.0f / static_cast<float>(top_k);
    for (uint32_t s = lane; s < top_k; s += 32) weights[static_cast<size_t>(t) * top_k + s] *= inv_sum;
}

// The same for up to 32 NV experts: a lane keeps its NV probabilities as keys in registers, and a round is two warp-wide reductions.
// A key is the order of the above: 0 taken or absent, 1 a NaN, from 2 on the bits of a probability (none is negative).  One token
// in the launch: 5.0 -> 3.0 us, 2048 tokens 7.4 -> 4.6.
template <bool SIGMOID, int NV>
__global__ void __launch_bounds__(WARPS * 32) topk_small_kernel(const float* logits, uint32_t ld, uint32_t* __restrict__ ids,
                                                                float* __restrict__ weights, uint32_t n_tokens, uint32_t n_experts, uint32_t top_k) {
    pdl_trigger();
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31, t = blockIdx.x * WARPS + (threadIdx.x >> 5);
    if (t >= n_tokens) return;
    const float* row = logits + static_cast<size_t>(t) * ld;
    float v[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = lane + 32 * j < n_experts ? row[lane + 32 * j] : -CUDART_INF_F;
    if constexpr (SIGMOID) {
#pragma unroll
        for (int j = 0; j < NV; ++j) v[j] = 1.0f / (1.0f + expf(-v[j]));
    } else {
        float mx = -CUDART_INF_F;
#pragma unroll
        for (int j = 0; j < NV; ++j) mx = fmaxf(mx, v[j]);
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float denom = 0.f;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            if (lane + 32 * j < n_experts) { v[j] = expf(v[j] - mx); denom += v[j]; }
        }
        for (int o = 16; o > 0; o >>= 1) denom += __shfl_xor_sync(0xffffffffu, denom, o);
        const float inv_d = denom > 1e-20f ? 1.0f / denom : 1.0f;
#pragma unroll
        for (int j = 0; j < NV; ++j) v[j] *= inv_d;
    }
    uint32_t key[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) key[j] = lane + 32 * j >= n_experts ? 0u : v[j] != v[j] ? 1u : __float_as_uint(v[j]) + 2u;
    float sum_sel = 0.f, my_w = 0.f;
    uint32_t my_id = 0;
    for (uint32_t s = 0; s < top_k; ++s) {
        uint32_t best = key[0], j_best = 0;
#pragma unroll
        for (int j = 1; j < NV; ++j)
            if (key[j] > best) { best = key[j]; j_best = j; }
        const uint32_t top = __reduce_max_sync(0xffffffffu, best), bi = __reduce_min_sync(0xffffffffu, best == top ? lane + 32 * j_best : 0xffffffffu);
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (bi == lane + 32 * j) key[j] = 0u;
        const float val = top == 1u ? CUDART_NAN_F : __uint_as_float(top - 2u);
        sum_sel += val;
        if ((s & 31u) == lane) { my_w = val; my_id = bi; }
        if ((s & 31u) == 31u || s + 1 == top_k) {
            const uint32_t base = s & ~31u;
            if (base + lane <= s) {
                ids[static_cast<size_t>(t) * top_k + base + lane] = my_id;
                weights[static_cast<size_t>(t) * top_k + base + lane] = my_w;
            }
        }
    }
    if constexpr (SIGMOID) return;
    __syncwarp();
    const float inv_sum = sum_sel > 1e-20f ? 1.0f / sum_sel : 1.0f / static_cast<float>(top_k);
    for (uint32_t s = lane; s < top_k; s += 32) weights[static_cast<size_t>(t) * top_k + s] *= inv_sum;
}

template <bool SIGMOID>
cudaError_t launch_topk(const float* logits, uint32_t ld, uint32_t* ids, float* weights, uint32_t n_tokens, uint32_t n_experts, uint32_t top_k, cudaStream_t st) {
    const size_t smem = static_cast<size_t>(WARPS) * n_experts * sizeof(float);
    if (smem > 48 * 1024) return cudaErrorInvalidValue;
    const dim3 grid((n_tokens + WARPS - 1) / WARPS), block(WARPS * 32);
    if (n_experts <= 32) return launch_pdl(topk_small_kernel<SIGMOID, 1>, grid, block, 0, st, logits, ld, ids, weights, n_tokens, n_experts, top_k);
    if (n_experts <= 64) return launch_pdl(topk_small_kernel<SIGMOID, 2>, grid, block, 0, st, logits, ld, ids, weights, n_tokens, n_experts, top_k);
    if (n_experts <= 128) return launch_pdl(topk_small_kernel<SIGMOID, 4>, grid, block, 0, st, logits, ld, ids, weights, n_tokens, n_experts, top_k);
    if (n_experts <= 256) return launch_pdl(topk_small_kernel<SIGMOID, 8>, grid, block, 0, st, logits, ld, ids, weights, n_tokens, n_experts, top_k);
    return launch_pdl(topk_kernel<SIGMOID>, grid, block, smem, st, logits, ld, ids, weights, n_tokens, n_experts, top_k);
}
}  // namespace

cudaError_t launch_softmax_topk(const float* logits, uint32_t* ids, float* weights, uint32_t n_tokens,
                                uint32_t n_experts, uint32_t top_k, cudaStream_t st) {
    return launch_topk<false>(logits, n_experts, ids, weights, n_tokens, n_experts, top_k, st);
}

cudaError_t launch_sigmoid_topk(const float* logits, uint32_t ld, uint32_t* ids, float* weights, uint32_t n_tokens,
                                uint32_t n_experts, uint32_t top_k, cudaStream_t st) {
    return launch_topk<true>(logits, ld, ids, weights, n_tokens, n_experts, top_k, st);
}

}  // namespace hf2q
