// Element-wise glue of the FFN builders that sit directly on the quantized products:
// SwiGLU (silu(gate) * up) and the MoE combine (weighted sum over the top-k slots, plus the
// sigmoid-gated shared expert and the residual).  Semantics follow hf2q's scalar references
// dense_swiglu_cpu_ref (src/inference/models/qwen35/ffn.rs:91-112) and moe_ffn_cpu_ref
// (ffn.rs:179-336); the reference's GPU builders dispatch dispatch_silu_mul /
// dispatch_moe_weighted_reduce for the same steps (gpu_ffn.rs:1086-1351, 2313-2802).
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"
#include "seq_common.cuh"

namespace hf2q {
namespace {
namespace cg = cooperative_groups;

__device__ __forceinline__ float silu(float x) { return x / (1.0f + expf(-x)); }     // ffn.rs:24-26

__global__ void __launch_bounds__(256) silu_mul_kernel(const float* __restrict__ gate, const float* __restrict__ up,
                                                       float* __restrict__ out, uint64_t n4) {
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += stride) {
        const float4 g = reinterpret_cast<const float4*>(gate)[i], u = reinterpret_cast<const float4*>(up)[i];
        reinterpret_cast<float4*>(out)[i] = make_float4(silu(g.x) * u.x, silu(g.y) * u.y, silu(g.z) * u.z, silu(g.w) * u.w);
    }
}
__global__ void __launch_bounds__(256) silu_mul_tail_kernel(const float* gate, const float* up, float* out, uint64_t from, uint64_t n) {
    const uint64_t i = from + blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = silu(gate[i]) * up[i];
}

// out[t, :] = sum_s w[t*k+s] * y[t*k+s, :]  (+ sigmoid(gate_logit[t]) * shared[t, :])  (+ residual[t, :])
// V: float, or float4 where rows are whole 16-byte groups.  Bound by memory: eight rows are asked for before they are added, in
// slot order, as the reference sums (2048 tokens, 8 rows of 2048 each: 151 MB, 30 -> 28 us).
// The next launch starts when this one ends: under it a following layer's router got SMs as they fell free, two CTAs to one (layers
// one behind the other, us with and without: 8 experts of 2048 x 2048, two a token, 200 tokens 69.8 and 62.4; 128 of 768, eight a token,
// 128 tokens 208 and 201; 256 of 512, 512 tokens 290 and 281).
__device__ __forceinline__ void add_scaled(float& a, float w, float v) { a += w * v; }
__device__ __forceinline__ void add_scaled(float4& a, float w, const float4& v) { a.x += w * v.x; a.y += w * v.y; a.z += w * v.z; a.w += w * v.w; }
template <typename V>
__global__ void __launch_bounds__(256) moe_combine_kernel(const float* y, const float* w,
                                                          const float* shared, const float* gate_logit,
                                                          const float* residual, float* __restrict__ out,
                                                          uint32_t top_k, uint32_t h) {
    constexpr uint32_t E = sizeof(V) / 4, AHEAD = 8;
    pdl_wait();
    const uint32_t t = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x, n = h / E;
    if (c >= n) return;
    auto at = [&](const float* p, size_t row) { return reinterpret_cast<const V*>(p + row * h)[c]; };
    V acc{};
    for (uint32_t s0 = 0; s0 < top_k; s0 += AHEAD) {
        V v[AHEAD];
        float f[AHEAD];
#pragma unroll
        for (uint32_t s = 0; s < AHEAD; ++s)
            if (s0 + s < top_k) { v[s] = at(y, static_cast<size_t>(t) * top_k + s0 + s); f[s] = w[static_cast<size_t>(t) * top_k + s0 + s]; }
#pragma unroll
        for (uint32_t s = 0; s < AHEAD; ++s)
            if (s0 + s < top_k) add_scaled(acc, f[s], v[s]);
    }
    if (shared) add_scaled(acc, gate_logit ? 1.0f / (1.0f + expf(-gate_logit[t])) : 1.0f, at(shared, t));      // ffn.rs:28-30
    if (residual) add_scaled(acc, 1.0f, at(residual, t));
    reinterpret_cast<V*>(out + static_cast<size_t>(t) * h)[c] = acc;
}

// out[t] = sum_i v[i] * x[t, i]   (the shared expert's gate logit, a [1, h] f32 matrix)
__global__ void __launch_bounds__(256) rowdot_kernel(const float* __restrict__ x, const float* __restrict__ v, float* __restrict__ out,
                                                     uint32_t n_tokens, uint32_t h) {
    __shared__ float part[8];
    const uint32_t t = blockIdx.x;
    float acc = 0.f;
    for (uint32_t i = threadIdx.x; i < h; i += 256) acc += v[i] * x[static_cast<size_t>(t) * h + i];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        for (int i = 0; i < 8; ++i) s += part[i];
        out[t] = s;
    }
    (void)n_tokens;
}

// Router logits of an MoE layer: out[t, e] = sum_h x[t, h] * w[e, h], all f32 (the router is a small
// dense f32 matrix in the reference as well: phase 1 of the six-phase graph at gpu_ffn.rs:2347-2359).
//
// Up to RV_TOKENS tokens: bound by the latency of one pass over the router (2 MB for 256 experts of 2048), so every
// expert has a CTA of its own whose threads request sixteen values of its row at a time (256 experts, one token: 2.6 us;
// tiles of 64 tokens, four CTAs in all, took 180 us).
constexpr int RV_TOKENS = 8, RV_THREADS = 128, RV_AHEAD = 4;

__device__ __forceinline__ float4 load4(const void* p, uint32_t bf16, size_t i) {
    if (!bf16) return *reinterpret_cast<const float4*>(static_cast<const float*>(p) + i);
    const uint2 u = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(p) + i);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float load1(const void* p, uint32_t bf16, size_t i) {
    return bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]) : static_cast<const float*>(p)[i];
}

// VEC: h is a multiple of 4, and x and w allow loads of four elements.
template <bool VEC>
__global__ void __launch_bounds__(RV_THREADS) router_vector_kernel(const void* x, uint32_t x_bf16, const float* w,
                                                                   float* __restrict__ out, uint32_t n_tokens, uint32_t n_experts, uint32_t h) {
    __shared__ float part[RV_TOKENS][RV_THREADS / 32];
    const uint32_t e = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* row = w + static_cast<size_t>(e) * h;
    float acc[RV_TOKENS] = {};
    pdl_trigger();
    pdl_wait();
    if constexpr (VEC) {
        for (uint32_t i0 = 4 * threadIdx.x; i0 < h; i0 += RV_AHEAD * 4 * RV_THREADS) {
            float4 wv[RV_AHEAD];
#pragma unroll
            for (int a = 0; a < RV_AHEAD; ++a) {
                const uint32_t i = i0 + a * 4 * RV_THREADS;
                wv[a] = i < h ? __ldg(reinterpret_cast<const float4*>(row + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int t = 0; t < RV_TOKENS; ++t) {
                if (t >= n_tokens) break;
#pragma unroll
                for (int a = 0; a < RV_AHEAD; ++a) {
                    const uint32_t i = i0 + a * 4 * RV_THREADS;
                    if (i >= h) break;
                    const float4 v = load4(x, x_bf16, static_cast<size_t>(t) * h + i);
                    acc[t] += wv[a].x * v.x + wv[a].y * v.y + wv[a].z * v.z + wv[a].w * v.w;
                }
            }
        }
    }
    if constexpr (!VEC) {
        for (uint32_t i = threadIdx.x; i < h; i += RV_THREADS) {
            const float wv = __ldg(row + i);
#pragma unroll
            for (int t = 0; t < RV_TOKENS; ++t)
                if (t < n_tokens) acc[t] += wv * load1(x, x_bf16, static_cast<size_t>(t) * h + i);
        }
    }
#pragma unroll
    for (int t = 0; t < RV_TOKENS; ++t) {
        for (int o = 16; o > 0; o >>= 1) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], o);
        if (lane == 0) part[t][warp] = acc[t];
    }
    __syncthreads();
    if (threadIdx.x < n_tokens) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < RV_THREADS / 32; ++i) s += part[threadIdx.x][i];
        out[static_cast<size_t>(threadIdx.x) * n_experts + e] = s;
    }
}

// More tokens: tiles of 64 R tokens x 64 R experts, R x R blocks of 4 x 4 outputs per thread in packed f32 arithmetic, the next 32
// columns on their way to registers while the present ones are used.  Bound by the f32 pipes (2048 tokens x 256 experts of 2048:
// 1.07 G multiply-adds, 29 us at their peak); with R = 1 by shared memory, 32 bytes for 16 multiply-adds, R = 2 halves that (86 -> 65 us).
// The CTAs of a cluster share a tile's columns where the tiles alone would leave the chip idle, and add
// their sums through distributed shared memory in rank order (2048 tokens, 256 experts of 2048, R = 1: 263 -> 86 us).  The line at
// RV_TOKENS is the number of sums a thread of the other kernel keeps in registers; there the tiles are still behind (us a CTA per
// expert / tiles, 8 and 16 tokens: 256 experts of 2048 7.9 / 13.9 and 12.6 / 13.9, 8 of 4096 10.7 / 20.9 and 19.7 / 21.1).
// Columns are stored with the group of four tokens (or experts) XORed by the column's own group of four, which keeps both the
// transposing stores and the reads free of conflicts.
constexpr int RT = 64, RKT = 32, RT_MAX_PARTS = 8;
constexpr size_t router_smem(int R) { return 4 * (2 * RKT * RT * R > RT * R * RT * R ? 2 * RKT * RT * R : RT * R * RT * R); }

template <bool VEC, int R>
__global__ void __launch_bounds__(256, 2) router_tile_kernel(const void* x, uint32_t x_bf16, const float* w,
                                                             float* __restrict__ out, uint32_t n_tokens, uint32_t n_experts, uint32_t h) {
    constexpr int TILE = RT * R;
    extern __shared__ __align__(16) float rsm[];
    float (*xs)[TILE] = reinterpret_cast<float (*)[TILE]>(rsm), (*ws)[TILE] = xs + RKT;
    const cg::cluster_group cl = cg::this_cluster();
    pdl_trigger();
    pdl_wait();
    const uint32_t parts = gridDim.z, part = blockIdx.z;             // the cluster is the whole z extent
    const uint32_t t0 = blockIdx.y * TILE, e0 = blockIdx.x * TILE;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;          // outputs: tokens 64 u + 4 ty .. + 3, experts 64 v + 4 tx .. + 3
    const uint32_t chunks = (h + RKT - 1) / RKT, per = (chunks + parts - 1) / parts;
    const uint32_t c0 = min(part * per, chunks), c1 = min(c0 + per, chunks);
    // a thread brings columns 4 kg .. 4 kg + 3 of every 32nd row of both tiles
    const uint32_t kg = threadIdx.x & 7, r = threadIdx.x >> 3;
    float4 xr[2 * R], wr[2 * R];
    auto fetch = [&](uint32_t c) {
        const uint32_t k = c * RKT + 4 * kg;
#pragma unroll
        for (int i = 0; i < 2 * R; ++i) {
            const uint32_t t = t0 + r + 32 * i, e = e0 + r + 32 * i;
            const size_t xo = static_cast<size_t>(t) * h + k, wo = static_cast<size_t>(e) * h + k;
            xr[i] = wr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if constexpr (VEC) {
                if (t < n_tokens && k < h) xr[i] = load4(x, x_bf16, xo);
                if (e < n_experts && k < h) wr[i] = __ldg(reinterpret_cast<const float4*>(w + wo));
            } else {
                float* xp = &xr[i].x;
                float* wp = &wr[i].x;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (t < n_tokens && k + j < h) xp[j] = load1(x, x_bf16, xo + j);
                    if (e < n_experts && k + j < h) wp[j] = __ldg(w + wo + j);
                }
            }
        }
    };
    f2 acc[4 * R][2 * R] = {};
    if (c0 < c1) fetch(c0);
    for (uint32_t c = c0; c < c1; ++c) {
#pragma unroll
        for (int i = 0; i < 2 * R; ++i) {
            const uint32_t row = r + 32 * i, at = 4 * ((row >> 2) ^ kg) + (row & 3);
            const float xv[4] = {xr[i].x, xr[i].y, xr[i].z, xr[i].w}, wv[4] = {wr[i].x, wr[i].y, wr[i].z, wr[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                xs[4 * kg + j][at] = xv[j];
                ws[4 * kg + j][at] = wv[j];
            }
        }
        __syncthreads();
        if (c + 1 < c1) fetch(c + 1);
#pragma unroll
        for (int k = 0; k < RKT; ++k) {
            float4 a[R];
            ulonglong2 b[R];
#pragma unroll
            for (int u = 0; u < R; ++u) {
                a[u] = *reinterpret_cast<const float4*>(&xs[k][RT * u + 4 * (ty ^ (k >> 2))]);
                b[u] = *reinterpret_cast<const ulonglong2*>(&ws[k][RT * u + 4 * (tx ^ (k >> 2))]);
            }
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const float av[4] = {a[u].x, a[u].y, a[u].z, a[u].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const f2 aa = f2_both(av[i]);
#pragma unroll
                    for (int v = 0; v < R; ++v) {
                        acc[4 * u + i][2 * v] = f2_fma(aa, b[v].x, acc[4 * u + i][2 * v]);
                        acc[4 * u + i][2 * v + 1] = f2_fma(aa, b[v].y, acc[4 * u + i][2 * v + 1]);
                    }
                }
            }
        }
        __syncthreads();
    }
    auto store = [&](uint32_t t, uint32_t e, const float4& v) {      // experts e .. e + 3 of token t
        if (t >= n_tokens) return;
        const float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (e + j < n_experts) out[static_cast<size_t>(t) * n_experts + e + j] = o[j];
    };
    // the tile's sums [token][expert], over the operands
    float* sums = rsm;
#pragma unroll
    for (int i = 0; i < 4 * R; ++i)
#pragma unroll
        for (int v = 0; v < R; ++v) {
            const uint32_t row = RT * (i / 4) + 4 * ty + i % 4, col = RT * v + 4 * tx;
            if (parts == 1) {
                const float2 lo = f2_parts(acc[i][2 * v]), hi = f2_parts(acc[i][2 * v + 1]);
                store(t0 + row, e0 + col, make_float4(lo.x, lo.y, hi.x, hi.y));
            } else {
                f2* d = reinterpret_cast<f2*>(sums + row * TILE + col);
                d[0] = acc[i][2 * v];
                d[1] = acc[i][2 * v + 1];
            }
        }
    if (parts == 1) return;
    cl.sync();
    // this CTA's share of the tile's rows
    const uint32_t rows = TILE / parts;
    for (uint32_t i = threadIdx.x; i < rows * (TILE / 4); i += 256) {
        const uint32_t row = part * rows + i / (TILE / 4), q = 4 * (i % (TILE / 4));
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t p = 0; p < parts; ++p) {
            const float4 v = *reinterpret_cast<const float4*>(cl.map_shared_rank(sums + row * TILE + q, p));
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        store(t0 + row, e0 + q, s);
    }
    cl.sync();                                                       // peers read this CTA's sums until here
}

uint64_t router_tiles(uint32_t n_tokens, uint32_t n_experts, uint32_t side) { return static_cast<uint64_t>((n_experts + side - 1) / side) * ((n_tokens + side - 1) / side); }
// Time of n tiles in so many parts, in eighths of what one tile takes an SM by itself: two CTAs that share an SM take twice as long.
uint64_t router_time(uint64_t n, uint32_t parts, uint64_t sms) { return (n * parts + sms - 1) / sms * (RT_MAX_PARTS / parts); }
// Parts of a tile: as many as keep two CTAs on every SM busy.  More tiles than SMs: halves or quarters where whole ones leave a last wave nearly
// empty (8192 tokens, 384 experts of 2048: 395 us in 192 large tiles, 302 in halves; 5000 tokens, 512 experts: 398 in 160, 249 in
// quarters; quarters for an eighth of the time were a little slower, 16384 tokens, 8 experts: 131 and 134).
uint32_t router_parts(uint64_t n, uint32_t h, uint64_t sms) {
    uint32_t parts = 1;
    while (parts < RT_MAX_PARTS && parts * n <= sms && h >= 2 * parts * RKT) parts *= 2;
    if (n > sms) {
        const uint64_t whole = router_time(n, 1, sms), halves = router_time(n, 2, sms), quarters = router_time(n, 4, sms);
        if (h >= 2 * RKT && 10 * halves < 9 * whole) parts = 2;
        if (h >= 4 * RKT && 10 * quarters < 8 * whole && quarters < router_time(n, parts, sms)) parts = 4;
    }
    return parts;
}

template <int R>
cudaError_t launch_router_tiles(bool vec, const void* x, uint32_t x_bf16, const float* w, float* out, uint32_t n_tokens, uint32_t n_experts, uint32_t h, int sm_count,
                                cudaStream_t st) {
    const dim3 tiles((n_experts + RT * R - 1) / (RT * R), (n_tokens + RT * R - 1) / (RT * R));
    const uint32_t parts = router_parts(router_tiles(n_tokens, n_experts, RT * R), h, static_cast<uint64_t>(sm_count));
    const auto kern = vec ? router_tile_kernel<true, R> : router_tile_kernel<false, R>;
    static PerDeviceFlag flag[2];
    if (const cudaError_t e = ensure_max_dynamic_smem(kern, static_cast<int>(router_smem(R)), flag[vec]); e != cudaSuccess) return e;
    return launch_pdl_cluster(kern, dim3(tiles.x, tiles.y, parts), dim3(256), dim3(1, 1, parts), router_smem(R), st, x, x_bf16, w, out, n_tokens, n_experts, h);
}

}  // namespace

cudaError_t launch_router_logits(const void* x, uint32_t x_bf16, const float* w, float* out, uint32_t n_tokens, uint32_t n_experts,
                                 uint32_t h, int sm_count, cudaStream_t st) {
    const bool vec = h % 4 == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0 && reinterpret_cast<uintptr_t>(x) % (x_bf16 ? 8 : 16) == 0;
    if (n_tokens <= RV_TOKENS)
        return launch_pdl(vec ? router_vector_kernel<true> : router_vector_kernel<false>, dim3(n_experts), dim3(RV_THREADS), 0, st, x, x_bf16, w, out,
                               n_tokens, n_experts, h);
    // The larger tiles take three times as long as the small ones (2048 columns: 200 and 66 us on an SM) for four times the work: where
    // their parts fill the chip and their waves, with the ragged edge, come out no longer (us small / large: 2048 tokens, 128 experts
    // 36.7 / 55.8, 256 experts 69.9 / 57.7; 1500 tokens, 192 experts 52.9 / 57.2; 8192 tokens, 256 experts 264 / 205).
    const uint64_t sms = static_cast<uint64_t>(sm_count), small = router_tiles(n_tokens, n_experts, RT), large = router_tiles(n_tokens, n_experts, 2 * RT);
    if (n_experts > RT && large * RT_MAX_PARTS >= sms && 3 * router_time(large, router_parts(large, h, sms), sms) <= router_time(small, router_parts(small, h, sms), sms))
        return launch_router_tiles<2>(vec, x, x_bf16, w, out, n_tokens, n_experts, h, sm_count, st);
    return launch_router_tiles<1>(vec, x, x_bf16, w, out, n_tokens, n_experts, h, sm_count, st);
}

cudaError_t launch_silu_mul(const float* gate, const float* up, float* out, uint64_t n, int sm_count, cudaStream_t st) {
    const bool vec = (reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(up) | reinterpret_cast<uintptr_t>(out)) % 16 == 0;
    const uint64_t n4 = vec ? n / 4 : 0;
    if (n4) {
        const uint64_t want = (n4 + 255) / 256, cap = static_cast<uint64_t>(sm_count) * 16;
        silu_mul_kernel<<<static_cast<unsigned>(want < cap ? want : cap), 256, 0, st>>>(gate, up, out, n4);
    }
    const uint64_t done = n4 * 4;
    if (done < n) silu_mul_tail_kernel<<<static_cast<unsigned>((n - done + 255) / 256), 256, 0, st>>>(gate, up, out, done, n);
    return cudaGetLastError();
}

cudaError_t launch_moe_combine(const float* y, const float* w, const float* shared, const float* gate_logit, const float* residual,
                               float* out, uint32_t n_tokens, uint32_t top_k, uint32_t h, cudaStream_t st) {
    const bool vec = h % 4 == 0 && (reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(shared) | reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(out)) % 16 == 0;
    const dim3 grid((h / (vec ? 4 : 1) + 255) / 256, n_tokens);
    return vec ? launch_pdl(moe_combine_kernel<float4>, grid, dim3(256), 0, st, y, w, shared, gate_logit, residual, out, top_k, h)
               : launch_pdl(moe_combine_kernel<float>, grid, dim3(256), 0, st, y, w, shared, gate_logit, residual, out, top_k, h);
}

cudaError_t launch_rowdot(const float* x, const float* v, float* out, uint32_t n_tokens, uint32_t h, cudaStream_t st) {
    rowdot_kernel<<<n_tokens, 256, 0, st>>>(x, v, out, n_tokens, h);
    return cudaGetLastError();
}

}  // namespace hf2q
