// Causal attention of a prompt portion over the 8-bit KV cache, on the 5th-generation tensor cores.
//
//   scores[t, p] = q[t] . (k_code[p] * k_scale[p])      out[t] = softmax(scores) . (v_code * v_scale)
//
// q is read rotated and scaled (rope_kv_append_kernel ran before).  Arithmetic: scores and weighted values are f16 products
// with fp32 accumulation; the codes are whole numbers below 128 and so exact in f16, q is rounded to f16 once, the scale of
// K is applied to the fp32 score, softmax and its sum run in fp32 and probability * v_scale is rounded to f16.
//
// One CTA owns 128 rows = 128 / G tokens x the G query heads of one KV head and walks the cached positions in blocks of 64:
//
//   warps 4-7   converters.  Read the block's K and V codes (16-byte loads, the next block's already under way), turn each
//               byte into an f16 whole number and store both operands with the 128-byte swizzle.  K is [position][dim], the
//               K-major B operand of the scores; V has the same layout, read MN-major as the B operand of the output.
//   warp 8      one lane issues the products: S(j+1) = Q K^T before O += P(j) V, so that the scores of the next block are
//               ready when the softmax of this one ends.  Two S buffers; P(j) takes the place of S(j) in tensor memory.
//   warps 0-3   softmax, a thread to a row: scores from tensor memory, fp32 exponentials, P back as the f16 A operand.  The
//               output row is rescaled only when the running maximum grew by more than 2^3 (the exponentials then stay
//               below 8, which f16 has room for as long as the V scales of the block are below 16; otherwise at any growth).
//
// 256 tensor-memory columns (S 2 x 64, O 128) and 100 KB of shared memory: two CTAs per SM, one converts and rescales while
// the other's products run.  The grid starts the tiles with the most positions first.
//
// What bounds it: shared-memory traffic and the exponentials, about level (a block of 64 positions moves 98 KB: Q and K
// of the scores 48, V 16, the converted operands 32; and takes 8192 exponentials, 512 cycles).  Measured: a prompt of 8192
// tokens in portions of 2048, 32 heads over 8, takes 269 us a portion and layer (137 GFLOP, 511 TFLOP/s); warp-level products
// with every warp converting its own codes took 1031 us.
//
// Up to 48 positions in all a kernel without tensor cores (attn_prefill_few_kernel).
#include <math_constants.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "tc_common.cuh"

namespace hf2q {
using namespace tc;
namespace {

constexpr uint32_t HD = 128, ROWS = 128, BP = 64;                  // head dim, rows of a CTA, positions of a block
constexpr uint32_t Q_BYTES = ROWS * HD * 2, KV_BYTES = BP * HD * 2, PANEL = BP * 128;
constexpr uint32_t AP_SMEM = Q_BYTES + 4 * KV_BYTES + 1024;        // Q, two K and two V blocks, alignment
constexpr uint32_t AP_THREADS = 288, COLS = 256, COL_O = 128;
// Scales of a block have a barrier per slot.  They are written up to two blocks ahead of the softmax, and no phase of sc_full
// passes its waiter: slot j % 4 is written next for block j + 4, after s_full of j + 2, which follows o_done of j, which follows
// the P(j) of every softmax warp.  (k_full, two deep, can run a phase ahead of the softmax: K(j + 2) waits for S(j) alone.)
constexpr uint32_t SLOTS = 4;
constexpr float LAZY_LOG2 = 3.0f, LAZY_VMAX = 16.0f;


// sixteen signed bytes -> sixteen f16 whole numbers, as the two 16-byte chunks of a swizzled row; odd panels store their
// chunks in the other order (the lanes of a quarter-warp then meet all banks)
__device__ __forceinline__ void store_codes(uint8_t* block, uint32_t row, uint32_t c16, const uint4& q) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    uint32_t h[8];
    const __half2 bias = __float2half2_rn(1152.0f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t x = w[i] ^ 0x80808080u;                     // code + 128; 0x6400 | b is 1024 + b
        h[2 * i] = h2_bits(codes01(x, bias));
        h[2 * i + 1] = h2_bits(codes23(x, bias));
    }
    uint8_t* at = block + (c16 >> 2) * PANEL + row * 128;
    const uint32_t c = (c16 & 3) * 2, flip = c16 >> 2;
    const uint4 lo = make_uint4(h[0], h[1], h[2], h[3]), hi = make_uint4(h[4], h[5], h[6], h[7]);
    *reinterpret_cast<uint4*>(at + (((c + flip) ^ (row & 7)) << 4)) = flip ? hi : lo;
    *reinterpret_cast<uint4*>(at + (((c + 1 - flip) ^ (row & 7)) << 4)) = flip ? lo : hi;
}

// two values of positions p and p + 1 for a row whose last position is `seen`: scores, or weights (what is hidden has none,
// also where its V scale is infinite or NaN)
__device__ __forceinline__ float2 hide(float2 x, uint32_t p, uint32_t seen, float hidden) {
    return make_float2(p <= seen ? x.x : hidden, p + 1 <= seen ? x.y : hidden);
}

// OUT __half: the f16 activation panel of the product that follows
template <typename OUT> __device__ __forceinline__ OUT out_value(float v, bool& clipped) {
    if constexpr (std::is_same_v<OUT, float>) return v;
    else if constexpr (std::is_same_v<OUT, __half>) return panel_f16(v, clipped);
    else return __float2bfloat16_rn(v);
}

template <int G, typename OUT>
__global__ void __launch_bounds__(AP_THREADS, 2) attn_prefill_kernel(const float* __restrict__ qkv, uint32_t row_stride, uint32_t m,
                                                                     const int8_t* __restrict__ k_codes, const float* __restrict__ k_scale,
                                                                     const int8_t* __restrict__ v_codes, const float* __restrict__ v_scale,
                                                                     uint32_t max_seq, uint32_t pos0, uint32_t n_kv, OUT* __restrict__ out,
                                                                     uint32_t out_stride, uint32_t* status) {
    extern __shared__ uint8_t ap_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ap_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t *qs = smem, *ks = smem + Q_BYTES, *vs = ks + 2 * KV_BYTES;
    __shared__ __align__(16) float s_ks[SLOTS][BP], s_vs[SLOTS][BP];
    __shared__ float s_vmax[SLOTS][2];
    __shared__ uint64_t k_full[2], v_full[2], s_full[2], p_full[2], o_done[2], sc_full[SLOTS];
    __shared__ uint32_t tmem_slot;
    constexpr uint32_t TOK = ROWS / G;
    const uint32_t kvh = blockIdx.x % n_kv, tok0 = ((gridDim.x - 1 - blockIdx.x) / n_kv) * TOK;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t last = pos0 + min(tok0 + TOK, m) - 1;           // the last position a row of this CTA sees
    const uint32_t nb = last / BP + 1;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 4);
            mbar_init(&v_full[i], 4);
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], 4);
            mbar_init(&o_done[i], 1);
        }
        for (uint32_t i = 0; i < SLOTS; ++i) mbar_init(&sc_full[i], 4);
        mbar_fence_init();
    }
    if (warp == 8) { tmem_alloc(&tmem_slot, COLS); tmem_relinquish(); }
    // Q: 128 rows of 128 dims as f16, two panels of 64 dims
    for (uint32_t r = warp; r < ROWS; r += AP_THREADS / 32) {
        const uint32_t tok = tok0 + r / G;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tok < m) v = __ldg(reinterpret_cast<const float4*>(qkv + static_cast<size_t>(tok) * row_stride + (static_cast<size_t>(kvh) * G + r % G) * HD) + lane);
        *reinterpret_cast<uint2*>(qs + (lane >> 4) * (ROWS * 128) + r * 128 + ((((lane & 15) >> 1) ^ (r & 7)) << 4) + (lane & 1) * 8) =
            make_uint2(pack_h2(v.x, v.y), pack_h2(v.z, v.w));
    }
    proxy_fence();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp >= 4 && warp < 8) {
        const uint32_t tid = threadIdx.x - 128, c16 = tid & 7, row0 = tid >> 3;
        const uint8_t* kc = reinterpret_cast<const uint8_t*>(k_codes) + static_cast<size_t>(kvh) * max_seq * HD + 16 * c16;
        const uint8_t* vc = reinterpret_cast<const uint8_t*>(v_codes) + static_cast<size_t>(kvh) * max_seq * HD + 16 * c16;
        const float* scale = (tid < BP ? k_scale : v_scale) + static_cast<size_t>(kvh) * max_seq;
        uint4 kq[4], vq[4];
        float sc;
        auto load = [&](const uint8_t* from, uint32_t j, uint4 (&q)[4]) {       // positions past the last visible one repeat it
#pragma unroll
            for (int i = 0; i < 4; ++i) q[i] = __ldg(reinterpret_cast<const uint4*>(from + static_cast<size_t>(min(j * BP + 16 * i + row0, last)) * HD));
        };
        load(kc, 0, kq);
        sc = __ldg(scale + min(tid & 63, last));
        load(vc, 0, vq);
        for (uint32_t j = 0; j < nb; ++j) {
            const uint32_t b = j & 1, par = ((j >> 1) - 1) & 1;
            bool ok = true;
            if (j >= 2) ok = mbar_wait_bounded(&s_full[b], par, status);        // S(j-2) is there: its K block and the scales of j-4 are free
            if (!__all_sync(0xffffffffu, ok)) break;
#pragma unroll
            for (int i = 0; i < 4; ++i) store_codes(ks + b * KV_BYTES, 16 * i + row0, c16, kq[i]);
            const uint32_t slot = j % SLOTS;
            if (tid < BP) {
                s_ks[slot][tid] = sc * 1.4426950408889634f;                     // scores in units of log2
            } else {
                s_vs[slot][tid - BP] = sc * 256.0f;                             // keeps small products out of the f16 subnormals
                float top = fabsf(sc);
                for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
                if (lane == 0) s_vmax[slot][(tid - BP) >> 5] = top;
            }
            proxy_fence();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&sc_full[slot]);
                mbar_arrive(&k_full[b]);
            }
            if (j + 1 < nb) {
                load(kc, j + 1, kq);
                sc = __ldg(scale + min((j + 1) * BP + (tid & 63), last));
            }
            if (j >= 2) ok = mbar_wait_bounded(&o_done[b], par, status);        // the output of j-2 is in: its V block is free
            if (!__all_sync(0xffffffffu, ok)) break;
#pragma unroll
            for (int i = 0; i < 4; ++i) store_codes(vs + b * KV_BYTES, 16 * i + row0, c16, vq[i]);
            proxy_fence();
            __syncwarp();
            if (lane == 0) mbar_arrive(&v_full[b]);
            if (j + 1 < nb) load(vc, j + 1, vq);
        }
    } else if (warp == 8) {
        if (lane == 0) {
            // D f32, A and B f16, M = 128; S: both K-major, N = 64; O: B MN-major, N = 128
            constexpr uint32_t ID = (1u << 4) | ((ROWS >> 4) << 24), ID_S = ID | ((BP >> 3) << 17), ID_O = ID | (1u << 16) | ((HD >> 3) << 17);
            bool ok = true;
            auto scores = [&](uint32_t j) {
                const uint32_t b = j & 1;
                ok = mbar_wait_bounded(&k_full[b], (j >> 1) & 1, status);
                if (ok && j >= 2) ok = mbar_wait_bounded(&o_done[b], ((j >> 1) - 1) & 1, status);   // P(j-2) is read: S(j) takes its place
                if (!ok) return;
                tc_fence_after();
#pragma unroll
                for (uint32_t kk = 0; kk < HD / 16; ++kk)
                    umma_ss(tmem + b * BP, smem_desc_sw128(smem_u32(qs + (kk >> 2) * (ROWS * 128))) + 2 * (kk & 3),
                            smem_desc_sw128(smem_u32(ks + b * KV_BYTES + (kk >> 2) * PANEL)) + 2 * (kk & 3), ID_S, kk ? 1u : 0u);
                tc_commit(&s_full[b]);
            };
            scores(0);
            for (uint32_t j = 0; j < nb && ok; ++j) {
                const uint32_t b = j & 1;
                if (j + 1 < nb) scores(j + 1);
                if (ok) ok = mbar_wait_bounded(&v_full[b], (j >> 1) & 1, status);
                if (ok) ok = mbar_wait_bounded(&p_full[b], (j >> 1) & 1, status);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (uint32_t kk = 0; kk < BP / 16; ++kk)
                    umma_ts(tmem + COL_O, tmem + b * BP + 8 * kk, smem_desc_mn_sw128(smem_u32(vs + b * KV_BYTES), PANEL) + kk * (16 * 128 >> 4), ID_O, (j | kk) ? 1u : 0u);
                tc_commit(&o_done[b]);
            }
        }
    } else {
        const uint32_t row = threadIdx.x, tok = tok0 + row / G, at = tmem + ((warp * 32u) << 16);
        const bool live = tok < m;
        const uint32_t seen = live ? pos0 + tok : last;            // (rows past the end compute on zeros and are not stored)
        float mx = -CUDART_INF_F;
        f2 sum = 0;
        bool ok = true;
        for (uint32_t j = 0; j < nb; ++j) {
            const uint32_t b = j & 1, slot = j % SLOTS;
            ok = mbar_wait_bounded(&s_full[b], (j >> 1) & 1, status);
            if (ok) ok = mbar_wait_bounded(&sc_full[slot], (j / SLOTS) & 1, status);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            // twice over the scores, 32 columns at a time: the maximum, then the exponentials (all 64 would not fit the registers)
            const ulonglong2 *k2 = reinterpret_cast<const ulonglong2*>(s_ks[slot]), *v2 = reinterpret_cast<const ulonglong2*>(s_vs[slot]);
            const bool diagonal = (j + 1) * BP > pos0 + tok0;      // only the blocks at the diagonal hold positions that a row must not see
            float top[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
            auto largest = [&](auto masked) {
#pragma unroll
                for (uint32_t half = 0; half < 2; ++half) {
                    uint32_t r[32];
                    tmem_ld32(at + b * BP + 32 * half, r);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const ulonglong2 k = k2[8 * half + i / 2];
                        float2 x = f2_parts(f2_mul(f2_of(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), i & 1 ? k.y : k.x));
                        if constexpr (decltype(masked)::value) x = hide(x, j * BP + 32 * half + 2 * i, seen, -CUDART_INF_F);
                        top[2 * (i & 1)] = fmaxf(top[2 * (i & 1)], x.x);
                        top[2 * (i & 1) + 1] = fmaxf(top[2 * (i & 1) + 1], x.y);
                    }
                }
            };
            if (diagonal) largest(std::true_type{}); else largest(std::false_type{});
            const float bm = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
            const float room = fmaxf(s_vmax[slot][0], s_vmax[slot][1]) < LAZY_VMAX ? LAZY_LOG2 : 0.0f;
            const bool grew = bm > mx + room;
            if (j == 0) {
                mx = bm;                                           // finite: position 0 is visible to every row
            } else if (__any_sync(0xffffffffu, grew)) {
                const float to = grew ? bm : mx, corr = grew ? ex2(mx - to) : 1.0f;
                mx = to;
                const f2 c2 = f2_both(corr);
                sum = f2_mul(sum, c2);
                ok = __all_sync(0xffffffffu, mbar_wait_bounded(&o_done[b ^ 1], ((j - 1) >> 1) & 1, status));
                if (!ok) break;
                tc_fence_after();
#pragma unroll 1
                for (uint32_t c = 0; c < HD; c += 16) {
                    uint32_t o[16];
                    tmem_ld16(at + COL_O + c, o);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                    tmem_st16(at + COL_O + c, o);
                }
            }
            const f2 nm = f2_both(-mx);
            f2 part = 0;
            auto weights = [&](auto masked) {
#pragma unroll
                for (uint32_t c = 0; c < 4; ++c) {
                    uint32_t r[16], p[8];
                    tmem_ld16(at + b * BP + 16 * c, r);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const ulonglong2 k = k2[4 * c + i / 2], v = v2[4 * c + i / 2];
                        float2 d = f2_parts(f2_fma(f2_of(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), i & 1 ? k.y : k.x, nm));
                        if constexpr (decltype(masked)::value) d = hide(d, j * BP + 16 * c + 2 * i, seen, -CUDART_INF_F);
                        const f2 e = f2_of(ex2(d.x), ex2(d.y));
                        part = f2_add(part, e);
                        float2 w = f2_parts(f2_mul(e, i & 1 ? v.y : v.x));
                        if constexpr (decltype(masked)::value) w = hide(w, j * BP + 16 * c + 2 * i, seen, 0.f);
                        p[i] = pack_h2(w.x, w.y);
                    }
                    tmem_st8(at + b * BP + 8 * c, p);          // over scores that have been read
                }
            };
            if (diagonal) weights(std::true_type{}); else weights(std::false_type{});
            sum = f2_add(sum, part);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[b]);
        }
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait_bounded(&o_done[(nb - 1) & 1], ((nb - 1) >> 1) & 1, status));
        if (ok) {
            tc_fence_after();
            const float l = f2_sum(sum), inv = l > 0.f ? (1.0f / 256.0f) / l : 0.f;
            OUT* dst = out + static_cast<size_t>(live ? tok : 0) * out_stride + (static_cast<size_t>(kvh) * G + row % G) * HD;
            const bool wide = reinterpret_cast<uintptr_t>(out) % 16 == 0;      // rows are whole numbers of heads
            bool clipped = false;
#pragma unroll 1
            for (uint32_t c = 0; c < HD; c += 32) {
                uint32_t o[32];
                tmem_ld32(at + COL_O + c, o);
                tmem_wait_ld();
                if (live) {
                    float v[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(o[i]) * inv;
                    if constexpr (std::is_same_v<OUT, float>) {
                        if (wide) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) reinterpret_cast<float4*>(dst + c)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                        } else {
                            for (int i = 0; i < 32; ++i) dst[c + i] = v[i];
                        }
                    } else {
                        __align__(16) OUT h[32];
#pragma unroll
                        for (int i = 0; i < 32; ++i) h[i] = out_value<OUT>(v[i], clipped);
                        if (wide) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) reinterpret_cast<uint4*>(dst + c)[i] = reinterpret_cast<const uint4*>(h)[i];
                        } else {
                            for (int i = 0; i < 32; ++i) dst[c + i] = h[i];
                        }
                    }
                }
                __syncwarp();                                  // the next load from tensor memory is the whole warp's
            }
            if (clipped) atomicOr(status, STATUS_X_CLIPPED);
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 8) { tc_fence_after(); tmem_dealloc(tmem, COLS); }
}

// Few positions in all: the tcgen05 kernel's start (barriers, tensor memory, one block's chain of four steps) takes 7 us however
// few there are.  Here the codes of one KV head go to shared memory and a warp takes a row in f32: lane = position for the
// scores, lane = four dims for the output.  Bound by the latency of its loads.  32 heads over 8, first portion of a sequence:
// 1 token 3.5 us (tcgen05 7.0), 17 tokens 5.1 (9.2), 33 tokens 5.7 (10.9).  The line: 64 heads over 8 take as long
// either way at 48 positions (10.1, 10.5); 32 over 8 would gain up to 64 of them (64: 9.0, 10.6).
constexpr uint32_t FEW = 48, FEW_WARPS = 8;

template <int G, typename OUT>
__global__ void __launch_bounds__(FEW_WARPS * 32) attn_prefill_few_kernel(const float* __restrict__ qkv, uint32_t row_stride, uint32_t m,
                                                                          const int8_t* __restrict__ k_codes, const float* __restrict__ k_scale,
                                                                          const int8_t* __restrict__ v_codes, const float* __restrict__ v_scale,
                                                                          uint32_t max_seq, uint32_t pos0, OUT* __restrict__ out, uint32_t out_stride,
                                                                          uint32_t* status) {
    __shared__ uint32_t ks[FEW][HD / 4 + 1], vs[FEW][HD / 4 + 1];  // code + 128 in every byte
    __shared__ float k_s[FEW], v_s[FEW];
    __shared__ __align__(16) float qs[FEW_WARPS][HD];
    const uint32_t kvh = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.x * FEW_WARPS + warp, tok = row / G;
    const uint32_t n = pos0 + min((blockIdx.x * FEW_WARPS + FEW_WARPS - 1) / G, m - 1) + 1;        // positions that a row of this CTA sees
    const size_t first = static_cast<size_t>(kvh) * max_seq;
    for (uint32_t i = threadIdx.x; i < n * 8; i += FEW_WARPS * 32) {
        const uint32_t p = i >> 3, c = i & 7;
        const uint4 k = __ldg(reinterpret_cast<const uint4*>(k_codes + (first + p) * HD) + c), v = __ldg(reinterpret_cast<const uint4*>(v_codes + (first + p) * HD) + c);
        const uint32_t kw[4] = {k.x, k.y, k.z, k.w}, vw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            ks[p][4 * c + j] = kw[j] ^ 0x80808080u;
            vs[p][4 * c + j] = vw[j] ^ 0x80808080u;
        }
    }
    if (threadIdx.x < n) {
        k_s[threadIdx.x] = __ldg(k_scale + first + threadIdx.x);
        v_s[threadIdx.x] = __ldg(v_scale + first + threadIdx.x);
    }
    if (tok < m)
        reinterpret_cast<float4*>(qs[warp])[lane] = __ldg(reinterpret_cast<const float4*>(qkv + static_cast<size_t>(tok) * row_stride + (static_cast<size_t>(kvh) * G + row % G) * HD) + lane);
    __syncthreads();
    if (tok >= m) return;
    const uint32_t seen = pos0 + tok, p0 = min(lane, n - 1), p1 = min(lane + 32, n - 1);
    float s0 = 0.f, s1 = 0.f;
#pragma unroll 8
    for (uint32_t w = 0; w < HD / 4; ++w) {
        const float4 q = reinterpret_cast<const float4*>(qs[warp])[w];
        const float qv[4] = {q.x, q.y, q.z, q.w};
        const uint32_t k0 = ks[p0][w], k1 = ks[p1][w];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            s0 = fmaf(qv[j], byte_to_float<128>(k0, j), s0);
            s1 = fmaf(qv[j], byte_to_float<128>(k1, j), s1);
        }
    }
    s0 = lane <= seen ? s0 * k_s[p0] : -CUDART_INF_F;
    s1 = lane + 32 <= seen ? s1 * k_s[p1] : -CUDART_INF_F;
    float mx = fmaxf(s0, s1);
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float e0 = expf(s0 - mx), e1 = expf(s1 - mx);
    float l = e0 + e1, o[4] = {0.f, 0.f, 0.f, 0.f};
    for (int d = 16; d > 0; d >>= 1) l += __shfl_xor_sync(0xffffffffu, l, d);
    for (uint32_t p = 0; p <= seen; ++p) {
        const float w = __shfl_sync(0xffffffffu, p < 32 ? e0 : e1, p & 31) * v_s[p];
        const uint32_t v = vs[p][lane];
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = fmaf(w, byte_to_float<128>(v, j), o[j]);
    }
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    OUT* dst = out + static_cast<size_t>(tok) * out_stride + (static_cast<size_t>(kvh) * G + row % G) * HD + 4 * lane;
    bool clipped = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) dst[j] = out_value<OUT>(o[j] * inv, clipped);
    if (clipped) atomicOr(status, STATUS_X_CLIPPED);
}

template <int G, typename OUT>
cudaError_t launch_prefill_g(const float* qkv, uint32_t row_stride, uint32_t m, const KvCacheView& kv, uint32_t n_kv, uint32_t pos0, OUT* out,
                             uint32_t out_stride, uint32_t* status, cudaStream_t st) {
    if (static_cast<uint64_t>(pos0) + m <= FEW) {
        attn_prefill_few_kernel<G, OUT><<<dim3((m * G + FEW_WARPS - 1) / FEW_WARPS, n_kv), FEW_WARPS * 32, 0, st>>>(
            qkv, row_stride, m, kv.k_codes, kv.k_scale, kv.v_codes, kv.v_scale, kv.max_seq, pos0, out, out_stride, status);
        return cudaGetLastError();
    }
    static PerDeviceFlag flag;
    if (const cudaError_t e = ensure_max_dynamic_smem(attn_prefill_kernel<G, OUT>, AP_SMEM, flag); e != cudaSuccess) return e;
    constexpr uint32_t TOK = ROWS / G;
    attn_prefill_kernel<G, OUT><<<n_kv * ((m + TOK - 1) / TOK), AP_THREADS, AP_SMEM, st>>>(
        qkv, row_stride, m, kv.k_codes, kv.k_scale, kv.v_codes, kv.v_scale, kv.max_seq, pos0, n_kv, out, out_stride, status);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_attn_prefill(const float* qkv, uint32_t row_stride, uint32_t m, uint32_t n_q, uint32_t n_kv, uint32_t hd,
                                const KvCacheView& kv, uint32_t pos0, void* out, uint32_t out_dtype, uint32_t out_stride, uint32_t* status,
                                cudaStream_t st) {
    if (hd != HD || n_kv == 0 || n_q % n_kv) return cudaErrorInvalidValue;
    switch (n_q / n_kv) {
#define HF2Q_CASE(GG) case GG: \
        if (out_dtype == HF2Q_DT_F32) return launch_prefill_g<GG, float>(qkv, row_stride, m, kv, n_kv, pos0, static_cast<float*>(out), out_stride, status, st); \
        if (out_dtype == HF2Q_DT_F16) return launch_prefill_g<GG, __half>(qkv, row_stride, m, kv, n_kv, pos0, static_cast<__half*>(out), out_stride, status, st); \
        if (out_dtype == HF2Q_DT_BF16) return launch_prefill_g<GG, __nv_bfloat16>(qkv, row_stride, m, kv, n_kv, pos0, static_cast<__nv_bfloat16*>(out), out_stride, status, st); \
        return cudaErrorInvalidValue;
        HF2Q_CASE(1) HF2Q_CASE(2) HF2Q_CASE(4) HF2Q_CASE(8)
#undef HF2Q_CASE
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace hf2q
