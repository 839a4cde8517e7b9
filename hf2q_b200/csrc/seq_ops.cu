// Row-wise steps around the products of a bf16-weight decoder: embedding rows with the hashed bigram table, the
// residual update + RMS norm + token shift in front of a product, the same for a residual in several streams, gated head outputs, and the hand-over of the
// shift / convolution state after a portion of several tokens.
#include <initializer_list>

#include "seq_common.cuh"

namespace hf2q {
namespace {
using namespace seq;

__global__ void __launch_bounds__(256) embed_kernel(const __grid_constant__ hf2q_embed e, const uint32_t* ids, uint32_t m,
                                                    float* __restrict__ x, uint32_t* status) {
    pdl_trigger();
    pdl_wait();
    const uint32_t t = blockIdx.x;
    const uint32_t id = ids[t], pos = *e.pos + t;
    const uint32_t before = t ? ids[t - 1] : *e.prev;
    const uint32_t last = ids[m - 1];
    __syncthreads();                                       // row 0 reads *prev before it replaces it
    if (t == 0 && threadIdx.x == 0) *e.prev = last;
    const bool bad = id >= e.vocab;
    if (bad && threadIdx.x == 0) atomicOr(status, STATUS_BAD_EXPERT_ID);
    const __nv_bfloat16* row = static_cast<const __nv_bfloat16*>(e.embed) + static_cast<size_t>(bad ? 0 : id) * e.ld;
    const __nv_bfloat16* big = nullptr;
    if (e.bigram) {
        const uint64_t r = pos == 0 ? e.buckets : (before * e.mul_prev + id * e.mul_cur) % e.buckets;
        big = static_cast<const __nv_bfloat16*>(e.bigram) + r * e.ld;
    }
    for (uint32_t i = threadIdx.x; i < e.width; i += blockDim.x) {
        float v = bad ? 0.f : to_f32(row[i]);
        if (big) v += to_f32(big[i]);
        x[static_cast<size_t>(t) * e.width + i] = v;
    }
}

// `run` consecutive rows per CTA; a token shift needs the row before the first as well, recomputed from the same inputs
template <typename OUT>
__global__ void __launch_bounds__(512) pre_norm_kernel(const __grid_constant__ hf2q_pre_norm p, uint32_t m, uint32_t run, OUT* __restrict__ out, uint32_t ldo,
                                                       float* __restrict__ h_last) {
    extern __shared__ __align__(16) float xs[];            // width, and another width with a shift: the h of the row before
    __shared__ float red[64];
    pdl_trigger();
    pdl_wait();
    const uint32_t t0 = blockIdx.x * run, t1 = min(t0 + run, m);
    const uint32_t pos = p.shift ? *p.pos : 0u;
    float* before = xs + p.width;                          // an element is read and written by one thread only
    if (p.shift) {
        if (t0 > 0) {
            const float inv = residual_row(p, t0 - 1, before, red);
            for (uint32_t i = threadIdx.x; i < p.width; i += blockDim.x) before[i] *= inv * p.norm[i];
        } else {
            for (uint32_t i = threadIdx.x; i < p.width; i += blockDim.x) before[i] = p.shift_state[static_cast<size_t>((pos + 1) & 1) * p.width + i];
        }
    }
    const bool quads = p.width % 4 == 0 && ldo == p.width &&
                       ((reinterpret_cast<uintptr_t>(p.norm) | reinterpret_cast<uintptr_t>(p.shift) | reinterpret_cast<uintptr_t>(p.x_out) |
                         reinterpret_cast<uintptr_t>(p.shift_state) | reinterpret_cast<uintptr_t>(h_last) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    if (quads) __syncthreads();                            // `before` changes hands: groups of four per thread from here on
    for (uint32_t t = t0; t < t1; ++t) {
        const float inv = residual_row(p, t, xs, red);
        if (quads) {
            for (uint32_t i = threadIdx.x; i < p.width / 4; i += blockDim.x) {
                const float4 x = reinterpret_cast<const float4*>(xs)[i], w = reinterpret_cast<const float4*>(p.norm)[i];
                if (p.x_out) reinterpret_cast<float4*>(p.x_out + static_cast<size_t>(t) * p.width)[i] = x;
                float4 h = make_float4(x.x * inv * w.x, x.y * inv * w.y, x.z * inv * w.z, x.w * inv * w.w);
                if (p.shift) {
                    const float4 b = reinterpret_cast<const float4*>(before)[i], mu = reinterpret_cast<const float4*>(p.shift)[i];
                    reinterpret_cast<float4*>(before)[i] = h;
                    if (m == 1) reinterpret_cast<float4*>(p.shift_state + static_cast<size_t>(pos & 1) * p.width)[i] = h;
                    else if (t == m - 1) reinterpret_cast<float4*>(h_last)[i] = h;
                    h = make_float4(h.x + (b.x - h.x) * mu.x, h.y + (b.y - h.y) * mu.y, h.z + (b.z - h.z) * mu.z, h.w + (b.w - h.w) * mu.w);
                }
                OUT* dst = out + static_cast<size_t>(t) * ldo + 4 * i;
                if constexpr (sizeof(OUT) == 4) {
                    *reinterpret_cast<float4*>(dst) = h;
                } else {
                    const __nv_bfloat162 lo = __floats2bfloat162_rn(h.x, h.y), hi = __floats2bfloat162_rn(h.z, h.w);
                    *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                }
            }
            __syncthreads();
            continue;
        }
        for (uint32_t i = threadIdx.x; i < ldo; i += blockDim.x) {
            float h = 0.f;
            if (i < p.width) {
                const float x = xs[i];
                if (p.x_out) p.x_out[static_cast<size_t>(t) * p.width + i] = x;
                h = x * inv * p.norm[i];
                if (p.shift) {
                    const float b = before[i];
                    before[i] = h;
                    if (m == 1) p.shift_state[static_cast<size_t>(pos & 1) * p.width + i] = h;
                    else if (t == m - 1) h_last[i] = h;
                    h += (b - h) * p.shift[i];
                }
            }
            out[static_cast<size_t>(t) * ldo + i] = from_f32<OUT>(h);
        }
        __syncthreads();                                   // xs is read across threads before the next row replaces it
    }
}

template <typename OUT>
__global__ void __launch_bounds__(512) hyper_norm_kernel(const __grid_constant__ hf2q_hyper p, OUT* __restrict__ out, uint32_t ldo) {
    extern __shared__ __align__(16) float xs[];
    __shared__ float coef[HYPER_COEF];
    __shared__ float red[32];
    pdl_trigger();
    pdl_wait();
    const uint32_t t = blockIdx.x;
    const float inv = hyper_row(p, t, xs, coef, red, 0, p.width);
    OUT* row = out + static_cast<size_t>(t) * ldo;
    if (p.width % 4 == 0 && ldo % 4 == 0 && ((reinterpret_cast<uintptr_t>(p.norm) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
        for (uint32_t i = threadIdx.x; i < ldo / 4; i += blockDim.x) {
            float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
            if (4 * i < p.width) {
                h = reinterpret_cast<const float4*>(xs)[i];
                if (p.norm) {
                    const float4 w = reinterpret_cast<const float4*>(p.norm)[i];
                    h = make_float4(h.x * inv * w.x, h.y * inv * w.y, h.z * inv * w.z, h.w * inv * w.w);
                }
            }
            if constexpr (sizeof(OUT) == 4) {
                reinterpret_cast<float4*>(row)[i] = h;
            } else {
                const __nv_bfloat162 a = __floats2bfloat162_rn(h.x, h.y), b = __floats2bfloat162_rn(h.z, h.w);
                reinterpret_cast<uint2*>(row)[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
            }
        }
        return;
    }
    for (uint32_t i = threadIdx.x; i < ldo; i += blockDim.x)
        row[i] = from_f32<OUT>(i < p.width ? (p.norm ? xs[i] * inv * p.norm[i] : xs[i]) : 0.f);
}

// ---- the same two for rows of whole 16-byte groups, one group per thread
// Bound by memory.  A CTA walks rows with everything of a row in registers and asks for the next row before it waits for the sums of
// this one; one row per CTA, through shared memory, left half of the time without a load in flight.  2048 rows of 2048:
// hyper_norm with four streams moves 160 MB, 47 - 53 us before, 30 - 32 now; pre_norm with a pending pair 76 MB, 28 and 17.7.
constexpr uint32_t ROW_THREADS = 1024;
template <typename OUT> __device__ __forceinline__ void store4(OUT* dst, const float4& h) {
    if constexpr (sizeof(OUT) == 4) {
        *reinterpret_cast<float4*>(dst) = h;
    } else {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(h.x, h.y), hi = __floats2bfloat162_rn(h.z, h.w);
        *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
}
template <typename OUT> __device__ __forceinline__ void clear_tail(OUT* row, uint32_t width, uint32_t ldo) {       // both multiples of four
    for (uint32_t i = width + 4 * threadIdx.x; i < ldo; i += 4 * blockDim.x) store4(row + i, make_float4(0.f, 0.f, 0.f, 0.f));
}
__device__ __forceinline__ float4 scaled(const float4& a, float c, const float4& b) { return make_float4(a.x * c * b.x, a.y * c * b.y, a.z * c * b.z, a.w * c * b.w); }
__device__ __forceinline__ float4 load4(const float* p, uint32_t i) { return *reinterpret_cast<const float4*>(p + 4 * i); }

// run consecutive rows per CTA
template <typename OUT, bool PAIR>
__global__ void __launch_bounds__(ROW_THREADS) pre_norm_rows_kernel(const __grid_constant__ hf2q_pre_norm p, uint32_t m, uint32_t run, OUT* __restrict__ out, uint32_t ldo,
                                                                    float* __restrict__ h_last) {
    __shared__ float red[2][3 * 32];
    pdl_trigger();
    pdl_wait();
    const uint32_t i = threadIdx.x, t0 = blockIdx.x * run, t1 = min(t0 + run, m);
    const bool has = i < p.width / 4;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto constant = [&](const float* q) { return q && has ? load4(q, i) : zero; };
    const float4 norm = constant(p.norm), mu = constant(p.shift), step = constant(p.step), an = constant(p.a_norm), bn = constant(p.b_norm);
    const float n = static_cast<float>(p.width);
    float4 x, a, b, add;
    auto load = [&](uint32_t t) {
        const size_t o = static_cast<size_t>(t) * p.width;
        x = has ? load4(p.x + o, i) : zero;
        if constexpr (PAIR) { a = has ? load4(p.a + o, i) : zero; b = has ? load4(p.b + o, i) : zero; }
        add = p.add0 && has ? load4(p.add0 + o, i) : zero;
    };
    const uint32_t pos = p.shift ? *p.pos : 0u, first = p.shift && t0 ? t0 - 1 : t0;      // a token shift needs the row before as well
    load(first);
    float4 before = p.shift && t0 == 0 && has ? load4(p.shift_state + static_cast<size_t>((pos + 1) & 1) * p.width, i) : zero;
    for (uint32_t t = first; t < t1; ++t) {
        float* r = red[t & 1];                             // (a warp may still read the other row's)
        float4 v = x;
        if constexpr (PAIR) {
            float s[2] = {square_sum(a), square_sum(b)};
            block_sum(s, r);
            const float ia = 0.5f / sqrtf(s[0] / n + p.eps), ib = 0.5f / sqrtf(s[1] / n + p.eps);
            v.x += a.x * ia * an.x + b.x * ib * bn.x; v.y += a.y * ia * an.y + b.y * ib * bn.y;
            v.z += a.z * ia * an.z + b.z * ib * bn.z; v.w += a.w * ia * an.w + b.w * ib * bn.w;
        }
        if (p.add0) { v.x += add.x; v.y += add.y; v.z += add.z; v.w += add.w; }
        if (p.step) { v.x += step.x; v.y += step.y; v.z += step.z; v.w += step.w; }
        if (t + 1 < t1) load(t + 1);
        float s[1] = {square_sum(v)};
        block_sum(s, r + 64);
        float4 h = scaled(v, 1.0f / sqrtf(s[0] / n + p.eps), norm);
        if (t >= t0 && has) {
            if (p.x_out) *reinterpret_cast<float4*>(p.x_out + static_cast<size_t>(t) * p.width + 4 * i) = v;
            float4 o = h;
            if (p.shift) {
                if (m == 1) *reinterpret_cast<float4*>(p.shift_state + static_cast<size_t>(pos & 1) * p.width + 4 * i) = h;
                else if (t == m - 1) *reinterpret_cast<float4*>(h_last + 4 * i) = h;
                o = make_float4(h.x + (before.x - h.x) * mu.x, h.y + (before.y - h.y) * mu.y, h.z + (before.z - h.z) * mu.z, h.w + (before.w - h.w) * mu.w);
            }
            store4(out + static_cast<size_t>(t) * ldo + 4 * i, o);
        }
        if (t >= t0) clear_tail(out + static_cast<size_t>(t) * ldo, p.width, ldo);
        before = h;
    }
}

// S: streams, at most; every gridDim.x-th row
constexpr int HELD_PARTS = 4;                              // rows of a pending output in flight at a time
template <int S, typename OUT>
__global__ void __launch_bounds__(ROW_THREADS) hyper_norm_rows_kernel(const __grid_constant__ hf2q_hyper p, uint32_t m, OUT* __restrict__ out, uint32_t ldo) {
    __shared__ float coef[S * S + 2 * S], red[2][32];
    pdl_trigger();
    pdl_wait();
    const uint32_t i = threadIdx.x, n = p.width / 4;
    const bool has = i < n;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), norm = p.norm && has ? load4(p.norm, i) : make_float4(1.f, 1.f, 1.f, 1.f);
    hyper_coefficients<S>(p, coef);
    const float *mix = coef, *gain = coef + S * S, *in = gain + S;
    float4 old[S], y[HELD_PARTS];
    auto load_y = [&](uint32_t t, uint32_t k0) {
#pragma unroll
        for (int k = 0; k < HELD_PARTS; ++k)
            y[k] = p.y && has && k0 + k < p.y_parts ? load4(p.y + (static_cast<size_t>(t) * p.y_parts + k0 + k) * p.width, i) : zero;
    };
    auto load = [&](uint32_t t) {
        const float* x = p.x + static_cast<size_t>(t) * p.x_streams * p.width;
#pragma unroll
        for (int s = 0; s < S; ++s) old[s] = has && s < static_cast<int>(p.streams) ? load4(x + (p.x_streams == 1 ? 0u : s * p.width), i) : zero;
        load_y(t, 0);
    };
    if (blockIdx.x < m) load(blockIdx.x);
    uint32_t turn = 0;
    for (uint32_t t = blockIdx.x; t < m; t += gridDim.x, turn ^= 1) {
        float4 yv = zero, u = zero;
        for (uint32_t k0 = 0;;) {
#pragma unroll
            for (int k = 0; k < HELD_PARTS; ++k) axpy(yv, 1.0f, y[k]);
            if (!p.y || (k0 += HELD_PARTS) >= p.y_parts) break;
            load_y(t, k0);
        }
#pragma unroll
        for (int d = 0; d < S; ++d) {
            if (d >= static_cast<int>(p.streams)) continue;
            float4 v = old[d];
            if (p.y) {
                v = zero;
#pragma unroll
                for (int s = 0; s < S; ++s) axpy(v, mix[s * S + d], old[s]);
                axpy(v, gain[d], yv);
            }
            if (p.x_out && has) *reinterpret_cast<float4*>(p.x_out + (static_cast<size_t>(t) * p.streams + d) * p.width + 4 * i) = v;
            axpy(u, in[d], v);
        }
        if (t + gridDim.x < m) load(t + gridDim.x);
        float s[1] = {square_sum(u)};
        block_sum(s, red[turn]);
        const float inv = p.norm ? 1.0f / sqrtf(s[0] / static_cast<float>(p.width) + p.eps) : 1.0f;
        OUT* row = out + static_cast<size_t>(t) * ldo;
        if (has) store4(row + 4 * i, scaled(u, inv, norm));
        clear_tail(row, p.width, ldo);
    }
}

template <typename OUT>
__global__ void __launch_bounds__(256) gated_heads_kernel(const __grid_constant__ hf2q_gated_heads g, OUT* __restrict__ out, uint32_t ldo) {
    pdl_trigger();
    pdl_wait();
    const uint32_t t = blockIdx.x;
    OUT* row = out + static_cast<size_t>(t) * ldo;
    for (uint32_t i = g.heads * g.head_dim + threadIdx.x; i < ldo; i += blockDim.x) row[i] = from_f32<OUT>(0.f);
    extern __shared__ __align__(16) float buf[];
    if (g.kind == HF2Q_GATE_SILU_FIRST) silu_group_norm_row<OUT>(g, t, buf, row);
    else gated_heads_row<OUT>(g, t, row, threadIdx.x >> 5, blockDim.x >> 5);
}

__global__ void __launch_bounds__(256) state_tail_kernel(const uint32_t* pos_dev, uint32_t m, const float* h_last,
                                                         float* __restrict__ shift_state, uint32_t width, const __grid_constant__ hf2q_delta d,
                                                         uint32_t channels) {
    pdl_trigger();
    pdl_wait();
    const uint32_t pos = *pos_dev;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (shift_state && i < width) shift_state[static_cast<size_t>((pos + m - 1) & 1) * width + i] = h_last[i];
    if (i < channels) {
        // inputs of the last taps - 1 positions; those before this portion are in the state already
        const uint32_t qk = d.kv_heads * d.dim;
        const uint32_t col = i < qk ? d.q_off + i : i < 2 * qk ? d.k_off + (i - qk) : d.v_off + (i - 2 * qk);
        const uint32_t keep = d.taps - 1 < m ? d.taps - 1 : m;
        for (uint32_t j = 0; j < keep; ++j) {
            const uint32_t t = m - 1 - j;
            d.conv_state[static_cast<size_t>(i) * d.taps + (pos + t) % d.taps] = d.proj[static_cast<size_t>(t) * d.ld + col];
        }
    }
}

// whole 16-byte groups, one per thread of a CTA
bool row_groups(uint32_t width, uint32_t ldo, std::initializer_list<const void*> all) {
    if (width % 4 || ldo % 4 || width > 4 * ROW_THREADS) return false;
    for (const void* q : all)
        if (reinterpret_cast<uintptr_t>(q) % 16) return false;
    return true;
}
// a thread per group; as many CTAs as stay on the chip
dim3 row_block(uint32_t width) { return dim3((width / 4 + 31) / 32 * 32); }
uint32_t row_ctas(uint32_t width, int sms) { return static_cast<uint32_t>(sms) * (ROW_THREADS / row_block(width).x); }

template <typename OUT>
cudaError_t launch_pre_norm(const hf2q_pre_norm& p, uint32_t m, OUT* out, uint32_t ldo, float* h_last, int sms, cudaStream_t st) {
    if (row_groups(p.width, ldo, {p.x, p.a, p.b, p.a_norm, p.b_norm, p.add0, p.step, p.norm, p.shift, p.x_out, p.shift_state, h_last, out})) {
        const uint32_t most = row_ctas(p.width, sms), run = (m + most - 1) / most;
        const dim3 grid((m + run - 1) / run);
        return p.a ? launch_pdl(pre_norm_rows_kernel<OUT, true>, grid, row_block(p.width), 0, st, p, m, run, out, ldo, h_last)
                   : launch_pdl(pre_norm_rows_kernel<OUT, false>, grid, row_block(p.width), 0, st, p, m, run, out, ldo, h_last);
    }
    const size_t smem = static_cast<size_t>(p.width) * (p.shift ? 8 : 4);
    static PerDeviceFlag flag;
    if (const cudaError_t e = ensure_max_dynamic_smem(pre_norm_kernel<OUT>, 200 * 1024, flag); e != cudaSuccess) return e;
    // long portions: a few rows per CTA while every SM keeps several CTAs
    const uint32_t run = p.shift && m >= 4u * 4u * static_cast<uint32_t>(sms) ? 8 : p.shift && m >= 512 ? 4 : 1;
    return launch_pdl(pre_norm_kernel<OUT>, dim3((m + run - 1) / run), dim3(p.width >= 2048 ? 512 : 256), smem, st, p, m, run, out, ldo, h_last);
}
template <typename OUT>
cudaError_t launch_hyper_norm(const hf2q_hyper& p, uint32_t m, OUT* out, uint32_t ldo, int sms, cudaStream_t st) {
    if (p.streams <= 4 && row_groups(p.width, ldo, {p.x, p.x_out, p.y, p.norm, out})) {
        const uint32_t most = row_ctas(p.width, sms);
        const dim3 grid(m < most ? m : most);
        return p.streams <= 2 ? launch_pdl(hyper_norm_rows_kernel<2, OUT>, grid, row_block(p.width), 0, st, p, m, out, ldo)
                              : launch_pdl(hyper_norm_rows_kernel<4, OUT>, grid, row_block(p.width), 0, st, p, m, out, ldo);
    }
    static PerDeviceFlag flag;
    if (const cudaError_t e = ensure_max_dynamic_smem(hyper_norm_kernel<OUT>, 200 * 1024, flag); e != cudaSuccess) return e;
    return launch_pdl(hyper_norm_kernel<OUT>, dim3(m), dim3(p.width >= 2048 ? 512 : 256), static_cast<size_t>(p.width) * 4, st, p, out, ldo);
}

}  // namespace
}  // namespace hf2q

using namespace hf2q;
using namespace hf2q::seq;

extern "C" {

HF2Q_API int32_t hf2q_cuda_embed(hf2q_ctx* ctx, void* stream, const hf2q_embed* e, const uint32_t* ids, uint32_t m, float* x) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!e || !e->embed || !e->pos || !e->prev || !ids || !x || e->vocab == 0 || e->width == 0 || e->ld < e->width || (e->bigram && e->buckets == 0))
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "embed: null pointer or empty table");
    if (m == 0) return HF2Q_OK;
    const cudaError_t r = launch_pdl(embed_kernel, dim3(m), dim3(256), 0, static_cast<cudaStream_t>(stream), *e, ids, m, x, ctx_status_word(ctx));
    return ctx_cuda_result(ctx, r, "embed", 1);
}

HF2Q_API int32_t hf2q_cuda_pre_norm(hf2q_ctx* ctx, void* stream, const hf2q_pre_norm* p, uint32_t m, void* out, uint32_t out_dtype, uint32_t ldo,
                                    float* h_last) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!p || !p->x || !p->norm || !out || p->width == 0 || ldo < p->width || p->x_out == p->x || (p->a && (!p->b || !p->a_norm || !p->b_norm)) ||
        (p->shift && (!p->shift_state || !p->pos || (m > 1 && !h_last))) || !pre_norm_aligned(*p))
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "pre_norm: null or unaligned pointer, or x_out is x");
    if (m == 0) return HF2Q_OK;
    const size_t smem = static_cast<size_t>(p->width) * (p->shift ? 8 : 4);
    if (smem > 200 * 1024) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "pre_norm: width too large");
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int sms = ctx_sm_count(ctx);
    cudaError_t e = cudaErrorInvalidValue;
    if (out_dtype == HF2Q_DT_F32) e = launch_pre_norm(*p, m, static_cast<float*>(out), ldo, h_last, sms, st);
    else if (out_dtype == HF2Q_DT_BF16) e = launch_pre_norm(*p, m, static_cast<__nv_bfloat16*>(out), ldo, h_last, sms, st);
    return ctx_cuda_result(ctx, e, "pre_norm", 1);
}

HF2Q_API int32_t hf2q_cuda_gated_heads(hf2q_ctx* ctx, void* stream, const hf2q_gated_heads* g, uint32_t m, void* out, uint32_t out_dtype, uint32_t ldo) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!g || !gated_ok(*g) || !out || ldo < g->heads * g->head_dim) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "gated_heads: null pointer or a short row");
    if (m == 0) return HF2Q_OK;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t smem = g->kind == HF2Q_GATE_SILU_FIRST ? static_cast<size_t>(g->heads) * g->head_dim * 4 : 0;
    if (smem > 200 * 1024) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "gated_heads: row too long");
    static PerDeviceFlag f32f, bff;
    cudaError_t e = cudaErrorInvalidValue;
    if (out_dtype == HF2Q_DT_F32) {
        e = ensure_max_dynamic_smem(gated_heads_kernel<float>, 200 * 1024, f32f);
        if (e == cudaSuccess) e = launch_pdl(gated_heads_kernel<float>, dim3(m), dim3(256), smem, st, *g, static_cast<float*>(out), ldo);
    } else if (out_dtype == HF2Q_DT_BF16) {
        e = ensure_max_dynamic_smem(gated_heads_kernel<__nv_bfloat16>, 200 * 1024, bff);
        if (e == cudaSuccess) e = launch_pdl(gated_heads_kernel<__nv_bfloat16>, dim3(m), dim3(256), smem, st, *g, static_cast<__nv_bfloat16*>(out), ldo);
    }
    return ctx_cuda_result(ctx, e, "gated_heads", 1);
}

HF2Q_API int32_t hf2q_cuda_hyper_norm(hf2q_ctx* ctx, void* stream, const hf2q_hyper* p, uint32_t m, void* out, uint32_t out_dtype, uint32_t ldo) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!p || !hyper_ok(*p) || !out || ldo < p->width) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "hyper_norm: null or unaligned pointer, a bad number of streams or a short row");
    if (m == 0) return HF2Q_OK;
    const size_t smem = static_cast<size_t>(p->width) * 4;
    if (smem > 200 * 1024) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "hyper_norm: width too large");
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int sms = ctx_sm_count(ctx);
    cudaError_t e = cudaErrorInvalidValue;
    if (out_dtype == HF2Q_DT_F32) e = launch_hyper_norm(*p, m, static_cast<float*>(out), ldo, sms, st);
    else if (out_dtype == HF2Q_DT_BF16) e = launch_hyper_norm(*p, m, static_cast<__nv_bfloat16*>(out), ldo, sms, st);
    return ctx_cuda_result(ctx, e, "hyper_norm", 1);
}

HF2Q_API int32_t hf2q_cuda_state_tail(hf2q_ctx* ctx, void* stream, const uint32_t* pos, uint32_t m, const float* h_last, float* shift_state,
                                      uint32_t width, const hf2q_delta* delta) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!pos || m == 0 || (shift_state && !h_last) || (delta && (!delta->proj || !delta->conv_state || delta->taps == 0)))
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "state_tail: null pointer");
    const uint32_t channels = delta && delta->taps > 1 ? 2 * delta->kv_heads * delta->dim + delta->heads * delta->vdim : 0;
    const uint32_t n = shift_state && width > channels ? width : channels;
    if (n == 0) return HF2Q_OK;
    const hf2q_delta none{};
    const cudaError_t e = launch_pdl(state_tail_kernel, dim3((n + 255) / 256), dim3(256), 0, static_cast<cudaStream_t>(stream), pos, m, h_last,
                                     shift_state, width, delta ? *delta : none, channels);
    return ctx_cuda_result(ctx, e, "state_tail", 1);
}

}  // extern "C"
