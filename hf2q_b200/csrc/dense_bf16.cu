// Products with bf16 weights: y[m][n] = epilogue(x[m][k] . w[n][k]^T), f32 accumulation.
//
//   dense_matvec_kernel   m = 1..8 rows; weights streamed with 16-byte loads, activations f32 in shared memory, fp32
//                         arithmetic (HBM-bound: 2 bytes per weight against one FMA per row).  With one row the
//                         layer's norm / token shift / gating runs in the kernel's own prologue.
//   dense_gemm_tc_kernel  more rows, bf16 activations: persistent tcgen05 kernel, both operands by TMA with 128-byte
//                         swizzle, two accumulator buffers in tensor memory so that the epilogue of a tile runs under
//                         the main loop of the next.
//   dense_gemm_f32_kernel more rows, f32 activations: CUDA-core tiles in full 32-bit arithmetic.
// Both take rows sorted by group (expert) with one weight matrix per group as well.
#include "matvec_stream.cuh"
#include "seq_common.cuh"
#include "tc_common.cuh"

namespace hf2q {
namespace {
using namespace seq;

__device__ __forceinline__ float epilogue_value(float v, uint32_t epi, float cap) {
    if (epi == HF2Q_EPI_GELU) return gelu_tanhf(v);
    if (epi == HF2Q_EPI_SOFTCAP) return cap * tanhf(v / cap);
    if (epi == HF2Q_EPI_SCALE) return v * cap;
    return v;
}

// ---------------------------------------------------------------- mat-vec
constexpr int MV_WARPS = 8;
constexpr int MV_THREADS = MV_WARPS * 32;

// acc[r][m] += w rows (row0 + r) . xs rows; one warp, RW weight rows, 8 elements per lane and step
template <int RW, int M>
__device__ __forceinline__ void matvec_rows(const __nv_bfloat16* __restrict__ w, uint32_t row0, uint32_t n, uint32_t k, const float* xs,
                                            float (&acc)[RW][M]) {
    const uint32_t lane = threadIdx.x & 31;
    const uint4* wr[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) wr[r] = reinterpret_cast<const uint4*>(w + static_cast<size_t>(min(row0 + r, n - 1)) * k);
    const uint32_t steps = k / 8;
    auto take = [&](const uint4& v, int r, uint32_t c) {
        const float f[8] = {bf_lo(v.x), bf_hi(v.x), bf_lo(v.y), bf_hi(v.y), bf_lo(v.z), bf_hi(v.z), bf_lo(v.w), bf_hi(v.w)};
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const float4 a = *reinterpret_cast<const float4*>(xs + static_cast<size_t>(m) * k + 8 * c);
            const float4 b = *reinterpret_cast<const float4*>(xs + static_cast<size_t>(m) * k + 8 * c + 4);
            float s = acc[r][m];
            s = fmaf(f[0], a.x, s); s = fmaf(f[1], a.y, s); s = fmaf(f[2], a.z, s); s = fmaf(f[3], a.w, s);
            s = fmaf(f[4], b.x, s); s = fmaf(f[5], b.y, s); s = fmaf(f[6], b.z, s); s = fmaf(f[7], b.w, s);
            acc[r][m] = s;
        }
    };
    constexpr int U = 4;
    uint32_t c = lane;
    for (; c + 32 * (U - 1) < steps; c += 32 * U) {
        uint4 v[U][RW];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int r = 0; r < RW; ++r) v[u][r] = __ldcs(wr[r] + c + 32 * u);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int r = 0; r < RW; ++r) take(v[u][r], r, c + 32 * u);
    }
    for (; c < steps; c += 32) {
#pragma unroll
        for (int r = 0; r < RW; ++r) take(__ldcs(wr[r] + c), r, c);
    }
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int m = 0; m < M; ++m) acc[r][m] = warp_sum(acc[r][m]);
}

struct MatvecSegs {
    hf2q_matvec s[2];
    MatvecPlan plan[2];
    uint32_t share[2];       // elements of the streams that a CTA stores
    uint32_t blocks0;        // CTAs of segment 0
};

// ---- row prologues with a row's 16-byte groups in registers, PRO_GROUPS per thread: constants are there before the wait for the
// launch in front, and everything that it wrote is asked for at once.
// Few instructions count as much, for they come cold: a prologue over four streams of 2048 took 3.5 us with an instruction per element
// and 2.0 with one per two, a gated row of 4096 5.2 and 3.0 with its head sums by a warp each.  Rows of 32 outputs, all of it: 7.2 -> 4.4
// us; 2048 outputs behind a gated row 10.5 -> 7.6.
constexpr int PRO_GROUPS = 3;
__device__ __forceinline__ float4 group4(const float* p, uint32_t i, bool in) { return p && in ? *reinterpret_cast<const float4*>(p + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ bool groups_fit(uint32_t width, uintptr_t pointers, int groups = PRO_GROUPS) { return width % 4 == 0 && width <= 4 * groups * MR_THREADS && pointers % 16 == 0; }
__device__ __forceinline__ uintptr_t bits(const void* p) { return reinterpret_cast<uintptr_t>(p); }

struct NormRow {
    const hf2q_pre_norm& q;
    float4 norm[PRO_GROUPS], mu[PRO_GROUPS], step[PRO_GROUPS], an[PRO_GROUPS], bn[PRO_GROUPS];
    static __device__ __forceinline__ bool fits(const hf2q_pre_norm& q) {
        return groups_fit(q.width, bits(q.x) | bits(q.a) | bits(q.b) | bits(q.a_norm) | bits(q.b_norm) | bits(q.add0) | bits(q.step) | bits(q.norm) | bits(q.shift) |
                                       bits(q.shift_state) | bits(q.x_out));
    }
    __device__ __forceinline__ explicit NormRow(const hf2q_pre_norm& p) : q(p) {
#pragma unroll
        for (int g = 0; g < PRO_GROUPS; ++g) {
            const uint32_t i = threadIdx.x + MR_THREADS * g;
            const bool in = 4 * i < q.width;
            norm[g] = group4(q.norm, i, in); mu[g] = group4(q.shift, i, in); step[g] = group4(q.step, i, in);
            an[g] = group4(q.a_norm, i, in); bn[g] = group4(q.b_norm, i, in);
        }
    }
    // the row into xs; with `keep` also x_out and the shift state.  red: 96 floats
    __device__ __forceinline__ void run(bool keep, float* xs, float* red) const {
        float4 v[PRO_GROUPS], a[PRO_GROUPS], b[PRO_GROUPS], add[PRO_GROUPS], even[PRO_GROUPS], odd[PRO_GROUPS];
#pragma unroll
        for (int g = 0; g < PRO_GROUPS; ++g) {
            const uint32_t i = threadIdx.x + MR_THREADS * g;
            const bool in = 4 * i < q.width;
            v[g] = group4(q.x, i, in); a[g] = group4(q.a, i, in); b[g] = group4(q.b, i, in); add[g] = group4(q.add0, i, in);
            even[g] = group4(q.shift ? q.shift_state : nullptr, i, in);     // (which of the two rows is the last one's follows from the position)
            odd[g] = group4(q.shift ? q.shift_state + q.width : nullptr, i, in);
        }
        const uint32_t pos = q.shift ? *q.pos : 0u;
        const float n = static_cast<float>(q.width);
        if (q.a) {
            float s[2] = {0.f, 0.f};
#pragma unroll
            for (int g = 0; g < PRO_GROUPS; ++g) { s[0] += square_sum(a[g]); s[1] += square_sum(b[g]); }
            block_sum(s, red);
            const float ia = 0.5f / sqrtf(s[0] / n + q.eps), ib = 0.5f / sqrtf(s[1] / n + q.eps);
#pragma unroll
            for (int g = 0; g < PRO_GROUPS; ++g) {
                v[g].x += a[g].x * ia * an[g].x + b[g].x * ib * bn[g].x; v[g].y += a[g].y * ia * an[g].y + b[g].y * ib * bn[g].y;
                v[g].z += a[g].z * ia * an[g].z + b[g].z * ib * bn[g].z; v[g].w += a[g].w * ia * an[g].w + b[g].w * ib * bn[g].w;
            }
        }
        float s[1] = {0.f};
#pragma unroll
        for (int g = 0; g < PRO_GROUPS; ++g) {
            if (q.add0) { v[g].x += add[g].x; v[g].y += add[g].y; v[g].z += add[g].z; v[g].w += add[g].w; }
            if (q.step) { v[g].x += step[g].x; v[g].y += step[g].y; v[g].z += step[g].z; v[g].w += step[g].w; }
            s[0] += square_sum(v[g]);
        }
        block_sum(s, red + 64);
        const float inv = 1.0f / sqrtf(s[0] / n + q.eps);
#pragma unroll
        for (int g = 0; g < PRO_GROUPS; ++g) {
            const uint32_t i = threadIdx.x + MR_THREADS * g;
            if (4 * i >= q.width) continue;
            if (keep && q.x_out) *reinterpret_cast<float4*>(q.x_out + 4 * i) = v[g];
            float4 h = make_float4(v[g].x * inv * norm[g].x, v[g].y * inv * norm[g].y, v[g].z * inv * norm[g].z, v[g].w * inv * norm[g].w);
            if (q.shift) {
                if (keep) *reinterpret_cast<float4*>(q.shift_state + static_cast<size_t>(pos & 1) * q.width + 4 * i) = h;
                const float4 was = pos & 1 ? even[g] : odd[g];              // row (pos + 1) & 1
                h = make_float4(h.x + (was.x - h.x) * mu[g].x, h.y + (was.y - h.y) * mu[g].y, h.z + (was.z - h.z) * mu[g].z, h.w + (was.w - h.w) * mu[g].w);
            }
            *reinterpret_cast<float4*>(xs + 4 * i) = h;
        }
    }
};

// up to four streams; two elements an instruction
struct HyperRow {
    static constexpr int S = 4;
    const hf2q_hyper& q;
    float4 norm[PRO_GROUPS];
    static __device__ __forceinline__ bool fits(const hf2q_hyper& q) {
        return q.streams <= S && groups_fit(q.width, bits(q.x) | bits(q.x_out) | bits(q.y) | bits(q.norm) | bits(q.h_out));
    }
    __device__ __forceinline__ HyperRow(const hf2q_hyper& p, f2* coef) : q(p) {
#pragma unroll
        for (int g = 0; g < PRO_GROUPS; ++g) norm[g] = group4(q.norm, threadIdx.x + MR_THREADS * g, 4 * (threadIdx.x + MR_THREADS * g) < q.width);
        hyper_coefficients<S>(q, coef);
    }
    static __device__ __forceinline__ ulonglong2 pairs(const float* p, uint32_t i, bool in) { return in ? *reinterpret_cast<const ulonglong2*>(p + 4 * i) : make_ulonglong2(0, 0); }
    static __device__ __forceinline__ void axpy2(ulonglong2& d, f2 a, const ulonglong2& x) { d.x = f2_fma(a, x.x, d.x); d.y = f2_fma(a, x.y, d.y); }
    // the row into xs, the new streams' elements [lo, hi) (multiples of four) and those of the row itself to memory
    __device__ __forceinline__ void run(float* xs, const f2* coef, float* red, uint32_t lo, uint32_t hi) const {
        const f2 *mix = coef, *gain = coef + S * S, *in = gain + S;
        const uint32_t step = q.x_streams == 1 ? 0u : q.width;
        ulonglong2 old[PRO_GROUPS][S], y[PRO_GROUPS], u[PRO_GROUPS];
#pragma unroll
        for (int g = 0; g < PRO_GROUPS; ++g) {
            if (4 * MR_THREADS * g >= q.width) break;
            const uint32_t i = threadIdx.x + MR_THREADS * g;
            const bool has = 4 * i < q.width;
#pragma unroll
            for (int s = 0; s < S; ++s) old[g][s] = pairs(q.x + s * step, i, has && s < static_cast<int>(q.streams));
            y[g] = pairs(q.y, i, has && q.y);
        }
        for (uint32_t k = 1; q.y && k < q.y_parts; ++k)
#pragma unroll
            for (int g = 0; g < PRO_GROUPS; ++g) {
                const uint32_t i = threadIdx.x + MR_THREADS * g;
                if (4 * i < q.width) axpy2(y[g], f2_both(1.0f), pairs(q.y + k * q.width, i, true));
            }
        float s1[1] = {0.f};
#pragma unroll
        for (int g = 0; g < PRO_GROUPS; ++g) {
            if (4 * MR_THREADS * g >= q.width) break;
            const uint32_t e = 4 * (threadIdx.x + MR_THREADS * g);
            const bool own = q.x_out && e >= lo && e < hi;
            u[g] = make_ulonglong2(0, 0);
#pragma unroll
            for (int d = 0; d < S; ++d) {
                if (d >= static_cast<int>(q.streams)) break;
                ulonglong2 v = old[g][d];
                if (q.y) {
                    v = make_ulonglong2(0, 0);
#pragma unroll
                    for (int s = 0; s < S; ++s) axpy2(v, mix[s * S + d], old[g][s]);
                    axpy2(v, gain[d], y[g]);
                }
                if (own) *reinterpret_cast<ulonglong2*>(q.x_out + static_cast<size_t>(d) * q.width + e) = v;
                axpy2(u[g], in[d], v);
            }
            const float2 a = f2_parts(u[g].x), b = f2_parts(u[g].y);
            s1[0] += a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y;
        }
        block_sum(s1, red);
        const float inv = 1.0f / sqrtf(s1[0] / static_cast<float>(q.width) + q.eps);
#pragma unroll
        for (int g = 0; g < PRO_GROUPS; ++g) {
            const uint32_t e = 4 * (threadIdx.x + MR_THREADS * g);
            if (e >= q.width) break;
            const float2 a = f2_parts(u[g].x), b = f2_parts(u[g].y);
            const float4 h = q.norm ? make_float4(a.x * inv * norm[g].x, a.y * inv * norm[g].y, b.x * inv * norm[g].z, b.y * inv * norm[g].w) : make_float4(a.x, a.y, b.x, b.y);
            *reinterpret_cast<float4*>(xs + e) = h;
            if (q.h_out && e >= lo && e < hi) *reinterpret_cast<float4*>(q.h_out + e) = h;
        }
    }
};

// Gated head outputs of heads of whole 128-element spans, a span to a warp (silu_group_norm_row and gated_heads_row take the others).
// G: groups a thread.
template <int G>
struct GatedRow {
    const hf2q_gated_heads& q;
    const bool silu;
    const uint32_t width, spans, inv;            // of a row; of a head; x / spans = x * inv >> 16
    float4 norm[G];
    static __device__ __forceinline__ bool fits(const hf2q_gated_heads& q) {
        return q.head_dim % 128 == 0 && groups_fit(q.heads * q.head_dim, bits(q.o) | bits(q.gate) | bits(q.norm), G);
    }
    __device__ __forceinline__ explicit GatedRow(const hf2q_gated_heads& p)
        : q(p), silu(p.kind == HF2Q_GATE_SILU_FIRST), width(p.heads * p.head_dim), spans(p.head_dim / 128), inv((65535 + spans) / spans) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const uint32_t i = threadIdx.x + MR_THREADS * g;
            norm[g] = group4(q.norm, silu || q.norm_all ? i : i - first_span(g) * 32, 4 * i < width);
        }
    }
    __device__ __forceinline__ uint32_t first_span(int g) const { return (((threadIdx.x + MR_THREADS * g) / 32 * inv) >> 16) * spans; }      // of the head
    __device__ __forceinline__ float gate_of(float x) const { return (silu ? x : 1.0f) / (1.0f + expf(-x)); }      // siluf, sigmoidf
    // the row into xs.  sums: a float per span
    __device__ __forceinline__ void run(float* xs, float* sums) const {
        const uint32_t lane = threadIdx.x & 31;
        float4 v[G], x[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const uint32_t i = threadIdx.x + MR_THREADS * g;
            v[g] = group4(q.o, i, 4 * i < width); x[g] = group4(q.gate, i, 4 * i < width);
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            if (4 * MR_THREADS * g >= width) break;
            x[g] = make_float4(gate_of(x[g].x), gate_of(x[g].y), gate_of(x[g].z), gate_of(x[g].w));
            if (silu) v[g] = make_float4(v[g].x * x[g].x, v[g].y * x[g].y, v[g].z * x[g].z, v[g].w * x[g].w);
            const float s = warp_sum(square_sum(v[g]));
            if (lane == 0) sums[(threadIdx.x + MR_THREADS * g) / 32] = s;
        }
        __syncthreads();
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const uint32_t i = threadIdx.x + MR_THREADS * g, first = first_span(g);
            if (4 * i >= width) break;                                      // (whole warps)
            float4 w = make_float4(1.f, 1.f, 1.f, 1.f);
            if (q.norm) {
                float part = (lane < spans ? sums[first + lane] : 0.f) + (lane + 32 < spans ? sums[first + lane + 32] : 0.f);
                if (G * MR_WARPS > 64 && lane + 64 < spans) part += sums[first + lane + 64];
                const float s = warp_sum(part);
                const float r = 1.0f / sqrtf(s / static_cast<float>(q.head_dim) + q.eps);
                w = make_float4(norm[g].x * r, norm[g].y * r, norm[g].z * r, norm[g].w * r);
            }
            float4 h = make_float4(v[g].x * w.x, v[g].y * w.y, v[g].z * w.z, v[g].w * w.w);
            if (!silu) h = make_float4(h.x * x[g].x, h.y * x[g].y, h.z * x[g].z, h.w * x[g].w);
            *reinterpret_cast<float4*>(xs + 4 * i) = h;
        }
    }
};

// One-row product: the CTA's weight rows run through a MatvecStream; the layer's row prologue fills x in front of it.
// WIDE: rows beyond PRO_GROUPS groups a thread, 16 bytes at a time through shared memory, gated ones with twice the groups (64 outputs behind
// rows of 8192, us element by element and now: norm 8.9 / 5.1, four streams 13.3 / 9.2, gated 7.6 / 6.6).  A form of its own, for with these
// paths beside the others a decode step of 200 products took 1.7 % longer.
template <int PRO, bool PAIRS, bool WIDE>
__global__ void __launch_bounds__(MR_THREADS, 1) dense_matvec_kernel(const __grid_constant__ MatvecSegs p, uint32_t* status) {
    extern __shared__ __align__(128) uint8_t mv_smem[];                 // ring, then x [k] f32
    __shared__ float red[96];                                           // (a float for every 128 elements of a gated row among them)
    static_assert(2 * PRO_GROUPS * MR_WARPS <= 96, "");
    __shared__ MatvecShared sh;
    pdl_trigger();
    const bool second = blockIdx.x >= p.blocks0;
    const hf2q_matvec& s = p.s[second];
    const MatvecPlan& plan = p.plan[second];
    const uint32_t blk = blockIdx.x - (second ? p.blocks0 : 0u);
    const uint32_t warp = threadIdx.x >> 5;
    float* xs = reinterpret_cast<float*>(mv_smem + MR_RING);
    constexpr uint32_t unit = PAIRS ? 2 : 1;
    const uint32_t row0 = unit * plan.first(blk), row1 = row0 + unit * plan.count(blk), piece = plan.piece;
    const __nv_bfloat16* w = static_cast<const __nv_bfloat16*>(s.w) + static_cast<size_t>(row0) * s.k;
    auto at = [&](uint32_t row, uint32_t col) {
        const uint32_t k0 = col * piece;
        return MatvecChunk{w + static_cast<size_t>(row) * s.k + k0, k0, min(piece, s.k - k0)};
    };
    MatvecStream stream(mv_smem, sh, row1 - row0, plan, status);
    stream.start(at);
    // what the first pass of the epilogue adds to this thread's row (or pair)
    const uint32_t mine = row0 + threadIdx.x * unit;
    float bias0 = 0.f, bias1 = 0.f, residual = 0.f;
    if (s.bias && mine < row1) {
        bias0 = s.bias[mine];
        if constexpr (PAIRS) bias1 = s.bias[mine + 1];
    }
    auto add_residual = [&] { if (s.epilogue == HF2Q_EPI_ADD && mine < row1) residual = s.residual[mine]; };
    if constexpr (PRO == HF2Q_PRO_NONE) {
        pdl_wait();
        add_residual();
        if (s.k % 4 == 0 && bits(s.x) % 16 == 0)
            for (uint32_t i = threadIdx.x; i < s.k / 4; i += MR_THREADS) reinterpret_cast<float4*>(xs)[i] = reinterpret_cast<const float4*>(s.x)[i];
        else
            for (uint32_t i = threadIdx.x; i < s.k; i += MR_THREADS) xs[i] = s.x[i];
    } else if constexpr (PRO == HF2Q_PRO_NORM) {
        const hf2q_pre_norm& q = s.pre;
        const bool keep = blk == 0;
        if (!WIDE && NormRow::fits(q)) {
            const NormRow row(q);
            pdl_wait();
            add_residual();
            row.run(keep, xs, red);
            for (uint32_t i = q.width + threadIdx.x; i < s.k; i += MR_THREADS) xs[i] = 0.f;
        } else {
            pdl_wait();
            add_residual();
            const float inv = residual_row(q, 0, xs, red);
            const uint32_t pos = q.shift ? *q.pos : 0u;
            const float* before = q.shift_state + static_cast<size_t>((pos + 1) & 1) * q.width;
            float* now = q.shift_state + static_cast<size_t>(pos & 1) * q.width;
            const uint32_t n4 = WIDE && q.width % 4 == 0 && (bits(q.norm) | bits(q.x_out) | bits(q.shift) | bits(q.shift_state)) % 16 == 0 ? q.width / 4 : 0u;
#pragma unroll 4
            for (uint32_t i = threadIdx.x; i < n4; i += MR_THREADS) {
                const float4 x = *reinterpret_cast<const float4*>(xs + 4 * i), w = group4(q.norm, i, true);
                if (keep && q.x_out) *reinterpret_cast<float4*>(q.x_out + 4 * i) = x;
                float4 h = make_float4(x.x * inv * w.x, x.y * inv * w.y, x.z * inv * w.z, x.w * inv * w.w);
                if (q.shift) {
                    const float4 was = group4(before, i, true), mu = group4(q.shift, i, true);
                    if (keep) *reinterpret_cast<float4*>(now + 4 * i) = h;
                    h = make_float4(h.x + (was.x - h.x) * mu.x, h.y + (was.y - h.y) * mu.y, h.z + (was.z - h.z) * mu.z, h.w + (was.w - h.w) * mu.w);
                }
                *reinterpret_cast<float4*>(xs + 4 * i) = h;
            }
            for (uint32_t i = 4 * n4 + threadIdx.x; i < s.k; i += MR_THREADS) {
                float h = 0.f;
                if (i < q.width) {
                    const float x = xs[i];
                    if (keep && q.x_out) q.x_out[i] = x;
                    h = x * inv * q.norm[i];
                    if (q.shift) {
                        if (keep) now[i] = h;
                        h += (before[i] - h) * q.shift[i];
                    }
                }
                xs[i] = h;
            }
        }
    } else if constexpr (PRO == HF2Q_PRO_HYPER) {
        const hf2q_hyper& q = s.hyper;
        __shared__ __align__(8) float coef[HYPER_COEF];
        // every CTA makes the whole row and stores its share of the new streams
        const uint32_t lo = min(p.share[second] * blk, q.width), hi = min(lo + p.share[second], q.width);
        if (!WIDE && HyperRow::fits(q)) {
            f2* pairs = reinterpret_cast<f2*>(coef);
            const HyperRow row(q, pairs);
            pdl_wait();
            add_residual();
            row.run(xs, pairs, red, lo, hi);
            for (uint32_t i = q.width + threadIdx.x; i < s.k; i += MR_THREADS) xs[i] = 0.f;
        } else {
            pdl_wait();
            add_residual();
            const float inv = hyper_row(q, 0, xs, coef, red, lo, hi);
            const uint32_t n4 = WIDE && q.width % 4 == 0 && (bits(q.norm) | bits(q.h_out)) % 16 == 0 ? q.width / 4 : 0u;      // (lo and hi are multiples of four)
#pragma unroll 4
            for (uint32_t i = threadIdx.x; i < n4; i += MR_THREADS) {
                float4 h = *reinterpret_cast<const float4*>(xs + 4 * i);
                if (q.norm) {
                    const float4 w = group4(q.norm, i, true);
                    h = make_float4(h.x * inv * w.x, h.y * inv * w.y, h.z * inv * w.z, h.w * inv * w.w);
                    *reinterpret_cast<float4*>(xs + 4 * i) = h;
                }
                if (q.h_out && 4 * i >= lo && 4 * i < hi) *reinterpret_cast<float4*>(q.h_out + 4 * i) = h;
            }
            for (uint32_t i = 4 * n4 + threadIdx.x; i < s.k; i += MR_THREADS) {
                const float h = i < q.width ? (q.norm ? xs[i] * inv * q.norm[i] : xs[i]) : 0.f;
                xs[i] = h;
                if (q.h_out && i >= lo && i < hi) q.h_out[i] = h;
            }
        }
    } else if (typedef GatedRow<(WIDE ? 2 : 1) * PRO_GROUPS> Row; Row::fits(s.gated)) {
        const Row row(s.gated);
        pdl_wait();
        add_residual();
        row.run(xs, red);
        for (uint32_t i = s.gated.heads * s.gated.head_dim + threadIdx.x; i < s.k; i += MR_THREADS) xs[i] = 0.f;
    } else {
        pdl_wait();
        add_residual();
        for (uint32_t i = s.gated.heads * s.gated.head_dim + threadIdx.x; i < s.k; i += MR_THREADS) xs[i] = 0.f;
        if (s.gated.kind == HF2Q_GATE_SILU_FIRST) silu_group_norm_row<float>(s.gated, 0, xs, xs);
        else gated_heads_row<float>(s.gated, 0, xs, warp, MR_WARPS);
    }
    __syncthreads();
    if constexpr (PAIRS) {
        stream.run<true>(at, xs, [&](uint32_t r, float gate, float up) {
            const uint32_t row = row0 + r;
            if (s.bias) { gate += row == mine ? bias0 : s.bias[row]; up += row == mine ? bias1 : s.bias[row + 1]; }
            s.y[row / 2] = glu_value(gate, up, s.epilogue, s.cap);
        });
    } else {
        stream.run<false>(at, xs, [&](uint32_t r, float v, float) {
            const uint32_t row = row0 + r;
            if (s.bias) v += row == mine ? bias0 : s.bias[row];
            v = epilogue_value(v, s.epilogue, s.cap);
            if (s.epilogue == HF2Q_EPI_ADD) v += row == mine ? residual : s.residual[row];
            s.y[row] = v;
        });
    }
}

struct DenseArgs {
    const void* x;
    const __nv_bfloat16* w;
    void* y;
    const float *residual, *bias;
    uint32_t ldx, ldy, m, n, k, epi;
    float cap;
    hf2q_row_groups g;       // grouped products: rows of x sorted by group, w [groups][n][k]
};
// where a grouped product's output row goes, and what it is scaled with before the activation
struct GroupRow { size_t out; float scale; };
__device__ __forceinline__ GroupRow group_row(const DenseArgs& p, uint32_t sorted) {
    const uint32_t routed = p.g.perm[sorted];
    return {p.g.scatter ? routed : sorted, p.g.row_scale ? p.g.row_scale[routed] : 1.0f};
}

template <typename X, typename Y, int M, int RW>
__global__ void __launch_bounds__(MV_THREADS) dense_matvec_m_kernel(const DenseArgs p) {          // RW = 2: rows are pairs
    extern __shared__ __align__(16) float xs[];
    pdl_trigger();
    pdl_wait();
    const X* x = static_cast<const X*>(p.x);
    for (int m = 0; m < M; ++m)
        for (uint32_t i = threadIdx.x; i < p.k; i += MV_THREADS)
            xs[static_cast<size_t>(m) * p.k + i] = m < static_cast<int>(p.m) ? to_f32(x[static_cast<size_t>(m) * p.ldx + i]) : 0.f;
    __syncthreads();
    const uint32_t row = (blockIdx.x * MV_WARPS + (threadIdx.x >> 5)) * RW;
    if (row >= p.n) return;
    float acc[RW][M];
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int m = 0; m < M; ++m) acc[r][m] = 0.f;
    matvec_rows<RW, M>(p.w, row, p.n, p.k, xs, acc);
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int m = 0; m < M; ++m)
            if (m < static_cast<int>(p.m)) {
                const size_t o = static_cast<size_t>(m) * p.ldy + row / RW;
                float v = acc[0][m] + (p.bias ? p.bias[row] : 0.f);
                if constexpr (RW == 2) {
                    v = glu_value(v, acc[1][m] + (p.bias ? p.bias[row + 1] : 0.f), p.epi, p.cap);
                } else {
                    v = epilogue_value(v, p.epi, p.cap);
                    if (p.epi == HF2Q_EPI_ADD) v += p.residual[o];
                }
                static_cast<Y*>(p.y)[o] = from_f32<Y>(v);
            }
    }
}

// ---------------------------------------------------------------- fp32 product on the CUDA cores
constexpr int FT = 64, FK = 16;

template <typename X, typename Y, bool GROUPED>
__global__ void __launch_bounds__(256) dense_gemm_f32_kernel(const DenseArgs p) {
    __shared__ float as[FK][FT + 4], bs[FK][FT + 4];
    pdl_trigger();
    pdl_wait();
    const X* x = static_cast<const X*>(p.x);
    uint32_t m0 = blockIdx.y * FT, m_end = p.m;
    const uint32_t n0 = blockIdx.x * FT;
    const __nv_bfloat16* w = p.w;
    if constexpr (GROUPED) {
        if (blockIdx.y >= p.g.header[0]) return;
        const uint4 tile = reinterpret_cast<const uint4*>(p.g.tiles)[blockIdx.y];           // group, first sorted row, rows
        w += static_cast<size_t>(tile.x) * p.n * p.k;
        m0 = tile.y;
        m_end = tile.y + tile.z;
    }
    const uint32_t tr = threadIdx.x / 16, tc = threadIdx.x % 16;
    float acc[4][4] = {};
    for (uint32_t k0 = 0; k0 < p.k; k0 += FK) {
        for (uint32_t i = threadIdx.x; i < FT * FK; i += 256) {
            const uint32_t r = i / FK, c = i % FK;
            as[c][r] = m0 + r < m_end && k0 + c < p.k ? to_f32(x[static_cast<size_t>(m0 + r) * p.ldx + k0 + c]) : 0.f;
            bs[c][r] = n0 + r < p.n && k0 + c < p.k ? to_f32(w[static_cast<size_t>(n0 + r) * p.k + k0 + c]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < FK; ++c) {
            const float4 a = *reinterpret_cast<const float4*>(&as[c][4 * tr]), b = *reinterpret_cast<const float4*>(&bs[c][4 * tc]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
    const bool pairs = epi_pairs(p.epi);
    for (int i = 0; i < 4; ++i) {
        const uint32_t r = m0 + 4 * tr + i;
        if (r >= m_end) continue;
        size_t row = r;
        float scale = 1.0f;
        if constexpr (GROUPED) { const GroupRow q = group_row(p, r); row = q.out; scale = q.scale; }
        for (int j = 0; j < 4; ++j) {
            const uint32_t c = n0 + 4 * tc + j;
            if (c >= p.n || (pairs && (j & 1))) continue;
            const size_t o = row * p.ldy + (pairs ? c / 2 : c);
            float v = acc[i][j] * scale + (p.bias ? p.bias[c] : 0.f);
            if (pairs) {
                v = glu_value(v, acc[i][j + 1 < 4 ? j + 1 : j] * scale + (p.bias ? p.bias[c + 1] : 0.f), p.epi, p.cap);
            } else {
                v = epilogue_value(v, p.epi, p.cap);
                if (p.epi == HF2Q_EPI_ADD) v += p.residual[o];
            }
            static_cast<Y*>(p.y)[o] = from_f32<Y>(v);
        }
    }
}

// ---------------------------------------------------------------- tcgen05 product
// One CTA per SM walks tiles of 128 activation rows x NT weight rows.  Warp 0: TMA producer; warp 1: tensor-memory
// owner and MMA issuer; warps 2..5: epilogue (thread = activation row).
constexpr int TC_M = 128, TC_K = 64, TC_THREADS = 192;
__host__ __device__ constexpr int tc_stages(int nt) { return nt == 256 ? 4 : nt == 128 ? 6 : 8; }
__host__ __device__ constexpr uint32_t tc_stage_bytes(int nt) { return (TC_M + nt) * TC_K * 2; }

__device__ __forceinline__ void st_global_v8(float* p, const float* v) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]),
                 "f"(v[6]), "f"(v[7])
                 : "memory");
}

// sixteen consecutive outputs, 32-byte aligned for f32 and 16-byte aligned for bf16
__device__ __forceinline__ void store16(float* y, const float* v) {
    st_global_v8(y, v);
    st_global_v8(y + 8, v + 8);
}
__device__ __forceinline__ void store16(__nv_bfloat16* y, const float* v) {
    uint32_t q[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        q[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    reinterpret_cast<uint4*>(y)[0] = make_uint4(q[0], q[1], q[2], q[3]);
    reinterpret_cast<uint4*>(y)[1] = make_uint4(q[4], q[5], q[6], q[7]);
}

template <int NT, typename Y, bool GROUPED>
__global__ void __launch_bounds__(TC_THREADS, 1) dense_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                                                      const DenseArgs p, uint32_t* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    constexpr int ST = tc_stages(NT);
    constexpr uint32_t SB = tc_stage_bytes(NT);
    __shared__ uint64_t full[ST], empty[ST], d_full[2], d_empty[2];
    __shared__ uint32_t tmem_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nkb = (p.k + TC_K - 1) / TC_K;
    if (threadIdx.x == 0) {
        for (int i = 0; i < ST; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&d_full[i], 1); mbar_init(&d_empty[i], 4); }
        mbar_fence_init();
    }
    if (warp == 1) { tc::tmem_alloc(&tmem_slot, 2 * NT); tc::tmem_relinquish(); }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_trigger();
    pdl_wait();
    const uint32_t mt = GROUPED ? p.g.header[0] : (p.m + TC_M - 1) / TC_M, n_tiles = mt * ((p.n + NT - 1) / NT);
    const uint4* group_tiles = reinterpret_cast<const uint4*>(p.g.tiles);                // group, first sorted row, rows
    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (uint32_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
                int row_x = static_cast<int>((tile % mt) * TC_M), row_w = static_cast<int>((tile / mt) * NT);
                if constexpr (GROUPED) {
                    const uint4 q = group_tiles[tile % mt];
                    row_x = static_cast<int>(q.y);
                    row_w += static_cast<int>(q.x * p.n);
                }
                for (uint32_t kb = 0; kb < nkb; ++kb, ++it) {
                    const uint32_t s = it % ST;
                    if (it >= ST) ok = mbar_wait_bounded(&empty[s], (it / ST - 1) & 1, status);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&full[s], SB);
                    tc::tma_2d(smem + s * SB, &map_x, static_cast<int>(kb * TC_K), row_x, &full[s]);
                    tc::tma_2d(smem + s * SB + TC_M * TC_K * 2, &map_w, static_cast<int>(kb * TC_K), row_w, &full[s]);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // D f32, A and B bf16, both K-major, M = 128, N = NT
            constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(NT >> 3) << 17) | (static_cast<uint32_t>(TC_M >> 4) << 24);
            uint32_t it = 0, li = 0;
            bool ok = true;
            for (uint32_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++li) {
                const uint32_t b = li & 1;
                if (li >= 2) ok = mbar_wait_bounded(&d_empty[b], (li / 2 - 1) & 1, status);
                if (!ok) break;
                tc::tc_fence_after();
                for (uint32_t kb = 0; kb < nkb; ++kb, ++it) {
                    const uint32_t s = it % ST;
                    ok = mbar_wait_bounded(&full[s], (it / ST) & 1, status);
                    if (!ok) break;
                    tc::tc_fence_after();
                    const uint64_t da = tc::smem_desc_sw128(smem_u32(smem + s * SB)), db = tc::smem_desc_sw128(smem_u32(smem + s * SB + TC_M * TC_K * 2));
#pragma unroll
                    for (uint32_t kk = 0; kk < TC_K / 16; ++kk) tc::umma_ss(tmem + b * NT, da + 2 * kk, db + 2 * kk, IDESC, (kb | kk) ? 1u : 0u);
                    tc::tc_commit(&empty[s]);
                }
                if (ok) tc::tc_commit(&d_full[b]);
            }
        }
    } else {
        const uint32_t quad = warp & 3;
        const bool wide = p.ldy % 8 == 0 && reinterpret_cast<uintptr_t>(p.y) % 32 == 0 &&
                          (p.epi != HF2Q_EPI_ADD || reinterpret_cast<uintptr_t>(p.residual) % 16 == 0);
        uint32_t li = 0;
        for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++li) {
            const uint32_t b = li & 1;
            bool ok = mbar_wait_bounded(&d_full[b], (li / 2) & 1, status);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc::tc_fence_after();
            const uint32_t n0 = (tile / mt) * NT, n_cols = min(static_cast<uint32_t>(NT), p.n - n0);
            size_t row = (tile % mt) * TC_M + quad * 32 + lane;
            bool live = row < p.m;
            float scale = 1.0f;
            if constexpr (GROUPED) {
                const uint4 q = group_tiles[tile % mt];
                live = quad * 32 + lane < q.z;
                if (live) { const GroupRow gr = group_row(p, q.y + quad * 32 + lane); row = gr.out; scale = gr.scale; }
            }
#pragma unroll 1
            for (uint32_t c0 = 0; c0 < n_cols; c0 += 32) {
                uint32_t r[32];
                tc::tmem_ld32(tmem + b * NT + ((quad * 32u) << 16) + c0, r);
                tc::tmem_wait_ld();
                if (live) {
                float v[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
                if constexpr (GROUPED) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] *= scale;
                }
                if (p.bias) {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (c0 + j < n_cols) v[j] += p.bias[n0 + c0 + j];
                }
                if (epi_pairs(p.epi)) {                                  // 32 columns -> 16 outputs
                    Y* y = static_cast<Y*>(p.y) + row * p.ldy + (n0 + c0) / 2;
                    float g[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) g[j] = glu_value(v[2 * j], v[2 * j + 1], p.epi, p.cap);
                    if (wide && c0 + 32 <= n_cols) {
                        store16(y, g);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (c0 + 2 * j < n_cols) y[j] = from_f32<Y>(g[j]);
                    }
                } else {
                const size_t o = row * p.ldy + n0 + c0;
                Y* y = static_cast<Y*>(p.y) + o;
                if (p.epi == HF2Q_EPI_GELU || p.epi == HF2Q_EPI_SOFTCAP || p.epi == HF2Q_EPI_SCALE) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = epilogue_value(v[j], p.epi, p.cap);
                }
                if (wide && c0 + 32 <= n_cols) {
                    if (p.epi == HF2Q_EPI_ADD) {
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            const float4 q = *reinterpret_cast<const float4*>(p.residual + o + j);
                            v[j] += q.x; v[j + 1] += q.y; v[j + 2] += q.z; v[j + 3] += q.w;
                        }
                    }
                    store16(y, v);
                    store16(y + 16, v + 16);
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (c0 + j < n_cols) {
                            float q = v[j];
                            if (p.epi == HF2Q_EPI_ADD) q += p.residual[o + j];
                            y[j] = from_f32<Y>(q);
                        }
                }
                }
                }
                __syncwarp();
            }
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&d_empty[b]);
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    if (warp == 1) tc::tmem_dealloc(tmem, 2 * NT);
}

// ---------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}
// rows x k bf16, `ld` elements between rows; box of 64 elements x box_rows, 128-byte swizzle
bool encode_rows(CUtensorMap* map, const void* base, uint32_t rows, uint32_t k, uint32_t ld, uint32_t box_rows) {
    const EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {k, rows}, strides[1] = {static_cast<cuuint64_t>(ld) * 2};
    const cuuint32_t box[2] = {TC_K, box_rows}, es[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NT, typename Y, bool GROUPED>
cudaError_t launch_tc(const DenseArgs& a, uint32_t m_tiles, int sms, uint32_t* status, cudaStream_t st) {
    CUtensorMap mx, mw;
    const uint32_t w_rows = GROUPED ? a.n * a.g.groups : a.n;
    if (!encode_rows(&mx, a.x, a.m, a.k, a.ldx, TC_M) || !encode_rows(&mw, a.w, w_rows, a.k, a.k, NT)) return cudaErrorInvalidValue;
    const size_t smem = 1024 + static_cast<size_t>(tc_stages(NT)) * tc_stage_bytes(NT);
    static PerDeviceFlag flag;
    if (const cudaError_t e = ensure_max_dynamic_smem(dense_gemm_tc_kernel<NT, Y, GROUPED>, static_cast<int>(smem), flag); e != cudaSuccess) return e;
    const uint32_t tiles = m_tiles * ((a.n + NT - 1) / NT);
    const uint32_t grid = tiles < static_cast<uint32_t>(sms) ? tiles : static_cast<uint32_t>(sms);
    return launch_pdl(dense_gemm_tc_kernel<NT, Y, GROUPED>, dim3(grid), dim3(TC_THREADS), smem, st, mx, mw, a, status);
}
// m_tiles: activation tiles, for a grouped product the most there can be
template <typename Y, bool GROUPED>
cudaError_t launch_tc_any(const DenseArgs& a, uint32_t m_tiles, int sms, uint32_t* status, cudaStream_t st) {
    // the widest tile that still gives (nearly) every SM work
    if (m_tiles * ((a.n + 255) / 256) >= static_cast<uint32_t>(sms) * 3 / 4) return launch_tc<256, Y, GROUPED>(a, m_tiles, sms, status, st);
    if (m_tiles * ((a.n + 127) / 128) >= static_cast<uint32_t>(sms) * 3 / 4) return launch_tc<128, Y, GROUPED>(a, m_tiles, sms, status, st);
    return launch_tc<64, Y, GROUPED>(a, m_tiles, sms, status, st);
}

constexpr uint32_t MV_SMEM = 200 * 1024;

template <typename X, typename Y, int M, int RW>
cudaError_t launch_mv_rw(const DenseArgs& a, cudaStream_t st) {
    static PerDeviceFlag flag;
    if (const cudaError_t e = ensure_max_dynamic_smem(dense_matvec_m_kernel<X, Y, M, RW>, MV_SMEM, flag); e != cudaSuccess) return e;
    return launch_pdl(dense_matvec_m_kernel<X, Y, M, RW>, dim3((a.n / RW + MV_WARPS - 1) / MV_WARPS), dim3(MV_THREADS),
                      static_cast<size_t>(M) * a.k * 4, st, a);
}
template <typename X, typename Y, int M>
cudaError_t launch_mv_m(const DenseArgs& a, cudaStream_t st) {
    return epi_pairs(a.epi) ? launch_mv_rw<X, Y, M, 2>(a, st) : launch_mv_rw<X, Y, M, 1>(a, st);
}
template <typename X, typename Y>
cudaError_t launch_mv(DenseArgs a, cudaStream_t st, uint64_t* launches) {
    const uint32_t fit = MV_SMEM / (a.k * 4);
    if (fit == 0) return cudaErrorInvalidValue;
    const uint32_t m_total = a.m;
    for (uint32_t m0 = 0; m0 < m_total;) {
        uint32_t step = fit < 8 ? fit : 8;
        if (step > m_total - m0) step = m_total - m0;
        DenseArgs b = a;
        b.m = step;
        b.x = static_cast<const X*>(a.x) + static_cast<size_t>(m0) * a.ldx;
        b.y = static_cast<Y*>(a.y) + static_cast<size_t>(m0) * a.ldy;
        if (a.residual) b.residual = a.residual + static_cast<size_t>(m0) * a.ldy;
        // the smallest kernel that holds `step` rows and fits
        const uint32_t mk = step <= 1 ? 1 : step <= 2 ? 2 : step <= 4 ? 4 : 8;
        cudaError_t e;
        if (mk > fit) { b.m = step = mk / 2; }
        switch (mk > fit ? mk / 2 : mk) {
            case 1: e = launch_mv_m<X, Y, 1>(b, st); break;
            case 2: e = launch_mv_m<X, Y, 2>(b, st); break;
            case 4: e = launch_mv_m<X, Y, 4>(b, st); break;
            default: e = launch_mv_m<X, Y, 8>(b, st); break;
        }
        if (e != cudaSuccess) return e;
        ++*launches;
        m0 += step;
    }
    return cudaSuccess;
}

template <typename X, typename Y>
cudaError_t dense_any(const DenseArgs& a, int sms, uint32_t* status, cudaStream_t st, uint64_t* launches) {
    if (a.m <= 8 && a.k * 4 <= MV_SMEM) return launch_mv<X, Y>(a, st, launches);
    *launches = 1;
    if constexpr (sizeof(X) == 2) {
        if (a.ldx % 8 == 0 && reinterpret_cast<uintptr_t>(a.x) % 16 == 0) return launch_tc_any<Y, false>(a, (a.m + TC_M - 1) / TC_M, sms, status, st);
    }
    return launch_pdl(dense_gemm_f32_kernel<X, Y, false>, dim3((a.n + FT - 1) / FT, (a.m + FT - 1) / FT), dim3(256), 0, st, a);
}

template <int PRO, bool PAIRS, bool WIDE>
cudaError_t launch_fused_as(const MatvecSegs& p, uint32_t blocks, size_t smem, uint32_t* status, cudaStream_t st) {
    static PerDeviceFlag flag;
    const auto kern = dense_matvec_kernel<PRO, PAIRS, WIDE>;
    if (const cudaError_t e = ensure_max_dynamic_smem(kern, MR_RING + MR_MAX_X, flag); e != cudaSuccess) return e;
    return launch_pdl(kern, dim3(blocks), dim3(MR_THREADS), smem, st, p, status);
}
// width: of the longest row in front of a product
template <int PRO>
cudaError_t launch_fused(const MatvecSegs& p, uint32_t width, uint32_t blocks, size_t smem, uint32_t* status, cudaStream_t st) {
    const bool pairs = epi_pairs(p.s[0].epilogue);
    if constexpr (PRO != HF2Q_PRO_NONE)
        if (width > 4 * PRO_GROUPS * MR_THREADS)
            return pairs ? launch_fused_as<PRO, true, true>(p, blocks, smem, status, st) : launch_fused_as<PRO, false, true>(p, blocks, smem, status, st);
    return pairs ? launch_fused_as<PRO, true, false>(p, blocks, smem, status, st) : launch_fused_as<PRO, false, false>(p, blocks, smem, status, st);
}

}  // namespace
}  // namespace hf2q

using namespace hf2q;

extern "C" {

HF2Q_API int32_t hf2q_cuda_dense_matmul(hf2q_ctx* ctx, void* stream, const void* x, uint32_t x_dtype, uint32_t ldx, const void* w, void* y,
                                        uint32_t y_dtype, uint32_t ldy, uint32_t m, uint32_t n, uint32_t k, uint32_t epilogue,
                                        const float* residual, float cap, const float* bias) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!x || !w || !y || n == 0 || k == 0 || k % 8 || ldx < k || ldy < (epi_pairs(epilogue) ? n / 2 : n) || reinterpret_cast<uintptr_t>(w) % 16)
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "dense_matmul: null pointer, k not a multiple of 8, a short row pitch or an unaligned weight");
    if (epilogue > HF2Q_EPI_CLAMP_GLU || (epilogue == HF2Q_EPI_ADD && !residual) || (epi_needs_cap(epilogue) && !(cap > 0.f)) || (epi_pairs(epilogue) && n % 2))
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "dense_matmul: bad epilogue");
    if (m == 0) return HF2Q_OK;
    if (m > 65535u * 64u) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "dense_matmul: too many rows");
    const DenseArgs a{x, static_cast<const __nv_bfloat16*>(w), y, residual, bias, ldx, ldy, m, n, k, epilogue, cap, {}};
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint32_t* status = ctx_status_word(ctx);
    const int sms = ctx_sm_count(ctx);
    uint64_t launches = 0;
    cudaError_t e = cudaErrorInvalidValue;
    if (x_dtype == HF2Q_DT_F32 && y_dtype == HF2Q_DT_F32) e = dense_any<float, float>(a, sms, status, st, &launches);
    else if (x_dtype == HF2Q_DT_BF16 && y_dtype == HF2Q_DT_F32) e = dense_any<__nv_bfloat16, float>(a, sms, status, st, &launches);
    else if (x_dtype == HF2Q_DT_BF16 && y_dtype == HF2Q_DT_BF16) e = dense_any<__nv_bfloat16, __nv_bfloat16>(a, sms, status, st, &launches);
    else if (x_dtype == HF2Q_DT_F32 && y_dtype == HF2Q_DT_BF16) e = dense_any<float, __nv_bfloat16>(a, sms, status, st, &launches);
    return ctx_cuda_result(ctx, e, "dense_matmul", launches);
}

HF2Q_API int32_t hf2q_cuda_dense_grouped(hf2q_ctx* ctx, void* stream, const hf2q_row_groups* g, const void* x, uint32_t dtype, uint32_t ldx, const void* w,
                                         void* y, uint32_t y_dtype, uint32_t ldy, uint32_t rows, uint32_t n, uint32_t k, uint32_t epilogue, float cap) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!g || !g->header || !g->tiles || !g->perm || g->groups == 0 || !x || !w || !y || n == 0 || k == 0 || k % 8 || ldx < k || ldx % 8 ||
        ldy < (epi_pairs(epilogue) ? n / 2 : n) || reinterpret_cast<uintptr_t>(w) % 16 || reinterpret_cast<uintptr_t>(x) % 16 || epilogue > HF2Q_EPI_CLAMP_GLU ||
        epilogue == HF2Q_EPI_ADD || (epi_needs_cap(epilogue) && !(cap > 0.f)) || (epi_pairs(epilogue) && n % 2) || static_cast<uint64_t>(g->groups) * n > 0x7fffffffu)
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "dense_grouped: null or unaligned pointer, or a bad size or epilogue");
    if (rows == 0) return HF2Q_OK;
    if (g->tile_rows != (dtype == HF2Q_DT_BF16 ? HF2Q_GROUP_TILE_BF16 : HF2Q_GROUP_TILE_F32))
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "dense_grouped: the rows were sorted for another tile height");
    DenseArgs a{x, static_cast<const __nv_bfloat16*>(w), y, nullptr, nullptr, ldx, ldy, rows, n, k, epilogue, cap, *g};
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t most = rows / g->tile_rows + (rows < g->groups ? rows : g->groups);     // sum of ceil(count / tile_rows)
    cudaError_t e = cudaErrorInvalidValue;
    if (dtype == HF2Q_DT_BF16 && y_dtype == HF2Q_DT_BF16) e = launch_tc_any<__nv_bfloat16, true>(a, most, ctx_sm_count(ctx), ctx_status_word(ctx), st);
    else if (dtype == HF2Q_DT_BF16 && y_dtype == HF2Q_DT_F32) e = launch_tc_any<float, true>(a, most, ctx_sm_count(ctx), ctx_status_word(ctx), st);
    else if (dtype == HF2Q_DT_F32 && y_dtype == HF2Q_DT_F32 && most <= 65535)
        e = launch_pdl(dense_gemm_f32_kernel<float, float, true>, dim3((n + FT - 1) / FT, most), dim3(256), 0, st, a);
    return ctx_cuda_result(ctx, e, "dense_grouped", 1);
}

HF2Q_API int32_t hf2q_cuda_dense_matvec(hf2q_ctx* ctx, void* stream, uint32_t prologue, const hf2q_matvec* segs, uint32_t n_segs) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!segs || n_segs == 0 || n_segs > 2 || prologue > HF2Q_PRO_HYPER) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "dense_matvec: bad segments");
    MatvecSegs p{};
    uint32_t kmax = 0;
    uint64_t chunks[2] = {0, 0};
    for (uint32_t i = 0; i < n_segs; ++i) {
        const hf2q_matvec& s = segs[i];
        if (!s.w || !s.y || s.n == 0 || s.k == 0 || s.k % 8 || reinterpret_cast<uintptr_t>(s.w) % 16 || s.k * 4ull > MR_MAX_X ||
            (prologue == HF2Q_PRO_NONE && !s.x) ||
            (prologue == HF2Q_PRO_NORM && (!s.pre.x || !s.pre.norm || s.pre.width > s.k || !pre_norm_aligned(s.pre) || (s.pre.a && (!s.pre.b || !s.pre.a_norm || !s.pre.b_norm)) || (s.pre.shift && (!s.pre.shift_state || !s.pre.pos)))) ||
            (prologue == HF2Q_PRO_GATED && (!gated_ok(s.gated) || s.gated.heads * s.gated.head_dim > s.k)) ||
            (prologue == HF2Q_PRO_HYPER && (!hyper_ok(s.hyper) || s.hyper.width > s.k || s.hyper.x_out == s.hyper.x)) || s.epilogue > HF2Q_EPI_CLAMP_GLU ||
            (s.epilogue == HF2Q_EPI_ADD && !s.residual) || (epi_needs_cap(s.epilogue) && !(s.cap > 0.f)) || (epi_pairs(s.epilogue) && s.n % 2) || epi_pairs(s.epilogue) != epi_pairs(segs[0].epilogue))
            return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "dense_matvec: bad segment");
        p.s[i] = s;
        chunks[i] = static_cast<uint64_t>(s.n) * ((s.k + MV_CHUNK - 1) / MV_CHUNK);
        kmax = s.k > kmax ? s.k : kmax;
    }
    // one CTA per SM, shared by the segments in proportion to their chunks; no more CTAs than rows
    const uint64_t total = chunks[0] + chunks[1], sms = static_cast<uint64_t>(ctx_sm_count(ctx));
    auto ctas = [&](uint32_t i, uint64_t want) { return static_cast<uint32_t>(want < 1 ? 1 : want > segs[i].n ? segs[i].n : want); };
    uint32_t blocks = p.blocks0 = ctas(0, n_segs == 1 ? sms : (sms * chunks[0] + total / 2) / total);
    if (n_segs == 2) blocks += ctas(1, sms > p.blocks0 ? sms - p.blocks0 : 1);
    for (uint32_t i = 0; i < n_segs; ++i) {
        const uint32_t mine = i ? blocks - p.blocks0 : p.blocks0;
        p.plan[i] = matvec_plan(segs[i].n, epi_pairs(segs[i].epilogue) ? 2 : 1, mine, segs[i].k);
        p.share[i] = ((segs[i].hyper.width + 3) / 4 + mine - 1) / mine * 4;
    }
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t smem = MR_RING + static_cast<size_t>(kmax) * 4;
    uint32_t* status = ctx_status_word(ctx);
    uint32_t width = 0;
    for (uint32_t i = 0; i < n_segs; ++i) {
        const hf2q_matvec& s = segs[i];
        const uint32_t w = prologue == HF2Q_PRO_NORM ? s.pre.width : prologue == HF2Q_PRO_HYPER ? s.hyper.width : s.gated.heads * s.gated.head_dim;
        width = w > width ? w : width;
    }
    cudaError_t e;
    switch (prologue) {
        case HF2Q_PRO_NONE: e = launch_fused<HF2Q_PRO_NONE>(p, width, blocks, smem, status, st); break;
        case HF2Q_PRO_NORM: e = launch_fused<HF2Q_PRO_NORM>(p, width, blocks, smem, status, st); break;
        case HF2Q_PRO_HYPER: e = launch_fused<HF2Q_PRO_HYPER>(p, width, blocks, smem, status, st); break;
        default: e = launch_fused<HF2Q_PRO_GATED>(p, width, blocks, smem, status, st); break;
    }
    return ctx_cuda_result(ctx, e, "dense_matvec", 1);
}

}  // extern "C"
