// Sliding-window attention over a ring cache (position p in slot p % capacity) with grouped query heads, optional
// per-head RMS norm of q and k and an optional logarithmic distance term taken off the scores.  The prefill also runs over
// plain rows of keys and values, with a part of every key shared by the heads (expanded latents).
//
//   append    prefill: normalised queries to a buffer, normalised keys and values to the cache
//   prefill   bf16 cache: tiles on the tensor cores (f32 scores, softmax and accumulators, bf16 product operands): of 128
//             queries on tcgen05 or of 64 on warps, by size (prefill_on_tcgen05); f32 cache: one warp per query in f32
//   decode    one launch: norm, append, window split over the CTAs of a cluster and merged by it
#include <cooperative_groups.h>
#include <math_constants.h>

#include "mma_sync.cuh"
#include "seq_common.cuh"
#include "tc_common.cuh"

namespace hf2q {
namespace {
using namespace seq;
namespace cg = cooperative_groups;

__host__ __device__ constexpr uint32_t pad8(uint32_t n) { return (n + 7) & ~7u; }

// q . k * scale - r1 ln(1 + r2 distance)
__device__ __forceinline__ float score_of(float dot, float scale, float r1, float r2, uint32_t dist, bool bias) {
    float s = dot * scale;
    if (bias) s -= r1 * logf(1.0f + r2 * static_cast<float>(dist));
    return s;
}

// where a KV head's keys and values are: rings, or with PLAIN rows that start at position `first` and a shared key part
template <typename T, bool PLAIN>
struct KeyRows {
    const T *k, *v, *shared;
    uint32_t capacity, dp, sp, k_row, v_row, first, s_row, s_capacity;      // sp: padded size of the shared part
    __device__ __forceinline__ KeyRows(const hf2q_window_attn& a, uint32_t kvh, uint32_t pos0) {
        const uint32_t dvp = pad8(a.vdim);
        dp = pad8(a.dim);
        capacity = a.capacity;
        if constexpr (PLAIN) {
            sp = pad8(a.shared_dim);
            k_row = v_row = a.row_stride;
            first = pos0 + 1 > a.window ? pos0 + 1 - a.window : 0u;
            k = static_cast<const T*>(a.k_cache) + static_cast<size_t>(kvh) * a.k_head_stride;
            v = static_cast<const T*>(a.v_cache) + static_cast<size_t>(kvh) * a.v_head_stride;
            shared = static_cast<const T*>(a.k_shared);
            s_row = a.shared_stride;
            s_capacity = a.shared_capacity;
        } else {
            sp = 0;
            k_row = dp;
            v_row = dvp;
            k = static_cast<const T*>(a.k_cache) + static_cast<size_t>(kvh) * a.capacity * dp;
            v = static_cast<const T*>(a.v_cache) + static_cast<size_t>(kvh) * a.capacity * dvp;
        }
    }
    __device__ __forceinline__ uint32_t slot(uint32_t p) const {
        if constexpr (PLAIN) return p - first;
        else return p % capacity;
    }
    __device__ __forceinline__ const T* key(uint32_t p) const { return k + static_cast<size_t>(slot(p)) * k_row; }
    __device__ __forceinline__ const T* value(uint32_t p) const { return v + static_cast<size_t>(slot(p)) * v_row; }
    __device__ __forceinline__ const T* shared_key(uint32_t p) const { return shared + static_cast<size_t>(p % s_capacity) * s_row; }
};

// one head vector of up to 256 elements held by a warp (element lane + 32 j), divided by its root mean square
struct HeadVec {
    float v[8];
    __device__ __forceinline__ void load(const float* p, uint32_t dim, uint32_t lane) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = lane + 32 * j < dim ? p[lane + 32 * j] : 0.f;
    }
    __device__ __forceinline__ void norm(const float* w, float eps, uint32_t dim, uint32_t lane) {
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) s += v[j] * v[j];
        const float inv = 1.0f / sqrtf(warp_sum(s) / static_cast<float>(dim) + eps);
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (lane + 32 * j < dim) v[j] *= inv * w[lane + 32 * j];
    }
    template <typename T> __device__ __forceinline__ void store(T* p, uint32_t dim, uint32_t lane) const {     // zero up to pad8(dim)
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (lane + 32 * j < pad8(dim)) p[lane + 32 * j] = from_f32<T>(v[j]);
    }
};

template <typename T>
__global__ void __launch_bounds__(256) window_append_kernel(const __grid_constant__ hf2q_window_attn a, uint32_t m, T* __restrict__ q_out) {
    pdl_trigger();
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31, heads = a.heads + 2 * a.kv_heads;
    const uint64_t wid = static_cast<uint64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (wid >= static_cast<uint64_t>(m) * heads) return;
    const uint32_t t = static_cast<uint32_t>(wid / heads), h = static_cast<uint32_t>(wid % heads);
    const float* row = a.qkv + static_cast<size_t>(t) * a.ld;
    const uint32_t dp = pad8(a.dim), dvp = pad8(a.vdim), slot = (*a.pos + t) % a.capacity;
    HeadVec v;
    if (h < a.heads) {
        v.load(row + a.q_off + h * a.dim, a.dim, lane);
        if (a.q_norm) v.norm(a.q_norm, a.eps, a.dim, lane);
        v.store(q_out + (static_cast<size_t>(t) * a.heads + h) * dp, a.dim, lane);
    } else if (h < a.heads + a.kv_heads) {
        const uint32_t g = h - a.heads;
        v.load(row + a.k_off + g * a.dim, a.dim, lane);
        if (a.k_norm) v.norm(a.k_norm, a.eps, a.dim, lane);
        v.store(static_cast<T*>(a.k_cache) + (static_cast<size_t>(g) * a.capacity + slot) * dp, a.dim, lane);
    } else {
        const uint32_t g = h - a.heads - a.kv_heads;
        v.load(row + a.v_off + g * a.vdim, a.vdim, lane);
        v.store(static_cast<T*>(a.v_cache) + (static_cast<size_t>(g) * a.capacity + slot) * dvp, a.vdim, lane);
    }
}

// Online softmax of one warp for a query against keys [lo, hi) of its KV head; qs: [dp] f32 in shared memory, ps: [32] of this
// warp.  Lane = key for the scores, lane = value columns 2 lane + 64 c for the sums.
template <typename T, int NC, bool PLAIN>
struct WarpAttn {
    float mx, l, acc[NC][2];
    __device__ __forceinline__ void init() {
        mx = -CUDART_INF_F;
        l = 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[c][0] = acc[c][1] = 0.f;
    }
    __device__ __forceinline__ void keys(const hf2q_window_attn& a, const T* kc, const T* vc, const KeyRows<T, PLAIN>* kv, const float* qs, float* ps, float r1, float r2,
                                         uint32_t pos, uint32_t p0, uint32_t hi) {
        const uint32_t lane = threadIdx.x & 31, dp = pad8(a.dim), dvp = pad8(a.vdim);
        uint32_t dq = dp;
        if constexpr (PLAIN) dq += kv->sp;
        const uint32_t p = p0 + lane;
        const bool live = p < hi;
        float s = 0.f;
        if (live) {
            const T* kr;
            if constexpr (PLAIN) kr = kv->key(p);
            else kr = kc + static_cast<size_t>(p % a.capacity) * dp;
#pragma unroll 4
            for (uint32_t c = 0; c < dp; c += 8) {
                float k[8];
                load8(kr + c, k);
                const float4 x = *reinterpret_cast<const float4*>(qs + c), y = *reinterpret_cast<const float4*>(qs + c + 4);
                s += k[0] * x.x + k[1] * x.y + k[2] * x.z + k[3] * x.w + k[4] * y.x + k[5] * y.y + k[6] * y.z + k[7] * y.w;
            }
            if constexpr (PLAIN) {
                kr = kv->shared_key(p) - dp;
#pragma unroll 4
                for (uint32_t c = dp; c < dq; c += 8) {
                    float k[8];
                    load8(kr + c, k);
                    const float4 x = *reinterpret_cast<const float4*>(qs + c), y = *reinterpret_cast<const float4*>(qs + c + 4);
                    s += k[0] * x.x + k[1] * x.y + k[2] * x.z + k[3] * x.w + k[4] * y.x + k[5] * y.y + k[6] * y.z + k[7] * y.w;
                }
            }
        }
        const float sc = live ? score_of(s, a.scale, r1, r2, pos - p, a.r1 != nullptr) : -CUDART_INF_F;
        float bm = sc;
        for (int o = 16; o > 0; o >>= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, o));
        const float nm = fmaxf(mx, bm);
        const float corr = expf(mx - nm), pr = live ? expf(sc - nm) : 0.f;
        l = l * corr + warp_sum(pr);
        mx = nm;
#pragma unroll
        for (int c = 0; c < NC; ++c) { acc[c][0] *= corr; acc[c][1] *= corr; }
        ps[lane] = pr;
        __syncwarp();
        const uint32_t cnt = min(32u, hi - p0);
#pragma unroll 4
        for (uint32_t i = 0; i < cnt; ++i) {
            const T* vr;
            if constexpr (PLAIN) vr = kv->value(p0 + i);
            else vr = vc + static_cast<size_t>((p0 + i) % a.capacity) * dvp;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const uint32_t d = 2 * lane + 64 * c;
                if (d < dvp) {
                    const float v0 = to_f32(vr[d]), v1 = to_f32(vr[d + 1]);
                    const float w = ps[i];
                    acc[c][0] = fmaf(w, v0, acc[c][0]);
                    acc[c][1] = fmaf(w, v1, acc[c][1]);
                }
            }
        }
        __syncwarp();
    }
};

// ---------------------------------------------------------------- decode
// One token: WD_WARPS warps of a CTA take 16 keys each, 256 a pass.  Bound by the latency of its dependent steps, so what can be
// is asked for at once: a pair of lanes holds a key's row and a lane four columns of 16 values in registers, and the first tile
// is on its way before the query is normed.  The splits of a short window are a cluster and merge through distributed shared
// memory; a long one has more splits, whose last CTA merges them (cluster_splits).  Window 2048, 530 tokens there, 16 heads over 4 of
// 128: 9.8 us in a decode step; a lane per key, rows read four at a time and a merge through memory took 22.8.
constexpr int WD_WARPS = 16, WD_KEYS = 16;
constexpr uint32_t WD_PASS = WD_WARPS * WD_KEYS, WD_CLUSTER = 8;
__host__ __device__ constexpr uint32_t wd_part(uint32_t vdim) { return 4 + pad8(vdim); }

// eight elements of a key row, four of a value row, as they lie in memory
template <typename T> struct Raw;
template <> struct Raw<__nv_bfloat16> {
    typedef uint4 Eight;
    typedef uint2 Four;
    static __device__ __forceinline__ void open(const uint4& v, float (&o)[8]) {
        o[0] = bf_lo(v.x); o[1] = bf_hi(v.x); o[2] = bf_lo(v.y); o[3] = bf_hi(v.y);
        o[4] = bf_lo(v.z); o[5] = bf_hi(v.z); o[6] = bf_lo(v.w); o[7] = bf_hi(v.w);
    }
    static __device__ __forceinline__ void open(const uint2& v, float (&o)[4]) { o[0] = bf_lo(v.x); o[1] = bf_hi(v.x); o[2] = bf_lo(v.y); o[3] = bf_hi(v.y); }
};
template <> struct Raw<float> {
    struct Eight { float4 a, b; };
    typedef float4 Four;
    static __device__ __forceinline__ void open(const Eight& v, float (&o)[8]) {
        o[0] = v.a.x; o[1] = v.a.y; o[2] = v.a.z; o[3] = v.a.w; o[4] = v.b.x; o[5] = v.b.y; o[6] = v.b.z; o[7] = v.b.w;
    }
    static __device__ __forceinline__ void open(const float4& v, float (&o)[4]) { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
};

// grid (kv_heads * groups of GR query heads, splits), NC: values of up to 128 NC elements.  CLUSTER: the splits are a cluster;
// else scratch: counters [grid.x] (256-byte multiple), then [grid.x][splits][GR][max, sum, 2 pad, acc].
template <typename T, int GR, int NC, bool CLUSTER>
__global__ void __launch_bounds__(WD_WARPS * 32) window_decode_kernel(const __grid_constant__ hf2q_window_attn a, uint32_t groups, float* __restrict__ out,
                                                                      uint32_t* __restrict__ counters, float* __restrict__ part) {
    typedef typename Raw<T>::Eight Eight;
    typedef typename Raw<T>::Four Four;
    constexpr int HOLD = GR * NC >= 16 ? 32 : GR * NC >= 8 ? 64 : 128;      // bytes of a key's half and of values that a lane holds
    constexpr int KB = HOLD / sizeof(Eight), VB = HOLD / (4 * NC * sizeof(T));       // groups of eight, value rows
    static_assert(VB >= 1 && WD_KEYS % VB == 0, "");
    extern __shared__ __align__(16) float sm[];
    const uint32_t dp = pad8(a.dim), dvp = pad8(a.vdim), PP = wd_part(a.vdim), n8 = dp / 8;
    float* qs = sm;                                        // [GR][dp]
    float* ps = qs + GR * dp;                              // [warps][GR][16]
    float* rm = ps + WD_WARPS * GR * WD_KEYS;              // [warps][GR] max, then sums
    float* rl = rm + WD_WARPS * GR;
    float* ra = rl + WD_WARPS * GR;                        // [warps][GR][dvp]
    float* sum = ra + WD_WARPS * GR * dvp;                 // CLUSTER: [GR][max, sum, 2 pad, acc] of this CTA
    __shared__ uint32_t is_last;
    pdl_trigger();
    pdl_wait();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t kvh = blockIdx.x / groups, rep = a.heads / a.kv_heads, g0 = (blockIdx.x % groups) * GR, n_g = min(static_cast<uint32_t>(GR), rep - g0);
    const uint32_t h0 = kvh * rep + g0, split = blockIdx.y, nsplit = gridDim.y;
    const uint32_t pos = *a.pos, n = min(pos + 1, a.window), first = pos + 1 - n;
    const uint32_t chunk = (n + nsplit - 1) / nsplit;
    const uint32_t lo = first + min(split * chunk, n), hi = first + min(split * chunk + chunk, n);
    T* kc = static_cast<T*>(a.k_cache) + static_cast<size_t>(kvh) * a.capacity * dp;
    T* vc = static_cast<T*>(a.v_cache) + static_cast<size_t>(kvh) * a.capacity * dvp;
    const uint32_t half = lane & 1;
    Eight kr[KB];
    Four vr[VB][NC];
    // groups 2 (c0 + j) + half of key p; rows v0 .. v0 + VB of the tile at p0 (columns past the row: the row's start)
    auto load_k = [&](uint32_t p, uint32_t c0) {
        const Eight* row = reinterpret_cast<const Eight*>(kc + static_cast<size_t>(p % a.capacity) * dp);
#pragma unroll
        for (int j = 0; j < KB; ++j)
            if (2 * (c0 + j) + half < n8) kr[j] = row[2 * (c0 + j) + half];
    };
    auto load_v = [&](uint32_t p, int i) {
        const T* row = vc + static_cast<size_t>(p % a.capacity) * dvp;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const uint32_t d = 4 * lane + 128 * c;
            vr[i][c] = *reinterpret_cast<const Four*>(row + (d < dvp ? d : 0u));
        }
    };
    auto load_rows = [&](uint32_t p0, uint32_t v0) {       // (past the end: the tile's first row, with weight zero)
#pragma unroll
        for (int i = 0; i < VB; ++i) load_v(p0 + v0 + i < hi ? p0 + v0 + i : p0, i);
    };
    // ahead of the query; the new position's row is not there yet
    uint32_t p0 = lo + warp * WD_KEYS;
    if (p0 < hi) {
        load_k(min(p0 + lane / 2, hi - 1), 0);
        load_rows(p0, 0);
    }
    if (warp < GR) {
        HeadVec v;
        v.load(a.qkv + a.q_off + (h0 + min(warp, n_g - 1)) * a.dim, a.dim, lane);
        if (a.q_norm) v.norm(a.q_norm, a.eps, a.dim, lane);
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (lane + 32 * j < dp) qs[warp * dp + lane + 32 * j] = to_f32(from_f32<T>(v.v[j]));      // the prefill's operand precision
    } else if (pos >= lo && pos < hi && warp < GR + 2) {   // the new position, by the CTAs whose range holds it
        const uint32_t slot = pos % a.capacity;
        HeadVec v;
        if (warp == GR) {
            v.load(a.qkv + a.k_off + kvh * a.dim, a.dim, lane);
            if (a.k_norm) v.norm(a.k_norm, a.eps, a.dim, lane);
            v.store(kc + static_cast<size_t>(slot) * dp, a.dim, lane);
        } else {
            v.load(a.qkv + a.v_off + kvh * a.vdim, a.vdim, lane);
            v.store(vc + static_cast<size_t>(slot) * dvp, a.vdim, lane);
        }
    }
    float r1[GR], r2[GR];
#pragma unroll
    for (int g = 0; g < GR; ++g) {
        r1[g] = a.r1 ? a.r1[h0 + min(static_cast<uint32_t>(g), n_g - 1)] : 0.f;
        r2[g] = a.r1 ? a.r2[h0 + min(static_cast<uint32_t>(g), n_g - 1)] : 0.f;
    }
    __syncthreads();
    if (p0 < hi && pos >= p0 && pos < p0 + WD_KEYS) {      // this tile holds the new position (its last key): its rows as they are now
        if (p0 + lane / 2 >= pos) load_k(pos, 0);
#pragma unroll
        for (int i = 0; i < VB; ++i)
            if (p0 + i == pos) load_v(pos, i);
    }
    float mx[GR], l[GR], acc[GR][NC][4];
#pragma unroll
    for (int g = 0; g < GR; ++g) {
        mx[g] = -CUDART_INF_F;
        l[g] = 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[g][c][0] = acc[g][c][1] = acc[g][c][2] = acc[g][c][3] = 0.f;
    }
    float* pw = ps + warp * GR * WD_KEYS;
    for (bool held = true; p0 < hi; p0 += WD_PASS, held = false) {
        const uint32_t p = min(p0 + lane / 2, hi - 1);
        const bool live = p0 + lane / 2 < hi;
        if (!held) { load_k(p, 0); load_rows(p0, 0); }
        float s[GR];
#pragma unroll
        for (int g = 0; g < GR; ++g) s[g] = 0.f;
        for (uint32_t c0 = 0; 2 * c0 < n8; c0 += KB) {
            if (c0) load_k(p, c0);
#pragma unroll
            for (int j = 0; j < KB; ++j) {
                const uint32_t c = 2 * (c0 + j) + half;
                if (c < n8) {
                    float k[8];
                    Raw<T>::open(kr[j], k);
#pragma unroll
                    for (int g = 0; g < GR; ++g) {
                        const float4 x = *reinterpret_cast<const float4*>(qs + g * dp + 8 * c), y = *reinterpret_cast<const float4*>(qs + g * dp + 8 * c + 4);
                        s[g] += k[0] * x.x + k[1] * x.y + k[2] * x.z + k[3] * x.w + k[4] * y.x + k[5] * y.y + k[6] * y.z + k[7] * y.w;
                    }
                }
            }
        }
#pragma unroll
        for (int g = 0; g < GR; ++g) {
            const float dot = s[g] + __shfl_xor_sync(0xffffffffu, s[g], 1);
            const float sc = live ? score_of(dot, a.scale, r1[g], r2[g], pos - p, a.r1 != nullptr) : -CUDART_INF_F;
            float bm = sc;
            for (int o = 16; o > 1; o >>= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, o));
            const float nm = fmaxf(mx[g], bm);
            const float corr = expf(mx[g] - nm), pr = live ? expf(sc - nm) : 0.f;
            float total = pr;
            for (int o = 16; o > 1; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
            l[g] = l[g] * corr + total;
            mx[g] = nm;
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int u = 0; u < 4; ++u) acc[g][c][u] *= corr;
            if (half == 0) pw[g * WD_KEYS + lane / 2] = pr;
        }
        __syncwarp();
#pragma unroll
        for (uint32_t v0 = 0; v0 < WD_KEYS; v0 += VB) {
            if (v0) load_rows(p0, v0);
#pragma unroll
            for (int i = 0; i < VB; ++i) {
                const bool there = p0 + v0 + i < hi;       // (a row past the end may hold anything: it does not enter, finite or not)
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    float v[4];
                    Raw<T>::open(vr[i][c], v);
                    if (there)
#pragma unroll
                        for (int g = 0; g < GR; ++g) {
                            const float w = pw[g * WD_KEYS + v0 + i];
#pragma unroll
                            for (int u = 0; u < 4; ++u) acc[g][c][u] = fmaf(w, v[u], acc[g][c][u]);
                        }
                }
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int g = 0; g < GR; ++g) {
        if (lane == 0) { rm[warp * GR + g] = mx[g]; rl[warp * GR + g] = l[g]; }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const uint32_t d = 4 * lane + 128 * c;
            if (d < dvp) *reinterpret_cast<float4*>(ra + (warp * GR + g) * dvp + d) = make_float4(acc[g][c][0], acc[g][c][1], acc[g][c][2], acc[g][c][3]);
        }
    }
    __syncthreads();
    float* mine = CLUSTER ? sum : part + (static_cast<size_t>(blockIdx.x) * nsplit + split) * GR * PP;
    for (uint32_t i = threadIdx.x; i < GR * dvp; i += WD_WARPS * 32) {
        const uint32_t g = i / dvp, d = i % dvp;
        float m = -CUDART_INF_F, t = 0.f, v = 0.f;
#pragma unroll
        for (int k = 0; k < WD_WARPS; ++k) m = fmaxf(m, rm[k * GR + g]);
#pragma unroll
        for (int k = 0; k < WD_WARPS; ++k) {
            const float c = rm[k * GR + g] == -CUDART_INF_F ? 0.f : expf(rm[k * GR + g] - m);
            t += rl[k * GR + g] * c;
            v += ra[(k * GR + g) * dvp + d] * c;
        }
        if (nsplit == 1) {
            if (g < n_g && d < a.vdim) out[(h0 + g) * a.vdim + d] = v / t;
        } else {
            if (d == 0) { mine[g * PP] = m; mine[g * PP + 1] = t; }
            mine[g * PP + 4 + d] = v;
        }
    }
    if (nsplit == 1) return;
    if constexpr (CLUSTER) {
        const cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        // the outputs are spread over the cluster; every CTA's sums in split order
        for (uint32_t i = split * (WD_WARPS * 32) + threadIdx.x; i < n_g * a.vdim; i += nsplit * (WD_WARPS * 32)) {
            const uint32_t g = i / a.vdim, d = i % a.vdim;
            float mk[WD_CLUSTER], lk[WD_CLUSTER], vk[WD_CLUSTER], m = -CUDART_INF_F, t = 0.f, v = 0.f;
#pragma unroll
            for (uint32_t k = 0; k < WD_CLUSTER; ++k) {
                const float* src = cl.map_shared_rank(sum, k < nsplit ? k : 0u) + g * PP;
                mk[k] = k < nsplit ? src[0] : -CUDART_INF_F; lk[k] = src[1]; vk[k] = src[4 + d];
                m = fmaxf(m, mk[k]);
            }
#pragma unroll
            for (uint32_t k = 0; k < WD_CLUSTER; ++k)
                if (mk[k] != -CUDART_INF_F) {
                    const float c = expf(mk[k] - m);
                    t += lk[k] * c;
                    v += vk[k] * c;
                }
            out[(h0 + g) * a.vdim + d] = v / t;
        }
        cl.sync();                                                   // the others read this CTA's sums until here
        return;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t old = atomicAdd(&counters[blockIdx.x], 1u);
        is_last = old == nsplit - 1;
        if (is_last) counters[blockIdx.x] = 0;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    const float* all = part + static_cast<size_t>(blockIdx.x) * nsplit * GR * PP;
    for (uint32_t i = threadIdx.x; i < n_g * a.vdim; i += WD_WARPS * 32) {
        const uint32_t g = i / a.vdim, d = i % a.vdim;
        float m = -CUDART_INF_F, t = 0.f, v = 0.f;
        for (uint32_t k = 0; k < nsplit; ++k) m = fmaxf(m, __ldcg(all + (k * GR + g) * PP));
        for (uint32_t k = 0; k < nsplit; ++k) {
            const float* src = all + (k * GR + g) * PP;
            const float mk = __ldcg(src), c = mk == -CUDART_INF_F ? 0.f : expf(mk - m);
            t += __ldcg(src + 1) * c;
            v += __ldcg(src + 4 + d) * c;
        }
        out[(h0 + g) * a.vdim + d] = v / t;
    }
}

constexpr uint32_t QK_MAX = 320;                        // dim and shared_dim together, padded

// ---------------------------------------------------------------- prefill, f32: one warp per (query, head)
// query t of head h by one warp; qs [QK_MAX] and ps [32] of this warp in shared memory
template <typename T, typename OUT, int NC, bool PLAIN>
__device__ __forceinline__ void f32_query(const hf2q_window_attn& a, uint32_t pos0, uint32_t t, uint32_t h, const T* q, const float* gate,
                                          uint32_t ldg, OUT* __restrict__ out, uint32_t ldo, float* qs, float* ps) {
    const uint32_t lane = threadIdx.x & 31;
    const KeyRows<T, PLAIN> kv(a, h / (a.heads / a.kv_heads), pos0);
    const uint32_t dq = kv.dp + kv.sp;
    for (uint32_t i = lane; i < dq; i += 32) qs[i] = to_f32(q[(static_cast<size_t>(t) * a.heads + h) * dq + i]);
    __syncwarp();
    const uint32_t pos = pos0 + t, n = min(pos + 1, a.window), hi = pos + 1;
    const float r1 = a.r1 ? a.r1[h] : 0.f, r2 = a.r1 ? a.r2[h] : 0.f;
    WarpAttn<T, NC, PLAIN> w;
    w.init();
    for (uint32_t p0 = hi - n; p0 < hi; p0 += 32) w.keys(a, kv.k, kv.v, &kv, qs, ps, r1, r2, pos, p0, hi);
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t d = 2 * lane + 64 * c + u;
            if (d < a.vdim) {
                float v = w.acc[c][u] / w.l;
                if (gate) v *= sigmoidf(gate[static_cast<size_t>(t) * ldg + h * a.vdim + d]);
                out[static_cast<size_t>(t) * ldo + h * a.vdim + d] = from_f32<OUT>(v);
            }
        }
    if (h == a.heads - 1)
        for (uint32_t i = a.heads * a.vdim + lane; i < ldo; i += 32) out[static_cast<size_t>(t) * ldo + i] = from_f32<OUT>(0.f);
}
template <typename T, typename OUT, int NC, bool PLAIN>
__global__ void __launch_bounds__(256) window_prefill_f32_kernel(const __grid_constant__ hf2q_window_attn a, uint32_t m, const T* q,
                                                                 const float* gate, uint32_t ldg, OUT* __restrict__ out, uint32_t ldo) {
    __shared__ __align__(16) float qs[8][QK_MAX];
    __shared__ float ps[8][32];
    pdl_trigger();
    pdl_wait();
    const uint32_t warp = threadIdx.x >> 5, t = blockIdx.x * 8 + warp;
    if (t >= m) return;
    f32_query<T, OUT, NC, PLAIN>(a, *a.pos, t, blockIdx.y, q, gate, ldg, out, ldo, qs[warp], ps[warp]);
}

// ---------------------------------------------------------------- prefill, bf16 cache, tcgen05
// One CTA owns 128 queries of one head and walks the keys from the first one that its first query sees, 64 at a time:
//
//   warps 4-7   copy keys and values (16 bytes a time, asynchronously) to shared memory with the 128-byte swizzle, two blocks
//               deep; K is the K-major B operand of the scores, V, in the same layout, the MN-major one of the output.
//   warp 8      one lane issues the products: the scores of the next block before the output of this one.
//   warps 0-3   softmax, a thread to a query: scores from tensor memory are scaled, biased, masked and put back, then read
//               again for the exponentials (64 of them would not fit the registers beside the rest); P takes their place.
//               The output rows of a warp are rescaled wherever one's running maximum grew: with the true maximum the largest
//               weight is 1, which bf16 holds exactly (an older one within 2^8 was no faster and doubled the error of peaked rows).
//
// The weight of a key that a query does not see is zero, but zero times a value that is not finite is NaN.  So warps 4-7 look
// for such values in the blocks that some query does not see whole; a tile that has one is done again in f32, a warp to a query.
//
// 256 tensor-memory columns (S 2 x 64, O 128).  Two CTAs per SM with keys of up to 128 elements, one with 192.  It is bound by
// the latency of a block's chain (scores, maximum, exponentials, output).  2048 queries x 16 heads of 128 with 2048 keys each
// take 168 us (the warp-level kernel below took 397), with keys of 192 elements 229 us (519).
constexpr uint32_t WT_Q = 128, WT_K = 64, WT_V = 128, WT_THREADS = 288, WT_COLS = 256, WT_O = 128, WT_PANEL = WT_K * 128;
constexpr uint32_t wt_smem(uint32_t dk) { return WT_Q * dk * 2 + 2 * WT_K * dk * 2 + 2 * WT_K * WT_V * 2 + 1024; }

__device__ __forceinline__ float lg2(float x) { float y; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
// 16-byte chunk c of a row, in panels of `rows` rows x 64 elements
__device__ __forceinline__ uint32_t wt_chunk(uint32_t rows, uint32_t row, uint32_t c) { return (c >> 3) * rows * 128 + row * 128 + (((c & 7) ^ (row & 7)) << 4); }

// the queries t0 .. t0 + n of head h again, in f32; work: WT_THREADS / 32 x (QK_MAX + 32) floats of shared memory
template <typename OUT, bool PLAIN>
__device__ __noinline__ void wt_again(const hf2q_window_attn& a, uint32_t pos0, uint32_t t0, uint32_t n, uint32_t h, const __nv_bfloat16* q, const float* gate,
                                      uint32_t ldg, OUT* out, uint32_t ldo, float* work) {
    float* qs = work + (threadIdx.x >> 5) * (QK_MAX + 32);
    for (uint32_t t = threadIdx.x >> 5; t < n; t += WT_THREADS / 32)
        f32_query<__nv_bfloat16, OUT, WT_V / 64, PLAIN>(a, pos0, t0 + t, h, q, gate, ldg, out, ldo, qs, qs + QK_MAX);
}

template <int DK, typename OUT, bool PLAIN>
__global__ void __launch_bounds__(WT_THREADS, DK <= 128 ? 2 : 1) window_prefill_tc_kernel(const __grid_constant__ hf2q_window_attn a, uint32_t m,
                                                                                          const __nv_bfloat16* q, const float* gate,
                                                                                          uint32_t ldg, OUT* __restrict__ out, uint32_t ldo, uint32_t* status) {
    extern __shared__ __align__(16) uint8_t wt_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(wt_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    constexpr uint32_t Q_BYTES = WT_Q * DK * 2, K_BYTES = WT_K * DK * 2, V_BYTES = WT_K * WT_V * 2;
    uint8_t *qs = smem, *ks = smem + Q_BYTES, *vs = ks + 2 * K_BYTES;
    __shared__ uint64_t k_full[2], v_full[2], s_full[2], p_full[2], o_done[2];
    __shared__ uint32_t tmem_slot, again;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t h = blockIdx.y, t0 = (gridDim.x - 1 - blockIdx.x) * WT_Q;
    if (threadIdx.x == 0) {
        again = 0;
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 4);
            mbar_init(&v_full[i], 4);
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], 4);
            mbar_init(&o_done[i], 1);
        }
        mbar_fence_init();
    }
    if (warp == 8) { tc::tmem_alloc(&tmem_slot, WT_COLS); tc::tmem_relinquish(); }
    __syncthreads();
    pdl_trigger();                                             // (dependents may claim tensor memory too: not before this CTA has its own)
    pdl_wait();
    const uint32_t pos0 = *a.pos;
    const KeyRows<__nv_bfloat16, PLAIN> rows(a, h / (a.heads / a.kv_heads), pos0);
    const uint32_t dq = rows.dp + rows.sp, dvp = pad8(a.vdim), nk = (dq + 15) / 16;
    const uint32_t q_lo = pos0 + t0, q_hi = pos0 + min(t0 + WT_Q, m) - 1;
    const uint32_t j0 = q_lo + 1 > a.window ? q_lo + 1 - a.window : 0u, nb = (q_hi - j0) / WT_K + 1;
    // some query of the tile (those past the end included) does not see all of block j
    auto edge = [&](uint32_t j) { return j0 + j * WT_K + WT_K - 1 > q_lo || q_lo + WT_Q - 1 - (j0 + j * WT_K) >= a.window; };
    if (dq < DK || dvp < WT_V) {                               // elements past dim / vdim must be finite zeros
        for (uint32_t i = threadIdx.x; i < (2 * K_BYTES + 2 * V_BYTES) / 16; i += WT_THREADS) reinterpret_cast<uint4*>(ks)[i] = make_uint4(0, 0, 0, 0);
    }
    const bool wide_q = reinterpret_cast<uintptr_t>(q) % 16 == 0;          // rows are whole 16-byte groups
    for (uint32_t i = threadIdx.x; i < WT_Q * (DK / 8); i += WT_THREADS) {
        const uint32_t r = i / (DK / 8), c = i % (DK / 8);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (t0 + r < m && 8 * c < dq) {
            const __nv_bfloat16* src = q + (static_cast<size_t>(t0 + r) * a.heads + h) * dq + 8 * c;
            if (wide_q) {
                v = *reinterpret_cast<const uint4*>(src);
            } else {
                const uint32_t* w = reinterpret_cast<const uint32_t*>(src);
                v = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        *reinterpret_cast<uint4*>(qs + wt_chunk(WT_Q, r, c)) = v;
    }
    tc::proxy_fence();
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp >= 4 && warp < 8) {
        const uint32_t tid = threadIdx.x - 128, c0 = tid & 7, row0 = tid >> 3, ck = dq / 8, cv = dvp / 8, cd = rows.dp / 8;
        bool ok = true;
        // iteration j starts the copies of block j and hands over those of block j - 1
        for (uint32_t j = 0; j <= nb; ++j) {
            const uint32_t b = j & 1, par = ((j >> 1) - 1) & 1;
            if (j < nb) {
                if (j >= 2) ok = __all_sync(0xffffffffu, mbar_wait_bounded(&s_full[b], par, status));        // S(j-2) is there: its K block is free
                if (!ok) break;
#pragma unroll
                for (uint32_t i = 0; i < WT_K / 16; ++i) {
                    const uint32_t r = row0 + 16 * i, key = min(j0 + j * WT_K + r, q_hi);             // keys past the last visible one repeat it
                    const __nv_bfloat16* src = rows.key(key);
                    for (uint32_t c = c0; c < ck; c += 8) {
                        const __nv_bfloat16* from = !PLAIN || c < cd ? src + 8 * c : rows.shared_key(key) + 8 * (c - cd);
                        cp_async16(ks + b * K_BYTES + wt_chunk(WT_K, r, c), from);
                    }
                }
            }
            cp_async_commit();
            if (j > 0) {
                cp_async_wait<2>();                            // all but the copies of V(j-1) and K(j)
                tc::proxy_fence();
                __syncwarp();
                if (lane == 0) mbar_arrive(&k_full[b ^ 1]);
                cp_async_wait<1>();
                tc::proxy_fence();
                __syncwarp();
                if (lane == 0) mbar_arrive(&v_full[b ^ 1]);
            }
            if (j < nb) {
                if (j >= 2) ok = __all_sync(0xffffffffu, mbar_wait_bounded(&o_done[b], par, status));        // the output of j-2 is in: its V block is free
                if (!ok) break;
#pragma unroll
                for (uint32_t i = 0; i < WT_K / 16; ++i) {
                    const uint32_t r = row0 + 16 * i;
                    const __nv_bfloat16* src = rows.value(min(j0 + j * WT_K + r, q_hi));
                    for (uint32_t c = c0; c < cv; c += 8) cp_async16(vs + b * V_BYTES + wt_chunk(WT_K, r, c), src + 8 * c);
                }
            }
            cp_async_commit();
            if (j > 0 && edge(j - 1)) {                        // this thread's copies of V(j-1): a value whose exponent is all ones?
                uint32_t top = 0;
                auto full = [](uint32_t w) { return (w & 0x7F807F80u) + 0x00800080u; };       // bit 15 of a half: its exponent was
#pragma unroll
                for (uint32_t i = 0; i < WT_K / 16; ++i)
                    for (uint32_t c = c0; c < cv; c += 8) {
                        const uint4 w = *reinterpret_cast<const uint4*>(vs + (b ^ 1) * V_BYTES + wt_chunk(WT_K, row0 + 16 * i, c));
                        top |= full(w.x) | full(w.y) | full(w.z) | full(w.w);
                    }
                if (top & 0x80008000u) again = 1;
            }
        }
        cp_async_wait<0>();
    } else if (warp == 8) {
        if (lane == 0) {
            // D f32, A and B bf16, M = 128; S: both K-major, N = 64; O: B MN-major, N = 128
            constexpr uint32_t ID = (1u << 4) | (1u << 7) | (1u << 10) | ((WT_Q >> 4) << 24), ID_S = ID | ((WT_K >> 3) << 17), ID_O = ID | (1u << 16) | ((WT_V >> 3) << 17);
            bool ok = true;
            auto scores = [&](uint32_t j) {
                const uint32_t b = j & 1;
                ok = mbar_wait_bounded(&k_full[b], (j >> 1) & 1, status);
                if (ok && j >= 2) ok = mbar_wait_bounded(&o_done[b], ((j >> 1) - 1) & 1, status);   // P(j-2) is read: S(j) takes its place
                if (!ok) return;
                tc::tc_fence_after();
#pragma unroll
                for (uint32_t kk = 0; kk < DK / 16; ++kk)
                    if (kk < nk)
                        tc::umma_ss(tmem + b * WT_K, tc::smem_desc_sw128(smem_u32(qs + (kk >> 2) * (WT_Q * 128))) + 2 * (kk & 3),
                                    tc::smem_desc_sw128(smem_u32(ks + b * K_BYTES + (kk >> 2) * WT_PANEL)) + 2 * (kk & 3), ID_S, kk ? 1u : 0u);
                tc::tc_commit(&s_full[b]);
            };
            scores(0);
            for (uint32_t j = 0; j < nb && ok; ++j) {
                const uint32_t b = j & 1;
                if (j + 1 < nb) scores(j + 1);
                if (ok) ok = mbar_wait_bounded(&v_full[b], (j >> 1) & 1, status);
                if (ok) ok = mbar_wait_bounded(&p_full[b], (j >> 1) & 1, status);
                if (!ok) break;
                tc::tc_fence_after();
#pragma unroll
                for (uint32_t kk = 0; kk < WT_K / 16; ++kk)
                    tc::umma_ts(tmem + WT_O, tmem + b * WT_K + 8 * kk, tc::smem_desc_mn_sw128(smem_u32(vs + b * V_BYTES), WT_PANEL) + kk * (16 * 128 >> 4), ID_O, (j | kk) ? 1u : 0u);
                tc::tc_commit(&o_done[b]);
            }
        }
    } else {
        const uint32_t t = t0 + threadIdx.x, at = tmem + ((warp * 32u) << 16), qp = pos0 + t;
        const bool live = t < m, bias = a.r1 != nullptr;       // (rows past the end compute on zeros and are not stored)
        const float r1 = bias ? a.r1[h] : 0.f, r2 = bias ? a.r2[h] : 0.f, scale = a.scale * 1.4426950408889634f;      // scores in units of log2
        float mx = -CUDART_INF_F, sum[2] = {0.f, 0.f};
        bool ok = true;
        for (uint32_t j = 0; j < nb; ++j) {
            const uint32_t b = j & 1, key0 = j0 + j * WT_K;
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&s_full[b], (j >> 1) & 1, status));
            if (!ok) break;
            tc::tc_fence_after();
            float top[2] = {-CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) {
                uint32_t r[32];
                tc::tmem_ld32(at + b * WT_K + 32 * half, r);
                tc::tmem_wait_ld();
                const uint32_t d0 = qp - key0 - 32 * half;     // distance to the first key; wraps for keys after the query
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * scale);
                if (bias) {
                    const float d0f = static_cast<float>(static_cast<int>(d0));        // (whole numbers; what is hidden may become NaN here)
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) - r1 * lg2(fmaf(r2, d0f - i, 1.0f)));
                }
                if (edge(j)) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = d0 - i < a.window ? r[i] : __float_as_uint(-CUDART_INF_F);
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) top[i & 1] = fmaxf(top[i & 1], __uint_as_float(r[i]));
                tc::tmem_st32(at + b * WT_K + 32 * half, r);
            }
            tc::tmem_wait_st();
            const float bm = fmaxf(top[0], top[1]);
            const bool grew = bm > mx;
            if (j == 0) {
                mx = bm;
            } else if (__any_sync(0xffffffffu, grew)) {
                const float to = grew ? bm : mx, corr = grew ? tc::ex2(mx - to) : 1.0f;
                mx = to;
                sum[0] *= corr;
                sum[1] *= corr;
                ok = __all_sync(0xffffffffu, mbar_wait_bounded(&o_done[b ^ 1], ((j - 1) >> 1) & 1, status));
                if (!ok) break;
                tc::tc_fence_after();
#pragma unroll 1
                for (uint32_t c = 0; c < WT_V; c += 32) {
                    uint32_t o[32];
                    tc::tmem_ld32(at + WT_O + c, o);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                    tc::tmem_st32(at + WT_O + c, o);
                }
            }
            const float nm = mx == -CUDART_INF_F ? 0.f : mx;   // nothing visible yet: every weight is 2^-inf = 0
#pragma unroll
            for (uint32_t c = 0; c < WT_K / 16; ++c) {
                uint32_t r[16], p[8];
                tc::tmem_ld16(at + b * WT_K + 16 * c, r);
                tc::tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float x = tc::ex2(__uint_as_float(r[2 * i]) - nm), y = tc::ex2(__uint_as_float(r[2 * i + 1]) - nm);
                    sum[0] += x;
                    sum[1] += y;
                    p[i] = pack_bf16(x, y);
                }
                tc::tmem_st8(at + b * WT_K + 8 * c, p);        // over scores that have been read
            }
            tc::tmem_wait_st();
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[b]);
        }
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait_bounded(&o_done[(nb - 1) & 1], ((nb - 1) >> 1) & 1, status));
        if (ok) {
            tc::tc_fence_after();
            const float inv = 1.0f / (sum[0] + sum[1]);
            OUT* dst = out + static_cast<size_t>(live ? t : 0) * ldo + h * a.vdim;
            const float* gr = gate ? gate + static_cast<size_t>(live ? t : 0) * ldg + h * a.vdim : nullptr;
            const bool wide = (reinterpret_cast<uintptr_t>(out) | ldo * sizeof(OUT) | a.vdim * sizeof(OUT)) % 16 == 0 &&
                              (!gate || (reinterpret_cast<uintptr_t>(gate) | ldg * sizeof(float) | a.vdim * sizeof(float)) % 16 == 0);
#pragma unroll 1
            for (uint32_t c = 0; c < a.vdim; c += 16) {
                uint32_t o[16];
                tc::tmem_ld16(at + WT_O + c, o);
                tc::tmem_wait_ld();
                if (live) {
                    float v[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(o[i]) * inv;
                    if (wide && c + 16 <= a.vdim) {
                        if (gr) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const float4 g = *reinterpret_cast<const float4*>(gr + c + 4 * i);
                                v[4 * i] *= sigmoidf(g.x);
                                v[4 * i + 1] *= sigmoidf(g.y);
                                v[4 * i + 2] *= sigmoidf(g.z);
                                v[4 * i + 3] *= sigmoidf(g.w);
                            }
                        }
                        if constexpr (sizeof(OUT) == 4) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(dst + c + 4 * i) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                        } else {
#pragma unroll
                            for (int i = 0; i < 2; ++i)
                                *reinterpret_cast<uint4*>(dst + c + 8 * i) = make_uint4(pack_bf16(v[8 * i], v[8 * i + 1]), pack_bf16(v[8 * i + 2], v[8 * i + 3]),
                                                                                        pack_bf16(v[8 * i + 4], v[8 * i + 5]), pack_bf16(v[8 * i + 6], v[8 * i + 7]));
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (c + i < a.vdim) dst[c + i] = from_f32<OUT>(gr ? v[i] * sigmoidf(gr[c + i]) : v[i]);
                    }
                }
                __syncwarp();                                  // the next load from tensor memory is the whole warp's
            }
            if (live && h == a.heads - 1)
                for (uint32_t i = a.heads * a.vdim; i < ldo; ++i) out[static_cast<size_t>(t) * ldo + i] = from_f32<OUT>(0.f);
        }
        tc::tc_fence_before();
    }
    __syncthreads();
    if (warp == 8) { tc::tc_fence_after(); tc::tmem_dealloc(tmem, WT_COLS); }
    if (again) wt_again<OUT, PLAIN>(a, pos0, t0, min(WT_Q, m - t0), h, q, gate, ldg, out, ldo, reinterpret_cast<float*>(smem));
}

// ---------------------------------------------------------------- prefill, bf16 cache: warp-level products
// 2048 queries x 16 heads with 2048 keys each take 147 us with 64 elements a key and value (on tcgen05, whose tiles hold 128 each,
// 146), 952 with ring keys of 192 (no tcgen05 form of those is built; rows: 229) and 1328 with 256.
constexpr int WP_WARPS = 4, WP_Q = 16 * WP_WARPS, WP_K = 64;

// grid (query tiles, heads); DK >= dim + shared_dim, DV >= vdim.  Keys are walked from the first one the tile's first
// query sees.
template <int DK, int DV, typename OUT, bool PLAIN>
__global__ void __launch_bounds__(WP_WARPS * 32) window_prefill_mma_kernel(const __grid_constant__ hf2q_window_attn a, uint32_t m,
                                                                           const __nv_bfloat16* q, const float* gate, uint32_t ldg,
                                                                           OUT* __restrict__ out, uint32_t ldo) {
    constexpr uint32_t KP = DK + 8, VP = DV + 8, K_TILE = WP_K * KP, TILES = K_TILE + WP_K * VP;      // pitches and sizes in elements
    extern __shared__ __align__(16) __nv_bfloat16 kv[];             // [2][K tile, V tile]
    pdl_trigger();
    pdl_wait();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, t4 = lane & 3;
    const uint32_t h = blockIdx.y, t0 = blockIdx.x * WP_Q;
    const uint32_t pos0 = *a.pos;
    const KeyRows<__nv_bfloat16, PLAIN> rows(a, h / (a.heads / a.kv_heads), pos0);
    const uint32_t dq = rows.dp + rows.sp, dvp = pad8(a.vdim), nk = (dq + 15) / 16, nv = (dvp + 15) / 16;
    const uint32_t q_lo = pos0 + t0, q_hi = pos0 + min(t0 + WP_Q, m) - 1;
    const uint32_t j0 = q_lo + 1 > a.window ? q_lo + 1 - a.window : 0u;
    // elements past dim / vdim, and keys never loaded, must be finite zeros
    for (uint32_t i = threadIdx.x; i < 2 * TILES / 8; i += WP_WARPS * 32) reinterpret_cast<uint4*>(kv)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    auto stage = [&](uint32_t key0, uint32_t b) {
        __nv_bfloat16* ks = kv + b * TILES;
        __nv_bfloat16* vs = ks + K_TILE;
        const uint32_t ck = dq / 8, cv = dvp / 8, cd = rows.dp / 8;
        for (uint32_t i = threadIdx.x; i < WP_K * ck; i += WP_WARPS * 32) {
            const uint32_t r = i / ck, c = i % ck;
            if (key0 + r <= q_hi) cp_async16(ks + r * KP + 8 * c, !PLAIN || c < cd ? rows.key(key0 + r) + 8 * c : rows.shared_key(key0 + r) + 8 * (c - cd));
        }
        for (uint32_t i = threadIdx.x; i < WP_K * cv; i += WP_WARPS * 32) {
            const uint32_t r = i / cv, c = i % cv;
            if (key0 + r <= q_hi) cp_async16(vs + r * VP + 8 * c, rows.value(key0 + r) + 8 * c);
        }
        cp_async_commit();
    };
    stage(j0, 0);
    uint32_t qa[DK / 16][4];
    uint32_t row[2], qpos[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) { row[u] = t0 + warp * 16 + gid + 8 * u; qpos[u] = pos0 + row[u]; }
#pragma unroll
    for (int k = 0; k < DK / 16; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t r = row[i & 1], c = 16 * k + 8 * (i >> 1) + 2 * t4;
            qa[k][i] = r < m && c < dq ? *reinterpret_cast<const uint32_t*>(q + (static_cast<size_t>(r) * a.heads + h) * dq + c) : 0u;
        }
    const bool bias = a.r1 != nullptr;
    const float r1 = bias ? a.r1[h] : 0.f, r2 = bias ? a.r2[h] : 0.f;
    float mx[2] = {-CUDART_INF_F, -CUDART_INF_F}, l[2] = {0.f, 0.f};
    float o[DV / 8][4];
#pragma unroll
    for (int i = 0; i < DV / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    const uint32_t n_tiles = (q_hi - j0) / WP_K + 1;
    const uint32_t w_lo = pos0 + t0 + warp * 16, w_hi = w_lo + 15;           // this warp's query positions
    for (uint32_t kt = 0; kt < n_tiles; ++kt) {
        const uint32_t key0 = j0 + kt * WP_K, b = kt & 1;
        if (kt + 1 < n_tiles) { stage(key0 + WP_K, b ^ 1); cp_async_wait<1>(); }
        else cp_async_wait<0>();
        __syncthreads();
        // keys above this warp's last query or below its first window edge touch none of its rows
        if (key0 <= w_hi && key0 + WP_K - 1 + a.window > w_lo) {
            const uint32_t ks = smem_u32(kv + b * TILES), vs = ks + K_TILE * 2;
            float s[WP_K / 8][4];
#pragma unroll
            for (int i = 0; i < WP_K / 8; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll
            for (int k = 0; k < DK / 16; ++k) {
                if (k < static_cast<int>(nk)) {
#pragma unroll
                    for (int n2 = 0; n2 < WP_K / 16; ++n2) {
                        uint32_t f[4];
                        ldmatrix4(f, ks + ((n2 * 16 + (lane >> 4) * 8 + (lane & 7)) * KP + 16 * k + ((lane >> 3) & 1) * 8) * 2);
                        mma_bf16(s[2 * n2], qa[k], f[0], f[1]);
                        mma_bf16(s[2 * n2 + 1], qa[k], f[2], f[3]);
                    }
                }
            }
            float bm[2] = {-CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
            for (int n = 0; n < WP_K / 8; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t key = key0 + 8 * n + 2 * t4 + (i & 1), qp = qpos[i >> 1];
                    const uint32_t dist = qp - key;                          // wraps to a huge value for keys after the query
                    float v = s[n][i] * a.scale;
                    if (bias) v -= r1 * __logf(fmaf(r2, static_cast<float>(dist), 1.0f));
                    v = dist < a.window ? v : -CUDART_INF_F;
                    s[n][i] = v;
                    bm[i >> 1] = fmaxf(bm[i >> 1], v);
                }
            float nm[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                bm[u] = fmaxf(bm[u], __shfl_xor_sync(0xffffffffu, bm[u], 1));
                bm[u] = fmaxf(bm[u], __shfl_xor_sync(0xffffffffu, bm[u], 2));
                const float top = fmaxf(mx[u], bm[u]);
                nm[u] = top == -CUDART_INF_F ? 0.f : top;                    // nothing visible yet: every weight is exp(-inf) = 0
                const float corr = __expf(mx[u] - nm[u]);
                l[u] *= corr;
                mx[u] = top;
#pragma unroll
                for (int i = 0; i < DV / 8; ++i) { o[i][2 * u] *= corr; o[i][2 * u + 1] *= corr; }
            }
#pragma unroll
            for (int n = 0; n < WP_K / 8; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    s[n][i] = __expf(s[n][i] - nm[i >> 1]);
                    l[i >> 1] += s[n][i];                                    // this lane's share; summed over the four lanes at the end
                }
#pragma unroll
            for (int k = 0; k < WP_K / 16; ++k) {
                uint32_t pa[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) pa[i] = pack_bf16(s[2 * k + (i >> 1)][2 * (i & 1)], s[2 * k + (i >> 1)][2 * (i & 1) + 1]);
#pragma unroll
                for (int n2 = 0; n2 < DV / 16; ++n2) {
                    if (n2 < static_cast<int>(nv)) {
                        uint32_t f[4];
                        ldmatrix4_trans(f, vs + ((16 * k + ((lane >> 3) & 1) * 8 + (lane & 7)) * VP + 16 * n2 + (lane >> 4) * 8) * 2);
                        mma_bf16(o[2 * n2], pa, f[0], f[1]);
                        mma_bf16(o[2 * n2 + 1], pa, f[2], f[3]);
                    }
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        l[u] += __shfl_xor_sync(0xffffffffu, l[u], 1);
        l[u] += __shfl_xor_sync(0xffffffffu, l[u], 2);
        if (row[u] >= m) continue;
        const float inv = 1.0f / l[u];
        OUT* dst = out + static_cast<size_t>(row[u]) * ldo + h * a.vdim;
        const float* gr = gate ? gate + static_cast<size_t>(row[u]) * ldg + h * a.vdim : nullptr;
#pragma unroll
        for (int n = 0; n < DV / 8; ++n)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t d = 8 * n + 2 * t4 + i;
                if (d < a.vdim) {
                    float v = o[n][2 * u + i] * inv;
                    if (gr) v *= sigmoidf(gr[d]);
                    dst[d] = from_f32<OUT>(v);
                }
            }
        if (h == a.heads - 1)
            for (uint32_t i = a.heads * a.vdim + t4; i < ldo; i += 4) out[static_cast<size_t>(row[u]) * ldo + i] = from_f32<OUT>(0.f);
    }
}

// ---------------------------------------------------------------- host side
bool window_ok(const hf2q_window_attn* a) {
    return a && a->qkv && a->k_cache && a->v_cache && a->pos && a->heads && a->kv_heads && a->heads % a->kv_heads == 0 && a->dim && a->dim <= 256 &&
           a->vdim && a->vdim <= 256 && a->window && a->capacity >= a->window && (a->r1 == nullptr) == (a->r2 == nullptr) &&
           (a->cache_dtype == HF2Q_DT_F32 || a->cache_dtype == HF2Q_DT_BF16) && reinterpret_cast<uintptr_t>(a->k_cache) % 16 == 0 &&
           reinterpret_cast<uintptr_t>(a->v_cache) % 16 == 0 && !a->linear && !a->shared_dim;
}
// what the prefill takes beyond that: plain rows, a shared part of the keys
bool window_rows_ok(const hf2q_window_attn* a) {
    if (!a || !a->linear) return window_ok(a);
    hf2q_window_attn b = *a;
    b.qkv = b.qkv ? b.qkv : static_cast<const float*>(a->k_cache);           // the queries come apart
    b.linear = b.shared_dim = 0;
    const bool shared = a->shared_dim == 0 || (a->k_shared && a->shared_capacity && a->shared_stride % 8 == 0 && a->shared_stride >= pad8(a->shared_dim) &&
                                               reinterpret_cast<uintptr_t>(a->k_shared) % 16 == 0 && pad8(a->dim) + pad8(a->shared_dim) <= QK_MAX);
    return window_ok(&b) && shared && (!a->linear || (a->row_stride % 8 == 0 && a->k_head_stride % 8 == 0 && a->v_head_stride % 8 == 0));
}
uint32_t decode_gr(const hf2q_window_attn& a) {
    const uint32_t rep = a.heads / a.kv_heads;
    return rep >= 5 ? 8 : rep >= 3 ? 4 : rep;
}
uint32_t decode_groups(const hf2q_window_attn& a) { const uint32_t gr = decode_gr(a); return (a.heads / a.kv_heads + gr - 1) / gr; }
// Splits of a window.  A CTA has an SM to itself and takes WD_PASS keys a pass, so the CTAs of all splits are one wave: eight splits a
// group of heads, whatever the number of groups, ran in several (bf16 heads of 128, us at 256 / 2048 keys of a window of 2048,
// eight splits and now: 32 heads of keys and values 15.0 / 23.5 and 5.5 / 13.6, 64 24.7 / 39.4 and 6.1 / 20.4, 128 45.4 / 71.1 and
// 6.5 / 32.1; 4 shared by 16 heads 8.8 / 12.1 as before).
// Merged through memory: whole passes, for with twice the CTAs and half a pass each a second wave waits with idle warps (window 16384, us at
// 256 / 8192 / 16384 keys, before and now: 16 heads of keys and values 16.2 / 35.6 / 55.2 and 7.9 / 22.7 / 35.2, 8 shared by 32
// 23.2 / 30.2 / 44.8 and 13.3 / 24.2 / 36.6, 4 by 16 26.4 / 29.3 / 34.2 and 16.0 / 19.3 / 26.5; 1 by 8 32.8 / 35.2 / 37.7 as before).
uint32_t decode_splits(const hf2q_window_attn& a, int sms) {
    const uint32_t ctas = a.kv_heads * decode_groups(a), by_sm = static_cast<uint32_t>(sms) / ctas, by_keys = (a.window + WD_PASS - 1) / WD_PASS;
    const uint32_t s = by_sm < by_keys ? by_sm : by_keys;
    return s < 1 ? 1 : s > 64 ? 64 : s;
}
size_t counter_bytes(const hf2q_window_attn& a) { return (static_cast<size_t>(a.kv_heads) * decode_groups(a) * 4 + 255) & ~static_cast<size_t>(255); }

// Splits as one cluster, 0 for windows of more than four passes for each of eight: up to there the cluster, which adds through shared
// memory, is ahead at short fills and at most level at full ones with as many CTAs again that merge through memory (us at 256 / 8192 keys of
// a window of 8192: 1 head of keys and values shared by 8 13.4 / 50.6, 16 splits through memory 19.0 / 34.3; 4 by 16 8.9 / 30.9 and 11.7 / 22.1;
// 10 heads 5.4 / 19.0 and 9.0 / 20.4).  One wave: clusters do not span the chip's groups of SMs, and with one CTA an SM those of more
// than four leave up to a quarter of it unused, smaller ones an eighth (16 heads, window 2048, 256 keys: clusters of 6 5.3 us, of 7 9.7).
uint32_t cluster_splits(const hf2q_window_attn& a, int sms) {
    const uint32_t ctas = a.kv_heads * decode_groups(a), n = static_cast<uint32_t>(sms), by_keys = (a.window + WD_PASS - 1) / WD_PASS;
    if (by_keys > 4 * WD_CLUSTER) return 0;
    uint32_t s = by_keys < WD_CLUSTER ? by_keys : WD_CLUSTER;
    while (s > 1 && ctas * s > (s > 4 ? n * 3 / 4 : n * 7 / 8)) --s;
    return s;
}
template <typename T, int GR, int NC>
cudaError_t launch_decode(const hf2q_window_attn& a, float* out, uint8_t* scratch, int sms, cudaStream_t st) {
    const size_t smem = (static_cast<size_t>(GR) * pad8(a.dim) + WD_WARPS * GR * (2 + WD_KEYS + pad8(a.vdim)) + GR * wd_part(a.vdim)) * sizeof(float);
    const uint32_t groups = decode_groups(a), cluster = cluster_splits(a, sms);
    uint32_t* counters = reinterpret_cast<uint32_t*>(scratch);
    float* part = reinterpret_cast<float*>(scratch + counter_bytes(a));
    if (cluster) {
        static PerDeviceFlag flag;
        const auto kern = window_decode_kernel<T, GR, NC, true>;
        if (const cudaError_t e = ensure_max_dynamic_smem(kern, 200 * 1024, flag); e != cudaSuccess) return e;
        return launch_pdl_cluster(kern, dim3(a.kv_heads * groups, cluster), dim3(WD_WARPS * 32), dim3(1, cluster, 1), smem, st, a, groups, out, counters, part);
    }
    static PerDeviceFlag flag;
    const auto kern = window_decode_kernel<T, GR, NC, false>;
    if (const cudaError_t e = ensure_max_dynamic_smem(kern, 200 * 1024, flag); e != cudaSuccess) return e;
    return launch_pdl(kern, dim3(a.kv_heads * groups, decode_splits(a, sms)), dim3(WD_WARPS * 32), smem, st, a, groups, out, counters, part);
}
template <typename T, int GR>
cudaError_t launch_decode_nc(const hf2q_window_attn& a, float* out, uint8_t* scratch, int sms, cudaStream_t st) {
    if (a.vdim <= 128) return launch_decode<T, GR, 1>(a, out, scratch, sms, st);
    return launch_decode<T, GR, 2>(a, out, scratch, sms, st);
}
template <typename T>
cudaError_t launch_decode_gr(const hf2q_window_attn& a, float* out, uint8_t* scratch, int sms, cudaStream_t st) {
    switch (decode_gr(a)) {
        case 1: return launch_decode_nc<T, 1>(a, out, scratch, sms, st);
        case 2: return launch_decode_nc<T, 2>(a, out, scratch, sms, st);
        case 4: return launch_decode_nc<T, 4>(a, out, scratch, sms, st);
        default: return launch_decode_nc<T, 8>(a, out, scratch, sms, st);
    }
}
template <typename T, typename OUT, bool PLAIN>
cudaError_t launch_prefill_f32(const hf2q_window_attn& a, uint32_t m, const void* q, const float* gate, uint32_t ldg, void* out, uint32_t ldo, cudaStream_t st) {
    const dim3 grid((m + 7) / 8, a.heads);
    const T* qt = static_cast<const T*>(q);
    OUT* o = static_cast<OUT*>(out);
    if (a.vdim <= 64) return launch_pdl(window_prefill_f32_kernel<T, OUT, 1, PLAIN>, grid, dim3(256), 0, st, a, m, qt, gate, ldg, o, ldo);
    if (a.vdim <= 128) return launch_pdl(window_prefill_f32_kernel<T, OUT, 2, PLAIN>, grid, dim3(256), 0, st, a, m, qt, gate, ldg, o, ldo);
    return launch_pdl(window_prefill_f32_kernel<T, OUT, 4, PLAIN>, grid, dim3(256), 0, st, a, m, qt, gate, ldg, o, ldo);
}
template <int DK, int DV, typename OUT, bool PLAIN>
cudaError_t launch_prefill_dm(const hf2q_window_attn& a, uint32_t m, const void* q, const float* gate, uint32_t ldg, void* out, uint32_t ldo, cudaStream_t st) {
    static PerDeviceFlag flag;
    const size_t smem = 2ull * WP_K * (DK + 8 + DV + 8) * 2;
    if (const cudaError_t e = ensure_max_dynamic_smem(window_prefill_mma_kernel<DK, DV, OUT, PLAIN>, static_cast<int>(smem), flag); e != cudaSuccess) return e;
    return launch_pdl(window_prefill_mma_kernel<DK, DV, OUT, PLAIN>, dim3((m + WP_Q - 1) / WP_Q, a.heads), dim3(WP_WARPS * 32), smem, st, a, m,
                      static_cast<const __nv_bfloat16*>(q), gate, ldg, static_cast<OUT*>(out), ldo);
}
template <int DK, typename OUT, bool PLAIN>
cudaError_t launch_prefill_tc(const hf2q_window_attn& a, uint32_t m, const void* q, const float* gate, uint32_t ldg, void* out, uint32_t ldo, uint32_t* status,
                              cudaStream_t st) {
    static PerDeviceFlag flag;
    constexpr uint32_t smem = wt_smem(DK);
    if (const cudaError_t e = ensure_max_dynamic_smem(window_prefill_tc_kernel<DK, OUT, PLAIN>, static_cast<int>(smem), flag); e != cudaSuccess) return e;
    return launch_pdl(window_prefill_tc_kernel<DK, OUT, PLAIN>, dim3((m + WT_Q - 1) / WT_Q, a.heads), dim3(WT_THREADS), smem, st, a, m,
                      static_cast<const __nv_bfloat16*>(q), gate, ldg, static_cast<OUT*>(out), ldo, status);
}
// Keys of 65..128 (or values of 65..128 beside shorter keys), in tiles of 64 queries on warps or of 128 on tcgen05?  While the
// tiles leave SMs idle both are bound by the latency of a block of 64 keys, 3.5 us on tcgen05 and, by the size of a key and a
// value, 3.6 to 4.6 on warps, and tcgen05 pays 2 us more at the start and walks the longer tile; once two of the smaller tiles
// stand on every SM it is the amount of work.  us, warps / tcgen05, with keys before the portion:
//   128 + 128 elements, 16 heads, 256 queries: window 256 26.6 / 29.9, window 512 44.7 / 43.8, window 2048 153 / 128
//                                2048 queries: window 64 30.5 / 24.7, window 2048 358 / 157
//   96 + 64 elements, 16 heads, 256 queries: window 512 36.8 / 43.8, window 2048 125 / 130
//                               1024 queries: window 256 30.4 / 33.7, window 512 50.9 / 49.9;  2048: window 256 50.2 / 37.1
// Rows with a shared key part cost the warps more (64 + 32 and 64 elements, window 2048: 127 / 99 with 64 queries).
bool prefill_on_tcgen05(const hf2q_window_attn& a, uint32_t m, int sms) {
    const uint64_t tiles = static_cast<uint64_t>((m + WP_Q - 1) / WP_Q) * a.heads;
    const uint32_t k = pad8(a.dim) + pad8(a.shared_dim);
    if (a.linear && a.shared_dim) return a.window > 256 || tiles > 2ull * sms;
    if (k + pad8(a.vdim) >= 224) return a.window > 256 || (a.window >= 64 && tiles > 2ull * sms);
    return (a.window >= 512 && tiles > static_cast<uint64_t>(sms)) || (a.window >= 256 && tiles > 2ull * sms);
}
template <typename OUT>
cudaError_t launch_prefill_bf16(const hf2q_window_attn& a, uint32_t m, const void* q, const float* gate, uint32_t ldg, void* out, uint32_t ldo, uint32_t* status,
                                int sms, cudaStream_t st) {
    const uint32_t k = pad8(a.dim) + pad8(a.shared_dim), v = a.vdim;
    const bool tc = prefill_on_tcgen05(a, m, sms);
    if (a.linear) {
        if (k <= 64 && v <= 64) return launch_prefill_dm<64, 64, OUT, true>(a, m, q, gate, ldg, out, ldo, st);
        if (k <= 128 && v <= 128) {
            if (tc) return launch_prefill_tc<128, OUT, true>(a, m, q, gate, ldg, out, ldo, status, st);
            return launch_prefill_dm<128, 128, OUT, true>(a, m, q, gate, ldg, out, ldo, st);
        }
        // 192: on warps a block of 64 keys takes 7 us, so tcgen05 from the second block on (one block: 8.2 / 7.7)
        if (k <= 192 && v <= 128) return launch_prefill_tc<192, OUT, true>(a, m, q, gate, ldg, out, ldo, status, st);
        return launch_prefill_dm<QK_MAX, 256, OUT, true>(a, m, q, gate, ldg, out, ldo, st);
    }
    if (k <= 64 && v <= 64) return launch_prefill_dm<64, 64, OUT, false>(a, m, q, gate, ldg, out, ldo, st);
    if (k <= 128 && v <= 128) {
        if (tc) return launch_prefill_tc<128, OUT, false>(a, m, q, gate, ldg, out, ldo, status, st);
        return launch_prefill_dm<128, 128, OUT, false>(a, m, q, gate, ldg, out, ldo, st);
    }
    return launch_prefill_dm<256, 256, OUT, false>(a, m, q, gate, ldg, out, ldo, st);
}

}  // namespace
}  // namespace hf2q

using namespace hf2q;
using namespace hf2q::seq;

extern "C" {

HF2Q_API int32_t hf2q_cuda_window_attn_scratch_bytes(hf2q_ctx* ctx, const hf2q_window_attn* a, uint64_t* out) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!a || !out || a->kv_heads == 0 || a->heads == 0 || a->heads % a->kv_heads || a->window == 0)
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "window_attn_scratch_bytes: bad sizes");
    *out = counter_bytes(*a) + static_cast<uint64_t>(a->kv_heads) * decode_groups(*a) * decode_splits(*a, ctx_sm_count(ctx)) * decode_gr(*a) * wd_part(a->vdim) * 4;
    return HF2Q_OK;
}

HF2Q_API int32_t hf2q_cuda_window_attn_decode(hf2q_ctx* ctx, void* stream, const hf2q_window_attn* a, float* out, void* scratch, uint64_t scratch_bytes) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    uint64_t need = 0;
    if (!window_ok(a) || !out || !scratch || hf2q_cuda_window_attn_scratch_bytes(ctx, a, &need) != HF2Q_OK)
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "window_attn_decode: null pointer or an unsupported size");
    if (scratch_bytes < need) return ctx_fail(ctx, HF2Q_ERR_WORKSPACE, "window_attn_decode: scratch too small");
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int sms = ctx_sm_count(ctx);
    const cudaError_t e = a->cache_dtype == HF2Q_DT_F32 ? launch_decode_gr<float>(*a, out, static_cast<uint8_t*>(scratch), sms, st)
                                                        : launch_decode_gr<__nv_bfloat16>(*a, out, static_cast<uint8_t*>(scratch), sms, st);
    return ctx_cuda_result(ctx, e, "window_attn_decode", 1);
}

HF2Q_API int32_t hf2q_cuda_window_attn_append(hf2q_ctx* ctx, void* stream, const hf2q_window_attn* a, uint32_t m, void* q_out) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!window_ok(a) || !q_out || a->window - 1 + static_cast<uint64_t>(m) > a->capacity)
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "window_attn_append: null pointer, an unsupported size or more tokens than the ring holds");
    if (m == 0) return HF2Q_OK;
    const uint64_t warps = static_cast<uint64_t>(m) * (a->heads + 2 * a->kv_heads);
    const dim3 grid(static_cast<unsigned>((warps + 7) / 8));
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const cudaError_t e = a->cache_dtype == HF2Q_DT_F32 ? launch_pdl(window_append_kernel<float>, grid, dim3(256), 0, st, *a, m, static_cast<float*>(q_out))
                                                        : launch_pdl(window_append_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, *a, m, static_cast<__nv_bfloat16*>(q_out));
    return ctx_cuda_result(ctx, e, "window_attn_append", 1);
}

HF2Q_API int32_t hf2q_cuda_window_attn_prefill(hf2q_ctx* ctx, void* stream, const hf2q_window_attn* a, uint32_t m, const void* q, const float* gate,
                                               uint32_t ldg, void* out, uint32_t out_dtype, uint32_t ldo) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!window_rows_ok(a) || !q || !out || ldo < a->heads * a->vdim || a->window - 1 + static_cast<uint64_t>(m) > a->capacity)
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "window_attn_prefill: null pointer, an unsupported size or more tokens than the ring holds");
    if (m == 0) return HF2Q_OK;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaErrorInvalidValue;
    if (a->cache_dtype == HF2Q_DT_F32) {
        if (out_dtype == HF2Q_DT_F32)
            e = a->linear ? launch_prefill_f32<float, float, true>(*a, m, q, gate, ldg, out, ldo, st) : launch_prefill_f32<float, float, false>(*a, m, q, gate, ldg, out, ldo, st);
    } else if (out_dtype == HF2Q_DT_BF16) {
        e = launch_prefill_bf16<__nv_bfloat16>(*a, m, q, gate, ldg, out, ldo, ctx_status_word(ctx), ctx_sm_count(ctx), st);
    } else if (out_dtype == HF2Q_DT_F32) {
        e = launch_prefill_bf16<float>(*a, m, q, gate, ldg, out, ldo, ctx_status_word(ctx), ctx_sm_count(ctx), st);
    }
    return ctx_cuda_result(ctx, e, "window_attn_prefill", 1);
}

}  // extern "C"
