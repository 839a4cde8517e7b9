// Recurrent mixers with a matrix state per head, token after token in 32-bit arithmetic:
//
//   mlstm   exponential input / forget gates with a running maximum (matrix memory of xLSTM)
//   delta   gated delta rule, one decay per head and key channel
//   ssd     scalar decay per head and token (Mamba-2)
//
// All keep S[key channel][value column] and treat a value column independently, so the state lives in registers:
// sixteen lanes share a column (each holds key channels 32 c + 2 l and + 1), and sums over the key channels are shuffles.
// The state in memory is [head][column][key channel, padded to 32] (f32), which makes a lane's channels consecutive.
//
// Prompt portions (the scans): a group of sixteen lanes carries C columns.  What a token costs a warp is the k, q (and g)
// words that each lane reads from shared memory -- the register file takes one 32-lane word per clock and SM, whether or
// not lanes read the same one -- so several columns share them; a column alone (two a warp, eight warps an SM) spent 260
// to 300 of its 490 to 570 clocks a token there.  One warp of the CTA only fetches: it stages the next batch of tokens by
// asynchronous copies (and makes the gate factors) while the others work through this one, with one barrier per batch.
// Portions of 2048 tokens: mlstm (8 heads of 128 x 128) 509 -> 217 us with two columns a group (one: 256 us), delta (16 of
// 128 x 128) 594 -> 314 us with two (346 us one token at a time), ssd (64 of 128 x 64) 547 -> 268 us with two in eight warps
// (280 us with four in four).  What bounds them now is the issue of a token's multiply-adds, two clocks for each pair.
#include <math_constants.h>

#include "seq_common.cuh"

namespace hf2q {
namespace {
using namespace seq;

constexpr int SC_WARPS = 8, SC_COLS = 16, SC_THREADS = SC_WARPS * 32;       // one-token kernels: a group to a column
constexpr int SC_TB = 32, SC_FEW = 8;                                       // scans: tokens of a batch, and of one of a short portion

__device__ __forceinline__ float group_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v;
}
// Sums of K values over the sixteen lanes of a group, transposed: lane l ends with the sum of v[l % K].
template <int K>
__device__ __forceinline__ float group_transpose_sum(float (&v)[K], uint32_t l) {
#pragma unroll
    for (int w = K / 2; w > 0; w >>= 1) {
        const bool up = l & w;
#pragma unroll
        for (int i = 0; i < w; ++i) {
            const float other = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + w], w);
            v[i] = (up ? v[i + w] : v[i]) + other;
        }
    }
#pragma unroll
    for (int w = K; w < 16; w *= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], w);
    return v[0];
}
// rows of `count` floats -> shared memory, asynchronously, by one warp; 16 bytes at a time where both sides allow it
__device__ __forceinline__ void stage_rows(float* dst, uint32_t dst_ld, const float* src, size_t src_ld, uint32_t rows, uint32_t count) {
    const uint32_t lane = threadIdx.x & 31;
    if (count % 4 == 0 && src_ld % 4 == 0 && dst_ld % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
        if (count <= 64) {                                   // several short rows at once
            const uint32_t per = count <= 8 ? 2 : count <= 16 ? 4 : count <= 32 ? 8 : 16, c = 4 * (lane % per);
            if (c < count)
                for (uint32_t r = lane / per; r < rows; r += 32 / per) cp_async16(dst + r * dst_ld + c, src + r * src_ld + c);
        } else {
            for (uint32_t c = 4 * lane; c < count; c += 128)
#pragma unroll 4
                for (uint32_t r = 0; r < rows; ++r) cp_async16(dst + r * dst_ld + c, src + r * src_ld + c);
        }
    } else {
        for (uint32_t c = lane; c < count; c += 32)
#pragma unroll 4
            for (uint32_t r = 0; r < rows; ++r) cp_async4(dst + r * dst_ld + c, src + r * src_ld + c);
    }
}
template <int C>
__device__ __forceinline__ void load_values(float (&v)[C], const float* p) {
    if constexpr (C == 4) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else if constexpr (C == 2) {
        const float2 x = *reinterpret_cast<const float2*>(p);
        v[0] = x.x; v[1] = x.y;
    } else {
        v[0] = *p;
    }
}

template <int RQ> struct Vec {                       // a lane's RQ pairs of key channels
    f2 v[RQ];
    __device__ __forceinline__ void load(const float* p) {
#pragma unroll
        for (int c = 0; c < RQ; ++c) v[c] = *reinterpret_cast<const f2*>(p + 32 * c);
    }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int c = 0; c < RQ; ++c) v[c] = 0ull;
    }
    __device__ __forceinline__ void store(float* p) const {
#pragma unroll
        for (int c = 0; c < RQ; ++c) *reinterpret_cast<f2*>(p + 32 * c) = v[c];
    }
    // sum over this lane's channels, in two interleaved pairs of partial sums
    __device__ __forceinline__ float dot(const Vec& k) const {
        f2 s[2] = {f2_mul(v[0], k.v[0]), 0ull};
#pragma unroll
        for (int c = 1; c < RQ; ++c) s[c & 1] = f2_fma(v[c], k.v[c], s[c & 1]);
        return f2_sum(RQ > 1 ? f2_add(s[0], s[1]) : s[0]);
    }
    __device__ __forceinline__ Vec operator*(const Vec& k) const {
        Vec r;
#pragma unroll
        for (int c = 0; c < RQ; ++c) r.v[c] = f2_mul(v[c], k.v[c]);
        return r;
    }
    __device__ __forceinline__ void scale(const Vec& k) {
#pragma unroll
        for (int c = 0; c < RQ; ++c) v[c] = f2_mul(v[c], k.v[c]);
    }
    __device__ __forceinline__ void axpy(const Vec& k, float a) {
        const f2 aa = f2_both(a);
#pragma unroll
        for (int c = 0; c < RQ; ++c) v[c] = f2_fma(k.v[c], aa, v[c]);
    }
    __device__ __forceinline__ void decay_axpy(float keep, const Vec& k, float a) {
        const f2 kk = f2_both(keep), aa = f2_both(a);
#pragma unroll
        for (int c = 0; c < RQ; ++c) v[c] = f2_fma(kk, v[c], f2_mul(k.v[c], aa));
    }
};

// Where a thread of a scan stands: W working warps of two groups with C columns each, then the fetching warp.
template <int RQ, int C, int W>
struct ScanPlace {
    static constexpr uint32_t DP = 32 * RQ, COLS = 2 * C * W, GROUP = 16 / C;        // GROUP: tokens whose sums fill a group's lanes
    uint32_t warp, lane, lg, group, col0, col, n_cols;
    bool fetches;
    __device__ __forceinline__ ScanPlace(uint32_t slice, uint32_t vdim) {
        warp = threadIdx.x >> 5;
        lane = threadIdx.x & 31;
        lg = lane & 15;
        group = warp * 2 + (lane >> 4);
        col0 = slice * COLS;
        col = col0 + group * C;                              // the group's first column
        n_cols = min(COLS, vdim - col0);
        fetches = warp == W;
    }
};
// Batches of TB tokens in two buffers: stage(t0, buffer) by the fetching warp, batch(t0, buffer, tokens) by the others.
template <uint32_t TB, typename Stage, typename Batch>
__device__ __forceinline__ void scan_batches(bool fetches, uint32_t m, Stage stage, Batch batch) {
    if (fetches) { stage(0u, 0u); cp_async_wait<0>(); }
    __syncthreads();
    for (uint32_t t0 = 0, b = 0; t0 < m; t0 += TB, b ^= 1) {
        if (fetches) {
            if (t0 + TB < m) { stage(t0 + TB, b ^ 1); cp_async_wait<0>(); }
        } else {
            batch(t0, b, min(TB, m - t0));
        }
        __syncthreads();
    }
}
// The whole groups of a batch's n tokens: form(j0, sums) makes a lane's partial sums, done(j0, sums) adds them up and stores.
// A group's sums are finished beside the next group's tokens, whose arithmetic hides the shuffles.  Returns the tokens taken.
template <typename Sums, uint32_t GROUP, uint32_t TB, typename Form, typename Done>
__device__ __forceinline__ uint32_t scan_groups(uint32_t n, Form form, Done done) {
    if (TB < GROUP || n < GROUP) return 0;
    Sums last;
    form(0u, last);
    uint32_t j0 = GROUP;
    for (; j0 + GROUP <= n; j0 += GROUP) {
        Sums now;
        form(j0, now);
        done(j0 - GROUP, last);
        last = now;
    }
    done(j0 - GROUP, last);
    return j0;
}
// channels past `dim` stay zero in shared memory, so the padded part of the state stays zero too
__device__ __forceinline__ void clear_padding(float* sm, uint32_t n, bool padded) {
    if (!padded) return;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) sm[i] = 0.f;
    __syncthreads();
}
// Shared memory of a scan's launch.  It asks for so much that no SM takes more CTAs than an even spread puts there: the CTAs
// start while the preceding kernel's last ones still run, and would otherwise pile up on the SMs that are free first.  The price:
// scans of two streams do not share SMs.  Two of 2048 tokens side by side: delta (16 heads) 512 us a pair, one alone 299; ssd (64
// heads) 443 and 256; mlstm (8 heads, both fit) 213 and 213.  (The former kernels shared SMs and took 1087, 869 and 586 a pair.)
constexpr size_t SCAN_STATIC = 9 * 1024, SCAN_MAX = 227 * 1024 - SCAN_STATIC;       // static arrays: at most
inline size_t scan_smem(size_t need, dim3 grid, int sms) {
    const size_t ctas = static_cast<size_t>(grid.x) * grid.y, per_sm = (ctas + sms - 1) / sms;
    const size_t even = 228 * 1024 / per_sm, claim = even > SCAN_STATIC + 1024 ? even - SCAN_STATIC - 1024 : 0;
    return claim > need ? claim : need;
}

// ---------------------------------------------------------------- mLSTM
// A CTA carries the 16 columns that share a normaliser and a maximum.
template <int RQ, int C, uint32_t TB>
__global__ void __launch_bounds__((8 / C + 1) * 32, TB == SC_TB ? 1 : 2) mlstm_kernel(const __grid_constant__ hf2q_mlstm a, uint32_t m, float* __restrict__ out) {
    constexpr uint32_t W = 8 / C;
    using Place = ScanPlace<RQ, C, W>;
    constexpr uint32_t DP = Place::DP;
    extern __shared__ __align__(16) float dsm[];                    // k, q: [2][TB][DP] each
    float* ks = dsm;
    float* qs = dsm + 2 * TB * DP;
    __shared__ __align__(16) float vs[2][TB][SC_COLS];
    __shared__ __align__(8) float2 gs[2][TB];                    // keep, write
    __shared__ float ge[2][TB];                                  // exp(-maximum)
    pdl_trigger();
    pdl_wait();
    const uint32_t h = blockIdx.x, slice = blockIdx.y, n_slices = gridDim.y;
    const Place at(slice, a.vdim);
    const float q_scale = 1.0f / sqrtf(static_cast<float>(a.dim));
    float* mp = a.mx + static_cast<size_t>(h) * n_slices + slice;
    float mx = *mp;                                          // carried by the fetching warp
    clear_padding(dsm, 4 * TB * DP, a.dim < DP);
    auto stage = [&](uint32_t t0, uint32_t b) {
        const uint32_t n = min(TB, m - t0), lane = at.lane;
        const float* row = a.proj + static_cast<size_t>(t0) * a.ld;
        stage_rows(ks + b * TB * DP, DP, row + a.k_off + h * a.dim, a.ld, n, a.dim);
        stage_rows(qs + b * TB * DP, DP, row + a.q_off + h * a.dim, a.ld, n, a.dim);
        stage_rows(vs[b][0], SC_COLS, row + a.v_off + h * a.vdim + at.col0, a.ld, n, at.n_cols);
        cp_async_commit();
        // gate factors of the batch (lane = token): the running maximum is a max-plus scan over the pairs (f, i),
        // m_t = max(m + f_1 + .. + f_t, max_s (i_s + f_(s+1) + .. + f_t))
        float f = 0.f, x = -CUDART_INF_F;
        if (lane < n) {
            const float* g = row + static_cast<size_t>(lane) * a.ld + h;
            x = a.gate_cap * tanhf((g[a.i_off] + a.i_bias[h]) / a.gate_cap);
            f = -softplusf(-a.gate_cap * tanhf((g[a.f_off] + a.f_bias[h]) / a.gate_cap));
        }
        const float f_own = f, x_own = x;
#pragma unroll
        for (int d = 1; d < TB; d *= 2) {
            const float fo = __shfl_up_sync(0xffffffffu, f, d), xo = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) { x = fmaxf(xo + f, x); f += fo; }
        }
        const float m_t = fmaxf(mx + f, x);
        float before = __shfl_up_sync(0xffffffffu, m_t, 1);
        if (lane == 0) before = mx;
        if (lane < n) {
            gs[b][lane] = make_float2(expf(f_own + before - m_t), expf(x_own - m_t));
            ge[b][lane] = expf(-m_t);
        }
        mx = __shfl_sync(0xffffffffu, m_t, n - 1);
    };
    Vec<RQ> S[C], N;
    float* sp = a.s + (static_cast<size_t>(h) * a.vdim + at.col) * DP + 2 * at.lg;
    float* np = a.n + (static_cast<size_t>(h) * n_slices + slice) * DP + 2 * at.lg;
    if (!at.fetches) {
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (at.col + c < a.vdim) S[c].load(sp + c * DP); else S[c].zero();
        N.load(np);
    }
    scan_batches<TB>(at.fetches, m, stage, [&](uint32_t t0, uint32_t b, uint32_t n) {
        // a token's operands are read one token ahead of their use
        struct Operands { Vec<RQ> k, q; float2 g; float v[C]; };
        auto fetch = [&](uint32_t j) {
            Operands t;
            t.k.load(ks + (b * TB + j) * DP + 2 * at.lg);
            t.q.load(qs + (b * TB + j) * DP + 2 * at.lg);
            t.g = gs[b][j];
            load_values(t.v, &vs[b][j][at.group * C]);
            return t;
        };
        auto token = [&](const Operands& t, float* num, float& den) {      // this lane's part of the sums
#pragma unroll
            for (int c = 0; c < C; ++c) {
                S[c].decay_axpy(t.g.x, t.k, t.g.y * t.v[c]);
                num[c] = S[c].dot(t.q);
            }
            N.decay_axpy(t.g.x, t.k, t.g.y);
            den = N.dot(t.q);
        };
        auto finish = [&](uint32_t j, uint32_t col, float num, float den) {
            if (col < a.vdim)
                out[static_cast<size_t>(t0 + j) * a.heads * a.vdim + static_cast<size_t>(h) * a.vdim + col] = num * q_scale / (fmaxf(fabsf(den * q_scale), ge[b][j]) + 1e-6f);
        };
        struct Sums { float num[16], den[Place::GROUP]; };
        uint32_t j0 = scan_groups<Sums, Place::GROUP, TB>(
            n,
            [&](uint32_t j, Sums& r) {
                Operands t = fetch(j);
#pragma unroll
                for (uint32_t u = 0; u < Place::GROUP; ++u) {
                    const Operands next = fetch(j + (u + 1 < Place::GROUP ? u + 1 : u));
                    token(t, r.num + u * C, r.den[u]);
                    t = next;
                }
            },
            [&](uint32_t j, Sums& r) {                           // lane i of a group finishes token i / C, column i % C
                const float x = group_transpose_sum(r.num, at.lg), y = group_transpose_sum(r.den, at.lg);
                finish(j + at.lg / C, at.col + at.lg % C, x, C == 1 ? y : __shfl_sync(0xffffffffu, y, (at.lane & 16) + at.lg / C));
            });
        for (; j0 < n; ++j0) {
            float num[C], den;
            token(fetch(j0), num, den);
            den = group_sum(den);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const float x = group_sum(num[c]);
                if (at.lg == c) finish(j0, at.col + c, x, den);
            }
        }
    });
    if (!at.fetches) {
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (at.col + c < a.vdim) S[c].store(sp + c * DP);
        if (at.warp == 0 && at.lane < 16) N.store(np);
    } else if (at.lane == 0) {
        *mp = mx;
    }
}

// One token: nothing is staged, each lane brings its own channels and every thread makes the gate factors for itself, so that the
// loads are one latency and no barrier stands in the chain.  8 heads of 128 x 128 1.95 us (a scan of one token 2.8, the kernel
// before the scans of several columns 2.7), 32 heads 2.7 (3.1; 3.0), 16 heads of 256 x 256 2.7 (3.8; 3.9).
template <int RQ>
__global__ void __launch_bounds__(SC_THREADS) mlstm_step_kernel(const __grid_constant__ hf2q_mlstm a, float* __restrict__ out) {
    constexpr uint32_t DP = 32 * RQ;
    pdl_trigger();
    pdl_wait();
    const uint32_t h = blockIdx.x, slice = blockIdx.y, n_slices = gridDim.y, lane = threadIdx.x & 31, lg = lane & 15;
    const uint32_t col = slice * SC_COLS + (threadIdx.x >> 4);
    const bool live = col < a.vdim;
    Vec<RQ> S, N, k, q;
    float* sp = a.s + (static_cast<size_t>(h) * a.vdim + (live ? col : 0)) * DP + 2 * lg;
    float* np = a.n + (static_cast<size_t>(h) * n_slices + slice) * DP + 2 * lg;
    float* mp = a.mx + static_cast<size_t>(h) * n_slices + slice;
    if (live) S.load(sp); else S.zero();
    N.load(np);
    const float *kr = a.proj + a.k_off + h * a.dim, *qr = a.proj + a.q_off + h * a.dim;
#pragma unroll
    for (int c = 0; c < RQ; ++c) {
        const uint32_t i = 32 * c + 2 * lg;
        const bool in0 = i < a.dim, in1 = i + 1 < a.dim;
        k.v[c] = f2_of(in0 ? kr[i] : 0.f, in1 ? kr[i + 1] : 0.f);
        q.v[c] = f2_of(in0 ? qr[i] : 0.f, in1 ? qr[i + 1] : 0.f);
    }
    const float v = live ? a.proj[a.v_off + h * a.vdim + col] : 0.f, mx = *mp;
    const float x = a.gate_cap * tanhf((a.proj[a.i_off + h] + a.i_bias[h]) / a.gate_cap);
    const float f = -softplusf(-a.gate_cap * tanhf((a.proj[a.f_off + h] + a.f_bias[h]) / a.gate_cap));
    const float top = fmaxf(mx + f, x), keep = expf(f + mx - top), write = expf(x - top);
    S.decay_axpy(keep, k, write * v);
    N.decay_axpy(keep, k, write);
    const float num = group_sum(S.dot(q)), den = group_sum(N.dot(q)), q_scale = 1.0f / sqrtf(static_cast<float>(a.dim));
    if (live) {
        S.store(sp);
        if (lg == 0) out[h * a.vdim + col] = num * q_scale / (fmaxf(fabsf(den * q_scale), expf(-top)) + 1e-6f);
    }
    __syncthreads();                                         // all threads have read the normaliser and the maximum
    if (threadIdx.x < 16) N.store(np);
    if (threadIdx.x == 0) *mp = top;
}

// ---------------------------------------------------------------- gated delta rule
// S <- g S;  u = beta (v - S^T k);  S <- S + k u;  o = S^T q
template <int RQ>
struct DeltaOperands {
    Vec<RQ> g, k, q;
    float v, beta;
};
template <int RQ>
__device__ __forceinline__ float delta_token(Vec<RQ>& S, const DeltaOperands<RQ>& t) {          // this lane's part of o
    S.scale(t.g);
    const float u = t.beta * (t.v - group_sum(S.dot(t.k)));
    S.axpy(t.k, u);
    return S.dot(t.q);
}

template <int RQ, int C, int W, uint32_t TB, int PER_SM>
__global__ void __launch_bounds__((W + 1) * 32, PER_SM) delta_scan_kernel(const __grid_constant__ hf2q_delta a, uint32_t m, const float* qkv,
                                                                  const float* beta, const float* g, float* __restrict__ out) {
    using Place = ScanPlace<RQ, C, W>;
    constexpr uint32_t DP = Place::DP;
    extern __shared__ __align__(16) float dsm[];                    // k, q, g: [2][TB][DP] each
    float* ks = dsm;
    float* qs = dsm + 2 * TB * DP;
    float* gs = dsm + 4 * TB * DP;
    __shared__ __align__(16) float vs[2][TB][Place::COLS];
    __shared__ float bs[2][TB];
    pdl_trigger();
    pdl_wait();
    const uint32_t h = blockIdx.x, kvh = h / (a.heads / a.kv_heads);
    const Place at(blockIdx.y, a.vdim);
    const uint32_t qk = a.kv_heads * a.dim, ld = 2 * qk + a.heads * a.vdim;
    clear_padding(dsm, 6 * TB * DP, a.dim < DP);
    auto stage = [&](uint32_t t0, uint32_t b) {
        const uint32_t n = min(TB, m - t0);
        const float* row = qkv + static_cast<size_t>(t0) * ld;
        stage_rows(qs + b * TB * DP, DP, row + kvh * a.dim, ld, n, a.dim);
        stage_rows(ks + b * TB * DP, DP, row + qk + kvh * a.dim, ld, n, a.dim);
        stage_rows(vs[b][0], Place::COLS, row + 2 * qk + h * a.vdim + at.col0, ld, n, at.n_cols);
        stage_rows(gs + b * TB * DP, DP, g + (static_cast<size_t>(t0) * a.heads + h) * a.dim, static_cast<size_t>(a.heads) * a.dim, n, a.dim);
        if (at.lane < n) cp_async4(&bs[b][at.lane], beta + static_cast<size_t>(t0 + at.lane) * a.heads + h);
        cp_async_commit();
    };
    Vec<RQ> S[C];
    float* sp = a.s + (static_cast<size_t>(h) * a.vdim + at.col) * DP + 2 * at.lg;
    if (!at.fetches) {
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (at.col + c < a.vdim) S[c].load(sp + c * DP); else S[c].zero();
    }
    scan_batches<TB>(at.fetches, m, stage, [&](uint32_t t0, uint32_t b, uint32_t n) {
        struct Operands { Vec<RQ> g, k, q; float v[C], beta; };
        auto fetch = [&](uint32_t j) {                       // read one step ahead of their use
            const uint32_t o = (b * TB + j) * DP + 2 * at.lg;
            Operands t;
            t.g.load(gs + o);
            t.k.load(ks + o);
            t.q.load(qs + o);
            load_values(t.v, &vs[b][j][at.group * C]);
            t.beta = bs[b][j];
            return t;
        };
        auto token = [&](const Operands& t, float* r) {      // this lane's part of o
#pragma unroll
            for (int c = 0; c < C; ++c) {
                S[c].scale(t.g);
                S[c].axpy(t.k, t.beta * (t.v[c] - group_sum(S[c].dot(t.k))));
                r[c] = S[c].dot(t.q);
            }
        };
        // Two tokens at a time: what the second one reads off the state is taken from the state before the first,
        //   S1^T (g2 k2) = S0^T (g1 g2 k2) + (k1 . g2 k2) u1,
        // so that one chain of shuffles serves both.
        auto pair = [&](const Operands& t1, const Operands& t2, float* r) {
            const Vec<RQ> gk = t1.g * t1.k, g2k = t2.g * t2.k, ggk = t1.g * g2k, gq = t1.g * t1.q, gg = t1.g * t2.g, kg = t1.k * t2.g;
            float d[2 * C + 1];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                d[2 * c] = S[c].dot(gk);
                d[2 * c + 1] = S[c].dot(ggk);
            }
            d[2 * C] = t1.k.dot(g2k);
            const float kq = t1.k.dot(t1.q);
#pragma unroll
            for (int w = 1; w < 16; w *= 2)
#pragma unroll
                for (int i = 0; i < 2 * C + 1; ++i) d[i] += __shfl_xor_sync(0xffffffffu, d[i], w);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const float u1 = t1.beta * (t1.v[c] - d[2 * c]), u2 = t2.beta * (t2.v[c] - fmaf(d[2 * C], u1, d[2 * c + 1]));
                r[c] = fmaf(kq, u1, S[c].dot(gq));
                S[c].scale(gg);
                S[c].axpy(kg, u1);
                S[c].axpy(t2.k, u2);
                r[C + c] = S[c].dot(t2.q);
            }
        };
        float* dst = out + static_cast<size_t>(t0) * a.heads * a.vdim + static_cast<size_t>(h) * a.vdim;
        const size_t row_o = static_cast<size_t>(a.heads) * a.vdim;
        struct Sums { float r[16]; };
        uint32_t j0 = scan_groups<Sums, Place::GROUP, TB>(
            n,
            [&](uint32_t j, Sums& s) {
                Operands t1 = fetch(j), t2 = fetch(j + 1);
#pragma unroll
                for (uint32_t u = 0; u < Place::GROUP; u += 2) {
                    const Operands n1 = fetch(j + (u + 2 < Place::GROUP ? u + 2 : u)), n2 = fetch(j + (u + 3 < Place::GROUP ? u + 3 : u));
                    pair(t1, t2, s.r + u * C);
                    t1 = n1;
                    t2 = n2;
                }
            },
            [&](uint32_t j, Sums& s) {                           // lane i of a group stores token i / C, column i % C
                const float x = group_transpose_sum(s.r, at.lg);
                const uint32_t col = at.col + at.lg % C;
                if (col < a.vdim) dst[(j + at.lg / C) * row_o + col] = x;
            });
        for (; j0 < n; ++j0) {
            float r[C];
            token(fetch(j0), r);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const float x = group_sum(r[c]);
                if (at.lg == c && at.col + c < a.vdim) dst[j0 * row_o + at.col + c] = x;
            }
        }
    });
    if (!at.fetches) {
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (at.col + c < a.vdim) S[c].store(sp + c * DP);
    }
}

// convolution + SiLU of channel `ch` (0 .. 2 qk + heads vdim) for one token; before(j): the input j tokens back
template <typename Before>
__device__ __forceinline__ float conv_silu(const float* w, uint32_t taps, float now, Before before) {
    float s = now * w[taps - 1];
    for (uint32_t j = 1; j < taps; ++j) s = fmaf(before(j), w[taps - 1 - j], s);
    return siluf(s);
}
__device__ __forceinline__ float decay_of(float a_log, float x) { return expf(-expf(a_log) * softplusf(x)); }
// The same for four taps from a channel's ring and its weights, both asked for before the position is known.
__device__ __forceinline__ float ring_at(const float4& r, uint32_t i) { return (i & 2) ? ((i & 1) ? r.w : r.z) : ((i & 1) ? r.y : r.x); }
__device__ __forceinline__ float conv4(const float4& w, const float4& ring, float now, uint32_t pos, float s0) {
    float s = fmaf(now, w.w, s0);
    s = fmaf(ring_at(ring, pos + 3), w.z, s);
    s = fmaf(ring_at(ring, pos + 2), w.y, s);
    return fmaf(ring_at(ring, pos + 1), w.x, s);
}

// Rows of a low-rank product, 16 lanes to a row: w holds the first 128 elements of N rows, fetch(c, w) brings those from c on.
// Every lane of the group gets the sums.
template <int N, typename F>
__device__ __forceinline__ void low_rank_dots(uint4 (&w)[N], uint32_t ld, const float* x, F fetch, float (&s)[N]) {
#pragma unroll
    for (int r = 0; r < N; ++r) s[r] = 0.f;
    for (uint32_t c = 0;;) {
        const uint32_t e = c + 8 * (threadIdx.x & 15);
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (e < ld) { a = *reinterpret_cast<const float4*>(x + e); b = *reinterpret_cast<const float4*>(x + e + 4); }
#pragma unroll
        for (int r = 0; r < N; ++r) {
            s[r] = fmaf(bf_lo(w[r].x), a.x, s[r]); s[r] = fmaf(bf_hi(w[r].x), a.y, s[r]); s[r] = fmaf(bf_lo(w[r].y), a.z, s[r]); s[r] = fmaf(bf_hi(w[r].y), a.w, s[r]);
            s[r] = fmaf(bf_lo(w[r].z), b.x, s[r]); s[r] = fmaf(bf_hi(w[r].z), b.y, s[r]); s[r] = fmaf(bf_lo(w[r].w), b.z, s[r]); s[r] = fmaf(bf_hi(w[r].w), b.w, s[r]);
        }
        if ((c += 128) >= ld) break;
        fetch(c, w);
    }
#pragma unroll
    for (int r = 0; r < N; ++r) s[r] = group_sum(s[r]);
}

// One token from the raw projection row: convolution, SiLU, unit norms, decays, gate and the state update.
// Bound by latency: one load behind another.  The rows of the low-rank products and the taps' weights are asked for before the wait,
// everything else right behind it; a row of a2 per thread, 16 bytes at a time, and rings read behind the position took most of a
// launch (16 heads of 128 x 128, rank 128: 10.2 -> 4.4 us a launch of many, 64 heads of rank 64 9.3 -> 8.8).
template <int RQ>
__global__ void __launch_bounds__(SC_THREADS, RQ <= 4 ? 2 : 1) delta_step_kernel(const __grid_constant__ hf2q_delta a, float* __restrict__ out, float* __restrict__ gate) {
    constexpr uint32_t DP = 32 * RQ, ROWS = DP / SC_COLS, ITEMS = (2 * DP + SC_COLS + SC_THREADS - 1) / SC_THREADS;
    __shared__ __align__(16) float xs[2 * DP + SC_COLS], gs[DP];    // q, k, v; decays
    __shared__ float red[64];
    extern __shared__ __align__(16) float lr[];                     // a1 [a_rank_ld], g1 [g_rank_ld]
    pdl_trigger();
    const uint32_t h = blockIdx.x, slice = blockIdx.y, rep = a.heads / a.kv_heads, kvh = h / rep, qk = a.kv_heads * a.dim;
    const uint32_t lg = threadIdx.x & 15, col_s = threadIdx.x >> 4, col0 = slice * SC_COLS, col = col0 + col_s;
    const uint32_t n_cols = min(static_cast<uint32_t>(SC_COLS), a.vdim - col0);
    const bool live = col < a.vdim;
    // decays: rows col_s + SC_COLS r of the head; the gate: the group's own column
    uint4 wa[ROWS], wg[1];
    auto fetch_a = [&](uint32_t c, uint4 (&w)[ROWS]) {
        const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(a.a2) + (static_cast<size_t>(h) * a.dim + col_s) * a.a_rank_ld + c + 8 * lg;
#pragma unroll
        for (uint32_t r = 0; r < ROWS; ++r)
            w[r] = col_s + SC_COLS * r < a.dim && c + 8 * lg < a.a_rank_ld ? *reinterpret_cast<const uint4*>(src + static_cast<size_t>(SC_COLS) * r * a.a_rank_ld) : make_uint4(0, 0, 0, 0);
    };
    auto fetch_g = [&](uint32_t c, uint4 (&w)[1]) {
        w[0] = live && c + 8 * lg < a.g_rank_ld
                   ? *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.g2) + (static_cast<size_t>(h) * a.vdim + col) * a.g_rank_ld + c + 8 * lg)
                   : make_uint4(0, 0, 0, 0);
    };
    fetch_a(0, wa);
    fetch_g(0, wg);
    // channel of an item: q, k, then the slice's v
    struct Channel { uint32_t ring, at; const float* w; bool in, keep; };
    auto channel = [&](uint32_t i) {
        const uint32_t j = i < DP ? i : i < 2 * DP ? i - DP : i - 2 * DP;
        if (i < 2 * DP) {
            const uint32_t c = kvh * a.dim + j;
            return Channel{i < DP ? c : qk + c, (i < DP ? a.q_off : a.k_off) + c, (i < DP ? a.q_conv : a.k_conv) + static_cast<size_t>(c) * a.taps, j < a.dim, slice == 0 && h % rep == 0};
        }
        const uint32_t c = h * a.vdim + col0 + j;
        return Channel{2 * qk + c, a.v_off + c, a.v_conv + static_cast<size_t>(c) * a.taps, j < n_cols, true};
    };
    const bool four = a.taps == 4 && ((reinterpret_cast<uintptr_t>(a.conv_state) | reinterpret_cast<uintptr_t>(a.q_conv) | reinterpret_cast<uintptr_t>(a.k_conv) |
                                       reinterpret_cast<uintptr_t>(a.v_conv)) & 15) == 0;
    float4 taps[ITEMS], ring[ITEMS];
    float now[ITEMS];
    if (four) {
#pragma unroll
        for (uint32_t n = 0; n < ITEMS; ++n) {
            const Channel c = channel(threadIdx.x + SC_THREADS * n);
            if (c.in) taps[n] = *reinterpret_cast<const float4*>(c.w);
        }
    }
    const uint32_t row = col_s + SC_COLS * lg;                      // whose decay this lane makes
    const bool decays = lg < ROWS && row < a.dim;
    const float bias = decays ? a.dt_bias[h * a.dim + row] : 0.f, a_log = a.a_log[h];
    pdl_wait();
    Vec<RQ> S;
    float* sp = a.s + (static_cast<size_t>(h) * a.vdim + (live ? col : 0)) * DP + 2 * lg;
    if (live) S.load(sp); else S.zero();
    const uint32_t pos = *a.pos;
    const float b = a.proj[a.b_off + h];
    for (uint32_t i = threadIdx.x; i < a.a_rank_ld; i += SC_THREADS) lr[i] = a.proj[a.a1_off + i];
    for (uint32_t i = threadIdx.x; i < a.g_rank_ld; i += SC_THREADS) lr[a.a_rank_ld + i] = a.proj[a.g1_off + i];
    // the state ring has one column more than the taps look back, so this token's column is read by nobody
#pragma unroll
    for (uint32_t n = 0; n < ITEMS; ++n) {
        const Channel c = channel(threadIdx.x + SC_THREADS * n);
        if (!c.in) continue;
        now[n] = a.proj[c.at];
        if (four) ring[n] = *reinterpret_cast<const float4*>(a.conv_state + static_cast<size_t>(c.ring) * 4);
    }
    float ss[2] = {0.f, 0.f};
#pragma unroll
    for (uint32_t n = 0; n < ITEMS; ++n) {
        const uint32_t i = threadIdx.x + SC_THREADS * n;
        const Channel c = channel(i);
        float v = 0.f;
        if (c.in) {
            float* st = a.conv_state + static_cast<size_t>(c.ring) * a.taps;
            v = four ? siluf(conv4(taps[n], ring[n], now[n], pos, 0.f)) : conv_silu(c.w, a.taps, now[n], [&](uint32_t j) { return st[(pos + a.taps - j) % a.taps]; });
            if (c.keep) st[pos % a.taps] = now[n];
        }
        if (i < 2 * DP + SC_COLS) xs[i] = v;
        if (i < 2 * DP) ss[i < DP ? 0 : 1] += v * v;
    }
    block_sum(ss, red);                                             // (its barrier also publishes lr and xs)
    float s[ROWS], sg[1];
    low_rank_dots(wa, a.a_rank_ld, lr, fetch_a, s);
    low_rank_dots(wg, a.g_rank_ld, lr + a.a_rank_ld, fetch_g, sg);
    float mine = 0.f;
#pragma unroll
    for (uint32_t r = 0; r < ROWS; ++r) mine = lg == r ? s[r] : mine;
    if (lg < ROWS) gs[row] = decays ? decay_of(a_log, mine + bias) : 0.f;
    if (live && lg == 0) gate[h * a.vdim + col] = sg[0];
    const float iq = 1.0f / sqrtf(ss[0] + 1e-6f) / sqrtf(static_cast<float>(a.dim)), ik = 1.0f / sqrtf(ss[1] + 1e-6f);
    for (uint32_t i = threadIdx.x; i < 2 * DP; i += SC_THREADS) xs[i] *= i < DP ? iq : ik;
    __syncthreads();
    DeltaOperands<RQ> t;
    t.g.load(gs + 2 * lg);
    t.k.load(xs + DP + 2 * lg);
    t.q.load(xs + 2 * lg);
    t.v = xs[2 * DP + col_s];
    t.beta = sigmoidf(b);
    const float r = group_sum(delta_token<RQ>(S, t));
    if (live) {
        S.store(sp);
        if (lg == 0) out[h * a.vdim + col] = r;
    }
}

// Tokens of a CTA of the four-tap kernels (`columns` CTAs to a run of tokens): 16, so that inputs and weights are read once and
// not four times through L2 (8 with wide heads, a lane of which has eight channels), or as few as put PREP_CTAS on every SM, for
// a CTA is a chain of its tokens.  delta, 8 + 8 + 16 heads of 128: 64 tokens 17.1 us a token a CTA, 20.6 at 16, 3.5 as here; 2048
// tokens 56.9, 41.0 and 41.0.  2 CTAs an SM: 4.6 at 64 tokens; 8: the same to 15 % slower at 128.  ssd, 64 heads of 128 x 64:
// 2048 tokens 57.8 us a token a CTA, 28.0 as here.
constexpr uint32_t PREP_CTAS = 4;
inline uint32_t prep_tokens(uint32_t m, uint32_t columns, int sms, bool wide = false) {
    uint32_t per = wide ? 8 : 16;
    while (per > 1 && static_cast<uint64_t>((m + per - 1) / per) * columns < static_cast<uint64_t>(PREP_CTAS) * sms) per /= 2;
    return per;
}
// f(t, x[t * ld]) for t = 0 .. n, the inputs of U tokens on their way together (a load behind each store would be a chain)
template <uint32_t U, typename F>
__device__ __forceinline__ void for_inputs(const float* x, size_t ld, uint32_t n, F f) {
    for (uint32_t t0 = 0; t0 < n; t0 += U) {
        float now[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u)
            if (t0 + u < n) now[u] = x[(t0 + u) * ld];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u)
            if (t0 + u < n) f(t0 + u, now[u]);
    }
}
// A channel's running window over the four taps of its convolution: the last three inputs and the weights in registers.
struct FourTaps {
    float w0, w1, w2, w3, x1, x2, x3;
    // x: the channel's input at the first token, `t0` tokens into the portion, rows ld apart; st: its ring of earlier inputs
    __device__ __forceinline__ void start(const float* w, const float* x, size_t ld, const float* st, uint32_t pos, uint32_t t0) {
        w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3];
        auto before = [&](uint32_t k) { return k <= t0 ? *(x - k * ld) : st[(pos + t0 + 4 - k) % 4]; };
        x1 = before(1), x2 = before(2), x3 = before(3);
    }
    __device__ __forceinline__ float next(float now, float first) {      // first: the newest tap's product (and bias)
        const float s = fmaf(x3, w0, fmaf(x2, w1, fmaf(x1, w2, first)));
        x3 = x2, x2 = x1, x1 = now;
        return siluf(s);
    }
};
// Four taps, `per` tokens a CTA.  Columns of CTAs: heads of q and k (a warp each, NJ channels a lane), channels of v (a thread
// each), then the gates and low-rank rows.
template <int NJ, typename LR>
__global__ void __launch_bounds__(256) delta_prep4_kernel(const __grid_constant__ hf2q_delta a, uint32_t m, uint32_t per, uint32_t qk_columns, float* __restrict__ qkv,
                                                          float* __restrict__ beta, LR* __restrict__ a1, LR* __restrict__ g1) {
    pdl_trigger();
    pdl_wait();
    const uint32_t t0 = blockIdx.x * per, n = min(per, m - t0), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t pos = *a.pos, qk = a.kv_heads * a.dim;
    const size_t ld = a.ld, ld_o = 2 * qk + a.heads * a.vdim;
    const float* rows = a.proj + t0 * ld;
    float* dst = qkv + t0 * ld_o;
    if (blockIdx.y < qk_columns) {
        const uint32_t hd = blockIdx.y * 8 + warp;
        if (hd >= 2 * a.kv_heads) return;
        const bool is_k = hd >= a.kv_heads;
        const uint32_t c0 = (is_k ? hd - a.kv_heads : hd) * a.dim;
        const float *w = is_k ? a.k_conv : a.q_conv, *x = rows + (is_k ? a.k_off : a.q_off) + c0;
        FourTaps tap[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const uint32_t i = lane + 32 * j;
            if (i < a.dim) tap[j].start(w + static_cast<size_t>(c0 + i) * 4, x + i, ld, a.conv_state + static_cast<size_t>((is_k ? qk : 0u) + c0 + i) * 4, pos, t0);
        }
        float* to = dst + (is_k ? qk : 0u) + c0;
        constexpr uint32_t U = NJ == 4 ? 4 : 2;                      // tokens whose inputs are on their way together
        for (uint32_t t1 = 0; t1 < n; t1 += U) {
            float now[U][NJ];
#pragma unroll
            for (uint32_t u = 0; u < U; ++u)
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    if (t1 + u < n && lane + 32 * j < a.dim) now[u][j] = x[(t1 + u) * ld + lane + 32 * j];
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t t = t1 + u;
                if (t >= n) break;
                float v[NJ], s = 0.f;
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    v[j] = lane + 32 * j < a.dim ? tap[j].next(now[u][j], now[u][j] * tap[j].w3) : 0.f;
                    s += v[j] * v[j];
                }
                float inv = 1.0f / sqrtf(warp_sum(s) + 1e-6f);
                if (!is_k) inv /= sqrtf(static_cast<float>(a.dim));
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    if (lane + 32 * j < a.dim) to[t * ld_o + lane + 32 * j] = v[j] * inv;
            }
        }
    } else if (blockIdx.y + 1 < gridDim.y) {
        const uint32_t c = (blockIdx.y - qk_columns) * 256 + threadIdx.x;
        if (c >= a.heads * a.vdim) return;
        const float* x = rows + a.v_off + c;
        FourTaps tap;
        tap.start(a.v_conv + static_cast<size_t>(c) * 4, x, ld, a.conv_state + static_cast<size_t>(2 * qk + c) * 4, pos, t0);
        for_inputs<8>(x, ld, n, [&](uint32_t t, float now) { dst[t * ld_o + 2 * qk + c] = tap.next(now, now * tap.w3); });
    } else {
        for (uint32_t t = 0; t < n; ++t) {
            const float* row = rows + t * ld;
            for (uint32_t h = threadIdx.x; h < a.heads; h += 256) beta[static_cast<size_t>(t0 + t) * a.heads + h] = sigmoidf(row[a.b_off + h]);
            for (uint32_t c = threadIdx.x; c < a.a_rank_ld; c += 256) a1[static_cast<size_t>(t0 + t) * a.a_rank_ld + c] = from_f32<LR>(row[a.a1_off + c]);
            for (uint32_t c = threadIdx.x; c < a.g_rank_ld; c += 256) g1[static_cast<size_t>(t0 + t) * a.g_rank_ld + c] = from_f32<LR>(row[a.g1_off + c]);
        }
    }
}

// One CTA per token: a warp takes one head of q or k (or a head of v) at a time.
template <typename LR>
__global__ void __launch_bounds__(256) delta_prep_kernel(const __grid_constant__ hf2q_delta a, float* __restrict__ qkv, float* __restrict__ beta,
                                                         LR* __restrict__ a1, LR* __restrict__ g1) {
    pdl_trigger();
    pdl_wait();
    const uint32_t t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t pos = *a.pos, qk = a.kv_heads * a.dim;
    const float* row = a.proj + static_cast<size_t>(t) * a.ld;
    float* dst = qkv + static_cast<size_t>(t) * (2 * qk + a.heads * a.vdim);
    auto channel = [&](uint32_t ch, const float* w, uint32_t off) {
        return conv_silu(w, a.taps, row[off], [&](uint32_t j) {
            return j <= t ? row[static_cast<ptrdiff_t>(off) - static_cast<ptrdiff_t>(j) * a.ld]
                          : a.conv_state[static_cast<size_t>(ch) * a.taps + (pos + t + a.taps - j) % a.taps];
        });
    };
    for (uint32_t hd = warp; hd < 2 * a.kv_heads; hd += 8) {
        const bool is_k = hd >= a.kv_heads;
        const uint32_t c0 = (is_k ? hd - a.kv_heads : hd) * a.dim;
        const float* w = is_k ? a.k_conv : a.q_conv;
        float v[8], s = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t i = lane + 32 * j;
            v[j] = i < a.dim ? channel((is_k ? qk : 0u) + c0 + i, w + static_cast<size_t>(c0 + i) * a.taps, (is_k ? a.k_off : a.q_off) + c0 + i) : 0.f;
            s += v[j] * v[j];
        }
        float inv = 1.0f / sqrtf(warp_sum(s) + 1e-6f);
        if (!is_k) inv /= sqrtf(static_cast<float>(a.dim));
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (lane + 32 * j < a.dim) dst[(is_k ? qk : 0u) + c0 + lane + 32 * j] = v[j] * inv;
    }
    for (uint32_t c = threadIdx.x; c < a.heads * a.vdim; c += 256)
        dst[2 * qk + c] = channel(2 * qk + c, a.v_conv + static_cast<size_t>(c) * a.taps, a.v_off + c);
    for (uint32_t h = threadIdx.x; h < a.heads; h += 256) beta[static_cast<size_t>(t) * a.heads + h] = sigmoidf(row[a.b_off + h]);
    for (uint32_t c = threadIdx.x; c < a.a_rank_ld; c += 256) a1[static_cast<size_t>(t) * a.a_rank_ld + c] = from_f32<LR>(row[a.a1_off + c]);
    for (uint32_t c = threadIdx.x; c < a.g_rank_ld; c += 256) g1[static_cast<size_t>(t) * a.g_rank_ld + c] = from_f32<LR>(row[a.g1_off + c]);
}

__global__ void __launch_bounds__(256) delta_decay_kernel(const float* a_log, const float* dt_bias, uint32_t dim, uint32_t per_token,
                                                          uint64_t n, float* __restrict__ g) {
    pdl_trigger();
    pdl_wait();
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint32_t c = static_cast<uint32_t>(i % per_token);
        g[i] = decay_of(a_log[c / dim], g[i] + dt_bias[c]);
    }
}

// ---------------------------------------------------------------- state space with a scalar decay
__device__ __forceinline__ uint32_t ssd_channels(const hf2q_ssd& a) { return a.heads * a.vdim + 2 * a.groups * a.state; }

// S <- keep S + dt B x^T;  y = S^T C + d x
template <int RQ, int C, int W, uint32_t TB>
__global__ void __launch_bounds__((W + 1) * 32, TB == SC_TB ? 1 : RQ <= 4 ? 4 : 2) ssd_scan_kernel(const __grid_constant__ hf2q_ssd a, uint32_t m, const float* xbc,
                                                                const float* dt, const float* la, float* __restrict__ y) {
    using Place = ScanPlace<RQ, C, W>;
    constexpr uint32_t DP = Place::DP;
    extern __shared__ __align__(16) float dsm[];                    // B, C: [2][TB][DP] each
    float* ks = dsm;
    float* qs = dsm + 2 * TB * DP;
    __shared__ __align__(16) float vs[2][TB][Place::COLS];
    __shared__ __align__(8) float2 gs[2][TB];                    // decay, step size
    pdl_trigger();
    pdl_wait();
    const uint32_t h = blockIdx.x, grp = h / (a.heads / a.groups);
    const Place at(blockIdx.y, a.vdim);
    const uint32_t channels = ssd_channels(a), inner = a.heads * a.vdim;
    // the convolution's reader has finished: the last inputs go to the state
    for (uint32_t i = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; i < channels; i += gridDim.x * gridDim.y * blockDim.x) {
        const uint32_t pos = *a.pos, keep = min(a.taps - 1, m);
        for (uint32_t j = 0; j < keep; ++j)
            a.conv_state[static_cast<size_t>(i) * a.taps + (pos + m - 1 - j) % a.taps] = a.proj[static_cast<size_t>(m - 1 - j) * a.ld + a.off + i];
    }
    clear_padding(dsm, 4 * TB * DP, a.state < DP);
    auto stage = [&](uint32_t t0, uint32_t b) {
        const uint32_t n = min(TB, m - t0);
        const float* row = xbc + static_cast<size_t>(t0) * channels;
        stage_rows(ks + b * TB * DP, DP, row + inner + grp * a.state, channels, n, a.state);
        stage_rows(qs + b * TB * DP, DP, row + inner + (a.groups + grp) * a.state, channels, n, a.state);
        stage_rows(vs[b][0], Place::COLS, row + h * a.vdim + at.col0, channels, n, at.n_cols);
        cp_async_commit();
        if (at.lane < n) {
            const size_t o = static_cast<size_t>(t0 + at.lane) * a.heads + h;
            gs[b][at.lane] = make_float2(expf(la[o]), dt[o]);
        }
    };
    Vec<RQ> S[C];
    float* sp = a.s + (static_cast<size_t>(h) * a.vdim + at.col) * DP + 2 * at.lg;
    const float skip = a.d[h];
    if (!at.fetches) {
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (at.col + c < a.vdim) S[c].load(sp + c * DP); else S[c].zero();
    }
    scan_batches<TB>(at.fetches, m, stage, [&](uint32_t t0, uint32_t b, uint32_t n) {
        struct Operands { Vec<RQ> k, q; float2 g; float v[C]; };
        auto fetch = [&](uint32_t j) {                       // read one token ahead of their use
            Operands t;
            t.k.load(ks + (b * TB + j) * DP + 2 * at.lg);
            t.q.load(qs + (b * TB + j) * DP + 2 * at.lg);
            t.g = gs[b][j];
            load_values(t.v, &vs[b][j][at.group * C]);
            return t;
        };
        auto token = [&](const Operands& t, float* r) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                S[c].decay_axpy(t.g.x, t.k, t.g.y * t.v[c]);
                r[c] = S[c].dot(t.q);
            }
        };
        auto finish = [&](uint32_t j, uint32_t c, float s) {     // column c of the group
            if (at.col + c < a.vdim) y[static_cast<size_t>(t0 + j) * inner + static_cast<size_t>(h) * a.vdim + at.col + c] = s + skip * vs[b][j][at.group * C + c];
        };
        struct Sums { float r[16]; };
        uint32_t j0 = scan_groups<Sums, Place::GROUP, TB>(
            n,
            [&](uint32_t j, Sums& s) {
                Operands t = fetch(j);
#pragma unroll
                for (uint32_t u = 0; u < Place::GROUP; ++u) {
                    const Operands next = fetch(j + (u + 1 < Place::GROUP ? u + 1 : u));
                    token(t, s.r + u * C);
                    t = next;
                }
            },
            [&](uint32_t j, Sums& s) { finish(j + at.lg / C, at.lg % C, group_transpose_sum(s.r, at.lg)); });    // lane i: token i / C, column i % C
        for (; j0 < n; ++j0) {
            float r[C];
            token(fetch(j0), r);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const float x = group_sum(r[c]);
                if (at.lg == c) finish(j0, c, x);
            }
        }
    });
    if (!at.fetches) {
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (at.col + c < a.vdim) S[c].store(sp + c * DP);
    }
}

__device__ __forceinline__ void ssd_gates(const hf2q_ssd& a, uint32_t h, float raw, float& dt, float& la) {
    dt = softplusf(raw + a.dt_bias[h]);
    la = -expf(a.a_log[h]) * dt;
}
template <typename Before>
__device__ __forceinline__ float conv_bias_silu(const float* w, float bias, uint32_t taps, float now, Before before) {
    float s = fmaf(now, w[taps - 1], bias);
    for (uint32_t j = 1; j < taps; ++j) s = fmaf(before(j), w[taps - 1 - j], s);
    return siluf(s);
}

// Four taps: a thread takes one channel over `per` tokens, with its taps and the last three inputs in registers (a token a CTA read
// every input and weight four times through L2).  Bound by memory; the last CTA column makes the gates.
__global__ void __launch_bounds__(256) ssd_prep4_kernel(const __grid_constant__ hf2q_ssd a, uint32_t m, uint32_t per, float* __restrict__ xbc, float* __restrict__ dt, float* __restrict__ la) {
    pdl_trigger();
    pdl_wait();
    const uint32_t t0 = blockIdx.x * per, n = min(per, m - t0), pos = *a.pos, channels = ssd_channels(a);
    const float* row = a.proj + static_cast<size_t>(t0) * a.ld + a.off;
    if (blockIdx.y + 1 == gridDim.y) {
        for (uint32_t i = threadIdx.x; i < n * a.heads; i += 256) {
            const uint32_t t = i / a.heads, h = i % a.heads;
            const size_t o = static_cast<size_t>(t0 + t) * a.heads + h;
            ssd_gates(a, h, row[static_cast<size_t>(t) * a.ld + channels + h], dt[o], la[o]);
        }
        return;
    }
    const uint32_t c = blockIdx.y * 256 + threadIdx.x;
    if (c >= channels) return;
    const float* x = row + c;
    FourTaps tap;
    tap.start(a.conv + static_cast<size_t>(c) * 4, x, a.ld, a.conv_state + static_cast<size_t>(c) * 4, pos, t0);
    const float bias = a.conv_bias[c];
    float* dst = xbc + static_cast<size_t>(t0) * channels + c;
    for_inputs<8>(x, a.ld, n, [&](uint32_t t, float now) { dst[static_cast<size_t>(t) * channels] = tap.next(now, fmaf(now, tap.w3, bias)); });
}

// One CTA per token.
__global__ void __launch_bounds__(256) ssd_prep_kernel(const __grid_constant__ hf2q_ssd a, float* __restrict__ xbc, float* __restrict__ dt, float* __restrict__ la) {
    pdl_trigger();
    pdl_wait();
    const uint32_t t = blockIdx.x, pos = *a.pos, channels = ssd_channels(a);
    const float* row = a.proj + static_cast<size_t>(t) * a.ld + a.off;
    float* dst = xbc + static_cast<size_t>(t) * channels;
    for (uint32_t c = threadIdx.x; c < channels; c += 256)
        dst[c] = conv_bias_silu(a.conv + static_cast<size_t>(c) * a.taps, a.conv_bias[c], a.taps, row[c], [&](uint32_t j) {
            return j <= t ? row[static_cast<ptrdiff_t>(c) - static_cast<ptrdiff_t>(j) * a.ld] : a.conv_state[static_cast<size_t>(c) * a.taps + (pos + t + a.taps - j) % a.taps];
        });
    for (uint32_t h = threadIdx.x; h < a.heads; h += 256) {
        const size_t o = static_cast<size_t>(t) * a.heads + h;
        ssd_gates(a, h, row[channels + h], dt[o], la[o]);
    }
}

// One token from the raw projection row: convolution, SiLU, step size and the state update.  Bound by latency: with four taps rings,
// weights and inputs of all channels are asked for at once, the weights before the wait (64 heads of 128 x 64: 4.7 -> 2.3 us a launch of many).
template <int RQ>
__global__ void __launch_bounds__(SC_THREADS, 2) ssd_step_kernel(const __grid_constant__ hf2q_ssd a, float* __restrict__ y) {
    constexpr uint32_t DP = 32 * RQ, ITEMS = (2 * DP + SC_COLS + SC_THREADS - 1) / SC_THREADS;
    __shared__ __align__(16) float xs[2 * DP + SC_COLS];            // k, q, v
    pdl_trigger();
    const uint32_t h = blockIdx.x, slice = blockIdx.y, rep = a.heads / a.groups, grp = h / rep;
    const uint32_t lg = threadIdx.x & 15, col_s = threadIdx.x >> 4, col0 = slice * SC_COLS, col = col0 + col_s;
    const uint32_t n_cols = min(static_cast<uint32_t>(SC_COLS), a.vdim - col0), channels = ssd_channels(a), inner = a.heads * a.vdim;
    const bool live = col < a.vdim, first = slice == 0 && h % rep == 0;
    struct Channel { uint32_t c; bool in, keep; };
    auto channel = [&](uint32_t i) {
        const uint32_t j = i < DP ? i : i < 2 * DP ? i - DP : i - 2 * DP;
        if (i < 2 * DP) return Channel{inner + (i < DP ? grp : a.groups + grp) * a.state + j, j < a.state, first};
        return Channel{h * a.vdim + col0 + j, j < n_cols, true};
    };
    const bool four = a.taps == 4 && ((reinterpret_cast<uintptr_t>(a.conv_state) | reinterpret_cast<uintptr_t>(a.conv)) & 15) == 0;
    float4 taps[ITEMS], ring[ITEMS];
    float now[ITEMS], bias[ITEMS];
#pragma unroll
    for (uint32_t n = 0; n < ITEMS; ++n) {
        const Channel c = channel(threadIdx.x + SC_THREADS * n);
        if (!c.in) continue;
        bias[n] = a.conv_bias[c.c];
        if (four) taps[n] = *reinterpret_cast<const float4*>(a.conv + static_cast<size_t>(c.c) * 4);
    }
    const float skip = a.d[h];
    pdl_wait();
    Vec<RQ> S;
    float* sp = a.s + (static_cast<size_t>(h) * a.vdim + (live ? col : 0)) * DP + 2 * lg;
    if (live) S.load(sp); else S.zero();
    const uint32_t pos = *a.pos;
    const float* row = a.proj + a.off;
    float dt, la;
    ssd_gates(a, h, row[channels + h], dt, la);
#pragma unroll
    for (uint32_t n = 0; n < ITEMS; ++n) {
        const Channel c = channel(threadIdx.x + SC_THREADS * n);
        if (!c.in) continue;
        now[n] = row[c.c];
        if (four) ring[n] = *reinterpret_cast<const float4*>(a.conv_state + static_cast<size_t>(c.c) * 4);
    }
    // the state ring has one column more than the taps look back, so this token's column is read by nobody
#pragma unroll
    for (uint32_t n = 0; n < ITEMS; ++n) {
        const uint32_t i = threadIdx.x + SC_THREADS * n;
        const Channel c = channel(i);
        float v = 0.f;
        if (c.in) {
            float* st = a.conv_state + static_cast<size_t>(c.c) * a.taps;
            v = four ? siluf(conv4(taps[n], ring[n], now[n], pos, bias[n]))
                     : conv_bias_silu(a.conv + static_cast<size_t>(c.c) * a.taps, bias[n], a.taps, now[n], [&](uint32_t j) { return st[(pos + a.taps - j) % a.taps]; });
            if (c.keep) st[pos % a.taps] = now[n];
        }
        if (i < 2 * DP + SC_COLS) xs[i] = v;
    }
    __syncthreads();
    Vec<RQ> k, q;
    k.load(xs + 2 * lg);
    q.load(xs + DP + 2 * lg);
    const float v = xs[2 * DP + col_s];
    S.decay_axpy(expf(la), k, dt * v);
    const float r = group_sum(S.dot(q));
    if (live) {
        S.store(sp);
        if (lg == 0) y[h * a.vdim + col] = r + skip * v;
    }
}

bool ssd_ok(const hf2q_ssd* a) {
    return a && a->proj && a->conv && a->conv_bias && a->dt_bias && a->a_log && a->d && a->conv_state && a->s && a->pos && a->heads && a->groups &&
           a->heads % a->groups == 0 && a->state && a->state <= 256 && a->vdim && a->taps;
}
template <int RQ, int C, int W, uint32_t TB>
cudaError_t launch_ssd_scan_as(const hf2q_ssd& a, uint32_t m, const float* xbc, const float* dt, const float* la, float* y, int sms, cudaStream_t st) {
    static PerDeviceFlag flag;
    constexpr size_t need = 4ull * TB * 32 * RQ * sizeof(float);
    constexpr uint32_t cols = ScanPlace<RQ, C, W>::COLS;
    const dim3 grid(a.heads, (a.vdim + cols - 1) / cols);
    if (const cudaError_t e = ensure_max_dynamic_smem(ssd_scan_kernel<RQ, C, W, TB>, SCAN_MAX, flag); e != cudaSuccess) return e;
    return launch_pdl(ssd_scan_kernel<RQ, C, W, TB>, grid, dim3((W + 1) * 32), TB == SC_TB ? scan_smem(need, grid, sms) : need, st, a, m, xbc, dt, la, y);
}
// Few tokens and more CTAs than SMs: one column a group in batches of 8, four CTAs to an SM (128 heads of 128 x 64, 5 tokens:
// 5.8 us, with two columns 6.6; 64 heads: 5.2 and 4.4).
template <int RQ>
cudaError_t launch_ssd_scan(const hf2q_ssd& a, uint32_t m, const float* xbc, const float* dt, const float* la, float* y, int sms, cudaStream_t st) {
    constexpr uint32_t cols = ScanPlace<RQ, 2, 8>::COLS;
    if (m < 8 && static_cast<uint64_t>(a.heads) * ((a.vdim + cols - 1) / cols) > static_cast<uint64_t>(sms))
        return launch_ssd_scan_as<RQ, 1, 8, SC_FEW>(a, m, xbc, dt, la, y, sms, st);
    return launch_ssd_scan_as<RQ, 2, 8, SC_TB>(a, m, xbc, dt, la, y, sms, st);
}

bool delta_ok(const hf2q_delta* a) {
    return a && a->proj && a->q_conv && a->k_conv && a->v_conv && a->a_log && a->dt_bias && a->a2 && a->g2 && a->conv_state && a->s && a->pos &&
           a->heads && a->kv_heads && a->heads % a->kv_heads == 0 && a->dim && a->dim <= 256 && a->vdim && a->taps && a->a_rank_ld % 8 == 0 &&
           a->g_rank_ld % 8 == 0 && a->a_rank_ld && a->g_rank_ld;
}
template <int RQ, int C, int W, uint32_t TB, int PER_SM>
cudaError_t launch_scan_as(const hf2q_delta& a, uint32_t m, const float* qkv, const float* beta, const float* g, float* out, int sms, cudaStream_t st) {
    static PerDeviceFlag flag;
    constexpr size_t need = 6ull * TB * 32 * RQ * sizeof(float);
    constexpr uint32_t cols = ScanPlace<RQ, C, W>::COLS;
    const dim3 grid(a.heads, (a.vdim + cols - 1) / cols);
    if (const cudaError_t e = ensure_max_dynamic_smem(delta_scan_kernel<RQ, C, W, TB, PER_SM>, SCAN_MAX, flag); e != cudaSuccess) return e;
    return launch_pdl(delta_scan_kernel<RQ, C, W, TB, PER_SM>, grid, dim3((W + 1) * 32), TB == SC_TB ? scan_smem(need, grid, sms) : need, st, a, m, qkv, beta, g, out);
}
// Few tokens: one column a group and batches of 8, as below (16 heads of 256 x 256: 33 tokens 27.3 us with two columns a group;
// of 128 x 128: 8 tokens 5.6 with one, 3.9 with two).  More CTAs than SMs: two to an SM where the batches of both fit (dim up to
// 128), which costs a CTA alone 6 % (200 registers).
template <int RQ>
cudaError_t launch_scan(const hf2q_delta& a, uint32_t m, const float* qkv, const float* beta, const float* g, float* out, int sms, cudaStream_t st) {
    if (m < (RQ > 4 ? 64u : 8u)) return launch_scan_as<RQ, 1, 8, SC_FEW, 2>(a, m, qkv, beta, g, out, sms, st);
    constexpr uint32_t cols = ScanPlace<RQ, 2, 4>::COLS;
    if (RQ <= 4 && static_cast<uint64_t>(a.heads) * ((a.vdim + cols - 1) / cols) > static_cast<uint64_t>(sms))
        return launch_scan_as<RQ, 2, 4, SC_TB, RQ <= 4 ? 2 : 1>(a, m, qkv, beta, g, out, sms, st);
    return launch_scan_as<RQ, 2, 4, SC_TB, 1>(a, m, qkv, beta, g, out, sms, st);
}

// four taps, as such layers are built; other counts a CTA a token
template <typename LR>
cudaError_t launch_delta_prep(const hf2q_delta& a, uint32_t m, float* qkv, float* beta, LR* a1, LR* g1, int sms, cudaStream_t st) {
    const uint32_t qk_columns = (2 * a.kv_heads + 7) / 8, columns = qk_columns + (a.heads * a.vdim + 255) / 256 + 1;
    if (a.taps != 4 || columns > 65535) return launch_pdl(delta_prep_kernel<LR>, dim3(m), dim3(256), 0, st, a, qkv, beta, a1, g1);
    const uint32_t per = prep_tokens(m, columns, sms, a.dim > 128);
    const dim3 grid((m + per - 1) / per, columns);
    if (a.dim <= 128) return launch_pdl(delta_prep4_kernel<4, LR>, grid, dim3(256), 0, st, a, m, per, qk_columns, qkv, beta, a1, g1);
    return launch_pdl(delta_prep4_kernel<8, LR>, grid, dim3(256), 0, st, a, m, per, qk_columns, qkv, beta, a1, g1);
}

template <int RQ, int C, uint32_t TB>
cudaError_t launch_mlstm_as(const hf2q_mlstm& a, uint32_t m, float* out, int sms, cudaStream_t st) {
    static PerDeviceFlag flag;
    constexpr size_t need = 4ull * TB * 32 * RQ * sizeof(float);
    const dim3 grid(a.heads, (a.vdim + SC_COLS - 1) / SC_COLS);
    if (const cudaError_t e = ensure_max_dynamic_smem(mlstm_kernel<RQ, C, TB>, SCAN_MAX, flag); e != cudaSuccess) return e;
    return launch_pdl(mlstm_kernel<RQ, C, TB>, grid, dim3((8 / C + 1) * 32), TB == SC_TB ? scan_smem(need, grid, sms) : need, st, a, m, out);
}
// Few tokens: what counts is how soon a token's chain starts and that the CTAs share the SMs, so one column a group, eight warps,
// and a batch of 8 tokens, whose buffers let several CTAs on an SM.  The line lies where two columns a group take whole groups of
// tokens: 16 heads of 128 x 128, 8 tokens 6.0 us with one column, 3.7 with two; 5 tokens 4.8 and 4.8.
template <int RQ>
cudaError_t launch_mlstm(const hf2q_mlstm& a, uint32_t m, float* out, int sms, cudaStream_t st) {
    if (m == 1) return launch_pdl(mlstm_step_kernel<RQ>, dim3(a.heads, (a.vdim + SC_COLS - 1) / SC_COLS), dim3(SC_THREADS), 0, st, a, out);
    if (m < (RQ > 4 ? 16u : 8u)) return launch_mlstm_as<RQ, 1, SC_FEW>(a, m, out, sms, st);
    return launch_mlstm_as<RQ, 2, SC_TB>(a, m, out, sms, st);
}

#define HF2Q_RQ_CASES(F) F(1) F(2) F(3) F(4) F(5) F(6) F(7) F(8)

}  // namespace
}  // namespace hf2q

using namespace hf2q;
using namespace hf2q::seq;

extern "C" {

HF2Q_API int32_t hf2q_cuda_mlstm(hf2q_ctx* ctx, void* stream, const hf2q_mlstm* a, uint32_t m, float* out) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!a || !a->proj || !a->i_bias || !a->f_bias || !a->s || !a->n || !a->mx || !out || a->heads == 0 || a->dim == 0 || a->vdim == 0 || a->dim > 256 ||
        !(a->gate_cap > 0.f))
        return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "mlstm: null pointer, or a size outside dim 1..256");
    if (m == 0) return HF2Q_OK;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaErrorInvalidValue;
    switch ((a->dim + 31) / 32) {
#define F(RQ) case RQ: e = launch_mlstm<RQ>(*a, m, out, ctx_sm_count(ctx), st); break;
        HF2Q_RQ_CASES(F)
#undef F
        default: break;
    }
    return ctx_cuda_result(ctx, e, "mlstm", 1);
}

HF2Q_API int32_t hf2q_cuda_delta_step(hf2q_ctx* ctx, void* stream, const hf2q_delta* a, float* out, float* gate) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!delta_ok(a) || !out || !gate) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "delta_step: null pointer or an unsupported size");
    const dim3 grid(a->heads, (a->vdim + SC_COLS - 1) / SC_COLS);
    const size_t smem = static_cast<size_t>(a->a_rank_ld + a->g_rank_ld) * 4;
    if (smem > 32 * 1024) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "delta_step: rank too large");
    cudaError_t e = cudaErrorInvalidValue;
    switch ((a->dim + 31) / 32) {
#define F(RQ) case RQ: e = launch_pdl(delta_step_kernel<RQ>, grid, dim3(SC_THREADS), smem, static_cast<cudaStream_t>(stream), *a, out, gate); break;
        HF2Q_RQ_CASES(F)
#undef F
        default: break;
    }
    return ctx_cuda_result(ctx, e, "delta_step", 1);
}

HF2Q_API int32_t hf2q_cuda_delta_prep(hf2q_ctx* ctx, void* stream, const hf2q_delta* a, uint32_t m, float* qkv, float* beta, void* a1, void* g1,
                                      uint32_t lr_dtype) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!delta_ok(a) || !qkv || !beta || !a1 || !g1) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "delta_prep: null pointer or an unsupported size");
    if (m == 0) return HF2Q_OK;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaErrorInvalidValue;
    if (lr_dtype == HF2Q_DT_F32) e = launch_delta_prep(*a, m, qkv, beta, static_cast<float*>(a1), static_cast<float*>(g1), ctx_sm_count(ctx), st);
    else if (lr_dtype == HF2Q_DT_BF16) e = launch_delta_prep(*a, m, qkv, beta, static_cast<__nv_bfloat16*>(a1), static_cast<__nv_bfloat16*>(g1), ctx_sm_count(ctx), st);
    return ctx_cuda_result(ctx, e, "delta_prep", 1);
}

HF2Q_API int32_t hf2q_cuda_delta_decay(hf2q_ctx* ctx, void* stream, const hf2q_delta* a, uint32_t m, float* g) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!delta_ok(a) || !g) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "delta_decay: null pointer or an unsupported size");
    if (m == 0) return HF2Q_OK;
    const uint64_t n = static_cast<uint64_t>(m) * a->heads * a->dim, want = (n + 255) / 256, cap = static_cast<uint64_t>(ctx_sm_count(ctx)) * 16;
    const cudaError_t e = launch_pdl(delta_decay_kernel, dim3(static_cast<unsigned>(want < cap ? want : cap)), dim3(256), 0, static_cast<cudaStream_t>(stream),
                                     a->a_log, a->dt_bias, a->dim, a->heads * a->dim, n, g);
    return ctx_cuda_result(ctx, e, "delta_decay", 1);
}

HF2Q_API int32_t hf2q_cuda_delta_scan(hf2q_ctx* ctx, void* stream, const hf2q_delta* a, uint32_t m, const float* qkv, const float* beta, const float* g,
                                      float* out) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!delta_ok(a) || !qkv || !beta || !g || !out) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "delta_scan: null pointer or an unsupported size");
    if (m == 0) return HF2Q_OK;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaErrorInvalidValue;
    switch ((a->dim + 31) / 32) {
#define F(RQ) case RQ: e = launch_scan<RQ>(*a, m, qkv, beta, g, out, ctx_sm_count(ctx), st); break;
        HF2Q_RQ_CASES(F)
#undef F
        default: break;
    }
    return ctx_cuda_result(ctx, e, "delta_scan", 1);
}

HF2Q_API int32_t hf2q_cuda_ssd_step(hf2q_ctx* ctx, void* stream, const hf2q_ssd* a, float* y) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!ssd_ok(a) || !y) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "ssd_step: null pointer or an unsupported size");
    const dim3 grid(a->heads, (a->vdim + SC_COLS - 1) / SC_COLS);
    cudaError_t e = cudaErrorInvalidValue;
    switch ((a->state + 31) / 32) {
#define F(RQ) case RQ: e = launch_pdl(ssd_step_kernel<RQ>, grid, dim3(SC_THREADS), 0, static_cast<cudaStream_t>(stream), *a, y); break;
        HF2Q_RQ_CASES(F)
#undef F
        default: break;
    }
    return ctx_cuda_result(ctx, e, "ssd_step", 1);
}

HF2Q_API int32_t hf2q_cuda_ssd_prep(hf2q_ctx* ctx, void* stream, const hf2q_ssd* a, uint32_t m, float* xbc, float* dt, float* la) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!ssd_ok(a) || !xbc || !dt || !la) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "ssd_prep: null pointer or an unsupported size");
    if (m == 0) return HF2Q_OK;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t columns = (a->heads * a->vdim + 2 * a->groups * a->state + 255) / 256 + 1;
    const uint32_t per = prep_tokens(m, columns, ctx_sm_count(ctx));
    const cudaError_t e = a->taps == 4 && columns <= 65535 ? launch_pdl(ssd_prep4_kernel, dim3((m + per - 1) / per, columns), dim3(256), 0, st, *a, m, per, xbc, dt, la)
                                                           : launch_pdl(ssd_prep_kernel, dim3(m), dim3(256), 0, st, *a, xbc, dt, la);
    return ctx_cuda_result(ctx, e, "ssd_prep", 1);
}

HF2Q_API int32_t hf2q_cuda_ssd_scan(hf2q_ctx* ctx, void* stream, const hf2q_ssd* a, uint32_t m, const float* xbc, const float* dt, const float* la, float* y) {
    if (!ctx) return HF2Q_ERR_INVALID_ARGUMENT;
    if (!ssd_ok(a) || !xbc || !dt || !la || !y) return ctx_fail(ctx, HF2Q_ERR_INVALID_ARGUMENT, "ssd_scan: null pointer or an unsupported size");
    if (m == 0) return HF2Q_OK;
    cudaError_t e = cudaErrorInvalidValue;
    switch ((a->state + 31) / 32) {
#define F(RQ) case RQ: e = launch_ssd_scan<RQ>(*a, m, xbc, dt, la, y, ctx_sm_count(ctx), static_cast<cudaStream_t>(stream)); break;
        HF2Q_RQ_CASES(F)
#undef F
        default: break;
    }
    return ctx_cuda_result(ctx, e, "ssd_scan", 1);
}

}  // extern "C"
