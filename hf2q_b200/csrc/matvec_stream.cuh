// Weight stream of the one-row products: a CTA's weights are cut into chunks of MV_CHUNK elements; its warps take the
// chunks in turn, each through a private ring of bulk copies.  Where the addresses do not depend on an earlier kernel the
// ring starts filling before the wait for it (weights never change).  Chunk sums of a block of rows meet in shared memory
// and are added in chunk order.
#pragma once
#include "seq_common.cuh"

namespace hf2q {
namespace seq {

// One CTA an SM; its kernels say so in their launch bounds, for with all registers to give ptxas asks for a chunk's 16-byte groups and
// a prologue's loads at once (16 warps, 25 MB: 9.4 us a product without, 7.6 with).  In a chain of up (norm prologue) and down
// products, us a product at 2048 x 6144 / 4096 x 11264 / 3072 x 9216 / 1536 x 4096: 12 warps of 3 stages 6.6 / 16.5 / 11.9 / 5.4, of 2
// 6.8 / 17.3 / 12.3 / 5.3, 16 of 3 7.3 / 16.9 / 12.9 / 5.6, 8 of 3 with chunks of 1536 7.5 / 17.3 / 11.3 / 5.3; two CTAs an SM 9.3 and
// more.  Before: 9.9 / 24.7 / 17.3 / 6.7.  (With the plan below 6.4 / 16.4 / - / 5.0.)
constexpr int MR_WARPS = 12, MR_THREADS = MR_WARPS * 32, MR_STAGES = 3, MV_CHUNK = 1024, MR_PART = 2048;
constexpr uint32_t MR_RING = MR_WARPS * MR_STAGES * MV_CHUNK * 2;      // bytes of dynamic shared memory
constexpr uint32_t MR_MAX_X = 112 * 1024;                              // bytes of activations

// A row of k weights is cut into pieces of this many elements: a divisor of the warps to a row, so that each warp keeps to one place
// of the rows and holds that place's activations in registers.  Longer rows: pieces of MV_CHUNK, activations from shared memory at
// every step (16 bytes of weights meet 32 of activations there).
constexpr uint32_t mv_piece(uint32_t k) {
    for (uint32_t n = 1; n <= MR_WARPS; ++n)
        if (MR_WARPS % n == 0 && k <= n * MV_CHUNK) return (k + 8 * n - 1) / (8 * n) * 8;
    return MV_CHUNK;
}
// Who does what, worked out on the host: a kernel's first instructions come cold, and its divisions were 0.5 us of every launch.
struct MatvecPlan {
    uint32_t rows, extra;        // rows (or pairs) of a CTA; the first `extra` CTAs have one more
    uint32_t piece, per_row;     // elements of a piece, pieces of a row
    uint32_t inv;                // x / per_row = x * inv >> 16 for x <= MR_WARPS
    uint32_t block_rows;         // rows whose sums meet at a time
    __device__ __forceinline__ uint32_t first(uint32_t cta) const { return rows * cta + min(cta, extra); }
    __device__ __forceinline__ uint32_t count(uint32_t cta) const { return rows + (cta < extra ? 1u : 0u); }
};
// rows of k weights, side of them to one sum; unit 2: in pairs
inline MatvecPlan matvec_plan(uint32_t rows, uint32_t unit, uint32_t ctas, uint32_t k, uint32_t side = 1) {
    const uint32_t piece = mv_piece(k), per_row = side * ((k + piece - 1) / piece), block = MR_PART / per_row / unit * unit;
    return {rows / unit / ctas, rows / unit % ctas, piece, per_row, (65536 + per_row - 1) / per_row, block ? block : unit};
}

struct MatvecShared {
    float part[2][MR_PART];
    uint64_t bars[MR_WARPS][MR_STAGES];
};
struct MatvecChunk {
    const __nv_bfloat16* w;      // global, 16-byte aligned
    uint32_t x0, len;            // its activations start at xs + x0; len a multiple of 8, at most MV_CHUNK
};

// What a step costs beside its 32 multiply-adds a lane is what this class is about: a chunk in 950 ns and more, with the weights long
// in shared memory, was 6 of the 10 us of a product of 25 MB.  Hence no division (places advance by a constant), no address but the
// issuing lane's, activations in registers.
class MatvecStream {
public:
    __device__ __forceinline__ MatvecStream(uint8_t* smem, MatvecShared& sh, uint32_t rows, const MatvecPlan& plan, uint32_t* status)
        : sh_(sh), rows_(rows), per_row_(plan.per_row), block_rows_(plan.block_rows), status_(status), warp_(threadIdx.x >> 5), lane_(threadIdx.x & 31),
          ring_(reinterpret_cast<__nv_bfloat16*>(smem) + static_cast<size_t>(warp_) * MR_STAGES * MV_CHUNK) {
        down_ = MR_WARPS * plan.inv >> 16;
        right_ = MR_WARPS - down_ * per_row_;
        now_.row = next_.row = warp_ * plan.inv >> 16;
        now_.col = next_.col = warp_ - now_.row * per_row_;
    }

    // fills the ring; at(row, col) -> MatvecChunk
    template <class F> __device__ __forceinline__ void start(F at) {
        if (lane_ == 0) {
            for (uint32_t i = 0; i < MR_STAGES; ++i) mbar_init(&sh_.bars[warp_][i], 1);
            mbar_fence_init();
        }
        for (uint32_t i = 0; i < MR_STAGES; ++i) issue(i, at);
    }
    // The rows, finished one (or with PAIRS two) at a time: finish(row, sum, sum of row + 1).  Every thread of the CTA calls it,
    // after a barrier behind the last write of xs.  x0 and len depend on the column only.
    template <bool PAIRS, class F, class G> __device__ __forceinline__ void run(F at, const float* xs, G finish) {
        if (right_ == 0) run_as<PAIRS, true>(at, xs, finish);
        else run_as<PAIRS, false>(at, xs, finish);
    }

private:
    struct Place { uint32_t row, col; };
    __device__ __forceinline__ void advance(Place& p) const {              // to the warp's next chunk
        p.row += down_;
        p.col += right_;
        if (p.col >= per_row_) { p.col -= per_row_; ++p.row; }
    }
    static constexpr int U = MV_CHUNK / 256;                               // 16-byte groups of a chunk per lane
    template <bool PAIRS, bool HELD, class F, class G> __device__ __forceinline__ void run_as(F at, const float* xs, G finish) {
        constexpr uint32_t unit = PAIRS ? 2 : 1;
        float held[HELD ? U : 1][8];
        uint32_t len = 0;
        if constexpr (HELD) {
            if (now_.row < rows_) {
                const MatvecChunk k = at(now_.row, now_.col);
                len = k.len;
#pragma unroll
                for (int u = 0; u < U; ++u) load_x(xs + k.x0, lane_ + 32 * u, len, held[u]);
            }
        }
        bool ok = true;
        uint32_t st = 0, ph = 0;                                            // ring slot and parity
        for (uint32_t r0 = 0, pb = 0; r0 < rows_; r0 += block_rows_, pb ^= 1) {
            const uint32_t nr = min(block_rows_, rows_ - r0);
            for (; now_.row < r0 + nr; advance(now_)) {
                const float* x = xs;
                if constexpr (!HELD) {
                    const MatvecChunk k = at(now_.row, now_.col);
                    len = k.len;
                    x += k.x0;
                }
                if (ok) ok = mbar_wait_bounded(&sh_.bars[warp_][st], ph, status_);
                ok = __all_sync(0xffffffffu, ok);
                uint4 v[U];
                const uint4* wv = reinterpret_cast<const uint4*>(ring_ + st * MV_CHUNK);
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = ok && 8 * (lane_ + 32 * u) < len ? wv[lane_ + 32 * u] : make_uint4(0, 0, 0, 0);
                __syncwarp();                                               // every lane has read the stage
                if (ok) issue(st, at);
                if (++st == MR_STAGES) { st = 0; ph ^= 1; }
                float acc[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    float mine[8];
                    if constexpr (!HELD) load_x(x, lane_ + 32 * u, len, mine);
                    const float (&f)[8] = HELD ? held[HELD ? u : 0] : mine;
                    float a = bf_lo(v[u].x) * f[0];
                    a = fmaf(bf_hi(v[u].x), f[1], a); a = fmaf(bf_lo(v[u].y), f[2], a); a = fmaf(bf_hi(v[u].y), f[3], a);
                    a = fmaf(bf_lo(v[u].z), f[4], a); a = fmaf(bf_hi(v[u].z), f[5], a); a = fmaf(bf_lo(v[u].w), f[6], a); a = fmaf(bf_hi(v[u].w), f[7], a);
                    acc[u] = a;
                }
                const float sum = warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
                if (lane_ == 0) sh_.part[pb][(now_.row - r0) * per_row_ + now_.col] = sum;
            }
            __syncthreads();                                                // (the other half of `part` is free: its readers passed this barrier)
            for (uint32_t r = threadIdx.x * unit; r < nr; r += MR_THREADS * unit) {
                float v = 0.f, w = 0.f;
                for (uint32_t kc = 0; kc < per_row_; ++kc) v += sh_.part[pb][r * per_row_ + kc];
                if constexpr (PAIRS)
                    for (uint32_t kc = 0; kc < per_row_; ++kc) w += sh_.part[pb][(r + 1) * per_row_ + kc];
                finish(r0 + r, v, w);
            }
        }
    }
    static __device__ __forceinline__ void load_x(const float* x, uint32_t e, uint32_t len, float (&out)[8]) {
        const bool in = 8 * e < len;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 a = in ? *reinterpret_cast<const float4*>(x + 8 * e) : zero, b = in ? *reinterpret_cast<const float4*>(x + 8 * e + 4) : zero;
        out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w; out[4] = b.x; out[5] = b.y; out[6] = b.z; out[7] = b.w;
    }
    template <class F> __device__ __forceinline__ void issue(uint32_t st, F& at) {      // the next chunk of this warp into slot st
        if (lane_ == 0 && next_.row < rows_) {
            const MatvecChunk k = at(next_.row, next_.col);
            uint64_t* bar = &sh_.bars[warp_][st];
            mbar_arrive_expect_tx(bar, k.len * 2);
            bulk_g2s(ring_ + st * MV_CHUNK, k.w, k.len * 2, bar);
        }
        advance(next_);
    }
    MatvecShared& sh_;
    const uint32_t rows_, per_row_, block_rows_;
    uint32_t* const status_;
    const uint32_t warp_, lane_;
    __nv_bfloat16* const ring_;
    uint32_t down_, right_;
    Place now_, next_;
};

}  // namespace seq
}  // namespace hf2q
