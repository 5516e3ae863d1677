// The routed experts of a step of few tokens: the matrices in use are streamed once, as csrc/gemv_bf16.cu streams a dense one.
//
//   expert_stream    for every (token, choice) pair p with unit e = ids[p] >= 0:  y[p] = act(W[e] x[row of p]), where the row is the
//                    pair's token (times its score, rounded, where the score scales the input) or the pair itself
//
// A block owns one unit and a tile of its rows; it finds the pairs that chose the unit among `ids` and leaves if there are
// none, so neither a plan of tiles nor gathered rows are needed, and the activation is the product's epilogue: two launches
// (gate|up, down) take the place of six. The arithmetic is the weight-streaming product's (mma.sync m16n8k16, weights as the
// 16-row operand, up to 8 pairs as the other, k positions permuted alike on both sides, the warps' partial sums added in warp
// order); a unit chosen by more than 8 pairs goes over its tile again. Rounding points are those of the grouped products:
// sums rounded, the unit's activation of the rounded sums rounded.
//
// Without `ids` it is the product with a matrix per head (csrc/gemm_tcgen05.cu's for steps of more tokens): unit h takes row h of every token.
//
// What bounds it: bytes of the matrices in use. Both products of 32 gated units of 1,024 x 2,048, each token in 4 of them and in two
// more that all take, against plan, gathered rows, grouped products and activation: 1 token 43 -> 21 us, 4 tokens 54 -> 45, 8 tokens
// 85 -> 62 (283 MB: 4.6 TB/s), 16 tokens 91 -> 89; plain units without the two: 1 token 40 -> 12 us, 8 tokens 56 -> 39.
#include "expert_stream.h"

#define ES_WARPS 8
#define ES_U 4                  // 32-wide k blocks of two row tiles in flight per warp: 16 16-byte weight loads per thread

__device__ __forceinline__ uint4 es_load_weights(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 es_load_rows(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.ca.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void es_mma(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// GATED: the unit's matrix holds `out` gate rows and then `out` up rows; a block's two row tiles are rows r of both. Otherwise they
// are 32 consecutive rows. SCALE: a pair's row is its token's times its score, rounded to bfloat16.
template <bool GATED, bool SCALE>
__global__ void __launch_bounds__(ES_WARPS * 32, 2) expert_stream_kernel(bf16* __restrict__ y, const bf16* x, const bf16* __restrict__ W,
                                                                      const int* ids, const float* scores, int* __restrict__ pair_row, int pairs,
                                                                      int per_row, int by_pair, int out, int K, int act, const float* __restrict__ limits,
                                                                      float slope, float shift, int ahead) {
    __shared__ float red[ES_WARPS][2][32][4];
    __shared__ int chosen[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int row0 = blockIdx.x * (GATED ? 16 : 32);
    bool waited = !ahead;
    if (waited) pdl_enter();
    const bool heads = ids == nullptr;                     // a matrix per head: pair p is token p / units, head p % units
    if (pair_row != nullptr && blockIdx.x == 0 && blockIdx.y == 0)     // a pair's result is its own row; a choice without a unit has none
        for (int p = threadIdx.x; p < pairs; p += ES_WARPS * 32) pair_row[p] = __ldcg(ids + p) >= 0 ? p : -1;
    // With `by_pair` a block's unit is that of pair blockIdx.y, if no pair before it chose the same one.
    const int unit = by_pair ? __ldcg(ids + blockIdx.y) : (int)blockIdx.y;
    if (unit < 0) {
        if (!waited) pdl_wait();                           // no block ends before the kernel ahead: the next one counts on that
        return;
    }
    const bf16* w = W + (size_t)unit * (GATED ? 2 : 1) * out * K;
    const int next = GATED ? out : 16;                     // rows between the two tiles
    const uint4* wr[2][2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = min(row0 + g + 8 * i + (GATED ? 0 : 16 * j), out - 1) + (GATED ? next * j : 0);
            wr[j][i] = reinterpret_cast<const uint4*>(w + (size_t)r * K);
        }
    const int blocks = (K + 31) >> 5;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (int first = 0;; first += 8) {
        // The pairs first .. first + 7 among those that chose this unit, in their order; a lane's is number first + g.
        int mine = -1, seen = 0, leader = -1;
        if (heads) {
            seen = pairs / (int)gridDim.y;
            if (first + g < seen) mine = (first + g) * (int)gridDim.y + unit;
        }
        for (int p0 = 0; !heads && p0 < pairs; p0 += 32) {
            unsigned m = __ballot_sync(0xffffffffu, p0 + lane < pairs && __ldcg(ids + p0 + lane) == unit);
            const int here = __popc(m), skip = first + g - seen;
            if (leader < 0 && m != 0) leader = p0 + __ffs(m) - 1;
            if (mine < 0 && skip >= 0 && skip < here) {
                for (int s = 0; s < skip; ++s) m &= m - 1;
                mine = p0 + __ffs(m) - 1;
            }
            seen += here;
        }
        if (first >= seen || (by_pair && leader != (int)blockIdx.y)) {           // the same for every thread of the block
            if (!waited) pdl_wait();
            return;
        }
        if (warp == 0 && t == 0) chosen[g] = mine;
        const bf16* xrow = x + (size_t)(mine < 0 ? 0 : mine / per_row) * K;
        const float score = SCALE && mine >= 0 ? __ldcg(scores + mine) : 1.f;
        float c[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) c[j][i] = 0.f;
        for (int b = warp; b < blocks; b += ES_WARPS * ES_U) {
            uint4 a[2][2][ES_U], v[ES_U];
#pragma unroll
            for (int u = 0; u < ES_U; ++u) {
                const int bb = b + u * ES_WARPS, idx = bb * 4 + t;
                const bool ok = bb < blocks && bb * 32 + 8 * t < K;          // K % 8 == 0: 8 consecutive k are inside the row or outside it
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int i = 0; i < 2; ++i) a[j][i][u] = ok ? es_load_weights(wr[j][i] + idx) : zero;
            }
            if (!waited) { pdl_enter(); waited = true; }   // the first weights are on their way
#pragma unroll
            for (int u = 0; u < ES_U; ++u) {
                const int bb = b + u * ES_WARPS, idx = bb * 4 + t;
                v[u] = bb < blocks && bb * 32 + 8 * t < K && mine >= 0 ? es_load_rows(reinterpret_cast<const uint4*>(xrow) + idx) : zero;
            }
#pragma unroll
            for (int u = 0; u < ES_U; ++u) {
                if (SCALE) {
                    Vec16<bf16> r;
                    r.unpack(v[u]);
                    unsigned q[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const __nv_bfloat162 s2 = __floats2bfloat162_rn(score * r.v[2 * e], score * r.v[2 * e + 1]);
                        q[e] = *reinterpret_cast<const unsigned*>(&s2);
                    }
                    v[u] = make_uint4(q[0], q[1], q[2], q[3]);
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    es_mma(c[j], a[j][0][u].x, a[j][1][u].x, a[j][0][u].y, a[j][1][u].y, v[u].x, v[u].y);
                    es_mma(c[j], a[j][0][u].z, a[j][1][u].z, a[j][0][u].w, a[j][1][u].w, v[u].z, v[u].w);
                }
            }
        }
        if (!waited) { pdl_enter(); waited = true; }       // a warp without work orders its writes after the kernel ahead too
#pragma unroll
        for (int j = 0; j < 2; ++j) *reinterpret_cast<float4*>(red[warp][j][lane]) = make_float4(c[j][0], c[j][1], c[j][2], c[j][3]);
        __syncthreads();
        for (int i = threadIdx.x; i < (GATED ? 128 : 256); i += ES_WARPS * 32) {
            const int j = i >> 7, l = (i & 127) >> 2, ci = i & 3;
            const int r = row0 + (l >> 2) + ((ci & 2) ? 8 : 0) + (GATED ? 0 : 16 * j), p = chosen[2 * (l & 3) + (ci & 1)];
            if (r >= out || p < 0) continue;
            float s[2] = {0.f, 0.f};
#pragma unroll
            for (int k = 0; k < ES_WARPS; ++k) {
                s[0] += red[k][GATED ? 0 : j][l][ci];
                if (GATED) s[1] += red[k][1][l][ci];
            }
            float o = rnd<bf16>(s[0]);
            if (GATED) {
                const float limit = limits[unit];
                const float a0 = fminf(o, limit), b0 = fminf(fmaxf(rnd<bf16>(s[1]), -limit), limit);
                o = a0 / (1.0f + __expf(-slope * a0)) * (b0 + shift);
            } else if (act == ES_ACT_RELU2) {
                o = fmaxf(o, 0.f);
                o *= o;
            }
            y[(size_t)p * out + r] = __float2bfloat16_rn(o);
        }
        if (first + 8 >= seen) return;
        __syncthreads();                                   // `chosen` and `red` are written again
    }
}

int expert_stream(void* y, const void* x, const void* W, const ExpertStream& e, int units, int out, int in, cudaStream_t stream) {
    if (e.pairs == 0) return 0;
    TI_REQUIRE(e.pairs > 0 && e.per_row >= 1 && units >= 1 && units <= 65535 && out > 0 && in > 0, "expert_stream: %d pairs, %d units, out %d, in %d", e.pairs,
               units, out, in);
    TI_REQUIRE(in % 8 == 0 && aligned16(x) && aligned16(W), "expert_stream: rows of %d must be 16-byte vectors", in);
    TI_REQUIRE(!e.gated || e.limits != nullptr, "expert_stream: a gated unit needs its limits");
    TI_REQUIRE(!e.ahead || (e.scores == nullptr && e.pair_row == nullptr), "expert_stream: scores and rows are the kernel before's");
    TI_REQUIRE(e.ids != nullptr || (e.pairs % units == 0 && e.pair_row == nullptr), "expert_stream: %d rows of %d heads", e.pairs, units);
    TI_REQUIRE(e.act == ES_ACT_NONE || e.act == ES_ACT_RELU2, "expert_stream: unknown activation %d", e.act);
    const int rows = e.gated ? 16 : 32;
    // Blocks of units that no pair chose leave at once but still take their turn (64 units, 1 token of 8 units: 20 us of 80), so with
    // fewer pairs than units there is a row of blocks per pair.
    const int by_pair = e.ids != nullptr && e.pairs < units;
    const dim3 grid((out + rows - 1) / rows, by_pair ? e.pairs : units), block(ES_WARPS * 32);
#define ES_LAUNCH(G, S) ti_launch(expert_stream_kernel<G, S>, grid, block, 0, stream, (bf16*)y, (const bf16*)x, (const bf16*)W, e.ids, e.scores, e.pair_row, \
                                  e.pairs, e.per_row, by_pair, out, in, e.act, e.limits, e.slope, e.shift, e.ahead)
    if (e.gated) { if (e.scores != nullptr) ES_LAUNCH(true, true); else ES_LAUNCH(true, false); }
    else { if (e.scores != nullptr) ES_LAUNCH(false, true); else ES_LAUNCH(false, false); }
#undef ES_LAUNCH
    return ti_check_launch("expert_stream");
}
