// The routed experts of a step of few tokens: the matrices in use are streamed once, as csrc/gemv_bf16.cu streams a dense one.
//
//   expert_stream    for every (token, choice) pair p with unit e = ids[p] >= 0:  y[p] = act(W[e] x[row of p]), where the row is the
//                    pair's token (times its score, rounded, where the score scales the input) or the pair itself
//
// Every block makes the same list of the units in use from `ids` (a unit that more than 8 pairs chose stands there once per 8, one entry behind the
// other, so that its later passes find its matrix in L2), and the blocks,
// two or three an SM, go over the tiles of 16 rows of all of them in turn: neither a plan of tiles nor gathered rows are needed, and the
// activation is the product's epilogue: two launches (gate|up, down) take the place of six. A gated tile is 8 gate rows and the 8 up rows that go with
// them. The arithmetic is the weight-streaming product's (mma.sync m16n8k16, weights as the 16-row operand, up to 8 pairs as the other, k
// positions permuted alike on both sides, the warps' partial sums added in warp order). Rounding points are those of the grouped
// products: sums rounded, the unit's activation of the rounded sums rounded.
//
// What bounds it: bytes of the matrices in use. A thread's loads of two sets of k blocks are always on their way: where one set is used, the one
// after the other is asked for, in the next tile where this one ends, so the sums over the warps and the epilogue of a tile cost little bandwidth.
// (Six sets of one k block took 31 % longer: a warp has few counters for loads in flight, and sets that share one wait for one another.) Both products
// of units of 1,024 x 2,048 out of 32, each token in 4, on weights that are not in L2, against a block per tile of 32 rows: plain units, 4 tokens
// 28.1 -> 24.1 us, 8 tokens 38.0 -> 30.2; gated ones with two more that every token takes, 8 tokens 61.5 -> 47.4 (289 MB: 6.1 TB/s), 16 tokens 86 -> 66.
#include "expert_stream.h"

#define ES_WARPS 8
#define ES_MAX_PAIRS 512        // pairs of one launch: two a thread
#define ES_RUNS (ES_MAX_PAIRS / 32)
#define ES_NONE 0xffff
// Rows of up to so many elements: two sets of two k blocks in flight and three blocks an SM, else two sets of four and two blocks (both products of 34
// gated units of 1,024 x 2,048, 8 tokens 47.4 against 48.9 us; of 8 of 4,096 x 4,096, 1 token 40.8 against 36.0).
#define ES_SHORT_ROW 2048
#define ES_U 4                  // the same of two row tiles, where a block has one unit

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

// GATED: the unit's matrix holds `out` gate rows and then `out` up rows. SCALE: a pair's row is its token's times its score, rounded to
// bfloat16. The pairs are p0 .. p0 + pairs - 1 of the caller's (at most ES_MAX_PAIRS).
template <bool GATED, bool SCALE, int B, int OCC>
__global__ void __launch_bounds__(ES_WARPS * 32, OCC) expert_stream_kernel(bf16* __restrict__ y, const bf16* x, const bf16* __restrict__ W, const int* ids,
                                                                      const float* scores, int* __restrict__ pair_row, int p0, int pairs, int per_row, int out,
                                                                      int K, int act, const float* __restrict__ limits, float slope, float shift, int ahead, int cells) {
    constexpr int ROWS = GATED ? 8 : 16, U = 2;             // sets of B k blocks in flight
    __shared__ float4 red[ES_WARPS][32];
    __shared__ int found[ES_RUNS];
    extern __shared__ __align__(16) unsigned char lists[];
    uint4* counts = reinterpret_cast<uint4*>(lists);        // [cells]: how many pairs of each run of 32 chose the cell's unit, a byte each
    unsigned short(*members)[8] = reinterpret_cast<unsigned short(*)[8]>(counts + cells);        // [pairs]: an entry's pairs, ES_NONE beyond the last
    int* unit_of = reinterpret_cast<int*>(members + pairs); // [pairs]: an entry's unit
    int* cell = unit_of + pairs;                            // [cells]: a unit's number, then its first entry
    float* score_of = reinterpret_cast<float*>(cell + cells);                                    // [pairs]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    if (!ahead) pdl_enter();
    auto take = [&](int p) {                               // the pair's unit; a pair's result is its own row, a choice without a unit has none
        const int e = __ldcg(ids + p0 + p);
        if (SCALE) score_of[p] = __ldcg(scores + p0 + p);
        if (pair_row != nullptr && blockIdx.x == 0) pair_row[p0 + p] = e >= 0 ? p0 + p : -1;
        *reinterpret_cast<uint4*>(members[p]) = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
        return e;
    };
    int entries = 0;
    if (pairs <= 32) {
        if (warp == 0) {
            const int e = lane < pairs ? take(lane) : -1;
            const unsigned same = __match_any_sync(0xffffffffu, e), below = (1u << lane) - 1;
            const int before = __popc(same & below);       // pairs with this unit ahead of this one
            const unsigned m = __ballot_sync(0xffffffffu, e >= 0 && (before & 7) == 0);
            __syncwarp();
            if (e >= 0) {
                unsigned led = same;                       // the first pair of this one's eight
                for (int i = 0; i < (before & ~7); ++i) led &= led - 1;
                const int entry = __popc(m & ((1u << (__ffs(led) - 1)) - 1));
                members[entry][before & 7] = (unsigned short)lane;
                if ((before & 7) == 0) unit_of[entry] = e;
            }
            if (lane == 0) found[0] = __popc(m);
        }
        __syncthreads();
        entries = found[0];
    } else {
        // A warp takes a run of 32 pairs, and a second one of more than 256 pairs. Their units' cells of a hash table receive how many of them chose the
        // unit; a pair's place among its unit's is the sum of the runs before and its place in its own run, whatever cell the unit got.
        int unit[2], at[2] = {0, 0}, before[2] = {0, 0}, first[2] = {0, 0};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int p = u * ES_WARPS * 32 + threadIdx.x;
            unit[u] = p < pairs ? take(p) : -1;
        }
        for (int i = threadIdx.x; i < cells; i += ES_WARPS * 32) {
            counts[i] = make_uint4(0, 0, 0, 0);
            cell[i] = -1;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int run = u * ES_WARPS + warp;
            if (run * 32 >= pairs) break;                  // the same for every thread of the warp
            const unsigned same = __match_any_sync(0xffffffffu, unit[u]);
            const int lead = __ffs(same) - 1;
            int i = unit[u] & (cells - 1);
            if (unit[u] >= 0 && lane == lead) {
                for (;; i = (i + 1) & (cells - 1)) {       // there are no more units than cells
                    const int was = atomicCAS(cell + i, -1, unit[u]);
                    if (was == -1 || was == unit[u]) break;
                }
                reinterpret_cast<unsigned char*>(counts + i)[run] = (unsigned char)__popc(same);
            }
            at[u] = __shfl_sync(0xffffffffu, i, lead);
            before[u] = __popc(same & ((1u << lane) - 1));
        }
        __syncthreads();
        int made[2] = {0, 0};                              // entries of a pair that is its unit's first
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int run = u * ES_WARPS + warp;
            if (run * 32 >= pairs) break;
            if (unit[u] >= 0) {
                const uint4 n = counts[at[u]];
                const unsigned words[4] = {n.x, n.y, n.z, n.w};
                unsigned sooner = 0, all = 0;
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const int bytes = min(max(run - 4 * w, 0), 4);
                    sooner = __dp4a(bytes == 4 ? words[w] : words[w] & ((1u << (8 * bytes)) - 1), 0x01010101u, sooner);
                    all = __dp4a(words[w], 0x01010101u, all);
                }
                before[u] += (int)sooner;
                if (before[u] == 0) made[u] = ((int)all + 7) / 8;
            }
            int upto = made[u];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            if (lane == 31) found[run] = upto;
            first[u] = upto - made[u];
        }
        __syncthreads();
        for (int r = 0; r * 32 < pairs; ++r) {
            if (r == warp) first[0] += entries;
            if (r == ES_WARPS + warp) first[1] += entries;
            entries += found[r];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (made[u] > 0) {
                cell[at[u]] = first[u];
                for (int i = 0; i < made[u]; ++i) unit_of[first[u] + i] = unit[u];
            }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (unit[u] >= 0) members[cell[at[u]] + (before[u] >> 3)][before[u] & 7] = (unsigned short)(u * ES_WARPS * 32 + threadIdx.x);
        __syncthreads();
    }
    const int tiles = (out + ROWS - 1) / ROWS, total = entries * tiles;
    const int blocks = (K + 31) >> 5, steps = (blocks + ES_WARPS * B - 1) / (ES_WARPS * B);          // k blocks of a row, of them a warp's (the last may lie beyond)
    const uint4 zero = make_uint4(0, 0, 0, 0);
    // Where a warp's loads stand: step `i` of tile `item`; the tile's two rows of this lane and its pair's row (null: none).
    struct Place {
        const uint4 *w0, *w1, *x;
        int item, i;
    };
    auto enter = [&](Place& c) {
        if (c.item >= total) return;
        const int entry = c.item / tiles, row0 = (c.item - entry * tiles) * ROWS, unit = unit_of[entry], mine = members[entry][g];
        const bf16* w = W + (size_t)unit * (GATED ? 2 : 1) * out * K;
        c.w0 = reinterpret_cast<const uint4*>(w + (size_t)min(row0 + g, out - 1) * K) + t;
        c.w1 = reinterpret_cast<const uint4*>(w + (size_t)(GATED ? out + min(row0 + g, out - 1) : min(row0 + g + 8, out - 1)) * K) + t;
        c.x = mine != ES_NONE ? reinterpret_cast<const uint4*>(x + (size_t)((p0 + mine) / per_row) * K) + t : nullptr;
    };
    auto next = [&](Place& c) {
        if (++c.i == steps) {
            c.i = 0;
            c.item += gridDim.x;
            enter(c);
        }
    };
    auto inside = [&](const Place& c, int j) { return c.item < total && (warp + (c.i * B + j) * ES_WARPS) * 32 + 8 * t < K; };      // K % 8 == 0: 8 consecutive k are inside the row or outside it
    auto load_w = [&](const Place& c, uint4 (&a0)[B], uint4 (&a1)[B]) {
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const int at = (warp + (c.i * B + j) * ES_WARPS) * 4;
            const bool ok = inside(c, j);
            a0[j] = ok ? es_load_weights(c.w0 + at) : zero;
            a1[j] = ok ? es_load_weights(c.w1 + at) : zero;
        }
    };
    auto load_x = [&](const Place& c, uint4 (&v)[B]) {
#pragma unroll
        for (int j = 0; j < B; ++j) v[j] = inside(c, j) && c.x != nullptr ? es_load_rows(c.x + (warp + (c.i * B + j) * ES_WARPS) * 4) : zero;
    };
    Place front;
    front.item = blockIdx.x;
    front.i = 0;
    front.w0 = front.w1 = front.x = nullptr;
    enter(front);
    uint4 a0[U][B], a1[U][B], v[U][B];
    {
        Place rows = front;                                // the first weights are on their way before the wait, the rows after it
#pragma unroll
        for (int u = 0; u < U; ++u) {
            load_w(front, a0[u], a1[u]);
            next(front);
        }
        if (ahead) pdl_enter();
#pragma unroll
        for (int u = 0; u < U; ++u) {
            load_x(rows, v[u]);
            next(rows);
        }
    }
    Place here;                                            // the tile that is worked on
    here.item = blockIdx.x;
    here.i = 0;
    float score = 1.f;
    auto start = [&] {
        if (SCALE && here.item < total) {
            const int mine = members[here.item / tiles][g];
            score = mine != ES_NONE ? score_of[mine] : 1.f;
        }
    };
    start();
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    while (here.item < total) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (here.item < total) {                       // the same for every thread of the block
#pragma unroll
                for (int j = 0; j < B; ++j) {
                    uint4 r = v[u][j];
                    if (SCALE) {
                        Vec16<bf16> f;
                        f.unpack(r);
                        unsigned q[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const __nv_bfloat162 s2 = __floats2bfloat162_rn(score * f.v[2 * e], score * f.v[2 * e + 1]);
                            q[e] = *reinterpret_cast<const unsigned*>(&s2);
                        }
                        r = make_uint4(q[0], q[1], q[2], q[3]);
                    }
                    es_mma(c, a0[u][j].x, a1[u][j].x, a0[u][j].y, a1[u][j].y, r.x, r.y);
                    es_mma(c, a0[u][j].z, a1[u][j].z, a0[u][j].w, a1[u][j].w, r.z, r.w);
                }
                load_w(front, a0[u], a1[u]);
                load_x(front, v[u]);
                next(front);
                if (++here.i == steps) {                   // the tile's last: the warps' sums, in warp order
                    __syncthreads();                       // the tile before has been read
                    red[warp][lane] = make_float4(c[0], c[1], c[2], c[3]);
                    c[0] = c[1] = c[2] = c[3] = 0.f;
                    __syncthreads();
                    if (threadIdx.x < (GATED ? 64 : 128)) {
                        const int l = threadIdx.x / (GATED ? 2 : 4), ci = threadIdx.x % (GATED ? 2 : 4);
                        const int entry = here.item / tiles, p = members[entry][2 * (l & 3) + (ci & 1)];
                        const int r = (here.item - entry * tiles) * ROWS + (l >> 2) + ((ci & 2) ? 8 : 0);
                        if (r < out && p != ES_NONE) {
                            const float* from = reinterpret_cast<const float*>(&red[0][l]) + ci;
                            float s0 = 0.f, s1 = 0.f;
#pragma unroll
                            for (int w = 0; w < ES_WARPS; ++w) {
                                s0 += from[w * 128];
                                if (GATED) s1 += from[w * 128 + 2];
                            }
                            float o = rnd<bf16>(s0);
                            if (GATED) {
                                const float limit = limits[unit_of[entry]];
                                const float a = fminf(o, limit), b = fminf(fmaxf(rnd<bf16>(s1), -limit), limit);
                                o = a / (1.0f + __expf(-slope * a)) * (b + shift);
                            } else if (act == ES_ACT_RELU2) {
                                o = fmaxf(o, 0.f);
                                o *= o;
                            }
                            y[(size_t)(p0 + p) * out + r] = __float2bfloat16_rn(o);
                        }
                    }
                    here.i = 0;
                    here.item += gridDim.x;
                    start();
                }
            }
        }
    }
}

// A block has one unit and a tile of its rows: 16 gate rows and the up rows that go with them, or 32 rows. It finds the unit's pairs among `ids` and goes over
// its tile again for every 8 of them. The same arithmetic. Without `ids` it is the product with a matrix per head: unit h takes row h of every token.
template <bool GATED, bool SCALE>
__global__ void __launch_bounds__(ES_WARPS * 32, 2) expert_block_kernel(bf16* __restrict__ y, const bf16* x, const bf16* __restrict__ W,
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
    const int rows = e.gated ? 8 : 16, occ = in <= ES_SHORT_ROW ? 3 : 2;
    const long long tiles = (out + rows - 1) / rows, place = (long long)occ * ti_sm_count(), in_use = (long long)(e.pairs < units ? e.pairs : units) * tiles;
    // The list costs its making and a round trip before the first weights, and blocks that take tiles in turn a round more where a few tiles are left over: with
    // up to 1.3 tiles a block, a block per unit and tile takes less (us, block / list: 34 gated units of 1,024 x 2,048, 4 pairs 7.7 / 9.3, 6 pairs 11.9 / 10.9;
    // plain, 8 pairs 7.6 / 8.6, 12 pairs 10.4 / 9.9; 64 plain units of 264 x 1,000, 16 pairs 3.7 / 4.6; 16 of 128 x 512, 48 pairs 3.4 / 4.5, 96 pairs
    // 5.3 / 5.0: there units are gone over again), unless so few are needed that the list's blocks are all there is (16 units of 128 x 512, 1 pair 2.9 / 2.8;
    // 64 units of 1,408 x 4,096, 2 pairs 9.3 / 8.1, 4 pairs 10.9 / 12.5).
    const bool few = 10 * in_use <= 13 * place && e.pairs <= 64 && ((occ == 3 ? 3 : 1) * in_use > place || e.pairs > 32);
    if (e.ids == nullptr || few) {
        // Blocks of units that no pair chose leave at once but still take their turn, so with fewer pairs than units there is a row of blocks per pair.
        const int by_pair = e.ids != nullptr && e.pairs < units, block_rows = e.gated ? 16 : 32;
#define ES_LAUNCH(G, S)                                                                                                                              \
    ti_launch(expert_block_kernel<G, S>, dim3((out + block_rows - 1) / block_rows, by_pair ? e.pairs : units), dim3(ES_WARPS * 32), 0, stream, (bf16*)y, \
              (const bf16*)x, (const bf16*)W, e.ids, e.scores, e.pair_row, e.pairs, e.per_row, by_pair, out, in, e.act, e.limits, e.slope, e.shift, e.ahead)
        if (e.gated) { if (e.scores != nullptr) ES_LAUNCH(true, true); else ES_LAUNCH(true, false); }
        else { if (e.scores != nullptr) ES_LAUNCH(false, true); else ES_LAUNCH(false, false); }
#undef ES_LAUNCH
        return ti_check_launch("expert_stream");
    }
    // As many blocks as fit the SMs, fewer where even a unit per pair has fewer tiles.
    for (int p0 = 0; p0 < e.pairs; p0 += ES_MAX_PAIRS) {
        const int pairs = e.pairs - p0 < ES_MAX_PAIRS ? e.pairs - p0 : ES_MAX_PAIRS;
        const long long most = pairs * tiles;
        // Cells of the hash table of units, for more pairs than a warp lists: a power of two, one for every unit or two for every pair.
        int cells = pairs > 32 ? 64 : 0;
        while (cells > 0 && cells < units && cells < 2 * pairs) cells *= 2;
        const size_t lists = (size_t)cells * (sizeof(uint4) + sizeof(int)) + (size_t)pairs * (8 * sizeof(unsigned short) + sizeof(int) + (e.scores != nullptr ? sizeof(float) : 0));
        TI_REQUIRE(most <= 0x7fffffffLL, "expert_stream: %d pairs of %d rows", pairs, out);
#define ES_LAUNCH(G, S, B, OCC)                                                                                                                         \
    ti_launch(expert_stream_kernel<G, S, B, OCC>, dim3((unsigned)(most < OCC * ti_sm_count() ? most : OCC * ti_sm_count())), dim3(ES_WARPS * 32), lists, stream, \
              (bf16*)y, (const bf16*)x, (const bf16*)W, e.ids, e.scores, e.pair_row, p0, pairs, e.per_row, out, in, e.act, e.limits, e.slope, e.shift, \
              e.ahead && p0 == 0, cells)
#define ES_SHAPE(G, S) do { if (in <= ES_SHORT_ROW) ES_LAUNCH(G, S, 2, 3); else ES_LAUNCH(G, S, 4, 2); } while (0)
        if (e.gated) { if (e.scores != nullptr) ES_SHAPE(true, true); else ES_SHAPE(true, false); }
        else { if (e.scores != nullptr) ES_SHAPE(false, true); else ES_SHAPE(false, false); }
#undef ES_SHAPE
#undef ES_LAUNCH
    }
    return ti_check_launch("expert_stream");
}
