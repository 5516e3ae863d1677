// Plain matrix product y[n, out] = x[n, in] · W[out, in]ᵀ on the CUDA cores, for any sizes
// and either element type. Inputs are widened to 32-bit, every product is a 32-bit fused
// multiply-add (no tensor-core or reduced-precision mode), and the order in which an output
// element adds its k terms is fixed by `in` alone: a row's result is bit-identical in a step of
// one token and in a step of thousands. It is the 32-bit path's product and the fallback of
// the bfloat16 path for sizes the tensor-core kernel refuses.
//
// The order, common to both kernels below: k is cut into segments of GP_SEGMENT terms. In a
// segment the terms of even k and those of odd k are two chains of fused multiply-adds from zero
// in ascending order (the two halves of a packed fma.rn.f32x2, which takes one issue slot where two
// fused multiply-adds take two); a segment's sum is even + odd, and the segments' sums are added in
// ascending order. Terms beyond `in` are zeros. Short chains are what lets several warps share one
// output row's k (a single chain of 21,504 terms is 44 us of latency alone), and they lose less to
// rounding than one long chain: against 64-bit sums a product of k = 4,096 is 2.9e-7 off.
//
// AntoineBut/TileInfer.jl: weights stay [out, in] row-major, y = Wᵀx with 32-bit
// accumulation and one rounding (src/ops/reference.jl:23-26, src/ops/tile/linear.jl:12-13);
// the logits leave in 32-bit after that rounding (src/ops/tile/linear.jl:26).
#include <type_traits>
#include "common.cuh"
#include "mma_util.cuh"
#include "packed_f32.cuh"

#define GP_SEGMENT 512

#define TI_EPI_NONE 0
#define TI_EPI_XIELU 1
#define TI_EPI_F32_OUT 2   // round to the storage type, store 32-bit (logits)

// One output: rounded to the storage type, through the epilogue, stored.
template <typename T>
__device__ __forceinline__ void store_output(void* y, long long ldy, int r, int c, float sum, int epilogue, const XieluParams& act) {
    float v = rnd<T>(sum);
    if (epilogue == TI_EPI_XIELU) v = xielu_value<T>(v, act);
    if (epilogue >= TI_EPI_GELU_ERF) v = gelu_epilogue(v, epilogue);
    if (epilogue == TI_EPI_F32_OUT) ((float*)y)[(size_t)r * ldy + c] = v;
    else ((T*)y)[(size_t)r * ldy + c] = from_f32<T>(v);
}

// Both kernels stage k blocks of 128 bytes a row (32 floats or 64 bfloat16 values) as they lie in memory, in pieces of PIECE bytes by
// cp.async: 16 where every row of both operands starts on such a boundary, else 4, and single bfloat16 values, which no asynchronous
// copy takes, through registers (as floats: the conversions are then one per element and not one per use). Rows are 144 bytes apart in
// shared memory, so eight consecutive rows' 16-byte pieces fall into different banks. Four consecutive k of a row are one read: the
// packed multiply-add's operands are (k, k + 1) pairs of both sides, with no transposition and no duplicated element.
#define GT_ROW 144
#define GT_BYTES 128

template <typename T> struct Quad;                         // four consecutive k of a row as two packed pairs
template <> struct Quad<float> {
    f32x2 p[2];
    static constexpr int BYTES = 16;
    __device__ __forceinline__ void load(const unsigned char* s) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(s);
        p[0] = t.x; p[1] = t.y;
    }
};
template <> struct Quad<bf16> {
    f32x2 p[2];
    static constexpr int BYTES = 8;
    __device__ __forceinline__ void load(const unsigned char* s) {
        const uint2 t = *reinterpret_cast<const uint2*>(s);
        p[0] = pack2(__uint_as_float(t.x << 16), __uint_as_float(t.x & 0xffff0000u));
        p[1] = pack2(__uint_as_float(t.y << 16), __uint_as_float(t.y & 0xffff0000u));
    }
};

// 16 or 4 bytes to shared memory, or as many zero bytes (nothing is read from `src` then).
__device__ __forceinline__ void stage16(unsigned dst, const void* src, bool inside) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(inside ? 16 : 0));
}
__device__ __forceinline__ void stage4(unsigned dst, const void* src, bool inside) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(inside ? 4 : 0));
}
// What lies in shared memory: the elements themselves, but single bfloat16 values, which pass through registers anyway, as floats.
template <typename T, int PIECE> struct Staged {
    typedef T type;
    static constexpr int BYTES = PIECE;                    // of a piece there
};
template <> struct Staged<bf16, 2> {
    typedef float type;
    static constexpr int BYTES = 4;
};
// COUNT pieces of fewer than 16 bytes: `at(i, dst, src)` says where piece i goes and comes from and whether it lies inside the matrix. Of
// single elements up to MOST loads leave together. (16-byte pieces, whose loops stand in the kernels, need no such care.)
template <typename T, int PIECE, int COUNT, int MOST, typename F> __device__ __forceinline__ void stage_pieces(F at) {
    if constexpr (PIECE == 4) {
#pragma unroll
        for (int i = 0; i < COUNT; ++i) {
            unsigned char* dst; const T* src;
            const bool inside = at(i, dst, src);
            stage4(smem_u32(dst), src, inside);
        }
    } else {
        constexpr int AT_ONCE = COUNT <= MOST ? COUNT : 8;
        static_assert(COUNT % AT_ONCE == 0 && sizeof(T) == PIECE, "whole rounds of single elements");
#pragma unroll 1
        for (int i0 = 0; i0 < COUNT; i0 += AT_ONCE) {
            unsigned char* dst[AT_ONCE];
            T v[AT_ONCE];
#pragma unroll
            for (int u = 0; u < AT_ONCE; ++u) {
                const T* src;
                v[u] = at(i0 + u, dst[u], src) ? __ldcg(src) : from_f32<T>(0.f);
            }
#pragma unroll
            for (int u = 0; u < AT_ONCE; ++u) *reinterpret_cast<float*>(dst[u]) = to_f32(v[u]);
        }
    }
}

// Steps of up to 32 tokens: weights are streamed once. A block owns 16 * RPT output rows, its warps take the segments of k in
// turn, each with a ring of STAGES k blocks of its own (no block barrier but one per round of segments, where the round's sums
// are added up in ascending order). A lane owns RPT rows and half of the tokens (TPL each), so a row's quad is read once for
// TPL tokens and a token's quad, the same for 16 lanes, is one broadcast.
// What bounds it: weight bytes and, from 8 tokens on, shared-memory reads (a row's quad is read by one lane pair, a token's by 16
// lanes; neighbouring lanes share both, which halves the reads' passes). Measured at 8 tokens: up projection (21,504 x 4,096, 352
// MB) 77 us, 4.6 TB/s, where one chain per output and 16 bytes per token and thread took 220; down (4,096 x 21,504) 83 us (335).
template <typename T, int TPL, int RPT, int STAGES, int PIECE>
__global__ void __launch_bounds__(256) gemv_plain_stream_kernel(void* __restrict__ y, long long ldy, const T* x, long long ldx,
                                                                const T* __restrict__ W, int n, int out, int in, int epilogue,
                                                                XieluParams act) {
    extern __shared__ __align__(16) unsigned char gv_smem[];
    constexpr int ROWS = 16 * RPT, TOKENS = 2 * TPL;
    typedef typename Staged<T, PIECE>::type E;
    constexpr int IN_ROW = Staged<T, PIECE>::BYTES, PER_ROW = GT_BYTES / IN_ROW, VEC = PIECE / (int)sizeof(T);
    constexpr int BK = GT_BYTES / (int)sizeof(E), PER_SEG = GP_SEGMENT / BK;
    constexpr int STAGE = (ROWS + TOKENS) * GT_ROW;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
    const int row = lane & 15, half = lane >> 4;
    const int m0 = blockIdx.x * ROWS, t0 = blockIdx.y * TOKENS;
    n = min(TOKENS, n - t0);
    x += (size_t)t0 * ldx;
    unsigned char* ring = gv_smem + (size_t)warp * (STAGES * STAGE);
    float* sums = reinterpret_cast<float*>(gv_smem + (size_t)warps * (STAGES * STAGE));     // [2][warps][TOKENS][ROWS]
    float* total = sums + 2 * warps * TOKENS * ROWS;                                         // [TOKENS][ROWS]
    const int segments = (in + GP_SEGMENT - 1) / GP_SEGMENT, rounds = (segments + warps - 1) / warps;
    // This warp's k blocks: segments warp, warp + warps, ..., each of PER_SEG blocks but perhaps the last one of all.
    const int mine = warp < segments ? (segments - 1 - warp) / warps + 1 : 0;
    const int last_blocks = (in - (segments - 1) * GP_SEGMENT + BK - 1) / BK;
    const bool has_last = mine > 0 && (mine - 1) * warps + warp == segments - 1;
    const int tiles = mine * PER_SEG - (has_last ? PER_SEG - last_blocks : 0);
    auto k_of = [&](int tile) { return ((tile / PER_SEG) * warps + warp) * GP_SEGMENT + (tile % PER_SEG) * BK; };
    // A warp's pieces of a k block: piece i * 32 + lane, PER_ROW of them a row; a piece is inside its row or outside it (in % VEC == 0).
    auto issue_w = [&](int tile) {
        if (tile < tiles) {
            const int k0 = k_of(tile);
            unsigned char* s = ring + (tile % STAGES) * STAGE;
            if constexpr (PIECE == 16) {
#pragma unroll
                for (int i = 0; i < ROWS * 8 / 32; ++i) {
                    const int r = (i * 32 + lane) >> 3, c = lane & 7, k = k0 + c * VEC;
                    const bool inside = m0 + r < out && k < in;
                    stage16(smem_u32(s + r * GT_ROW + c * 16), inside ? W + (size_t)(m0 + r) * in + k : W, inside);
                }
            } else {
                stage_pieces<T, PIECE, ROWS * PER_ROW / 32, 16>([&](int i, unsigned char*& dst, const T*& src) {
                    const int r = (i * 32 + lane) / PER_ROW, c = (i * 32 + lane) % PER_ROW, k = k0 + c * VEC;
                    const bool inside = m0 + r < out && k < in;
                    dst = s + r * GT_ROW + c * IN_ROW;
                    src = inside ? W + (size_t)(m0 + r) * in + k : W;
                    return inside;
                });
            }
        }
    };
    auto issue_x = [&](int tile) {
        if (tile < tiles) {
            const int k0 = k_of(tile);
            unsigned char* s = ring + (tile % STAGES) * STAGE + ROWS * GT_ROW;
            if constexpr (PIECE == 16) {
#pragma unroll
                for (int i = 0; i < (TOKENS * 8 + 31) / 32; ++i) {
                    const int r = (i * 32 + lane) >> 3, c = lane & 7, k = k0 + c * VEC;
                    if (TOKENS * 8 < 32 && r >= TOKENS) continue;
                    const bool inside = r < n && k < in;
                    stage16(smem_u32(s + r * GT_ROW + c * 16), inside ? x + (size_t)r * ldx + k : x, inside);
                }
            } else {
                stage_pieces<T, PIECE, TOKENS * PER_ROW / 32, 16>([&](int i, unsigned char*& dst, const T*& src) {
                    const int r = (i * 32 + lane) / PER_ROW, c = (i * 32 + lane) % PER_ROW, k = k0 + c * VEC;
                    const bool inside = r < n && k < in;
                    dst = s + r * GT_ROW + c * IN_ROW;
                    src = inside ? x + (size_t)r * ldx + k : x;
                    return inside;
                });
            }
        }
    };
    // Weights do not depend on the kernel before: the first k blocks are on their way before the wait.
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) issue_w(s);
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) { issue_x(s); cp_async_commit(); }
    f32x2 acc[RPT][TPL];
    int tile = 0;
    for (int round = 0; round < rounds; ++round) {
#pragma unroll
        for (int q = 0; q < RPT; ++q)
#pragma unroll
            for (int j = 0; j < TPL; ++j) acc[q][j] = 0ull;
        const int end = min(tiles, (round + 1) * PER_SEG);
        for (; tile < end; ++tile) {
            cp_async_wait<STAGES - 2>();
            __syncwarp();                                   // every lane's copies of this k block have landed, and the stage refilled below is no longer read
            issue_w(tile + STAGES - 1);
            issue_x(tile + STAGES - 1);
            cp_async_commit();
            const unsigned char* s = ring + (tile % STAGES) * STAGE;
            const unsigned char* ws = s + row * GT_ROW;
            const unsigned char* xs = s + (ROWS + half) * GT_ROW;
#pragma unroll
            for (int c = 0; c < BK / 4; ++c) {
                Quad<E> w[RPT];
#pragma unroll
                for (int q = 0; q < RPT; ++q) w[q].load(ws + q * 16 * GT_ROW + c * Quad<E>::BYTES);
#pragma unroll
                for (int j = 0; j < TPL; ++j) {
                    Quad<E> v;
                    v.load(xs + 2 * j * GT_ROW + c * Quad<E>::BYTES);
#pragma unroll
                    for (int q = 0; q < RPT; ++q) acc[q][j] = fma2(v.p[1], w[q].p[1], fma2(v.p[0], w[q].p[0], acc[q][j]));
                }
            }
        }
        if (round < mine) {
            float* to = sums + ((round & 1) * warps + warp) * (TOKENS * ROWS);
#pragma unroll
            for (int q = 0; q < RPT; ++q)
#pragma unroll
                for (int j = 0; j < TPL; ++j) {
                    float e, o;
                    unpack2(acc[q][j], e, o);
                    to[(2 * j + half) * ROWS + q * 16 + row] = e + o;
                }
        }
        __syncthreads();                                    // the other buffer is written in the next round, after every thread has read it
        const int here = min(warps, segments - round * warps);
        for (int i = tid; i < n * ROWS; i += blockDim.x) {
            const float* from = sums + (round & 1) * warps * (TOKENS * ROWS) + i;
            float t = round == 0 ? from[0] : total[i] + from[0];
            for (int w = 1; w < here; ++w) t += from[w * (TOKENS * ROWS)];
            if (round + 1 < rounds) total[i] = t;
            else if (m0 + i % ROWS < out) store_output<T>(y, ldy, t0 + i / ROWS, m0 + i % ROWS, t, epilogue, act);
        }
    }
    cp_async_wait<0>();
}

// Steps of more tokens: tiles of 16 TI tokens x 16 TJ features, 256 threads with TI x TJ outputs each, k blocks in a ring of
// shared-memory stages. A thread's tokens and features are 16 apart, so the lanes of a warp (8 features x 4 tokens) read
// consecutive rows. The sums of the segments before the current one wait in shared memory.
// What bounds it: the FMA units, at 0.7 of their rate at the clock that a long run of them settles at (ncu: 1.6 GHz; a
// thread's fragments come in 16-byte reads of which every second or fourth lane's is its own). 512 tokens x 21,504 x 4,096: 2,230
// us, 40 TFLOP/s; tiles staged with k outermost, 8 x 8 outputs a thread and single multiply-adds took 4,500.
// (Single elements are not on their way while a k block is worked on, so two or three blocks share an SM; a lower bound of one block for
// the others makes the compiler spend more registers: 512 tokens of the 32-bit model at 8B sizes 0.4 % longer.)
// bfloat16 in the largest tiles is widened once, into floats in shared memory, instead of by each of the 16 threads that read a row: 512 /
// 1,000 tokens x 21,504 x 4,096 2,288 / 4,578 us (2,574 / 5,156 without). Smaller tiles would lose the blocks that share an SM to the floats' room.
template <typename T, int TI, int TJ, int PIECE> struct Widens { static constexpr bool value = sizeof(typename Staged<T, PIECE>::type) == 2 && TI * TJ >= 64; };
#define GT_WIDE_ROW (2 * GT_BYTES + 16)
template <typename T, int TI, int TJ, int STAGES, int PIECE>
__global__ void __launch_bounds__(256, PIECE == 2 ? (TI * TJ <= 16 ? 3 : 2) : 0) gemm_plain_tile_kernel(void* __restrict__ y, long long ldy, const T* x, long long ldx,
                                                             const T* __restrict__ W, int n, int out, int in, int epilogue,
                                                             XieluParams act) {
    extern __shared__ __align__(16) unsigned char gt_smem[];
    constexpr int TM = 16 * TI, TN = 16 * TJ;
    typedef typename Staged<T, PIECE>::type E;
    constexpr bool WIDE = Widens<T, TI, TJ, PIECE>::value;
    typedef std::conditional_t<WIDE, float, E> F;           // what the products are taken of
    constexpr int IN_ROW = Staged<T, PIECE>::BYTES, PER_ROW = GT_BYTES / IN_ROW, VEC = PIECE / (int)sizeof(T);
    constexpr int BK = GT_BYTES / (int)sizeof(E), PER_SEG = GP_SEGMENT / BK;
    constexpr int STAGE = (TM + TN) * GT_ROW, STEP = 256 / PER_ROW;            // staging: STEP rows at a time
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int tx = (lane & 7) + 8 * (warp & 1), ty = (lane >> 3) + 4 * (warp >> 1);
    float* total = reinterpret_cast<float*>(gt_smem + STAGES * STAGE);        // [TI * TJ][256]
    const int blocks = (in + BK - 1) / BK;
    const int lrow = tid / PER_ROW, lc = tid % PER_ROW;
    auto issue = [&](int b, bool weights, bool tokens) {
        if (b < blocks) {
            unsigned char* s = gt_smem + (b % STAGES) * STAGE + lrow * GT_ROW + lc * IN_ROW;
            const int k = b * BK + lc * VEC;
            const bool k_ok = k < in;
            if constexpr (PIECE == 16) {
                if (tokens) {
#pragma unroll
                    for (int i = 0; i < TM / 32; ++i) {
                        const int r = m0 + lrow + 32 * i;
                        const bool inside = k_ok && r < n;
                        stage16(smem_u32(s + 32 * i * GT_ROW), inside ? x + (size_t)r * ldx + k : x, inside);
                    }
                }
                if (weights) {
#pragma unroll
                    for (int i = 0; i < TN / 32; ++i) {
                        const int c = n0 + lrow + 32 * i;
                        const bool inside = k_ok && c < out;
                        stage16(smem_u32(s + (TM + 32 * i) * GT_ROW), inside ? W + (size_t)c * in + k : W, inside);
                    }
                }
            } else {
                if (tokens)
                    stage_pieces<T, PIECE, TM / STEP, 8>([&](int i, unsigned char*& dst, const T*& src) {
                        const int r = m0 + lrow + STEP * i;
                        const bool inside = k_ok && r < n;
                        dst = s + STEP * i * GT_ROW;
                        src = inside ? x + (size_t)r * ldx + k : x;
                        return inside;
                    });
                if (weights)
                    stage_pieces<T, PIECE, TN / STEP, 8>([&](int i, unsigned char*& dst, const T*& src) {
                        const int c = n0 + lrow + STEP * i;
                        const bool inside = k_ok && c < out;
                        dst = s + (TM + STEP * i) * GT_ROW;
                        src = inside ? W + (size_t)c * in + k : W;
                        return inside;
                    });
            }
        }
    };
#pragma unroll
    for (int b = 0; b < STAGES - 1; ++b) issue(b, true, false);
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int b = 0; b < STAGES - 1; ++b) { issue(b, false, true); cp_async_commit(); }
    f32x2 acc[TI][TJ];
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j) acc[i][j] = 0ull;
    for (int b = 0; b < blocks; ++b) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();                                    // this k block has landed, and the stage refilled below is no longer read
        issue(b + STAGES - 1, true, true);
        cp_async_commit();
        const unsigned char* from = gt_smem + (b % STAGES) * STAGE;
        if constexpr (WIDE) {
            unsigned char* wide = gt_smem + STAGES * STAGE + TI * TJ * 256 * sizeof(float);
#pragma unroll
            for (int i = 0; i < (TM + TN) / 16; ++i) {
                const int r = (tid >> 4) + 16 * i, c = tid & 15;
                const uint2 t = *reinterpret_cast<const uint2*>(from + r * GT_ROW + c * 8);
                *reinterpret_cast<uint4*>(wide + r * GT_WIDE_ROW + c * 16) = make_uint4(t.x << 16, t.x & 0xffff0000u, t.y << 16, t.y & 0xffff0000u);
            }
            __syncthreads();
            from = wide;
        }
        constexpr int ROW = WIDE ? GT_WIDE_ROW : GT_ROW;
        const unsigned char* as = from + ty * ROW;
        const unsigned char* bs = from + (TM + tx) * ROW;
#pragma unroll
        for (int c = 0; c < BK / 4; ++c) {
            Quad<F> w[TJ];
#pragma unroll
            for (int j = 0; j < TJ; ++j) w[j].load(bs + j * 16 * ROW + c * Quad<F>::BYTES);
#pragma unroll
            for (int i = 0; i < TI; ++i) {
                Quad<F> v;
                v.load(as + i * 16 * ROW + c * Quad<F>::BYTES);
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int j = 0; j < TJ; ++j) acc[i][j] = fma2(v.p[h], w[j].p[h], acc[i][j]);
            }
        }
        if ((b + 1) % PER_SEG == 0 && b + 1 < blocks) {     // a segment ends, and more follow
#pragma unroll
            for (int i = 0; i < TI; ++i)
#pragma unroll
                for (int j = 0; j < TJ; ++j) {
                    float e, o;
                    unpack2(acc[i][j], e, o);
                    float* t = total + (i * TJ + j) * 256 + tid;
                    *t = b < PER_SEG ? e + o : *t + (e + o);
                    acc[i][j] = 0ull;
                }
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < TI; ++i) {
        const int r = m0 + ty + 16 * i;
#pragma unroll
        for (int j = 0; j < TJ; ++j) {
            const int c = n0 + tx + 16 * j;
            float e, o;
            unpack2(acc[i][j], e, o);
            const float s = blocks > PER_SEG ? total[(i * TJ + j) * 256 + tid] + (e + o) : e + o;
            if (r < n && c < out) store_output<T>(y, ldy, r, c, s, epilogue, act);
        }
    }
}

template <typename K> static cudaError_t allow_smem(K kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <typename T, int TPL, int RPT, int STAGES, int PIECE>
static int launch_stream(void* y, long long ldy, const T* x, long long ldx, const T* W, int n, int out, int in, int epilogue,
                         const XieluParams& act, cudaStream_t stream) {
    constexpr int ROWS = 16 * RPT, MAX_WARPS = 8;
    constexpr size_t PER_WARP = (size_t)STAGES * (ROWS + 2 * TPL) * GT_ROW + 2 * 2 * TPL * ROWS * sizeof(float);
    constexpr size_t TOTAL = 2 * TPL * ROWS * sizeof(float);
    static const cudaError_t allowed = allow_smem(gemv_plain_stream_kernel<T, TPL, RPT, STAGES, PIECE>, MAX_WARPS * PER_WARP + TOTAL);
    if (allowed != cudaSuccess) return ti_fail("gemv_plain: %s", cudaGetErrorString(allowed));
    const int segments = (in + GP_SEGMENT - 1) / GP_SEGMENT, rounds = (segments + MAX_WARPS - 1) / MAX_WARPS;
    const int warps = (segments + rounds - 1) / rounds;                        // as few as the rounds need: the last round is full
    ti_launch(gemv_plain_stream_kernel<T, TPL, RPT, STAGES, PIECE>, dim3((out + ROWS - 1) / ROWS, (n + 2 * TPL - 1) / (2 * TPL)), dim3(32 * warps), warps * PER_WARP + TOTAL, stream, y,
              ldy, x, ldx, W, n, out, in, epilogue, act);
    return ti_check_launch("gemv_plain");
}

template <typename T, int TI, int TJ, int STAGES, int PIECE>
static int launch_tile(void* y, long long ldy, const T* x, long long ldx, const T* W, int n, int out, int in, int epilogue,
                       const XieluParams& act, cudaStream_t stream) {
    constexpr size_t SMEM = (size_t)STAGES * 16 * (TI + TJ) * GT_ROW + (size_t)TI * TJ * 256 * sizeof(float) +
                            (Widens<T, TI, TJ, PIECE>::value ? (size_t)16 * (TI + TJ) * GT_WIDE_ROW : 0);
    static const cudaError_t allowed = allow_smem(gemm_plain_tile_kernel<T, TI, TJ, STAGES, PIECE>, SMEM);
    if (allowed != cudaSuccess) return ti_fail("gemm_plain: %s", cudaGetErrorString(allowed));
    const dim3 grid((out + 16 * TJ - 1) / (16 * TJ), (n + 16 * TI - 1) / (16 * TI));
    TI_REQUIRE(grid.y <= 65535, "gemm: too many rows (%d) for one launch", n);
    ti_launch(gemm_plain_tile_kernel<T, TI, TJ, STAGES, PIECE>, grid, dim3(256), SMEM, stream, y, ldy, x, ldx, W, n, out, in, epilogue, act);
    return ti_check_launch("gemm_plain_tile");
}

// Tokens x features per thread of the tile kernel: the shape whose rounds of tiles over the SMs take the least time, by what a
// round and a launch's first and last tile cost (in units of k, from sweeps of 64 to 2,048 tokens x 2,048 to 21,504 features at k =
// 4,096: microseconds per round 447 / 235 / 132 / 92, and 0 / 15 / 23 / 22 once; 512 tokens x 4,096 features take 449 / 471 / 518 / 660
// us, 128 x 4,096 take 448 / 255 / 155 / 260, 512 x 6,144 take 893 / 691 / 771 / 1,027). It does not ask for k: over k = 512 to 21,504,
// 70 to 1,024 tokens and 1,024 to 21,504 features the choice takes 1.3 % longer than the best shape on average (3.2 % at k = 512, 0.0 at
// 21,504; 20 % at worst, 1,024 tokens x 21,504 x 512), with the second cost weighed by k 1.9 %. The sums do not depend on the shape.
struct TileShape { int ti, tj; float round, once; };
static const TileShape TILE_SHAPES[] = {{8, 8, 447.f, 0.f}, {8, 4, 235.f, 15.f}, {4, 4, 132.f, 23.f}, {2, 4, 92.f, 22.f}};

extern "C" int ti_gemm_plain_shape(int n, int out, int sms) {
    int best = 0;
    float least = 0.f;
    for (int s = 0; s < 4; ++s) {
        const TileShape& t = TILE_SHAPES[s];
        const long long tiles = (long long)((n + 16 * t.ti - 1) / (16 * t.ti)) * ((out + 16 * t.tj - 1) / (16 * t.tj));
        const float time = (float)((tiles + sms - 1) / sms) * t.round + t.once;
        if (s == 0 || time < least) { best = s; least = time; }
    }
    return best;
}

// Up to 64 tokens the weight-streaming kernel is the faster one (two token groups of 32 read the weights twice, the second time from
// L2): 64 tokens x 4,096 / 21,504 features of k = 4,096 take 74 / 355 us against 115 / 402 in tiles; at 100 tokens the two are level.
#define GT_STREAM_TOKENS 64

template <typename T, int PIECE>
static int launch_product(void* y, long long ldy, const T* x, long long ldx, const T* W, int n, int out, int in, int epilogue,
                          const XieluParams& act, cudaStream_t stream) {
#define GT_ARGS y, ldy, x, ldx, W, n, out, in, epilogue, act, stream
    if (n <= GT_STREAM_TOKENS) {
        // One segment of k is one warp a block, whose chain is the time: its tokens are shared out, four to a block, while the blocks take
        // no more than about three rounds, of 1 KB rows (32-bit, 32 / 64 tokens: 512 x 512 22.5 / 22.5 -> 6.8 / 7.1 us, 300 x 64 6.8 / 6.9 -> 2.7 / 2.6,
        // but 8,192 x 512 24.5 -> 25.2 with 32).
        const long long row = in * (long long)sizeof(T) < 1024 ? 1024 : in * (long long)sizeof(T), fours = (long long)((out + 15) / 16) * ((n + 3) / 4);
        if (in <= GP_SEGMENT && n > 4 && fours * row <= 42LL * 1024 * ti_sm_count()) return launch_stream<T, 2, 1, PIECE == 16 ? 5 : 4, PIECE>(GT_ARGS);
        if constexpr (PIECE == 16) {
            // 32 rows a block halve what is read of the tokens, where that leaves blocks for six tenths of the SMs (8 tokens: 4,096
            // rows 17.8 us against 24.5 with 16 rows a block, 2,048 rows of k = 2,048 13.8 against 10.7). More blocks than SMs take two
            // stages, so that two blocks fit an SM (6,144 rows: 26.9 us against 33.0); fewer take a deeper ring (4,096 rows x 21,504: 83 us against 98).
            const int sms = ti_sm_count(), groups = (n + 31) / 32, blocks = (out + 31) / 32 * groups;
            const bool tall = 5 * blocks >= 3 * sms, many = blocks > sms;
            if (n <= 2) return !tall ? launch_stream<T, 1, 1, 6, 16>(GT_ARGS) : many ? launch_stream<T, 1, 2, 2, 16>(GT_ARGS) : launch_stream<T, 1, 2, 5, 16>(GT_ARGS);
            if (n <= 4) return !tall ? launch_stream<T, 2, 1, 5, 16>(GT_ARGS) : many ? launch_stream<T, 2, 2, 2, 16>(GT_ARGS) : launch_stream<T, 2, 2, 4, 16>(GT_ARGS);
            if (n <= 8) return !tall ? launch_stream<T, 4, 1, 5, 16>(GT_ARGS) : many ? launch_stream<T, 4, 2, 2, 16>(GT_ARGS) : launch_stream<T, 4, 2, 4, 16>(GT_ARGS);
            if (n <= 16) return tall ? launch_stream<T, 8, 2, 3, 16>(GT_ARGS) : launch_stream<T, 8, 1, 4, 16>(GT_ARGS);
            return tall ? launch_stream<T, 16, 2, 2, 16>(GT_ARGS) : launch_stream<T, 16, 1, 3, 16>(GT_ARGS);
        } else {
            // Other rows, one set of blocks (microseconds; in brackets with blocks of 16 rows or tiles of 64 x 64 that staged element by element, 8-byte
            // loads and tiles of 128 x 128 for bfloat16 rows of 4 modulo 8): bfloat16, 8 tokens x 4,096 x 4,100 35 (195), 512 tokens 536 (763);
            // x 4,099 58 (199), 512 tokens 651 (865), 700 tokens 844 (879); 32-bit x 4,099, 8 tokens 48 (253), 512 tokens 510 (859).
            if (n <= 2) return launch_stream<T, 1, 1, 4, PIECE>(GT_ARGS);
            if (n <= 8) return launch_stream<T, 4, 1, 4, PIECE>(GT_ARGS);
            if (n <= 16) return launch_stream<T, 8, 1, 4, PIECE>(GT_ARGS);
            return launch_stream<T, 16, 2, 2, PIECE>(GT_ARGS);
        }
    }
    const int shape = ti_gemm_plain_shape(n, out, ti_sm_count());
    if constexpr (PIECE == 2) {                            // (8 x 8 outputs take longer at every size)
        if (shape <= 1) return launch_tile<T, 8, 4, 2, 2>(GT_ARGS);
        if (shape == 2) return launch_tile<T, 4, 4, 2, 2>(GT_ARGS);
        return launch_tile<T, 2, 4, 2, 2>(GT_ARGS);
    } else {
        if (shape == 0) return launch_tile<T, 8, 8, 2, PIECE>(GT_ARGS);
        if (shape == 1) return launch_tile<T, 8, 4, 2, PIECE>(GT_ARGS);
        if (shape == 2) return launch_tile<T, 4, 4, 3, PIECE>(GT_ARGS);
        return launch_tile<T, 2, 4, 4, PIECE>(GT_ARGS);
    }
#undef GT_ARGS
}

extern "C" int ti_gemm_plain(void* y, long long ldy, const void* x, long long ldx, const void* W, int n, int out, int in,
                             int epilogue, float alpha_p, float alpha_n, float beta, float eps, int dtype,
                             cudaStream_t stream) {
    if (n == 0) return 0;
    TI_REQUIRE(n > 0 && out > 0 && in > 0, "gemm: bad sizes n=%d out=%d in=%d", n, out, in);
    TI_REQUIRE((epilogue >= 0 && epilogue <= 2) || (epilogue >= TI_EPI_GELU_ERF && epilogue <= TI_EPI_LAST), "gemm: unknown epilogue %d", epilogue);
    XieluParams act{alpha_p, alpha_n, beta, eps};
    // The widest piece on whose boundaries all rows of both operands start.
    const unsigned long long size = dtype == TI_F32 ? 4 : 2;
    const unsigned long long off = (unsigned long long)in * size | (unsigned long long)ldx * size | (uintptr_t)x | (uintptr_t)W;
#define GP_PRODUCT(T, PIECE) launch_product<T, PIECE>(y, ldy, (const T*)x, ldx, (const T*)W, n, out, in, epilogue, act, stream)
    if (dtype == TI_F32) return off % 16 == 0 ? GP_PRODUCT(float, 16) : GP_PRODUCT(float, 4);
    if (dtype == TI_BF16) return off % 16 == 0 ? GP_PRODUCT(bf16, 16) : off % 4 == 0 ? GP_PRODUCT(bf16, 4) : GP_PRODUCT(bf16, 2);
#undef GP_PRODUCT
    return ti_fail("unknown element type code %d", dtype);
}
