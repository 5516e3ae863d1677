// Two recurrences whose only memory is a matrix state per (sequence, head), kept in 32-bit, and the small kernels around them.
//
//   decay scan (time mixing with a decay per key channel that depends on the token, and a bonus for the current token):
//       o_t = (S + diag(u) k_t v_t^T)^T r_t ;   S <- diag(w_t) S + k_t v_t^T ;   w_t = exp(-exp(d_t + w0))
//   delta scan (gated delta rule):
//       S <- g_t S ;  e = beta_t (v_t - S^T k_t) ;  S <- S + k_t e^T ;  o_t = S^T q_t
//       beta_t = sigmoid(b_t),  g_t = exp(-exp(A_log) * softplus(a_t + dt_bias))
//
// S is [dim][vdim] (key rows, value columns). A warp owns CB value columns of one (sequence, head) with all their key rows: G = 32 / CB groups
// of R rows a column, a lane has the rows of one group in registers (G is the least power of two that holds the key size). What a token
// reads out of the state is added up over a column's groups by shuffles, so the warps of a block share nothing but the staged inputs. (The decay
// scan of keys above 64 shares a column's rows out among warps instead: see there.) A step's tokens are walked in order from the state that earlier
// steps left, in batches of RS_BATCH tokens staged in shared memory. The groups' sums are added in ascending order everywhere, in the one-token
// kernels too, and only those of groups that have rows of the key, so a result depends on the token's place in its sequence alone, not on the
// batch or on how the prompt was cut.
#include "mma_util.cuh"
#include "packed_f32.cuh"

#define RS_ROWS 16                 // key rows of a lane of the delta scan
#define RS_BATCH 16
#define RS_MAX_KEY 256

__device__ __forceinline__ float rs_silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float rs_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// Where the RUN tokens from `first` on lie: every token's sequence's first token of the step, that sequence's slot and the one after its last token.
// Asked by a whole block ahead of the wait (the step's tables were uploaded before its first kernel). One warp looks, a lane per token:
// thousands of warps that each go through the same few words queue for them at L2. Where the step has as many sequences as tokens, token t is
// sequence t's only one, unless some sequence has none.
template <int RUN> struct TokenRun {
    int t0[RUN], t1[RUN], slot[RUN];
    __device__ __forceinline__ void find(const int* cu, const int* slots, int B, int n, int first) {
        if (threadIdx.x < RUN && first + (int)threadIdx.x < n) {
            const int i = threadIdx.x, t = first + i;
            bool found = false;
            if (n == B) {
                t0[i] = __ldcg(cu + t);
                t1[i] = __ldcg(cu + t + 1);
                slot[i] = __ldcg(slots + t);
                found = t0[i] == t && t1[i] == t + 1;
            }
            if (!found) {
                int lo = 0, hi = B - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (__ldcg(cu + mid) <= t) lo = mid; else hi = mid - 1;
                }
                t0[i] = __ldcg(cu + lo);
                t1[i] = __ldcg(cu + lo + 1);
                slot[i] = __ldcg(slots + lo);
            }
        }
        __syncthreads();
    }
};

// ------------------------------------------------------------------------------------------------ what both scans share
// The launch of a scan: G groups of R rows hold a key of D elements; a block has `warps` warps of 32 / G columns.
struct ScanShape { int groups, warps, through; };
// Blocks of `most` warps share the staged rows of a head; where so few leave most SMs idle, smaller ones (a token's time is its warp's own
// chain, and staging takes a small part of it).
static ScanShape scan_shape(int rows, int D, int cols, long long heads, int most, int least) {
    ScanShape s = {1, most, 0};
    while (s.groups * rows < D) s.groups *= 2;
    auto blocks = [&] { const int per = s.warps * (32 / s.groups); return (cols + per - 1) / per * heads; };
    if (blocks() > 4LL * ti_sm_count())                     // so many that warps without a column, which help with staging, take room from others
        while (s.warps > 1 && s.warps / 2 * (32 / s.groups) >= cols) s.warps /= 2;
    while (s.warps > least && 2 * blocks() < ti_sm_count()) s.warps /= 2;
    s.through = s.groups >= 8 && blocks() > 4LL * ti_sm_count();
    return s;
}
// The sum over the groups of a column, whose lanes are 32 / G apart, in every lane of it; groups without rows of the key give zero. (One shuffle a
// group: they do not wait for one another as a tree's would, and their additions in a row take no longer than its round trips.)
template <int G> __device__ __forceinline__ float groups_sum(float v) {
    const int first = (threadIdx.x & 31) % (32 / G);
    float t[G], total = 0.f;
#pragma unroll
    for (int i = 0; i < G; ++i) t[i] = __shfl_sync(0xffffffffu, v, first + i * (32 / G));
#pragma unroll
    for (int i = 0; i < G; ++i) total += t[i];
    return total;
}
// The same of the first `used` groups' values, which lie `stride` apart.
__device__ __forceinline__ float groups_sum(const float* from, int stride, int used) {
    float total = 0.f;
    for (int i = 0; i < used; ++i) total += from[i * stride];
    return total;
}
// All G of them.
template <int G> __device__ __forceinline__ float groups_sum(const float* from, int stride) {
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < G; ++i) total += from[i * stride];
    return total;
}
// A staged row: a group's rows lie four floats further apart than they are many, so that a warp's 16-byte reads fall into different banks.
template <int R> __device__ __forceinline__ int staged_at(int d) { return d + d / R * 4; }
template <int R> __device__ __forceinline__ void read_rows(f32x2 (&to)[R / 2], const float* from) {
#pragma unroll
    for (int r = 0; r < R; r += 4) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(from + r);
        to[r / 2] = t.x; to[r / 2 + 1] = t.y;
    }
}
__device__ __forceinline__ float rows_sum(f32x2 a, f32x2 b) {
    float p0, p1, p2, p3;
    unpack2(a, p0, p1);
    unpack2(b, p2, p3);
    return (p0 + p1) + (p2 + p3);
}
// A load that stays where it is written (the compiler would move it down to its use, past the work that hides its latency).
__device__ __forceinline__ float load_now(const float* p) {
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bf16 load_now(const bf16* p) {
    unsigned short v;
    asm volatile("ld.global.cg.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
    return __ushort_as_bfloat16(v);
}
__device__ __forceinline__ void copy4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src));
}
// A block's columns of the state. Where many blocks have few tokens each and a warp few columns (`through`), they pass through shared memory: a warp's
// own columns are 8 or 16 bytes of a row, the block's a whole sector or more (64 sequences of two tokens, straight into the lanes / through: 16 heads of
// 256 x 256 726 / 301 us, 32 of 128 x 128 225 / 144). A group's rows lie CB floats further apart than they are long, so that a warp's reads fall into
// different banks. A thread carries R elements.
template <int R, int G> struct StateTile {
    static constexpr int CB = 32 / G;
    float* area;                                   // [R * G][cols] and the gaps: 32 R floats a warp and 32 more
    float* S;                                      // [D][V], from the block's first column on
    int cols_log2, D, V, cols_left;
    __device__ __forceinline__ int place(int row, int c) const { return (row << cols_log2) + row / R * CB + c; }
    __device__ __forceinline__ void ask(float (&t)[R]) const {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int e = threadIdx.x + j * blockDim.x, row = e >> cols_log2, c = e & ((1 << cols_log2) - 1);
            t[j] = row < D && c < cols_left ? load_now(S + (size_t)row * V + c) : 0.f;
        }
    }
    __device__ __forceinline__ void lay(const float (&t)[R]) const {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int e = threadIdx.x + j * blockDim.x;
            area[place(e >> cols_log2, e & ((1 << cols_log2) - 1))] = t[j];
        }
    }
    __device__ __forceinline__ void take(f32x2 (&s)[R / 2], int row0, int cl) const {
#pragma unroll
        for (int r = 0; r < R; r += 2) s[r / 2] = pack2(area[place(row0 + r, cl)], area[place(row0 + r + 1, cl)]);
    }
    __device__ __forceinline__ void give(const f32x2 (&s)[R / 2], int row0, int cl) const {
#pragma unroll
        for (int r = 0; r < R; r += 2) unpack2(s[r / 2], area[place(row0 + r, cl)], area[place(row0 + r + 1, cl)]);
    }
    __device__ __forceinline__ void leave() const {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int e = threadIdx.x + j * blockDim.x, row = e >> cols_log2, c = e & ((1 << cols_log2) - 1);
            if (row < D && c < cols_left) S[(size_t)row * V + c] = area[place(row, c)];
        }
    }
    // Straight between global memory and the lanes.
    __device__ __forceinline__ void load(f32x2 (&s)[R / 2], int row0, int cl) const {
#pragma unroll
        for (int r = 0; r < R; r += 2)
            s[r / 2] = pack2(row0 + r < D && cl < cols_left ? __ldcg(S + (size_t)(row0 + r) * V + cl) : 0.f,
                             row0 + r + 1 < D && cl < cols_left ? __ldcg(S + (size_t)(row0 + r + 1) * V + cl) : 0.f);
    }
    __device__ __forceinline__ void store(const f32x2 (&s)[R / 2], int row0, int cl) const {
#pragma unroll
        for (int r = 0; r < R; r += 2) {
            float lo, hi;
            unpack2(s[r / 2], lo, hi);
            if (row0 + r < D && cl < cols_left) S[(size_t)(row0 + r) * V + cl] = lo;
            if (row0 + r + 1 < D && cl < cols_left) S[(size_t)(row0 + r + 1) * V + cl] = hi;
        }
    }
};

// ------------------------------------------------------------------------------------------------ decay scan
// rkv [n][ld] of T: r at r_off, k at k_off, v at v_off, heads of `D` side by side; dlog [n][H * D] float: the decay's logit
// before w0 [H * D] is added; u [H * D] float; state rows `state_stride` floats apart, a head's matrix at h * D * D.
// The next batch's rows are fetched into registers before this batch is worked on and laid into the other half of the staging buffers
// after it, so their latency hides behind the recurrence; one barrier per batch. A thread stages one channel of tokens STEP apart.
// What bounds it: instructions issued, a warp or two per scheduler, a third of them staging. The lanes' sums of a token meet in shared memory once
// per batch. A prompt of 1,500 tokens (with 333, 64 and 7 beside it), 32 heads of 64, alone 373 -> 270 us, against blocks of 32 columns
// whose warps shared a column's rows; 2,048 tokens 406 -> 274, 8 heads 799 -> 355.
template <typename T, int R, int G, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, WARPS == 4 ? 4 : 1) decay_scan_kernel(float* __restrict__ o, const T* rkv, long long ld, int r_off, int k_off, int v_off, const float* dlog,
                                  const float* __restrict__ w0, const float* __restrict__ u, float* state, long long state_stride,
                                  const int* cu_seqlens, const int* seq_slots, int H, int D, int through) {
    extern __shared__ __align__(16) float sm[];
    constexpr int CB = 32 / G, Dp = R * G, ROW = G * (R + 4), THREADS = 32 * WARPS, COLS = WARPS * CB;
    constexpr int AT_ONCE = 4;                                                             // tokens whose reads are in flight
    constexpr int CHANNELS = Dp < THREADS ? Dp : THREADS, STEP = THREADS / CHANNELS;       // threads of a row, rows at a time
    constexpr int PER = RS_BATCH / STEP, PASSES = Dp / CHANNELS;                           // rows of a thread's channel, channels of a thread
    constexpr int PV = (RS_BATCH * COLS + THREADS - 1) / THREADS;
    float* sr = sm;                               // [2][RS_BATCH][ROW]
    float* sk = sr + 2 * RS_BATCH * ROW;
    float* sw = sk + 2 * RS_BATCH * ROW;
    float* sv = sw + 2 * RS_BATCH * ROW;          // [2][RS_BATCH][COLS]
    float* so = sv + 2 * RS_BATCH * COLS;         // [WARPS][RS_BATCH][32], and before and after the tokens the state
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cl = warp * CB + lane % CB, sub = lane / CB;
    const int col0 = blockIdx.x * COLS, h = blockIdx.y, b = blockIdx.z, row0 = sub * R, used = (D + R - 1) / R;
    const int t0 = __ldcg(cu_seqlens + b), t1 = __ldcg(cu_seqlens + b + 1);
    const StateTile<R, G> tile = {so, state + (size_t)__ldcg(seq_slots + b) * state_stride + (size_t)h * D * D + col0, __ffs(COLS) - 1, D, D, D - col0};
    const int ch = threadIdx.x % CHANNELS, i0 = threadIdx.x / CHANNELS;
    float shift[PASSES];
#pragma unroll
    for (int q = 0; q < PASSES; ++q) shift[q] = ch + q * CHANNELS < D ? w0[h * D + ch + q * CHANNELS] : 0.f;
    f32x2 bonus[R / 2];
#pragma unroll
    for (int r = 0; r < R; r += 2)
        bonus[r / 2] = pack2(row0 + r < D ? u[h * D + row0 + r] : 0.f, row0 + r + 1 < D ? u[h * D + row0 + r + 1] : 0.f);
    pdl_enter();
    f32x2 s[R / 2];
    float asked[R];
    if (through) tile.ask(asked); else tile.load(s, row0, cl);
    // Fetched values stay as they were loaded (no conversion, no branch): a use right behind a load would make the warp wait for it,
    // one round trip to memory per load instead of one per batch. Rows outside the batch or the head read a valid address and
    // are zeroed when they are laid into shared memory.
    T fr[PER], fk[PER], fv[PV];
    float fd[PER];
    auto fetch = [&](int base, int count, int q) {
        const int d = min(ch + q * CHANNELS, D - 1);
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const size_t t = base + min(i0 + j * STEP, count - 1);
            fr[j] = load_now(rkv + t * ld + (r_off + h * D + d));
            fk[j] = load_now(rkv + t * ld + (k_off + h * D + d));
            fd[j] = load_now(dlog + t * (H * D) + (h * D + d));
        }
    };
    auto stash = [&](int buf, int count, int q) {
        const bool in_head = ch + q * CHANNELS < D;
        const int to = buf * RS_BATCH * ROW + i0 * ROW + staged_at<R>(ch + q * CHANNELS);
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const bool in = in_head && i0 + j * STEP < count;
            sr[to + j * STEP * ROW] = in ? to_f32(fr[j]) : 0.f;
            sk[to + j * STEP * ROW] = in ? to_f32(fk[j]) : 0.f;
            sw[to + j * STEP * ROW] = in ? expf(-expf(fd[j] + shift[q])) : 1.f;
        }
    };
    auto fetch_values = [&](int base, int count) {
#pragma unroll
        for (int j = 0; j < PV; ++j) {
            const int e = threadIdx.x + j * THREADS, i = e / COLS, c = col0 + e % COLS;
            fv[j] = load_now(rkv + (size_t)(base + min(i, count - 1)) * ld + (v_off + h * D + min(c, D - 1)));
        }
    };
    auto stash_values = [&](int buf, int count) {
#pragma unroll
        for (int j = 0; j < PV; ++j) {
            const int e = threadIdx.x + j * THREADS, i = e / COLS, c = col0 + e % COLS;
            if (e < RS_BATCH * COLS) sv[buf * RS_BATCH * COLS + e] = i < count && c < D ? to_f32(fv[j]) : 0.f;
        }
    };
    auto rest = [&](int buf, int base, int count) {      // the channels that a thread has beyond its first
#pragma unroll
        for (int q = 1; q < PASSES; ++q) {
            fetch(base, count, q);
            stash(buf, count, q);
        }
    };
    if (t0 < t1) {
        const int count = min(RS_BATCH, t1 - t0);
        fetch(t0, count, 0);
        fetch_values(t0, count);
        if (through) tile.lay(asked);
        stash(0, count, 0);
        stash_values(0, count);
        rest(0, t0, count);
    } else {
        return;                                   // no token: the state stays as it is
    }
    __syncthreads();
    if (through) {
        tile.take(s, row0, cl);
        __syncthreads();
    }
    int buf = 0;
    float* mine = so + warp * RS_BATCH * 32;
    for (int base = t0; base < t1; base += RS_BATCH, buf ^= 1) {
        const int count = min(RS_BATCH, t1 - base), next = base + RS_BATCH, next_count = min(RS_BATCH, t1 - next);
        if (next < t1) {
            fetch(next, next_count, 0);
            fetch_values(next, next_count);
        }
        // Tokens AT_ONCE at a time (those beyond the last leave the state as it is: k = 0, v = 0, w = 1), their reads in flight together: a token
        // waits for the one before only in the state, one multiply-add an element. (A loop of known length lets the next reads start earlier.)
        auto token = [&](int i) {
            const int at = (buf * RS_BATCH + i) * ROW + sub * (R + 4);
            const float v = sv[(buf * RS_BATCH + i) * COLS + cl];
            const f32x2 v2 = pack2(v, v);
            f32x2 rr[R / 2], kk[R / 2], ww[R / 2], part[2] = {0ull, 0ull};
            read_rows<R>(rr, sr + at);
            read_rows<R>(kk, sk + at);
            read_rows<R>(ww, sw + at);
#pragma unroll
            for (int r = 0; r < R / 2; ++r) {
                const f32x2 kv = mul2(kk[r], v2);
                part[r & 1] = fma2(fma2(bonus[r], kv, s[r]), rr[r], part[r & 1]);
                s[r] = fma2(ww[r], s[r], kv);
            }
            mine[i * 32 + lane] = rows_sum(part[0], part[1]);
        };
        if (count == RS_BATCH) {
#pragma unroll AT_ONCE
            for (int i = 0; i < RS_BATCH; ++i) token(i);
        } else {
            for (int i0 = 0; i0 < count; i0 += AT_ONCE)
#pragma unroll
                for (int i1 = 0; i1 < AT_ONCE; ++i1) token(i0 + i1);
        }
        __syncwarp();
        for (int e = lane; e < count * CB; e += 32) {         // a warp's own columns leave once per batch
            const int i = e / CB, c = e % CB, to = col0 + warp * CB + c;
            if (to < D) o[(size_t)(base + i) * H * D + h * D + to] = used == G ? groups_sum<G>(mine + i * 32 + c, CB) : groups_sum(mine + i * 32 + c, CB, used);
        }
        if (next < t1) {
            stash(buf ^ 1, next_count, 0);
            stash_values(buf ^ 1, next_count);
            rest(buf ^ 1, next, next_count);
        }
        __syncthreads();
    }
    if (through) {
        tile.give(s, row0, cl);
        __syncthreads();
        tile.leave();
    } else {
        tile.store(s, row0, cl);
    }
}

// Keys above 64. Every block stages all key rows of its head, and what that takes grows with the key, so a block has 32 columns here (8 or 16 where few
// blocks would leave most SMs idle): R rows a lane, a column's rows shared out among the warps, and among a warp's lanes too where the columns are
// fewer; their sums meet in shared memory once per batch. 2,048 tokens here / in the kernel above: 32 heads of 128 576 / 1,111 us, 16 of 256 986 / 4,027;
// for 64 and less the other way round (32 heads of 64 406 / 274).
template <typename T, int R, int CB>
__global__ void decay_scan_wide_kernel(float* __restrict__ o, const T* rkv, long long ld, int r_off, int k_off, int v_off, const float* dlog,
                                  const float* __restrict__ w0, const float* __restrict__ u, float* state, long long state_stride,
                                  const int* cu_seqlens, const int* seq_slots, int H, int D) {
    extern __shared__ __align__(16) float sm[];
    constexpr int SUBS = 32 / CB;                 // a warp's lanes: CB columns x SUBS groups of R rows
    constexpr int PER = RS_BATCH * R * SUBS / 32; // staged elements of r, k, w per thread and batch: RS_BATCH * Dp / threads
    constexpr int PV = (RS_BATCH * CB + 127) / 128;
    const int warps = blockDim.x >> 5, Dp = warps * R * SUBS, threads = blockDim.x;
    float* sr = sm;                               // [2][RS_BATCH][Dp]
    float* sk = sr + 2 * RS_BATCH * Dp;
    float* sw = sk + 2 * RS_BATCH * Dp;
    float* sv = sw + 2 * RS_BATCH * Dp;           // [2][RS_BATCH][CB]
    float* red = sv + 2 * RS_BATCH * CB;          // [2][RS_BATCH][warps][32]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cl = lane % CB, sub = lane / CB;
    const int col0 = blockIdx.x * CB, col = col0 + cl, h = blockIdx.y, b = blockIdx.z;
    const int row0 = (warp * SUBS + sub) * R;
    const int used = (D + R - 1) / R;
    const bool early_v = threads >= 128;          // enough threads to fetch a batch's values ahead in PV registers each
    pdl_enter();
    const int t0 = __ldcg(cu_seqlens + b), t1 = __ldcg(cu_seqlens + b + 1);
    float* S = state + (size_t)__ldcg(seq_slots + b) * state_stride + (size_t)h * D * D;
    float s[R], bonus[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const bool in = row0 + r < D && col < D;
        s[r] = in ? __ldcg(S + (size_t)(row0 + r) * D + col) : 0.f;
        bonus[r] = row0 + r < D ? u[h * D + row0 + r] : 0.f;
    }
    // Fetched values stay as they were loaded (no conversion, no branch): a use right behind a load would make the warp wait for it,
    // one round trip to memory per load instead of one per batch. Rows outside the batch or the head read a valid address and
    // are zeroed when they are laid into shared memory.
    T fr[PER], fk[PER], fv[PV];
    float fd[PER];
    auto fetch = [&](int base, int count) {
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int e = threadIdx.x + j * threads, i = e / Dp, d = e - i * Dp;
            const bool in = i < count && d < D;
            const size_t at = in ? (size_t)(base + i) * ld + h * D + d : 0;
            fr[j] = __ldcg(rkv + at + r_off);
            fk[j] = __ldcg(rkv + at + k_off);
            fd[j] = __ldcg(dlog + (in ? (size_t)(base + i) * H * D + h * D + d : 0));
        }
        if (early_v) {
#pragma unroll
            for (int j = 0; j < PV; ++j) {
                const int e = threadIdx.x + j * threads, i = e / CB, c = col0 + e % CB;
                const bool in = e < RS_BATCH * CB && i < count && c < D;
                fv[j] = __ldcg(rkv + (in ? (size_t)(base + i) * ld + v_off + h * D + c : 0));
            }
        }
    };
    auto stash = [&](int buf, int base, int count) {
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int e = threadIdx.x + j * threads, i = e / Dp, d = e - i * Dp;
            const bool in = i < count && d < D;
            sr[buf * RS_BATCH * Dp + e] = in ? to_f32(fr[j]) : 0.f;
            sk[buf * RS_BATCH * Dp + e] = in ? to_f32(fk[j]) : 0.f;
            sw[buf * RS_BATCH * Dp + e] = in ? expf(-expf(fd[j] + w0[h * D + d])) : 1.f;
        }
        if (early_v) {
#pragma unroll
            for (int j = 0; j < PV; ++j) {
                const int e = threadIdx.x + j * threads, i = e / CB, c = col0 + e % CB;
                if (e < RS_BATCH * CB) sv[buf * RS_BATCH * CB + e] = (i < count && c < D) ? to_f32(fv[j]) : 0.f;
            }
        } else {                                  // a block of few threads (a small key size) reads its values late
            for (int e = threadIdx.x; e < RS_BATCH * CB; e += threads) {
                const int i = e / CB, c = col0 + e % CB;
                sv[buf * RS_BATCH * CB + e] = (i < count && c < D) ? to_f32(__ldcg(rkv + (size_t)(base + i) * ld + v_off + h * D + c)) : 0.f;
            }
        }
    };
    if (t0 < t1) {
        fetch(t0, min(RS_BATCH, t1 - t0));
        stash(0, t0, min(RS_BATCH, t1 - t0));
    }
    __syncthreads();
    int it = 0;
    for (int base = t0; base < t1; base += RS_BATCH, ++it) {
        const int count = min(RS_BATCH, t1 - base), buf = it & 1;
        const int next = base + RS_BATCH, next_count = min(RS_BATCH, t1 - next);
        if (next < t1) fetch(next, next_count);
        float* my_red = red + (size_t)buf * RS_BATCH * warps * 32;
        for (int i = 0; i < count; ++i) {
            const float v = sv[(buf * RS_BATCH + i) * CB + cl];
            const float4* pr = reinterpret_cast<const float4*>(sr + (buf * RS_BATCH + i) * Dp + row0);
            const float4* pk = reinterpret_cast<const float4*>(sk + (buf * RS_BATCH + i) * Dp + row0);
            const float4* pw = reinterpret_cast<const float4*>(sw + (buf * RS_BATCH + i) * Dp + row0);
            float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int q = 0; q < R / 4; ++q) {
                const float4 r4 = pr[q], k4 = pk[q], w4 = pw[q];
                const float rr[4] = {r4.x, r4.y, r4.z, r4.w}, kk[4] = {k4.x, k4.y, k4.z, k4.w}, ww[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float kv = kk[c] * v;
                    part[c] = fmaf(fmaf(bonus[4 * q + c], kv, s[4 * q + c]), rr[c], part[c]);
                    s[4 * q + c] = fmaf(ww[c], s[4 * q + c], kv);
                }
            }
            my_red[(i * warps + warp) * 32 + lane] = (part[0] + part[1]) + (part[2] + part[3]);
        }
        if (next < t1) stash(buf ^ 1, next, next_count);
        __syncthreads();
        for (int e = threadIdx.x; e < count * CB; e += threads) {
            const int i = e / CB, c = col0 + e % CB;
            if (c < D) o[(size_t)(base + i) * H * D + h * D + c] = groups_sum(my_red + i * warps * 32 + e % CB, CB, used);
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (row0 + r < D && col < D) S[(size_t)(row0 + r) * D + col] = s[r];
}

// One token per sequence (a decode step): no staging; a warp has one group of rows of 32 columns, its lanes read the same r, k and decay
// logits; the groups' sums meet in a small array and are added in the scan's order.
template <typename T, int R>
__global__ void decay_token_kernel(float* __restrict__ o, const T* rkv, long long ld, int r_off, int k_off, int v_off, const float* dlog,
                                   const float* __restrict__ w0, const float* __restrict__ u, float* state, long long state_stride,
                                   const int* seq_slots, int H, int D) {
    __shared__ float red[RS_MAX_KEY / R * 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int col = blockIdx.x * 32 + lane, h = blockIdx.y, t = blockIdx.z;
    const int row0 = warp * R;
    float* S = state + (size_t)__ldg(seq_slots + t) * state_stride + (size_t)h * D * D;
    float s[R], bonus[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {                 // the state does not depend on the step's other kernels: read before the wait
        s[r] = (row0 + r < D && col < D) ? __ldcg(S + (size_t)(row0 + r) * D + col) : 0.f;
        bonus[r] = row0 + r < D ? u[h * D + row0 + r] : 0.f;
    }
    pdl_enter();
    const T* row = rkv + (size_t)t * ld + h * D;
    const float v = col < D ? to_f32(__ldcg(row + v_off + col)) : 0.f;
    float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int d = row0 + r;
        float rr = 0.f, kk = 0.f, ww = 1.f;
        if (d < D) {
            rr = to_f32(__ldcg(row + r_off + d));
            kk = to_f32(__ldcg(row + k_off + d));
            ww = expf(-expf(__ldcg(dlog + (size_t)t * H * D + h * D + d) + w0[h * D + d]));
        }
        const float kv = kk * v;
        part[r & 3] = fmaf(fmaf(bonus[r], kv, s[r]), rr, part[r & 3]);
        s[r] = fmaf(ww, s[r], kv);
    }
    red[warp * 32 + lane] = (part[0] + part[1]) + (part[2] + part[3]);
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (row0 + r < D && col < D) S[(size_t)(row0 + r) * D + col] = s[r];
    __syncthreads();
    if (warp == 0 && col < D) o[(size_t)t * H * D + h * D + col] = groups_sum(red + lane, 32, blockDim.x >> 5);
}

template <typename T, int G>
static void launch_decay_scan(float* o, const T* rkv, long long ld, int r_off, int k_off, int v_off, const float* dlog, const float* w0, const float* u,
                              float* state, long long state_stride, const int* cu_seqlens, const int* seq_slots, int B, int H, int D, ScanShape shape, cudaStream_t stream) {
    constexpr int R = 8;
    const int warps = shape.warps, cols = warps * (32 / G);
    const size_t smem = (size_t)(2 * 3 * RS_BATCH * G * (R + 4) + 2 * RS_BATCH * cols + RS_BATCH * warps * 32 + 32) * sizeof(float);
    auto launch = [&](auto kernel) {
        if (smem > TI_SMEM_UNASKED) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        ti_launch_after(kernel, dim3((D + cols - 1) / cols, H, B), dim3(warps * 32), smem, stream, o, rkv, ld, r_off, k_off, v_off, dlog, w0, u, state, state_stride,
                        cu_seqlens, seq_slots, H, D, shape.through);
    };
    if constexpr (G <= 2) {                       // a warp or two hold all columns of such heads
        if (warps == 1) return launch(decay_scan_kernel<T, R, G, 1>);
    }
    if (warps == 4) launch(decay_scan_kernel<T, R, G, 4>);
    else launch(decay_scan_kernel<T, R, G, 2>);
}

template <typename T, int R, int CB>
static void launch_decay_scan_wide(float* o, const T* rkv, long long ld, int r_off, int k_off, int v_off, const float* dlog, const float* w0, const float* u,
                                   float* state, long long state_stride, const int* cu_seqlens, const int* seq_slots, int B, int H, int D, cudaStream_t stream) {
    constexpr int RW = R * (32 / CB);             // key rows of a warp
    const int warps = (D + RW - 1) / RW;
    const size_t smem = (size_t)(2 * 3 * RS_BATCH * warps * RW + 2 * RS_BATCH * CB + 2 * RS_BATCH * warps * 32) * sizeof(float);
    if (smem > TI_SMEM_UNASKED) cudaFuncSetAttribute(decay_scan_wide_kernel<T, R, CB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    ti_launch_after(decay_scan_wide_kernel<T, R, CB>, dim3((D + CB - 1) / CB, H, B), dim3(warps * 32), smem, stream, o, rkv, ld, r_off, k_off, v_off, dlog, w0, u,
                    state, state_stride, cu_seqlens, seq_slots, H, D);
}

extern "C" int ti_decay_scan(float* o, const void* rkv, long long ld, int r_off, int k_off, int v_off, const float* dlog, const float* w0,
                             const float* u, float* state, long long state_stride, const int* cu_seqlens, const int* seq_slots, int n, int B,
                             int H, int D, int dtype, cudaStream_t stream) {
    if (n == 0 || B == 0) return 0;
    TI_REQUIRE(D > 0 && D <= RS_MAX_KEY && H > 0, "decay_scan: %d heads of %d (at most %d)", H, D, RS_MAX_KEY);
    if (n == B) {                                 // one token per sequence
        TI_DISPATCH_DTYPE(dtype, {
            auto launch = [&](auto kernel, int rows) {
                ti_launch(kernel, dim3((D + 31) / 32, H, B), dim3((D + rows - 1) / rows * 32), 0, stream, o, (const T*)rkv, ld, r_off, k_off, v_off, dlog, w0, u,
                          state, state_stride, seq_slots, H, D);
            };
            if (D <= 128) launch(decay_token_kernel<T, 8>, 8); else launch(decay_token_kernel<T, 16>, 16);
        });
        return ti_check_launch("decay_token");
    }
    const ScanShape shape = scan_shape(8, D, D, (long long)H * B, 4, 2);
    const long long blocks32 = (long long)((D + 31) / 32) * H * B;
    const int sms = ti_sm_count();
#define RS_ARGS o, (const T*)rkv, ld, r_off, k_off, v_off, dlog, w0, u, state, state_stride, cu_seqlens, seq_slots, B, H, D
    TI_DISPATCH_DTYPE(dtype, {
        if (D > 128) launch_decay_scan_wide<T, 16, 32>(RS_ARGS, stream);
        else if (D > 64 && blocks32 * 4 >= sms) launch_decay_scan_wide<T, 8, 32>(RS_ARGS, stream);
        else if (D > 64 && blocks32 * 8 >= sms) launch_decay_scan_wide<T, 8, 16>(RS_ARGS, stream);
        else if (D > 64) launch_decay_scan_wide<T, 8, 8>(RS_ARGS, stream);
        else if (shape.groups == 8) launch_decay_scan<T, 8>(RS_ARGS, shape, stream);
        else if (shape.groups == 4) launch_decay_scan<T, 4>(RS_ARGS, shape, stream);
        else if (shape.groups == 2) launch_decay_scan<T, 2>(RS_ARGS, shape, stream);
        else launch_decay_scan<T, 1>(RS_ARGS, shape, stream);
    });
#undef RS_ARGS
    return ti_check_launch("decay_scan");
}

// ------------------------------------------------------------------------------------------------ delta scan
// qkv [n][ld] float: q heads (GQ of D) at 0, k heads (GQ of D) at GQ * D, v heads (H of V) at 2 GQ D, already activated and
// normalised; ba [n][2 H] float: the logits of beta, then of the decay; head h reads q/k head h / (H / GQ). The next batch's rows are
// on their way (cp.async, 16 bytes where `vec` says that all rows allow it) while this batch is worked on; one barrier per batch.
// What bounds it: one token's chain, decay, products with k, their sum over the lanes of a column, the write. So the next token's k is read
// ahead, the products with q are off the chain, and pairs of rows share an instruction. A prompt of 1,500 tokens
// (with 333, 64 and 7 beside it), 16 heads of 128 x 128, alone 804 -> 405 us, against blocks of 32 columns whose warps shared a column's rows
// and met at a barrier per token; 2,048 tokens 973 -> 402, 4 heads 1,408 -> 405.
// FULL: every group has rows of the key. FEW: so few blocks that a token's chain is all that counts; the state then always goes through shared memory, which
// leaves the compiler twice the registers to read ahead into (2 heads of 256 x 256, 2,048 tokens 741 -> 476 us; 16 heads, with more warps an SM, 1,282 -> 1,411).
template <int G, bool FULL, bool FEW>
__global__ void __launch_bounds__(G == 16 ? 256 : 128) delta_scan_kernel(float* __restrict__ o, const float* qkv, long long ld, const float* ba, const float* __restrict__ a_log,
                                  const float* __restrict__ dt_bias, float* state, long long state_stride, const int* cu_seqlens,
                                  const int* seq_slots, int H, int GQ, int D, int V, int vec, int many) {
    extern __shared__ __align__(16) float sm[];
    constexpr int R = RS_ROWS, CB = 32 / G, ROW = G * (R + 4);
    const bool through = FEW || many;
    const int threads = blockDim.x, cols = (threads >> 5) * CB;
    float* sq = sm;                               // [2][RS_BATCH][ROW]
    float* sk = sq + 2 * RS_BATCH * ROW;
    float* sv = sk + 2 * RS_BATCH * ROW;          // [2][RS_BATCH][cols]
    float* sg = sv + 2 * RS_BATCH * cols;         // [2][RS_BATCH][2]: decay, beta
    float* so = sg + 2 * RS_BATCH * 2;            // [warps][RS_BATCH][32], and before and after the tokens the state
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cl = warp * CB + lane % CB, sub = lane / CB;
    const int col0 = blockIdx.x * cols, h = blockIdx.y, b = blockIdx.z;
    const int g = h / (H / GQ), row0 = sub * R, used = (D + R - 1) / R;
    const int t0 = __ldcg(cu_seqlens + b), t1 = __ldcg(cu_seqlens + b + 1);
    if (t0 >= t1) return;                         // no token: the state stays as it is
    const StateTile<R, G> tile = {so, state + (size_t)__ldcg(seq_slots + b) * state_stride + (size_t)h * D * V + col0, __ffs(cols) - 1, D, V, V - col0};
    const float rate = expf(a_log[h]), shift = dt_bias[h];
    // 16-byte pieces: a thread has one column of rows `vec_rows` apart (threads beyond whole rows have none).
    const int pieces = max(1, D >> 2), vec_rows = threads / pieces, vec_col = (int)threadIdx.x % pieces * 4;
    const int vec_row = (int)threadIdx.x < vec_rows * pieces ? (int)threadIdx.x / pieces : RS_BATCH;
    // What lies beyond the last key or column stays zero, in the rows that the step's tokens use.
    if (D < R * G) {
        const int rows = min(RS_BATCH, t1 - t0), rest = R * G - D, bits = 32 - __clz(rest - 1);
#pragma unroll 4
        for (int e = threadIdx.x; e < rows << bits; e += threads) {
            const int d = D + (e & ((1 << bits) - 1)), at = (e >> bits) * ROW + staged_at<R>(d);
            if (d < R * G)
#pragma unroll
                for (int k = 0; k < 4; ++k) sm[k * RS_BATCH * ROW + at] = 0.f;      // both halves of q and of k
        }
    }
    if (col0 + cols > V)
        for (int e = threadIdx.x; e < 2 * RS_BATCH * cols; e += threads) sv[e] = 0.f;
    pdl_enter();
    f32x2 s[R / 2];
    float asked[R];
    if (through) tile.ask(asked); else tile.load(s, row0, cl);
    float fg[2] = {0.f, 0.f};
    auto fetch = [&](int buf, int base, int count) {
        const float* from = qkv + (size_t)base * ld + g * D;
        if (vec) {
            for (int i = vec_row; i < count; i += vec_rows) {
                const int to = (buf * RS_BATCH + i) * ROW + staged_at<R>(vec_col);
                cp_async16(smem_u32(sq + to), from + (size_t)i * ld + vec_col);
                cp_async16(smem_u32(sk + to), from + (size_t)i * ld + GQ * D + vec_col);
            }
        } else {
            for (int e = threadIdx.x; e < count * D; e += threads) {
                const int i = e / D, d = e - i * D, to = (buf * RS_BATCH + i) * ROW + staged_at<R>(d);
                copy4(sq + to, from + (size_t)i * ld + d);
                copy4(sk + to, from + (size_t)i * ld + GQ * D + d);
            }
        }
        for (int e = threadIdx.x; e < count * cols; e += threads) {
            const int i = e / cols, c = col0 + e % cols;
            if (c < V) copy4(sv + buf * RS_BATCH * cols + e, qkv + (size_t)(base + i) * ld + 2 * GQ * D + h * V + c);
        }
        cp_async_commit();
        if (threadIdx.x < count) {
            const float* row = ba + (size_t)(base + threadIdx.x) * 2 * H;
            fg[0] = load_now(row + H + h); fg[1] = load_now(row + h);
        }
    };
    auto land = [&](int buf, int count) {
        if (threadIdx.x < count) {
            sg[(buf * RS_BATCH + threadIdx.x) * 2] = expf(-rate * rs_softplus(fg[0] + shift));
            sg[(buf * RS_BATCH + threadIdx.x) * 2 + 1] = 1.0f / (1.0f + expf(-fg[1]));
        }
        cp_async_wait<0>();
        __syncthreads();
    };
    if (col0 + cols > V) __syncthreads();         // the zeros lie before the values
    fetch(0, t0, min(RS_BATCH, t1 - t0));
    if (through) tile.lay(asked);
    land(0, min(RS_BATCH, t1 - t0));
    if (through) {
        tile.take(s, row0, cl);
        __syncthreads();
    }
    int buf = 0;
    float* mine = so + warp * RS_BATCH * 32;
    for (int base = t0; base < t1; base += RS_BATCH, buf ^= 1) {
        const int count = min(RS_BATCH, t1 - base), next = base + RS_BATCH, next_count = min(RS_BATCH, t1 - next);
        if (next < t1) fetch(buf ^ 1, next, next_count);
        const float* rows_q = sq + buf * RS_BATCH * ROW + sub * (R + 4);
        const float* rows_k = sk + buf * RS_BATCH * ROW + sub * (R + 4);
        const float* gates = sg + buf * RS_BATCH * 2;
        // One token: `kk` and `decay` are its key rows and decay, `kn` and `decay_n` become the next one's.
        auto token = [&](int i, const f32x2 (&kk)[R / 2], float decay, f32x2 (&kn)[R / 2], float& decay_n) {
            const int after = min(i + 1, RS_BATCH - 1);
            const float beta = gates[i * 2 + 1], v = sv[(buf * RS_BATCH + i) * cols + cl];
            f32x2 qq[R / 2], part[2] = {0ull, 0ull}, out[2] = {0ull, 0ull};
            const f32x2 decay2 = pack2(decay, decay);
#pragma unroll
            for (int r = 0; r < R / 2; ++r) {
                s[r] = mul2(s[r], decay2);
                part[r & 1] = fma2(s[r], kk[r], part[r & 1]);
            }
            read_rows<R>(kn, rows_k + after * ROW);
            read_rows<R>(qq, rows_q + i * ROW);
            decay_n = gates[after * 2];
            const float write = beta * (v - groups_sum<G>(FULL || sub < used ? rows_sum(part[0], part[1]) : 0.f));
            const f32x2 write2 = pack2(write, write);
#pragma unroll
            for (int r = 0; r < R / 2; ++r) {
                s[r] = fma2(kk[r], write2, s[r]);
                out[r & 1] = fma2(s[r], qq[r], out[r & 1]);
            }
            mine[i * 32 + lane] = rows_sum(out[0], out[1]);
        };
        f32x2 ka[R / 2], kb[R / 2];
        float decay_a = gates[0], decay_b;
        read_rows<R>(ka, rows_k);
        int i = 0;
        for (; i + 1 < count; i += 2) {
            token(i, ka, decay_a, kb, decay_b);
            token(i + 1, kb, decay_b, ka, decay_a);
        }
        if (i < count) token(i, ka, decay_a, kb, decay_b);
        __syncwarp();
        for (int e = lane; e < count * CB; e += 32) {         // a warp's own columns leave once per batch
            const int i = e / CB, c = e % CB, to = col0 + warp * CB + c;
            if (to < V) o[(size_t)(base + i) * H * V + h * V + to] = FULL ? groups_sum<G>(mine + i * 32 + c, CB) : groups_sum(mine + i * 32 + c, CB, used);
        }
        __syncwarp();
        if (next < t1) land(buf ^ 1, next_count);
    }
    if (through) {
        __syncthreads();
        tile.give(s, row0, cl);
        __syncthreads();
        tile.leave();
    } else {
        tile.store(s, row0, cl);
    }
}

// One token per sequence: as the scan's step for one token, without staging; a warp has one group of rows of 32 columns.
__global__ void delta_token_kernel(float* __restrict__ o, const float* qkv, long long ld, const float* ba, const float* __restrict__ a_log,
                                   const float* __restrict__ dt_bias, float* state, long long state_stride, const int* seq_slots, int H, int GQ,
                                   int D, int V) {
    constexpr int R = RS_ROWS;
    __shared__ float red[2 * (RS_MAX_KEY / RS_ROWS) * 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, used = blockDim.x >> 5;
    const int col = blockIdx.x * 32 + lane, h = blockIdx.y, t = blockIdx.z;
    const int g = h / (H / GQ), row0 = warp * R;
    float* S = state + (size_t)__ldg(seq_slots + t) * state_stride + (size_t)h * D * V;
    float s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] = (row0 + r < D && col < V) ? __ldcg(S + (size_t)(row0 + r) * V + col) : 0.f;
    pdl_enter();
    const float* row = qkv + (size_t)t * ld;
    const float decay = expf(-expf(a_log[h]) * rs_softplus(__ldcg(ba + (size_t)t * 2 * H + H + h) + dt_bias[h]));
    const float beta = 1.0f / (1.0f + expf(-__ldcg(ba + (size_t)t * 2 * H + h)));
    const float v = col < V ? __ldcg(row + 2 * GQ * D + h * V + col) : 0.f;
    float kk[R], part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r = 0; r < R; ++r) {
        kk[r] = row0 + r < D ? __ldcg(row + GQ * D + g * D + row0 + r) : 0.f;
        s[r] *= decay;
        part[r & 3] = fmaf(s[r], kk[r], part[r & 3]);
    }
    red[warp * 32 + lane] = (part[0] + part[1]) + (part[2] + part[3]);
    __syncthreads();
    const float write = beta * (v - groups_sum(red + lane, 32, used));
    float out[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float qq = row0 + r < D ? __ldcg(row + g * D + row0 + r) : 0.f;
        s[r] = fmaf(kk[r], write, s[r]);
        out[r & 3] = fmaf(s[r], qq, out[r & 3]);
        if (row0 + r < D && col < V) S[(size_t)(row0 + r) * V + col] = s[r];
    }
    float* red_o = red + used * 32;
    red_o[warp * 32 + lane] = (out[0] + out[1]) + (out[2] + out[3]);
    __syncthreads();
    if (warp == 0 && col < V) o[(size_t)t * H * V + h * V + col] = groups_sum(red_o + lane, 32, used);
}

template <int G>
static void launch_delta_scan(float* o, const float* qkv, long long ld, const float* ba, const float* a_log, const float* dt_bias, float* state,
                              long long state_stride, const int* cu_seqlens, const int* seq_slots, int B, int H, int GQ, int D, int V, bool one_token,
                              ScanShape shape, cudaStream_t stream) {
    if (one_token) {
        ti_launch(delta_token_kernel, dim3((V + 31) / 32, H, B), dim3((D + RS_ROWS - 1) / RS_ROWS * 32), 0, stream, o, qkv, ld, ba, a_log, dt_bias, state, state_stride, seq_slots,
                  H, GQ, D, V);
        return;
    }
    const int warps = shape.warps, cols = warps * (32 / G);
    const size_t smem = (size_t)(4 * RS_BATCH * G * (RS_ROWS + 4) + 2 * RS_BATCH * cols + 4 * RS_BATCH + RS_BATCH * warps * 32 + 32) * sizeof(float);
    const int vec = D % 4 == 0 && ld % 4 == 0 && aligned16(qkv) && warps * 32 >= D / 4;
    auto launch = [&](auto kernel) {
        if (smem > TI_SMEM_UNASKED) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        ti_launch_after(kernel, dim3((V + cols - 1) / cols, H, B), dim3(warps * 32), smem, stream, o, qkv, ld, ba, a_log, dt_bias, state, state_stride,
                        cu_seqlens, seq_slots, H, GQ, D, V, vec, shape.through);
    };
    const bool full = D > RS_ROWS * (G - 1);
    if constexpr (G == 16) {
        if (!shape.through) return full ? launch(delta_scan_kernel<G, true, true>) : launch(delta_scan_kernel<G, false, true>);
    }
    if (full) launch(delta_scan_kernel<G, true, false>); else launch(delta_scan_kernel<G, false, false>);
}

extern "C" int ti_delta_scan(float* o, const float* qkv, long long ld, const float* ba, const float* a_log, const float* dt_bias, float* state,
                             long long state_stride, const int* cu_seqlens, const int* seq_slots, int n, int B, int H, int G, int D, int V,
                             cudaStream_t stream) {
    if (n == 0 || B == 0) return 0;
    TI_REQUIRE(D > 0 && V > 0 && D <= RS_MAX_KEY, "delta_scan: keys of %d (at most %d)", D, RS_MAX_KEY);
    TI_REQUIRE(H > 0 && G > 0 && H % G == 0, "delta_scan: %d heads do not divide into %d query/key heads", H, G);
    const ScanShape shape = scan_shape(RS_ROWS, D, V, (long long)H * B, D > 128 ? 8 : 4, 1);
#define RS_DELTA(GROUPS) launch_delta_scan<GROUPS>(o, qkv, ld, ba, a_log, dt_bias, state, state_stride, cu_seqlens, seq_slots, B, H, G, D, V, n == B, shape, stream)
    if (shape.groups == 1) RS_DELTA(1);
    else if (shape.groups == 2) RS_DELTA(2);
    else if (shape.groups == 4) RS_DELTA(4);
    else if (shape.groups == 8) RS_DELTA(8);
    else RS_DELTA(16);
#undef RS_DELTA
    return ti_check_launch("delta_scan");
}

// ------------------------------------------------------------------------------------------------ blends with the token before
// out [K][n][W] of T (every blend a matrix of its own): out[k][t] = h_t + (h_(t-1) - h_t) * mu[k], h_(t-1) being the row before in the step, or for a sequence's
// first token of the step the row `prev` [slots] (state rows `prev_stride` floats apart; zeros at a sequence's start). The
// block of a sequence's first token then moves the state on to the sequence's last row of the step (it alone reads the state).
// A thread has one channel of RUN tokens in a row: their rows and the blends' weights are read once, all loads in flight together
// (five blends of 2,048 channels, against a block that goes through a token's channels: 4 tokens 8.0 -> 2.3 us, 2,048 tokens 30 -> 24).
#define SB_BLENDS 8
template <typename T, int RUN>
__global__ void shift_blend_kernel(T* __restrict__ out, const T* h, const T* __restrict__ mu, int K, float* prev, long long prev_stride,
                                   const int* cu_seqlens, const int* seq_slots, int B, int n, int W) {
    __shared__ TokenRun<RUN> run;
    const int t = blockIdx.x * RUN, c = blockIdx.y * blockDim.x + threadIdx.x;
    run.find(cu_seqlens, seq_slots, B, n, t);
    const int count = min(RUN, n - t);
    float weight[SB_BLENDS];
#pragma unroll
    for (int k = 0; k < SB_BLENDS; ++k) weight[k] = k < K && c < W ? to_f32(mu[(size_t)k * W + c]) : 0.f;
    pdl_enter();
    if (c >= W) return;
    float row[RUN + 1];
#pragma unroll
    for (int i = 0; i <= RUN; ++i) row[i] = t + i >= 1 && i <= count ? to_f32(__ldcg(h + (size_t)(t + i - 1) * W + c)) : 0.f;
#pragma unroll
    for (int i = 0; i < RUN; ++i) {
        if (i >= count) break;
        const float cur = row[i + 1];
        float before = row[i];
        if (t + i == run.t0[i]) {                            // the sequence's first token of the step
            float* st = prev + (size_t)run.slot[i] * prev_stride + c;
            before = __ldcg(st);
            *st = to_f32(__ldcg(h + (size_t)(run.t1[i] - 1) * W + c));
        }
#pragma unroll
        for (int k = 0; k < SB_BLENDS; ++k)
            if (k < K) out[((size_t)k * n + t + i) * W + c] = from_f32<T>(fmaf(before - cur, weight[k], cur));
        for (int k = SB_BLENDS; k < K; ++k) out[((size_t)k * n + t + i) * W + c] = from_f32<T>(fmaf(before - cur, to_f32(mu[(size_t)k * W + c]), cur));
    }
}

extern "C" int ti_shift_blend(void* out, const void* h, const void* mu, int K, float* prev, long long prev_stride, const int* cu_seqlens,
                              const int* seq_slots, int n, int B, int W, int dtype, cudaStream_t stream) {
    if (n == 0) return 0;
    TI_REQUIRE(K > 0 && W > 0 && B > 0, "shift_blend: %d blends of rows of %d", K, W);
    const int threads = W >= 1024 ? 256 : 128, parts = (W + threads - 1) / threads;
    // Eight tokens in a row once single ones would be some 14 blocks an SM (2,048 channels, single / eight: 100 tokens 3.2 / 4.5 us, 300 6.7 / 5.8,
    // 2,048 33 / 24; 384 channels, 600 tokens 4.1 / 4.7, 1,000 5.6 / 4.7), but not where every token begins its sequence (200 x 4,096: 9.2 / 11.8).
    const bool runs = n > B && (long long)n * parts > 14LL * ti_sm_count();
    TI_DISPATCH_DTYPE(dtype, {
        if (runs)
            ti_launch(shift_blend_kernel<T, 8>, dim3((n + 7) / 8, parts), dim3(threads), 0, stream, (T*)out, (const T*)h, (const T*)mu, K, prev, prev_stride,
                      cu_seqlens, seq_slots, B, n, W);
        else
            ti_launch(shift_blend_kernel<T, 1>, dim3(n, parts), dim3(threads), 0, stream, (T*)out, (const T*)h, (const T*)mu, K, prev, prev_stride, cu_seqlens,
                      seq_slots, B, n, W);
    });
    return ti_check_launch("shift_blend");
}

// ------------------------------------------------------------------------------------------------ inputs of the delta scan
// proj [n][ld] of T: the projections' rows, C = 2 G D + H V channels (q heads, k heads, v heads). Every channel passes a causal
// convolution over time (conv [C][taps] of T, the last tap the current token's, zeros before the sequence's start; history from
// the step's own rows or from `hist`: the sequence's last taps - 1 rows, state rows `hist_stride` floats apart) and SiLU; then
// every q and k head becomes a unit vector x / sqrt(sum x^2 + unit_eps), q also times D^(-1/2). out [n][C] float.
// A block has RUN tokens in a row and `per` channels, whole heads among the q and k channels. A thread reads a channel's rows and weights once
// for all of them (TAPS weights; -1: more than 4, four at a time), its loads in flight together
// (4,096 channels, 4 taps, against a block that goes through a token's channels: 4 tokens 13.6 -> 2.3 us, 2,048 tokens 60 -> 54).
#define DI_THREADS 256
#define DI_MOST_THREADS 512
template <typename T, int RUN, int TAPS>
__global__ void __launch_bounds__(DI_MOST_THREADS) delta_inputs_kernel(float* __restrict__ out, const T* proj, long long ld, const T* __restrict__ conv,
                                                                   int taps, const float* hist, long long hist_stride, const int* cu_seqlens,
                                                                   const int* seq_slots, int B, int n, int G, int D, int HV, float unit_eps, int per) {
    extern __shared__ float y[];                             // [RUN][per]
    __shared__ TokenRun<RUN> run;
    const int t = blockIdx.x * RUN, C = 2 * G * D + HV, c0 = blockIdx.y * per, channels = min(per, C - c0), count = min(RUN, n - t);
    run.find(cu_seqlens, seq_slots, B, n, t);
    pdl_enter();
    for (int i = threadIdx.x; i < channels; i += blockDim.x) {
        const int c = c0 + i;
        // The row `back` before token t + j: of the step, or of the sequence's history, whose row taps - 1 - (t0 - token) counts back from the newest.
        auto older = [&](int j, int back) {
            return __ldcg(hist + (size_t)run.slot[j] * hist_stride + (size_t)(taps - 1 - (run.t0[j] - (t + j - back))) * C + c);
        };
        if (TAPS >= 0) {
            constexpr int KEEP = TAPS > 0 ? TAPS - 1 : 0;
            float row[RUN + KEEP], weight[KEEP + 1];
#pragma unroll
            for (int k = 0; k < (TAPS > 0 ? TAPS : 0); ++k) weight[k] = to_f32(conv[(size_t)c * taps + k]);
#pragma unroll
            for (int j = 0; j < RUN + KEEP; ++j) {
                const int tj = t + j - KEEP;
                row[j] = tj >= run.t0[0] && tj < t + count ? to_f32(__ldcg(proj + (size_t)tj * ld + c)) : 0.f;
            }
#pragma unroll
            for (int j = 0; j < RUN; ++j) {
                if (j >= count) break;
                float acc = TAPS == 0 ? row[j] : 0.f;
#pragma unroll
                for (int k = 0; k < (TAPS > 0 ? TAPS : 0); ++k) {
                    const int back = KEEP - k;
                    acc = fmaf(weight[k], t + j - back >= run.t0[j] ? row[j + k] : older(j, back), acc);
                }
                y[j * per + i] = rs_silu(acc);
            }
        } else if (RUN == 1) {
            float acc = 0.f;
            for (int k = 0; k < taps; ++k) {
                const int back = taps - 1 - k;
                const float x = t - back >= run.t0[0] ? to_f32(__ldcg(proj + (size_t)(t - back) * ld + c)) : older(0, back);
                acc = fmaf(to_f32(conv[(size_t)c * taps + k]), x, acc);
            }
            y[i] = rs_silu(acc);
        } else {
            // Four taps at a time: their rows lie in a row, a token's one after the one before's.
            float acc[RUN];
#pragma unroll
            for (int j = 0; j < RUN; ++j) acc[j] = 0.f;
            for (int k0 = 0; k0 < taps; k0 += 4) {
                const int far = taps - 1 - k0;               // rows back of the first of them
                float row[RUN + 3], weight[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) weight[k] = k0 + k < taps ? to_f32(conv[(size_t)c * taps + k0 + k]) : 0.f;
#pragma unroll
                for (int j = 0; j < RUN + 3; ++j) {
                    const int tj = t + j - far;
                    row[j] = tj >= run.t0[0] && tj < t + count ? to_f32(__ldcg(proj + (size_t)tj * ld + c)) : 0.f;
                }
#pragma unroll
                for (int j = 0; j < RUN; ++j) {
                    if (j >= count) break;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (k0 + k < taps) acc[j] = fmaf(weight[k], t + j - far + k >= run.t0[j] ? row[j + k] : older(j, far - k), acc[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < RUN; ++j)
                if (j < count) y[j * per + i] = rs_silu(acc[j]);
        }
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, head0 = D > 0 ? c0 / D : 0, heads = D > 0 ? max(0, min(2 * G - head0, channels / D)) : 0;
    for (int e = warp; e < heads * count; e += blockDim.x >> 5) {              // a warp per q or k head of a token
        const int hd = head0 + e % heads;
        float* src = y + (e / heads) * per + (size_t)hd * D - c0;
        float ss = 0.f;
        for (int d = lane; d < D; d += 32) ss = fmaf(src[d], src[d], ss);
        float inv = 1.0f / sqrtf(warp_sum(ss) + unit_eps);
        if (hd < G) inv *= 1.0f / sqrtf((float)D);
        for (int d = lane; d < D; d += 32) src[d] *= inv;
    }
    __syncthreads();
    for (int j = 0; j < count; ++j)
        for (int i = threadIdx.x; i < channels; i += blockDim.x) out[(size_t)(t + j) * C + c0 + i] = y[j * per + i];
}

extern "C" int ti_delta_inputs(float* out, const void* proj, long long ld, const void* conv, int taps, const float* hist, long long hist_stride,
                               const int* cu_seqlens, const int* seq_slots, int n, int B, int G, int D, int HV, float unit_eps, int dtype,
                               cudaStream_t stream) {
    if (n == 0) return 0;
    const int C = 2 * G * D + HV;
    TI_REQUIRE(G >= 0 && D >= 0 && HV >= 0, "delta_inputs: %d heads of %d, %d values", G, D, HV);
    TI_REQUIRE(taps >= 0 && taps <= 64 && (taps <= 1 || hist != nullptr) && (taps == 0 || conv != nullptr), "delta_inputs: %d taps", taps);
    TI_REQUIRE((size_t)C * sizeof(float) <= 160 * 1024, "delta_inputs: %d channels", C);
    if (C == 0) return 0;
    // Heads' worth of channels a block: about DI_THREADS of them; eight tokens in a row once single ones would be some 20 blocks an SM (4,096
    // channels, single / eight: 100 tokens 5.7 / 6.8 us, 200 10.5 / 9.8, 2,048 89 / 54; 2,048 channels, 300 tokens 8.0 / 8.9, 600 14.7 / 11.9).
    const int whole = D == 0 || D >= DI_THREADS ? 1 : DI_THREADS / D, want = D > 0 ? whole * D : DI_THREADS, per = want < C ? want : C, parts = (C + per - 1) / per;
    const bool runs = (long long)n * parts > 20LL * ti_sm_count() && (size_t)8 * per * sizeof(float) <= TI_SMEM_UNASKED;
    const size_t smem = (size_t)(runs ? 8 : 1) * per * sizeof(float);
    const int threads = per > DI_MOST_THREADS ? DI_MOST_THREADS : (per + 31) / 32 * 32;
#define DI_TAPS(TAPS) do { if (runs) launch(delta_inputs_kernel<T, 8, TAPS>); else launch(delta_inputs_kernel<T, 1, TAPS>); } while (0)
    TI_DISPATCH_DTYPE(dtype, {
        auto launch = [&](auto kernel) {
            if (smem > TI_SMEM_UNASKED) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            ti_launch(kernel, dim3(runs ? (n + 7) / 8 : n, parts), dim3(threads), smem, stream, out, (const T*)proj, ld, (const T*)conv, taps, hist, hist_stride,
                      cu_seqlens, seq_slots, B, n, G, D, HV, unit_eps, per);
        };
        switch (taps) {
            case 0: DI_TAPS(0); break;
            case 1: DI_TAPS(1); break;
            case 2: DI_TAPS(2); break;
            case 3: DI_TAPS(3); break;
            case 4: DI_TAPS(4); break;
            default: DI_TAPS(-1); break;
        }
    });
#undef DI_TAPS
    return ti_check_launch("delta_inputs");
}

// After the step: a sequence's history becomes its last taps - 1 projected rows (rows of this step where it brought enough, older
// ones moved up otherwise). A thread owns one channel of one sequence: it reads all it needs, then writes.
template <typename T>
__global__ void history_update_kernel(float* hist, long long hist_stride, const T* proj, long long ld, int taps, const int* cu_seqlens,
                                      const int* seq_slots, int C) {
    const int b = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_enter();
    if (c >= C) return;
    const int t0 = __ldcg(cu_seqlens + b), t1 = __ldcg(cu_seqlens + b + 1), n = t1 - t0, keep = taps - 1;
    float* st = hist + (size_t)__ldcg(seq_slots + b) * hist_stride;
    float rows[64];
    for (int j = 0; j < keep; ++j) {
        const int back = keep - 1 - j;                       // row j of the new history lies `back` rows before the newest
        rows[j] = back < n ? to_f32(__ldcg(proj + (size_t)(t1 - 1 - back) * ld + c)) : __ldcg(st + (size_t)(j + n) * C + c);
    }
    for (int j = 0; j < keep; ++j) st[(size_t)j * C + c] = rows[j];
}

extern "C" int ti_history_update(float* hist, long long hist_stride, const void* proj, long long ld, int taps, const int* cu_seqlens,
                                 const int* seq_slots, int B, int C, int dtype, cudaStream_t stream) {
    if (B == 0 || taps <= 1) return 0;
    TI_REQUIRE(taps <= 64, "history_update: %d taps", taps);
    TI_DISPATCH_DTYPE(dtype, (ti_launch(history_update_kernel<T>, dim3((C + 127) / 128, B), dim3(128), 0, stream, hist, hist_stride, (const T*)proj,
                                        ld, taps, cu_seqlens, seq_slots, C)));
    return ti_check_launch("history_update");
}

// ------------------------------------------------------------------------------------------------ a scan's output
// y [n][H * V] of T = o / rms(o over a head) * w * act(gate): every head normed by itself in 32-bit; w is [V] (one weight for all
// heads, `shared_w`) or [H * V], or null (no weight); gate [n][ldg] of T holds the gate's projection, act is SiLU or, with
// `gate_sigmoid`, the sigmoid. With nq and em [n][H] (a gated matrix memory) o is divided by max(|nq|, em) + 1e-6 first. With m_new [n][H]
// (one-token steps) the sequences' running maxima at m_state + slot * state_stride are moved on. A warp per (token, head).
struct HeadsOut {
    const float* nq;
    const float* em;
    const float* m_new;
    float* m_state;
    long long state_stride;
    const int* seq_slots;
    int gate_sigmoid;
};
template <typename T>
__global__ void heads_norm_gate_kernel(T* __restrict__ y, const float* o, const T* gate, long long ldg, const T* __restrict__ w, int shared_w,
                                       float eps, int H, int V, size_t heads_total, HeadsOut ex) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const size_t item = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= heads_total) return;
    const size_t t = item / H;
    const int h = (int)(item % H);
    const float* src = o + (t * H + h) * V;
    const float div = ex.nq != nullptr ? fmaxf(fabsf(__ldcg(ex.nq + item)), __ldcg(ex.em + item)) + 1e-6f : 1.f;
    if (ex.m_new != nullptr && lane == 0) ex.m_state[(size_t)__ldcg(ex.seq_slots + t) * ex.state_stride + h] = __ldcg(ex.m_new + item);
    float ss = 0.f;
    for (int d = lane; d < V; d += 32) {
        const float v = __ldcg(src + d) / div;
        ss = fmaf(v, v, ss);
    }
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)V + eps);
    for (int d = lane; d < V; d += 32) {
        float v = __ldcg(src + d) / div * inv;
        if (w != nullptr) v *= to_f32(w[shared_w ? d : h * V + d]);
        if (gate != nullptr) {
            const float g = to_f32(__ldcg(gate + t * ldg + h * V + d));
            v *= ex.gate_sigmoid ? 1.0f / (1.0f + expf(-g)) : rs_silu(g);
        }
        y[(t * H + h) * V + d] = from_f32<T>(v);
    }
}

extern "C" int ti_heads_norm_gate(void* y, const float* o, const void* gate, long long ldg, const void* w, int shared_w, float eps, const float* nq,
                                  const float* em, const float* m_new, float* m_state, long long state_stride, const int* seq_slots,
                                  int gate_sigmoid, int n, int H, int V, int dtype, cudaStream_t stream) {
    if (n == 0) return 0;
    TI_REQUIRE((nq != nullptr) == (em != nullptr) && (m_new == nullptr || (m_state != nullptr && seq_slots != nullptr)), "heads_norm_gate: nq comes with em, m_new with a state");
    const HeadsOut ex = {nq, em, m_new, m_state, state_stride, seq_slots, gate_sigmoid};
    const size_t total = (size_t)n * H;
    TI_DISPATCH_DTYPE(dtype, (ti_launch(heads_norm_gate_kernel<T>, dim3((unsigned)((total + 3) / 4)), dim3(128), 0, stream, (T*)y, o, (const T*)gate,
                                        ldg, (const T*)w, shared_w, eps, H, V, total, ex)));
    return ti_check_launch("heads_norm_gate");
}

// ------------------------------------------------------------------------------------------------ two mixers side by side
// out [n][size] float = sa * A' + sb * B'; A' = A / rms(A over the row) * wa with `normed`, else A (the same for B). A and B are rows
// of T or the sum of 32-bit partial sums (a product cut over k). One block per token.
template <typename T>
__device__ __forceinline__ float pair_value(const T* d, const float* partials, int n_partials, size_t stride, size_t at) {
    if (partials != nullptr) {
        float v = __ldcg(partials + at);
        for (int s = 1; s < n_partials; ++s) v += __ldcg(partials + (size_t)s * stride + at);
        return v;
    }
    return to_f32(__ldcg(d + at));
}

// Squares are added as by `sum_threads` threads, element i by thread i modulo it, whatever a block's size is. With no more rows than SMs a block
// has up to 1,024 threads, so that a row is a round trip or two
// (4 rows of 2,048, two slices of sums each: 7.5 -> 4.1 us).
template <typename T>
__global__ void __launch_bounds__(1024) pair_combine_kernel(float* __restrict__ out, const T* a, const float* pa, int na, size_t sa_stride, const T* b, const float* pb,
                                    int nb, size_t sb_stride, const T* __restrict__ wa, const T* __restrict__ wb, int normed, float eps,
                                    float scale_a, float scale_b, int size, int sum_threads) {
    extern __shared__ float rows[];                // [2][size]
    __shared__ float scratch[33];
    pdl_enter();
    float ssa = 0.f, ssb = 0.f;
    for (int i = threadIdx.x; i < size; i += blockDim.x) {
        const size_t at = (size_t)blockIdx.x * size + i;
        const float va = pair_value<T>(a, pa, na, sa_stride, at), vb = pair_value<T>(b, pb, nb, sb_stride, at);
        rows[i] = va; rows[size + i] = vb;
        ssa = fmaf(va, va, ssa); ssb = fmaf(vb, vb, ssb);
    }
    float ia = 1.f, ib = 1.f;
    if (normed) {
        if (blockDim.x != sum_threads) {
            __syncthreads();
            ssa = ssb = 0.f;
#pragma unroll 4
            for (int i = threadIdx.x < sum_threads ? threadIdx.x : size; i < size; i += sum_threads) {
                ssa = fmaf(rows[i], rows[i], ssa);
                ssb = fmaf(rows[size + i], rows[size + i], ssb);
            }
        }
        ia = 1.0f / sqrtf(block_sum(ssa, scratch) / (float)size + eps);
        ib = 1.0f / sqrtf(block_sum(ssb, scratch) / (float)size + eps);
    }
    for (int i = threadIdx.x; i < size; i += blockDim.x) {
        float va = rows[i], vb = rows[size + i];
        if (normed) { va = va * ia * to_f32(wa[i]); vb = vb * ib * to_f32(wb[i]); }
        out[(size_t)blockIdx.x * size + i] = fmaf(scale_a, va, scale_b * vb);
    }
}

extern "C" int ti_pair_combine(float* out, const void* a, const float* pa, int na, long long sa_stride, const void* b, const float* pb, int nb,
                               long long sb_stride, const void* wa, const void* wb, int normed, float eps, float scale_a, float scale_b, int n,
                               int size, int dtype, cudaStream_t stream) {
    if (n == 0) return 0;
    TI_REQUIRE(!normed || (wa != nullptr && wb != nullptr), "pair_combine: normed outputs need their weights");
    const size_t smem = (size_t)2 * size * sizeof(float);
    TI_REQUIRE(smem <= 160 * 1024, "pair_combine: rows of %d", size);
    TI_DISPATCH_DTYPE(dtype, {
        if (smem > TI_SMEM_UNASKED) cudaFuncSetAttribute(pair_combine_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        const int sum_threads = size >= 1024 ? 256 : 128, all = size > 1024 ? 1024 : (size + 31) / 32 * 32;
        const int threads = n <= ti_sm_count() && all > sum_threads ? all : sum_threads;
        ti_launch(pair_combine_kernel<T>, dim3(n), dim3(threads), smem, stream, out, (const T*)a, pa, na, (size_t)sa_stride, (const T*)b,
                  pb, nb, (size_t)sb_stride, (const T*)wa, (const T*)wb, normed, eps, scale_a, scale_b, size, sum_threads);
    });
    return ti_check_launch("pair_combine");
}
