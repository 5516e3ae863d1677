// Linear attention with a decay per head ("lightning" attention): a matrix state per (sequence, head) that is carried
// from token to token,
//
//   S_t = a_h S_(t-1) + k_t v_t^T        S [dim, vdim], 32-bit, zero at the start of a sequence
//   o_t = S_t^T q_t                      [vdim]
//
// with q, k, v = act(projection) (act: SiLU or none; the activation is applied, and rounded to T, as the rows are read).
//
//   lightning_scan   the recurrence over the tokens a step brings, from the state the earlier steps left; the new state is
//                    written back. One kernel serves prompts and one-token steps.
//   lightning_out    y = T( o / rms(o) * w * sigmoid(g) ): the RMS norm over all heads' outputs together, in 32-bit, times
//                    the output gate; the input of the output projection.
//
// The scan: the columns of S are independent (column j of S sees v_t[j] only), so a block owns 32 columns of one
// (sequence, head) and walks the sequence's tokens in order; its 8 or 16 warps split the rows of S (warp w owns DP rows in a
// row, read from shared memory four at a time), a lane owns one column, the state lives in registers. Tokens are staged 32 at a time in shared memory; the
// warps' partial sums of o meet there once per 32 tokens. A launch of few blocks (one prompt, few heads) shares the rows of S
// out between two blocks per column block, whose two shares of o are added in global memory. A token's result depends on
// the sequence's earlier tokens alone; the order of its sums depends on the sizes and on whether the launch was shared
// out, so results agree to rounding, not bit for bit, between a prompt alone and the same prompt in a large batch.
// Everything is 32-bit arithmetic; nothing of the state, the decay or o is rounded.
#include "lightning_scan.cuh"

// One token per sequence: the step reads and writes every state once and is bound by that traffic. A block owns 128 columns
// of one (sequence, head): a lane owns four of them (16 bytes of a row), the warps take the rows in turn with several rows'
// loads in flight, and their shares of o meet in shared memory. The arithmetic per element is the scan's.
#define LT_WARPS 8
template <typename T, int LT_ROWS>
__global__ void __launch_bounds__(LT_WARPS * 32) lightning_token_kernel(float* __restrict__ o, const T* qkv, long long ld, int q_off, int k_off,
                                                                        int v_off, float* state, const float* __restrict__ decay,
                                                                        const int* seq_slots, int H, int D, int V, int act) {
    extern __shared__ float smem[];
    float* qs = smem;                                   // [D]
    float* ks = qs + D;                                 // [D]
    float* part = ks + D;                               // [LT_WARPS][128]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int col = blockIdx.x * 128 + lane * 4, h = blockIdx.y, b = blockIdx.z;
    const float a = decay[h];
    float* S = state + ((size_t)__ldcg(seq_slots + b) * H + h) * D * V;
    pdl_enter();
    const T* row = qkv + (size_t)b * ld;
    // The state is most of what is read: LT_ROWS rows of it a warp are asked for at once, the first ahead of everything else (16 heads of 128 x 128, four
    // rows at once behind q, k and v: 1 / 8 sequences 7.6 / 6.6 us, now 4.3 / 4.5; 32 heads, 64 sequences 55.7, 46.7).
    float4 s4[LT_ROWS];
    auto load = [&](int d0) {
#pragma unroll
        for (int i = 0; i < LT_ROWS; ++i) {
            const int d = d0 + i * LT_WARPS;
            s4[i] = d < D && col < V ? __ldcg(reinterpret_cast<const float4*>(S + (size_t)d * V + col)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    load(w);
    for (int d = threadIdx.x; d < D; d += LT_WARPS * 32) {
        float qv = to_f32(__ldcg(row + q_off + (size_t)h * D + d)), kv = to_f32(__ldcg(row + k_off + (size_t)h * D + d));
        if (act) { qv = rnd<T>(silu_value(qv)); kv = rnd<T>(silu_value(kv)); }
        qs[d] = qv;
        ks[d] = kv;
    }
    float v4[4] = {0.f, 0.f, 0.f, 0.f};
    if (col < V) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            v4[e] = to_f32(__ldcg(row + v_off + (size_t)h * V + col + e));
            if (act) v4[e] = rnd<T>(silu_value(v4[e]));
        }
    }
    __syncthreads();
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int d0 = w; d0 < D; d0 += LT_ROWS * LT_WARPS) {
        if (d0 > w) load(d0);
#pragma unroll
        for (int i = 0; i < LT_ROWS; ++i) {
            const int d = d0 + i * LT_WARPS;
            if (d >= D || col >= V) break;
            const float kd = ks[d], qd = qs[d];
            float4 t = s4[i];
            t.x = fmaf(a, t.x, kd * v4[0]); t.y = fmaf(a, t.y, kd * v4[1]);
            t.z = fmaf(a, t.z, kd * v4[2]); t.w = fmaf(a, t.w, kd * v4[3]);
            acc[0] = fmaf(t.x, qd, acc[0]); acc[1] = fmaf(t.y, qd, acc[1]);
            acc[2] = fmaf(t.z, qd, acc[2]); acc[3] = fmaf(t.w, qd, acc[3]);
            *reinterpret_cast<float4*>(S + (size_t)d * V + col) = t;
        }
    }
    *reinterpret_cast<float4*>(part + w * 128 + lane * 4) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    __syncthreads();
    for (int c = threadIdx.x; c < 128; c += LT_WARPS * 32) {
        if (blockIdx.x * 128 + c >= V) continue;
        float sum = 0.f;
#pragma unroll
        for (int p = 0; p < LT_WARPS; ++p) sum += part[p * 128 + c];
        o[(size_t)b * H * V + (size_t)h * V + blockIdx.x * 128 + c] = sum;
    }
}

// Prompts in chunks of 64 tokens that are worked on side by side (csrc/memory_chunks.cu), for decays above zero.
int lightning_chunks(float* o, const void* rows, long long ld, int q_off, int k_off, int v_off, float* state, const float* decay, const int* cu_seqlens,
                     const int* seq_slots, int B, int H, int D, int V, int act, float* ws, float* total, int chunks, int dtype, cudaStream_t stream);

// With work space `ws` [chunks, H, ti_memory_chunk_pitch(D, V)] and `total` [chunks, H] (chunks = sum over the sequences of ceil(tokens
// / 64)) a prompt goes through the chunks: 2,048 tokens of 16 heads of 128 x 128, 387 us in one scan, 170 in chunks. Whoever calls
// decides; short portions and many sequences take less time token by token.
// o [n, H * V] float; qkv [n, ld] of T with the heads' queries from column q_off on (H * D of them), keys from k_off, values
// from v_off (H * V); state [slots, H, D, V] float; decay [H] float; cu_seqlens [B + 1], seq_slots [B] (n_tokens in all). act: 1 = SiLU.
extern "C" int ti_lightning_scan(float* o, const void* qkv, long long ld, int q_off, int k_off, int v_off, float* state, const float* decay,
                                 const int* cu_seqlens, const int* seq_slots, int n_tokens, int B, int H, int D, int V, int act, float* ws, float* total,
                                 int chunks, int dtype, cudaStream_t stream) {
    if (B == 0) return 0;
    TI_REQUIRE(H > 0 && D > 0 && V > 0 && D <= LS_MAX_DIM, "lightning_scan: %d heads of %d x %d (the key size is at most %d)", H, D, V, LS_MAX_DIM);
    TI_REQUIRE(H <= 65535 && B <= 65535, "lightning_scan: %d heads, %d sequences", H, B);
    if (n_tokens == B && V % 4 == 0 && D <= 2048) {      // one token per sequence: the kernel that streams the states
        const size_t smem1 = (size_t)(2 * D + LT_WARPS * 128) * sizeof(float);
        // Eight rows at once are all of a warp's up to 64, and leave room for more blocks (64 sequences of 16 heads of 64 x 64 13.6 us with 16); four once there
        // are blocks for many rounds of heads whose values are few, where an SM's blocks hide one another's latency (256 sequences of them 26.7, with eight 30.5).
        const bool many = V <= 72 && (long long)((V + 127) / 128) * H * B > 5LL * ti_sm_count();
        TI_DISPATCH_DTYPE(dtype, {
            auto launch = [&](auto kernel) {
                ti_launch(kernel, dim3((V + 127) / 128, H, B), dim3(LT_WARPS * 32), smem1, stream, o, (const T*)qkv, ld, q_off, k_off, v_off, state, decay,
                          seq_slots, H, D, V, act);
            };
            if (many) launch(lightning_token_kernel<T, 4>);
            else if (D <= 8 * LT_WARPS) launch(lightning_token_kernel<T, 8>);
            else launch(lightning_token_kernel<T, 16>);
        });
        return ti_check_launch("lightning_scan");
    }
    if (ws != nullptr) {
        TI_REQUIRE(chunks > 0 && total != nullptr, "lightning_scan: %d chunks", chunks);
        return lightning_chunks(o, qkv, ld, q_off, k_off, v_off, state, decay, cu_seqlens, seq_slots, B, H, D, V, act, ws, total, chunks, dtype, stream);
    }
    ScanExtras ex = {};
    ex.state_stride = (long long)H * D * V;
    ex.q_scale = ex.k_scale = 1.f;
    return launch_lightning_scan<0>("lightning_scan", o, qkv, ld, q_off, k_off, v_off, state, decay, cu_seqlens, seq_slots, n_tokens, B, H, D, V, act, ex,
                                    dtype, stream);
}

// The squares are added as by `sum_threads` threads, element i by thread i modulo it, whatever a block's size is. The first LO_AHEAD elements of a thread
// and their gates are asked for at once and kept. With no more rows than SMs a block has up to 1,024 threads (2,048 elements, 1 / 2,048 rows 5.7 / 14.1 -> 3.1 / 12.2 us).
#define LO_AHEAD 4                 // (1 where a thread has no more)
template <typename T, int AHEAD>
__global__ void __launch_bounds__(1024) lightning_out_kernel(T* __restrict__ y, const float* o, const T* g, long long ldg, const T* __restrict__ w, float eps, int size,
                                                             int sum_threads) {
    extern __shared__ float squares[];                  // [size], where the block is larger than sum_threads
    __shared__ float scratch[33];
    const float* row = o + (size_t)blockIdx.x * size;
    const T* gate = g != nullptr ? g + (size_t)blockIdx.x * ldg : nullptr;
    pdl_enter();
    float v[AHEAD], gv[AHEAD], ss = 0.f;
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
        const int i = threadIdx.x + k * blockDim.x;
        v[k] = i < size ? __ldcg(row + i) : 0.f;
        gv[k] = gate != nullptr && i < size ? to_f32(__ldcg(gate + i)) : 0.f;
    }
    if (blockDim.x == sum_threads) {
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) ss = fmaf(v[k], v[k], ss);
        for (int i = threadIdx.x + AHEAD * blockDim.x; i < size; i += blockDim.x) {
            const float t = __ldcg(row + i);
            ss = fmaf(t, t, ss);
        }
    } else {
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
            if (threadIdx.x + k * blockDim.x < size) squares[threadIdx.x + k * blockDim.x] = v[k];
        for (int i = threadIdx.x + AHEAD * blockDim.x; i < size; i += blockDim.x) squares[i] = __ldcg(row + i);
        __syncthreads();
        for (int i = threadIdx.x < sum_threads ? threadIdx.x : size; i < size; i += sum_threads) ss = fmaf(squares[i], squares[i], ss);
    }
    ss = block_sum(ss, scratch);
    const float inv = 1.0f / sqrtf(ss / (float)size + eps);
    auto leave = [&](int i, float value, float z) {
        float r = value * inv * to_f32(w[i]);
        if (gate != nullptr) r = r / (1.0f + expf(-z));
        y[(size_t)blockIdx.x * size + i] = from_f32<T>(r);
    };
#pragma unroll
    for (int k = 0; k < AHEAD; ++k)
        if (threadIdx.x + k * blockDim.x < size) leave(threadIdx.x + k * blockDim.x, v[k], gv[k]);
    for (int i = threadIdx.x + AHEAD * blockDim.x; i < size; i += blockDim.x) leave(i, __ldcg(row + i), gate != nullptr ? to_f32(__ldcg(gate + i)) : 0.f);
}

// y [n, size] = T(o / rms(o) * w * sigmoid(g)); o [n, size] float, g [n, ldg] of T (null: no gate), w [size].
extern "C" int ti_lightning_out(void* y, const float* o, const void* g, long long ldg, const void* w, float eps, int n, int size, int dtype,
                                cudaStream_t stream) {
    if (n == 0) return 0;
    TI_REQUIRE(size > 0, "lightning_out: size %d", size);
    const int sum_threads = size >= 4096 ? 512 : size >= 1024 ? 256 : 128, all = size > 1024 ? 1024 : (size + 31) / 32 * 32;
    const size_t kept = (size_t)size * sizeof(float);
    // (Kept rows and the kernel's static arrays, less than 256 bytes, fit the 48 KB that a launch may have unasked.)
    const int threads = n <= ti_sm_count() && all > sum_threads && kept + 256 <= 48 * 1024 ? all : sum_threads;
    TI_DISPATCH_DTYPE(dtype, {
        auto launch = [&](auto kernel) {
            ti_launch(kernel, dim3(n), dim3(threads), threads > sum_threads ? kept : 0, stream, (T*)y, o, (const T*)g, ldg, (const T*)w, eps, size, sum_threads);
        };
        if (size <= threads) launch(lightning_out_kernel<T, 1>);
        else launch(lightning_out_kernel<T, LO_AHEAD>);
    });
    return ti_check_launch("lightning_out");
}
