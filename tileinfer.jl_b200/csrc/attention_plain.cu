// Plain attention over the paged cache, for any element type, head size and number of
// tokens per sequence: one block per (token, KV head, a few of its query heads), keys walked in position
// order in chunks of 256 with an online softmax. It is the 32-bit path's attention and the fallback
// of the bfloat16 path for sizes the tensor-core kernels refuse.
//
// The order of every sum depends only on the query's position, never on which other tokens
// or sequences share the launch, so a position's result is bit-identical however the work
// is cut into steps or batches.
//
// AntoineBut/TileInfer.jl: query head h reads KV head h div group
// (src/ops/reference.jl:108-112); the key at position i is visible to the query at
// position p iff i <= p, over all cached positions (reference.jl:98-107); scores, softmax
// and the accumulator are 32-bit, P is rounded to the storage type only for the PV product,
// O is rounded once (src/ops/tile/attention.jl:1-3, 34-59).
#include "common.cuh"

#define AP_THREADS 256
#define AP_WARPS (AP_THREADS / 32)
#define AP_CHUNK 256      // keys of one step of the online softmax, one per thread; borders are multiples of it in absolute positions
#define AP_MAX_D 512
#define AP_HEADS 4        // query heads of one KV head that a block serves together

// Four consecutive elements of a row, widened; through L2 (the row may have been written by the kernel before).
__device__ __forceinline__ void load_quad(const float* p, float (&v)[4]) {
    const float4 t = __ldcg(reinterpret_cast<const float4*>(p));
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void load_quad(const bf16* p, float (&v)[4]) {
    const uint2 t = __ldcg(reinterpret_cast<const uint2*>(p));
    v[0] = __uint_as_float(t.x << 16); v[1] = __uint_as_float(t.x & 0xffff0000u);
    v[2] = __uint_as_float(t.y << 16); v[3] = __uint_as_float(t.y & 0xffff0000u);
}
// A quad of a row that cannot be read so, element by element, zeros beyond the row's end.
template <typename T> __device__ __forceinline__ void load_elements(const T* row, int d, int D, float (&v)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = d + e < D ? to_f32(__ldcg(row + d + e)) : 0.f;
}
// A set's HN probabilities of one key.
template <int HN> __device__ __forceinline__ void load_set(const float* p, float (&v)[HN]) {
    if constexpr (HN == 4) { const float4 t = *reinterpret_cast<const float4*>(p); v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w; }
    else if constexpr (HN == 2) { const float2 t = *reinterpret_cast<const float2*>(p); v[0] = t.x; v[1] = t.y; }
    else v[0] = *p;
}
// N quads of a key into the scores of a set's heads, terms in ascending dimension. `q`: the heads' queries, Dq apart, from the first quad on.
template <int HN, int N> __device__ __forceinline__ void add_scores(const float (&k)[N][4], const float* q, int Dq, float (&s)[HN]) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int h = 0; h < HN; ++h) {
            const float4 qv = *reinterpret_cast<const float4*>(q + h * Dq + 4 * i);
            s[h] = fmaf(qv.w, k[i][3], fmaf(qv.z, k[i][2], fmaf(qv.y, k[i][1], fmaf(qv.x, k[i][0], s[h]))));
        }
}
template <typename T, int HN, int N> __device__ __forceinline__ void score_quads(const T* k, const float* q, int Dq, float (&s)[HN]) {
    float v[N][4];
#pragma unroll
    for (int i = 0; i < N; ++i) load_quad(k + 4 * i, v[i]);                        // all on their way before the first is used
    add_scores<HN, N>(v, q, Dq, s);
}

// A key's quads of the value row, times its probabilities, into the sums of a set's heads.
template <int NI, int HN> __device__ __forceinline__ void add_values(const float* p, const float (&v)[NI][4], float (&acc)[HN][NI][4]) {
    float w[HN];
    load_set<HN>(p, w);
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int h = 0; h < HN; ++h)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[h][i][e] = fmaf(w[h], v[i][e], acc[h][i][e]);
}

// One block per (token, KV head, set of up to AP_HEADS of its query heads): a key's and a value's row is read once for all the
// heads of the set. A chunk's scores are one key per thread (the products of a score added in ascending dimension); for the sums over
// keys warp w has the w-th 32 positions of every chunk and keeps a sum of its own over all chunks, and within a warp 128 / D
// groups of lanes take keys in turn when a value row is shorter than a warp's 128 elements. The groups' and then the warps' sums are
// added in a fixed order at the end. Per head the arithmetic is what it would be alone, so a head's result does not depend on how
// the heads are grouped.
// What bounds it: the latency of a few dependent reads per chunk at decode, reads of keys and values from L2 over prompts. Keys' row
// numbers come from the block table once per chunk, and value rows are asked for eight at a time: 8 sequences of 12 to 255
// positions, 32 / 8 heads of 128 take 35 us; with 128 threads, a table lookup ahead of every value row and one chain per
// dimension over all keys they took 127 us.
// NI: quads of a value row per lane (rows of up to 128 NI elements). HN: heads of a set, 1, 2 or 4 (the last set may have fewer).
// AT_ONCE: quads that a thread has in flight. BLOCKS: what an SM is to hold.
template <typename T, int NI, int HN, int AT_ONCE, int BLOCKS>
__global__ void __launch_bounds__(AP_THREADS, BLOCKS) attention_plain_kernel(T* __restrict__ out, const T* q, const T* k_cache,
                                       const T* v_cache, const int* block_table,
                                       int table_stride, const int* tok_slot,
                                       const int* positions, float scale, int nq, int nkv, int D,
                                       int page_size, int window, const float* __restrict__ sink, int chunk,
                                       const float* __restrict__ dist_bias, int bias_len, float cap,
                                       const float* __restrict__ slope, int keep) {
    extern __shared__ __align__(16) float smem[];
    const int Dq = (D + 3) & ~3;
    float* qs = smem;                                 // [HN][Dq], zeros beyond D
    float* ps = smem + HN * Dq;                 // [AP_CHUNK][HN]
    float* part_sums = ps + AP_CHUNK * HN;            // [AP_WARPS][Dq]
    __shared__ long long rows[AP_CHUNK];              // a key's row in the cache, in rows of D elements (pools of small heads hold more than 2^31)
    __shared__ float maxima[AP_WARPS][HN], sums[AP_WARPS][HN];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int group = nq / nkv;
    const int sets = (group + HN - 1) / HN;
    const int t = blockIdx.x, kvh = blockIdx.y / sets;
    const int h0 = kvh * group + (blockIdx.y % sets) * HN;           // first query head of the set
    const int heads = min(HN, kvh * group + group - h0);
    // Lanes that share a value row, and how many rows a warp takes at a time.
    int lanes = 32;
    if (NI == 1) while (lanes > 1 && lanes * 2 >= Dq) lanes >>= 1;          // lanes * 4 >= Dq still holds
    const int takes = 32 / lanes, sub = lane / lanes, dl = (lane % lanes) * 4;
    const bool quads = D % 4 == 0 && ((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & (4 * sizeof(T) - 1)) == 0;
    pdl_wait();
    pdl_launch_dependents();
    const int p = __ldcg(positions + t);
    const int* table = block_table + (size_t)__ldcg(tok_slot + t) * table_stride;
    for (int i = tid; i < HN * Dq; i += AP_THREADS) {
        const int h = i / Dq, d = i % Dq;
        qs[i] = h < heads && d < D ? to_f32(__ldcg(q + ((size_t)t * nq + h0 + h) * D + d)) : 0.f;
    }

    float acc[HN][NI][4];
    float m[HN], l[HN];
#pragma unroll
    for (int h = 0; h < HN; ++h) {
        m[h] = -INFINITY; l[h] = 0.f;
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[h][i][e] = 0.f;
    }
    int first = (window > 0 && p + 1 > window) ? p + 1 - window : 0;
    // Chunked visibility: only the keys of the query's own chunk of `chunk` positions, counted from the sequence's start.
    if (chunk > 0) first = max(first, (p / chunk) * chunk);
    // The kept first keys that lie before the window's come first.
    const int kept = min(keep, first);
    for (int part = kept > 0 ? 0 : 1; part < 2; ++part)
    for (int begin = part == 0 ? 0 : first, end = part == 0 ? kept - 1 : p, c0 = (begin / AP_CHUNK) * AP_CHUNK; c0 <= end; c0 += AP_CHUNK) {
        const int lo = c0 > begin ? c0 : begin;
        const int hi = (c0 + AP_CHUNK - 1 < end) ? c0 + AP_CHUNK - 1 : end;       // inclusive
        const int j = c0 + tid;
        const bool mine = j >= lo && j <= hi;
        const long long row = mine ? ((long long)__ldcg(table + j / page_size) * nkv + kvh) * page_size + j % page_size : 0;
        __syncthreads();                              // the chunk before is done with rows and ps; q is there
        rows[tid] = row;
        float s[HN];
#pragma unroll
        for (int h = 0; h < HN; ++h) s[h] = 0.f;
        if (mine) {
            const T* krow = k_cache + row * D;
            int d = 0;
            if (quads) {
#pragma unroll 1
                for (; d + 4 * AT_ONCE <= D; d += 4 * AT_ONCE) score_quads<T, HN, AT_ONCE>(krow + d, qs + d, Dq, s);
#pragma unroll 1
                for (; d < D; d += 4) score_quads<T, HN, 1>(krow + d, qs + d, Dq, s);
            } else {
#pragma unroll 1
                for (; d < Dq; d += 4) {
                    float kv[1][4];
                    load_elements(krow, d, D, kv[0]);
                    add_scores<HN, 1>(kv, qs + d, Dq, s);
                }
            }
        }
#pragma unroll
        for (int h = 0; h < HN; ++h) {
            if (h >= heads) continue;
            if (mine) {
                s[h] *= scale;
                if (cap > 0.f) s[h] = cap * tanhf(s[h] / cap);
                // A learned bias per (head, distance), added after the scale; distances beyond the table take its last entry.
                if (dist_bias != nullptr) s[h] += dist_bias[(size_t)(h0 + h) * bias_len + min(p - j, bias_len - 1)];
                if (slope != nullptr) s[h] = fmaf(-slope[h0 + h], (float)(p - j), s[h]);
            } else {
                s[h] = -INFINITY;
            }
            const float wm = warp_max(s[h]);
            if (lane == 0) maxima[warp][h] = wm;
        }
        __syncthreads();
        float factor[HN];
#pragma unroll
        for (int h = 0; h < HN; ++h) {
            if (h >= heads) continue;
            float m_new = m[h];
#pragma unroll
            for (int w = 0; w < AP_WARPS; ++w) m_new = fmaxf(m_new, maxima[w][h]);
            factor[h] = (m[h] == -INFINITY) ? 0.f : expf(m[h] - m_new);
            const float e = mine ? expf(s[h] - m_new) : 0.f;
            ps[tid * HN + h] = rnd<T>(e);
            const float ws = warp_sum(e);
            if (lane == 0) sums[warp][h] = ws;
            m[h] = m_new;
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < HN; ++h) {
            if (h >= heads) continue;
            float total = 0.f;
#pragma unroll
            for (int w = 0; w < AP_WARPS; ++w) total += sums[w][h];
            l[h] = l[h] * factor[h] + total;
#pragma unroll
            for (int i = 0; i < NI; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[h][i][e] *= factor[h];
        }
        // This warp's keys of the chunk that are visible: from the first row group that holds one on.
        const int w0 = c0 + 32 * warp, a = max(lo, w0) - w0, b = min(hi, w0 + 31) - w0;
        const int g0 = a > 0 ? a / takes * takes : 0;
        if (quads) {
            // Rows in flight together: AT_ONCE quads a lane. In the place of a key that is not visible stands the cache's first row; nothing is added.
            constexpr int ROWS = AT_ONCE / NI;
#pragma unroll 1
            for (int g = g0; g <= b; g += takes * ROWS) {
                float v[ROWS][NI][4];
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const T* vrow = v_cache + rows[32 * warp + min(g + r * takes + sub, 31)] * D;
#pragma unroll
                    for (int i = 0; i < NI; ++i) load_quad(vrow + (dl + 128 * i < D ? dl + 128 * i : 0), v[r][i]);
                }
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    const int k = g + r * takes + sub;
                    if (k >= a && k <= b) add_values<NI, HN>(ps + (32 * warp + k) * HN, v[r], acc);
                }
            }
        } else {
#pragma unroll 1
            for (int g = g0; g <= b; g += takes) {
                const int k = g + sub;
                if (k < a || k > b) continue;
                float v[NI][4];
#pragma unroll
                for (int i = 0; i < NI; ++i) load_elements(v_cache + rows[32 * warp + k] * D, dl + 128 * i, D, v[i]);
                add_values<NI, HN>(ps + (32 * warp + k) * HN, v, acc);
            }
        }
    }
#pragma unroll
    for (int h = 0; h < HN; ++h) {
        if (h >= heads) continue;
        // A sink: one more term exp(sink_h) in the softmax's denominator, with no key and no value.
        if (sink != nullptr) l[h] += expf(sink[h0 + h] - m[h]);
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                for (int o = lanes; o < 32; o <<= 1) acc[h][i][e] += __shfl_xor_sync(0xffffffffu, acc[h][i][e], o);
        __syncthreads();
        if (sub == 0)
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int d = dl + 128 * i;
                if (d < Dq) *reinterpret_cast<float4*>(part_sums + warp * Dq + d) = make_float4(acc[h][i][0], acc[h][i][1], acc[h][i][2], acc[h][i][3]);
            }
        __syncthreads();
        for (int d = tid; d < D; d += AP_THREADS) {
            float o = part_sums[d];
#pragma unroll
            for (int w = 1; w < AP_WARPS; ++w) o += part_sums[w * Dq + d];
            out[((size_t)t * nq + h0 + h) * D + d] = from_f32<T>(o / l[h]);
        }
    }
}

// `chunk` > 0: a key is visible only inside the query's chunk of so many positions; `dist_bias` [nq][bias_len] float: added to
// the scaled score by the distance between query and key (null: none). `cap` > 0: the scaled score s becomes cap tanh(s / cap) before
// any bias; `slope` [nq] float (null: none): slope[head] * distance is taken off after the cap.
// `keep`: beside a window, the first `keep` positions stay visible.
extern "C" int ti_attention_plain_kept(void* out, const void* q, const void* k_cache, const void* v_cache,
                                        const int* block_table, int table_stride, const int* tok_slot, const int* positions,
                                         float scale, int n_tokens, int nq, int nkv, int D, int page_size, int window,
                                         const float* sink, int chunk, const float* dist_bias, int bias_len, float cap, const float* slope,
                                        int keep, int dtype, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    TI_REQUIRE(chunk >= 0 && (dist_bias == nullptr || bias_len > 0), "attention: chunk %d, bias table of %d", chunk, bias_len);
    TI_REQUIRE(keep >= 0 && (keep == 0 || chunk == 0), "attention: kept positions beside a window, not beside chunks");
    TI_REQUIRE(D > 0 && D <= AP_MAX_D, "attention: head_dim %d exceeds %d", D, AP_MAX_D);
    TI_REQUIRE(nq > 0 && nkv > 0 && nq % nkv == 0, "attention: %d query heads do not divide into %d KV heads", nq, nkv);
    // The query heads of a KV head go in sets of up to four, which share the loads of its keys and values; in smaller sets while an SM has no more than
    // one of their blocks (a head's sums do not depend on its set; 32 heads on 8 of 128, 32-bit, one sequence of 64 / 300 positions 10.1 / 23.5 -> 7.0 / 16.1 us;
    // with two blocks an SM eight sequences of up to 255 take no less than in sets of four).
    const int group = nq / nkv;
    int hn = group <= 2 ? group : AP_HEADS;
    while (hn > 1 && (long long)n_tokens * nkv * ((group + hn / 2 - 1) / (hn / 2)) <= ti_sm_count()) hn /= 2;
    const int sets = (group + hn - 1) / hn;
    TI_REQUIRE((long long)nkv * sets <= 65535, "attention: too many heads (%d)", nq);
    dim3 grid(n_tokens, nkv * sets);
    const int Dq = (D + 3) & ~3;
    const size_t smem = (size_t)(hn * Dq + AP_CHUNK * hn + AP_WARPS * Dq) * sizeof(float);       // 28 KB at the largest head
    // Many blocks hide one another's latency: more of them on an SM (8 prompts of 60 tokens, 32-bit, 8 / 16 heads of 64 / 128 on as many: 42 / 111 us, 129 / 439
    // with two blocks an SM). Few have the longer run of loads each (one sequence of 20 / 2,000 positions, 32 / 4 heads of 64: 9 / 62 us).
    const bool many = (long long)n_tokens * nkv * sets > 3LL * ti_sm_count();
#define AP_ONE(NI, HN, AT_ONCE, BLOCKS) ti_launch(attention_plain_kernel<T, NI, HN, AT_ONCE, BLOCKS>, dim3(grid), dim3(AP_THREADS), smem, stream, (T*)out, (const T*)q, (const T*)k_cache,  \
                                (const T*)v_cache, block_table, table_stride, tok_slot, positions, scale, nq, nkv, D, page_size, window, sink, chunk, \
                                dist_bias, bias_len, cap, slope, window > 0 ? keep : 0)
#define AP_LAUNCH(NI, HN, LITTLE, BLOCKS) do { if (many) AP_ONE(NI, HN, LITTLE, BLOCKS); else AP_ONE(NI, HN, 8, 2); } while (0)
    TI_DISPATCH_DTYPE(dtype, {
        if (D <= 128) { if (hn == 1) AP_LAUNCH(1, 1, 4, 4); else if (hn == 2) AP_LAUNCH(1, 2, 4, 4); else AP_LAUNCH(1, 4, 4, 3); }
        else if (D <= 256) { if (hn == 1) AP_LAUNCH(2, 1, 4, 4); else if (hn == 2) AP_LAUNCH(2, 2, 4, 3); else AP_LAUNCH(2, 4, 4, 2); }
        else { if (hn == 1) AP_LAUNCH(4, 1, 4, 3); else if (hn == 2) AP_LAUNCH(4, 2, 4, 2); else AP_ONE(4, 4, 4, 2); }
    });
#undef AP_LAUNCH
#undef AP_ONE
    return ti_check_launch("attention_plain");
}

extern "C" int ti_attention_plain_ruled(void* out, const void* q, const void* k_cache, const void* v_cache,
                                        const int* block_table, int table_stride, const int* tok_slot, const int* positions,
                                        float scale, int n_tokens, int nq, int nkv, int D, int page_size, int window,
                                        const float* sink, int chunk, const float* dist_bias, int bias_len, float cap, const float* slope,
                                        int dtype, cudaStream_t stream) {
    return ti_attention_plain_kept(out, q, k_cache, v_cache, block_table, table_stride, tok_slot, positions, scale, n_tokens, nq, nkv, D, page_size,
                                   window, sink, chunk, dist_bias, bias_len, cap, slope, 0, dtype, stream);
}

extern "C" int ti_attention_plain_biased(void* out, const void* q, const void* k_cache, const void* v_cache,
                                         const int* block_table, int table_stride, const int* tok_slot, const int* positions,
                                         float scale, int n_tokens, int nq, int nkv, int D, int page_size, int window,
                                         const float* sink, int chunk, const float* dist_bias, int bias_len, int dtype, cudaStream_t stream) {
    return ti_attention_plain_ruled(out, q, k_cache, v_cache, block_table, table_stride, tok_slot, positions, scale, n_tokens, nq, nkv, D,
                                    page_size, window, sink, chunk, dist_bias, bias_len, 0.f, nullptr, dtype, stream);
}

extern "C" int ti_attention_plain(void* out, const void* q, const void* k_cache, const void* v_cache,
                                  const int* block_table, int table_stride, const int* tok_slot, const int* positions,
                                  float scale, int n_tokens, int nq, int nkv, int D, int page_size, int window,
                                  const float* sink, int dtype, cudaStream_t stream) {
    return ti_attention_plain_biased(out, q, k_cache, v_cache, block_table, table_stride, tok_slot, positions, scale, n_tokens, nq, nkv, D,
                                     page_size, window, sink, 0, nullptr, 0, dtype, stream);
}
