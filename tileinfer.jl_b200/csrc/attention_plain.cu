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
template <typename T> __device__ __forceinline__ void load_quad_any(const T* row, int d, int D, bool quads, float (&v)[4]) {
    if (quads) { load_quad(row + d, v); return; }
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = d + e < D ? to_f32(__ldcg(row + d + e)) : 0.f;
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
template <typename T, int NI>                     // NI: quads of a value row per lane (rows of up to 128 NI elements)
__global__ void __launch_bounds__(AP_THREADS) attention_plain_kernel(T* __restrict__ out, const T* q, const T* k_cache,
                                       const T* v_cache, const int* block_table,
                                       int table_stride, const int* tok_slot,
                                       const int* positions, float scale, int nq, int nkv, int D,
                                       int page_size, int window, const float* __restrict__ sink, int chunk,
                                       const float* __restrict__ dist_bias, int bias_len, float cap,
                                       const float* __restrict__ slope, int keep) {
    extern __shared__ __align__(16) float smem[];
    const int Dq = (D + 3) & ~3;
    float* qs = smem;                                 // [AP_HEADS][Dq], zeros beyond D
    float* ps = smem + AP_HEADS * Dq;                 // [AP_CHUNK][AP_HEADS]
    float* part_sums = ps + AP_CHUNK * AP_HEADS;      // [AP_WARPS][Dq]
    __shared__ long long rows[AP_CHUNK];              // a key's row in the cache, in rows of D elements (pools of small heads hold more than 2^31)
    __shared__ float maxima[AP_WARPS][AP_HEADS], sums[AP_WARPS][AP_HEADS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int group = nq / nkv;
    const int sets = (group + AP_HEADS - 1) / AP_HEADS;
    const int t = blockIdx.x, kvh = blockIdx.y / sets;
    const int h0 = kvh * group + (blockIdx.y % sets) * AP_HEADS;           // first query head of the set
    const int heads = min(AP_HEADS, kvh * group + group - h0);
    // Lanes that share a value row, and how many rows a warp takes at a time.
    int lanes = 32;
    if (NI == 1) while (lanes > 1 && lanes * 2 >= Dq) lanes >>= 1;          // lanes * 4 >= Dq still holds
    const int takes = 32 / lanes, sub = lane / lanes, dl = (lane % lanes) * 4;
    const bool quads = D % 4 == 0 && ((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & (4 * sizeof(T) - 1)) == 0;
    pdl_wait();
    pdl_launch_dependents();
    const int p = __ldcg(positions + t);
    const int* table = block_table + (size_t)__ldcg(tok_slot + t) * table_stride;
    for (int i = tid; i < AP_HEADS * Dq; i += AP_THREADS) {
        const int h = i / Dq, d = i % Dq;
        qs[i] = h < heads && d < D ? to_f32(__ldcg(q + ((size_t)t * nq + h0 + h) * D + d)) : 0.f;
    }

    float acc[AP_HEADS][NI][4];
    float m[AP_HEADS], l[AP_HEADS];
#pragma unroll
    for (int h = 0; h < AP_HEADS; ++h) {
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
        float s[AP_HEADS];
#pragma unroll
        for (int h = 0; h < AP_HEADS; ++h) s[h] = 0.f;
        if (mine) {
            const T* krow = k_cache + row * D;
#pragma unroll 8
            for (int d0 = 0; d0 < Dq; d0 += 4) {
                float kv[4];
                load_quad_any(krow, d0, D, quads, kv);
#pragma unroll
                for (int h = 0; h < AP_HEADS; ++h) {
                    if (h >= heads) continue;                                      // uniform across the block
                    const float4 qv = *reinterpret_cast<const float4*>(qs + h * Dq + d0);
                    s[h] = fmaf(qv.w, kv[3], fmaf(qv.z, kv[2], fmaf(qv.y, kv[1], fmaf(qv.x, kv[0], s[h]))));
                }
            }
        }
#pragma unroll
        for (int h = 0; h < AP_HEADS; ++h) {
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
        float factor[AP_HEADS];
#pragma unroll
        for (int h = 0; h < AP_HEADS; ++h) {
            if (h >= heads) continue;
            float m_new = m[h];
#pragma unroll
            for (int w = 0; w < AP_WARPS; ++w) m_new = fmaxf(m_new, maxima[w][h]);
            factor[h] = (m[h] == -INFINITY) ? 0.f : expf(m[h] - m_new);
            const float e = mine ? expf(s[h] - m_new) : 0.f;
            ps[tid * AP_HEADS + h] = rnd<T>(e);
            const float ws = warp_sum(e);
            if (lane == 0) sums[warp][h] = ws;
            m[h] = m_new;
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < AP_HEADS; ++h) {
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
#pragma unroll 8
        for (int g = a > 0 ? a / takes * takes : 0; g <= b; g += takes) {
            const int k = g + sub, i0 = 32 * warp + k;
            if (k < a || k > b) continue;
            const T* vrow = v_cache + rows[i0] * D;
            const float4 pv = *reinterpret_cast<const float4*>(ps + i0 * AP_HEADS);
            const float w[AP_HEADS] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int d = dl + 128 * i;
                if (d >= D) continue;
                float v[4];
                load_quad_any(vrow, d, D, quads, v);
#pragma unroll
                for (int h = 0; h < AP_HEADS; ++h) {
                    if (h >= heads) continue;
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[h][i][e] = fmaf(w[h], v[e], acc[h][i][e]);
                }
            }
        }
    }
#pragma unroll
    for (int h = 0; h < AP_HEADS; ++h) {
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
    const int sets = (nq / nkv + AP_HEADS - 1) / AP_HEADS;
    TI_REQUIRE((long long)nkv * sets <= 65535, "attention: too many heads (%d)", nq);
    dim3 grid(n_tokens, nkv * sets);
    const int Dq = (D + 3) & ~3;
    const size_t smem = (size_t)(AP_HEADS * Dq + AP_CHUNK * AP_HEADS + AP_WARPS * Dq) * sizeof(float);       // 28 KB at the largest head
#define AP_LAUNCH(NI) ti_launch(attention_plain_kernel<T, NI>, dim3(grid), dim3(AP_THREADS), smem, stream, (T*)out, (const T*)q, (const T*)k_cache,  \
                                (const T*)v_cache, block_table, table_stride, tok_slot, positions, scale, nq, nkv, D, page_size, window, sink, chunk, \
                                dist_bias, bias_len, cap, slope, window > 0 ? keep : 0)
    TI_DISPATCH_DTYPE(dtype, { if (D <= 128) AP_LAUNCH(1); else if (D <= 256) AP_LAUNCH(2); else AP_LAUNCH(4); });
#undef AP_LAUNCH
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
