// Inputs of latent attention: the two down-projected latents of a token, each RMS-normed in 32-bit with a plain
// weight; the query latent goes to a dense buffer, the key/value latent to the token's place in the paged pool
// (one "head" of kv_rank elements per position: pool[slot * kv_rank + i], slot = page * page_size + offset).
//
//   cq = T(a / rms(a) * wq),  a = row[0 : q_rank]
//   c  = T(b / rms(b) * wkv), b = row[q_rank : q_rank + kv_rank]          (q_rank 0: no query latent)
//
// With a rotated key part (rot > 0) the row has rot more elements after the two latents: one key part shared by all heads,
// not normed, rotated by the position's angles (cos_sin [positions, rot / 2, 2] float; pairs (2i, 2i + 1) or (i, i + rot / 2)) in
// 32-bit and written behind the latent in the same row of the pool, whose rows are pool_row >= kv_rank + rot long (zeros after).
// rotate_heads does the same rotation in place for a part of every head of a [n, heads, row] tensor (the queries' rotated part).
//
// The row is the fused down projection's output [n, q_rank + kv_rank] in T, or its 32-bit partial sums
// [s, n, q_rank + kv_rank] (a product cut over k), added in split order. One block per token.
#include "row_quads.cuh"

#define LI_THREADS 128

template <typename T>
__global__ void latent_inputs_kernel(const T* rows, size_t row_stride, const float* partials, int n_partials, size_t partial_stride,
                                     T* __restrict__ cq, T* pool, const T* __restrict__ wq, const T* __restrict__ wkv, float eps,
                                     const int* slots, int q_rank, int kv_rank, int rot, const float* __restrict__ cos_sin, int interleaved,
                                     const int* positions, int pool_row, size_t in_row) {
    extern __shared__ float row[];             // [q_rank + kv_rank + rot]
    __shared__ float scratch[33];
    const int t = blockIdx.x, size = q_rank + kv_rank + rot, normed = q_rank + kv_rank;
    pdl_enter();
    float sq = 0.f, sk = 0.f;
    for (int i = threadIdx.x; i < size; i += LI_THREADS) {
        float v;
        if (partials != nullptr) {
            const float* p = partials + (size_t)t * in_row + i;
            v = __ldcg(p);
            for (int s = 1; s < n_partials; ++s) v += __ldcg(p + (size_t)s * partial_stride);
        } else {
            v = to_f32(__ldcg(rows + (size_t)t * row_stride + i));
        }
        row[i] = v;
        if (i < q_rank) sq = fmaf(v, v, sq);
        else if (i < normed) sk = fmaf(v, v, sk);
    }
    sq = block_sum(sq, scratch);
    sk = block_sum(sk, scratch);
    const float iq = q_rank > 0 ? 1.0f / sqrtf(sq / (float)q_rank + eps) : 0.f, ik = 1.0f / sqrtf(sk / (float)kv_rank + eps);
    const size_t slot = (size_t)__ldcg(slots + t);
    for (int i = threadIdx.x; i < normed; i += LI_THREADS) {
        if (i < q_rank) cq[(size_t)t * q_rank + i] = from_f32<T>(row[i] * iq * to_f32(wq[i]));
        else pool[slot * pool_row + (i - q_rank)] = from_f32<T>(row[i] * ik * to_f32(wkv[i - q_rank]));
    }
    if (pool_row == kv_rank) return;
    const float* cs = rot > 0 ? cos_sin + (size_t)__ldcg(positions + t) * rot : nullptr;      // [rot / 2][2] = (cos, sin)
    const float* kr = row + normed;
    const int half = rot >> 1;
    for (int j = threadIdx.x; j < pool_row - kv_rank; j += LI_THREADS) {
        float v = 0.f;
        if (j < rot) {
            const int i = interleaved ? j >> 1 : (j < half ? j : j - half);
            const bool first = interleaved ? !(j & 1) : j < half;
            const float other = interleaved ? (first ? -kr[j + 1] : kr[j - 1]) : (first ? -kr[j + half] : kr[j - half]);
            v = kr[j] * cs[2 * i] + other * cs[2 * i + 1];
        }
        pool[slot * pool_row + kv_rank + j] = from_f32<T>(v);
    }
}

// The same for ranks of whole quads: a thread owns up to LQ_PER quads of the row, kept in registers; the two sums meet in one reduction
// and the weights are there before the kernel ahead has finished. A decode step of 8 rows of 768 + 128: 6.9 -> 2.3 us. With two quads a thread the
// block is as small as they allow: 8,192 rows of 768 + 256 + 32 take 19.8 us, in blocks of 256, where few threads have a second quad, 30.8.
#define LQ_THREADS 256
#define LQ_PER 2                                   // rows of up to 2,048 elements
template <typename T>
__global__ void __launch_bounds__(LQ_THREADS) latent_inputs_quads_kernel(const T* rows, size_t row_stride, const float* partials, int n_partials,
                                                                         size_t partial_stride, T* __restrict__ cq, T* pool, const T* __restrict__ wq,
                                                                         const T* __restrict__ wkv, float eps, const int* slots, int q_rank, int kv_rank,
                                                                         int rot, const float* __restrict__ cos_sin, int interleaved,
                                                                         const int* positions, int pool_row, size_t in_row) {
    __shared__ float sums[2][LQ_THREADS / 32];
    extern __shared__ __align__(16) float key_part[];          // [rot]
    const int t = blockIdx.x, size = q_rank + kv_rank + rot, normed = q_rank + kv_rank, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float4 w[LQ_PER], v[LQ_PER];
#pragma unroll
    for (int k = 0; k < LQ_PER; ++k) {
        const int i = (tid + k * (int)blockDim.x) * 4;
        w[k] = i < q_rank ? load_weight4(wq + i) : i < normed ? load_weight4(wkv + i - q_rank) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    pdl_enter();
    const size_t slot = (size_t)__ldcg(slots + t);
    const float* cs = rot > 0 ? cos_sin + (size_t)__ldcg(positions + t) * rot : nullptr;      // [rot / 2][2] = (cos, sin)
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int k = 0; k < LQ_PER; ++k) {
        const int i = (tid + k * (int)blockDim.x) * 4;
        v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i >= size) continue;
        if (partials != nullptr) {
            const float* p = partials + (size_t)t * in_row + i;
            v[k] = load_row4(p);
            for (int s = 1; s < n_partials; ++s) {
                const float4 q = load_row4(p + (size_t)s * partial_stride);
                v[k].x += q.x; v[k].y += q.y; v[k].z += q.z; v[k].w += q.w;
            }
        } else {
            v[k] = load_row4(rows + (size_t)t * row_stride + i);
        }
        const float ss = v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
        if (i < q_rank) sq += ss;
        else if (i < normed) sk += ss;
        else *reinterpret_cast<float4*>(key_part + i - normed) = v[k];
    }
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    if (lane == 0) { sums[0][warp] = sq; sums[1][warp] = sk; }
    __syncthreads();
    sq = sk = 0.f;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) { sq += sums[0][i]; sk += sums[1][i]; }
    const float iq = q_rank > 0 ? 1.0f / sqrtf(sq / (float)q_rank + eps) : 0.f, ik = 1.0f / sqrtf(sk / (float)kv_rank + eps);
#pragma unroll
    for (int k = 0; k < LQ_PER; ++k) {
        const int i = (tid + k * (int)blockDim.x) * 4;
        if (i >= normed) continue;
        const float s = i < q_rank ? iq : ik;
        const float o[4] = {v[k].x * s * w[k].x, v[k].y * s * w[k].y, v[k].z * s * w[k].z, v[k].w * s * w[k].w};
        store_row4(i < q_rank ? cq + (size_t)t * q_rank + i : pool + slot * pool_row + (i - q_rank), o);
    }
    const int half = rot >> 1;
    for (int j = tid; j < pool_row - kv_rank; j += blockDim.x) {
        float o = 0.f;
        if (j < rot) {
            const int i = interleaved ? j >> 1 : (j < half ? j : j - half);
            const bool first = interleaved ? !(j & 1) : j < half;
            const float other = interleaved ? (first ? -key_part[j + 1] : key_part[j - 1]) : (first ? -key_part[j + half] : key_part[j - half]);
            o = key_part[j] * cs[2 * i] + other * cs[2 * i + 1];
        }
        pool[slot * pool_row + kv_rank + j] = from_f32<T>(o);
    }
}

// x [n, heads, row] of T: elements [first, first + rot) of every head are rotated in place, a thread per pair, in 32-bit.
template <typename T>
__global__ void rotate_heads_kernel(T* x, const float* __restrict__ cos_sin, const int* positions, int heads, int row, int first, int rot,
                                    int interleaved, size_t pairs) {
    const int half = rot >> 1;
    pdl_enter();
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < pairs; e += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(e % half);
        const size_t th = e / half;                    // token * heads + head
        const size_t t = th / heads;
        const float* cs = cos_sin + ((size_t)__ldcg(positions + t) * half + i) * 2;
        T* base = x + th * row + first;
        const int a = interleaved ? 2 * i : i, b = interleaved ? 2 * i + 1 : i + half;
        const float u = to_f32(base[a]), v = to_f32(base[b]);
        base[a] = from_f32<T>(u * cs[0] - v * cs[1]);
        base[b] = from_f32<T>(v * cs[0] + u * cs[1]);
    }
}

extern "C" int ti_rotate_heads(void* x, const float* cos_sin, const int* positions, int n, int heads, int row, int first, int rot, int interleaved,
                               int dtype, cudaStream_t stream) {
    if (n == 0) return 0;
    TI_REQUIRE(rot >= 2 && rot % 2 == 0 && first >= 0 && first + rot <= row && heads > 0, "rotate_heads: %d elements from %d in heads of %d", rot, first, row);
    const long long pairs = (long long)n * heads * (rot / 2);
    long long blocks = (pairs + 255) / 256;
    if (blocks > ti_sm_count() * 16) blocks = ti_sm_count() * 16;
    TI_DISPATCH_DTYPE(dtype, (ti_launch(rotate_heads_kernel<T>, dim3((int)blocks), dim3(256), 0, stream, (T*)x, cos_sin, positions, heads, row, first,
                                        rot, interleaved, (size_t)pairs)));
    return ti_check_launch("rotate_heads");
}

extern "C" int ti_latent_inputs(const void* rows, long long row_stride, const float* partials, int n_partials, long long partial_stride,
                                void* cq, void* pool, const void* wq, const void* wkv, float eps, const int* slots, int n_tokens,
                                int q_rank, int kv_rank, int rot, const float* cos_sin, int interleaved, const int* positions, int pool_row,
                                long long in_row, int dtype, cudaStream_t stream) {
    if (n_tokens == 0) return 0;
    TI_REQUIRE(q_rank >= 0 && kv_rank > 0 && rot >= 0 && q_rank + kv_rank + rot <= 12000, "latent_inputs: ranks %d and %d, %d rotated", q_rank, kv_rank, rot);
    TI_REQUIRE((rows != nullptr) != (partials != nullptr), "latent_inputs: give rows or partial sums, not both");
    TI_REQUIRE(pool_row >= kv_rank + rot && in_row >= q_rank + kv_rank + rot, "latent_inputs: pool rows of %d for %d + %d", pool_row, kv_rank, rot);
    TI_REQUIRE(rot == 0 || (rot % 2 == 0 && cos_sin != nullptr && positions != nullptr), "latent_inputs: %d rotated elements need a table and positions", rot);
    const int quads = (q_rank + kv_rank + rot) / 4;
    if (q_rank % 4 == 0 && kv_rank % 4 == 0 && rot % 4 == 0 && pool_row % 4 == 0 && quads <= LQ_PER * LQ_THREADS && row_stride % 4 == 0 && in_row % 4 == 0 &&
        partial_stride % 4 == 0 && aligned16(rows) && aligned16(partials) && aligned16(cq) && aligned16(pool) && aligned16(wq) && aligned16(wkv)) {
        const int per = quads > LQ_THREADS ? LQ_PER : 1, threads = ((quads + per - 1) / per + 31) / 32 * 32;
        TI_DISPATCH_DTYPE(dtype, (ti_launch(latent_inputs_quads_kernel<T>, dim3(n_tokens), dim3(threads), (size_t)rot * sizeof(float), stream, (const T*)rows,
                                            (size_t)row_stride, partials, n_partials, (size_t)partial_stride, (T*)cq, (T*)pool, (const T*)wq,
                                            (const T*)wkv, eps, slots, q_rank, kv_rank, rot, cos_sin, interleaved, positions, pool_row, (size_t)in_row)));
        return ti_check_launch("latent_inputs");
    }
    const size_t smem = (size_t)(q_rank + kv_rank + rot) * sizeof(float);
    TI_DISPATCH_DTYPE(dtype, (ti_launch(latent_inputs_kernel<T>, dim3(n_tokens), dim3(LI_THREADS), smem, stream, (const T*)rows,
                                        (size_t)row_stride, partials, n_partials, (size_t)partial_stride, (T*)cq, (T*)pool, (const T*)wq,
                                        (const T*)wkv, eps, slots, q_rank, kv_rank, rot, cos_sin, interleaved, positions, pool_row,
                                        (size_t)in_row)));
    return ti_check_launch("latent_inputs");
}
