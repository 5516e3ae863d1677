// Several copies of the residual stream (hyper-connections), kept in 32-bit: x [n][S][size].
//
// A sublayer reads u = sum_s a[s] x_s through a layer norm (weight, optional bias); its output y [n][size] is written back to all
// copies at once from the old ones:  x_t <- sum_s M[s][t] x_s + m * c[t] * y  (M indexed [from][to]). The kernel that writes a
// sublayer's output back also makes the next reader's input: u' = sum_t a'[t] x_t of the new copies, normed and rounded once.
// With S = 1, M = [[1]], a = c = [1] this is the plain residual sum x += m y followed by the next norm, so one kernel serves
// both arrangements. One block per token; everything is 32-bit arithmetic until the one rounding of the reader's input.
#include "common.cuh"

#define HS_MAX_STREAMS 8

// Sums over a row are added as by this many threads, element i by thread i modulo it, whatever a block's size is: a token's bits do not
// depend on the step it is in.
static int hs_threads(int size) { return size >= 4096 ? 512 : size >= 1024 ? 256 : 128; }
// Threads of a row's block. With no more rows than SMs a row's time is the round trips of one thread's loads, one after the other: blocks as
// large as the row, up to 1,024 threads (4 rows of 2,048, two copies: update 8.4 -> 3.7 us, read 6.1 -> 3.6).
static int hs_block(int size, int n) {
    if (n > ti_sm_count()) return hs_threads(size);
    const int all = (size + 31) / 32 * 32;
    return all > 1024 ? 1024 : all > hs_threads(size) ? all : hs_threads(size);
}

// x [n][S][size] <- x0 [n][size] in every copy.
__global__ void streams_begin_kernel(float* __restrict__ x, const float* x0, int S, int size, size_t count) {
    pdl_enter();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
        const size_t t = i / size;
        const int c = (int)(i % size);
        const float v = __ldcg(x0 + i);
        for (int s = 0; s < S; ++s) x[(t * S + s) * size + c] = v;
    }
}

extern "C" int ti_streams_begin(float* x, const float* x0, int n, int S, int size, cudaStream_t stream) {
    if (n == 0) return 0;
    TI_REQUIRE(S >= 1 && S <= HS_MAX_STREAMS && size > 0, "streams_begin: %d copies of rows of %d", S, size);
    const size_t count = (size_t)n * size;
    long long blocks = (count + 255) / 256;
    if (blocks > ti_sm_count() * 16) blocks = ti_sm_count() * 16;
    ti_launch(streams_begin_kernel, dim3((int)blocks), dim3(256), 0, stream, x, x0, S, size, count);
    return ti_check_launch("streams_begin");
}

struct StreamTables {
    float mix[HS_MAX_STREAMS * HS_MAX_STREAMS];   // [from][to]
    float out[HS_MAX_STREAMS];                     // m * c[t]
    float in_next[HS_MAX_STREAMS];                 // a'[t]
};

// The layer norm of `row_u` [size] (shared memory) into dst. Element i was written by thread i modulo the block's size, which added its own up
// in `sum`; a block of more than `sum_threads` threads adds again in the order of so many, and so does one that did not (ADD).
template <typename T, bool ADD>
__device__ __forceinline__ void norm_row(T* __restrict__ dst, const float* row_u, float sum, const T* __restrict__ w, const T* __restrict__ b,
                                         float eps, int centred, int size, int sum_threads, float* scratch) {
    const int first = threadIdx.x < sum_threads ? threadIdx.x : size;
    if (ADD || blockDim.x != sum_threads) {
        __syncthreads();
        sum = 0.f;
#pragma unroll 4
        for (int i = centred ? first : size; i < size; i += sum_threads) sum += row_u[i];
    }
    float mean = 0.f;
    if (centred) mean = block_sum(sum, scratch) / (float)size;
    float ss = 0.f;
#pragma unroll 4
    for (int i = first; i < size; i += sum_threads) {
        const float d = row_u[i] - mean;
        ss = fmaf(d, d, ss);
    }
    ss = block_sum(ss, scratch);
    const float inv = 1.0f / sqrtf(ss / (float)size + eps);
    for (int i = threadIdx.x; i < size; i += blockDim.x) {
        float v = (row_u[i] - mean) * inv * to_f32(w[i]);
        if (b != nullptr) v += to_f32(b[i]);
        dst[i] = from_f32<T>(v);
    }
}
// The norm's weights do not depend on the step's kernels: on their way to L2 before the wait, one request per 128 bytes. (Of many blocks the first
// do it for all, and the others' requests for the same lines only queue.)
#define HS_PREFETCH_ROWS 64
template <typename T> __device__ __forceinline__ void prefetch_row(const T* p, int size) {
    constexpr int PER = 128 / (int)sizeof(T);
    if (p != nullptr && gridDim.x <= HS_PREFETCH_ROWS)
        for (int i = threadIdx.x * PER; i < size; i += blockDim.x * PER) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + i));
}

// h = norm(sum_s a[s] x_s): the first reader's input (nothing to write back yet).
template <typename T>
__global__ void __launch_bounds__(1024) streams_read_norm_kernel(T* __restrict__ h, const float* x, const float* __restrict__ a, int S, const T* __restrict__ w,
                                         const T* __restrict__ b, float eps, int centred, int size, int sum_threads) {
    extern __shared__ float row_u[];
    __shared__ float scratch[33];
    const float* rows = x + (size_t)blockIdx.x * S * size;
    prefetch_row(w, size);
    prefetch_row(b, size);
    pdl_enter();
    float sum = 0.f;
    for (int i = threadIdx.x; i < size; i += blockDim.x) {
        float u = 0.f;
        for (int s = 0; s < S; ++s) u = fmaf(a[s], __ldcg(rows + (size_t)s * size + i), u);
        row_u[i] = u;
        sum += u;
    }
    norm_row<T, false>(h + (size_t)blockIdx.x * size, row_u, sum, w, b, eps, centred, size, sum_threads, scratch);
}

// Write a sublayer's output back and make the next reader's input. The output is `delta` [n][size] of T, or the sum of
// `n_partials` 32-bit arrays [n][size] `partial_stride` apart (a product cut over k, or one unrounded 32-bit result).
template <typename T>
__global__ void streams_update_kernel(float* x, const T* delta, const float* partials, int n_partials, size_t partial_stride, StreamTables tab,
                                      int S, T* __restrict__ h, const T* __restrict__ w, const T* __restrict__ b, float eps, int centred, int size,
                                      int sum_threads) {
    extern __shared__ float row_u[];
    __shared__ float scratch[33];
    float* rows = x + (size_t)blockIdx.x * S * size;
    pdl_enter();
    float sum = 0.f;
    for (int i = threadIdx.x; i < size; i += blockDim.x) {
        float y;
        if (partials != nullptr) {
            const float* p = partials + (size_t)blockIdx.x * size + i;
            y = __ldcg(p);
            for (int s = 1; s < n_partials; ++s) y += __ldcg(p + (size_t)s * partial_stride);
        } else {
            y = to_f32(__ldcg(delta + (size_t)blockIdx.x * size + i));
        }
        float old[HS_MAX_STREAMS];
#pragma unroll
        for (int s = 0; s < HS_MAX_STREAMS; ++s) old[s] = s < S ? __ldcg(rows + (size_t)s * size + i) : 0.f;
        float u = 0.f;
#pragma unroll
        for (int t = 0; t < HS_MAX_STREAMS; ++t) {
            if (t >= S) break;
            float v = 0.f;
#pragma unroll
            for (int s = 0; s < HS_MAX_STREAMS; ++s)
                if (s < S) v = fmaf(tab.mix[s * HS_MAX_STREAMS + t], old[s], v);
            v = fmaf(tab.out[t], y, v);
            rows[(size_t)t * size + i] = v;
            u = fmaf(tab.in_next[t], v, u);
        }
        row_u[i] = u;
        sum += u;
    }
    if (h == nullptr) return;
    norm_row<T, false>(h + (size_t)blockIdx.x * size, row_u, sum, w, b, eps, centred, size, sum_threads, scratch);
}

// The same, at most MAXS copies; a thread asks for AT_ONCE elements of all of them before it works on the first (2,048 rows, two copies of 2,048: 32.0 ->
// 23.4 us).
template <typename T, int MAXS, int AT_ONCE, int MOST>
__global__ void __launch_bounds__(MOST) streams_update_rows_kernel(float* x, const T* delta, const float* partials, int n_partials, size_t partial_stride, StreamTables tab,
                                      int S, T* __restrict__ h, const T* __restrict__ w, const T* __restrict__ b, float eps, int centred, int size,
                                      int sum_threads) {
    extern __shared__ float row_u[];
    __shared__ float scratch[33];
    float* rows = x + (size_t)blockIdx.x * S * size;
    if (h != nullptr) {
        prefetch_row(w, size);
        prefetch_row(b, size);
    }
    pdl_enter();
    for (int i0 = threadIdx.x; i0 < size; i0 += blockDim.x * AT_ONCE) {
        float y[AT_ONCE], old[AT_ONCE][MAXS];
#pragma unroll
        for (int k = 0; k < AT_ONCE; ++k) {
            const int i = i0 + k * blockDim.x, in = i < size ? i : 0;
            y[k] = partials != nullptr ? __ldcg(partials + (size_t)blockIdx.x * size + in) : to_f32(__ldcg(delta + (size_t)blockIdx.x * size + in));
#pragma unroll
            for (int s = 0; s < MAXS; ++s) old[k][s] = s < S ? __ldcg(rows + (size_t)s * size + in) : 0.f;
        }
        for (int s = 1; s < n_partials; ++s)
#pragma unroll
            for (int k = 0; k < AT_ONCE; ++k) {
                const int i = i0 + k * blockDim.x;
                y[k] += __ldcg(partials + (size_t)s * partial_stride + (size_t)blockIdx.x * size + (i < size ? i : 0));
            }
#pragma unroll
        for (int k = 0; k < AT_ONCE; ++k) {
            const int i = i0 + k * blockDim.x;
            float u = 0.f;
#pragma unroll
            for (int t = 0; t < MAXS; ++t) {
                if (t >= S) break;
                float v = 0.f;
#pragma unroll
                for (int s = 0; s < MAXS; ++s)
                    if (s < S) v = fmaf(tab.mix[s * HS_MAX_STREAMS + t], old[k][s], v);
                v = fmaf(tab.out[t], y[k], v);
                if (i < size) rows[(size_t)t * size + i] = v;
                u = fmaf(tab.in_next[t], v, u);
            }
            if (i < size) row_u[i] = u;
        }
    }
    if (h == nullptr) return;
    norm_row<T, true>(h + (size_t)blockIdx.x * size, row_u, 0.f, w, b, eps, centred, size, sum_threads, scratch);
}

extern "C" int ti_streams_read_norm(void* h, const float* x, const float* a, int S, const void* w, const void* b, float eps, int centred, int n,
                                    int size, int dtype, cudaStream_t stream) {
    if (n == 0) return 0;
    TI_REQUIRE(S >= 1 && S <= HS_MAX_STREAMS && size > 0, "streams_read_norm: %d copies of rows of %d", S, size);
    const size_t smem = (size_t)size * sizeof(float);
    TI_REQUIRE(smem <= 160 * 1024, "streams_read_norm: rows of %d", size);
    TI_DISPATCH_DTYPE(dtype, {
        if (smem > TI_SMEM_UNASKED) cudaFuncSetAttribute(streams_read_norm_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        ti_launch(streams_read_norm_kernel<T>, dim3(n), dim3(hs_block(size, n)), smem, stream, (T*)h, x, a, S, (const T*)w, (const T*)b, eps, centred, size,
                  hs_threads(size));
    });
    return ti_check_launch("streams_read_norm");
}

// mix [S][S] (from, to), out [S] (already times the multiplier), in_next [S]: host arrays, passed by value.
extern "C" int ti_streams_update(float* x, const void* delta, const float* partials, int n_partials, long long partial_stride, const float* mix,
                                 const float* out, const float* in_next, int S, void* h, const void* w, const void* b, float eps, int centred,
                                 int n, int size, int dtype, cudaStream_t stream) {
    if (n == 0) return 0;
    TI_REQUIRE(S >= 1 && S <= HS_MAX_STREAMS && size > 0, "streams_update: %d copies of rows of %d", S, size);
    TI_REQUIRE((delta != nullptr) != (partials != nullptr && n_partials > 0), "streams_update: rows or partial sums, one of them");
    StreamTables tab = {};
    for (int s = 0; s < S; ++s) {
        for (int t = 0; t < S; ++t) tab.mix[s * HS_MAX_STREAMS + t] = mix[s * S + t];
        tab.out[s] = out[s];
        tab.in_next[s] = in_next != nullptr ? in_next[s] : 0.f;
    }
    const size_t smem = (size_t)size * sizeof(float);
    TI_REQUIRE(smem <= 160 * 1024, "streams_update: rows of %d", size);
    const int threads = hs_block(size, n);
    TI_DISPATCH_DTYPE(dtype, {
        auto launch = [&](auto kernel, int block) {
            if (smem > TI_SMEM_UNASKED) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            ti_launch(kernel, dim3(n), dim3(block), smem, stream, x, (const T*)delta, partials, n_partials, (size_t)partial_stride, tab, S, (T*)h,
                      (const T*)w, (const T*)b, eps, centred, size, hs_threads(size));
        };
        // A thread asks for no more elements at once than it has: one in blocks as large as the row, four of rows up to 4,096 in blocks of 512 (two copies of
        // 2,048, 4 rows: 5.3 us in blocks of 1,024 with four, whose 64 registers do not hold them, 3.7 so; longer rows take less all the same in blocks of
        // 1,024: 4,096 9.1 and 5.7). Three copies and more: one at a time (four of 8,192, 4 rows 13.1 us with two, 10.2).
        // Many rows of 4,096 and more, or of many copies: their blocks' memory traffic is the bound, and a thread that asks for more at once only
        // takes room from other blocks (2,048 rows of 4,096, two copies, four elements at once: 73 us
        // against 65; four copies, two elements: 112 against 80); rows of one or two elements a thread have none to ask for.
        if (threads > hs_threads(size)) {
            if (S <= 2 && size <= 1024) launch(streams_update_rows_kernel<T, 2, 1, 1024>, threads);
            else if (S <= 2 && size < 4096) launch(streams_update_rows_kernel<T, 2, 4, 512>, 512);
            else if (S <= 2) launch(streams_update_rows_kernel<T, 2, 4, 1024>, threads);
            else if (S <= 4) launch(streams_update_rows_kernel<T, 4, 1, 1024>, threads);
            else launch(streams_update_rows_kernel<T, HS_MAX_STREAMS, 1, 1024>, threads);
        } else if (n > ti_sm_count() && S <= 2 && size < 4096 && size > 2 * threads) launch(streams_update_rows_kernel<T, 2, 4, 256>, threads);
        else launch(streams_update_kernel<T>, threads);
    });
    return ti_check_launch("streams_update");
}
