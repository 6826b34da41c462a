// Plain kernels: one simple kernel per operation, all arithmetic in IEEE float32
// (no fast-math in this file), a fixed order of summation that depends only on
// the element's own position, never on what else is in the batch.
//
// They are the whole float32 path of the engine and the reference beside each
// fast kernel.  Templated on the storage type so that the same code also runs
// with bfloat16 storage.  Formulas as the reference computes them:
//   embedding   kernels/full_attention_cuda.cuh:2012-2034
//   rmsnorm     kernels/full_attention_cuda.cuh:2826-2873
//   matmul      kernels/full_attention_4b_cuda.cuh:2671-2743 (out[m,n] = sum_k a[m,k] w[n,k])
//   rope        kernels/prefill_helpers_cuda.cuh:80-111 (half-split pairs)
//   kv append   kernels/certified_kv_bridge_cuda.cu:32-51
//   attention   kernels/full_attention_cuda.cuh:360-474, 476-576
//   swiglu      kernels/full_attention_cuda.cuh:1995-2010
//   argmax      kernels/prefill_helpers_bridge_cuda.cu:247-287 (lowest index wins ties)
#include "common.cuh"
#include "gemm_f32.cuh"
#include "attention_f32.cuh"
#include <math.h>

typedef __nv_bfloat16 bf16;

// ---------------------------------------------------------------------------------------
// embedding: out[t, :] = table[ids[t], :] * scale, written into the float32 residual stream; optionally the same row in
// the table's type (what a first sublayer without a norm in front of it reads)
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void embed_kernel(const int* __restrict__ ids, const T* __restrict__ table,
                             float* __restrict__ out, T* __restrict__ rounded, int hidden, int vocab, float scale) {
    const int t = blockIdx.x;
    const int id = ids[t];
    float* dst = out + (size_t)t * hidden;
    T* dst_r = rounded ? rounded + (size_t)t * hidden : nullptr;
    if (id < 0 || id >= vocab) {          // the host refuses such ids; never read out of range
        for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
            dst[c] = 0.f;
            if (dst_r) dst_r[c] = ssb_from_float<T>(0.f);
        }
        return;
    }
    const T* src = table + (size_t)id * hidden;
    if (dst_r) {
        for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
            const float v = ssb_to_float(src[c]) * scale;
            dst[c] = v;
            dst_r[c] = ssb_from_float<T>(v);
        }
        return;
    }
    if (scale == 1.0f)
        for (int c = threadIdx.x; c < hidden; c += blockDim.x) dst[c] = ssb_to_float(src[c]);
    else
        for (int c = threadIdx.x; c < hidden; c += blockDim.x) dst[c] = ssb_to_float(src[c]) * scale;
}

SSB_API int ssb_embed_scaled(const int* ids, const void* table, int table_dtype, float* out, void* rounded, int n_tokens,
                             int hidden, int vocab, float scale, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (table_dtype == SSB_F32)
        embed_kernel<float><<<n_tokens, 256, 0, stream>>>(ids, (const float*)table, out, (float*)rounded, hidden, vocab, scale);
    else if (table_dtype == SSB_BF16)
        embed_kernel<bf16><<<n_tokens, 256, 0, stream>>>(ids, (const bf16*)table, out, (bf16*)rounded, hidden, vocab, scale);
    else
        return SSB_ERR_BAD_DTYPE;
    return ssb_launch_status();
}

// out[t, :] = e / sqrt(mean(e^2) + eps) * w with e = table[ids[t], :] * scale: an embedding whose rows pass an RMS
// norm on their way into the stream (w float32, the multiplier itself).  One block per token, two passes over the row.
template <typename T>
__global__ void __launch_bounds__(256)
embed_norm_kernel(const int* __restrict__ ids, const T* __restrict__ table, const float* __restrict__ w, float eps,
                  float* __restrict__ out, int hidden, int vocab, float scale) {
    __shared__ float red[8];
    const int t = blockIdx.x;
    const int id = ids[t];
    float* dst = out + (size_t)t * hidden;
    const bool ok = id >= 0 && id < vocab;               // the host refuses other ids; never read out of range
    const T* src = table + (size_t)(ok ? id : 0) * hidden;
    float sq = 0.f;
    for (int c = threadIdx.x; c < hidden; c += 256) {
        const float v = ok ? ssb_to_float(src[c]) * scale : 0.f;
        sq = fmaf(v, v, sq);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) total += red[i];
    const float inv = 1.0f / sqrtf(total / (float)hidden + eps);
    for (int c = threadIdx.x; c < hidden; c += 256) dst[c] = ok ? ssb_to_float(src[c]) * scale * inv * w[c] : 0.f;
}

SSB_API int ssb_embed_norm(const int* ids, const void* table, int table_dtype, const float* w, float eps, float* out,
                           int n_tokens, int hidden, int vocab, float scale, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (table_dtype == SSB_F32)
        embed_norm_kernel<float><<<n_tokens, 256, 0, stream>>>(ids, (const float*)table, w, eps, out, hidden, vocab, scale);
    else if (table_dtype == SSB_BF16)
        embed_norm_kernel<bf16><<<n_tokens, 256, 0, stream>>>(ids, (const bf16*)table, w, eps, out, hidden, vocab, scale);
    else
        return SSB_ERR_BAD_DTYPE;
    return ssb_launch_status();
}

SSB_API int ssb_embed(const int* ids, const void* table, int table_dtype, float* out, int n_tokens,
                      int hidden, int vocab, cudaStream_t stream) {
    return ssb_embed_scaled(ids, table, table_dtype, out, nullptr, n_tokens, hidden, vocab, 1.0f, stream);
}

// ---------------------------------------------------------------------------------------
// rmsnorm over rows of the float32 residual stream; optional row gather
// ---------------------------------------------------------------------------------------
template <typename TO, typename TW>
__global__ void rmsnorm_kernel(const float* __restrict__ x, const int* __restrict__ rows,
                               const TW* __restrict__ w, float eps, TO* __restrict__ out, int hidden) {
    __shared__ float red[256];
    const int r = blockIdx.x;
    ssb_pdl_launch_dependents();
    ssb_pdl_wait();
    const float* src = x + (size_t)(rows ? rows[r] : r) * hidden;
    float part = 0.f;
    for (int c = threadIdx.x; c < hidden; c += 256) {
        const float v = src[c];
        part = fmaf(v, v, part);
    }
    red[threadIdx.x] = part;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    const float inv = 1.0f / sqrtf(red[0] / (float)hidden + eps);
    TO* dst = out + (size_t)r * hidden;
    for (int c = threadIdx.x; c < hidden; c += 256)
        dst[c] = ssb_from_float<TO>(src[c] * inv * ssb_to_float(w[c]));
}

SSB_API int ssb_rmsnorm(const float* x, const int* rows, const void* w, int w_dtype, float eps,
                        void* out, int out_dtype, int n_rows, int hidden, int pdl, cudaStream_t stream) {
    if (n_rows <= 0) return 0;
    int rc = 0;
#define SSB_RMS(TO, TW) \
    rc = ssb_launch(rmsnorm_kernel<TO, TW>, dim3(n_rows), dim3(256), 0, stream, pdl != 0, x, rows, (const TW*)w, eps, \
                    (TO*)out, hidden)
    if (out_dtype == SSB_F32 && w_dtype == SSB_F32) SSB_RMS(float, float);
    else if (out_dtype == SSB_F32 && w_dtype == SSB_BF16) SSB_RMS(float, bf16);
    else if (out_dtype == SSB_BF16 && w_dtype == SSB_F32) SSB_RMS(bf16, float);
    else if (out_dtype == SSB_BF16 && w_dtype == SSB_BF16) SSB_RMS(bf16, bf16);
    else return SSB_ERR_BAD_DTYPE;
#undef SSB_RMS
    return rc ? rc : ssb_launch_status();
}

// ---------------------------------------------------------------------------------------
// C[m, n] (+)= sum_k A[m, k] * W[n, k]; 64x64 tile, 16-wide k steps.  float32 throughout, in a
// fixed order: the 16 products of a k step are summed with FMAs, and the steps' sums are added
// with compensation (Kahan), so that the rounding error of a long row (14,336 terms in a
// feed-forward) stays at a few units in the last place instead of growing with its length.
// ---------------------------------------------------------------------------------------
template <typename TA, typename TC, bool ACCUMULATE>
__global__ void __launch_bounds__(256)
gemm_nt_plain_kernel(const TA* __restrict__ A, int lda, const TA* __restrict__ W, int ldw,
                     TC* __restrict__ C, int ldc, int M, int N, int K,
                     long long a_batch, long long w_batch, long long c_batch) {
    constexpr int BM = 64, BN = 64, BK = 16;
    A += (size_t)blockIdx.z * a_batch;        // one product per blockIdx.z (heads of a per-head projection)
    W += (size_t)blockIdx.z * w_batch;
    C += (size_t)blockIdx.z * c_batch;
    __shared__ float As[BK][BM + 1];
    __shared__ float Ws[BK][BN + 1];
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[4][4], lost[4][4];          // running sums and what their last additions rounded away
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) { acc[i][j] = 0.f; lost[i][j] = 0.f; }

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int idx = tid + e * 256;         // 0..1023
            const int r = idx / BK, c = idx % BK;
            const int k = k0 + c;
            const int m = m0 + r, n = n0 + r;
            As[c][r] = (m < M && k < K) ? ssb_to_float(A[(size_t)m * lda + k]) : 0.f;
            Ws[c][r] = (n < N && k < K) ? ssb_to_float(W[(size_t)n * ldw + k]) : 0.f;
        }
        __syncthreads();
        float part[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) part[i][j] = 0.f;
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) part[i][j] = fmaf(a[i], b[j], part[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float y = __fsub_rn(part[i][j], lost[i][j]);       // explicit roundings: nothing is re-associated
                const float t = __fadd_rn(acc[i][j], y);
                lost[i][j] = __fsub_rn(__fsub_rn(t, acc[i][j]), y);
                acc[i][j] = t;
            }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            TC* dst = C + (size_t)m * ldc + n;
            if (ACCUMULATE) *dst = ssb_from_float<TC>(ssb_to_float(*dst) + acc[i][j]);
            else *dst = ssb_from_float<TC>(acc[i][j]);
        }
    }
}

// ``n_batch`` products of the same sizes whose operands lie ``*_batch`` elements apart (per-head
// projections: a head's columns of a packed row, a head's own matrix); 1 and zeros: one product
static int gemm_nt_plain_launch(const void* A, int lda, long long a_batch, const void* W, int ldw,
                                long long w_batch, int in_dtype, void* C, int ldc, long long c_batch,
                                int out_dtype, int n_batch, int M, int N, int K, int accumulate, bool pdl,
                                cudaStream_t stream) {
    if (M <= 0 || N <= 0 || n_batch <= 0) return 0;
    if (K <= 0 || n_batch > 65535) return SSB_ERR_BAD_SIZE;
    if (accumulate && out_dtype != SSB_F32) return SSB_ERR_BAD_DTYPE;
    // float32 operands in whole 16-byte pieces: the same sums, bit for bit, from kernels made for their number of rows
    if (in_dtype == SSB_F32 && out_dtype == SSB_F32 && gemm_f32_ok(A, lda, a_batch, W, ldw, w_batch, K))
        return gemm_f32_launch((const float*)A, lda, a_batch, (const float*)W, ldw, w_batch, (float*)C, ldc, c_batch, n_batch,
                               M, N, K, accumulate, 0, stream, pdl);
    dim3 grid((N + 63) / 64, (M + 63) / 64, n_batch);
#define SSB_GEMM(TA, TC, ACC) \
    gemm_nt_plain_kernel<TA, TC, ACC><<<grid, 256, 0, stream>>>( \
        (const TA*)A, lda, (const TA*)W, ldw, (TC*)C, ldc, M, N, K, a_batch, w_batch, c_batch)
    if (in_dtype == SSB_F32 && out_dtype == SSB_F32) {
        if (accumulate) SSB_GEMM(float, float, true); else SSB_GEMM(float, float, false);
    } else if (in_dtype == SSB_BF16 && out_dtype == SSB_F32) {
        if (accumulate) SSB_GEMM(bf16, float, true); else SSB_GEMM(bf16, float, false);
    } else if (in_dtype == SSB_BF16 && out_dtype == SSB_BF16) {
        SSB_GEMM(bf16, bf16, false);
    } else {
        return SSB_ERR_BAD_DTYPE;
    }
#undef SSB_GEMM
    return ssb_launch_status();
}

// pdl: W is written by no kernel of the step, and the kernels of a few rows may start as dependents of the one before
SSB_API int ssb_gemm_nt_plain(const void* A, int lda, const void* W, int ldw, int in_dtype, void* C,
                              int ldc, int out_dtype, int M, int N, int K, int accumulate, int pdl,
                              cudaStream_t stream) {
    return gemm_nt_plain_launch(A, lda, 0, W, ldw, 0, in_dtype, C, ldc, 0, out_dtype, 1, M, N, K, accumulate, pdl != 0, stream);
}

// z = gate_fn(x gate^T, x up^T) * row_scale for a few float32 rows, in one launch; the bits of the product and the kernel behind it
SSB_API int ssb_gemm_f32_gated_ok(const void* A, int lda, const void* W, int ldw, int M, int N, int K) {
    return M > 0 && N > 0 && K > 0 && gemm_f32_ok(A, lda, 0, W, ldw, 0, K) && gemm_f32_gated_ok(M, N, K);
}
SSB_API int ssb_gemm_f32_gated(const float* A, int lda, const float* W, int ldw, float* z, int ldz, int M, int N, int K, int kind,
                               float limit, const float* row_scale, int pdl, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (kind < 0 || kind > SSB_GATE_LAST || !ssb_gemm_f32_gated_ok(A, lda, W, ldw, M, N, K)) return SSB_ERR_BAD_SIZE;
    const GfGate gate = {kind, limit, row_scale};
    return gemm_f32_launch(A, lda, 0, W, ldw, 0, z, ldz, 0, 1, M, N, K, 0, 0, stream, pdl != 0, &gate);
}

SSB_API int ssb_gemm_nt_plain_batched(const void* A, int lda, long long a_batch, const void* W, int ldw,
                                      long long w_batch, int in_dtype, void* C, int ldc, long long c_batch,
                                      int out_dtype, int n_batch, int M, int N, int K, cudaStream_t stream) {
    return gemm_nt_plain_launch(A, lda, a_batch, W, ldw, w_batch, in_dtype, C, ldc, c_batch, out_dtype, n_batch,
                                M, N, K, 0, false, stream);
}

// ---------------------------------------------------------------------------------------
// rotary position encoding on q (in place) and k, then k and v into the paged cache
// qkv row layout: [q heads | k heads | v heads], each head_dim wide
// ---------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void rotate_pair(float x1, float x2, float c, float sn, T& y1, T& y2) {
    y1 = ssb_from_float<T>(x1 * c - x2 * sn);
    y2 = ssb_from_float<T>(x1 * sn + x2 * c);
}

// Heads (of q, k and v) a block where tokens are few, so that they make many: all of a token's where that makes more than eight
// blocks an SM.  us with all and with eight, 48 heads of 64 in all: 1 token 3.3 and 1.8, 131 3.5 and 3.1, 900 7.1 and 10.1, 8,000 55
// and 82; 48 of 128: 5.2 and 2.2, 5.3 and 3.9, 11.9 and 13.7, 102 and 124.
constexpr int RO_HEADS = 8;

template <typename T>
__global__ void __launch_bounds__(256)
rope_append_kernel(T* __restrict__ qkv, int ld, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                   int table_positions, const int* __restrict__ pos, const int* __restrict__ slot,
                   const int* __restrict__ page_table, int max_pages, T* __restrict__ k_cache, T* __restrict__ v_cache, int n_q,
                   int n_kv, int head_dim, int rotary_dim, int page_shift, int write_cache, int interleaved, int per_block) {
    ssb_pdl_launch_dependents();
    ssb_pdl_wait();
    const int t = blockIdx.x, h0 = blockIdx.y * per_block;
    const int s = slot[t], p = pos[t];
    if (s < 0) return;                                   // padding row
    const int half = rotary_dim / 2, rest = head_dim - rotary_dim;
    T* row = qkv + (size_t)t * ld;
    const bool have_table = (cos_t != nullptr) && p < table_positions;
    const float* c_row = have_table ? cos_t + (size_t)p * half : nullptr;
    const float* s_row = have_table ? sin_t + (size_t)p * half : nullptr;
    size_t tok = 0;                                      // the token's row of kv head 0 in the cache entry
    if (write_cache) tok = ssb_cache_row(page_table, max_pages, s, p, page_shift, n_kv, 0, 1);
    const size_t head_rows = (size_t)1 << page_shift;
    // rotate q heads (and k heads): pairs (i, i + half) of the first rotary_dim elements, or (interleaved) pairs
    // (2i, 2i + 1); what a thread has rotated of a key it also appends
    const int rot_end = min(h0 + per_block, write_cache ? n_q + n_kv : n_q);
    for (int e = threadIdx.x; e < (rot_end - h0) * half; e += blockDim.x) {
        const int h = h0 + e / half, i = e % half;
        T* x = row + (size_t)h * head_dim;
        const int ia = interleaved ? 2 * i : i, ib = interleaved ? 2 * i + 1 : i + half;
        const float c = have_table ? c_row[i] : 1.f, sn = have_table ? s_row[i] : 0.f;
        const float x1 = ssb_to_float(x[ia]), x2 = ssb_to_float(x[ib]);
        T y1, y2;
        rotate_pair(x1, x2, c, sn, y1, y2);
        x[ia] = y1;
        x[ib] = y2;
        if (h >= n_q) {
            T* dst = k_cache + (tok + (h - n_q) * head_rows) * head_dim;
            dst[ia] = y1;
            dst[ib] = y2;
        }
    }
    if (!write_cache) return;
    // what is appended as it is: a key's elements behind the rotated ones, and values
    const int k_first = max(h0, n_q), k_end = min(h0 + per_block, n_q + n_kv);
    for (int e = threadIdx.x; e < (k_end - k_first) * rest; e += blockDim.x) {
        const int h = k_first + e / rest, d = rotary_dim + e % rest;
        k_cache[(tok + (h - n_q) * head_rows) * head_dim + d] = row[(size_t)h * head_dim + d];
    }
    const int v_first = max(h0, n_q + n_kv), v_end = min(h0 + per_block, n_q + 2 * n_kv);
    for (int e = threadIdx.x; e < (v_end - v_first) * head_dim; e += blockDim.x) {
        const int h = v_first + e / head_dim, d = e % head_dim;
        v_cache[(tok + (h - n_q - n_kv) * head_rows) * head_dim + d] = row[(size_t)h * head_dim + d];
    }
}

SSB_API int ssb_rope_append(void* qkv, int ld, int dtype, const float* cos_t, const float* sin_t,
                            int table_positions, const int* pos, const int* slot,
                            const int* page_table, int max_pages, void* k_cache, void* v_cache,
                            int n_tokens, int n_q, int n_kv, int head_dim, int rotary_dim,
                            int page_shift, int write_cache, int interleaved, int pdl, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (rotary_dim % 2 || rotary_dim > head_dim || rotary_dim < 0) return SSB_ERR_BAD_SIZE;
    const int heads = write_cache ? n_q + 2 * n_kv : n_q;
    if (heads > RO_HEADS * 65535) return SSB_ERR_BAD_SIZE;
    const int groups = (heads + RO_HEADS - 1) / RO_HEADS, per_block = (long long)n_tokens * groups <= 8 * ssb_sm_count() ? RO_HEADS : heads;
    const dim3 grid(n_tokens, (heads + per_block - 1) / per_block);
    int rc;
    if (dtype == SSB_F32)
        rc = ssb_launch(rope_append_kernel<float>, grid, dim3(256), 0, stream, pdl != 0, (float*)qkv, ld, cos_t, sin_t,
                        table_positions, pos, slot, page_table, max_pages, (float*)k_cache, (float*)v_cache, n_q, n_kv, head_dim,
                        rotary_dim, page_shift, write_cache, interleaved, per_block);
    else if (dtype == SSB_BF16)
        rc = ssb_launch(rope_append_kernel<bf16>, grid, dim3(256), 0, stream, pdl != 0, (bf16*)qkv, ld, cos_t, sin_t,
                        table_positions, pos, slot, page_table, max_pages, (bf16*)k_cache, (bf16*)v_cache, n_q, n_kv, head_dim,
                        rotary_dim, page_shift, write_cache, interleaved, per_block);
    else
        return SSB_ERR_BAD_DTYPE;
    return rc ? rc : ssb_launch_status();
}

// ---------------------------------------------------------------------------------------
// attention of each token over its sequence's cached keys: one block per (token, head).
// Keys are visited in chunks of 128 starting at the first visible key, so the order of
// every sum depends on the token's own position and window only.
// ---------------------------------------------------------------------------------------
constexpr int ATT_THREADS = 128;
constexpr int ATT_MAX_HEAD_DIM = 1024;

__device__ __forceinline__ float block_reduce_max(float v, float* red) {
    red[threadIdx.x] = v;
    __syncthreads();
    for (int s = ATT_THREADS / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + s]);
        __syncthreads();
    }
    const float r = red[0];
    __syncthreads();
    return r;
}

__device__ __forceinline__ float block_reduce_sum(float v, float* red) {
    red[threadIdx.x] = v;
    __syncthreads();
    for (int s = ATT_THREADS / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    const float r = red[0];
    __syncthreads();
    return r;
}

template <typename T>
__global__ void __launch_bounds__(ATT_THREADS)
attention_plain_kernel(const T* __restrict__ q, int ldq, const T* __restrict__ k_cache,
                       const T* __restrict__ v_cache, const int* __restrict__ pos,
                       const int* __restrict__ slot, const int* __restrict__ page_table, int max_pages,
                       T* __restrict__ out, int ldo, int n_q, int n_kv, int head_dim, int page_shift,
                       int window, float scale, int v_dim, int v_row, const float* __restrict__ sinks) {
    __shared__ __align__(16) float q_s[ATT_MAX_HEAD_DIM];
    __shared__ float p_s[ATT_THREADS];
    __shared__ float red[ATT_THREADS];
    const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const bool pieces = sizeof(T) == 4 && head_dim % 4 == 0 && ((uintptr_t)k_cache & 15) == 0;
    T* o = out + (size_t)t * ldo + (size_t)h * v_dim;
    const int s = slot[t];
    if (s < 0) {
        for (int d = tid; d < v_dim; d += ATT_THREADS) o[d] = ssb_from_float<T>(0.f);
        return;
    }
    const int p = pos[t];
    const int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
    const int kvh = h / (n_q / n_kv);
    const T* qp = q + (size_t)t * ldq + (size_t)h * head_dim;
    for (int d = tid; d < head_dim; d += ATT_THREADS) q_s[d] = ssb_to_float(qp[d]);
    __syncthreads();

    float m = -INFINITY, l = 0.f;
    float acc[ATT_MAX_HEAD_DIM / ATT_THREADS];
#pragma unroll
    for (int i = 0; i < ATT_MAX_HEAD_DIM / ATT_THREADS; ++i) acc[i] = 0.f;

    for (int base = lo; base <= p; base += ATT_THREADS) {
        const int j = base + tid;
        float sc = -INFINITY;
        if (j <= p) {
            const T* kr = k_cache + ssb_cache_row(page_table, max_pages, s, j, page_shift, n_kv, kvh, head_dim);
            float dot = 0.f;
            if (pieces) {                                // the same chain, four elements a load
#pragma unroll 4
                for (int d = 0; d < head_dim; d += 4) {
                    const float4 k4 = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(kr) + d);
                    const float4 q4 = *reinterpret_cast<const float4*>(q_s + d);
                    dot = fmaf(q4.x, k4.x, dot);
                    dot = fmaf(q4.y, k4.y, dot);
                    dot = fmaf(q4.z, k4.z, dot);
                    dot = fmaf(q4.w, k4.w, dot);
                }
            } else {
                for (int d = 0; d < head_dim; ++d) dot = fmaf(q_s[d], ssb_to_float(kr[d]), dot);
            }
            sc = dot * scale;
        }
        const float cm = block_reduce_max(sc, red);
        const float m_new = fmaxf(m, cm);
        const float pj = (j <= p) ? expf(sc - m_new) : 0.f;
        p_s[tid] = pj;
        const float cs = block_reduce_sum(pj, red);      // also orders p_s writes before reads
        const float alpha = (m == -INFINITY) ? 0.f : expf(m - m_new);
        l = l * alpha + cs;
        const int n_in = min(ATT_THREADS, p - base + 1);
#pragma unroll
        for (int i = 0; i < ATT_MAX_HEAD_DIM / ATT_THREADS; ++i) {
            const int d = tid + i * ATT_THREADS;
            if (d < v_dim) {
                float a = acc[i] * alpha;
#pragma unroll 8
                for (int jj = 0; jj < n_in; ++jj) {
                    const T* vr = v_cache + ssb_cache_row(page_table, max_pages, s, base + jj, page_shift,
                                                          n_kv, kvh, v_row);
                    a = fmaf(p_s[jj], ssb_to_float(vr[d]), a);
                }
                acc[i] = a;
            }
        }
        m = m_new;
        __syncthreads();
    }
    // a sink adds exp(sink) to the denominator and nothing to the numerator
    float keep = 1.f;
    if (sinks != nullptr) {
        const float sk = sinks[h];
        const float m_all = fmaxf(m, sk);
        keep = (m == -INFINITY) ? 0.f : expf(m - m_all);
        l = l * keep + expf(sk - m_all);
    }
#pragma unroll
    for (int i = 0; i < ATT_MAX_HEAD_DIM / ATT_THREADS; ++i) {
        const int d = tid + i * ATT_THREADS;
        if (d < v_dim) o[d] = ssb_from_float<T>(l > 0.f ? acc[i] * keep / l : 0.f);
    }
}

// The same sums for float32 rows of up to 128 elements in whole 16-byte pieces, which come through shared memory; a key's place is
// looked up once.  ROPE (decode steps): q comes as the projection left it, [q | k | v] in a row; the block rotates its query and its
// token's key (pairs i, i + rotary_dim / 2), and the first head of a kv head appends key and value.
constexpr int AS_MAX_DIM = 128;
struct AsRope { const float *cos_t, *sin_t; int table_positions, rotary_dim; float *k_cache, *v_cache; };

// The block's query, rotated where ROPE, and this thread's element of the token's own key and value.
template <bool ROPE>
__device__ __forceinline__ void attention_own_rows(const float* __restrict__ q, int ldq, int t, int h, int s, int p, int n_q, int n_kv,
                                                   int head_dim, const int* __restrict__ page_table, int max_pages, int page_shift,
                                                   const AsRope& rope, float* q_s, float& own_k, float& own_v) {
    const int tid = threadIdx.x, kvh = h / (n_q / n_kv);
    const float* qp = q + (size_t)t * ldq + (size_t)h * head_dim;
    if (tid >= head_dim) return;
    float own_q = qp[tid];
    if constexpr (ROPE) {
        const float* row = q + (size_t)t * ldq;
        const float* kp = row + (size_t)(n_q + kvh) * head_dim;
        own_v = row[(size_t)(n_q + n_kv + kvh) * head_dim + tid];
        own_k = kp[tid];
        if (tid < rope.rotary_dim) {
            const int half = rope.rotary_dim / 2, i = tid < half ? tid : tid - half;
            const bool have = p < rope.table_positions;
            const float c = have ? rope.cos_t[(size_t)p * half + i] : 1.f, sn = have ? rope.sin_t[(size_t)p * half + i] : 0.f;
            float y1, y2;
            rotate_pair(qp[i], qp[i + half], c, sn, y1, y2);
            own_q = tid < half ? y1 : y2;
            rotate_pair(kp[i], kp[i + half], c, sn, y1, y2);
            own_k = tid < half ? y1 : y2;
        }
        if (h % (n_q / n_kv) == 0) {
            const size_t at = ssb_cache_row(page_table, max_pages, s, p, page_shift, n_kv, kvh, head_dim) + tid;
            rope.k_cache[at] = own_k;
            rope.v_cache[at] = own_v;
        }
    }
    q_s[tid] = own_q;
}

// Where rows are few: all of a chunk's values and the next chunk's keys are on their way while the scores and their sums are made.
static size_t attention_staged_smem(int head_dim, int v_dim) {
    return sizeof(float) * (size_t)ATT_THREADS * (head_dim + 4 + v_dim);
}

template <bool ROPE>
__global__ void __launch_bounds__(ATT_THREADS)
attention_staged_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                        const int* __restrict__ pos, const int* __restrict__ slot, const int* __restrict__ page_table,
                        int max_pages, float* __restrict__ out, int ldo, int n_q, int n_kv, int head_dim, int page_shift,
                        int window, float scale, int v_dim, int v_row, const float* __restrict__ sinks, AsRope rope) {
    extern __shared__ __align__(16) float as_smem[];
    __shared__ __align__(16) float q_s[AS_MAX_DIM];
    __shared__ __align__(16) float p_s[ATT_THREADS];
    __shared__ size_t tok_s[2][ATT_THREADS];             // a chunk's keys: their rows in the cache entry
    __shared__ float red[ATT_THREADS / 32 + 1];
    const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ld = head_dim + 4;
    float* k_s = as_smem;                                // [key][head_dim + 4]
    float* v_s = k_s + ATT_THREADS * ld;                 // [key][v_dim]
    float* o = out + (size_t)t * ldo + (size_t)h * v_dim;
    ssb_pdl_launch_dependents();
    ssb_pdl_wait();
    const int s = slot[t];
    if (s < 0) {
        for (int d = tid; d < v_dim; d += ATT_THREADS) o[d] = 0.f;
        return;
    }
    const int p = pos[t];
    const int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
    const int kvh = h / (n_q / n_kv);
    const int kq = head_dim / 4, vq = v_dim / 4;
    auto look_up = [&](int base, int buf) {
        if (base + tid <= p) tok_s[buf][tid] = ssb_cache_row(page_table, max_pages, s, base + tid, page_shift, n_kv, kvh, 1);
    };
    auto fetch = [&](const float* src, int row, int quads, float* dst, int dst_ld, int base, int buf) {
        const int n = min(ATT_THREADS, p - base + (ROPE ? 0 : 1)) * quads;           // ROPE: the token's own is not there yet
        for (int e = tid; e < n; e += ATT_THREADS) {
            const int r = e / quads, c = e % quads * 4;
            gf_cp16(dst + r * dst_ld + c, src + tok_s[buf][r] * row + c, 16);
        }
        gf_commit();
    };
    look_up(lo, 0);
    float own_k = 0.f, own_v = 0.f;                      // ROPE: an element of the token's key and value
    attention_own_rows<ROPE>(q, ldq, t, h, s, p, n_q, n_kv, head_dim, page_table, max_pages, page_shift, rope, q_s, own_k, own_v);
    __syncthreads();
    fetch(k_cache, head_dim, kq, k_s, ld, lo, 0);
    float m = -INFINITY, l = 0.f, acc = 0.f;
    int buf = 0;
    for (int base = lo; base <= p; base += ATT_THREADS, buf ^= 1) {
        fetch(v_cache, v_row, vq, v_s, v_dim, base, buf);
        look_up(base + ATT_THREADS, buf ^ 1);
        if (ROPE && p - base < ATT_THREADS && tid < head_dim) {
            k_s[(p - base) * ld + tid] = own_k;
            v_s[(p - base) * v_dim + tid] = own_v;
        }
        gf_wait<1>();
        __syncthreads();                                 // the keys have landed
        float sc = -INFINITY;
        if (base + tid <= p) {
            const float* kr = k_s + tid * ld;
            float dot = 0.f;
#pragma unroll 8
            for (int d = 0; d < head_dim; d += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(kr + d);
                const float4 q4 = *reinterpret_cast<const float4*>(q_s + d);
                dot = fmaf(q4.x, k4.x, dot);
                dot = fmaf(q4.y, k4.y, dot);
                dot = fmaf(q4.z, k4.z, dot);
                dot = fmaf(q4.w, k4.w, dot);
            }
            sc = dot * scale;
        }
        float cm = sc;
#pragma unroll
        for (int i = 16; i > 0; i >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, i));
        if (lane == 0) red[warp] = cm;
        __syncthreads();                                 // and everyone is done with the keys
        if (base + ATT_THREADS <= p) fetch(k_cache, head_dim, kq, k_s, ld, base + ATT_THREADS, buf ^ 1);
        else gf_commit();
        const float m_new = fmaxf(m, fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3])));
        p_s[tid] = (base + tid <= p) ? expf(sc - m_new) : 0.f;
        __syncthreads();
        if (warp == 0) {                                 // the tree of block_reduce_sum: i with i + 64, then i + 32, ...
            float cs = (p_s[lane] + p_s[lane + 64]) + (p_s[lane + 32] + p_s[lane + 96]);
#pragma unroll
            for (int i = 16; i > 0; i >>= 1) cs += __shfl_down_sync(0xffffffffu, cs, i);
            if (lane == 0) red[ATT_THREADS / 32] = cs;
        }
        gf_wait<1>();
        __syncthreads();                                 // the values have landed, the sum is there
        const float alpha = (m == -INFINITY) ? 0.f : expf(m - m_new);
        l = l * alpha + red[ATT_THREADS / 32];
        if (tid < v_dim) {
            const int n_in = min(ATT_THREADS, p - base + 1);
            acc *= alpha;
            int j = 0;
            for (; j + 8 <= n_in; j += 8) {
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = v_s[(j + i) * v_dim + tid];
                const float4 a = *reinterpret_cast<const float4*>(p_s + j), b = *reinterpret_cast<const float4*>(p_s + j + 4);
                acc = fmaf(a.x, v[0], acc); acc = fmaf(a.y, v[1], acc); acc = fmaf(a.z, v[2], acc); acc = fmaf(a.w, v[3], acc);
                acc = fmaf(b.x, v[4], acc); acc = fmaf(b.y, v[5], acc); acc = fmaf(b.z, v[6], acc); acc = fmaf(b.w, v[7], acc);
            }
            for (; j < n_in; ++j) acc = fmaf(p_s[j], v_s[j * v_dim + tid], acc);
        }
        m = m_new;
        __syncthreads();                                 // everyone is done with the values and the weights
    }
    float keep = 1.f;
    if (sinks != nullptr) {
        const float sk = sinks[h];
        const float m_all = fmaxf(m, sk);
        keep = (m == -INFINITY) ? 0.f : expf(m - m_all);
        l = l * keep + expf(sk - m_all);
    }
    if (tid < v_dim) o[tid] = l > 0.f ? acc * keep / l : 0.f;
}

// Where rows are many: a chunk's keys come in slices of SL dims, then its values in as many bytes a time, through a ring of STAGES
// of them that runs across chunks, 32 to 96 KB where whole chunks take 66 (heads of 64) or 132 (128), so that two to six blocks
// share an SM.  A block that is alone on its SM takes longer so: a meeting of the block and the addresses of a fetch for every slice
// (one sequence of 1,000 tokens, 32 heads of 128, 56 us and 46).  Bound by the issue slots where rows are many (64 sequences of
// 1,000 tokens, 32 heads over 8 of 128: 77 % busy, 47 % of the shared memory's cycles, 9.2 TB/s from L2), by a chunk's chain of
// products and meetings where few.
template <bool ROPE, int SL, int STAGES>
__global__ void __launch_bounds__(ATT_THREADS)
attention_ring_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                        const int* __restrict__ pos, const int* __restrict__ slot, const int* __restrict__ page_table,
                        int max_pages, float* __restrict__ out, int ldo, int n_q, int n_kv, int head_dim, int page_shift,
                        int window, float scale, int v_dim, int v_row, const float* __restrict__ sinks, AsRope rope) {
    static_assert(SL % 32 == 0, "pieces are exchanged so that eight neighbouring keys' start in eight groups of banks");
    constexpr int STAGE = ATT_THREADS * SL, PIECES = SL / 4;
    extern __shared__ __align__(16) float ar_smem[];     // [stage]: keys as [key][SL], values as [key][v_dim]
    __shared__ __align__(16) float q_s[AS_MAX_DIM];
    __shared__ __align__(16) float p_s[ATT_THREADS];
    __shared__ size_t tok_s[2][ATT_THREADS];             // a chunk's keys: their rows in the cache entry
    __shared__ float red[ATT_THREADS / 32 + 1];
    const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* o = out + (size_t)t * ldo + (size_t)h * v_dim;
    ssb_pdl_launch_dependents();
    ssb_pdl_wait();
    const int s = slot[t], p = pos[t];
    if (s < 0) {
        for (int d = tid; d < v_dim; d += ATT_THREADS) o[d] = 0.f;
        return;
    }
    const int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
    const int kvh = h / (n_q / n_kv);
    auto look_up = [&](int base, int buf) {
        if (base + tid <= p) tok_s[buf][tid] = ssb_cache_row(page_table, max_pages, s, base + tid, page_shift, n_kv, kvh, 1);
    };
    look_up(lo, 0);
    float own_k = 0.f, own_v = 0.f;                      // ROPE: an element of the token's key and value
    attention_own_rows<ROPE>(q, ldq, t, h, s, p, n_q, n_kv, head_dim, page_table, max_pages, page_shift, rope, q_s, own_k, own_v);
    __syncthreads();

    int v_keys = ATT_THREADS;                            // keys a stage of values holds: a multiple of 8
    while (v_keys * v_dim > STAGE) v_keys >>= 1;
    const int k_stages = (head_dim + SL - 1) / SL, v_stages = ATT_THREADS / v_keys, quads = v_dim / 4;
    auto place = [&](int key, int piece) {               // of a slice of a key's elements
        return key * SL + ((piece ^ (key & 7)) << 2);
    };
    int ahead_base = lo, ahead_stage = 0, ahead_slot = 0, ahead_buf = 0;          // the stage that is fetched next
    auto fetch = [&]() {
        // the chunk's keys, and those of them that are in the cache (ROPE: the token's own is not there yet)
        const int n = min(ATT_THREADS, p - ahead_base + 1), cached = ROPE ? min(n, p - ahead_base) : n;
        const int j0 = (ahead_stage - k_stages) * v_keys;
        if (n > 0 && j0 < n) {
            float* dst = ar_smem + ahead_slot * STAGE;
            if (j0 < 0) {
                if (ahead_stage == 0) look_up(ahead_base + ATT_THREADS, ahead_buf ^ 1);        // read from the next turn on
                const int d0 = ahead_stage * SL;
                for (int e = tid; e < cached * PIECES; e += ATT_THREADS) {
                    const int r = e / PIECES, c = e % PIECES;
                    if (d0 + c * 4 < head_dim) gf_cp16(dst + place(r, c), k_cache + tok_s[ahead_buf][r] * head_dim + d0 + c * 4, 16);
                }
                if (ROPE && cached < n && tid >= d0 && tid < min(d0 + SL, head_dim)) dst[place(cached, (tid - d0) / 4) + tid % 4] = own_k;
            } else {
                const int here = min(v_keys, cached - j0);
                for (int e = tid; e < here * quads; e += ATT_THREADS) {
                    const int r = e / quads, c = e % quads * 4;
                    gf_cp16(dst + r * v_dim + c, v_cache + tok_s[ahead_buf][j0 + r] * v_row + c, 16);
                }
                if (ROPE && cached < n && cached - j0 < v_keys && tid < v_dim) dst[(cached - j0) * v_dim + tid] = own_v;
            }
        }
        gf_commit();
        if (++ahead_slot == STAGES) ahead_slot = 0;
        if (++ahead_stage == k_stages + v_stages) { ahead_stage = 0; ahead_base += ATT_THREADS; ahead_buf ^= 1; }
    };
#pragma unroll 1
    for (int i = 0; i < STAGES - 1; ++i) {
        fetch();
        __syncthreads();                                 // the next chunk's places, where one was begun
    }
    int at = 0;                                          // the stage in work
    auto turn = [&]() -> const float* {
        gf_wait<STAGES - 2>();
        __syncthreads();                                 // it has landed, and everyone is done with the one before
        fetch();
        const float* src = ar_smem + at * STAGE;
        if (++at == STAGES) at = 0;
        return src;
    };
    float m = -INFINITY, l = 0.f, acc = 0.f;
    for (int base = lo; base <= p; base += ATT_THREADS) {
        const int n_in = min(ATT_THREADS, p - base + 1);
        float dot = 0.f;
        for (int st = 0; st < k_stages; ++st) {
            const float* src = turn();
            const float* qs = q_s + st * SL;
            if (tid < n_in) {
                auto add = [&](int c) {
                    const float4 k4 = *reinterpret_cast<const float4*>(src + place(tid, c));
                    const float4 q4 = *reinterpret_cast<const float4*>(qs + c * 4);
                    dot = fmaf(q4.x, k4.x, dot);
                    dot = fmaf(q4.y, k4.y, dot);
                    dot = fmaf(q4.z, k4.z, dot);
                    dot = fmaf(q4.w, k4.w, dot);
                };
                if (head_dim - st * SL >= SL) {
#pragma unroll 8
                    for (int c = 0; c < PIECES; ++c) add(c);
                } else {
                    for (int c = 0; c < (head_dim - st * SL) / 4; ++c) add(c);
                }
            }
        }
        const float sc = tid < n_in ? dot * scale : -INFINITY;
        float cm = sc;
#pragma unroll
        for (int i = 16; i > 0; i >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, i));
        if (lane == 0) red[warp] = cm;
        __syncthreads();
        const float m_new = fmaxf(m, fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3])));
        p_s[tid] = tid < n_in ? expf(sc - m_new) : 0.f;
        __syncthreads();
        if (warp == 0) {                                 // the tree of block_reduce_sum: i with i + 64, then i + 32, ...
            float cs = (p_s[lane] + p_s[lane + 64]) + (p_s[lane + 32] + p_s[lane + 96]);
#pragma unroll
            for (int i = 16; i > 0; i >>= 1) cs += __shfl_down_sync(0xffffffffu, cs, i);
            if (lane == 0) red[ATT_THREADS / 32] = cs;
        }
        const float alpha = (m == -INFINITY) ? 0.f : expf(m - m_new);
        acc *= alpha;
        for (int st = 0; st < v_stages; ++st) {
            const int j0 = st * v_keys, here = min(v_keys, n_in - j0);
            if (here <= 0) break;                        // the last chunk's keys
            const float* src = turn() + tid;
            if (st == 0) l = l * alpha + red[ATT_THREADS / 32];
            if (tid < v_dim) {
                int j = 0;
                for (; j + 8 <= here; j += 8) {
                    float v[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = src[(j + i) * v_dim];
                    const float4 a = *reinterpret_cast<const float4*>(p_s + j0 + j), b = *reinterpret_cast<const float4*>(p_s + j0 + j + 4);
                    acc = fmaf(a.x, v[0], acc); acc = fmaf(a.y, v[1], acc); acc = fmaf(a.z, v[2], acc); acc = fmaf(a.w, v[3], acc);
                    acc = fmaf(b.x, v[4], acc); acc = fmaf(b.y, v[5], acc); acc = fmaf(b.z, v[6], acc); acc = fmaf(b.w, v[7], acc);
                }
                for (; j < here; ++j) acc = fmaf(p_s[j0 + j], src[j * v_dim], acc);
            }
        }
        m = m_new;
    }
    gf_wait<0>();
    float keep = 1.f;
    if (sinks != nullptr) {
        const float sk = sinks[h];
        const float m_all = fmaxf(m, sk);
        keep = (m == -INFINITY) ? 0.f : expf(m - m_all);
        l = l * keep + expf(sk - m_all);
    }
    if (tid < v_dim) o[tid] = l > 0.f ? acc * keep / l : 0.f;
}

static bool attention_staged_takes(const void* k_cache, const void* v_cache, int head_dim, int v_dim, int v_row) {
    return head_dim <= AS_MAX_DIM && v_dim <= AS_MAX_DIM && !((head_dim | v_dim | v_row) & 3)
        && !(((uintptr_t)k_cache | (uintptr_t)v_cache) & 15);
}

// Whole chunks while the device holds all the blocks at once, else the ring, as deep as leaves the blocks of an SM room.  us of a
// decode step's launch, 1,000 tokens a sequence, 32 heads of 64 / 128, of a plain row a block (and its rotation), whole chunks and
// the ring: 4 sequences 91, 40, 37 / 109, 46, 60; 8 101, 41, 37 / 122, 92, 64; 16 120, 70, 56 / 203, 184, 103; 64 360, 193, 167 /
// 474, 643, 309.  Where heads of 64 still fit, the ring gains on long contexts and loses on short ones (8 sequences of 5 tokens
// 3.3 and 3.6).
template <bool ROPE>
static int attention_staged_launch(const float* q, int ldq, const float* k_cache, const float* v_cache, const int* pos, const int* slot,
                                   const int* page_table, int max_pages, float* out, int ldo, int n_tokens, int n_q, int n_kv,
                                   int head_dim, int page_shift, int window, float scale, int v_dim, int v_row, const float* sinks,
                                   AsRope rope, bool pdl, cudaStream_t stream) {
#define AS_LAUNCH(MOST, SMEM, ...) do { \
        auto kernel = __VA_ARGS__; \
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(MOST)); \
        if (e != cudaSuccess) return (int)e; \
        const int rc = ssb_launch(kernel, dim3(n_tokens, n_q), dim3(ATT_THREADS), SMEM, stream, pdl, q, ldq, k_cache, v_cache, pos, slot, \
                                  page_table, max_pages, out, ldo, n_q, n_kv, head_dim, page_shift, window, scale, v_dim, v_row, sinks, rope); \
        return rc ? rc : ssb_launch_status(); \
    } while (0)
#define AS_RING(SL, STAGES) AS_LAUNCH(STAGES * ATT_THREADS * SL * 4, STAGES * ATT_THREADS * SL * 4, attention_ring_kernel<ROPE, SL, STAGES>)
    const size_t whole = attention_staged_smem(head_dim, v_dim);
    const long long blocks = (long long)n_tokens * n_q, sms = ssb_sm_count(), room = (227 * 1024) / (whole + 4 * 1024);
    if (blocks <= room * sms)
        AS_LAUNCH(attention_staged_smem(AS_MAX_DIM, AS_MAX_DIM), whole, attention_staged_kernel<ROPE>);
    if (blocks <= 2 * sms) AS_RING(64, 3);
    if (blocks <= 3 * sms) AS_RING(64, 2);
    if (blocks <= 4 * sms) AS_RING(32, 3);
    AS_RING(32, 2);
#undef AS_RING
#undef AS_LAUNCH
}

// A float32 decode step: rotation, append and attention of one token a sequence in one launch, the bits of ssb_rope_append and
// ssb_attention_plain.  qkv: [q heads | k heads | v heads] a row, left as it is; rotary_dim even, up to head_dim.
SSB_API int ssb_attention_f32_decode(const float* qkv, int ld, const float* cos_t, const float* sin_t, int table_positions,
                                     int rotary_dim, float* k_cache, float* v_cache, const int* pos, const int* slot,
                                     const int* page_table, int max_pages, float* out, int ldo, int n_tokens, int n_q, int n_kv,
                                     int head_dim, int page_shift, int window, float scale, int pdl, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (head_dim <= 0 || n_kv <= 0 || n_q % n_kv || n_q > 65535 || rotary_dim < 0 || rotary_dim % 2 || rotary_dim > head_dim
        || (rotary_dim && (!cos_t || !sin_t)) || !attention_staged_takes(k_cache, v_cache, head_dim, head_dim, head_dim))
        return SSB_ERR_BAD_SIZE;
    const AsRope rope = {cos_t, sin_t, table_positions, rotary_dim, k_cache, v_cache};
    return attention_staged_launch<true>(qkv, ld, k_cache, v_cache, pos, slot, page_table, max_pages, out, ldo, n_tokens, n_q, n_kv,
                                         head_dim, page_shift, window, scale, head_dim, head_dim, nullptr, rope, pdl != 0, stream);
}

SSB_API int ssb_attention_plain(const void* q, int ldq, int dtype, const void* k_cache,
                                const void* v_cache, const int* pos, const int* slot,
                                const int* page_table, int max_pages, void* out, int ldo, int n_tokens,
                                int n_q, int n_kv, int head_dim, int page_shift, int window, float scale,
                                int v_dim, int v_row, const float* sinks, int pdl, cudaStream_t stream) {
    // v_dim: width of a value and of a head's output; v_row: elements between the value rows of
    // consecutive tokens (values may be the first v_dim elements of the key rows: pass the key
    // store as v_cache and v_row = head_dim); sinks: one float per query head, or null
    if (n_tokens <= 0) return 0;
    if (head_dim > ATT_MAX_HEAD_DIM || head_dim <= 0 || n_kv <= 0 || n_q % n_kv) return SSB_ERR_BAD_SIZE;
    if (v_dim <= 0 || v_dim > ATT_MAX_HEAD_DIM || v_row < v_dim) return SSB_ERR_BAD_SIZE;
    dim3 grid(n_tokens, n_q);
    if (dtype == SSB_F32 && attention_staged_takes(k_cache, v_cache, head_dim, v_dim, v_row))
        return attention_staged_launch<false>((const float*)q, ldq, (const float*)k_cache, (const float*)v_cache, pos, slot,
                                              page_table, max_pages, (float*)out, ldo, n_tokens, n_q, n_kv, head_dim, page_shift,
                                              window, scale, v_dim, v_row, sinks, AsRope{}, pdl != 0, stream);
    if (dtype == SSB_F32)
        attention_plain_kernel<float><<<grid, ATT_THREADS, 0, stream>>>(
            (const float*)q, ldq, (const float*)k_cache, (const float*)v_cache, pos, slot, page_table,
            max_pages, (float*)out, ldo, n_q, n_kv, head_dim, page_shift, window, scale, v_dim, v_row, sinks);
    else if (dtype == SSB_BF16)
        attention_plain_kernel<bf16><<<grid, ATT_THREADS, 0, stream>>>(
            (const bf16*)q, ldq, (const bf16*)k_cache, (const bf16*)v_cache, pos, slot, page_table,
            max_pages, (bf16*)out, ldo, n_q, n_kv, head_dim, page_shift, window, scale, v_dim, v_row, sinks);
    else
        return SSB_ERR_BAD_DTYPE;
    return ssb_launch_status();
}

// The same attention for a step of float32 prompts: the new tokens of each sequence seq_start .. of slot seq_slot, at packed
// rows cu_new[b] .. cu_new[b + 1] - 1 (attention_f32.cuh).  head_dim 64 or 128, values as wide as keys.
SSB_API int ssb_attention_f32_prompt(const float* q, int ldq, const float* k_cache, const float* v_cache, const int* cu_new,
                                     const int* seq_start, const int* seq_slot, const int* page_table, int max_pages,
                                     float* out, int ldo, int n_seqs, int max_new, int n_q, int n_kv, int head_dim,
                                     int page_shift, float scale, cudaStream_t stream) {
    if (n_seqs <= 0 || max_new <= 0) return 0;
    if ((head_dim != 64 && head_dim != 128) || n_kv <= 0 || n_kv > 65535 || n_seqs > 65535 || n_q % n_kv) return SSB_ERR_BAD_SIZE;
    if ((((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) & 15) || ((ldq | ldo) & 3)) return SSB_ERR_BAD_SIZE;
    const long long tiles = ((long long)max_new * (n_q / n_kv) + AF_ROWS - 1) / AF_ROWS;
    if (tiles > 0x7fffffffLL) return SSB_ERR_BAD_SIZE;
    const dim3 grid((unsigned)tiles, n_kv, n_seqs);
#define SSB_AF(HD) do { \
        const cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                   (int)attention_f32_smem<HD>()); \
        if (e != cudaSuccess) return (int)e; \
        attention_f32_kernel<HD><<<grid, AF_THREADS, attention_f32_smem<HD>(), stream>>>( \
            q, ldq, k_cache, v_cache, cu_new, seq_start, seq_slot, page_table, max_pages, out, ldo, n_q, n_kv, page_shift, scale); \
    } while (0)
    if (head_dim == 64) SSB_AF(64); else SSB_AF(128);
#undef SSB_AF
    return ssb_launch_status();
}

// ---------------------------------------------------------------------------------------
// A gated unit's inner step: z[t, c] = gate_fn(gate[t, c], up[t, c]) * row_scale[t] (ssb_gate: silu(g) u, or the
// clamped form g' sigmoid(1.702 g') (u' + 1), or gelu(g) u).  Gate and up are the two halves of a row, or (interleaved) come as
// [8 gate | 8 up] per 16 columns.  row_scale: one float32 factor per row, or none.
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void gated_activation_kernel(const T* __restrict__ gu, int ld, T* __restrict__ z, int ldz, int inter,
                                        size_t total, int interleaved, int kind, float limit,
                                        const float* __restrict__ row_scale) {
    ssb_pdl_launch_dependents();
    ssb_pdl_wait();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const size_t t = idx / inter;
    const int c = (int)(idx % inter);
    const int cg = interleaved ? (c / 8) * 16 + (c % 8) : c;
    const int cu = interleaved ? cg + 8 : inter + c;
    const float g = ssb_to_float(gu[t * ld + cg]);
    const float u = ssb_to_float(gu[t * ld + cu]);
    const float r = row_scale ? row_scale[t] : 1.0f;
    z[t * ldz + c] = ssb_from_float<T>(ssb_gate(g, u, kind, limit) * r);
}

SSB_API int ssb_gated_activation(const void* gate_up, int ld, void* z, int ldz, int dtype, int n_tokens, int inter,
                                 int interleaved, int kind, float limit, const float* row_scale, int pdl,
                                 cudaStream_t stream) {
    if ((interleaved && inter % 8) || kind < 0 || kind > SSB_GATE_LAST) return SSB_ERR_BAD_SIZE;
    const size_t total = (size_t)n_tokens * inter;
    if (total == 0) return 0;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    int rc;
    if (dtype == SSB_F32)
        rc = ssb_launch(gated_activation_kernel<float>, dim3(blocks), dim3(256), 0, stream, pdl != 0, (const float*)gate_up,
                        ld, (float*)z, ldz, inter, total, interleaved, kind, limit, row_scale);
    else if (dtype == SSB_BF16)
        rc = ssb_launch(gated_activation_kernel<bf16>, dim3(blocks), dim3(256), 0, stream, pdl != 0, (const bf16*)gate_up,
                        ld, (bf16*)z, ldz, inter, total, interleaved, kind, limit, row_scale);
    else
        return SSB_ERR_BAD_DTYPE;
    return rc ? rc : ssb_launch_status();
}

SSB_API int ssb_swiglu(const void* gate_up, int ld, void* z, int ldz, int dtype, int n_tokens, int inter,
                       int interleaved, cudaStream_t stream) {
    return ssb_gated_activation(gate_up, ld, z, ldz, dtype, n_tokens, inter, interleaved, SSB_GATE_SILU, 0.f, nullptr, 0,
                                stream);
}

// ---------------------------------------------------------------------------------------
// A sublayer's result joins the stream through a norm of its own:
//     residual[t] += branch[t] / sqrt(mean(branch[t]^2) + eps) * w
// (w float32, the multiplier itself: a weight stored around zero arrives as 1 + w).  Optionally the branch row is
// zeroed behind the read, so that the next sublayer's products can add into it again, and optionally the norm
// that the next sublayer reads is taken of the new stream in the same pass:
//     next_out[t] = residual[t] / sqrt(mean(residual[t]^2) + next_eps) * next_w,
// or, where the next sublayer reads the stream without a norm (no next_w), the new stream itself in its type.
// One block per token, the row in shared memory, sums in a fixed order.
// ---------------------------------------------------------------------------------------
constexpr int RA_THREADS = 256;

__device__ __forceinline__ float ra_block_sum(float v, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < RA_THREADS / 32; ++w) s += red[w];
    return s;
}

template <typename T>
__global__ void __launch_bounds__(RA_THREADS)
rms_add_kernel(float* __restrict__ residual, float* __restrict__ branch, const float* __restrict__ w, float eps, int width,
               int clear, const float* __restrict__ next_w, float next_eps, T* __restrict__ next_out) {
    extern __shared__ float ra_row[];
    __shared__ float red[RA_THREADS / 32];
    ssb_pdl_launch_dependents();
    ssb_pdl_wait();
    const size_t t = blockIdx.x;
    const int tid = threadIdx.x;
    float* br = branch + t * width;
    float* rr = residual + t * width;
    // four-byte accesses a thread, the stream's row read behind the branch's sum: 33 us for 2,048 rows of 2,048; with
    // sixteen-byte accesses the same kernel took 87 us, with both rows staged in shared memory up front 49
    float sq = 0.f;
    for (int c = tid; c < width; c += RA_THREADS) {
        const float v = br[c];
        ra_row[c] = v;
        sq = fmaf(v, v, sq);
        if (clear) br[c] = 0.f;
    }
    const float inv = 1.0f / sqrtf(ra_block_sum(sq, red) / (float)width + eps);
    float sq2 = 0.f;
    for (int c = tid; c < width; c += RA_THREADS) {
        const float v = rr[c] + ra_row[c] * inv * w[c];
        rr[c] = v;
        ra_row[c] = v;
        sq2 = fmaf(v, v, sq2);
    }
    if (next_out == nullptr) return;
    if (next_w == nullptr) {
        for (int c = tid; c < width; c += RA_THREADS) next_out[t * width + c] = ssb_from_float<T>(ra_row[c]);
        return;
    }
    const float inv2 = 1.0f / sqrtf(ra_block_sum(sq2, red) / (float)width + next_eps);
    for (int c = tid; c < width; c += RA_THREADS)
        next_out[t * width + c] = ssb_from_float<T>(ra_row[c] * inv2 * next_w[c]);
}

SSB_API int ssb_rms_add(float* residual, float* branch, const float* w, float eps, int n_tokens, int width, int clear,
                        const float* next_w, float next_eps, void* next_out, int next_dtype, int pdl, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (width <= 0 || (size_t)width * sizeof(float) > 200 * 1024) return SSB_ERR_BAD_SIZE;
    const size_t smem = (size_t)width * sizeof(float);
    int rc;
#define SSB_RA(TYPE)                                                                                                 \
    {                                                                                                                \
        auto kern = rms_add_kernel<TYPE>;                                                                            \
        if (smem > 48 * 1024) {                                                                                      \
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);      \
            if (e != cudaSuccess) return (int)e;                                                                     \
        }                                                                                                            \
        rc = ssb_launch(kern, dim3(n_tokens), dim3(RA_THREADS), smem, stream, pdl != 0, residual, branch, w, eps,    \
                        width, clear, next_w, next_eps, (TYPE*)next_out);                                            \
    }
    if (next_out == nullptr || next_dtype == SSB_F32) SSB_RA(float)
    else if (next_dtype == SSB_BF16) SSB_RA(bf16)
    else return SSB_ERR_BAD_DTYPE;
#undef SSB_RA
    return rc ? rc : ssb_launch_status();
}

// ---------------------------------------------------------------------------------------
// y[t, c] *= sigmoid(g[t, c]): concatenated heads times a gate of their own, element by element
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void sigmoid_gate_kernel(T* __restrict__ y, int ldy, const T* __restrict__ g, int ldg, int width, size_t total) {
    ssb_pdl_launch_dependents();
    ssb_pdl_wait();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const size_t t = idx / width;
    const int c = (int)(idx % width);
    T* p = y + t * ldy + c;
    *p = ssb_from_float<T>(ssb_to_float(*p) / (1.0f + expf(-ssb_to_float(g[t * ldg + c]))));
}

// float32 rows in another type: a stream read without a norm
template <typename T>
__global__ void round_rows_kernel(const float* __restrict__ x, T* __restrict__ out, size_t total) {
    ssb_pdl_launch_dependents();
    ssb_pdl_wait();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < total) out[idx] = ssb_from_float<T>(x[idx]);
}

SSB_API int ssb_round_rows(const float* x, void* out, int dtype, long long total, int pdl, cudaStream_t stream) {
    if (total <= 0) return 0;
    if (total > (1ll << 38)) return SSB_ERR_BAD_SIZE;
    const dim3 grid((unsigned)((total + 255) / 256));
    int rc;
    if (dtype == SSB_F32)
        rc = ssb_launch(round_rows_kernel<float>, grid, dim3(256), 0, stream, pdl != 0, x, (float*)out, (size_t)total);
    else if (dtype == SSB_BF16)
        rc = ssb_launch(round_rows_kernel<bf16>, grid, dim3(256), 0, stream, pdl != 0, x, (bf16*)out, (size_t)total);
    else
        return SSB_ERR_BAD_DTYPE;
    return rc ? rc : ssb_launch_status();
}

SSB_API int ssb_sigmoid_gate(void* y, int ldy, const void* g, int ldg, int dtype, int n_tokens, int width, int pdl,
                             cudaStream_t stream) {
    const size_t total = (size_t)n_tokens * width;
    if (n_tokens <= 0 || width <= 0) return 0;
    const dim3 grid((unsigned)((total + 255) / 256));
    int rc;
    if (dtype == SSB_F32)
        rc = ssb_launch(sigmoid_gate_kernel<float>, grid, dim3(256), 0, stream, pdl != 0, (float*)y, ldy, (const float*)g, ldg,
                        width, total);
    else if (dtype == SSB_BF16)
        rc = ssb_launch(sigmoid_gate_kernel<bf16>, grid, dim3(256), 0, stream, pdl != 0, (bf16*)y, ldy, (const bf16*)g, ldg,
                        width, total);
    else
        return SSB_ERR_BAD_DTYPE;
    return rc ? rc : ssb_launch_status();
}

// ---------------------------------------------------------------------------------------
// An activation between two dense products: z[t, c] = act(u[t, c]) * scale, in float32.
//   kind 0: relu(u)^2;  1: gelu with tanh, 0.5 u (1 + tanh(sqrt(2/pi) (u + 0.044715 u^3)));  2: silu
//   (ssb_activate, shared with the kernels that apply it where they finish a product)
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void activation_kernel(const T* __restrict__ u, int ld, T* __restrict__ z, int ldz, int width, size_t total,
                                  int kind, float scale) {
    ssb_pdl_launch_dependents();
    ssb_pdl_wait();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const size_t t = idx / width;
    const int c = (int)(idx % width);
    z[t * ldz + c] = ssb_from_float<T>(ssb_activate(ssb_to_float(u[t * ld + c]), kind) * scale);
}

SSB_API int ssb_activation(const void* u, int ld, void* z, int ldz, int dtype, int n_tokens, int width, int kind,
                           float scale, int pdl, cudaStream_t stream) {
    if (kind < 0 || kind > 2) return SSB_ERR_BAD_SIZE;
    const size_t total = (size_t)n_tokens * width;
    if (total == 0) return 0;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    int rc;
    if (dtype == SSB_F32)
        rc = ssb_launch(activation_kernel<float>, dim3(blocks), dim3(256), 0, stream, pdl != 0, (const float*)u, ld, (float*)z,
                        ldz, width, total, kind, scale);
    else if (dtype == SSB_BF16)
        rc = ssb_launch(activation_kernel<bf16>, dim3(blocks), dim3(256), 0, stream, pdl != 0, (const bf16*)u, ld, (bf16*)z,
                        ldz, width, total, kind, scale);
    else
        return SSB_ERR_BAD_DTYPE;
    return rc ? rc : ssb_launch_status();
}

// ---------------------------------------------------------------------------------------
// out (float32) += x
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void add_into_kernel(float* __restrict__ out, const T* __restrict__ x, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += ssb_to_float(x[i]);
}

SSB_API int ssb_add_into(float* out, const void* x, int x_dtype, long long n, cudaStream_t stream) {
    if (n <= 0) return 0;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (x_dtype == SSB_F32) add_into_kernel<float><<<blocks, 256, 0, stream>>>(out, (const float*)x, (size_t)n);
    else if (x_dtype == SSB_BF16) add_into_kernel<bf16><<<blocks, 256, 0, stream>>>(out, (const bf16*)x, (size_t)n);
    else return SSB_ERR_BAD_DTYPE;
    return ssb_launch_status();
}

// ---------------------------------------------------------------------------------------
// x (float32) *= s
// ---------------------------------------------------------------------------------------
__global__ void scale_kernel(float* __restrict__ x, float s, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] *= s;
}

SSB_API int ssb_scale(float* x, float s, long long n, cudaStream_t stream) {
    if (n <= 0) return 0;
    scale_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(x, s, (size_t)n);
    return ssb_launch_status();
}

// ---------------------------------------------------------------------------------------
// out[e] = sum_{j < n_terms} w[j] * streams[j * stride + e]: a weighted sum of the first n_terms of a
// stack of float32 streams, added in the order of j
// ---------------------------------------------------------------------------------------
__global__ void stream_mix_kernel(const float* __restrict__ streams, size_t stride, const float* __restrict__ w,
                                  int n_terms, float* __restrict__ out, size_t n) {
    ssb_pdl_launch_dependents();
    ssb_pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float acc = 0.f;
    for (int j = 0; j < n_terms; ++j) acc = fmaf(w[j], streams[(size_t)j * stride + i], acc);
    out[i] = acc;
}

// The same sums, four elements a thread and the terms' loads in groups of four (2,048 x 2,048,
// two to five terms: 35 us a launch with one element a thread, 25 so).
__global__ void __launch_bounds__(256)
stream_mix_vec_kernel(const float4* __restrict__ streams, size_t stride, const float* __restrict__ w, int n_terms,
                      float4* __restrict__ out, size_t n) {
    constexpr int AHEAD = 4;
    ssb_pdl_launch_dependents();
    ssb_pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j0 = 0; j0 < n_terms; j0 += AHEAD) {
        float4 v[AHEAD];
#pragma unroll
        for (int j = 0; j < AHEAD; ++j)
            if (j0 + j < n_terms) v[j] = streams[(size_t)(j0 + j) * stride + i];
#pragma unroll
        for (int j = 0; j < AHEAD; ++j)
            if (j0 + j < n_terms) {
                const float s = w[j0 + j];
                acc.x = fmaf(s, v[j].x, acc.x);
                acc.y = fmaf(s, v[j].y, acc.y);
                acc.z = fmaf(s, v[j].z, acc.z);
                acc.w = fmaf(s, v[j].w, acc.w);
            }
    }
    out[i] = acc;
}

SSB_API int ssb_stream_mix(const float* streams, long long stride, const float* w, int n_terms, float* out,
                           long long n, int pdl, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (n_terms <= 0) return SSB_ERR_BAD_SIZE;
    if (n % 4 == 0 && stride % 4 == 0 && (((uintptr_t)streams | (uintptr_t)out) & 15) == 0) {
        const int st = ssb_launch(stream_mix_vec_kernel, dim3((unsigned)((n / 4 + 255) / 256)), dim3(256), 0, stream, pdl != 0,
                                  (const float4*)streams, (size_t)stride / 4, w, n_terms, (float4*)out, (size_t)n / 4);
        return st ? st : ssb_launch_status();
    }
    const int rc = ssb_launch(stream_mix_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, pdl != 0,
                              streams, (size_t)stride, w, n_terms, out, (size_t)n);
    return rc ? rc : ssb_launch_status();
}
