// Causal attention of float32 prompts over the paged cache, many rows of one kv head a block.
//
// Every sum is attention_plain_kernel's, bit for bit: keys in chunks of 128 from the sequence's first one, a score one FMA
// chain over the head's dims, a chunk's weights added in the same tree (key i with i + 64, then i + 32, ..., i + 1), the
// weighted values one FMA chain over the chunk's keys on the rescaled sum.  What changes is the work that is shared: a
// chunk's keys and values are fetched once for 64 (token, head) rows instead of once a row, and the products run in
// register tiles.  Prompts of 100, 500, 333, 1 and 9 tokens, 32 heads over 8 of 64: 1,976 us a row a block, 105 us here.
#pragma once
#include "common.cuh"
#include "gemm_f32.cuh"
#include <math.h>

constexpr int AF_ROWS = 64, AF_KEYS = 128, AF_THREADS = 256;

template <bool V> struct AfFlag { static constexpr bool value = V; };

template <int HD>
constexpr size_t attention_f32_smem() {
    return sizeof(float) * ((size_t)(AF_ROWS + AF_KEYS) * (HD + 4) + (size_t)AF_ROWS * (AF_KEYS + 4));
}

template <int HD>
__global__ void __launch_bounds__(AF_THREADS)
attention_f32_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                     const int* __restrict__ cu_new, const int* __restrict__ seq_start, const int* __restrict__ seq_slot,
                     const int* __restrict__ page_table, int max_pages, float* __restrict__ out, int ldo, int n_q, int n_kv,
                     int page_shift, float scale) {
    constexpr int LD = HD + 4, PLD = AF_KEYS + 4, DQ = HD / 64;       // DQ: groups of four dims a thread owns
    extern __shared__ __align__(16) float af_smem[];
    float* q_s = af_smem;                                             // [row][dim]
    float* kv_s = q_s + AF_ROWS * LD;                                 // [key][dim]: a chunk's keys, then its values
    float* p_s = kv_s + AF_KEYS * LD;                                 // [row][key]
    const int b = blockIdx.z, kvh = blockIdx.y, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int t0 = cu_new[b], n_new = cu_new[b + 1] - t0, start = seq_start[b], slot = seq_slot[b];
    const int G = n_q / n_kv, n_rows = n_new * G;
    const int row0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * AF_ROWS;          // the longest rows first
    if (row0 >= n_rows) return;
    const int* pt = page_table + (size_t)(slot < 0 ? 0 : slot) * max_pages;

    int tok[4], head[4], pos[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int R = row0 + ty + 16 * i;
        tok[i] = R < n_rows ? R / G : -1;
        head[i] = kvh * G + R % G;
        pos[i] = R < n_rows && slot >= 0 ? start + tok[i] : -1;
    }
    const int p_last = slot < 0 ? -1 : start + min(n_rows - 1, row0 + AF_ROWS - 1) / G;
    const int p_first = start + row0 / G;
    for (int e = tid; e < AF_ROWS * (HD / 4); e += AF_THREADS) {
        const int r = e / (HD / 4), c = e % (HD / 4), R = row0 + r;
        const bool in = R < n_rows;
        const float* src = in ? q + (size_t)(t0 + R / G) * ldq + (size_t)(kvh * G + R % G) * HD + c * 4 : q;
        gf_cp16(q_s + r * LD + c * 4, src, in ? 16 : 0);
    }
    // keys or values base .. base + 127 of the sequence; zeros past the block's last position
    auto load = [&](const float* cache, int base) {
        for (int e = tid; e < AF_KEYS * (HD / 4); e += AF_THREADS) {
            const int r = e / (HD / 4), c = e % (HD / 4), key = base + r;
            const bool in = key <= p_last;
            const float* src = cache;
            if (in) {
                const size_t tk = (((size_t)pt[key >> page_shift] * n_kv + kvh) << page_shift) + (key & ((1 << page_shift) - 1));
                src = cache + tk * HD + c * 4;
            }
            gf_cp16(kv_s + r * LD + c * 4, src, in ? 16 : 0);
        }
        gf_commit();
    };

    float m[4], l[4], acc[4][DQ * 4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
        for (int d = 0; d < DQ * 4; ++d) acc[i][d] = 0.f;
    }
    for (int base = 0; base <= p_last; base += AF_KEYS) {
        __syncthreads();                                              // the values of the chunk before are done with
        load(k_cache, base);
        gf_wait<0>();
        __syncthreads();
        float s[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) s[i][j] = 0.f;
#pragma unroll 2
        for (int d = 0; d < HD; d += 4) {
            float4 kk[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) kk[j] = *reinterpret_cast<const float4*>(kv_s + (tx + 16 * j) * LD + d);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(q_s + (ty + 16 * i) * LD + d);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    s[i][j] = fmaf(a.x, kk[j].x, s[i][j]);
                    s[i][j] = fmaf(a.y, kk[j].y, s[i][j]);
                    s[i][j] = fmaf(a.z, kk[j].z, s[i][j]);
                    s[i][j] = fmaf(a.w, kk[j].w, s[i][j]);
                }
            }
        }
        __syncthreads();                                              // the keys are done with: the values come over them
        load(v_cache, base);
        float alpha[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                s[i][j] = base + tx + 16 * j <= pos[i] ? s[i][j] * scale : -INFINITY;
                mx = fmaxf(mx, s[i][j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(m[i], mx);
            float p[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                p[j] = base + tx + 16 * j <= pos[i] ? expf(s[i][j] - m_new) : 0.f;
                p_s[(ty + 16 * i) * PLD + tx + 16 * j] = p[j];
            }
            // the tree over 128 keys: 64 and 32 and 16 apart in this thread, then 8, 4, 2, 1 across the lanes
#pragma unroll
            for (int h = 4; h > 0; h >>= 1)
#pragma unroll
                for (int j = 0; j < h; ++j) p[j] = __fadd_rn(p[j], p[j + h]);
            float sum = p[0];
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
            alpha[i] = (m[i] == -INFINITY) ? 0.f : expf(m[i] - m_new);
            if (base <= pos[i]) {                                     // a row that ends before this chunk stays as it is
                l[i] = fmaf(l[i], alpha[i], sum);
                m[i] = m_new;
            } else {
                alpha[i] = 1.f;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int d = 0; d < DQ * 4; ++d) acc[i][d] *= alpha[i];
        gf_wait<0>();
        __syncthreads();
        const int n_keys = min(AF_KEYS, p_last + 1 - base);
        // on the diagonal a row takes the keys it sees and no other (a weight of zero would still spread an infinity)
        const bool edge = base + n_keys - 1 > p_first || row0 + AF_ROWS > n_rows;
        auto add = [&](int jj, auto guarded) {
#pragma unroll
            for (int g = 0; g < DQ; ++g) {
                const float4 v = *reinterpret_cast<const float4*>(kv_s + jj * LD + g * 64 + tx * 4);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float p = p_s[(ty + 16 * i) * PLD + jj];
                    if (!decltype(guarded)::value || base + jj <= pos[i]) {
                        acc[i][g * 4] = fmaf(p, v.x, acc[i][g * 4]);
                        acc[i][g * 4 + 1] = fmaf(p, v.y, acc[i][g * 4 + 1]);
                        acc[i][g * 4 + 2] = fmaf(p, v.z, acc[i][g * 4 + 2]);
                        acc[i][g * 4 + 3] = fmaf(p, v.w, acc[i][g * 4 + 3]);
                    }
                }
            }
        };
        if (edge) {
#pragma unroll 2
            for (int jj = 0; jj < n_keys; ++jj) add(jj, AfFlag<true>());
        } else {
#pragma unroll 4
            for (int jj = 0; jj < AF_KEYS; ++jj) add(jj, AfFlag<false>());
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (tok[i] < 0) continue;
        float* dst = out + (size_t)(t0 + tok[i]) * ldo + (size_t)head[i] * HD + tx * 4;
#pragma unroll
        for (int g = 0; g < DQ; ++g) {
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            if (l[i] > 0.f)
                o = make_float4(acc[i][g * 4] / l[i], acc[i][g * 4 + 1] / l[i], acc[i][g * 4 + 2] / l[i], acc[i][g * 4 + 3] / l[i]);
            *reinterpret_cast<float4*>(dst + g * 64) = o;
        }
    }
}
