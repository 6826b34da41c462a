// Latent attention of prompts on the fifth-generation tensor cores.
//
// Every head of a token attends over the same cached rows [latent (dv) | rotated key part] (dk elements, the values are
// the first dv of them).  A block takes 128 (token, head) rows of one sequence and up to 256 value columns: its query
// rows stay in shared memory, the sequence's keys come a page (64) at a time through a TMA ring (128-byte swizzle, boxes of 64
// dims) and serve twice, K-major for the scores and MN-major as the values.  A width above 256 is shared by two blocks
// that take the scores twice: the output of 128 rows and 512 columns alone would fill tensor memory.  Of the query rows
// the first 256 dims move to the columns of tensor memory that are left (an operand there costs no shared memory, neither
// room nor bandwidth), so that two pages of 576 elements a key fit beside the rest.  A tcgen05.mma of 128 rows takes about
// 70 cycles whether it has 32, 64 or 128 columns: with turns of 32 keys the scores alone bounded the kernel.
//
// Warp 0 feeds TMA, warp 1 issues tcgen05.mma as its inputs become ready (scores of the next page, or the weighted
// sum of the last), warps 2-5 own a row a thread: scores leave tensor memory, are masked on the edges, and return as
// weights over the place of the scores.  A weight enters the second product as the sum of two bfloat16 numbers (two
// MMAs), so that it keeps 16 bits of mantissa, as in latent_attention.cu.  A row's reference maximum is set by its first
// keys and moves only when later weights against it sum to more than 2^8; only then is the output rescaled.
//
// One prompt of 2,048 tokens, 16 heads, rows of 576: 705 us on mma.sync, 178 here (0.42 PFLOP/s; every weight goes through the
// second product twice); 8,192 tokens 9,718 and 2,381 us; 8 prompts of 300 tokens 168 and 73.  Bound by the chain of a turn:
// scores, weights and sum wait for one another, and tensor memory holds one output and one pair of turns (tensor pipe 39 % of
// the active cycles, issue slots 17 %, a warp's waits for what it loads 4.5 cycles an instruction).
#include "common.cuh"
#include "tc_helpers.cuh"
#include <math.h>

typedef __nv_bfloat16 bf16;

constexpr int LT_BM = 128;                 // (token, head) rows a block
constexpr int LT_BN = 64;                  // keys a turn: a page
constexpr int LT_NV = 256;                 // most value columns a block
constexpr int LT_MAX_STAGES = 5;
constexpr int LT_THREADS = 192;
constexpr float LT_LAZY_P = 256.f;         // how far a turn's weights may sum before a row's reference moves
constexpr uint32_t LT_BOX_Q = LT_BM * 128, LT_BOX_K = LT_BN * 128;     // 64 dims of the query rows; of a turn's keys
// tensor-memory columns: the output, the scores of two turns, 64 dims of the query rows per 32 columns
constexpr uint32_t LT_S0 = 256, LT_Q0 = 384;
constexpr int LT_TMEM_BOXES = 4;           // query boxes that fit behind them
constexpr int LT_NBARS = 2 + 2 * LT_MAX_STAGES + 6;
constexpr float LT_LOG2E = 1.4426950408889634f;

__device__ __forceinline__ bool lt_ready(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred P1;\nmbarrier.test_wait.parity.shared::cta.b64 P1, [%1], %2;\nselp.b32 %0, 1, 0, P1;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void lt_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void lt_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void lt_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void lt_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
                 "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                   "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                   "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
                 : "memory");
}
__device__ __forceinline__ void lt_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float lt_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Half of a turn's weighted sum: the weights' high (or low) parts, 32 columns of tensor memory, four steps of 16 keys, over
// the page's values (16 keys of 128 bytes a step).
__device__ __forceinline__ void lt_mma_values(uint32_t tmem_d, uint32_t tmem_p, uint64_t desc_v, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p, q;\n.reg .b32 a1, a2, a3;\n.reg .b64 b1, b2, b3;\n"
                 "setp.ne.b32 p, %4, 0;\nsetp.eq.b32 q, %5, 0;\n"
                 "add.u32 a1, %1, 8;\nadd.u32 a2, %1, 16;\nadd.u32 a3, %1, 24;\n"
                 "add.u64 b1, %2, 128;\nadd.u64 b2, %2, 256;\nadd.u64 b3, %2, 384;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, {%5, %5, %5, %5}, q;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, {%5, %5, %5, %5}, q;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, {%5, %5, %5, %5}, q;\n}"
                 ::"r"(tmem_d), "r"(tmem_p), "l"(desc_v), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// Four k-steps of 16 dims of the scores with the query rows in tensor memory (8 columns a step).
__device__ __forceinline__ void lt_mma_scores(uint32_t tmem_d, uint32_t tmem_q, uint64_t desc_k, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p, q;\n.reg .b32 a1, a2, a3;\n.reg .b64 b1, b2, b3;\n"
                 "setp.ne.b32 p, %4, 0;\nsetp.eq.b32 q, %5, 0;\n"
                 "add.u32 a1, %1, 8;\nadd.u32 a2, %1, 16;\nadd.u32 a3, %1, 24;\n"
                 "add.u64 b1, %2, 2;\nadd.u64 b2, %2, 4;\nadd.u64 b3, %2, 6;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, {%5, %5, %5, %5}, q;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, {%5, %5, %5, %5}, q;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, {%5, %5, %5, %5}, q;\n}"
                 ::"r"(tmem_d), "r"(tmem_q), "l"(desc_k), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// MN-major operand [key][dim] in boxes of 64 dims LT_BOX_K bytes apart (leading offset), groups of 8 keys 1024 bytes apart.
__device__ __forceinline__ uint64_t lt_desc_values(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(LT_BOX_K >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

__global__ void __launch_bounds__(LT_THREADS, 1)
latent_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                           const int* __restrict__ cu_new, const int* __restrict__ seq_start, const int* __restrict__ seq_slot,
                           const int* __restrict__ page_table, int max_pages, bf16* __restrict__ out,
                           const float* __restrict__ sinks, int n_heads, int boxes, int dv, int parts, int stages, int window,
                           float scale_log2, int* __restrict__ error_word) {
    extern __shared__ unsigned char lt_smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)lt_smem_raw + 1023) & ~(uintptr_t)1023);
    // query boxes that stay in shared memory, then the ring; the others pass through the ring on their way to tensor memory
    const int tm_boxes = min(boxes, LT_TMEM_BOXES), ss_boxes = boxes - tm_boxes;
    const uint32_t stage_bytes = boxes * LT_BOX_K, ring_bytes = max(stages * stage_bytes, tm_boxes * LT_BOX_Q);
    const uint32_t q_s = smem_u32(smem), k_s = q_s + ss_boxes * LT_BOX_Q;
    uint64_t* bars = (uint64_t*)(smem + ss_boxes * LT_BOX_Q + ring_bytes);
    // q_full, q_moved, k_full[stage], k_empty[stage], then one each for even and odd turns: s_full[2], p_full[2], o_full[2].  A
    // wait by parity tells a phase from the next one only.  The scores of a turn are issued after the weighted sum of the turn
    // two before, and that sum after the row's weights of its turn: whoever waits for a turn's barrier waits for the phase that
    // is open or for the last one that closed.  One o_full for all turns would not do: after the last weights two sums may
    // both end before a warp first looks.
    const uint32_t q_full = smem_u32(bars), q_moved = q_full + 8, k_full0 = q_moved + 8, k_empty0 = k_full0 + 8 * LT_MAX_STAGES,
                   s_full0 = k_empty0 + 8 * LT_MAX_STAGES, p_full0 = s_full0 + 16, o_full0 = p_full0 + 16;
    uint32_t* tmem_slot = (uint32_t*)(bars + LT_NBARS);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);   // [0]: a role gave up; [1]: stays zero

    const int b = blockIdx.x / parts, part = blockIdx.x % parts;
    const int t0 = cu_new[b], n_rows = (cu_new[b + 1] - t0) * n_heads, slot = seq_slot[b], start = seq_start[b];
    const int row0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * LT_BM;         // the tiles with most keys start first
    if (slot < 0 || row0 >= n_rows) return;
    const int rows_here = min(LT_BM, n_rows - row0);
    const int pos_first = start + row0 / n_heads, pos_last = start + (row0 + rows_here - 1) / n_heads;
    const int kb_lo = window > 0 ? max(0, pos_first - window + 1) / LT_BN : 0;
    const int turns = pos_last / LT_BN - kb_lo + 1;
    const int v0 = part * LT_NV, nv = min(LT_NV, dv - v0);
    const int* pt = page_table + (size_t)slot * max_pages;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        mbar_init(q_moved, 4);
        for (int s = 0; s < stages; ++s) { mbar_init(k_full0 + 8 * s, 1); mbar_init(k_empty0 + 8 * s, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(s_full0 + 8 * i, 1); mbar_init(p_full0 + 8 * i, 4); mbar_init(o_full0 + 8 * i, 1); }
        abort_flag[0] = 0;
        abort_flag[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            const int grow0 = t0 * n_heads + row0;               // rows past the sequence's are another's, or zeros: not written
            mbar_expect_tx(q_full, boxes * LT_BOX_Q);
            for (int h = 0; h < tm_boxes; ++h) tma_load_2d(k_s + h * LT_BOX_Q, &map_q, q_full, 64 * h, grow0);
            for (int h = 0; h < ss_boxes; ++h) tma_load_2d(q_s + h * LT_BOX_Q, &map_q, q_full, 64 * (tm_boxes + h), grow0);
            int issued = 0;
            const bool moved = mbar_wait(q_moved, 0, abort_flag);        // the ring is free of query rows
            if (!moved) { *abort_flag = 1; atomicCAS(error_word, 0, TC_ERR_PRODUCER); }
            for (int j = 0; moved && j < turns; ++j) {
                const int s = j % stages;
                if (!mbar_wait(k_empty0 + 8 * s, ((j / stages) & 1) ^ 1, abort_flag)) {
                    *abort_flag = 1; atomicCAS(error_word, 0, TC_ERR_PRODUCER); break;
                }
                const int y = pt[kb_lo + j] * LT_BN;
                mbar_expect_tx(k_full0 + 8 * s, stage_bytes);
                for (int h = 0; h < boxes; ++h) tma_load_2d(k_s + s * stage_bytes + h * LT_BOX_K, &map_k, k_full0 + 8 * s, 64 * h, y);
                issued = j + 1;
            }
            if (*abort_flag) {                                   // let issued copies land
                mbar_wait(q_full, 0, abort_flag + 1);
                for (int j = max(0, issued - stages); j < issued; ++j) mbar_wait(k_full0 + 8 * (j % stages), (j / stages) & 1, abort_flag + 1);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // scores: D float32, A and B bfloat16 K-major, M 128, N 64; weighted sum: B MN-major (bit 16), N nv
            const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LT_BN >> 3) << 17) | ((uint32_t)(LT_BM >> 4) << 24);
            const uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(nv >> 3) << 17) | ((uint32_t)(LT_BM >> 4) << 24);
            const uint64_t q_desc = smem_desc(q_s), k_desc = smem_desc(k_s);
            const uint64_t v_desc = lt_desc_values(k_s + (uint32_t)(v0 / 64) * LT_BOX_K);
            bool ok = mbar_wait(q_full, 0, abort_flag) && mbar_wait(q_moved, 0, abort_flag);
            int next_s = 0, next_o = 0;
            long long since = clock64();
            while (ok && next_o < turns) {
                if (next_s < turns && next_s - next_o < 2 && lt_ready(k_full0 + 8 * (next_s % stages), (next_s / stages) & 1)) {
                    tc_fence_after();
                    const uint64_t db = k_desc + (uint64_t)((next_s % stages) * (stage_bytes >> 4));
                    const uint32_t d = tmem + LT_S0 + (next_s & 1) * LT_BN;
                    for (int h = 0; h < tm_boxes; ++h)
                        lt_mma_scores(d, tmem + LT_Q0 + h * 32, db + (uint64_t)(h * (LT_BOX_K >> 4)), idesc_s, h ? 1u : 0u);
                    for (int h = 0; h < ss_boxes; ++h)
                        tc_mma_x4(d, q_desc + (uint64_t)(h * (LT_BOX_Q >> 4)),
                                  db + (uint64_t)((tm_boxes + h) * (LT_BOX_K >> 4)), idesc_s, 1u);
                    tc_commit(s_full0 + 8 * (next_s & 1));
                    ++next_s;
                    since = clock64();
                } else if (next_o < next_s && lt_ready(p_full0 + 8 * (next_o & 1), (next_o >> 1) & 1)) {
                    tc_fence_after();
                    const uint32_t p = tmem + LT_S0 + (next_o & 1) * LT_BN;
                    const uint64_t dv = v_desc + (uint64_t)((next_o % stages) * (stage_bytes >> 4));
                    lt_mma_values(tmem, p, dv, idesc_o, next_o ? 1u : 0u);
                    lt_mma_values(tmem, p + LT_BN / 2, dv, idesc_o, 1u);
                    tc_commit(k_empty0 + 8 * (next_o % stages));
                    tc_commit(o_full0 + 8 * (next_o & 1));
                    ++next_o;
                    since = clock64();
                } else if (*abort_flag || clock64() - since > 2000000000LL) {
                    ok = false;
                }
            }
            if (!ok) { *abort_flag = 1; atomicCAS(error_word, 0, TC_ERR_MMA); }
        }
    } else {
        const int quarter = warp & 3;                            // the lanes of tensor memory this warp may touch
        const int r = quarter * 32 + lane;
        const bool mine = r < rows_here;
        const int pos = mine ? start + (row0 + r) / n_heads : -1;
        const uint32_t t_lane = tmem + ((uint32_t)(quarter * 32) << 16);
        float m_ref = -INFINITY, l_run = 0.f;
        bool ok = mbar_wait(q_full, 0, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            // this row's first dims from the ring (rows of 128 bytes, 16-byte pieces exchanged by the swizzle) to tensor memory
            for (int h = 0; h < tm_boxes; ++h) {
                const unsigned char* row = smem + (k_s - smem_u32(smem)) + h * LT_BOX_Q + r * 128;
                uint32_t v[32];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 x = *reinterpret_cast<const uint4*>(row + ((c ^ (r & 7)) << 4));
                    v[4 * c] = x.x; v[4 * c + 1] = x.y; v[4 * c + 2] = x.z; v[4 * c + 3] = x.w;
                }
                lt_st32(t_lane + LT_Q0 + h * 32, v);
            }
            lt_st_wait();
            tc_fence_before();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");         // the reads come before the ring's next loads
            __syncwarp();
            if (lane == 0) lt_arrive(q_moved);
        }
        for (int j = 0; ok && j < turns; ++j) {
            bool w = mbar_wait(s_full0 + 8 * (j & 1), (j >> 1) & 1, abort_flag);
            w = __all_sync(0xffffffffu, w);
            if (!w) { ok = false; break; }
            tc_fence_after();
            const uint32_t t_s = t_lane + LT_S0 + (j & 1) * LT_BN;
            const int key0 = (kb_lo + j) * LT_BN;
            uint32_t raw[LT_BN];
            lt_ld32(t_s, raw);
            lt_ld32(t_s + 32, raw + 32);
            lt_ld_wait();
            if (key0 + LT_BN - 1 > pos_first || window > 0) {    // on the diagonal or at a window's edge
                const int hi = pos - key0, lo = window > 0 ? hi - window + 1 : 0;
#pragma unroll
                for (int i = 0; i < LT_BN; ++i)
                    if (i > hi || i < lo) raw[i] = 0xff800000u;
            }
            // weights 2^(score * scale - reference): 32 columns of high parts, 32 of low parts; returns their sum
            auto weights = [&](float neg_ref) -> float {
                float sum[4] = {0.f, 0.f, 0.f, 0.f};
                uint32_t packed[LT_BN];
#pragma unroll
                for (int i = 0; i < LT_BN; i += 2) {
                    const float pa = lt_ex2(fmaf(__uint_as_float(raw[i]), scale_log2, neg_ref));
                    const float pb = lt_ex2(fmaf(__uint_as_float(raw[i + 1]), scale_log2, neg_ref));
                    sum[(i >> 1) & 3] += pa + pb;
                    const __nv_bfloat162 hi = __floats2bfloat162_rn(pa, pb);
                    const __nv_bfloat162 lo = __floats2bfloat162_rn(pa - __low2float(hi), pb - __high2float(hi));
                    packed[i / 2] = *reinterpret_cast<const uint32_t*>(&hi);
                    packed[LT_BN / 2 + i / 2] = *reinterpret_cast<const uint32_t*>(&lo);
                }
                lt_st32(t_s, packed);
                lt_st32(t_s + 32, packed + 32);
                return (sum[0] + sum[1]) + (sum[2] + sum[3]);
            };
            float sum = 0.f;
            bool find_max = j == 0;
            if (!find_max) {
                sum = weights(m_ref == -INFINITY ? 0.f : -m_ref);
                find_max = __any_sync(0xffffffffu, mine && (!(sum <= LT_LAZY_P) || m_ref == -INFINITY));
            }
            if (find_max) {
                float mx = -INFINITY;
#pragma unroll
                for (int i = 0; i < LT_BN; ++i) mx = fmaxf(mx, __uint_as_float(raw[i]));
                const float m_new = fmaxf(m_ref, mx * scale_log2);
                if (j > 0 && __any_sync(0xffffffffu, m_new > m_ref)) {
                    // rescale what this warp's rows have summed so far to their new maxima
                    bool wo = mbar_wait(o_full0 + 8 * ((j - 1) & 1), ((j - 1) >> 1) & 1, abort_flag);
                    wo = __all_sync(0xffffffffu, wo);
                    if (!wo) { ok = false; break; }
                    tc_fence_after();
                    const float alpha = (m_new == -INFINITY) ? 1.f : lt_ex2(m_ref - m_new);
#pragma unroll 1
                    for (int c = 0; c < nv; c += 32) {
                        uint32_t o[32];
                        lt_ld32(t_lane + c, o);
                        lt_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        lt_st32(t_lane + c, o);
                    }
                    l_run *= alpha;
                }
                m_ref = m_new;
                lt_st_wait();                                    // what was written against the old reference has landed
                sum = weights(m_ref == -INFINITY ? 0.f : -m_ref);
            }
            lt_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) lt_arrive(p_full0 + 8 * (j & 1));
            l_run += sum;
        }
        if (ok) {
            // the last weighted sum: its commit counts every product issued before it
            const bool w = mbar_wait(o_full0 + 8 * ((turns - 1) & 1), ((turns - 1) >> 1) & 1, abort_flag);
            ok = __all_sync(0xffffffffu, w);
        }
        if (!ok) {
            if (lane == 0) { *abort_flag = 1; atomicCAS(error_word, 0, TC_ERR_EPILOGUE); }
        } else {
            tc_fence_after();
            // a sink adds exp(sink) to the denominator and nothing to the numerator
            float keep = 1.f, l = l_run;
            if (sinks != nullptr && mine) {
                const float sk = sinks[(row0 + r) % n_heads] * LT_LOG2E;
                const float m_all = fmaxf(m_ref, sk);
                keep = (m_ref == -INFINITY) ? 0.f : exp2f(m_ref - m_all);
                l = l * keep + exp2f(sk - m_all);
            }
            const float inv = l > 0.f ? keep / l : 0.f;
            bf16* dst = out + ((size_t)t0 * n_heads + row0 + r) * dv + v0;
#pragma unroll 1
            for (int c = 0; c < nv; c += 32) {
                uint32_t o[32];
                lt_ld32(t_lane + c, o);
                lt_ld_wait();
                if (mine) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        if (c + i >= nv) break;
                        uint32_t v[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const __nv_bfloat162 x = __floats2bfloat162_rn(__uint_as_float(o[i + 2 * e]) * inv, __uint_as_float(o[i + 2 * e + 1]) * inv);
                            v[e] = *reinterpret_cast<const uint32_t*>(&x);
                        }
                        *reinterpret_cast<uint4*>(dst + c + i) = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

static inline long long lt_smem(int boxes, int stages) {
    const int tm = boxes < LT_TMEM_BOXES ? boxes : LT_TMEM_BOXES;
    const long long ring = (long long)stages * boxes * LT_BOX_K, pass = (long long)tm * LT_BOX_Q;
    return (long long)(boxes - tm) * LT_BOX_Q + (ring > pass ? ring : pass) + LT_NBARS * 8 + 32 + 1024;
}

// Whether rows of dk elements and values of dv fit: two stages beside the query rows in shared memory.
SSB_API int ssb_latent_attention_tc_fits(int dk, int dv) {
    const int boxes = (dk + 63) / 64;
    return dk > 0 && dk % 8 == 0 && dv > 0 && dv % 16 == 0 && dv <= dk && dv <= 2 * LT_NV && lt_smem(boxes, 2) <= 227 * 1024;
}

// q [tokens, heads x dk] and out [tokens, heads x dv] contiguous bfloat16; cache [pages][64][dk]; sinks: one float32 a head, or null
SSB_API int ssb_latent_attention_tc(const void* q, const void* cache, int n_pages, const int* cu_new, const int* seq_start,
                                    const int* seq_slot, const int* page_table, int max_pages, void* out, const float* sinks,
                                    int n_seqs, int max_new, int n_tokens, int n_heads, int dk, int dv, int page_shift, int window,
                                    float scale, int* error_word, cudaStream_t stream) {
    if (n_seqs <= 0 || max_new <= 0) return 0;
    if (page_shift != 6 || n_heads <= 0 || !error_word || !ssb_latent_attention_tc_fits(dk, dv)) return SSB_ERR_BAD_SIZE;
    if (((uintptr_t)q | (uintptr_t)cache | (uintptr_t)out) & 15) return SSB_ERR_BAD_SIZE;
    const long long q_rows = (long long)n_tokens * n_heads, k_rows = (long long)n_pages * 64;
    const long long tiles = ((long long)max_new * n_heads + LT_BM - 1) / LT_BM;
    const int parts = (dv + LT_NV - 1) / LT_NV, boxes = (dk + 63) / 64;
    if (q_rows > 0x7fffffffLL || k_rows > 0x7fffffffLL || tiles > 65535 || (long long)n_seqs * parts > 0x7fffffffLL) return SSB_ERR_BAD_SIZE;
    int stages = 2;
    while (stages < LT_MAX_STAGES && lt_smem(boxes, stages + 1) <= 227 * 1024) ++stages;
    CUtensorMap mq, mk;
    int rc = make_map(&mq, q, (int)q_rows, dk, dk, LT_BM);
    if (rc) return rc;
    rc = make_map(&mk, cache, (int)k_rows, dk, dk, LT_BN);
    if (rc) return rc;
    const long long smem = lt_smem(boxes, stages);
    static long long configured = 0;
    if (smem > configured) {
        cudaError_t e = cudaFuncSetAttribute(latent_attention_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = smem;
    }
    latent_attention_tc_kernel<<<dim3((unsigned)(n_seqs * parts), (unsigned)tiles), LT_THREADS, (size_t)smem, stream>>>(
        mq, mk, cu_new, seq_start, seq_slot, page_table, max_pages, (bf16*)out, sinks, n_heads, boxes, dv, parts, stages, window,
        scale * LT_LOG2E, error_word);
    return ssb_launch_status();
}
