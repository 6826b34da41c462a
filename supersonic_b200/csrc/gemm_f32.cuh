// Float32 products C[m, n] (+)= sum_k A[m, k] W[n, k] whose operands can be fetched in 16-byte pieces.
//
// The sums are those of gemm_nt_plain_kernel bit for bit: 16 products a chunk, one FMA chain in k order, the chunks'
// sums added in k order with compensation (Kahan).  Nothing here is re-associated, so a row's result does not depend on
// which kernel took it, how many rows it came with or which tile it lay in.
#pragma once
#include "packed_f32.cuh"

constexpr int GF_CHUNK = 16;               // products of one FMA chain
constexpr int GF_LD = GF_CHUNK + 4;        // a chunk's place in shared memory: 80 bytes, so that eight neighbouring chunks
                                           // (or rows) start in eight different groups of four banks

__device__ __forceinline__ void gf_cp16(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gf_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void gf_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One compensated addition, its roundings written out: nothing is re-associated.
__device__ __forceinline__ void gf_kahan(float& acc, float& lost, float part) {
    const float y = __fsub_rn(part, lost);
    const float t = __fadd_rn(acc, y);
    lost = __fsub_rn(__fsub_rn(t, acc), y);
    acc = t;
}

// ---------------------------------------------------------------------------------------------------------------------
// Few rows (a decode step, a short prompt): the weights are streamed once per group of MB rows.  A block takes 8 R rows
// of W and 512 columns a turn: a lane of the eight product warps makes the sum of one chunk of R rows of W with all MB rows
// of A; the chunks' sums go through shared memory, two turns deep, to further warps whose threads add them in order, one
// result each: 32 additions of four dependent steps a turn, which nobody else waits for.  W and A come by cp.async, STAGES
// turns deep, in one stream over all the tiles that a block of the grid walks.
// Bound by the shared-memory reads of the products from 8 rows on; the general kernel read the weights again for every row and
// spent a dependent chain of 4 additions per 16 products in every thread.  Weights of 16384 x 2048 (134 MB), us: 8 rows 270 on
// the general kernel and 54 here, 16 rows 270 and 91.  Up to four rows take the kernel below, but where they are too long for it.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int GF_PRODUCT_THREADS = 256;
constexpr int GF_SKINNY_CHUNKS = 32;                                  // chunks a turn: one a lane
__host__ __device__ constexpr int gf_adders(int mb, int r) { return (8 * r * mb + 31) / 32 * 32; }      // threads that add

template <int MB, int R, int STAGES>
constexpr size_t gf_skinny_smem() {
    return sizeof(float) * ((size_t)STAGES * (8 * R + MB) * GF_SKINNY_CHUNKS * GF_LD + 2 * 8 * R * MB * (GF_SKINNY_CHUNKS + 1));
}
__device__ __forceinline__ void gf_bar_sync(int id, int count) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory"); }
__device__ __forceinline__ void gf_bar_arrive(int id, int count) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory"); }

template <int MB, int R, int STAGES>
__global__ void __launch_bounds__(GF_PRODUCT_THREADS + gf_adders(MB, R))
gemm_f32_skinny_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C,
                       int ldc, int M, int N, int K, long long a_batch, long long w_batch, long long c_batch, int m_groups,
                       int accumulate) {
    constexpr int NB = 8 * R, CH = GF_SKINNY_CHUNKS, TURN = CH * GF_CHUNK, PIECES = TURN / 4;
    constexpr int ALL = GF_PRODUCT_THREADS + gf_adders(MB, R), SUMS = NB * MB * (CH + 1);
    // named barriers: the product warps among themselves; a turn's sums are written; a turn's sums have been added (two each)
    constexpr int BAR_PRODUCTS = 1, BAR_WRITTEN = 2, BAR_ADDED = 4;
    extern __shared__ __align__(16) float gf_smem[];
    float* w_s = gf_smem;                                             // [stage][row of W][chunk]
    float* a_s = w_s + STAGES * NB * CH * GF_LD;                      // [stage][row of A][chunk]
    float* sums = a_s + STAGES * MB * CH * GF_LD;                     // [2][row of W][row of A][chunk]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    A += (size_t)blockIdx.z * a_batch;
    W += (size_t)blockIdx.z * w_batch;
    C += (size_t)blockIdx.z * c_batch;
    const int turns = (K + TURN - 1) / TURN, tiles = m_groups * ((N + NB - 1) / NB);
    // this block's tiles, every gridDim.x-th (the groups of rows of A that share rows of W lie side by side), and their turns
    const int total = ((tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x) * turns;
    auto m_of = [&](int tile) { return tile % m_groups * MB; };
    auto n_of = [&](int tile) { return tile / m_groups * NB; };

    if (tid >= GF_PRODUCT_THREADS) {
        const int o = tid - GF_PRODUCT_THREADS, n = o / MB, m = o % MB;
        const bool mine = o < NB * MB;
        float acc = 0.f, lost = 0.f;
        int turn = 0, tile = blockIdx.x;
        for (int g = 0; g < total; ++g) {
            const int buf = g & 1;
            gf_bar_sync(BAR_WRITTEN + buf, ALL);
            if (mine) {
                const int n_chunks = min(CH, (K - turn * TURN + GF_CHUNK - 1) / GF_CHUNK);
                const float* sp = sums + buf * SUMS + o * (CH + 1);
                if (n_chunks == CH) {
#pragma unroll
                    for (int c = 0; c < CH; ++c) gf_kahan(acc, lost, sp[c]);
                } else {
                    for (int c = 0; c < n_chunks; ++c) gf_kahan(acc, lost, sp[c]);
                }
            }
            __syncwarp();
            if (g + 2 < total) gf_bar_arrive(BAR_ADDED + buf, ALL);
            if (++turn == turns) {                                    // the tile's last turn
                const int row = m_of(tile) + m, col = n_of(tile) + n;
                if (mine && row < M && col < N) {
                    float* dst = C + (size_t)row * ldc + col;
                    *dst = accumulate ? *dst + acc : acc;
                }
                acc = lost = 0.f;
                turn = 0;
                tile += gridDim.x;
            }
        }
        return;
    }
    // what lies outside the operands arrives as zeros (a copy of no bytes)
    int ahead_turn = 0, ahead_tile = blockIdx.x;                      // of the next load
    auto load = [&](int s) {
        const int k0 = ahead_turn * TURN, m0 = m_of(ahead_tile), n0 = n_of(ahead_tile);
        const int m_here = M - m0, n_here = N - n0;
        const float* At = A + (size_t)m0 * lda;
        const float* Wt = W + (size_t)n0 * ldw;
#pragma unroll
        for (int e = 0; e < NB * PIECES / GF_PRODUCT_THREADS; ++e) {
            const int p = tid + e * GF_PRODUCT_THREADS, r = p / PIECES, c = p % PIECES, k = k0 + c * 4;
            const bool in = r < n_here && k < K;
            gf_cp16(w_s + ((s * NB + r) * CH + c / 4) * GF_LD + (c % 4) * 4, in ? Wt + (size_t)r * ldw + k : W, in ? 16 : 0);
        }
#pragma unroll
        for (int e = 0; e < (MB * PIECES + GF_PRODUCT_THREADS - 1) / GF_PRODUCT_THREADS; ++e) {
            const int p = tid + e * GF_PRODUCT_THREADS, r = p / PIECES, c = p % PIECES, k = k0 + c * 4;
            const bool in = r < m_here && k < K;
            if (MB * PIECES % GF_PRODUCT_THREADS == 0 || p < MB * PIECES)
                gf_cp16(a_s + ((s * MB + r) * CH + c / 4) * GF_LD + (c % 4) * 4, in ? At + (size_t)r * lda + k : A, in ? 16 : 0);
        }
        if (++ahead_turn == turns) { ahead_turn = 0; ahead_tile += gridDim.x; }
    };
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t) {
        if (t < total) load(t);
        gf_commit();
    }
    for (int g = 0; g < total; ++g) {
        const int buf = g & 1;
        gf_wait<STAGES - 2>();
        gf_bar_sync(BAR_PRODUCTS, GF_PRODUCT_THREADS);                // the turn has landed; everyone is done with the one before
        if (g + STAGES - 1 < total) load((g + STAGES - 1) % STAGES);
        gf_commit();
        const int s = g % STAGES;
        const float* wp = w_s + ((s * NB + warp * R) * CH + lane) * GF_LD;
        const float* ap = a_s + (s * MB * CH + lane) * GF_LD;
        float part[R][MB];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int m = 0; m < MB; ++m) part[r][m] = 0.f;
#pragma unroll
        for (int q = 0; q < GF_CHUNK / 4; ++q) {
            float4 w[R];
#pragma unroll
            for (int r = 0; r < R; ++r) w[r] = *reinterpret_cast<const float4*>(wp + r * CH * GF_LD + q * 4);
#pragma unroll
            for (int m = 0; m < MB; ++m) {
                const float4 a = *reinterpret_cast<const float4*>(ap + m * CH * GF_LD + q * 4);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    part[r][m] = fmaf(a.x, w[r].x, part[r][m]);
                    part[r][m] = fmaf(a.y, w[r].y, part[r][m]);
                    part[r][m] = fmaf(a.z, w[r].z, part[r][m]);
                    part[r][m] = fmaf(a.w, w[r].w, part[r][m]);
                }
            }
        }
        if (g >= 2) gf_bar_sync(BAR_ADDED + buf, ALL);                // the sums of two turns ago have been added
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int m = 0; m < MB; ++m) sums[buf * SUMS + ((warp * R + r) * MB + m) * (CH + 1) + lane] = part[r][m];
        gf_bar_arrive(BAR_WRITTEN + buf, ALL);
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Up to four rows (decode steps): a warp walks RW rows of W from end to end on its own.  32 / RW lanes a row take a chunk each,
// hand the sums of a step to one another by shuffles and add them in k order, the step before while this one multiplies: no
// barrier and no exchange through shared memory between the warps of a block.  W comes by cp.async into a ring of the warp's
// own, its first turns before the dependency wait (no kernel of a step writes weights); A lies whole in shared memory.  16-byte
// pieces are permuted within their chunk, so that the eight lanes of an access start in eight different groups of four banks.
// Many columns are bound by the memory, few by a warp's chain: a step's fetches, 16 products, shuffles and additions (16
// clocks a chunk), one after another, so that few columns take few rows a warp and long steps.  us on the kernel above and
// here, 1, 2 and 4 rows: 128256 x 2048 202, 236, 301 and 153, 164, 205; 16384 x 2048 30, 34, 42 and 24, 27, 32; 3072 x 2048
// 10.7, 12.0, 14.3 and 9.3, 10.0, 11.2; 1 and 2 rows, 2048 x 8192 18.0, 20.3 and 15.9, 16.8, 4096 x 14336 56, 64 and 38, 44.
// Four rows of W a warp, 2 x 2048 x 8192: 22.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int GF_WALK_WARPS = 8, GF_WALK_STAGES = 4, GF_WALK_TURN = 1024;        // a turn: 1024 / RW columns of RW rows, two steps
constexpr size_t GF_WALK_RING = sizeof(float) * GF_WALK_STAGES * GF_WALK_TURN;   // a warp's
constexpr size_t GF_WALK_SMEM = 227 * 1024;
static inline size_t gf_walk_rows(int mb, int K) { return sizeof(float) * (size_t)mb * (((size_t)K + 511) / 512 * 512); }
// Whether the rows of A leave room for the rings of seven warps (4 x 2048 x 8192 with six: 31.7 us, 25.0 on the kernel above).
static inline bool gf_walk_ok(int M, int K) {
    return M <= 4 && gf_walk_rows(M <= 2 ? M : 4, K) + 7 * GF_WALK_RING <= GF_WALK_SMEM;
}
// Rows of W a warp: as many as leave six warps an SM something to do.
static inline int gf_walk_width(int N) { return N > 24 * ssb_sm_count() ? 4 : N > 12 * ssb_sm_count() ? 2 : 1; }

// The chunks' sums of a step, one of each of MB rows a lane, in; those of this lane's row (its chunk modulo MB) in k order out.
template <int MB, int RW>
__device__ __forceinline__ void gf_walk_exchange(const float (&part)[MB], float (&v)[32 / RW], int lane) {
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int CL = 32 / RW;
    const int n = lane % RW, c = lane / RW;
    if constexpr (MB == 1) {
#pragma unroll
        for (int j = 0; j < CL; ++j) v[j] = __shfl_sync(ALL, part[0], j * RW + n);
    } else if constexpr (MB == 2) {
        const bool odd = c & 1;
        const float got = __shfl_xor_sync(ALL, odd ? part[0] : part[1], RW);
        const float t0 = odd ? got : part[0], t1 = odd ? part[1] : got;
#pragma unroll
        for (int p = 0; p < CL / 2; ++p) {
            v[2 * p] = __shfl_sync(ALL, t0, (2 * p + (c & 1)) * RW + n);
            v[2 * p + 1] = __shfl_sync(ALL, t1, (2 * p + (c & 1)) * RW + n);
        }
    } else {
        const bool odd = c & 1, high = c & 2;
        const float g0 = __shfl_xor_sync(ALL, odd ? part[0] : part[1], RW);
        const float g1 = __shfl_xor_sync(ALL, odd ? part[2] : part[3], RW);
        const float t0 = odd ? g0 : part[0], t1 = odd ? part[1] : g0;          // row c & 1, the pair's two chunks
        const float u0 = odd ? g1 : part[2], u1 = odd ? part[3] : g1;          // row 2 + (c & 1)
        const float h0 = __shfl_xor_sync(ALL, high ? t0 : u0, 2 * RW);
        const float h1 = __shfl_xor_sync(ALL, high ? t1 : u1, 2 * RW);
        const float w[4] = {high ? h0 : t0, high ? h1 : t1, high ? u0 : h0, high ? u1 : h1};
#pragma unroll
        for (int p = 0; p < CL / 4; ++p)
#pragma unroll
            for (int i = 0; i < 4; ++i) v[4 * p + i] = __shfl_sync(ALL, w[i], (4 * p + (c & 3)) * RW + n);
    }
}

// How a row's 16-byte pieces are permuted: a piece's place is its number xor this, of its chunk and row.
template <int RW>
__device__ __forceinline__ int gf_walk_key(int chunk, int row) {
    return RW == 4 ? row : RW == 2 ? ((chunk >> 1) & 1) ^ (row << 1) : (chunk >> 1) & 3;
}

// A gated unit's first product: W holds its gate rows, then as many up rows (N in all); a warp's rows are half of either, and
// what is stored is ssb_gate of the two sums, times the row's factor.
struct GfGate { int kind; float limit; const float* row_scale; };

template <int MB, int RW, bool GATED = false>
__global__ void __launch_bounds__(32 * GF_WALK_WARPS)
gemm_f32_walk_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C, int ldc,
                     int M, int N, int K, long long a_batch, long long w_batch, long long c_batch, int accumulate, GfGate gate) {
    static_assert(!GATED || RW >= 2, "gate and up rows in one warp");
    constexpr int OUT = GATED ? RW / 2 : RW;                           // columns of the result a warp makes
    const int n_out = GATED ? N / 2 : N;
    constexpr int CL = 32 / RW, STEP = CL * GF_CHUNK, SEG = GF_WALK_TURN / RW, ROW_LOADS = 8 / RW, STAGES = GF_WALK_STAGES;
    static_assert(SEG == 2 * STEP && GF_WALK_TURN == 8 * 32 * 4, "two steps a turn, eight pieces a lane");
    extern __shared__ __align__(16) float gf_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    const int n = lane % RW, c = lane / RW, Kp = (K + 511) / 512 * 512;
    float* a_s = gf_smem;                                              // [row of A][Kp], zeros from K on
    float* ring = a_s + MB * Kp + warp * STAGES * GF_WALK_TURN;        // this warp's: [stage][row of W][SEG]
    A += (size_t)blockIdx.z * a_batch;
    W += (size_t)blockIdx.z * w_batch;
    C += (size_t)blockIdx.z * c_batch;
    const int tasks = (n_out + OUT - 1) / OUT, first = warp * (int)gridDim.x + (int)blockIdx.x, stride = warps * (int)gridDim.x;
    const int turns = (K + SEG - 1) / SEG;
    const int total = first < tasks ? (tasks - first + stride - 1) / stride * turns : 0;

    int ahead_turn = 0, ahead_task = first, ahead_slot = 0;            // of the next load
    auto load = [&]() {
        const int k = ahead_turn * SEG + lane * 4, rows = n_out - ahead_task * OUT;
        const float* src = W + (size_t)ahead_task * OUT * ldw + k;
        float* dst = ring + ahead_slot * GF_WALK_TURN;
#pragma unroll
        for (int e = 0; e < 8; ++e) {                                  // what lies outside arrives as zeros
            const int r = e / ROW_LOADS, s = e % ROW_LOADS * 32;       // row, and the row's piece lane + s
            const bool in = r % OUT < rows && k + s * 4 < K;
            gf_cp16(dst + r * SEG + ((s + lane) ^ gf_walk_key<RW>(lane / 4, r)) * 4,
                    in ? src + (size_t)(r % OUT + r / OUT * n_out) * ldw + s * 4 : W, in ? 16 : 0);
        }
        if (++ahead_slot == STAGES) ahead_slot = 0;
        if (++ahead_turn == turns) { ahead_turn = 0; ahead_task += stride; }
    };
    ssb_pdl_launch_dependents();
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t) {
        if (t < total) load();
        gf_commit();
    }
    ssb_pdl_wait();                                                    // A and C are the predecessor's
    for (int p = tid; p < MB * (Kp / 4); p += blockDim.x) {
        const int m = p / (Kp / 4), u = p % (Kp / 4);
        const bool in = m < M && u * 4 < K;
        gf_cp16(a_s + m * Kp + (u ^ gf_walk_key<1>(u / 4, 0)) * 4, in ? A + (size_t)m * lda + u * 4 : A, in ? 16 : 0);
    }
    gf_commit();
    gf_wait<0>();
    __syncthreads();

    int w_at[4], a_at[4];                                              // this lane's chunk of a step: its pieces' places
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        w_at[q] = n * SEG + ((c * 4 + q) ^ gf_walk_key<RW>(c, n)) * 4;
        a_at[q] = ((c * 4 + q) ^ gf_walk_key<1>(c, 0)) * 4;
    }
    float acc = 0.f, lost = 0.f, held[CL];                             // held: the step before's chunks of this lane's row of A
#pragma unroll
    for (int j = 0; j < CL; ++j) held[j] = 0.f;
    int turn = 0, task = first, slot = 0;
    for (int g = 0; g < total; ++g) {
        gf_wait<STAGES - 2>();
        __syncwarp();                                                  // the turn has landed; all lanes are done with the one before
        if (g + STAGES - 1 < total) load();
        gf_commit();
        int here = 0;                                                  // chunks of the last step
#pragma unroll
        for (int st = 0; st < 2; ++st) {
            const int k0 = turn * SEG + st * STEP;
            if (k0 >= K) break;
            here = (K - k0 + GF_CHUNK - 1) / GF_CHUNK;
            const float* w_t = ring + slot * GF_WALK_TURN + st * STEP;
            const float* a_t = a_s + k0;
            float part[MB];
#pragma unroll
            for (int m = 0; m < MB; ++m) part[m] = 0.f;
#pragma unroll
            for (int q = 0; q < GF_CHUNK / 4; ++q) {
                const float4 w = *reinterpret_cast<const float4*>(w_t + w_at[q]);
#pragma unroll
                for (int m = 0; m < MB; ++m) {
                    const float4 a = *reinterpret_cast<const float4*>(a_t + m * Kp + a_at[q]);
                    part[m] = fmaf(a.x, w.x, part[m]);
                    part[m] = fmaf(a.y, w.y, part[m]);
                    part[m] = fmaf(a.z, w.z, part[m]);
                    part[m] = fmaf(a.w, w.w, part[m]);
                }
            }
            // whole steps, and zeros before a row's first: adding a zero to the zeros it starts from changes nothing
#pragma unroll
            for (int j = 0; j < CL; ++j) gf_kahan(acc, lost, held[j]);
            gf_walk_exchange<MB, RW>(part, held, lane);
        }
        if (++slot == STAGES) slot = 0;
        if (++turn == turns) {                                         // the row's last step, which may have fewer chunks
#pragma unroll
            for (int j = 0; j < CL; ++j) {
                if (j < here) gf_kahan(acc, lost, held[j]);
                held[j] = 0.f;
            }
            const float up = GATED ? __shfl_down_sync(0xffffffffu, acc, OUT) : 0.f;
            const int col = task * OUT + n;
            if (c < MB && c < M && n < OUT && col < n_out) {
                float* dst = C + (size_t)c * ldc + col;
                if constexpr (GATED) *dst = ssb_gate(acc, up, gate.kind, gate.limit) * (gate.row_scale ? gate.row_scale[c] : 1.0f);
                else *dst = accumulate ? *dst + acc : acc;
            }
            acc = lost = 0.f;
            turn = 0;
            task += stride;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// A few hundred rows of many columns: tiles of 64 x 64 and 128 x 64, 4 x 4 and 8 x 4 results a thread, one chunk of k a turn, two or
// three blocks an SM.  A chunk comes by cp.async as it lies in memory, GF_RAW deep, and is turned k-major in shared memory on the
// way to its two buffers, so that a thread reads four neighbouring columns at a time and the multiply-adds go two columns an
// instruction (fma.rn.f32x2: each half rounds as the scalar one does).  Bound by the FP32 pipes and the shared-memory reads beside
// them: a chunk's 16 multiply-adds of a result are followed by the four steps of its compensated addition, so 4/5 of the peak
// is what this sum leaves.  500 rows by 2048 x 2048, us on the general kernel and here: 257 and 181.
// ---------------------------------------------------------------------------------------------------------------------
// Two compensated additions; `kept` is what the last ones rounded away, with the sign it is added back with.
__device__ __forceinline__ void gf_kahan2(unsigned long long& acc, unsigned long long& kept, unsigned long long part,
                                          unsigned long long minus_one) {
    const unsigned long long y = f2_add(part, kept);
    const unsigned long long t = f2_add(acc, y);
    kept = f2_add(y, f2_fma(t, minus_one, acc));
    acc = t;
}

constexpr int GF_TILE_THREADS = 256, GF_RAW = 3;                     // GF_RAW: chunks on their way from memory, and at work

template <int RM, int RN>
constexpr size_t gf_tile_smem() { return sizeof(float) * (size_t)(2 + GF_RAW) * GF_CHUNK * 16 * (RM + RN); }

template <int RM, int RN, int MIN_BLOCKS>                // results a thread; tiles of 16 RM x 16 RN
__global__ void __launch_bounds__(GF_TILE_THREADS, MIN_BLOCKS)
gemm_f32_tile_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C,
                     int ldc, int M, int N, int K, long long a_batch, long long w_batch, long long c_batch, int accumulate) {
    constexpr int TM = 16 * RM, TN = 16 * RN, PA = TM / 64, PW = TN / 64;     // PA, PW: 16-byte pieces of A and W a thread fetches
    extern __shared__ __align__(16) float gf_smem[];
    float (*a_s)[GF_CHUNK][TM] = reinterpret_cast<float (*)[GF_CHUNK][TM]>(gf_smem);                       // [2]: a chunk, k-major
    float (*w_s)[GF_CHUNK][TN] = reinterpret_cast<float (*)[GF_CHUNK][TN]>(gf_smem + 2 * GF_CHUNK * TM);   // [2]
    float4* raw = reinterpret_cast<float4*>(gf_smem + 2 * GF_CHUNK * (TM + TN));       // [GF_RAW][piece][thread]: as it lay
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane % 8 + 8 * (warp % 2), ty = lane / 8 + 4 * (warp / 2);    // columns 4 tx .. + 3 (and + 64); rows likewise
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    A += (size_t)blockIdx.z * a_batch + (size_t)m0 * lda;
    W += (size_t)blockIdx.z * w_batch + (size_t)n0 * ldw;
    C += (size_t)blockIdx.z * c_batch;
    const int m_here = min(TM, M - m0), n_here = min(TN, N - n0);
    const int turns = (K + GF_CHUNK - 1) / GF_CHUNK;
    // a thread's pieces: neighbouring k of one row of A and of one of W
    const int a_row = tid % TM, a_k = tid / TM * 4 * PA, w_row = tid % TN, w_k = tid / TN * 4 * PW;
    const bool a_in = a_row < m_here, w_in = w_row < n_here;
    const float* a_src = A + (size_t)(a_in ? a_row : 0) * lda + a_k;
    const float* w_src = W + (size_t)(w_in ? w_row : 0) * ldw + w_k;
    auto fetch = [&](int turn) {
        float4* dst = raw + (turn % GF_RAW) * (PA + PW) * GF_TILE_THREADS + tid;
        const int k = turn * GF_CHUNK;
#pragma unroll
        for (int e = 0; e < PA; ++e) {
            const bool in = a_in && k + a_k + 4 * e < K;
            gf_cp16(reinterpret_cast<float*>(dst + e * GF_TILE_THREADS), in ? a_src + k + 4 * e : A, in ? 16 : 0);
        }
#pragma unroll
        for (int e = 0; e < PW; ++e) {
            const bool in = w_in && k + w_k + 4 * e < K;
            gf_cp16(reinterpret_cast<float*>(dst + (PA + e) * GF_TILE_THREADS), in ? w_src + k + 4 * e : W, in ? 16 : 0);
        }
    };
    // k-major: a thread turns over what it fetched itself, so its own wait is all that comes between
    auto stage = [&](int turn) {
        const float4* src = raw + (turn % GF_RAW) * (PA + PW) * GF_TILE_THREADS + tid;
#pragma unroll
        for (int e = 0; e < PA; ++e) {
            const float4 x = src[e * GF_TILE_THREADS];
            float* dst = &a_s[turn & 1][a_k + 4 * e][a_row];
            dst[0] = x.x; dst[TM] = x.y; dst[2 * TM] = x.z; dst[3 * TM] = x.w;
        }
#pragma unroll
        for (int e = 0; e < PW; ++e) {
            const float4 x = src[(PA + e) * GF_TILE_THREADS];
            float* dst = &w_s[turn & 1][w_k + 4 * e][w_row];
            dst[0] = x.x; dst[TN] = x.y; dst[2 * TN] = x.z; dst[3 * TN] = x.w;
        }
    };
    unsigned long long acc[RM][RN / 2], kept[RM][RN / 2];             // two columns each
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN / 2; ++j) { acc[i][j] = 0ull; kept[i][j] = 0ull; }
    const unsigned long long minus_one = f2_twice(-1.0f);
#pragma unroll
    for (int t = 0; t < GF_RAW - 1; ++t) {
        if (t < turns) fetch(t);
        gf_commit();
    }
    gf_wait<GF_RAW - 2>();
    stage(0);
    __syncthreads();
    for (int turn = 0; turn < turns; ++turn) {
        if (turn + GF_RAW - 1 < turns) fetch(turn + GF_RAW - 1);
        gf_commit();
        const float (*ab)[TM] = a_s[turn & 1];
        const float (*wb)[TN] = w_s[turn & 1];
        unsigned long long part[RM][RN / 2];
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN / 2; ++j) part[i][j] = 0ull;
#pragma unroll
        for (int k = 0; k < GF_CHUNK; ++k) {
            float a[RM];
            unsigned long long w[RN / 2];
#pragma unroll
            for (int g = 0; g < RM / 4; ++g) {
                const float4 x = *reinterpret_cast<const float4*>(&ab[k][64 * g + 4 * ty]);
                a[4 * g] = x.x; a[4 * g + 1] = x.y; a[4 * g + 2] = x.z; a[4 * g + 3] = x.w;
            }
#pragma unroll
            for (int g = 0; g < RN / 4; ++g) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(&wb[k][64 * g + 4 * tx]);
                w[2 * g] = x.x; w[2 * g + 1] = x.y;
            }
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                const unsigned long long aa = f2_twice(a[i]);
#pragma unroll
                for (int j = 0; j < RN / 2; ++j) part[i][j] = f2_fma(aa, w[j], part[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN / 2; ++j) gf_kahan2(acc[i][j], kept[i][j], part[i][j], minus_one);
        gf_wait<GF_RAW - 2>();
        if (turn + 1 < turns) stage(turn + 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int m = 64 * (i / 4) + 4 * ty + i % 4;
        if (m >= m_here) continue;
#pragma unroll
        for (int j = 0; j < RN / 2; ++j) {
            const int n = 64 * (j / 2) + 4 * tx + 2 * (j % 2);
            float* dst = C + (size_t)(m0 + m) * ldc + n0 + n;
            const float lo = __uint_as_float((unsigned)acc[i][j]), hi = __uint_as_float((unsigned)(acc[i][j] >> 32));
            if (n < n_here) dst[0] = accumulate ? dst[0] + lo : lo;
            if (n + 1 < n_here) dst[1] = accumulate ? dst[1] + hi : hi;
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Many rows, tiles of 128 x 128, one block an SM that walks its share of them.  Warps have roles: eight do nothing but multiply and
// add, 8 x 8 results a thread in registers, and four others keep a ring of turns of 32 k ahead of them, k-major in shared memory.
// Rows come as they lie, 128 bytes of one at a time, and are turned by scalar stores whose column is exchanged by the quarter
// of k they belong to, so that neither the stores nor the reads meet on a bank.  Hardware barriers by number say when a turn is full
// and when it is free; nothing waits in a loop.  Bound by the FP32 pipe: a chunk's 640 multiply-adds and compensated additions of a
// warp in packed pairs take 2560 clocks an SM, 3200 are spent (a ninth of them in the meeting a turn).  With the same warps fetching,
// turning and multiplying by turns: 1000 rows, 2048 x 2048 288 us and 217 here, 3072 x 2048 435 (64 x 64 tiles) and 430, 16384 x 2048
// 1777 (two blocks an SM, their sums in tensor memory) and 1491, 45 TFLOP/s; 2048 x 8192 1142 and 850.  Turns of 64 k: 265 for the first.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int GF_ROLE_COMPUTE = 256, GF_ROLE_FETCH = 128, GF_ROLE_ALL = GF_ROLE_COMPUTE + GF_ROLE_FETCH, GF_ROLE_STAGES = 4, GF_ROLE_K = 32;
template <int RM, int RN>
constexpr size_t gf_role_smem() { return sizeof(float) * (size_t)GF_ROLE_STAGES * GF_ROLE_K * 16 * (RM + RN); }

template <int RM, int RN>
__global__ void __launch_bounds__(GF_ROLE_ALL, 1)
gemm_f32_role_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C, int ldc,
                     int M, int N, int K, long long a_batch, long long w_batch, long long c_batch, int accumulate) {
    constexpr int TM = 16 * RM, TN = 16 * RN, STAGES = GF_ROLE_STAGES, TK = GF_ROLE_K, STAGE = TK * (TM + TN);
    constexpr int BAR_FULL = 1, BAR_FREE = 1 + STAGES;
    extern __shared__ __align__(16) float gf_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    A += (size_t)blockIdx.z * a_batch;
    W += (size_t)blockIdx.z * w_batch;
    C += (size_t)blockIdx.z * c_batch;
    const int m_tiles = (M + TM - 1) / TM, tiles = m_tiles * ((N + TN - 1) / TN), turns = (K + TK - 1) / TK;
    if (warp >= GF_ROLE_COMPUTE / 32) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");        // 4 x 32 x 40 + 8 x 32 x 232 = 384 x 168, what the block has
        const int f = tid - GF_ROLE_COMPUTE, q = f % 8, r0 = f / 8;      // 16 bytes of a row's 128; rows r0, r0 + 16, ...
        int turn_no = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const int m0 = tile % m_tiles * TM, n0 = tile / m_tiles * TN;
            for (int turn = 0; turn < turns; ++turn, ++turn_no) {
                const int s = turn_no % STAGES, k = turn * TK + q * 4;
                float* a_s = gf_smem + s * STAGE;                        // [k][TM]
                float* w_s = a_s + TK * TM;                              // [k][TN]
                float4 x[TM / 16];
#pragma unroll
                for (int i = 0; i < TM / 16; ++i) {
                    const int m = m0 + r0 + 16 * i;
                    x[i] = m < M && k < K ? *reinterpret_cast<const float4*>(A + (size_t)m * lda + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                if (turn_no >= STAGES) gf_bar_sync(BAR_FREE + s, GF_ROLE_ALL);
#pragma unroll
                for (int i = 0; i < TM / 16; ++i) {
                    float* dst = a_s + q * 4 * TM + ((r0 + 16 * i) ^ (q * 4));
                    dst[0] = x[i].x; dst[TM] = x[i].y; dst[2 * TM] = x[i].z; dst[3 * TM] = x[i].w;
                }
                float4 y[TN / 16];
#pragma unroll
                for (int i = 0; i < TN / 16; ++i) {
                    const int n = n0 + r0 + 16 * i;
                    y[i] = n < N && k < K ? *reinterpret_cast<const float4*>(W + (size_t)n * ldw + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int i = 0; i < TN / 16; ++i) {
                    float* dst = w_s + q * 4 * TN + ((r0 + 16 * i) ^ (q * 4));
                    dst[0] = y[i].x; dst[TN] = y[i].y; dst[2 * TN] = y[i].z; dst[3 * TN] = y[i].w;
                }
                gf_bar_arrive(BAR_FULL + s, GF_ROLE_ALL);
            }
        }
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    const int tx = lane % 8 + 8 * (warp % 2), ty = lane / 8 + 4 * (warp / 2);    // columns 4 tx .. + 3 (and + 64); rows likewise
    const unsigned long long minus_one = f2_twice(-1.0f);
    const int all_turns = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * turns;
    int turn_no = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int m0 = tile % m_tiles * TM, n0 = tile / m_tiles * TN;
        unsigned long long acc[RM][RN / 2], kept[RM][RN / 2];            // two columns each
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN / 2; ++j) { acc[i][j] = 0ull; kept[i][j] = 0ull; }
        for (int turn = 0; turn < turns; ++turn, ++turn_no) {
            const int s = turn_no % STAGES;
            const float* a_s = gf_smem + s * STAGE;
            const float* w_s = a_s + TK * TM;
            gf_bar_sync(BAR_FULL + s, GF_ROLE_ALL);
#pragma unroll
            for (int half = 0; half < TK / GF_CHUNK; ++half) {
                if (turn * TK + half * GF_CHUNK >= K) break;
                unsigned long long part[RM][RN / 2];
#pragma unroll
                for (int i = 0; i < RM; ++i)
#pragma unroll
                    for (int j = 0; j < RN / 2; ++j) part[i][j] = 0ull;
#pragma unroll
                for (int k4 = 0; k4 < GF_CHUNK / 4; ++k4) {
                    const int swap = (half * 4 + k4) * 4;
                    const float* ab = a_s + (half * GF_CHUNK + k4 * 4) * TM + ((4 * ty) ^ swap);
                    const float* wb = w_s + (half * GF_CHUNK + k4 * 4) * TN + ((4 * tx) ^ swap);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        float a[RM];
                        unsigned long long w[RN / 2];
#pragma unroll
                        for (int g = 0; g < RM / 4; ++g) {
                            const float4 x = *reinterpret_cast<const float4*>(ab + k * TM + 64 * g);
                            a[4 * g] = x.x; a[4 * g + 1] = x.y; a[4 * g + 2] = x.z; a[4 * g + 3] = x.w;
                        }
#pragma unroll
                        for (int g = 0; g < RN / 4; ++g) {
                            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(wb + k * TN + 64 * g);
                            w[2 * g] = x.x; w[2 * g + 1] = x.y;
                        }
#pragma unroll
                        for (int i = 0; i < RM; ++i) {
                            const unsigned long long aa = f2_twice(a[i]);
#pragma unroll
                            for (int j = 0; j < RN / 2; ++j) part[i][j] = f2_fma(aa, w[j], part[i][j]);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < RM; ++i)
#pragma unroll
                    for (int j = 0; j < RN / 2; ++j) gf_kahan2(acc[i][j], kept[i][j], part[i][j], minus_one);
            }
            if (turn_no + STAGES < all_turns) gf_bar_arrive(BAR_FREE + s, GF_ROLE_ALL);
        }
#pragma unroll
        for (int i = 0; i < RM; ++i) {
            const int m = m0 + 64 * (i / 4) + 4 * ty + i % 4;
            if (m >= M) continue;
#pragma unroll
            for (int j = 0; j < RN / 2; ++j) {
                const int n = n0 + 64 * (j / 2) + 4 * tx + 2 * (j % 2);
                float* dst = C + (size_t)m * ldc + n;
                const float lo = f2_lo(acc[i][j]), hi = f2_hi(acc[i][j]);
                if (n < N) dst[0] = accumulate ? dst[0] + lo : lo;
                if (n + 1 < N) dst[1] = accumulate ? dst[1] + hi : hi;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// 17 to 300 rows: too few for tiles of 64 columns to fill the SMs, too many to stream the weights 16 rows at a time.  A block's
// warps take a chunk of k each of one tile of 8 RM x 4 RN results, RM x RN a lane, from rows as they lie in memory; the chunks' sums
// go through shared memory to the threads that own the results, which add them in k order while the next turn is multiplied.
// Bound by the shared-memory reads beside the multiply-adds (12 of 16 bytes for 128 multiply-adds a lane, then a chunk's sums
// written and read).  us before (16 rows at a time, or tiles of 64 x 64) and here, rows x columns x k:
//   tiles of 64 x 16: 64 x 2048 x 2048 51 and 34, 64 x 2048 x 8192 193 and 125, 100 x 2048 x 8192 333 and 246, 300 x 2048 x 2048 181
//   and 155, 200 x 512 x 128 9.4 and 4.3;
//   tiles of 32 x 32: 32 x 16384 x 2048 170 and 152, 32 x 4096 x 4096 98 and 77.
// Tiles of 64 x 32, 8 x 8 results a lane: 64 x 2048 x 2048 72, 64 x 16384 x 2048 284 (191 with tiles of 64 x 64, 219 of 64 x 16).
// ---------------------------------------------------------------------------------------------------------------------
constexpr int GF_PART_WARPS = 8, GF_PART_K = GF_PART_WARPS * GF_CHUNK, GF_PART_LD = GF_PART_K + 4, GF_PART_STAGES = 3;
template <int RM, int RN>
constexpr size_t gf_part_smem() {
    return sizeof(float) * ((size_t)GF_PART_STAGES * (8 * RM + 4 * RN) * GF_PART_LD + (size_t)2 * GF_PART_WARPS * 32 * RM * RN);
}

template <int RM, int RN>
__global__ void __launch_bounds__(32 * GF_PART_WARPS, 1)
gemm_f32_part_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C, int ldc,
                     int M, int N, int K, long long a_batch, long long w_batch, long long c_batch, int accumulate) {
    constexpr int TM = 8 * RM, TN = 4 * RN, TILE = TM * TN;
    static_assert(TILE == 4 * 32 * GF_PART_WARPS, "a thread owns four results");
    extern __shared__ __align__(16) float gf_smem[];
    float* sums = gf_smem + GF_PART_STAGES * (TM + TN) * GF_PART_LD;     // [2][chunk of the turn][row][4 RN columns, exchanged]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane % 8, lc = lane / 8;
    A += (size_t)blockIdx.z * a_batch;
    W += (size_t)blockIdx.z * w_batch;
    C += (size_t)blockIdx.z * c_batch;
    const int m_tiles = (M + TM - 1) / TM, tiles = m_tiles * ((N + TN - 1) / TN);
    const int chunks = (K + GF_CHUNK - 1) / GF_CHUNK, turns = (K + GF_PART_K - 1) / GF_PART_K;
    const int all = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * turns;
    int f_tile = blockIdx.x, f_turn = 0;                             // what is fetched next
    auto fetch = [&](int stage) {
        if (f_tile < tiles) {
            const int m0 = f_tile % m_tiles * TM, n0 = f_tile / m_tiles * TN, k = f_turn * GF_PART_K + 4 * lane;
            float* dst = gf_smem + stage * (TM + TN) * GF_PART_LD + warp * GF_PART_LD + 4 * lane;    // a warp fetches 512 bytes of a row
#pragma unroll
            for (int e = 0; e < (TM + TN) / GF_PART_WARPS; ++e) {
                const int r = warp + e * GF_PART_WARPS;
                const bool of_a = e < TM / GF_PART_WARPS;
                const int row = of_a ? m0 + r : n0 + r - TM;
                const bool in = k < K && row < (of_a ? M : N);
                gf_cp16(dst + e * GF_PART_WARPS * GF_PART_LD, !in ? A : of_a ? A + (size_t)row * lda + k : W + (size_t)row * ldw + k, in ? 16 : 0);
            }
            if (++f_turn == turns) { f_turn = 0; f_tile += gridDim.x; }
        }
        gf_commit();
    };
#pragma unroll
    for (int s = 0; s < GF_PART_STAGES - 1; ++s) fetch(s);
    const unsigned long long minus_one = f2_twice(-1.0f);
    unsigned long long acc[2] = {0, 0}, kept[2] = {0, 0};            // four results
    int a_tile = blockIdx.x, a_turn = 0, stage = 0;
    auto add = [&](int buffer) {                                     // a turn's sums
        const float* src = sums + buffer * GF_PART_WARPS * TILE + 4 * tid;
        const int here = min(GF_PART_WARPS, chunks - a_turn * GF_PART_WARPS);
#pragma unroll
        for (int c = 0; c < GF_PART_WARPS; ++c) {
            if (c >= here) break;
            const ulonglong2 part = *reinterpret_cast<const ulonglong2*>(src + c * TILE);
            gf_kahan2(acc[0], kept[0], part.x, minus_one);
            gf_kahan2(acc[1], kept[1], part.y, minus_one);
        }
        if (++a_turn < turns) return;
        // a row's results lie [column / 16][column % 4][column / 4 % 4]
        const int m = a_tile % m_tiles * TM + 4 * tid / TN, place = 4 * tid % TN, n0 = a_tile / m_tiles * TN + place / 16 * 16 + place % 16 / 4;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float x = __uint_as_float((unsigned)(acc[e / 2] >> (32 * (e % 2))));
            if (m < M && n0 + 4 * e < N) {
                float* dst = C + (size_t)m * ldc + n0 + 4 * e;
                *dst = accumulate ? *dst + x : x;
            }
        }
        acc[0] = acc[1] = kept[0] = kept[1] = 0;
        a_turn = 0;
        a_tile += gridDim.x;
    };
    for (int turn = 0; turn < all; ++turn) {
        gf_wait<GF_PART_STAGES - 2>();
        __syncthreads();                                             // this turn has landed, the one before is multiplied
        fetch(stage == 0 ? GF_PART_STAGES - 1 : stage - 1);
        if (turn > 0) add((turn - 1) & 1);
        float part[RM][RN];
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN; ++j) part[i][j] = 0.f;
        const float* a_s = gf_smem + stage * (TM + TN) * GF_PART_LD + lr * GF_PART_LD + warp * GF_CHUNK;
        const float* w_s = gf_smem + stage * (TM + TN) * GF_PART_LD + (TM + lc) * GF_PART_LD + warp * GF_CHUNK;
#pragma unroll
        for (int k = 0; k < GF_CHUNK; k += 4) {
            float4 w[RN];
#pragma unroll
            for (int j = 0; j < RN; ++j) w[j] = *reinterpret_cast<const float4*>(w_s + j * 4 * GF_PART_LD + k);
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(a_s + i * 8 * GF_PART_LD + k);
#pragma unroll
                for (int j = 0; j < RN; ++j) {
                    part[i][j] = fmaf(a.x, w[j].x, part[i][j]);
                    part[i][j] = fmaf(a.y, w[j].y, part[i][j]);
                    part[i][j] = fmaf(a.z, w[j].z, part[i][j]);
                    part[i][j] = fmaf(a.w, w[j].w, part[i][j]);
                }
            }
        }
        float* dst = sums + ((turn & 1) * GF_PART_WARPS + warp) * TILE + lr * TN + 4 * lc;
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN; j += 4)
                *reinterpret_cast<float4*>(dst + i * 8 * TN + 4 * j) = make_float4(part[i][j], part[i][j + 1], part[i][j + 2], part[i][j + 3]);
        stage = stage + 1 == GF_PART_STAGES ? 0 : stage + 1;
    }
    __syncthreads();
    add((all - 1) & 1);
    gf_wait<0>();
}

// ---------------------------------------------------------------------------------------------------------------------
// Whether the operands can be fetched in 16-byte pieces (rows of W and A start on 16-byte boundaries, K in whole pieces).
static inline bool gemm_f32_ok(const void* A, int lda, long long a_batch, const void* W, int ldw, long long w_batch, int K) {
    return !(((uintptr_t)A | (uintptr_t)W) & 15) && !((lda | ldw | K) & 3) && !((a_batch | w_batch) & 3);
}

// Which kernel takes a product: one that streams the weights once for up to 16 rows at a time, or one of the tiles, whichever
// is done first by the time a chunk of 16 k takes it: the blocks run in waves over the SMs, and tiles that are too large leave
// SMs idle where tiles that are too small fetch more often than they multiply.  Hundredths of a microsecond a chunk, measured
// for 1 and for each further wave: up to 4, 8 and 16 rows x 16 columns a block 5 to 3 + 3.8, 5 and 10, whole turns of 32 chunks
// whatever K is; tiles of 64 x 64 90 + 60, of 128 x 64 145 + 115, of 128 x 128 167 + 167, of 64 x 16 and 32 x 32 by chunks 24 and 29 (whole turns of 8),
// and 3 us to start and end.  A walking warp's turn: 4 rows of W 65, 70 and 85 (1, 2, 4 rows of A), 2 rows 80, 1 row 130,
// and 3 us.  Sides of the lines it draws (us; rows x columns, k 2048): 32 x 2048 27 with 16 rows and 33 by chunks of 64 x 16; 64 x 2048
// 51 and 34; 64 x 16384 219 by chunks and 191 with tiles of 64; 128 x 3072 95 by chunks, 114 with tiles of 64; 300 x 2048 155 by
// chunks, 181 with 128 x 64; 300 x 3072 182 with 128 x 64, 189 with 64 x 64, 217 with 128 x 128; 500 x 3072 217 with 128 x 128, 266
// with 64 x 64; 500 x 2048 181 with 128 x 64, 217; 1000 x 2048 217 and 318.  K 64: 300 x 64 5.3 with 16 rows, 6.5 with tiles of
// 64; 16 x 8192 14.3 and 6.1.  16 x 128256, k 256 155 and 141, k 512 171 and 274.  Blocks of 16 rows that stay for many waves take 9.3
// a wave and 4.2 us in all (of whole chunks; k 1500 is 10 % above that): 32 x 6144, k 4096 146 and 153 with 32 x 32, 32 x 3072 75 and
// 78, 33 x 5120, k 8192 330 and 366 by chunks of 64 x 16, 48 x 10240, k 5120 390 and 382.
static inline int gemm_f32_form(int n_batch, int M, int N, int K) {
    const long long sms = ssb_sm_count(), chunks = (K + 15) / 16, turns = (K + 511) / 512;
    const auto waves = [&](int rows, int cols) {
        return ((long long)((M + rows - 1) / rows) * ((N + cols - 1) / cols) * n_batch + sms - 1) / sms;
    };
    const bool walk = gf_walk_ok(M, K);
    const int rows = M <= 4 ? 4 : M <= 8 ? 8 : 16;
    const int first = rows < 16 ? 50 : 30, each = rows == 4 ? 38 : rows == 8 ? 50 : 100;
    const int forms[6] = {walk ? (M <= 2 ? M : 4) : M <= 4 ? 5 : rows, 100, 101, 102, 103, 104};
    const long long parts = (chunks + GF_PART_WARPS - 1) / GF_PART_WARPS * GF_PART_WARPS;
    long long cost[6] = {32 * turns * (first + each * waves(rows, 16)), 3000 + 10 * chunks * (30 + 60 * waves(64, 64)),
                         3000 + 10 * chunks * (30 + 115 * waves(128, 64)), 3000 + 10 * chunks * 167 * waves(128, 128),
                         3000 + 10 * parts * 24 * waves(64, 16), 3000 + 10 * parts * 29 * waves(32, 32)};
    if (rows == 16 && n_batch == 1 && K % 16 == 0) {
        const long long steady = 4200 + 32 * turns * 93 * waves(16, 16);
        if (steady < cost[0]) cost[0] = steady;
    }
    if (walk) {
        const int width = gf_walk_width(N), turn = width == 1 ? 1300 : width == 2 ? 800 : M <= 1 ? 650 : M <= 2 ? 700 : 850;
        const long long held = sms * GF_WALK_WARPS, rounds = ((long long)((N + width - 1) / width) * n_batch + held - 1) / held;
        cost[0] = 3000 + ((K + GF_WALK_TURN / width - 1) / (GF_WALK_TURN / width)) * rounds * turn;
    }
    int best = 0;
    for (int f = 1; f < 6; ++f)
        if (cost[f] < cost[best]) best = f;
    return forms[best];
}

// Whether a gated unit's first product is made by walking warps, which finish it.
static inline bool gemm_f32_gated_ok(int M, int N, int K) { return N % 2 == 0 && gemm_f32_form(1, M, N, K) <= 4; }

// form 0: chosen by the sizes; else one of the kernels: 1, 2, 4 (a warp walks), 5, 8, 16 (few rows, 4, 8, 16 a group), 100, 101, 102 (tiles of
// 64 x 64, 128 x 64 and 128 x 128), 103, 104 (a tile of 64 x 16, 32 x 32 by chunks of k)
static inline int gemm_f32_launch(const float* A, int lda, long long a_batch, const float* W, int ldw, long long w_batch,
                                  float* C, int ldc, long long c_batch, int n_batch, int M, int N, int K, int accumulate,
                                  int form, cudaStream_t stream, bool pdl = false, const GfGate* gate = nullptr) {
    if (form == 0) form = gemm_f32_form(n_batch, M, N, K);
    if (gate && (form > 4 || n_batch != 1 || N % 2)) return SSB_ERR_UNSUPPORTED;
#define GF_CONFIGURE(kernel, smem) do { \
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem)); \
        if (e != cudaSuccess) return (int)e; \
    } while (0)
#define GF_SKINNY(MB, R, STAGES) do { \
        constexpr size_t smem = gf_skinny_smem<MB, R, STAGES>(); \
        auto kernel = gemm_f32_skinny_kernel<MB, R, STAGES>; \
        GF_CONFIGURE(kernel, smem); \
        const int groups = (M + MB - 1) / MB; \
        const long long tiles = (long long)groups * ((N + 8 * R - 1) / (8 * R)); \
        if (tiles > 0x7fffffffLL) return SSB_ERR_BAD_SIZE; \
        /* as many blocks as are resident at once (by shared memory), each walking its share of the tiles */ \
        const long long held = ssb_sm_count() * (228 * 1024 / (long long)(smem + 1024)); \
        const long long blocks = tiles < held ? tiles : held; \
        kernel<<<dim3((unsigned)blocks, 1, n_batch), GF_PRODUCT_THREADS + gf_adders(MB, R), smem, stream>>>( \
            A, lda, W, ldw, C, ldc, M, N, K, a_batch, w_batch, c_batch, groups, accumulate); \
    } while (0)
#define GF_TILES(RM, RN, ...) do { \
        constexpr size_t smem = gf_tile_smem<RM, RN>(); \
        auto kernel = gemm_f32_tile_kernel<RM, RN, __VA_ARGS__>; \
        GF_CONFIGURE(kernel, smem); \
        const int rows = 16 * RM, cols = 16 * RN; \
        if ((M + rows - 1) / rows > 65535) return SSB_ERR_BAD_SIZE; \
        kernel<<<dim3((N + cols - 1) / cols, (M + rows - 1) / rows, n_batch), GF_TILE_THREADS, smem, stream>>>( \
            A, lda, W, ldw, C, ldc, M, N, K, a_batch, w_batch, c_batch, accumulate); \
    } while (0)
#define GF_WALK(MB, RW, ...) do { \
        const size_t rows = gf_walk_rows(MB, K); \
        auto kernel = gemm_f32_walk_kernel<MB, RW, ##__VA_ARGS__>; \
        GF_CONFIGURE(kernel, GF_WALK_SMEM); \
        const int tasks = (N + RW - 1) / RW, blocks = tasks < ssb_sm_count() ? tasks : ssb_sm_count(), room = (int)((GF_WALK_SMEM - rows) / GF_WALK_RING); \
        int warps = (tasks + blocks - 1) / blocks; \
        warps = warps > GF_WALK_WARPS ? GF_WALK_WARPS : warps; \
        warps = warps > room ? room : warps; \
        const int rc = ssb_launch(kernel, dim3((unsigned)blocks, 1, n_batch), dim3(32 * warps), rows + warps * GF_WALK_RING, \
                                  stream, pdl, A, lda, W, ldw, C, ldc, M, N, K, a_batch, w_batch, c_batch, accumulate, gate ? *gate : GfGate{}); \
        if (rc) return rc; \
    } while (0)
#define GF_WALKS(MB) do { \
        const int width = gf_walk_width(N); \
        if (gate) { if (width == 4) GF_WALK(MB, 4, true); else GF_WALK(MB, 2, true); } \
        else if (width == 4) GF_WALK(MB, 4); else if (width == 2) GF_WALK(MB, 2); else GF_WALK(MB, 1); \
    } while (0)
#define GF_ROLES(RM, RN) do { \
        constexpr size_t smem = gf_role_smem<RM, RN>(); \
        auto kernel = gemm_f32_role_kernel<RM, RN>; \
        GF_CONFIGURE(kernel, smem); \
        const long long tiles = (long long)((N + 16 * RN - 1) / (16 * RN)) * ((M + 16 * RM - 1) / (16 * RM)); \
        if (tiles > 0x7fffffffLL) return SSB_ERR_BAD_SIZE; \
        kernel<<<dim3((unsigned)(tiles < ssb_sm_count() ? tiles : ssb_sm_count()), 1, n_batch), GF_ROLE_ALL, smem, stream>>>( \
            A, lda, W, ldw, C, ldc, M, N, K, a_batch, w_batch, c_batch, accumulate); \
    } while (0)
#define GF_PARTS(RM, RN) do { \
        constexpr size_t smem = gf_part_smem<RM, RN>(); \
        auto kernel = gemm_f32_part_kernel<RM, RN>; \
        GF_CONFIGURE(kernel, smem); \
        const long long tiles = (long long)((N + 4 * RN - 1) / (4 * RN)) * ((M + 8 * RM - 1) / (8 * RM)); \
        if (tiles > 0x7fffffffLL) return SSB_ERR_BAD_SIZE; \
        kernel<<<dim3((unsigned)(tiles < ssb_sm_count() ? tiles : ssb_sm_count()), 1, n_batch), 32 * GF_PART_WARPS, smem, stream>>>( \
            A, lda, W, ldw, C, ldc, M, N, K, a_batch, w_batch, c_batch, accumulate); \
    } while (0)
    switch (form) {
        case 1: GF_WALKS(1); break;
        case 2: GF_WALKS(2); break;
        case 4: GF_WALKS(4); break;
        case 5: GF_SKINNY(4, 2, 3); break;
        case 8: GF_SKINNY(8, 2, 3); break;
        case 16: GF_SKINNY(16, 2, 2); break;
        case 100: GF_TILES(4, 4, 3); break;
        case 101: GF_TILES(8, 4, 2); break;
        case 102: GF_ROLES(8, 8); break;
        case 103: GF_PARTS(8, 4); break;
        case 104: GF_PARTS(4, 8); break;
        default: return SSB_ERR_BAD_SIZE;
    }
#undef GF_SKINNY
#undef GF_WALK
#undef GF_WALKS
#undef GF_ROLES
#undef GF_PARTS
#undef GF_TILES
#undef GF_CONFIGURE
    return ssb_launch_status();
}
