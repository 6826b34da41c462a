// What the host hands a step or a new sequence, as kernel arguments: a step's token ids, positions and slots, a sequence's
// generator seed.  A copy from host memory, however small, goes through a copy engine: between two steps of a decode loop the
// device stood still 14 us before it and 10 us behind it (a 1B model's step takes 640), and a scalar written into a tensor is a
// copy from pageable memory, 24 us for each sequence that is opened.  A launch's arguments are taken when it is made, so that
// no staging buffer has to outlive it.
#include "common.cuh"

template <int N>
struct StepInts { int v[N]; };

template <int N>
__global__ void __launch_bounds__(256)
put_ints_kernel(const __grid_constant__ StepInts<N> x, int n, const int* __restrict__ before, int n_before, int* __restrict__ dst) {
    for (int i = threadIdx.x; i < n_before + n; i += 256) dst[i] = i < n_before ? before[i] : x.v[i - n_before];
}

constexpr int PUT_FEW = 128, PUT_MOST = 960;             // arguments of half and of four kilobytes

// dst = the n_before ints at ``before`` on the device, then the n host values; n up to ssb_put_ints_most()
SSB_API int ssb_put_ints_most() { return PUT_MOST; }
SSB_API int ssb_put_ints(const int* values, int n, const int* before, int n_before, int* dst, cudaStream_t stream) {
    if (n < 0 || n > PUT_MOST || n_before < 0) return SSB_ERR_BAD_SIZE;
    if (n + n_before == 0) return 0;
    if (n <= PUT_FEW) {
        StepInts<PUT_FEW> x = {};
        for (int i = 0; i < n; ++i) x.v[i] = values[i];
        put_ints_kernel<PUT_FEW><<<1, 256, 0, stream>>>(x, n, before, n_before, dst);
    } else {
        StepInts<PUT_MOST> x = {};
        for (int i = 0; i < n; ++i) x.v[i] = values[i];
        put_ints_kernel<PUT_MOST><<<1, 256, 0, stream>>>(x, n, before, n_before, dst);
    }
    return ssb_launch_status();
}

// A sequence's slot: its generator's state, and the rows of fixed state (words of four bytes) zeroed.
constexpr int OPEN_STATES = 96;                          // rows a launch
struct OpenRows { unsigned* row[OPEN_STATES]; int words[OPEN_STATES]; };

__global__ void __launch_bounds__(256)
open_sequence_kernel(const __grid_constant__ OpenRows x, long long* __restrict__ rng, long long seed) {
    if (rng && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *rng = seed;
    unsigned* row = x.row[blockIdx.y];
    const int n = x.words[blockIdx.y];
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) row[i] = 0u;
}

SSB_API int ssb_open_sequence(long long* rng, long long seed, void* const* rows, const int* words, int n_rows, cudaStream_t stream) {
    if (n_rows < 0 || (n_rows > 0 && (!rows || !words))) return SSB_ERR_BAD_SIZE;
    for (int at = 0; at == 0 || at < n_rows; at += OPEN_STATES) {
        OpenRows x = {};
        const int n = n_rows - at < OPEN_STATES ? n_rows - at : OPEN_STATES;
        int most = 0;
        for (int i = 0; i < n; ++i) {
            x.row[i] = (unsigned*)rows[at + i];
            x.words[i] = words[at + i];
            most = words[at + i] > most ? words[at + i] : most;
        }
        const int blocks = (most + 2047) / 2048;
        open_sequence_kernel<<<dim3(blocks < 1 ? 1 : blocks > 148 ? 148 : blocks, n < 1 ? 1 : n), 256, 0, stream>>>(
            x, at == 0 ? rng : nullptr, seed);
        const int rc = ssb_launch_status();
        if (rc) return rc;
    }
    return 0;
}
