// Order statistics of a device array (the payoff distribution's percentiles,
// OptionPricer.hpp:340-360, which sorts every path's payoff on the host for 15 of them).
//
// Radix selection, eight bits of the values' ordered bit patterns a pass: one launch per
// pass histograms the next digit of the values that share a wanted rank's prefix so far
// (at most kSelectRanks distinct prefixes), and the last block to finish picks each rank's
// digit.  Exact: the selected values are elements of the array.  Bound by launch latency
// for small arrays (nine launches) and by eight reads of the array for large ones.  A
// configuration's run with percentiles (FP64 Asian, 100,000 x 128): 4.57 ms when every
// payoff was copied to the host and sorted there, 0.49 ms with a first form of these passes,
// 0.27 ms now, with the payoffs taken from the pricing's own paths.
#include <cuda_runtime.h>

#include "qk_kernels.h"

namespace qk {

namespace {

struct SelectState {
    unsigned long long prefix[kSelectRanks];  // digits fixed so far
    unsigned long long rank[kSelectRanks];    // rank among the values with that prefix
    unsigned int hist[kSelectRanks][256];     // by group: ranks with equal prefixes share one
    unsigned int done;
};

// Bit pattern whose unsigned order is the values' order.
__device__ __forceinline__ unsigned long long ordered_bits(double x) {
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x));
    return (b >> 63) ? ~b : b | 0x8000000000000000ull;
}
__device__ __forceinline__ double from_ordered_bits(unsigned long long k) {
    return __longlong_as_double(static_cast<long long>((k >> 63) ? k & 0x7FFFFFFFFFFFFFFFull : ~k));
}

constexpr int kSelectBlock = 256;

__global__ void __launch_bounds__(kSelectBlock) select_pass_kernel(const double *__restrict__ x, int64_t n, int n_ranks,
                                                                   int pass, SelectState *st, double *__restrict__ out) {
    __shared__ unsigned int s_hist[kSelectRanks][256];
    __shared__ unsigned long long s_prefix[kSelectRanks];  // by group
    __shared__ int s_group[kSelectRanks];                  // by rank
    __shared__ int s_n_groups;
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) {  // a lane per rank: one load latency
        const unsigned long long p = lane < n_ranks ? st->prefix[lane] : 0ull;
        const unsigned long long before = __shfl_up_sync(0xffffffffu, p, 1);
        const bool first = lane < n_ranks && (lane == 0 || p != before);
        const unsigned heads = __ballot_sync(0xffffffffu, first);
        const int g = __popc(heads & (0xffffffffu >> (31 - lane))) - 1;
        if (first) s_prefix[g] = p;
        if (lane < n_ranks) s_group[lane] = g;
        if (lane == 0) s_n_groups = __popc(heads);
    }
    for (int i = threadIdx.x; i < kSelectRanks * 256; i += kSelectBlock) (&s_hist[0][0])[i] = 0u;
    __syncthreads();
    const int groups = s_n_groups;
    const int shift = 56 - 8 * pass;
    // whole warps: the lanes of a warp with the same bin add once
    for (int64_t i0 = static_cast<int64_t>(blockIdx.x) * kSelectBlock + warp * 32; i0 < n;
         i0 += static_cast<int64_t>(gridDim.x) * kSelectBlock) {
        const bool have = i0 + lane < n;
        const unsigned long long k = have ? ordered_bits(x[i0 + lane]) : 0ull;
        const unsigned long long head = pass == 0 ? 0ull : k >> (shift + 8);
        int bin = -1;
        for (int g = 0; g < groups; ++g)
            if (have && head == s_prefix[g]) bin = g * 256 + static_cast<int>((k >> shift) & 255u);
        const unsigned same = __match_any_sync(0xffffffffu, bin);
        if (bin >= 0 && lane == __ffs(same) - 1) atomicAdd(&s_hist[0][0] + bin, static_cast<unsigned>(__popc(same)));
    }
    __syncthreads();
    for (int i = threadIdx.x; i < groups * 256; i += kSelectBlock) {
        const unsigned v = (&s_hist[0][0])[i];
        if (v) atomicAdd(&st->hist[0][0] + i, v);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&st->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    // last block: rank r's digit, a warp per rank, eight bins per lane
    __threadfence();
    for (int r = warp; r < n_ranks; r += kSelectBlock / 32) {
        const int g = s_group[r];
        // one lane reads the rank that one lane replaces below: the shuffle orders the two
        const unsigned long long want = __shfl_sync(0xffffffffu, lane == 0 ? st->rank[r] : 0ull, 0);
        unsigned c[8], sum = 0;
        for (int j = 0; j < 8; ++j) sum += c[j] = __ldcg(&st->hist[g][8 * lane + j]);
        unsigned before = sum;  // inclusive, then exclusive, sum over the lanes
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned o = __shfl_up_sync(0xffffffffu, before, off);
            if (lane >= off) before += o;
        }
        before -= sum;
        if (want >= before && want < static_cast<unsigned long long>(before) + sum) {
            unsigned long long left = want - before;
            int j = 0;
            while (left >= c[j]) left -= c[j++];
            const unsigned long long prefix = (pass == 0 ? 0ull : s_prefix[g] << 8) | static_cast<unsigned>(8 * lane + j);
            st->prefix[r] = prefix;
            st->rank[r] = left;
            if (pass == 7) out[r] = from_ordered_bits(prefix);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < groups * 256; i += kSelectBlock) (&st->hist[0][0])[i] = 0u;
    if (threadIdx.x == 0) st->done = 0u;
}

__global__ void select_init_kernel(SelectState *st, SelectRanks ranks) {
    for (int i = threadIdx.x; i < kSelectRanks * 256; i += blockDim.x) (&st->hist[0][0])[i] = 0u;
    if (threadIdx.x < kSelectRanks) {
        st->prefix[threadIdx.x] = 0ull;
        st->rank[threadIdx.x] = ranks.r[threadIdx.x];
    }
    if (threadIdx.x == 0) st->done = 0u;
}

}  // namespace

size_t select_scratch_bytes() { return (sizeof(SelectState) + 255) / 256 * 256; }

cudaError_t launch_select(cudaStream_t s, int sm_count, const double *x, int64_t n, const SelectRanks &ranks, int n_ranks,
                          void *scratch, double *out) {
    SelectState *st = static_cast<SelectState *>(scratch);
    select_init_kernel<<<1, 256, 0, s>>>(st, ranks);
    // a value per thread where that is at most four blocks per SM: a pass over few values is a
    // chain of latencies, and each value a thread takes adds one (100,000 values, eight passes:
    // 147 us with eight values a thread, the prefixes read one after another and the results
    // copied from the device; 90 us)
    const int64_t blocks = (n + kSelectBlock - 1) / kSelectBlock;
    const int grid = static_cast<int>(blocks < 4 * sm_count ? (blocks < 1 ? 1 : blocks) : 4 * sm_count);
    for (int pass = 0; pass < 8; ++pass)
        select_pass_kernel<<<grid, kSelectBlock, 0, s>>>(x, n, n_ranks, pass, st, out);
    return cudaGetLastError();
}

cudaError_t preload_select_kernels() {
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, select_pass_kernel);
    return e == cudaSuccess ? cudaFuncGetAttributes(&fa, select_init_kernel) : e;
}

}  // namespace qk
