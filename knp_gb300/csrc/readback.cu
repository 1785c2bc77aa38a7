// Read-back of recorded spikes: turns steps' bitmaps on the device into lists of ascending indexes in
// pinned host memory, so that neither whole bitmaps cross to the host nor the host looks for the bits.
//
// A step's bitmap of W words is cut into segments of kSegWords words. The first kernel counts each
// segment's spikes; the second, one block per segment again, knows from the counts where its indexes
// start, compacts them in shared memory and stores them coalesced into the step's span of W words of
// the host buffer. A step with more than W spikes keeps its bitmap (the list would be longer): the host
// copies it. Bound by latency at low rates (20 steps of 10^6 neurons, 5300 spikes each: 1.3 MB of lists'
// sectors against 2.5 MB of bitmaps and 0.6 M words for the host to scan).
#include <cstdint>

#include <cuda_runtime.h>

#include "kernels.h"

namespace knp_gb300
{
namespace
{

constexpr int kSegThreads = 256;
constexpr uint32_t kSegWords = kReadbackSegWords;
constexpr uint32_t kWordsPerThread = kSegWords / kSegThreads;
constexpr uint32_t kStageCap = 4096;  // indexes compacted in shared memory; a denser segment stores directly

__device__ __forceinline__ uint32_t block_sum(uint32_t v)
{
    __shared__ uint32_t part[kSegThreads / 32];
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t s = 0;
    for (int i = 0; i < kSegThreads / 32; ++i) s += part[i];
    __syncthreads();
    return s;
}

// Words of this thread in segment `seg` of the bitmap of step first + blockIdx.y (zeros past W).
__device__ __forceinline__ void load_words(const uint32_t *bits, uint32_t W, uint32_t slots, unsigned long long first,
                                           uint32_t (&w)[kWordsPerThread])
{
    const uint32_t *row = bits + static_cast<size_t>((first + blockIdx.y) % slots) * W;
    const uint32_t w0 = blockIdx.x * kSegWords + threadIdx.x * kWordsPerThread;
#pragma unroll
    for (uint32_t i = 0; i < kWordsPerThread; ++i) w[i] = w0 + i < W ? row[w0 + i] : 0u;
}

__global__ void __launch_bounds__(kSegThreads) segment_count_kernel(const uint32_t *bits, uint32_t W, uint32_t slots,
                                                                   unsigned long long first, uint32_t *counts,
                                                                   uint32_t *counts_host)
{
    uint32_t w[kWordsPerThread];
    load_words(bits, W, slots, first, w);
    uint32_t c = 0;
#pragma unroll
    for (uint32_t i = 0; i < kWordsPerThread; ++i) c += __popc(w[i]);
    const uint32_t total = block_sum(c);
    if (threadIdx.x == 0)
    {
        const size_t at = static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x;
        counts[at] = total;
        counts_host[at] = total;
    }
}

__global__ void __launch_bounds__(kSegThreads) segment_list_kernel(const uint32_t *bits, uint32_t W, uint32_t slots,
                                                                  unsigned long long first, const uint32_t *counts,
                                                                  uint32_t *lists)
{
    __shared__ uint32_t stage[kStageCap];
    __shared__ uint32_t warp_base[kSegThreads / 32];
    const uint32_t *seg_counts = counts + static_cast<size_t>(blockIdx.y) * gridDim.x;
    uint32_t before = 0, all = 0;
    for (uint32_t i = threadIdx.x; i < gridDim.x; i += kSegThreads)
    {
        const uint32_t c = seg_counts[i];
        all += c;
        if (i < blockIdx.x) before += c;
    }
    before = block_sum(before);
    all = block_sum(all);
    const uint32_t mine = seg_counts[blockIdx.x];
    if (all > W || mine == 0) return;  // the same in every thread
    uint32_t w[kWordsPerThread];
    load_words(bits, W, slots, first, w);
    uint32_t c = 0;
#pragma unroll
    for (uint32_t i = 0; i < kWordsPerThread; ++i) c += __popc(w[i]);
    // Exclusive prefix over the block's threads.
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) warp_base[warp] = incl;
    __syncthreads();
    uint32_t k = incl - c;
    for (int i = 0; i < warp; ++i) k += warp_base[i];
    uint32_t *out = lists + static_cast<size_t>(blockIdx.y) * W + before;
    const bool staged = mine <= kStageCap;
    uint32_t *dst = staged ? stage : out;
    const uint32_t n0 = 32 * (blockIdx.x * kSegWords + threadIdx.x * kWordsPerThread);
#pragma unroll
    for (uint32_t i = 0; i < kWordsPerThread; ++i)
        for (uint32_t x = w[i]; x; x &= x - 1) dst[k++] = n0 + 32 * i + __ffs(x) - 1;
    if (!staged) return;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < mine; i += kSegThreads) out[i] = stage[i];
}

}  // namespace

uint32_t readback_segments(uint32_t W) { return (W + kSegWords - 1) / kSegWords; }

cudaError_t launch_spike_lists(const uint32_t *bits, uint32_t W, uint32_t slots, uint64_t first, uint32_t n_steps,
                               uint32_t *counts, uint32_t *counts_host, uint32_t *lists_host, cudaStream_t s)
{
    const dim3 grid(readback_segments(W), n_steps);
    segment_count_kernel<<<grid, kSegThreads, 0, s>>>(bits, W, slots, first, counts, counts_host);
    segment_list_kernel<<<grid, kSegThreads, 0, s>>>(bits, W, slots, first, counts, lists_host);
    return cudaGetLastError();
}

}  // namespace knp_gb300
