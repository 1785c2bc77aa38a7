// Device code of the gather ("pull") form of a delta projection, shared by the per-step gather
// kernel (pull.cu) and the persistent grid step kernel (grid_net.cu).
//
// For the step tn whose input it completes, a block walks, for every delay d whose step tn - d was
// recorded in the projection's spike bitmap, the slices of its range of 256-target windows in the
// sliced ELL layout of kernels.h: each lane owns one target of a slice and sums, down its list, the
// weights of the synapses whose presynaptic bit is set (bitmap staged in shared memory), then adds
// the sum to the target's accumulator; the accumulators are added once to the targets' input-ring
// slot of step tn. The sums are the impacts the scatter would have delivered at step tn (delay
// convention of delta_impl.h:78-79 of the reference CPU library), added in another order, which is
// exact for the FP32 ring (dyadic weights); populations with the fixed-point ring never use this form.
#pragma once

#include <cstdint>
#include <type_traits>

#include <cuda_fp16.h>

#include "kernels.h"

namespace knp_gb300
{
namespace
{

constexpr int kGatherThreads = 1024;
constexpr int kDepth = 16;  // list entries per lane in flight

// Hint: bring [p, p + bytes) into L2 (16-byte aligned address and size; no completion to wait for).
__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// Slices ahead of the one a warp takes whose entries it asks L2 to fetch: by the time a warp takes
// that slice its loads hit L2 instead of DRAM (full-size step: 8 and 16 give 0.80 ms, 32 0.81 ms,
// 64 0.84 ms).
constexpr uint32_t kPrefetchAhead = 16;

enum WeightForm
{
    kDict = 0,     // 8-bit dictionary index in the top bits of the packed entry
    kHalf = 1,     // FP16
    kFull = 2,     // FP32
    kDictRep = 3,  // as kDict, with 32 copies of the dictionary in shared memory (PullDev::tab_rep)
};


// The gather's work is cut over G blocks in units of (window, delay), window-major: block `block` takes units
// [u0, u1), so that the blocks' shares are equal to within one unit, and for each delay a run of windows that
// differs by one at either end at most. (Without split_delays: whole windows.) A window cut between two
// blocks is summed by both.
struct GatherShare
{
    uint32_t u0, u1, q0, r0, q1, r1;  // u = q D + r
    GatherShare() = default;
    __host__ __device__ GatherShare(const PullDev &p, uint32_t block, uint32_t G)
    {
        const uint32_t D = p.split_delays ? p.max_delay : 1u;
        u0 = static_cast<uint32_t>(static_cast<uint64_t>(block) * p.n_windows * D / G);
        u1 = static_cast<uint32_t>(static_cast<uint64_t>(block + 1) * p.n_windows * D / G);
        q0 = u0 / D;
        r0 = u0 % D;
        q1 = u1 / D;
        r1 = u1 % D;
    }
    // The block's windows of delay d (1 ..): [first(d), last(d)); unit (w, d) is w D + d - 1. Whole windows have
    // r = 0. Of all delays: [q0, end()).
    __device__ uint32_t first(uint32_t d) const { return q0 + (r0 >= d ? 1u : 0u); }
    __device__ uint32_t last(uint32_t d) const { return q1 + (r1 >= d ? 1u : 0u); }
    __device__ uint32_t end() const { return q1 + (r1 ? 1u : 0u); }
};

// Largest number of windows that a block's share touches.
__host__ __device__ inline uint32_t gather_windows(const PullDev &p, uint32_t G)
{
    return (p.n_windows + G - 1) / G + (p.split_delays ? 1u : 0u);
}

// Shared memory of one gather block: the spike bitmaps of n_bm steps, the accumulators of the block's
// windows and (dictionary weights) 32 replicas of the dictionary.
__host__ __device__ inline size_t gather_smem_for(const PullDev &p, uint32_t G)
{
    return static_cast<size_t>(p.n_bm) * p.words * 4 + static_cast<size_t>(gather_windows(p, G)) * kPullWindow * 4 +
           (p.tab_rep ? static_cast<size_t>(p.n_tab) * 32 * 4 : 0);
}

// Whether the gather of step tn has work: some delay d in 1..max_delay whose step tn - d was pulled.
__device__ __forceinline__ bool gather_needed(const PullDev &g, unsigned long long tn)
{
    for (uint32_t d = 1; d <= g.max_delay && d <= tn; ++d)
        if (g.pulled[static_cast<uint32_t>((tn - d) % g.hist_slots)]) return true;
    return false;
}

// Clears block `block`'s share (of G) of the bitmap slot that the scatter kernel of step tn will
// fill; it holds step tn - hist_slots, which no gather reads any more.
__device__ __forceinline__ void clear_bitmap_slot(const PullDev &g, unsigned long long tn, uint32_t block, uint32_t G)
{
    const uint32_t sl_next = static_cast<uint32_t>(tn % g.hist_slots);
    uint32_t *dst = g.bitmap + static_cast<size_t>(sl_next) * g.words;
    const uint32_t b0 = static_cast<uint32_t>(static_cast<uint64_t>(block) * g.words / G);
    const uint32_t b1 = static_cast<uint32_t>(static_cast<uint64_t>(block + 1) * g.words / G);
    for (uint32_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) dst[i] = 0u;
}

// Static shared memory of a gather block (one copy, whichever weight form runs).
struct GatherTables
{
    // The descriptor: the gather's loops write memory, so the compiler reads the fields they use again for every
    // slice. (From a descriptor in global memory, as the whole-step kernel has it, 226 us a step against 218 for
    // 200k neurons of which a third fire, and 710 against 699 for 10^6 that all fire.)
    alignas(16) uint32_t desc[sizeof(PullDev) / 4];
    GatherShare share;
    uint8_t pflag[256];  // pulled flag of step tn - d, d = 1 .. max_delay (max_delay <= 255)
    // The group's delays, its slices before each, and the first window of each; their number; the first pulled
    // delay after them, its first slice of this block in the layout (of the delay) and its number of them. (One thread's work: in every thread's registers it made the slices' loop spill, 237 us
    // against 218 and 720 against 676.)
    uint32_t delay[kGatherBitmaps], before[kGatherBitmaps + 1], window[kGatherBitmaps];
    uint32_t n_group, delay_next, q_next, slices_next;
    uint32_t next;  // next slice of the current group to hand out
};
static_assert(sizeof(GatherTables) + 256 * sizeof(float) <= kGatherStaticSmem, "reserved beside the dynamic part");
static_assert(sizeof(PullDev) % 4 == 0, "copied by words");

__device__ __forceinline__ GatherTables &gather_tables()
{
    __shared__ GatherTables tables;
    return tables;
}

// Block `block` of G gather blocks completes the input of step tn (every thread of the block calls
// it; it contains block barriers), and clears its share of the bitmap slot that step tn's spikes
// will be recorded in. smem_u4: gather_smem_for(p.pull, G) bytes of dynamic shared memory.
//
// The delays are walked in groups of n_bm, whose bitmaps are in shared memory together: the slices of a group
// are handed out from one pool, so that the block's 32 warps wait for one another once per group. (One
// delay at a time, a block of 200k neurons' gather had 48 slices a delay for 32 warps, half a round of idle
// warps at each of 20 barriers, and 5 or 6 whole windows a block: 271 us a step at a third of the neurons
// firing, against 218 us. Loading the next round's entries during the current one gave 226 us at 8 entries
// a round and 253 at 16, 64 registers being too few for both.)
template <int kForm>
__device__ __forceinline__ void gather_block(const ProjectionDev &p, unsigned long long tn, uint32_t block, uint32_t G,
                                             uint4 *smem_u4)
{
    __shared__ float s_dict[256];  // kDict only
    GatherTables &tab = gather_tables();
    for (uint32_t i = threadIdx.x; i < sizeof(PullDev) / 4; i += blockDim.x)
        tab.desc[i] = reinterpret_cast<const uint32_t *>(&p.pull)[i];
    __syncthreads();
    const PullDev &g = *reinterpret_cast<const PullDev *>(tab.desc);
    uint32_t *bm0 = reinterpret_cast<uint32_t *>(smem_u4);
    float *acc = reinterpret_cast<float *>(bm0 + static_cast<size_t>(g.n_bm) * g.words);
    float *rep = acc + static_cast<size_t>(gather_windows(g, G)) * kPullWindow;  // after the largest acc
    if (kForm == kDictRep)
        for (uint32_t i = threadIdx.x; i < g.n_tab * 32u; i += blockDim.x) rep[i] = g.wtab[i >> 5];
    if (kForm == kDict)
        for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) s_dict[i] = g.wtab[i];
    if (threadIdx.x == 0)
    {
        tab.share = GatherShare(g, block, G);
        tab.delay_next = 1;
    }
    const int lane = threadIdx.x & 31;
    for (uint32_t d = 1 + threadIdx.x; d <= g.max_delay; d += blockDim.x)
        tab.pflag[d] = d <= tn ? static_cast<uint8_t>(g.pulled[static_cast<uint32_t>((tn - d) % g.hist_slots)]) : 0;
    __syncthreads();
    const uint32_t w0 = tab.share.q0;
    const uint32_t n_acc = tab.share.u1 > tab.share.u0 ? (tab.share.end() - w0) * kPullWindow : 0u;
    for (uint32_t i = threadIdx.x; i < n_acc; i += blockDim.x) acc[i] = 0.0f;

    bool any = false;
    while (n_acc)
    {
        __syncthreads();  // the previous group's bitmaps and tables are no longer read
        if (threadIdx.x == 0)
        {
            // The next n_bm delays whose step was pulled.
            const GatherShare share = tab.share;
            uint32_t n = 0, before = 0, d = tab.delay_next;
            for (; d <= g.max_delay && n < g.n_bm; ++d)
            {
                if (!tab.pflag[d]) continue;
                tab.delay[n] = d;
                tab.window[n] = share.first(d);
                tab.before[n] = before;
                before += (share.last(d) - share.first(d)) * kPullSlicesPerWindow;
                ++n;
            }
            tab.before[n] = before;
            while (d <= g.max_delay && !tab.pflag[d]) ++d;
            tab.delay_next = d;
            tab.q_next = share.first(d) * kPullSlicesPerWindow;
            tab.slices_next = d <= g.max_delay ? (share.last(d) - share.first(d)) * kPullSlicesPerWindow : 0u;
            tab.n_group = n;
            tab.next = 0;
        }
        __syncthreads();
        const uint32_t n_in = tab.n_group;
        if (!n_in) break;
        any = true;
        for (uint32_t k = 0; k < n_in; ++k)
        {
            const uint32_t d = tab.delay[k];
            if (tab.pflag[d] == 2u) continue;  // every presynaptic neuron fired: no bitmap needed
            const uint32_t sl = static_cast<uint32_t>((tn - d) % g.hist_slots);
            const uint4 *src = reinterpret_cast<const uint4 *>(g.bitmap + static_cast<size_t>(sl) * g.words);
            uint4 *dst = smem_u4 + static_cast<size_t>(k) * (g.words / 4);
            for (uint32_t i = threadIdx.x; i < g.words / 4; i += blockDim.x) dst[i] = src[i];
        }
        __syncthreads();
        const uint32_t n_q = tab.before[n_in];
        // Index in the layout of slice qi of the group, which is one of its k-th delay's.
        auto slice_at = [&](uint32_t qi, uint32_t k) -> size_t
        {
            return (static_cast<size_t>(tab.delay[k] - 1) * g.n_windows + tab.window[k]) * kPullSlicesPerWindow +
                   (qi - tab.before[k]);
        };
        // The delay of this warp's slice (slices are handed out in order), kept in registers until it changes:
        // its place in the group, its slices in the pool, its first slice in the layout, its first window's
        // accumulators and its bitmap.
        uint32_t in_group = 0, before = 0, end = 0;
        size_t q_first = 0;
        float *acc_first = acc;
        const uint32_t *bm = bm0;
        bool all = false;
        // Slices are handed out one at a time (lists differ in length: longest first within a window).
        for (;;)
        {
            uint32_t qi = 0;
            if (lane == 0) qi = atomicAdd(&tab.next, 1u);
            qi = __shfl_sync(0xffffffffu, qi, 0);
            if (qi >= n_q) break;
            if (qi >= end)
            {
                while (qi >= tab.before[in_group + 1]) ++in_group;
                before = tab.before[in_group];
                end = tab.before[in_group + 1];
                q_first = slice_at(before, in_group);
                acc_first = acc + static_cast<size_t>(tab.window[in_group] - w0) * kPullWindow;
                bm = bm0 + static_cast<size_t>(in_group) * g.words;
                all = tab.pflag[tab.delay[in_group]] == 2u;
            }
            const size_t q = q_first + (qi - before);
            if (lane == 0)
            {
                // Ask L2 for the slice kPrefetchAhead further on; at the end of the group, for the first
                // ones of the next pulled delay.
                const uint32_t ahead = qi + kPrefetchAhead;
                size_t qa = q + kPrefetchAhead;
                bool ask = ahead < end;
                if (!ask)
                {
                    if (ahead < n_q)
                    {
                        uint32_t k = in_group + 1;
                        while (ahead >= tab.before[k + 1]) ++k;
                        qa = slice_at(ahead, k);
                        ask = true;
                    }
                    else if (ahead - n_q < tab.slices_next)
                    {
                        qa = static_cast<size_t>(tab.delay_next - 1) * g.n_windows * kPullSlicesPerWindow + tab.q_next +
                             (ahead - n_q);
                        ask = true;
                    }
                }
                const uint32_t la = ask ? g.slice_len[qa] : 0u;
                if (la)
                {
                    // Slices start on 32-entry boundaries; one slice is len x 32 entries.
                    prefetch_l2(g.packed + g.slice_ptr[qa], la * kPullSlice * 4u);
                    if (kForm == kHalf) prefetch_l2(g.w16 + g.slice_ptr[qa], la * kPullSlice * 2u);
                    if (kForm == kFull) prefetch_l2(g.w + g.slice_ptr[qa], la * kPullSlice * 4u);
                }
            }
            const uint32_t len = g.slice_len[q];
            if (len == 0) continue;
            // Entry k of this lane's list is at slice_ptr + 32 k + lane (a warp load reads 128
            // consecutive bytes).
            const long long off = g.slice_ptr[q] + lane;
            const uint32_t *pk = g.packed + off;
            const uint16_t *ph = kForm == kHalf ? g.w16 + off : nullptr;
            const float *pf = kForm == kFull ? g.w + off : nullptr;
            const float *rep_lane = rep + lane;
            // This lane's target, read before the walk (after it, one more trip to memory in turn: 748 us for 10^6
            // that all fire, against 699). Where the group has several delays, another warp may hold it for another of
            // them (the sums are exact in any order).
            float *mine = acc_first + (qi - before) / kPullSlicesPerWindow * kPullWindow + g.perm[q * kPullSlice + lane];
            // Two copies of the walk: with the bit test, and without it for a step in which every
            // presynaptic neuron fired (the test would always pass).
            auto walk = [&](auto all_tag) -> float
            {
                constexpr bool kAll = decltype(all_tag)::value;
                float sum = 0.0f;
                // One entry: its weight, and (the shift takes its amount modulo 32) its presynaptic bit.
                auto take = [&](uint32_t pn, float wi)
                {
                    if (kForm == kDictRep) wi = rep_lane[(pn >> 24) * 32u];
                    if (kForm == kDict) wi = s_dict[pn >> 24];
                    if (kAll)
                        sum = __fadd_rn(sum, wi);
                    else if (__funnelshift_r(bm[(pn >> 5) & 0x7FFFFu], 0u, pn) & 1u)
                        sum = __fadd_rn(sum, wi);
                };
                // Entries k0 .. k0 + kN - 1 in one round of loads; kTail leaves out those past the list's end.
                auto round = [&](auto n_tag, auto tail_tag, uint32_t k0)
                {
                    constexpr int kN = decltype(n_tag)::value;
                    constexpr bool kTail = decltype(tail_tag)::value;
                    const size_t o = static_cast<size_t>(k0) * kPullSlice;
                    uint32_t pre[kN];
                    float w[kN];
#pragma unroll
                    for (int i = 0; i < kN; ++i)
                    {
                        pre[i] = 0u;
                        w[i] = 0.0f;
                        if (kTail && k0 + i >= len) continue;
                        pre[i] = __ldcs(pk + o + i * kPullSlice);
                        if (kForm == kHalf) w[i] = __half2float(__ushort_as_half(__ldcs(ph + o + i * kPullSlice)));
                        if (kForm == kFull) w[i] = __ldcs(pf + o + i * kPullSlice);
                    }
#pragma unroll
                    for (int i = 0; i < kN; ++i)
                        if (!kTail || k0 + i < len) take(pre[i], w[i]);
                };
                // Rounds of kDepth, then the rest in one more round of about its size (len is the same in every
                // lane): lists of about 10 are one trip to memory, and 50 pay for 2 entries at the end, not 16.
                uint32_t k0 = 0;
                for (; k0 + kDepth <= len; k0 += kDepth)
                    round(std::integral_constant<int, kDepth>{}, std::false_type{}, k0);
                const uint32_t rest = len - k0;
                if (rest > 8u)
                    round(std::integral_constant<int, kDepth>{}, std::true_type{}, k0);
                else if (rest > 4u)
                    round(std::integral_constant<int, 8>{}, std::true_type{}, k0);
                else if (rest)
                    round(std::integral_constant<int, 4>{}, std::true_type{}, k0);
                return sum;
            };
            const float sum = all ? walk(std::true_type{}) : walk(std::false_type{});
            if (sum != 0.0f)
            {
                if (g.n_bm == 1u)
                    *mine += sum;
                else
                    atomicAdd(mine, sum);
            }
        }
    }
    __syncthreads();
    if (any)
    {
        const uint32_t slot = static_cast<uint32_t>(tn % p.ring.slots);
        float *ring = p.ring.v32 + static_cast<size_t>(slot) * p.ring.pitch;
        for (uint32_t i = threadIdx.x; i < n_acc; i += blockDim.x)
        {
            const uint32_t j = w0 * kPullWindow + i;
            // The window may be another block's too: of this projection where delays are split, or of another
            // projection into the same population, whose gather the grid kernel runs without waiting for this one.
            if (j < g.n_post && acc[i] != 0.0f) atomicAdd(ring + j, acc[i]);
        }
    }
    clear_bitmap_slot(g, tn, block, G);
}

}  // namespace
}  // namespace knp_gb300
