// Device code that scatters a step's spikes as one list of synapses per CTA, shared by the fused step kernel
// (small_net.cu) and the persistent grid step kernel (grid_net.cu).
#pragma once

#include <cstdint>

#include "kernels.h"
#include "population_dev.cuh"
#include "projection_dev.cuh"

namespace knp_gb300
{
namespace
{

constexpr uint32_t kSourcesAtATime = 32;  // one warp resolves and scans them
constexpr uint32_t kLongRow = 1u << 20;   // rows above it are walked one by one (32-bit list positions)

// A step's projections: the spikes of all sources, then the synapses of the CTA's share of their rows as one
// list over the CTA's threads.
template <int kThreads>
struct ScatterTables
{
    static constexpr uint32_t kRows = kThreads;  // rows of a CTA's list at a time, one a thread
    static constexpr uint32_t kHead = kRows / 32;
    const uint32_t *idx[kSourcesAtATime];  // a source's spikes of this step
    uint32_t count[kSourcesAtATime];
    uint32_t first[kSourcesAtATime + 1];  // its first row among all sources' rows
    // The listed rows (those with synapses), in order.
    long long shift[kRows];          // CSR position of a row's synapse = shift + position in the list
    uint32_t start[kRows + 64];      // list position of a row's first synapse; above all past the last row
    uint32_t head[32];  // start[] of every kHead-th row
    uint2 place[kRows];              // its projection, and that one's ring slot of this step
    uint2 warp_total[kThreads / 32];  // a warp's rows' synapses, and its listed rows
    long long long_row;  // synapses of the long row being walked
};

struct Synapse
{
    int32_t col;
    float w;
    uint32_t delay;
    int type;
};
__device__ __forceinline__ Synapse load_synapse(const ProjectionDev &p, long long e)
{
    return {__ldg(p.col + e), p.w[e], __ldg(p.delay + e), p.type ? __ldg(p.type + e) : p.uniform_type};
}
__device__ __forceinline__ void deliver_synapse(const ProjectionDev &p, uint32_t slot, long long e, const Synapse &y)
{
    if (p.ring.fixed)
        deliver<true, false>(p, slot, e, y.col, y.w, y.delay, y.type);
    else
        deliver<false, false>(p, slot, e, y.col, y.w, y.delay, y.type);
}

// The projections of step t: this is CTA `rank` of C. Every thread of the CTA calls it (it contains block
// barriers). tab.idx / tab.count of the first kSourcesAtATime sources that are channels are filled already.
// listed_of(projection, spikes of one of its sources) is how many of them the list takes. kAtHand: what the plain
// case of the adds needs is read with the synapses, not field by field between the adds (6.6 us a step against 6.9
// for the network below); it takes registers.
// Returns (in thread 0) the synapses of the CTA's rows.
//
// A step of a small network is a few hundred rows of about a hundred synapses: a chain of trips to L2 (spike
// list, row bounds, synapses, adds), whose length is what the step takes. So the trips are made once for the
// rows of all projections together, a row a thread, and the synapses once, kInFlight a thread, whatever the
// rows' lengths. (A warp a row, projection after projection, went through the chain 4 to 6 times: 25200 cycles
// a step on 8 CTAs, against 13000, and 8500 on 16, for 1000 neurons with 260 rows of 100.) The whole step of that
// network went from 16.5 us to 6.6, one with 784 inputs, 800 neurons and additive STDP from 13 to 6.8.
//
// In a large one (10^6 neurons with 1000 synapses, 5000 of them firing) the adds are most of the time, 5 10^6 of them
// in 56 us with the rest; what the list gives is that every warp has as many. (A warp for a third of a row: 68.5 us
// for the phase. With rows of 100, 18.7 us against 35.) Its loads want L1 to be in flight: see where the gather's
// shared memory is sized.
template <int kThreads, int kInFlight, bool kAtHand, bool kLongLists, typename Listed>
__device__ __forceinline__ unsigned long long project_rows(const ProjectionDev *projs, const SmallSource *sources,
                                                           uint32_t n_sources, unsigned long long t, uint32_t rank,
                                                           uint32_t C, ScatterTables<kThreads> &tab, Listed listed_of)
{
    constexpr uint32_t kRowsAtATime = ScatterTables<kThreads>::kRows, kHead = ScatterTables<kThreads>::kHead;
    constexpr uint32_t kWarps = kThreads / 32;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long events = 0;
    for (uint32_t b0 = 0; b0 < n_sources; b0 += kSourcesAtATime)
    {
        const uint32_t n = min(kSourcesAtATime, n_sources - b0);
        if (warp == 0)
        {
            uint32_t cnt = 0;
            if (lane < n)
            {
                const SpikeSource &src = sources[b0 + lane].src;
                if (b0 > 0 || !src.channel)
                    resolve_source(src, t, tab.idx[lane], cnt);
                else
                    cnt = tab.count[lane];
                cnt = listed_of(projs[sources[b0 + lane].proj], cnt);
            }
            uint32_t run = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const uint32_t v = __shfl_up_sync(0xffffffffu, run, o);
                if (lane >= static_cast<uint32_t>(o)) run += v;
            }
            tab.first[lane] = run - cnt;
            if (lane == 31) tab.first[kSourcesAtATime] = run;
        }
        __syncthreads();
        // Rows are dealt to the CTAs in turn; a few, cut into 2^cut parts each, so that every CTA gets some (ten rows
        // of 10^5 synapses: 18.8 us a step on 152 CTAs, 89 uncut, 174 as up to eight warps a row).
        const uint32_t rows_all = tab.first[kSourcesAtATime];
        uint32_t cut = 0;
        while (cut < 6 && rows_all <= 4 * C >> cut) ++cut;
        const uint32_t total = rows_all << cut;
        for (uint32_t r0 = rank; r0 < total; r0 += C * kRowsAtATime)
        {
            const uint32_t i = r0 + C * tid, j = i >> cut, part = i & ((1u << cut) - 1u);
            long long a = 0;
            long long len = 0;
            uint32_t pj = 0, slot0 = 0;
            if (i < total)
            {
                uint32_t k = 0;
                while (j >= tab.first[k + 1]) ++k;
                pj = sources[b0 + k].proj;
                const ProjectionDev &p = projs[pj];
                const uint32_t pre = tab.idx[k][j - tab.first[k]];
                slot0 = step_slot(t, p.ring.slots);
                if (pre < p.n_rows)
                {
                    a = p.row_ptr[pre];
                    len = p.row_ptr[pre + 1] - a;
                    const long long from = len * part >> cut;
                    len = (len * (part + 1) >> cut) - from;
                    a += from;
                }
            }
            const bool is_long = len > static_cast<long long>(kLongRow);
            const uint32_t listed = is_long ? 0u : static_cast<uint32_t>(len);
            const uint32_t rows = __ballot_sync(0xffffffffu, listed != 0);
            uint32_t run = listed;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const uint32_t v = __shfl_up_sync(0xffffffffu, run, o);
                if (lane >= static_cast<uint32_t>(o)) run += v;
            }
            if (lane == 31) tab.warp_total[warp] = make_uint2(run, __popc(rows));
            const bool any_long = __syncthreads_or(is_long);
            uint32_t before = 0, all = 0, r = 0, n_rows = 0;
#pragma unroll
            for (uint32_t w = 0; w < kWarps; ++w)
            {
                const uint2 x = tab.warp_total[w];
                if (w < warp) before += x.x, r += x.y;
                all += x.x;
                n_rows += x.y;
            }
            r += __popc(rows & ((1u << lane) - 1u));
            if (listed)
            {
                const uint32_t start = before + run - listed;
                tab.start[r] = start;
                tab.shift[r] = a - start;
                tab.place[r] = make_uint2(pj, slot0);
                if (r % kHead == 0) tab.head[r / kHead] = start;
            }
            // The rows past the last start above every position of the list.
            for (uint32_t i = n_rows + tid; i < kRowsAtATime + 64; i += kThreads)
            {
                tab.start[i] = 0xFFFFFFFFu;
                if (i % kHead == 0 && i < kRowsAtATime) tab.head[i / kHead] = 0xFFFFFFFFu;
            }
            __syncthreads();
            if (tid == 0) events += all;
            // The row of position e (the same in the warp's lanes), by the lanes together: every kHead-th row, then its
            // kHead. (A search by each lane met itself in the banks: 3700 cycles against 2400 for 1450 synapses a CTA.)
            auto row_at = [&](uint32_t e) -> uint32_t
            {
                const uint32_t h = kHead * (__popc(__ballot_sync(0xffffffffu, tab.head[lane] <= e)) - 1);
                return h + __popc(__ballot_sync(0xffffffffu, lane < kHead && tab.start[h + lane] <= e)) - 1;
            };
            // The row of position e + lane: the rows that start within the warp's 32 positions, as bits.
            auto row_of_lane = [&](uint32_t e, uint32_t r0) -> uint32_t
            {
                const uint32_t ahead = tab.start[r0 + 1 + lane] - e;
                const uint32_t starts = __reduce_or_sync(0xffffffffu, ahead < 32 ? 1u << ahead : 0u);
                return r0 + __popc(starts & (0xFFFFFFFFu >> (31 - lane)));
            };
            // Long lists: a warp takes kRun positions in a row, mostly of one row (rows of 1000: 7 in 8 are), whose
            // projection and bounds are then the same in all lanes. It is a third fewer instructions, which is what
            // counts where the adds are of neighbouring targets (459 10^6 synapses all to all, 1.2 10^5 a CTA and
            // step: 18.9 ms for 200 steps against 25.0); with random targets, 3.3 10^4 a CTA, the adds count and
            // come better spread from 32 positions at a time (56.7 us against 63).
            constexpr uint32_t kRun = 128, kLongList = 1u << 16;
            const uint32_t by_runs = kLongLists && all >= kLongList ? all - all % (kRun * kWarps) : 0u;
            for (uint32_t e0 = kRun * warp; kLongLists && e0 < by_runs; e0 += kRun * kWarps)
            {
                const uint32_t r0 = row_at(e0);
                const uint2 at = tab.place[r0];
                const ProjectionDev &p = projs[at.x];
                if (min(tab.start[r0 + 1], all) >= e0 + kRun && !p.type && p.uniform_type == 0 && !p.ring.fixed &&
                    !(p.forcing && p.ring.forced))
                {
                    const long long e = tab.shift[r0] + e0 + lane;
                    const int32_t *col = p.col + e;
                    const float *w = p.w + e;
                    const uint8_t *delay = p.delay + e;
                    const uint32_t n_slots = p.ring.slots, pitch = p.ring.pitch;
                    float *ring = p.ring.v32;
                    int32_t c[4];
                    float x[4];
                    uint32_t d[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                    {
                        c[u] = __ldg(col + 32 * u);
                        x[u] = w[32 * u];
                        d[u] = __ldg(delay + 32 * u);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                    {
                        if (d[u] == 0u) continue;  // lost, as in deliver()
                        uint32_t to = at.y + d[u];
                        while (to >= n_slots) to -= n_slots;
                        atomicAdd(ring + static_cast<size_t>(to) * pitch + static_cast<uint32_t>(c[u]), x[u]);
                    }
                    continue;
                }
                for (uint32_t e = e0; e < e0 + kRun; e += 32)
                {
                    const uint32_t r = row_of_lane(e, row_at(e));
                    const uint2 mine = tab.place[r];
                    const long long k = tab.shift[r] + e + lane;
                    deliver_synapse(projs[mine.x], mine.y, k, load_synapse(projs[mine.x], k));
                }
            }
            for (uint32_t e0 = by_runs + tid - lane; e0 < all; e0 += kInFlight * kThreads)
            {
                Synapse y[kInFlight];
                uint32_t row[kInFlight], slot[kInFlight], n_slots[kInFlight], pitch[kInFlight];
                float *ring[kInFlight];
#pragma unroll
                for (int u = 0; u < kInFlight; ++u)
                {
                    const uint32_t e = e0 + u * kThreads;
                    row[u] = row_of_lane(e, row_at(e));
                }
#pragma unroll
                for (int u = 0; u < kInFlight; ++u)
                {
                    const uint32_t e = e0 + lane + u * kThreads;
                    if (e >= all) continue;
                    const uint2 at = tab.place[row[u]];
                    const ProjectionDev &p = projs[at.x];
                    y[u] = load_synapse(p, tab.shift[row[u]] + e);
                    if (!kAtHand) continue;
                    slot[u] = at.y;
                    n_slots[u] = p.ring.slots;
                    pitch[u] = p.ring.pitch;
                    ring[u] = p.ring.fixed || (p.forcing && p.ring.forced) ? nullptr : p.ring.v32;
                }
#pragma unroll
                for (int u = 0; u < kInFlight; ++u)
                {
                    const uint32_t e = e0 + lane + u * kThreads;
                    if (e >= all) continue;
                    if (!kAtHand || !ring[u] || static_cast<uint32_t>(y[u].type) > 1u)
                    {
                        const uint2 at = tab.place[row[u]];
                        deliver_synapse(projs[at.x], at.y, tab.shift[row[u]] + e, y[u]);
                        continue;
                    }
                    // The plain case of deliver(), with what it needs at hand.
                    if (y[u].delay == 0u) continue;
                    uint32_t to = slot[u] + y[u].delay;
                    while (to >= n_slots[u]) to -= n_slots[u];
                    atomicAdd(ring[u] + static_cast<size_t>(to) * pitch[u] + static_cast<uint32_t>(y[u].col),
                              y[u].type == 1 ? -y[u].w : y[u].w);
                }
            }
            if (any_long)
            {
                // One row after another, its bounds from the thread that has them.
                for (uint32_t i = 0; i < kRowsAtATime; ++i)
                {
                    const bool mine = tid == i && is_long;
                    __syncthreads();
                    if (mine)
                    {
                        tab.shift[0] = a;
                        tab.place[0] = make_uint2(pj, slot0);
                        tab.long_row = len;
                    }
                    if (!__syncthreads_or(mine)) continue;
                    const long long n_e = tab.long_row;
                    const uint2 at = tab.place[0];
                    const ProjectionDev &p = projs[at.x];
                    for (long long e = tab.shift[0] + tid; e < tab.shift[0] + n_e; e += kThreads)
                        deliver_synapse(p, at.y, e, load_synapse(p, e));
                    if (tid == 0) events += n_e;
                }
            }
            __syncthreads();  // the tables are used again
        }
        __syncthreads();
    }
    return events;
}

}  // namespace
}  // namespace knp_gb300
