// Fused step kernel for small networks: one thread-block cluster runs whole steps of every
// population, projection and STDP rule of a backend, `n_steps` steps per launch, with the phases of
// a step separated by cluster barriers instead of kernel boundaries.
//
// A step of the per-phase path is five to six dependent launches (population, scatter per
// projection, STDP append and modify, end of step); below ~10^4 neurons each phase is a few
// microseconds of latency and the launches, not the work, set the step time. Here a step is two
// phases inside one cluster of up to 16 CTAs on 16 SMs (the adds into the input ring leave an SM at a
// lane or so a cycle: 1000 neurons with 260 rows of 100 a step take 8.1 us on 16, 9.7 on 8): the populations of step t beside the STDP rules of step t - 1,
// then the projections of step t. That keeps the order of the single-threaded backend's step
// (backend.cpp:89-141 of the reference: populations, projections, then the STDP rules, whose
// weights the next step's projections read) for every datum, and no wait spins: every ordering is a
// hardware cluster barrier (barrier.cluster arrive.release / wait.acquire, which also orders the
// CTAs' global-memory accesses) or a block barrier.
//
// The per-neuron, per-synapse and per-column code is the per-phase kernels' own (population_dev.cuh,
// projection_dev.cuh, stdp_dev.cuh), and the cluster walks the same device layout, so results are
// those of the per-phase path. Only projections without a gather layout take part (the host selects
// this kernel only then).
#include <cstdint>

#include "kernels.h"
#include "population_dev.cuh"
#include "projection_dev.cuh"
#include "stdp_dev.cuh"
#include "tcgen05.cuh"

namespace knp_gb300
{
namespace
{

constexpr int kSmallThreads = 512;
constexpr uint32_t kSmallWarps = kSmallThreads / 32;

constexpr uint32_t kSourcesAtATime = 32;        // one warp resolves and scans them
constexpr uint32_t kRowsAtATime = kSmallThreads;  // rows of a CTA's list, one a thread
constexpr uint32_t kLongRow = 1u << 20;          // rows above it are walked one by one (32-bit list positions)
constexpr int kInFlight = 3;                     // synapses a thread loads at a time

// A step's projections: the spikes of all sources, then the synapses of the CTA's share of their rows as one
// list over the CTA's threads.
struct ScatterTables
{
    const uint32_t *idx[kSourcesAtATime];   // a source's spikes of this step
    uint32_t count[kSourcesAtATime];
    uint32_t first[kSourcesAtATime + 1];    // its first row among all sources' rows
    // The listed rows (those with synapses), in order.
    long long shift[kRowsAtATime];          // CSR position of a row's synapse = shift + position in the list
    uint32_t start[kRowsAtATime + 64];      // list position of a row's first synapse; above all past the last row
    uint32_t head[32];                      // start[] of every 16th row
    uint2 place[kRowsAtATime];              // its projection, and that one's ring slot of this step
    uint2 warp_total[kSmallWarps];          // a warp's rows' synapses, and its listed rows
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
// Returns (in thread 0) the synapses of the CTA's rows.
//
// A step of a small network is a few hundred rows of about a hundred synapses: a chain of trips to L2 (spike
// list, row bounds, synapses, adds), whose length is what the step takes. So the trips are made once for the
// rows of all projections together, a row a thread, and the synapses once, kInFlight a thread, whatever the
// rows' lengths. (A warp a row, projection after projection, went through the chain 4 to 6 times: 25200 cycles
// a step on 8 CTAs, against 13000, and 8500 on 16, for 1000 neurons with 260 rows of 100.) The whole step of that
// network went from 16.5 us to 6.6, one with 784 inputs, 800 neurons and additive STDP from 13 to 6.8.
__device__ __forceinline__ unsigned long long project_rows(const SmallNet &net, const ProjectionDev *projs,
                                                           const SmallSource *sources, unsigned long long t,
                                                           uint32_t rank, uint32_t C, ScatterTables &tab)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long events = 0;
    for (uint32_t b0 = 0; b0 < net.n_sources; b0 += kSourcesAtATime)
    {
        const uint32_t n = min(kSourcesAtATime, net.n_sources - b0);
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
        // Rows are dealt to the CTAs in turn.
        const uint32_t total = tab.first[kSourcesAtATime];
        for (uint32_t r0 = rank; r0 < total; r0 += C * kRowsAtATime)
        {
            const uint32_t j = r0 + C * tid;
            long long a = 0;
            long long len = 0;
            uint32_t pj = 0, slot0 = 0;
            if (j < total)
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
            for (uint32_t w = 0; w < kSmallWarps; ++w)
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
                if (r % 16 == 0) tab.head[r / 16] = start;
            }
            // The rows past the last start above every position of the list.
            for (uint32_t i = n_rows + tid; i < kRowsAtATime + 64; i += kSmallThreads)
            {
                tab.start[i] = 0xFFFFFFFFu;
                if (i % 16 == 0 && i < kRowsAtATime) tab.head[i / 16] = 0xFFFFFFFFu;
            }
            __syncthreads();
            if (tid == 0) events += all;
            for (uint32_t e0 = tid - lane; e0 < all; e0 += kInFlight * kSmallThreads)
            {
                Synapse y[kInFlight];
                uint32_t row[kInFlight], slot[kInFlight], n_slots[kInFlight], pitch[kInFlight];
                float *ring[kInFlight];
#pragma unroll
                for (int u = 0; u < kInFlight; ++u)
                {
                    // The row of the warp's first position, by its lanes together (every 16th row, then the 16);
                    // then the rows that start within the warp's 32 positions, as bits. (A search by each lane
                    // met itself in the banks: 3700 cycles against 2400 for 1450 synapses a CTA.)
                    const uint32_t e = e0 + u * kSmallThreads;
                    const uint32_t h = 16 * (__popc(__ballot_sync(0xffffffffu, tab.head[lane] <= e)) - 1);
                    const uint32_t r0 =
                        h + __popc(__ballot_sync(0xffffffffu, lane < 16 && tab.start[h + lane] <= e)) - 1;
                    const uint32_t ahead = tab.start[r0 + 1 + lane] - e;
                    const uint32_t starts = __reduce_or_sync(0xffffffffu, ahead < 32 ? 1u << ahead : 0u);
                    row[u] = r0 + __popc(starts & (0xFFFFFFFFu >> (31 - lane)));
                }
#pragma unroll
                for (int u = 0; u < kInFlight; ++u)
                {
                    const uint32_t e = e0 + lane + u * kSmallThreads;
                    if (e >= all) continue;
                    const uint2 at = tab.place[row[u]];
                    const ProjectionDev &p = projs[at.x];
                    y[u] = load_synapse(p, tab.shift[row[u]] + e);
                    slot[u] = at.y;
                    n_slots[u] = p.ring.slots;
                    pitch[u] = p.ring.pitch;
                    ring[u] = p.ring.fixed || (p.forcing && p.ring.forced) ? nullptr : p.ring.v32;
                }
#pragma unroll
                for (int u = 0; u < kInFlight; ++u)
                {
                    const uint32_t e = e0 + lane + u * kSmallThreads;
                    if (e >= all) continue;
                    if (!ring[u] || static_cast<uint32_t>(y[u].type) > 1u)
                    {
                        deliver_synapse(projs[tab.place[row[u]].x], slot[u], tab.shift[row[u]] + e, y[u]);
                        continue;
                    }
                    // The plain case of deliver(), with what it needs at hand (read field by field between the
                    // adds it took longer than the synapses' trip).
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
                    for (long long e = tab.shift[0] + tid; e < tab.shift[0] + n_e; e += kSmallThreads)
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

// Lists and records a population's spikes: a warp's with one atomic if it has a neuron a lane, else a block's.
template <int kN, typename Pop>
__device__ __forceinline__ void emit(const Pop &p, uint32_t mask, uint32_t i0, unsigned long long t)
{
    uint32_t *rec = record_slot(p.rec_bits, p.rec_words, p.rec_slots, t);
    if (kN == 4)
        emit_spikes<kSmallThreads>(mask, i0, p.spikes, p.spike_count, rec, p.rec_words);
    else
        emit_warp(mask, i0, p.spikes, p.spike_count, rec, p.rec_words);
}

// One population's step t, kN neurons a thread: 1 while the cluster has a thread for every neuron (the chain of
// a neuron's operations is what the pass takes then: 5600 cycles against 11500 for 800 neurons with a fixed-point
// ring), else 4, for the wider loads and the fewer passes.
template <int kN>
__device__ __forceinline__ void step_population(const SmallPop &q, unsigned long long t, uint32_t gthread,
                                                uint32_t n_threads)
{
    if (q.kind == kSmallLif)
    {
        const LifDev &p = q.lif;
        for (uint32_t base = 0; base < p.n; base += kN * n_threads)
        {
            const uint32_t i0 = base + kN * gthread;
            emit<kN>(p, lif_quad<kN>(p, t, i0), i0, t);
        }
    }
    else
    {
        const BlifatDev &p = q.blifat;
        for (uint32_t base = 0; base < p.n; base += kN * n_threads)
        {
            const uint32_t i0 = base + kN * gthread;
            emit<kN>(p, blifat_quad_any<kN>(p, t, i0), i0, t);
        }
    }
}

// Reads (into the CTA's spike total) and zeroes the per-step counters of one descriptor set; one warp's work.
__device__ __forceinline__ void retire_counters(const StepEnd &e, uint32_t lane, unsigned long long *spikes)
{
    for (uint32_t k = lane; k < e.n_zero_u32; k += 32)
    {
        const uint32_t v = e.zero_u32[k];
        if (k < e.n_spike_counts && v) atomicAdd(spikes, static_cast<unsigned long long>(v));
        if (v) e.zero_u32[k] = 0;
    }
}

// The STDP rules of step t (descriptor set of step t): a one-source rule appends and updates in one
// pass; otherwise the sources' appends in order, then the weight update of the touched columns that
// are full. `thread` / `warp` are this thread's ids rotated by half the cluster, so that the rules'
// work lands on other SMs than the first neurons' population work it runs beside.
__device__ __forceinline__ void stdp_rules(const SmallStdp *rules, uint32_t n_rules, unsigned long long t,
                                           uint32_t thread, uint32_t n_threads, int lane)
{
    const uint32_t warp = thread >> 5, n_warps = n_threads >> 5;
    for (uint32_t k = 0; k < n_rules; ++k)
    {
        const SmallStdp &r = rules[k];
        if (r.n_src == 1 && !r.src[0].channel)
        {
            stdp_append_update_range(r.d, r.src[0], r.both[0], t, thread, n_threads);
            continue;
        }
        for (uint32_t j = 0; j < r.n_src; ++j)
        {
            stdp_append_range(r.d, r.src[j], r.both[j], t, thread, n_threads);
            tc::cluster_sync();
        }
        stdp_modify_range(r.d, warp, n_warps, lane);
    }
}

// The first CTA's copy of what p, in this CTA's shared memory, points to (as a generic address).
template <typename T>
__device__ __forceinline__ T *first_cta(T *p)
{
    T *r;
    asm("mapa.u64 %0, %1, 0;" : "=l"(r) : "l"(p));
    return r;
}

// Copies n descriptors to `to` (and moves it past them), all threads of the CTA together.
template <typename T>
__device__ __forceinline__ const T *copy_in(uint8_t *&to, const T *from, uint32_t n)
{
    static_assert(sizeof(T) % 8 == 0 && alignof(T) <= 8, "copied by 8-byte words");
    const uint32_t words = n * (sizeof(T) / 8);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(to);
    for (uint32_t i = threadIdx.x; i < words; i += kSmallThreads)
        dst[i] = reinterpret_cast<const unsigned long long *>(from)[i];
    to += static_cast<size_t>(words) * 8;
    return reinterpret_cast<const T *>(dst);
}

// Bytes of the copies with the counters, and of the spike lists, two sets of each.
inline size_t desc_copy_bytes(const SmallNet &net)
{
    const size_t counters = (net.end[0].n_zero_u32 + 3) / 4 * 16;
    return 2 * (net.n_pops * sizeof(SmallPop) + net.n_projs * sizeof(ProjectionDev) + net.n_stdp * sizeof(SmallStdp) +
                net.n_sources * sizeof(SmallSource) + counters);
}
constexpr size_t kDescCopyMax = 96 * 1024;  // beside the static tables and the lists, within an SM's shared memory
constexpr size_t kListMax = 64 * 1024;

__device__ __forceinline__ uint32_t pop_size(const SmallPop &q) { return q.kind == kSmallLif ? q.lif.n : q.blifat.n; }
__device__ __forceinline__ const uint32_t *pop_list(const SmallPop &q)
{
    return q.kind == kSmallLif ? q.lif.spikes : q.blifat.spikes;
}

// The launch's own copies, in shared memory, of what a step reads and writes from phase to phase: in every CTA
// the descriptors (their fields are read all over a step, between writes that make the compiler read them again,
// and what L1 holds is dropped at every cluster barrier); in the first CTA's the per-step counters and (list_bytes)
// the spike lists, which the others reach over the cluster: a trip of a third of the way to L2, several of which
// follow one another in a step (count reserved, list written, count read, list read). All is zero or unused between
// launches, so nothing is written back. Every thread of the CTA calls it; a cluster barrier has to follow.
__device__ __forceinline__ void own_descriptors(SmallNet &net, uint4 *smem, uint32_t list_bytes)
{
    const SmallPop *const global_pops[2] = {net.pops[0], net.pops[1]};
    uint8_t *to = reinterpret_cast<uint8_t *>(smem);
    for (int set = 0; set < 2; ++set)
    {
        net.pops[set] = copy_in(to, net.pops[set], net.n_pops);
        net.projs[set] = copy_in(to, net.projs[set], net.n_projs);
        net.stdp[set] = copy_in(to, net.stdp[set], net.n_stdp);
        net.sources[set] = copy_in(to, net.sources[set], net.n_sources);
    }
    const uint32_t n_counters = net.end[0].n_zero_u32;
    for (int set = 0; set < 2; ++set)
    {
        uint32_t *counters = reinterpret_cast<uint32_t *>(to);
        to += (n_counters + 3) / 4 * 16;
        for (uint32_t i = threadIdx.x; i < n_counters; i += kSmallThreads) counters[i] = 0u;
        uint32_t *const first = first_cta(counters), *const from = net.end[set].zero_u32;
        net.end[set].zero_u32 = first;
        uint32_t *const lists = first_cta(reinterpret_cast<uint32_t *>(to));
        if (list_bytes) to += list_bytes / 2;
        if (set == 0) __syncthreads();  // the copies are there
        auto counter = [&](const uint32_t *c) -> uint32_t *
        { return c >= from && c < from + n_counters ? first + (c - from) : const_cast<uint32_t *>(c); };
        auto list = [&](const uint32_t *l) -> uint32_t *
        {
            uint32_t at = 0;
            for (uint32_t k = 0; list_bytes && l && k < net.n_pops; ++k)
            {
                if (pop_list(global_pops[set][k]) == l) return lists + at;
                at += (pop_size(global_pops[set][k]) + 3) / 4 * 4;
            }
            return const_cast<uint32_t *>(l);
        };
        for (uint32_t i = threadIdx.x; i < net.n_pops; i += kSmallThreads)
        {
            SmallPop &q = const_cast<SmallPop &>(net.pops[set][i]);
            q.blifat.spike_count = counter(q.blifat.spike_count);
            q.blifat.spikes = list(q.blifat.spikes);
            q.lif.spike_count = counter(q.lif.spike_count);
            q.lif.spikes = list(q.lif.spikes);
        }
        for (uint32_t i = threadIdx.x; i < net.n_sources; i += kSmallThreads)
        {
            SpikeSource &src = const_cast<SmallSource &>(net.sources[set][i]).src;
            src.count = counter(src.count);
            src.idx = list(src.idx);
        }
        for (uint32_t i = threadIdx.x; i < net.n_stdp; i += kSmallThreads)
        {
            SmallStdp &r = const_cast<SmallStdp &>(net.stdp[set][i]);
            r.d.touched_count = counter(r.d.touched_count);
            for (uint32_t j = 0; j < r.n_src; ++j)
            {
                r.src[j].count = counter(r.src[j].count);
                r.src[j].idx = list(r.src[j].idx);
            }
        }
    }
}

// Launched as one cluster of C CTAs (C = cluster size, 1 to 16); every thread of the cluster passes
// the same sequence of cluster barriers (all loop bounds below are the same in every thread).
// Step t is two phases, each closed by a cluster barrier:
//   A: the populations of step t, beside the STDP rules of step t - 1 (they read step t - 1's spike
//      lists and counters, the other descriptor set, and change weights no one reads in phase A);
//   B: the projections of step t (reading the weights after step t - 1's STDP update, as the
//      reference's order requires), beside the retirement of step t - 1's counters.
// A launch ends with the STDP rules of its last step, so both descriptor sets' counters are zero and
// every update is done between launches.
__global__ void __launch_bounds__(kSmallThreads, 1) small_net_kernel(SmallNet net, Control *ctl, uint32_t n_steps,
                                                                      uint32_t desc_bytes, uint32_t list_bytes)
{
    extern __shared__ uint4 s_desc[];
    __shared__ unsigned long long s_spikes;
    __shared__ ScatterTables tab;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t C = gridDim.x;
    const uint32_t rank = blockIdx.x;
    const uint32_t n_threads = C * kSmallThreads;
    // Warps are dealt to the CTAs in turn: the populations' from the first up, the STDP rules' from the last down.
    const uint32_t gthread = 32 * (warp * C + rank) + lane;
    const uint32_t sthread = 32 * ((kSmallWarps - 1 - warp) * C + rank) + lane;
    if (threadIdx.x == 0) s_spikes = 0;
    if (desc_bytes) own_descriptors(net, s_desc, list_bytes);
    unsigned long long t = ctl->step;
    unsigned long long events = 0;
    // Every CTA has read the step number before CTA 0 may advance it (at the end).
    tc::cluster_sync();
    for (uint32_t s = 0; s < n_steps; ++s, ++t)
    {
        // Descriptor sets of this step and of the previous one (selects, not a dynamic index into
        // the parameter block).
        const bool odd = t & 1u;
        const SmallPop *pops = odd ? net.pops[1] : net.pops[0];
        const ProjectionDev *projs = odd ? net.projs[1] : net.projs[0];
        const SmallSource *sources = odd ? net.sources[1] : net.sources[0];
        // ---- phase A
        // What the channels send at step t is known already.
        if (warp == kSmallWarps - 1 && lane < net.n_sources && sources[lane].src.channel)
            resolve_source(sources[lane].src, t, tab.idx[lane], tab.count[lane]);
        // Populations (a pass of the cluster covers n_threads neurons or four times as many; each CTA compacts
        // its own spikes into the list).
        for (uint32_t k = 0; k < net.n_pops; ++k)
        {
            if (pop_size(pops[k]) <= n_threads)
                step_population<1>(pops[k], t, gthread, n_threads);
            else
                step_population<4>(pops[k], t, gthread, n_threads);
        }
        // The STDP rules of step t - 1 (done by the previous launch for its first step).
        if (s > 0 && net.n_stdp) stdp_rules(odd ? net.stdp[0] : net.stdp[1], net.n_stdp, t - 1, sthread, n_threads, lane);
        tc::cluster_sync();
        // ---- phase B
        // Step t - 1's counters are no longer read by anyone. (Beside the first warp's look at the sources.)
        if (rank == 0 && warp == kSmallWarps - 1) retire_counters(odd ? net.end[0] : net.end[1], lane, &s_spikes);
        events += project_rows(net, projs, sources, t, rank, C, tab);
        tc::cluster_sync();
    }
    // The last step's STDP rules, then its counters: both sets are zero between launches.
    const bool last_odd = (t - 1) & 1u;
    if (net.n_stdp)
    {
        stdp_rules(last_odd ? net.stdp[1] : net.stdp[0], net.n_stdp, t - 1, sthread, n_threads, lane);
        tc::cluster_sync();
    }
    if (rank == 0 && warp == kSmallWarps - 1) retire_counters(last_odd ? net.end[1] : net.end[0], lane, &s_spikes);
    if (events) atomicAdd(&ctl->events_total, events);  // thread 0
    __syncthreads();
    if (threadIdx.x == 0 && s_spikes) atomicAdd(&ctl->spikes_total, s_spikes);
    if (rank == 0 && threadIdx.x == 0) ctl->step = t;
}

}  // namespace

int small_net_cluster()
{
    static int c = [] {
        cudaLaunchConfig_t cfg{};
        cfg.blockDim = dim3(kSmallThreads);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        // 16 CTAs are more than every device schedules; the query below says.
        cudaFuncSetAttribute(small_net_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        for (int size = 16; size > 1; size /= 2)
        {
            cfg.gridDim = dim3(size);
            attr[0].val.clusterDim.x = size;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, small_net_kernel, &cfg) == cudaSuccess && n > 0) return size;
            cudaGetLastError();
        }
        return 1;
    }();
    return c;
}

cudaError_t launch_small_net(const SmallNet &net, Control *ctl, uint32_t n_steps, int cluster, cudaStream_t s)
{
    if (!n_steps) return cudaSuccess;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cluster);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    size_t desc = desc_copy_bytes(net), lists = 2 * static_cast<size_t>(net.list_words) * 4;
    if (desc > kDescCopyMax) desc = 0;
    if (!desc || lists > kListMax) lists = 0;
    cfg.dynamicSmemBytes = desc + lists;
    if (cfg.dynamicSmemBytes > 32 * 1024)
    {
        const cudaError_t err = cudaFuncSetAttribute(small_net_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     static_cast<int>(kDescCopyMax + kListMax));
        if (err != cudaSuccess) return err;
    }
    return cudaLaunchKernelEx(&cfg, small_net_kernel, net, ctl, n_steps, static_cast<uint32_t>(desc),
                              static_cast<uint32_t>(lists));
}

}  // namespace knp_gb300
