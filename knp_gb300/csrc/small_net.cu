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
#include "scatter_list.cuh"
#include "stdp_dev.cuh"
#include "tcgen05.cuh"

namespace knp_gb300
{
namespace
{

constexpr int kSmallThreads = 512;
constexpr uint32_t kSmallWarps = kSmallThreads / 32;
constexpr int kInFlight = 3;  // synapses a thread loads at a time (2: 6.7 us a step, 3: 6.6, 4: 6.65)

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
    __shared__ ScatterTables<kSmallThreads> tab;
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
        events += project_rows<kSmallThreads, kInFlight, true, false>(projs, sources, net.n_sources, t, rank, C, tab,
                                                         [](const ProjectionDev &, uint32_t count) { return count; });
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

namespace
{

// Shared memory of a launch beside the kernel's own: the copies, as far as they fit.
struct SmallSmem
{
    size_t desc, lists;
    explicit SmallSmem(const SmallNet &net) : desc(desc_copy_bytes(net)), lists(2 * static_cast<size_t>(net.list_words) * 4)
    {
        if (desc > kDescCopyMax) desc = 0;
        if (!desc || lists > kListMax) lists = 0;
    }
};

cudaLaunchConfig_t small_net_config(const SmallSmem &smem, int cluster, cudaStream_t s, cudaLaunchAttribute *attr)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cluster);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = smem.desc + smem.lists;
    cfg.stream = s;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = cluster;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

int small_net_cluster(const SmallNet &net)
{
    // 16 CTAs are more than the portable size: allowed per device, so asked for and set for the current one.
    if (cudaFuncSetAttribute(small_net_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        allow_dynamic_smem(small_net_kernel) != cudaSuccess)
        cudaGetLastError();
    const SmallSmem smem(net);
    for (int size = 16; size > 1; size /= 2)
    {
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = small_net_config(smem, size, nullptr, &attr);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, small_net_kernel, &cfg) == cudaSuccess && n > 0) return size;
        cudaGetLastError();
    }
    return 1;
}

cudaError_t launch_small_net(const SmallNet &net, Control *ctl, uint32_t n_steps, int cluster, cudaStream_t s)
{
    if (!n_steps) return cudaSuccess;
    const SmallSmem smem(net);
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = small_net_config(smem, cluster, s, &attr);
    return cudaLaunchKernelEx(&cfg, small_net_kernel, net, ctl, n_steps, static_cast<uint32_t>(smem.desc),
                              static_cast<uint32_t>(smem.lists));
}

}  // namespace knp_gb300
