// Neuron-side training of resource-STDP BLIFAT and AltAI-LIF populations over their
// SynapticResourceSTDPDeltaSynapse projections, after the population step and before the
// projections (the population's step in populations_old.h:195-217 ends with train_population; the
// AltAI-LIF training of altai/altai_stdp.h is the same computation):
//   process_spiking_neurons_impl (knp/backends/cpu/cpu-library/include/knp/backends/cpu-library/impl/
//     populations/blifat/blifat_stdp.h:35-103) for every neuron that spiked,
//   do_dopamine_plasticity_impl (:106-155) and renormalize_resource (impl/populations/training/
//     stdp.h:152-186) for every neuron, with recalculate_synapse_weights (training/stdp.h:40-52).
//
// Neurons are independent (a neuron's synapses are the ones into it), so one warp, or one block, trains one
// neuron through all three stages in the reference's order. The work list is this step's spike list
// followed by the non-spiking neurons the population kernel found with dopamine or renormalisation
// work; every other neuron would be left unchanged. A neuron's synapses are its entries of the
// column index, in get_all_connected_synapses order (projection load order, then synapse index),
// skipping locked projections. Per-synapse updates run on its threads; the two quantities the
// reference accumulates across synapses (the FP64 additional threshold and the FP32 free
// resource) are accumulated in synapse order, so every rounding is the reference's (or in another
// order where none rounds).
#include <cstdint>

#include "kernels.h"
#include "population_dev.cuh"

namespace knp_gb300
{
namespace
{

constexpr int kTrainThreads = 256;
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr unsigned long long kPosMask = (1ull << kResSlotShift) - 1;

// std::min(static_cast<float>(std::pow(2, -stability)), 1.F): the power in FP64 (CUDA's exp2),
// rounded to FP32.
__device__ __forceinline__ float resource_factor(float stability)
{
    const float v = __double2float_rn(exp2(-static_cast<double>(stability)));
    return 1.0f < v ? 1.0f : v;
}

// recalculate_synapse_weights (training/stdp.h:40-52) for one synapse.
__device__ __forceinline__ float synapse_weight(float resource, float w_min, float w_max)
{
    const float syn_w = resource < 0.0f ? 0.0f : resource;  // std::max(resource, 0.F)
    const float diff = __fsub_rn(w_max, w_min);
    return __fadd_rn(w_min, __fdiv_rn(__fmul_rn(diff, syn_w), __fadd_rn(diff, syn_w)));
}

// is_point_in_interval (training/stdp.h:129-133), unsigned.
__device__ __forceinline__ bool in_interval(unsigned long long a, unsigned long long b, unsigned long long x)
{
    if (a > b)
    {
        const unsigned long long c = a;
        a = b;
        b = c;
    }
    return a <= x && x <= b;
}

// Synapse `e` of the column range [a, b): its position in the concatenated arrays, and whether it
// belongs to an unlocked projection (is in the working list).
__device__ __forceinline__ bool working_synapse(const ResSynDev &y, long long e, long long b, unsigned long long &pos)
{
    if (e >= b) return false;
    const unsigned long long ent = y.col_pos[e];
    pos = ent & kPosMask;
    return y.locked[ent >> kResSlotShift] == 0u;
}

constexpr int kPer = 4;  // synapses of a thread in a tile

// Exponents that bound the additional threshold's FP64 sum: every term is a multiple of 2^lo and less than 2^hi.
struct SumRange
{
    int lo = 1 << 20, hi = -(1 << 20);
    __device__ void add(float x)
    {
        const uint32_t u = __float_as_uint(x) & 0x7FFFFFFFu;
        if (!u) return;
        const int e = static_cast<int>(u >> 23);
        if (e == 0xFF)  // infinite or NaN: no order is free
        {
            hi = 1 << 20;
            return;
        }
        const uint32_t m = e ? (u & 0x7FFFFFu) | 0x800000u : u;
        const int ulp = (e ? e : 1) - 150;
        lo = min(lo, ulp + __ffs(static_cast<int>(m)) - 1);
        hi = max(hi, ulp + 24);
    }
    __device__ void join(int l, int h)
    {
        lo = min(lo, l);
        hi = max(hi, h);
    }
    // Whether sums of up to n such terms are exact in FP64, in whatever order.
    __device__ bool exact(unsigned long long n) const { return hi + 64 - __clzll(static_cast<long long>(n)) - lo <= 53; }
};

// Shared memory of the kT threads that train a neuron together.
template <int kT>
struct TrainShared
{
    float x[kT * kPer], du[kT * kPer];  // a tile's terms of the additional threshold and changes of the resource
    uint32_t ok[kT * kPer / 32], hebb[kT * kPer / 32];
    double part[kT / 32];
    int lo[kT / 32], hi[kT / 32];
    uint32_t count[kT / 32];
    float f, g;  // values that one thread makes for all
};

template <int kT>
__device__ __forceinline__ void group_sync()
{
    if (kT == 32)
        __syncwarp();
    else
        __syncthreads();
}

// Sum of v over the group, in every thread.
template <int kT>
__device__ __forceinline__ uint32_t group_sum(TrainShared<kT> &sh, uint32_t v, int tid)
{
    v = __reduce_add_sync(kFull, v);
    if (kT == 32) return v;
    if ((tid & 31) == 0) sh.count[tid >> 5] = v;
    __syncthreads();
    uint32_t all = 0;
#pragma unroll
    for (int k = 0; k < kT / 32; ++k) all += sh.count[k];
    __syncthreads();
    return all;
}

// Trains neuron i with kT threads (this is thread tid of them): a warp for neurons of few synapses, a block for ones
// of many, whose per-synapse work is then one round of loads instead of one per 32. What has to be taken in synapse
// order is done by the first warp from shared memory: the free resource (FP32, a chain of adds), and the additional
// threshold where its FP64 sum would round (else it is the same in any order, and FP64 is a slow unit). A label step
// of 200 neurons with 784 synapses each took 182 us by warps that shuffled every synapse's terms to all lanes, and
// takes 19.
template <int kT>
__device__ void train_neuron(const TrainView &p, uint32_t i, unsigned long long t, bool spiked, int tid, TrainShared<kT> &sh)
{
    const ResourceDev &r = p.res;
    const ResSynDev &y = p.syn;
    const int lane = tid & 31, warp = tid >> 5;
    int32_t status = r.isi_status[i];
    const bool forced = r.is_forced[i] != 0;
    const float dopa = p.dopa[i];
    float stab = r.stability[i], fr = r.free_resource[i];
    unsigned long long last_step = r.last_step[i], first = r.first_isi_spike[i], last_spike = r.last_spike_step[i];
    const uint32_t isi_max = pu(r.isi_max, i);
    const long long a = y.col_ptr[i], b = y.col_ptr[i + 1];

    if (spiked)
    {
        // process_spiking_neurons_impl: ISI status, stability at a new ISI period, then one pass over
        // the synapses (additional-threshold term from the weight before this step's change,
        // contribution flag, Hebbian flag reset, resource change, new weight).
        last_spike = t;
        status = update_isi(status, forced, dopa, isi_max, t, last_step, first);
        if (status == 1) stab = __fsub_rn(stab, pf(r.stability_change_at_isi, i));
        if (tid == 0) sh.g = __fmul_rn(pf(r.d_h, i), resource_factor(stab));
        group_sync<kT>();
        const float d_h = sh.g;
        double add = 0.0;
        SumRange range;
        for (long long base = a; base < b; base += kT * kPer)
        {
            double part = 0.0;
            SumRange mine;
#pragma unroll
            for (int u = 0; u < kPer; ++u)
            {
                const int q = u * kT + tid;
                unsigned long long pos = 0;
                const bool ok = working_synapse(y, base + q, b, pos);
                float x = 0.0f, du = 0.0f;
                bool hebb = false;
                if (ok)
                {
                    const float w = y.w[pos];
                    x = __fmul_rn(w, w > 0.0f ? 1.0f : 0.0f);
                    const bool had_spike = in_interval(t - y.period[pos], t, y.last_spike[pos] + y.delay[pos] - 1ull);
                    uint32_t fl = y.flags[pos];
                    if (status != 2 || had_spike) fl = had_spike ? (fl | 2u) : (fl & ~2u);
                    if (status != 2) fl &= ~1u;
                    float res = y.resource[pos];
                    if (status != 0)
                    {
                        du = y.d_u[pos];
                        res = __fsub_rn(res, du);
                        if ((fl & 2u) && !(fl & 1u))
                        {
                            res = __fadd_rn(res, d_h);
                            fl |= 1u;
                            hebb = true;
                        }
                    }
                    y.resource[pos] = res;
                    y.flags[pos] = static_cast<uint8_t>(fl);
                    y.w[pos] = synapse_weight(res, y.w_min[pos], y.w_max[pos]);
                    mine.add(x);
                    part = __dadd_rn(part, static_cast<double>(x));
                }
                sh.x[q] = x;
                sh.du[q] = du;
                const unsigned okm = __ballot_sync(kFull, ok), hm = __ballot_sync(kFull, hebb);
                if (lane == 0)
                {
                    sh.ok[q >> 5] = okm;
                    sh.hebb[q >> 5] = hm;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) part = __dadd_rn(part, __shfl_xor_sync(kFull, part, o));
            const int lo = __reduce_min_sync(kFull, mine.lo), hi = __reduce_max_sync(kFull, mine.hi);
            if (lane == 0)
            {
                sh.part[warp] = part;
                sh.lo[warp] = lo;
                sh.hi[warp] = hi;
            }
            group_sync<kT>();
            if (warp == 0)
            {
                const long long left = b - base;
                const int n = left < kT * kPer ? static_cast<int>(left) : kT * kPer;
#pragma unroll
                for (int k = 0; k < kT / 32; ++k) range.join(sh.lo[k], sh.hi[k]);
                if (range.exact(static_cast<unsigned long long>(base - a) + n + 1))
                {
#pragma unroll
                    for (int k = 0; k < kT / 32; ++k) add = __dadd_rn(add, sh.part[k]);
                }
                else
                {
                    for (int q = 0; q < n; ++q)
                        if ((sh.ok[q >> 5] >> (q & 31)) & 1u) add = __dadd_rn(add, static_cast<double>(sh.x[q]));
                }
                for (int w = 0; status != 0 && w * 32 < n; ++w)
                {
                    const uint32_t okm = sh.ok[w], hm = sh.hebb[w];
                    const float *du = sh.du + 32 * w;
                    if (okm == kFull && hm == 0u)
                    {
#pragma unroll
                        for (int q = 0; q < 32; ++q) fr = __fadd_rn(fr, du[q]);
                    }
                    else
                    {
#pragma unroll
                        for (int q = 0; q < 32; ++q)
                        {
                            if ((okm >> q) & 1u) fr = __fadd_rn(fr, du[q]);
                            if ((hm >> q) & 1u) fr = __fsub_rn(fr, d_h);
                        }
                    }
                }
            }
            group_sync<kT>();  // the tile is used again
        }
        if (tid == 0)
        {
            y.add_thr[i] = __dmul_rn(add, static_cast<double>(pf(r.add_thr_coef, i)));
            sh.f = fr;
        }
        group_sync<kT>();
        fr = sh.f;
    }

    if (dopa > 0.0f || (dopa < 0.0f && status != 0))
    {
        // do_dopamine_plasticity_impl: resource change of contributing synapses while the last spike
        // is recent, stability change, new weights of every synapse.
        const bool recent = t - last_spike <= pu(r.dopamine_time, i);
        group_sync<kT>();  // sh.g and sh.f have been read
        if (tid == 0) sh.g = __fmul_rn(dopa, resource_factor(stab));
        group_sync<kT>();
        const float change = sh.g;
        uint32_t n_app = 0;
#pragma unroll 4
        for (long long e = a + tid; e < b; e += kT)
        {
            unsigned long long pos = 0;
            if (working_synapse(y, e, b, pos))
            {
                float res = y.resource[pos];
                if (recent && (y.flags[pos] & 2u))
                {
                    res = __fadd_rn(res, change);
                    y.resource[pos] = res;
                    ++n_app;
                }
                y.w[pos] = synapse_weight(res, y.w_min[pos], y.w_max[pos]);
            }
        }
        n_app = group_sum<kT>(sh, n_app, tid);
        for (uint32_t k = 0; k < n_app; ++k) fr = __fsub_rn(fr, change);
        if (tid == 0) stab = dopamine_stability(stab, dopa, pf(r.stability_change_param, i), forced, t, first, isi_max);
    }

    if (!(t - last_step <= isi_max && status != 0) && !(fabsf(fr) < pf(r.resource_threshold, i)))
    {
        // renormalize_resource: the free resource divided over the working synapses and the drain.
        uint32_t mine = 0;
        for (long long e = a + tid; e < b; e += kT)
        {
            unsigned long long pos = 0;
            mine += working_synapse(y, e, b, pos) ? 1u : 0u;
        }
        const unsigned long long n_syn = group_sum<kT>(sh, mine, tid);
        const float add_v = __fdiv_rn(fr, __ull2float_rn(n_syn + pu(r.drain, i)));
#pragma unroll 4
        for (long long e = a + tid; e < b; e += kT)
        {
            unsigned long long pos = 0;
            if (working_synapse(y, e, b, pos))
            {
                const float res = __fadd_rn(y.resource[pos], add_v);
                y.resource[pos] = res;
                y.w[pos] = synapse_weight(res, y.w_min[pos], y.w_max[pos]);
            }
        }
        fr = 0.0f;
    }

    if (tid == 0)
    {
        r.isi_status[i] = status;
        r.last_step[i] = last_step;
        r.first_isi_spike[i] = first;
        r.last_spike_step[i] = last_spike;
        r.stability[i] = stab;
        r.free_resource[i] = fr;
    }
    group_sync<kT>();  // the shared memory is the next neuron's
}

template <int kT>
__device__ __forceinline__ void train_groups(const TrainView &p, unsigned long long t, uint32_t block, uint32_t n_blocks,
                                             TrainShared<kT> *shared)
{
    constexpr uint32_t kGroups = kTrainThreads / kT;
    const uint32_t n_spk = *p.spike_count, n_work = *p.syn.work_count;
    const uint32_t group = threadIdx.x / kT;
    for (uint32_t j = block * kGroups + group; j < n_spk + n_work; j += n_blocks * kGroups)
    {
        const bool spiked = j < n_spk;
        train_neuron<kT>(p, spiked ? p.spikes[j] : p.syn.work[j - n_spk], t, spiked, static_cast<int>(threadIdx.x % kT),
                         shared[group]);
    }
}

// A neuron of kBlockSynapses synapses or more on average is a block's work, else a warp's.
constexpr uint32_t kBlockSynapses = 128;
__device__ __forceinline__ void train_block(const TrainView &p, unsigned long long t, uint32_t block, uint32_t n_blocks)
{
    __shared__ union Shared
    {
        TrainShared<kTrainThreads> block;
        TrainShared<32> warp[kTrainThreads / 32];
        __device__ Shared() {}
    } shared;
    if (p.per_neuron >= kBlockSynapses)
        train_groups<kTrainThreads>(p, t, block, n_blocks, &shared.block);
    else
        train_groups<32>(p, t, block, n_blocks, shared.warp);
}

__global__ void __launch_bounds__(kTrainThreads) resource_train_kernel(TrainView p, Control *ctl)
{
    pdl_begin();
    train_block(p, ctl->step, blockIdx.x, gridDim.x);
}

// Several populations' training in one launch.
__global__ void __launch_bounds__(kTrainThreads) train_batch_kernel(const __grid_constant__ TrainBatch b, Control *ctl)
{
    pdl_begin();
    const uint32_t k = b.of_block(blockIdx.x);
    train_block(b.item[k], ctl->step, blockIdx.x - b.first[k], b.first[k + 1] - b.first[k]);
}

}  // namespace

void launch_resource_train(const TrainView &p, int blocks, Control *ctl, cudaStream_t s)
{
    launch_pdl(resource_train_kernel, dim3(blocks > 0 ? blocks : 1), dim3(kTrainThreads), 0, s, p, ctl);
}

void launch_train_batch(const TrainBatch &b, Control *ctl, cudaStream_t s)
{
    launch_pdl(train_batch_kernel, dim3(b.blocks()), dim3(kTrainThreads), 0, s, b, ctl);
}

}  // namespace knp_gb300
