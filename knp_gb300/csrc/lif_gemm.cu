// Differentiation form: a LIF layer's input product with its recurrence in the epilogue, forward and
// backward, on the tcgen05 tensor cores.
//
// I[t][b][n] = sum_k S_in[t][b][k] W[k][n] is formed as D[neuron][column] = W^T * S_in^T: an accumulator row
// (tensor-memory lane) is a neuron and its columns are consecutive steps of a sample, so the thread that
// owns the lane runs the recurrence (the arithmetic of bptt.cu's scans, operation by operation) down its
// row, and I is never written to memory:
//   forward   U_t = beta V_{t-1} + I_t, S_t = [U_t > theta], V_t = U_t - theta S_t; S and the checkpoints of V out;
//   backward  the same product again, each checkpoint segment's U from its V, then the surrogate-gradient
//             recurrence from the segment's last step to its first; dI goes out as two BF16 terms
//             hi = bf16(dI), lo = bf16(dI - hi), the rows that the products for dW and ds_in read.
// A layer of 2048 x 2048 over 16384 rows: forward 100 us, backward 131 us (tensor time 70 us each), where product
// and scan took 90 + 79 and 90 + 128 us and the gradient's BF16 rows another 53 + 89. The forward is bound by the
// product beside the stores of S, the backward by the latency of its scan (an IEEE division and two dependent
// chains a step), hence two sets of scan warps per half (one: 170 us).
// Layers whose product fills few tiles and has many inputs take product and scan apart instead (apart_is_faster).
// Columns: a CTA pair takes a tile of 256 neurons (128 a CTA) and two halves of up to 128 columns, one per
// CTA's share of the spike operand: whole samples while T fits a half (box_b samples of T steps; a 3-D
// TMA box brings rows (b, t) in that order from [T][B][K]), else one sample's steps tile by tile, forward in
// time or, for the backward, from the last tile (starting on a checkpoint) to the first, the state in
// registers.
#include <algorithm>
#include <cstdint>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "kernels.h"
#include "tcgen05.cuh"

namespace knp_gb300
{
namespace
{

constexpr int kStages = 6;
constexpr uint32_t kOperand = 128 * 64 * 2;  // this CTA's 128 neurons, or its half of the columns, by 64 of K
constexpr uint32_t kStage = 2 * kOperand;
constexpr uint32_t kSmem = kStages * kStage + 1024;
constexpr uint32_t kWait = 1u << 22, kDrainWait = 1u << 14;  // polls
constexpr int kIssuerWarp = 0, kCopyWarp = 1, kScanWarp0 = 4;
constexpr int kScanWarps = 16;  // two sets of four per half, taking its samples in turn
constexpr int kThreads = 32 * (kScanWarp0 + kScanWarps);
constexpr int kMaxSeg = 16;

struct LifGemmArgs
{
    CUtensorMap w;  // BF16 W [K][wp], 64 x 64 boxes (columns from N on reach no neuron)
    CUtensorMap s;  // BF16 S_in [T][B][K], 64 x box_t x box_b boxes
    int T, B, N, w2;
    int chunks;                 // of K
    int splits, cps;            // K in `splits` runs of cps chunks, each its own accumulator
    int half_cols;              // columns of a half: 128 .. 16
    int acc_cols, bufs;         // tensor-memory columns of a tile's accumulators; 2 sets of them if they fit
    int box_t, box_b, t_tiles;  // steps and samples of a half; tiles along time (box_b == 1 if more than one)
    int n_tiles, items;         // pairs of neuron tiles; items = n_tiles * sample groups
    float beta, theta, k;
    int seg;                    // checkpoint interval
    float *S;                   // forward: [T][B][N]
    float *ckpt;                // [ceil(T / seg)][B][N]
    const float *dS;            // backward: [T][B][N]
    __nv_bfloat16 *dI2;         // backward: [T B][2 w2], halves hi and lo
    unsigned int *err;
};

__device__ __forceinline__ bool wait_or_fail(uint64_t *mbar, uint32_t parity, const volatile int *fail)
{
    for (uint32_t i = 0; i < kWait; ++i)
    {
        if (tc::mbar_try_wait(mbar, parity)) return true;
        if (*fail) return false;
    }
    return false;
}

// One thread's neuron over the columns of one sample in the accumulator: steps [t0, t0 + steps), the first at
// tensor-memory address `col`. `V` carries over from tile to tile.
struct Lane
{
    uint32_t col;
    int n, b;
    bool real;  // the neuron exists
};

// kN columns of I from `col`: the runs' sums added in order (as split_sum_kernel of gemm.cu adds them).
template <int kN, bool kSplit>
__device__ __forceinline__ void load_cols(const LifGemmArgs &a, uint32_t col, float *x)
{
    auto ld = [](uint32_t c, float *v)
    {
        if (kN == 16)
            tc::tmem_ld16(c, v);
        else if (kN == 8)
            tc::tmem_ld8(c, v);
        else
            v[0] = tc::tmem_ld1(c);
    };
    ld(col, x);
    if (!kSplit) return;
    for (int p = 1; p < a.splits; ++p)
    {
        float y[kN];
        ld(col + p * 2 * a.half_cols, y);
#pragma unroll
        for (int i = 0; i < kN; ++i) x[i] = __fadd_rn(x[i], y[i]);
    }
}

template <bool kSplit>
__device__ __forceinline__ void forward_sample(const LifGemmArgs &a, const Lane &l, int t0, int steps, float &V)
{
    const size_t stride = static_cast<size_t>(a.B) * a.N;
    const size_t at = static_cast<size_t>(l.b) * a.N + l.n;
    float *S = a.S + static_cast<size_t>(t0) * stride + at;
    float *ck = a.ckpt + static_cast<size_t>((t0 + a.seg - 1) / a.seg) * stride + at;
    int to_ck = (a.seg - t0 % a.seg) % a.seg;  // steps until the next checkpoint
    auto step = [&](float x)
    {
        if (to_ck == 0)
        {
            if (l.real) *ck = V;
            ck += stride;
            to_ck = a.seg;
        }
        --to_ck;
        const float U = __fadd_rn(__fmul_rn(a.beta, V), x);
        const float s = U > a.theta ? 1.0f : 0.0f;
        if (l.real) *S = s;
        S += stride;
        V = __fsub_rn(U, __fmul_rn(a.theta, s));
    };
    int u = 0;
    for (; u + 16 <= steps; u += 16)
    {
        float x[16];
        load_cols<16, kSplit>(a, l.col + u, x);
#pragma unroll
        for (int i = 0; i < 16; ++i) step(x[i]);
    }
    if (u + 8 <= steps)
    {
        float x[8];
        load_cols<8, kSplit>(a, l.col + u, x);
#pragma unroll
        for (int i = 0; i < 8; ++i) step(x[i]);
        u += 8;
    }
    for (; u < steps; ++u)
    {
        float x[1];
        load_cols<1, kSplit>(a, l.col + u, x);
        step(x[0]);
    }
}

// kSeg: the checkpoint interval when it is 8 (whole segments read as 8 columns), else 0.
template <int kSeg, bool kSplit>
__device__ __forceinline__ void backward_sample(const LifGemmArgs &a, const Lane &l, int t0, int steps, float &dV)
{
    constexpr int kMost = kSeg ? kSeg : kMaxSeg;
    const int seg = kSeg ? kSeg : a.seg;
    const size_t stride = static_cast<size_t>(a.B) * a.N;
    const size_t at = static_cast<size_t>(l.b) * a.N + l.n;
    const size_t row = 2 * static_cast<size_t>(a.w2);
    const bool pad = l.n < a.w2;  // columns N .. w2 - 1 of the halves are written as zeros
    // t0 is a multiple of the interval; the segments of the tile from the last to the first.
    const int n_seg = (steps + seg - 1) / seg;
    float g_out[kMost], ck = 0.0f;
    auto fetch = [&](int c)
    {
        const int t = t0 + c * seg, len = min(seg, t0 + steps - t);
        ck = l.real ? a.ckpt[static_cast<size_t>(t / seg) * stride + at] : 0.0f;
#pragma unroll
        for (int u = 0; u < kMost; ++u)
            g_out[u] = (l.real && u < len) ? __ldcs(a.dS + static_cast<size_t>(t + u) * stride + at) : 0.0f;
    };
    fetch(n_seg - 1);
    for (int c = n_seg - 1; c >= 0; --c)
    {
        const int t = t0 + c * seg, len = min(seg, t0 + steps - t);
        float U[kMost], g[kMost];
        if (kSeg == 8 && len == 8)
        {
            load_cols<8, kSplit>(a, l.col + c * seg, U);
        }
        else
        {
#pragma unroll
            for (int u = 0; u < kMost; ++u)
                if (u < len) load_cols<1, kSplit>(a, l.col + c * seg + u, U + u);
        }
        float V = ck;
#pragma unroll
        for (int u = 0; u < kMost; ++u) g[u] = g_out[u];
        if (c > 0) fetch(c - 1);  // used after this segment
#pragma unroll
        for (int u = 0; u < kMost; ++u)
        {
            if (u < len)
            {
                U[u] = __fadd_rn(__fmul_rn(a.beta, V), U[u]);
                const float s = U[u] > a.theta ? 1.0f : 0.0f;
                V = __fsub_rn(U[u], __fmul_rn(a.theta, s));
            }
        }
        __nv_bfloat16 *o = a.dI2 + (static_cast<size_t>(t) * a.B + l.b) * row + l.n;
#pragma unroll
        for (int u = kMost - 1; u >= 0; --u)
        {
            if (u < len)
            {
                const float d = __fadd_rn(1.0f, __fmul_rn(a.k, fabsf(__fsub_rn(U[u], a.theta))));
                const float sg = __fdiv_rn(__fmul_rn(0.5f, a.k), __fmul_rn(d, d));
                const float dU = __fadd_rn(__fmul_rn(g[u], sg), __fmul_rn(dV, __fsub_rn(1.0f, __fmul_rn(a.theta, sg))));
                dV = __fmul_rn(a.beta, dU);
                const float v = l.real ? dU : 0.0f;
                const __nv_bfloat16 hi = __float2bfloat16_rn(v);
                const __nv_bfloat16 lo = __float2bfloat16_rn(__fsub_rn(v, __bfloat162float(hi)));
                if (pad)
                {
                    __nv_bfloat16 *p = o + static_cast<size_t>(u) * a.B * row;
                    p[0] = hi;
                    p[a.w2] = lo;
                }
            }
        }
    }
}

// Roles in each CTA of a pair: warp 0 issues the pair's MMAs (even rank), warp 1 loads this CTA's operands,
// warps 4-19 scan the two halves' columns (thread = neuron; per half two sets of four warps take its samples
// in turn: the scans are bound by latency). Two accumulators: the scan of a tile
// runs beside the product of the next. Persistent over items (a pair of neuron tiles and a group of
// samples). Waits and their failure are gemm_pair_kernel's (gemm.cu).
template <bool kBackward, int kSeg, bool kSplit>
__global__ void __launch_bounds__(kThreads, 1) __cluster_dims__(2, 1, 1)
    lif_gemm_kernel(const __grid_constant__ LifGemmArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages];  // full, acc_empty: of the even CTA
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], drain;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = tc::cluster_rank();
    const uint32_t peer_fail = tc::mapa(tc::smem_u32(&s_fail), rank ^ 1u);
    auto fail = [&]()
    {
        s_fail = 1;
        tc::st_cluster_u32(peer_fail, 1u);
        atomicOr(a.err, 1u);
    };
    if (warp == kIssuerWarp) tc::tmem_alloc_pair(&tmem_slot, 512);
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < kStages; ++s)
        {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int i = 0; i < 2; ++i)
        {
            tc::mbar_init(&acc_full[i], 1);
            tc::mbar_init(&acc_empty[i], 2 * kScanWarps);
        }
        tc::mbar_init(&drain, 1);
        s_fail = 0;
    }
    // What is above overlaps the end of the kernel before (programmatic dependent launch), nothing below does; a
    // training iteration of about twenty such launches went from 190 us to 177.
    pdl_begin();
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();  // both CTAs' barriers and tensor memory are set up
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    const uint32_t base = (tc::smem_u32(smem) + 1023u) & ~1023u;
    const int pairs = gridDim.x / 2, pair = blockIdx.x / 2;
    // Tile q of an item: its time tile, from the last for the backward.
    auto time_tile = [&](int q) { return kBackward ? a.t_tiles - 1 - q : q; };

    if (warp == kCopyWarp)
    {
        if (lane == 0)
        {
            const uint32_t full0 = tc::mapa(tc::smem_u32(full), 0);
            const uint32_t s_bytes = static_cast<uint32_t>(a.box_t * a.box_b) * 128u;
            int issued = 0, s = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int it = pair; it < a.items && ok; it += pairs)
            {
                const int n0 = (it % a.n_tiles) * 256 + 128 * static_cast<int>(rank);
                const int b0 = ((it / a.n_tiles) * 2 + static_cast<int>(rank)) * a.box_b;
                for (int q = 0; q < a.t_tiles && ok; ++q)
                {
                    const int t0 = time_tile(q) * a.box_t;
                    for (int c = 0; c < a.chunks; ++c)
                    {
                        if (!wait_or_fail(&empty[s], ph, &s_fail))
                        {
                            ok = false;
                            break;
                        }
                        const uint32_t dst = base + s * kStage;
                        if (rank == 0) tc::mbar_expect_tx(&full[s], 2 * (kOperand + s_bytes));
                        tc::tma_load_2d_pair(dst, &a.w, n0, c * 64, full0 + s * 8u);
                        tc::tma_load_2d_pair(dst + kOperand / 2, &a.w, n0 + 64, c * 64, full0 + s * 8u);
                        tc::tma_load_3d_pair(dst + kOperand, &a.s, c * 64, t0, b0, full0 + s * 8u);
                        ++issued;
                        if (++s == kStages)
                        {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
                }
            }
            if (!ok) fail();
            // Both CTAs' copies in flight after a failed wait land before either leaves (bounded).
            if (s_fail && rank == 0)
                for (int i = max(0, issued - kStages); i < issued; ++i)
                    tc::mbar_wait(&full[i % kStages], (i / kStages) & 1, kDrainWait);
        }
    }
    else if (warp == kIssuerWarp)
    {
        if (lane == 0 && rank == 0)
        {
            const uint32_t idesc = tc::idesc_bf16_f32(256, 2 * a.half_cols) | tc::kIdescAMn;
            const uint64_t dw = tc::smem_desc_sw128_mn(base, kOperand / 2), ds = tc::smem_desc_sw128(base + kOperand, 1024);
            int s = 0, n = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int it = pair; it < a.items && ok; it += pairs)
                for (int q = 0; q < a.t_tiles && ok; ++q, ++n)
                {
                    const int acc = n % a.bufs, use = n / a.bufs;
                    if (use >= 1 && !wait_or_fail(&acc_empty[acc], (use - 1) & 1, &s_fail))
                    {
                        ok = false;
                        break;
                    }
                    uint32_t d = tmem + acc * a.acc_cols;
                    int in_run = 0;  // chunk of the run
                    for (int c = 0; c < a.chunks; ++c)
                    {
                        if (!wait_or_fail(&full[s], ph, &s_fail))
                        {
                            ok = false;
                            break;
                        }
                        tc::fence_after_sync();
                        const uint64_t off = static_cast<uint64_t>(s) * (kStage >> 4);
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            tc::mma_bf16_pair(d, dw + off + j * (2048 >> 4), ds + off + j * (32 >> 4), idesc,
                                              (in_run > 0 || j > 0) ? 1u : 0u);
                        tc::commit_pair(&empty[s]);
                        if (++in_run == a.cps)
                        {
                            in_run = 0;
                            d += 2 * a.half_cols;
                        }
                        if (++s == kStages)
                        {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
                    if (ok) tc::commit_pair(&acc_full[acc]);
                }
            if (!ok) fail();
            tc::commit_pair(&drain);
            if (!tc::mbar_wait(&drain, 0, kWait)) fail();
        }
        else if (lane == 0)
        {
            // Odd rank: the issuer's last arrivals reach this CTA before it leaves.
            if (!tc::mbar_wait(&drain, 0, kWait)) fail();
        }
    }
    else if (warp >= kScanWarp0)
    {
        const int half = ((warp - kScanWarp0) >> 2) & 1, set = (warp - kScanWarp0) >> 3;
        const uint32_t lanes = tmem + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + half * a.half_cols;
        const uint32_t acc_empty0 = tc::mapa(tc::smem_u32(acc_empty), 0);
        int n = 0;
        bool ok = true;
        for (int it = pair; it < a.items && ok; it += pairs)
        {
            Lane l;
            l.n = (it % a.n_tiles) * 256 + 128 * static_cast<int>(rank) + 32 * (warp & 3) + lane;
            l.real = l.n < a.N;
            const int b0 = ((it / a.n_tiles) * 2 + half) * a.box_b;
            float carry = 0.0f;  // V, or dV, from tile to tile of one sample
            for (int q = 0; q < a.t_tiles; ++q, ++n)
            {
                const int acc = n % a.bufs;
                int got = 1;
                if (lane == 0) got = wait_or_fail(&acc_full[acc], (n / a.bufs) & 1, &s_fail);
                if (!__shfl_sync(0xffffffffu, got, 0))
                {
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                const int t0 = time_tile(q) * a.box_t, steps = min(a.box_t, a.T - t0);
                for (int i = set; i < a.box_b && b0 + i < a.B; i += 2)
                {
                    if (a.t_tiles == 1) carry = 0.0f;
                    l.b = b0 + i;
                    l.col = lanes + acc * a.acc_cols + i * a.box_t;
                    if (kBackward)
                        backward_sample<kSeg, kSplit>(a, l, t0, steps, carry);
                    else
                        forward_sample<kSplit>(a, l, t0, steps, carry);
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive_cluster(acc_empty0 + acc * 8u);
            }
        }
        if (!ok && lane == 0) fail();
    }
    __syncwarp();
    tc::fence_before_sync();
    __syncthreads();
    // Neither CTA leaves while the other's MMAs may read its shared memory or arrivals may reach it.
    tc::cluster_sync();
    if (warp == kIssuerWarp) tc::tmem_dealloc_pair(tmem, 512);
}

// The layer as a product, the scan of bptt.cu and (backward) the gradient's BF16 rows: the same bits.
int launch_apart(const LifGemmArgs &a, const void *S_in, const void *W, int K, int k8, int wp, bool backward, cudaStream_t s)
{
    const int rows = a.T * a.B;
    const size_t n = (static_cast<size_t>(rows) * a.N + 3) / 4 * 4;
    const long long BN = static_cast<long long>(a.B) * a.N;
    float *I = nullptr;
    if (workspace_alloc(reinterpret_cast<void **>(&I), (backward ? 2 : 1) * n * sizeof(float), s) != cudaSuccess)
    {
        cudaGetLastError();
        return -3;
    }
    int rc = lif_input_gemm(S_in, W, I, rows, K, k8, a.N, wp, a.err, s);
    if (rc == 0 && !backward) rc = lif_scan_forward(I, a.S, a.ckpt, a.T, BN, a.beta, a.theta, a.seg, 0, 0.0f, s);
    if (rc == 0 && backward)
    {
        rc = lif_scan_backward(I, a.ckpt, a.dS, I + n, a.T, BN, a.beta, a.theta, a.seg, 0, a.k, s);
        if (rc == 0) rc = bf16_operand(I + n, 0, rows, a.N, 2, 0, a.w2, a.dI2, s);
    }
    cudaFreeAsync(I, s);
    return rc;
}

// Where the product alone would split K over CTAs, a pair here takes the runs one after another, and a time tile after
// another, while most of the device idles; the product apart takes a run in parallel with the others, and then the scan
// takes a segment after another on threads that have little else to hide its loads. What either does in sequence, in
// units of a chunk of a pair's product (0.37 us): fitted to 400 layers of 1..1000 steps, 1..300 samples, 200..8000
// inputs, 4..2000 neurons and intervals of 1..16 (50 x 2, 5000 -> 300: forward 135 us here, 27 apart; 64 x 8, 2048 -> 10: 37
// and 22; 27 x 12, 526 -> 1585: 12 and 25; 559 x 1, 561 -> 173, interval 1: 44 and 460). The form taken was the slower one by 8 % or
// more in one of 20.
bool apart_is_faster(const LifGemmArgs &a, int waves, bool backward)
{
    const long long tiles = static_cast<long long>(waves) * a.t_tiles;
    const long long samples = tiles * ((a.box_b + 1) / 2);  // that a set of scan warps takes, tile by tile
    const int t = a.box_t, n_seg = (a.T + a.seg - 1) / a.seg;
    const int reads = a.splits * (backward ? (a.seg == 8 ? t / 8 + t % 8 : t) : t / 16 + t % 16 / 8 + t % 8);
    const double here = static_cast<double>(tiles) * a.chunks +
                        static_cast<double>(samples) * (backward ? reads / 6.0 + 3.0 * ((t + a.seg - 1) / a.seg)
                                                                 : reads / 7.0 + t / 23.0);
    const double apart = backward ? 4 + 2.0 * a.cps + 2.5 * n_seg + a.T / 4.0 : 7 + 1.7 * a.cps + 2.0 * n_seg + a.T / 12.0;
    return here > apart;
}

int launch(LifGemmArgs &a, const void *S_in, const void *W, int K, int k8, int wp, bool backward, cudaStream_t s)
{
    if (a.T < 1 || a.B < 1 || a.N < 1 || K < 1 || a.seg < 1 || a.seg > kMaxSeg) return -1;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int pairs = std::max(1, sms / 2);
    a.chunks = (K + 63) / 64;
    // The product alone would split K here when its 128 x 128 tiles leave most SMs idle; the runs are kept
    // apart and added in the same order, so that I has the same bits.
    const long long tiles = ((static_cast<long long>(a.T) * a.B + 127) / 128) * ((a.N + 127) / 128);
    a.splits = gemm_splits(static_cast<int>(std::min<long long>(tiles, 1 << 20)), a.chunks, sms, a.cps);
    // The backward writes its rows up to their width, which a caller may have chosen above the neurons' last tile.
    a.n_tiles = ((backward ? std::max(a.N, a.w2) : a.N) + 255) / 256;
    auto plan = [&](int cols)
    {
        a.half_cols = cols;
        a.acc_cols = 2 * cols * a.splits;
        a.bufs = 2 * a.acc_cols <= 512 ? 2 : 1;
        // Tiles along time start on a checkpoint.
        a.box_t = a.T <= cols ? a.T : cols / a.seg * a.seg;
        a.box_b = a.T <= cols ? std::min(cols / a.T, a.B) : 1;
        a.t_tiles = (a.T + a.box_t - 1) / a.box_t;
        a.items = a.n_tiles * ((a.B + 2 * a.box_b - 1) / (2 * a.box_b));
        return (a.items + pairs - 1) / pairs;
    };
    int waves;
    if (a.splits > 1)
    {
        waves = plan(a.splits <= 4 ? 64 : a.splits <= 8 ? 32 : 16);  // at most 16 runs: 512 columns
    }
    else
    {
        // Halves of 64 columns when they spread the samples over more of the device: a tile of them takes
        // about half as long, so they win while they need fewer than twice the waves.
        waves = plan(128);
        const int narrow = a.T > 64 ? 2 * waves : plan(64);
        if (narrow < 2 * waves)
            waves = narrow;
        else
            plan(128);
    }
    // (A product of one wave: its time is one tile's. The gradient's rows are stored 16 bytes at a time then.)
    if (tiles <= sms && (reinterpret_cast<uintptr_t>(a.dI2) & 15u) == 0 && apart_is_faster(a, waves, backward)) return launch_apart(a, S_in, W, K, k8, wp, backward, s);
    if (!sw128_map(&a.w, W, K, wp, 64) || !sw128_map_3d(&a.s, S_in, a.T, a.B, k8, a.box_t, a.box_b)) return -3;
    auto kernel = !backward   ? (a.splits > 1 ? lif_gemm_kernel<false, 0, true> : lif_gemm_kernel<false, 0, false>)
                  : a.seg == 8 ? (a.splits > 1 ? lif_gemm_kernel<true, 8, true> : lif_gemm_kernel<true, 8, false>)
                               : (a.splits > 1 ? lif_gemm_kernel<true, 0, true> : lif_gemm_kernel<true, 0, false>);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) return -3;
    launch_pdl(kernel, dim3(2 * std::min(a.items, pairs)), dim3(kThreads), kSmem, s, a);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace

// S_in: BF16 [T B][k8], W: BF16 [K][wp] with the weights in columns 0 .. N - 1 and zeros up to w2 (rows of
// whole 16-byte units).
int lif_layer_forward(const void *S_in, const void *W, float *S, float *ckpt, int T, int B, int K, int k8, int N, int w2, int wp,
                      float beta, float theta, int seg, unsigned int *err, cudaStream_t s)
{
    LifGemmArgs a{};
    a.T = T;
    a.B = B;
    a.N = N;
    a.w2 = w2;
    a.beta = beta;
    a.theta = theta;
    a.seg = seg;
    a.S = S;
    a.ckpt = ckpt;
    a.err = err;
    return launch(a, S_in, W, K, k8, wp, false, s);
}

int lif_layer_backward(const void *S_in, const void *W, const float *ckpt, const float *dS, void *dI2, int T, int B, int K,
                       int k8, int N, int w2, int wp, float beta, float theta, int seg, float k, unsigned int *err, cudaStream_t s)
{
    LifGemmArgs a{};
    a.T = T;
    a.B = B;
    a.N = N;
    a.w2 = w2;
    a.beta = beta;
    a.theta = theta;
    a.k = k;
    a.seg = seg;
    a.ckpt = const_cast<float *>(ckpt);
    a.dS = dS;
    a.dI2 = static_cast<__nv_bfloat16 *>(dI2);
    a.err = err;
    return launch(a, S_in, W, K, k8, wp, true, s);
}

}  // namespace knp_gb300
