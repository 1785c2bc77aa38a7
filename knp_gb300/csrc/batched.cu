// Batched form on 5th-generation tensor cores.
//
// bf16_gemm_tn_simple: D[M x N] (FP32) = A[M x K] * B[N x K]^T with BF16 operands (row-major, K
// contiguous), tcgen05.mma kind::f16 with the accumulator in tensor memory, single stage; the
// pipelined GEMM is gemm.cu.
#include <algorithm>
#include <cstdlib>
#include <cstdint>
#include <functional>
#include <memory>
#include <mutex>
#include <queue>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "kernels.h"
#include "tcgen05.cuh"

namespace knp_gb300
{
namespace
{

constexpr int kGemmM = 128;
constexpr int kGemmN = 64;
constexpr int kGemmK = 64;  // K chunk staged in shared memory
constexpr uint32_t kWaitLimit = 1u << 22;  // try_wait calls of up to kSuspendNs each

// Stage rows [r0, r0 + rows) x K-chunk [k0, k0 + kGemmK) of a row-major BF16 matrix into the
// canonical no-swizzle K-major layout (zero outside the matrix).
__device__ __forceinline__ void stage_tile(
    const __nv_bfloat16 *__restrict__ src, int n_rows, int K, int r0, int k0, int rows, uint8_t *dst, uint32_t lbo,
    uint32_t sbo)
{
    // 16-byte units: (row, 8-element K group)
    const int groups = kGemmK / 8;
    for (int u = threadIdx.x; u < rows * groups; u += blockDim.x)
    {
        const int r = u / groups, g = u % groups;
        const int gr = r0 + r, gk = k0 + g * 8;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (gr < n_rows)
        {
            if (gk + 8 <= K && (reinterpret_cast<uintptr_t>(src + static_cast<size_t>(gr) * K + gk) & 15u) == 0)
            {
                v = *reinterpret_cast<const uint4 *>(src + static_cast<size_t>(gr) * K + gk);
            }
            else
            {
                __nv_bfloat16 tmp[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    tmp[e] = (gk + e < K) ? src[static_cast<size_t>(gr) * K + gk + e] : __float2bfloat16(0.0f);
                v = *reinterpret_cast<uint4 *>(tmp);
            }
        }
        *reinterpret_cast<uint4 *>(dst + tc::core_offset(r, g * 8, lbo, sbo)) = v;
    }
}

__global__ void __launch_bounds__(128) gemm_tn_kernel(
    const __nv_bfloat16 *__restrict__ A, const __nv_bfloat16 *__restrict__ B, float *__restrict__ D, int M, int N,
    int K, unsigned int *err)
{
    __shared__ __align__(128) uint8_t sa[kGemmM * kGemmK * 2];
    __shared__ __align__(128) uint8_t sb[kGemmN * kGemmK * 2];
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t mbar;
    const int m0 = blockIdx.x * kGemmM, n0 = blockIdx.y * kGemmN;
    const uint32_t lbo = 128, sbo_a = (kGemmK / 8) * 128, sbo_b = (kGemmK / 8) * 128;
    if (threadIdx.x < 32) tc::tmem_alloc(&tmem_slot, kGemmN);
    if (threadIdx.x == 0) tc::mbar_init(&mbar, 1);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    constexpr uint32_t idesc = tc::idesc_bf16_f32(kGemmM, kGemmN);
    bool ok = true;
    uint32_t phase = 0;
    for (int k0 = 0; k0 < K; k0 += kGemmK)
    {
        stage_tile(A, M, K, m0, k0, kGemmM, sa, lbo, sbo_a);
        stage_tile(B, N, K, n0, k0, kGemmN, sb, lbo, sbo_b);
        tc::fence_async_smem();
        __syncthreads();
        if (threadIdx.x == 0)
        {
            tc::fence_after_sync();
            for (int j = 0; j < kGemmK / 16; ++j)
            {
                const uint64_t da = tc::smem_desc(tc::smem_u32(sa) + j * 256, lbo, sbo_a);
                const uint64_t db = tc::smem_desc(tc::smem_u32(sb) + j * 256, lbo, sbo_b);
                tc::mma_bf16(tmem, da, db, idesc, (k0 > 0 || j > 0) ? 1u : 0u);
            }
            tc::commit(&mbar);
        }
        // Every thread waits for the MMAs of this chunk before the buffers are overwritten; the
        // outcome is made block-uniform so that no warp-collective instruction runs partially.
        const bool waited = tc::mbar_wait(&mbar, phase, kWaitLimit);
        phase ^= 1u;
        tc::fence_after_sync();
        ok = (__syncthreads_and(waited ? 1 : 0) != 0) && ok;
    }
    if (!ok)
    {
        if (threadIdx.x == 0) atomicOr(err, 1u);
    }
    else
    {
        const int row = m0 + (threadIdx.x >> 5) * 32 + (threadIdx.x & 31);
        const uint32_t lane_base = static_cast<uint32_t>((threadIdx.x >> 5) * 32) << 16;
        for (int c = 0; c < kGemmN; c += 16)
        {
            float v[16];
            tc::tmem_ld16(tmem + lane_base + c, v);
            if (row < M)
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (n0 + c + i < N) D[static_cast<size_t>(row) * N + n0 + c + i] = v[i];
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) tc::tmem_dealloc(tmem, kGemmN);
}

}  // namespace

// The single-stage GEMM: any K and alignment (bf16_gemm_tn in gemm.cu takes it for shapes the
// pipelined kernel does not).
int bf16_gemm_tn_simple(const void *A, const void *B, float *D, int M, int N, int K, unsigned int *d_err, cudaStream_t s)
{
    if (M < 1 || N < 1 || K < 1 || !A || !B || !D || !d_err) return -1;
    dim3 grid((M + kGemmM - 1) / kGemmM, (N + kGemmN - 1) / kGemmN);
    gemm_tn_kernel<<<grid, 128, 0, s>>>(static_cast<const __nv_bfloat16 *>(A), static_cast<const __nv_bfloat16 *>(B),
                                        D, M, N, K, d_err);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace knp_gb300

// ------------------------------------------------------------------------------------------------
// Batched LIF network (batched / precision form).
//
// B independent samples of a feed-forward LIF network (layers of sizes n_0 -> n_1 -> ... -> n_L,
// all-to-all, delay 1). Semantics per neuron are the reference LIF
// (knp/backends/cpu/cpu-library/include/knp/backends/cpu-library/impl/populations/lif/lif_impl.h:33-86):
// outside the refractory period V = V * leak + I, spike iff V > threshold, then V = reset and the
// counter = period; inside it the counter counts down and input is ignored. Layer l's input at
// step t is the spikes of layer l - 1 at step t - 1 times W_l (delay 1); layer 0 is the input,
// whose spike of source i for sample b at step t is the counter-based Bernoulli draw
// rand64(key, (t * B + b) * n_0 + i) >> 11 < rate[b][i] * 2^53. Sample b runs steps [0, T_b).
//
// The network is feed-forward, so a layer's input of every step is known once the layer below has
// run all of its steps: the layers run one after another, and a layer is one matrix product over all
// (sample, step) columns with the LIF recurrence in its epilogue. The product is taken as
// D[neuron][column] = W[neuron][k] * S[column][k]: an accumulator row (tensor-memory lane) is one
// neuron and its columns are consecutive steps of one sample, so the thread that owns the lane runs
// the recurrence down its row with the membrane state in registers, and no step waits for another
// CTA. (Stepping all layers together, one step at a time, costs a chain of expansion, product,
// exchange and hand-over per step: 0.95 ms for 256 samples of 784-1000-1000-10 and 50-200 steps, the
// tensor cores idle for most of it; this form takes 0.218 ms.)
//
// Spikes travel between layers as bitmaps: per layer one row of wpad words (bit j of word w = neuron
// 32 w + j) for every (sample, step) of a segment of steps, a sample's rows consecutive:
// row_base[s] + j is what the step t0 + j of the layer above reads, i.e. the spikes of step
// t0 + j - 1. Long runs are cut into segments; LIF state and each sample's last spikes carry over.
namespace knp_gb300
{
namespace
{

constexpr int kMaxLayers = 4;
constexpr uint32_t kTileN = 128;  // neurons of a CTA (its accumulator rows); a CTA pair has two tiles
constexpr uint32_t kStreamCols = 128;  // columns of one stream in a tile (two streams per pair)
constexpr uint32_t kCols = 2 * kStreamCols;
constexpr uint32_t kChunk = 64;                          // K of a staged chunk
constexpr uint32_t kAChunk = kTileN * kChunk * 2;       // 16 KB of packed weights
constexpr uint32_t kBChunk = kStreamCols * kChunk * 2;  // 16 KB of expanded spikes, this CTA's stream
// A stage of the operand ring holds two chunks (weights of both, then spikes of both); the issuer
// spends as long on a wait and a commit as on two MMAs, so it waits once for eight of them.
constexpr uint32_t kLayerStage = 2 * (kAChunk + kBChunk);
constexpr int kMinStages = 2, kMaxStages = 4;  // operand ring depths the autotuner tries
constexpr int kMaxRing = 3;
constexpr int ring_stages(int depth) { return depth - 1; }
constexpr int kExpandWarps = 8, kScanWarps = 8, kRowWarps = 2;
constexpr int kExpandGroups = 2;  // groups of expander warps, one per chunk of a stage
constexpr uint32_t kGroupThreads = 32 * kExpandWarps / kExpandGroups;
constexpr int kIssuerWarp = 0, kCopyWarp = 1, kRowWarp0 = 2, kScanWarp0 = 4, kExpandWarp0 = kScanWarp0 + kScanWarps;
constexpr int kLayerThreads = 32 * (kExpandWarp0 + kExpandWarps);
constexpr uint32_t kRowSlots = 4;  // tiles of row indexes kept ahead of the expanders
constexpr uint32_t kDrainWait = 1u << 14;  // polls, about 0.06 s
static_assert(kGroupThreads == kStreamCols, "an expander thread has one row of a chunk");
constexpr uint32_t kTmemCols = 512;  // two accumulators of kCols columns per CTA
constexpr uint32_t kScanCols = 32;   // columns a scan thread reads from its accumulator at a time
constexpr uint32_t kPad = 8;         // a sample's columns in a stream are padded to a multiple of this
constexpr uint32_t kNoRow = 0xFFFFFFFFu;
constexpr uint32_t kMaxFanIn = 2048;
constexpr size_t kMinDynSmem = size_t(120) << 10;  // one CTA per SM (a second would wait for tensor memory)
constexpr size_t kRowBudget = size_t(256) << 20;   // bytes of a layer's rows per segment
constexpr uint32_t kMaxTiles = 512;  // see the size limit in batched_plan_create

// What one launch of a layer needs. A stream is a list of samples whose columns follow one another;
// CTA pair (pair of n tiles, g) runs streams 2 g and 2 g + 1 side by side, one per half of its columns:
// each CTA expands one stream's spikes and scans its own neurons in both.
struct LayerArgs
{
    CUtensorMap w;            // packed weights as rows of kChunk elements: block [n tile][chunk] is 128 rows
    const uint32_t *bits_in;  // rows of the layer below
    uint32_t wp_in;           // words per row (a multiple of 4)
    uint32_t *bits_out;       // this layer's rows (null for the last layer)
    uint32_t wp_out;
    uint32_t n;               // neurons
    uint32_t kp;              // fan-in rounded up to 16
    uint32_t chunks;          // ceil(kp / kChunk)
    uint32_t n_groups;        // CTA pairs per pair of neuron tiles
    float leak, thr, reset;
    uint32_t refract;
    const uint32_t *st_off;   // [2 n_groups + 1] first entry of each stream
    const uint32_t *st_len;   // [2 n_groups] columns of each stream (padding included)
    const uint32_t *st_start;  // per entry: the sample's first column in its stream
    const uint4 *st_info;     // per entry: sample, its first row, its columns in this segment, its steps in all
    const uint32_t *own_size, *next_size;  // per-sample sizes of this layer and of the next, or null
    uint32_t next_n;          // fan-out of a spike (0 for the last layer)
    uint32_t t0, t1;
    uint32_t *carry;          // [batch][wp_out] last spikes of a sample that goes on in the next segment
    uint32_t *state;          // [batch][n][3] its potentials, refractory counters and spike counts
    int *counts;              // [batch][n], last layer only
    uint32_t *record;         // or null
    unsigned long long rec_off, rec_stride;
    uint32_t wn;              // words of a recorded row
    unsigned long long *events;
    unsigned int *err;        // bit 0: a wait gave up
    uint32_t poll_limit;
    uint32_t stall;           // failure test: the issuer waits for this many more expanders than exist
    uint32_t ring;            // stages of the operand ring
};

// Position p of a 16-wide K block holds input (p >> 1) + 8 (p & 1) of the block, in the packed
// weights and in the expanded spikes alike: one word of two BF16 elements then comes from bits i and
// 8 + i of the block's 16 spike bits, which one shift and one mask isolate.
__host__ __device__ constexpr uint32_t k_of(uint32_t p) { return (p >> 1) + 8u * (p & 1u); }

// Weights of one layer, BF16 [n][k] row-major (any k), to [n tile][chunk] blocks of 128 rows of 64
// elements, zero past n and k, which TMA loads with the 128-byte swizzle. One thread per 16 bytes.
// Repacked in every run (the caller may rewrite the weights between runs): 4 MB, 5 us at
// 784-1000-1000-10.
struct PackArgs
{
    const __nv_bfloat16 *w[kMaxLayers];
    uint8_t *out[kMaxLayers];
    uint32_t n[kMaxLayers], k[kMaxLayers], chunks[kMaxLayers];
    unsigned long long first[kMaxLayers + 1];  // first unit of each layer
    int n_layers;
};

__global__ void pack_weights_kernel(const __grid_constant__ PackArgs a)
{
    const unsigned long long total = a.first[a.n_layers];
    for (unsigned long long u = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; u < total;
         u += static_cast<unsigned long long>(gridDim.x) * blockDim.x)
    {
        int l = 0;
        while (u >= a.first[l + 1]) ++l;
        const unsigned long long v = u - a.first[l];
        const uint32_t slot = static_cast<uint32_t>(v & 7u);
        const uint32_t r = static_cast<uint32_t>((v >> 3) & (kTileN - 1));
        const unsigned long long blk = v >> 10;  // n tile * chunks + chunk
        const uint32_t chunk = static_cast<uint32_t>(blk % a.chunks[l]);
        const uint32_t row = static_cast<uint32_t>(blk / a.chunks[l]) * kTileN + r;
        __nv_bfloat16 e[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i)
        {
            const uint32_t k = chunk * kChunk + (slot >> 1) * 16u + k_of((slot & 1u) * 8u + i);
            e[i] = (row < a.n[l] && k < a.k[l]) ? a.w[l][static_cast<size_t>(row) * a.k[l] + k] : __float2bfloat16(0.0f);
        }
        *reinterpret_cast<uint4 *>(a.out[l] + blk * kAChunk + r * 128u + (slot << 4)) =
            *reinterpret_cast<uint4 *>(e);
    }
}

// The 53-bit threshold an input draw is compared with, rate * 2^53 truncated, computed exactly from
// the FP32 rate's fields (no FP64 on the device): m * 2^(e - 97) for a normal rate in (0, 1) with
// 24-bit significand m and biased exponent e; 0 for rates <= 0, subnormal or NaN; 2^53 (every draw is
// below it) for rates >= 1.
__device__ __forceinline__ unsigned long long rate_threshold(float rate)
{
    const uint32_t bits = __float_as_uint(rate);
    const uint32_t e = (bits >> 23) & 0xFFu;
    if (bits >> 31) return 0ull;
    if (e == 0xFFu) return (bits & 0x7FFFFFu) ? 0ull : 1ull << 53;  // NaN, +infinity
    if (e == 0u) return 0ull;
    const unsigned long long m = (bits & 0x7FFFFFu) | 0x800000u;
    if (e >= 127u) return 1ull << 53;
    if (e >= 97u) return m << (e - 97u);
    return 97u - e < 64u ? m >> (97u - e) : 0ull;
}

// Transposes a 32 x 32 bit matrix held one row per lane: afterwards bit j of lane c is what bit c of
// lane j was.
__device__ __forceinline__ uint32_t warp_transpose_bits(uint32_t x, uint32_t lane)
{
    uint32_t mask = 0x0000FFFFu;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1)
    {
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, m);
        x = (lane & m) ? ((x & ~mask) | ((y & ~mask) >> m)) : ((x & mask) | ((y & mask) << m));
        mask ^= mask << (m >> 1);
    }
    return x;
}

struct DrawArgs
{
    const float *rates;  // [batch][n_in]
    uint32_t n_in, wp, words, batch;
    const uint32_t *size0, *size1;  // per-sample sizes or null
    uint32_t n1;
    const uint4 *rows;  // per sample: first row, columns in this segment
    uint32_t t0, blocks;  // blocks of 32 rows per sample
    unsigned long long key;
    uint32_t *bits;
    uint32_t *record;
    unsigned long long rec_stride;
    unsigned long long *events;
};

// Layer 0's rows: row j of a sample = the inputs drawn at step t0 + j - 1 (zero before step 0), for j
// in [0, columns]. A warp takes one word (32 inputs, a lane each, the threshold in a register) of 32
// consecutive rows, a bit per row, and one transposition across the warp gives the rows' words; a draw is
// counted and recorded in the segment where it is not row 0. Bound by the draws' integer instructions (two
// 64-bit products each, half-rate pipes): one lane per input keeps the rate loads coalesced and one
// threshold serves 32 draws. 26 M draws: 49 us (one thread per word of 32 draws: 56 us).
__global__ void __launch_bounds__(256, 6) input_rows_kernel(const __grid_constant__ DrawArgs a)
{
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned long long items = static_cast<unsigned long long>(a.batch) * a.blocks * a.wp;
    const unsigned long long warps = static_cast<unsigned long long>(gridDim.x) * (blockDim.x >> 5);
    unsigned long long ev = 0;
    for (unsigned long long it = blockIdx.x * static_cast<unsigned long long>(blockDim.x >> 5) + (threadIdx.x >> 5);
         it < items; it += warps)
    {
        const uint32_t w = static_cast<uint32_t>(it % a.wp);
        const unsigned long long sb = it / a.wp;
        const uint32_t smp = static_cast<uint32_t>(sb / a.blocks), j0 = 32u * static_cast<uint32_t>(sb % a.blocks);
        const uint4 info = a.rows[smp];
        const uint32_t cols = info.y;
        if (cols == 0u || j0 > cols) continue;
        const uint32_t i = 32u * w + lane;
        const uint32_t lim = a.size0 ? min(a.n_in, a.size0[smp]) : a.n_in;
        const unsigned long long thr = i < lim ? rate_threshold(a.rates[static_cast<size_t>(smp) * a.n_in + i]) : 0ull;
        uint32_t word = 0;  // of row j0 + lane
        if (w < a.words)
        {
            const uint32_t n_rows = min(32u, cols + 1u - j0);
            // The draw of row j is that of step t0 + j - 1; row 0 of the first segment has none.
            const uint32_t c0 = a.t0 + j0 == 0u ? 1u : 0u;
            // rand64(key, ctr) with ctr * G + C carried from step to step by one addition; its first mixing
            // step y ^ (y >> 30) of y = x ^ key is x ^ (x >> 30) ^ (key ^ (key >> 30)); and (r >> 11) < thr
            // is r < thr << 11, which the high words decide unless they are equal (2^-32 of the draws), so
            // the last mixing step's low word is rarely formed.
            constexpr unsigned long long kG = 0x9E3779B97F4A7C15ull, kC = 0x632BE59BD9B4E019ull;
            const unsigned long long inc = static_cast<unsigned long long>(a.batch) * a.n_in * kG;
            const unsigned long long key1 = a.key ^ (a.key >> 30);
            unsigned long long x =
                ((static_cast<unsigned long long>(a.t0 + j0 + c0 - 1u) * a.batch + smp) * a.n_in + i) * kG + kC;
            const bool always = thr >> 53;  // thr << 11 would be 2^64
            const uint32_t t_hi = always ? 0xFFFFFFFFu : static_cast<uint32_t>(thr >> 21);
            const uint32_t t_lo = always ? 0xFFFFFFFFu : static_cast<uint32_t>(thr << 11);
            uint32_t fired = 0;  // bit c: this input fires in row j0 + c
            auto draw = [&](uint32_t c)
            {
                unsigned long long y = (x ^ (x >> 30) ^ key1) * 0xBF58476D1CE4E5B9ull;
                y = (y ^ (y >> 27)) * 0x94D049BB133111EBull;
                const uint32_t hi = static_cast<uint32_t>(y >> 32), r_hi = hi ^ (hi >> 31);
                if (r_hi < t_hi) fired |= 1u << c;
                if (r_hi == t_hi && (always || static_cast<uint32_t>(y ^ (y >> 31)) < t_lo)) fired |= 1u << c;
                x += inc;
            };
            if (c0 == 0u && n_rows == 32u)
            {
#pragma unroll
                for (uint32_t c = 0; c < 32; ++c) draw(c);
            }
            else
            {
                for (uint32_t c = c0; c < n_rows; ++c) draw(c);
            }
            word = warp_transpose_bits(fired, lane);
        }
        const uint32_t j = j0 + lane;
        if (j > cols) continue;
        a.bits[(static_cast<size_t>(info.x) + j) * a.wp + w] = word;
        if (j >= 1u && w < a.words)
        {
            if (a.record)
                a.record[static_cast<size_t>(a.t0 + j - 1u) * a.rec_stride + static_cast<size_t>(smp) * a.words + w] = word;
            ev += static_cast<unsigned long long>(__popc(word)) * (a.size1 ? a.size1[smp] : a.n1);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ev += __shfl_down_sync(0xffffffffu, ev, o);
    if (lane == 0 && ev) atomicAdd(a.events, ev);
}

// mbar_wait that also gives up as soon as another role of the CTA has.
__device__ __forceinline__ bool wait_or_fail(uint64_t *mbar, uint32_t parity, uint32_t limit, const volatile int *fail)
{
    for (uint32_t i = 0; i < limit; ++i)
    {
        if (tc::mbar_try_wait(mbar, parity)) return true;
        if (*fail) return false;
    }
    return false;
}

// wait_or_fail for a whole warp: one lane polls (32 lanes suspended on a barrier cost its other users),
// every lane gets the outcome. The whole warp calls it.
__device__ __forceinline__ bool warp_wait(uint64_t *mbar, uint32_t parity, uint32_t limit, const volatile int *fail,
                                          uint32_t lane)
{
    int ok = 1;
    if (lane == 0) ok = wait_or_fail(mbar, parity, limit, fail);
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// The 16 spike bits `h` of a K block as its 16 BF16 elements (8 words): word i = bit i in the low half
// and bit 8 + i in the high half, as 1.0 (0x3F80 = 127 << 7) or 0.
__device__ __forceinline__ void expand16(uint32_t h, uint32_t *v)
{
    const uint32_t z = __byte_perm(h, 0u, 0x4140);  // byte 0 to the low half, byte 1 to the high half
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = ((z << (7 - i)) & 0x00800080u) * 127u;
}

__device__ __forceinline__ void st_shared_v4(uint32_t dst, const uint32_t *v)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
                 : "memory");
}

// One scan warp's share of a layer: 32 neurons of one stream.
struct ScanTarget
{
    uint32_t tmem;      // its lanes and its stream's columns of accumulator 0
    uint32_t off, len;  // its stream's first entry and its columns
    uint32_t neuron, wq;  // this thread's neuron, the warp's word in a row
    uint32_t n_tiles;
    uint32_t acc_empty;  // the even CTA's acc_empty barriers (shared::cluster address)
};

// The LIF recurrence of one stream down its accumulator columns (lif_impl.h:33-86: leak and input only
// outside the refractory period; strict '>'; reset to a value). A thread reads kScanCols columns at a
// time and collects its spikes as one word, a bit per column; a transposition across the warp turns 32
// neurons' words into the columns' bitmap words, so a step costs five instructions and no vote. A
// sample's columns are padded to a multiple of kPad, so that kPad steps at a time need no check
// for its end. Returns false if a wait gave up.
template <bool kRefract, bool kLeak>
__device__ __forceinline__ bool scan_stream(const LayerArgs &a, const ScanTarget &tgt, uint32_t lane, uint64_t *acc_full,
                                            const volatile int *fail, unsigned long long &events)
{
    const float leak = a.leak, thr = a.thr, reset = a.reset;
    // The sample being scanned (sample, first row, columns, steps in all), its next step (from t0), and
    // this neuron's state; the next sample's entry is loaded ahead.
    uint32_t entry = tgt.off, j = 0, fan = 0;
    uint4 info = make_uint4(0, 0, 0, 0), next = info;
    bool exists = false;
    float V = 0.0f;
    bool spiked = false;
    const float reset_leak = __fmul_rn(reset, leak);
    float limit = thr;  // thr, or +infinity for a neuron its sample does not have
    uint32_t RC = 0, count = 0, last_word = 0;
    uint32_t end = 0;  // the stream column after the sample's last (padded)
    auto open_sample = [&]()
    {
        info = next;
        j = 0;
        end += (info.z + kPad - 1) / kPad * kPad;
        if (end < tgt.len) next = a.st_info[entry + 1];
        const uint32_t smp = info.x;
        exists = tgt.neuron < (a.own_size ? a.own_size[smp] : a.n);
        limit = exists ? thr : __int_as_float(0x7F800000);
        spiked = false;
        fan = a.next_size ? a.next_size[smp] : a.next_n;
        V = 0.0f;
        RC = count = 0;
        if (a.t0 != 0u && tgt.neuron < a.n)
        {
            const uint32_t *st = a.state + (static_cast<size_t>(smp) * a.n + tgt.neuron) * 3;
            V = __uint_as_float(st[0]);
            RC = st[1];
            count = st[2];
        }
        // The row before the segment's first step: the last spikes of the previous segment.
        if (a.bits_out && lane == 0)
            a.bits_out[static_cast<size_t>(info.y) * a.wp_out + tgt.wq] =
                a.t0 ? a.carry[static_cast<size_t>(smp) * a.wp_out + tgt.wq] : 0u;
    };
    auto close_sample = [&]()
    {
        const uint32_t smp = info.x;
        if (info.w <= a.t1)
        {
            if (a.counts && tgt.neuron < a.n)
                a.counts[static_cast<size_t>(smp) * a.n + tgt.neuron] = static_cast<int>(count);
        }
        else
        {
            if (tgt.neuron < a.n)
            {
                uint32_t *st = a.state + (static_cast<size_t>(smp) * a.n + tgt.neuron) * 3;
                st[0] = __float_as_uint(spiked ? reset : V);
                st[1] = RC;
                st[2] = count;
            }
            if (a.bits_out && lane == 0) a.carry[static_cast<size_t>(smp) * a.wp_out + tgt.wq] = last_word;
        }
        ++entry;
    };
    if (tgt.len)
    {
        next = a.st_info[entry];
        open_sample();
    }
    for (uint32_t tile = 0; tile < tgt.n_tiles; ++tile)
    {
        const uint32_t acc = tile & 1u;
        if (!warp_wait(&acc_full[acc], (tile >> 1) & 1u, a.poll_limit, fail, lane)) return false;
        tc::fence_after_sync();
        const uint32_t p0 = tile * kStreamCols;
        const uint32_t valid = tgt.len > p0 ? min(kStreamCols, tgt.len - p0) : 0u;  // a multiple of kPad
        for (uint32_t c0 = 0; c0 < kStreamCols; c0 += kScanCols)
        {
            const uint32_t here = valid > c0 ? min(kScanCols, valid - c0) : 0u;  // uniform
            float x[kScanCols];
            if (here) tc::tmem_ld32(tgt.tmem + acc * kCols + c0, x);
            if (here < kScanCols || c0 + kScanCols == kStreamCols)
            {
                // The last columns of this tile are in registers: the accumulator may be reused.
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive_cluster(tgt.acc_empty + acc * 8u);
            }
            if (!here) break;
            uint32_t bits = 0;  // bit c: this neuron fired at column c0 + c
            // V is the potential before its reset: `spiked` says whether the last step reset it. The sum
            // with the reset value is formed beside the sum with the kept one, so the chain from step to
            // step is a product (leak only; V * 1 is V), a sum and a choice.
            auto step = [&](uint32_t c)
            {
                if (kRefract)
                {
                    const float v = __fadd_rn(__fmul_rn(V, leak), x[c]);
                    const bool free_ = RC == 0u;
                    const bool spike = exists && free_ && v > thr;
                    V = spike ? reset : (free_ ? v : V);
                    RC = spike ? a.refract : (free_ ? 0u : RC - 1u);
                    if (spike) bits |= 1u << c;
                }
                else
                {
                    const float kept = __fadd_rn(kLeak ? __fmul_rn(V, leak) : V, x[c]);
                    const float fresh = __fadd_rn(reset_leak, x[c]);
                    V = spiked ? fresh : kept;
                    spiked = V > limit;
                    if (spiked) bits |= 1u << c;
                }
            };
            // Columns [from, to) of this block, steps j0 .. of the sample, are done: their bitmap words go
            // out, one lane each.
            auto flush = [&](uint32_t from, uint32_t to, uint32_t j0)
            {
                const uint32_t span = to - from == 32u ? 0xFFFFFFFFu : ((1u << (to - from)) - 1u) << from;
                count += __popc(bits & span);
                const uint32_t word = warp_transpose_bits(bits & span, lane);
                last_word = __shfl_sync(0xffffffffu, word, static_cast<int>(to - 1u));
                if (lane >= from && lane < to)
                {
                    const uint32_t jj = j0 + (lane - from);
                    if (a.bits_out)
                    {
                        a.bits_out[(static_cast<size_t>(info.y) + jj + 1u) * a.wp_out + tgt.wq] = word;
                        events += static_cast<unsigned long long>(__popc(word)) * fan;
                    }
                    if (a.record && tgt.wq < a.wn)
                        a.record[static_cast<size_t>(a.t0 + jj) * a.rec_stride + a.rec_off +
                                 static_cast<size_t>(info.x) * a.wn + tgt.wq] = word;
                }
            };
            uint32_t from = 0, j_from = j;  // first column not flushed, and its step
#pragma unroll
            for (uint32_t sb = 0; sb < kScanCols; sb += kPad)
            {
                if (sb >= here) break;
                const uint32_t left = info.z - j;
                if (left >= kPad)
                {
#pragma unroll
                    for (uint32_t i = 0; i < kPad; ++i) step(sb + i);
                    j += kPad;
                }
                else
                {
#pragma unroll
                    for (uint32_t i = 0; i < kPad; ++i)
                        if (i < left) step(sb + i);
                    j += left;
                }
                if (j == info.z)
                {
                    flush(from, sb + min(left, kPad), j_from);
                    close_sample();
                    if (p0 + c0 + sb + kPad < tgt.len) open_sample();
                    from = sb + kPad;
                    j_from = 0;
                }
            }
            if (from < here) flush(from, here, j_from);
            if (here < kScanCols) break;
        }
    }
    return true;
}

// One layer over a segment of steps, on CTA pairs. Roles in each CTA: warp 0 issues the pair's MMAs (even
// rank; M = 256 neurons, N = 256 columns, FP32 accumulators in tensor memory, two of them, so the scan of a
// tile runs beside the product of the next), warp 1 copies packed weight chunks, warps 2-3 look up the
// columns' spike rows a few tiles ahead, warps 4-11 scan (thread = neuron; 4-7 the first stream's half of
// the accumulator, 8-11 the second's), warps 12-19 expand this CTA's stream into the BF16 operand. Every wait
// is bounded; a wait that gives up sets bit 0 of *err and stops the roles of both CTAs, copies and MMAs in
// flight land, and the tensor memory is freed.
// A pair rather than one CTA per tile: each CTA expands one stream instead of both, and shared memory
// carries 128 KB per 128-deep stage instead of 192 KB (1024 cycles of tensor work either way). 256 samples of
// 784-1000-1000-10, 50-200 steps: the three layers take 66, 73 and 27 us (one CTA per 128 x 256 tile: 93,
// 112, 33); what is left above the tensor time (about 58 us in all) is a stage's hand-over (wait, eight MMAs
// and commit take the issuing thread about as long as they run), the scan (about 60 cycles a step beside the
// expansion) and some 10 us of start and end per launch.
__global__ void __launch_bounds__(kLayerThreads, 1) __cluster_dims__(2, 1, 1)
    lif_layer_kernel(const __grid_constant__ LayerArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    // Of the even CTA alone: full (both CTAs' weights and spikes of a stage are in place: its copy warp's
    // arrival with the bytes of both, and one arrival per expander group) and acc_empty (the scan warps of
    // both). Of each CTA: empty, acc_full and drain (commits reach both), the row indexes.
    __shared__ __align__(8) uint64_t full[kMaxRing], empty[kMaxRing];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], drain;
    __shared__ __align__(8) uint64_t row_full[kRowSlots], row_empty[kRowSlots];
    __shared__ uint32_t s_row[kRowSlots][kStreamCols];  // a column's row of bits_in, or kNoRow
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    __shared__ unsigned long long s_events;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t rank = tc::cluster_rank();
    const uint32_t pair = blockIdx.x >> 1;
    const uint32_t n_pair = pair / a.n_groups, group = pair - n_pair * a.n_groups;
    const uint32_t n_tile = 2 * n_pair + rank;
    const uint32_t peer_fail = tc::mapa(tc::smem_u32(&s_fail), rank ^ 1u);
    auto fail = [&]()
    {
        s_fail = 1;
        tc::st_cluster_u32(peer_fail, 1u);
        atomicOr(a.err, 1u);
    };
    if (warp == kIssuerWarp) tc::tmem_alloc_pair(&tmem_slot, kTmemCols);
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < kMaxRing; ++s)
        {
            tc::mbar_init(&full[s], 1 + 2 * kExpandGroups + a.stall);
            tc::mbar_init(&empty[s], 1);
        }
        for (int i = 0; i < 2; ++i)
        {
            tc::mbar_init(&acc_full[i], 1);
            tc::mbar_init(&acc_empty[i], 2 * kScanWarps);
        }
        for (uint32_t i = 0; i < kRowSlots; ++i)
        {
            tc::mbar_init(&row_full[i], kRowWarps);
            tc::mbar_init(&row_empty[i], kExpandWarps);
        }
        tc::mbar_init(&drain, 1);
        s_events = 0;
        s_fail = 0;
    }
    // Everything above overlaps the preceding kernel; from here on its results are read.
    pdl_begin();
    __syncthreads();
    if (threadIdx.x == 0 && *reinterpret_cast<volatile unsigned int *>(a.err) != 0u) s_fail = 1;
    tc::fence_before_sync();
    tc::cluster_sync();  // both CTAs' barriers and tensor memory are set up
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    const uint32_t base = (tc::smem_u32(smem) + 1023u) & ~1023u;  // swizzle atoms on 1024-byte boundaries
    const uint32_t ring = a.ring, chunks = a.chunks, per_tile = (chunks + 1) / 2;  // stages of a tile
    const uint32_t n_tiles =
        (max(a.st_len[2 * group], a.st_len[2 * group + 1]) + kStreamCols - 1) / kStreamCols;
    unsigned long long my_events = 0;

    if (warp >= kExpandWarp0)
    {
        // Expanders: group g of four warps expands chunk g of every stage, a thread one of its 128 rows.
        const uint32_t e = threadIdx.x - 32 * kExpandWarp0, r = e & (kStreamCols - 1), sw = r & 7u;
        const uint32_t g = e / kGroupThreads;
        const uint32_t full0 = tc::mapa(tc::smem_u32(full), 0);
        const uint32_t dst0 = base + 2 * kAChunk + g * kBChunk + r * 128u;
        bool ok = true;
        // The stage being loaded (tile lt, stage lc of it) runs one ahead of the one being expanded.
        uint32_t lt = 0, lc = 0;
        const uint32_t *row = nullptr;
        auto open_tile = [&]()
        {
            row = nullptr;
            if (lt >= n_tiles || !ok) return;
            const uint32_t slot = lt % kRowSlots;
            if (!warp_wait(&row_full[slot], (lt / kRowSlots) & 1u, a.poll_limit, &s_fail, lane))
            {
                ok = false;
                return;
            }
            const uint32_t q = s_row[slot][r];
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&row_empty[slot]);
            if (q != kNoRow) row = a.bits_in + static_cast<size_t>(q) * a.wp_in + 2 * g;
        };
        // Rows are padded to whole stages (wp_in is a multiple of 4 words).
        auto load = [&]() { return row ? __ldcg(reinterpret_cast<const uint2 *>(row + 4 * lc)) : make_uint2(0, 0); };
        open_tile();
        uint32_t s = 0, ph = 1;  // the stage and its parity (the first pass finds it free)
        bool have = n_tiles > 0;
        uint2 h = have ? load() : make_uint2(0, 0);
        while (have)
        {
            const uint2 now = h;
            if (++lc == per_tile)
            {
                lc = 0;
                ++lt;
                open_tile();
            }
            have = lt < n_tiles;
            if (have) h = load();
            ok = ok && warp_wait(&empty[s], ph, a.poll_limit, &s_fail, lane);
            if (ok)
            {
                const uint32_t dst = dst0 + s * kLayerStage;
#pragma unroll
                for (uint32_t b = 0; b < 4; ++b)
                {
                    uint32_t v[8];
                    const uint32_t word = b < 2 ? now.x : now.y;
                    expand16((b & 1u) ? word >> 16 : word, v);
                    st_shared_v4(dst + (((2 * b) ^ sw) << 4), v);
                    st_shared_v4(dst + (((2 * b + 1) ^ sw) << 4), v + 4);
                }
            }
            tc::fence_async_smem();
            // The group's decision is uniform; one thread tells the issuer.
            if (!tc::named_sync_and(1 + g, kGroupThreads, ok))
            {
                ok = false;
                break;
            }
            if (r == 0) tc::mbar_arrive_cluster(full0 + s * 8u);
            if (++s == ring)
            {
                s = 0;
                ph ^= 1u;
            }
        }
        if (!ok && lane == 0) fail();
    }
    else if (warp >= kScanWarp0)
    {
        const uint32_t half = (warp - kScanWarp0) >> 2;
        const uint32_t stream = 2 * group + half;
        ScanTarget tgt;
        tgt.tmem = tmem + ((32u * (warp & 3u)) << 16) + half * kStreamCols;
        tgt.off = a.st_off[stream];
        tgt.neuron = n_tile * kTileN + 32u * (warp & 3u) + lane;
        tgt.wq = 4u * n_tile + (warp & 3u);
        // A tile wholly past the layer (an odd number of tiles): nothing to scan.
        tgt.len = n_tile * kTileN < a.n ? a.st_len[stream] : 0u;
        tgt.n_tiles = n_tiles;
        tgt.acc_empty = tc::mapa(tc::smem_u32(acc_empty), 0);
        const bool ok = a.refract         ? scan_stream<true, true>(a, tgt, lane, acc_full, &s_fail, my_events)
                        : a.leak == 1.0f ? scan_stream<false, false>(a, tgt, lane, acc_full, &s_fail, my_events)
                                         : scan_stream<false, true>(a, tgt, lane, acc_full, &s_fail, my_events);
        if (!ok && lane == 0) fail();
    }
    else if (warp >= kRowWarp0)
    {
        // Row lookups of this CTA's stream: each thread two columns of a tile.
        const uint32_t stream = 2 * group + rank;
        const uint32_t off = a.st_off[stream], entries = a.st_off[stream + 1] - off, len = a.st_len[stream];
        bool ok = true;
        for (uint32_t tile = 0; tile < n_tiles && ok; ++tile)
        {
            const uint32_t slot = tile % kRowSlots;
            uint32_t found[2];
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i)
            {
                const uint32_t p = tile * kStreamCols + (threadIdx.x - 32 * kRowWarp0) + 64 * i;
                found[i] = kNoRow;
                if (p < len)
                {
                    uint32_t lo = 0, hi = entries;  // the last entry that starts at or before p
                    while (hi - lo > 1)
                    {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (a.st_start[off + mid] <= p) lo = mid;
                        else hi = mid;
                    }
                    const uint4 info = a.st_info[off + lo];
                    const uint32_t j = p - a.st_start[off + lo];
                    if (j < info.z) found[i] = info.y + j;
                }
            }
            ok = warp_wait(&row_empty[slot], ((tile / kRowSlots) & 1u) ^ 1u, a.poll_limit, &s_fail, lane);
            if (!ok) break;
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) s_row[slot][(threadIdx.x - 32 * kRowWarp0) + 64 * i] = found[i];
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&row_full[slot]);
        }
        if (!ok && lane == 0) fail();
    }
    else if (warp == kCopyWarp)
    {
        if (lane == 0)
        {
            const uint32_t full0 = tc::mapa(tc::smem_u32(full), 0);
            const uint32_t total = n_tiles * per_tile;
            const int y0 = static_cast<int>(n_tile * chunks * kTileN);  // past the weights: zeros
            uint32_t issued = 0;
            for (uint32_t u = 0, c = 0, s = 0, ph = 1; u < total; ++u)
            {
                if (!wait_or_fail(&empty[s], ph, a.poll_limit, &s_fail))
                {
                    fail();
                    break;
                }
                const bool two = c + 1 < chunks;
                if (rank == 0) tc::mbar_expect_tx(&full[s], two ? 4 * kAChunk : 2 * kAChunk);
                const uint32_t dst = base + s * kLayerStage;
                tc::tma_load_2d_pair(dst, &a.w, 0, y0 + static_cast<int>(c * kTileN), full0 + s * 8u);
                if (two)
                    tc::tma_load_2d_pair(dst + kAChunk, &a.w, 0, y0 + static_cast<int>((c + 1) * kTileN), full0 + s * 8u);
                issued = u + 1;
                c = c + 2 < chunks ? c + 2 : 0;
                if (++s == ring)
                {
                    s = 0;
                    ph ^= 1u;
                }
            }
            // After a failure: both CTAs' copies in flight land before either leaves (bounded; a chunk that
            // not every role reached does not complete, so the limit is short).
            if (s_fail && rank == 0)
                for (uint32_t u = issued > ring ? issued - ring : 0u; u < issued; ++u)
                    tc::mbar_wait(&full[u % ring], (u / ring) & 1u, kDrainWait);
        }
    }
    else if (lane == 0 && rank == 0)
    {
        constexpr uint32_t idesc = tc::idesc_bf16_f32(2 * kTileN, kCols);
        const uint64_t d_w = tc::smem_desc_sw128(base, 1024), d_s = tc::smem_desc_sw128(base + 2 * kAChunk, 1024);
        bool stop = false;
        uint32_t s = 0, ph = 0;
        for (uint32_t tile = 0; tile < n_tiles && !stop; ++tile)
        {
            const uint32_t acc = tile & 1u;
            if (tile >= 2 && !wait_or_fail(&acc_empty[acc], ((tile >> 1) - 1u) & 1u, a.poll_limit, &s_fail))
            {
                stop = true;
                break;
            }
            const uint32_t d_acc = tmem + acc * kCols;
            for (uint32_t c = 0; c < per_tile; ++c)
            {
                if (!wait_or_fail(&full[s], ph, a.poll_limit, &s_fail))
                {
                    stop = true;
                    break;
                }
                tc::fence_after_sync();
                // The stage's descriptors follow from the first one's by their start addresses (in
                // 16-byte units).
                const uint64_t dw = d_w + s * (kLayerStage >> 4), ds = d_s + s * (kLayerStage >> 4);
                const uint32_t blocks = (a.kp - c * 2 * kChunk) >> 4;
                tc::mma_bf16_pair(d_acc, dw, ds, idesc, c ? 1u : 0u);
                if (blocks >= 8)
                {
#pragma unroll
                    for (uint32_t b = 1; b < 8; ++b)
                        tc::mma_bf16_pair(d_acc, dw + (b >> 2) * (kAChunk >> 4) + 2 * (b & 3u),
                                          ds + (b >> 2) * (kBChunk >> 4) + 2 * (b & 3u), idesc, 1u);
                }
                else
                {
                    for (uint32_t b = 1; b < blocks; ++b)
                        tc::mma_bf16_pair(d_acc, dw + (b >> 2) * (kAChunk >> 4) + 2 * (b & 3u),
                                          ds + (b >> 2) * (kBChunk >> 4) + 2 * (b & 3u), idesc, 1u);
                }
                tc::commit_pair(&empty[s]);
                if (c + 1 == per_tile) tc::commit_pair(&acc_full[acc]);
                if (++s == ring)
                {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
        if (stop) fail();
        // Every issued MMA completes (bounded wait) before the tensor memory is freed.
        tc::commit_pair(&drain);
        if (!tc::mbar_wait(&drain, 0, kWaitLimit)) fail();
    }
    else if (lane == 0)
    {
        // Odd rank: the issuer's last arrivals reach this CTA before it leaves.
        if (!tc::mbar_wait(&drain, 0, kWaitLimit)) fail();
    }
    __syncwarp();
    if (my_events) atomicAdd(&s_events, my_events);
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0 && s_events) atomicAdd(a.events, s_events);
    // Neither CTA leaves while the other's MMAs may read its shared memory or arrivals may reach it.
    tc::cluster_sync();
    if (warp == kIssuerWarp) tc::tmem_dealloc_pair(tmem, kTmemCols);
}

// Pinned words that runs leave their totals in: one page of them for the process, handed out two words a plan (pinning
// a plan's own costs 130 us and unpinning it 160, as much as the rest of a small plan's life); plans past its 256 have
// their own.
class PinnedTotals
{
public:
    unsigned long long *take()
    {
        std::lock_guard<std::mutex> lock(mu_);
        if (!page_)
        {
            if (cudaHostAlloc(reinterpret_cast<void **>(&page_), kSlots * 16, cudaHostAllocPortable) != cudaSuccess)
                return page_ = nullptr;
            for (int i = kSlots; i-- > 0;) free_.push_back(page_ + 2 * i);
        }
        unsigned long long *p = nullptr;
        if (free_.empty())
            return cudaHostAlloc(reinterpret_cast<void **>(&p), 16, cudaHostAllocPortable) == cudaSuccess ? p : nullptr;
        p = free_.back();
        free_.pop_back();
        return p;
    }
    void give_back(unsigned long long *p)
    {
        std::lock_guard<std::mutex> lock(mu_);
        if (p >= page_ && p < page_ + 2 * kSlots)
            free_.push_back(p);
        else
            cudaFreeHost(p);
    }

private:
    static constexpr int kSlots = 256;
    std::mutex mu_;
    unsigned long long *page_ = nullptr;
    std::vector<unsigned long long *> free_;
};
PinnedTotals &pinned_totals()
{
    static PinnedTotals *t = new PinnedTotals();  // outlives every plan
    return *t;
}

}  // namespace

// A batch prepared once and run as one CUDA-graph launch: a memset of the run's totals, the weight
// packing, then per segment of steps the input draws and one kernel per layer. Reusable: every run
// starts from zero state, so repeated runs of the same plan give identical results.
struct BatchedPlan
{
    struct Segment
    {
        DrawArgs draw{};
        LayerArgs layer[kMaxLayers]{};
        unsigned grid[kMaxLayers]{};
    };
    int n_layers = 0;
    std::vector<Segment> segs;
    PackArgs pack{};
    cudaStream_t caller = nullptr;  // the caller's stream: a run starts after its queued work
    cudaStream_t stream = nullptr;  // the plan's own stream (graphs cannot be captured on the legacy stream)
    cudaEvent_t ready = nullptr, begin = nullptr, end = nullptr;
    uint8_t *memory = nullptr;  // all of the plan's buffers and tables
    unsigned long long *totals = nullptr;       // device: events, then the error word
    unsigned long long *totals_host = nullptr;  // pinned copy, written by the run
    uint32_t *record = nullptr;
    size_t record_bytes = 0;
    cudaGraphExec_t exec = nullptr;
    int stages = 0;
    float tune_ms[kMaxStages + 1] = {};  // by operand ring depth

    ~BatchedPlan()
    {
        if (exec) cudaGraphExecDestroy(exec);
        if (stream) cudaStreamSynchronize(stream);
        if (memory) cudaFree(memory);
        if (totals_host) pinned_totals().give_back(totals_host);
        if (ready) cudaEventDestroy(ready);
        if (begin) cudaEventDestroy(begin);
        if (end) cudaEventDestroy(end);
        if (stream) cudaStreamDestroy(stream);
    }
};

namespace
{

size_t smem_bytes(int stages) { return std::max(ring_stages(stages) * size_t(kLayerStage) + 1024, kMinDynSmem); }

// Captures one run with a ring of `stages` chunks into p.exec.
cudaError_t capture(BatchedPlan &p, int stages)
{
    if (p.exec)
    {
        cudaGraphExecDestroy(p.exec);
        p.exec = nullptr;
    }
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const size_t smem = smem_bytes(stages);
    cudaError_t err = allow_dynamic_smem(lif_layer_kernel);
    if (err != cudaSuccess) return err;
    cudaStream_t s = p.stream;
    err = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    if (err != cudaSuccess) return err;
    cudaError_t lerr = cudaSuccess;
    auto note = [&](cudaError_t e)
    {
        if (lerr == cudaSuccess) lerr = e;
    };
    note(cudaMemsetAsync(p.totals, 0, 16, s));
    if (p.record) note(cudaMemsetAsync(p.record, 0, p.record_bytes, s));
    const unsigned long long units = p.pack.first[p.pack.n_layers];
    pack_weights_kernel<<<static_cast<unsigned>(std::min<unsigned long long>((units + 255) / 256, 16ull * sms)), 256, 0,
                          s>>>(p.pack);
    note(cudaGetLastError());
    for (auto &seg : p.segs)
    {
        const unsigned long long warps = static_cast<unsigned long long>(seg.draw.batch) * seg.draw.blocks * seg.draw.wp;
        input_rows_kernel<<<static_cast<unsigned>(std::min<unsigned long long>((warps + 7) / 8, 1ull << 20)), 256, 0, s>>>(
            seg.draw);
        note(cudaGetLastError());
        for (int l = 0; l < p.n_layers; ++l)
        {
            LayerArgs a = seg.layer[l];
            a.ring = static_cast<uint32_t>(ring_stages(stages));
            note(launch_pdl(lif_layer_kernel, dim3(seg.grid[l]), dim3(kLayerThreads), smem, s, a));
        }
    }
    note(cudaMemcpyAsync(p.totals_host, p.totals, 16, cudaMemcpyDeviceToHost, s));
    cudaGraph_t g = nullptr;
    err = cudaStreamEndCapture(s, &g);
    if (lerr != cudaSuccess) err = lerr;
    if (err == cudaSuccess) err = cudaGraphInstantiate(&p.exec, g, 0);
    if (g) cudaGraphDestroy(g);
    if (err == cudaSuccess) p.stages = stages;
    return err;
}

cudaError_t launch_timed(BatchedPlan &p, float *ms)
{
    // Order the run after the caller's queued work (weights, rates written on its stream).
    cudaError_t err = cudaEventRecord(p.ready, p.caller);
    if (err == cudaSuccess) err = cudaStreamWaitEvent(p.stream, p.ready, 0);
    if (err == cudaSuccess) err = cudaEventRecord(p.begin, p.stream);
    if (err == cudaSuccess) err = cudaGraphLaunch(p.exec, p.stream);
    if (err == cudaSuccess) err = cudaEventRecord(p.end, p.stream);
    if (err == cudaSuccess) err = cudaEventSynchronize(p.end);
    float t = 0.f;
    if (err == cudaSuccess) err = cudaEventElapsedTime(&t, p.begin, p.end);
    if (ms) *ms = t;
    return err;
}

}  // namespace

// Prepares a batch. Host arrays: sizes[n_layers + 1], leak/threshold/reset/refract[n_layers],
// steps[batch], sample_sizes[(n_layers + 1) * batch] (layer-major, optional); device arrays:
// weights[l] (BF16 [sizes[l + 1]][sizes[l]]), rates [batch][sizes[0]], counts [batch][sizes[n_layers]]
// and record (optional; layouts in knp_gb300.h). With `autotune` > 0, each operand ring depth is run
// twice and the fastest kept; < 0 uses depth -autotune; 0 the deepest. Every depth computes the same
// results. `segment_steps` > 0 caps the steps per segment (0: as many as the row budget allows).
int batched_plan_create(
    int n_layers, const uint32_t *sizes, const void *const *weights, const float *leak, const float *threshold,
    const float *reset, const uint32_t *refract, uint32_t batch, const uint32_t *steps, const uint32_t *sample_sizes,
    const float *rates, unsigned long long key, int *counts, uint32_t *record, int autotune, uint32_t segment_steps,
    cudaStream_t s, BatchedPlan **out, const char **why)
{
    *out = nullptr;
    if (n_layers < 1 || n_layers > kMaxLayers || batch == 0 || !sizes || !weights || !steps || !rates || !counts)
    {
        *why = "bad arguments";
        return -1;
    }
    std::unique_ptr<BatchedPlan> plan(new BatchedPlan());
    BatchedPlan &p = *plan;
    p.n_layers = n_layers;
    p.caller = s;
    if (cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&p.ready, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreate(&p.begin) != cudaSuccess || cudaEventCreate(&p.end) != cudaSuccess)
    {
        *why = "could not create the plan's stream";
        return -3;
    }
    // Failure test (KNP_GB300_BATCHED_STALL=1): the MMA issuer waits for one expander group more per chunk
    // than exists, so its first operand wait runs out (after a short poll limit) and the run ends with the
    // error word set instead of results.
    const char *stall_env = std::getenv("KNP_GB300_BATCHED_STALL");
    const uint32_t stall = (stall_env && stall_env[0] == '1') ? 1u : 0u;
    const uint32_t poll_limit = stall ? (1u << 16) : kWaitLimit;
    for (int l = 0; l <= n_layers; ++l)
    {
        if (sizes[l] == 0 || sizes[l] > 4096)
        {
            *why = "layer sizes must be in [1, 4096]";
            return -1;
        }
        if (l < n_layers && sizes[l] > kMaxFanIn)
        {
            *why = "a layer's fan-in exceeds 2048";
            return -1;
        }
    }
    for (uint32_t b = 0; b < batch; ++b)
    {
        if (steps[b] == 0 || steps[b] > 1000000)
        {
            *why = "per-sample step counts must be in [1, 1000000]";
            return -1;
        }
        if (sample_sizes)
            for (int l = 0; l <= n_layers; ++l)
                if (sample_sizes[static_cast<size_t>(l) * batch + b] > sizes[l])
                {
                    *why = "a sample's layer size exceeds the layer size";
                    return -1;
                }
    }
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    // The size limit of the interface (knp_gb300.h), kept as it was: pairs of 128-sample and 64-neuron tiles, two a
    // layer, at most one per SM. The kernel itself takes any number of columns.
    unsigned long long units = 0;
    for (int l = 1; l <= n_layers; ++l) units += 2ull * ((batch + 127) / 128) * ((sizes[l] + 63) / 64);
    if (units > kMaxTiles)
    {
        *why = "too many (layer, sample tile, neuron tile) work items";
        return -1;
    }
    if (units > static_cast<unsigned long long>(sms))
    {
        *why = "the batch does not fit: its (layer, sample tile, neuron tile) work items exceed the device";
        return -1;
    }
    int best = kMaxStages;
    if (autotune < 0)
    {
        // A fixed ring depth (-autotune).
        if (-autotune < kMinStages || -autotune > kMaxStages)
        {
            *why = "the requested operand ring depth is out of range or does not fit";
            return -1;
        }
        best = -autotune;
        autotune = 0;
    }
    const uint32_t t_max = *std::max_element(steps, steps + batch);
    // Rows of layer l have wp[l] words: whole 128-neuron tiles, 16-byte aligned.
    uint32_t wp[kMaxLayers + 1], words[kMaxLayers + 1], tiles[kMaxLayers + 1], wp_most = 4;
    unsigned long long rec_off[kMaxLayers + 1], rec_stride = 0;
    for (int l = 0; l <= n_layers; ++l)
    {
        tiles[l] = (sizes[l] + kTileN - 1) / kTileN;
        wp[l] = 4 * tiles[l];
        words[l] = (sizes[l] + 31) / 32;
        if (l < n_layers) wp_most = std::max(wp_most, wp[l]);
        rec_off[l] = rec_stride;
        rec_stride += static_cast<unsigned long long>(batch) * words[l];
    }
    uint32_t seg_steps = static_cast<uint32_t>(
        std::max<size_t>(1, std::min<size_t>(t_max, kRowBudget / (static_cast<size_t>(batch) * wp_most * 4))));
    if (segment_steps) seg_steps = std::min(seg_steps, segment_steps);
    const uint32_t n_segs = (t_max + seg_steps - 1) / seg_steps;

    // One device allocation and one copy for all of the plan's buffers and tables (one each cost 10 us and
    // more: 11 ms instead of 3 for a plan of 300 segments). Below, what
    // will be device pointers are offsets from its start until it is there.
    std::vector<uint8_t> tables;
    auto table = [&](const void *src, size_t bytes) -> size_t
    {
        tables.resize((tables.size() + 15) / 16 * 16);
        const size_t at = tables.size();
        tables.insert(tables.end(), static_cast<const uint8_t *>(src), static_cast<const uint8_t *>(src) + bytes);
        return at;
    };
    // Packed weights.
    p.pack.n_layers = n_layers;
    for (int l = 0; l < n_layers; ++l)
    {
        const uint32_t kp = (sizes[l] + 15) / 16 * 16, chunks = (kp + kChunk - 1) / kChunk;
        p.pack.w[l] = static_cast<const __nv_bfloat16 *>(weights[l]);
        p.pack.n[l] = sizes[l + 1];
        p.pack.k[l] = sizes[l];
        p.pack.chunks[l] = chunks;
        p.pack.first[l + 1] = p.pack.first[l] + static_cast<unsigned long long>(tiles[l + 1]) * chunks * kTileN * 8;
    }
    size_t size_at[kMaxLayers + 1] = {};
    for (int l = 0; sample_sizes && l <= n_layers; ++l)
        size_at[l] = table(sample_sizes + static_cast<size_t>(l) * batch, batch * 4ull);

    // Segments: every sample's columns and rows; per layer the streams, samples dealt longest first to
    // the shortest stream so far.
    size_t rows_most = 0;
    std::vector<uint32_t> order(batch);
    for (uint32_t b = 0; b < batch; ++b) order[b] = b;
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return steps[x] > steps[y]; });
    struct SegmentTables
    {
        size_t rows, tab[kMaxLayers], info[kMaxLayers];
    };
    std::vector<SegmentTables> seg_at(n_segs);
    p.segs.resize(n_segs);
    for (uint32_t sg = 0; sg < n_segs; ++sg)
    {
        BatchedPlan::Segment &seg = p.segs[sg];
        const uint32_t t0 = sg * seg_steps, t1 = std::min(t_max, t0 + seg_steps);
        std::vector<uint4> rows(batch);
        size_t at = 0;
        for (uint32_t b = 0; b < batch; ++b)
        {
            const uint32_t cols = steps[b] > t0 ? std::min(steps[b], t1) - t0 : 0u;
            rows[b] = make_uint4(static_cast<uint32_t>(at), cols, 0, 0);
            at += cols ? cols + 1 : 0;
        }
        rows_most = std::max(rows_most, at);
        seg_at[sg].rows = table(rows.data(), batch * sizeof(uint4));
        seg.draw.t0 = t0;
        seg.draw.blocks = (t1 - t0 + 1 + 31) / 32;
        size_t tab = 0, info_at = 0;
        uint32_t groups = 0;
        for (int l = 0; l < n_layers; ++l)
        {
            const uint32_t n_pairs = (tiles[l + 1] + 1) / 2;
            const uint32_t want = std::max(1u, std::min((batch + 1) / 2, static_cast<uint32_t>(sms) / 2 / n_pairs));
            if (want != groups)  // layers of equal width share their streams
            {
                groups = want;
                std::vector<std::vector<uint32_t>> streams(2 * groups);
                std::vector<uint64_t> load(2 * groups, 0);
                std::priority_queue<std::pair<uint64_t, uint32_t>, std::vector<std::pair<uint64_t, uint32_t>>,
                                    std::greater<>>
                    shortest;
                for (uint32_t q = 0; q < 2 * groups; ++q) shortest.emplace(0, q);
                for (uint32_t b : order)
                {
                    if (!rows[b].y) continue;
                    const uint32_t q = shortest.top().second;
                    shortest.pop();
                    streams[q].push_back(b);
                    load[q] += (rows[b].y + kPad - 1) / kPad * kPad;
                    shortest.emplace(load[q], q);
                }
                // [off: 2 G + 1][len: 2 G][start: entries]
                std::vector<uint32_t> t(4 * groups + 1), start;
                std::vector<uint4> info;
                for (uint32_t q = 0; q < 2 * groups; ++q)
                {
                    t[q] = static_cast<uint32_t>(start.size());
                    t[2 * groups + 1 + q] = static_cast<uint32_t>(load[q]);
                    uint32_t pos = 0;
                    for (uint32_t b : streams[q])
                    {
                        start.push_back(pos);
                        info.push_back(make_uint4(b, rows[b].x, rows[b].y, steps[b]));
                        pos += (rows[b].y + kPad - 1) / kPad * kPad;
                    }
                }
                t[2 * groups] = static_cast<uint32_t>(start.size());
                t.insert(t.end(), start.begin(), start.end());
                tab = table(t.data(), t.size() * 4);
                info_at = table(info.data(), info.size() * sizeof(uint4));
            }
            LayerArgs &a = seg.layer[l];
            seg_at[sg].tab[l] = tab;
            seg_at[sg].info[l] = info_at;
            a.n_groups = groups;
            a.t0 = t0;
            a.t1 = t1;
            seg.grid[l] = 2 * n_pairs * groups;
        }
    }
    size_t total = 0;
    auto carve = [&](size_t bytes)
    {
        const size_t at = total;
        total += (std::max<size_t>(bytes, 1) + 255) / 256 * 256;
        return at;
    };
    const size_t totals_at = carve(16), tables_at = carve(tables.size());
    size_t pack_at[kMaxLayers], bits_at[kMaxLayers], state_at[kMaxLayers] = {}, carry_at[kMaxLayers] = {};
    for (int l = 0; l < n_layers; ++l)
    {
        pack_at[l] = carve(static_cast<size_t>(tiles[l + 1]) * p.pack.chunks[l] * kAChunk);
        bits_at[l] = carve(rows_most * wp[l] * 4);
        if (n_segs == 1) continue;
        state_at[l] = carve(static_cast<size_t>(batch) * sizes[l + 1] * 12);
        carry_at[l] = carve(static_cast<size_t>(batch) * wp[l + 1] * 4);
    }
    if (cudaMalloc(reinterpret_cast<void **>(&p.memory), total) != cudaSuccess ||
        cudaMemcpyAsync(p.memory + tables_at, tables.data(), tables.size(), cudaMemcpyHostToDevice, p.stream) != cudaSuccess ||
        cudaStreamSynchronize(p.stream) != cudaSuccess ||
        !(p.totals_host = pinned_totals().take()))
    {
        *why = "device allocation failed";
        return -5;
    }
    p.totals = reinterpret_cast<unsigned long long *>(p.memory + totals_at);
    auto *d_err = reinterpret_cast<unsigned int *>(p.totals + 1);
    auto words_at = [&](size_t at) { return reinterpret_cast<uint32_t *>(p.memory + at); };
    auto table_at = [&](size_t at) { return reinterpret_cast<const uint32_t *>(p.memory + tables_at + at); };
    for (int l = 0; l < n_layers; ++l) p.pack.out[l] = p.memory + pack_at[l];
    p.record = record;
    p.record_bytes = static_cast<size_t>(t_max) * rec_stride * 4;
    for (uint32_t sg = 0; sg < n_segs; ++sg)
    {
        BatchedPlan::Segment &seg = p.segs[sg];
        const SegmentTables &at = seg_at[sg];
        DrawArgs &d = seg.draw;
        d.rows = reinterpret_cast<const uint4 *>(table_at(at.rows));
        d.rates = rates;
        d.n_in = sizes[0];
        d.wp = wp[0];
        d.words = words[0];
        d.batch = batch;
        d.size0 = sample_sizes ? table_at(size_at[0]) : nullptr;
        d.size1 = sample_sizes ? table_at(size_at[1]) : nullptr;
        d.n1 = sizes[1];
        d.key = key;
        d.bits = words_at(bits_at[0]);
        d.record = record;
        d.rec_stride = rec_stride;
        d.events = p.totals;
        for (int l = 0; l < n_layers; ++l)
        {
            LayerArgs &a = seg.layer[l];
            const bool last = l + 1 == n_layers;
            if (!sw128_map(&a.w, p.pack.out[l], static_cast<int>(tiles[l + 1] * p.pack.chunks[l] * kTileN), kChunk,
                           kTileN))
            {
                *why = "could not describe the packed weights to the TMA unit";
                return -3;
            }
            a.st_off = table_at(at.tab[l]);
            a.st_len = a.st_off + 2 * a.n_groups + 1;
            a.st_start = a.st_off + 4 * a.n_groups + 1;
            a.st_info = reinterpret_cast<const uint4 *>(table_at(at.info[l]));
            a.bits_in = words_at(bits_at[l]);
            a.wp_in = wp[l];
            a.bits_out = last ? nullptr : words_at(bits_at[l + 1]);
            a.wp_out = wp[l + 1];
            a.n = sizes[l + 1];
            a.kp = (sizes[l] + 15) / 16 * 16;
            a.chunks = p.pack.chunks[l];
            a.leak = leak ? leak[l] : 1.0f;
            a.thr = threshold ? threshold[l] : 1.0f;
            a.reset = reset ? reset[l] : 0.0f;
            a.refract = refract ? refract[l] : 0u;
            a.own_size = sample_sizes ? table_at(size_at[l + 1]) : nullptr;
            a.next_size = last || !sample_sizes ? nullptr : table_at(size_at[l + 2]);
            a.next_n = last ? 0u : sizes[l + 2];
            a.carry = n_segs > 1 ? words_at(carry_at[l]) : nullptr;
            a.state = n_segs > 1 ? words_at(state_at[l]) : nullptr;
            a.counts = last ? counts : nullptr;
            a.record = record;
            a.rec_off = rec_off[l + 1];
            a.rec_stride = rec_stride;
            a.wn = words[l + 1];
            a.events = p.totals;
            a.err = d_err;
            a.poll_limit = poll_limit;
            a.stall = stall;
        }
    }
    cudaError_t err = cudaSuccess;
    if (autotune)
    {
        float best_ms = 0.f;
        for (int stg = kMinStages; stg <= kMaxStages && err == cudaSuccess; ++stg)
        {
            float t = 0.f;
            err = capture(p, stg);
            if (err == cudaSuccess) err = launch_timed(p, &t);
            if (err == cudaSuccess) err = launch_timed(p, &t);
            p.tune_ms[stg] = t;
            if (err == cudaSuccess && (!best_ms || t < best_ms))
            {
                best_ms = t;
                best = stg;
            }
        }
    }
    if (err == cudaSuccess) err = capture(p, best);
    if (err != cudaSuccess)
    {
        *why = cudaGetErrorString(err);
        return -3;
    }
    *out = plan.release();
    return 0;
}

int batched_plan_run(BatchedPlan *p, unsigned long long *events_out, float *ms, const char **why)
{
    const cudaError_t err = launch_timed(*p, ms);
    if (err != cudaSuccess)
    {
        if (events_out) *events_out = 0;
        *why = cudaGetErrorString(err);
        return -3;
    }
    if (events_out) *events_out = p->totals_host[0];
    if (static_cast<uint32_t>(p->totals_host[1]))
    {
        *why = "a wait of the batched layer kernel (operands, accumulator or tensor-core completion) timed out";
        return -4;
    }
    return 0;
}

// tune_ms: [3][kMaxStages - kMinStages + 1]; the second and third rows stay 0 (depths alone are tuned).
void batched_plan_info(const BatchedPlan *p, int *stages, int *ring_steps, float *tune_ms)
{
    if (stages) *stages = p->stages;
    if (ring_steps) *ring_steps = 4;
    if (tune_ms)
        for (int ri = 0; ri < 3; ++ri)
            for (int i = kMinStages; i <= kMaxStages; ++i)
                tune_ms[ri * (kMaxStages - kMinStages + 1) + (i - kMinStages)] = ri ? 0.f : p->tune_ms[i];
}

void batched_plan_destroy(BatchedPlan *p) { delete p; }

// One-shot form: prepare, run once, release.
int batched_lif_run(
    int n_layers, const uint32_t *sizes, const void *const *weights, const float *leak, const float *threshold,
    const float *reset, const uint32_t *refract, uint32_t batch, const uint32_t *steps, const float *rates,
    unsigned long long key, int *counts, uint32_t *record, unsigned long long *events_out, float *ms,
    cudaStream_t s, const char **why)
{
    BatchedPlan *p = nullptr;
    int rc = batched_plan_create(n_layers, sizes, weights, leak, threshold, reset, refract, batch, steps, nullptr,
                                 rates, key, counts, record, 0, 0, s, &p, why);
    if (rc == 0) rc = batched_plan_run(p, events_out, ms, why);
    if (p) batched_plan_destroy(p);
    return rc;
}

}  // namespace knp_gb300
