// BF16 GEMM on the tcgen05 tensor cores, pipelined: D[M x N] (FP32, row-major) = A[M x K] * B[N x K]^T
// with A and B BF16, row-major, K contiguous.
//
// One CTA computes one 128 x 128 tile of D over the whole K range in chunks of 64. Four warps copy
// the chunks of A and B into a ring of kStages shared-memory stages (cp.async, 16 bytes per thread
// and copy, zero-filled past the matrix edges) in the canonical no-swizzle K-major layout of
// tcgen05.cuh; one thread of a fifth warp issues the MMAs of each staged chunk (four K = 16 slices,
// FP32 accumulator in tensor memory) and commits them to the stage's `empty` barrier, so the copies
// of later chunks overlap the MMAs of earlier ones. The same four warps then read the accumulator
// (tcgen05.ld, one row per thread) and store it. Every wait is bounded: a timeout sets bit 0 of
// *err, stops the loops, drains the issued MMAs (bounded) and frees the tensor memory.
//
// When K is a multiple of 8, the chunks are loaded by TMA instead (gemm_tma_kernel): each operand is
// described to the TMA unit as a 2-D tensor (K, rows) whose 64 x 128 box (128 bytes of K per row)
// lands in shared memory in the 128-byte swizzled K-major layout the MMA reads directly; one thread
// issues the two copies of a stage and the stage's mbarrier counts their bytes; rows and K past the
// matrix edge arrive as zeros. Tiles are few when M and N are small and K large (weight gradients):
// the K range is then split over up to 16 CTAs per tile, each writing its partial tile to a
// workspace, and a second kernel adds the partials in split order, so results
// do not depend on scheduling.
#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "kernels.h"
#include "tcgen05.cuh"

namespace knp_gb300
{
namespace
{

constexpr int kBM = 128, kBN = 128, kBK = 64;
constexpr int kStages = 4;
constexpr int kCopyWarps = 4;
constexpr int kCopyThreads = 32 * kCopyWarps;
constexpr int kThreads = kCopyThreads + 32;  // + the MMA warp
constexpr uint32_t kTileBytes = kBM * kBK * 2;  // 16 KB: one operand chunk (kBN == kBM)
constexpr uint32_t kStageBytes = 2 * kTileBytes;
constexpr uint32_t kSbo = (kBK / 8) * 128;  // bytes between core matrices adjacent along M / N
constexpr uint32_t kLbo = 128;              // bytes between core matrices adjacent along K
constexpr uint32_t kWait = 1u << 22;        // polls (of up to tc::kSuspendNs each) before a wait gives up
static_assert(kBN == kBM, "A and B chunks share one layout");

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t src_bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Copies chunk [k0, k0 + 64) of rows [r0, r0 + 128) of a row-major [rows][K] BF16 matrix into the
// stage tile at `dst` (shared address). Copy thread t handles 16-byte units u = t + 128 i: row
// r0 + 8 (u / 64) + u % 8, K group (u / 8) % 8, so a warp's 32 units fill 512 contiguous bytes.
__device__ __forceinline__ void copy_chunk(const __nv_bfloat16 *__restrict__ m, int rows, int K, int r0, int k0,
                                           uint32_t dst, int t)
{
#pragma unroll
    for (int i = 0; i < (kBM * kBK / 8) / kCopyThreads; ++i)
    {
        const int u = t + kCopyThreads * i;
        const int r = 8 * (u >> 6) + (u & 7), g = (u >> 3) & 7;
        const int gr = r0 + r, gk = k0 + 8 * g;
        const int left = K - gk;
        const uint32_t bytes = (gr < rows && left > 0) ? (left >= 8 ? 16u : 2u * static_cast<uint32_t>(left)) : 0u;
        const __nv_bfloat16 *src = bytes ? m + static_cast<size_t>(gr) * K + gk : m;
        cp_async16(dst + tc::core_offset(r, 8 * g, kLbo, kSbo), src, bytes);
    }
}

// mbar_wait that also stops as soon as another role of the CTA has given up.
__device__ __forceinline__ bool wait_or_fail(uint64_t *mbar, uint32_t parity, const volatile int *fail)
{
    for (uint32_t i = 0; i < kWait; ++i)
    {
        if (tc::mbar_try_wait(mbar, parity)) return true;
        if (*fail) return false;
    }
    return false;
}

__global__ void __launch_bounds__(kThreads, 1) gemm_pipe_kernel(
    const __nv_bfloat16 *__restrict__ A, const __nv_bfloat16 *__restrict__ B, float *__restrict__ D, int M, int N,
    int K, unsigned int *err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages], acc_full, drain;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * kBN;
    const int nk = (K + kBK - 1) / kBK;
    if (warp == 0) tc::tmem_alloc(&tmem_slot, kBN);
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < kStages; ++s)
        {
            tc::mbar_init(&full[s], kCopyThreads);
            tc::mbar_init(&empty[s], 1);
        }
        tc::mbar_init(&acc_full, 1);
        tc::mbar_init(&drain, 1);
        s_fail = 0;
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    const uint32_t base = tc::smem_u32(smem);

    if (warp < kCopyWarps)
    {
        // Copies: chunk c into stage c % kStages once the MMAs of chunk c - kStages are done; the
        // stage is published (after its copies landed and are made visible to the tensor cores)
        // kStages - 1 chunks later, so that many chunks' copies are in flight.
        const int t = threadIdx.x;
        bool ok = true;
        int published = 0;
        auto publish = [&](int c)
        {
            tc::fence_async_smem();
            tc::mbar_arrive(&full[c % kStages]);
        };
        for (int c = 0; c < nk; ++c)
        {
            const int s = c % kStages;
            if (c >= kStages && ok && !wait_or_fail(&empty[s], ((c / kStages) - 1) & 1, &s_fail))
            {
                ok = false;
                s_fail = 1;
            }
            if (!ok || s_fail) break;  // no copies into a stage the tensor cores may still read
            copy_chunk(A, M, K, m0, c * kBK, base + s * kStageBytes, t);
            copy_chunk(B, N, K, n0, c * kBK, base + s * kStageBytes + kTileBytes, t);
            cp_async_commit();
            if (c >= kStages - 1)
            {
                cp_async_wait<kStages - 1>();
                publish(published++);
            }
        }
        cp_async_wait<0>();
        while (published < nk && ok && !s_fail) publish(published++);
        if (!ok) atomicOr(err, 1u);

        // Epilogue: thread t reads accumulator lane t (row m0 + t) and stores its kBN columns. The
        // decision to read is the same in all four warps (bar.red.and over their 128 threads).
        const bool done = wait_or_fail(&acc_full, 0, &s_fail);
        tc::fence_after_sync();
        if (tc::named_sync_and(1, kCopyThreads, done && !s_fail))
        {
            const int row = m0 + t;
            const uint32_t lane_base = static_cast<uint32_t>(32 * warp) << 16;
#pragma unroll 1
            for (int c0 = 0; c0 < kBN; c0 += 16)
            {
                float v[16];
                tc::tmem_ld16(tmem + lane_base + c0, v);
                if (row < M)
                {
                    float *d = D + static_cast<size_t>(row) * N + n0 + c0;
                    if (n0 + c0 + 16 <= N && (reinterpret_cast<uintptr_t>(d) & 15u) == 0)
                    {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            reinterpret_cast<float4 *>(d)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                    }
                    else
                    {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (n0 + c0 + i < N) d[i] = v[i];
                    }
                }
            }
        }
        else if (t == 0)
        {
            atomicOr(err, 1u);
        }
    }
    else if (lane == 0)
    {
        // MMA issuer: the four K = 16 slices of each staged chunk, then one commit that frees the stage.
        constexpr uint32_t idesc = tc::idesc_bf16_f32(kBM, kBN);
        for (int c = 0; c < nk; ++c)
        {
            const int s = c % kStages;
            if (!wait_or_fail(&full[s], (c / kStages) & 1, &s_fail))
            {
                s_fail = 1;
                break;
            }
            tc::fence_after_sync();
            const uint32_t sa = base + s * kStageBytes, sb = sa + kTileBytes;
#pragma unroll
            for (int j = 0; j < kBK / 16; ++j)
                tc::mma_bf16(tmem, tc::smem_desc(sa + j * 256, kLbo, kSbo), tc::smem_desc(sb + j * 256, kLbo, kSbo),
                             idesc, (c > 0 || j > 0) ? 1u : 0u);
            tc::commit(&empty[s]);
        }
        tc::commit(&acc_full);
        // Every issued MMA completes (bounded wait) before the tensor memory is freed.
        tc::commit(&drain);
        if (!tc::mbar_wait(&drain, 0, kWait)) s_fail = 1;
        if (s_fail) atomicOr(err, 1u);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, kBN);
}

// How a GEMM's K is read: nk chunks of 64 positions. Positions from `half` on are the second half of an
// operand of two: they start over at K 0, in a K-major operand `step` elements further along K, in an
// MN-major one `step` elements further along M or N (0: both halves share the operand). `half` is a multiple
// of 64 for K-major operands and of 8 for MN-major ones, or above every position.
struct KPlan
{
    int nk, half, a_step, b_step;
};
constexpr int kOneHalf = 0x7FFFFFFF;

// The operands' tensor maps: 64 x 128 boxes (K-major), or 64 x 64 boxes and 64 x 8 boxes (MN-major).
struct GemmMaps
{
    CUtensorMap a, b, a8, b8;
};

template <bool kPair>
__device__ __forceinline__ void load_box(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t pair_mbar,
                                         uint64_t *mbar)
{
    if (kPair)
        tc::tma_load_2d_pair(dst, map, x, y, pair_mbar);
    else
        tc::tma_load_2d(dst, map, x, y, mbar);
}

// Stages chunk c of the 128 rows from r0 of an operand: K-major (row-major [rows][K]) as one 64 x 128 box,
// MN-major (row-major [K][rows]) as two 64 x 64 boxes, one per 64 rows, or, where the halves meet in the
// chunk, eight 64 x 8 boxes each. Rows and K past the matrix are zeros.
template <bool kMn, bool kPair>
__device__ __forceinline__ void load_operand(uint32_t dst, const CUtensorMap *map, const CUtensorMap *map8, int c, int half,
                                             int step, int r0, uint32_t pair_mbar, uint64_t *mbar)
{
    const int pos = c * kBK;
    const int second = pos >= half ? 1 : 0;
    if (!kMn)
    {
        load_box<kPair>(dst, map, pos - second * (half - step), r0, pair_mbar, mbar);
    }
    else if (second || half - pos >= kBK)
    {
        const int x = r0 + second * step, y = second ? pos - half : pos;
        load_box<kPair>(dst, map, x, y, pair_mbar, mbar);
        load_box<kPair>(dst + kTileBytes / 2, map, x + 64, y, pair_mbar, mbar);
    }
    else
    {
        for (int i = 0; i < kBK / 8; ++i)
        {
            const bool s = pos + 8 * i >= half;
            const int x = r0 + (s ? step : 0), y = pos + 8 * i - (s ? half : 0);
            load_box<kPair>(dst + i * 1024, map8, x, y, pair_mbar, mbar);
            load_box<kPair>(dst + kTileBytes / 2 + i * 1024, map8, x + 64, y, pair_mbar, mbar);
        }
    }
}

// Descriptor of a staged operand at shared address `a`, and the step of its start address per 16 of K.
template <bool kMn>
__device__ __forceinline__ uint64_t operand_desc(uint32_t a)
{
    return kMn ? tc::smem_desc_sw128_mn(a, kTileBytes / 2) : tc::smem_desc_sw128(a, 1024);
}
template <bool kMn>
constexpr uint32_t kDescStep = kMn ? 2048 >> 4 : 32 >> 4;

constexpr int kTmaThreads = 128;

constexpr int kTmaStages = 6;
constexpr uint32_t kTmaSmem = kTmaStages * kStageBytes + 1024;  // + alignment slack

// One 128 x 128 tile of D (or of split blockIdx.z's partial, into `out` with row stride N) over
// chunks [blockIdx.z * cps, min(nk, (blockIdx.z + 1) * cps)). Warp 0 lane 0 issues the TMA copies,
// warp 1 lane 0 the MMAs; all four warps read the accumulator back.
template <bool kAMn, bool kBMn>
__global__ void __launch_bounds__(kTmaThreads, 1) gemm_tma_kernel(
    const __grid_constant__ GemmMaps maps, float *__restrict__ out, int M,
    int N, KPlan kp, int cps, size_t split_stride, unsigned int *err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[kTmaStages], empty[kTmaStages], acc_full, drain;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * kBN;
    const int c0 = blockIdx.z * cps, c1 = min(kp.nk, c0 + cps);
    float *dst = out + blockIdx.z * split_stride;
    if (warp == 0) tc::tmem_alloc(&tmem_slot, kBN);
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < kTmaStages; ++s)
        {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        tc::mbar_init(&acc_full, 1);
        tc::mbar_init(&drain, 1);
        s_fail = 0;
    }
    // What is above overlaps the end of the kernel before (programmatic dependent launch); nothing below does.
    pdl_begin();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    const uint32_t base = (tc::smem_u32(smem) + 1023u) & ~1023u;  // TMA boxes on 1024-byte boundaries

    if (warp == 0 && lane == 0)
    {
        int issued = 0;
        for (int c = c0; c < c1; ++c)
        {
            const int i = c - c0, s = i % kTmaStages;
            if (i >= kTmaStages && !wait_or_fail(&empty[s], ((i / kTmaStages) - 1) & 1, &s_fail))
            {
                s_fail = 1;
                break;
            }
            const uint32_t sa = base + s * kStageBytes;
            tc::mbar_expect_tx(&full[s], kStageBytes);
            load_operand<kAMn, false>(sa, &maps.a, &maps.a8, c, kp.half, kp.a_step, m0, 0u, &full[s]);
            load_operand<kBMn, false>(sa + kTileBytes, &maps.b, &maps.b8, c, kp.half, kp.b_step, n0, 0u, &full[s]);
            issued = i + 1;
        }
        // Copies still in flight after a failed wait land before the CTA leaves (bounded).
        for (int i = max(0, issued - kTmaStages); i < issued; ++i)
            if (!tc::mbar_wait(&full[i % kTmaStages], (i / kTmaStages) & 1, kWait)) s_fail = 1;
    }
    else if (warp == 1 && lane == 0)
    {
        constexpr uint32_t idesc =
            tc::idesc_bf16_f32(kBM, kBN) | (kAMn ? tc::kIdescAMn : 0u) | (kBMn ? tc::kIdescBMn : 0u);
        for (int c = c0; c < c1; ++c)
        {
            const int i = c - c0, s = i % kTmaStages;
            if (!wait_or_fail(&full[s], (i / kTmaStages) & 1, &s_fail))
            {
                s_fail = 1;
                break;
            }
            tc::fence_after_sync();
            const uint32_t sa = base + s * kStageBytes, sb = sa + kTileBytes;
#pragma unroll
            for (int j = 0; j < kBK / 16; ++j)
                tc::mma_bf16(tmem, operand_desc<kAMn>(sa) + j * kDescStep<kAMn>,
                             operand_desc<kBMn>(sb) + j * kDescStep<kBMn>, idesc, (i > 0 || j > 0) ? 1u : 0u);
            tc::commit(&empty[s]);
        }
        tc::commit(&acc_full);
        tc::commit(&drain);
        if (!tc::mbar_wait(&drain, 0, kWait)) s_fail = 1;
    }
    __syncwarp();
    // Epilogue: thread t reads accumulator lane t (row m0 + t); an empty chunk range leaves zeros.
    const bool done = c1 <= c0 || wait_or_fail(&acc_full, 0, &s_fail);
    tc::fence_after_sync();
    const bool ok = tc::named_sync_and(1, kTmaThreads, done && !s_fail);
    if (ok)
    {
        const int row = m0 + threadIdx.x;
        const uint32_t lane_base = static_cast<uint32_t>(32 * warp) << 16;
#pragma unroll 1
        for (int q0 = 0; q0 < kBN; q0 += 16)
        {
            float v[16];
            if (c1 > c0)
                tc::tmem_ld16(tmem + lane_base + q0, v);
            else
                for (int i = 0; i < 16; ++i) v[i] = 0.0f;
            if (row < M)
            {
                float *d = dst + static_cast<size_t>(row) * N + n0 + q0;
                if (n0 + q0 + 16 <= N && (reinterpret_cast<uintptr_t>(d) & 15u) == 0)
                {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        reinterpret_cast<float4 *>(d)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                }
                else
                {
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (n0 + q0 + i < N) d[i] = v[i];
                }
            }
        }
    }
    else if (threadIdx.x == 0)
    {
        atomicOr(err, 1u);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, kBN);
}

// ---- Large GEMMs: 256 x 256 tiles on CTA pairs. Shared memory bounds a tile that one CTA multiplies
// alone: for a 64-deep chunk of a 128 x 256 tile TMA writes 48 KB and the MMAs read 48 KB, 768 cycles at
// 128 B a cycle where the tensor core needs 512 (8192^3: 784 us, 1.40 PFLOP/s). Of a pair's 256 x 256
// tile each CTA stages 128 rows of A and 128 of B and the tensor cores of both read B's two halves: 64 KB
// and 512 cycles per CTA. Persistent (one pair per two SMs) with two accumulators, so the read-back of a
// tile overlaps the next tile's product; tiles are taken in bands of kPairBand rows of tiles, so that
// the pairs at work share A and B in L2. Calls in a row: 8192^3 629-640 us, 1.72-1.75 PFLOP/s (among other work, under
// the power cap, 720 against 840); 2048 x 2048 x 32768: 325 -> 172 us; 16384 x 2048 x 2048: 133 -> 90 us. Both CTAs' copies are counted on the even CTA's barriers, whose
// issuer waits with CTA-scope acquire: a relay of the odd CTA's copies by a cluster-scope wait and arrival
// cost 2.2 ms at 8192^3.
constexpr int kPairM = 256, kPairN = 256, kPairStages = 6, kPairBand = 8;
constexpr uint32_t kPairStage = 2 * kTileBytes;  // this CTA's 128 x 64 of A and of B
constexpr uint32_t kTurn = 32 * 33 * 4;  // a read-back warp's 32 x 32 of the accumulator, rows 33 words apart
constexpr uint32_t kPairSmem = kPairStages * kPairStage + 1024 + 4 * kTurn;
constexpr uint32_t kDrainWait = 1u << 14;  // polls, about 0.06 s
constexpr int kPairThreads = 224;  // warps 0-3 read back, 4 and 6 load A and B, 5 issues (even rank)

template <bool kAMn, bool kBMn>
__global__ void __launch_bounds__(kPairThreads, 1) __cluster_dims__(2, 1, 1) gemm_pair_kernel(
    const __grid_constant__ GemmMaps maps, float *__restrict__ D, int M, int N, KPlan kp, unsigned int *err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    // Of the even CTA alone: full (both CTAs' halves of a chunk have landed) and acc_empty (4 read-back
    // warps of each CTA). Of both: empty (the pair's MMAs have read the stage), acc_full.
    __shared__ __align__(8) uint64_t full[kPairStages], empty[kPairStages];
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
        atomicOr(err, 1u);
    };
    if (warp == 5) tc::tmem_alloc_pair(&tmem_slot, 2 * kPairN);
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < kPairStages; ++s)
        {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a)
        {
            tc::mbar_init(&acc_full[a], 1);
            tc::mbar_init(&acc_empty[a], 8);
        }
        tc::mbar_init(&drain, 1);
        s_fail = 0;
    }
    pdl_begin();
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync();  // both CTAs' barriers and tensor memory are set up
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    const uint32_t base = (tc::smem_u32(smem) + 1023u) & ~1023u;
    const int nk = kp.nk;
    const int tiles_m = (M + kPairM - 1) / kPairM, tiles_n = (N + kPairN - 1) / kPairN;
    const int tiles = tiles_m * tiles_n, pairs = gridDim.x / 2, pair = blockIdx.x / 2;
    auto place = [&](int t, int &m0, int &n0)
    {
        const int band = t / (kPairBand * tiles_n), in = t - band * kPairBand * tiles_n;
        const int rows = min(kPairBand, tiles_m - band * kPairBand);
        m0 = (band * kPairBand + in % rows) * kPairM;
        n0 = (in / rows) * kPairN;
    };
    auto wait = [&](uint64_t *mbar, uint32_t parity) { return wait_or_fail(mbar, parity, &s_fail); };

    if (warp == 4 || warp == 6)
    {
        if (lane == 0)
        {
            // One thread issuing the four boxes of MN-major operands sets the pace (2048 x 2048 x 32768: 197 us
            // against 173 with a thread for each operand).
            const bool is_a = warp == 4;
            const CUtensorMap *map = is_a ? &maps.a : &maps.b, *map8 = is_a ? &maps.a8 : &maps.b8;
            const int step = is_a ? kp.a_step : kp.b_step;
            const uint32_t full0 = tc::mapa(tc::smem_u32(full), 0);  // the even CTA's
            int issued = 0, s = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs)
            {
                int m0, n0;
                place(t, m0, n0);
                const int r0 = (is_a ? m0 : n0) + 128 * static_cast<int>(rank);
                for (int c = 0; c < nk; ++c)
                {
                    if (!wait(&empty[s], ph))
                    {
                        ok = false;
                        break;
                    }
                    if (is_a && rank == 0) tc::mbar_expect_tx(&full[s], 2 * kPairStage);
                    const uint32_t dst = base + s * kPairStage + (is_a ? 0u : kTileBytes);
                    if (is_a ? kAMn : kBMn)
                        load_operand<true, true>(dst, map, map8, c, kp.half, step, r0, full0 + s * 8u, nullptr);
                    else
                        load_operand<false, true>(dst, map, map8, c, kp.half, step, r0, full0 + s * 8u, nullptr);
                    ++issued;
                    if (++s == kPairStages)
                    {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (!ok) fail();
            // Both CTAs' copies in flight after a failed wait land before either leaves (bounded; a chunk that
            // only one of them asked for does not complete, so the limit is short).
            for (int i = max(0, issued - kPairStages); i < issued && rank == 0; ++i)
                if (!tc::mbar_wait(&full[i % kPairStages], (i / kPairStages) & 1, kDrainWait)) fail();
        }
    }
    else if (warp == 5)
    {
        if (lane == 0 && rank == 0)
        {
            constexpr uint32_t idesc =
                tc::idesc_bf16_f32(kPairM, kPairN) | (kAMn ? tc::kIdescAMn : 0u) | (kBMn ? tc::kIdescBMn : 0u);
            const uint64_t da = operand_desc<kAMn>(base), db = operand_desc<kBMn>(base + kTileBytes);
            int s = 0, n = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs, ++n)
            {
                const int a = n & 1;
                if (n >= 2 && !wait(&acc_empty[a], ((n >> 1) - 1) & 1))
                {
                    ok = false;
                    break;
                }
                for (int c = 0; c < nk; ++c)
                {
                    if (!wait(&full[s], ph))
                    {
                        ok = false;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint64_t off = static_cast<uint64_t>(s) * (kPairStage >> 4);
#pragma unroll
                    for (int j = 0; j < kBK / 16; ++j)
                        tc::mma_bf16_pair(tmem + a * kPairN, da + off + j * kDescStep<kAMn>, db + off + j * kDescStep<kBMn>,
                                          idesc, (c > 0 || j > 0) ? 1u : 0u);
                    tc::commit_pair(&empty[s]);
                    if (++s == kPairStages)
                    {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                if (ok) tc::commit_pair(&acc_full[a]);
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
    else
    {
        // Read-back: thread t of the CTA has accumulator lane t, row m0 + 128 rank + t of the tile. Where D's rows are
        // whole 16-byte units a thread stores its row; else a warp turns its 32 x 32 values in shared memory and
        // stores row after row, 128 bytes at a time: a thread's 4-byte stores touch 32 rows at a time (8192 x 8190 x 64:
        // 410 us that way, 76 so; 8192 x 8190 x 8192: 768 and 628). Turned, whole rows are no better where the product
        // carries the time (2500^3: 83 us against 79; 16384 x 2048 x 2048: 91.5 against 89.7).
        const uint32_t lane_base = static_cast<uint32_t>(32 * warp) << 16;
        float *turn = reinterpret_cast<float *>(smem + (base - tc::smem_u32(smem)) + kPairStages * kPairStage + warp * kTurn);
        int n = 0;
        for (int t = pair; t < tiles; t += pairs, ++n)
        {
            const int a = n & 1;
            if (!__all_sync(0xffffffffu, wait(&acc_full[a], (n >> 1) & 1)))
            {
                if (lane == 0) fail();
                break;
            }
            tc::fence_after_sync();
            int m0, n0;
            place(t, m0, n0);
            const int row = m0 + 128 * static_cast<int>(rank) + static_cast<int>(threadIdx.x);
            float *d = D + static_cast<size_t>(row) * N + n0;
            const bool vec = N % 4 == 0 && (reinterpret_cast<uintptr_t>(D) & 15u) == 0;
#pragma unroll 1
            for (int q0 = 0; q0 < kPairN; q0 += 32)
            {
                float v[32];
                tc::tmem_ld32(tmem + a * kPairN + lane_base + q0, v);
                if (q0 + 32 == kPairN)
                {
                    // The whole accumulator has been read: the issuer may start the tile after next in it.
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive_cluster(tc::mapa(tc::smem_u32(&acc_empty[a]), 0));
                }
                if (vec && n0 + q0 + 32 <= N)
                {
                    if (row < M)
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            reinterpret_cast<float4 *>(d + q0)[q] =
                                make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                    __syncwarp();  // the next read is warp-collective
                    continue;
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) turn[lane * 33 + i] = v[i];
                __syncwarp();
                const int col = n0 + q0 + lane, rows = min(32, M - (row - lane));
                float *out = D + static_cast<size_t>(row - lane) * N + col;
                if (col < N)
                    for (int r = 0; r < rows; ++r) out[static_cast<size_t>(r) * N] = turn[r * 33 + lane];
                __syncwarp();
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    // Neither CTA leaves while the other's MMAs may read its shared memory or arrivals may reach it.
    tc::cluster_sync();
    if (warp == 5) tc::tmem_dealloc_pair(tmem, 2 * kPairN);
}

// D = sum over the splits of ws[z] (split order), n elements.
__global__ void split_sum_kernel(const float *__restrict__ ws, float *__restrict__ D, size_t n, int splits)
{
    pdl_begin();
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x)
    {
        float s = ws[i];
        for (int z = 1; z < splits; ++z) s = __fadd_rn(s, ws[z * n + i]);
        D[i] = s;
    }
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled()
{
    static EncodeTiled fn = []
    {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
        {
            cudaGetLastError();
            return static_cast<EncodeTiled>(nullptr);
        }
        return reinterpret_cast<EncodeTiled>(p);
    }();
    return fn;
}

// Stream-ordered pool of the split-K workspaces of device `dev` (memory kept by the pool between
// calls). Allocating on the call's stream keeps concurrent streams apart and lets a call be captured
// in a CUDA graph (the allocation becomes a graph memory node).
cudaMemPool_t split_pool(int dev)
{
    static std::mutex mu;
    static std::map<int, cudaMemPool_t> pools;
    std::lock_guard<std::mutex> lock(mu);
    const auto it = pools.find(dev);
    if (it != pools.end()) return it->second;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess)
    {
        cudaGetLastError();
        return pools[dev] = nullptr;
    }
    uint64_t keep = UINT64_MAX;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    return pools[dev] = pool;
}

}  // namespace
}  // namespace knp_gb300

namespace knp_gb300
{
namespace
{

// A BF16 tensor of `rank` dimensions (K contiguous), loaded in boxes of 64 x ... with the 128-byte swizzle.
bool sw128_map_nd(void *map, const void *ptr, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
                  const cuuint32_t *box)
{
    const EncodeTiled fn = encode_tiled();
    if (!fn) return false;
    const cuuint32_t estr[3] = {1, 1, 1};
    auto encode = [&]
    {
        return fn(static_cast<CUtensorMap *>(map), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void *>(ptr), dims,
                  strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r = encode();
    if (r == CUDA_ERROR_INVALID_CONTEXT)
    {
        // A thread whose first CUDA call this is (an autograd thread, say) has no current context yet.
        int dev = 0;
        if (cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) r = encode();
    }
    return r == CUDA_SUCCESS;
}

}  // namespace

// The (K, rows) view of a row-major [rows][K] BF16 matrix (K a multiple of 8), in 64 x box_rows boxes.
bool sw128_map(void *map, const void *ptr, int rows, int K, int box_rows)
{
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * 2};
    const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)};
    return sw128_map_nd(map, ptr, 2, dims, strides, box);
}

// The (K, t, b) view of the rows t * batch + b of such a matrix, in 64 x box_t x box_b boxes.
bool sw128_map_3d(void *map, const void *ptr, int T, int batch, int K, int box_t, int box_b)
{
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(T), static_cast<cuuint64_t>(batch)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(batch) * K * 2, static_cast<cuuint64_t>(K) * 2};
    const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_t), static_cast<cuuint32_t>(box_b)};
    return sw128_map_nd(map, ptr, 3, dims, strides, box);
}

int bf16_gemm_tn_simple(const void *A, const void *B, float *D, int M, int N, int K, unsigned int *d_err, cudaStream_t s);

// K is split when the tiles leave most SMs idle and each split keeps at least 4 chunks: the number of
// splits of nk chunks over `tiles` 128 x 128 tiles, and the chunks of each but the last.
int gemm_splits(int tiles, int nk, int sms, int &cps)
{
    int splits = 1;
    if (tiles * 2 <= sms) splits = std::max(1, std::min({16, nk / 4, sms / tiles}));
    cps = (nk + splits - 1) / splits;
    return (nk + cps - 1) / cps;
}

namespace
{

// D[M x N] from operands that are K-major or (kAMn, kBMn) MN-major.
template <bool kAMn, bool kBMn>
int launch_gemm(const GemmMaps &maps, float *D, int M, int N, KPlan kp, unsigned int *d_err, cudaStream_t s)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int tiles_m = (M + kBM - 1) / kBM, tiles_n = (N + kBN - 1) / kBN, tiles = tiles_m * tiles_n;
    const int pair_tiles = ((M + kPairM - 1) / kPairM) * ((N + kPairN - 1) / kPairN);
    // A 128 x 128 tile on one CTA (bound by shared memory) and a 256 x 256 tile on a pair (bound by the
    // tensor core) take the same 512 cycles per 64-deep chunk, so the form with fewer waves is the faster
    // (2500^3: 3 waves 86 us, 2 waves 74 us; 2048 x 2048 x 32768: 2 waves 325 us, 1 wave 169 us); at the
    // same number of waves the small tiles start and end sooner and may split K.
    const int waves = (tiles + sms - 1) / sms, pair_waves = (pair_tiles + sms / 2 - 1) / (sms / 2);
    if (pair_waves < waves)
    {
        if (allow_dynamic_smem(gemm_pair_kernel<kAMn, kBMn>) != cudaSuccess) return -3;
        launch_pdl(gemm_pair_kernel<kAMn, kBMn>, dim3(2 * std::min(pair_tiles, sms / 2)), dim3(kPairThreads), kPairSmem, s, maps, D, M, N,
                   kp, d_err);
        return cudaGetLastError() == cudaSuccess ? 0 : -3;
    }
    if (allow_dynamic_smem(gemm_tma_kernel<kAMn, kBMn>) != cudaSuccess) return -3;
    int cps = 0;
    int splits = gemm_splits(tiles, kp.nk, sms, cps);
    const size_t mn = static_cast<size_t>(M) * N;
    float *ws = nullptr;
    if (splits > 1)
    {
        const cudaMemPool_t pool = split_pool(dev);
        if (!pool || cudaMallocFromPoolAsync(reinterpret_cast<void **>(&ws), mn * splits * sizeof(float), pool, s) !=
                         cudaSuccess)
        {
            cudaGetLastError();
            ws = nullptr;
            splits = 1;
        }
    }
    const int cps_used = splits > 1 ? cps : kp.nk;
    dim3 grid(tiles_m, tiles_n, splits);
    launch_pdl(gemm_tma_kernel<kAMn, kBMn>, grid, dim3(kTmaThreads), kTmaSmem, s, maps, splits > 1 ? ws : D, M, N, kp, cps_used,
               splits > 1 ? mn : 0, d_err);
    if (splits > 1)
    {
        const int blocks = static_cast<int>(std::min<size_t>((mn + 255) / 256, 8ull * sms));
        launch_pdl(split_sum_kernel, dim3(blocks), dim3(256), 0, s, static_cast<const float *>(ws), D, mn, splits);
        cudaFreeAsync(ws, s);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace

// D = A * B^T (see knp_gb300_bf16_gemm_tn). The TMA-fed kernels need 16-byte aligned rows (K a multiple
// of 8, 16-byte aligned A and B); other shapes take the single-stage kernel.
int bf16_gemm_tn(const void *A, const void *B, float *D, int M, int N, int K, unsigned int *d_err, cudaStream_t s)
{
    if (M < 1 || N < 1 || K < 1 || !A || !B || !D || !d_err) return -1;
    const bool aligned = K % 8 == 0 && (reinterpret_cast<uintptr_t>(A) & 15u) == 0 && (reinterpret_cast<uintptr_t>(B) & 15u) == 0;
    if (!aligned) return bf16_gemm_tn_simple(A, B, D, M, N, K, d_err, s);
    GemmMaps maps{};
    if (sw128_map(&maps.a, A, M, K, kBM) && sw128_map(&maps.b, B, N, K, kBN))
        return launch_gemm<false, false>(maps, D, M, N, KPlan{(K + kBK - 1) / kBK, kOneHalf, 0, 0}, d_err, s);
    if (allow_dynamic_smem(gemm_pipe_kernel) != cudaSuccess) return -3;
    dim3 grid((M + kBM - 1) / kBM, (N + kBN - 1) / kBN);
    gemm_pipe_kernel<<<grid, kThreads, kStages * kStageBytes, s>>>(static_cast<const __nv_bfloat16 *>(A),
                                                                   static_cast<const __nv_bfloat16 *>(B), D, M, N, K, d_err);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// The two products of a LIF layer's backward, with the gradient dI given as rows of two BF16 halves
// [hi | lo] of width w2 (knp_gb300_lif_layer_backward), summed over hi, then over lo:
//   ds[rows][n_in] = (hi + lo) W^T   from W as [n_in][w2] (w2 a multiple of 64: both halves read the same W):
// both operands K-major;
//   dW[n_in][n_out] = S^T (hi + lo)  from S as [rows][n_in8]: both operands MN-major, so neither S nor dI is
// transposed in memory (a transposed copy of each cost 89 us of the 1.03 ms of a 16384-row layer of
// 2048 x 2048). Positions along K, and so the order of every sum, are those of operands concatenated along K
// with the rows padded to a multiple of 8.
int lif_ds_gemm(const void *dI2, const void *W, float *ds, int rows, int n_in, int w2, unsigned int *d_err, cudaStream_t s)
{
    if (w2 % kBK) return -1;
    GemmMaps maps{};
    if (!sw128_map(&maps.a, dI2, rows, 2 * w2, kBM) || !sw128_map(&maps.b, W, n_in, w2, kBN)) return -3;
    return launch_gemm<false, false>(maps, ds, rows, n_in, KPlan{2 * w2 / kBK, w2, w2, 0}, d_err, s);
}

int lif_dw_gemm(const void *S, const void *dI2, float *dW, int rows, int n_in, int n_in8, int n_out, int w2,
                unsigned int *d_err, cudaStream_t s)
{
    GemmMaps maps{};
    const int padded = (rows + 7) / 8 * 8;
    if (!sw128_map(&maps.a, S, rows, n_in8, kBK) || !sw128_map(&maps.b, dI2, rows, 2 * w2, kBK) ||
        !sw128_map(&maps.a8, S, rows, n_in8, 8) || !sw128_map(&maps.b8, dI2, rows, 2 * w2, 8))
        return -3;
    return launch_gemm<true, true>(maps, dW, n_in, n_out, KPlan{(2 * padded + kBK - 1) / kBK, padded, 0, w2}, d_err, s);
}

// I[rows][N] = S W from S as [rows][k8] (K-major) and W as [K][wp] (MN-major, columns from N on unused).
int lif_input_gemm(const void *S, const void *W, float *I, int rows, int K, int k8, int N, int wp, unsigned int *d_err,
                   cudaStream_t s)
{
    GemmMaps maps{};
    if (!sw128_map(&maps.a, S, rows, k8, kBM) || !sw128_map(&maps.b, W, K, wp, kBK)) return -3;
    return launch_gemm<false, true>(maps, I, rows, N, KPlan{(K + kBK - 1) / kBK, kOneHalf, 0, 0}, d_err, s);
}

cudaError_t workspace_alloc(void **p, size_t bytes, cudaStream_t s)
{
    int dev = 0;
    cudaGetDevice(&dev);
    const cudaMemPool_t pool = split_pool(dev);
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaErrorMemoryAllocation;
}
}  // namespace knp_gb300
