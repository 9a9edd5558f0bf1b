// moe_kernels.cu - expert-parallel all-to-all for mixture-of-experts layers: dispatch (tokens to the
// ranks that own their experts, quantised on the fly to fp8 e4m3 with one fp32 scale per 128 values) and
// combine (expert outputs back to the token's rank with the gate-weighted sum fused).  One kernel each;
// all traffic is remote stores into symmetric buffers.  The reference only offers AlltoAll(V/VC) for this
// (pkg_inc/legacy/hccl/hccl_inner.h:55-66); routing, quantisation and the weighted sum are fused here.
//
// Dispatch, rank r - two ordinary launches (no CTA of a launch waits for another CTA of it, so they can share the GPU
// with expert GEMMs on other streams):
//   route    (1 CTA)  histogram of the experts its tokens chose, the counts published to the rank that owns each expert,
//                     one cross-rank barrier, the per-expert offsets of this rank's own experts for its grouped GEMM
//   dispatch (N CTAs) every CTA reads the owners' count tables and derives, for each expert, where this rank's rows
//                     start in the owner's receive buffer (rows are grouped by expert, inside an expert by source rank);
//                     the CTA's threads claim the rows of its tokens' experts in parallel (atomics on the row cursors),
//                     then its warps quantise 512 values of a token at a time and store them to the token's k rows;
//                     each CTA ends with one cross-rank barrier with its namesakes
// A single rank has no counts to exchange: one launch, in which CTAs count all choices alone or in pairs.
// Combine, rank r (owner of experts) - two ordinary launches, one when there is a single rank:
//   send  one warp per row received from ANOTHER rank: the bf16 expert output goes to slot (token, k) of the token's rank;
//         cross-rank barrier
//   sum   out = sum_k gate[k] * row(token, k) over the k that were sent, fp32 accumulation in the order of k; a row whose
//         expert lives on the token's own rank is read where the expert wrote it (dispatch noted which row that is)
// Rows of this rank's own tokens go through their slots as well (and a single rank has both launches) when the result may
// overlap the experts' output, whose rows would otherwise be overwritten before they are read, and once the caller has
// asked for the address of the slots.
//
// Device scratch (beyond inputs and outputs): numExperts u32 row cursors, cleared by the route launch and left as they are by
// the dispatch (a single rank has none); the local row of every (token, k).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <map>

#include "../comm/comm.h"
#include "../core/log.h"
#include "emu_launch.h"
#include "hccl/hccl_sym_win.h"
#include "hcomm_res.h"
#include "hcomm_device.cuh"
#include "hcomm_moe.h"

namespace hc {
namespace {

namespace cg = cooperative_groups;
using namespace hcdev;

constexpr int kMaxExperts = 1024;
constexpr int kBlock = 128;            // quantisation block

struct MoeParams {
    CommDev *dev;
    char *peerBuf[HC_KERNEL_MAX_RANKS];   // symmetric buffer of every rank as mapped here
    MoeLayout lay;
    // dispatch
    const __nv_bfloat16 *x;
    const int32_t *topkIdx;
    int numTokens;
    uint32_t *scratch;                    // [numExperts]: row cursors
    // combine
    const __nv_bfloat16 *y;
    const float *gates;
    __nv_bfloat16 *out;
    uint32_t *overflow;                   // device words: rows that did not fit the receive capacity, tokens of the last dispatch
    uint32_t *localRow;                   // [maxTokens * topk]: 1 + row of (token, k) in this rank's receive buffer, 0 when it went elsewhere or nowhere
    int segsPerItem;                      // sum: 256-column segments that a warp takes at a time
    int countsLaunch;                     // sum: this launch is the whole operator (single rank) and advances the launch state
    int allThroughSlots;                  // combine: rows of this rank's own tokens go through the landing area too
    int overlaps;                         // single rank: the kernel behind may take SMs early (see MOE_ARGS)
};
constexpr uint32_t kNoRow = 0xffffffffu;

// A single rank launches with the stream-serialization attribute: the CTAs are resident before the kernel in front has ended
// and idle until it has, and the kernel behind may do the same.  Kernels that meet other ranks let nothing start early: what is
// resident behind them would hold its SMs for as long as a peer is late.
#define MOE_ARGS MOE_ARGS_OF(table != nullptr)
#define MOE_ARGS_OF(merged)                                                                    \
    const MoeParams &p = (merged) ? table[blockIdx.y] : byval;                                 \
    if (p.overlaps) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");            \
    asm volatile("griddepcontrol.wait;" ::: "memory")

__device__ __forceinline__ uint32_t *Counts(const MoeParams &p, int rank) { return (uint32_t *)(p.peerBuf[rank] + p.lay.offCounts); }
__device__ __forceinline__ uint8_t *Rows(const MoeParams &p, int rank) { return (uint8_t *)(p.peerBuf[rank] + p.lay.offRows); }
__device__ __forceinline__ float *Scales(const MoeParams &p, int rank) { return (float *)(p.peerBuf[rank] + p.lay.offScales); }
__device__ __forceinline__ uint64_t *Origin(const MoeParams &p, int rank) { return (uint64_t *)(p.peerBuf[rank] + p.lay.offOrigin); }
__device__ __forceinline__ uint32_t *ExpertOffsets(const MoeParams &p, int rank) { return (uint32_t *)(p.peerBuf[rank] + p.lay.offExpertOffsets); }
__device__ __forceinline__ __nv_bfloat16 *Comb(const MoeParams &p, int rank) { return (__nv_bfloat16 *)(p.peerBuf[rank] + p.lay.offCombine); }
// one byte per (token, k) of the LOCAL tokens: 1 when dispatch sent that row, 0 when the expert index was out of range
// (masked) or the owner's receive capacity was exhausted; combine leaves such rows out of the sum
__device__ __forceinline__ uint8_t *Valid(const MoeParams &p, int rank) { return (uint8_t *)(p.peerBuf[rank] + p.lay.offValid); }

// Streamed once, not worth a line of L1.  Data that peers wrote has landed in this GPU's memory before the kernel began.
__device__ __forceinline__ uint4 LdStream16(const void *p)
{
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// Exclusive prefix sums of v over the CTA's threads (a multiple of 32, at most 1024); warpSums: one word per warp.
__device__ __forceinline__ uint32_t BlockExclusiveScan(uint32_t v, uint32_t *warpSums)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warpSums[warp] = x;
    __syncthreads();
    uint32_t below = 0;
    for (int w = 0; w < warps; ++w) below += w < warp ? warpSums[w] : 0u;
    return below + x - v;
}

// Dispatch, first launch (one CTA per rank): routing histogram, counts published to the experts' owners, one cross-rank
// barrier, the offsets of this rank's own experts, row cursors cleared for the second launch.  Bound by latency and by
// shared-memory atomics: 32768 choices 10.5 us (28 with one histogram and a serial prefix), 512 choices 6 (12).
__global__ void __launch_bounds__(1024) MoeRouteKernel(const __grid_constant__ MoeParams byval, const MoeParams *table)
{
    MOE_ARGS;
    const CommDev *d = p.dev;
    const LaunchState ls = KernelBegin(d);
    const int n = d->nRanks, me = d->rank;
    const int E = p.lay.numExperts, El = E / n, K = p.lay.topk;
    const int tid = threadIdx.x;
    // four histograms, warps dealt over them: neighbouring lanes often hold the same expert and would queue for its counter
    __shared__ uint32_t sHist[4][kMaxExperts], sWarp[32];
    uint32_t *cursor = p.scratch;
    for (int e = tid; e < E; e += blockDim.x) {
#pragma unroll
        for (int h = 0; h < 4; ++h) sHist[h][e] = 0;
        cursor[e] = 0;
    }
    __syncthreads();
    uint32_t *hist = sHist[(tid >> 5) & 3];
    const int total = p.numTokens * K, stride = blockDim.x;
    for (int i = tid; i < total; i += 16 * stride) {        // sixteen loads in flight
        int e[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) e[u] = i + u * stride < total ? p.topkIdx[i + u * stride] : -1;
#pragma unroll
        for (int u = 0; u < 16; ++u)
            if (e[u] >= 0 && e[u] < E) atomicAdd(&hist[e[u]], 1u);
    }
    __syncthreads();
    for (int e = tid; e < E; e += blockDim.x) Counts(p, e / El)[me * El + (e % El)] = sHist[0][e] + sHist[1][e] + sHist[2][e] + sHist[3][e];
    CrossRankBarrier(d, ls.epoch0 + 1);
    // the offsets of my own experts for the grouped GEMM that follows (the table may be overwritten by a peer's next
    // dispatch as soon as the second launch's barrier is passed, so derive them now): one thread per local expert sums
    // its column.  Every entry is clamped to the receive capacity: a grouped GEMM that walks [off[el], off[el + 1]) never
    // leaves the buffer.
    uint32_t sum = 0;
    if (tid < El) {
        const volatile uint32_t *c = Counts(p, me);
        for (int s = 0; s < n; ++s) sum += c[s * El + tid];
    }
    const uint32_t before = BlockExclusiveScan(sum, sWarp), capRows = (uint32_t)p.lay.maxRecvRows;
    uint32_t *off = ExpertOffsets(p, me);
    if (tid < El) off[tid] = before < capRows ? before : capRows;
    if (tid == El - 1) off[El] = before + sum < capRows ? before + sum : capRows;
    KernelEnd(d, ls, 1, 0);
}

// A lane's 16 values as fp8, the scale of their block of 128: the eight lanes that share a block sit next to each other.
__device__ __forceinline__ uint4 Quantise(const uint4 &lo, const uint4 &hi, float *blockScale)
{
    // the largest magnitude of the lane's 16 values (a maximum of bf16 values is exact in bf16)
    const uint4 cur[2] = {lo, hi};
    const __nv_bfloat162 *x2 = (const __nv_bfloat162 *)cur;
    __nv_bfloat162 m2 = __habs2(x2[0]);
#pragma unroll
    for (int j = 1; j < 8; ++j) m2 = __hmax2(m2, __habs2(x2[j]));
    float amax = fmaxf(0.f, fmaxf(__low2float(m2), __high2float(m2)));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
    const float scale = fmaxf(amax, 1e-4f) / 448.0f;   // values are divided (not multiplied by a reciprocal): bit-exact with x / scale
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f0 = __bfloat1622float2(x2[2 * j]), f1 = __bfloat1622float2(x2[2 * j + 1]);
        const __nv_fp8x2_storage_t first = __nv_cvt_float2_to_fp8x2(make_float2(f0.x / scale, f0.y / scale), __NV_SATFINITE, __NV_E4M3);
        const __nv_fp8x2_storage_t second = __nv_cvt_float2_to_fp8x2(make_float2(f1.x / scale, f1.y / scale), __NV_SATFINITE, __NV_E4M3);
        w[j] = (uint32_t)first | ((uint32_t)second << 16);
    }
    *blockScale = scale;
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Dispatch, second launch (any number of CTAs, an ordinary launch that can share the GPU with expert GEMMs): every CTA
// derives from the owners' count tables where this rank's rows of each expert start, claims the rows of its tokens, then
// quantises and sends them, and meets its namesakes on the other ranks once all of its rows are on their way.
// Bound by memory, by its scattered 512-byte stores: 4096 x 7168 to 8 experts each take 69 us (86 with one warp per token), 46
// at HBM rate, and no less with a sixth of the divisions; 64 tokens 9 us (39).  A CTA owns whole tokens and its 16 warps share them in
// pieces of 512 values, so that few tokens still occupy many warps and the claims cost one round of atomics per CTA, not one
// per token.
constexpr int kClaims = 512;           // (token, k) pairs that a CTA claims at a time: one per thread
__global__ void __launch_bounds__(512, 2) MoeDispatchKernel(const __grid_constant__ MoeParams byval, const MoeParams *table)
{
    MOE_ARGS;
    const CommDev *d = p.dev;
    const LaunchState ls = KernelBegin(d);
    const int n = d->nRanks, me = d->rank;
    const int E = p.lay.numExperts, El = E / n, K = p.lay.topk, H = p.lay.hidden;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
    __shared__ uint32_t sBase[kMaxExperts], sWarp[16];
    __shared__ uint8_t *sRow[kClaims];
    __shared__ float *sScale[kClaims];
    uint32_t *cursor = p.scratch;
    const int t0 = (int)((int64_t)p.numTokens * blockIdx.x / gridDim.x), t1 = (int)((int64_t)p.numTokens * (blockIdx.x + 1) / gridDim.x);
    const int segs = H / 512, perRound = kClaims / K;

    // the first piece of this warp is on its way while the rows are being found
    uint4 a = make_uint4(0, 0, 0, 0), b = a;
    const int firstItems = (t1 - t0 < perRound ? t1 - t0 : perRound) * segs;
    if (warp < firstItems) {
        const __nv_bfloat16 *src = p.x + (size_t)t0 * H + (size_t)warp * 512 + lane * 16;     // pieces of consecutive tokens are consecutive in x
        a = LdStream16(src); b = LdStream16(src + 8);
    }

    // where do my rows of expert e start at its owner?  before them: all rows of the owner's earlier experts,
    // and the rows of this expert that come from lower ranks.  Every thread fetches the n counts of two experts
    // from their owner (independent loads, one NVLink round trip), then the prefix runs inside the CTA.
    {
        uint32_t tot[2] = {0, 0}, below[2] = {0, 0};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int e = 2 * tid + j;
            if (e < E) {
                const volatile uint32_t *c = Counts(p, e / El) + e % El;
                for (int s = 0; s < n; ++s) {
                    const uint32_t v = c[s * El];
                    tot[j] += v;
                    if (s < me) below[j] += v;
                }
            }
        }
        const uint32_t before = BlockExclusiveScan(tot[0] + tot[1], sWarp);
        if (2 * tid < E) sBase[2 * tid] = before;
        if (2 * tid + 1 < E) sBase[2 * tid + 1] = before + tot[0];
        __syncthreads();
        uint32_t base[2] = {0, 0};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int e = 2 * tid + j;
            if (e < E) base[j] = sBase[e] - sBase[e / El * El] + below[j];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (2 * tid + j < E) sBase[2 * tid + j] = base[j];
        __syncthreads();
    }

    if (blockIdx.x == 0 && tid == 0) p.overflow[1] = (uint32_t)p.numTokens;
    for (int r0 = t0; r0 < t1; r0 += perRound) {
        const int tokens = t1 - r0 < perRound ? t1 - r0 : perRound;
        if (tid < tokens * K) {
            const size_t tk = (size_t)r0 * K + tid;
            const int e = p.topkIdx[tk];
            uint32_t slot = kNoRow, local = 0;
            if (e >= 0 && e < E) {
                slot = sBase[e] + atomicAdd(&cursor[e], 1u);
                if (slot >= (uint32_t)p.lay.maxRecvRows) { atomicAdd(p.overflow, 1u); slot = kNoRow; }
            }
            Valid(p, me)[tk] = slot != kNoRow ? 1 : 0;
            sRow[tid] = nullptr;
            if (slot != kNoRow) {
                const int owner = e / El;
                sRow[tid] = Rows(p, owner) + (size_t)slot * H;
                sScale[tid] = Scales(p, owner) + (size_t)slot * (H / kBlock);
                Origin(p, owner)[slot] = ((uint64_t)me << 32) | (uint32_t)tk;
                if (owner == me) local = slot + 1;
            }
            p.localRow[tk] = local;
        }
        __syncthreads();
        const int items = tokens * segs;
        const __nv_bfloat16 *src = p.x + (size_t)r0 * H + lane * 16;
        if (r0 != t0 && warp < items) { a = LdStream16(src + (size_t)warp * 512); b = LdStream16(src + (size_t)warp * 512 + 8); }
        for (int it = warp; it < items; it += warps) {
            const uint4 ca = a, cb = b;
            if (it + warps < items) { a = LdStream16(src + (size_t)(it + warps) * 512); b = LdStream16(src + (size_t)(it + warps) * 512 + 8); }
            float scale;
            const uint4 q = Quantise(ca, cb, &scale);
            const int tok = it / segs, seg = it - tok * segs, c0 = tok * K;
            for (int k = 0; k < K; ++k) {
                uint8_t *row = sRow[c0 + k];
                if (!row) continue;
                *(uint4 *)(row + seg * 512 + lane * 16) = q;
                if ((lane & 7) == 0) sScale[c0 + k][seg * 4 + (lane >> 3)] = scale;
            }
        }
        __syncthreads();        // the claims of the next round overwrite these
    }
    // all rows of this CTA are on their way; once every local CTA has passed its barrier (= the kernel has ended) all
    // CTAs of all ranks have sent
    CrossRankBarrier(d, ls.epoch0 + 1);
    KernelEnd(d, ls, 1);
}

// Dispatch of a single rank: one launch, nobody to exchange counts with.  The two CTAs of a cluster count the choices of all tokens
// together, half of them each, those of tokens before the cluster's apart, and read one another's counts: offsets and the first
// row of every expert for every CTA follow without a word from another cluster, and rows are claimed from counters in shared
// memory.  Then as above: the warps share the CTA's tokens in pieces of 512 values.
// Bound by memory, and before that by the shared-memory atomics that count, during which memory is idle: hence, with many choices,
// one CTA of 1024 threads per SM and pairs of them, a quarter of the atomics of two CTAs of 512 that each count alone (the rule stands
// at LocalDispatchShape).  4096 x 7168 to 8 of 256 experts 68.5 us (71.8 with every CTA counting alone), 9000 x 512 to 16 of 1024 29.6 (49.2), 64
// tokens 7.1 (8.4).  Tried and no faster: rows put together in shared memory and sent with one bulk copy each (73 - 87 us), loads four
// pieces ahead through shared memory (74.7), clusters of four CTAs of 512 (not all resident: 87).
constexpr int kLocalThreads = 1024;

__device__ __forceinline__ uint32_t LdClusterWord(const uint32_t *mine, uint32_t rank)
{
    uint32_t addr, v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// PER: experts of a thread.
template <int PER>
__global__ void __launch_bounds__(kLocalThreads, 1) MoeDispatchLocalKernel(const __grid_constant__ MoeParams byval, const MoeParams *)
{
    const MoeParams &p = byval;         // never merged with another rank's launch
    if (p.overlaps) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const CommDev *d = p.dev;
    const LaunchState ls = KernelBeginAlone(d);
    const int E = p.lay.numExperts, K = p.lay.topk, H = p.lay.hidden;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
    // choices of tokens before the cluster's and of the others, each twice: neighbouring lanes often hold the same expert and would
    // queue for its counter, so the warps are dealt over two; and those of this CTA's tokens
    __shared__ uint32_t sCount[2][2][kMaxExperts], sOwn[kMaxExperts], sBase[kMaxExperts], sWarp[32], sSlot[kLocalThreads];      // one claim of a row per thread at a time
    uint32_t rank, ranks;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(ranks));
    const auto firstToken = [&](uint32_t cta) { return (int)((int64_t)p.numTokens * cta / gridDim.x); };
    const int t0 = firstToken(blockIdx.x), t1 = firstToken(blockIdx.x + 1), segs = H / 512, pieces = (t1 - t0) * segs;

    // the first piece of this warp, and the choice that this thread claims a row for, are on their way while the rows are being found
    uint4 a = make_uint4(0, 0, 0, 0), b = a;
    const __nv_bfloat16 *src = p.x + (size_t)t0 * H + lane * 16;         // pieces of consecutive tokens are consecutive in x
    auto fetch = [&](int item) { if (item < pieces) { a = LdStream16(src + (size_t)item * 512); b = LdStream16(src + (size_t)item * 512 + 8); } };
    fetch(warp);
    const int perRound = (int)blockDim.x / K, claimed = (t1 - t0 < perRound ? t1 - t0 : perRound) * K;
    const int choice = tid < claimed ? p.topkIdx[(size_t)t0 * K + tid] : -1;

    for (int e = tid; e < E; e += blockDim.x) sCount[0][0][e] = sCount[0][1][e] = sCount[1][0][e] = sCount[1][1][e] = sOwn[e] = 0;
    __syncthreads();
    {
        const int total = p.numTokens * K, stride = blockDim.x, before = firstToken(blockIdx.x - rank) * K;
        const int lo = (int)((int64_t)total * rank / ranks), hi = (int)((int64_t)total * (rank + 1) / ranks);
        for (int i = lo + tid; i < hi; i += 16 * stride) {        // sixteen loads in flight
            int e[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) e[u] = i + u * stride < hi ? p.topkIdx[i + u * stride] : -1;
#pragma unroll
            for (int u = 0; u < 16; ++u)
                if (e[u] >= 0 && e[u] < E) atomicAdd(&sCount[warp & 1][i + u * stride < before ? 0 : 1][e[u]], 1u);
        }
        if (ranks > 1)
            for (int i = t0 * K + tid; i < t1 * K; i += stride) {
                const int e = p.topkIdx[i];
                if (e >= 0 && e < E) atomicAdd(&sOwn[e], 1u);
            }
    }
    if (ranks > 1) cg::this_cluster().sync();
    else __syncthreads();
    uint32_t first[PER], tot[PER], all = 0;         // of this thread's experts: choices of tokens before this CTA's, of all
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int e = tid * PER + j;
        first[j] = tot[j] = 0;
        if (e < E) {
            first[j] = sCount[0][0][e] + sCount[1][0][e];
            tot[j] = sCount[0][1][e] + sCount[1][1][e];
            if (ranks > 1) {
                const uint32_t peer = rank ^ 1u;
                const uint32_t b0 = LdClusterWord(&sCount[0][0][e], peer), b1 = LdClusterWord(&sCount[1][0][e], peer);
                const uint32_t a0 = LdClusterWord(&sCount[0][1][e], peer), a1 = LdClusterWord(&sCount[1][1][e], peer), own = LdClusterWord(&sOwn[e], peer);
                first[j] += b0 + b1;
                tot[j] += a0 + a1 + first[j];
                if (rank) first[j] += own;
            } else {
                tot[j] += first[j];
            }
        }
        all += tot[j];
    }
    uint32_t start = BlockExclusiveScan(all, sWarp);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int e = tid * PER + j;
        if (e < E) {
            sBase[e] = start + first[j];
            if (blockIdx.x == 0) {
                // offsets for the grouped GEMM, clamped to the receive capacity like the route launch's
                const uint32_t cap = (uint32_t)p.lay.maxRecvRows;
                Counts(p, 0)[e] = tot[j];
                ExpertOffsets(p, 0)[e] = start < cap ? start : cap;
                if (e == E - 1) ExpertOffsets(p, 0)[E] = start + tot[j] < cap ? start + tot[j] : cap;
            }
        }
        start += tot[j];
    }
    if (ranks > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");       // its partner's counts have been read
    __syncthreads();

    if (blockIdx.x == 0 && tid == 0) p.overflow[1] = (uint32_t)p.numTokens;
    int it = warp;
    for (int r0 = t0; r0 < t1; r0 += perRound) {
        const int tokens = t1 - r0 < perRound ? t1 - r0 : perRound;
        if (tid < tokens * K) {
            const size_t tk = (size_t)r0 * K + tid;
            const int e = r0 == t0 ? choice : p.topkIdx[tk];
            uint32_t slot = kNoRow;
            if (e >= 0 && e < E) {
                slot = atomicAdd(&sBase[e], 1u);
                if (slot >= (uint32_t)p.lay.maxRecvRows) { atomicAdd(p.overflow, 1u); slot = kNoRow; }
            }
            Valid(p, 0)[tk] = slot != kNoRow ? 1 : 0;
            if (slot != kNoRow) Origin(p, 0)[slot] = (uint32_t)tk;
            p.localRow[tk] = slot + 1;          // kNoRow + 1 = 0: nowhere
            sSlot[tid] = slot;
        }
        __syncthreads();
        for (const int end = (r0 - t0 + tokens) * segs; it < end; it += warps) {
            const uint4 ca = a, cb = b;
            fetch(it + warps);
            float scale;
            const uint4 q = Quantise(ca, cb, &scale);
            const int tok = it / segs - (r0 - t0), seg = it % segs;
            uint8_t *row = Rows(p, 0) + seg * 512 + lane * 16;
            float *rowScale = Scales(p, 0) + seg * 4 + (lane >> 3);
            for (int k = 0; k < K; ++k) {
                const uint32_t slot = sSlot[tok * K + k];
                if (slot == kNoRow) continue;
                *(uint4 *)(row + (size_t)slot * H) = q;
                if ((lane & 7) == 0) rowScale[(size_t)slot * (H / kBlock)] = scale;
            }
        }
        __syncthreads();        // the claims of the next round overwrite these
    }
    if (ranks > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // nobody leaves while another reads its counts
    KernelEndAlone(d, ls);
}

// Combine, first launch: every expert output row of another rank's token (all rows with allThroughSlots) goes home, into slot (token, k) of that rank; each
// CTA then meets its namesakes on the other ranks.  When the kernel has ended on a rank, every rank's rows for it have landed.
__global__ void __launch_bounds__(512) MoeCombineSendKernel(const __grid_constant__ MoeParams byval, const MoeParams *table)
{
    MOE_ARGS;
    const CommDev *d = p.dev;
    const LaunchState ls = KernelBegin(d);
    const int n = d->nRanks, me = d->rank;
    const int El = p.lay.numExperts / n, H = p.lay.hidden;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warpsPerCta = blockDim.x >> 5;
    const int rows = (int)ExpertOffsets(p, me)[El];
    const int vecs = H / 8;                          // 16-byte vectors of bf16 per row
    for (int r = blockIdx.x * warpsPerCta + warp; r < rows; r += gridDim.x * warpsPerCta) {
        const uint64_t o = Origin(p, me)[r];
        const int src = (int)(o >> 32);
        if (src == me && !p.allThroughSlots) continue;       // the sum reads it where it is
        const uint32_t tk = (uint32_t)o;
        const uint4 *in = (const uint4 *)(p.y + (size_t)r * H);
        uint4 *dst = (uint4 *)(Comb(p, src) + (size_t)tk * H);
        // eight loads of the row in flight per lane, then their stores back to back
        for (int v0 = lane; v0 < vecs; v0 += 32 * 8) {
            uint4 buf[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (v0 + 32 * u < vecs) buf[u] = in[v0 + 32 * u];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (v0 + 32 * u < vecs) dst[v0 + 32 * u] = buf[u];
        }
    }
    CrossRankBarrier(d, ls.epoch0 + 1);
    KernelEnd(d, ls, 1);
}

// Combine, second launch (local): gate-weighted sum of the K rows of every local token, fp32 accumulation in the order of k.
// Bound by memory: 2 k H bytes in, 2 H out per token; 3001 x 7168, 8 experts each, a tenth masked, 57 us (205 with every row
// copied to its slot first), 54 at HBM rate; 64 tokens 4.5 us (13 + 43).  A warp takes segsPerItem segments of 256 columns of a token; lane k
// finds the k-th row's address one item ahead, and every lane keeps the loads of eight rows of a segment in flight.
constexpr int kSumThreads = 256, kSumCtasPerSm = 2;     // 128 registers a thread: eight addresses and gates of rows beside their loads; three CTAs spill and take 67 us for 58
// BATCHES: groups of eight rows that K calls for.  MERGED: ranks of one GPU in one launch; a choice at run time would put the
// arguments behind a pointer.
template <int BATCHES, bool MERGED>
__global__ void __launch_bounds__(kSumThreads, kSumCtasPerSm) MoeCombineSumKernel(const __grid_constant__ MoeParams byval, const MoeParams *table)
{
    MOE_ARGS_OF(MERGED);
    const CommDev *d = p.dev;
    LaunchState ls = {};
    if (p.countsLaunch) ls = KernelBeginAlone(d);
    const int me = d->rank, K = p.lay.topk, H = p.lay.hidden;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warpsPerCta = blockDim.x >> 5;
    const int segs = H / 256, perToken = (segs + p.segsPerItem - 1) / p.segsPerItem;
    const int items = p.numTokens * perToken;
    const int step = gridDim.x * warpsPerCta;
    // row, mark and gate of (token of item i, lane): looked up while the item before is being summed
    uint32_t nextRow = 0;
    uint8_t nextValid = 0;
    float nextGate = 0.f;
    const int dispatched = (int)p.overflow[1];      // marks and rows of later tokens are an older dispatch's: nothing is added for them
    auto lookUp = [&](int i) {
        const int t = i / perToken;
        nextRow = 0;
        nextValid = 0;
        if (i < items && lane < K && t < dispatched) {
            const size_t tk = (size_t)t * K + lane;
            nextRow = p.allThroughSlots ? 0u : p.localRow[tk];
            nextValid = Valid(p, me)[tk];
            nextGate = p.gates[tk];
        }
    };
    int it = blockIdx.x * warpsPerCta + warp;
    lookUp(it);
    for (; it < items; it += step) {
        const int t = it / perToken, seg0 = (it - t * perToken) * p.segsPerItem;
        const int seg1 = seg0 + p.segsPerItem < segs ? seg0 + p.segsPerItem : segs;
        uint64_t mine = 0;                          // address of row (t, lane); zero when nothing was sent: the slot then holds an older step's row
        if (lane < K) {
            if (nextRow != 0) mine = (uint64_t)(p.y + (size_t)(nextRow - 1) * H);
            else if (nextValid != 0) mine = (uint64_t)(Comb(p, me) + ((size_t)t * K + lane) * H);
        }
        const float myGate = nextGate;
        lookUp(it + step);
        const uint32_t live = __ballot_sync(0xffffffffu, mine != 0);
        for (int seg = seg0; seg < seg1; ++seg) {
            const uint32_t col = seg * 512 + lane * 16;         // bytes
            float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
            for (int kb = 0; kb < 8 * BATCHES; kb += 8) {
                uint4 pk[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint64_t row = __shfl_sync(0xffffffffu, mine, kb + k);
                    if (live >> (kb + k) & 1u) pk[k] = LdStream16((const char *)row + col);
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float g = __shfl_sync(0xffffffffu, myGate, kb + k);
                    if (!(live >> (kb + k) & 1u)) continue;
                    const __nv_bfloat162 *ph = (const __nv_bfloat162 *)&pk[k];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float2 f = __bfloat1622float2(ph[j]);
                        acc[2 * j] += g * f.x;
                        acc[2 * j + 1] += g * f.y;
                    }
                }
            }
            uint4 outv;
            uint32_t *pw = (uint32_t *)&outv;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                __nv_bfloat162 h = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
                pw[j] = *(uint32_t *)&h;
            }
            *(uint4 *)((char *)(p.out + (size_t)t * H) + col) = outv;
        }
    }
    if (p.countsLaunch) KernelEndAlone(d, ls);
}

void *SumKernel(int topk, bool merged)
{
    if (topk <= 8) return merged ? (void *)MoeCombineSumKernel<1, true> : (void *)MoeCombineSumKernel<1, false>;
    return merged ? (void *)MoeCombineSumKernel<2, true> : (void *)MoeCombineSumKernel<2, false>;
}

struct MoeCtx {
    Comm *comm;
    MoeLayout lay;
    void *buf = nullptr;          // local symmetric buffer
    HcclCommSymWindow win = nullptr;
    char *peer[HC_KERNEL_MAX_RANKS] = {nullptr};
    uint32_t *scratch = nullptr;
    uint32_t *staticScratch = nullptr;   // device address of the built-in counter table on this exchange's GPU
    int device = -1;                     // the GPU this exchange was created on
    uint32_t *overflow = nullptr;
    uint32_t *localRow = nullptr;        // [maxTokens * topk], see MoeParams
    std::atomic<bool> slotsAsked{false}; // HcommMoeGetBuffers has handed out the landing area: combine fills all of it
};
std::mutex g_mu;
std::map<void *, MoeCtx *> g_ctx;

// Where an exchange's own device block comes from; a test puts failing functions in their place.
struct DeviceBlocks {
    cudaError_t (*take)(void **, size_t);
    cudaError_t (*clear)(void *, int, size_t);
    cudaError_t (*give)(void *);
};
// One block: the row cursors, the overflow count and the last dispatch's tokens, the local rows.  On failure nothing is kept.
HcclResult MakeScratch(const DeviceBlocks &from, MoeCtx *m, int numExperts, int maxTokens, int topk)
{
    const size_t bytes = sizeof(uint32_t) * ((size_t)numExperts + 64 + (size_t)maxTokens * topk);
    void *block = nullptr;
    cudaError_t e = from.take(&block, bytes);
    if (e != cudaSuccess || !block) {
        HCCL_ERROR("MoE exchange: no device memory for its %zu bytes of counters and row numbers: %s", bytes, cudaGetErrorString(e));
        cudaGetLastError();
        return HCCL_E_MEMORY;
    }
    e = from.clear(block, 0, bytes);
    if (e != cudaSuccess) {
        HCCL_ERROR("MoE exchange: clearing its counters failed: %s", cudaGetErrorString(e));
        cudaGetLastError();
        from.give(block);
        return HCCL_E_RUNTIME;
    }
    m->scratch = (uint32_t *)block;
    m->overflow = m->scratch + numExperts;
    m->localRow = m->overflow + 64;
    return HCCL_SUCCESS;
}

uint64_t Align256(uint64_t v) { return (v + 255) & ~255ull; }

// HCOMM_MOE_CTAS: CTAs of the data-moving launches, to leave SMs to kernels running beside them (0 = not set).
int ForcedMoeCtas()
{
    static const int forced = [] { const char *e = getenv("HCOMM_MOE_CTAS"); return e ? std::max(0, atoi(e)) : 0; }();
    return std::min(forced, HC_MAX_CTAS);
}
int MoeSms()
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}
// CTAs of a launch that meets its namesakes on the other ranks: the same number on every rank, whatever it has to do.  A
// single rank meets nobody: two CTAs per SM, no more than there is work for.
int MoeCtas(const Comm *c, int sms, int64_t useful)
{
    const int forced = ForcedMoeCtas();
    if (c->nRanks > 1) return forced > 0 ? forced : std::min(sms, HC_MAX_CTAS);
    return (int)std::max<int64_t>(1, std::min<int64_t>(forced > 0 ? forced : 2 * sms, useful));
}

// One launch of `kernel` with `ctas` CTAs of `threads` threads.  Ordinary launches: nothing in these kernels waits for
// another CTA of the same launch.  Ranks that share a GPU (tests) are merged into one cooperative launch with `emuCtas`
// CTAs per rank, because their kernels wait for each other.
HcclResult LaunchMoe(MoeCtx *m, void *kernel, const MoeParams &hp, int id, void *stream, int ctas, int emuCtas, int threads, int cluster = 1)
{
    Comm *c = m->comm;
    const MoeParams *none = nullptr;
    if (c->emuSameDevice && c->nRanks > 1) {
        return EmuLaunchGeneric(c->identifier + "#moe" + std::to_string(c->group.id), c->nRanks, c->rank, id, &hp, sizeof(hp), stream,
                                [=](const void *devTable, uint32_t n, void *st) {
                                    MoeParams unused = hp;
                                    void *args[] = {(void *)&unused, (void *)&devTable};
                                    cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(emuCtas, n, 1), dim3(threads, 1, 1), args, 0, (cudaStream_t)st);
                                    if (e != cudaSuccess) { HCCL_ERROR("MoE launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
                                    return HCCL_SUCCESS;
                                });
    }
    void *args[] = {(void *)&hp, (void *)&none};
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, 1, 1); cfg.blockDim = dim3(threads, 1, 1); cfg.stream = (cudaStream_t)stream;
    cfg.attrs = at;
    if (hp.overlaps) {          // kernels that meet other ranks hold no SM before their turn
        at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        at[cfg.numAttrs].val.clusterDim.x = cluster; at[cfg.numAttrs].val.clusterDim.y = 1; at[cfg.numAttrs++].val.clusterDim.z = 1;
    }
    cudaError_t e = cudaLaunchKernelExC(&cfg, kernel, args);
    if (e != cudaSuccess) { HCCL_ERROR("MoE launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

// The launch of a single rank's dispatch; `ctas`: as many as it may have.
// Counting alone and in pairs, us: counting takes time by the choice and is the larger part where rows are small (256 experts, 8 each,
// 512 wide: 2048 tokens 11.3 and 11.4, 4096 15.7 and 13.7; 4096 wide: 2048 21.7 and 24.1, 3072 33.0 and 33.0), until there is so much to move that half as many, larger CTAs
// do it better whatever the counting (8 experts, 1 each, 8192 wide: 10000 tokens 69.6 and 67.2; 2 each: 6144 49.8 and 50.3, 8192 63.2 and 62.5).
// Beyond 512 experts a thread of 512 has two, which beats half as many CTAs of 1024 (1024 experts, 8 each: 64 x 2048 6.3 us and 7.7, 512
// x 8192 14.7 and 16.8, 1750 x 4096 19.9 and 22.7) but for many choices of small rows (1536 x 512 11.0 and 10.3).
struct DispatchShape {
    int ctas, threads, cluster;
};
DispatchShape LocalDispatchShape(int64_t tokens, int topk, int experts, int hidden, int ctas, int sms)
{
    const bool many = tokens * topk > (hidden <= 1024 ? 17000 : 24000) || tokens * hidden > 55000000;
    const bool smallRows = experts > kLocalThreads / 2 && hidden < 1024 && tokens * topk > 9000;
    const int threads = many || smallRows ? kLocalThreads : kLocalThreads / 2;
    const int mine = threads == kLocalThreads ? std::min(ctas, sms) : ctas, cluster = many && mine >= 2 ? 2 : 1;
    return {mine / cluster * cluster, threads, cluster};
}

// The launches of a dispatch; hp.scratch holds the row cursors (a single rank needs none).
HcclResult LaunchDispatch(MoeCtx *m, const MoeParams &hp, int routeId, int dispatchId, void *stream)
{
    const int sms = MoeSms(), ctas = MoeCtas(m->comm, sms, hp.numTokens), emuCtas = std::max(1, sms / (int)m->comm->nRanks);
    if (m->comm->nRanks == 1) {
        const DispatchShape l = LocalDispatchShape(hp.numTokens, m->lay.topk, m->lay.numExperts, m->lay.hidden, ctas, sms);
        void *kernel = m->lay.numExperts > l.threads ? (void *)MoeDispatchLocalKernel<2> : (void *)MoeDispatchLocalKernel<1>;
        return LaunchMoe(m, kernel, hp, dispatchId, stream, l.ctas, emuCtas, l.threads, l.cluster);
    }
    CHK_RET(LaunchMoe(m, (void *)MoeRouteKernel, hp, routeId, stream, 1, 1, 1024));
    return LaunchMoe(m, (void *)MoeDispatchKernel, hp, dispatchId, stream, ctas, emuCtas, 512);
}

}  // namespace

HcclResult LaunchBarrierIfNeeded(Comm *c, void *stream);

}  // namespace hc

using namespace hc;

// ------------------------------------------------------------------ built-in scratch of HcommMoeDispatchStaticScratch
//
// The dispatch kernel counts rows per expert in a small table of global-memory counters.  HcommMoeDispatch keeps
// that table in a cudaMalloc'ed block owned by the exchange object.  HcommMoeDispatchStaticScratch runs the SAME kernel
// with the table placed in the array below, which is part of this library's device image, so that nothing on its path
// asks any allocator for memory - neither the CUDA runtime's nor a framework's caching one.
//
// It exists for callers that must not allocate at the moment they dispatch:
//   * a serving process whose memory pool has already claimed all of the GPU, where a late cudaMalloc fails;
//   * a step in which other streams (or other ranks' kernels waiting on this rank) are in flight, where the
//     implicit device-wide synchronisation of cudaMalloc / cudaFree stalls them or lengthens a peer's wait;
//   * code that owns no handle it could hang a buffer on and would otherwise allocate and free around each call.
//
// Limits and rules:
//   * a single rank counts in shared memory and neither clears nor reads the table; the limits below hold for it all the
//     same, so that a program meets them at any number of ranks;
//   * at most kStaticScratchExperts experts (a counter each, kStaticScratchBytes of device memory per process and
//     GPU, reserved when the library is loaded); larger exchanges are refused with HCCL_E_PARA;
//   * the array's device address is looked up (cudaGetSymbolAddress) by HcommMoeCreate, which runs at set-up on the
//     exchange's GPU; the dispatch call itself does no look-up, and it refuses (HCCL_E_PARA, before anything is queued)
//     a call made while another device is current - the address belongs to the exchange's GPU only;
//   * the array is shared by every call from this process on the same GPU and keeps whatever the previous call
//     left (a call that ran out of time leaves counts behind); each call therefore zeroes the part it uses, on
//     the caller's stream, before the kernel runs;
//   * because the array is shared, two calls that overlap in time on one GPU (different streams, different
//     exchange objects) race on it: keep calls of this entry point ordered one after another per GPU;
//   * ranks of one process that share a GPU (the single-GPU test arrangement) are refused: their launches are
//     merged through a table that is created on demand, which this entry point promises not to do.
constexpr int kStaticScratchExperts = 256;
constexpr size_t kStaticScratchBytes = sizeof(uint32_t) * kStaticScratchExperts;
static __device__ __align__(256) uint32_t g_staticDispatchScratch[kStaticScratchExperts];

// Device address of the table on the CURRENT device (in host code the array's name is only a stand-in for it).
static uint32_t *ResolveStaticScratch()
{
    uint32_t *ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void **)&ptr, g_staticDispatchScratch);
    if (e != cudaSuccess || !ptr) {
        HCCL_WARNING("built-in dispatch scratch: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
        cudaGetLastError();
        return nullptr;
    }
    return ptr;
}

extern "C" {

// Collective: every rank allocates the same symmetric buffer and maps its peers'.
int HcommMoeCreate(HcclComm comm, int numExperts, int topk, int hidden, int maxTokens, float capacityFactor, void **handle, MoeLayout *layoutOut)
{
    Comm *c = AsComm(comm);
    if (!c || !handle) return HCCL_E_PTR;
    if (c->plat->kind() != PlatKind::CUDA || c->nRanks > HC_KERNEL_MAX_RANKS) return HCCL_E_NOT_SUPPORT;
    const int n = (int)c->nRanks;
    if (numExperts <= 0 || numExperts > kMaxExperts || numExperts % n || topk <= 0 || topk > 16 || hidden % 512 || hidden > 8192 || maxTokens <= 0) {
        RPT_ERR("EI0003", "MoE geometry not supported: experts %d (multiple of %d, <= %d), top-k %d (<= 16), hidden %d (multiple of 512, <= 8192)", numExperts, n, kMaxExperts, topk, hidden);
        return HCCL_E_PARA;
    }
    MoeCtx *m = new MoeCtx();
    m->comm = c;
    MoeLayout &L = m->lay;
    L.numExperts = numExperts; L.topk = topk; L.hidden = hidden; L.maxTokens = maxTokens;
    L.maxRecvRows = (int)std::max<int64_t>(1, (int64_t)((double)maxTokens * topk * (capacityFactor > 0 ? capacityFactor : 2.0)));
    uint64_t off = 0;
    L.offCounts = off; off = Align256(off + (uint64_t)n * (numExperts / n) * 4);
    L.offExpertOffsets = off; off = Align256(off + (uint64_t)(numExperts / n + 1) * 4);
    L.offOrigin = off; off = Align256(off + (uint64_t)L.maxRecvRows * 8);
    L.offScales = off; off = Align256(off + (uint64_t)L.maxRecvRows * (hidden / 128) * 4);
    L.offRows = off; off = Align256(off + (uint64_t)L.maxRecvRows * hidden);
    L.offCombine = off; off = Align256(off + (uint64_t)maxTokens * topk * hidden * 2);
    L.offValid = off; off = Align256(off + (uint64_t)maxTokens * topk);
    L.totalBytes = off;
    HcclResult r = (HcclResult)HcommMemAlloc(&m->buf, L.totalBytes);
    if (r != HCCL_SUCCESS) { delete m; return r; }
    // Taking device memory waits for the GPU, so a single rank does it last, when what the caller has queued has run beside the
    // registration.  With several ranks it comes first: taking a window back needs all of them.
    const DeviceBlocks device = {[](void **p, size_t bytes) { return cudaMalloc(p, bytes); }, cudaMemset, cudaFree};
    if (n > 1) r = MakeScratch(device, m, numExperts, maxTokens, topk);
    if (r != HCCL_SUCCESS) { HcommMemFree(m->buf); delete m; return r; }
    cudaMemset(m->buf, 0, L.offOrigin);
    r = HcclCommSymWinRegister(comm, m->buf, L.totalBytes, &m->win, 0);
    if (r == HCCL_SUCCESS && n == 1) {
        r = MakeScratch(device, m, numExperts, maxTokens, topk);
        if (r != HCCL_SUCCESS) HcclCommSymWinDeregister(m->win);
    }
    if (r != HCCL_SUCCESS) { cudaFree(m->scratch); HcommMemFree(m->buf); delete m; return r; }
    for (int q = 0; q < n; ++q) {
        void *pp = nullptr;
        HcclSymWinGetPeerPointer(m->win, 0, (uint32_t)q, &pp);
        m->peer[q] = (char *)pp;
    }
    cudaGetDevice(&m->device);
    m->staticScratch = ResolveStaticScratch();       // set-up time, the exchange's GPU is current
    cudaFuncAttributes fa;
    cudaFuncGetAttributes(&fa, MoeRouteKernel);
    cudaFuncGetAttributes(&fa, MoeDispatchKernel);
    cudaFuncGetAttributes(&fa, MoeDispatchLocalKernel<1>);
    cudaFuncGetAttributes(&fa, MoeDispatchLocalKernel<2>);
    cudaFuncGetAttributes(&fa, MoeCombineSendKernel);
    for (bool merged : {false, true}) cudaFuncGetAttributes(&fa, SumKernel(topk, merged));
    cudaDeviceSynchronize();
    *handle = m;
    if (layoutOut) *layoutOut = L;
    std::lock_guard<std::mutex> lk(g_mu);
    g_ctx[m] = m;
    return HCCL_SUCCESS;
}

int HcommMoeDestroy(void *handle)
{
    MoeCtx *m = (MoeCtx *)handle;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (!g_ctx.erase(handle)) return HCCL_E_NOT_FOUND;
    }
    cudaDeviceSynchronize();
    HcclCommSymWinDeregister(m->win);
    HcommMemFree(m->buf);
    cudaFree(m->scratch);
    delete m;
    return HCCL_SUCCESS;
}

// Local addresses of the receive-side arrays (valid after a dispatch on the same stream).
int HcommMoeGetBuffers(void *handle, void **rows, void **scales, void **origin, void **expertOffsets, void **combine)
{
    MoeCtx *m = (MoeCtx *)handle;
    if (!m) return HCCL_E_PTR;
    char *b = (char *)m->buf;
    if (rows) *rows = b + m->lay.offRows;
    if (scales) *scales = b + m->lay.offScales;
    if (origin) *origin = b + m->lay.offOrigin;
    if (expertOffsets) *expertOffsets = b + m->lay.offExpertOffsets;
    if (combine) {
        *combine = b + m->lay.offCombine;
        m->slotsAsked.store(true);
    }
    return HCCL_SUCCESS;
}

static void FillCommon(MoeCtx *m, MoeParams &hp)
{
    memset(&hp, 0, sizeof(hp));
    hp.dev = m->comm->devStruct;
    for (uint32_t q = 0; q < m->comm->nRanks; ++q) hp.peerBuf[q] = m->peer[q];
    hp.lay = m->lay;
    hp.scratch = m->scratch;
    hp.overflow = m->overflow;
    hp.localRow = m->localRow;
    hp.overlaps = m->comm->nRanks == 1;
}

int HcommMoeDispatch(void *handle, const void *x, const int32_t *topkIdx, int numTokens, void *stream)
{
    MoeCtx *m = (MoeCtx *)handle;
    if (!m || !x || !topkIdx) return HCCL_E_PTR;
    if (numTokens < 0 || numTokens > m->lay.maxTokens) return HCCL_E_PARA;
    Comm *c = m->comm;
    std::lock_guard<std::mutex> lk(c->opMu);
    int st = c->state.load();
    if (st == (int)CommState::SUSPENDING || st == (int)CommState::SUSPENDED) return HCCL_E_SUSPENDING;
    CHK_RET(LaunchBarrierIfNeeded(c, stream));
    MoeParams hp;
    FillCommon(m, hp);
    hp.x = (const __nv_bfloat16 *)x; hp.topkIdx = topkIdx; hp.numTokens = numTokens;
    ++c->opSeq;
    return LaunchDispatch(m, hp, 9100, 9101, stream);
}

int HcommMoeCombine(void *handle, const void *y, const float *gates, void *out, int numTokens, void *stream)
{
    // how many rows y has is not known here: as many as can be received
    return HcommMoeCombineRows(handle, y, handle ? (uint64_t)((MoeCtx *)handle)->lay.maxRecvRows : 0, gates, out, numTokens, stream);
}

int HcommMoeCombineRows(void *handle, const void *y, uint64_t yRows, const float *gates, void *out, int numTokens, void *stream)
{
    MoeCtx *m = (MoeCtx *)handle;
    if (!m || !y || !gates || !out) return HCCL_E_PTR;
    if (numTokens < 0 || numTokens > m->lay.maxTokens) return HCCL_E_PARA;
    Comm *c = m->comm;
    std::lock_guard<std::mutex> lk(c->opMu);
    int st = c->state.load();
    if (st == (int)CommState::SUSPENDING || st == (int)CommState::SUSPENDED) return HCCL_E_SUSPENDING;
    CHK_RET(LaunchBarrierIfNeeded(c, stream));
    MoeParams hp;
    FillCommon(m, hp);
    hp.y = (const __nv_bfloat16 *)y; hp.gates = gates; hp.out = (__nv_bfloat16 *)out; hp.numTokens = numTokens;
    ++c->opSeq;
    const uintptr_t yBegin = (uintptr_t)y, yEnd = yBegin + yRows * m->lay.hidden * 2;
    const uintptr_t outBegin = (uintptr_t)out, outEnd = outBegin + (uint64_t)numTokens * m->lay.hidden * 2;
    hp.allThroughSlots = m->slotsAsked.load() || (outBegin < yEnd && yBegin < outEnd);
    const int sms = MoeSms(), emuCtas = std::max(1, sms / (int)c->nRanks), segs = m->lay.hidden / 256;
    if (c->nRanks > 1 || hp.allThroughSlots) {
        const int forced = ForcedMoeCtas();
        CHK_RET(LaunchMoe(m, (void *)MoeCombineSendKernel, hp, 9102, stream, forced > 0 ? forced : std::min(sms, HC_MAX_CTAS), emuCtas, 512));
    } else {
        hp.countsLaunch = 1;
    }
    // four segments to a warp where that still fills every SM's warps (the row addresses are then found once for all four),
    // single segments below
    constexpr int warps = kSumThreads / 32;
    hp.segsPerItem = (int64_t)numTokens * ((segs + 3) / 4) >= (int64_t)warps * kSumCtasPerSm * sms ? 4 : 1;
    const int64_t items = (int64_t)numTokens * ((segs + hp.segsPerItem - 1) / hp.segsPerItem);
    const int forced = ForcedMoeCtas(), most = forced > 0 ? forced : kSumCtasPerSm * sms;
    return LaunchMoe(m, SumKernel(m->lay.topk, c->emuSameDevice && c->nRanks > 1), hp, 9104, stream, (int)std::max<int64_t>(1, std::min<int64_t>(most, (items + warps - 1) / warps)), emuCtas, kSumThreads);
}

// ------------------------------------------------------------------ dispatch without any allocation
//
// See the comment at g_staticDispatchScratch (top of the host section) for what this entry point is for and its rules.
int HcommMoeDispatchStaticScratch(void *handle, const void *x, const int32_t *topkIdx, int numTokens, void *stream)
{
    MoeCtx *m = (MoeCtx *)handle;
    if (!m || !x || !topkIdx) return HCCL_E_PTR;
    if (numTokens < 0 || numTokens > m->lay.maxTokens) return HCCL_E_PARA;
    Comm *c = m->comm;
    if (m->lay.numExperts > kStaticScratchExperts) {
        RPT_ERR("EI0003", "HcommMoeDispatchStaticScratch serves at most %d experts (%zu bytes of built-in scratch); this exchange has %d - use HcommMoeDispatch",
                kStaticScratchExperts, kStaticScratchBytes, m->lay.numExperts);
        return HCCL_E_PARA;
    }
    if (c->emuSameDevice && c->nRanks > 1) {
        RPT_ERR("EI0003", "HcommMoeDispatchStaticScratch does not serve several ranks of one process on one GPU - use HcommMoeDispatch");
        return HCCL_E_NOT_SUPPORT;
    }
    // The table's address belongs to the GPU the exchange was created on; with another device current the launch
    // below would go elsewhere.  Checked before anything is queued or counted.
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != m->device) {
        RPT_ERR("EI0003", "HcommMoeDispatchStaticScratch called with device %d current; the exchange lives on device %d", dev, m->device);
        return HCCL_E_PARA;
    }
    if (!m->staticScratch) {
        RPT_ERR("EI0003", "the built-in dispatch scratch could not be resolved when this exchange was created - use HcommMoeDispatch");
        return HCCL_E_NOT_SUPPORT;
    }
    std::lock_guard<std::mutex> lk(c->opMu);
    int st = c->state.load();
    if (st == (int)CommState::SUSPENDING || st == (int)CommState::SUSPENDED) return HCCL_E_SUSPENDING;
    CHK_RET(LaunchBarrierIfNeeded(c, stream));
    // the array may hold a previous call's leftovers
    if (c->nRanks > 1 && cudaMemsetAsync(m->staticScratch, 0, sizeof(uint32_t) * (size_t)m->lay.numExperts, (cudaStream_t)stream) != cudaSuccess) {
        HCCL_ERROR("built-in dispatch scratch: clearing failed: %s", cudaGetErrorString(cudaGetLastError()));
        return HCCL_E_RUNTIME;
    }
    MoeParams hp;
    FillCommon(m, hp);
    hp.scratch = m->staticScratch;
    hp.x = (const __nv_bfloat16 *)x; hp.topkIdx = topkIdx; hp.numTokens = numTokens;
    ++c->opSeq;
    return LaunchDispatch(m, hp, 9105, 9103, stream);
}

// The launch of a single rank's dispatch: shape = CTAs, threads of each, CTAs that count together.
void HcommToolMoeDispatchShape(int tokens, int topk, int experts, int hidden, int ctas, int sms, int *shape)
{
    const DispatchShape l = LocalDispatchShape(tokens, topk, experts, hidden, ctas, sms);
    shape[0] = l.ctas; shape[1] = l.threads; shape[2] = l.cluster;
}

// An exchange's device block from stand-in allocators in host memory: failing 0 = none, 1 = taking it, 2 = clearing it.
// *blocksLeft: blocks taken and not given back.  Returns what HcommMoeCreate would; on success the parts' offsets in words.
int HcommToolMoeScratch(int numExperts, int maxTokens, int topk, int failing, int *blocksLeft, uint64_t *overflowAt, uint64_t *localRowAt)
{
    static thread_local int fail, taken;
    fail = failing;
    taken = 0;
    const DeviceBlocks host = {[](void **p, size_t n) { if (fail == 1) return cudaErrorMemoryAllocation; ++taken; *p = malloc(n); return *p ? cudaSuccess : cudaErrorMemoryAllocation; },
                               [](void *p, int v, size_t n) { if (fail == 2) return cudaErrorUnknown; memset(p, v, n); return cudaSuccess; },
                               [](void *p) { --taken; free(p); return cudaSuccess; }};
    MoeCtx m;
    const HcclResult r = MakeScratch(host, &m, numExperts, maxTokens, topk);
    if (blocksLeft) *blocksLeft = taken;
    if (r == HCCL_SUCCESS) {
        if (overflowAt) *overflowAt = (uint64_t)(m.overflow - m.scratch);
        if (localRowAt) *localRowAt = (uint64_t)(m.localRow - m.scratch);
        free(m.scratch);
    } else if (m.scratch || m.overflow || m.localRow) {
        return HCCL_E_INTERNAL;             // a part of a block that is not there
    }
    return r;
}

// Rows dropped because a rank received more than its capacity since the last call (clears the counter).
int HcommMoeTakeOverflow(void *handle)
{
    MoeCtx *m = (MoeCtx *)handle;
    if (!m) return -1;
    uint32_t v = 0, zero = 0;
    cudaMemcpy(&v, m->overflow, 4, cudaMemcpyDeviceToHost);
    if (v) cudaMemcpy(m->overflow, &zero, 4, cudaMemcpyHostToDevice);
    return (int)v;
}

}  // extern "C"
