// gemm_sm100_swap.cuh - the CTA-pair bf16 GEMM with the operands' roles exchanged: the rows of B (a layer's weights, N of
// them) are the 256 rows of the MMA tile and the rows of A (tokens, M of them) its columns.
//
//   C[M,N] = A[M,K] * B[N,K]^T      tile = 256 weights x bn tokens, bn = 32 .. 256 in steps of 32, chosen at launch
//
// Same machinery as gemm_sm100_2sm.cuh (tcgen05 cta_group::2, both CTAs' loads completing on the pair leader's barrier,
// two-CTA commits).  What the exchange buys:
//   * the tensor core's row count is 128 or 256, whatever is asked of it, but its column count follows in steps of 32.
//     Weights come in multiples of 256 nearly always, tokens in any number: 16 decoded tokens cost a 32-column tile
//     instead of 128 or 256 rows of which 16 are real, and 777 tokens cost 800 columns instead of 1024 rows;
//   * edges need no other kernel: TMA fills rows beyond M and N with zeros and the epilogue leaves them out.
// SPLIT pairs of one cluster share a tile along K (1 to 4 pairs): each multiplies its part of K, parks its fp32
// accumulator in its own shared memory (the ring is idle by then), and after one cluster barrier every pair adds the
// SPLIT partial sums of its share of the tokens over distributed shared memory, in the order of K.  Nothing goes through
// global memory, nothing has to be cleared, no CTA waits for one that may not be resident, and the result does not
// depend on timing.  It is for shapes with fewer tiles than the chip has pairs, where most SMs would stand idle while
// a few read a deep K.
// Every wait is bounded; all CTAs of a cluster meet at the barriers behind the roles whether their waits held or not.
#pragma once
#include "gemm_sm100_2sm.cuh"

namespace hcgemm {

constexpr int kSwapThreads = 320;       // producer, MMA issuer and eight epilogue warps: two per 32-lane quarter of tensor memory
constexpr int kSwapMaxStages = 12;
constexpr int kSwapSlab = 16 * 32 * 4;  // per epilogue warp: 16 pairs of tokens x 32 weights, one word per pair and weight

struct SwapState {
    uint64_t full[kSwapMaxStages], empty[kSwapMaxStages], tmemFull[2], tmemEmpty[2];
    uint32_t tmemBase;
    volatile uint32_t abort;
};

struct SwapShape {
    int M, N, K;
    int tilesW, tilesT;      // blocks of 256 weights, of bn tokens
    int bn, stages;
    int group;               // weight blocks per rasterisation group, 1 .. tilesW
    __nv_bfloat16 *C;
    int ldc;
    uint32_t *errFlag;
};

// Tile t's block of weights and of tokens: walks the weight blocks of a group for one token block, then for the next, so that
// the pairs in flight share both operands' panels in L2.
__host__ __device__ inline void SwapOrder(const SwapShape &g, int t, int *wb, int *tb)
{
    const int perGroup = g.group * g.tilesT, gi = t / perGroup, rem = t % perGroup;
    const int left = g.tilesW - gi * g.group, here = left < g.group ? left : g.group;
    *tb = rem / here;
    *wb = gi * g.group + rem % here;
}

__host__ __device__ constexpr int SwapStageBytes(int bn) { return (kBlockM + bn / 2) * kBlockK * 2; }
constexpr int kSwapFixedSmem = 8 * kSwapSlab + (int)sizeof(SwapState) + 1024 /* alignment slack */;
// Ring depth: what 227 KB hold.  A split tile parks bn x 128 fp32 values in the ring, which any depth of these covers.
__host__ __device__ constexpr int SwapStages(int bn)
{
    const int n = (227 * 1024 - kSwapFixedSmem) / SwapStageBytes(bn);
    return n < kSwapMaxStages ? n : kSwapMaxStages;
}
__host__ __device__ constexpr int SwapSmemBytes(int bn) { return SwapStages(bn) * SwapStageBytes(bn) + kSwapFixedSmem; }

namespace pair {
__device__ __forceinline__ void MmaCommitPairMask(uint64_t *bar, uint16_t mask)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(SmemAddr(bar)), "h"(mask) : "memory");
}
__device__ __forceinline__ float4 LdCluster16(uint32_t clusterAddr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(clusterAddr) : "memory");
    return v;
}
}  // namespace pair

__device__ __forceinline__ uint32_t PackBf16(float lo, float hi)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *(const uint32_t *)&h;
}

// Launch with clusters of 2 * SPLIT CTAs along x; with SPLIT > 1 one cluster per tile.
template <int SPLIT>
__device__ __forceinline__ void GemmMainLoopSwap(const CUtensorMap *tmW, const CUtensorMap *tmX, const SwapShape &g)
{
    using namespace pair;
    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
    const int stageBytes = SwapStageBytes(g.bn), aBytes = kBlockM * kBlockK * 2;
    uint8_t *slabs = smem + g.stages * stageBytes;
    SwapState *st = (SwapState *)(slabs + 8 * kSwapSlab);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rankInCluster = ClusterCtaRank();
    const int half = (int)(rankInCluster & 1u), part = SPLIT > 1 ? (int)(rankInCluster >> 1) : 0;
    const uint32_t leaderRank = rankInCluster & ~1u;
    const bool leader = half == 0;
    const int numTiles = g.tilesW * g.tilesT;
    const int kBlocks = (g.K + kBlockK - 1) / kBlockK;
    const int kFirst = kBlocks * part / SPLIT, kLast = kBlocks * (part + 1) / SPLIT;
    const int firstTile = (int)ClusterId(), tileStep = (int)NumClusters();

    if (threadIdx.x < (unsigned)g.stages) {
        MbarInit(&st->full[threadIdx.x], 1);
        MbarInit(&st->empty[threadIdx.x], 1);
        if (threadIdx.x < 2) {
            MbarInit(&st->tmemFull[threadIdx.x], 1);
            MbarInit(&st->tmemEmpty[threadIdx.x], 16);      // 8 epilogue warps x 2 CTAs
        }
        if (threadIdx.x == 0) st->abort = 0;
        MbarFenceInit();
    }
    if (threadIdx.x == 64) { TmaPrefetchDescriptor(tmW); TmaPrefetchDescriptor(tmX); }
    if (warp == 1) {
        TmemAlloc2(&st->tmemBase, 512);
        TmemRelinquish2();
    }
    GridDependentsLaunch();
    TcFenceBefore();
    __syncthreads();
    ClusterSync();          // every barrier of the cluster is initialised before anything signals it
    TcFenceAfter();
    const uint32_t tmemBase = st->tmemBase;

    // Every role waits for the kernel in front before its first bounded wait, not only the producer: the bound must not run
    // down while that kernel still works.
    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer (both CTAs of a pair)
        if (ElectOne()) {
            int s = 0;
            uint32_t ph = 0;
            bool alive = true;
            GridDependencyWait();           // up to here a CTA may run beside the tail of the kernel in front; all it writes follows its loads
            for (int t = firstTile; t < numTiles && alive; t += tileStep) {
                int wb, tb;
                SwapOrder(g, t, &wb, &tb);
                const int wRow = (wb * 2 + half) * kBlockM, xRow = tb * g.bn + half * (g.bn / 2);
                for (int kb = kFirst; kb < kLast; ++kb) {
                    if (!MbarWait(&st->empty[s], ph ^ 1, &st->abort)) { alive = false; break; }
                    uint8_t *sa = smem + s * stageBytes;
                    if (leader) MbarExpectTx(&st->full[s], 2 * stageBytes);      // both CTAs' loads land on this barrier
                    const uint32_t bar = MapToCta(&st->full[s], leaderRank);
                    TmaLoad2dPair(sa, tmW, bar, kb * kBlockK, wRow);
                    TmaLoad2dPair(sa + aBytes, tmX, bar, kb * kBlockK, xRow);
                    if (++s == g.stages) { s = 0; ph ^= 1; }
                }
            }
            if (!alive) __nanosleep(500000);        // copies already issued land long before this ends
        }
    } else if (warp == 1) {
        // -------------------------------------------------------------------- MMA issuer (the pair's leader only)
        if (leader && ElectOne()) {
            const uint32_t idesc = InstrDescBf16(kPairM, (uint32_t)g.bn);
            const uint16_t mask = (uint16_t)(3u << leaderRank);
            int s = 0;
            uint32_t ph = 0, tileIter = 0;
            bool alive = true;
            GridDependencyWait();
            for (int t = firstTile; t < numTiles && alive; t += tileStep, ++tileIter) {
                const uint32_t acc = tileIter & 1, accPh = (tileIter >> 1) & 1;
                if (!MbarWait(&st->tmemEmpty[acc], accPh ^ 1, &st->abort)) { alive = false; break; }
                TcFenceAfter();
                const uint32_t tmemD = tmemBase + acc * 256;
                for (int kb = kFirst; kb < kLast; ++kb) {
                    if (!MbarWait(&st->full[s], ph, &st->abort)) { alive = false; break; }
                    TcFenceAfter();
                    uint8_t *sa = smem + s * stageBytes;
                    const uint64_t da = SmemDescKMajorSw128(sa), db = SmemDescKMajorSw128(sa + aBytes);
#pragma unroll
                    for (int k = 0; k < kBlockK / kUmmaK; ++k) MmaBf16Pair(tmemD, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, kb != kFirst || k != 0);
                    MmaCommitPairMask(&st->empty[s], mask);
                    if (++s == g.stages) { s = 0; ph ^= 1; }
                }
                if (alive) MmaCommitPairMask(&st->tmemFull[acc], mask);
            }
        }
    } else if constexpr (SPLIT == 1) {
        // ---------------------------------------------------------------------- epilogue (both CTAs)
        // A lane holds one weight's column of results; C wants the weights of a token side by side.  Each warp turns
        // blocks of 32 tokens x 32 weights through a 2 KB slab, two tokens to a word (16 word writes, free of bank
        // conflicts), and writes 64-byte pieces of token rows.  The two warps of a quarter take every second block.
        const int q = warp & 3, odd = (warp - 2) >> 2;
        uint32_t *slab = (uint32_t *)(slabs + (warp - 2) * kSwapSlab);
        const int chunk = lane & 3, pair0 = lane >> 2;
        uint32_t tileIter = 0;
        bool alive = true;
        GridDependencyWait();
        for (int t = firstTile; t < numTiles && alive; t += tileStep, ++tileIter) {
            int wb, tb;
            SwapOrder(g, t, &wb, &tb);
            const uint32_t acc = tileIter & 1, accPh = (tileIter >> 1) & 1;
            if (!MbarWait(&st->tmemFull[acc], accPh, &st->abort)) { alive = false; break; }
            TcFenceAfter();
            const int n0 = wb * kPairM + half * kBlockM + q * 32, t0 = tb * g.bn;
            const int tokens = g.M - t0 < g.bn ? g.M - t0 : g.bn;
            const int col = n0 + chunk * 8;
            if (n0 < g.N) {
#pragma unroll 1
                for (int c = odd * 32; c < tokens; c += 64) {
                    uint32_t f[32];
                    TmemLoad32x32(tmemBase + ((uint32_t)(q * 32) << 16) + acc * 256 + c, f);
                    TmemLoadWait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) slab[j * 32 + lane] = PackBf16(__uint_as_float(f[2 * j]), __uint_as_float(f[2 * j + 1]));
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int pr = pair0 + 8 * i, tok = c + 2 * pr;
                        const uint4 a = *(const uint4 *)(slab + pr * 32 + chunk * 8), b = *(const uint4 *)(slab + pr * 32 + chunk * 8 + 4);
                        if (col < g.N) {
                            __nv_bfloat16 *dst = g.C + (size_t)(t0 + tok) * g.ldc + col;
                            if (tok < tokens)
                                *(uint4 *)dst = make_uint4(__byte_perm(a.x, a.y, 0x5410), __byte_perm(a.z, a.w, 0x5410), __byte_perm(b.x, b.y, 0x5410), __byte_perm(b.z, b.w, 0x5410));
                            if (tok + 1 < tokens)
                                *(uint4 *)(dst + g.ldc) = make_uint4(__byte_perm(a.x, a.y, 0x7632), __byte_perm(a.z, a.w, 0x7632), __byte_perm(b.x, b.y, 0x7632), __byte_perm(b.z, b.w, 0x7632));
                        }
                    }
                    __syncwarp();
                }
            }
            TcFenceBefore();
            __syncwarp();
            if (lane == 0) {
                if (leader) MbarArrive(&st->tmemEmpty[acc]);
                else RemoteArrive(MapToCta(&st->tmemEmpty[acc], leaderRank));
            }
        }
    } else {
        // ------------------------------------------- split along K: the accumulator goes to this CTA's shared memory
        // as fp32 rows of 128 weights per token.  The ring is free: the accumulator is complete, so all loads have
        // landed and all MMAs that read them have finished.
        const int q = warp & 3, odd = (warp - 2) >> 2;
        int wb, tb;
        SwapOrder(g, firstTile, &wb, &tb);
        const int tokens = g.M - tb * g.bn < g.bn ? g.M - tb * g.bn : g.bn;
        GridDependencyWait();
        if (MbarWait(&st->tmemFull[0], 0, &st->abort)) {
            TcFenceAfter();
            float *mine = (float *)smem + q * 32 + lane;
#pragma unroll 1
            for (int c = odd * 32; c < tokens; c += 64) {
                uint32_t f[32];
                TmemLoad32x32(tmemBase + ((uint32_t)(q * 32) << 16) + c, f);
                TmemLoadWait();
#pragma unroll
                for (int j = 0; j < 32; ++j) mine[(c + j) * 128] = __uint_as_float(f[j]);
            }
        }
    }
    TcFenceBefore();
    __syncthreads();
    ClusterSync();
    if constexpr (SPLIT > 1) {
        int wb, tb;
        SwapOrder(g, firstTile, &wb, &tb);
        const int t0 = tb * g.bn, tokens = g.M - t0 < g.bn ? g.M - t0 : g.bn;
        const int per = (tokens + SPLIT - 1) / SPLIT, lo = part * per, hi = lo + per < tokens ? lo + per : tokens;
        const int n = wb * kPairM + half * kBlockM + lane * 4;
        uint32_t base[SPLIT];
#pragma unroll
        for (int s = 0; s < SPLIT; ++s) base[s] = MapToCta(smem + lane * 16, (uint32_t)(2 * s + half));
        // a pair whose wait ran out has parked nothing: the error flag below says so, and what is written here is void
        for (int t = lo + warp; t < hi; t += kSwapThreads / 32) {
            float4 v[SPLIT];
#pragma unroll
            for (int s = 0; s < SPLIT; ++s) v[s] = LdCluster16(base[s] + (uint32_t)t * 512u);
#pragma unroll
            for (int s = 1; s < SPLIT; ++s) { v[0].x += v[s].x; v[0].y += v[s].y; v[0].z += v[s].z; v[0].w += v[s].w; }
            if (n < g.N) *(uint2 *)(g.C + (size_t)(t0 + t) * g.ldc + n) = make_uint2(PackBf16(v[0].x, v[0].y), PackBf16(v[0].z, v[0].w));
        }
        ClusterSync();      // nobody leaves while its shared memory is being read
    }
    if (warp == 1) TmemDealloc2(tmemBase, 512);
    if (threadIdx.x == 0 && st->abort && g.errFlag) atomicExch(g.errFlag, 1u);
}

}  // namespace hcgemm
