// gemm_sm100.cu - the plain bf16 GEMM on the tcgen05 main loop, and the host-side tensor-map helper
// used by every kernel that loads tiles with TMA.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "../core/log.h"
#include "../core/per_device.h"
#include "gemm_api.h"
#include "gemm_sm100.cuh"
#include "gemm_sm100_2sm.cuh"
#include "gemm_sm100_2sm_wide.cuh"
#include "gemm_sm100_swap.cuh"

namespace hc {

namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
std::once_flag g_encodeOnce;

template <int BN>
__global__ void __launch_bounds__(hcgemm::kThreads, 1)
GemmBf16Kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, hcgemm::GemmShape shape, hcgemm::StoreBf16 epi)
{
    hcgemm::GemmMainLoop<BN>(&tmA, &tmB, shape, hcgemm::GroupedOrder{shape.tilesM < 16 ? shape.tilesM : 16}, hcgemm::NoGate(), epi);
}
// 256 x 512 tiles, one accumulator per CTA (see gemm_sm100_2sm_wide.cuh).
__global__ void __launch_bounds__(hcgemm::kWideThreads, 1)
GemmBf16PairWideKernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC, hcgemm::GemmShape shape, int gm)
{
    hcgemm::GemmMainLoopPairWide<4>(&tmA, &tmB, &tmC, shape, hcgemm::GroupedOrder{shape.tilesM < gm ? shape.tilesM : gm});
}

// 256 x 224 tiles with the tokens as rows (see gemm_sm100_2sm.cuh).
__global__ void __launch_bounds__(hcgemm::kThreads, 1)
GemmBf16Pair224Kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, hcgemm::GemmShape shape, hcgemm::StoreBf16 epi, int gm)
{
    hcgemm::GemmMainLoopPair<224, 7>(&tmA, &tmB, shape, hcgemm::GroupedOrder{shape.tilesM < gm ? shape.tilesM : gm}, epi);
}

// 256 weights x bn tokens, SPLIT pairs of a cluster along K (see gemm_sm100_swap.cuh).
template <int SPLIT>
__global__ void __launch_bounds__(hcgemm::kSwapThreads, 1)
GemmBf16SwapKernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, hcgemm::SwapShape shape)
{
    hcgemm::GemmMainLoopSwap<SPLIT>(&tmW, &tmX, shape);
}

// What the plain GEMM's kernels find on a device: clusters of 1 to 4 CTA pairs that it holds at once, 0 where a kernel
// cannot run, and whether the kernels without pairs have their shared memory.
struct GemmLimits {
    int cap[4];
    bool single;
};
template <typename Kernel> bool AllowShared(Kernel *kernel, int bytes)
{
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}
template <int SPLIT> bool ClustersAtOnce(int *n)
{
    *n = 0;
    if (!AllowShared(GemmBf16SwapKernel<SPLIT>, 227 * 1024)) return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * SPLIT * 148, 1, 1);
    cfg.blockDim = dim3(hcgemm::kSwapThreads, 1, 1);
    cfg.dynamicSmemBytes = hcgemm::SwapSmemBytes(256);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2 * SPLIT; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(n, GemmBf16SwapKernel<SPLIT>, &cfg) != cudaSuccess) { cudaGetLastError(); *n = 0; return false; }
    HCCL_INFO("GEMM clusters of %d CTAs resident at once: %d", 2 * SPLIT, *n);
    return true;
}
// cap[i] = what ask(pairs of a cluster, &n) says of i + 1; false where one of them failed: that is no answer to keep, unlike none at once.
template <typename Ask> bool ClusterCaps(int *cap, Ask ask)
{
    bool all = true;
    for (int pairs = 1; pairs <= 4; ++pairs) all = ask(pairs, &cap[pairs - 1]) && all;
    return all;
}
// The limits of the current device: shared memory limits are a device's own, so its first call sets them.
GemmLimits Limits()
{
    static PerDevice<GemmLimits> limits;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return {}; }
    return limits.Get(dev, [](GemmLimits *l) {
        const bool wide = AllowShared(GemmBf16PairWideKernel, hcgemm::ConfigWide<4>::kSmemBytes) && AllowShared(GemmBf16Pair224Kernel, hcgemm::Config2<224, 7>::kSmemBytes);
        const bool clusters = ClusterCaps(l->cap, [](int pairs, int *n) {
            return pairs == 1 ? ClustersAtOnce<1>(n) : pairs == 2 ? ClustersAtOnce<2>(n) : pairs == 3 ? ClustersAtOnce<3>(n) : ClustersAtOnce<4>(n);
        });
        if (!wide) l->cap[0] = 0;
        l->single = AllowShared(GemmBf16Kernel<256>, hcgemm::Config<256>::kSmemBytes) && AllowShared(GemmBf16Kernel<128>, hcgemm::Config<128>::kSmemBytes);
        return wide && clusters && l->single;
    });
}

}  // namespace

HcclResult MakeTensorMap2dBf16(CUtensorMap *map, const void *base, uint64_t rows, uint64_t cols, uint64_t ldElems, uint32_t boxRows, uint32_t boxCols)
{
    std::call_once(g_encodeOnce, [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess) g_encode = (EncodeTiledFn)fn;
        cudaGetLastError();
    });
    if (!g_encode) {
        HCCL_ERROR("cuTensorMapEncodeTiled is not available from this driver");
        return HCCL_E_DRV;
    }
    if (((uintptr_t)base & 15) != 0 || (ldElems * 2) % 16 != 0) {
        HCCL_ERROR("TMA needs a 16-byte aligned base and row pitch (base %p, pitch %llu bytes)", base, (unsigned long long)(ldElems * 2));
        return HCCL_E_PARA;
    }
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {ldElems * 2};
    cuuint32_t box[2] = {boxCols, boxRows};
    cuuint32_t elemStrides[2] = {1, 1};
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, elemStrides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        HCCL_ERROR("cuTensorMapEncodeTiled failed with %d (rows %llu cols %llu ld %llu box %ux%u)", (int)r, (unsigned long long)rows,
                   (unsigned long long)cols, (unsigned long long)ldElems, boxRows, boxCols);
        return HCCL_E_DRV;
    }
    return HCCL_SUCCESS;
}

// Row blocks (256 rows) per rasterisation group of the CTA-pair kernels.  The tiles in flight cover gm row blocks by
// pairs / gm column blocks; the gm A panels are what consecutive waves share, so they should stay in L2.  The L2 is two
// partitions and a panel that both halves of the chip read occupies both, so the budget is about half the nominal 126 MB.
// HCOMM_GEMM_GM or HcommGemmSetTuning override the choice.
namespace {
std::atomic<int> g_forceGm{-1}, g_forceBn{-1}, g_forceSplit{0};
}
int PairGroupRows(int K)
{
    int forced = g_forceGm.load();
    if (forced < 0) {
        const char *e = getenv("HCOMM_GEMM_GM");
        forced = e ? atoi(e) : 0;
        g_forceGm.store(forced);
    }
    if (forced > 0) return forced;
    // Never below 8: a wave of 74 tiles laid out as r rows x c columns loads r + c panels, least at r = c = 8.6, and DRAM
    // counters on B200 confirm it for deep K too, where the group's A panels exceed the L2 anyway (8192 x 8192 x 28672:
    // 6.5 GB read at 8 or 16 row blocks per group, 8.8 GB at 4, 9.7 GB at 2; ideal 0.9 GB).
    const double panelMB = 256.0 * K * 2 / (1 << 20);
    int gm = 16;
    while (gm > 8 && gm * panelMB > 40.0) gm /= 2;
    return gm;
}
int ForcedPairTileWidth()
{
    int forced = g_forceBn.load();
    if (forced < 0) {
        const char *e = getenv("HCOMM_GEMM_BN");
        forced = e ? atoi(e) : 0;
        g_forceBn.store(forced);
    }
    return forced;
}

int GemmSmCount()
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    return sms;
}

uint32_t *GemmErrorFlag()
{
    static thread_local uint32_t *flag[16] = {nullptr};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 16) dev = 0;
    if (!flag[dev]) {
        cudaMalloc(&flag[dev], sizeof(uint32_t));
        cudaMemset(flag[dev], 0, sizeof(uint32_t));
    }
    return flag[dev];
}

namespace {

// Tile of the CTA-pair kernels for a shape: tokens per tile and pairs that share a tile along K for the one with exchanged
// operands (gemm_sm100_swap.cuh), or 256 x 512 (gemm_sm100_2sm_wide.cuh).  The estimate below, in nanoseconds, was fitted to
// timings of every tile at about 1600 shapes (M 1 .. 65536, N 8 .. 128256, K 64 .. 28672).  It is not the best everywhere: of
// 150 shapes up to 700 tokens 11 are 4 - 13 % off their best tile.
//   * a 64-deep step of a 256 x bn tile takes 48 + 1.28 bn ns on the tensor core at the clock that a GPU under such load
//     holds, but never less than its operands (16 KB of weights, 128 bytes per token and CTA) at 120 bytes per ns and SM;
//   * tiles come in whole waves of the clusters that fit at once (74 of two CTAs, 33 of four, 22 of six, 15 of eight);
//   * a tile's accumulator is emptied while the next tile is multiplied, in 1 us and 0.5 for every 64 tokens begun.  Where K is
//     shallow neither hides the other: measured, the two add up like the sides of a right angle (256 tokens, K of 64 / 256 /
//     512: 2.7 / 3.1 / 4.2 us a tile; multiplying alone 0.4 / 1.5 / 3.0), which makes wide tiles the better ones:
//     65536 x 4096 x 64 takes 119 us with 512/1, 310 with 64/1;
//   * all operand traffic passes L2 at 13.5 TB/s, half as much again where K is no multiple of 64, so that rows straddle
//     128-byte lines (seen from the third wave on: 16384 x 4096 x 1000 512/1 107 us, 256/1 122); every operand comes from HBM
//     once at 6.5 TB/s, a tenth less when only a few SMs ask for it;
//     up to 256 tokens, where weights come from HBM and go to every token tile, a fifth of the L2 time adds to that of HBM
//     (64 x 4096 x 4096 64/3 10.4 us, not 32/2 11.4);
//   * a launch costs 3 us, emptying the last accumulator 6 ns per token, exchanging partial sums 0.6 us and 10 ns per token (three
//     pairs up to 128 tokens only: beyond them they won nothing).
//     Tiles are shared along K only where their clusters all fit at once: a further wave starts from nothing.
//     Beyond 128 tokens the exchange costs more than this where a call follows its like: 8192 x 3584, 174 tokens 192/2 18.1 us, 96/1 17.8;
//     227 256/2 20.4, 128/1 19.7.  Priced at 18 ns for each such token a first call takes longer (33.5 us for 30.5) and two layers together
//     no less (176 and 223 tokens through 8192 / 3584 37.4 and 41.0 for 37.2 and 40.8), so the price stays;
//   * a 256 x 512 tile moves a quarter less operand data than two of 256 x 256, and under the power cap that sets the clock:
//     690 ns a step against 752, but 4 us in which nothing overlaps the emptying of its one accumulator.
// Examples, us, against the fixed choice before (128 x 256 tiles of one CTA below 256 rows or at ragged ones):
// 16 x 8192 x 28672 32/2 71 (165), 96 x 3584 x 8192 96/4 15 (51), 777 x 4096 x 14336 224/1 82 (97), 33 x 128256 x 4096
// 64/1 165 (185), 5003 x 8192 x 3584 224/1 210 (235).  Half a second into a run at the power cap 8192 x 28672 x 8192 takes
// 2929 with 256 x 512 and 3149 with 256 x 256 tiles (from a cool start 2988 and 2783), 8192 x 3584 x 8192 414 and 395.
//
// Results of at most 128 columns fill less than half of a tile's 256 weights, and all clusters read the same few lines of B at
// the same time, which costs each step some ns for every cluster beyond 30.  The kernel without pairs (128 x 128 tiles, one
// per SM) is the better one there from 2048 rows and up to a K of 1024, beyond 148 tiles up to 512: 16384 x 8 x 256 5.1 us (6.9
// with the best exchanged tile), 8192 x 64 x 512 5.2 (6.1), 5956 x 24 x 936 7.8 (8.2); but 2048 x 64 x 1000 8.8 (6.4) where
// few clusters do, 65536 x 8 x 1000 49 (38).  Below 2048 rows the exchanged tiles are ahead by a tenth and more.
//
// Layers are often a multiple of 224 wide (3584, 7168, 14336, 28672) and batches a multiple of 256 tokens.  Tiles of 256 tokens x
// 224 weights, the roles not exchanged, then come out whole where 256 weights x any number of tokens leaves part of a wave
// empty: 512 x 14336 x 8192 91 us (101 with 512/1), 256 x 14336 x 8192 52.8 (56), half a second into a run at the power cap
// 2048 x 14336 x 8192 373 (390).  With a shallower K its result, stored by the lanes at a row stride, holds it up: 4096 x
// 14336 x 1000 146 (111 with 256/1); the line is a K of 4096.
enum class GemmKernel { EXCHANGED = 0, WIDE = 1, SINGLE = 2, ROWS224 = 3 };     // SINGLE: without pairs
struct PairTile {
    int bn, split;              // WIDE: bn = 512
    GemmKernel kernel;
    int group = 0;              // rasterisation group, 0 = by rule
};
// Calls f(tile, estimate in ns) for every tile that can take the shape.
template <typename F> void EachTile(int M, int N, int K, const int (&cap)[4], bool wide, F f)
{
    const double kBlocks = (K + hcgemm::kBlockK - 1) / hcgemm::kBlockK, tilesW = (N + hcgemm::kPairM - 1) / hcgemm::kPairM;
    const double straddle = K % hcgemm::kBlockK ? 1.5 : 1;
    const bool few = N <= 128 && (N < 64 || K % hcgemm::kBlockK);       // from 64 columns on, lines of B that do not straddle suffice
    const double hbmNs = 2.0 * ((double)M * K + (double)N * K + (double)M * N) / 6500.0;
    for (int split = 1; split <= 4; ++split) {
        const int fit = cap[split - 1];
        if (fit <= 0 || (split == 3 && M > 128) || (split > 1 && kBlocks < 4 * split)) continue;
        for (int bn = 256; bn >= 32; bn -= 32) {
            if (bn - 32 >= M) continue;                             // a narrower tile holds every token
            const double tiles = tilesW * ((M + bn - 1) / bn), x = std::min(bn, M);
            const double waves = std::ceil(tiles / fit), active = std::min(tiles, (double)fit) * split / cap[0];
            if (split > 1 && waves > 1) continue;
            const double crowd = few ? (K <= 1024 ? 4 : 2) * std::max(0.0, std::min(tiles, (double)fit) - 30) : 0;
            const double step = std::max(48 + 1.28 * bn, (16384 + 64 * x) / 120) + crowd;
            const double multiply = std::ceil(kBlocks / split) * step, empty = 1000 + 500 * std::ceil(x / 64);
            const double l2Ns = tiles * kBlocks * (32768 + 128 * x) / 13500 * (M > 256 && waves > 2 ? straddle : 1);
            const double loop = std::max(waves > 1 ? waves * std::max(multiply, std::sqrt(0.94 * multiply * multiply + empty * empty)) : multiply, l2Ns);
            f(PairTile{bn, split, GemmKernel::EXCHANGED},
              std::max(loop, hbmNs / (0.9 + 0.1 * std::min(1.0, active))) + (M <= 256 ? 0.2 * l2Ns : 0) + 3000 + 6 * x + (split > 1 ? 600 + 10 * x : 0));
        }
    }
    if (cap[0] <= 0) return;
    if (wide && M > 256) {
        const double tiles = (double)((M + hcgemm::kPairM - 1) / hcgemm::kPairM) * ((N + hcgemm::kWideN - 1) / hcgemm::kWideN);
        const double waves = std::ceil(tiles / cap[0]), l2Ns = tiles * kBlocks * 98304 / 13500 * (waves > 2 ? straddle : 1);
        f(PairTile{hcgemm::kWideN, 1, GemmKernel::WIDE}, std::max({waves * (kBlocks * 690 + 4000), l2Ns, hbmNs}) + 3000);
    }
    if (M % hcgemm::kPairM == 0 && N % 224 == 0 && N % 128 == 0 && K >= 4096) {
        const double tiles = (double)(M / hcgemm::kPairM) * (N / 224), waves = std::ceil(tiles / cap[0]);
        const double multiply = kBlocks * (48 + 1.28 * 224), l2Ns = tiles * kBlocks * (32768 + 128 * 224) / 13500;
        // ahead by three hundredths, less is chance
        f(PairTile{224, 1, GemmKernel::ROWS224},
          (std::max({waves * std::max(multiply, std::sqrt(0.94 * multiply * multiply + 3000.0 * 3000.0)), l2Ns, hbmNs}) + 3000 + 6 * 224) / 0.97);
    }
    const double rows = (M + hcgemm::kBlockM - 1) / hcgemm::kBlockM, sms = 2.0 * cap[0];
    if (N <= 128 && M >= 2048 && K <= (rows <= sms ? 1024 : 512)) {
        const double tile = std::max(kBlocks * (K % hcgemm::kBlockK ? 240 : 200), 700.0);
        f(PairTile{128, 1, GemmKernel::SINGLE}, std::max(std::ceil(rows / sms) * tile, hbmNs) + 2900);
    }
}
// HCOMM_GEMM_WIDE=0 keeps the tiles at 256 columns or fewer.
bool WideTiles()
{
    static const bool on = [] { const char *e = getenv("HCOMM_GEMM_WIDE"); return !(e && e[0] == '0'); }();
    return on;
}
PairTile PickPairTile(int M, int N, int K, const int (&cap)[4], double *estimate = nullptr)
{
    PairTile best{32, 1, GemmKernel::EXCHANGED};
    double bestNs = 0;
    EachTile(M, N, K, cap, WideTiles(), [&](const PairTile &t, double ns) {
        if (bestNs == 0 || ns < bestNs) { bestNs = ns; best = t; }
    });
    if (estimate) *estimate = bestNs;
    return best;
}

cudaLaunchConfig_t PairConfig(cudaLaunchAttribute *at, int clusters, int clusterCtas, int threads, int smemBytes, void *stream)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * clusterCtas, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smemBytes;
    cfg.stream = (cudaStream_t)stream;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = clusterCtas; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    // Calls follow one another on a stream: the next GEMM's barriers, tensor memory and descriptors are set up while this
    // one's last tiles finish.  Measured between two calls: 1.3 us at 96 x 8192 x 3584 (16.0 -> 14.7), 2.7 at 200 x 136 x 72.
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 2;
    return cfg;
}

hcgemm::SwapShape ShapeOf(int M, int N, int K, int bn, int group = 0)
{
    hcgemm::SwapShape g = {};
    g.M = M; g.N = N; g.K = K;
    g.tilesW = (N + hcgemm::kPairM - 1) / hcgemm::kPairM;
    g.tilesT = (M + bn - 1) / bn;
    g.bn = bn; g.stages = hcgemm::SwapStages(bn);
    g.group = std::min(group > 0 ? group : PairGroupRows(K), g.tilesW);     // a group that the caller forces may be any number
    return g;
}

HcclResult LaunchSwapGemm(const void *A, const void *B, void *C, int M, int N, int K, int lda, int ldb, int ldc, const PairTile &tile, void *stream)
{
    CUtensorMap tmW, tmX;
    CHK_RET(MakeTensorMap2dBf16(&tmW, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, hcgemm::kBlockM, hcgemm::kBlockK));
    CHK_RET(MakeTensorMap2dBf16(&tmX, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, (uint32_t)(tile.bn / 2), hcgemm::kBlockK));
    hcgemm::SwapShape g = ShapeOf(M, N, K, tile.bn, tile.group);
    g.C = (__nv_bfloat16 *)C; g.ldc = ldc;
    g.errFlag = GemmErrorFlag();
    const int tiles = g.tilesW * g.tilesT;
    cudaLaunchAttribute at[2];
    const cudaLaunchConfig_t cfg = PairConfig(at, tile.split > 1 ? tiles : std::min(Limits().cap[0], tiles), 2 * tile.split, hcgemm::kSwapThreads,
                                              hcgemm::SwapSmemBytes(tile.bn), stream);
    cudaError_t e;
    switch (tile.split) {
        case 4: e = cudaLaunchKernelEx(&cfg, GemmBf16SwapKernel<4>, tmW, tmX, g); break;
        case 3: e = cudaLaunchKernelEx(&cfg, GemmBf16SwapKernel<3>, tmW, tmX, g); break;
        case 2: e = cudaLaunchKernelEx(&cfg, GemmBf16SwapKernel<2>, tmW, tmX, g); break;
        default: e = cudaLaunchKernelEx(&cfg, GemmBf16SwapKernel<1>, tmW, tmX, g); break;
    }
    if (e != cudaSuccess) {
        HCCL_ERROR("GemmBf16 (tiles of %d tokens, %d CTA pairs along K) launch failed: %s", tile.bn, tile.split, cudaGetErrorString(e));
        return HCCL_E_RUNTIME;
    }
    return HCCL_SUCCESS;
}

HcclResult LaunchWideGemm(const void *A, const void *B, void *C, int M, int N, int K, int lda, int ldb, int ldc, const PairTile &tile, void *stream)
{
    CUtensorMap tmA, tmB, tmC;            // result tiles leave through TMA stores: boxes of 32 rows x 64 columns
    CHK_RET(MakeTensorMap2dBf16(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, hcgemm::kBlockM, hcgemm::kBlockK));
    CHK_RET(MakeTensorMap2dBf16(&tmB, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 128u, hcgemm::kBlockK));
    CHK_RET(MakeTensorMap2dBf16(&tmC, C, (uint64_t)M, (uint64_t)N, (uint64_t)ldc, 32, 64));
    hcgemm::GemmShape shape;
    shape.M = M; shape.N = N; shape.K = K;
    shape.tilesM = (M + hcgemm::kPairM - 1) / hcgemm::kPairM;
    shape.tilesN = (N + hcgemm::kWideN - 1) / hcgemm::kWideN;
    shape.errFlag = GemmErrorFlag();
    shape.phase = nullptr;
    // a wave of 74 such tiles loads the fewest panels at 12 rows x 6 columns
    const int rows = PairGroupRows(K), group = tile.group > 0 ? tile.group : g_forceGm.load() > 0 || rows >= 16 ? rows : 12;
    cudaLaunchAttribute at[2];
    const cudaLaunchConfig_t cfg = PairConfig(at, std::min(Limits().cap[0], shape.tilesM * shape.tilesN), 2, hcgemm::kWideThreads, hcgemm::ConfigWide<4>::kSmemBytes, stream);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, GemmBf16PairWideKernel, tmA, tmB, tmC, shape, group);
    if (e != cudaSuccess) { HCCL_ERROR("GemmBf16 (256 x 512 tiles) launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

HcclResult LaunchPair224Gemm(const void *A, const void *B, void *C, int M, int N, int K, int lda, int ldb, int ldc, const PairTile &tile, void *stream)
{
    CUtensorMap tmA, tmB;
    CHK_RET(MakeTensorMap2dBf16(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, hcgemm::kBlockM, hcgemm::kBlockK));
    CHK_RET(MakeTensorMap2dBf16(&tmB, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 224u / 2, hcgemm::kBlockK));
    hcgemm::GemmShape shape;
    shape.M = M; shape.N = N; shape.K = K;
    shape.tilesM = M / hcgemm::kPairM;
    shape.tilesN = N / 224;
    shape.errFlag = GemmErrorFlag();
    shape.phase = nullptr;
    const hcgemm::StoreBf16 epi{(__nv_bfloat16 *)C, ldc, M, N};
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t cfg = PairConfig(at, std::min(Limits().cap[0], shape.tilesM * shape.tilesN), 2, hcgemm::kThreads, hcgemm::Config2<224, 7>::kSmemBytes, stream);
    cfg.numAttrs = 1;           // the loop is the fused kernels', which do not wait for a kernel in front: an ordinary launch
    const cudaError_t e = cudaLaunchKernelEx(&cfg, GemmBf16Pair224Kernel, tmA, tmB, shape, epi, tile.group > 0 ? tile.group : PairGroupRows(K));
    if (e != cudaSuccess) { HCCL_ERROR("GemmBf16 (256 x 224 tiles) launch failed: %s", cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}

// One launch of a tile's kernel on CTA pairs (all but SINGLE).
HcclResult LaunchTile(const void *A, const void *B, void *C, int M, int N, int K, int lda, int ldb, int ldc, const PairTile &tile, void *stream)
{
    if (tile.kernel == GemmKernel::WIDE) return LaunchWideGemm(A, B, C, M, N, K, lda, ldb, ldc, tile, stream);
    if (tile.kernel == GemmKernel::ROWS224) return LaunchPair224Gemm(A, B, C, M, N, K, lda, ldb, ldc, tile, stream);
    return LaunchSwapGemm(A, B, C, M, N, K, lda, ldb, ldc, tile, stream);
}

// HCOMM_GEMM_AUTOTUNE=1: a large shape (2 M N K of 2e11 and more) seen for the first time is timed once with the tiles whose
// estimates come within 15 % of the best, each with the rasterisation group halved, kept and doubled, on the caller's stream,
// and the fastest is kept for the process.  Never while the stream is being captured, nor with a forced width, group or split.
// Off by default: at the power cap the variants differ mostly through the clock that they leave the chip at, and timings of a
// few launches each did not rank them the same from run to run.
struct ShapeKey {
    int M, N, K;
    bool operator<(const ShapeKey &o) const { return M != o.M ? M < o.M : (N != o.N ? N < o.N : K < o.K); }
};
std::mutex g_tuneMu;
std::map<ShapeKey, PairTile> g_tuned;

PairTile MeasuredTile(const void *A, const void *B, void *C, int M, int N, int K, int lda, int ldb, int ldc, const int (&cap)[4], const PairTile &rule, double estimate,
                      void *stream)
{
    const ShapeKey key{M, N, K};
    {
        std::lock_guard<std::mutex> lk(g_tuneMu);
        auto it = g_tuned.find(key);
        if (it != g_tuned.end()) return it->second;
    }
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing((cudaStream_t)stream, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone) { cudaGetLastError(); return rule; }
    std::vector<PairTile> cands;
    EachTile(M, N, K, cap, WideTiles(), [&](PairTile t, double ns) {
        if (ns > 1.15 * estimate || t.kernel == GemmKernel::SINGLE) return;
        const int group = PairGroupRows(K);
        for (int g : {group / 2, group, group * 2})
            if (g >= 2 && g <= 32) { t.group = g; cands.push_back(t); }
    });
    if (cands.size() < 2) return rule;
    // Five rounds over all candidates, two back-to-back launches each; the first round only warms up (module load, L2,
    // clocks).  Odd rounds walk the list backwards so that a drift over a round does not favour one end of it, and a
    // candidate's figure is the median of its four counted rounds, not its luckiest one.
    cudaEvent_t ev[2];
    if (cudaEventCreate(&ev[0]) != cudaSuccess) { cudaGetLastError(); return rule; }
    if (cudaEventCreate(&ev[1]) != cudaSuccess) { cudaGetLastError(); cudaEventDestroy(ev[0]); return rule; }
    const int count = (int)cands.size();
    std::vector<std::vector<float>> samples(count);
    bool ok = true;
    for (int round = 0; round < 5 && ok; ++round) {
        for (int i = 0; i < count && ok; ++i) {
            const int c = (round & 1) ? count - 1 - i : i;
            cudaEventRecord(ev[0], (cudaStream_t)stream);
            for (int r = 0; r < 2 && ok; ++r) ok = LaunchTile(A, B, C, M, N, K, lda, ldb, ldc, cands[c], stream) == HCCL_SUCCESS;
            cudaEventRecord(ev[1], (cudaStream_t)stream);
            float ms = 0;
            if (!ok || cudaEventSynchronize(ev[1]) != cudaSuccess || cudaEventElapsedTime(&ms, ev[0], ev[1]) != cudaSuccess) { cudaGetLastError(); ok = false; break; }
            if (round > 0) samples[c].push_back(ms * 0.5f);
        }
    }
    cudaEventDestroy(ev[0]);
    cudaEventDestroy(ev[1]);
    if (!ok) return rule;
    int win = 0;
    std::vector<float> median(count);
    for (int i = 0; i < count; ++i) {
        std::sort(samples[i].begin(), samples[i].end());
        median[i] = 0.5f * (samples[i][1] + samples[i][2]);
        if (median[i] < median[win]) win = i;
    }
    HCCL_INFO("GEMM %d x %d x %d: tile width %d, %d pairs along K, group %d chosen by measurement (%.3f ms; the estimate said %d / %d)", M, N, K, cands[win].bn,
              cands[win].split, cands[win].group, median[win], rule.bn, rule.split);
    std::lock_guard<std::mutex> lk(g_tuneMu);
    return g_tuned.emplace(key, cands[win]).first->second;
}

PairTile ChoosePairTile(const void *A, const void *B, void *C, int M, int N, int K, int lda, int ldb, int ldc, const int (&cap)[4], void *stream)
{
    static const bool measure = [] { const char *e = getenv("HCOMM_GEMM_AUTOTUNE"); return e && e[0] == '1'; }();
    double estimate = 0;
    PairTile t = PickPairTile(M, N, K, cap, &estimate);
    const int bn = ForcedPairTileWidth(), split = g_forceSplit.load(), kBlocks = (K + hcgemm::kBlockK - 1) / hcgemm::kBlockK;
    if (measure && bn <= 0 && split <= 0 && 2.0 * M * N * K >= 2e11) {
        PairGroupRows(K);               // the first call reads HCOMM_GEMM_GM
        if (g_forceGm.load() <= 0) return MeasuredTile(A, B, C, M, N, K, lda, ldb, ldc, cap, t, estimate, stream);
    }
    if (bn >= hcgemm::kWideN) t = {hcgemm::kWideN, 1, GemmKernel::WIDE};
    else if (bn > 0) t = {std::min(256, std::max(32, bn / 32 * 32)), t.split, GemmKernel::EXCHANGED};
    else if (split > 0 && t.kernel != GemmKernel::WIDE) t.kernel = GemmKernel::EXCHANGED;
    if (t.bn <= 256 && split >= 1 && split <= 4 && split <= kBlocks && cap[split - 1] > 0) t.split = split;
    return t;
}

}  // namespace

HcclResult GemmBf16(const void *A, const void *B, void *C, int M, int N, int K, int lda, int ldb, int ldc, void *stream)
{
    if (M <= 0 || N <= 0 || K <= 0) return HCCL_SUCCESS;
    if (N % 8 != 0 || K % 8 != 0 || ((uintptr_t)C & 15) != 0 || (ldc % 8) != 0) {
        HCCL_ERROR("GemmBf16: N, K and ldc must be multiples of 8 and C 16-byte aligned (N=%d K=%d ldc=%d)", N, K, ldc);
        return HCCL_E_PARA;
    }
    static const bool pairEnabled = [] { const char *e = getenv("HCOMM_GEMM_PAIR"); return !(e && e[0] == '0'); }();
    const GemmLimits limits = Limits();
    if (pairEnabled && limits.cap[0] > 0) {
        const PairTile tile = ChoosePairTile(A, B, C, M, N, K, lda, ldb, ldc, limits.cap, stream);
        if (tile.kernel != GemmKernel::SINGLE) return LaunchTile(A, B, C, M, N, K, lda, ldb, ldc, tile, stream);
    }
    // one CTA per 128-row tile: few columns, HCOMM_GEMM_PAIR=0, or a device that cannot hold a cluster
    const int BN = (N % 256 == 0 || N >= 2048) ? 256 : 128;
    CUtensorMap tmA, tmB;
    CHK_RET(MakeTensorMap2dBf16(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, hcgemm::kBlockM, hcgemm::kBlockK));
    CHK_RET(MakeTensorMap2dBf16(&tmB, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, (uint32_t)BN, hcgemm::kBlockK));
    hcgemm::GemmShape shape;
    shape.M = M; shape.N = N; shape.K = K;
    shape.tilesM = (M + hcgemm::kBlockM - 1) / hcgemm::kBlockM;
    shape.tilesN = (N + BN - 1) / BN;
    shape.errFlag = GemmErrorFlag();
    shape.phase = nullptr;
    hcgemm::StoreBf16 epi{(__nv_bfloat16 *)C, ldc, M, N};
    int grid = std::min(GemmSmCount(), shape.tilesM * shape.tilesN);
    cudaError_t e;
    if (BN == 256) {
        GemmBf16Kernel<256><<<grid, hcgemm::kThreads, hcgemm::Config<256>::kSmemBytes, (cudaStream_t)stream>>>(tmA, tmB, shape, epi);
    } else {
        GemmBf16Kernel<128><<<grid, hcgemm::kThreads, hcgemm::Config<128>::kSmemBytes, (cudaStream_t)stream>>>(tmA, tmB, shape, epi);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        HCCL_ERROR("GemmBf16 launch failed: %s", cudaGetErrorString(e));
        return HCCL_E_RUNTIME;
    }
    return HCCL_SUCCESS;
}

}  // namespace hc

// C entry points (used from Python through ctypes).
extern "C" int HcommGemmBf16(const void *A, const void *B, void *C, int M, int N, int K, int lda, int ldb, int ldc, void *stream)
{
    return (int)hc::GemmBf16(A, B, C, M, N, K, lda, ldb, ldc, stream);
}
// Reads and clears the "a bounded wait expired inside a GEMM kernel" flag of the current device.
// Overrides the rasterisation group (row blocks of 256 rows) and the tile width of the CTA-pair GEMM kernels; 0 = automatic.
extern "C" void HcommGemmSetTuning(int groupRows, int tileWidth)
{
    hc::g_forceGm.store(groupRows > 0 ? groupRows : 0);
    hc::g_forceBn.store(tileWidth > 0 ? tileWidth : 0);
}
// CTA pairs (1 to 4) that share a tile along K; 0 = automatic.
extern "C" void HcommGemmSetSplit(int pairsAlongK)
{
    hc::g_forceSplit.store(pairsAlongK);
}
// The rule behind the automatic choice, for a device that holds cap1, cap2 and cap4 clusters of 1, 2 and 4 CTA pairs at once and none of 3.
extern "C" void HcommToolGemmTile(int M, int N, int K, int cap1, int cap2, int cap4, int *tileWidth, int *pairsAlongK)
{
    const int cap[4] = {cap1, cap2, 0, cap4};
    const hc::PairTile t = hc::PickPairTile(M, N, K, cap);
    if (tileWidth) *tileWidth = t.bn;
    if (pairsAlongK) *pairsAlongK = t.split;
}
// The same for a device that holds caps[0] .. caps[3] clusters of 1 .. 4 pairs.  Returns which kernel, numbered as below.
extern "C" int HcommToolGemmTileOf(int M, int N, int K, const int *caps, int *tileWidth, int *pairsAlongK)
{
    const int cap[4] = {caps[0], caps[1], caps[2], caps[3]};
    const hc::PairTile t = hc::PickPairTile(M, N, K, cap);
    if (tileWidth) *tileWidth = t.bn;
    if (pairsAlongK) *pairsAlongK = t.split;
    return (int)t.kernel;
}
// What is made of a device's answers, the clusters of 1 to 4 pairs that it holds at once, negative ones failures; whether they are kept.
extern "C" int HcommToolGemmClusterCaps(const int *answers, int *caps)
{
    return hc::ClusterCaps(caps, [&](int pairs, int *n) { *n = std::max(0, answers[pairs - 1]); return answers[pairs - 1] >= 0; });
}
// What the current device holds.
extern "C" void HcommToolGemmCaps(int *caps)
{
    const hc::GemmLimits l = hc::Limits();
    for (int i = 0; i < 4; ++i) caps[i] = l.cap[i];
}
// Which kernel that rule takes: 0 exchanged operands, 1 tiles of 256 x 512, 2 without pairs, 3 tiles of 256 tokens x 224 weights.
extern "C" int HcommToolGemmKernel(int M, int N, int K, int cap1, int cap2, int cap4)
{
    const int cap[4] = {cap1, cap2, 0, cap4};
    return (int)hc::PickPairTile(M, N, K, cap).kernel;
}
// The blocks (256 weights, tileWidth tokens) of tile t of the GEMM with exchanged operands; returns the number of tiles.
extern "C" int HcommToolGemmOrder(int M, int N, int K, int tileWidth, int t, int *weightBlock, int *tokenBlock)
{
    const hcgemm::SwapShape g = hc::ShapeOf(M, N, K, tileWidth);
    if (t >= 0 && t < g.tilesW * g.tilesT) hcgemm::SwapOrder(g, t, weightBlock, tokenBlock);
    return g.tilesW * g.tilesT;
}
// Tile width and rasterisation group that the measurement at first use chose for a shape (0 / 0: none was made).
extern "C" void HcommGemmGetTuned(int M, int N, int K, int *tileWidth, int *groupRows)
{
    std::lock_guard<std::mutex> lk(hc::g_tuneMu);
    auto it = hc::g_tuned.find(hc::ShapeKey{M, N, K});
    if (tileWidth) *tileWidth = it == hc::g_tuned.end() ? 0 : it->second.bn;
    if (groupRows) *groupRows = it == hc::g_tuned.end() ? 0 : it->second.group;
}
extern "C" int HcommGemmTakeError(void)
{
    uint32_t v = 0, zero = 0;
    uint32_t *f = hc::GemmErrorFlag();
    if (cudaMemcpy(&v, f, sizeof(v), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    if (v) cudaMemcpy(f, &zero, sizeof(zero), cudaMemcpyHostToDevice);
    return (int)v;
}
