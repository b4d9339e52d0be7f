// RL weight reshard: training layout (one flat bf16 parameter vector, evenly sharded over R ranks — the FSDP layout) →
// inference layout of one rank (its tensor-parallel sub-block of every parameter), optionally cast to e4m3 with 128x128
// block scales, as ONE gather kernel that pulls exactly the bytes this rank needs from the owners' shards over NVLink.
// The reference names parameter resharding for reinforcement learning only as a use case of its global address space
// (README.md:53 of the reference); the all-gather-then-slice it replaces moves R x more data.
//
// Bound by memory traffic, so: loads run a tile ahead of the arithmetic (cp.async into shared memory, every thread its own
// slots), one barrier round per tile for the block maxima, and what is not cast goes through the bulk copy engine. Two tiles of
// 64 KiB in flight per SM are better than three (1620 against 1689 us; the DRAM turns between reading and writing less
// often), L2 eviction hints were worse. 8 layers + embedding + head to e4m3, 9.4 GB of traffic: 2150 us with loads, arithmetic and
// stores in turn -> 1591 us (5.9 TB/s).
//
// The host describes the destination as a table of parameter sub-blocks (origin + shape inside the full parameter, where
// the parameter sits in the flat vector, where the sub-block goes). The kernel enumerates 128x256 tiles over the table
// (binary search of a prefix of tile counts), and for each tile: computes, per 16-byte vector or run, which rank's shard holds it
// (shards are multiples of 8 elements, so a vector never straddles two ranks), loads it from that rank's heap, and either
// stores it (bf16) or reduces the tile's absolute maximum, scales and converts to e4m3 (one fp32 scale per tile).
// A barrier over all ranks opens the kernel (every shard is final) and closes it (nobody reuses its shard while it is read).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <atomic>

#include "mf/device/mf_shm_device.cuh"
#include "mf_kernels.h"

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kTile = 128;           // quantisation block edge and tile height
constexpr int kTileCols = 256;       // tile width: a warp reads 512 contiguous bytes of a row (two quantisation blocks)
constexpr int kVecPerThread = (kTile * kTileCols / 8) / kThreads;  // 8
constexpr uint32_t kTileElems = kTile * kTileCols;
constexpr int kStages = 2;           // tiles of 64 KiB in shared memory
constexpr int kSmemBytes = kStages * kTileElems * 2;
constexpr uint32_t kLinearMinCols = 1024;  // narrowest row segment that is worth a bulk copy of its own (2 KiB)

// What has to be known of a tile when its data has arrived.
struct TileInfo {
    uint64_t dst;         // byte offset of this thread's first vector in the destination
    uint64_t scale;       // index of the scale of this thread's quantisation block
    uint32_t rowBytes;    // bytes from one destination row to the next
    uint32_t rows;        // rows of the tile that exist, 0 where this thread's columns do not
    uint32_t quant;
    uint32_t linear;      // bytes of a tile that is moved as it is, dst being the tile's offset; 0: rows and columns
};

// Walks the tiles of a table in ascending order; the descriptor is looked up again only where a tile leaves it.
struct TileCursor {
    uint32_t begin{1}, end{0};  // tiles of the current descriptor
    uint32_t index{0};
    __device__ __forceinline__ const mf_reshard_desc_t &Find(const mf_reshard_args_t &a, uint32_t tile)
    {
        if (tile < begin || tile >= end) {
            uint32_t lo = 0, hi = a.ndesc;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (a.descs[mid].tileStart <= tile) {
                    lo = mid;
                } else {
                    hi = mid;
                }
            }
            index = lo;
            begin = a.descs[lo].tileStart;
            end = lo + 1 < a.ndesc ? a.descs[lo + 1].tileStart : a.totalTiles;
        }
        return a.descs[index];
    }
};

__device__ __forceinline__ void CopyAsync16(uint32_t smem, const void *src, bool valid)
{
    // Nothing is read and zeros are stored where the element does not exist.
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

__device__ __forceinline__ uint32_t SmemAddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void MbarInit(uint64_t *bar) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(SmemAddr(bar))); }

__device__ __forceinline__ void MbarExpect(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(SmemAddr(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool MbarWait(uint64_t *bar, uint32_t parity)
{
    for (uint32_t i = 0; i < (1u << 24); i++) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(SmemAddr(bar)), "r"(parity)
            : "memory");
        if (ok) {
            return true;
        }
    }
    return false;
}

__device__ __forceinline__ void BulkLoad(uint32_t smem, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem), "l"(src), "r"(bytes),
                 "r"(SmemAddr(bar))
                 : "memory");
}

// Stores and waits until the shared memory may be overwritten.
__device__ __forceinline__ void BulkStore(void *dst, uint32_t smem, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.commit_group;\ncp.async.bulk.wait_group.read 0;" ::: "memory");
}

// Largest magnitudes so far and of eight further bf16, exact (a NaN is passed over, as fmaxf does).
__device__ __forceinline__ __nv_bfloat162 MaxMagnitude2(const uint4 &v, __nv_bfloat162 m)
{
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        m = __hmax2(m, __habs2(h[q]));
    }
    return m;
}

__global__ void __launch_bounds__(kThreads, 1)
mf_reshard_kernel(const mf_reshard_args_t *__restrict__ args, uint32_t channel, uint64_t epoch, uint64_t timeoutNs)
{
    cg::grid_group grid = cg::this_grid();
    const mf_reshard_args_t a = args[blockIdx.y];
    const MfDeviceMeta *m = reinterpret_cast<const MfDeviceMeta *>(a.meta);
    extern __shared__ uint4 stageMem[];
    __shared__ uint64_t landed[kStages];
    __shared__ __nv_bfloat162 warpMax[2][2][kWarps];  // per parity of the tile, quantisation block and warp
    __shared__ int abortFlag;
    if (mf_check_bounds_enabled(m) && !mf_shm_in_own_window(m, a.srcShard, a.shardElems * 2)) {
        if (threadIdx.x == 0 && a.status != nullptr) {
            atomicCAS(a.status, 0, MF_DEV_ERR_BOUNDS);
        }
        return;
    }

    if (blockIdx.x == 0) {
        int rc = mf_barrier_cta(m, channel, 0, 2 * epoch - 1, timeoutNs);
        if (rc != MF_DEV_OK && threadIdx.x == 0 && a.status != nullptr) {
            atomicCAS(a.status, 0, rc);
        }
    }
    grid.sync();
    if (threadIdx.x == 0) {
        abortFlag = a.status != nullptr ? *(volatile int *)a.status : 0;
    }
    __syncthreads();
    const bool dead = abortFlag != 0;

    // rank 0's copy of the shard buffer: rank r's is r * symmetricSize further
    const char *shard0 = reinterpret_cast<const char *>(a.srcShard) - (uint64_t)m->rankId * m->symmetricSize;
    if (!dead) {
        // Several ranks: every CTA walks a contiguous run of tiles (same rows, neighbouring columns, then the next rows), so its
        // reads stay inside a few pages of one owner at a time instead of hopping across all peers' shards. One rank: the CTAs
        // stand next to each other, which keeps more of a DRAM page's accesses together (5.2 GB of blocks cast to e4m3 and 4.2 GB
        // moved as they are: 1640 -> 1591 us).
        const bool strided = m->rankCount == 1;
        const uint32_t tileBegin = strided ? blockIdx.x : (uint32_t)((uint64_t)blockIdx.x * a.totalTiles / gridDim.x);
        const uint32_t tileEnd = strided ? a.totalTiles : (uint32_t)((uint64_t)(blockIdx.x + 1) * a.totalTiles / gridDim.x);
        const uint32_t tileStep = strided ? gridDim.x : 1;
        const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = lane >> 4;
        const uint32_t smem = (uint32_t)__cvta_generic_to_shared(stageMem);
        TileCursor cursor;
        if (threadIdx.x == 0) {
            for (int i = 0; i < kStages; i++) {
                MbarInit(&landed[i]);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        asm volatile("fence.proxy.async;" ::: "memory");  // what peers stored before the barrier is read by the bulk copy engine below
        __syncthreads();
        uint32_t parity = 0;  // bit i: parity of the next bulk load into stage i

        // Asks for tile `tile`. A warp reads one row segment of 512 bytes per vector: lane l owns columns colBase + 8l .. +7 of rows
        // rowBase + warp, + 16, + 32, ... (16 warps, 8 vectors). A thread later takes only what it asked for itself. Parameters that
        // are not quantised are moved in destination order instead, 64 KiB a tile, by bulk copies in and out.
        auto request = [&](uint32_t tile, uint32_t turn) {
            TileInfo t{};
            if (tile < tileEnd) {
                const mf_reshard_desc_t &d = cursor.Find(a, tile);
                const uint32_t nrows = d.nrows, ncols = d.ncols, colsFull = d.colsFull;
                const uint32_t local = tile - d.tileStart, stage = smem + turn % kStages * (kTileElems * 2);
                if (!d.quant && (ncols == colsFull || ncols >= kLinearMinCols)) {
                    const uint64_t total = (uint64_t)nrows * ncols, first = (uint64_t)local * kTileElems;
                    t.linear = first < total ? (uint32_t)min((uint64_t)kTileElems, total - first) * 2 : 0;
                    t.dst = d.dstOff + first * 2;
                    t.quant = 2;
                    if (threadIdx.x < 32 && t.linear != 0) {
                        if (lane == 0) {
                            MbarExpect(&landed[turn % kStages], t.linear);
                        }
                        __syncwarp();
                        // One lane per source run: the rest of the first row, then whole rows; a single run where the rows follow
                        // one another in the source too.
                        const uint32_t elems = t.linear / 2, width = ncols == colsFull ? kTileElems : ncols;
                        const uint64_t row0 = first / ncols;
                        const uint32_t col0 = (uint32_t)(first - row0 * ncols), lead = ncols == colsFull ? kTileElems : ncols - col0;
                        for (uint32_t s = lane;; s += 32) {
                            const uint32_t at = s == 0 ? 0 : lead + (s - 1) * width;
                            if (at >= elems) {
                                break;
                            }
                            uint32_t len = min(elems - at, s == 0 ? lead : width), to = stage + at * 2;
                            uint64_t flat = d.srcFlatOff + (d.r0 + row0 + s) * colsFull + d.c0 + (s == 0 ? col0 : 0);
                            while (len > 0) {  // cut where a shard ends
                                const uint64_t owner = flat < a.shardElems ? 0 : flat / a.shardElems, within = flat - owner * a.shardElems;
                                const uint32_t run = (uint32_t)min((uint64_t)len, a.shardElems - within);
                                BulkLoad(to, shard0 + owner * m->symmetricSize + within * 2, run * 2, &landed[turn % kStages]);
                                flat += run;
                                to += run * 2;
                                len -= run;
                            }
                        }
                    }
                } else {
                    const uint32_t tilesPerRow = (ncols + kTileCols - 1) / kTileCols;
                    const uint32_t tr = local / tilesPerRow, tc = local % tilesPerRow;
                    const uint32_t rowBase = tr * kTile, colBase = tc * kTileCols;
                    const uint32_t c = colBase + lane * 8;
                    t.quant = d.quant;
                    t.rows = c < ncols ? min(nrows - rowBase, (uint32_t)kTile) : 0;
                    const uint32_t elem = d.quant ? 1 : 2;
                    t.rowBytes = ncols * elem;
                    t.dst = d.dstOff + ((uint64_t)(rowBase + warp) * ncols + c) * elem;
                    t.scale = d.scaleOff + (uint64_t)tr * (ncols / kTile) + tc * 2 + half;
                    // Which shard holds the tile's first element: ONE 64-bit division per tile, none where it is the first shard. A
                    // tile spans far fewer elements than a shard, so every other element of it lives in that shard or in the next;
                    // the loop below walks on in the rare case of tiny shards.
                    const uint64_t tileFlat = d.srcFlatOff + (uint64_t)(d.r0 + rowBase) * colsFull + d.c0 + colBase;
                    const uint64_t owner0 = tileFlat < a.shardElems ? 0 : tileFlat / a.shardElems;
                    const uint64_t rel0 = tileFlat - owner0 * a.shardElems + (uint64_t)warp * colsFull + lane * 8;
                    const uint64_t relStep = (uint64_t)kWarps * colsFull;
                    const char *ownerBase = shard0 + owner0 * m->symmetricSize;
#pragma unroll
                    for (int i = 0; i < kVecPerThread; i++) {
                        const bool valid = warp + i * kWarps < t.rows;
                        uint64_t within = valid ? rel0 + (uint64_t)i * relStep : 0;
                        const char *base = ownerBase;
                        while (within >= a.shardElems) {
                            within -= a.shardElems;
                            base += m->symmetricSize;
                        }
                        CopyAsync16(stage + (i * kThreads + threadIdx.x) * 16, base + within * 2, valid);
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            return t;
        };

        TileInfo now = request(tileBegin, 0);
        for (uint32_t tile = tileBegin, turn = 0; tile < tileEnd; tile += tileStep, turn++) {
            // Everybody has taken the previous tile out of the stage that is filled next.
            __syncthreads();
            const TileInfo next = request(tile + tileStep, turn + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            if (now.quant == 2) {
                if (threadIdx.x == 0 && now.linear != 0) {
                    const uint32_t st = turn % kStages;
                    if (!MbarWait(&landed[st], (parity >> st) & 1)) {
                        if (a.status != nullptr) {
                            atomicCAS(a.status, 0, MF_DEV_ERR_TIMEOUT);
                        }
                    } else {
                        BulkStore(reinterpret_cast<unsigned char *>(a.dst) + now.dst, smem + st * (kTileElems * 2), now.linear);
                    }
                    parity ^= 1u << st;
                }
                now = next;
                continue;
            }
            uint4 v[kVecPerThread];
            const uint4 *slot = stageMem + turn % kStages * (kTileElems / 8) + threadIdx.x;
#pragma unroll
            for (int i = 0; i < kVecPerThread; i++) {
                v[i] = slot[i * kThreads];
            }
            unsigned char *dst = reinterpret_cast<unsigned char *>(a.dst) + now.dst;
            const size_t step = (size_t)kWarps * now.rowBytes;
            if (now.quant) {
                __nv_bfloat162 m2 = __float2bfloat162_rn(0.f);
#pragma unroll
                for (int i = 0; i < kVecPerThread; i++) {
                    m2 = MaxMagnitude2(v[i], m2);
                }
                // Lanes 0-15 of every warp hold columns of the tile's left quantisation block, lanes 16-31 of the right one.
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) {
                    m2 = __hmax2(m2, __shfl_xor_sync(0xffffffffu, m2, o));
                }
                __nv_bfloat162 *maxima = warpMax[turn & 1][half];
                if ((lane & 15) == 0) {
                    maxima[warp] = m2;
                }
                __syncthreads();  // one per tile: the other parity's maxima are rewritten before everybody is past this one again
                m2 = maxima[lane & 15];
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) {
                    m2 = __hmax2(m2, __shfl_xor_sync(0xffffffffu, m2, o));
                }
                const float2 ends = __bfloat1622float2(m2);
                const float tmax = fmaxf(ends.x, ends.y);
                const float sc = fmaxf(tmax, 1e-10f) * (1.f / 448.f);
                const float inv = 1.f / sc;
#pragma unroll
                for (int i = 0; i < kVecPerThread; i++) {
                    if (warp + i * kWarps < now.rows) {
                        const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v[i]);
                        uint2 pk;
                        unsigned short *ps = reinterpret_cast<unsigned short *>(&pk);
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            float2 f = __bfloat1622float2(h[q]);
                            ps[q] = __nv_cvt_float2_to_fp8x2(make_float2(f.x * inv, f.y * inv), __NV_SATFINITE, __NV_E4M3);
                        }
                        *reinterpret_cast<uint2 *>(dst + i * step) = pk;
                    }
                }
                if ((lane & 15) == 0 && warp == 0 && now.rows != 0) {
                    a.dstScale[now.scale] = sc;
                }
            } else {
#pragma unroll
                for (int i = 0; i < kVecPerThread; i++) {
                    if (warp + i * kWarps < now.rows) {
                        mf_st16(dst + i * step, v[i]);
                    }
                }
            }
            now = next;
        }
        if (threadIdx.x == 0) {
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // every bulk store has landed
        }
    }
    grid.sync();
    if (blockIdx.x == 0 && !dead) {
        int rc = mf_barrier_cta(m, channel, 0, 2 * epoch, timeoutNs);
        if (rc != MF_DEV_OK && threadIdx.x == 0 && a.status != nullptr) {
            atomicCAS(a.status, 0, rc);
        }
    }
}

}  // namespace

extern "C" int mf_k_reshard(const mf_reshard_args_t *argsDev, int nEmulatedRanks, int rankCount, uint32_t channel, uint64_t epoch, uint64_t timeoutNs,
                            int ctas, mf_stream_t stream)
{
    if (argsDev == nullptr || nEmulatedRanks < 1 || rankCount < 1 || rankCount > (int)MF_SIGNAL_MAX_RANKS || channel >= MF_SIGNAL_CHANNELS || epoch == 0) {
        return MF_K_INVALID;
    }
    if (timeoutNs == 0) {
        timeoutNs = 2000000000ull;
    }
    // How many CTAs fit the GPU is asked once per device.
    static std::atomic<int> resident[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        (void)cudaGetLastError();
        return MF_K_LAUNCH_FAILED;
    }
    int fit = resident[dev].load(std::memory_order_relaxed);
    if (fit == 0) {
        int perSm = 0, sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaFuncSetAttribute(mf_reshard_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, mf_reshard_kernel, kThreads, kSmemBytes) != cudaSuccess || perSm * sms <= 0) {
            (void)cudaGetLastError();
            return MF_K_LAUNCH_FAILED;
        }
        fit = perSm * sms;
        resident[dev].store(fit, std::memory_order_relaxed);
    }
    int grid = fit / nEmulatedRanks;
    if (ctas > 0 && ctas < grid) {
        grid = ctas;
    }
    if (grid < 1) {
        return MF_K_TOO_LARGE;
    }
    void *kargs[] = {(void *)&argsDev, (void *)&channel, (void *)&epoch, (void *)&timeoutNs};
    dim3 g((unsigned)grid, (unsigned)nEmulatedRanks, 1), b(kThreads, 1, 1);
    cudaError_t e = cudaLaunchCooperativeKernel((const void *)mf_reshard_kernel, g, b, kargs, kSmemBytes, (cudaStream_t)stream);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return MF_K_LAUNCH_FAILED;
    }
    return MF_K_OK;
}
