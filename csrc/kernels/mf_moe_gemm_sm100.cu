// Grouped FP8 GEMM for the MoE expert FFN on Blackwell tensor cores (tcgen05 + TMEM + TMA), block-scaled:
//     out[g-rows, :] = (A[g-rows, :] * sa) x (B[g] * sb)^T
// A: received tokens, fp8 e4m3 with one fp32 scale per (row, 128 K-elements); B[g]: expert weights [N, K] fp8 e4m3 with one
// fp32 scale per 128x128 block. The reference library has no GEMM (MoE is only named as a use case, README.md:53 of the
// reference); the contract here is the DeepSeek-V3 block-scaled FFN of the workload definition.
//
// Mapping to the hardware, per CTA (one persistent CTA per SM; tiles of 128 x BN, BN = 256 or 128):
//   warp 0     TMA producer: cp.async.bulk.tensor 2-D loads of a 128x128-byte A tile and a BNx128-byte B tile per K-block
//              into a shared-memory ring (128-byte swizzle), completion on mbarriers. Loads are per-CTA, no multicast.
//   warp 1     one elected thread issues tcgen05.mma.kind::f8f6f4 (M128, N = BN, K32, four per K-block) into one of 512 / BN
//              TMEM accumulators (all 512 columns) and tcgen05.commit's to "stage free" and "partial ready" mbarriers.
//   warps 4..  read each K-block's partial product from TMEM (tcgen05.ld 32x32b, 64 columns per thread: every four warps one
//              64-column part of the tile), multiply by sa[row, kb] * sb[tile, kb] and add into fp32 registers (two columns per
//              packed FMA) while the MMAs fill the other accumulators. After the last K-block they apply the epilogue (plain,
//              or SwiGLU on interleaved gate/up columns) and store bf16.
//   warps 2-3  bring the products sa * sb of four K-blocks at a time into a ring of two such groups, one group ahead and across
//              tiles: a row's scales are a line of their own for every thread, and waiting for them once per K-block on the
//              promotion path took longer than the MMAs. It also leaves the promotion threads few enough registers.
// 8191 rows over 32 experts, SwiGLU GEMM N 4096 / K 7168: 486 -> 353 us; N 7168 / K 2048: 281 -> 196 us. What bounds it now is the
// promotion: a K-block takes about 950 cycles of the wide tile and 720 of the narrow one, whose four accumulators leave the hand-over
// out of the way, against 512 and 256 of its MMAs. Each warp reads its 64 columns by four loads that it waits for one by one.
// Tiles are enumerated on the device from group_offset/group_count (the host does not know the routing result), n fastest so
// that concurrently running CTAs share an A tile and stream one expert's weights through L2.
// Every mbarrier wait is bounded; on expiry the CTA sets *status, all roles drain and the CTA frees its TMEM and exits.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <cstdlib>

#include "mf_kernels.h"
#include "mf_launch.cuh"
#include "mf_sm100_ptx.cuh"

using namespace mf::sm100;
using mf::AllowSmem;

namespace {

constexpr int BM = 128, BK = 128;
constexpr int HC = 64;               // columns per promotion thread
constexpr int kTileBytes = BM * BK;  // fp8: 16 KiB of A per K-block
constexpr int kMaxGroups = 256;
constexpr uint32_t kTmemCols = 512;

template <int BN>
struct Cfg {
    static constexpr int kStages = BN == 256 ? 4 : 6;
    static constexpr int kAccBufs = (int)kTmemCols / BN;  // TMEM accumulator buffers
    static constexpr int kEpiWarps = 4 * (BN / HC);       // warps 4 and up
    static constexpr int kThreads = 128 + 32 * kEpiWarps;
    static constexpr int kBTile = BN * BK;
};

template <int BN>
struct SharedStorage {
    alignas(1024) unsigned char a[Cfg<BN>::kStages][kTileBytes];
    alignas(1024) unsigned char b[Cfg<BN>::kStages][Cfg<BN>::kBTile];
    // Read per K-block, not four at a time: with those in registers the promotion threads spilled (12 bytes, 389 instead of 353 us).
    float scale[2][BN / 128][4][BM];  // [group of four K-blocks][weight block][K-block][row]
    uint64_t scaleFull[2];
    uint64_t scaleEmpty[2];
    uint64_t full[Cfg<BN>::kStages];
    uint64_t empty[Cfg<BN>::kStages];
    uint64_t tmemFull[Cfg<BN>::kAccBufs];
    uint64_t tmemEmpty[Cfg<BN>::kAccBufs];
    uint32_t tmemBase;
    int abortFlag;
    int tilePrefix[kMaxGroups + 1];
    int groupOffset[kMaxGroups];  // of the caller's tables: looked up for every tile by every role
    int groupCount[kMaxGroups];
};

struct GemmParams {
    const float *aScale;
    const float *bScale;
    __nv_bfloat16 *out;
    const int *groupOffset;
    const int *groupCount;
    int *status;
    int G, N, K, mode, outStride, rowsTotal;
    int wideStores;  // out is 32-byte aligned: the epilogue stores whole sectors
    int vecScales;   // the scales of four K-blocks of a row are one aligned 16-byte word
};

__device__ __forceinline__ uint32_t PackBf16(float lo, float hi)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}
// Sixteen bf16 of one row: one whole sector where the address allows it (the lanes of a warp store to 32 different rows).
__device__ __forceinline__ void Store16(__nv_bfloat16 *o, const uint32_t (&pk)[8], bool wide)
{
    if (wide) {
        StGlobal32B(o, pk);
    } else {
        reinterpret_cast<uint4 *>(o)[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        reinterpret_cast<uint4 *>(o)[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
    }
}

__device__ __forceinline__ uint64_t PackF32x2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void UnpackF32x2(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
// acc = a * b + acc on two floats at once, each as fmaf does it.
__device__ __forceinline__ void FmaF32x2(uint64_t &acc, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }

__device__ __forceinline__ float Silu(float x) { return x / (1.f + __expf(-x)); }

template <int BN>
__global__ void __launch_bounds__(Cfg<BN>::kThreads, 1)
mf_moe_grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmapA, const __grid_constant__ CUtensorMap tmapB, const GemmParams p)
{
    using C = Cfg<BN>;
    extern __shared__ unsigned char smemRaw[];
    SharedStorage<BN> &s = *reinterpret_cast<SharedStorage<BN> *>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int KB = p.K / BK, NT = p.N / BN;

    if (threadIdx.x == 0) {
        for (int i = 0; i < C::kStages; i++) {
            MbarInit(&s.full[i], 1);
            MbarInit(&s.empty[i], 1);
        }
        for (int i = 0; i < C::kAccBufs; i++) {
            MbarInit(&s.tmemFull[i], 1);
            MbarInit(&s.tmemEmpty[i], C::kEpiWarps);  // one arrival per promotion warp
        }
        for (int i = 0; i < 2; i++) {
            MbarInit(&s.scaleFull[i], 2);
            MbarInit(&s.scaleEmpty[i], C::kEpiWarps);
        }
        s.abortFlag = 0;
        MbarInitFence();
        TmaPrefetchDesc(&tmapA);
        TmaPrefetchDesc(&tmapB);
    }
    if (warp == 0) {
        TmemAlloc(&s.tmemBase, kTmemCols);
    }
    GridDependency();  // what stands above ran under the end of the kernel before
    for (int g = threadIdx.x; g < p.G; g += C::kThreads) {
        s.groupOffset[g] = p.groupOffset[g];
        s.groupCount[g] = p.groupCount[g];
        s.tilePrefix[g + 1] = ((s.groupCount[g] + BM - 1) / BM) * NT;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0;
        s.tilePrefix[0] = 0;
        for (int g = 0; g < p.G; g++) {
            acc += s.tilePrefix[g + 1];
            s.tilePrefix[g + 1] = acc;
        }
    }
    TcFenceBefore();
    __syncthreads();
    TcFenceAfter();
    const uint32_t tmemBase = s.tmemBase;
    const int totalTiles = s.tilePrefix[p.G];
    volatile int *abortFlag = &s.abortFlag;

    auto decode = [&](int tile, int &g, int &mt, int &nt) {
        int lo = 0, hi = p.G;  // last group whose first tile is <= tile (empty groups share a prefix value: take the last)
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s.tilePrefix[mid] <= tile) {
                lo = mid;
            } else {
                hi = mid;
            }
        }
        g = lo;
        const int local = tile - s.tilePrefix[g];
        mt = local / NT;
        nt = local % NT;
    };

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        const bool elected = ElectOne();
        uint32_t st = 0, ph = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && __any_sync(0xffffffffu, tile < totalTiles); tile += gridDim.x) {
            int g, mt, nt;
            decode(tile, g, mt, nt);
            const int rowA = __reduce_max_sync(0xffffffffu, s.groupOffset[g] + mt * BM);
            const int rowB = __reduce_max_sync(0xffffffffu, g * p.N + nt * BN);
            for (int kb = 0; kb < KB; kb++) {
                if (!MbarWaitWarp(&s.empty[st], ph ^ 1, abortFlag)) {
                    ok = false;
                    break;
                }
                if (elected) {
                    MbarExpectTx(&s.full[st], kTileBytes + C::kBTile);
                    TmaLoad2D(s.a[st], &tmapA, &s.full[st], kb * BK, rowA);
                    TmaLoad2D(s.b[st], &tmapB, &s.full[st], kb * BK, rowB);
                }
                if (++st == C::kStages) {
                    st = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        constexpr uint32_t idesc = InstrDescF8(BM, BN);
        const bool elected = ElectOne();
        const uint32_t tmem = __reduce_or_sync(0xffffffffu, tmemBase);
        const uint64_t aDesc0 = SmemDescSw128(SmemAddr(s.a[0])), bDesc0 = SmemDescSw128(SmemAddr(s.b[0]));
        uint32_t st = 0, ph = 0, buf = 0, bph = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && __any_sync(0xffffffffu, tile < totalTiles); tile += gridDim.x) {
            for (int kb = 0; kb < KB; kb++) {
                if (!MbarWaitWarp(&s.tmemEmpty[buf], bph ^ 1, abortFlag) || !MbarWaitWarp(&s.full[st], ph, abortFlag)) {
                    ok = false;
                    break;
                }
                TcFenceAfter();
                if (elected) {
                    const uint64_t aDesc = aDesc0 + (uint64_t)(st * (uint32_t)(kTileBytes >> 4)), bDesc = bDesc0 + (uint64_t)(st * (uint32_t)(C::kBTile >> 4));
#pragma unroll
                    for (int k = 0; k < BK / 32; k++) {
                        // 32 fp8 elements = 32 bytes further along K inside the 128-byte swizzled row: +2 in 16-byte units.
                        MmaF8(tmem + buf * BN, aDesc + (uint64_t)(k * 2), bDesc + (uint64_t)(k * 2), idesc, k > 0 ? 1u : 0u);
                    }
                    MmaCommit(&s.empty[st]);      // the smem stage may be refilled once these MMAs have read it
                    MmaCommit(&s.tmemFull[buf]);  // the partial product is complete in TMEM
                }
                if (++st == C::kStages) {
                    st = 0;
                    ph ^= 1;
                }
                if (++buf == C::kAccBufs) {
                    buf = 0;
                    bph ^= 1;
                }
            }
        }
    } else if (warp < 4) {
        // ------------------------------------------------------------------ scales: a work item is a tile and four of its K-blocks
        const int row0 = (warp - 2) * (BM / 2) + lane;  // and row0 + 32
        struct Words {
            float a[2][4], b[BN / 128][4];
        };
        auto load4 = [&](const float *src, int kb0, bool valid, float (&f)[4]) {
            if (p.vecScales) {
                const float4 q = valid ? *reinterpret_cast<const float4 *>(src + kb0) : make_float4(0.f, 0.f, 0.f, 0.f);
                f[0] = q.x;
                f[1] = q.y;
                f[2] = q.z;
                f[3] = q.w;
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    f[k] = valid && kb0 + k < KB ? src[kb0 + k] : 0.f;
                }
            }
        };
        auto fetch = [&](int tile, int kb0, Words &w) {
            int g, mt, nt;
            decode(tile, g, mt, nt);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int rowInTile = row0 + 32 * j;
                const int row = s.groupOffset[g] + mt * BM + rowInTile;
                load4(p.aScale + (size_t)row * KB, kb0, mt * BM + rowInTile < s.groupCount[g] && row < p.rowsTotal, w.a[j]);
            }
#pragma unroll
            for (int c = 0; c < BN / 128; c++) {
                load4(p.bScale + ((size_t)g * (p.N / 128) + (size_t)(nt * (BN / 128) + c)) * KB, kb0, true, w.b[c]);
            }
        };
        Words cur, nxt;
        uint32_t it = 0;
        int tile = blockIdx.x, kb0 = 0;
        bool have = tile < totalTiles;
        if (have) {
            fetch(tile, kb0, cur);
        }
        for (; have && *abortFlag == 0; it++) {
            const int tileN = kb0 + 4 < KB ? tile : tile + (int)gridDim.x, kbN = kb0 + 4 < KB ? kb0 + 4 : 0;
            const bool haveNext = tileN < totalTiles;
            if (haveNext) {
                fetch(tileN, kbN, nxt);
            }
            const uint32_t buf = it & 1, ph = (it >> 1) & 1;
            if (!MbarWaitBounded(&s.scaleEmpty[buf], ph ^ 1, abortFlag)) {
                break;
            }
#pragma unroll
            for (int c = 0; c < BN / 128; c++) {
#pragma unroll
                for (int j = 0; j < 2; j++) {
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        s.scale[buf][c][k][row0 + 32 * j] = cur.a[j][k] * cur.b[c][k];
                    }
                }
            }
            __syncwarp();
            if (lane == 0) {
                MbarArrive(&s.scaleFull[buf]);
            }
            cur = nxt;
            tile = tileN;
            kb0 = kbN;
            have = haveNext;
        }
    } else {
        // ------------------------------------------------------------------ promotion + epilogue (one row, 64 columns per thread)
        const int quad = warp & 3;         // TMEM lanes this warp may touch: 32*quad .. 32*quad+31
        const int part = (warp - 4) >> 2;  // tile columns [64 * part, 64 * part + 64)
        const int rowInTile = quad * 32 + lane;
        uint64_t acc2[HC / 2];  // two fp32 sums each
#pragma unroll
        for (int i = 0; i < HC / 2; i++) {
            acc2[i] = 0;
        }
        uint32_t it = 0, item = 0;
        int tile = blockIdx.x, kb0 = 0;
        while (tile < totalTiles && *abortFlag == 0) {
            if (!MbarWaitBounded(&s.scaleFull[item & 1], (item >> 1) & 1, abortFlag)) {
                break;
            }
            const int n = min(4, KB - kb0);
            bool ok = true;
#pragma unroll 1
            for (int k = 0; k < n; k++, it++) {
                const uint32_t buf = it % C::kAccBufs, bph = (it / C::kAccBufs) & 1;
                if (!MbarWaitBounded(&s.tmemFull[buf], bph, abortFlag)) {
                    ok = false;
                    break;
                }
                TcFenceAfter();
                const uint32_t taddr = tmemBase + ((uint32_t)(quad * 32) << 16) + buf * BN + part * HC;
                const float scale = s.scale[item & 1][part / 2][k][rowInTile];
                const uint64_t sc = PackF32x2(scale, scale);
#pragma unroll
                for (int c = 0; c < HC; c += 16) {
                    float v[16];
                    TmemLd16Issue(taddr + c, v);
                    TmemLdWait16(v);
                    if (c == HC - 16) {
                        TcFenceBefore();
                        __syncwarp();
                        if (lane == 0) {
                            MbarArrive(&s.tmemEmpty[buf]);  // the warp's values are in registers: one arrival per warp keeps the barrier cheap
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        FmaF32x2(acc2[(c + i) / 2], PackF32x2(v[i], v[i + 1]), sc);
                    }
                }
            }
            if (!ok) {
                break;
            }
            __syncwarp();
            if (lane == 0) {
                MbarArrive(&s.scaleEmpty[item & 1]);
            }
            item++;
            kb0 += 4;
            if (kb0 >= KB) {
                int g, mt, nt;
                decode(tile, g, mt, nt);
                const int row = s.groupOffset[g] + mt * BM + rowInTile;
                // Rows past the end of A (group tables that overrun the buffer) are never read or written.
                if (mt * BM + rowInTile < s.groupCount[g] && row < p.rowsTotal) {
                    float acc[HC];
#pragma unroll
                    for (int i = 0; i < HC; i += 2) {
                        UnpackF32x2(acc2[i / 2], acc[i], acc[i + 1]);
                    }
                    const int col = nt * BN + part * HC;
                    const bool swiglu = (p.mode & 15) == MF_GEMM_EPI_SWIGLU;
                    __nv_bfloat16 *o = p.out + (size_t)row * p.outStride + (swiglu ? col / 2 : col);
                    if (swiglu) {
                        // Every 64 columns hold 32 gate projections followed by the 32 matching up projections.
#pragma unroll
                        for (int j = 0; j < HC / 2; j += 16) {
                            uint32_t pk[8];
#pragma unroll
                            for (int q = 0; q < 8; q++) {
                                const int c = j + 2 * q;
                                pk[q] = PackBf16(Silu(acc[c]) * acc[HC / 2 + c], Silu(acc[c + 1]) * acc[HC / 2 + c + 1]);
                            }
                            Store16(o + j, pk, p.wideStores);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < HC; j += 16) {
                            uint32_t pk[8];
#pragma unroll
                            for (int q = 0; q < 8; q++) {
                                pk[q] = PackBf16(acc[j + 2 * q], acc[j + 2 * q + 1]);
                            }
                            Store16(o + j, pk, p.wideStores);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < HC / 2; i++) {
                    acc2[i] = 0;
                }
                tile += gridDim.x;
                kb0 = 0;
            }
        }
    }
    // ---------------------------------------------------------------------- teardown
    TcFenceBefore();
    __syncthreads();
    if (s.abortFlag != 0 && threadIdx.x == 0 && p.status != nullptr) {
        atomicCAS(p.status, 0, 3 /* MF_DEV_ERR_PIPELINE */);
    }
    if (warp == 0) {
        TcFenceAfter();
        TmemDealloc(tmemBase, kTmemCols);
    }
}

// ---------------------------------------------------------------------------------------------- row quantisation (bf16 → fp8, 1x128 scales)

// x / sc as IEEE division rounds it, from rcp = the rounded 1 / sc: with FMAs one correction step of the product is enough
// (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990). Needs 0 < sc < infinity and
// a normal rcp; where the correction underflows, the quotient is far below the smallest e4m3 value.
__device__ __forceinline__ float DivByRcp(float x, float sc, float rcp)
{
    const float q = x * rcp;
    return q == 0.f ? q : fmaf(fmaf(-q, sc, x), rcp, q);  // the sum would lose the sign of a zero
}

constexpr int kQuantUnroll = 4;

// Bound by DRAM: 12288 x 7168 in 57 us = 4.6 TB/s (96 us with one load in flight and divisions). K is a multiple of 128, so the rows are one sequence of 128-element blocks; sixteen lanes own a block, eight elements
// each, and a warp takes 2 x kQuantUnroll consecutive blocks at once so that four 16-byte loads per lane are in flight.
__global__ void __launch_bounds__(256) mf_quant_rows_fp8_kernel(const __nv_bfloat16 *x, unsigned char *q, float *scale, int rows, int blocksPerRow,
                                                                const int *rowLimit)
{
    // No __restrict__: x and *rowLimit are written by kernels that this one may be resident with, so they must not be read by the
    // non-coherent path.
    GridDependency();
    const int lane = threadIdx.x & 31;
    const int limit = rowLimit != nullptr ? min(*rowLimit, rows) : rows;
    const long long total = (long long)limit * blocksPerRow;
    constexpr int kStep = 2 * kQuantUnroll;
    for (long long b0 = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kStep; b0 < total;
         b0 += (long long)gridDim.x * (blockDim.x >> 5) * kStep) {
        const long long first = b0 + (lane >> 4);
        uint4 raw[kQuantUnroll];
#pragma unroll
        for (int u = 0; u < kQuantUnroll; u++) {
            raw[u] = make_uint4(0u, 0u, 0u, 0u);  // past the end: a zero vector, so that the full-mask shuffles below stay convergent
            if (first + 2 * u < total) {
                raw[u] = *reinterpret_cast<const uint4 *>(x + (first + 2 * u) * 128 + (lane & 15) * 8);
            }
        }
#pragma unroll
        for (int u = 0; u < kQuantUnroll; u++) {
            const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw[u]);
            float f[8];
            float amax = 0.f;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float2 t = __bfloat1622float2(h[i]);
                f[2 * i] = t.x;
                f[2 * i + 1] = t.y;
                amax = fmaxf(amax, fmaxf(fabsf(t.x), fabsf(t.y)));
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            }
            const float sc = fmaxf(amax, 1e-10f) * (1.f / 448.f);
            if (sc < __int_as_float(0x7f800000)) {
                const float rcp = 1.f / sc;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    f[i] = DivByRcp(f[i], sc, rcp);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    f[i] = f[i] / sc;
                }
            }
            uint2 packed;
            unsigned short *ps = reinterpret_cast<unsigned short *>(&packed);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                ps[i] = __nv_cvt_float2_to_fp8x2(make_float2(f[2 * i], f[2 * i + 1]), __NV_SATFINITE, __NV_E4M3);
            }
            if (first + 2 * u < total) {
                *reinterpret_cast<uint2 *>(q + (first + 2 * u) * 128 + (lane & 15) * 8) = packed;
                if ((lane & 15) == 0) {
                    scale[first + 2 * u] = sc;
                }
            }
        }
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn GetEncodeTiled()
{
    static EncodeTiledFn fn = []() -> EncodeTiledFn {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult st;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &st) != cudaSuccess || st != cudaDriverEntryPointSuccess) {
            (void)cudaGetLastError();
            return nullptr;
        }
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// [rows, K] uint8 row-major, boxes of 128 (K) x boxRows, 128-byte swizzle.
bool MakeMap(CUtensorMap *m, const void *base, uint64_t rows, uint64_t K, uint32_t boxRows)
{
    EncodeTiledFn enc = GetEncodeTiled();
    if (enc == nullptr) {
        return false;
    }
    cuuint64_t dims[2] = {K, rows};
    cuuint64_t strides[1] = {K};
    cuuint32_t box[2] = {BK, boxRows};
    cuuint32_t estr[2] = {1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN>
int Launch(const void *a, const void *b, const GemmParams &p, int ctas, cudaStream_t stream)
{
    CUtensorMap mapA, mapB;
    if (!MakeMap(&mapA, a, (uint64_t)p.rowsTotal, (uint64_t)p.K, BM) || !MakeMap(&mapB, b, (uint64_t)p.G * p.N, (uint64_t)p.K, BN)) {
        return MF_K_LAUNCH_FAILED;
    }
    const size_t smem = sizeof(SharedStorage<BN>) + 1024;
    if (!AllowSmem<mf_moe_grouped_gemm_kernel<BN>>(smem)) {
        return MF_K_LAUNCH_FAILED;
    }
    const int sms = mf_k_sm_count();
    if (sms <= 0) {
        return MF_K_LAUNCH_FAILED;
    }
    const int grid = ctas > 0 && ctas < sms ? ctas : sms;
    if (LaunchDependent(mf_moe_grouped_gemm_kernel<BN>, (unsigned)grid, Cfg<BN>::kThreads, smem, stream, mapA, mapB, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return MF_K_LAUNCH_FAILED;
    }
    return MF_K_OK;
}

}  // namespace

extern "C" int mf_k_moe_grouped_gemm(const void *a, const float *aScale, const void *b, const float *bScale, void *out, const int *groupOffset,
                                     const int *groupCount, int G, int rowsTotal, int N, int K, int mode, int *status, int ctas, mf_stream_t stream)
{
    if (a == nullptr || b == nullptr || out == nullptr || aScale == nullptr || bScale == nullptr || groupOffset == nullptr || groupCount == nullptr ||
        G < 1 || G > kMaxGroups || rowsTotal < 1 || N % 128 != 0 || K % BK != 0 || N <= 0 || K <= 0) {
        return MF_K_INVALID;
    }
    if (((uintptr_t)a & 15) || ((uintptr_t)b & 15) || ((uintptr_t)out & 15)) {
        return MF_K_INVALID;  // TMA base addresses and the 16-byte epilogue stores need 16-byte alignment
    }
    if (ctas < 0) {
        ctas = 0;
    }
    GemmParams p;
    p.aScale = aScale;
    p.bScale = bScale;
    p.out = (__nv_bfloat16 *)out;
    p.groupOffset = groupOffset;
    p.groupCount = groupCount;
    p.status = status;
    p.G = G;
    p.N = N;
    p.K = K;
    p.mode = mode;
    p.outStride = (mode & 15) == MF_GEMM_EPI_SWIGLU ? N / 2 : N;
    p.rowsTotal = rowsTotal;
    p.wideStores = ((uintptr_t)out & 31) == 0 ? 1 : 0;
    p.vecScales = (K / BK) % 4 == 0 && ((uintptr_t)aScale & 15) == 0 && ((uintptr_t)bScale & 15) == 0 ? 1 : 0;
    const int sms = mf_k_sm_count();
    const bool wide = mf_k_gemm_tile(G, rowsTotal, N, ctas > 0 && ctas < sms ? ctas : sms) == 256;
    return wide ? Launch<256>(a, b, p, ctas, (cudaStream_t)stream) : Launch<128>(a, b, p, ctas, (cudaStream_t)stream);
}

extern "C" int mf_k_gemm_tile(int G, int rowsTotal, int N, int ctas)
{
    // The wide tile reads A half as often and hands a partial product over half as often: one K-block takes about 950 cycles instead
    // of 2 x 720. It pays from two m-tiles per expert on if every SM still gets two tiles (8191 rows over 32 experts, N 4096 / K 7168: 353
    // against 455 us); below that the weights' stream is what counts and the finer tiles end more evenly (2048 rows: 201 against 197 us).
    const long long mTiles = (rowsTotal + BM - 1) / BM;
    return N % 256 == 0 && mTiles >= 2LL * G && mTiles * (N / 256) >= 2LL * ctas ? 256 : 128;
}

extern "C" int mf_k_quant_rows_fp8(const void *x, void *q, float *scale, int rows, int K, const int *rowLimit, mf_stream_t stream)
{
    if (x == nullptr || q == nullptr || scale == nullptr || rows < 1 || K % 128 != 0) {
        return MF_K_INVALID;
    }
    const long long perCta = 8LL * 2 * kQuantUnroll;  // eight warps
    long long blocks = ((long long)rows * (K / 128) + perCta - 1) / perCta;
    if (blocks > 148 * 16) {
        blocks = 148 * 16;
    }
    if (LaunchDependent(mf_quant_rows_fp8_kernel, (unsigned)blocks, 256, 0, (cudaStream_t)stream, (const __nv_bfloat16 *)x, (unsigned char *)q, scale, rows,
                        K / 128, rowLimit) != cudaSuccess) {
        (void)cudaGetLastError();
        return MF_K_LAUNCH_FAILED;
    }
    return MF_K_OK;
}
