// MoE expert-parallel dispatch and combine over the symmetric heap, each as ONE kernel that computes and communicates.
//
// dispatch  (a) histogram of this rank's (token, k) pairs per global expert, pushed to every rank; (b) after a cross-rank
//           barrier every rank knows the full count matrix and derives, without any further message, the row of the
//           destination rank's receive buffer where each of its pairs lands (experts contiguous, starts aligned to the
//           128-row GEMM tile, sources in rank order); (c) each token is quantised ONCE to e4m3 with 1x128 power-of-two
//           scales (UE8M0 exponent bytes, the format the block-scaled tensor-core GEMM consumes) in shared memory and its
//           bytes, scale words and routing record are stored straight into the receive buffers of the owners of its top-k
//           experts over NVLink; (d) a closing barrier tells the owners that everything has landed.
//           The owner-side tables (expert_offset / expert_count) that the grouped GEMM consumes are written on the way,
//           clamped to the capacity of the receive buffer: on overflow the call reports MF_DEV_ERR_BOUNDS and what was
//           published never points past the buffer.
//           A token whose top-k holds several experts of the same owner tells that owner, in the record of the first of
//           them (the "leader"), where its sibling rows are.
//           Arrival mode (args.arrive set): instead of (d) every row that has landed is counted, with release semantics, in a
//           counter of its 128-row tile on the owner; the kernel ends without a closing barrier and the grouped GEMM that
//           follows starts each tile when the counter of that tile is complete (mf_k_moe_grouped_gemm_mx_gated), so an owner
//           computes on what has arrived while slower senders are still pushing. Every pair carries its payload in this mode.
// combine   each expert owner reduces the sibling rows of a token with their routing weights (fp32) and pushes ONE row
//           per (token, owner) back to the source rank's landing zone [token][k of the leader][hidden]; after a barrier the
//           source adds the partial sums of the owners in fixed k order (fp32, deterministic) and writes bf16. A top-8
//           token over 8 ranks reaches 5.25 distinct owners on average, so a third of the return traffic never leaves
//           the owner.
// The reference library names MoE dispatch/combine only as a use case of its symmetric heap (README.md:53 of the reference);
// the flag/barrier discipline follows its sample kernel (example/shm/AllReduce/shm_all_reduce.cpp:69-112) with bounded waits.
// Like the all-reduce, both kernels take a rank's argument block by value, or an array of blocks in device memory so that tests can
// run all ranks of a fake heap as gridDim.y slices of one cooperative launch on a single GPU.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <mutex>

#include "mf/device/mf_shm_device.cuh"
#include "mf_kernels.h"
#include "mf_sm100_ptx.cuh"

namespace cg = cooperative_groups;
using mf::sm100::GridDependency;
using mf::sm100::LaunchDependent;

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxExperts = 1024;
constexpr int kMaxTopk = 32;
// A token routed to several experts of one owner crosses the link once and is replicated by the owner when the call moves at
// least this many (token, expert) pairs per rank on average; below it the scan of the receive buffer that the replication
// needs costs more than the link time it saves. Measured on two GPUs, top-8 of 64 experts, with the dispatch that worked a token per
// warp: 128 tokens per rank 45 us without and 109 us with it, 4096 tokens per rank 233 us without and 190 us with it. The
// present form (a CTA per token, the replication unchanged) has not run on several GPUs; the line stands where it was.
constexpr int kDedupMinPairsPerRank = 8192;

__device__ __forceinline__ void FailD(int *status, int code)
{
    if (threadIdx.x == 0 && status != nullptr) {
        atomicCAS(status, 0, code);
    }
}

// UE8M0 byte (biased exponent) of the smallest power of two >= t, clamped to [1, 253] so that its reciprocal is a normal float.
__device__ __forceinline__ uint32_t Ue8m0Ceil(float t)
{
    const uint32_t bits = __float_as_uint(t);
    const uint32_t e = ((bits >> 23) & 0xffu) + ((bits & 0x7fffffu) != 0u ? 1u : 0u);
    return e < 1u ? 1u : (e > 253u ? 253u : e);
}

__device__ __forceinline__ int ReadAbort(int *status, int *smemFlag)
{
    if (threadIdx.x == 0) {
        *smemFlag = status != nullptr ? *(volatile int *)status : 0;
    }
    __syncthreads();
    int v = *smemFlag;
    __syncthreads();
    return v;
}

// Epoch of this call: the kernel argument, or (argument 0) one more than the device-resident count of finished calls. Every CTA
// of the launch reads the same value: the count only moves when the LAST CTA of a launch retires (FinishEpochD).
template <typename Args>
__device__ __forceinline__ uint64_t ResolveEpochD(const Args &a, uint64_t epochArg)
{
    if (epochArg != 0 || a.epochState == nullptr) {
        return epochArg;
    }
    return *(volatile unsigned long long *)a.epochState + 1;
}

// Called by every thread of every CTA on every way out of the kernel (after its last use of the epoch).
template <typename Args>
__device__ __forceinline__ void FinishEpochD(const Args &a, uint64_t epochArg, uint64_t epoch)
{
    if (epochArg != 0 || a.epochState == nullptr) {
        return;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned long long done = atomicAdd(a.epochState + 1, 1ull);
        if (done == (unsigned long long)gridDim.x - 1) {
            a.epochState[1] = 0;
            *(volatile unsigned long long *)a.epochState = epoch;
            __threadfence();
        }
    }
}

// Meta words are written by other GPUs during this kernel: read them past the non-coherent path.
__device__ __forceinline__ int4 mf_ld_meta(const int4 *p)
{
    const uint4 u = mf_ld16_coherent(p);
    return make_int4((int)u.x, (int)u.y, (int)u.z, (int)u.w);
}

// A CTA works on one token at a time: every thread quantises 16 consecutive elements (32 bytes in, 16 out, the eight lanes of a
// 128-element block share the maximum) and stores them straight from registers to every row that gets them, while warp 0
// finds the rows. One warp per token with a stage in shared memory took 28 dependent loads a token; with one CTA per token and
// four per SM the small call is a few latencies long (128 tokens: 55 -> 15 us on one rank) and the large one is bound by its stores
// (4096 tokens, top-8 of 32 experts on one rank, 300 MB: 158 -> 75 us).
template <bool EMULATED>
__global__ void __launch_bounds__(kThreads, 4)
mf_moe_dispatch_kernel(const __grid_constant__ mf_moe_dispatch_args_t own, const mf_moe_dispatch_args_t *__restrict__ emulated, int H, int K, int E, uint32_t channel, uint64_t epochArg, uint64_t timeoutNs)
{
    GridDependency();
    cg::grid_group grid = cg::this_grid();
    const mf_moe_dispatch_args_t &a = EMULATED ? emulated[blockIdx.y] : own;
    const uint64_t epoch = ResolveEpochD(a, epochArg);
    if (epoch == 0) {
        FailD(a.status, MF_DEV_ERR_BOUNDS);  // neither an epoch argument nor a device-resident epoch
        return;
    }
    const MfDeviceMeta *m = reinterpret_cast<const MfDeviceMeta *>(a.meta);
    const int R = (int)m->rankCount, me = (int)m->rankId, EL = E / R;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nblk = H / 128;
    extern __shared__ unsigned char smem[];
    int *sendBase = reinterpret_cast<int *>(smem);                              // [E]
    int *totals = sendBase + kMaxExperts;                                       // [E] pairs per expert over all sources
    int *starts = totals + kMaxExperts;                                         // [E] first row of the expert on its owner
    __shared__ int2 target[2][kMaxTopk];  // per parity of the token: row on the owner (-1: none) and owner of each pair
    __shared__ int abortFlag;
    __shared__ int grandTotal;
    __shared__ int overflow;  // rows did not fit an owner's buffer: reported when no CTA reads the status any more to see whether to go on
    if (threadIdx.x == 0) {
        overflow = 0;
    }
    if (mf_check_bounds_enabled(m) &&
        !(mf_shm_in_own_window(m, a.cnt, (uint64_t)(a.arrive != nullptr ? 2 : 1) * R * E * 4) &&
          (a.arrive == nullptr || mf_shm_in_own_window(m, a.arrive, (uint64_t)(a.cap / 128) * 4)) && mf_shm_in_own_window(m, a.recvX, (uint64_t)a.cap * H) &&
          mf_shm_in_own_window(m, a.recvSf, (uint64_t)a.cap * nblk * 4) && mf_shm_in_own_window(m, a.recvMeta, (uint64_t)a.cap * 16) &&
          mf_shm_in_own_window(m, a.recvSib, (uint64_t)a.cap * MF_MOE_MAX_SIBLINGS * 8))) {
        FailD(a.status, MF_DEV_ERR_BOUNDS);  // the receive buffers are addressed by offset on every owner: they must be heap memory
        FinishEpochD(a, epochArg, epoch);
        return;
    }

    // ---- (a) histogram of my pairs per global expert
    const bool arrival = a.arrive != nullptr;
    const int *myCnt = a.cnt + (arrival ? (size_t)(epoch & 1) * R * E : 0);
    if (arrival) {
        // My tile counters start from zero before anybody is told (by the barrier below) that it may send.
        for (int i = blockIdx.x * kThreads + threadIdx.x; i < a.cap / 128; i += gridDim.x * kThreads) {
            a.arrive[i] = 0;
        }
    }
    const int pairs = a.T * K;
    if (blockIdx.x * kThreads < pairs) {
        for (int e = threadIdx.x; e < E; e += kThreads) {
            totals[e] = 0;
        }
        __syncthreads();
        for (int i = blockIdx.x * kThreads + threadIdx.x; i < pairs; i += gridDim.x * kThreads) {
            const int e = a.topkIdx[i];
            if (e >= 0 && e < E) {
                atomicAdd(&totals[e], 1);
            }
        }
        __syncthreads();
        for (int e = threadIdx.x; e < E; e += kThreads) {
            if (totals[e] != 0) {
                atomicAdd(&a.localCnt[e], totals[e]);
            }
        }
    }
    __threadfence();
    grid.sync();
    if (R == 1) {
        myCnt = a.localCnt;  // one rank: its own histogram is the count matrix, there is nobody to publish it to or wait for
    } else if (blockIdx.x == 0) {
        for (int i = threadIdx.x; i < E * R; i += kThreads) {
            const int r = i / E, e = i % E;
            int *peerCnt = mf_shm_peer(m, const_cast<int *>(myCnt), (uint32_t)r);
            peerCnt[me * E + e] = ((volatile int *)a.localCnt)[e];
        }
        // Nobody sends before every rank is inside this call (its receive buffers are free) and has published its counts.
        int rc = mf_barrier_cta(m, channel, 0, 2 * epoch - 1, timeoutNs);
        if (rc != MF_DEV_OK) {
            FailD(a.status, rc);
        }
    }
    if (R > 1) {
        grid.sync();
    }
    const bool dead = ReadAbort(a.status, &abortFlag) != 0;
    bool dedup = false;

    if (!dead) {
        // ---- (b) where my pairs land: sendBase[e] = start of expert e on its owner + pairs of lower ranks for e.
        // Column sums of the count matrix first (one expert per thread, R loads each), then short prefix walks in shared memory.
        for (int e = threadIdx.x; e < E; e += kThreads) {
            int tot = 0, before = 0;
            for (int s = 0; s < R; s++) {
                const int c = ((volatile const int *)myCnt)[s * E + e];
                tot += c;
                before += s < me ? c : 0;
            }
            totals[e] = tot;
            sendBase[e] = before;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < E; e += kThreads) {
            int start = 0;
            for (int e2 = (e / EL) * EL; e2 < e; e2++) {
                start += (totals[e2] + 127) & ~127;
            }
            starts[e] = start;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < E; e += kThreads) {
            sendBase[e] += starts[e];
        }
        if (warp == 0) {
            // Every rank holds the same count matrix, so every CTA of every rank takes the same decision.
            int sum = 0;
            for (int e = lane; e < E; e += 32) {
                sum += totals[e];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sum += __shfl_xor_sync(0xffffffffu, sum, o);
            }
            if (lane == 0) {
                grandTotal = sum;
            }
        }
        __syncthreads();
        dedup = !arrival && R > 1 && (long long)grandTotal >= (long long)R * (a.dedupMinPairs > 0 ? a.dedupMinPairs : kDedupMinPairsPerRank);
        if (blockIdx.x == 0) {
            // What the GEMM and combine consume never points past the receive buffer: an expert that starts beyond the
            // capacity is published empty, one that straddles it is cut. The senders skip the same rows.
            for (int el = threadIdx.x; el < EL; el += kThreads) {
                const int off = min(starts[me * EL + el], a.cap);
                a.expertOffset[el] = off;
                a.expertCount[el] = min(totals[me * EL + el], a.cap - off);
            }
            if (threadIdx.x == 0) {
                const int last = me * EL + EL - 1;
                const int off = starts[last] + ((totals[last] + 127) & ~127);
                a.expertOffset[EL] = min(off, a.cap);
                if (off > a.cap) {
                    overflow = 1;
                }
            }
        }
        __syncthreads();

        // ---- (c) quantise each token once, store it to the owners of its experts
        const int pieces = H / 16;
        for (int t = blockIdx.x, turn = 0; t < a.T; t += gridDim.x, turn ^= 1) {
            const unsigned char *row = reinterpret_cast<const unsigned char *>(a.x) + (size_t)t * H * 2;
            int2 *to = target[turn];
            uint4 raw[2][2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int p = threadIdx.x + i * kThreads;
                if (p < pieces) {
                    raw[i][0] = *reinterpret_cast<const uint4 *>(row + (size_t)p * 32);
                    raw[i][1] = *reinterpret_cast<const uint4 *>(row + (size_t)p * 32 + 16);
                }
            }
            int mySlot = -1, myOwner = -1;
            if (warp == 0) {
                // Lane k owns pair (t, k): its row on the owner, and whether it leads the pairs of this token on that owner.
                float myW = 0.f;
                if (lane < K) {
                    const int myE = a.topkIdx[t * K + lane];
                    myW = a.topkW[t * K + lane];
                    if (myE >= 0 && myE < E) {
                        mySlot = sendBase[myE] + atomicAdd(&a.cursor[myE], 1);
                        myOwner = myE / EL;
                        if (mySlot >= a.cap) {
                            overflow = 1;
                            mySlot = -1;  // the owner's buffer is full: this pair is dropped and the call reports the overflow
                        }
                    }
                    a.routed[t * K + lane] = make_int4(mySlot, myOwner, __float_as_int(myW), 0);
                }
                // Pairs of one (token, owner) form groups of up to 1 + MF_MOE_MAX_SIBLINGS in k order; the first of a group leads it.
                int before = 0, nsib = 0;
                const uint32_t leadDst = (uint32_t)(mySlot >= 0 ? myOwner : me);
                for (int j = 0; j < K; j++) {
                    const int oj = __shfl_sync(0xffffffffu, myOwner, j);
                    const int sj = __shfl_sync(0xffffffffu, mySlot, j);
                    if (mySlot >= 0 && sj >= 0 && oj == myOwner && j < lane) {
                        before++;
                    }
                }
                const bool leader = mySlot >= 0 && before % (MF_MOE_MAX_SIBLINGS + 1) == 0;
                int2 *sd = mf_shm_peer(m, a.recvSib, leadDst) + (size_t)(mySlot >= 0 ? mySlot : 0) * MF_MOE_MAX_SIBLINGS;
                for (int j = 0; j < K; j++) {
                    const int oj = __shfl_sync(0xffffffffu, myOwner, j);
                    const int sj = __shfl_sync(0xffffffffu, mySlot, j);
                    const float wj = __shfl_sync(0xffffffffu, myW, j);
                    if (leader && sj >= 0 && oj == myOwner && j > lane && nsib < MF_MOE_MAX_SIBLINGS) {
                        sd[nsib++] = make_int2(sj, __float_as_int(wj));
                    }
                }
                // In a large call only the leader of a (token, owner) group carries the payload over the link; the owner copies it
                // into the followers' rows after everything has landed (phase (e)): a token routed to several experts of one
                // other rank crosses NVLink once. Rows of this rank itself are written here one and all.
                if (lane < K) {
                    to[lane] = make_int2(dedup && myOwner != me && !leader ? -1 : mySlot, myOwner);
                }
                if (mySlot >= 0) {
                    // Followers of a (token, owner) group are marked; the leader carries the number of siblings and their rows.
                    const int kField = lane | (leader ? (nsib << 8) : MF_MOE_META_FOLLOWER);
                    mf_shm_peer(m, a.recvMeta, (uint32_t)myOwner)[mySlot] = make_int4(me, t, kField, __float_as_int(myW));
                }
            }
            __syncthreads();  // the targets are known; those of the token after next go into the same place only after the next round
            for (int p0 = 0; p0 < pieces; p0 += 2 * kThreads) {
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int p = p0 + threadIdx.x + i * kThreads;
                    const bool active = p < pieces;
                    if (p0 > 0 && active) {
                        raw[i][0] = *reinterpret_cast<const uint4 *>(row + (size_t)p * 32);
                        raw[i][1] = *reinterpret_cast<const uint4 *>(row + (size_t)p * 32 + 16);
                    }
                    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(raw[i]);
                    __nv_bfloat162 m2 = __float2bfloat162_rn(0.f);
                    if (active) {
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            m2 = __hmax2(m2, __habs2(h[q]));
                        }
                    }
                    const float2 ends = __bfloat1622float2(m2);
                    float amax = fmaxf(ends.x, ends.y);
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) {
                        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
                    }
                    if (!active) {
                        continue;
                    }
                    // Scale = smallest power of two >= amax / 448, as a biased exponent byte; multiplying by its reciprocal is exact.
                    const uint32_t eb = Ue8m0Ceil(amax * (1.f / 448.f));
                    const float inv = __uint_as_float((254u - eb) << 23);
                    uint4 packed;
                    unsigned short *ps = reinterpret_cast<unsigned short *>(&packed);
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const float2 f = __bfloat1622float2(h[q]);
                        ps[q] = __nv_cvt_float2_to_fp8x2(make_float2(f.x * inv, f.y * inv), __NV_SATFINITE, __NV_E4M3);
                    }
                    for (int k = 0; k < K; k++) {
                        const int2 d = to[k];
                        if (d.x < 0) {
                            continue;
                        }
                        mf_st16(reinterpret_cast<unsigned char *>(mf_shm_peer(m, a.recvX, (uint32_t)d.y)) + (size_t)d.x * H + (size_t)p * 16, packed);
                        if ((lane & 7) == 0) {
                            // the same exponent for the four 32-element steps of the block
                            mf_shm_peer(m, a.recvSf, (uint32_t)d.y)[(size_t)d.x * nblk + (p >> 3)] = eb * 0x01010101u;
                        }
                    }
                }
            }
            if (arrival) {
                // Everything this CTA stored for the token is visible system-wide before any of its rows is counted.
                __threadfence_system();
                __syncthreads();
                if (mySlot >= 0) {
                    atomicAdd_system(mf_shm_peer(m, a.arrive, (uint32_t)myOwner) + (mySlot >> 7), 1);
                }
            }
        }
    }
    // ---- (d) everything I sent is visible before my arrival is; when all have arrived, all receive buffers are complete
    if (R > 1) {
        __threadfence_system();
    }
    grid.sync();
    if (overflow != 0) {
        FailD(a.status, MF_DEV_ERR_BOUNDS);
    }
    if (blockIdx.x == 0) {
        if (!dead && !arrival && R > 1) {
            int rc = mf_barrier_cta(m, channel, 0, 2 * epoch, timeoutNs);
            if (rc != MF_DEV_OK) {
                FailD(a.status, rc);
            }
        }
        // leave the scratch counters clean for the next call
        for (int e = threadIdx.x; e < E; e += kThreads) {
            a.localCnt[e] = 0;
            a.cursor[e] = 0;
        }
    }
    if (!dedup) {
        FinishEpochD(a, epochArg, epoch);
        return;  // every row came with its payload (in arrival mode the consumers wait on the tile counters)
    }
    // ---- (e) every leader row that arrived here from another rank is copied into the rows of its followers (local memory only)
    grid.sync();
    if (dead || ReadAbort(a.status, &abortFlag) != 0) {
        FinishEpochD(a, epochArg, epoch);
        return;
    }
    {
        const int warpsTotal = gridDim.x * kWarps;
        const int rowsHere = min(starts[me * EL + EL - 1] + ((totals[me * EL + EL - 1] + 127) & ~127), a.cap);
        const unsigned char *rx = reinterpret_cast<const unsigned char *>(a.recvX);
        for (int r = blockIdx.x * kWarps + warp; r < rowsHere; r += warpsTotal) {
            int el = 0;
            while (el + 1 < EL && starts[me * EL + el + 1] <= r) {
                el++;
            }
            if (r - starts[me * EL + el] >= totals[me * EL + el]) {
                continue;  // padding row: whatever it holds is from an earlier call
            }
            const int4 meta = mf_ld_meta(a.recvMeta + r);
            const int nsib = (meta.z >> 8) & 0xff;
            if ((meta.z & MF_MOE_META_FOLLOWER) != 0 || meta.x == me || nsib == 0 || nsib > MF_MOE_MAX_SIBLINGS) {
                continue;
            }
            const int2 *sd = a.recvSib + (size_t)r * MF_MOE_MAX_SIBLINGS;
            int rowsOf[MF_MOE_MAX_SIBLINGS];
            int nf = 0;
            for (int i = 0; i < nsib; i++) {
                const int fr = sd[i].x;
                if (fr >= 0 && fr < rowsHere && fr != r) {
                    rowsOf[nf++] = fr;
                }
            }
            // The leader's row is read once, four vectors per lane at a time, and stored to every follower.
            const unsigned char *srcRow = rx + (size_t)r * H;
            for (int vb = lane; vb < H / 16; vb += 128) {
                uint4 raw[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    raw[j] = vb + 32 * j < H / 16 ? mf_ld16_coherent(srcRow + (size_t)(vb + 32 * j) * 16) : make_uint4(0u, 0u, 0u, 0u);
                }
                for (int i = 0; i < nf; i++) {
                    unsigned char *dx = reinterpret_cast<unsigned char *>(a.recvX) + (size_t)rowsOf[i] * H;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        if (vb + 32 * j < H / 16) {
                            mf_st16(dx + (size_t)(vb + 32 * j) * 16, raw[j]);
                        }
                    }
                }
            }
            for (int v = lane; v < nblk; v += 32) {
                const uint32_t w = ((volatile uint32_t *)a.recvSf)[(size_t)r * nblk + v];
                for (int i = 0; i < nf; i++) {
                    a.recvSf[(size_t)rowsOf[i] * nblk + v] = w;
                }
            }
        }
    }
    FinishEpochD(a, epochArg, epoch);
}

// Eight fp32 values as bf16, and two such vectors added to fp32 sums.
__device__ __forceinline__ uint4 PackRow(const float (&v)[8])
{
    uint4 pk;
    __nv_bfloat162 *hp = reinterpret_cast<__nv_bfloat162 *>(&pk);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        hp[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
    }
    return pk;
}

__device__ __forceinline__ void AddRow(float (&acc)[2][8], const uint4 (&raw)[2])
{
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw[c]);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float2 f = __bfloat1622float2(h[q]);
            acc[c][2 * q] += f.x;
            acc[c][2 * q + 1] += f.y;
        }
    }
}

// Weighted sum of up to `left` rows of y, in ascending lane order over the lanes in `group`, each of which holds a row and its
// weight. Four rows of two vectors are in flight per lane (the rows of a group lie far apart: latency, not bandwidth, would
// pace a one-at-a-time loop).
__device__ __forceinline__ void GatherGroup(float (&part)[2][8], uint32_t group, int left, int myRow, float myW, const void *y, size_t rowBytes, int rows,
                                            int v0, int vecs)
{
#pragma unroll
    for (int q = 0; q < 8; q++) {
        part[0][q] = part[1][q] = 0.f;
    }
    while (group != 0 && left > 0) {
        uint4 raw[4][2];
        float w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const bool any = group != 0 && left > 0;
            const int j = any ? __ffs(group) - 1 : 0;
            const int row = __shfl_sync(0xffffffffu, myRow, j);
            const float weight = __shfl_sync(0xffffffffu, myW, j);
            const bool taken = any && row >= 0 && row < rows;
            w[i] = taken ? weight : 0.f;  // an infinite weight must not meet the zeros of a slot that holds no row
            group &= group - 1;
            left--;
            raw[i][0] = raw[i][1] = make_uint4(0u, 0u, 0u, 0u);
            if (taken) {
                const char *rowp = reinterpret_cast<const char *>(y) + (size_t)row * rowBytes + (size_t)v0 * 16;
                if (v0 < vecs) {
                    raw[i][0] = mf_ld16_ordered(rowp);
                }
                if (v0 + 32 < vecs) {
                    raw[i][1] = mf_ld16_ordered(rowp + 512);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw[i][c]);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float2 f = __bfloat1622float2(h[q]);
                    part[c][2 * q] = fmaf(w[i], f.x, part[c][2 * q]);
                    part[c][2 * q + 1] = fmaf(w[i], f.y, part[c][2 * q + 1]);
                }
            }
        }
    }
}

// One rank. Bound by the traffic of the expert outputs: they are gathered by token from where dispatch put them, no landing zone is
// written and read and no receive buffer is scanned for leaders (7 of 8 of its rows are followers). Nothing waits on anything, so it
// is an ordinary launch. Top-8, hidden 7168, in a loop: 128 tokens 61 -> 6 us, 4096 tokens (530 MB) 247 -> 85 us.
template <bool MANY>  // more pairs a token than one group holds
__global__ void __launch_bounds__(kThreads, 3)
mf_moe_combine_alone_kernel(const __grid_constant__ mf_moe_combine_args_t a, int H, int K, uint64_t epochArg)
{
    GridDependency();
    const uint64_t epoch = ResolveEpochD(a, epochArg);
    if (epoch == 0) {
        FailD(a.status, MF_DEV_ERR_BOUNDS);  // neither an epoch argument nor a device-resident epoch
        return;
    }
    const MfDeviceMeta *m = reinterpret_cast<const MfDeviceMeta *>(a.meta);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int warpsTotal = gridDim.x * kWarps;
    __shared__ int abortFlag;
    if (mf_check_bounds_enabled(m) && !mf_shm_in_own_window(m, a.retY, (uint64_t)a.retRows * H * 2)) {
        FailD(a.status, MF_DEV_ERR_BOUNDS);
        FinishEpochD(a, epochArg, epoch);
        return;
    }
    if (ReadAbort(a.status, &abortFlag) != 0) {  // a call whose dispatch failed (overflow) moves no data
        FinishEpochD(a, epochArg, epoch);
        return;
    }
    // Work unit = (token, chunk of 64 vectors); lane k holds pair k.
    const int vecs = H / 8, units = (vecs + 63) / 64;
    for (long long u = (long long)blockIdx.x * kWarps + warp; u < (long long)a.T * units; u += warpsTotal) {
        const int t = (int)(u / units), v0 = (int)(u % units) * 64 + lane;
        int mySlot = -1, myOwner = -1;
        float myW = 0.f;
        if (lane < K) {
            const int4 pair = a.routed[t * K + lane];
            mySlot = pair.x;
            myOwner = pair.y;
            myW = __int_as_float(pair.z);
        }
        uint32_t pairs = __ballot_sync(0xffffffffu, myOwner >= 0);
        float acc[2][8];
        if (!MANY) {
            GatherGroup(acc, pairs, MF_MOE_MAX_SIBLINGS + 1, mySlot, myW, a.y, (size_t)H * 2, a.cap, v0, vecs);
        } else {
            // Groups of eight in k order, each rounded like a partial sum that travels.
#pragma unroll
            for (int q = 0; q < 8; q++) {
                acc[0][q] = acc[1][q] = 0.f;
            }
            while (pairs != 0) {
                float part[2][8];
                GatherGroup(part, pairs, MF_MOE_MAX_SIBLINGS + 1, mySlot, myW, a.y, (size_t)H * 2, a.cap, v0, vecs);
                const uint4 rounded[2] = {PackRow(part[0]), PackRow(part[1])};
                AddRow(acc, rounded);
                for (int i = 0; i < MF_MOE_MAX_SIBLINGS + 1; i++) {
                    pairs &= pairs - 1;
                }
            }
        }
        char *o = reinterpret_cast<char *>(a.out) + ((size_t)t * H + (size_t)v0 * 8) * 2;
        if (v0 < vecs) {
            mf_st16(o, PackRow(acc[0]));
        }
        if (v0 + 32 < vecs) {
            mf_st16(o + 512, PackRow(acc[1]));
        }
    }
    FinishEpochD(a, epochArg, epoch);
}

// Several ranks. Every pair travels as a partial sum through the landing zone, those of a rank's own tokens too: a form that gathered these
// directly, in units of 64 instead of 128 vectors, left too few loads in flight for groups of one or two rows (emulated ranks, 4096
// tokens in all, hidden 7168, top-8 of 32: 2 / 4 / 8 ranks 220 / 238 / 263 us, that form 308 / 346 / 421 us).
template <bool EMULATED>
__global__ void __launch_bounds__(kThreads, 3)
mf_moe_combine_kernel(const __grid_constant__ mf_moe_combine_args_t own, const mf_moe_combine_args_t *__restrict__ emulated, int H, int K, int EL, uint32_t channel, uint64_t epochArg, uint64_t timeoutNs)
{
    cg::grid_group grid = cg::this_grid();
    const mf_moe_combine_args_t a = EMULATED ? emulated[blockIdx.y] : own;
    const uint64_t epoch = ResolveEpochD(a, epochArg);
    if (epoch == 0) {
        FailD(a.status, MF_DEV_ERR_BOUNDS);  // neither an epoch argument nor a device-resident epoch
        return;
    }
    const MfDeviceMeta *m = reinterpret_cast<const MfDeviceMeta *>(a.meta);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int warpsTotal = gridDim.x * kWarps;
    __shared__ int offs[kMaxExperts + 1];
    __shared__ int cnts[kMaxExperts];
    __shared__ int abortFlag;
    if (mf_check_bounds_enabled(m) && !mf_shm_in_own_window(m, a.retY, (uint64_t)a.retRows * H * 2)) {
        FailD(a.status, MF_DEV_ERR_BOUNDS);
        FinishEpochD(a, epochArg, epoch);
        return;
    }
    for (int i = threadIdx.x; i <= EL; i += kThreads) {
        offs[i] = a.expertOffset[i];
        if (i < EL) {
            cnts[i] = a.expertCount[i];
        }
    }
    __syncthreads();
    const int rows = min(offs[EL], a.cap);
    const int vecs = H / 8;
    const uint32_t R = m->rankCount;
    // A call whose dispatch failed (overflow, timeout) moves no data; it still walks through the barriers so that the
    // peers' waits complete.
    const bool dead = ReadAbort(a.status, &abortFlag) != 0;

    // ---- push: one row per (token, owner): the leader's output plus its siblings', weighted, to the source rank's
    //      landing zone [token][k of the leader][:]
    // Work unit = (row, chunk of 128 vectors): a leader with many siblings is spread over several warps.
    const int chunks = (vecs + 127) / 128;
    for (long long u = (long long)blockIdx.x * kWarps + warp; u < (long long)rows * chunks && !dead; u += warpsTotal) {
        const int r = (int)(u / chunks), ch = (int)(u % chunks);
        int el = 0;
        while (el + 1 < EL && offs[el + 1] <= r) {
            el++;
        }
        if (r - offs[el] >= cnts[el]) {
            continue;  // padding row of the tile grid
        }
        const int4 meta = a.recvMeta[r];
        const uint32_t src = (uint32_t)meta.x;
        const int k = meta.z & 0xff, nsib = (meta.z >> 8) & 0xff;
        if ((meta.z & MF_MOE_META_FOLLOWER) != 0 || src >= R || meta.y < 0 || k >= K || (long long)meta.y * K + k >= a.retRows ||
            nsib > MF_MOE_MAX_SIBLINGS) {
            continue;
        }
        const int2 *sd = a.recvSib + (size_t)r * MF_MOE_MAX_SIBLINGS;
        int rowOf[MF_MOE_MAX_SIBLINGS + 1];
        float wOf[MF_MOE_MAX_SIBLINGS + 1];
        rowOf[0] = r;
        wOf[0] = __int_as_float(meta.w);
        int n = 1;
        for (int i = 0; i < nsib; i++) {
            const int2 e = sd[i];
            if (e.x >= 0 && e.x < rows) {
                rowOf[n] = e.x;
                wOf[n] = __int_as_float(e.y);
                n++;
            }
        }
        char *dst = reinterpret_cast<char *>(mf_shm_peer(m, a.retY, src)) + ((size_t)meta.y * K + k) * H * 2;
        // The lane's four vectors of the chunk are loaded together for every addend, so that four 16-byte loads per lane are
        // in flight (the rows of a group lie far apart: latency, not bandwidth, would pace a one-at-a-time loop).
        const int vEnd = min(vecs, (ch + 1) * 128);
        const int v0 = ch * 128 + lane;
        float acc[4][8];
#pragma unroll
        for (int j = 0; j < 4; j++) {
#pragma unroll
            for (int q = 0; q < 8; q++) {
                acc[j][q] = 0.f;
            }
        }
        for (int i = 0; i < n; i++) {
            const char *rowp = reinterpret_cast<const char *>(a.y) + (size_t)rowOf[i] * H * 2;
            uint4 raw[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                raw[j] = v0 + 32 * j < vEnd ? mf_ld16(rowp + (size_t)(v0 + 32 * j) * 16) : make_uint4(0u, 0u, 0u, 0u);
            }
            const float w = wOf[i];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw[j]);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    float2 f = __bfloat1622float2(h[q]);
                    acc[j][2 * q] = fmaf(w, f.x, acc[j][2 * q]);
                    acc[j][2 * q + 1] = fmaf(w, f.y, acc[j][2 * q + 1]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (v0 + 32 * j < vEnd) {
                uint4 pk;
                __nv_bfloat162 *hp = reinterpret_cast<__nv_bfloat162 *>(&pk);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    hp[q] = __floats2bfloat162_rn(acc[j][2 * q], acc[j][2 * q + 1]);
                }
                mf_st16(dst + (size_t)(v0 + 32 * j) * 16, pk);
            }
        }
    }
    __threadfence_system();
    grid.sync();
    if (blockIdx.x == 0) {
        int rc = mf_barrier_cta(m, channel, 0, epoch, timeoutNs);
        if (rc != MF_DEV_OK) {
            FailD(a.status, rc);
        }
    }
    grid.sync();
    if (ReadAbort(a.status, &abortFlag) != 0) {
        FinishEpochD(a, epochArg, epoch);
        return;
    }
    // ---- add the owners' partial sums (fp32, fixed order): pair k carries one iff no earlier pair of the token has the same owner
    for (int t = blockIdx.x * kWarps + warp; t < a.T; t += warpsTotal) {
        const char *base = reinterpret_cast<const char *>(a.retY) + (size_t)t * K * H * 2;
        char *o = reinterpret_cast<char *>(a.out) + (size_t)t * H * 2;
        const int myOwner = lane < K ? a.routed[t * K + lane].y : -1;  // lane k holds pair k
        int before = 0;
        for (int j = 0; j < K; j++) {
            before += __shfl_sync(0xffffffffu, myOwner, j) == myOwner && j < lane ? 1 : 0;
        }
        const uint32_t leaders = __ballot_sync(0xffffffffu, myOwner >= 0 && before % (MF_MOE_MAX_SIBLINGS + 1) == 0);
        // Four vectors per lane and trip, loaded together for every partial sum (same reason as above).
        for (int vb = lane; vb < vecs; vb += 128) {
            float acc[4][8];
#pragma unroll
            for (int j = 0; j < 4; j++) {
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    acc[j][q] = 0.f;
                }
            }
            for (int k = 0; k < K; k++) {
                if ((leaders >> k & 1u) == 0) {
                    continue;
                }
                const char *rowp = base + (size_t)k * H * 2;
                uint4 raw[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    raw[j] = vb + 32 * j < vecs ? mf_ld16_coherent(rowp + (size_t)(vb + 32 * j) * 16) : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw[j]);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        float2 f = __bfloat1622float2(h[i]);
                        acc[j][2 * i] += f.x;
                        acc[j][2 * i + 1] += f.y;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (vb + 32 * j < vecs) {
                    uint4 pk;
                    __nv_bfloat162 *hp = reinterpret_cast<__nv_bfloat162 *>(&pk);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        hp[i] = __floats2bfloat162_rn(acc[j][2 * i], acc[j][2 * i + 1]);
                    }
                    mf_st16(o + (size_t)(vb + 32 * j) * 16, pk);
                }
            }
        }
    }
    FinishEpochD(a, epochArg, epoch);
}

// Resident-CTA capacity of a kernel on the current device for a given dynamic shared-memory size; remembered per (device,
// kernel, size) because the occupancy query costs microseconds on a latency-critical call path.
int CoopCap(const void *kernel, size_t smem)
{
    struct Entry {
        const void *kernel;
        size_t smem;
        int dev;
        int capacity;
    };
    static Entry cache[32];
    static int used = 0;
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    {
        std::lock_guard<std::mutex> g(mu);
        for (int i = 0; i < used; i++) {
            if (cache[i].kernel == kernel && cache[i].smem == smem && cache[i].dev == dev) {
                return cache[i].capacity;
            }
        }
    }
    int perSm = 0, sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, kThreads, smem) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    const int cap = perSm * sms;
    if (cap > 0) {
        std::lock_guard<std::mutex> g(mu);
        if (used < 32) {
            cache[used++] = Entry{kernel, smem, dev, cap};
        }
    }
    return cap;
}

}  // namespace

// argsHost: the block of a real rank, by value; argsDev: nEmulatedRanks blocks in device memory. One of the two.
static int LaunchDispatch(const mf_moe_dispatch_args_t *argsHost, const mf_moe_dispatch_args_t *argsDev, int nEmulatedRanks, int rankCount, int H, int K,
                          int E, uint32_t channel, uint64_t epoch, uint64_t timeoutNs, int ctas, mf_stream_t stream)
{
    if ((argsHost == nullptr) == (argsDev == nullptr) || nEmulatedRanks < 1 || rankCount < 1 || rankCount > (int)MF_SIGNAL_MAX_RANKS || H <= 0 || H % 128 != 0 || K < 1 ||
        K > kMaxTopk || E < rankCount || E % rankCount != 0 || E > kMaxExperts || channel >= MF_SIGNAL_CHANNELS) {
        return MF_K_INVALID;
    }
    if (timeoutNs == 0) {
        timeoutNs = 2000000000ull;
    }
    const size_t smem = (size_t)3 * kMaxExperts * sizeof(int);
    const void *kernel = argsHost != nullptr ? (const void *)mf_moe_dispatch_kernel<false> : (const void *)mf_moe_dispatch_kernel<true>;
    const mf_moe_dispatch_args_t own = argsHost != nullptr ? *argsHost : mf_moe_dispatch_args_t{};
    int cap = CoopCap(kernel, smem);
    if (cap <= 0) {
        return MF_K_LAUNCH_FAILED;
    }
    int grid = cap / nEmulatedRanks;
    if (ctas > 0 && ctas < grid) {
        grid = ctas;
    }
    if (grid < 1) {
        return MF_K_TOO_LARGE;
    }
    void *kargs[] = {(void *)&own, (void *)&argsDev, (void *)&H, (void *)&K, (void *)&E, (void *)&channel, (void *)&epoch, (void *)&timeoutNs};
    dim3 g((unsigned)grid, (unsigned)nEmulatedRanks, 1), b(kThreads, 1, 1);
    cudaError_t e = cudaLaunchCooperativeKernel(kernel, g, b, kargs, smem, (cudaStream_t)stream);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return MF_K_LAUNCH_FAILED;
    }
    return MF_K_OK;
}

static int LaunchCombine(const mf_moe_combine_args_t *argsHost, const mf_moe_combine_args_t *argsDev, int nEmulatedRanks, int rankCount, int H, int K,
                         int EL, uint32_t channel, uint64_t epoch, uint64_t timeoutNs, int ctas, mf_stream_t stream)
{
    if ((argsHost == nullptr) == (argsDev == nullptr) || nEmulatedRanks < 1 || rankCount < 1 || rankCount > (int)MF_SIGNAL_MAX_RANKS || H <= 0 || H % 8 != 0 || K < 1 || K > 32 ||
        EL < 1 || EL > kMaxExperts || channel >= MF_SIGNAL_CHANNELS) {
        return MF_K_INVALID;
    }
    if (timeoutNs == 0) {
        timeoutNs = 2000000000ull;
    }
    const bool alone = argsHost != nullptr && rankCount == 1;
    auto aloneKernel = K > MF_MOE_MAX_SIBLINGS + 1 ? mf_moe_combine_alone_kernel<true> : mf_moe_combine_alone_kernel<false>;
    const void *kernel = alone                 ? (const void *)aloneKernel
                         : argsHost != nullptr ? (const void *)mf_moe_combine_kernel<false>
                                               : (const void *)mf_moe_combine_kernel<true>;
    const mf_moe_combine_args_t own = argsHost != nullptr ? *argsHost : mf_moe_combine_args_t{};
    int cap = CoopCap(kernel, 0);
    if (cap <= 0) {
        return MF_K_LAUNCH_FAILED;
    }
    int grid = cap / nEmulatedRanks;
    if (ctas > 0 && ctas < grid) {
        grid = ctas;
    }
    if (grid < 1) {
        return MF_K_TOO_LARGE;
    }
    void *kargs[] = {(void *)&own, (void *)&argsDev, (void *)&H, (void *)&K, (void *)&EL, (void *)&channel, (void *)&epoch, (void *)&timeoutNs};
    dim3 g((unsigned)grid, (unsigned)nEmulatedRanks, 1), b(kThreads, 1, 1);
    cudaError_t e = alone ? LaunchDependent(aloneKernel, (unsigned)grid, kThreads, 0, (cudaStream_t)stream, own, H, K, epoch)
                          : cudaLaunchCooperativeKernel(kernel, g, b, kargs, 0, (cudaStream_t)stream);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return MF_K_LAUNCH_FAILED;
    }
    return MF_K_OK;
}

extern "C" int mf_k_moe_dispatch(const mf_moe_dispatch_args_t *argsDev, int nEmulatedRanks, int rankCount, int H, int K, int E, uint32_t channel,
                                 uint64_t epoch, uint64_t timeoutNs, int ctas, mf_stream_t stream)
{
    return LaunchDispatch(nullptr, argsDev, nEmulatedRanks, rankCount, H, K, E, channel, epoch, timeoutNs, ctas, stream);
}

extern "C" int mf_k_moe_dispatch_rank(const mf_moe_dispatch_args_t *argsHost, int rankCount, int H, int K, int E, uint32_t channel, uint64_t epoch,
                                      uint64_t timeoutNs, int ctas, mf_stream_t stream)
{
    return LaunchDispatch(argsHost, nullptr, 1, rankCount, H, K, E, channel, epoch, timeoutNs, ctas, stream);
}

extern "C" int mf_k_moe_combine(const mf_moe_combine_args_t *argsDev, int nEmulatedRanks, int rankCount, int H, int K, int EL, uint32_t channel,
                                uint64_t epoch, uint64_t timeoutNs, int ctas, mf_stream_t stream)
{
    return LaunchCombine(nullptr, argsDev, nEmulatedRanks, rankCount, H, K, EL, channel, epoch, timeoutNs, ctas, stream);
}

extern "C" int mf_k_moe_combine_rank(const mf_moe_combine_args_t *argsHost, int rankCount, int H, int K, int EL, uint32_t channel, uint64_t epoch,
                                     uint64_t timeoutNs, int ctas, mf_stream_t stream)
{
    return LaunchCombine(argsHost, nullptr, 1, rankCount, H, K, EL, channel, epoch, timeoutNs, ctas, stream);
}
