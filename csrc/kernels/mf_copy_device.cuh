// Device-side building blocks of the copy kernels: cache-hinted vector loads/stores and a CTA-cooperative span copy
// that handles any pair of byte alignments. Sources may be local HBM, a peer GPU's HBM mapped over NVLink, or pinned
// host memory; all are plain generic addresses in the global virtual address space.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace mf {
namespace dev {

// Streaming 16-byte load without L1 allocation (every byte is touched once). An ordinary load, not the non-coherent one: the copy kernels
// are launched as programmatic dependents, so a copy may be resident while the ones before it still write what it reads.
__device__ __forceinline__ uint4 LdStream16(const void *p)
{
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void StStream16(void *p, const uint4 &v)
{
    asm volatile("st.global.L1::no_allocate.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Copies n aligned 16-byte vectors with THREADS cooperating threads (this thread is `tid`), UNROLL independent loads in flight per
// thread before the first store; what is left at the end takes less than one trip and has the same loads in flight, each
// under its own bound.
template <int UNROLL, int THREADS>
__device__ __forceinline__ void CopyVec(uint4 *dst, const uint4 *src, unsigned n, unsigned tid)
{
    dst += tid;
    src += tid;
    int left = (int)n - (int)tid;  // this thread's vectors are those below it in steps of THREADS
    for (; left > 0; left -= UNROLL * THREADS, dst += UNROLL * THREADS, src += UNROLL * THREADS) {
        uint4 v[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            if (left > u * THREADS) {
                v[u] = LdStream16(src + u * THREADS);
            }
        }
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            if (left > u * THREADS) {
                StStream16(dst + u * THREADS, v[u]);
            }
        }
    }
}

// The same through the L1: for vectors that two threads read.
__device__ __forceinline__ uint4 LdShared16(const void *p)
{
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

// The 16 bytes that start `rel` (0..15) bytes into the 32 bytes of two neighbouring vectors: by two words, by one, by bits.
__device__ __forceinline__ uint4 Realign16(const uint4 &a, const uint4 &b, unsigned rel)
{
    const bool two = (rel & 8) != 0, one = (rel & 4) != 0;
    const uint32_t t0 = two ? a.z : a.x, t1 = two ? a.w : a.y, t2 = two ? b.x : a.z, t3 = two ? b.y : a.w, t4 = two ? b.z : b.x, t5 = two ? b.w : b.y;
    const uint32_t w0 = one ? t1 : t0, w1 = one ? t2 : t1, w2 = one ? t3 : t2, w3 = one ? t4 : t3, w4 = one ? t5 : t4;
    const unsigned bits = (rel & 3) * 8;
    return make_uint4(__funnelshift_r(w0, w1, bits), __funnelshift_r(w1, w2, bits), __funnelshift_r(w2, w3, bits), __funnelshift_r(w3, w4, bits));
}

// nv 16-byte vectors to a 16-byte boundary from an address `rel` (1..15) bytes past `src`, a boundary. Memory is read and written
// in aligned vectors only: an output takes the source vector that it starts in and the following one, which the L1 holds for the
// neighbouring thread. Every source vector that is touched has at least one wanted byte, so nothing outside the pages of
// the source is read. Narrow loads (two bytes for a bf16 slice at an odd element) need eight times the instructions.
template <int UNROLL, int THREADS>
__device__ __forceinline__ void CopyRealigned(uint4 *dst, const uint4 *src, unsigned nv, unsigned rel, unsigned tid)
{
    dst += tid;
    src += tid;
    for (int left = (int)nv - (int)tid; left > 0; left -= UNROLL * THREADS, dst += UNROLL * THREADS, src += UNROLL * THREADS) {
        uint4 v[UNROLL], n[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            if (left > u * THREADS) {
                v[u] = LdShared16(src + u * THREADS);
                n[u] = LdShared16(src + u * THREADS + 1);
            }
        }
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            if (left > u * THREADS) {
                StStream16(dst + u * THREADS, Realign16(v[u], n[u], rel));
            }
        }
    }
}

// Copies [src, src+n), at most 1 GiB, to [dst, dst+n) with the threads (tid of THREADS). The destination is brought to a 16-byte
// boundary with byte stores; the body moves in 16-byte vectors whatever the two addresses are modulo 16.
template <int UNROLL, int THREADS>
__device__ __forceinline__ void CopySpan(unsigned char *dst, const unsigned char *src, unsigned n, unsigned tid)
{
    unsigned head = (16 - (unsigned)((uintptr_t)dst & 15)) & 15;
    if (head > n) {
        head = n;
    }
    if (tid < head) {
        dst[tid] = src[tid];
    }
    dst += head;
    src += head;
    n -= head;
    const unsigned body = n & ~15u;
    const unsigned rel = (unsigned)((uintptr_t)src & 15);
    uint4 *d16 = (uint4 *)dst;
    const uint4 *s16 = (const uint4 *)(src - rel);
    if (rel == 0) {
        CopyVec<UNROLL, THREADS>(d16, s16, body >> 4, tid);
    } else {
        CopyRealigned<UNROLL / 2, THREADS>(d16, s16, body >> 4, rel, tid);
    }
    const unsigned tail = n - body;
    if (tid < tail) {
        dst[body + tid] = src[body + tid];
    }
}

}  // namespace dev
}  // namespace mf
