// twins-b200: the words that the slot barriers arrive at and wait for.
//
// What an entity sends in a slot (link messages and their tags, the RDMA model's frames, bucket tags and
// tail nodes) and what its world's controller is told (activity, wake-ups, messages done) is read by other
// SMs in the next slot; its own records are not. An arrival releases what its block, or its warp, wrote
// (the lanes' writes are ordered before it by the block's or the warp's barrier). The arrival that
// closes the slot acquires what the others released before it reads the slot's sums and publishes the
// next, and so does every wait before its block, or its warp, reads its entities' messages.
//
// A wait polls with relaxed loads and acquires once, when it is over: an acquire empties the SM's L1,
// which holds the records of the entities of all its warps, and an entity's first events of the slot
// then read them from L2. Measured, against waits without an acquire (the same results on every world
// tried, but PTX then orders none of what is read after the wait): 3-10% of a TCP run (k=8 NewReno 69.6 /
// 75.7 ms, 96 k=8 worlds 99.2 / 106 ms, k=16 68.6 / 70.5 ms), 0-2% of an RDMA run. A fence at the arrival that
// closes the slot instead of the acquiring load costs up to 3% more, acquiring polls up to 10% more (k=16
// 77.9 ms), and bringing the records back by loads ahead of the events gains nothing.
#pragma once
#include <cstdint>

namespace tb
{

__device__ __forceinline__ unsigned add_release(unsigned *p, unsigned v)
{
    unsigned o;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(o) : "l"(p), "r"(v) : "memory");
    return o;
}
__device__ __forceinline__ unsigned add_acq_rel(unsigned *p, unsigned v)
{
    unsigned o;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(o) : "l"(p), "r"(v) : "memory");
    return o;
}
__device__ __forceinline__ unsigned ld_acq(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
#ifdef X1
#define POLL ld_acq
#else
#define POLL ld_relaxed
#endif
__device__ __forceinline__ void st_release(int64_t *p, int64_t v)
{
    asm volatile("st.release.gpu.global.s64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_relaxed(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int64_t ld_relaxed(const int64_t *p)
{
    int64_t v;
    asm volatile("ld.relaxed.gpu.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
// (the value read is the one waited for: the word does not move on before its reader has arrived again)
__device__ __forceinline__ void acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    (void)v;
}
__device__ __forceinline__ void acquire(const int64_t *p)
{
    int64_t v;
    asm volatile("ld.acquire.gpu.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    (void)v;
}

} // namespace tb
