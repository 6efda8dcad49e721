// Device pieces shared by the pair-test kernels (ig_graph.cu, ig_prefix.cu):
// mbarriers and bulk copies, the pass status, record slots, the look-back of
// the row-offset scans.
#pragma once

#include <cstdint>

namespace ig {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// Pass status word: a bounded wait ran out (the CTA left after its copies in
// flight had landed), or, worse, a copy in flight never landed either.
enum : int { kStatusOk = 0, kStatusTimeout = 1, kStatusCopyLost = 2 };

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// 1-D TMA bulk copy global -> this CTA's shared memory (16-byte aligned,
// size a multiple of 16).  Plain copy: no cluster multicast.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// Record slots.  Each warp takes slots from the global counter in chunks of
// kSlotChunk (one atomic per chunk instead of one per hit group: a single
// counter address is otherwise the limit on dense graphs) and keeps the rest
// of its chunk, the same in every lane's registers.  Slots a warp never fills
// are written as sentinels (cell = kNoCell) when the kernel ends; the scatter
// skips them.
constexpr unsigned kSlotChunk = 64;
constexpr uint32_t kNoCell = 0xffffffffu;

struct WarpSlots {
    unsigned long long base;  // next free slot of the warp's chunk
    unsigned left;            // free slots left in it
};

// Slots of the warp's next `total` records (warp-uniform call): record j goes
// to b0 + j for j < n0, else to b1 + j (b1 already less n0).
struct Slots {
    unsigned long long b0, b1;
    unsigned n0;
};

__device__ __forceinline__ Slots take_slots(unsigned long long *rec_count, WarpSlots &w, unsigned total, int lane)
{
    Slots s;
    s.b0 = w.base;
    s.b1 = 0;
    s.n0 = total;
    if (w.left >= total) {
        w.base += total;
        w.left -= total;
        return s;
    }
    s.n0 = w.left;
    const unsigned need = total - w.left;
    const unsigned take = need > kSlotChunk ? need : kSlotChunk;
    unsigned long long b1 = 0;
    if (lane == 0)
        b1 = atomicAdd(rec_count, (unsigned long long)take);
    b1 = __shfl_sync(kFull, b1, 0);
    s.b1 = b1 - s.n0;
    w.base = b1 + need;
    w.left = take - need;
    return s;
}

// Warp total of cnt and this lane's exclusive prefix.  When no lane has more
// than one hit (the usual case on sparse graphs) one ballot gives both,
// otherwise a shuffle scan does.
__device__ __forceinline__ void warp_count_prefix(uint32_t cnt, int lane, unsigned &total, unsigned &pre)
{
    const unsigned some = __ballot_sync(kFull, cnt != 0u);
    if (__all_sync(kFull, cnt <= 1u)) {
        total = (unsigned)__popc(some);
        pre = (unsigned)__popc(some & ((1u << lane) - 1u));
        return;
    }
    unsigned incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o)
            incl += t;
    }
    total = __shfl_sync(kFull, incl, 31);
    pre = incl - cnt;
}

// Words of a scan by decoupled look-back (Merrill and Garland, 2016): a block's word is a sum in 62 bits
// under two bits saying what it is (0 nothing, 1 the block's own sum, 2 the
// prefix up to and including the block).
constexpr unsigned long long kOwnSum = 1ull << 62, kPrefixSum = 2ull << 62, kSumMask = (1ull << 62) - 1;

// Sum of the degrees of all blocks before block b; lane-parallel in one warp.
// False when the wait ran out.
__device__ __forceinline__ bool look_back(const unsigned long long *words, int64_t b, long long wait_cycles,
                                          int *status, unsigned long long &before)
{
    const int lane = threadIdx.x & 31;
    before = 0ull;
    const long long t0 = clock64();
    for (int64_t end = b; end > 0; end -= 32) {
        const int64_t i = end - 1 - lane;
        unsigned long long w = kPrefixSum;  // before block 0: an empty prefix
        for (;;) {
            if (i >= 0)
                w = *reinterpret_cast<const volatile unsigned long long *>(words + i);
            if (__all_sync(kFull, w != 0ull))
                break;
            // every lane sees lane 0's view of the clock and of the status
            const bool stop = clock64() - t0 > wait_cycles ||
                              *reinterpret_cast<const volatile int *>(status) != kStatusOk;
            if (__shfl_sync(kFull, (int)stop, 0))
                return false;
        }
        const unsigned full = __ballot_sync(kFull, (w & kPrefixSum) != 0ull);
        // lanes up to the nearest complete prefix count
        const int last = full != 0u ? __ffs(full) - 1 : 31;
        unsigned long long v = lane <= last ? (w & kSumMask) : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            v += __shfl_xor_sync(kFull, v, o);
        before += v;
        if (full != 0u)
            break;
    }
    return true;
}

}  // namespace
}  // namespace ig
