// Pair pass of one large sparse job, with the work of shared prefixes done
// once.
//
// The level words of a row's prefix against a set of columns do not depend on
// what follows the prefix, and among many words most rows share a long prefix
// with another row: of 300,000 uniform words of length 16, 4.6 share their
// first eight characters.  So the words are sorted by their first characters
// (a bucket sort by the first D2), a warp holds 2,048 columns (a lane the
// tables of 64) and walks the sorted rows, one row at a time, all lanes the
// same row: the levels of the first D1 = D2 - 2 characters are kept while rows
// share them, those of the first D2 likewise, and only the rest is run for
// every row.
//
//   bucket_zero     bucket counts, flag words, degrees, scan words
//   bucket_count    words per bucket, each word's number in its bucket
//   bucket_scan     first sorted place of every bucket
//   bucket_place    sorted words and their original ids
//   column_tables   per 2,048 sorted columns: one-hot words by position,
//                   character and lane
//   row_records     per sorted row: the table offset of each character, and
//                   whether its first D1 / D2 characters differ from the row
//                   before
//   prefix_pairs    the pair tests; hits as (row, column) records in sorted
//                   numbers
//   count_degrees, degree_offsets, place_columns, sort_rows
//                   the upper CSR in original ids: a record's edge belongs to
//                   the smaller id; degrees, their scan, columns into their
//                   rows in any order, rows sorted
//
// Bound by the ALU pipe (k = 3, 4: 78 and 90 % active) and, at k = 2, the
// shared-memory pipe (86 %).  Three-input operations per 2,048 pair tests: 94
// of 123 issued at L = 12, k = 3 (200,000 code words), 331 of 359 at L = 16,
// k = 4 (100,000 uniform words), where the general pass needs 226 and 516.
// Measured against the general pass on a B200, whole builds: 201,601 words
// L = 12 k = 3 4.65 -> 3.28 ms, 150,001 L = 15 k = 2 1.89 -> 1.39 ms, 300,000
// L = 16 k = 4 21.9 -> 13.6 ms; the count of 100,003 L = 16 k = 3 1.58 -> 1.14 ms.
//
// The result is the same CSR as the general pass's (ig_graph.cu): it depends
// neither on the order inside a bucket nor on the order of the records.
#include <algorithm>
#include <cstdio>

#include "ig_internal.h"
#include "ig_pairs.cuh"
#include "ig_slice.cuh"

namespace ig {
namespace {

using slice::imad;
using slice::Words2;

// One warp per CTA: warps of a CTA share nothing but would wait for each other
// at every row tile (2 / 4 warps and tiles of 32: 3.9 / 4.1 ms instead of 3.3 on
// 201,601 code words at L = 12, k = 3).  Tiles of 32 rows instead of 16 cost 5 %
// there, of 8 saved 0.5 % at k = 3 and 4 and cost 2 % at k = 2.
constexpr int kWarps = 1;                        // warps of a CTA
constexpr int kWarpCols = 2048;                  // columns of a warp
constexpr int kBlockCols = kWarps * kWarpCols;   // columns of a CTA
static_assert(kBlockCols == kPrefixBlockCols, "the tiling that a graph reports");
constexpr int kTileRows = 16;                    // rows per staged tile
constexpr int kRowBytes = 64;                    // a row record: 16 table offsets
constexpr int kPosBytes = 1024;                  // table bytes per position: 4 characters x 32 lanes x 2 words
constexpr uint32_t kNewD2 = 1u, kNewD1 = 2u;     // row flags, in the low bits of offset 0

// Flag words of a pass (same places as the general pass reports them from).
enum : int { kFlagWork = 0, kFlagSlots = 1, kFlagStatus = 2, kFlagHits = 3, kFlagBig = 4, kFlagCount = 8 };

struct PrefixArgs {
    const uint4 *tables;       // [columns / 2048][L][4][32][2] words
    const uint4 *records;      // row records
    int32_t n, seg_rows;       // rows per item (a multiple of kTileRows, dividing kBlockCols)
    long long items;
    uint32_t one;
    int emit;
    unsigned long long *flags;
    uint2 *rec;
    unsigned long long rec_cap;
    long long wait_cycles;
    int skip_first_copy;       // test hook: withhold the first row tile of the first item
};

// Sorted place of a word's bucket: the first D1 characters, then those up to D2.
__device__ __forceinline__ uint32_t bucket_key(uint32_t w, int d1, int d2)
{
    return ((w & ((1u << (2 * d1)) - 1u)) << (2 * (d2 - d1))) | ((w >> (2 * d1)) & ((1u << (2 * (d2 - d1))) - 1u));
}

__global__ void bucket_zero(uint32_t *counts, int nbuckets, unsigned long long *flags, uint32_t *degrees,
                            long long ndegrees, unsigned long long *scan_words, long long nscan, int64_t *row_ptr)
{
    const long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long step = gridDim.x * (long long)blockDim.x;
    for (long long k = id; k < nbuckets; k += step)
        counts[k] = 0u;
    for (long long k = id; k < ndegrees; k += step)
        degrees[k] = 0u;
    for (long long k = id; k < nscan; k += step)
        scan_words[k] = 0ull;
    if (id < kFlagCount)
        flags[id] = 0ull;
    if (row_ptr && id == 0)
        row_ptr[0] = 0;
}

__global__ void bucket_count(const uint32_t *__restrict__ words, int32_t n, int d1, int d2, uint32_t *counts,
                             uint32_t *__restrict__ number)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n)
        number[i] = atomicAdd(&counts[bucket_key(words[i], d1, d2)], 1u);
}

// Exclusive scan of the bucket counts in place, one block of 1,024 threads,
// 4,096 counts (four a thread) at a time.
__global__ void __launch_bounds__(1024) bucket_scan(uint4 *counts, int nvec)
{
    __shared__ uint32_t warp_sum[2][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (int k = 0; k * 1024 < nvec; ++k) {
        uint4 c = counts[k * 1024 + threadIdx.x];
        const uint32_t sum = c.x + c.y + c.z + c.w;
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o)
                incl += t;
        }
        if (lane == 31)
            warp_sum[k & 1][wid] = incl;
        __syncthreads();
        const uint32_t w = warp_sum[k & 1][lane];
        uint32_t winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFull, winc, o);
            if (lane >= o)
                winc += t;
        }
        const uint32_t before = carry + __shfl_sync(kFull, winc - w, wid) + incl - sum;
        carry += __shfl_sync(kFull, winc, 31);
        counts[k * 1024 + threadIdx.x] = make_uint4(before, before + c.x, before + c.x + c.y, before + c.x + c.y + c.z);
    }
}

__global__ void bucket_place(const uint32_t *__restrict__ words, int32_t n, int d1, int d2,
                             const uint32_t *__restrict__ start, const uint32_t *__restrict__ number,
                             uint32_t *__restrict__ sorted, uint32_t *__restrict__ ids)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const uint32_t w = words[i];
    const uint32_t p = start[bucket_key(w, d1, d2)] + number[i];
    sorted[p] = w;
    ids[p] = (uint32_t)i;
}

// One warp per 32 columns: word (j, c) of lane l, half h of a 2,048-column
// block has bit b set where column 1,024 h + 32 l + b has character c at j.
__global__ void column_tables(const uint32_t *__restrict__ sorted, int32_t n, int L, uint32_t *__restrict__ tables)
{
    const int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;  // group of 32 columns
    const int lane = threadIdx.x & 31;
    const int64_t block = g / (kWarpCols / 32);
    if (block * kWarpCols >= n)
        return;
    const int in = (int)(g % (kWarpCols / 32));
    const int h = in >> 5, l = in & 31;
    const int64_t col = g * 32 + lane;
    const bool ok = col < n;
    const uint32_t w = ok ? sorted[col] : 0u;
    const uint32_t valid = __ballot_sync(kFull, ok);
    uint32_t *out = tables + block * (int64_t)(L * (kPosBytes / 4)) + l * 2 + h;
    const uint32_t clo = (lane & 1) ? kFull : 0u, chi = (lane & 2) ? kFull : 0u;
    for (int j0 = 0; j0 < L; j0 += 8) {
        uint32_t mine = 0u;
        for (int j = j0; j < min(j0 + 8, L); ++j) {
            const uint32_t lo = __ballot_sync(kFull, (w >> (2 * j)) & 1u);
            const uint32_t hi = __ballot_sync(kFull, (w >> (2 * j + 1)) & 1u);
            if ((lane >> 2) == j - j0)
                mine = ~((lo ^ clo) | (hi ^ chi)) & valid;
        }
        const int j = j0 + (lane >> 2);
        if (j < L)
            out[j * (kPosBytes / 4) + (lane & 3) * 64] = mine;
    }
}

__global__ void row_records(const uint32_t *__restrict__ sorted, int32_t n, int d1, int d2, uint4 *__restrict__ records)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;  // four threads a row
    const int64_t r = t >> 2;
    const int v = (int)(t & 3);
    if (r >= n)
        return;
    const uint32_t w = sorted[r];
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        o[k] = ((w >> (2 * (4 * v + k))) & 3u) * 256u;
    if (v == 0) {
        const uint32_t x = r > 0 ? w ^ sorted[r - 1] : kFull;
        if ((x & ((1u << (2 * d2)) - 1u)) != 0u)
            o[0] |= kNewD2;
        if ((x & ((1u << (2 * d1)) - 1u)) != 0u)
            o[0] |= kNewD1;
    }
    records[t] = make_uint4(o[0], o[1], o[2], o[3]);
}

// Shared memory of a CTA: the column tables of its warps, then a ring of two
// row tiles.
constexpr int kTileVec = kTileRows * kRowBytes / 16;
constexpr size_t prefix_smem(int L) { return (size_t)kWarps * L * kPosBytes + 2 * kTileVec * 16; }

// A row's match words against the lane's 64 columns.
template <int L>
struct PrefixEq {
    const char *smem;
    const uint32_t *rec;  // the row's offsets, in the ring
    uint32_t lane_base, one;
    __device__ __forceinline__ Words2 operator()(int i, int j) const
    {
        const uint32_t off = i == 0 ? rec[0] & ~3u : rec[i];
        const uint2 v = *reinterpret_cast<const uint2 *>(smem + imad(off, one, lane_base) + j * kPosBytes);
        return Words2{v.x, v.y};
    }
};

template <int L, int K, int D1, int D2>
__global__ void __launch_bounds__(kWarps * 32, 12) prefix_pairs(const PrefixArgs a)
{
    extern __shared__ __align__(128) uint4 smem4[];
    __shared__ __align__(8) uint64_t bar[3];  // two ring slots, the tables
    __shared__ long long item_sh;
    constexpr int kTableVec = L * kPosBytes / 16;  // uint4 per warp
    uint4 *ring = smem4 + kWarps * kTableVec;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const char *smem = reinterpret_cast<const char *>(smem4);
    const uint32_t lane_base = (uint32_t)(wid * kTableVec * 16 + lane * 8);
    int *status = reinterpret_cast<int *>(a.flags + kFlagStatus);
    if (tid == 0) {
        for (int b = 0; b < 3; ++b)
            mbar_init(&bar[b], 1);
        mbar_fence_init();
    }
    __syncthreads();
    WarpSlots ws{0ull, 0u};
    uint32_t parity = 0u;   // bit b: phase barrier b waits for next
    uint32_t flying = 0u;   // thread 0: barriers with a copy in flight
    bool aborted = false;
    unsigned long long hits = 0ull;
    const int segs = kBlockCols / a.seg_rows;  // row segments per block of columns

    for (;;) {
        if (tid == 0)
            item_sh = (long long)atomicAdd(a.flags + kFlagWork, 1ull);
        __syncthreads();
        const long long item = item_sh;
        if (item >= a.items)
            break;
        // column block cb owns the segments of rows below its end, (cb + 1) segs of them
        int cb = 0;
        {
            int lo = 0, hi = (a.n - 1) / kBlockCols;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if ((long long)segs * mid * (mid + 1) / 2 <= item)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            cb = lo;
        }
        const int32_t r0 = (int32_t)(item - (long long)segs * cb * (cb + 1) / 2) * a.seg_rows;
        const int32_t r1 = min(r0 + a.seg_rows, a.n);
        const int32_t wc0 = cb * kBlockCols + wid * kWarpCols;     // the warp's columns
        const int32_t wc1 = wc0 < a.n ? min(wc0 + kWarpCols, a.n) : 0;
        const int ntiles = (r1 - r0 + kTileRows - 1) / kTileRows;  // 0: a segment past the last row
        const bool skip = a.skip_first_copy && item == 0;
        auto issue = [&](int t) {
            const int32_t first = r0 + t * kTileRows;
            const uint32_t bytes = (uint32_t)min(kTileRows, r1 - first) * kRowBytes;
            mbar_arrive_expect_tx(&bar[t & 1], bytes);
            bulk_g2s(ring + (t & 1) * kTileVec, a.records + (size_t)first * (kRowBytes / 16), bytes, &bar[t & 1]);
            flying |= 1u << (t & 1);
        };
        // bounded wait on barrier b by every thread; false: all leave
        auto wait = [&](int b) -> bool {
            bool timed_out = false;
            const long long t0 = clock64();
            while (!mbar_try_wait(&bar[b], (parity >> b) & 1u)) {
                if (clock64() - t0 > a.wait_cycles) {
                    timed_out = true;
                    break;
                }
            }
            if (__syncthreads_or(timed_out)) {
                if (tid == 0)
                    atomicCAS(status, kStatusOk, kStatusTimeout);
                return false;
            }
            parity ^= 1u << b;
            flying &= ~(1u << b);
            return true;
        };
        if (ntiles > 0) {
            if (tid == 0) {
                const int blocks = (a.n - cb * kBlockCols + kWarpCols - 1) / kWarpCols;
                const uint32_t bytes = (uint32_t)(min(blocks, kWarps) * kTableVec * 16);
                mbar_arrive_expect_tx(&bar[2], bytes);
                bulk_g2s(smem4, a.tables + (size_t)cb * kWarps * kTableVec, bytes, &bar[2]);
                flying |= 4u;
                for (int t = 0; t < 2 && t < ntiles; ++t)
                    if (!(skip && t == 0))
                        issue(t);
            }
            if (!wait(2)) {
                aborted = true;
                break;
            }
        }
        slice::Levels<K> S1, S2;  // levels of the first D1 and D2 characters of the row before
        slice::levels_start<K>(S1);
        slice::levels_start<K>(S2);
        for (int t = 0; t < ntiles; ++t) {
            if (!wait(t & 1)) {
                aborted = true;
                break;
            }
            const int32_t first = r0 + t * kTileRows;
            const int nr = min(min(kTileRows, r1 - first), wc1 - first);  // rows with a column to their right
            const bool diagonal = first + kTileRows > wc0;
#pragma unroll 1
            for (int q = 0; q < nr; ++q) {
                PrefixEq<L> eq;
                eq.smem = smem;
                eq.rec = reinterpret_cast<const uint32_t *>(ring + (t & 1) * kTileVec) + q * (kRowBytes / 4);
                eq.lane_base = lane_base;
                eq.one = a.one;
                // the item's first row runs from the start whatever the row before it
                const uint32_t changed = (t | q) == 0 ? (kNewD1 | kNewD2) : eq.rec[0] & 3u;
                if (changed) {
                    if (changed & kNewD1) {
                        slice::levels_start<K>(S1);
                        slice::levels_advance<L, K, 0, D1>(eq, S1);
                    }
#pragma unroll
                    for (int d = 0; d < 2 * (K / 2) + 1; ++d)
#pragma unroll
                        for (int e = 0; e <= K; ++e)
                            S2[d][e] = S1[d][e];
                    slice::levels_advance<L, K, D1, D2>(eq, S2);
                }
                slice::Levels<K> S;
#pragma unroll
                for (int d = 0; d < 2 * (K / 2) + 1; ++d)
#pragma unroll
                    for (int e = 0; e <= K; ++e)
                        S[d][e] = S2[d][e];
                slice::levels_advance<L, K, D2, L>(eq, S);
                Words2 m = S[K / 2][K];
                if (!__any_sync(kFull, (m.a | m.b) != 0u))
                    continue;
                const int32_t row = first + q;
                if (diagonal) {  // columns beyond the row only
                    const int lo = min(max(row + 1 - (wc0 + lane * 32), 0), 32);
                    const int lob = min(max(row + 1 - (wc0 + 1024 + lane * 32), 0), 32);
                    m.a &= lo >= 32 ? 0u : kFull << lo;
                    m.b &= lob >= 32 ? 0u : kFull << lob;
                }
                const uint32_t cnt = (uint32_t)(__popc(m.a) + __popc(m.b));
                if (!a.emit) {
                    hits += cnt;
                    continue;
                }
                unsigned total, j;
                warp_count_prefix(cnt, lane, total, j);
                if (total == 0u)
                    continue;
                if (lane == 0)
                    hits += total;
                const Slots sl = take_slots(a.flags + kFlagSlots, ws, total, lane);
                uint32_t col = (uint32_t)(wc0 + lane * 32);
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    uint32_t bits = h ? m.b : m.a;
                    while (bits) {
                        const uint32_t c = (uint32_t)__ffs(bits) - 1u;
                        bits &= bits - 1u;
                        const unsigned long long idx = (j < sl.n0 ? sl.b0 : sl.b1) + j;
                        if (idx < a.rec_cap)
                            a.rec[idx] = make_uint2((uint32_t)row, col + c);
                        ++j;
                    }
                    col += 1024u;
                }
            }
            __syncthreads();
            if (tid == 0 && t + 2 < ntiles)
                issue(t + 2);
        }
        if (aborted)
            break;
        __syncthreads();
    }
    if (aborted && tid == 0) {
        // no copy may land after the CTA is gone
        for (int b = 0; b < 3; ++b) {
            if (!((flying >> b) & 1u))
                continue;
            const long long t0 = clock64();
            while (!mbar_try_wait(&bar[b], (parity >> b) & 1u)) {
                if (clock64() - t0 > a.wait_cycles) {
                    atomicExch(status, kStatusCopyLost);
                    break;
                }
            }
        }
    }
    if (a.emit && !aborted)
        for (unsigned k = lane; k < ws.left; k += 32)
            if (ws.base + k < a.rec_cap)
                a.rec[ws.base + k] = make_uint2(kNoCell, 0u);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        hits += __shfl_xor_sync(kFull, hits, o);
    if (lane == 0 && hits != 0ull)
        atomicAdd(a.flags + kFlagHits, hits);
}

// ---- the CSR in original ids ----

__device__ __forceinline__ bool complete(const unsigned long long *flags, unsigned long long rec_cap,
                                         unsigned long long col_cap)
{
    return *reinterpret_cast<const int *>(flags + kFlagStatus) == kStatusOk && flags[kFlagSlots] <= rec_cap &&
           flags[kFlagHits] <= col_cap;
}

// Upper degrees: a record's edge counts for the smaller original id.
__global__ void count_degrees(const uint2 *__restrict__ rec, const unsigned long long *__restrict__ flags,
                              unsigned long long rec_cap, unsigned long long col_cap, const uint32_t *__restrict__ ids,
                              uint32_t *__restrict__ degrees)
{
    if (!complete(flags, rec_cap, col_cap))
        return;
    const unsigned long long nrec = flags[kFlagSlots];
    const unsigned long long step = gridDim.x * (unsigned long long)blockDim.x;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < nrec; i += step) {
        const uint2 r = rec[i];
        if (r.x != kNoCell)
            atomicAdd(&degrees[min(ids[r.x], ids[r.y])], 1u);
    }
}

// row_ptr[r + 1] = sum of the degrees of rows 0..r: 1,024 rows a block, one
// look-back (ig_pairs.cuh).
constexpr int kOffsetRows = 1024;

__global__ void __launch_bounds__(256) degree_offsets(const uint32_t *__restrict__ degrees, int64_t rows,
                                                      int64_t *__restrict__ row_ptr, unsigned long long *words,
                                                      int *status, long long wait_cycles)
{
    __shared__ unsigned long long warp_sum[8], before_sh;
    __shared__ int64_t block_sh;
    if (threadIdx.x == 0)
        block_sh = (int64_t)atomicAdd(words, 1ull);
    __syncthreads();
    const int64_t block = block_sh;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t first = block * kOffsetRows + threadIdx.x * 4;
    unsigned long long d[4], sum = 0ull;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        sum += first + k < rows ? degrees[first + k] : 0u;
        d[k] = sum;
    }
    unsigned long long incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o)
            incl += t;
    }
    if (lane == 31)
        warp_sum[wid] = incl;
    __syncthreads();
    unsigned long long ahead = 0ull, total = 0ull;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < wid)
            ahead += warp_sum[w];
        total += warp_sum[w];
    }
    if (wid == 0) {
        if (lane == 0)
            *reinterpret_cast<volatile unsigned long long *>(words + 1 + block) =
                (block == 0 ? kPrefixSum : kOwnSum) | total;
        unsigned long long before = 0ull;
        const bool ok = look_back(words + 1, block, wait_cycles, status, before);
        if (lane == 0) {
            if (!ok)
                atomicCAS(status, kStatusOk, kStatusTimeout);
            else if (block > 0)
                *reinterpret_cast<volatile unsigned long long *>(words + 1 + block) = kPrefixSum | (before + total);
            before_sh = before;
        }
    }
    __syncthreads();
    const unsigned long long base = before_sh + ahead + (incl - sum);
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (first + k < rows)
            row_ptr[first + k + 1] = (int64_t)(base + d[k]);
}

// Columns into their rows, in any order (the degrees count down to 0).
__global__ void place_columns(const uint2 *__restrict__ rec, const unsigned long long *__restrict__ flags,
                              unsigned long long rec_cap, unsigned long long col_cap, const uint32_t *__restrict__ ids,
                              const int64_t *__restrict__ row_ptr, uint32_t *__restrict__ degrees,
                              int32_t *__restrict__ cols)
{
    if (!complete(flags, rec_cap, col_cap))
        return;
    const unsigned long long nrec = flags[kFlagSlots];
    const unsigned long long step = gridDim.x * (unsigned long long)blockDim.x;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < nrec; i += step) {
        const uint2 r = __ldcs(rec + i);
        if (r.x == kNoCell)
            continue;
        const uint32_t u = ids[r.x], v = ids[r.y];
        const uint32_t lo = min(u, v);
        const int64_t pos = row_ptr[lo] + (int64_t)atomicSub(&degrees[lo], 1u) - 1;
        if (pos >= 0 && (unsigned long long)pos < col_cap)
            cols[pos] = (int32_t)max(u, v);
    }
}

// Ascending bitonic sort (Batcher, 1968) of 32 E values, value e * 32 + lane in v[e].
template <int E>
__device__ __forceinline__ void warp_sort(int32_t (&v)[E], int lane)
{
#pragma unroll
    for (int k = 2; k <= 32 * E; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const int f = e ^ (j >> 5);
                    if (f > e) {
                        const bool up = ((e * 32) & k) == 0;
                        const int32_t lo = min(v[e], v[f]), hi = max(v[e], v[f]);
                        v[e] = up ? lo : hi;
                        v[f] = up ? hi : lo;
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const int32_t o = __shfl_xor_sync(kFull, v[e], j);
                    const bool up = ((e * 32 + lane) & k) == 0;
                    const bool lower = (lane & j) == 0;
                    v[e] = (up == lower) ? min(v[e], o) : max(v[e], o);
                }
            }
        }
    }
}

template <int E>
__device__ __forceinline__ void sort_in_registers(int32_t *row, int len, int lane)
{
    int32_t v[E];
#pragma unroll
    for (int e = 0; e < E; ++e)
        v[e] = e * 32 + lane < len ? row[e * 32 + lane] : INT32_MAX;
    warp_sort<E>(v, lane);
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (e * 32 + lane < len)
            row[e * 32 + lane] = v[e];
}

// Rows of up to 256 columns, a warp each, in registers; longer ones are listed
// for sort_long_rows.
__global__ void __launch_bounds__(256) sort_rows(const int64_t *__restrict__ row_ptr, int32_t n,
                                                 unsigned long long *__restrict__ flags, unsigned long long rec_cap,
                                                 unsigned long long col_cap, int32_t *__restrict__ cols,
                                                 uint32_t *__restrict__ list)
{
    if (!complete(flags, rec_cap, col_cap))
        return;
    const int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= n)
        return;
    const int64_t b = row_ptr[r];
    const int64_t len = row_ptr[r + 1] - b;
    if (len < 2)
        return;
    if (len <= 32)
        sort_in_registers<1>(cols + b, (int)len, lane);
    else if (len <= 64)
        sort_in_registers<2>(cols + b, (int)len, lane);
    else if (len <= 128)
        sort_in_registers<4>(cols + b, (int)len, lane);
    else if (len <= 256)
        sort_in_registers<8>(cols + b, (int)len, lane);
    else if (lane == 0)
        list[atomicAdd(flags + kFlagBig, 1ull)] = (uint32_t)r;
}

// Longer rows, a CTA each: the row's values (distinct ids) set bits of a
// bitmap over 128 Ki ids at a time and are read back in order.  `scratch` is
// as long as cols.  The last kernel of a pass: its first block reports.
constexpr int kMapWords = 4096;  // 16 KiB

__global__ void __launch_bounds__(1024) sort_long_rows(const int64_t *__restrict__ row_ptr, int32_t n,
                                                       const unsigned long long *__restrict__ flags,
                                                       unsigned long long rec_cap, unsigned long long col_cap,
                                                       int32_t *__restrict__ cols, const uint32_t *__restrict__ list,
                                                       int32_t *__restrict__ scratch, unsigned long long *host_flags,
                                                       int64_t *host_bounds)
{
    __shared__ uint32_t map[kMapWords];
    __shared__ uint32_t warp_sum[32];
    if (blockIdx.x == 0) {
        if (threadIdx.x < 4)
            host_flags[threadIdx.x] = flags[threadIdx.x];
        if (threadIdx.x < 2)
            host_bounds[threadIdx.x] = row_ptr[threadIdx.x == 0 ? 0 : n];
    }
    if (!complete(flags, rec_cap, col_cap))
        return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (unsigned long long q = blockIdx.x; q < flags[kFlagBig]; q += gridDim.x) {
        const uint32_t r = list[q];
        const int64_t b = row_ptr[r], len = row_ptr[r + 1] - b;
        for (int64_t i = threadIdx.x; i < len; i += blockDim.x)
            scratch[b + i] = cols[b + i];
        int64_t out = b;
        for (int64_t v0 = (int64_t)r / (kMapWords * 32) * (kMapWords * 32); v0 < n; v0 += kMapWords * 32) {
            for (int k = threadIdx.x; k < kMapWords; k += blockDim.x)
                map[k] = 0u;
            __syncthreads();
            for (int64_t i = threadIdx.x; i < len; i += blockDim.x) {
                const int64_t v = scratch[b + i] - v0;
                if (v >= 0 && v < kMapWords * 32)
                    atomicOr(&map[v >> 5], 1u << (v & 31));
            }
            __syncthreads();
            uint32_t w[kMapWords / 1024];
            uint32_t mine = 0;
#pragma unroll
            for (int k = 0; k < kMapWords / 1024; ++k) {
                w[k] = map[threadIdx.x * (kMapWords / 1024) + k];
                mine += __popc(w[k]);
            }
            uint32_t incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(kFull, incl, o);
                if (lane >= o)
                    incl += t;
            }
            if (lane == 31)
                warp_sum[wid] = incl;
            __syncthreads();
            uint32_t ahead = 0, total = 0;
            for (int k = 0; k < 32; ++k) {
                if (k < wid)
                    ahead += warp_sum[k];
                total += warp_sum[k];
            }
            int64_t p = out + ahead + (incl - mine);
#pragma unroll
            for (int k = 0; k < kMapWords / 1024; ++k) {
                uint32_t bits = w[k];
                while (bits) {
                    const int c = __ffs(bits) - 1;
                    bits &= bits - 1u;
                    cols[p++] = (int32_t)(v0 + (threadIdx.x * (kMapWords / 1024) + k) * 32 + c);
                }
            }
            out += total;
            __syncthreads();
        }
    }
}

using PairsKernel = void (*)(PrefixArgs);

template <int L, int K>
PairsKernel pairs_kernel_of(int d2)
{
    return d2 == 8 ? prefix_pairs<L, K, 6, 8> : prefix_pairs<L, K, 5, 7>;
}

template <int K, int... Ls>
PairsKernel pairs_kernel(int L, int d2, std::integer_sequence<int, Ls...>)
{
    PairsKernel k = nullptr;
    ((L == Ls + kPrefixMinLen ? (void)(k = pairs_kernel_of<Ls + kPrefixMinLen, K>(d2)) : void()), ...);
    return k;
}

PairsKernel pairs_kernel(int L, int k, int d2)
{
    using Lens = std::make_integer_sequence<int, IG_MAX_LEN - kPrefixMinLen + 1>;
    return k == 2 ? pairs_kernel<2>(L, d2, Lens{}) : k == 3 ? pairs_kernel<3>(L, d2, Lens{}) : pairs_kernel<4>(L, d2, Lens{});
}

#define IG_CUDA(call)                                                                                          \
    do {                                                                                                       \
        cudaError_t e_ = (call);                                                                               \
        if (e_ != cudaSuccess)                                                                                 \
            return cuda_error(ctx, e_, #call);                                                                 \
    } while (0)

}  // namespace

bool prefix_job(const JobSpec &j)
{
    const slice::Test t = slice::test_of(j.len, j.min_ed);
    return j.n >= kPrefixMinWords && j.len >= kPrefixMinLen && t.L == j.len && t.levels && t.k >= 2;
}

// The saving grows with the pair tests (0.06 to 0.2 ns each), the cost of
// degrees, placing and sorting with the edges: 15 to 30 ps each up to about 130
// edges a word, 45 at 156, 65 to 135 at 220, where half of the rows are too
// long for a warp's registers.  What decides is the share of pairs that are
// edges, for uniform words a matter of length and threshold, and the word
// count.  Whole builds of uniform words on a B200, this pass against the general
// one, ms:
//   L = 10, k = 2  400,000 6.5 / 11.6   800,000 46.7 / 45.7
//   L = 10, k = 3   33,000 0.34 / 0.25   60,000 1.04 / 0.62
//   L = 11, k = 3   50,000 0.40 / 0.45  130,000 2.07 / 2.26  145,000 2.87 / 2.83  160,000 3.71 / 3.47
//   L = 12, k = 3  300,000 6.7 / 11.6   600,000 37.3 / 45.6
//   L = 12, k = 4   33,000 0.41 / 0.34   60,000 1.30 / 0.95
//   L = 13, k = 4   60,000 0.82 / 0.90  209,000 9.65 / 10.08
//   L = 14, k = 4  300,000 13.2 / 20.6  500,000 41.4 / 56.3
// So: never at (10, 3) and (12, 4), up to 140,000 and 750,000 words at (11, 3)
// and (10, 2), elsewhere up to 256 edges a word (densities of 8 x 10^8 uniform
// pairs per length and threshold); jobs of editDist >= L/2 keep hit words.
bool prefix_build(const JobSpec &j)
{
    constexpr int32_t any = kMaxJobWords;
    static const int32_t most[IG_MAX_LEN - kPrefixMinLen + 1][3] = {  // by length and k = 2..4
        {750000, 0, 0},        {2988000, 140000, 0},   {10026000, 705000, 0}, {any, 2136000, 206000},
        {any, 6616000, 572000}, {any, any, 1638000},    {any, any, 4776000},
    };
    return prefix_job(j) && j.n <= most[j.len - kPrefixMinLen][j.min_ed - 3];
}

ig_status prefix_pass(Ctx *ctx, const uint32_t *d_words, const JobSpec &job, const PrefixOut *out,
                      unsigned long long *slots, unsigned long long *hits, int64_t *bounds)
{
    cudaStream_t st = ctx->stream;
    const int32_t n = job.n;
    const int L = job.len;
    const slice::Test test = slice::test_of(job.len, job.min_ed);
    // Below about two words per bucket the longer prefix saves nothing, as its
    // levels then run for most rows (150,000 words: 7 and 8 characters equal;
    // 300,000 words: 14.8 ms at 7, 13.6 at 8).
    const int d2 = n >= kPrefixLongWords ? 8 : 7, d1 = d2 - 2;
    const int nbuckets = 1 << (2 * d2);
    const PairsKernel kernel = pairs_kernel(L, test.k, d2);
    const size_t smem = prefix_smem(L);
    int per_sm = 0;
    IG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    IG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kWarps * 32, smem));
    const int grid = std::max(per_sm, 1) * ctx->sm_count;
    // workspace: tables | row records | sorted words | ids (also place numbers
    // within a bucket, before they are known) | degrees | list of long rows | buckets
    const int64_t blocks = ((int64_t)n + kWarpCols - 1) / kWarpCols;
    const size_t table_bytes = (size_t)blocks * L * kPosBytes;
    const size_t word_bytes = ((size_t)n * sizeof(uint32_t) + 255) & ~size_t(255);
    size_t off = 0;
    auto place = [&](size_t bytes) {
        const size_t at = off;
        off += (bytes + 255) & ~size_t(255);
        return at;
    };
    const size_t o_tab = place(table_bytes), o_rec = place((size_t)n * kRowBytes), o_sorted = place(word_bytes),
                 o_ids = place(word_bytes), o_num = place(word_bytes), o_deg = place(word_bytes),
                 o_bkt = place((size_t)nbuckets * sizeof(uint32_t));
    ig_status s = ensure_buffer(ctx, ctx->sel, off, "column tables");
    if (s != IG_OK)
        return s;
    if ((s = ensure_buffer(ctx, ctx->flags, kFlagCount * sizeof(unsigned long long), "flags")) != IG_OK)
        return s;
    const int64_t scan_blocks = ((int64_t)n + kOffsetRows - 1) / kOffsetRows;
    if ((s = ensure_buffer(ctx, ctx->scan_tmp, (size_t)(scan_blocks + 1) * sizeof(unsigned long long),
                           "scan workspace")) != IG_OK)
        return s;
    if ((s = ensure_staging(ctx, 128)) != IG_OK)
        return s;
    unsigned long long *host_flags = static_cast<unsigned long long *>(ctx->stage);
    int64_t *host_bounds = reinterpret_cast<int64_t *>(host_flags + 8);
    char *ws = static_cast<char *>(ctx->sel.ptr);
    uint32_t *tables = reinterpret_cast<uint32_t *>(ws + o_tab);
    uint4 *records = reinterpret_cast<uint4 *>(ws + o_rec);
    uint32_t *sorted = reinterpret_cast<uint32_t *>(ws + o_sorted), *ids = reinterpret_cast<uint32_t *>(ws + o_ids);
    uint32_t *number = reinterpret_cast<uint32_t *>(ws + o_num), *degrees = reinterpret_cast<uint32_t *>(ws + o_deg);
    uint32_t *buckets = reinterpret_cast<uint32_t *>(ws + o_bkt);
    unsigned long long *flags = static_cast<unsigned long long *>(ctx->flags.ptr);
    unsigned long long *scan_words = static_cast<unsigned long long *>(ctx->scan_tmp.ptr);
    int *status = reinterpret_cast<int *>(flags + kFlagStatus);

    PrefixArgs a{};
    a.tables = reinterpret_cast<const uint4 *>(tables);
    a.records = records;
    a.n = n;
    // about twenty items per CTA, of one row tile to 2,048 rows (ten cost 2 %,
    // forty gave 1 % on the largest)
    const long double pairs = (long double)n * (n - 1) / 2;
    a.seg_rows = 2048;
    while (a.seg_rows > kTileRows && pairs / ((long double)a.seg_rows * kBlockCols) < 20.0L * grid)
        a.seg_rows /= 2;
    const long long cblocks = ((long long)n + kBlockCols - 1) / kBlockCols;
    a.items = (kBlockCols / a.seg_rows) * cblocks * (cblocks + 1) / 2;
    a.one = 1u;
    a.emit = out ? 1 : 0;
    a.flags = flags;
    a.rec = out ? static_cast<uint2 *>(ctx->records.ptr) : nullptr;
    a.rec_cap = out ? rec_capacity(ctx) : 0;
    a.wait_cycles = ctx->wait_cycles;
    a.skip_first_copy = ctx->fault_tile_copy ? 1 : 0;
    ctx->fault_tile_copy = false;  // the injected fault is one-shot

    const unsigned word_grid = (unsigned)(((int64_t)n + 255) / 256);
    phase_begin(ctx, IG_PHASE_PREP);
    bucket_zero<<<ctx->sm_count, 256, 0, st>>>(buckets, nbuckets, flags, degrees, out ? n : 0, scan_words,
                                               out ? scan_blocks + 1 : 0, out ? out->row_ptr : nullptr);
    bucket_count<<<word_grid, 256, 0, st>>>(d_words + job.word_off, n, d1, d2, buckets, number);
    bucket_scan<<<1, 1024, 0, st>>>(reinterpret_cast<uint4 *>(buckets), nbuckets / 4);
    bucket_place<<<word_grid, 256, 0, st>>>(d_words + job.word_off, n, d1, d2, buckets, number, sorted, ids);
    column_tables<<<(unsigned)(blocks * (kWarpCols / 256)), 256, 0, st>>>(sorted, n, L, tables);
    row_records<<<(unsigned)(((int64_t)n * 4 + 255) / 256), 256, 0, st>>>(sorted, n, d1, d2, records);
    phase_end(ctx, IG_PHASE_PREP);
    IG_CUDA(cudaGetLastError());
    phase_begin(ctx, IG_PHASE_PAIRS);
    kernel<<<grid, kWarps * 32, smem, st>>>(a);
    phase_end(ctx, IG_PHASE_PAIRS);
    IG_CUDA(cudaGetLastError());
    ctx->launches += 7;
    if (out) {
        const int wide = ctx->sm_count * 16;
        phase_begin(ctx, IG_PHASE_COMPACT);
        phase_begin(ctx, IG_PHASE_PREFIX);
        count_degrees<<<wide, 256, 0, st>>>(a.rec, flags, a.rec_cap, out->col_cap, ids, degrees);
        degree_offsets<<<(unsigned)scan_blocks, 256, 0, st>>>(degrees, n, out->row_ptr, scan_words, status,
                                                              a.wait_cycles);
        phase_end(ctx, IG_PHASE_PREFIX);
        phase_begin(ctx, IG_PHASE_SCATTER);
        place_columns<<<wide, 256, 0, st>>>(a.rec, flags, a.rec_cap, out->col_cap, ids, out->row_ptr, degrees,
                                            out->cols);
        sort_rows<<<(unsigned)(((int64_t)n * 32 + 255) / 256), 256, 0, st>>>(out->row_ptr, n, flags, a.rec_cap,
                                                                             out->col_cap, out->cols, number);
        // the records are used up: their buffer is the scratch (8 bytes a slot, 4 a column)
        sort_long_rows<<<ctx->sm_count * 2, 1024, 0, st>>>(out->row_ptr, n, flags, a.rec_cap, out->col_cap, out->cols,
                                                           number, reinterpret_cast<int32_t *>(a.rec), host_flags,
                                                           host_bounds);
        phase_end(ctx, IG_PHASE_SCATTER);
        phase_end(ctx, IG_PHASE_COMPACT);
        IG_CUDA(cudaGetLastError());
        ctx->launches += 5;
    } else {
        IG_CUDA(cudaMemcpyAsync(host_flags, flags, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
    }
    IG_CUDA(cudaStreamSynchronize(st));
    phase_collect(ctx);
    s = pass_status(ctx, static_cast<int>(host_flags[kFlagStatus] & 0xffffffffu));
    if (s != IG_OK)
        return s;
    *slots = host_flags[kFlagSlots];
    *hits = host_flags[kFlagHits];
    if (bounds) {
        bounds[0] = host_bounds[0];
        bounds[1] = host_bounds[1];
    }
    return IG_OK;
}

}  // namespace ig
