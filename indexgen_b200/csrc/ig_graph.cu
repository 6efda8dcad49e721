// Conflict-graph construction on sm_100a.
//
// Replaces compute_chunk_kernel + the tile loop of src/cuda_edit_distance.py
// (:20-226, :278-446) and the Python edge writer (src/gpu_graph_generator.py:49-77).
//
// Pipeline for a batch of independent jobs (one job = n words of one length L
// and a threshold d; edge iff ED < d).  A single job is a batch of one; the
// clustered solve (src/SparseMat.cpp:927-1095) submits all clusters at once.
//   prep_units      words -> units of 64 columns: four one-hot words per
//                   position and 32 columns (ig_slice.cuh)
//   pair_kernel     ONE persistent launch per form for the whole batch: CTAs
//                   take (job, row band, column segment) items from an atomic
//                   queue and dispatch on the job's length and threshold; 256
//                   rows per band, one per thread; column tiles of the segment
//                   are staged into shared memory by cp.async.bulk (TMA bulk
//                   copy, no multicast) with a two-slot mbarrier pipeline; each
//                   thread tests its row against 64 columns at a time, bit-
//                   sliced (pair_levels: editDist <= 5, pair_deltas: above),
//                   and emits hits as (cell, column offset, rank) records into
//                   slots its warp takes in chunks, plus a per-(row, segment)
//                   count.
//   row_offsets     per-row exclusive prefix over its segments + degree, and
//                   the scan of the degrees -> row_ptr (int64)
//   scatter         cols[row_ptr[r] + prefix[cell] + rank] = col
//   (dense jobs: the pair kernel stores every hit word instead of records, and
//   expand_bits turns a cell's words into its columns at row_ptr + prefix)
// The result is one upper CSR over the concatenated rows with global column
// ids (block diagonal: jobs never share an edge), ascending per row and
// bit-exact by construction (no sort, no dependence on scheduling).
#include <algorithm>
#include <cstdio>
#include <cstring>

#include "ig_internal.h"
#include "ig_pairs.cuh"
#include "ig_slice.cuh"

namespace ig {

namespace {

using slice::imad;
using slice::kUnitCols;
using slice::Words2;

// Index of the job whose `key` range contains v (jobs sorted by key).
__device__ __forceinline__ int find_job_by_item(const JobDesc *jobs, int njobs, long long v)
{
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].item_off <= v)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ int find_job_by_unit(const JobDesc *jobs, int njobs, long long v)
{
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].unit_start <= v)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ int find_job_by_row(const JobDesc *jobs, int njobs, long long v)
{
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].word_off <= v)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// What a pass starts from zero: its flag words, row_ptr[0] and the words of the
// row-offset scan.  The first kernel clears them (a memset each costs a
// graph node and its gap).
constexpr int kFlagWords = 8;
struct PassZero {
    unsigned long long *flags;
    int64_t *row_ptr;                // null: count-only pass
    unsigned long long *scan_words;
    long long scan_count;
};

// A small job table travels as an argument of the first kernel, which writes it
// to device memory for the others: a copy node before it would cost every
// small build some 4 us.
constexpr int kInlineVecs = 224;
struct InlineTable {
    uint4 v[kInlineVecs];
    int vecs;  // 0: the table has been copied
};
static_assert(sizeof(JobDesc) % sizeof(uint4) == 0, "tables are whole vectors");

// Column units of every job, one warp per unit of 64 columns: word (j, c, h)
// has bit b set where column 32 h + b of the unit has character c at position j.
__global__ void prep_units(const uint32_t *__restrict__ words, JobDesc *__restrict__ table, int njobs,
                           long long total_units, uint4 *__restrict__ units, PassZero zero,
                           const __grid_constant__ InlineTable given)
{
    const long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const JobDesc *jobs = given.vecs > 0 ? reinterpret_cast<const JobDesc *>(given.v) : table;
    for (int k = (int)id; k < given.vecs && id < kInlineVecs; k += kInlineVecs)
        reinterpret_cast<uint4 *>(table)[k] = given.v[k];
    if (id < kFlagWords)
        zero.flags[id] = 0ull;
    if (zero.row_ptr && id == 0)
        zero.row_ptr[0] = 0;
    for (long long k = id; k < zero.scan_count; k += gridDim.x * (long long)blockDim.x)
        zero.scan_words[k] = 0ull;
    const long long u = id >> 5;
    const int lane = threadIdx.x & 31;
    if (u >= total_units)
        return;
    const JobDesc &J = jobs[find_job_by_unit(jobs, njobs, u)];
    const long long p = u - J.unit_start;
    const long long c0 = p * kUnitCols;
    const uint32_t *w = words + J.word_off;
    const bool oka = c0 + lane < J.n, okb = c0 + 32 + lane < J.n;
    slice::write_unit(oka ? w[c0 + lane] : 0u, okb ? w[c0 + 32 + lane] : 0u, oka, okb, J.L, lane,
                      reinterpret_cast<uint2 *>(units + J.unit_off + p * slice::unit_vec(J.L)));
}

struct PairArgs {
    const uint4 *units;
    const uint32_t *words;
    const JobDesc *jobs;
    int njobs;
    long long items;
    uint32_t one;     // 1, as an operand the compiler cannot see (imad)
    unsigned long long *work;
    unsigned long long *rec_count;  // record slots handed out (chunks of kSlotChunk)
    unsigned long long *hit_count;  // pair tests that are edges (exact)
    EdgeRecord *rec;
    unsigned long long rec_cap;
    uint2 *bits;  // hit words of the dense jobs
    uint32_t *counts;
    int *status;
    int emit;
    long long wait_cycles;  // bound on every mbarrier wait (SM clock cycles)
    int skip_first_copy;    // test hook: withhold the first tile copy of the kernel's first item
};

// A pair CTA's shared state.  The item functions below are calls, not inlined
// (one per length and threshold: together in one body they cost the register
// allocator a stack frame of 1.8 KB), so what they share is at file scope,
// where its loads stay shared-memory loads; each kernel's thread 0 copies its
// arguments in.
constexpr int kTileCols = 1024;                                        // columns per staged tile
constexpr int kSlotVec = kTileCols / kUnitCols * slice::unit_vec(IG_MAX_LEN);  // uint4 per ring slot (8 KiB)
__shared__ __align__(128) uint4 g_tile[2][kSlotVec];
__shared__ __align__(8) uint64_t g_bar[2];
__shared__ PairArgs g_args;
__shared__ long long g_item[2];  // the next item, alternating

// Thread 0: copy the tile of units starting at column c0 (at most kTileCols
// columns, up to c_hi) into ring slot `slot`.
template <int L>
__device__ __forceinline__ void ring_issue(int slot, const uint4 *units, int32_t c0, int32_t c_hi)
{
    const int nu = (min(kTileCols, c_hi - c0) + kUnitCols - 1) / kUnitCols;
    const uint32_t bytes = (uint32_t)nu * slice::unit_vec(L) * 16;
    mbar_arrive_expect_tx(&g_bar[slot], bytes);
    bulk_g2s(&g_tile[slot][0], units + (size_t)(c0 / kUnitCols) * slice::unit_vec(L), bytes, &g_bar[slot]);
}

// Ring state bits: bit s (s = 0, 1) is the phase parity slot s waits for
// next; kSkipped marks an item whose first tile copy the test hook withheld
// (cleared by that tile's wait).
constexpr uint32_t kSkipped = 4u;

// A CTA whose wait on a staged tile ran out leaves its item loop, but not
// before thread 0 has waited (bounded) for the copies it issued that may still
// be in flight into the CTA's shared memory -- slot b's, unless the test hook
// withheld it, and the other slot's, when the next tile was issued -- so that
// no bulk copy lands after the CTA is gone.  The wait happens once per kernel,
// after the item loop (ring_drain), where it costs the pair loop no
// registers; ring_note_abort leaves it what it needs: bit 0 = slot b, bit 1 =
// slot b's copy was issued, bit 2 = the other slot's copy was issued.
__shared__ uint32_t g_drain;

__device__ __forceinline__ void ring_note_abort(int b, bool b_issued, bool other_issued)
{
    atomicCAS(g_args.status, kStatusOk, kStatusTimeout);
    g_drain = (uint32_t)b | (b_issued ? 2u : 0u) | (other_issued ? 4u : 0u);
}

// Thread 0, after the item loop of an aborted CTA.  `parity` has slot b's bit
// already advanced past the phase that timed out.  Waiting on a phase that
// has completed returns at once; a copy that never lands is reported as
// kStatusCopyLost.
__device__ __forceinline__ void ring_drain(uint32_t parity)
{
    const uint32_t d = g_drain;
    const int b = (int)(d & 1u);
    const uint32_t pend = parity ^ (1u << b);  // the phase each slot still waits for
    for (int slot = 0; slot < 2; ++slot) {
        if (!((d >> (slot == b ? 1 : 2)) & 1u))
            continue;
        const long long t0 = clock64();
        while (!mbar_try_wait(&g_bar[slot], (pend >> slot) & 1u)) {
            if (clock64() - t0 > g_args.wait_cycles) {
                atomicExch(g_args.status, kStatusCopyLost);
                break;
            }
        }
    }
}

// Bits [0, 32) of the columns col0 + c that lie in the strict upper triangle
// of the job (col > row, col < n) for a valid row.
__device__ __forceinline__ uint32_t upper_mask(int32_t row, int32_t n, int32_t col0)
{
    const int lo = min(max(row + 1 - col0, 0), 32);
    const int hi = min(max(n - col0, 0), 32);
    const uint32_t below_lo = lo >= 32 ? kFull : (1u << lo) - 1u;
    const uint32_t below_hi = hi >= 32 ? kFull : (1u << hi) - 1u;
    return row < n ? below_hi & ~below_lo : 0u;
}

// Hit words of a dense job: the words of 64-column unit u for rows 0.. up to
// the end of the band whose diagonal the unit meets, unit after unit (the
// triangle, in blocks of 256 x 256), so that a warp's 32 rows store 256
// consecutive bytes.  Entry of (unit, row 0):
__host__ __device__ __forceinline__ long long unit_bits(long long u)
{
    const long long c = u >> 2;
    static_assert(kBandRows == 4 * slice::kUnitCols, "a band meets the diagonal in four units");
    return 2 * kBandRows * c * (c + 1) + (u & 3) * kBandRows * (c + 1);
}

// Records of one word's hits m (bit c: column offset off0 + c in the segment)
// at warp record numbers j, j+1, ... of the slots sl.  Ranks count the row's
// hits in its (row, segment) cell in column order, so the scatter needs no
// sort.
__device__ __forceinline__ void write_hits(EdgeRecord *rec, unsigned long long cap, uint32_t m, uint32_t cell, uint32_t off0,
                                           uint32_t &rank, const Slots &sl, unsigned &j)
{
    while (m) {
        const uint32_t c = (uint32_t)__ffs(m) - 1u;
        m &= m - 1u;
        const unsigned long long idx = (j < sl.n0 ? sl.b0 : sl.b1) + j;
        if (idx < cap)
            *reinterpret_cast<uint2 *>(rec + idx) = make_uint2(cell, (off0 + c) << 16 | rank);
        ++rank;
        ++j;
    }
}

// A row's match words in one staged unit: the unit's table at the offsets of
// the row's characters.
template <int L>
struct TileEq {
    uint32_t at[L];  // byte offsets in the ring
    __device__ __forceinline__ Words2 operator()(int i, int j) const
    {
        const uint2 v = *reinterpret_cast<const uint2 *>(reinterpret_cast<const char *>(&g_tile[0][0]) + at[i] +
                                                         j * slice::unit_pos_bytes());
        return Words2{v.x, v.y};
    }
};

template <int L_, int K>
struct LevelForm {
    static constexpr int L = L_;
    uint32_t k0;
    __device__ __forceinline__ explicit LevelForm(const JobDesc &J) : k0(J.k > 0 ? kFull : 0u) {}
    __device__ __forceinline__ Words2 hits(const TileEq<L> &eq) const { return slice::levels<L, K>(eq, k0); }
};

template <int L_, int W>
struct DeltaForm {
    static constexpr int L = L_;
    uint32_t nk[5];
    __device__ __forceinline__ explicit DeltaForm(const JobDesc &J)
    {
#pragma unroll
        for (int b = 0; b < 5; ++b)
            nk[b] = ((J.k >> b) & 1) ? 0u : kFull;
    }
    __device__ __forceinline__ Words2 hits(const TileEq<L> &eq) const
    {
        slice::Planes da, db;
        slice::deltas<L, W>(eq, da, db);
        return Words2{slice::at_most(da, nk), slice::at_most(db, nk)};
    }
};

// What a thread carries from item to item.
struct LoopState {
    WarpSlots ws;
    uint32_t parity;  // bit b: phase parity of ring slot b; kSkipped
    int turn;         // items run so far, modulo 2
    bool aborted;
};

// What is the same for a whole item and only needed now and then: kept in
// shared memory and read where it is used, not held in registers through the
// pair loop (which is short of them).
struct ItemShared {
    const uint4 *units;
    uint2 *bits;       // dense job: entry of (unit 0, first row of the band)
    uint32_t cell;     // count cell of the band's first row
    int32_t n, row0, seg0, c_lo, c_hi;
};
__shared__ ItemShared g_it;

template <class T>
__device__ __forceinline__ T now(const T &x)
{
    return *const_cast<const volatile T *>(&x);
}

// Units tested before the warp looks for hits: the vote, the branches and the
// loop cost some 35 of 200 ALU-pipe operations per unit at k = 2; two units a
// vote took 150,001 words at L = 15, k = 2 from 1.94 to 1.90 ms and 300,000 at
// L = 16, k = 4 from 22.1 to 21.9.
constexpr int kUnitsPerVote = 2;

// Ways out of the pair loop's common path (records of an item inside the
// triangle): uniform bits.
constexpr unsigned kCheck = 1u, kDense = 2u, kCountOnly = 4u;

// One (band, segment) item of job J: stream the segment's column tiles through
// the two-slot ring and test them against the band's rows, one per thread.
template <class Form>
__device__ __noinline__ LoopState run_item(const JobDesc *job, int band, int seg, LoopState state)
{
    constexpr int L = Form::L;
    const JobDesc &J = *job;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    uint32_t at[L];  // table offset of the row's character at each position
    const Form form(J);
    unsigned way = 0u;
    int ntiles;
    {
        const int32_t n = J.n;
        const int32_t row0 = band * kBandRows;
        // c_lo is a multiple of 256 (segments and bands are), so units never
        // straddle a segment
        const int32_t c_lo = (int32_t)max((long long)seg << J.seg_shift, (long long)row0);
        const int32_t c_hi = (int32_t)min((long long)(seg + 1) << J.seg_shift, (long long)n);
        ntiles = (c_hi - c_lo + kTileCols - 1) / kTileCols;
        // col > row, row < n and col < n only need a look on diagonal items,
        // the last (partial) band and a partial last unit
        const long long row_end = (long long)row0 + kBandRows;
        if ((long long)c_lo < row_end || row_end > (long long)n || (c_hi % kUnitCols) != 0)
            way |= kCheck;
        if (!g_args.emit)
            way |= kCountOnly;
        else if (J.bit_off >= 0)
            way |= kDense;
        const uint32_t w = g_args.words[J.word_off + (row0 + tid < n ? row0 + tid : 0)];
#pragma unroll
        for (int i = 0; i < L; ++i)
            at[i] = ((w >> (2 * i)) & 3u) * 8u;
        // test hook: the first tile of the kernel's first item is never copied
        if (g_args.skip_first_copy && J.item_off == 0 && band == 0 && seg == 0)
            state.parity |= kSkipped;
        if (tid == 0) {
            g_it.units = g_args.units + J.unit_off;
            g_it.bits = g_args.bits + J.bit_off + row0;
            g_it.cell = (uint32_t)(J.count_off + (long long)seg * n + row0);
            g_it.n = n;
            g_it.row0 = row0;
            g_it.seg0 = seg << J.seg_shift;
            g_it.c_lo = c_lo;
            g_it.c_hi = c_hi;
            for (int t = 0; t < 2 && t < ntiles; ++t)
                if (!(t == 0 && (state.parity & kSkipped)))
                    ring_issue<L>(t, g_it.units, c_lo + t * kTileCols, c_hi);
            // the next item's number, while the tile is on its way
            g_item[state.turn] = (long long)gridDim.x + (long long)atomicAdd(g_args.work, 1ull);
        }
    }
    const uint32_t one = g_args.one;
    uint32_t rank = 0;
    for (int t = 0; t < ntiles; ++t) {
        const int b = t & 1;
        bool timed_out = false;
        const long long t_start = clock64();
        while (!mbar_try_wait(&g_bar[b], (state.parity >> b) & 1u)) {
            if (clock64() - t_start > now(g_args.wait_cycles)) {
                timed_out = true;
                break;
            }
        }
        state.parity ^= 1u << b;
        // uniform decision: every thread leaves together if any gave up (and
        // the item's shared values are there for all)
        if (__syncthreads_or(timed_out)) {
            if (tid == 0)
                ring_note_abort(b, !(t == 0 && (state.parity & kSkipped)), t + 1 < ntiles);
            state.parity &= ~kSkipped;
            state.aborted = true;
            return state;
        }
        state.parity &= ~kSkipped;
        const int32_t c0 = now(g_it.c_lo) + t * kTileCols;
        const int nu = (min(kTileCols, now(g_it.c_hi) - c0) + kUnitCols - 1) / kUnitCols;
        const uint32_t at0 = (uint32_t)b * (kSlotVec * 16);
        TileEq<L> eq;
#pragma unroll 1
        for (int u0 = 0; u0 < nu; u0 += kUnitsPerVote) {
            // an odd last unit's partner is whatever the slot holds, left out below
            Words2 hit[kUnitsPerVote];
            uint32_t some = 0u;
#pragma unroll
            for (int q = 0; q < kUnitsPerVote; ++q) {
#pragma unroll
                for (int i = 0; i < L; ++i)
                    eq.at[i] = imad(at[i], one, at0 + (uint32_t)(u0 + q) * (slice::unit_vec(L) * 16));
                hit[q] = form.hits(eq);
                some |= hit[q].a | hit[q].b;
            }
            if (!(way & kDense) && !__any_sync(kFull, some != 0u))
                continue;
#pragma unroll 1
            for (int q = 0; q < kUnitsPerVote; ++q) {
                if (u0 + q >= nu)
                    break;
                Words2 m = q == 0 ? hit[0] : hit[kUnitsPerVote - 1];
                const int32_t col0 = c0 + (u0 + q) * kUnitCols;
                if (way & (kCheck | kDense)) {
                    const int32_t n = now(g_it.n), row = now(g_it.row0) + tid;
                    if (way & kCheck) {
                        m.a &= upper_mask(row, n, col0);
                        m.b &= upper_mask(row, n, col0 + 32);
                    }
                    if (way & kDense) {
                        if (row < n)
                            now(g_it.bits)[unit_bits(col0 / kUnitCols) + tid] = make_uint2(m.a, m.b);
                        rank += (uint32_t)(__popc(m.a) + __popc(m.b));
                        continue;
                    }
                }
                const uint32_t cnt = (uint32_t)(__popc(m.a) + __popc(m.b));
                if (way & kCountOnly) {
                    rank += cnt;
                    continue;
                }
                unsigned total, j;
                warp_count_prefix(cnt, lane, total, j);
                if (total == 0u)
                    continue;
                const Slots sl = take_slots(now(g_args.rec_count), state.ws, total, lane);
                const uint32_t cell = now(g_it.cell) + (uint32_t)tid;
                const uint32_t off = (uint32_t)(col0 - now(g_it.seg0));
                EdgeRecord *rec = now(g_args.rec);
                const unsigned long long cap = now(g_args.rec_cap);
                write_hits(rec, cap, m.a, cell, off, rank, sl, j);
                write_hits(rec, cap, m.b, cell, off + 32u, rank, sl, j);
            }
        }
        __syncthreads();
        if (tid == 0 && t + 2 < ntiles)
            ring_issue<L>(b, now(g_it.units), c0 + 2 * kTileCols, now(g_it.c_hi));
    }
    const bool live = now(g_it.row0) + tid < now(g_it.n);
    if (live)
        g_args.counts[now(g_it.cell) + (uint32_t)tid] = rank;
    const unsigned hits = __reduce_add_sync(kFull, live ? rank : 0u);
    if (lane == 0 && hits != 0u)
        atomicAdd(g_args.hit_count, (unsigned long long)hits);
    return state;
}

// Local item -> (band, segment): bands are grouped by their first segment g;
// a band of group g owns segments g..nseg-1.  Every group before the last is
// full, so group g starts at item bands_per_seg * (g * nseg - g (g - 1) / 2);
// g is found by bisection.
__device__ __forceinline__ void decode_item(const JobDesc &J, long long local, int &band, int &seg)
{
    // a job has at most 65,536 bands x 256 segments: 32 bits
    const uint32_t li = (uint32_t)local, nseg = (uint32_t)J.nseg, bps = (uint32_t)J.bands_per_seg;
    uint32_t lo = 0, hi = nseg - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (bps * (mid * nseg - mid * (mid - 1) / 2) <= li)
            lo = mid;
        else
            hi = mid - 1;
    }
    const uint32_t q = li - bps * (lo * nseg - lo * (lo - 1) / 2);
    const uint32_t per = nseg - lo;
    band = (int)(lo * bps + q / per);
    seg = (int)(lo + q % per);
}

// The unused rest of each warp's record-slot chunk becomes sentinels.
__device__ __forceinline__ void fill_slot_tails(const WarpSlots &w)
{
    for (unsigned k = threadIdx.x & 31; k < w.left; k += 32) {
        const unsigned long long idx = w.base + k;
        if (idx < g_args.rec_cap)
            *reinterpret_cast<uint2 *>(g_args.rec + idx) = make_uint2(kNoCell, 0u);
    }
}

// The item function of a job's (length, threshold class): level form K = 1
// for every L, K = 2..4 for L > K, delta form W = 2..7 for L > 2 W.
template <int K, int... Ls>
__device__ __forceinline__ void dispatch_levels(const JobDesc *J, int band, int seg, LoopState &st,
                                                std::integer_sequence<int, Ls...>)
{
    constexpr int kFirst = K == 1 ? 1 : K + 1;
    ((J->L == Ls + kFirst ? (void)(st = run_item<LevelForm<Ls + kFirst, K>>(J, band, seg, st)) : void()), ...);
}

template <int W, int... Ls>
__device__ __forceinline__ void dispatch_deltas(const JobDesc *J, int band, int seg, LoopState &st,
                                                std::integer_sequence<int, Ls...>)
{
    constexpr int kFirst = 2 * W + 1;
    ((J->L == Ls + kFirst ? (void)(st = run_item<DeltaForm<Ls + kFirst, W>>(J, band, seg, st)) : void()), ...);
}

// Persistent item loop: the CTA takes (job, band, segment) items of its job
// table from its work counter and runs them.
template <bool kLevels>
__device__ __forceinline__ void pair_loop(const PairArgs &args)
{
    const int tid = threadIdx.x;
    if (tid == 0) {
        g_args = args;
        mbar_init(&g_bar[0], 1);
        mbar_init(&g_bar[1], 1);
        mbar_fence_init();
    }
    __syncthreads();
    LoopState st;
    st.ws.base = 0ull;
    st.ws.left = 0u;
    st.parity = 0u;
    st.turn = 0;
    st.aborted = false;

    // the first item by the CTA's number, the others from the counter, each
    // fetched while the one before it is under way (run_item)
    for (long long item = blockIdx.x; item < args.items; item = g_item[st.turn ^ 1]) {
        const JobDesc *J = args.jobs + find_job_by_item(args.jobs, args.njobs, item);
        int band = 0, seg = 0;
        decode_item(*J, item - J->item_off, band, seg);
#define IG_LEVELS(K)                                                                                      \
    case K:                                                                                               \
        dispatch_levels<K>(J, band, seg, st, std::make_integer_sequence<int, IG_MAX_LEN - (K > 1 ? K : 0)>{}); \
        break;
#define IG_DELTAS(W)                                                                                      \
    case W:                                                                                               \
        dispatch_deltas<W>(J, band, seg, st, std::make_integer_sequence<int, IG_MAX_LEN - 2 * W>{});      \
        break;
        if constexpr (kLevels) {
            switch (J->cls) {
                IG_LEVELS(1)
                IG_LEVELS(2)
                IG_LEVELS(3)
                IG_LEVELS(4)
            }
        } else {
            switch (J->cls) {
                IG_DELTAS(2)
                IG_DELTAS(3)
                IG_DELTAS(4)
                IG_DELTAS(5)
                IG_DELTAS(6)
                IG_DELTAS(7)
            }
        }
#undef IG_LEVELS
#undef IG_DELTAS
        if (st.aborted)
            break;
        __syncthreads();  // the item is done with its shared values, and the next one's number is there
        st.turn ^= 1;     // (the number after it goes to the other place: slow warps may still read this one)
    }
    if (st.aborted && tid == 0)
        ring_drain(st.parity);
    if (args.emit && !st.aborted)
        fill_slot_tails(st.ws);
}

// Level form (editDist <= 5).
__global__ void __launch_bounds__(kBandRows, 3) pair_levels(PairArgs a) { pair_loop<true>(a); }

// Delta form (editDist 6..16).
__global__ void __launch_bounds__(kBandRows, 2) pair_deltas(PairArgs a) { pair_loop<false>(a); }

// Per row: in-place exclusive prefix of its segment counts, and the row
// offsets row_ptr of all rows, in one launch (a row's degree, a scan of the
// degrees over the blocks by decoupled look-back).
//
// A row's cells (one per segment from its band's first segment on, a
// [segment][row] array) are split into kPrefixParts consecutive chunks, each
// taken by its own thread: the threads of a warp hold 32 consecutive rows of
// one chunk, so every access is coalesced, and four times as many loads are
// in flight as with one thread per row (which left the kernel waiting on
// memory with a quarter of the SM's warps).  Phase one sums each chunk, phase
// two rewrites it with prefixes that start at the sum of the chunks before it
// (its cells come back from L2).
// (8 and 16 threads per row measured slower on the headline job: 0.048 and
// 0.084 ms against 0.038 ms, the shorter chunks leaving each thread less to
// overlap.)
//
// One launch where there were five (prefix, three of a scan, job bounds): with
// the memsets and read-backs also folded into the first and last kernels a
// build went from 13 graph nodes to 5, and 2,000 words at L = 12, editDist 4
// from 122 to 100 us, 19,999 at L = 13, editDist 7 from 378 to 346.
//
// Look-back (decoupled look-back: Merrill and Garland, "Single-pass Parallel
// Prefix Scan with Decoupled Look-back", 2016): a block takes its number from a ticket, so every block before it
// is already running; it publishes its own degree sum, then adds up the
// blocks before it from their published words, 32 at a time, until one holds
// a complete prefix, and publishes its own.  A word is the sum in 62 bits
// under two bits saying what it is (0 nothing, 1 the block's own sum, 2 the
// prefix up to and including the block).  The wait is bounded like the pair
// kernels' and ends in the same status.
constexpr int kPrefixParts = 4;
constexpr int kPrefixRows = 256 / kPrefixParts;
__global__ void __launch_bounds__(256) row_offsets(uint32_t *__restrict__ counts, const JobDesc *__restrict__ jobs,
                                                   int njobs, int64_t rows, int64_t *__restrict__ out,
                                                   unsigned long long *__restrict__ words, int *status,
                                                   long long wait_cycles)
{
    __shared__ uint32_t part_sum[kPrefixParts][kPrefixRows];
    __shared__ unsigned long long half_sum, before_sh;
    __shared__ int64_t block_sh;
    if (threadIdx.x == 0)
        block_sh = (int64_t)atomicAdd(words, 1ull);  // the ticket; block b's word is words[1 + b]
    __syncthreads();
    const int64_t block = block_sh;
    const int r = threadIdx.x % kPrefixRows, q = threadIdx.x / kPrefixRows;
    const int64_t gr = block * kPrefixRows + r;
    const bool live = gr < rows;
    uint32_t *p = nullptr;
    int64_t stride = 0;
    int len = 0;
    if (live) {
        const JobDesc &J = jobs[find_job_by_row(jobs, njobs, gr)];
        const int64_t row = gr - J.word_off;
        const int g = (int)(((row / kBandRows) * kBandRows) >> J.seg_shift);
        const int m = max(J.nseg - g, 0);
        const int chunk = (m + kPrefixParts - 1) / kPrefixParts;
        const int s0 = min(q * chunk, m), s1 = min(s0 + chunk, m);
        stride = J.n;
        p = counts + J.count_off + (int64_t)(g + s0) * J.n + row;
        len = s1 - s0;
    }
    uint32_t sum = 0;
    {
        int k = 0;
        for (; k + 8 <= len; k += 8) {
            uint32_t c[8];
#pragma unroll
            for (int t = 0; t < 8; ++t)
                c[t] = p[(int64_t)(k + t) * stride];
#pragma unroll
            for (int t = 0; t < 8; ++t)
                sum += c[t];
        }
        for (; k < len; ++k)
            sum += p[(int64_t)k * stride];
    }
    part_sum[q][r] = sum;
    __syncthreads();
    // warps 0 and 1: the block's rows' degrees and their inclusive sums
    unsigned long long incl = 0ull;
    if (threadIdx.x < kPrefixRows) {
        static_assert(kPrefixRows == 64, "two warps hold the block's rows");
#pragma unroll
        for (int t = 0; t < kPrefixParts; ++t)
            incl += part_sum[t][r];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(kFull, incl, o);
            if ((threadIdx.x & 31) >= o)
                incl += t;
        }
        if (threadIdx.x == 31)
            half_sum = incl;
    }
    __syncthreads();
    if (threadIdx.x >= 32 && threadIdx.x < kPrefixRows)
        incl += half_sum;
    if (threadIdx.x == kPrefixRows - 1)
        *reinterpret_cast<volatile unsigned long long *>(words + 1 + block) = (block == 0 ? kPrefixSum : kOwnSum) | incl;
    if (threadIdx.x >= 32 && threadIdx.x < 64) {  // the warp that holds the block's sum
        unsigned long long before = 0ull;
        const bool ok = look_back(words + 1, block, wait_cycles, status, before);
        if (threadIdx.x == kPrefixRows - 1) {
            if (!ok)
                atomicCAS(status, kStatusOk, kStatusTimeout);
            else if (block > 0)
                *reinterpret_cast<volatile unsigned long long *>(words + 1 + block) = kPrefixSum | (before + incl);
            before_sh = before;
        }
    }
    // meanwhile the cells
    uint32_t acc = 0;
    for (int t = 0; t < q; ++t)
        acc += part_sum[t][r];
    {
        int k = 0;
        for (; k + 8 <= len; k += 8) {
            uint32_t c[8];
#pragma unroll
            for (int t = 0; t < 8; ++t)
                c[t] = p[(int64_t)(k + t) * stride];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                p[(int64_t)(k + t) * stride] = acc;
                acc += c[t];
            }
        }
        for (; k < len; ++k) {
            const uint32_t c = p[(int64_t)k * stride];
            p[(int64_t)k * stride] = acc;
            acc += c;
        }
    }
    __syncthreads();
    if (threadIdx.x < kPrefixRows && live)
        out[gr + 1] = (int64_t)(before_sh + incl);
}

// What a pass reports to the host, written by one block of its last kernel
// straight into page-locked host memory: the four flag words, and row_ptr at
// the job boundaries (out[j] = row_ptr[word_off_j], out[k] = row_ptr[rows]).
struct Report {
    const unsigned long long *flags;
    unsigned long long *host_flags;
    int64_t *host_bounds;
    int64_t rows;
};

__device__ __forceinline__ void report(const Report &to, const int64_t *__restrict__ row_ptr,
                                       const JobDesc *__restrict__ jobs, int njobs)
{
    for (int j = threadIdx.x; j <= njobs; j += blockDim.x)
        to.host_bounds[j] = row_ptr[j < njobs ? jobs[j].word_off : to.rows];
    if (threadIdx.x < 4)
        to.host_flags[threadIdx.x] = to.flags[threadIdx.x];
}

// ---- inclusive scan of int64 in place: block scan, scan of block sums, add ----
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanChunk = kScanThreads * kScanItems;

__device__ __forceinline__ int64_t block_inclusive(int64_t v, int64_t *warp_tot)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t t = __shfl_up_sync(kFull, v, o);
        if (lane >= o)
            v += t;
    }
    if (lane == 31)
        warp_tot[wid] = v;
    __syncthreads();
    if (wid == 0) {
        int64_t w = (lane < kScanThreads / 32) ? warp_tot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t t = __shfl_up_sync(kFull, w, o);
            if (lane >= o)
                w += t;
        }
        if (lane < kScanThreads / 32)
            warp_tot[lane] = w;
    }
    __syncthreads();
    if (wid > 0)
        v += warp_tot[wid - 1];
    return v;
}

__global__ void scan_blocks(int64_t *__restrict__ x, int64_t m, int64_t *__restrict__ block_sums)
{
    __shared__ int64_t warp_tot[kScanThreads / 32];
    const int64_t base = blockIdx.x * (int64_t)kScanChunk + (int64_t)threadIdx.x * kScanItems;
    int64_t v[kScanItems];
    int64_t run = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = (base + k < m) ? x[base + k] : 0;
        run += v[k];
        v[k] = run;
    }
    const int64_t incl = block_inclusive(run, warp_tot);
    const int64_t excl = incl - run;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
        if (base + k < m)
            x[base + k] = v[k] + excl;
    if (threadIdx.x == kScanThreads - 1)
        block_sums[blockIdx.x] = incl;
}

// Exclusive scan of the block sums, one block, sequential over chunks.
__global__ void scan_sums(int64_t *__restrict__ s, int64_t nb)
{
    __shared__ int64_t warp_tot[kScanThreads / 32];
    __shared__ int64_t carry;
    if (threadIdx.x == 0)
        carry = 0;
    __syncthreads();
    for (int64_t off = 0; off < nb; off += kScanThreads) {
        const int64_t i = off + threadIdx.x;
        const int64_t v = (i < nb) ? s[i] : 0;
        const int64_t incl = block_inclusive(v, warp_tot);
        const int64_t c = carry;
        if (i < nb)
            s[i] = c + incl - v;
        __syncthreads();
        if (threadIdx.x == kScanThreads - 1)
            carry = c + incl;
        __syncthreads();
    }
}

__global__ void scan_add(int64_t *__restrict__ x, int64_t m, const int64_t *__restrict__ block_off)
{
    const int64_t base = blockIdx.x * (int64_t)kScanChunk;
    const int64_t add = block_off[blockIdx.x];
    for (int k = threadIdx.x; k < kScanChunk; k += kScanThreads)
        if (base + k < m)
            x[base + k] += add;
}

// Job owning count cell v: the last job with count_off <= v (a job without
// cells shares the next job's count_off and so never wins).
__device__ __forceinline__ int find_job_by_cell(const JobDesc *jobs, int njobs, uint32_t v)
{
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].count_off <= (long long)v)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// cols[row_ptr[row] + prefix[cell] + rank] = column, for every record.  The
// cell gives the job, the segment and the row; the record's high half is the
// column's offset in its segment.  The slot count comes from the pair pass's
// counter on the device (the scatter is queued in the same graph, before the
// host has seen it); a pass whose slots overflowed the record buffer is
// rerun, so it scatters nothing, and so does a pass whose pair kernel
// reported a timeout (its counts and records are incomplete).  Records are
// read once, with the streaming hint (evict first), so that the columns being
// written stay in L2 while their sectors fill; each thread keeps kScatterIlp
// records in flight.  A record whose cell or destination lies outside the
// arrays is skipped (sentinels, and nothing else on a complete pass).
constexpr int kScatterIlp = 8;

__device__ __forceinline__ void scatter_one(uint2 r, const JobDesc *__restrict__ jobs, int njobs,
                                            unsigned long long ncells, const int64_t *__restrict__ row_ptr,
                                            const uint32_t *__restrict__ counts, int32_t *__restrict__ cols,
                                            unsigned long long col_cap)
{
    if (r.x >= ncells)
        return;
    const JobDesc &J = jobs[find_job_by_cell(jobs, njobs, r.x)];
    const uint32_t local = r.x - (uint32_t)J.count_off;
    const uint32_t seg = local / (uint32_t)J.n;
    const uint32_t row = local - seg * (uint32_t)J.n;
    const int64_t pos = row_ptr[J.word_off + row] + (int64_t)counts[r.x] + (int64_t)(r.y & 0xffffu);
    if ((unsigned long long)pos < col_cap)
        cols[pos] = (int32_t)(J.word_off + ((int64_t)seg << J.seg_shift) + (int64_t)(r.y >> 16));
}

__global__ void scatter_records(const EdgeRecord *__restrict__ rec, const unsigned long long *__restrict__ d_slots,
                                const int *__restrict__ status, unsigned long long cap, const JobDesc *__restrict__ jobs,
                                int njobs, unsigned long long ncells, const int64_t *__restrict__ row_ptr,
                                const uint32_t *__restrict__ counts, int32_t *__restrict__ cols,
                                unsigned long long col_cap, Report to)
{
    if (blockIdx.x == 0)
        report(to, row_ptr, jobs, njobs);
    const unsigned long long nrec = *d_slots;
    if (nrec > cap || *status != kStatusOk)
        return;
    const uint2 *r2 = reinterpret_cast<const uint2 *>(rec);
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    for (; i + (kScatterIlp - 1) * stride < nrec; i += kScatterIlp * stride) {
        uint2 r[kScatterIlp];
#pragma unroll
        for (int k = 0; k < kScatterIlp; ++k)
            r[k] = __ldcs(r2 + i + k * stride);
#pragma unroll
        for (int k = 0; k < kScatterIlp; ++k)
            scatter_one(r[k], jobs, njobs, ncells, row_ptr, counts, cols, col_cap);
    }
    for (; i < nrec; i += stride)
        scatter_one(__ldcs(r2 + i), jobs, njobs, ncells, row_ptr, counts, cols, col_cap);
}

// The columns of a dense job's (band, segment) item from its hit words, one
// row per lane: every 256 columns a lane counts its hits, the warp lists them
// row by row in shared memory (13 bits each: lane and column offset) and
// copies the list out, so that a row's run of columns is written by
// neighbouring lanes.  A list too long for the buffer (more than a quarter of
// the pairs) is written by each lane on its own.
//
// Why words and not records: a record costs 16 bytes of traffic and some 45
// instructions per hit (slot handling, a scattered 4-byte store), 17 ps a hit
// on the 33 million of 40,000 words at L = 10, editDist 5; the words cost a
// quarter of a byte per pair test and about 3 ps a hit.  The two meet near one
// hit in 250 pair tests; dense_job takes the words from about one in 128.
constexpr int kListMax = 2048;

__global__ void __launch_bounds__(kBandRows) expand_bits(const uint2 *__restrict__ bits, const JobDesc *__restrict__ jobs,
                                                         int njobs, const unsigned long long *__restrict__ hits,
                                                         const int *__restrict__ status,
                                                         const int64_t *__restrict__ row_ptr,
                                                         const uint32_t *__restrict__ counts, int32_t *__restrict__ cols,
                                                         unsigned long long col_cap, const JobDesc *__restrict__ all_jobs,
                                                         int nall, Report to)
{
    __shared__ uint16_t list[kBandRows / 32][kListMax];
    __shared__ int64_t run[kBandRows / 32][32];  // where list entry 0 would go if it were lane l's
    if (blockIdx.x == 0 && to.host_flags)  // null: scatter_records reports
        report(to, row_ptr, all_jobs, nall);
    if (*hits > col_cap || *status != kStatusOk)
        return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long item = blockIdx.x;
    const JobDesc &J = jobs[find_job_by_item(jobs, njobs, item)];
    int band = 0, seg = 0;
    decode_item(J, item - J.item_off, band, seg);
    const int32_t row = band * kBandRows + threadIdx.x;
    const bool live = row < J.n;
    const int blocks = (J.n + kBandRows - 1) / kBandRows;
    const int per_seg = J.bands_per_seg;
    int64_t at = 0;  // where the row's next column goes
    if (live)
        at = row_ptr[J.word_off + row] + (int64_t)counts[J.count_off + (long long)seg * J.n + row];
    for (int cb = max(seg * per_seg, band); cb < min((seg + 1) * per_seg, blocks); ++cb) {
        const int32_t col0 = cb * kBandRows;
        uint2 w[4];
        int cnt = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            w[q] = make_uint2(0u, 0u);
            if (live && col0 + q * kUnitCols < J.n)
                w[q] = __ldcs(bits + J.bit_off + unit_bits(4ll * cb + q) + row);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            cnt += __popc(w[q].x) + __popc(w[q].y);
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o)
                incl += t;
        }
        const int total = __shfl_sync(kFull, incl, 31);
        if (total == 0)
            continue;
        const int64_t base = J.word_off + col0;
        if (total <= kListMax) {
            int p = incl - cnt;
            run[wid][lane] = at - p;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                uint32_t m = (q & 1) ? w[q >> 1].y : w[q >> 1].x;
                while (m) {
                    list[wid][p++] = (uint16_t)(lane << 8 | (q * 32 + __ffs(m) - 1));
                    m &= m - 1u;
                }
            }
            __syncwarp();
            for (int e = lane; e < total; e += 32) {
                const uint32_t v = list[wid][e];
                cols[run[wid][v >> 8] + e] = (int32_t)(base + (v & 255u));
            }
            __syncwarp();
        } else {
            int64_t p = at;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                uint32_t m = (q & 1) ? w[q >> 1].y : w[q >> 1].x;
                while (m) {
                    cols[p++] = (int32_t)(base + q * 32 + __ffs(m) - 1);
                    m &= m - 1u;
                }
            }
        }
        at += cnt;
    }
}

ig_status ensure(Ctx *ctx, DevBuf &b, size_t bytes, const char *what)
{
    if (b.bytes >= bytes && b.ptr)
        return IG_OK;
    // A buffer that has to grow again grows by at least half: every growth
    // of a workspace costs a stream-ordered free + allocation, and growth of
    // the edge records also a second pair pass.
    size_t want = std::max<size_t>(bytes, 256);
    if (b.ptr) {
        want = std::max(want, b.bytes + b.bytes / 2);
        cudaFreeAsync(b.ptr, ctx->stream);
        b.ptr = nullptr;
        b.bytes = 0;
    }
    cudaError_t e = dev_malloc(ctx, &b.ptr, want, ctx->stream);
    if (e != cudaSuccess && want > bytes) {  // the headroom does not fit: the exact size may
        cudaGetLastError();
        want = std::max<size_t>(bytes, 256);
        e = dev_malloc(ctx, &b.ptr, want, ctx->stream);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        b.ptr = nullptr;
        return set_error(ctx, IG_ERR_OOM, std::string("device allocation failed for ") + what + ": " +
                                              cudaGetErrorString(e));
    }
    b.bytes = want;
    return IG_OK;
}

#define IG_CUDA(call)                                                                                          \
    do {                                                                                                       \
        cudaError_t e_ = (call);                                                                               \
        if (e_ != cudaSuccess)                                                                                 \
            return cuda_error(ctx, e_, #call);                                                                 \
    } while (0)

// Page-locked staging of at least `bytes` (the context stream must be idle:
// a graph in flight may still read the old block).
ig_status ensure_stage(Ctx *ctx, size_t bytes)
{
    if (ctx->stage && ctx->stage_bytes >= bytes)
        return IG_OK;
    const size_t want = std::max<size_t>({bytes, ctx->stage_bytes + ctx->stage_bytes / 2, 4096});
    if (ctx->stage) {
        cudaFreeHost(ctx->stage);
        ctx->stage = nullptr;
        ctx->stage_bytes = 0;
    }
    cudaError_t e = cudaHostAlloc(&ctx->stage, want, cudaHostAllocDefault);
    if (e != cudaSuccess) {
        cudaGetLastError();
        ctx->stage = nullptr;
        return set_error(ctx, IG_ERR_OOM, "page-locked staging allocation failed");
    }
    ctx->stage_bytes = want;
    return IG_OK;
}

// Queues the work of `enqueue` (a callable that queues onto ctx->stream and
// returns the first CUDA error) as one CUDA graph launch: the calls are
// captured, the capture is applied to the context's cached executable graph
// `slot` by cudaGraphExecUpdate when the topology is unchanged (only kernel
// arguments, grids and copy addresses differ between batches) or
// instantiated afresh, and the executable graph is launched on the stream.
// With graphs off, or with per-phase event timing on (events recorded inside
// a capture are not timed), the calls run directly on the stream; so they do
// for good on a context where capturing or instantiating failed.
//
// `sig` lists every pointer, size, grid and scalar argument the calls bake
// into the graph (not the contents of the staging block, which the graph's
// copy reads when it runs); when it equals the one of the cached graph, the
// cached graph is launched as it is, without a capture.
template <class F>
ig_status run_graph(Ctx *ctx, int slot, const std::vector<uint64_t> &sig, const char *what, F &&enqueue)
{
    cudaStream_t st = ctx->stream;
    if (!ctx->use_graphs || ctx->profiling) {
        const cudaError_t e = enqueue();
        return e == cudaSuccess ? IG_OK : cuda_error(ctx, e, what);
    }
    if (ctx->graph_exec[slot] && ctx->graph_sig[slot] == sig) {
        const cudaError_t e = cudaGraphLaunch(ctx->graph_exec[slot], st);
        if (e != cudaSuccess)
            return cuda_error(ctx, e, what);
        ctx->graph_launches++;
        return IG_OK;
    }
    ctx->graph_sig[slot].clear();
    // Nothing captured has run, so when the graph machinery itself fails the
    // context turns graphs off and queues the same calls directly.
    auto direct = [&]() -> ig_status {
        cudaGetLastError();
        ctx->use_graphs = false;
        const cudaError_t de = enqueue();
        return de == cudaSuccess ? IG_OK : cuda_error(ctx, de, what);
    };
    cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess)
        return direct();
    const cudaError_t qe = enqueue();
    cudaGraph_t graph = nullptr;
    e = cudaStreamEndCapture(st, &graph);
    if (qe != cudaSuccess || e != cudaSuccess) {
        if (graph)
            cudaGraphDestroy(graph);
        cudaGetLastError();
        if (qe != cudaSuccess && qe != cudaErrorStreamCaptureUnsupported && qe != cudaErrorStreamCaptureInvalidated)
            return cuda_error(ctx, qe, what);  // a launch error of the calls themselves
        return direct();
    }
    cudaGraphExec_t &exec = ctx->graph_exec[slot];
    if (exec) {
        cudaGraphExecUpdateResultInfo info;
        if (cudaGraphExecUpdate(exec, graph, &info) == cudaSuccess) {
            ctx->graph_updates++;
        } else {
            cudaGetLastError();
            cudaGraphExecDestroy(exec);
            exec = nullptr;
        }
    }
    if (!exec) {
        e = cudaGraphInstantiate(&exec, graph, 0);
        if (e != cudaSuccess) {
            exec = nullptr;
            cudaGraphDestroy(graph);
            return direct();
        }
        ctx->graph_instantiations++;
    }
    cudaGraphDestroy(graph);
    ctx->graph_sig[slot] = sig;
    e = cudaGraphLaunch(exec, st);
    if (e != cudaSuccess)
        return cuda_error(ctx, e, what);
    ctx->graph_launches++;
    return IG_OK;
}

int pair_grid(Ctx *ctx)
{
    if (ctx->pair_grid == 0) {
        int bps = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, pair_deltas, kBandRows, 0);
        cudaGetLastError();
        ctx->pair_grid = std::max(bps, 1) * ctx->sm_count;
        bps = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, pair_levels, kBandRows, 0);
        cudaGetLastError();
        ctx->pair_grid_levels = std::max(bps, 1) * ctx->sm_count;
    }
    return ctx->pair_grid;
}

// Device-side layout of a batch.
struct BatchLayout {
    std::vector<JobDesc> desc;      // every job, in batch order
    std::vector<JobDesc> desc_levels;  // level-form jobs with items, item_off over their own items
    std::vector<JobDesc> desc_deltas;  // the other jobs with items (pair_deltas)
    std::vector<JobDesc> desc_dense;  // dense jobs, item_off over their own items (expand_bits)
    long long items_levels = 0, items_deltas = 0, items_dense = 0;
    long long bits = 0;          // hit-word entries (8 bytes) of the dense jobs
    long long record_pairs = 0;  // pair tests of the jobs that emit records
    long long items = 0;
    long long units = 0;       // column units over all jobs
    long long pairs = 0;       // pair tests over the jobs with items (bounds the edges)
    long long unit_vec = 0;    // uint4 of all unit streams
    long long counts = 0;      // per-(segment, row) cells
    int64_t rows = 0;
};

// Jobs whose pair tests hit often enough for hit words (expand_bits): on
// uniform words the share of pairs with distance < min_ed passes 1/128 between
// min_ed = L/2 - 1 and L/2 for every length (10^6 sampled pairs each: 0.6 and
// 4.2 % at L = 10, 0.2 and 1.7 % at L = 11, 0.7 and 3.7 % at L = 16).  Small
// jobs are bound by launches, which a second kernel would add to.
bool dense_job(const JobSpec &j) { return j.n >= 8192 && j.min_ed >= 1 && j.min_ed >= j.len / 2; }

// Hit-word entries of a job of n words: the triangle of 256 x 256 blocks.
long long job_bits(int32_t n)
{
    const long long blocks = ((long long)n + kBandRows - 1) / kBandRows;
    return unit_bits(4 * blocks);
}

// Hit words take the record buffer's place: up to this much of it is allocated
// for them (126,000 words), more only where the buffer has grown for records.
constexpr size_t kBitsRoom = (size_t)1 << 30;

// Each kernel (level form / delta form) gets items_per_cta[lane form] items
// per CTA of its grid (the work split, 24 unless the autotuner chose
// another), shared among its jobs in proportion to their pair tests.
//
// With `bits_limit` above 0, dense jobs (dense_job) keep hit words instead of
// records as long as all of them fit that many bytes.
bool plan_batch(const std::vector<JobSpec> &jobs, int grid_deltas, int grid_levels, const int (&items_per_cta)[3],
                size_t bits_limit, BatchLayout &out)
{
    long double bits_total = 0;
    for (const JobSpec &j : jobs)
        if (dense_job(j))
            bits_total += (long double)job_bits(j.n);
    const bool use_bits = bits_total > 0 && bits_total * sizeof(uint2) <= (long double)bits_limit;
    long double pairs_total[2] = {0, 0};
    for (const JobSpec &j : jobs)
        pairs_total[slice::test_of(j.len, j.min_ed).levels] += (long double)j.n * (j.n > 0 ? j.n - 1 : 0) / 2;
    const long long grids[2] = {grid_deltas, grid_levels};
    out = BatchLayout();
    for (const JobSpec &j : jobs) {
        JobDesc d{};
        const slice::Test test = slice::test_of(j.len, j.min_ed);
        const int kn = test.levels;
        const long double share = pairs_total[kn] > 0 ? ((long double)j.n * (j.n - 1) / 2) / pairs_total[kn] : 0;
        const long long want = (long long)items_per_cta[lane_form(j.len, j.min_ed)] * grids[kn];
        const PairPlan p = make_plan(j.n, std::max<long long>(1, (long long)(share * want)));
        d.word_off = j.word_off;
        d.n = j.n;
        d.L = test.L;
        d.k = test.k;
        d.cls = test.levels ? test.K : test.W;
        d.seg_shift = p.seg_shift;
        d.nseg = p.nseg;
        d.bands_per_seg = p.bands_per_seg;
        d.nbands = p.nbands;
        d.item_off = out.items;
        d.unit_start = out.units;
        d.unit_off = out.unit_vec;
        d.count_off = out.counts;
        const long long units = ((long long)j.n + kUnitCols - 1) / kUnitCols;
        const long long vec = slice::unit_vec(d.L);
        // n < 2 or min_ed <= 0: no pair can be an edge.  The job gets no items
        // and no segments, so its rows read no count cells (degree 0).
        const bool active = j.n >= 2 && j.min_ed >= 1;
        if (!active)
            d.nseg = 0;
        d.bit_off = -1;
        if (active && use_bits && dense_job(j)) {
            d.bit_off = out.bits;
            out.bits += job_bits(j.n);
        }
        out.items += active ? p.items : 0;
        out.pairs += active ? (long long)j.n * (j.n - 1) / 2 : 0;
        out.units += units;
        out.unit_vec += units * vec;
        out.counts += (long long)d.nseg * j.n;
        out.rows = std::max<int64_t>(out.rows, j.word_off + j.n);
        out.desc.push_back(d);
        if (active && p.items > 0) {  // the kernel of its form takes its items
            JobDesc k = d;
            if (d.bit_off >= 0) {
                k.item_off = out.items_dense;
                out.items_dense += p.items;
                out.desc_dense.push_back(k);
            } else {
                out.record_pairs += (long long)j.n * (j.n - 1) / 2;
            }
            long long &space = kn ? out.items_levels : out.items_deltas;
            k.item_off = space;
            space += p.items;
            (kn ? out.desc_levels : out.desc_deltas).push_back(k);
        }
    }
    return out.counts < (1ll << 32);
}

// Compaction of a build pass: the CSR it fills.
struct CompactOut {
    int64_t *row_ptr = nullptr;  // n + 1
    int32_t *cols = nullptr;     // room for min(record capacity, pair tests) columns
    unsigned long long col_cap = 0;
    int32_t n = 0;
};

// One pass over a planned batch: column units (with the job table, uploaded
// before them when it is long), the pair kernel(s) and, for a build (`out`
// set), the compaction into out's CSR (row offsets from the per-(row, segment)
// counts, records or hit words into columns, job bounds) -- queued as ONE graph
// launch with one host wait at the end.
// *slots = record slots handed out (>= *hits; the pass is complete iff they
// fit the record buffer -- otherwise its CSR is void and the caller grows the
// buffer and reruns), *hits = edges; bounds (build only) = row_ptr at the
// job boundaries.
ig_status run_pass(Ctx *ctx, const uint32_t *d_words, const BatchLayout &B, int grid, const CompactOut *out,
                   unsigned long long *slots, unsigned long long *hits, int64_t *bounds)
{
    cudaStream_t st = ctx->stream;
    ig_status s;
    if ((s = ensure(ctx, ctx->sel, (size_t)B.unit_vec * sizeof(uint4), "column streams")) != IG_OK)
        return s;
    if ((s = ensure(ctx, ctx->counts, (size_t)B.counts * sizeof(uint32_t), "segment counts")) != IG_OK)
        return s;
    if ((s = ensure(ctx, ctx->flags, kFlagWords * sizeof(unsigned long long), "flags")) != IG_OK)
        return s;
    // the scan workspace is sized here: nothing allocates inside a capture
    const int64_t row_blocks = out ? ((int64_t)out->n + kPrefixRows - 1) / kPrefixRows : 0;
    if (out && (s = ensure(ctx, ctx->scan_tmp, (size_t)(row_blocks + 1) * sizeof(unsigned long long),
                           "scan workspace")) != IG_OK)
        return s;
    // job buffer: all jobs | pair_levels jobs | pair_deltas jobs | dense jobs
    const size_t jbytes = B.desc.size() * sizeof(JobDesc);
    const size_t bbytes = (B.desc.size() + 1) * sizeof(int64_t);
    const size_t nbytes = B.desc_levels.size() * sizeof(JobDesc), gbytes = B.desc_deltas.size() * sizeof(JobDesc);
    const size_t dbytes = out ? B.desc_dense.size() * sizeof(JobDesc) : 0;
    const size_t table = jbytes + nbytes + gbytes + dbytes;
    if ((s = ensure(ctx, ctx->jobs, table, "job table")) != IG_OK)
        return s;
    // staging: the job table image | 4 flag words and the job bounds, written by the pass
    const size_t flag_off = (table + 63) & ~size_t(63), bound_off = flag_off + 64;
    if ((s = ensure_stage(ctx, bound_off + bbytes)) != IG_OK)
        return s;
    char *stage = static_cast<char *>(ctx->stage);
    std::memcpy(stage, B.desc.data(), jbytes);
    if (nbytes)
        std::memcpy(stage + jbytes, B.desc_levels.data(), nbytes);
    if (gbytes)
        std::memcpy(stage + jbytes + nbytes, B.desc_deltas.data(), gbytes);
    if (dbytes)
        std::memcpy(stage + jbytes + nbytes + gbytes, B.desc_dense.data(), dbytes);
    unsigned long long *host_flags = reinterpret_cast<unsigned long long *>(stage + flag_off);
    int64_t *host_bounds = reinterpret_cast<int64_t *>(stage + bound_off);
    char *jbase = static_cast<char *>(ctx->jobs.ptr);
    JobDesc *d_jobs = reinterpret_cast<JobDesc *>(jbase);
    const int njobs = (int)B.desc.size();
    unsigned long long *flags = static_cast<unsigned long long *>(ctx->flags.ptr);
    PairArgs a;
    a.units = static_cast<const uint4 *>(ctx->sel.ptr);
    a.words = d_words;
    a.one = 1u;
    a.work = flags + 0;
    a.rec_count = flags + 1;
    a.status = reinterpret_cast<int *>(flags + 2);
    a.hit_count = flags + 3;
    // record buffer: hit words of the dense jobs | edge records
    const size_t bits_bytes = out ? (size_t)B.bits * sizeof(uint2) : 0;
    a.bits = static_cast<uint2 *>(ctx->records.ptr);
    a.rec = reinterpret_cast<EdgeRecord *>(static_cast<char *>(ctx->records.ptr) + bits_bytes);
    a.rec_cap = out ? rec_capacity(ctx) - bits_bytes / sizeof(EdgeRecord) : 0;
    a.counts = static_cast<uint32_t *>(ctx->counts.ptr);
    a.emit = out ? 1 : 0;
    a.wait_cycles = ctx->wait_cycles;
    a.skip_first_copy = ctx->fault_tile_copy ? 1 : 0;
    const int grid_levels = ctx->pair_grid_levels;
    const unsigned prep_grid = (unsigned)((B.units + 7) / 8);  // one warp per unit
    const int n = out ? out->n : 0;
    // scatter grid: enough threads for the slots the pass can hand out
    const unsigned long long cap = a.rec_cap;
    const int sgrid = (int)std::min<unsigned long long>(
        (std::min<unsigned long long>(cap, (unsigned long long)B.record_pairs) + 255) / 256 + 1,
        (unsigned long long)ctx->sm_count * 16);
    InlineTable given;
    given.vecs = table <= sizeof(given.v) && B.units > 0 ? (int)(table / sizeof(uint4)) : 0;
    std::memcpy(given.v, stage, given.vecs * sizeof(uint4));
    std::vector<uint64_t> sig = {
        (uint64_t)(uintptr_t)stage,  table, (uint64_t)(uintptr_t)jbase, (uint64_t)(uintptr_t)d_words,
        (uint64_t)B.units,           (uint64_t)njobs, (uint64_t)(uintptr_t)ctx->sel.ptr,
        (uint64_t)(uintptr_t)flags,  (uint64_t)(uintptr_t)ctx->records.ptr, cap,
        (uint64_t)(uintptr_t)ctx->counts.ptr, (uint64_t)a.emit, (uint64_t)B.items_deltas, (uint64_t)B.items_levels,
        B.desc_levels.size(),           B.desc_deltas.size(), (uint64_t)grid, (uint64_t)grid_levels,
        out ? (uint64_t)(uintptr_t)out->row_ptr : 0, out ? (uint64_t)(uintptr_t)out->cols : 0, (uint64_t)n,
        (uint64_t)sgrid,             (uint64_t)(uintptr_t)ctx->scan_tmp.ptr, (uint64_t)B.counts,
        out ? (uint64_t)out->col_cap : 0, (uint64_t)a.wait_cycles, (uint64_t)a.skip_first_copy,
        (uint64_t)bits_bytes, (uint64_t)B.items_dense, dbytes, (uint64_t)(B.record_pairs > 0)};
    {  // an inline table is an argument too
        const size_t at = sig.size();
        sig.resize(at + given.vecs * 2);
        std::memcpy(sig.data() + at, given.v, given.vecs * sizeof(uint4));
    }
    ctx->fault_tile_copy = false;  // the injected fault is one-shot
    const PassZero zero{flags, out ? out->row_ptr : nullptr,
                        out ? static_cast<unsigned long long *>(ctx->scan_tmp.ptr) : nullptr,
                        out ? (long long)row_blocks + 1 : 0};
    const Report to{flags, host_flags, host_bounds, n};
    int64_t launched = 0;
    s = run_graph(ctx, out ? 0 : 1, sig, out ? "build pass" : "count pass", [&]() -> cudaError_t {
        launched = 0;
        cudaError_t e = cudaSuccess;
        if (given.vecs == 0 && (e = cudaMemcpyAsync(jbase, stage, table, cudaMemcpyHostToDevice, st)) != cudaSuccess)
            return e;
        phase_begin(ctx, IG_PHASE_PREP);
        if (B.units > 0) {
            prep_units<<<prep_grid, 256, 0, st>>>(d_words, d_jobs, njobs, B.units, static_cast<uint4 *>(ctx->sel.ptr),
                                                   zero, given);
            launched++;
        }
        phase_end(ctx, IG_PHASE_PREP);
        if ((e = cudaGetLastError()) != cudaSuccess)
            return e;
        phase_begin(ctx, IG_PHASE_PAIRS);
        PairArgs k = a;
        if (B.items_deltas > 0) {
            k.jobs = reinterpret_cast<const JobDesc *>(jbase + jbytes + nbytes);
            k.njobs = (int)B.desc_deltas.size();
            k.items = B.items_deltas;
            pair_deltas<<<grid, kBandRows, 0, st>>>(k);
            launched++;
            if ((e = cudaGetLastError()) != cudaSuccess)
                return e;
        }
        if (B.items_levels > 0) {
            k.jobs = reinterpret_cast<const JobDesc *>(jbase + jbytes);
            k.njobs = (int)B.desc_levels.size();
            k.items = B.items_levels;
            k.work = flags + 4;
            pair_levels<<<grid_levels, kBandRows, 0, st>>>(k);
            launched++;
            if ((e = cudaGetLastError()) != cudaSuccess)
                return e;
        }
        phase_end(ctx, IG_PHASE_PAIRS);
        if (out) {
            phase_begin(ctx, IG_PHASE_COMPACT);
            phase_begin(ctx, IG_PHASE_PREFIX);
            row_offsets<<<(unsigned)row_blocks, 256, 0, st>>>(static_cast<uint32_t *>(ctx->counts.ptr), d_jobs, njobs, n,
                                                              out->row_ptr, zero.scan_words, a.status, a.wait_cycles);
            launched++;
            if ((e = cudaGetLastError()) != cudaSuccess)
                return e;
            phase_end(ctx, IG_PHASE_PREFIX);
            phase_begin(ctx, IG_PHASE_SCATTER);
            if (B.record_pairs > 0) {
                scatter_records<<<sgrid, 256, 0, st>>>(a.rec, flags + 1, a.status, cap, d_jobs, njobs,
                                                        (unsigned long long)B.counts, out->row_ptr,
                                                        static_cast<const uint32_t *>(ctx->counts.ptr), out->cols,
                                                        out->col_cap, to);
                launched++;
                if ((e = cudaGetLastError()) != cudaSuccess)
                    return e;
            }
            if (B.items_dense > 0) {
                expand_bits<<<(unsigned)B.items_dense, kBandRows, 0, st>>>(
                    a.bits, reinterpret_cast<const JobDesc *>(jbase + jbytes + nbytes + gbytes),
                    (int)B.desc_dense.size(), a.hit_count, a.status, out->row_ptr,
                    static_cast<const uint32_t *>(ctx->counts.ptr), out->cols, out->col_cap, d_jobs, njobs,
                    B.record_pairs > 0 ? Report{} : to);
                launched++;
                if ((e = cudaGetLastError()) != cudaSuccess)
                    return e;
            }
            phase_end(ctx, IG_PHASE_SCATTER);
            phase_end(ctx, IG_PHASE_COMPACT);
            return cudaSuccess;
        }
        return cudaMemcpyAsync(host_flags, flags, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
    });
    ctx->launches += launched;
    if (s != IG_OK)
        return s;
    IG_CUDA(cudaStreamSynchronize(st));
    phase_collect(ctx);
    if ((s = pass_status(ctx, static_cast<int>(host_flags[2] & 0xffffffffu))) != IG_OK)
        return s;
    *slots = host_flags[1];
    *hits = host_flags[3];
    if (bounds)
        std::memcpy(bounds, host_bounds, bbytes);
    return IG_OK;
}

ig_status check_jobs(Ctx *ctx, const std::vector<JobSpec> &jobs)
{
    int64_t rows = 0;
    for (const JobSpec &j : jobs) {
        if (j.n < 0 || j.len < 1 || j.len > IG_MAX_LEN || j.word_off < 0)
            return set_error(ctx, IG_ERR_INPUT, "job: n >= 0 and 1 <= len <= 16 required");
        if (j.n > kMaxJobWords)
            return set_error(ctx, IG_ERR_CAPACITY, "a job holds at most 16,777,215 words");
        rows = std::max<int64_t>(rows, j.word_off + j.n);
    }
    if (rows > (int64_t)INT32_MAX)
        return set_error(ctx, IG_ERR_CAPACITY, "more than 2^31-1 words in one batch");
    return IG_OK;
}

}  // namespace

ig_status inclusive_scan_i64(Ctx *ctx, int64_t *x, int64_t m)
{
    cudaStream_t st = ctx->stream;
    const int64_t nb = (m + kScanChunk - 1) / kScanChunk;
    ig_status s = ensure(ctx, ctx->scan_tmp, (size_t)nb * sizeof(int64_t), "scan workspace");
    if (s != IG_OK)
        return s;
    int64_t *sums = static_cast<int64_t *>(ctx->scan_tmp.ptr);
    scan_blocks<<<(unsigned)nb, kScanThreads, 0, st>>>(x, m, sums);
    scan_sums<<<1, kScanThreads, 0, st>>>(sums, nb);
    scan_add<<<(unsigned)nb, kScanThreads, 0, st>>>(x, m, sums);
    ctx->launches += 3;
    IG_CUDA(cudaGetLastError());
    return IG_OK;
}

ig_status pass_status(Ctx *ctx, int status)
{
    if (status == kStatusTimeout)
        return set_error(ctx, IG_ERR_TIMEOUT, "pair kernel: a staged tile did not arrive within the wait limit");
    if (status == kStatusCopyLost)
        return set_error(ctx, IG_ERR_TIMEOUT,
                         "pair kernel: a staged tile did not arrive within the wait limit, and a copy still in flight "
                         "did not land either");
    return IG_OK;
}

ig_status ensure_staging(Ctx *ctx, size_t bytes) { return ensure_stage(ctx, bytes); }

ig_status ensure_buffer(Ctx *ctx, DevBuf &b, size_t bytes, const char *what) { return ensure(ctx, b, bytes, what); }

size_t workspace_bytes(const Ctx *ctx)
{
    return ctx->sel.bytes + ctx->counts.bytes + ctx->records.bytes + ctx->cols_ws.bytes + ctx->adj_tmp.bytes;
}

void trim_workspaces(Ctx *ctx, size_t keep_bytes)
{
    if (workspace_bytes(ctx) <= keep_bytes)
        return;
    for (DevBuf *b : {&ctx->sel, &ctx->counts, &ctx->records, &ctx->cols_ws, &ctx->adj_tmp}) {
        if (b->ptr)
            cudaFreeAsync(b->ptr, ctx->stream);
        b->ptr = nullptr;
        b->bytes = 0;
    }
    ctx->col_room = 0;
    cudaGetLastError();
}

void phase_begin(Ctx *ctx, int phase)
{
    if (!ctx->profiling)
        return;
    cudaEventRecord(ctx->ev[2 * phase], ctx->stream);
}

void phase_end(Ctx *ctx, int phase)
{
    if (!ctx->profiling)
        return;
    cudaEventRecord(ctx->ev[2 * phase + 1], ctx->stream);
    ctx->phase_pending[phase] = true;
}

void phase_collect(Ctx *ctx)
{
    if (!ctx->profiling)
        return;
    for (int p = 0; p < Ctx::kPhases; ++p) {
        if (!ctx->phase_pending[p])
            continue;
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, ctx->ev[2 * p], ctx->ev[2 * p + 1]) == cudaSuccess) {
            ctx->phase_ms[p] += ms;
            ctx->phase_launches[p] += 1;
        }
        cudaGetLastError();
        ctx->phase_pending[p] = false;
    }
}

PairPlan make_plan(int32_t n, long long target_items)
{
    PairPlan p;
    p.n = n;
    // Segment width: a power of two >= one band, small enough that the job
    // yields about target_items items, large enough that at most 256 segments
    // exist and the per-(row, segment) counts stay under 1 GiB where a
    // segment of at most 2^16 columns allows it (an edge record holds the
    // column offset and the rank in 16 bits each; jobs of up to 2^24 - 1
    // words fit 256 such segments).
    int shift = 8;  // 256 columns
    while (shift < kMaxSegShift && ((int64_t)n + (1ll << shift) - 1) >> shift > 256)
        shift++;
    while (shift < kMaxSegShift && (((int64_t)n + (1ll << shift) - 1) >> shift) * (int64_t)n * 4 > (1ll << 30))
        shift++;
    // Prefer wider segments (fewer per-item overheads) while the target holds.
    for (;;) {
        const int s2 = shift + 1;
        const int64_t nseg2 = ((int64_t)n + (1ll << s2) - 1) >> s2;
        const int64_t nb = ((int64_t)n + kBandRows - 1) / kBandRows;
        const int64_t items2 = nb * (nseg2 + 1) / 2;
        if (s2 > 14 || items2 < target_items)
            break;
        shift = s2;
    }
    p.seg_shift = shift;
    p.nseg = (int)(((int64_t)n + (1ll << shift) - 1) >> shift);
    p.bands_per_seg = (1 << shift) / kBandRows;
    p.nbands = (int)(((int64_t)n + kBandRows - 1) / kBandRows);
    long long items = 0;
    for (int g = 0; g < p.nseg; ++g) {
        const int b_lo = g * p.bands_per_seg;
        const int b_hi = std::min(b_lo + p.bands_per_seg, p.nbands);
        items += (long long)std::max(b_hi - b_lo, 0) * (p.nseg - g);
    }
    p.items = items;
    return p;
}

namespace {

// `general`: by the general pass whatever the jobs (the work split is timed on it).
ig_status count_jobs(Ctx *ctx, const uint32_t *d_words, const std::vector<JobSpec> &jobs, bool general, int64_t *edges)
{
    ig_status s = check_jobs(ctx, jobs);
    if (s != IG_OK)
        return s;
    const int grid = pair_grid(ctx);
    BatchLayout B;
    if (!plan_batch(jobs, grid, ctx->pair_grid_levels, ctx->items_per_cta, 0, B))
        return set_error(ctx, IG_ERR_CAPACITY, "batch too large for one launch");
    if (B.items == 0) {
        *edges = 0;
        return IG_OK;
    }
    unsigned long long slots = 0, hits = 0;
    if (!general && jobs.size() == 1 && prefix_job(jobs[0]))
        s = prefix_pass(ctx, d_words, jobs[0], nullptr, &slots, &hits, nullptr);
    else
        s = run_pass(ctx, d_words, B, grid, nullptr, &slots, &hits, nullptr);
    if (s != IG_OK)
        return s;
    *edges = (int64_t)hits;
    return IG_OK;
}

}  // namespace

ig_status count_batch(Ctx *ctx, const uint32_t *d_words, const std::vector<JobSpec> &jobs, int64_t *edges)
{
    return count_jobs(ctx, d_words, jobs, false, edges);
}

// Work-split autotuner.  The pair kernels walk (256-row band x segment) item
// tiles; items_per_cta sets how many a batch is cut into, and so the segment
// width (256 .. 16,384 columns) of each job's item tiles: wide tiles amortise
// the per-item row setup and tile staging, narrow ones even out the end of the
// persistent launch.  The tuner times the count-only pair pass of `jobs` (all
// of one lane form) with CUDA events on the context's stream for each
// candidate whose plan differs from the ones already timed (best of two runs
// after one warm-up) and keeps the fastest for that lane form.
ig_status autotune(Ctx *ctx, const uint32_t *d_words, const std::vector<JobSpec> &jobs, int *chosen)
{
    static const int kCandidates[] = {6, 12, 24, 48, 96};
    if (jobs.empty())
        return set_error(ctx, IG_ERR_INPUT, "autotune needs a job");
    const int mode = lane_form(jobs[0].len, jobs[0].min_ed);
    for (const JobSpec &j : jobs)
        if (lane_form(j.len, j.min_ed) != mode)
            return set_error(ctx, IG_ERR_INPUT, "autotune jobs must share one lane form");
    ig_status s = check_jobs(ctx, jobs);
    if (s != IG_OK)
        return s;
    const int grid = pair_grid(ctx);
    const int before = ctx->items_per_cta[mode];
    // distinct plans only: candidates that cut the jobs identically are one
    std::vector<int> cands;
    std::vector<std::vector<int>> shifts;
    for (int c : kCandidates) {
        int tune[3] = {ctx->items_per_cta[0], ctx->items_per_cta[1], ctx->items_per_cta[2]};
        tune[mode] = c;
        BatchLayout B;
        if (!plan_batch(jobs, grid, ctx->pair_grid_levels, tune, 0, B))
            return set_error(ctx, IG_ERR_CAPACITY, "batch too large for one launch");
        std::vector<int> sh;
        for (const JobDesc &d : B.desc)
            sh.push_back(d.seg_shift);
        if (std::find(shifts.begin(), shifts.end(), sh) == shifts.end()) {
            shifts.push_back(sh);
            cands.push_back(c);
        }
    }
    int best = before;
    if (cands.size() > 1) {
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
            if (e0)
                cudaEventDestroy(e0);
            return cuda_error(ctx, cudaGetLastError(), "autotune events");
        }
        float best_ms = 1e30f;
        int64_t edges = 0;
        for (size_t k = 0; k < cands.size() && s == IG_OK; ++k) {
            ctx->items_per_cta[mode] = cands[k];
            if (k == 0)
                s = count_jobs(ctx, d_words, jobs, true, &edges);  // warm-up: workspaces grow here
            float ms = 1e30f;
            for (int rep = 0; rep < 2 && s == IG_OK; ++rep) {
                cudaEventRecord(e0, ctx->stream);
                s = count_jobs(ctx, d_words, jobs, true, &edges);
                cudaEventRecord(e1, ctx->stream);
                const cudaError_t e = cudaEventSynchronize(e1);
                float t = 0.f;
                if (e != cudaSuccess || cudaEventElapsedTime(&t, e0, e1) != cudaSuccess)
                    s = cuda_error(ctx, e != cudaSuccess ? e : cudaGetLastError(), "autotune timing");
                ms = std::min(ms, t);
            }
            if (s == IG_OK && ms < best_ms) {
                best_ms = ms;
                best = cands[k];
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    } else if (!cands.empty()) {
        best = before;  // every candidate gives the same plan: nothing to choose
    }
    ctx->items_per_cta[mode] = s == IG_OK ? best : before;
    if (s == IG_OK && cands.size() > 1) {
        ctx->tuned[mode] = true;
        ctx->tune_runs++;
    }
    if (chosen)
        *chosen = ctx->items_per_cta[mode];
    return s;
}

// The classes of thresholds that the work split is kept for, as callers name
// them (IG_LANES_*): editDist 1..4, 5..8 and the rest.
int lane_form(int len, int min_ed)
{
    (void)len;
    return min_ed >= 1 && min_ed <= 4 ? 1 : (min_ed >= 5 && min_ed <= 8 ? 2 : 0);
}

ig_status autotune_jobs(Ctx *ctx, const uint32_t *d_words, const std::vector<JobSpec> &jobs)
{
    // Batches only: their uneven jobs are where the split matters, and a
    // one-job build (often the only one of a process) would pay the timing
    // passes up front; ig_ctx_autotune tunes for single jobs on request.
    if (!ctx->autotune || jobs.size() < 2)
        return IG_OK;
    for (int mode = 0; mode < 3; ++mode) {
        if (ctx->tuned[mode])
            continue;
        std::vector<JobSpec> sub;
        long double pairs = 0;
        size_t largest = 0;
        for (const JobSpec &j : jobs)
            if (j.n > 1 && j.min_ed > 0 && lane_form(j.len, j.min_ed) == mode) {
                sub.push_back(j);
                pairs += (long double)j.n * (j.n - 1) / 2;
                if (j.n > sub[largest].n)
                    largest = sub.size() - 1;
            }
        if (sub.empty())
            continue;
        // Time the real jobs when a pass is short (<= 2^33 pair tests, 2 to 4 ms
        // at editDist 4 and 5); otherwise the first 131,072 words of the
        // largest job stand in for them.
        if (pairs > (long double)(1ull << 33)) {
            JobSpec one = sub[largest];
            one.n = std::min<int32_t>(one.n, 131072);
            sub.assign(1, one);
        }
        ig_status s = autotune(ctx, d_words, sub, nullptr);
        if (s != IG_OK)
            return s;
    }
    return IG_OK;
}

// Edges per word beyond which a prefix build is done over by the general pass.
// prefix_build lets uniform words have 256 at most and filtered ones, up to 1.2
// times as dense, 307; beyond that only words of many near neighbours go, whose
// compaction then does not run: 50,000 words of 60 distinct ones (417 a word)
// would take 1.13 ms for it, the general pass 0.69 for everything; 150,000 of
// 150 (500 a word) 4.7 against 4.0 (k = 2) to 7.6 (k = 4).
constexpr unsigned long long kPrefixMaxDegree = 320;

namespace {

// build_batch with hit words in at most bits_limit bytes; *hit_words: whether
// any job keeps them.
ig_status build_planned(Ctx *ctx, const uint32_t *d_words, const std::vector<JobSpec> &jobs, size_t bits_limit,
                        Graph *g, bool *hit_words)
{
    cudaStream_t st = ctx->stream;
    ig_status s = IG_OK;
    const int grid = pair_grid(ctx);
    BatchLayout B;
    if (!plan_batch(jobs, grid, ctx->pair_grid_levels, ctx->items_per_cta, bits_limit, B))
        return set_error(ctx, IG_ERR_CAPACITY, "batch too large for one launch");
    *hit_words = B.bits > 0;
    const int32_t n = (int32_t)B.rows;
    g->ctx = ctx;
    g->n = n;
    g->jobs = jobs;
    g->job_edge_off.assign(jobs.size() + 1, 0);
    g->job_seg_shift.clear();
    g->job_nseg.clear();
    if (!g->d_row_ptr)
        IG_CUDA(dev_malloc(ctx, (void **)&g->d_row_ptr, ((size_t)n + 1) * sizeof(int64_t), st));
    if (B.items == 0) {
        IG_CUDA(cudaMemsetAsync(g->d_row_ptr, 0, ((size_t)n + 1) * sizeof(int64_t), st));
        IG_CUDA(cudaStreamSynchronize(st));
        g->edges = 0;
        return IG_OK;
    }
    const size_t bits_bytes = (size_t)B.bits * sizeof(uint2);
    const size_t first_records = B.record_pairs > 0 ? (size_t)(1u << 22) * sizeof(EdgeRecord) : 0;
    if (rec_capacity(ctx) == 0 || ctx->records.bytes < bits_bytes) {
        s = ensure(ctx, ctx->records, bits_bytes + first_records, "edge records");
        if (s != IG_OK)
            return s;
    }
    // A lone large sparse job runs its shared prefixes once, unless it turns out
    // to have so many edges that sorting its rows would cost more than that saves.
    bool prefix = jobs.size() == 1 && !dense_job(jobs[0]) && prefix_build(jobs[0]);
    const unsigned long long prefix_most = kPrefixMaxDegree * (unsigned long long)n;
    unsigned long long slots = 0, total = 0;
    for (int attempt = 0;; ++attempt) {
        // columns go to a context workspace with room for every record slot
        // the pass may fill (at most one per pair test), or as many columns as
        // a build on this context has needed, so the compaction runs in the
        // same graph as the pair kernels, before the host has seen the edge
        // count; the graph then gets an exact copy
        const unsigned long long room = std::max(rec_capacity(ctx), ctx->col_room);
        const size_t col_cap = (size_t)std::min<unsigned long long>(room, (unsigned long long)B.pairs);
        if ((s = ensure(ctx, ctx->cols_ws, std::max<size_t>(col_cap, 1) * sizeof(int32_t), "column workspace")) !=
            IG_OK)
            return s;
        CompactOut out;
        out.row_ptr = g->d_row_ptr;
        out.cols = static_cast<int32_t *>(ctx->cols_ws.ptr);
        out.col_cap = ctx->cols_ws.bytes / sizeof(int32_t);
        out.n = n;
        if (prefix) {
            // more edges than it may keep: nothing is compacted
            const PrefixOut po{out.row_ptr, out.cols, std::min<unsigned long long>(out.col_cap, prefix_most)};
            s = prefix_pass(ctx, d_words, jobs[0], &po, &slots, &total, g->job_edge_off.data());
        } else {
            s = run_pass(ctx, d_words, B, grid, &out, &slots, &total, g->job_edge_off.data());
        }
        if (s != IG_OK)
            return s;
        const size_t tails = ((size_t)grid + (size_t)ctx->pair_grid_levels) * (kBandRows / 32) * kSlotChunk;
        if (prefix && total > prefix_most) {
            prefix = false;
            attempt = -1;
            ctx->col_room = std::max(ctx->col_room, total + total / 8);
            const size_t want = (size_t)(total + total / 8) + tails + 1024;
            if ((s = ensure(ctx, ctx->records, want * sizeof(EdgeRecord), "edge records")) != IG_OK)
                return s;
            continue;
        }
        const unsigned long long record_cap = rec_capacity(ctx) - bits_bytes / sizeof(EdgeRecord);
        if (slots <= record_cap && total <= out.col_cap)
            break;
        if (attempt > 0)
            return set_error(ctx, IG_ERR_STATE, "record slots exceeded a buffer sized for them twice");
        ctx->col_room = std::max(ctx->col_room, total + total / 8);
        if (slots > record_cap) {
            // slots of a rerun differ from this pass only by the chunk tails
            // of the warps (scheduling), so leave room for all of them
            const size_t want = (size_t)(slots + slots / 8) + tails + 1024;
            s = ensure(ctx, ctx->records, bits_bytes + want * sizeof(EdgeRecord), "edge records");
            if (s != IG_OK)
                return s;
        }
    }
    g->edges = (int64_t)total;
    g->shared_prefixes = prefix;
    if (!prefix)
        for (const JobDesc &d : B.desc) {
            g->job_seg_shift.push_back(d.seg_shift);
            g->job_nseg.push_back(d.nseg);
        }
    const int njobs = (int)B.desc.size();
    if (g->job_edge_off[(size_t)njobs] != (int64_t)total)
        return set_error(ctx, IG_ERR_STATE, "row offsets disagree with the edge count");
    if ((size_t)total * sizeof(int32_t) * 2 >= ctx->cols_ws.bytes) {
        // the columns fill most of the workspace: the graph takes it over
        // (no copy, no second array of that size) and the next build
        // allocates a new one
        g->d_cols = static_cast<int32_t *>(ctx->cols_ws.ptr);
        ctx->cols_ws.ptr = nullptr;
        ctx->cols_ws.bytes = 0;
        return IG_OK;
    }
    IG_CUDA(dev_malloc(ctx, (void **)&g->d_cols, std::max<size_t>((size_t)total, 1) * sizeof(int32_t), st));
    if (total > 0)
        // in order with everything the library does on the stream; the public
        // builds wait for it
        IG_CUDA(cudaMemcpyAsync(g->d_cols, ctx->cols_ws.ptr, (size_t)total * sizeof(int32_t), cudaMemcpyDeviceToDevice,
                                st));
    return IG_OK;
}

}  // namespace

ig_status build_batch(Ctx *ctx, const uint32_t *d_words, const std::vector<JobSpec> &jobs, Graph *g)
{
    ig_status s = check_jobs(ctx, jobs);
    if (s == IG_OK)
        s = autotune_jobs(ctx, d_words, jobs);
    if (s != IG_OK)
        return s;
    bool hit_words = false;
    s = build_planned(ctx, d_words, jobs, std::max(ctx->records.bytes, kBitsRoom), g, &hit_words);
    if (s != IG_ERR_OOM || !hit_words)
        return s;
    // Hit words take n^2/16 bytes whatever the edges are, and the columns get
    // room to match: where that does not fit, records may.
    for (DevBuf *b : {&ctx->records, &ctx->cols_ws}) {
        if (b->ptr)
            cudaFreeAsync(b->ptr, ctx->stream);
        b->ptr = nullptr;
        b->bytes = 0;
    }
    ctx->col_room = 0;
    IG_CUDA(cudaStreamSynchronize(ctx->stream));
    return build_planned(ctx, d_words, jobs, 0, g, &hit_words);
}

}  // namespace ig
