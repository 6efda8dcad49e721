// Nearest-centre assignment for random_cluster on sm_100a.
//
// Replaces compute_distance_matrix_kernel + the host argmin of
// src/gpu_cluster.py (:16-193, :239-300), which RandomCluster::fit runs through
// system() (src/clustering/impl/random_cluster/RandomCluster.cpp:42-136): the
// reference fills a dense K x N uint8 distance matrix per 32768-word batch,
// copies it to the host and takes np.argmin over the centres.  Here one kernel
// computes each word's Levenshtein distance to every centre and keeps the
// running minimum in registers; only the N int32 assignments leave the device.
// Ties go to the lowest centre index, as np.argmin's first occurrence does.
//
// Two kernels.  assign_sliced (from 9 to 13 centres on, by length and word
// count): one word per thread against 64 centres per step, bit-sliced
// (ig_slice.cuh), centre tables staged in shared memory, 2,048 per pass.
// assign_kernel (fewer, where most of a word's bits would stand for no centre):
// centres are the Myers patterns (their Peq pools in shared memory), words the
// texts: each thread holds the selector stream of two words (two 16-bit lanes,
// L <= 15) or one (L = 16) in registers and walks all centres with the full
// Myers recurrence of ig_myers.cuh, reading the exact distance at the end.
#include <algorithm>
#include <climits>

#include "ig_internal.h"
#include "ig_myers.cuh"
#include "ig_slice.cuh"

namespace ig {
namespace {

using myers::Unit;
using myers::nib;
using myers::row_pools;

constexpr int kAssignThreads = 256;
constexpr int kCentreChunk = 2048;  // centre pools per shared-memory pass (16 KiB)

// The running minimum of the two-lane form as one key per word: distance in
// bits 26..30, centre index in bits 0..25, so one unsigned min keeps the
// nearest centre and, among equals, the lowest index (np.argmin's first
// occurrence).  The key is formed by two IMADs on the FMA pipe from the two
// popcounts, with the multipliers 2^26 and -2^26 passed in as arguments so
// that they stay multiplies; the ALU pipe, which the recurrence saturates,
// then spends one min per distance instead of an add, a compare and two
// selects.
constexpr int kKeyShift = 26;
constexpr uint32_t kKeyIndexMask = (1u << kKeyShift) - 1u;

template <int L, bool kKeyed>
__global__ void __launch_bounds__(kAssignThreads) assign_kernel(const uint32_t *__restrict__ words, long long n,
                                                               const uint32_t *__restrict__ centres, int k,
                                                               int32_t *__restrict__ out, uint32_t one,
                                                               uint32_t two, uint32_t hi, uint32_t unit,
                                                               uint32_t neg_unit)
{
    __shared__ uint2 pools[kCentreChunk];
    using U = Unit<L>;
    const long long first = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * U::kCols;
    const uint32_t wa = first < n ? words[first] : 0u;
    const uint32_t wb = (U::kTwo && first + 1 < n) ? words[first + 1] : wa;
    // this thread's selector stream, in the column-unit layout of ig_myers.cuh
    uint32_t sel[16];
    if constexpr (U::kTwo) {
#pragma unroll
        for (int p = 0; p < 16; ++p)
            sel[p] = (p < L) ? (nib((wa >> (2 * p)) & 3u) | (nib((wb >> (2 * p)) & 3u) << 8)) : 0u;
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            sel[j] = nib((wa >> (4 * j)) & 3u) | (nib((wa >> (4 * j + 2)) & 3u) << 16);
#pragma unroll
        for (int j = 8; j < 16; ++j)
            sel[j] = 0u;
    }
    int best0 = INT_MAX, best1 = INT_MAX, arg0 = 0, arg1 = 0;
    uint32_t key0 = 0xffffffffu, key1 = 0xffffffffu;  // kKeyed: two-lane form, k <= 2^26
    for (int c0 = 0; c0 < k; c0 += kCentreChunk) {
        const int cn = min(kCentreChunk, k - c0);
        __syncthreads();  // the previous pass is done with the pools
        for (int i = threadIdx.x; i < cn; i += blockDim.x) {
            uint32_t p01, p23;
            row_pools<L>(centres[c0 + i], p01, p23);
            pools[i] = make_uint2(p01, p23);
        }
        __syncthreads();
        for (int i = 0; i < cn; ++i) {
            const uint2 p = pools[i];
            if constexpr (U::kTwo) {
                if constexpr (kKeyed) {
                    uint32_t pv, mv;
                    myers::myers_two_vectors<L>(p.x, p.y, sel, one, two, pv, mv);
                    constexpr uint32_t M0 = (1u << L) - 1u;
                    constexpr uint32_t M1 = M0 << 16;
                    // (L + popc(Pv) - popc(Mv)) << 26 | index, modulo 2^32
                    const uint32_t base = ((uint32_t)L << kKeyShift) + (uint32_t)(c0 + i);
                    const uint32_t k0 = myers::imad((uint32_t)__popc(mv & M0), neg_unit,
                                                    myers::imad((uint32_t)__popc(pv & M0), unit, base));
                    const uint32_t k1 = myers::imad((uint32_t)__popc(mv & M1), neg_unit,
                                                    myers::imad((uint32_t)__popc(pv & M1), unit, base));
                    key0 = min(key0, k0);
                    key1 = min(key1, k1);
                } else {
                    int d0, d1;
                    myers::myers_two_dist<L>(p.x, p.y, sel, one, two, d0, d1);
                    if (d0 < best0) {
                        best0 = d0;
                        arg0 = c0 + i;
                    }
                    if (d1 < best1) {
                        best1 = d1;
                        arg1 = c0 + i;
                    }
                }
            } else {
                uint32_t s8[8];
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    s8[j] = sel[j];
                const int d0 = myers::myers_one_dist<L>(p.x, p.y, s8, one, two, hi);
                if (d0 < best0) {
                    best0 = d0;
                    arg0 = c0 + i;
                }
            }
        }
    }
    if constexpr (kKeyed) {
        arg0 = (int)(key0 & kKeyIndexMask);
        arg1 = (int)(key1 & kKeyIndexMask);
    }
    if (first < n)
        out[first] = arg0;
    if (U::kTwo && first + 1 < n)
        out[first + 1] = arg1;
}

// ---- bit-sliced over the centres ----
//
// The distances to 64 centres come out as bit planes (the delta form on a band
// of half-width W), the nearest among them by one pass over the planes.  A
// band distance of at most 2W + 1 is the true distance and a larger one means
// a truly larger distance, so the nearest centre found is exact, ties
// included, as soon as it is that near; a thread whose nearest is farther goes
// over all centres again with the full matrix (full_nearest).  W is chosen so
// that this happens to fewer than 1 thread in 1,000 on uniform words
// (min_centres below).
//
// ALU-pipe bound: about 31 (W = 3) LOP3 per row position and 32 centres, 14.5
// per distance at L = 14 with 64 centres, against 68.6 operations in
// assign_kernel.  1,000,000 words on a B200, the whole call: L = 14, k = 64
// 278.5 -> 76.5 us; L = 10 / 13 / 16, k = 64 214 / 263 / 638 -> 57 / 74 / 99 us,
// k = 16 69 / 82 / 177 -> 41 / 52 / 68 us.
constexpr int kUnitsPerPass = kCentreChunk / slice::kUnitCols;
__shared__ __align__(16) uint4 g_centres[kUnitsPerPass * slice::unit_vec(IG_MAX_LEN)];  // 16 KiB

template <int L, bool kHalf>
struct CentreEq {
    uint32_t at[L];  // byte offsets in the table
    __device__ __forceinline__ slice::Words2 operator()(int i, int j) const
    {
        const char *p = reinterpret_cast<const char *>(g_centres) + at[i] + j * slice::unit_pos_bytes();
        if constexpr (kHalf)
            return slice::Words2{*reinterpret_cast<const uint32_t *>(p), 0u};
        const uint2 v = *reinterpret_cast<const uint2 *>(p);
        return slice::Words2{v.x, v.y};
    }
};

// One word against a unit (or its first 32 centres) at byte offset `unit` of
// the table; va / vb: its valid centres.
template <int L, int W, bool kHalf>
__device__ __forceinline__ void nearest_in_unit(const uint32_t (&at)[L], uint32_t one, uint32_t unit, uint32_t va,
                                                uint32_t vb, int base, int &best, int &arg)
{
    CentreEq<L, kHalf> eq;
#pragma unroll
    for (int i = 0; i < L; ++i)
        eq.at[i] = slice::imad(at[i], one, unit);
    slice::Planes da, db;
    slice::deltas<L, W>(eq, da, db);
    int dist, col;
    slice::smallest<L>(da, db, va, kHalf ? 0u : vb, dist, col);
    if (dist < best) {
        best = dist;
        arg = base + col;
    }
}

__device__ __forceinline__ uint32_t first_bits(int m) { return m >= 32 ? 0xffffffffu : (1u << m) - 1u; }

// The staged pass's `cn` centres (global index of the first: c0).
template <int L, int W>
__device__ __forceinline__ void nearest_in_pass(const uint32_t (&at)[L], uint32_t one, int c0, int cn, int &best,
                                                int &arg)
{
    constexpr uint32_t kBytes = slice::unit_vec(L) * 16;
    int u = 0;
#pragma unroll 1
    for (; cn - u * slice::kUnitCols > 32; ++u)
        nearest_in_unit<L, W, false>(at, one, (uint32_t)u * kBytes, 0xffffffffu,
                                     first_bits(cn - u * slice::kUnitCols - 32), c0 + u * slice::kUnitCols, best, arg);
    const int rest = cn - u * slice::kUnitCols;
    if (rest > 0)
        nearest_in_unit<L, W, true>(at, one, (uint32_t)u * kBytes, first_bits(rest), 0u, c0 + u * slice::kUnitCols,
                                    best, arg);
}

// The same with the full matrix, 32 centres at a time (rare: kept out of the
// main kernel's registers).
template <int L>
__device__ __noinline__ int2 full_nearest(uint32_t word, uint32_t one, int c0, int cn, int2 so_far)
{
    constexpr uint32_t kBytes = slice::unit_vec(L) * 16;
    uint32_t at[L];
#pragma unroll
    for (int i = 0; i < L; ++i)
        at[i] = ((word >> (2 * i)) & 3u) * 8u;
#pragma unroll 1
    for (int c = 0; c < cn; c += 32)
        nearest_in_unit<L, L - 1, true>(at, one, (uint32_t)(c / slice::kUnitCols) * kBytes + (c & 32 ? 4u : 0u),
                                        first_bits(cn - c), 0u, c0 + c, so_far.x, so_far.y);
    return so_far;
}

// Stages the tables of centres [c0, c0 + cn).
__device__ __forceinline__ void stage_centres(const uint32_t *__restrict__ centres, int c0, int cn, int L)
{
    const int lane = threadIdx.x & 31;
    for (int u = threadIdx.x >> 5; u * slice::kUnitCols < cn; u += kAssignThreads / 32) {
        const int a = u * slice::kUnitCols + lane, b = a + 32;
        slice::write_unit(a < cn ? centres[c0 + a] : 0u, b < cn ? centres[c0 + b] : 0u, a < cn, b < cn, L, lane,
                          reinterpret_cast<uint2 *>(g_centres + u * slice::unit_vec(L)));
    }
}

template <int L, int W>
__global__ void __launch_bounds__(kAssignThreads, 3) assign_sliced(const uint32_t *__restrict__ words, long long n,
                                                                  const uint32_t *__restrict__ centres, int k,
                                                                  int32_t *__restrict__ out, uint32_t one)
{
    const bool staged_once = k <= kCentreChunk;
    if (staged_once) {
        stage_centres(centres, 0, k, L);
        __syncthreads();
    }
    for (long long first = blockIdx.x * (long long)kAssignThreads; first < n;
         first += gridDim.x * (long long)kAssignThreads) {
        const long long i = first + threadIdx.x;
        const uint32_t word = i < n ? words[i] : 0u;
        uint32_t at[L];
#pragma unroll
        for (int q = 0; q < L; ++q)
            at[q] = ((word >> (2 * q)) & 3u) * 8u;
        int best = INT_MAX, arg = 0;
        for (int c0 = 0; c0 < k; c0 += kCentreChunk) {
            const int cn = min(kCentreChunk, k - c0);
            if (!staged_once) {
                __syncthreads();  // the previous pass is done with the tables
                stage_centres(centres, c0, cn, L);
                __syncthreads();
            }
            nearest_in_pass<L, W>(at, one, c0, cn, best, arg);
        }
        if constexpr (2 * W + 1 < L) {
            bool far = best > 2 * W + 1;
            if (staged_once ? __any_sync(0xffffffffu, far) : __syncthreads_or(far)) {
                int2 full = make_int2(INT_MAX, 0);
                for (int c0 = 0; c0 < k; c0 += kCentreChunk) {
                    const int cn = min(kCentreChunk, k - c0);
                    if (!staged_once) {
                        __syncthreads();
                        stage_centres(centres, c0, cn, L);
                        __syncthreads();
                    }
                    full = full_nearest<L>(word, one, c0, cn, full);
                }
                arg = full.y;
            }
        }
        if (i < n)
            out[i] = arg;
    }
}

// Centres needed for a word's nearest to lie within 2W + 1 in all but 1 of
// 1,000 cases (distances of 10^6 uniform word pairs per length): below that a
// wider band is faster than the repeats.  W = 3 covers every distance up to
// L = 7.
//
// A word costs the same for 1 to 32 centres, so below some count assign_kernel
// wins; later for fewer words, whose last wave of persistent blocks is emptier.
// assign_kernel / assign_sliced, us:
//            300,000 words               1,000,000 words
//   L = 10   k = 9 26.3 / 25.4           k = 9 47.9 / 40.0
//   L = 11   k = 9 27.7 / 29.0           k = 9 51.6 / 45.2
//            k = 11 29.4 / 29.0
//   L = 12   k = 9 28.6 / 27.8           k = 9 54.1 / 56.4, k = 10 57.5 / 49.4
//   L = 13   k = 9 28.9 / 29.6           k = 9 55.1 / 53.1
//            k = 10 30.1 / 29.6
//   L = 14   k = 9 29.8 / 33.0           k = 9 58.5 / 62.4
//            k = 11 32.1 / 30.9          k = 11 66.3 / 57.4
//   L = 15   k = 9 30.5 / 33.3           k = 9 61.3 / 63.9
//            k = 12 34.4 / 36.7          k = 12 73.8 / 67.6
//            k = 13 35.7 / 34.2
//   L = 16   k = 9 45.6 / 33.9           k = 9 110 / 67
constexpr long long kManyWords = 1 << 19;

__host__ __device__ constexpr int sliced_from(int L, bool many)
{
    return L == 11 ? (many ? 9 : 11) : L == 12 ? 10 : L == 13 ? (many ? 9 : 10) : L == 14 ? (many ? 10 : 11)
           : L == 15 ? (many ? 12 : 13) : 9;
}

__host__ __device__ constexpr int min_centres(int L, int W)
{
    constexpr int w3[17] = {0, 1, 1, 1, 1, 1, 1, 1, 2, 3, 5, 8, 14, 24, 45, 89, 182};
    constexpr int w4[17] = {0, 1, 1, 1, 1, 1, 1, 1, 1, 1, 2, 2, 3, 5, 7, 11, 17};
    return W == 3 ? w3[L] : W == 4 ? w4[L] : 1;
}

template <int L, int W>
void launch_sliced(Ctx *ctx, const uint32_t *words, long long n, const uint32_t *centres, int k, int32_t *out)
{
    const long long blocks = std::min<long long>((n + kAssignThreads - 1) / kAssignThreads, 3ll * ctx->sm_count);
    assign_sliced<L, W><<<(unsigned)blocks, kAssignThreads, 0, ctx->stream>>>(words, n, centres, k, out, 1u);
}

// The narrowest band whose repeats are rare; lengths whose fewest centres
// always suffice for W = 3 or 4 have no wider variant.
template <int L>
void launch_sliced_len(Ctx *ctx, const uint32_t *words, long long n, const uint32_t *centres, int k, int32_t *out)
{
    if (k >= min_centres(L, 3)) {
        launch_sliced<L, 3>(ctx, words, n, centres, k, out);
        return;
    }
    if constexpr (min_centres(L, 3) > sliced_from(L, true)) {
        if (k >= min_centres(L, 4)) {
            launch_sliced<L, 4>(ctx, words, n, centres, k, out);
            return;
        }
        if constexpr (min_centres(L, 4) > sliced_from(L, true))
            launch_sliced<L, 5>(ctx, words, n, centres, k, out);
    }
}

// The keyed minimum for the two-lane lengths (L <= 15) with at most 2^26
// centres; the compare-and-select form otherwise.
template <int L>
void launch_assign_len(Ctx *ctx, int grid, const uint32_t *words, long long n, const uint32_t *centres, int k,
                       int32_t *out)
{
    const cudaStream_t st = ctx->stream;
    if (k >= sliced_from(L, n >= kManyWords)) {
        launch_sliced_len<L>(ctx, words, n, centres, k, out);
        return;
    }
    constexpr uint32_t unit = 1u << kKeyShift;
    if constexpr (Unit<L>::kTwo) {
        if (k <= (int)kKeyIndexMask + 1) {
            assign_kernel<L, true><<<grid, kAssignThreads, 0, st>>>(words, n, centres, k, out, 1u, 2u, 1u << 16,
                                                                    unit, 0u - unit);
            return;
        }
    }
    assign_kernel<L, false><<<grid, kAssignThreads, 0, st>>>(words, n, centres, k, out, 1u, 2u, 1u << 16, unit,
                                                             0u - unit);
}

template <int... Ls>
void launch_assign(Ctx *ctx, int L, int grid, const uint32_t *words, long long n, const uint32_t *centres, int k,
                   int32_t *out, std::integer_sequence<int, Ls...>)
{
    ((L == Ls + 1 ? launch_assign_len<Ls + 1>(ctx, grid, words, n, centres, k, out) : void()), ...);
}

__global__ void gather_words_kernel(const uint32_t *__restrict__ src, const int32_t *__restrict__ idx, long long n,
                                    uint32_t *__restrict__ dst)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = src[idx[i]];
}

}  // namespace

ig_status gather_words(Ctx *ctx, const uint32_t *d_src, const int32_t *d_idx, int64_t n, uint32_t *d_dst)
{
    if (n == 0)
        return IG_OK;
    const long long blocks = std::min<long long>((n + 255) / 256, (long long)ctx->sm_count * 8);
    gather_words_kernel<<<(int)blocks, 256, 0, ctx->stream>>>(d_src, d_idx, n, d_dst);
    ctx->launches++;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? IG_OK : cuda_error(ctx, e, "gather_words launch");
}

ig_status assign_centers(Ctx *ctx, const uint32_t *d_words, int64_t n, const uint32_t *d_centres, int32_t k, int len,
                         int32_t *d_out)
{
    if (n == 0)
        return IG_OK;
    const int per_thread = len <= 15 ? 2 : 1;
    const long long threads = (n + per_thread - 1) / per_thread;
    const long long grid = (threads + kAssignThreads - 1) / kAssignThreads;
    if (grid > INT32_MAX)
        return set_error(ctx, IG_ERR_CAPACITY, "too many words for one assignment launch");
    launch_assign(ctx, len, (int)grid, d_words, n, d_centres, k, d_out,
                  std::make_integer_sequence<int, IG_MAX_LEN>{});
    ctx->launches++;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return cuda_error(ctx, e, "assign_kernel launch");
    return IG_OK;
}

}  // namespace ig
