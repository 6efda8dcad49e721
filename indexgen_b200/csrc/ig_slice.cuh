// Bit-sliced pair test: one row against 32 columns per 32-bit word.
//
// Every word below holds one truth value for 32 columns, so an operation of
// the distance recurrence is a three-input logic operation (LOP3) that serves
// 32 pair tests.  What a thread needs of a column tile is, for row position i
// and column position j, the word "which columns have the row's character x_i
// at j": a lookup in a table of four one-hot words per column position, which
// runs on the load/store pipe beside the logic.
//
// Two forms decide ED(x, y) <= k for words of one length L, both on the
// diagonals |j - i| <= k/2 only: an alignment of equal-length words that
// leaves them costs more than k (Ukkonen).
//
//  * levels (k <= 4): for every diagonal t and every e with |t| <= e <= k-|t|
//    (less than |t| cannot be there, more cannot come back to the end) one
//    word "the prefixes of lengths i and i+t are within e":
//      S[t][e](i) = S[t][e](i-1) & Eq | S[t][e-1](i-1) | S[t+1][e-1](i-1)
//                   | S[t-1][e-1](i)
//    1 or 2 LOP3 each: 2, 6, 12, 20 per row position for k = 1..4, less what
//    is constant at the start or never reaches S[0][k](L) at the end.
//  * deltas (any k): Myers' horizontal and vertical differences, one bit pair
//    per cell of the band:
//      D0 = Eq | Mh | Mv;  Ph' = Mv | ~(D0 | Pv);  Mh' = Pv & D0
//      Pv' = Mh | ~(D0 | Ph);  Mv' = Ph & D0
//    5 LOP3 per cell (3 at the band's ends, where the difference to the cell
//    outside is taken as +1: one more edit along the band's edge, never less
//    than the true distance), and a carry-save sum of the main diagonal's
//    steps, which is the distance.
//
// Counted with the constants of the start folded and what never reaches the
// end left out, the levels take 113 LOP3 for 32 pair tests at L = 12, k = 3
// (3.5 each), 258 at L = 16, k = 4 (8.1) and 80 at L = 15, k = 2 (2.5).  Bound
// by the ALU pipe (64 lanes per clock and SM) except at k = 2, whose 43 table
// words per 32 pair tests fill the shared-memory pipe (128 B per clock and SM)
// first.  Measured on a B200 against the recurrence with one 4- or 8-bit lane
// per pair test that this replaced (17.1, 43.3 and 21.3 operations per pair
// test): builds of 201,601 words at L = 12, k = 3 21.56 -> 4.77 ms; 300,000 at
// L = 16, k = 4 117.5 -> 21.8 ms; 150,001 at L = 15, k = 2 14.59 -> 2.08 ms;
// 19,999 at L = 13, k = 6 (deltas) 0.95 -> 0.54 ms.
#pragma once

#include <cstdint>

// host compilers warn about the pragma
#ifdef __CUDA_ARCH__
#define IG_UNROLL _Pragma("unroll")
#else
#define IG_UNROLL
#endif

namespace ig {
namespace slice {

constexpr int kMaxLevelK = 4;   // thresholds the level form is built for
constexpr int kUnitCols = 64;   // columns per unit: two words, loaded together

// 32 or 64 columns' truth values.
struct Words2 {
    uint32_t a, b;
};

// Unit of 64 columns as the kernels stage it: four one-hot pairs of words per
// position, 32 L bytes.
__host__ __device__ constexpr int unit_vec(int L) { return 2 * L; }  // uint4 per unit
__host__ __device__ constexpr int unit_pos_bytes() { return 32; }

#ifdef __CUDACC__
// A warp writes the unit of the 64 words it holds (wa in columns 0..31, wb in
// 32..63, one per lane; lanes out of range, oka / okb false, match nothing) to
// out: each position's two character bits become two ballots per 32 columns,
// from which lane 4 (j % 8) + c forms character c's words.
__device__ __forceinline__ void write_unit(uint32_t wa, uint32_t wb, bool oka, bool okb, int L, int lane, uint2 *out)
{
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t va = __ballot_sync(kAll, oka), vb = __ballot_sync(kAll, okb);
    const uint32_t clo = (lane & 1) ? kAll : 0u, chi = (lane & 2) ? kAll : 0u;
    for (int j0 = 0; j0 < L; j0 += 8) {
        uint2 mine = make_uint2(0u, 0u);
        for (int j = j0; j < min(j0 + 8, L); ++j) {
            const uint32_t la = __ballot_sync(kAll, (wa >> (2 * j)) & 1u);
            const uint32_t ha = __ballot_sync(kAll, (wa >> (2 * j + 1)) & 1u);
            const uint32_t lb = __ballot_sync(kAll, (wb >> (2 * j)) & 1u);
            const uint32_t hb = __ballot_sync(kAll, (wb >> (2 * j + 1)) & 1u);
            if ((lane >> 2) == j - j0) {
                mine.x = ~((la ^ clo) | (ha ^ chi)) & va;
                mine.y = ~((lb ^ clo) | (hb ^ chi)) & vb;
            }
        }
        if (j0 + (lane >> 2) < L)
            out[4 * j0 + lane] = mine;
    }
}

// Integer multiply-add with an operand the compiler cannot see as a constant,
// so it stays an IMAD on the FMA pipe instead of an add on the ALU pipe (the
// pipe the logic operations saturate).
__device__ __forceinline__ uint32_t imad(uint32_t a, uint32_t b, uint32_t c)
{
    uint32_t d;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
#endif

// (a & m) | b and a | b | c, one operation each: left to itself the compiler
// regroups the terms into more of them (spelled out, k = 2 at L = 15 went from
// 2.07 to 1.94 ms on 150,001 words, k = 3 at L = 16 from 1.67 to 1.60 ms on
// 100,003).
__host__ __device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t m, uint32_t b)
{
#ifdef __CUDA_ARCH__
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(d) : "r"(a), "r"(m), "r"(b));
    return d;
#else
    return (a & m) | b;
#endif
}

__host__ __device__ __forceinline__ uint32_t or3(uint32_t a, uint32_t b, uint32_t c)
{
#ifdef __CUDA_ARCH__
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xfe;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
#else
    return a | b | c;
#endif
}

// (prev & m) | the OR of the `n` first terms; all[] true: prev is all ones.
__host__ __device__ __forceinline__ uint32_t level_step(bool all, uint32_t prev, uint32_t m, int n, uint32_t x,
                                                        uint32_t y, uint32_t z)
{
    if (all)
        return n == 0 ? m : n == 1 ? m | x : n == 2 ? or3(m, x, y) : or3(m, x, y) | z;
    return n == 0 ? prev & m : n == 1 ? and_or(prev, m, x) : n == 2 ? and_or(prev, m, x) | y
                                                                   : or3(and_or(prev, m, x), y, z);
}

// The level words S[t + W][e] of a row's prefix.
template <int K>
using Levels = Words2[2 * (K / 2) + 1][K + 1];

template <int K>
__host__ __device__ __forceinline__ void levels_start(Levels<K> &S)
{
    IG_UNROLL
    for (int t = 0; t < 2 * (K / 2) + 1; ++t)
        IG_UNROLL
        for (int e = 0; e <= K; ++e)
            S[t][e] = Words2{0xffffffffu, 0xffffffffu};
}

// S from the prefix of I0 characters to that of I1.  eq(i, j): the columns
// whose character at j equals the row's at i.
template <int L, int K, int I0, int I1, class Eq>
__host__ __device__ __forceinline__ void levels_advance(const Eq &eq, Levels<K> &S)
{
    constexpr int W = K / 2;
    IG_UNROLL
    for (int i = I0 + 1; i <= I1; ++i) {
        IG_UNROLL
        for (int t = -W; t <= W; ++t) {
            const int j = i + t;
            if (j < 1 || j > L)
                continue;
            const int at = t < 0 ? -t : t;
            const int lower = t - 1 < 0 ? 1 - t : t - 1, upper = t + 1 < 0 ? -t - 1 : t + 1;  // |t - 1|, |t + 1|
            const Words2 m = eq(i - 1, j - 1);
            IG_UNROLL
            for (int e = K; e >= 0; --e) {
                // max(i, j) edits always suffice: those words stay all ones
                if (e < at || e > K - at || e >= (i > j ? i : j))
                    continue;
                // the terms that exist, and whether the word so far is all ones
                const bool all = e >= (i > j ? i : j) - 1;
                const bool sub = e - 1 >= at;
                const bool down = t + 1 <= W && e - 1 >= upper && e - 1 <= K - upper;
                const bool left = t - 1 >= -W && e - 1 >= lower && e - 1 <= K - lower;
                Words2 x{0u, 0u}, y{0u, 0u}, z{0u, 0u};
                int n = 0;
                if (sub) {
                    x = S[t + W][e - 1];
                    n = 1;
                }
                if (down) {
                    (n == 0 ? x : y) = S[t + 1 + W][e - 1];
                    ++n;
                }
                if (left) {
                    (n == 0 ? x : n == 1 ? y : z) = S[t - 1 + W][e - 1];
                    ++n;
                }
                S[t + W][e] = Words2{level_step(all, S[t + W][e].a, m.a, n, x.a, y.a, z.a),
                                     level_step(all, S[t + W][e].b, m.b, n, x.b, y.b, z.b)};
            }
        }
    }
}

// The hits S[0][k](L).  For k = 0 and 1 (K = 1) `k0` is 0 or all ones: hits at
// distance 1 only count when it is set.
template <int L, int K, class Eq>
__host__ __device__ __forceinline__ Words2 levels(const Eq &eq, uint32_t k0)
{
    Levels<K> S;
    levels_start<K>(S);
    levels_advance<L, K, 0, L>(eq, S);
    Words2 r = S[K / 2][K];
    if (K == 1) {
        r.a &= S[K / 2][0].a | k0;
        r.b &= S[K / 2][0].b | k0;
    }
    return r;
}

// Counts of up to 16 one-bit words: p[b] is bit b of the count.
struct Planes {
    uint32_t p[5];
};

// Carry-save counter (a column of full adders per bit weight, as in Wallace's
// multiplier, 1964).  Level l keeps one or two words of weight 2^l; a third
// goes through a full adder, whose carry arrives at the next level.  Which of
// these a word meets depends only on how many arrived before it, so with the
// row loop unrolled it is all known at compile time.
struct Counter {
    Words2 one[5], two[5];
    int arrived[5];

    __host__ __device__ __forceinline__ Counter()
    {
        IG_UNROLL
        for (int l = 0; l < 5; ++l)
            arrived[l] = 0;
    }

    __host__ __device__ __forceinline__ void add(int level, Words2 c)
    {
        bool moving = true;
        IG_UNROLL
        for (int l = 0; l < 5; ++l) {
            if (l >= level && moving) {
                arrived[l] += 1;
                if (arrived[l] == 1) {
                    one[l] = c;
                    moving = false;
                } else if (arrived[l] % 2 == 0) {
                    two[l] = c;
                    moving = false;
                } else {
                    const Words2 x = one[l], y = two[l];
                    one[l].a = x.a ^ y.a ^ c.a;
                    one[l].b = x.b ^ y.b ^ c.b;
                    c.a = (x.a & y.a) | (x.a & c.a) | (y.a & c.a);
                    c.b = (x.b & y.b) | (x.b & c.b) | (y.b & c.b);
                }
            }
        }
    }

    // The count, by half adders from the lowest level up.
    __host__ __device__ __forceinline__ void settle(Planes &da, Planes &db)
    {
        IG_UNROLL
        for (int l = 0; l < 5; ++l) {
            if (arrived[l] == 0) {
                da.p[l] = db.p[l] = 0u;
            } else if (arrived[l] % 2 == 1) {
                da.p[l] = one[l].a;
                db.p[l] = one[l].b;
            } else {
                da.p[l] = one[l].a ^ two[l].a;
                db.p[l] = one[l].b ^ two[l].b;
                add(l + 1, Words2{one[l].a & two[l].a, one[l].b & two[l].b});
            }
        }
    }
};

// The distance in five bit planes, exact where it is at most 2W + 1 and
// otherwise an upper bound greater than that (the band's own distance).
template <int L, int W, class Eq>
__host__ __device__ __forceinline__ void deltas(const Eq &eq, Planes &da, Planes &db)
{
    // horizontal differences of the row above, by diagonal (constant +1 at the top)
    Words2 ph[2 * W + 1], mh[2 * W + 1];
    IG_UNROLL
    for (int t = 0; t <= 2 * W; ++t) {
        ph[t].a = ph[t].b = 0xffffffffu;
        mh[t].a = mh[t].b = 0u;
    }
    Counter steps;  // of the main diagonal
    IG_UNROLL
    for (int i = 1; i <= L; ++i) {
        Words2 pv, mv;  // vertical difference left of the cell
        pv.a = pv.b = 0xffffffffu;
        mv.a = mv.b = 0u;
        Words2 nph[2 * W + 1], nmh[2 * W + 1];
        IG_UNROLL
        for (int t = -W; t <= W; ++t) {
            const int j = i + t;
            nph[t + W].a = nph[t + W].b = 0xffffffffu;
            nmh[t + W].a = nmh[t + W].b = 0u;
            if (j < 1 || j > L)
                continue;
            const Words2 m = eq(i - 1, j - 1);
            // the cell above lies on diagonal t + 1 of the row above; outside
            // the band its difference is +1
            uint32_t Pa = 0xffffffffu, Pb = 0xffffffffu, Ma = 0u, Mb = 0u;
            if (t + 1 <= W) {
                Pa = ph[t + 1 + W].a;
                Pb = ph[t + 1 + W].b;
                Ma = mh[t + 1 + W].a;
                Mb = mh[t + 1 + W].b;
            }
            const uint32_t d0a = m.a | Ma | mv.a, d0b = m.b | Mb | mv.b;
            nph[t + W].a = mv.a | ~(d0a | pv.a);
            nph[t + W].b = mv.b | ~(d0b | pv.b);
            nmh[t + W].a = pv.a & d0a;
            nmh[t + W].b = pv.b & d0b;
            pv.a = Ma | ~(d0a | Pa);
            pv.b = Mb | ~(d0b | Pb);
            mv.a = Pa & d0a;
            mv.b = Pb & d0b;
            if (t == 0)
                steps.add(0, Words2{~d0a, ~d0b});
        }
        IG_UNROLL
        for (int t = 0; t <= 2 * W; ++t) {
            ph[t] = nph[t];
            mh[t] = nmh[t];
        }
    }
    steps.settle(da, db);
}

// The smallest distance among the columns ca | cb (at least one) and the first
// column that has it, planes read from the highest down.
template <int L>
__host__ __device__ __forceinline__ void smallest(const Planes &da, const Planes &db, uint32_t ca, uint32_t cb,
                                                  int &dist, int &col)
{
    dist = 0;
    IG_UNROLL
    for (int b = L < 16 ? 3 : 4; b >= 0; --b) {
        const uint32_t za = ca & ~da.p[b], zb = cb & ~db.p[b];
        const bool some = (za | zb) != 0u;
        ca = some ? za : ca;
        cb = some ? zb : cb;
        dist |= some ? 0 : 1 << b;
    }
#ifdef __CUDA_ARCH__
    col = ca != 0u ? __ffs(ca) - 1 : __ffs(cb) + 31;
#else
    col = ca != 0u ? __builtin_ctz(ca) : 32 + __builtin_ctz(cb);
#endif
}

// Columns whose count is at most k: nk[b] is 0 where bit b of k is set, else
// all ones.
__host__ __device__ __forceinline__ uint32_t at_most(const Planes &d, const uint32_t (&nk)[5])
{
    uint32_t gt = 0u;
    IG_UNROLL
    for (int b = 0; b < 5; ++b)
        gt = (d.p[b] & gt) | (d.p[b] & nk[b]) | (gt & nk[b]);
    return ~gt;
}

// How a job's test runs: the length it is compared at, its threshold and its
// form.  ED <= L always holds, so a threshold of L or more makes every pair a
// hit: such a job runs as length 1 with threshold 1.
struct Test {
    int L, k;     // length and threshold of the form
    int levels;   // 1 level form, 0 delta form
    int K, W;     // level form: threshold class (1..4); delta form: half-width
};

__host__ __device__ inline Test test_of(int len, int min_ed)
{
    Test t;
    t.L = len;
    t.k = min_ed < 1 ? 0 : min_ed - 1;  // below 1 nothing is a hit and the job gets no items
    if (t.k >= len) {
        t.L = 1;
        t.k = 1;
    }
    t.levels = t.k <= kMaxLevelK;
    t.K = t.k < 1 ? 1 : t.k;
    t.W = t.k / 2;
    return t;
}

}  // namespace slice
}  // namespace ig
