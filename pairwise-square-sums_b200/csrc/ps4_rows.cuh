// ps4_rows.cuh -- the divisor pairs of a difference as rows of two short lists: what the extension
// engine (ps4_extend.cu) and the triple extension (ps4_triples.cu) share.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ps4_device.cuh"

namespace ps4 {

constexpr int LCAP = 128;                // divisors per list at most (longer ones take the per-lane walk)
constexpr int FSIDE = 7;                 // odd primes of a number below 2^23 at most

// The odd part of a difference D = m1*m2 is kept factored as two coprime numbers below 2^32 (m1's
// odd primes, with the powers that m2 adds to them, and m2's others; a prime moves to the other side
// where that evens out the divisor counts).  The longer of their divisor lists is the row list x[0..L),
// the other y[0..H), each in mixed-radix order of its primes.  The odd divisor (l, h) is x[l]*y[h], its
// complement x[L-1-l]*y[H-1-h].  With D = 2^E2 * odd, the candidates -- complementary divisor pairs (f,
// g) of equal parity -- are (l, h, d): f = x[l]*y[h] << s, g = the complement << E2-s, with s = d + 1, 0 <= d <
// E2 - 1, for even D and s = 0 for odd D.  In the order l fastest, then h, then d, complements lie at
// mirrored places, so the first half of the sequence visits each pair once: full rows of L
// candidates, and half a row at the end when the number of rows is odd.
struct PairLists {
    uint32_t L, H;                       // divisors of the row list and of the other one
    uint32_t slots;                      // row list: first prime slot | primes << 8, the other << 16
    bool wide;                           // an entry may exceed 32 bits
};

// Whether the product of a lane's n prime powers from slot `first` exceeds 32 bits.
static __device__ __noinline__ bool side_is_wide(const uint32_t (*fp)[32], int lane, uint32_t first, uint32_t n) {
    uint64_t x = 1;
    for (uint32_t i = first; i < first + n; i++)
        for (uint32_t e = fp[i][lane] >> 24; e && x <= 0xFFFFFFFFull; e--) x *= fp[i][lane] & 0xFFFFFFu;
    return x > 0xFFFFFFFFull;
}

// The odd primes of m1 and m2 (p | e << 24, from slots 0 and FSIDE): those of m2 that divide m1 too
// add to m1's exponents.  The slow form, for numbers with more primes than a table entry holds.
// Returns the primes and divisors of each side: na | nb << 8 | L << 16 | H << 40.
static __device__ __noinline__ uint64_t merge_slow(const uint64_t *spfq, uint32_t m1, uint32_t m2, uint32_t (*fp)[32],
                                                   int lane) {
    uint32_t na = 0, nb = 0, L = 1, H = 1;
    while (m1 > 1) {
        const uint64_t t = __ldg(&spfq[m1]);
        fp[na++][lane] = (uint32_t)t;                          // p | e << 24, as the table stores it
        m1 = spf_cof(t);
    }
    while (m2 > 1) {
        const uint64_t t = __ldg(&spfq[m2]);
        const uint32_t x = (uint32_t)t, p = x & 0xFFFFFFu;
        m2 = spf_cof(t);
        uint32_t i = 0;
        while (i < na && (fp[i][lane] & 0xFFFFFFu) != p) i++;
        if (i < na) {
            fp[i][lane] += x & 0xFF000000u;
        } else {
            fp[FSIDE + nb++][lane] = x;
            H *= (x >> 24) + 1;
        }
    }
    for (uint32_t i = 0; i < na; i++) L *= (fp[i][lane] >> 24) + 1;
    return (uint64_t)na | (uint64_t)nb << 8 | (uint64_t)L << 16 | (uint64_t)H << 40;
}

// The two lists of m1 * m2 (odd, m1, m2 < 2^23), fa and fb their table entries: primes into the
// lane's slots of fp (p | e << 24; m1's from slot 0, m2's others from FSIDE).
__device__ __forceinline__ void split_pair(const uint64_t *spfq, uint4 fa, uint4 fb, uint32_t m1, uint32_t m2,
                                           uint32_t (*fp)[32], int lane, PairLists &pl) {
    uint32_t na = 0, nb = 0, L = 1, H = 1, common = 0;
    if ((fa.w | fb.w) >> 31) {                     // more than four primes on a side
        const uint64_t s = merge_slow(spfq, m1, m2, fp, lane);
        na = (uint32_t)s & 0xFFu;
        nb = (uint32_t)(s >> 8) & 0xFFu;
        L = (uint32_t)(s >> 16) & 0xFFFFFFu;
        H = (uint32_t)(s >> 40);
        common = 1;
    } else {
        uint32_t x[4] = {fa.x, fa.y, fa.z, fa.w}, y[4] = {fb.x, fb.y, fb.z, fb.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t e = y[k] & 0xFF000000u;
            bool eq = false;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const bool s = ((x[i] ^ y[k]) & 0xFFFFFFu) == 0;     // two zeros: nothing moves
                x[i] += s ? e : 0u;
                eq |= s;
            }
            common |= eq ? e : 0u;
            y[k] = eq ? 0u : y[k];
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (x[i]) fp[i][lane] = x[i];
            na += x[i] != 0;
            L += L * (x[i] >> 24);
            if (y[i]) fp[FSIDE + nb][lane] = y[i];
            nb += y[i] != 0;
            H += H * (y[i] >> 24);
        }
    }
    // the row list is the longer one; its last prime moves over while that leaves both shorter
    uint32_t sr = 0, so = FSIDE, nr = na, no = nb;
    if (H > L) {
        sr = FSIDE; so = 0; nr = nb; no = na;
        const uint32_t s = L; L = H; H = s;
    }
    pl.wide = false;
    if ((uint64_t)m1 * m2 <= 0xFFFFFFFFull) {      // then no list entry is above 32 bits
        while (nr > 1 && no < FSIDE) {
            const uint32_t x = fp[sr + nr - 1][lane], k = (x >> 24) + 1;
            if (H * k >= L) break;
            fp[so + no++][lane] = x;
            nr--;
            L = (uint32_t)(__fdividef((float)L, (float)k) + 0.5f);   // exact: k divides L < 2^14
            H *= k;
        }
        if (H > L) {
            uint32_t s = L; L = H; H = s;
            s = sr; sr = so; so = s;
            s = nr; nr = no; no = s;
        }
    } else if (common) {
        pl.wide = side_is_wide(fp, lane, 0, na);   // m2's side is a divisor of m2
    }
    pl.L = L;
    pl.H = H;
    pl.slots = sr | nr << 8 | so << 16 | no << 24;
}

// The divisors of the n prime powers from slot q, in mixed-radix order (first prime fastest): prime
// after prime, the list so far is repeated e times, each copy p times the one before.  After the first
// prime two entries at a time, whose loads do not wait for each other's stores.
__device__ __forceinline__ void gen_list(uint32_t *d, const uint32_t (*fp)[32], int lane, uint32_t q, uint32_t n) {
    d[0] = 1;
    if (n == 0) return;
    uint32_t cur = 1;
    {
        const uint32_t x = fp[q][lane], p = x & 0xFFFFFFu, e = x >> 24;
        for (uint32_t v = p; cur <= e; v *= p) d[cur++] = v;
    }
    for (uint32_t i = 1; i < n; i++) {
        const uint32_t x = fp[q + i][lane], p = x & 0xFFFFFFu, add = cur * (x >> 24);
#pragma unroll 1
        for (uint32_t j = 0; j < add; j += 2) {
            const uint32_t a = d[j] * p, b = d[j + 1] * p;
            d[cur + j] = a;
            if (j + 1 < add) d[cur + j + 1] = b;
        }
        cur += add;
    }
}

// Residue masks of a candidate's w = f + g + 32 = 2u + 32.  e + C = u^2 + (C - A) must be a square mod
// 64, 63 and 65 for every remaining member C (s4.c:192-194): one bit test per modulus, against the AND of
// the members' masks q_m[(C - A) mod m].
//  * mod 64: u^2 mod 64 depends on u mod 32, bit w/2 mod 32.
//  * mod 63 and 65: bit w mod 63, and bit (w mod 65) mod 64: w = 0 and 64 mod 65 are 2u = -32 and 32, whose
//    squares are equal, so 65 residues fit 64 bits.
struct VResTabs {
    uint64_t q63[63], q65[65];
    uint32_t q64[64];
};
constexpr bool is_qr_mod(int m, int r) {
    return r < 64 ? ((qr_bits(m) >> r) & 1) != 0 : true;          // r = 64 (m = 65) is 8^2
}
constexpr VResTabs make_vres() {
    VResTabs t{};
    for (int a = 0; a < 64; a++)
        for (int u = 0; u < 32; u++)
            if (is_qr_mod(64, (u * u + a) % 64)) t.q64[a] |= 1u << ((u + 16) % 32);
    for (int a = 0; a < 63; a++)
        for (int x = 0; x < 63; x++) {
            const int u = (x + 31) * 32 % 63;                     // (x - 32) / 2; 1/2 = 32
            if (is_qr_mod(63, (u * u + a) % 63)) t.q63[a] |= 1ull << x;
        }
    for (int a = 0; a < 65; a++)
        for (int x = 0; x < 64; x++) {
            const int u = (x + 33) * 33 % 65;                     // (x - 32) / 2; 1/2 = 33
            if (is_qr_mod(65, (u * u + a) % 65)) t.q65[a] |= 1ull << x;
        }
    return t;
}
__device__ const VResTabs VQ = make_vres();

// x mod 63 and mod 65 for x < 2^26, by the ceilings of 2^32/63 and 2^32/65 (exact there)
__device__ __forceinline__ uint32_t mod63(uint32_t x) { return x - 63u * __umulhi(x, 68174085u); }
__device__ __forceinline__ uint32_t mod65(uint32_t x) { return x - 65u * __umulhi(x, 66076420u); }

// a 4-set's masks for C - A = d, |d| < 2^44
__device__ __forceinline__ void and_masks(int64_t d, uint32_t &m64, uint64_t &m63, uint64_t &m65) {
    const uint64_t x = (uint64_t)(d + (int64_t)(4095ull << 33));  // positive; 4095 = 63 * 65, 2^12 = 1 in both
    const uint32_t r = (uint32_t)(x >> 24) + ((uint32_t)x & 0xFFFFFFu);
    m64 &= __ldg(&VQ.q64[(uint32_t)d & 63u]);
    m63 &= __ldg(&VQ.q63[mod63(r)]);
    m65 &= __ldg(&VQ.q65[mod65(r)]);
}

// One candidate of a row: w = f + g + c = x*fy + y*gy + c, and whether it passes the filters (bit 0).  c is 32
// with a tag from bit 58 up, which the sum (below 2^46) does not reach: an entry for the queue as it is.
// The filters' index is w folded at 24 bits, lo - (lo >> 24)(2^24 - 1) + 256 hi (2^24 = 2^12 = 1 mod 63 and 65), in
// multiplications, which have a pipe to themselves, and modulo 2^32, where the tag times 256 vanishes.
__device__ __forceinline__ uint32_t candidate(uint32_t x, uint32_t y, uint64_t fy, uint64_t gy, uint64_t c, uint32_t m64,
                                              uint64_t m63, uint64_t m65, uint64_t &w) {
    const uint64_t s = (uint64_t)y * (uint32_t)gy + ((uint64_t)x * (uint32_t)fy + c);
    const uint32_t lo = (uint32_t)s, hi = y * (uint32_t)(gy >> 32) + (x * (uint32_t)(fy >> 32) + (uint32_t)(s >> 32));
    w = (uint64_t)hi << 32 | lo;
    const uint32_t z = (lo >> 24) * (1u - (1u << 24)) + (hi * 256u + lo);        // below 2^25
    return __funnelshift_r(m64, m64, lo >> 1) & (uint32_t)(m63 >> mod63(z)) & (uint32_t)(m65 >> (mod65(z) & 63u));
}
constexpr uint64_t W_SUM = (1ull << 58) - 1;                 // f + g + 32 of an entry

// Whether n = u^2 + d is a square; n > 0, u < 2^44, |d| < 2^44, n's low 64 bits given.  If n = s^2
// then s < 2^45; the double of n is one rounding off (2^-53), and two Newton steps from the single-precision
// reciprocal root (relative error e < 2^-22) leave 1.5 e^2, then e times that, plus roundings: below 2^-50,
// so the root is less than 1/4 off and rounds to s.  A number r that passes r^2 = n mod 2^64 for r
// within 1/2 of sqrt(n) has |r^2 - n| <= sqrt(n) + 1 < 2^46, so r^2 = n.  Hence the result is exact.
__device__ __forceinline__ bool is_square_near(uint64_t u, int64_t d, uint64_t n_lo) {
    const double two52 = 4503599627370496.0, b = 6755399441055744.0;             // 2^52, 1.5 * 2^52
    const double ud = __longlong_as_double((long long)(u | 0x4330000000000000ull)) - two52;
    const double dd = __longlong_as_double(0x4338000000000000ll + d) - b;
    const double x = fma(ud, ud, dd);
    float yf;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"((float)x));
    const double y = (double)yf, h = 0.5 * y;
    double s = x * y;
    s = fma(fma(-s, s, x), h, s);
    s = fma(fma(-s, s, x), h, s);
    const uint64_t r = ((uint64_t)__double_as_longlong(s + b) & 0xFFFFFFFFFFFFFull) ^ 0x8000000000000ull;
    return r * r == n_lo;
}

// a warp's exclusive prefix of n, and its total
__device__ __forceinline__ uint32_t warp_prefix(uint32_t n, int lane, uint32_t &total) {
    uint32_t i = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, i, o);
        if (lane >= o) i += y;
    }
    total = __shfl_sync(0xffffffffu, i, 31);
    return i - n;
}

// The rows of a warp's 4-sets (or triples), one per lane with `rows` of them, row list L long: longest
// first, so that the 32 rows of a turn are about equally long.
struct RowPlan {
    uint32_t start, lane_of, total;      // in rank order: first row of a job, the job's lane; all rows
};
__device__ __forceinline__ void plan_rows(uint32_t rows, uint32_t L, uint8_t *order, int lane, RowPlan &pl) {
    const unsigned FULL = 0xffffffffu;
    // each lane's rank by (length, lane), then the rows' prefix in rank order
    uint32_t rank = 0;
    const uint32_t key = rows ? min(L, 31u) : 0u;
    unsigned eq = FULL;
#pragma unroll
    for (int b = 4; b >= 0; b--) {
        const unsigned m = __ballot_sync(FULL, key >> b & 1u);
        if (key >> b & 1u) eq &= m;
        else { rank += __popc(eq & m); eq &= ~m; }
    }
    rank += __popc(eq & ((1u << lane) - 1u));
    order[rank] = (uint8_t)lane;
    __syncwarp();                                            // lists, records and order written
    pl.lane_of = order[lane];
    const uint32_t n = __shfl_sync(FULL, rows, pl.lane_of);
    pl.start = warp_prefix(n, lane, pl.total);
    if (!n) pl.start = 0xFFFFFFFFu;                          // no row: after every row
}

// The lane whose job has row g0 + lane, and the row's number r within the job: the last job (in rank
// order) that starts at or before it; starts within these 32 rows as a bit mask.
__device__ __forceinline__ uint32_t row_job(const RowPlan &pl, uint32_t g0, int lane, uint32_t &r) {
    const unsigned FULL = 0xffffffffu;
    const uint32_t rel0 = pl.start - g0;
    const unsigned before = __ballot_sync(FULL, pl.start < g0);
    const unsigned starts = __reduce_or_sync(FULL, rel0 < 32u ? 1u << rel0 : 0u);
    const int o = __popc(before) + __popc(starts & (0xFFFFFFFFu >> (31 - lane))) - 1;
    r = g0 + lane - __shfl_sync(FULL, pl.start, o);
    return __shfl_sync(FULL, pl.lane_of, o);
}

struct Row {
    uint64_t fy, gy;                     // f = x[l] * fy, g = x[L-1-l] * gy
    const uint32_t *xf, *xg;             // x[0], x[L-1]
    int len;                             // candidates (0 for a lane without a row)
};
// Row r = (h, d), h fastest, of a job with lists at `geo`'s place of dbuf.  (r + 1/2) / H is 1/(2H) >= 2^-9
// from an integer, and below R/2 + 1 < 32: far more than the division's error (2^-21 relative).
__device__ __forceinline__ void row_start(uint32_t geo, uint32_t r, bool live, const uint32_t *dbuf, Row &row) {
    const uint32_t L = geo & 0xFFu, H = geo >> 8 & 0xFFu, E2 = geo >> 16 & 0x3Fu, x0 = geo >> 22;
    const uint32_t d = (uint32_t)__fdividef((float)r + 0.5f, (float)H), h = r - d * H;
    const uint32_t sf = E2 ? d + 1 : 0, sg = E2 - sf;
    const uint32_t full = H * (E2 ? E2 - 1 : 1) >> 1;        // full rows, then half a one
    row.len = live ? (int)(r < full ? L : L >> 1) : 0;
    row.fy = live ? (uint64_t)dbuf[x0 + L + h] << sf : 0;
    row.gy = live ? (uint64_t)dbuf[x0 + L + H - 1 - h] << sg : 0;
    // a lane past the end of its row reads on, within the warp's area, and passes nothing
    row.xf = dbuf + (live ? x0 : 0);
    row.xg = dbuf + (live ? x0 + L - 1 : 0);
}

}  // namespace ps4
