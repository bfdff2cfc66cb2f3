// ps4_triples.cu -- batched triple extension: for each square-sum triple {a,b,c}, every d with
// 0 < d <= dmax, d not in the triple, and d+a, d+b, d+c all squares.
//
// The reference has no function for this query; it is its extension step (exhaustive/s4.c:160-207)
// applied to three members instead of four: with A > B two members and C the third,
// e + A = u^2 and e + B = w^2 give (u-w)(u+w) = A - B = D, and D = r_AC^2 - r_BC^2 =
// (r_AC - r_BC)(r_AC + r_BC) factors through the smallest-prime-factor table.  Every pair of
// complementary divisors f, g of equal parity gives u = (f+g)/2 and e = u^2 - A; e + B is then
// a square by construction and e + C is tested exactly.  The pair of members to extend by is
// the one with the fewest estimated divisors, as s4.c:163-171 chooses it.
//
// One triple per lane (fewer lanes per warp when there are few triples): the lane checks it, picks the
// pair and factors its difference; the warp then walks the candidates of all its triples as rows of
// two short divisor lists, 32 rows at a time (ps4_rows.cuh), as the extension engine does.  A triple has
// about ten candidates, so a warp per triple left most lanes idle and repeated the factoring 32 times:
// 1e5 triples (x, y, z below 1e5, d <= 1e12) took 201 us, now 29 us; 50 triples 14.5 us, now 11.8.

#include <cuda_runtime.h>
#include <stdint.h>

#include "ps4_device.cuh"
#include "ps4_rows.cuh"

namespace ps4 {

constexpr int TBS = 128;                 // threads per CTA of the triple kernel
constexpr int TDCAP = 640;               // divisor-list entries per warp (u32)

struct __align__(16) TJob {              // one lane's triple: d = u^2 - A
    uint64_t m63, m65;                   // residue masks of f + g + 32 for the third member
    uint32_t m64, geo;                   // geo: L | H << 8 | E2 << 16 | list place << 22
    uint64_t A, B, C;
    uint64_t uA, umax;                   // u <= uA: d <= 0; u > umax: d > dmax
    uint32_t item, nsq;                  // index of the triple; its square tests
};

struct TriWarp {
    TJob job[32];
    uint32_t dbuf[TDCAP];                // read up to LCAP entries past a list's ends (see the engine)
    uint32_t fp[2 * FSIDE][32];
    uint8_t order[32];
};
static_assert(TDCAP <= 1024 && sizeof(TJob) * 32 >= 4 * LCAP && 4 * 32 * 2 * FSIDE >= 4 * LCAP, "as the engine's");

// d = u^2 - A of lane jl's triple, 0 < d <= dmax and a filtered candidate: the exact test (s4.c:197-203)
__device__ __forceinline__ bool tri_test(const TriArgs &t, const TJob &j, uint64_t u) {
    const uint64_t e = u * u - j.A;                               // 0 < e <= dmax <= 2^62
    if (e == j.A || e == j.B || e == j.C) return false;
    const int64_t d = (int64_t)j.C - (int64_t)j.A;
    if (is_square_near(u, d, u * u + (uint64_t)d)) {
        const unsigned long long slot = atomicAdd(t.n_out, 1ull);
        if (slot < t.out_cap) {
            ps4_tri_ext rec;
            rec.d = e; rec.item = t.item_base + j.item; rec.reserved = 0;
            t.out[slot] = rec;
        }
    }
    return true;
}

// A triple whose lists the buffers cannot hold (a list of more than LCAP divisors, or an entry above 32
// bits): one lane walks its divisors with an odometer.  Returns its square tests.
static __device__ __noinline__ uint32_t tri_walk(const TriArgs &t, const TJob &j, uint32_t m1, uint32_t m2) {
    uint32_t pr[MAXP], nsq = 0;
    uint8_t ex[MAXP], dig[MAXP];
    int np = 0;
    factor_merge(t.spfq, m1, pr, ex, np);
    factor_merge(t.spfq, m2, pr, ex, np);
    const bool has2 = np > 0 && pr[0] == 2;                       // D even => both factors even, 4 | D
    const int E2 = has2 ? ex[0] : 0, j0 = has2 ? 1 : 0;
    uint64_t qinv[MAXP], ndo = 1, fo = 1, go = 1;
    for (int i = j0; i < np; i++) {
        qinv[i] = inv64(pr[i]);
        for (int e = 0; e < ex[i]; e++) go *= pr[i];
        ndo *= (uint64_t)ex[i] + 1;
        dig[i] = 0;
    }
    const int dlo = has2 ? 1 : 0, dhi = has2 ? E2 - 1 : 0;
    uint32_t m64 = j.m64;
    for (uint64_t todd = 0; 2 * todd + 1 <= ndo; todd++) {        // todd <= its complement
        for (int d2 = dlo; d2 <= dhi; d2++) {
            if (2 * todd + 1 == ndo && 2 * d2 >= E2) break;       // self-complementary half already seen
            const uint64_t v = (fo << d2) + (go << (E2 - d2)), u = v >> 1;
            if (u <= j.uA || u > j.umax) continue;
            const uint64_t w = v + 32;
            const uint32_t z = (uint32_t)(w >> 24) + ((uint32_t)w & 0xFFFFFFu);
            if (__funnelshift_r(m64, m64, (uint32_t)w >> 1) & (uint32_t)(j.m63 >> mod63(z)) &
                (uint32_t)(j.m65 >> (mod65(z) & 63u)) & 1u)
                nsq += tri_test(t, j, u);
        }
        for (int i = j0; i < np; i++) {                           // odometer over the odd primes
            if (dig[i] < ex[i]) { dig[i]++; fo *= pr[i]; go *= qinv[i]; break; }
            for (int e = 0; e < dig[i]; e++) { fo *= qinv[i]; go *= pr[i]; }
            dig[i] = 0;
        }
    }
    return nsq;
}

__global__ void __launch_bounds__(TBS) extend_triples_kernel(const __grid_constant__ TriArgs t) {
    __shared__ TriWarp area[TBS / 32];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    TriWarp *w = &area[threadIdx.x >> 5];
    const uint64_t nwarps = ((uint64_t)gridDim.x * TBS) >> 5, warp = ((uint64_t)blockIdx.x * TBS + threadIdx.x) >> 5;
    const uint32_t per = (uint32_t)min((t.n + nwarps - 1) / nwarps, (uint64_t)32);      // triples per warp and round
    ull cand = 0, nsqrt = 0;
    for (uint64_t i0 = warp * per; i0 < t.n; i0 += nwarps * per) {                       // warp-uniform
        const uint64_t i = i0 + lane;
        TJob &E = w->job[lane];
        bool pending = false;
        PairLists pl;
        pl.L = pl.H = pl.slots = 0;
        uint32_t rows = 0;
        ull tcand = 0;
        if ((uint32_t)lane < per && i < t.n) {
            uint64_t m[3] = {t.abc[3 * i], t.abc[3 * i + 1], t.abc[3 * i + 2]};
            if (m[0] > m[1]) { const uint64_t s = m[0]; m[0] = m[1]; m[1] = s; }
            if (m[1] > m[2]) { const uint64_t s = m[1]; m[1] = m[2]; m[2] = s; }
            if (m[0] > m[1]) { const uint64_t s = m[0]; m[0] = m[1]; m[1] = s; }
            // m[0] < m[1] < m[2] from here on, or the triple is rejected
            int st = TRI_OK;
            uint64_t r01 = 0, r02 = 0, r12 = 0;
            if (m[0] == 0 || m[0] == m[1] || m[1] == m[2]) {
                st = TRI_INVALID;
            } else if (m[2] >= (1ull << 44)) {
                st = TRI_RANGE;
            } else {
                r01 = isqrt64(m[0] + m[1]); r02 = isqrt64(m[0] + m[2]); r12 = isqrt64(m[1] + m[2]);
                if (r01 * r01 != m[0] + m[1] || r02 * r02 != m[0] + m[2] || r12 * r12 != m[1] + m[2]) st = TRI_INVALID;
                else if (r12 + r02 >= t.tab_n) st = TRI_RANGE;
            }
            t.state[i] = (uint8_t)st;
            if (st != TRI_OK && t.cand_per) { t.cand_per[i] = 0; t.sqrt_per[i] = 0; }
            if (st == TRI_OK) {
                // the three differences A - B with third member C; roots ra = r_AC > rb = r_BC
                uint32_t ra = 0, rb = 0, best = 0xFFFFFFFFu;
                uint64_t A = 0, B = 0, C = 0;
                auto pair = [&](uint64_t a, uint64_t b, uint64_t c, uint32_t x, uint32_t y) {
                    const uint32_t est = (uint32_t)__ldg(&t.ndiv[x - y]) * __ldg(&t.ndiv[x + y]);
                    if (est < best) { best = est; A = a; B = b; C = c; ra = x; rb = y; }
                };
                pair(m[2], m[1], m[0], (uint32_t)r02, (uint32_t)r01);
                pair(m[2], m[0], m[1], (uint32_t)r12, (uint32_t)r01);
                pair(m[1], m[0], m[2], (uint32_t)r12, (uint32_t)r02);
                uint32_t m1 = ra - rb, m2 = ra + rb, E2 = 0;
                if (!(m1 & 1)) {                                  // D even => both factors even
                    const uint32_t z1 = (uint32_t)__ffs((int)m1) - 1, z2 = (uint32_t)__ffs((int)m2) - 1;
                    E2 = z1 + z2;
                    m1 >>= z1;
                    m2 >>= z2;
                }
                const uint4 fa = __ldg(&t.fac[m1 >> 1]), fb = __ldg(&t.fac[m2 >> 1]);
                E.A = A; E.B = B; E.C = C;
                E.uA = isqrt64(A);
                E.umax = isqrt64(t.dmax + A);                     // dmax + A < 2^63
                E.item = (uint32_t)i;
                E.nsq = 0;
                uint32_t m64 = 0xFFFFFFFFu;
                uint64_t m63 = ~0ull, m65 = ~0ull;
                and_masks((int64_t)C - (int64_t)A, m64, m63, m65);
                E.m64 = m64; E.m63 = m63; E.m65 = m65;
                split_pair(t.spfq, fa, fb, m1, m2, w->fp, lane, pl);
                const uint32_t R = E2 ? E2 - 1 : 1;               // 2-exponents of f: 1 .. E2-1, or 0
                // same-parity complementary pairs f < g, the reference's ext_cand (s4.c:191)
                tcand = (ull)pl.L * pl.H * R >> 1;
                cand += tcand;
                rows = (pl.H * R + (pl.L > 1 ? 1u : 0u)) >> 1;
                E.geo = pl.L | pl.H << 8 | E2 << 16;
                pending = true;
                if (pl.wide || pl.L > (uint32_t)LCAP) {           // rare
                    E.nsq = tri_walk(t, E, ra - rb, ra + rb);
                    rows = 0;
                }
            }
        }
        // rounds until every lane's lists have had room (one, nearly always)
        bool waiting = rows != 0;
        while (__any_sync(FULL, waiting)) {
            uint32_t total;
            const uint32_t want = waiting ? pl.L + pl.H : 0;
            const uint32_t base = warp_prefix(want, lane, total);
            const bool fits = waiting && base + want <= (uint32_t)TDCAP;   // the first one always does
            if (fits) {
                E.geo |= base << 22;
                gen_list(w->dbuf + base, w->fp, lane, pl.slots & 0xFFu, pl.slots >> 8 & 0xFFu);
                gen_list(w->dbuf + base + pl.L, w->fp, lane, pl.slots >> 16 & 0xFFu, pl.slots >> 24);
            }
            RowPlan plan;
            plan_rows(fits ? rows : 0, pl.L, w->order, lane, plan);
            for (uint32_t g0 = 0; g0 < plan.total; g0 += 32) {
                uint32_t r;
                const uint32_t jl = row_job(plan, g0, lane, r);
                const TJob &j = w->job[jl];
                Row row;
                row_start(j.geo, r, g0 + lane < plan.total, w->dbuf, row);
                const uint64_t m63 = j.m63, m65 = j.m65, uA = j.uA, umax = j.umax;
                const uint32_t m64 = j.m64;
                const int turns = (int)__reduce_max_sync(FULL, (unsigned)row.len);
                for (int l = 0; l < turns; l++) {
                    uint64_t v;
                    const uint32_t p = candidate(*row.xf, *row.xg, row.fy, row.gy, 32u, m64, m63, m65, v);
                    row.xf++;
                    row.xg--;
                    const uint64_t u = (v - 32) >> 1;
                    if (l < row.len && (p & 1u) && u > uA && u <= umax && tri_test(t, j, u))
                        atomicAdd(&w->job[jl].nsq, 1u);
                }
            }
            __syncwarp();
            if (fits) waiting = false;
        }
        if (pending) {
            nsqrt += E.nsq;
            if (t.cand_per) { t.cand_per[i] = tcand; t.sqrt_per[i] = E.nsq; }            // per triple (serving)
        }
        __syncwarp();
    }
    cand = warp_sum(cand);
    nsqrt = warp_sum(nsqrt);
    if (lane == 0) {
        if (cand) atomicAdd(t.n_cand, cand);
        if (nsqrt) atomicAdd(t.n_sqrt, nsqrt);
    }
}

int launch_triples(const TriArgs &t, void *stream) {
    if (t.n == 0) return 0;
    // a warp per triple up to the device's residency (8 CTAs per SM), then more triples per warp
    const uint64_t want = (t.n + (TBS / 32) - 1) / (TBS / 32);
    const int grid = (int)(want < 1184 ? want : 1184);
    extend_triples_kernel<<<grid, TBS, 0, (cudaStream_t)stream>>>(t);
    return (int)cudaGetLastError();
}

}  // namespace ps4
