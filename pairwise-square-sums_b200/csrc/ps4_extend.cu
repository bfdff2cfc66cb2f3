// ps4_extend.cu -- the batched search as two persistent kernels per batch of S:
//
//   gen_jobs<TL,NT,SIDE>  tiles of 2^TL S in shared memory (P1-P4 of ps4_device.cuh), then every
//                 4-set of the tile (P5: two searches per representation pair give the z intervals)
//                 is written to a global job queue, each warp into stretches it reserves.
//                                                                             (s4.c:280-341)
//   extend_jobs   the extension engine.  Each lane of a warp takes one queued 4-set, picks the
//                 difference to extend by and factors it (phase A).  The candidates of the
//                 round's 4-sets -- the complementary divisor pairs (f,g), f<g, of equal parity,
//                 each visited once -- are products of two short divisor lists in shared memory,
//                 and come in rows: one divisor of the shorter list (and power of two) against
//                 the whole longer list.  Rows are taken longest first, 32 at a time, one per
//                 lane, so a row's factors are set up once and its candidates take two
//                 multiplications each.  Residue filters mod 64/63/65 are bit tests against
//                 per-4-set masks indexed by residues of f + g = 2u; the candidates that pass go
//                 through a warp queue, where those that are the reference's ext_sqrt are
//                 square-tested 64 at a time.                                  (s4.c:160-207)
//
// The engine is bound by instruction issue (74 % of issue slots busy, 30.0 of 32 threads active; DRAM 3.0 %).
// Per [1,1e10) search its launches take 163 ms; with candidates spread over the lanes in 32 equal
// runs, u64 lists, per-candidate member tests and IEEE double square roots they took 313 ms (25.5 -> 14.8 warp
// instructions per S).  Rows cost a partly empty turn (30.2 turns of 32 candidates per round against
// 24.9 full ones) and save the per-candidate bookkeeping, half of the 85 instructions of the old loop.
//
// Every counter and every reported line is identical to the reference's.

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "ps4_device.cuh"
#include "ps4_rows.cuh"

namespace cg = cooperative_groups;

namespace ps4 {

// ================================================================== job records

// A queued 4-set: its six pair roots (< 2^22), one 24-byte record per 4-set (three 8-byte
// stores and loads; six u32 arrays took 2.2 % more tile-kernel and 1.2 % more engine time per
// [1,1e10) step).  The query item id (< 2^30, MAX_ITEMS) rides in the spare top bits of r_ac (bits 0..9
// of the id), r_ad (bits 10..19) and r_bc (bits 20..29).  The queue of cap records is 6 * cap u32.
__device__ __forceinline__ void put_job(uint32_t *jobs, uint64_t j, const uint32_t r[6], uint32_t item) {
    uint2 *p = (uint2 *)(jobs + 6 * j);               // 8-byte aligned: 24 * j
    p[0] = make_uint2(r[0], r[1] | item << 22);
    p[1] = make_uint2(r[2] | item >> 10 << 22, r[3] | item >> 20 << 22);
    p[2] = make_uint2(r[4], r[5]);
}

// COH: the queue is a ring whose slots are rewritten while the kernel runs, so its words are read
// through L2 (coherent), not the read-only path that may hold a slot's previous 4-set.
template <bool COH = false>
__device__ __forceinline__ void get_job(const uint32_t *jobs, uint64_t j, uint32_t r[6], uint32_t &item) {
    const uint2 *p = (const uint2 *)(jobs + 6 * j);
    const uint2 x = COH ? __ldcg(p) : __ldg(p), y = COH ? __ldcg(p + 1) : __ldg(p + 1),
                z = COH ? __ldcg(p + 2) : __ldg(p + 2);
    r[0] = x.x;
    r[1] = x.y & 0x3FFFFFu;
    r[2] = y.x & 0x3FFFFFu;
    r[3] = y.y & 0x3FFFFFu;
    r[4] = z.x;
    r[5] = z.y;
    item = x.y >> 22 | y.x >> 22 << 10 | y.y >> 22 << 20;
}

// ================================================================== the persistent kernel's ring
//
// Producing CTAs reserve positions (q_tail), wait until each position's slot is free of its
// previous lap, write the 4-set, and publish it: seq[slot] = pos + 1 after a fence.  Consuming
// warps claim positions below q_tail (q_head), wait until each is published, and after the 4-set
// is extended and reported free its slot: seq[slot] = pos + ring size.  Every wait is bounded in
// time (WAIT_NS); a wait that gives up sets the error word to E_TIMEOUT (with which wait in the S
// field: 1 published, 2 slot free, 3 ring room, 4 idle) and the kernel ends, the host re-running
// the call on the two-kernel pipeline.

__device__ __forceinline__ uint64_t gtimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t ld_vol(const uint32_t *p) { return *(const volatile uint32_t *)p; }
__device__ __forceinline__ ull ld_vol(const ull *p) { return *(const volatile ull *)p; }

// Tracks one wait's elapsed time: true once it has lasted WAIT_NS (and records the timeout).
struct WaitClock {
    uint64_t t0 = 0;
    __device__ __forceinline__ bool expired(const SearchArgs &a, unsigned which) {
        const uint64_t t = gtimer();
        if (!t0) { t0 = t; return false; }
        if (t - t0 <= WAIT_NS) return false;
        raise_error(a.status, E_TIMEOUT, which);
        return true;
    }
};

// A producer's slot: wait until it is free for position pos.  False if the call stopped.
__device__ __noinline__ bool ring_wait_free(const SearchArgs &a, uint64_t pos) {
    const uint32_t *f = a.seq + (pos & a.ring_mask);
    WaitClock wc;
    for (uint32_t k = 0;; k++) {
        if (ld_vol(f) == (uint32_t)pos) return true;
        if ((k & 15) == 15 && (ld_vol(&a.status->err) != 0ull || wc.expired(a, 2))) return false;
        __nanosleep(64);
    }
}

// A consumer's claimed position: wait until its 4-set is published.  False if the call stopped,
// or if the position will never be written (every tile is produced and the position lies past
// the last reserved one: a claim that overtook the reservations, see ring_claim).
__device__ __noinline__ bool ring_wait_ready(const SearchArgs &a, uint64_t pos) {
    const uint32_t *f = a.seq + (pos & a.ring_mask);
    WaitClock wc;
    for (uint32_t k = 0;; k++) {
        if (ld_vol(f) == (uint32_t)(pos + 1)) {
            __threadfence();                       // the 4-set's words after its flag
            return true;
        }
        if ((k & 15) == 15) {
            if (ld_vol(&a.status->err) != 0ull) return false;
            if (ld_vol(&a.status->q_produced) >= a.n_tiles && pos >= ld_vol(&a.status->q_tail)) return false;
            if (wc.expired(a, 1)) return false;
        }
        __nanosleep(32);
    }
}

__device__ __forceinline__ void ring_release(const SearchArgs &a, uint64_t pos) {
    __threadfence();                               // every read of the slot before it is handed back
    *(volatile uint32_t *)&a.seq[pos & a.ring_mask] = (uint32_t)(pos + a.ring_mask + 1);
}

// Claim up to n positions below q_tail (one lane of a warp).  The thresholds count published
// 4-sets (q_pub), so that claims rarely land on positions still being written.  While tiles are
// left, fewer than ring_low published 4-sets are left for later (the warp stops consuming, its
// CTA turns to tiles).  While at least ring_fast published positions are unclaimed, an add cannot
// overtake the reservations (every warp of the grid claiming at once takes fewer), so it is
// used; closer to q_tail a compare-and-swap claims only what is reserved.  *got receives the count, the first
// position is returned.
__device__ __forceinline__ uint64_t ring_claim(const SearchArgs &a, uint32_t n, uint32_t *got) {
    ull *head = &a.status->q_head;
    ull h = ld_vol(head);
    const ull t = ld_vol(&a.status->q_tail);
    const long long pub = (long long)(ld_vol(&a.status->q_pub) - h);   // published and unclaimed (about)
    *got = 0;
    if ((long long)(t - h) <= 0) return 0;
    if (pub < (long long)a.ring_low && ld_vol(&a.status->tile_next) < a.n_tiles) return 0;
    if (pub >= (long long)a.ring_fast) {
        *got = n;
        return atomicAdd(head, (ull)n);
    }
    for (int k = 0; k < 16; k++) {
        const ull tt = ld_vol(&a.status->q_tail);
        if ((long long)(tt - h) <= 0) break;
        const ull take = tt - h < n ? tt - h : n;
        const ull prev = atomicCAS(head, h, h + take);
        if (prev == h) {
            *got = (uint32_t)take;
            return h;
        }
        h = prev;
    }
    return 0;
}

// ================================================================== gen_jobs

// P5: the 4-sets of a representation pair x < y are its z > y with, in class 0, P_z < P_x + P_y (P =
// p^2) and p_z of p_x + p_y's parity, and, in class 1, P_z > S - P_x - P_y, p_z of that parity or, for
// odd S, the other, and q_z != p_z (which only the last z can violate).  Both are intervals of the
// sorted list, found by two binary searches, and the list's parity index turns them into a count and
// the j-th z of each.  (A loop over z per pair, once to count and once to write, took 42 % of the
// tile kernel: 82,000 of a tile's 190,000 cycles at S = 4e11.  Per [1,1e10) step of the tile kernel
// 141.4 -> 99.5 ms with this and the lane-wise sort of P4; 2e8 S at 1e12 4.76 -> 3.36, 3e7 at 1.2e13 1.63 -> 1.10.)
struct TileView {
    const uint16_t *off, *k, *start;
    const uint32_t *pbase, *rep_p, *rep_q;
    const uint16_t *ev, *pp;
    uint32_t n_is;
};
struct PairSets {
    uint32_t sx;                       // list start | x << 16
    uint32_t ya;                       // y | 4-sets of class 0 << 16
    uint32_t ab;                       // first z of class 0 | of class 1 << 16, as places in the parity index
};

// The selected S of the pairs g0 + lane, as its place `lo` in the list and its first pair `base` (lanes past the last
// pair get the last S).  pbase[lo]: pairs before the S at lo, n_is of them and the total.  lo0, warp-uniform:
// the S of pair g0; moved on to pair g0 + 32's.  Every selected S has a pair at least, so 32 consecutive
// pairs lie in 32 consecutive S from the first one's.
__device__ __forceinline__ void pair_owner(const uint32_t *pbase, uint32_t n_is, uint32_t g0, int lane, uint32_t &lo0,
                                           uint32_t &lo, uint32_t &base) {
    const uint32_t pb = lo0 + lane < n_is ? pbase[lo0 + lane] : 0xFFFFFFFFu;
    const uint32_t rel = pb - g0;                          // starts behind the first pair, as a bit mask
    const unsigned starts = __reduce_or_sync(0xffffffffu, rel - 1u < 31u ? 1u << rel : 0u);
    const uint32_t o = __popc(starts & (0xFFFFFFFFu >> (31 - lane)));
    base = __shfl_sync(0xffffffffu, pb, o);
    lo = lo0 + o;
    lo0 += __popc(starts);
    if (pbase[lo0 + 1] <= g0 + 32) lo0++;                  // its pairs end with this step
}

// The pairs g of a warp, one per lane (32 consecutive ones; ge ends the warp's block): each lane's
// number of 4-sets and where they are.  lo0: as for pair_owner.
__device__ __forceinline__ uint32_t pair_sets(const TileView &v, uint64_t S0, uint32_t g, uint32_t ge, int lane,
                                              uint32_t &lo0, PairSets &ps) {
    uint32_t lo, base;
    pair_owner(v.pbase, v.n_is, g - lane, lane, lo0, lo, base);
    if (g >= ge) return 0;
    const uint32_t st = v.start[lo], k = v.k[lo];
    const uint64_t S = S0 + v.off[lo];
    uint32_t x, y;
    decode_pair(g - base, x, y);
    const uint32_t *p = v.rep_p + st;
    const uint16_t *ev = v.ev + st + lo;
    const uint32_t px = p[x], py = p[y];
    const uint64_t T = (uint64_t)px * px + (uint64_t)py * py, U = S - T;
    uint32_t za = y + 1, zb = y + 1, n = k - 1 - y;        // first z with P_z >= T / with P_z > U
    while (n > 1) {
        const uint32_t h = n >> 1, pa = p[za + h - 1], pb2 = p[zb + h - 1];
        if ((uint64_t)pa * pa < T) za += h;
        if ((uint64_t)pb2 * pb2 <= U) zb += h;
        n -= h;
    }
    {
        const uint32_t pa = p[za], pb2 = p[zb];
        if ((uint64_t)pa * pa < T) za++;
        if ((uint64_t)pb2 * pb2 <= U) zb++;
    }
    const uint32_t oa = (px + py) & 1u, ob = oa ^ ((uint32_t)S & 1u);     // the parity of p_z in each class
    const uint32_t ne = ev[k];
    const uint32_t e0 = ev[y + 1], ea = ev[za], eb = ev[zb];
    const uint32_t a0 = oa ? y + 1 - e0 : e0, a1 = oa ? za - ea : ea;
    const uint32_t b0 = ob ? zb - eb : eb, b1 = ob ? k - ne : ne;
    const uint32_t na = a1 - a0;
    uint32_t nb = b1 - b0;
    if (nb && !(S & 1) && p[k - 1] == v.rep_q[st + k - 1]) nb--;         // even S: ob is every p's parity
    ps.sx = st | x << 16;
    ps.ya = y | na << 16;
    ps.ab = (st + (oa ? ne : 0) + a0) | (st + (ob ? ne : 0) + b0) << 16;
    return na + nb;
}

// The write pass of one warp step: the lanes' 4-sets (n each, places ps) are spread evenly over the
// warp, 32 per turn, checked and dumped where asked, and queued (when `store`): the first `rem` at
// `cur`, those after them at `next`.
template <bool RING>
__device__ __forceinline__ void write_sets(const SearchArgs &a, const TileView &v, uint32_t n, const PairSets &ps,
                                           uint32_t first, uint32_t total, int lane, uint64_t S0, uint32_t item,
                                           bool store, uint64_t cur, uint32_t rem, uint64_t next) {
    for (uint32_t t = 0; t < total; t += 32) {
        const uint32_t s = t + lane;
        uint32_t o = 0;                                                  // the last lane with first <= s
#pragma unroll
        for (uint32_t step = 16; step; step >>= 1)
            if (__shfl_sync(0xffffffffu, first, o + step) <= s) o += step;
        const uint32_t f = __shfl_sync(0xffffffffu, first, o), sx = __shfl_sync(0xffffffffu, ps.sx, o),
                       ya = __shfl_sync(0xffffffffu, ps.ya, o), ab = __shfl_sync(0xffffffffu, ps.ab, o);
        if (s >= total) continue;
        const uint32_t st = sx & 0xFFFFu, x = st + (sx >> 16), y = st + (ya & 0xFFFFu), na = ya >> 16;
        uint32_t j = s - f;
        const bool one = j >= na;                                        // class 1
        j = one ? (ab >> 16) + j - na : (ab & 0xFFFFu) + j;
        const uint32_t z = st + v.pp[j];
        const uint32_t pz = v.rep_p[z], qz = v.rep_q[z];
        uint32_t r[6];
        r[0] = v.rep_q[x]; r[1] = v.rep_q[y]; r[4] = v.rep_p[y]; r[5] = v.rep_p[x];
        r[2] = one ? pz : qz;
        r[3] = one ? qz : pz;
        if (a.flags & (PS4_F_VERIFY | PS4_F_DUMP4)) {
            uint64_t m[4], S;
            quad_values(r, m, S);
            if ((a.flags & PS4_F_VERIFY) && !quad_roots_ok(m, r)) record_verify_failure(a, S, m);
            if (a.flags & PS4_F_DUMP4) dump_quad(a, r);
        }
        if (store) {
            const uint64_t pos = s < rem ? cur + s : next + (s - rem);
            if (!RING) {
                put_job(a.jobs, pos, r, item);
            } else if (ring_wait_free(a, pos)) {
                put_job(a.jobs, pos & a.ring_mask, r, item);
                __threadfence();
                *(volatile uint32_t *)&a.seq[pos & a.ring_mask] = (uint32_t)(pos + 1);
            }
        }
    }
}

// A warp's open stretch of the job queue: a.chunk records at a time are reserved (one atomic), so that
// the tile needs no count pass and no barrier before its 4-sets are written.  What is left at the
// kernel's end is filled with empty records, which the engine passes over.
struct JobSpan {
    uint64_t cur = 0;
    uint32_t rem = 0;
};
// A tile's positions in the persistent kernel's ring, in shared memory: the first one, and whether there is room.
struct RingSpan {
    ull base;
    int store;
};

// One tile [S0, S0+n) of query item `item`: P1-P4 (from its list's parts, or by scanning when list
// is null), then P5: each warp takes a contiguous block of the tile's pairs, 32 at a time.  NT threads.
// The tile kernel (RING false) queues what a step finds in the warp's open stretch.  The persistent
// kernel counts first and reserves the tile's 4-sets at once (the ring's room is waited for), and
// each 4-set is published after a fence.
template <int TL, int NT, bool RING, bool SIDE>
__device__ __forceinline__ void produce_tile(const SearchArgs &a, TileShared &ts, unsigned char *smem, uint64_t S0,
                                             uint32_t n, uint32_t item, const uint64_t *list,
                                             const uint32_t *list_n, uint32_t parts, uint32_t cap,
                                             std::conditional_t<RING, RingSpan, JobSpan> &span) {
    using L = TileLayout<TL>;
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const bool noext = (a.flags & PS4_F_NOEXT) != 0;
    const bool need_write_pass = !noext || (a.flags & (PS4_F_DUMP4 | PS4_F_VERIFY));
    tile_reset(ts);
    __syncthreads();
    if (!tile_reps<TL, NT, true, SIDE>(a, ts, smem, S0, n, list, list_n, parts, cap)) { __syncthreads(); return; }
    TileView v;
    v.off = (const uint16_t *)(smem + L::OFF_IS_OFF);
    v.k = (const uint16_t *)(smem + L::OFF_IS_K);
    v.start = (const uint16_t *)(smem + L::OFF_IS_START);
    v.pbase = (const uint32_t *)(smem + L::OFF_IS_PBASE);
    v.rep_p = (const uint32_t *)(smem + L::OFF_REP_P);
    v.rep_q = (const uint32_t *)(smem + L::OFF_REP_Q);
    v.ev = (const uint16_t *)(smem + TileIndex<TL>::OFF_EV);
    v.pp = (const uint16_t *)(smem + TileIndex<TL>::OFF_PP);
    v.n_is = ts.n_is;
    const uint32_t nPairs = ts.n_pairs;
    // each warp a contiguous block of pairs (whole multiples of 32), and the S of its first one
    const uint32_t blk = ((nPairs + NW * 32 - 1) / (NW * 32)) * 32;
    const uint32_t gw = (uint32_t)wid * blk, ge = min(nPairs, gw + blk);
    uint32_t lo0 = 0;
    if (gw < ge) {
        uint32_t hi = v.n_is;
        while (hi - lo0 > 1) {
            const uint32_t mid = (lo0 + hi) >> 1;
            if (v.pbase[mid] <= gw) lo0 = mid; else hi = mid;
        }
    }
    PairSets ps;
    uint32_t mine = 0, total;
    if constexpr (RING) {
        const uint32_t lo_first = lo0;
        for (uint32_t g = gw; g < ge; g += 32) mine += pair_sets(v, S0, g + lane, ge, lane, lo0, ps);
        lo0 = lo_first;
        uint32_t off, d1, d2, tot[3];
        block_scan3<NT>(mine, 0u, 0u, off, d1, d2, tot, ts.wsum);
        if (tid == 0) {
            span.base = 0;
            span.store = 0;
            if (!noext && tot[0]) {
                // room: the ring holds the reserved-but-unfinished 4-sets plus this tile's
                WaitClock wc;
                bool ok = true;
                while (ld_vol(&a.status->q_tail) + tot[0] - ld_vol(&a.status->q_freed) > a.jobs_cap) {
                    if (ld_vol(&a.status->err) != 0ull || wc.expired(a, 3)) { ok = false; break; }
                    __nanosleep(256);
                }
                if (ok) {
                    span.base = atomicAdd(&a.status->q_tail, (ull)tot[0]);
                    span.store = 1;
                }
            }
        }
        __syncthreads();
        if (need_write_pass) {
            uint64_t cur = span.base + __shfl_sync(0xffffffffu, off, 0);
            for (uint32_t g = gw; g < ge; g += 32) {
                const uint32_t m = pair_sets(v, S0, g + lane, ge, lane, lo0, ps);
                const uint32_t first = warp_prefix(m, lane, total);
                write_sets<true>(a, v, m, ps, first, total, lane, S0, item, span.store != 0, cur, total, 0);
                cur += total;
            }
        }
        __syncthreads();
        if (tid == 0 && span.store && tot[0]) atomicAdd(&a.status->q_pub, (ull)tot[0]);
    } else {
        for (uint32_t g = gw; g < ge; g += 32) {
            const uint32_t m = pair_sets(v, S0, g + lane, ge, lane, lo0, ps);
            mine += m;
            if (!need_write_pass) continue;                              // warp-uniform
            const uint32_t first = warp_prefix(m, lane, total);
            if (total == 0) continue;
            uint64_t next = 0;
            uint32_t room = 0;
            bool store = !noext;
            if (store && total > span.rem) {
                room = max(a.chunk, total - span.rem);
                if (lane == 0) next = atomicAdd(&a.status->n_jobs, (ull)room);
                next = __shfl_sync(0xffffffffu, next, 0);
                if (next + room > a.jobs_cap) {
                    if (lane == 0) raise_capacity(a.status, E_QUEUE, 5, next + room, a.jobs_cap, S0);
                    store = false;
                }
            }
            write_sets<false>(a, v, m, ps, first, total, lane, S0, item, store, span.cur, span.rem, next);
            if (store) {
                if (room) {
                    span.cur = next + (total - span.rem);
                    span.rem = room - (total - span.rem);
                } else {
                    span.cur += total;
                    span.rem -= total;
                }
            }
        }
    }
    const ull found = warp_sum((ull)mine);
    if (lane == 0 && found) atomicAdd(&ts.cnt[K_SETS4], found);
    __syncthreads();
    tile_flush_counters(a, ts, item);
    __syncthreads();
}

// The persistent kernel's claim of SUPER_K tiles, the last-but-c0 ones of the launch (tiles are
// taken from the last one down, costliest first): per segment among them one scan for all its
// tiles, then tile by tile.  Returns the number of tiles.
template <int TL, int NT>
__device__ uint32_t produce_group(const SearchArgs &a, TileShared &ts, unsigned char *smem, uint64_t c0,
                                  uint64_t *lists, uint32_t *raw_n, RingSpan &span) {
    using L = TileLayout<TL>;
    const uint64_t cn = min((uint64_t)SUPER_K, a.n_tiles - c0);
    uint64_t ti = a.n_tiles - c0 - cn;
    const uint64_t ti_end = a.n_tiles - c0;
    while (ti < ti_end) {
        const Item it = segment_of(a, ti);
        const uint64_t seg_tiles = (it.hi - it.lo + (1ull << TL) - 1) >> TL;
        const uint64_t g_end = min(ti_end, it.tile_base + seg_tiles);
        const uint32_t ng = (uint32_t)(g_end - ti);
        const uint64_t SA = it.lo + ((ti - it.tile_base) << TL);
        const uint64_t SB = min(it.hi, SA + ((uint64_t)ng << TL));
        if (threadIdx.x < SUPER_K) raw_n[threadIdx.x] = 0;
        __syncthreads();
        scan_group<NT>(SA, SB, TL, lists, a.raw_cap, raw_n, 0, 1);
        __syncthreads();
        for (uint32_t j = 0; j < ng; j++) {
            const uint64_t S0 = SA + ((uint64_t)j << TL);
            produce_tile<TL, NT, true, false>(a, ts, smem, S0, (uint32_t)min((uint64_t)L::W, SB - S0), it.id,
                                       raw_n[j] <= a.raw_cap ? lists + (size_t)j * a.raw_cap : nullptr, &raw_n[j], 1,
                                       a.raw_cap, span);
        }
        ti = g_end;
    }
    return (uint32_t)cn;
}

// The tile kernel: clusters of CTAs claim `a.group` tiles at a time (from the last one down,
// costliest first).  Per segment among them the cluster's CTAs share one scan -- each takes every
// nc-th q and appends what it finds to its part of the tiles' lists -- and then take the tiles one
// by one from a common counter.  A scan costs ~0.29 sqrt(S) steps however few S it covers, and a
// narrow call has too few tiles for one CTA each on a scan of its own, so both ends gain from sharing it.
template <int TL, int NT, bool SIDE>
__global__ void __launch_bounds__(NT, NT > BS ? 1 : BS / NT * 2) gen_jobs(const __grid_constant__ SearchArgs a) {
    using L = TileLayout<TL>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ TileShared ts;
    __shared__ unsigned long long s_claim;
    JobSpan span;
    __shared__ uint32_t s_tile, s_fit;
    // entries that this CTA's scan appended to each tile's list, and the next tile to take (CTA 0's
    // is used).  Two sets, one for each parity of the group: a set is cleared while the other one's
    // group is scanned, between the two cluster barriers that no CTA passes before all have
    // finished the group that used it last.
    __shared__ uint32_t raw_n[2][GEN_CLUSTER * SUPER_K];
    __shared__ uint32_t s_take[2];
    __shared__ uint32_t s_n[GEN_CLUSTER];                                // the parts' entries of the tile at hand
    const int tid = threadIdx.x;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), nc = cluster.num_blocks();
    const uint32_t cap = a.raw_cap / nc;
    uint64_t *lists = a.raw + (size_t)(blockIdx.x / nc) * nc * a.raw_lists * a.raw_cap;
    for (uint32_t i = tid; i < GEN_CLUSTER * SUPER_K; i += NT) raw_n[0][i] = 0;
    if (tid == 0) s_take[0] = 0;
    uint64_t ti = 0, ti_end = 0;
    for (uint32_t par = 0;; par ^= 1) {                                  // every CTA of the cluster alike
        if (ti == ti_end) {
            if (rank == 0 && tid == 0)
                s_claim = *(volatile ull *)&a.status->err != 0ull ? a.n_tiles
                                                                  : (ull)atomicAdd(&a.status->tile_next, a.group);
            cluster.sync();
            const uint64_t c0 = *cluster.map_shared_rank(&s_claim, 0);
            if (c0 >= a.n_tiles) break;
            ti_end = a.n_tiles - c0;
            ti = ti_end - min((uint64_t)a.group, ti_end);
        } else {
            cluster.sync();
        }
        for (uint32_t i = tid; i < GEN_CLUSTER * SUPER_K; i += NT) raw_n[par ^ 1][i] = 0;
        if (tid == 0) s_take[par ^ 1] = 0;
        const Item it = segment_of(a, ti);
        const uint64_t seg_tiles = (it.hi - it.lo + (1ull << TL) - 1) >> TL;
        const uint64_t g_end = min(ti_end, it.tile_base + seg_tiles);
        const uint32_t ng = (uint32_t)(g_end - ti);
        const uint64_t SA = it.lo + ((ti - it.tile_base) << TL);
        const uint64_t SB = min(it.hi, SA + ((uint64_t)ng << TL));
        scan_group<NT>(SA, SB, TL, lists, cap, raw_n[par], rank, nc);
        cluster.sync();
        for (;;) {
            if (tid == 0) {
                s_tile = atomicAdd(cluster.map_shared_rank(&s_take[par], 0), 1u);
                s_fit = 1;
            }
            __syncthreads();
            const uint32_t j = s_tile;
            if (j >= ng) break;                                          // block-uniform
            if (tid < nc) {
                const uint32_t c = *cluster.map_shared_rank(&raw_n[par][j], tid);
                s_n[tid] = c;
                if (c > cap) s_fit = 0;
            }
            __syncthreads();
            const uint64_t S0 = SA + ((uint64_t)j << TL);
            produce_tile<TL, NT, false, SIDE>(a, ts, smem, S0, (uint32_t)min((uint64_t)L::W, SB - S0), it.id,
                                        s_fit ? lists + (size_t)j * nc * cap : nullptr, s_n, nc, cap, span);
        }
        __syncthreads();                                                 // s_tile read by all
        ti = g_end;
    }
    const uint32_t none[6] = {0, 0, 0, 0, 0, 0};
    for (uint32_t i = tid & 31; i < span.rem; i += 32) put_job(a.jobs, span.cur + i, none, 0);
    cluster.sync();                          // no CTA leaves while another may read its shared memory
}

// ================================================================== extend_jobs

constexpr int EBS = 256;                 // threads per CTA
constexpr int EWARPS = EBS / 32;
constexpr int DCAP = 640;                // divisor-list entries per warp (u32)
constexpr int CPT = 4;                   // candidates of a row per turn: independent chains (4 / 3 / 2: 175.5 / 181.8 /
                                         //   179.2 ms per [1,1e10) search)
constexpr int QCAP = 64 + 32 * CPT;      // square-test queue per warp
constexpr int EXCAP = 8;                 // extensions found in a warp's round
constexpr int ICACHE = 8;                // items whose counters a warp holds back

struct __align__(16) EJob {              // one lane's 4-set
    uint64_t m63, m65;                   // residue masks of f + g + 32 = 2u + 32 (see VResTabs)
    uint32_t m64, geo;                   // geo: L | H << 8 | E2 << 16 | list place << 22
    uint64_t A;                          // extend by D = A - B: e = u^2 - A
    int64_t d1, d2;                      // C - A of the other two members (square tests of u^2 + (C - A))
    uint32_t rA0, rA1, rA2;              // the roots sqrt(A + v) of the three other members: e is one of
                                         //   them iff u is one of these
    uint32_t item;
    uint32_t nsq;                        // ext_sqrt, where the round's items differ
    uint32_t pad[3];                     // 80 bytes: vector accesses of eight jobs meet no bank twice (64
                                         //   bytes: engine 189.3 -> 182.7 ms per [1,1e10) search)
};
static_assert(sizeof(EJob) == 80 && offsetof(EJob, d1) == 32 && offsetof(EJob, rA0) == 48, "vector loads of job fields");
static_assert(LCAP <= 255 && DCAP <= 1024, "fields of geo");

struct ItemCount {                       // counters of an item that the warp holds back
    uint32_t item, mdiv;
    ull cand, sqrt_;
};

struct WarpArea {
    EJob job[32];
    uint32_t dbuf[DCAP];                 // turns may read LCAP + CPT entries past a list's ends: the
                                         //   neighbours on both sides are longer than that
    union {                              // primes until the lists are made, then the queue
        uint32_t fp[2 * FSIDE][32];      // each lane's odd primes of D (p | e << 24), m1's from slot 0, m2's
                                         //   others from FSIDE, lane-minor (no bank conflicts)
        uint64_t q[QCAP];                // candidates that pass the filters: f + g + 32 | job << 58
    };
    ItemCount ic[ICACHE];
    uint64_t hit_u[EXCAP];               // what rare_work is left with: the round's extensions u, their
    uint32_t hit_jid[EXCAP];             //   4-sets,
    uint32_t big[64];                    //   and the 4-sets for the per-lane divisor walk (queue indices)
    uint32_t n_hit, n_big, n_ext;
    uint32_t pend, rel, took;            // the rounds' state while rare_work runs (lane masks)
    uint32_t jid[32];                    // queue index of each lane's 4-set
    // the loop's own state, out of the registers between its claims (the same for all lanes)
    uint32_t njobs, quota, stretch;      // queue length; lanes that hold a 4-set; 4-sets per stretch
    uint32_t st_cur, st_rem, last;       // the stretch at hand; whether it is the last
    uint32_t claimed;                    // 4-sets in the warps' first stretches
    uint8_t order[32];                   // lanes by row length, longest first
};
static_assert(sizeof(EJob) * 32 >= 4 * (LCAP + CPT) && 4 * 32 * 2 * FSIDE >= 4 * (LCAP + CPT), "neighbours of dbuf");
static_assert(EWARPS * sizeof(WarpArea) + 1024 <= 228 * 1024 / 3, "three engine CTAs per SM");

constexpr int EXTCAP = 4 * DCAP / (int)sizeof(ExtEntry);     // a report's extensions, in dbuf
static_assert(offsetof(WarpArea, dbuf) % 8 == 0 && EXTCAP >= EXCAP, "room for a report");

constexpr uint32_t NO_ITEM = 0xFFFFFFFFu;

__device__ __forceinline__ void count_global(const SearchArgs &a, uint32_t item, ull cand, ull sq, uint32_t mdiv) {
    ull *k = a.counters + (size_t)item * K_SLOTS;
    if (cand) atomicAdd(&k[K_EXT_CAND], cand);
    if (sq) atomicAdd(&k[K_EXT_SQRT], sq);
    if (mdiv) atomicMax(&k[K_MAX_DIVS], (ull)mdiv);
}

// A warp's counters: one item at a time (queries of a batch are separate items; the queue's
// neighbours mostly belong to one), summed over the lanes and, when the item changes, put into the
// warp's small cache of items, which reaches the items' counter blocks when an entry is pushed out and
// at the end.  (Every lane's own atomics to one block took most of a small call's engine time: 2e5
// 4-sets 0.28 -> 0.08 ms; without the cache, claims that alternate between the items in production
// cost 64 uneven subranges 20 ms of 50 in atomics.)
struct WarpCounters {
    uint32_t item = NO_ITEM;                     // warp-uniform
    uint32_t cand = 0, sqrt_ = 0, mdiv = 0;      // a lane meets 2^29 / 32 4-sets of a few dozen candidates at most
    __device__ __forceinline__ void flush(const SearchArgs &a, WarpArea *w, int lane) {      // the whole warp
        // sums of 32-bit values by halves (at most 32 * 65535 each)
        const ull c = (ull)__reduce_add_sync(0xffffffffu, cand & 0xFFFFu) +
                      ((ull)__reduce_add_sync(0xffffffffu, cand >> 16) << 16);
        const ull s = (ull)__reduce_add_sync(0xffffffffu, sqrt_ & 0xFFFFu) +
                      ((ull)__reduce_add_sync(0xffffffffu, sqrt_ >> 16) << 16);
        const uint32_t d = __reduce_max_sync(0xffffffffu, mdiv);
        if (lane == 0 && item != NO_ITEM) {
            ItemCount &e = w->ic[item * 0x9E3779B1u >> 29];
            if (e.item == item) {
                e.cand += c;
                e.sqrt_ += s;
                e.mdiv = max(e.mdiv, d);
            } else {
                if (e.item != NO_ITEM) count_global(a, e.item, e.cand, e.sqrt_, e.mdiv);
                e.item = item;
                e.cand = c;
                e.sqrt_ = s;
                e.mdiv = d;
            }
        }
        cand = 0; sqrt_ = 0; mdiv = 0;
    }
    // the whole warp: the lanes with `have` count c, s and d for their item `it`
    __device__ __forceinline__ void add(const SearchArgs &a, WarpArea *w, int lane, bool have, uint32_t it, uint32_t c,
                                        uint32_t s, uint32_t d) {
        for (;;) {
            if (have && it == item) {
                cand += c;
                sqrt_ += s;
                mdiv = max(mdiv, d);
                have = false;
            }
            const unsigned m = __ballot_sync(0xffffffffu, have);
            if (!m) break;
            flush(a, w, lane);
            item = __shfl_sync(0xffffffffu, it, __ffs((int)m) - 1);
        }
    }
};
static_assert(ICACHE == 8, "the cache index is a 3-bit hash");

// Report a warp's extensions: group them per 4-set, emit hit / ext / six
// records and the counters sets5 / multi / sets6 / hist5 / max_extensions (s4.c:243-277).
template <bool COH>
static __device__ void report_warp_exts(const SearchArgs &a, ExtEntry *el, uint32_t n) {
    for (uint32_t x = 1; x < n; x++) {
        ExtEntry k = el[x];
        uint32_t y = x;
        while (y > 0 && (el[y - 1].qid > k.qid || (el[y - 1].qid == k.qid && el[y - 1].key > k.key))) {
            el[y] = el[y - 1];
            y--;
        }
        el[y] = k;
    }
    for (uint32_t g0 = 0; g0 < n;) {
        uint32_t g1 = g0 + 1;
        while (g1 < n && el[g1].qid == el[g0].qid) g1++;
        const uint32_t ne = g1 - g0;
        uint32_t roots[6], item;                              // the 4-set and its item, from the queue
        get_job<COH>(a.jobs, el[g0].qid, roots, item);
        ull *cnt = a.counters + (size_t)item * K_SLOTS;
        uint64_t v[4], S;
        quad_values(roots, v, S);
        if (ne > a.cap_ext) { raise_error(a.status, E_CAP_EXT, S); g0 = g1; continue; }
        atomicMax(&cnt[K_MAX_EXT], (ull)ne);
        uint64_t vmax = v[0];
        for (int i = 1; i < 4; i++) vmax = v[i] > vmax ? v[i] : vmax;
        bool prints = ne >= 2;
        for (uint32_t t = 0; t < ne; t++) prints |= (el[g0 + t].hi != 0 || el[g0 + t].lo > vmax);
        uint32_t hslot = 0, eslot = 0;
        if (prints) {
            hslot = atomicAdd(&a.status->n_hits, 1u);
            eslot = atomicAdd(&a.status->n_exts, ne);
        }
        uint32_t hflags = 0;
        if (ne >= 2) {
            hflags |= PS4_HIT_MULTI;
            atomicAdd(&cnt[K_MULTI], 1ull);
            u128 x[6] = {v[0], v[1], v[2], v[3], ((u128)el[g0].hi << 64) | el[g0].lo,
                         ((u128)el[g0 + 1].hi << 64) | el[g0 + 1].lo};
            if (verify_set(x, 6)) hflags |= PS4_HIT_DRILL_OK;
        }
        for (uint32_t t = 0; t < ne; t++) {
            const u128 e = ((u128)el[g0 + t].hi << 64) | el[g0 + t].lo;
            uint32_t ef = 0;
            if (e > vmax) {
                ef |= PS4_EXT_FIVE;
                atomicAdd(&cnt[K_SETS5], 1ull);
                int lg = 0;
                for (u128 z = e; z > 1; z >>= 1) lg++;
                atomicAdd(&cnt[K_HIST5 + (lg > 99 ? 99 : lg)], 1ull);
                u128 x[5] = {v[0], v[1], v[2], v[3], e};
                if (verify_set(x, 5)) ef |= PS4_EXT_FIVE_OK;
            }
            if (prints && eslot + t < a.exts_cap) {
                ps4_ext rec;
                rec.lo = el[g0 + t].lo; rec.hi = el[g0 + t].hi; rec.key = el[g0 + t].key; rec.flags = ef;
                a.exts[eslot + t] = rec;
            }
        }
        for (uint32_t t = 0; t < ne; t++)
            for (uint32_t s = t + 1; s < ne; s++) {
                const u128 et = ((u128)el[g0 + t].hi << 64) | el[g0 + t].lo;
                const u128 es = ((u128)el[g0 + s].hi << 64) | el[g0 + s].lo;
                if (!is_square_exact(et + es)) continue;
                atomicAdd(&cnt[K_SETS6], 1ull);
                u128 x[6] = {v[0], v[1], v[2], v[3], et, es};
                const uint32_t sslot = atomicAdd(&a.status->n_sixes, 1u);
                if (sslot < a.sixes_cap) {
                    ps4_six rec;
                    rec.hit = hslot; rec.t = t; rec.s = s; rec.flags = verify_set(x, 6) ? 1u : 0u;
                    a.sixes[sslot] = rec;
                }
            }
        if (prints && hslot < a.hits_cap) {
            ps4_hit h;
            h.S = S;
            for (int i = 0; i < 4; i++) h.v[i] = v[i];
            h.n_ext = ne; h.first_ext = eslot; h.flags = hflags; h.item = item;
            h.order[0] = roots[5]; h.order[1] = roots[4];
            h.order[2] = roots[2] < roots[3] ? roots[2] : roots[3];
            h.order[3] = roots[2] < roots[3] ? 1u : 0u;
            a.hits[hslot] = h;
        }
        g0 = g1;
    }
}

struct LaneJob {                                 // a lane's 4-set in its round
    uint32_t item, ncand, nd;
    uint32_t L, H, rows;                         // list lengths; full rows and the last half one
    uint32_t slots;                              // row list: first prime slot | primes << 8, the other << 16
    bool big;                                    // for the per-lane divisor walk
};

// p[i] by a 32-bit byte offset (tables are below 2^32 bytes): one register for an address in flight, not two
template <class T>
__device__ __forceinline__ T ldg_at(const T *p, uint32_t i) {
    return __ldg((const T *)((const char *)p + (uint32_t)(i * (uint32_t)sizeof(T))));
}

// Phase A: one 4-set per lane.  Picks the difference to extend by (the fewest estimated divisors, in
// the candidate order and with the tie-break of s4.c:163-171), factors it and writes the lane's
// EJob.  False: an empty record, or more divisors than the cap.
template <bool COH>
__device__ __forceinline__ bool job_setup(const SearchArgs &a, uint64_t j, LaneJob &J, WarpArea *w, int lane) {
    uint32_t r[6];
    get_job<COH>(a.jobs, j, r, J.item);
    if (r[0] == 0) return false;                   // an empty record (the end of a tile warp's stretch)
    // The six candidate pairs (i, j) with third member k: v_i - v_j = r_ik^2 - r_jk^2.  (0,1;2) (2,3;0)
    // (0,2;1) (1,3;0) (0,3;1) (1,2;0), the first of the least kept.
    uint32_t best = 0xFFFFFFFFu, rik = 0, rjk = 0;
    auto pair = [&](int t, uint32_t x, uint32_t y) {
        const uint32_t hi = max(x, y), lo = min(x, y);
        const uint32_t est = (uint32_t)ldg_at(a.ndiv, hi - lo) * (uint32_t)ldg_at(a.ndiv, hi + lo);
        const uint32_t key = est * 8u + t;                                       // est < 2^26
        if (key < best) { best = key; rik = x; rjk = y; }
    };
    pair(0, r[1], r[3]);
    pair(1, r[1], r[2]);
    pair(2, r[0], r[3]);
    pair(3, r[0], r[2]);
    pair(4, r[0], r[4]);
    pair(5, r[0], r[1]);
    const uint32_t t = best & 7u;
    // D = m1 * m2; D even => both even.  The factors are loaded while the members are worked out.
    uint32_t m1 = max(rik, rjk) - min(rik, rjk), m2 = rik + rjk, E2 = 0;
    if (!(m1 & 1)) {
        const uint32_t z1 = (uint32_t)__ffs((int)m1) - 1, z2 = (uint32_t)__ffs((int)m2) - 1;
        E2 = z1 + z2;
        m1 >>= z1;
        m2 >>= z2;
    }
    const uint4 fa = ldg_at(a.fac, m1 >> 1), fb = ldg_at(a.fac, m2 >> 1);
    EJob &E = w->job[lane];
    {
        uint64_t v[4];
        const uint64_t ab = (uint64_t)r[0] * r[0], ac = (uint64_t)r[1] * r[1], ad = (uint64_t)r[2] * r[2],
                       bc = (uint64_t)r[3] * r[3];
        v[0] = (ab + ac - bc) >> 1; v[1] = ab - v[0]; v[2] = ac - v[0]; v[3] = ad - v[0];
        // i = 0,2,0,1,0,1 and j = 1,3,2,3,3,2 for t = 0..5; the other two are 2,3 / 0,1 / 1,3 / 0,2 / 1,2 / 0,3
        const bool i0 = (0x15u >> t) & 1u, i1 = (0x28u >> t) & 1u;               // i = 0; i = 1; else 2
        const bool j3 = (0x1Au >> t) & 1u, j2 = (0x24u >> t) & 1u;               // j = 3; j = 2; else 1
        const bool sw = rik < rjk;                                               // v_i < v_j
        const uint64_t A = sw ? (j3 ? v[3] : j2 ? v[2] : v[1]) : (i0 ? v[0] : i1 ? v[1] : v[2]);
        const uint64_t C1 = t == 0 ? v[2] : (0x14u >> t) & 1u ? v[1] : v[0];     // t = 2, 4: 1; t = 1, 3, 5: 0
        const uint64_t C2 = (0x25u >> t) & 1u ? v[3] : t == 1 ? v[1] : v[2];     // t = 0, 2, 5: 3; t = 3, 4: 2
        const uint32_t bi = sw ? (j3 ? 3u : j2 ? 2u : 1u) : (i0 ? 0u : i1 ? 1u : 2u);
        E.A = A;
        const int64_t d1 = (int64_t)C1 - (int64_t)A, d2 = (int64_t)C2 - (int64_t)A;
        E.d1 = d1;
        E.d2 = d2;
        // the roots through member bi: r_ab r_ac r_ad / r_ab r_bc r_bd / r_ac r_bc r_cd / r_ad r_bd r_cd
        E.rA0 = bi <= 1 ? r[0] : bi == 2 ? r[1] : r[2];
        E.rA1 = bi == 0 ? r[1] : bi == 3 ? r[4] : r[3];
        E.rA2 = bi == 0 ? r[2] : bi == 1 ? r[4] : r[5];
        E.item = J.item;
        E.nsq = 0;
        uint32_t m64 = 0xFFFFFFFFu;
        uint64_t m63 = ~0ull, m65 = ~0ull;
        and_masks(d1, m64, m63, m65);
        and_masks(d2, m64, m63, m65);
        E.m64 = m64; E.m63 = m63; E.m65 = m65;
    }
    PairLists pl;
    split_pair(a.spfq, fa, fb, m1, m2, w->fp, lane, pl);
    const uint32_t L = pl.L, H = pl.H, ndo = L * H;
    const uint64_t nd = (uint64_t)ndo * (E2 + 1);
    if (nd > a.cap_divs) {
        raise_error(a.status, E_CAP_DIVS, (uint64_t)r[0] * r[0] + (uint64_t)r[5] * r[5]);
        return false;
    }
    J.nd = (uint32_t)nd;
    J.slots = pl.slots;
    J.L = L;
    J.H = H;
    // same-parity complementary pairs with f < g: the reference's ext_cand (s4.c:191)
    const uint32_t R = E2 ? E2 - 1 : 1;            // 2-exponents of f: 1 .. E2-1, or 0
    J.ncand = ndo * R >> 1;
    J.rows = (H * R + (L > 1 ? 1u : 0u)) >> 1;
    E.geo = L | H << 8 | E2 << 16;
    // a list longer than the fields and buffers allow, or one side above 32 bits: the per-lane walk
    J.big = pl.wide || L > (uint32_t)LCAP;
    return true;
}

// A 4-set whose factored divisor lists exceed the warp buffer or 32 bits: the per-lane divisor walk.
// Returns its ext_sqrt and its item.
template <bool COH>
__device__ __forceinline__ uint32_t extend_big(const SearchArgs &a, uint32_t qid, ExtEntry *el, uint32_t *el_n,
                                               uint32_t &item) {
    ull cand = 0, sq = 0;
    uint32_t r[6], best, md = 0;
    uint64_t v[4], S;
    int bi, bj, bk;
    get_job<COH>(a.jobs, qid, r, item);
    quad_values(r, v, S);
    choose_pair(v, r, a.ndiv, bi, bj, bk, best);
    extend_quad(a, r, v, S, bi, bj, bk, qid, cand, sq, md, el, el_n, EXTCAP);
    return (uint32_t)sq;
}

// The extension e = u^2 - A of the 4-set at queue index qid.  Its order key is the reference's mixed-radix
// index of the smaller divisor f = u - w, w^2 = e + B, over the primes in first-seen order: 2, m1's, then
// m2's others (s4.c:141-156).
__device__ __forceinline__ void record_ext(const SearchArgs &a, ExtEntry *el, uint32_t *el_n, uint32_t qid,
                                           uint64_t u) {
    uint32_t rt[6], item, best;
    uint64_t v[4], S;
    int bi, bj, bk;
    get_job<true>(a.jobs, qid, rt, item);
    quad_values(rt, v, S);
    choose_pair(v, rt, a.ndiv, bi, bj, bk, best);
    const uint32_t ra = pick6(rt, pair_slot(bi, bk)), rb = pick6(rt, pair_slot(bj, bk));
    uint32_t m1 = ra - rb, m2 = ra + rb, key = 0, mult = 1;
    const u128 e = (u128)u * u - pick4(v, bi);
    uint64_t f = u - isqrt128(e + pick4(v, bj));
    if (!(m1 & 1)) {
        const uint32_t z1 = (uint32_t)__ffs((int)m1) - 1, z2 = (uint32_t)__ffs((int)m2) - 1;
        while (!(f & 1)) { f >>= 1; key++; }
        mult = z1 + z2 + 1;
        m1 >>= z1;
        m2 >>= z2;
    }
    for (int side = 0; side < 2; side++) {
        const uint32_t other = side ? m1 : m2;
        for (uint32_t m = side ? m2 : m1; m > 1;) {
            const uint64_t t = __ldg(&a.spfq[m]);
            const uint32_t p = spf_p(t);
            uint32_t ex = spf_e(t), o = other;
            m = spf_cof(t);
            if (side && o % p == 0) continue;                        // one of m1's
            while (o % p == 0) { o /= p; ex++; }
            while (f % p == 0) { f /= p; key += mult; }
            mult *= ex + 1;
        }
    }
    const uint32_t slot = atomicAdd(el_n, 1u);
    if (slot < EXTCAP) {
        ExtEntry &x = el[slot];
        x.qid = qid;
        x.key = key;
        x.lo = (uint64_t)e;
        x.hi = (uint64_t)(e >> 64);
    } else {
        raise_capacity(a.status, E_EXTLIST, 4, slot + 1, EXTCAP, 0);
    }
}

// What a round seldom has, between two runs of rounds: the 4-sets for the divisor walk, one per lane, and
// the round's extensions, which are recorded and reported.  Called where nothing of a round is live:
// with these calls inside the rounds the compiler kept the rounds' values in local memory (58 M of
// 4.5 G instructions and half of the waiting on loads per 3e8 S at 5e9; [1,1e10) engine 175.5 ->
// 163.4 ms), and one lane walked alone while the others waited (2e8 S at 1e12: 11.4 -> 10.5 ms).
template <bool COH>
static __device__ __noinline__ void rare_work(const SearchArgs &a, WarpArea *w) {
    const unsigned FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31, nb = w->n_big, nh = w->n_hit;
    ExtEntry *el = (ExtEntry *)w->dbuf;          // free between rounds
    if (lane == 0) w->n_ext = 0;
    __syncwarp();
    for (uint32_t b = 0; b < nb; b += 32) {
        const bool have = b + lane < nb;
        uint32_t item = 0, sq = 0;
        if (have) sq = extend_big<COH>(a, w->big[b + lane], el, &w->n_ext, item);
        const uint32_t it0 = __shfl_sync(FULL, item, 0);
        if (__all_sync(FULL, !have || item == it0)) {
            sq = __reduce_add_sync(FULL, sq);
            if (lane == 0) count_global(a, it0, 0, sq, 0);
        } else if (have) {
            count_global(a, item, 0, sq, 0);
        }
    }
    if (lane < min(nh, (uint32_t)EXCAP)) record_ext(a, el, &w->n_ext, w->hit_jid[lane], w->hit_u[lane]);
    __syncwarp();
    if (lane == 0) {
        if (nh > (uint32_t)EXCAP) raise_capacity(a.status, E_EXTLIST, 4, nh, EXCAP, 0);
        if (w->n_ext) report_warp_exts<COH>(a, el, min(w->n_ext, (uint32_t)EXTCAP));
        w->n_hit = w->n_big = 0;
    }
    __syncwarp();
}

// Queue entries [first, first+count), two per lane (their chains of double arithmetic overlap): those
// with 0 < e = u^2 - A not in the 4-set are the reference's ext_sqrt (s4.c:195-198) and are
// square-tested (s4.c:199-203).
__device__ __forceinline__ void process_queue(WarpArea *w, uint32_t first, uint32_t count, int lane,
                                              WarpCounters &cnt) {
    uint32_t jl[2];
    uint64_t u[2], u2[2];
    bool hit[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const uint32_t at = lane + 32 * k;
        const uint64_t ent = w->q[first + (at < count ? at : 0)];
        jl[k] = (uint32_t)(ent >> 58);
        u[k] = ((ent & W_SUM) - 32) >> 1;                                        // below 2^44
        u2[k] = u[k] * u[k];                                                     // mod 2^64
        const EJob &E = w->job[jl[k]];
        const uint64_t A = E.A;
        const uint4 ro = *(const uint4 *)&E.rA0;
        const int64_t d1 = E.d1;
        const uint32_t ul = (uint32_t)u[k];
        // u below 2^32: e > 0 iff u2 > A; e = A iff u2 = 2A; e another member iff u one of A's roots
        const bool test = at < count && ((u[k] >> 32) != 0 || (u2[k] > A && u2[k] != 2 * A && ul != ro.x &&
                                                               ul != ro.y && ul != ro.z));
        const bool here = ro.w == cnt.item;
        cnt.sqrt_ += test && here;
        if (test && !here) atomicAdd(&w->job[jl[k]].nsq, 1u);
        hit[k] = is_square_near(u[k], d1, u2[k] + (uint64_t)d1) && test;
    }
#pragma unroll
    for (int k = 0; k < 2; k++)
        if (hit[k]) {                                                            // rare
            const int64_t d2 = w->job[jl[k]].d2;
            if (is_square_near(u[k], d2, u2[k] + (uint64_t)d2)) {
                const uint32_t slot = atomicAdd(&w->n_hit, 1u);
                if (slot < EXCAP) {
                    w->hit_u[slot] = u[k];
                    w->hit_jid[slot] = w->jid[jl[k]];
                }
            }
        }
}

// Runs rounds until rare_work is due (true), or the queue is drained or an error is raised (false).
template <bool RING>
__device__ __forceinline__ bool engine_rounds(const SearchArgs &a, WarpArea *w, int lane) {
    const unsigned FULL = 0xffffffffu;
    WarpCounters cnt;
    bool pending = w->pend >> lane & 1u, drained = false, took = false, more = false;
    bool rel = RING && (w->rel >> lane & 1u);
    uint64_t mypos = RING ? w->q[lane] : 0;
    auto release = [&]() {                     // finished 4-sets hand their slots back, after their report
        const unsigned rm = __ballot_sync(FULL, rel);
        if (rel) ring_release(a, mypos);
        rel = false;
        if (lane == 0 && rm) atomicAdd(&a.status->q_freed, (ull)__popc(rm));
    };
    if (RING) release();

    // Rounds: every lane without a 4-set takes the next one from the queue; a lane whose divisor lists
    // did not fit keeps its 4-set, sets it up again and goes first in the next round's placement.
    for (;;) {
        const bool old = pending;
        if (!drained) {
            const bool need = !pending && (uint32_t)lane < w->quota;
            const unsigned m = __ballot_sync(FULL, need);
            const uint32_t n = (uint32_t)__popc(m), rank = (uint32_t)__popc(m & ((1u << lane) - 1u));
            int stop = 0;
            if (RING) {
                uint64_t base = 0;
                uint32_t got = 0;
                if (lane == 0) {
                    if (m) base = ring_claim(a, n, &got);
                    stop = *(volatile ull *)&a.status->err != 0ull;
                }
                base = __shfl_sync(FULL, base, 0);
                got = __shfl_sync(FULL, got, 0);
                stop = __shfl_sync(FULL, stop, 0);
                if (stop) break;                                         // warp-uniform
                if (got < n) drained = true;                             // the ring is empty for now
                if (need && rank < got && ring_wait_ready(a, base + rank)) {
                    pending = true;
                    mypos = base + rank;
                    w->jid[lane] = (uint32_t)(mypos & a.ring_mask);
                }
                took |= pending;
            } else {
                const uint32_t cur = w->st_cur, rem = w->st_rem, size = w->stretch;
                bool last = w->last != 0;
                uint32_t nx = 0, avail = 0;
                if (rem < n && !last) {                                  // a new stretch behind the old one
                    if (lane == 0) {
                        nx = w->claimed + atomicAdd(&a.status->ext_next, size);
                        stop = *(volatile ull *)&a.status->err != 0ull;
                    }
                    nx = __shfl_sync(FULL, nx, 0);
                    stop = __shfl_sync(FULL, stop, 0);
                    if (stop) break;                                     // warp-uniform
                    avail = nx < w->njobs ? min(size, w->njobs - nx) : 0u;
                    last = avail < size;
                }
                if (need && rank < rem + avail) {
                    pending = true;
                    w->jid[lane] = rank < rem ? cur + rank : nx + (rank - rem);
                }
                const uint32_t used = min(n, rem + avail);
                __syncwarp();                                            // read by all
                if (lane == 0) {
                    w->st_cur = used < rem ? cur + used : nx + (used - rem);
                    w->st_rem = rem + avail - used;
                    w->last = last;
                }
                drained = last && rem + avail == used;                   // warp-uniform
            }
        }
        // ---- phase A: one 4-set per lane
        LaneJob J;
        J.item = J.ncand = J.nd = 0;
        J.big = false;
        const bool mine = pending;
        if (pending) pending = job_setup<RING>(a, w->jid[lane], J, w, lane);
        const bool fresh = pending && !old;                              // counted once
        if (pending && J.big) {                                          // rare
            w->big[atomicAdd(&w->n_big, 1u)] = w->jid[lane];             // fewer than 32 are there
            pending = false;
        }
        if (RING && mine && !pending) rel = true;
        cnt.add(a, w, lane, fresh, J.item, J.ncand, 0, J.nd);
        const bool round = __any_sync(FULL, pending);
        if (round) {
            // place the factored divisor lists of as many pending lanes as fit: lanes left over
            // from the last round first, then the new ones, each in lane order
            const uint32_t want = pending ? J.L + J.H : 0;
            uint32_t tot_old = 0, tot_new, base = 0;
            if (__any_sync(FULL, old)) base = warp_prefix(old ? want : 0, lane, tot_old);
            const uint32_t bn = warp_prefix(old ? 0 : want, lane, tot_new);
            if (!old) base = tot_old + bn;
            const bool fits = pending && base + want <= (uint32_t)DCAP;
            if (fits) {
                w->job[lane].geo |= base << 22;
                gen_list(w->dbuf + base, w->fp, lane, J.slots & 0xFFu, J.slots >> 8 & 0xFFu);      // rows: L entries
                gen_list(w->dbuf + base + J.L, w->fp, lane, J.slots >> 16 & 0xFFu, J.slots >> 24); // H entries
            }
            RowPlan plan;
            plan_rows(fits ? J.rows : 0, J.L, w->order, lane, plan);
            // ---- phase B: 32 rows at a time, one per lane, CPT candidates of each per turn
            uint32_t qn = 0;
            for (uint32_t g0 = 0; g0 < plan.total; g0 += 32) {
                uint32_t r;
                const uint32_t jl = row_job(plan, g0, lane, r);
                const ulonglong2 mm = *(const ulonglong2 *)&w->job[jl].m63;
                const uint2 jj = *(const uint2 *)&w->job[jl].m64;        // m64, geo
                Row row;
                row_start(jj.y, r, g0 + lane < plan.total, w->dbuf, row);
                const int turns = (int)__reduce_max_sync(FULL, (unsigned)row.len);
                const uint64_t tag = (uint64_t)jl << 58 | 32u;
#pragma unroll 1
                for (int l = 0; l < turns; l += CPT) {
                    uint64_t v[CPT];
                    bool ok[CPT];
                    const unsigned below = (1u << lane) - 1u;
#pragma unroll
                    for (int k = 0; k < CPT; k++) {
                        const uint32_t p = candidate(row.xf[k], row.xg[-k], row.fy, row.gy, tag, jj.x, mm.x, mm.y, v[k]);
                        ok[k] = l + k < row.len && (p & 1u);
                    }
                    row.xf += CPT;
                    row.xg -= CPT;
#pragma unroll
                    for (int k = 0; k < CPT; k++) {
                        const unsigned m = __ballot_sync(FULL, ok[k]);
                        if (ok[k]) w->q[qn + __popc(m & below)] = v[k];
                        qn += __popc(m);
                    }
                    // the queue is emptied 64 at a time, and whole after the round's last turn
                    const uint32_t least = l + CPT >= turns && g0 + 32 >= plan.total ? 1u : 64u;
                    while (qn >= least) {
                        const uint32_t n = min(qn, 64u);
                        qn -= n;
                        __syncwarp();
                        process_queue(w, qn, n, lane, cnt);
                        __syncwarp();
                    }
                }
            }
            const uint32_t it = w->job[lane].item;
            const bool other = fits && it != cnt.item;                   // counted with its 4-set
            if (__any_sync(FULL, other)) cnt.add(a, w, lane, other, it, 0, w->job[lane].nsq, 0);
            if (fits) pending = false;
            if (RING && fits) rel = true;
        }
        __syncwarp();
        const bool end = !round && drained;                              // warp-uniform
        more = w->n_hit || w->n_big >= (RING || end ? 1u : 32u);         // warp-uniform
        __syncwarp();                                                    // read by all
        if (more) break;
        if (RING) release();
        if (end) break;
    }
    cnt.flush(a, w, lane);
    const unsigned pm = __ballot_sync(FULL, pending), rm = __ballot_sync(FULL, rel);
    const bool tm = __any_sync(FULL, took);
    if (RING) w->q[lane] = mypos;
    if (lane == 0) {
        w->pend = pm;
        w->rel = rm;
        w->took |= tm;
    }
    __syncwarp();
    return more;
}

// The engine loop of one warp.  Linear (RING false): the batch's queue [0, njobs), filled before
// the launch, taken in stretches of `stretch` 4-sets; the loop ends when it is drained.  RING: the
// persistent kernel's ring; positions are claimed below q_tail and waited for until published, each
// finished 4-set's slot is handed back after the round's report, and the loop ends when a claim finds
// the ring empty and no lane holds a 4-set.  quota: lanes that hold a 4-set (32 unless the queue is too
// short to fill every warp of the launch; the candidates of few 4-sets are still walked by all
// lanes).  The first `claimed` stretches belong to the warps in order, this one is number `first`.  Returns
// whether the warp took any 4-set.
template <bool RING>
__device__ __forceinline__ bool engine_loop(const SearchArgs &a, WarpArea *w, int lane, uint32_t njobs, uint32_t quota,
                                            uint32_t stretch, uint32_t first, uint32_t claimed) {
    if (lane == 0) {
        w->n_hit = w->n_big = 0;
        w->pend = w->rel = w->took = 0;
        w->njobs = njobs; w->quota = quota; w->stretch = stretch;
        // the warp's first stretch is its own place in the grid (a short queue needs no atomics, whose turns
        // on one address took 12 of a small call's 29 us), the later ones are claimed behind them
        const uint32_t at = min(first * stretch, njobs);
        w->st_cur = at;
        w->st_rem = RING ? 0 : min(stretch, njobs - at);
        w->last = (uint64_t)claimed * stretch >= njobs;
        w->claimed = claimed * stretch;
    }
    if (lane < ICACHE) w->ic[lane].item = NO_ITEM;
    __syncwarp();
    while (engine_rounds<RING>(a, w, lane)) rare_work<RING>(a, w);
    if (lane < ICACHE && w->ic[lane].item != NO_ITEM)
        count_global(a, w->ic[lane].item, w->ic[lane].cand, w->ic[lane].sqrt_, w->ic[lane].mdiv);
    const bool took = w->took != 0;
    __syncwarp();
    return took;
}

__global__ void __launch_bounds__(EBS, 3) extend_jobs(const __grid_constant__ SearchArgs a) {
    extern __shared__ __align__(16) unsigned char esmem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    WarpArea *w = (WarpArea *)(esmem + (size_t)wid * sizeof(WarpArea));
    // An overflown queue (more reserved than it holds) ends with unwritten records; its search is repeated.  (A look at
    // the error word instead, which covers that too, is a second load: 2 of 34 us of the smallest calls.)
    const ull queued = *(volatile ull *)&a.status->n_jobs;
    if (queued == 0 || queued > a.jobs_cap) return;
    const uint32_t njobs = (uint32_t)queued;
    const uint32_t warps = gridDim.x * EWARPS;
    const uint32_t quota = min((njobs + warps - 1) / warps, 32u);                // 1 at least
    // a stretch is a 32nd of a warp's share, 32 to 256 4-sets (one atomic each)
    const uint32_t stretch = quota < 32 ? quota : 32u * min(max(njobs / (warps * 1024), 1u), 8u);
    engine_loop<false>(a, w, lane, njobs, quota, stretch, blockIdx.x * EWARPS + wid, warps);
}

// ================================================================== the persistent kernel

// One launch for a whole call.  Every CTA (PBS threads, three per SM) loops over two roles:
// producing -- claim the next group of SUPER_K tiles of 2^13 S (highest cost first), run P1-P5
// and write the 4-sets into the ring -- or consuming -- its warps run the extension engine on
// 4-sets claimed from the ring.  A CTA consumes while at least CONSUME_AT 4-sets are queued,
// produces while tiles are left and the ring is less than half full, and ends when every tile is
// produced and every 4-set claimed.  The roles switch with hysteresis: a CTA turns to the engine
// when ring_high 4-sets are queued, and its warps keep claiming until fewer than ring_low are
// left (while tiles remain), so that every warp has 4-sets to pool, claims take the add path,
// and role changes are rare next to the work between them.  A call of any number of subranges is
// one launch.  The tile layout and the engine's warp areas share the CTA's shared memory (one
// role at a time).
constexpr int PTL = 13;
constexpr int PWARPS = PBS / 32;
// the tile state of the producing role sits in the dynamic area too, after the tile layout and
// the group's list counters, so that the kernel's static shared memory stays a few words and three
// CTAs (each with the 1 KB the hardware reserves per block) fit in the SM's 228 KB
constexpr size_t P_TS_OFF = (TileLayout<PTL>::OFF_ELIST + SUPER_K * sizeof(uint32_t) + 15) & ~(size_t)15;
static_assert(P_TS_OFF + sizeof(TileShared) <= PWARPS * sizeof(WarpArea),
              "the tile layout and tile state fit in the engine's warp areas");
static_assert(PWARPS * sizeof(WarpArea) + 1024 + 128 <= 228 * 1024 / 3, "three persistent CTAs per SM");

__global__ void __launch_bounds__(PBS, 3) search_persist(const __grid_constant__ SearchArgs a) {
    using L = TileLayout<PTL>;
    extern __shared__ __align__(16) unsigned char smem[];
    TileShared &ts = *reinterpret_cast<TileShared *>(smem + P_TS_OFF);
    __shared__ unsigned long long s_idle0;
    __shared__ RingSpan s_span;
    __shared__ unsigned int s_claim;
    __shared__ int s_role, s_busy;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint64_t *lists = a.raw + (size_t)blockIdx.x * SUPER_K * a.raw_cap;
    uint32_t *raw_n = (uint32_t *)(smem + L::OFF_ELIST);
    if (tid == 0) s_idle0 = 0;
    for (;;) {
        if (tid == 0) {
            int role = 2;                                    // 0 end, 1 produce, 2 consume
            if (ld_vol(&a.status->err) != 0ull) {
                role = 0;
            } else {
                const ull tail = ld_vol(&a.status->q_tail), head = ld_vol(&a.status->q_head);
                const ull freed = ld_vol(&a.status->q_freed), pub = ld_vol(&a.status->q_pub);
                const uint32_t tn = ld_vol(&a.status->tile_next);
                const long long queued = (long long)(tail - head);
                if ((long long)(pub - head) >= (long long)a.ring_high || (tn >= a.n_tiles && queued > 0)) {
                    role = 2;
                } else if (tn < a.n_tiles && tail - freed < (a.jobs_cap >> 1)) {
                    const uint32_t c = atomicAdd(&a.status->tile_next, SUPER_K);
                    if (c < a.n_tiles) {
                        role = 1;
                        s_claim = c;
                    }
                } else if (tn >= a.n_tiles && ld_vol(&a.status->q_produced) >= a.n_tiles && queued <= 0) {
                    role = 0;
                }
            }
            s_role = role;
            s_busy = 0;
        }
        __syncthreads();
        const int role = s_role;
        if (role == 0) break;                                // block-uniform
        if (role == 1) {
            const uint32_t cn = produce_group<PTL, PBS>(a, ts, smem, s_claim, lists, raw_n, s_span);
            if (tid == 0) {
                __threadfence();
                atomicAdd(&a.status->q_produced, (ull)cn);
                s_idle0 = 0;
            }
        } else {
            WarpArea *w = (WarpArea *)(smem + (size_t)wid * sizeof(WarpArea));
            if (engine_loop<true>(a, w, lane, 0u, 32u, 0u, 0u, 0u) && lane == 0) s_busy = 1;
            __syncthreads();
            if (tid == 0) {
                if (s_busy) {
                    s_idle0 = 0;
                } else {                                     // nothing to take: wait a little, bounded
                    const uint64_t t = gtimer();
                    if (!s_idle0) s_idle0 = t;
                    else if (t - s_idle0 > 2 * WAIT_NS) raise_error(a.status, E_TIMEOUT, 4);
                    __nanosleep(1000);
                }
            }
        }
        __syncthreads();
    }
}

// One consumer wait on position 0 of a one-slot ring that nothing publishes, with tiles still
// unproduced: the wait must give up after WAIT_NS and record E_TIMEOUT (ps4_check_ring_wait).
__global__ void ring_wait_probe(const SearchArgs a, unsigned long long *out) {
    const uint64_t t0 = gtimer();
    out[0] = ring_wait_ready(a, 0) ? 1ull : 0ull;
    out[1] = gtimer() - t0;
}

// The owners of all pairs, as one warp of the tile kernel finds them (ps4_check_pair_owners).
__global__ void pair_owner_probe(const uint32_t *pbase, uint32_t n_is, unsigned long long *out) {
    const uint32_t total = pbase[n_is];
    uint32_t lo0 = 0, lo, base;
    for (uint32_t g = 0; g < total; g += 32) {
        pair_owner(pbase, n_is, g, threadIdx.x, lo0, lo, base);
        if (g + threadIdx.x < total) out[g + threadIdx.x] = (ull)base << 32 | lo;
    }
}

// seq[i] = i: every slot free for its first lap
__global__ void ring_init(uint32_t *seq, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        seq[i] = (uint32_t)i;
}

// ================================================================== launchers

// the tile kernel's full residency for 2^TL-S tiles
int gen_grid(int num_sms, unsigned TL) { return num_sms * (BS / gen_threads(TL)) * 2; }
int ext_grid(int num_sms) { return num_sms * 3; }

template <int TL, int NT>
static int launch_gen_tl(const SearchArgs &a, int grid, uint32_t cluster, cudaStream_t s) {
    const size_t smem = TileLayout<TL>::OFF_ELIST;       // up to the extension-list area, which it does not use
    const auto kernel = cluster > 2 ? gen_jobs<TL, NT, true> : gen_jobs<TL, NT, false>;
    const int e = (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = cluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, a);
}

// up to this many tiles each has an SM to itself, and CTAs of 1024 threads
constexpr uint64_t FEW_TILES = 128;

// Launch shape of the tile kernel.  A group's scan visits 0.29 sqrt(S) q, as much work as s tiles
// (34,000 q cost about what a tile of 2^13 S does).
//  * Cluster: 8 CTAs where scans weigh, i.e. for high S and for calls with few tiles, else 2.  Measured,
//    tile kernel with 8 / 2 / 1 CTAs: [1,1e10) 98.9 / 80.9 / 80.0 ms; 2e8 S at 1e12 2.79 / 3.05 / 3.82; 3e7 S at
//    1.2e13 1.05 / 1.65 / 2.45; 64 subranges below 1e11 10.3 / 9.0 / 9.3; 2e4 S at 4e11 0.042 / 0.066 / 0.096
//    (all with parts read one by one; side by side, as eight are now, 2.57, 0.99 and 0.040 at 1e12, 1.2e13 and 4e11).
//  * Segments of fewer tiles than a cluster has CTAs share no more than their own scan: a cluster of c takes s / c +
//    ceil(t / c) for one of t tiles, and K clusters take segs / K rounds, half of the last one idle.  Where that promises a
//    fifth at least, the c with the least of it.  Tile kernel, one scan per CTA and 16 tiles / the rule above / this
//    one: 8000 subranges of 8000 S at 1e12 8.50 / 9.39 / 6.87 ms, 40000 of 30 S at 1e7 1.02 / 1.67 / 0.83, 1000 of 8000 S at 1e9
//    1.14 / 0.44 / 0.10, 200 of 1000 S at 1e7 0.31 / 0.11 / 0.03.  (Without the fifth: 200 of 30000 S at 1e12 0.40 -> 0.54.)
//  * Tiles per claim: n tiles in groups of G on K clusters take n + s n / G of work and about G K / 2 of
//    idling at the end, least at G = sqrt(2 n s / K).
// `grid`: the CTAs that the lists of a.raw are sized for; whole clusters of them are launched, no more
// than there are tiles to take.
int launch_gen(SearchArgs a, int grid, void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    const double n = (double)std::max<uint64_t>(a.n_tiles, 1);
    const double scan = 0.29 * std::sqrt((double)a.s_top) / (34e3 * std::ldexp(1.0, (int)a.log2_tile - 13));
    uint32_t cl = n < 11e3 * scan || grid < 16 ? GEN_CLUSTER : 2;
    const double segs = a.n_items, t = n / segs;
    if (segs > 1 && t < GEN_CLUSTER) {
        auto cost = [&](uint32_t c) {
            const double rounds = segs / std::min(std::max(grid / (int)c, 1) * 1.0, std::ceil(n / c));
            return (rounds > 1 ? rounds + 0.5 : 1.0) * (scan / c + std::ceil(t / c));
        };
        double least = 0.8 * cost(cl);
        for (const uint32_t c : {1u, 2u, GEN_CLUSTER})
            if (cost(c) < least) { least = cost(c); cl = c; }
    }
    const uint64_t fit = std::max<uint64_t>((uint64_t)grid / cl, 1), want = ((uint64_t)n + cl - 1) / cl;
    const uint64_t K = std::min(fit, want), ctas = K * cl;
    const double G = std::min(std::sqrt(2 * n * scan / (double)K), std::ceil(n / (double)K));
    a.group = (uint32_t)std::min<double>(std::max<double>(G, cl), cl * a.raw_lists);
    // a warp's reservations: a sixteenth of its expected share of about 0.2 4-sets per S, so that the
    // empty records at the end stay below a few percent, 128 at most (one atomic per 128 4-sets)
    const bool few = a.log2_tile == 12 && a.n_tiles <= FEW_TILES;
    const double warps = (double)ctas * (few ? 1024 : gen_threads(a.log2_tile)) / 32;
    const double share = 0.2 * std::ldexp(n, (int)a.log2_tile) / warps;
    a.chunk = (uint32_t)std::min<double>(std::max<double>(share / 16, 8), 128);
    switch (a.log2_tile) {
        case 12:
            if (few) return launch_gen_tl<12, 1024>(a, (int)ctas, cl, s);
            return launch_gen_tl<12, gen_threads(12)>(a, (int)ctas, cl, s);
        case 13: return launch_gen_tl<13, gen_threads(13)>(a, (int)ctas, cl, s);
        default: return launch_gen_tl<14, gen_threads(14)>(a, (int)ctas, cl, s);
    }
}

// resident CTAs per SM of the persistent kernel (three by design; fewer if the device says so, so
// that no CTA of the grid waits for another to exit)
int persist_ctas_per_sm() {
    int n = 0;
    if (cudaFuncSetAttribute(search_persist, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(PWARPS * sizeof(WarpArea))) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, search_persist, PBS, PWARPS * sizeof(WarpArea)) !=
            cudaSuccess)
        n = 1;
    return n < 1 ? 1 : (n > 3 ? 3 : n);
}

int launch_persist(const SearchArgs &a, int grid, void *stream) {
    const size_t smem = PWARPS * sizeof(WarpArea);
    cudaFuncSetAttribute(search_persist, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    search_persist<<<grid, PBS, smem, (cudaStream_t)stream>>>(a);
    return (int)cudaGetLastError();
}

int launch_ring_wait_probe(const SearchArgs &a, unsigned long long *out, void *stream) {
    ring_wait_probe<<<1, 1, 0, (cudaStream_t)stream>>>(a, out);
    return (int)cudaGetLastError();
}

int launch_pair_owner_probe(const uint32_t *pbase, uint32_t n_is, unsigned long long *out) {
    pair_owner_probe<<<1, 32>>>(pbase, n_is, out);
    return (int)cudaGetLastError();
}

int launch_ring_init(uint32_t *seq, uint64_t n, void *stream) {
    ring_init<<<1184, 256, 0, (cudaStream_t)stream>>>(seq, n);
    return (int)cudaGetLastError();
}

int launch_ext(const SearchArgs &a, int grid, void *stream) {
    const size_t smem = EWARPS * sizeof(WarpArea);
    cudaFuncSetAttribute(extend_jobs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    extend_jobs<<<grid, EBS, smem, (cudaStream_t)stream>>>(a);
    return (int)cudaGetLastError();
}

}  // namespace ps4
