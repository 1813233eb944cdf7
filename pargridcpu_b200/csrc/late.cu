// The last levels of a peel (or all levels of a small graph), on the rows that
// are left.
//
// Late in a peel a level is a chain of small rounds, and a round's time is its
// chain of dependent memory accesses, not its work.  So the nodes still alive
// are given ids 0 .. m-1, their rows are copied without the entries that name
// removed nodes, and the rounds run on a form with the shortest chain: an item
// holds its node, chunk and columns, a row's place and length are one load, an
// entry is (neighbour, layer) with no division, and no alive test stands before
// a decrement.
//
// The alive test is not needed for the result.  A degree field counts at
// least the neighbours not yet expanded, so it never falls below 0.  A layer's
// degree falls from K+1 to K while the level is K at most once (degrees only
// fall and levels only rise), so after its removal a column's count falls by
// at most L: it starts below lambda, as the layers that could still do so, or
// at LT_DEAD (columns removed before, whose degrees the peel stopped keeping),
// and neither falls below 0 nor reaches lambda.
#include <algorithm>

#include "device.h"
#include "peel_common.h"

namespace fc {

constexpr uint32_t LT_CHUNK = LATE_CHUNK;
constexpr uint32_t LT_FILL_LONG = 4096;   // longer source rows are a block's to copy
// An item: node, columns (and LT_OWNER on a row's first chunk), the chunk's
// first entry and entries.
constexpr uint32_t LT_OWNER = 0x80000000u;
// With more than LT_FILTER items a warp a round is bound by its decrements
// (125 G/s at most), and testing whether a neighbour is still alive saves half
// of them; with fewer the test is one access more in the chain (180,001 nodes,
// 17 layers: 26.8 against 28.0 ms).
constexpr uint32_t LT_FILTER = 1;
// With up to LT_DIRECT items a block, removals go straight to the list instead
// of through the block's stage: two block barriers less (hub graph of 2.5M
// nodes, 4 layers: 15.8 against 16.1 ms; 8 and 32 measure the same).
constexpr uint32_t LT_DIRECT = 16;
// Levels with at most LT_SMALL nodes run on blocks of LT_SMALL_T threads: a
// barrier of fewer warps (5.1 against 6.1 us a small round at 1024 threads; 256
// threads are too few where the rounds are not small: 25.9 against 24.5 ms).
constexpr uint32_t LT_SMALL = 16384;
constexpr int LT_SMALL_T = 512;
constexpr uint32_t LT_NONE = 0xFFFFFFFFu;   // no entry (a node has at most 20 bits)
constexpr u64 LT_DEAD = 0x4000400040004000ull;
// an entry: neighbour << 9 | layer
constexpr uint32_t LT_LAYER_BITS = 9;
static_assert(LATE_MAX_LAYERS == 1u << LT_LAYER_BITS, "");

struct LateJob {
    uint32_t L, Q, col0, G;      // single segment: layers, words per layer; G: count words per node
    const uint2* row;            // m: first entry, entries
    const uint2* meta;           // several segments: first degree word, Q | col0 << 8
    const uint32_t* adj;
    // G planes of `plane` words, one per word of four columns, a node's layers
    // side by side in each: as the higher columns empty, their planes leave L2
    // to the others (interleaved, 180,001 nodes x 17 layers is 122 MB to the
    // end, and a decrement a random atomic at 56 G/s instead of 125).
    u64* deg;
    uint64_t plane;
    u64* cnt;                    // m * G
    uint32_t* M;                 // m: columns not yet expanded
    const uint32_t* x_of;
    const uint32_t* node_seg;
    uint32_t* alive[2];
    uint4* q[2];
    uint32_t q_cap, cap;
    LateCtl* ctl0;               // the first launch's
    LateCtl* ctl;                // this launch's: where it starts, its counters
    SegP seg0;
    const SegP* segs;
    uint32_t max_level;
    uint32_t stop_alive;         // leave levels with this many nodes or fewer to the next launch
    uint64_t timeout_ns, deadline_ns;
    unsigned long long* trace;
    uint32_t trace_levels;
};

struct LateView {
    uint32_t err, items, alive;
};

template <bool MULTI>
__device__ __forceinline__ uint2 lt_meta(const LateJob& j, uint32_t i) {
    if (!MULTI) return make_uint2(i * j.L, j.Q | (j.col0 << 8));
    return __ldg(j.meta + i);
}

// chunk ch of the row r of node x, removed in the columns cols
__device__ __forceinline__ uint4 lt_item(uint32_t x, uint32_t cols, uint2 r, uint32_t ch) {
    const uint32_t o = ch * LT_CHUNK;
    return make_uint4(x, ch ? cols : cols | LT_OWNER, r.x + o, min(LT_CHUNK, r.y - o));
}

// A block's part of a list that all blocks write: collected in shared memory
// and appended with one reservation at the end of the step.  Counters that the
// whole grid adds to are the limit otherwise: atomics on one address take
// turns, about 1.3 ns each.
constexpr uint32_t LT_STAGE = 1536, LT_STAGE_ALIVE = 1024;
template <class T, uint32_t CAP>
struct Stage {
    T item[CAP];
    uint32_t n;
};
struct LateBlock {
    Stage<uint4, LT_STAGE> q;
    Stage<uint32_t, LT_STAGE_ALIVE> alive;
    uint32_t base[2];
    LateView sv;
};

// Reserves `want` places for each lane; the lane's k-th thing then goes to
// place at + k (stage_put).  `at` counts staged places; what lies past the
// stage's end has its places in the list itself, from `over`.
template <class T, uint32_t CAP, class C>
__device__ __forceinline__ uint32_t stage_reserve(Stage<T, CAP>& st, C* count, uint32_t want,
                                                  uint32_t* over, bool direct) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t in = want;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, in, o);
        if (lane >= (uint32_t)o) in += y;
    }
    uint32_t at = 0, ov = 0;
    if (lane == 31) {
        // (a light round's few go to the list at once: no barrier in between)
        at = direct ? CAP : atomicAdd(&st.n, in);
        if (at + in > CAP) {
            const uint32_t from = max(at, CAP);
            ov = (uint32_t)atomicAdd(count, (C)(at + in - from)) - from;  // place p of the list is ov + p
        }
    }
    *over = __shfl_sync(0xffffffffu, ov, 31);
    return __shfl_sync(0xffffffffu, at, 31) + in - want;
}
template <class T, uint32_t CAP>
__device__ __forceinline__ void stage_put(const LateJob& j, Stage<T, CAP>& st, T* list, uint32_t cap,
                                          uint32_t at, uint32_t over, T v) {
    if (at < CAP) st.item[at] = v;
    else if (over + at < cap) list[over + at] = v;
    else atomicExch(&j.ctl->err.v, PEEL_ERR_QUEUE);
}
template <class T, uint32_t CAP>
__device__ __forceinline__ void stage_copy(const LateJob& j, const Stage<T, CAP>& st, uint32_t n,
                                           T* list, uint32_t cap, uint32_t base) {
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        if (base + i < cap) list[base + i] = st.item[i];
        else atomicExch(&j.ctl->err.v, PEEL_ERR_QUEUE);
    }
}
// The block's staged items and survivors to their lists, both reservations at
// once; all threads of the block call it.
__device__ __forceinline__ void stage_flush(const LateJob& j, LateBlock& sb, u64* tail, uint4* q,
                                            uint32_t* kept, uint32_t* alive) {
    __syncthreads();
    const uint32_t nq = min(sb.q.n, LT_STAGE), na = min(sb.alive.n, LT_STAGE_ALIVE);
    if (!(nq | na)) return;  // the same on every thread
    if (threadIdx.x == 0) {
        const uint32_t bq = nq ? (uint32_t)atomicAdd(tail, (u64)nq) : 0u;
        sb.base[1] = na ? atomicAdd(kept, na) : 0u;
        sb.base[0] = bq;
    }
    __syncthreads();
    stage_copy(j, sb.q, nq, q, j.q_cap, sb.base[0]);
    stage_copy(j, sb.alive, na, alive, j.cap, sb.base[1]);
    __syncthreads();
    if (threadIdx.x == 0) sb.q.n = sb.alive.n = 0;
}

// The nch items of each lane's node x (row r), removed in the columns cols, at
// the places reserved.  All 32 lanes call it together: long rows by the whole
// warp.
__device__ __forceinline__ void lt_put(const LateJob& j, LateBlock& sb, uint4* out, uint32_t x,
                                       uint32_t cols, uint2 r, uint32_t nch, uint32_t at,
                                       uint32_t over) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t todo = __ballot_sync(0xffffffffu, nch > 4); todo; todo &= todo - 1) {
        const uint32_t src = __ffs(todo) - 1;
        const uint32_t rx = __shfl_sync(0xffffffffu, x, src);
        const uint32_t rc = __shfl_sync(0xffffffffu, cols, src);
        const uint2 rr = make_uint2(__shfl_sync(0xffffffffu, r.x, src),
                                    __shfl_sync(0xffffffffu, r.y, src));
        const uint32_t ra = __shfl_sync(0xffffffffu, at, src);
        const uint32_t rn = __shfl_sync(0xffffffffu, nch, src);
        for (uint32_t c = lane; c < rn; c += 32)
            stage_put(j, sb.q, out, j.q_cap, ra + c, over, lt_item(rx, rc, rr, c));
    }
    if (nch <= 4)
        for (uint32_t c = 0; c < nch; c++)
            stage_put(j, sb.q, out, j.q_cap, at + c, over, lt_item(x, cols, r, c));
}

__device__ __forceinline__ uint32_t lt_chunks(uint32_t len) {
    return len ? (len + LT_CHUNK - 1) / LT_CHUNK : 1u;
}

// SCAN(k) (peel.cu) over the alive list.
template <bool MULTI>
__device__ __forceinline__ void lt_scan(const LateJob& j, LateBlock& sb, uint32_t k, const uint32_t* src,
                                        uint32_t n, uint32_t* out, uint32_t* out_cnt, u64* tail,
                                        uint4* qout) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t G = j.G, npw = 32u / G;
    const uint32_t sub = lane / G, q = lane - sub * G, gbase = sub * G;
    const uint32_t nwarps = blockDim.x >> 5;
    const uint32_t nw = gridDim.x * nwarps, gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const uint32_t t2 = (k + 1) | ((k + 1) << 16);
    const uint32_t groups = (n + npw - 1) / npw;
    const bool direct = groups <= LT_DIRECT * gridDim.x;
    for (uint32_t b = gw; b < groups; b += nw) {
        const uint32_t idx = b * npw + sub;
        bool live = sub < npw && idx < n;
        const uint32_t x = live ? src[idx] : 0u;
        const uint32_t m = live ? j.M[x] : 0u;
        const uint2 mt = lt_meta<MULTI>(j, x);
        const uint32_t Q = mt.y & 0xFFu, col0 = mt.y >> 8;
        live = live && m;
        uint32_t L = j.L;
        if (MULTI) L = __ldg(&j.segs[j.node_seg[x]].L);
        const uint32_t m4 = live && q < Q ? (m >> (4 * q)) & 15u : 0u;
        u64 c4 = 0;
        if (m4 && k < FIELD_MAX) {
            const u64* dw = j.deg + q * j.plane + mt.x;
#pragma unroll 4
            for (uint32_t l = 0; l < L; l++) c4 += geq4(dw[l], t2);
        }
        uint32_t r4 = 0;
#pragma unroll
        for (uint32_t f = 0; f < 4; f++)
            if (((m4 >> f) & 1u) && ((uint32_t)(c4 >> (16 * f)) & 0xFFFFu) < col0 + 4 * q + f + 1)
                r4 |= 1u << f;
        if (m4) {
            const u64 kept = spread4(m4 & ~r4) * 0xFFFFull;
            j.cnt[(uint64_t)x * G + q] = (c4 & kept) | (LT_DEAD & ~kept);
        }
        if (r4) {
            const SegP g = MULTI ? j.segs[j.node_seg[x]] : j.seg0;
            const uint32_t v = j.x_of[x] - g.xbase;
#pragma unroll
            for (uint32_t f = 0; f < 4; f++)
                if ((r4 >> f) & 1u) g.t[(uint64_t)(4 * q + f) * g.n + v] = k;
        }
        uint32_t rem = 0;
        for (uint32_t t = 0; t < G; t++)
            rem |= __shfl_sync(0xffffffffu, r4, (gbase + t) & 31) << (4 * t);
        const bool lead = live && q == 0;
        const bool keep = lead && (m & ~rem);
        uint32_t nch = 0;
        uint2 r = make_uint2(0, 0);
        if (lead && rem) {
            j.M[x] = m & ~rem;
            r = j.row[x];
            nch = lt_chunks(r.y);
        }
        if (__any_sync(0xffffffffu, keep)) {
            uint32_t over;
            const uint32_t at = stage_reserve(sb.alive, out_cnt, keep ? 1u : 0u, &over, direct);
            if (keep) stage_put(j, sb.alive, out, j.cap, at, over, x);
        }
        if (__any_sync(0xffffffffu, nch != 0)) {
            uint32_t over;
            const uint32_t at = stage_reserve(sb.q, tail, nch, &over, direct);
            lt_put(j, sb, qout, x, rem, r, nch, at, over);
        }
    }
    if (!direct) stage_flush(j, sb, tail, qout, out_cnt, out);
}

// An item and its entries.
struct LateItem {
    uint4 it;
    uint32_t a[4];
};
__device__ __forceinline__ uint4 lt_fetch(const uint4* in, uint32_t i, uint32_t items) {
    return i < items ? in[i] : make_uint4(0, 0, 0, 0);
}
__device__ __forceinline__ void lt_entries_of(const LateJob& j, LateItem& t) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const uint32_t p = 32 * e + (threadIdx.x & 31);
        t.a[e] = p < t.it.w ? __ldg(j.adj + t.it.z + p) : LT_NONE;
    }
}
// drops the entries whose neighbour is left in none of the columns
__device__ __forceinline__ void lt_filter(const LateJob& j, LateItem& t) {
    uint32_t m[4];
#pragma unroll
    for (int e = 0; e < 4; e++)
        m[e] = t.a[e] != LT_NONE ? ld_either(j.M + (t.a[e] >> LT_LAYER_BITS)) : 0u;
#pragma unroll
    for (int e = 0; e < 4; e++)
        if (!(m[e] & t.it.y)) t.a[e] = LT_NONE;  // (no mask has LT_OWNER)
}

// One item by a warp, four entries per lane, their decrements in flight
// together.
template <bool MULTI>
__device__ __forceinline__ void lt_item_run(const LateJob& j, LateBlock& sb, uint32_t k, const LateItem& t,
                                            bool scanned, bool direct, u64* tail, uint4* out) {
    const uint32_t S = t.it.y & ~LT_OWNER;
    uint32_t rb[4] = {0, 0, 0, 0};
    uint2 row[4];
    if (!(S & (S - 1))) {
        // Removed in one column: one word of a neighbour's, one field of it.
        // The atomics take the whole word here too: other items of the round
        // decrement several of its fields at once, and atomics of two widths
        // on the same bytes are not atomic to each other.
        const uint32_t c = __ffs(S) - 1, sh = (c & 3) * 16;
        const u64 minus = 0ull - (1ull << sh);
        u64 old[4], oc[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            old[e] = 0;
            if (t.a[e] != LT_NONE) {
                const uint2 mt = lt_meta<MULTI>(j, t.a[e] >> LT_LAYER_BITS);
                const uint64_t w = (c >> 2) * j.plane + mt.x +
                                   (t.a[e] & ((1u << LT_LAYER_BITS) - 1u));
                old[e] = atomicAdd(j.deg + w, minus);
            }
        }
        // (results are only looked at once all are on their way)
        uint32_t crossed = 0;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            row[e] = make_uint2(0, 0);
            if (t.a[e] == LT_NONE || ((uint32_t)(old[e] >> sh) & 0xFFFFu) != k + 1) continue;
            const uint32_t u = t.a[e] >> LT_LAYER_BITS;
            crossed |= 1u << e;
            row[e] = __ldg(j.row + u);
            oc[e] = atomicAdd(j.cnt + (uint64_t)u * j.G + (c >> 2), minus);
        }
#pragma unroll
        for (int e = 0; e < 4; e++)
            if ((crossed >> e) & 1u)
                if (((uint32_t)(oc[e] >> sh) & 0xFFFFu) ==
                    (lt_meta<MULTI>(j, t.a[e] >> LT_LAYER_BITS).y >> 8) + c + 1)
                    rb[e] = S;
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++) row[e] = make_uint2(0, 0);
        for (uint32_t q = 0; (S >> (4 * q)) != 0; q++) {
            const uint32_t s4 = (S >> (4 * q)) & 15u;
            if (!s4) continue;
            const u64 dec = spread4(s4), kk = all4(k + 1);
            u64 old[4], cross[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                old[e] = 0;
                if (t.a[e] != LT_NONE) {
                    const uint2 mt = lt_meta<MULTI>(j, t.a[e] >> LT_LAYER_BITS);
                    const uint64_t w =
                        q * j.plane + mt.x + (t.a[e] & ((1u << LT_LAYER_BITS) - 1u));
                    old[e] = atomicAdd(j.deg + w, 0ull - dec);
                }
            }
            // (results are only looked at once all are on their way)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                cross[e] = t.a[e] != LT_NONE ? zero4(old[e] ^ kk) & dec : 0ull;
                if (!cross[e]) continue;
                const uint32_t u = t.a[e] >> LT_LAYER_BITS;
                row[e] = __ldg(j.row + u);
                old[e] = atomicAdd(j.cnt + (uint64_t)u * j.G + q, 0ull - cross[e]);
            }
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if (!cross[e]) continue;
                const u64 lm = all4((lt_meta<MULTI>(j, t.a[e] >> LT_LAYER_BITS).y >> 8) + 4 * q) +
                               0x0004000300020001ull;
                rb[e] |= gather4(zero4(old[e] ^ lm) & cross[e]) << (4 * q);
            }
        }
    }
    // one reservation for the item
    if (__any_sync(0xffffffffu, (rb[0] | rb[1] | rb[2] | rb[3]) != 0)) {
        uint32_t want = 0, most = 0, nch[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            nch[e] = rb[e] ? lt_chunks(row[e].y) : 0u;
            want += nch[e];
            most = max(most, nch[e]);
        }
        uint32_t over;
        uint32_t at = stage_reserve(sb.q, tail, want, &over, direct);
        if (__any_sync(0xffffffffu, most > 4)) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                lt_put(j, sb, out, t.a[e] >> LT_LAYER_BITS, rb[e], row[e], nch[e], at, over);
                at += nch[e];
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
                for (uint32_t c = 0; c < nch[e]; c++)
                    stage_put(j, sb.q, out, j.q_cap, at++, over,
                              lt_item(t.a[e] >> LT_LAYER_BITS, rb[e], row[e], c));
        }
    }
    // (the scan has done this for its own removals)
    if ((t.it.y & LT_OWNER) && !scanned && (threadIdx.x & 31) == 0) {
        const uint32_t x = t.it.x;
        atomicAnd(j.M + x, ~S);
        const SegP g = MULTI ? j.segs[j.node_seg[x]] : j.seg0;
        const uint32_t v = j.x_of[x] - g.xbase;
        for (uint32_t b = S; b; b &= b - 1) g.t[(uint64_t)(__ffs(b) - 1) * g.n + v] = k;
    }
}

// The removals of one round: a warp per item.  While an item's decrements are
// in flight, the next item's entries and the one after are on their way.
template <bool MULTI>
__device__ __forceinline__ void lt_expand(const LateJob& j, LateBlock& sb, uint32_t k,
                                          const uint4* in, uint32_t items, bool scanned, u64* tail,
                                          uint4* out) {
    const uint32_t nwarps = blockDim.x >> 5;
    const uint32_t nw = gridDim.x * nwarps, gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    // with several items a warp the grid is short of atomics, not of time
    const bool filter = items > LT_FILTER * nw;  // the same on every warp
    const bool direct = items <= LT_DIRECT * gridDim.x;
    if (gw < items) {
        LateItem cur, nxt;
        cur.it = lt_fetch(in, gw, items);
        nxt.it = lt_fetch(in, gw + nw, items);
        lt_entries_of(j, cur);
        for (uint32_t i = gw; i < items; i += nw) {
            const uint4 after = lt_fetch(in, i + 2 * nw, items);
            lt_entries_of(j, nxt);
            if (filter) lt_filter(j, cur);
            lt_item_run<MULTI>(j, sb, k, cur, scanned, direct, tail, out);
            cur = nxt;
            nxt.it = after;
        }
    }
    if (!direct) stage_flush(j, sb, tail, out, nullptr, nullptr);
}

// Grid barrier with a bounded wait, as in peel.cu; returns the items queued in
// the step (one load tells them and that every block has come).
__device__ __forceinline__ uint32_t lt_barrier(const LateJob& j, uint64_t t_start, u64* word,
                                               const uint32_t* alive, LateView* out) {
    LateCtl* const c = j.ctl;
    __syncthreads();
    if (threadIdx.x == 0) {
        if (blockIdx.x == 0 && past_deadline(t_start, j.deadline_ns))
            atomicCAS(&c->err.v, PEEL_OK, PEEL_ERR_DEADLINE);
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(1ull << 32)
                     : "memory");
        uint64_t t0 = 0;
        u64 w;
        uint32_t err = PEEL_OK;
        for (uint32_t spins = 1;; spins++) {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(word) : "memory");
            if ((uint32_t)(w >> 32) >= gridDim.x) break;
            if ((spins & 255) == 0) {
                const uint64_t now = global_ns();
                if (!t0) t0 = now;
                if (now - t0 > j.timeout_ns) atomicCAS(&c->err.v, PEEL_OK, PEEL_ERR_BARRIER);
                // an error ends the run: some blocks may have left already
                if ((err = ld_relaxed(&c->err.v)) != PEEL_OK) break;
            }
        }
        out->items = (uint32_t)w;
        // the error flag is looked at once a level
        out->err = alive ? ld_relaxed(&c->err.v) : err;
        if (alive) out->alive = ld_relaxed(alive);
    }
    __syncthreads();
    return min(out->items, j.q_cap);  // (past it: PEEL_ERR_QUEUE)
}

template <int T, bool MULTI>
__global__ void __launch_bounds__(T, 1) k_late(const __grid_constant__ LateJob j) {
    __shared__ LateBlock sb;
    LateView& sv = sb.sv;
    LateCtl* const c = j.ctl;
    // the rows are not what their degrees say, or the launch before ended with
    // an error: nothing reads them
    if (j.ctl0->err.v) return;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    const uint64_t t_start = lead ? j.ctl0->t_start : 0;
    uint64_t t_last = lead ? global_ns() : 0, t_scan = 0;
    uint32_t step = 0, level = 0;
    const uint32_t k0 = c->first_level, list0 = c->list;
    uint32_t alive_n = c->m;
    if (threadIdx.x == 0) sb.q.n = sb.alive.n = 0;
    __syncthreads();
    while (alive_n > j.stop_alive) {
        const uint32_t k = k0 + level, la = level % 3;
        if (lead) {  // read for the last time before the last barrier
            c->step[(step + 1) % 3].v = 0;
            c->alive_cnt[(level + 1) % 3].v = 0;
        }
        lt_scan<MULTI>(j, sb, k, j.alive[(list0 + level) & 1], alive_n,
                       j.alive[(list0 + level + 1) & 1],
                       &c->alive_cnt[la].v, &c->step[step % 3].v, j.q[(step + 1) & 1]);
        uint32_t items = lt_barrier(j, t_start, &c->step[step % 3].v, &c->alive_cnt[la].v, &sv);
        step++;
        uint32_t err = sv.err, rounds = 0, lv_items = 0;
        alive_n = sv.alive;
        if (lead) t_scan = global_ns();
        bool scanned = true;
        // with no survivor left the rows of this scan's removals name no node
        // that could still change
        while (!err && alive_n && items) {
            if (lead) c->step[(step + 1) % 3].v = 0;
            lt_expand<MULTI>(j, sb, k, j.q[step & 1], items, scanned, &c->step[step % 3].v,
                             j.q[(step + 1) & 1]);
            lv_items += items;
            rounds++;
            items = lt_barrier(j, t_start, &c->step[step % 3].v, nullptr, &sv);
            step++;
            err = sv.err;
            scanned = false;
        }
        if (lead) {
            const uint64_t now = global_ns();
            c->ph_ns[0] += t_scan - t_last;
            c->ph_ns[1] += now - t_scan;
            c->queued += lv_items;
            if (j.trace && k < j.trace_levels) {
                unsigned long long* r = j.trace + (uint64_t)TRACE_W * k;
                r[0] = t_scan - t_last;
                r[1] = now - t_scan;
                r[2] = rounds;
                r[3] = lv_items;
                r[4] = alive_n;
            }
            t_last = now;
            c->levels = level + 1;
        }
        level++;
        if (err) return;
        if (alive_n && k + 1 > j.max_level) {  // the same on every block
            if (lead) atomicCAS(&c->err.v, PEEL_OK, PEEL_ERR_LIMIT);
            return;
        }
    }
    if (j.stop_alive && lead) {  // the next launch goes on from here
        c[1].m = alive_n;
        c[1].first_level = k0 + level;
        c[1].list = (list0 + level) & 1;
    }
}

// ---- the rows that are left --------------------------------------------------
//
// Ids in the order in which blocks reserve them.  A node alive in any column
// of a group is alive in its first (core_{lambda+1} <= core_lambda), so the
// degrees of the first column are the rows' lengths.

struct LateBuild {
    uint32_t fresh;              // no peel ran: every node, from its full degrees
    uint32_t cap, adj_cap, G;
    uint2* row;
    uint2* meta;
    uint32_t* adj;
    u64* deg;
    uint64_t plane;
    u64* cnt;
    uint32_t* M;
    uint32_t* x_of;              // the launch index of node i
    uint32_t* id_of;             // the id of launch index x (unless fresh: then the same)
    uint32_t* node_seg;
    uint32_t* alive;
    uint32_t* fills;             // nodes whose source row is a block's to copy
    LateCtl* ctl;
};

constexpr uint32_t FB_THREADS = 256;

// exclusive scan over the block's 256 threads; every thread gets the total
__device__ __forceinline__ uint32_t fb_scan(uint32_t v, uint32_t* excl, uint32_t* s_w) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t in = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, in, o);
        if (lane >= (uint32_t)o) in += y;
    }
    __syncthreads();
    if (lane == 31) s_w[w] = in;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (uint32_t i = 0; i < FB_THREADS / 32; i++) {
        const uint32_t x = s_w[i];
        if (i < w) before += x;
        total += x;
    }
    *excl = before + in - v;
    return total;
}

// The row length of node v of segment g: its alive neighbours.
__device__ __forceinline__ uint32_t lt_row_len(const PeelJob& j, const SegP& g, bool fresh,
                                               uint32_t x, uint32_t v) {
    if (fresh) return __ldg(g.node_ptr + v + 1) - __ldg(g.node_ptr + v);
    const u64* dw = (const u64*)g.deg + (uint64_t)v * g.L * g.Q;
    uint32_t row = 0;
    for (uint32_t l = 0; l < g.L; l++) row += (uint32_t)dw[(uint64_t)l * g.Q] & 0xFFFFu;
    return row;
}

// Ids, row places, masks, and the list of nodes; the degree words are copied
// by k_lt_degrees.
template <bool MULTI>
__global__ void __launch_bounds__(FB_THREADS) k_lt_rows(const __grid_constant__ PeelJob j,
                                                        const __grid_constant__ LateBuild b) {
    __shared__ uint32_t s_w[FB_THREADS / 32], s_base[3];
    const PeelCtl* const pc = j.ctl;
    const uint32_t n_in = b.fresh ? j.nx : pc->stopped ? pc->stop_alive : 0u;
    const uint32_t* const list = b.fresh ? nullptr : j.alive[pc->stop_list & 1u];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        b.ctl->first_level = b.fresh ? 0u : pc->stop_level + 1;
        b.ctl->t_start = !b.fresh ? pc->t_start : j.t_start ? j.t_start : global_ns();
    }
    for (uint32_t i0 = blockIdx.x * FB_THREADS; i0 < n_in; i0 += gridDim.x * FB_THREADS) {
        const uint32_t i = i0 + threadIdx.x;
        uint32_t x = 0, s = 0, row = 0, v = 0, M = 0;
        bool live = i < n_in;
        if (live) {
            x = list ? list[i] : i;
            if (!b.fresh) {
                M = j.M[x] & COLS_MASK;
                live = M != 0;
            }
        }
        SegP g = seg_load<MULTI>(j, 0);
        if (live) {
            s = seg_of<MULTI>(j, x);
            g = seg_load<MULTI>(j, s);
            v = x - g.xbase;
            if (b.fresh) M = (1u << g.ncols) - 1u;
            row = lt_row_len(j, g, b.fresh, x, v);
        }
        uint32_t id, at, wt = 0;
        const uint32_t tid = fb_scan(live ? 1u : 0u, &id, s_w);
        const uint32_t tat = fb_scan(row, &at, s_w);
        const uint32_t twt = MULTI ? fb_scan(live ? g.L : 0u, &wt, s_w) : 0u;
        if (threadIdx.x == 0) {
            // (when fresh, ids are launch indices: neighbours are named without a map)
            s_base[0] = b.fresh ? i0 : tid ? atomicAdd(&b.ctl->m, tid) : 0u;
            s_base[1] = tat ? atomicAdd(&b.ctl->entries, tat) : 0u;
            s_base[2] = twt ? atomicAdd(&b.ctl->words, twt) : 0u;
            if (b.fresh && i0 == 0) b.ctl->m = n_in;
        }
        __syncthreads();
        if (live) {
            id += s_base[0];
            b.row[id] = make_uint2(at + s_base[1], row);
            b.x_of[id] = x;
            b.M[id] = M;
            b.alive[id] = id;
            if (!b.fresh) b.id_of[x] = id;
            if (MULTI) {
                b.node_seg[id] = s;
                b.meta[id] = make_uint2(wt + s_base[2], g.Q | (g.col0 << 8));
            }
        }
    }
}

// The degree words: copied, or every column's from the full degrees; the
// counts of the columns that no scan will look at.  A word whose columns have
// all left the node was perhaps never written (the first scan writes none
// whose columns all go there): it starts with full fields, which count more
// than the neighbours left, as the rounds' bounds ask.
template <bool MULTI>
__global__ void __launch_bounds__(FB_THREADS) k_lt_degrees(const __grid_constant__ PeelJob j,
                                                           const __grid_constant__ LateBuild b) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t m = b.ctl->m;
    const uint32_t warps = gridDim.x * (FB_THREADS / 32);
    for (uint32_t i = blockIdx.x * (FB_THREADS / 32) + (threadIdx.x >> 5); i < m; i += warps) {
        const SegP g = seg_load<MULTI>(j, MULTI ? b.node_seg[i] : 0u);
        const uint32_t v = b.x_of[i] - g.xbase, words = g.L * g.Q;
        const uint32_t M = b.M[i];
        u64* const dst = b.deg + (MULTI ? b.meta[i].x : i * g.L);
        const u64* const src = (const u64*)g.deg + (uint64_t)v * words;
        for (uint32_t w = lane; w < words; w += 32) {
            const uint32_t q = g.divL.div(w), l = w - q * g.L;
            u64 d = ~0ull;
            if (b.fresh) d = all4(__ldg(g.deg0 + (uint64_t)v * g.L + l));
            else if ((M >> (4 * q)) & 15u) d = src[l * g.Q + q];
            dst[q * b.plane + l] = d;
        }
        if (lane < b.G) b.cnt[(uint64_t)i * b.G + lane] = LT_DEAD;
    }
}

// The part of node v's row that can name alive nodes: an ordered row
// (device.h) only as far as its entries of bucket >= bucket_of(k), the rest
// name nodes whose bound, hence core, is below it.
__device__ __forceinline__ uint32_t lt_need(const SegP& g, uint32_t v, uint32_t k,
                                            uint32_t* start) {
    const uint32_t id = g.big_id ? __ldg(g.big_id + v) : NO_BIG_ROW;
    const uint32_t rb = __ldg(g.node_ptr + v), len = __ldg(g.node_ptr + v + 1) - rb;
    *start = rb;
    if (id == NO_BIG_ROW) return len;
    return min(len, __ldg(g.ptab + (uint64_t)id * BUCKETS + bucket_of(k)));
}

// 32 entries of a row (each lane's slot, or none): the ones that name alive
// nodes go to the row's next places, at `at`; returns how many.
__device__ __forceinline__ uint32_t lt_entry(const PeelJob& j, const LateBuild& b, const SegP& g,
                                             uint32_t slot, bool& in) {
    const uint32_t u = g.divL.div(slot), l = slot - u * g.L, xu = g.xbase + u;
    uint32_t id = xu;
    if (!b.fresh && in) {
        in = (j.M[xu] & COLS_MASK) != 0;
        if (in) id = b.id_of[xu];
    }
    return (id << LT_LAYER_BITS) | l;
}

// One warp per node copies its row; a row of more than LT_FILL_LONG source
// entries is listed for k_lt_fill_long.  A row that does not come out as long
// as its degrees say is an error (found before anything reads the rows).
template <bool MULTI>
__global__ void __launch_bounds__(FB_THREADS) k_lt_fill(const __grid_constant__ PeelJob j,
                                                        const __grid_constant__ LateBuild b) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t m = b.ctl->m, k = b.ctl->first_level;
    const uint32_t warps = gridDim.x * (FB_THREADS / 32);
    for (uint32_t i = blockIdx.x * (FB_THREADS / 32) + (threadIdx.x >> 5); i < m; i += warps) {
        const SegP g = seg_load<MULTI>(j, MULTI ? b.node_seg[i] : 0u);
        const uint32_t v = b.x_of[i] - g.xbase;
        const uint2 r = b.row[i];
        uint32_t rb;
        const uint32_t need = lt_need(g, v, k, &rb);
        if (need > LT_FILL_LONG) {
            if (lane == 0) {
                const uint32_t at = atomicAdd(&b.ctl->nfill, 1u);
                if (at < b.cap) b.fills[at] = i;
                else atomicExch(&b.ctl->err.v, PEEL_ERR_ITEM);
            }
            continue;
        }
        uint32_t got = 0;
        for (uint32_t p0 = 0; p0 < need; p0 += 128) {
            uint32_t e[4];
            bool in[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const uint32_t p = p0 + 32 * t + lane;
                in[t] = p < need;
                e[t] = in[t] ? __ldg(g.adj + rb + p) : 0u;
            }
#pragma unroll
            for (int t = 0; t < 4; t++) e[t] = lt_entry(j, b, g, e[t], in[t]);
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const uint32_t am = __ballot_sync(0xffffffffu, in[t]);
                const uint32_t at = r.x + got + __popc(am & ((1u << lane) - 1u));
                if (in[t] && at < b.adj_cap) b.adj[at] = e[t];
                got += __popc(am);
            }
        }
        if (lane == 0 && got != r.y) atomicExch(&b.ctl->err.v, PEEL_ERR_ITEM);
    }
}

constexpr uint32_t FL_THREADS = 1024;
template <bool MULTI>
__global__ void __launch_bounds__(FL_THREADS) k_lt_fill_long(const __grid_constant__ PeelJob j,
                                                             const __grid_constant__ LateBuild b) {
    __shared__ uint32_t s_got;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nf = min(b.ctl->nfill, b.cap), k = b.ctl->first_level;
    for (uint32_t f = blockIdx.x; f < nf; f += gridDim.x) {
        const uint32_t i = b.fills[f];
        const SegP g = seg_load<MULTI>(j, MULTI ? b.node_seg[i] : 0u);
        const uint32_t v = b.x_of[i] - g.xbase;
        const uint2 r = b.row[i];
        uint32_t rb;
        const uint32_t need = lt_need(g, v, k, &rb);
        __syncthreads();
        if (threadIdx.x == 0) s_got = 0;
        __syncthreads();
        for (uint32_t p0 = (threadIdx.x & ~31u) * 4; p0 < need; p0 += 4 * FL_THREADS) {
            uint32_t e[4], am[4], n = 0;
            bool in[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const uint32_t p = p0 + 32 * t + lane;
                in[t] = p < need;
                e[t] = in[t] ? __ldg(g.adj + rb + p) : 0u;
            }
#pragma unroll
            for (int t = 0; t < 4; t++) e[t] = lt_entry(j, b, g, e[t], in[t]);
#pragma unroll
            for (int t = 0; t < 4; t++) {
                am[t] = __ballot_sync(0xffffffffu, in[t]);
                n += __popc(am[t]);
            }
            uint32_t at = 0;  // the entries of a row may stand in any order
            if (lane == 0 && n) at = atomicAdd(&s_got, n);
            at = r.x + __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const uint32_t p = at + __popc(am[t] & ((1u << lane) - 1u));
                if (in[t] && p < b.adj_cap) b.adj[p] = e[t];
                at += __popc(am[t]);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0 && s_got != r.y) atomicExch(&b.ctl->err.v, PEEL_ERR_ITEM);
    }
}

// ---- host ---------------------------------------------------------------------

// Whether a launch's graphs are within what the late form holds: 9-bit layers
// and 32-bit row and word positions.
bool late_takes(const PeelSegSpec* specs, size_t count) {
    uint64_t e = 0;
    for (size_t i = 0; i < count; i++) {
        if (specs[i].g.L > LATE_MAX_LAYERS) return false;
        e += specs[i].g.entries * ((specs[i].ncols + MAX_COLS - 1) / MAX_COLS);
    }
    return e < (1ull << 32);
}

void LatePlan::init(uint64_t nx, uint64_t nodes_, uint64_t words, uint64_t entries_,
                    uint64_t items, uint32_t G_, bool fresh_) {
    nodes = nodes_;
    entries = entries_;
    q_cap = items;
    G = G_;
    fresh = fresh_;
    uint64_t at = 0;
    auto take = [&](uint64_t bytes) {
        const uint64_t o = at;
        at = (at + bytes + 255) & ~255ull;
        return o;
    };
    o_ctl = take(2 * sizeof(LateCtl));
    o_row = take(8 * nodes);
    o_meta = take(8 * nodes);
    o_adj = take(4 * entries);
    plane = words;
    o_deg = take(8ull * G * plane);
    o_cnt = take(8ull * G * nodes);
    o_M = take(4 * nodes);
    o_x = take(4 * nodes);
    o_id = take(fresh ? 0 : 4 * nx);
    o_seg = take(4 * nodes);
    o_alive = take(8 * nodes);
    o_fill = take(4 * nodes);
    o_q = take(32 * q_cap);
    total = at;
}

template <bool MULTI>
static fc_status late_launch_t(const PeelJob& pj, const LatePlan& p, char* w, cudaStream_t s) {
    LateBuild b{};
    b.fresh = p.fresh;
    b.cap = (uint32_t)p.nodes;
    b.adj_cap = (uint32_t)p.entries;
    b.G = p.G;
    b.row = (uint2*)(w + p.o_row);
    b.meta = (uint2*)(w + p.o_meta);
    b.adj = (uint32_t*)(w + p.o_adj);
    b.deg = (u64*)(w + p.o_deg);
    b.plane = p.plane;
    b.cnt = (u64*)(w + p.o_cnt);
    b.M = (uint32_t*)(w + p.o_M);
    b.x_of = (uint32_t*)(w + p.o_x);
    b.id_of = (uint32_t*)(w + p.o_id);
    b.node_seg = (uint32_t*)(w + p.o_seg);
    b.alive = (uint32_t*)(w + p.o_alive);
    b.fills = (uint32_t*)(w + p.o_fill);
    b.ctl = (LateCtl*)(w + p.o_ctl);
    LateJob j{};
    j.L = pj.seg0.L;
    j.Q = pj.seg0.Q;
    j.col0 = pj.seg0.col0;
    j.G = p.G;
    j.row = b.row;
    j.meta = b.meta;
    j.adj = b.adj;
    j.deg = b.deg;
    j.plane = p.plane;
    j.cnt = b.cnt;
    j.M = b.M;
    j.x_of = b.x_of;
    j.node_seg = b.node_seg;
    j.alive[0] = (uint32_t*)(w + p.o_alive);
    j.alive[1] = j.alive[0] + p.nodes;
    j.q[0] = (uint4*)(w + p.o_q);
    j.q[1] = j.q[0] + p.q_cap;
    j.q_cap = (uint32_t)p.q_cap;
    j.cap = (uint32_t)p.nodes;
    j.ctl0 = j.ctl = b.ctl;
    j.seg0 = pj.seg0;
    j.segs = pj.segs;
    j.max_level = pj.max_level;
    j.timeout_ns = pj.timeout_ns;
    j.deadline_ns = pj.deadline_ns;
    j.trace = pj.trace;
    j.trace_levels = pj.trace_levels;
    int dev = 0, sms = 0;
    FC_CUDA_TRY(cudaGetDevice(&dev));
    FC_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (pj.max_sms && (int)pj.max_sms < sms) sms = (int)pj.max_sms;
    const uint32_t node_blocks =
        (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(8ull * sms, (p.nodes + 255) / 256));
    const uint32_t warp_blocks =
        (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(8ull * sms, (p.nodes + 7) / 8));
    FC_CUDA_TRY(cudaMemsetAsync(b.ctl, 0, 2 * sizeof(LateCtl), s));
    k_lt_rows<MULTI><<<node_blocks, FB_THREADS, 0, s>>>(pj, b);
    FC_CUDA_TRY(cudaGetLastError());
    k_lt_degrees<MULTI><<<warp_blocks, FB_THREADS, 0, s>>>(pj, b);
    FC_CUDA_TRY(cudaGetLastError());
    k_lt_fill<MULTI><<<warp_blocks, FB_THREADS, 0, s>>>(pj, b);
    FC_CUDA_TRY(cudaGetLastError());
    k_lt_fill_long<MULTI><<<2 * sms, FL_THREADS, 0, s>>>(pj, b);
    FC_CUDA_TRY(cudaGetLastError());
    void* args[] = {&j};
    if (p.nodes > LT_SMALL) {
        j.stop_alive = LT_SMALL;
        FC_CUDA_TRY(cudaLaunchCooperativeKernel((void*)k_late<1024, MULTI>, dim3(sms), dim3(1024),
                                                args, 0, s));
        j.stop_alive = 0;
        j.ctl = b.ctl + 1;
        count_launch();
    }
    FC_CUDA_TRY(cudaLaunchCooperativeKernel((void*)k_late<LT_SMALL_T, MULTI>, dim3(sms),
                                            dim3(LT_SMALL_T), args, 0, s));
    count_launch(5);
    return FC_OK;
}

fc_status late_launch(const PeelJob& pj, const LatePlan& p, char* w, cudaStream_t s) {
    return pj.nseg > 1 ? late_launch_t<true>(pj, p, w, s) : late_launch_t<false>(pj, p, w, s);
}

void late_preload() {
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, k_late<1024, false>);
    cudaFuncGetAttributes(&a, k_late<1024, true>);
    cudaFuncGetAttributes(&a, k_late<LT_SMALL_T, false>);
    cudaFuncGetAttributes(&a, k_late<LT_SMALL_T, true>);
    cudaFuncGetAttributes(&a, k_lt_rows<false>);
    cudaFuncGetAttributes(&a, k_lt_rows<true>);
    cudaFuncGetAttributes(&a, k_lt_degrees<false>);
    cudaFuncGetAttributes(&a, k_lt_degrees<true>);
    cudaFuncGetAttributes(&a, k_lt_fill<false>);
    cudaFuncGetAttributes(&a, k_lt_fill<true>);
    cudaFuncGetAttributes(&a, k_lt_fill_long<false>);
    cudaFuncGetAttributes(&a, k_lt_fill_long<true>);
    cudaGetLastError();
}

}  // namespace fc
