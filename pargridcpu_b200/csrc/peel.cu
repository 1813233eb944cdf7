// The fcgrid peel: core_lambda(v) for groups of lambda columns of one or many
// graphs, in one persistent cooperative kernel with the level loop inside.
//
// A launch covers segments; a segment is one graph's group of up to MAX_COLS
// lambda columns (lambda = col0+c+1 for c < ncols).  The segments' nodes are
// laid end to end in one index space x, so one launch peels many graphs at
// once and they share the level loop.  All columns advance together, level by
// level, K = 0, 1, 2, ...:
//
//   SCAN(K)    every alive x counts, per column, its layers with degree >=
//              K+1 inside the column's alive set.  A column whose count is
//              below lambda removes x at level K (core = K).  Survivors keep
//              their counts.
//   EXPAND     every adjacency slot (u,l) of a removed x decrements
//              deg[u][l] of the removed columns in which u is alive; a
//              decrement from exactly K+1 to K lowers u's count, and the
//              decrement that takes the count from lambda to lambda-1 removes
//              u in that column at level K too -- ParGrid's own trigger
//              (CoreParallel/FCSyncLeft.cpp:99-103).  Each of those crossings
//              happens exactly once.  What a round removes, the next round
//              expands, until a round removes nothing.
//
// This computes the same table as the reference's get_index2 bucket peel
// (CoreIndexParallel/CoreIndex.cpp:62-109) and ParGrid's per-cell PeelSync:
// core_lambda is the unique fixpoint, whatever the removal order.
//
// Columns are packed.  The degrees of (u,l) in four columns are the 16-bit
// fields of one 64-bit word, so one atomic decrements all four; a node's alive
// columns are one mask word, so one load tells a visit which columns are left;
// and a node removed in several columns in one round is expanded once for all
// of them (at a node's low levels most of its columns go together: on a
// 2.6M-node, 24-layer graph a row is read 6.7 times instead of 24).
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "peel_common.h"

namespace fc {

// ---- the grid barrier ---------------------------------------------------------

// What thread 0 reads after a barrier, for the whole block.
struct StepView {
    uint32_t err, ns, nc, alive;
};

// Grid barrier with a bounded wait.  Every block counts itself in; the wait
// ends when all have (the counter only grows).  `out` (shared) receives the
// error flag, the items queued for step slot `slot` and the survivors counted
// at parity `ap`, read once by thread 0.  Block 0 also checks the run's
// deadline.  A block that sees the error flag leaves; the others' waits end by
// the flag or by their own bound.
__device__ void grid_barrier(const PeelJob& j, uint32_t& nbar, uint64_t t_start, uint32_t slot,
                             uint32_t ap, StepView* out) {
    PeelCtl* c = j.ctl;
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t target = ++nbar * gridDim.x;
        if (blockIdx.x == 0 && past_deadline(t_start, j.deadline_ns))
            atomicCAS(&c->err.v, PEEL_OK, PEEL_ERR_DEADLINE);
        red_add_release(&c->arrive.v, 1u);
        uint64_t t0 = 0;
        for (uint32_t spins = 1; (int)(ld_relaxed(&c->arrive.v) - target) < 0; spins++) {
            if ((spins & 255) == 0) {
                const uint64_t now = global_ns();
                if (!t0) t0 = now;
                if (now - t0 > j.timeout_ns) atomicCAS(&c->err.v, PEEL_OK, PEEL_ERR_BARRIER);
                // an error ends the run: some blocks may have left already
                if (ld_relaxed(&c->err.v) != PEEL_OK) break;
            }
        }
        (void)ld_acquire(&c->arrive.v);
        out->err = ld_relaxed(&c->err.v);
        out->ns = ld_relaxed(&c->tail[slot][0].v);
        out->nc = ld_relaxed(&c->tail[slot][1].v);
        out->alive = ld_relaxed(&c->alive_cnt[ap].v);
    }
    __syncthreads();
}

// ---- queues -----------------------------------------------------------------

// Where a step's items go, and the level they are removed at.  The packed form
// keeps three steps' queues apart (the step after next clears what a step
// marked); the unpacked form appends, as a node is removed only once.
struct Step {
    uint32_t k;
    uint32_t slot;      // step mod 3: the items read
    uint32_t next;      // (step + 1) mod 3: the items written
    const uint32_t* s_in;           // the items read
    const unsigned long long* c_in;
    uint32_t* s_out;                // the items written, at most s_cap and c_cap
    unsigned long long* c_out;
    uint32_t s_cap, c_cap;
};

// A node removed at level k is queued as one short item when its row has at
// most small_row entries, else as chunk items; returns the chunk count (0 for
// a short row).  An ordered row (device.h) needs only the chunks covering its
// entries of bucket >= bucket_of(k): every later entry names a neighbour whose
// bound is below k, removed at an earlier level.  At least one chunk is
// queued, so that every removal of a long row is one or more chunk items.
__device__ __forceinline__ uint32_t chunks_of(const SegP& g, uint32_t v, uint32_t small_row,
                                              uint32_t k) {
    // the three loads are independent: one round trip
    const uint32_t id = g.big_id ? __ldg(g.big_id + v) : NO_BIG_ROW;
    const uint32_t len = __ldg(g.node_ptr + v + 1) - __ldg(g.node_ptr + v);
    if (len <= small_row) return 0u;
    uint32_t need = len;
    if (id != NO_BIG_ROW) need = min(len, __ldg(g.ptab + (uint64_t)id * BUCKETS + bucket_of(k)));
    return need ? (need + CHUNK - 1) / CHUNK : 1u;
}

// The high word of chunk item c of a row queued as nch chunks at level k.
// From level 16 on (where the ordered rows' pruning acts) a row of 2 .. 32767
// chunks is visited strided: chunk c takes the 8-entry groups c, c + nch,
// c + 2 nch, ... (one group per lane), so that the front of an ordered row --
// the neighbours that may still be alive -- is spread over all of its chunks
// rather than loading its first one.  Otherwise chunk c is the CHUNK entries
// from c * CHUNK.  Either way the row's first 256 * nch entries (clipped to
// the row) are visited once each.
constexpr uint32_t STRIDED = 0x80000000u;
__device__ __forceinline__ uint32_t chunk_word(uint32_t c, uint32_t nch, uint32_t k) {
    return (k >= 16 && nch > 1 && nch < 32768) ? (STRIDED | (nch << 16) | c) : c;
}
// whether a chunk item is its row's first
__device__ __forceinline__ bool first_chunk(uint32_t w) {
    return (w & STRIDED) ? (w & 0xFFFFu) == 0 : w == 0;
}

__device__ __forceinline__ void write_short(const PeelJob& j, const Step& st, uint32_t idx,
                                            uint32_t x) {
    if (idx < st.s_cap) st.s_out[idx] = x;
    else atomicExch(&j.ctl->err.v, PEEL_ERR_QUEUE);
}

// The chunk items of the lanes with nch > 0 (row x, first queue index at), one
// row after another, 32 items at a time: a hub's thousands of items are not
// one lane's serial loop.  All 32 lanes call it together.
__device__ __forceinline__ void write_chunks(const PeelJob& j, const Step& st, uint32_t x,
                                             uint32_t at, uint32_t nch) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t todo = __ballot_sync(0xffffffffu, nch != 0); todo; todo &= todo - 1) {
        const uint32_t src = __ffs(todo) - 1;
        const uint32_t rx = __shfl_sync(0xffffffffu, x, src);
        const uint32_t ra = __shfl_sync(0xffffffffu, at, src);
        const uint32_t rn = __shfl_sync(0xffffffffu, nch, src);
        for (uint32_t c = lane; c < rn; c += 32) {
            if (ra + c < st.c_cap)
                st.c_out[ra + c] = (u64)rx | ((u64)chunk_word(c, rn, st.k) << 32);
            else
                atomicExch(&j.ctl->err.v, PEEL_ERR_QUEUE);
        }
    }
}

// Warp-wide inclusive scan.
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (uint32_t)o) v += y;
    }
    return v;
}

// A queued item that names no node of the launch, or no chunk of its row:
// the first one is recorded and the run ends with PEEL_ERR_ITEM; the item itself
// is skipped.
__device__ __noinline__ void record_bad(const PeelJob& j, uint32_t item, uint32_t where) {
    if (atomicCAS(&j.ctl->err.v, PEEL_OK, PEEL_ERR_ITEM) == PEEL_OK) {
        j.ctl->bad_item = item;
        j.ctl->bad_where = where;
    }
}

// ---- SCAN -----------------------------------------------------------------

// Degrees of a HUB node above what its fields hold: per layer and column how
// many decrements the counters take before the fields do.
__device__ __noinline__ void make_hub(const PeelJob& j, const SegP& g, uint32_t x, uint32_t v) {
    const uint32_t h = atomicAdd(&j.ctl->nhub, 1u);
    if (h >= j.hub_cap) {  // more than the entries allow
        record_bad(j, x, 5);
        return;
    }
    j.hub_idx[x] = h;
    int* ex = j.hub_ex + (uint64_t)h * j.hub_stride * j.hub_pad;
    for (uint32_t l = 0; l < g.L; l++) {
        const uint32_t d = __ldg(g.deg0 + (uint64_t)v * g.L + l);
        const int e = d > FIELD_MAX ? (int)(d - FIELD_MAX) : 0;
        for (uint32_t c = 0; c < g.ncols; c++) ex[(l * g.ncols + c) * j.hub_pad] = e;
    }
}

// SCAN(K) over `cnt_nodes` alive nodes taken from `src` (or 0..nx-1 when src
// is null: the first level, which starts every column from the full degrees).
// G lanes per node (one per degree word of a layer, so a node's row is read in
// whole sectors), NPT nodes per lane group and block iteration; survivors and
// queue items of a block are reserved with one atomic each per iteration (the
// counters are shared by the whole grid).
template <bool MULTI, bool PACK, int NPT>
__device__ __forceinline__ void scan_nodes(const PeelJob& j, const Step& st, const uint32_t* src,
                                           uint32_t cnt_nodes, uint32_t* out, uint32_t* out_cnt) {
    __shared__ uint32_t s_keep[32], s_short[32], s_chunk[32], s_kbase, s_sbase, s_cbase;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t nwarps = blockDim.x >> 5;
    const uint32_t G = PACK ? j.G : 1u;
    const uint32_t npw = PACK ? 32u / G : 32u;  // nodes per warp and pass
    const uint32_t sub = PACK ? lane / G : lane, q = PACK ? lane - sub * G : 0u;
    const uint32_t gbase = PACK ? sub * G : lane;
    const uint32_t per_pass = nwarps * npw;
    const uint32_t per_block = per_pass * NPT;
    const bool first = src == nullptr;
    const uint32_t t2 = (st.k + 1) | ((st.k + 1) << 16);
    for (uint32_t base = blockIdx.x * per_block; base < cnt_nodes; base += gridDim.x * per_block) {
        uint32_t xs[NPT], nchs[NPT], tk = 0, tsh = 0, tch = 0;
        uint32_t flags = 0;  // per pass: 1 keep, 2 short item
#pragma unroll
        for (int i = 0; i < NPT; i++) {
            const uint32_t idx = base + i * per_pass + warp * npw + sub;
            bool live = sub < npw && idx < cnt_nodes;
            const uint32_t x = live ? (src ? src[idx] : idx) : 0;
            const SegP g = seg_load<MULTI>(j, seg_of<MULTI>(j, x));
            const uint32_t v = x - g.xbase;
            const uint32_t full = (1u << g.ncols) - 1u;
            const uint32_t m = !live ? 0u : first ? full : j.M[x];
            if (!(m & COLS_MASK)) live = false;  // removed in the last level's rounds
            uint32_t rem = 0;
            bool hub = false;
            if (PACK) {
                const uint32_t m4 = live && q < g.Q ? (m >> (4 * q)) & 15u : 0u;
                u64 c4 = 0;
                u64* const dw = (u64*)g.deg + (uint64_t)v * g.L * g.Q + q;
                if (m4) {
                    if (first) {
                        const uint32_t* d0 = g.deg0 + (uint64_t)v * g.L;
                        uint32_t c = 0;
#pragma unroll 4
                        for (uint32_t l = 0; l < g.L; l++) {
                            const uint32_t d = __ldg(d0 + l);
                            c += d >= st.k + 1;
                            hub |= d > FIELD_MAX;
                        }
                        c4 = all4(c);
                    } else if (st.k < FIELD_MAX) {  // no core is larger: entries < 2^32
#pragma unroll 4
                        for (uint32_t l = 0; l < g.L; l++)
                            c4 += geq4(dw[(uint64_t)l * g.Q], t2);
                    }
                }
                uint32_t r4 = 0;
#pragma unroll
                for (uint32_t f = 0; f < 4; f++)
                    if (((m4 >> f) & 1u) && ((uint32_t)(c4 >> (16 * f)) & 0xFFFFu) < g.col0 + 4 * q + f + 1)
                        r4 |= 1u << f;
                const uint32_t k4 = m4 & ~r4;
                if (k4) {
                    ((u64*)g.cnt)[(uint64_t)v * g.Q + q] = c4;
                    if (first) {
                        const uint32_t* d0 = g.deg0 + (uint64_t)v * g.L;
#pragma unroll 4
                        for (uint32_t l = 0; l < g.L; l++)
                            dw[(uint64_t)l * g.Q] = all4(min(__ldg(d0 + l), FIELD_MAX));
                    }
                }
#pragma unroll
                for (uint32_t f = 0; f < 4; f++)
                    if ((r4 >> f) & 1u) g.t[(uint64_t)(4 * q + f) * g.n + v] = st.k;
                for (uint32_t t = 0; t < G; t++)
                    rem |= __shfl_sync(0xffffffffu, r4, (gbase + t) & 31) << (4 * t);
            } else if (live) {
                uint32_t* const dw = (uint32_t*)g.deg + (uint64_t)v * g.L;
                const uint32_t* const d = first ? g.deg0 + (uint64_t)v * g.L : dw;
                uint32_t c = 0;
#pragma unroll 4
                for (uint32_t l = 0; l < g.L; l++) c += d[l] >= st.k + 1;
                if (c < g.col0 + 1) {
                    rem = 1;
                    g.t[v] = st.k;
                } else {
                    ((uint32_t*)g.cnt)[v] = c;
                    if (first)
                        for (uint32_t l = 0; l < g.L; l++) dw[l] = d[l];
                }
            }
            const bool lead = live && q == 0;
            uint32_t nch = 0;
            bool keep = false, ns = false;
            if (lead) {
                const uint32_t left = m & ~rem;
                keep = (left & COLS_MASK) != 0;
                if (first || rem) j.M[x] = left | (hub && keep ? HUB : 0u);
                if (hub && keep) make_hub(j, g, x, v);
                if (rem) {
                    if (PACK) j.P[st.next][x] = rem;
                    nch = chunks_of(g, v, j.small_row, st.k);
                    ns = nch == 0;
                }
            }
            xs[i] = x;
            nchs[i] = nch;
            flags |= (keep ? 1u : 0u) << (2 * i) | (ns ? 2u : 0u) << (2 * i);
            tk += keep;
            tsh += ns;
            tch += nch;
        }
        const uint32_t kin = warp_incl_scan(tk);
        const uint32_t sin = warp_incl_scan(tsh);
        const uint32_t cin = warp_incl_scan(tch);
        if (lane == 31) {
            s_keep[warp] = kin;
            s_short[warp] = sin;
            s_chunk[warp] = cin;
        }
        __syncthreads();
        if (warp == 0) {  // nwarps <= 32: one value per lane
            const uint32_t a = lane < nwarps ? s_keep[lane] : 0u;
            const uint32_t b = lane < nwarps ? s_short[lane] : 0u;
            const uint32_t d = lane < nwarps ? s_chunk[lane] : 0u;
            const uint32_t ai = warp_incl_scan(a), bi = warp_incl_scan(b), di = warp_incl_scan(d);
            s_keep[lane] = ai - a;
            s_short[lane] = bi - b;
            s_chunk[lane] = di - d;
            if (lane == 31) {
                s_kbase = ai ? atomicAdd(out_cnt, ai) : 0u;
                s_sbase = bi ? atomicAdd(&j.ctl->tail[st.next][0].v, bi) : 0u;
                s_cbase = di ? atomicAdd(&j.ctl->tail[st.next][1].v, di) : 0u;
            }
        }
        __syncthreads();
        uint32_t kp = s_kbase + s_keep[warp] + kin - tk;
        uint32_t sp = s_sbase + s_short[warp] + sin - tsh;
        uint32_t cp = s_cbase + s_chunk[warp] + cin - tch;
#pragma unroll
        for (int i = 0; i < NPT; i++) {
            if ((flags >> (2 * i)) & 1u) out[kp++] = xs[i];
            if ((flags >> (2 * i)) & 2u) write_short(j, st, sp++, xs[i]);
            write_chunks(j, st, xs[i], cp, nchs[i]);
            cp += nchs[i];
        }
        __syncthreads();
    }
}

// ---- EXPAND ---------------------------------------------------------------

// Entry (u,l) of a HUB node u, columns m: the counters take the decrements
// that the fields cannot hold (the true degree is the field plus what is left
// in the counter, and the fields only move once it has run out).  Returns the
// columns whose field takes the decrement.
__device__ __noinline__ uint32_t absorb(const PeelJob& j, const SegP& g, uint32_t xu, uint32_t l,
                                        uint32_t m) {
    const uint32_t h = j.hub_idx[xu];
    if (h >= j.hub_cap) return m;  // recorded by make_hub
    int* ex = j.hub_ex + ((uint64_t)h * j.hub_stride + l * g.ncols) * j.hub_pad;
    if (__ldg(g.deg0 + (uint64_t)(xu - g.xbase) * g.L + l) <= FIELD_MAX) return m;
    uint32_t left = m;
    for (uint32_t b = m; b; b &= b - 1) {
        const uint32_t c = __ffs(b) - 1;
        if (atomicSub(ex + c * j.hub_pad, 1) > 0) left &= ~(1u << c);
    }
    return left;
}

// N row entries per lane at once (loads first, then the atomics) so that each
// lane keeps several memory operations in flight.  Entry i is slot slot[i] of
// segment seg[i], removed in the columns S[i].  All 32 lanes call it together.
//
// Columns in which the neighbour is already removed are skipped.  A column
// removed in this round may still take a decrement; that is harmless: its
// fields are not read again, a degree field counts neighbours not yet expanded
// and so never falls below 0, and the count, at least the number of layers
// that can still cross at this level, neither falls below 0 nor passes lambda
// again.
template <bool MULTI, bool PACK, int N>
__device__ __forceinline__ void visit(const PeelJob& j, const Step& st, const uint32_t (&seg)[N],
                                      const uint32_t (&S)[N], const uint32_t (&slot)[N]) {
    uint32_t xu[N], m[N], um = 0;
#pragma unroll
    for (int i = 0; i < N; i++) {
        const SegP g = seg_load<MULTI>(j, seg[i]);
        xu[i] = g.xbase + g.divL.div(slot[i]);
        m[i] = S[i] ? ld_either(j.M + xu[i]) : 0u;
    }
    uint32_t rb[N];
    if (PACK) {
        if (j.hub_idx) {
#pragma unroll
            for (int i = 0; i < N; i++)
                if ((m[i] & HUB) && (m[i] & S[i])) {
                    const SegP g = seg_load<MULTI>(j, seg[i]);
                    const uint32_t u = xu[i] - g.xbase;
                    m[i] = absorb(j, g, xu[i], slot[i] - u * g.L, m[i] & S[i]);
                }
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            m[i] &= S[i];
            um |= m[i];
            rb[i] = 0;
        }
        const uint32_t wm = __reduce_or_sync(0xffffffffu, um);
        for (uint32_t q = 0; q < j.G; q++) {
            if (!((wm >> (4 * q)) & 15u)) continue;
            u64 old[N];
#pragma unroll
            for (int i = 0; i < N; i++) {
                const uint32_t m4 = (m[i] >> (4 * q)) & 15u;
                old[i] = 0;
                if (m4) {
                    const SegP g = seg_load<MULTI>(j, seg[i]);
                    old[i] = atomicAdd((u64*)g.deg + ((uint64_t)slot[i] * g.Q + q),
                                       0ull - spread4(m4));
                }
            }
            const u64 kk = all4(st.k + 1);
            // (results are only looked at once all are on their way)
            u64 cross[N];
#pragma unroll
            for (int i = 0; i < N; i++) {
                cross[i] = zero4(old[i] ^ kk) & spread4((m[i] >> (4 * q)) & 15u);
                if (cross[i]) {
                    const SegP g = seg_load<MULTI>(j, seg[i]);
                    old[i] = atomicAdd(
                        (u64*)g.cnt + ((uint64_t)(xu[i] - g.xbase) * g.Q + q), 0ull - cross[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < N; i++)
                if (cross[i]) {
                    const SegP g = seg_load<MULTI>(j, seg[i]);
                    const u64 lm = all4(g.col0 + 4 * q) + 0x0004000300020001ull;
                    rb[i] |= gather4(zero4(old[i] ^ lm) & cross[i]) << (4 * q);
                }
        }
    } else {
        uint32_t old[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            old[i] = 0;
            if (m[i] & S[i]) {
                const SegP g = seg_load<MULTI>(j, seg[i]);
                old[i] = atomicSub((uint32_t*)g.deg + slot[i], 1u);
            }
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            rb[i] = 0;
            if (old[i] == st.k + 1) {
                const SegP g = seg_load<MULTI>(j, seg[i]);
                rb[i] = atomicSub((uint32_t*)g.cnt + (xu[i] - g.xbase), 1u) == g.col0 + 1;
            }
        }
    }
    // queue the nodes removed: the first column to remove a node in this
    // round queues it, the others join its mask
    uint32_t ur = 0;
#pragma unroll
    for (int i = 0; i < N; i++) ur |= rb[i];
    if (!__any_sync(0xffffffffu, ur != 0)) return;
    uint32_t nch[N], my_s = 0, my_c = 0;
#pragma unroll
    for (int i = 0; i < N; i++) {
        nch[i] = 0;
        if (PACK && rb[i] && atomicOr(j.P[st.next] + xu[i], rb[i]) != 0) rb[i] = 0;
        if (rb[i]) {
            const SegP g = seg_load<MULTI>(j, seg[i]);
            nch[i] = chunks_of(g, xu[i] - g.xbase, j.small_row, st.k);
            my_s += nch[i] == 0;
            my_c += nch[i];
        }
    }
    const uint32_t is = warp_incl_scan(my_s);
    const uint32_t ic = warp_incl_scan(my_c);
    uint32_t bs = 0, bc = 0;
    if ((threadIdx.x & 31) == 31) {
        if (is) bs = atomicAdd(&j.ctl->tail[st.next][0].v, is);
        if (ic) bc = atomicAdd(&j.ctl->tail[st.next][1].v, ic);
    }
    bs = __shfl_sync(0xffffffffu, bs, 31) + is - my_s;
    bc = __shfl_sync(0xffffffffu, bc, 31) + ic - my_c;
#pragma unroll
    for (int i = 0; i < N; i++) {
        if (rb[i] && nch[i] == 0) write_short(j, st, bs++, xu[i]);
        write_chunks(j, st, xu[i], bc, nch[i]);
        bc += nch[i];
    }
}

// x's removal in the columns S takes effect for the rounds to come; the
// table's entries are written unless the scan has written them.
__device__ __forceinline__ void retire(const PeelJob& j, const SegP& g, const Step& st, uint32_t x,
                                       uint32_t S, bool scanned) {
    st_either(j.M + x, ld_either(j.M + x) & ~S);  // its only writer in this step
    if (scanned) return;
    const uint32_t v = x - g.xbase;
    for (uint32_t b = S; b; b &= b - 1)
        g.t[(uint64_t)(__ffs(b) - 1) * g.n + v] = st.k;
}

// The short rows of up to 32 queued nodes, flattened over the warp's lanes;
// the owner of entry q is found by binary search over the warp's exclusive
// scan of row lengths.
template <bool MULTI, bool PACK>
__device__ __forceinline__ void expand_short(const PeelJob& j, const Step& st, uint32_t i0,
                                             uint32_t cnt, bool scanned) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t x = lane < cnt ? st.s_in[i0 + lane] : 0u;
    bool ready = lane < cnt;
    if (ready && x >= j.nx) {
        record_bad(j, x, 4);
        ready = false;
        x = 0;
    }
    const uint32_t s = seg_of<MULTI>(j, x);
    const SegP g = seg_load<MULTI>(j, s);
    uint32_t b = 0, len = 0, S = 0;
    if (ready) {
        const uint32_t v = x - g.xbase;
        b = __ldg(g.node_ptr + v);
        len = __ldg(g.node_ptr + v + 1) - b;
        S = PACK ? j.P[st.slot][x] : 1u;
        if (len > j.small_row) {  // long rows are never queued as short items
            record_bad(j, x, 1);
            len = 0;
        }
        retire(j, g, st, x, S, scanned);
    }
    const uint32_t incl = warp_incl_scan(len);
    const uint32_t excl = incl - len;
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    for (uint32_t jb = 0; jb < total; jb += 128) {
        uint32_t segs[4], slot[4], Ss[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t qq = jb + 32 * i + lane;
            uint32_t own = 0;
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1) {
                const uint32_t cand = own + step;
                const uint32_t ex = __shfl_sync(0xffffffffu, excl, cand & 31);
                if (cand < 32 && ex <= qq) own = cand;
            }
            const uint32_t ob = __shfl_sync(0xffffffffu, b, own);
            const uint32_t oe = __shfl_sync(0xffffffffu, excl, own);
            const uint32_t oS = __shfl_sync(0xffffffffu, S, own);
            segs[i] = MULTI ? __shfl_sync(0xffffffffu, s, own) : 0u;
            const uint32_t* oadj =
                MULTI ? (const uint32_t*)__shfl_sync(0xffffffffu, (u64)g.adj, own) : g.adj;
            const bool ok = qq < total;
            Ss[i] = ok ? oS : 0u;
            slot[i] = ok ? __ldg(oadj + ob + (qq - oe)) : 0u;
        }
        visit<MULTI, PACK, 4>(j, st, segs, Ss, slot);
    }
}

// One chunk of a long row (chunk_word), by the whole warp, CHUNK / 32 entries
// per lane, four at a time.
template <bool MULTI, bool PACK>
__device__ __forceinline__ void expand_chunk(const PeelJob& j, const Step& st, uint32_t i0,
                                             bool scanned) {
    constexpr int PER_LANE = CHUNK / 32;
    const uint32_t lane = threadIdx.x & 31;
    const u64 it = st.c_in[i0];
    const uint32_t x = (uint32_t)it, w = (uint32_t)(it >> 32);
    if (x >= j.nx) {
        if (lane == 0) record_bad(j, x, 3);
        return;
    }
    const uint32_t s = seg_of<MULTI>(j, x);
    const SegP g = seg_load<MULTI>(j, s);
    const uint32_t v = x - g.xbase;
    const uint32_t rb = __ldg(g.node_ptr + v), re = __ldg(g.node_ptr + v + 1);
    const uint32_t S = PACK ? j.P[st.slot][x] : 1u;
    const uint32_t len = re - rb, full = (len + CHUNK - 1) / CHUNK;
    const bool strided = (w & STRIDED) != 0;
    const uint32_t nch = strided ? (w >> 16) & 0x7FFFu : 0u;
    const uint32_t ch = strided ? (w & 0xFFFFu) : w;
    if (strided ? (ch >= nch || nch > full) : ch >= full) {  // no such chunk of the row
        if (lane == 0) record_bad(j, x, 2);
        return;
    }
    if (ch == 0 && lane == 0) retire(j, g, st, x, S, scanned);
    // row offset of this lane's first entry and the step between its entries;
    // offsets stay below 256 * full, under 2^24 when strided
    const uint32_t o0 = strided ? 8u * (ch + lane * nch) : ch * CHUNK + lane;
    const uint32_t step = strided ? 1u : 32u;
    uint32_t slots[PER_LANE];
    uint32_t okm = 0;
#pragma unroll
    for (int i = 0; i < PER_LANE; i++) {
        const uint32_t o = o0 + step * i;
        const bool ok = o < len && (strided || o < (ch + 1) * CHUNK);
        okm |= (ok ? 1u : 0u) << i;
        slots[i] = ok ? __ldg(g.adj + rb + o) : 0u;
    }
#pragma unroll
    for (int h = 0; h < PER_LANE; h += 4) {
        uint32_t segs[4], slot[4], Ss[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            segs[i] = s;
            slot[i] = slots[h + i];
            Ss[i] = (okm >> (h + i)) & 1u ? S : 0u;
        }
        visit<MULTI, PACK, 4>(j, st, segs, Ss, slot);
    }
}

// The items of one round: chunk items first (the larger ones), then the short
// items in tiles of up to 32, dealt over the grid's warps so that consecutive
// items go to different SMs; with few short items a tile is one row.
template <bool MULTI, bool PACK>
__device__ __forceinline__ void phase_expand(const PeelJob& j, const Step& st, uint32_t ns,
                                             uint32_t nc, bool scanned) {
    const uint32_t nw = gridDim.x * (blockDim.x >> 5);
    const uint32_t gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const uint32_t tile = max(1u, min(32u, (ns + nw - 1) / nw));
    const uint32_t tiles = (ns + tile - 1) / tile;
    const uint32_t total = nc + tiles;
    for (uint32_t i = gw; i < total; i += nw) {
        if (i < nc) {
            expand_chunk<MULTI, PACK>(j, st, i, scanned);
        } else {
            const uint32_t i0 = (i - nc) * tile;
            expand_short<MULTI, PACK>(j, st, i0, min(tile, ns - i0), scanned);
        }
    }
}

// The masks that the step before the last marked are empty again before the
// next step's removals use them.
__device__ __forceinline__ void clear_masks(const PeelJob& j, uint32_t slot, uint32_t ns,
                                            uint32_t nc) {
    uint32_t* P = j.P[slot];
    const uint32_t* qs = j.qs + (uint64_t)slot * j.qs_cap;
    const u64* qc = j.qc + (uint64_t)slot * j.qc_cap;
    const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x, st = gridDim.x * blockDim.x;
    for (uint32_t i = t0; i < ns; i += st) {
        const uint32_t x = qs[i];
        if (x < j.nx) P[x] = 0;
    }
    for (uint32_t i = t0; i < nc; i += st) {
        const u64 it = qc[i];
        if ((uint32_t)it < j.nx && first_chunk((uint32_t)(it >> 32))) P[(uint32_t)it] = 0;
    }
}

// T threads per block, 1024 threads resident per SM (512 x 2 or 1024 x 1):
// at most 64 registers a thread.
template <int T, bool MULTI, bool PACK, int BPS = 1024 / T>
__global__ void __launch_bounds__(T, BPS) k_peel(const __grid_constant__ PeelJob j) {
    __shared__ StepView sv;
    PeelCtl* const c = j.ctl;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    uint64_t t_last = lead ? global_ns() : 0, t_scan = 0, ph0 = 0, ph1 = 0;
    const uint64_t t_start = j.t_start ? j.t_start : t_last;
    if (lead) c->t_start = t_start;
    uint32_t nbar = 0, items = 0;
    uint32_t step = 0, level = 0;
    uint32_t alive_n = j.nx, pns = 0, pnc = 0;  // pns, pnc: items the last step read
    for (;;) {
        Step st;
        st.k = level;
        st.slot = step % 3;
        st.next = (step + 1) % 3;
        st.s_in = nullptr;
        st.c_in = nullptr;
        st.s_out = j.qs + (PACK ? (uint64_t)st.next * j.qs_cap : 0u);
        st.c_out = j.qc + (PACK ? (uint64_t)st.next * j.qc_cap : 0u);
        st.s_cap = j.qs_cap;
        st.c_cap = j.qc_cap;
        const uint32_t la = level % 3;
        if (lead) {
            // read for the last time before the last barrier
            c->tail[(step + 2) % 3][0].v = 0;
            c->tail[(step + 2) % 3][1].v = 0;
            c->alive_cnt[(level + 1) % 3].v = 0;
        }
        if (PACK) clear_masks(j, (step + 2) % 3, pns, pnc);
        const uint32_t* const src = level ? j.alive[(level + 1) & 1] : nullptr;
        uint32_t* const out = j.alive[level & 1];
        // grid-uniform choice (every block sees the same count)
        if ((uint64_t)alive_n * (PACK ? j.G : 1u) >= 4ull * gridDim.x * blockDim.x)
            scan_nodes<MULTI, PACK, 4>(j, st, src, alive_n, out, &c->alive_cnt[la].v);
        else
            scan_nodes<MULTI, PACK, 1>(j, st, src, alive_n, out, &c->alive_cnt[la].v);
        grid_barrier(j, nbar, t_start, st.next, la, &sv);
        step++;
        pns = pnc = 0;
        const uint32_t err = sv.err;
        alive_n = sv.alive;
        uint32_t ns = sv.ns, nc = sv.nc, rounds = 0, lv_items = 0;
        if (lead) {
            t_scan = global_ns();
            ph0 += t_scan - t_last;
        }
        bool scanned = true;
        uint32_t e2 = err;
        // with no survivor left the rows of this scan's removals name no node
        // that could still change
        while (!e2 && alive_n && (ns | nc)) {
            st.slot = step % 3;
            st.next = (step + 1) % 3;
            st.s_in = st.s_out;
            st.c_in = st.c_out;
            if (PACK) {
                st.s_out = j.qs + (uint64_t)st.next * j.qs_cap;
                st.c_out = j.qc + (uint64_t)st.next * j.qc_cap;
            } else {  // the items of one level, step after step
                ns = min(ns, st.s_cap);
                nc = min(nc, st.c_cap);
                st.s_out += ns;
                st.c_out += nc;
                st.s_cap -= ns;
                st.c_cap -= nc;
            }
            if (lead) {
                c->tail[(step + 2) % 3][0].v = 0;
                c->tail[(step + 2) % 3][1].v = 0;
            }
            if (PACK) clear_masks(j, (step + 2) % 3, pns, pnc);
            phase_expand<MULTI, PACK>(j, st, ns, nc, scanned);
            grid_barrier(j, nbar, t_start, st.next, la, &sv);
            step++;
            pns = ns;
            pnc = nc;
            lv_items += ns + nc;
            rounds++;
            ns = sv.ns;
            nc = sv.nc;
            e2 = sv.err;
            scanned = false;
        }
        if (lead) {
            const uint64_t now = global_ns();
            if (j.trace && level < j.trace_levels) {
                unsigned long long* r = j.trace + (uint64_t)TRACE_W * level;
                r[0] = t_scan - t_last;
                r[1] = now - t_scan;
                r[2] = rounds;
                r[3] = lv_items;
                r[4] = alive_n;
            }
            ph1 += now - t_scan;
            t_last = now;
            items += lv_items;
        }
        const bool stop = alive_n && alive_n <= j.stop_alive;  // the same on every block
        level++;
        const bool done = e2 || alive_n == 0 || stop;
        if (!done && level > j.max_level) e2 = PEEL_ERR_LIMIT;  // the same on every block
        if (done || e2) {
            if (lead) {
                c->ph_ns[0] = ph0;
                c->ph_ns[1] = ph1;
                c->levels = level;
                c->items = items;
                c->err_level = level - 1;
                if (stop && !e2) {
                    c->stopped = 1;
                    c->stop_level = level - 1;
                    c->stop_list = (level - 1) & 1;
                    c->stop_alive = alive_n;
                }
                if (e2 == PEEL_ERR_LIMIT) atomicCAS(&c->err.v, PEEL_OK, PEEL_ERR_LIMIT);
            }
            return;
        }
    }
}

// ---- host ---------------------------------------------------------------------

static uint32_t env_u32(const char* name, uint32_t dflt) {
    const char* s = getenv(name);
    return s && *s ? (uint32_t)strtoul(s, nullptr, 10) : dflt;
}

template <int T, bool MULTI, bool PACK, int BPS = 1024 / T>
static fc_status launch_t(PeelJob& j, cudaStream_t s) {
    int dev = 0, sms = 0, occ = 0;
    FC_CUDA_TRY(cudaGetDevice(&dev));
    FC_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    FC_CUDA_TRY(
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_peel<T, MULTI, PACK, BPS>, T, 0));
    if (occ < 1) return FC_ERR_DEVICE;
    uint32_t want_occ = env_u32("FC_PEEL_BLOCKS_PER_SM", BPS);
    if (want_occ >= 1 && (int)want_occ < occ) occ = (int)want_occ;
    if (j.max_sms && (int)j.max_sms < sms) sms = (int)j.max_sms;
    dim3 grid(sms * occ), block(T);
    void* args[] = {&j};
    FC_CUDA_TRY(cudaLaunchCooperativeKernel((void*)k_peel<T, MULTI, PACK, BPS>, grid, block, args,
                                            0, s));
    return FC_OK;
}

template <int T>
static fc_status launch_m(PeelJob& j, bool pack, cudaStream_t s) {
    if (j.nseg > 1) return pack ? launch_t<T, true, true>(j, s) : launch_t<T, true, false>(j, s);
    return pack ? launch_t<T, false, true>(j, s) : launch_t<T, false, false>(j, s);
}

static fc_status launch(PeelJob& j, bool pack, uint32_t threads, cudaStream_t s) {
    return threads == 512 ? launch_m<512>(j, pack, s) : launch_m<1024>(j, pack, s);
}

static uint32_t default_threads() { return env_u32("FC_PEEL_THREADS", 1024) == 512 ? 512 : 1024; }

// Nodes at which late.cu takes over from the peel (FC_PEEL_LATE; 0: never; at
// most the 2^20 an item of late.cu can name).  Its rounds have the shorter
// chain, but it writes the rows that are left once more and its rows are not
// ordered.  A graph that it can take from the first level it should, unless
// its degrees are far more than L2 holds, where both forms wait for memory and
// the copy is for nothing: 300,001 nodes x 10 layers 5.36 ms against 6.43 with
// 262,144 of them, 900,000 x 13 (374 MB of degrees) 12.8 against 14.2, but
// 600,000 x 24 (691 MB) 14.5 against 13.7.  With more nodes than it can take
// it should start late: 2.6M x 24 33.0 ms at 262,144 and 34.7 at 2^20, 180,001
// x 17 26.7 at 131,072 (24.8 from the first level).  With several segments the
// peel looks up an entry's segment at each access: 24 graphs of 546,404 nodes
// together 31.5 ms at 262,144 and 27.5 at 2^20.
static uint64_t late_nodes(bool several, uint64_t nodes, uint64_t degree_bytes) {
    const bool all = nodes <= (1u << 20) && degree_bytes <= (512ull << 20);
    const uint32_t most = several || all ? 1u << 20 : 262144u;
    const uint64_t n = env_u32("FC_PEEL_ENDGAME", 1) ? env_u32("FC_PEEL_LATE", most) : 0;
    return n < (1u << 20) ? n : (1u << 20);
}

uint32_t peel_kind(const PeelGraph& g) {
    return g.L > MAX_PACKED_LAYERS ? 2u : g.L > LATE_MAX_LAYERS ? 1u : 0u;
}

// Packed: four columns' degrees share a word, a step's queues and masks are
// kept apart from those of the steps around it.  Unpacked (one column per
// segment, 32-bit degrees, one queue): when every spec is a single column and
// no late form follows, where packing would only waste the other three fields,
// when a count of layers does not fit a field, and when a degree may pass it
// without as many nodes.
static bool packs(const PeelSegSpec* specs, size_t count, bool late) {
    bool several = late;
    for (size_t i = 0; i < count; i++) {
        if (specs[i].g.L > MAX_PACKED_LAYERS || specs[i].g.repeats) return false;
        several |= specs[i].ncols > 1;
    }
    return several;
}

// One launch over some columns of some graphs: its segments and where its
// scratch lies in one workspace.
struct PeelPlan {
    std::vector<SegP> segs;      // scratch pointers as offsets until carved
    std::vector<uint32_t> xb;
    bool pack = false;
    uint64_t nx = 0, qc_cap = 0, hub_cap = 0, hub_stride = 0;
    uint64_t total = 0;          // bytes
    uint64_t o_segs = 0, o_xb = 0, o_M = 0, o_P = 0, o_alive = 0, o_qs = 0, o_qc = 0, o_hub = 0,
             o_ex = 0, o_ctl = 0;
    std::vector<uint64_t> o_deg, o_cnt;
    uint32_t G = 1, max_level = 1;
    // each counter of a HUB node on a 128-byte line of its own while that is
    // little (64 MB): the whole grid decrements a few hubs, and atomics on one
    // line take turns (2.5M nodes x 4 layers, 16 hub counters: the levels that
    // remove the leaves take half the time)
    static constexpr uint64_t HUB_PAD_MOST = 1ull << 19;
    uint32_t hub_pad() const { return hub_cap * hub_stride <= HUB_PAD_MOST ? 32u : 1u; }
    bool late = false;           // late.cu takes the last levels, or all of them
    bool split = false;          // late.cu's scratch is not in the workspace but at late_ws
    void* late_ws = nullptr;
    uint64_t o_late = 0;
    LatePlan lp;
};

static void plan_peel(const PeelSegSpec* specs, size_t count, PeelPlan* p, bool late = false,
                      bool split = false) {
    uint64_t deg_bytes = 0, all_nodes = 0;
    for (size_t i = 0; i < count; i++) {
        all_nodes += specs[i].g.n;
        deg_bytes += 8ull * specs[i].g.n * specs[i].g.L * ((specs[i].ncols + 3) / 4);
    }
    const uint64_t stop =
        late_nodes(count > 1 || (count && specs[0].ncols > MAX_COLS), all_nodes, deg_bytes);
    late = late && stop && late_takes(specs, count);
    p->pack = packs(specs, count, late);
    uint64_t at = 0;
    auto take = [&](uint64_t bytes) {
        const uint64_t o = at;
        at = (at + bytes + 255) & ~255ull;
        return o;
    };
    const uint32_t word = p->pack ? 8 : 4;
    const uint32_t most = p->pack ? MAX_COLS : 1u;
    // what late.cu may be handed: every node when there are few (no peel runs
    // then), else the nodes left when the peel stops
    uint64_t lt_nodes = 0, lt_words = 0, lt_entries = 0, lt_items = 0, lt_most = 0;
    for (size_t i = 0; i < count; i++)
        lt_nodes += (uint64_t)specs[i].g.n * ((specs[i].ncols + most - 1) / most);
    p->late = late && p->pack;
    uint32_t max_deg = 0;
    bool bound = false;
    for (size_t i = 0; i < count; i++) {
        max_deg = std::max(max_deg, specs[i].g.max_level);
        bound |= specs[i].g.bound;
    }
    const bool fresh = p->late && lt_nodes <= stop && max_deg <= FIELD_MAX + 1;
    if (!fresh && lt_nodes > stop) lt_nodes = stop;
    for (size_t i = 0; i < count; i++) {
        const PeelSegSpec& sp = specs[i];
        const PeelGraph& g = sp.g;
        // groups of columns of about equal size, whole words
        const uint32_t ng = (sp.ncols + most - 1) / most;
        uint32_t per = (sp.ncols + ng - 1) / ng;
        if (p->pack) per = (per + 3) & ~3u;
        for (uint32_t c = 0; c < sp.ncols; c += per) {
            SegP s{};
            s.n = g.n;
            s.L = g.L;
            s.col0 = sp.col0 + c;
            s.ncols = sp.ncols - c < per ? sp.ncols - c : per;
            s.Q = p->pack ? (s.ncols + 3) / 4 : 1u;
            s.xbase = (uint32_t)p->nx;
            s.divL.init(g.L);
            s.node_ptr = g.node_ptr;
            s.adj = g.adj;
            s.deg0 = g.deg0;
            s.t = sp.table + (uint64_t)s.col0 * g.n;
            s.big_id = g.big_id;
            s.ptab = g.ptab;
            p->segs.push_back(s);
            p->xb.push_back((uint32_t)p->nx);
            // (a run that starts in the late form has no peel)
            p->o_deg.push_back(take(fresh ? 0 : (uint64_t)g.n * g.L * s.Q * word));
            p->o_cnt.push_back(take(fresh ? 0 : (uint64_t)g.n * s.Q * word));
            lt_words += (uint64_t)g.n * g.L;
            lt_most = std::max<uint64_t>(lt_most, g.L);
            lt_entries += g.entries;
            // A step may queue a node once per column, but rarely does: a run
            // that needs more than this is done again without the late form.
            lt_items += 2 * (g.entries / LATE_CHUNK + std::min<uint64_t>(g.n, lt_nodes));
            p->nx += g.n;
            // a step queues each node at most once: as one short item, or as
            // at most entries/CHUNK + 1 chunk items
            p->qc_cap += g.n + (g.entries + CHUNK - 1) / CHUNK;
            p->G = s.Q > p->G ? s.Q : p->G;
            if (p->pack && g.max_level > FIELD_MAX + 1) {  // a degree may pass a field
                p->hub_cap += g.entries / (FIELD_MAX + 1) + 1;
                const uint64_t st = (uint64_t)g.L * s.ncols;
                p->hub_stride = st > p->hub_stride ? st : p->hub_stride;
            }
        }
        p->max_level = g.max_level > p->max_level ? g.max_level : p->max_level;
    }
    p->xb.push_back((uint32_t)p->nx);
    const uint64_t keep = p->pack ? 3 : 1;
    if (p->segs.size() > 1) {
        p->o_segs = take(p->segs.size() * sizeof(SegP));
        p->o_xb = take(4ull * (p->segs.size() + 1));
    }
    if (!fresh) {
        p->o_M = take(4 * p->nx);
        p->o_alive = take(8 * p->nx);
        p->o_qs = take(4 * keep * p->nx);
        p->o_qc = take(8 * keep * p->qc_cap);
        if (p->hub_cap) {
            p->o_hub = take(4 * p->nx);
            uint64_t ex = p->hub_pad() * p->hub_cap * p->hub_stride;
            if (bound) ex = std::max(ex, 32 * std::min(p->hub_cap * p->hub_stride,
                                                       PeelPlan::HUB_PAD_MOST));
            p->o_ex = take(4 * ex);
        }
    }
    if (p->late) {
        const uint32_t most_items = env_u32("FC_PEEL_LATE_ITEMS", 0);
        if (most_items && lt_items > most_items) lt_items = most_items;
        p->lp.init(p->nx, lt_nodes, std::min(lt_words, lt_nodes * lt_most), lt_entries, lt_items,
                   p->G, fresh);
        p->split = split && !fresh;
        if (!p->split) p->o_late = take(p->lp.total);
    }
    p->o_P = p->pack && !fresh ? take(12 * p->nx) : at;  // cleared with the control block
    p->o_ctl = take(sizeof(PeelCtl));
    p->total = at + 256;  // the workspace may start anywhere
}

// what a run may need: with the late form, also its repetition without
static uint64_t run_bytes(const PeelSegSpec* specs, size_t count, bool late) {
    PeelPlan p;
    plan_peel(specs, count, &p, false);
    uint64_t bytes = p.total;
    if (late) {
        PeelPlan q;
        plan_peel(specs, count, &q, true);
        bytes = std::max(bytes, q.total);
    }
    return bytes;
}

// As many columns as keep the peel's scratch within a budget
// (FC_PEEL_GROUP_MB, default 4 GiB); the late form's comes on top.
uint32_t peel_columns_per_group(const DeviceGraph* d) {
    const PeelGraph g{d->n, d->L, d->entries, nullptr, nullptr, nullptr, d->max_deg + 1};
    const uint64_t budget = (uint64_t)env_u32("FC_PEEL_GROUP_MB", 4096) << 20;
    uint32_t cols = std::min(env_u32("FC_PEEL_GROUP_COLS", 0), d->L);
    if (!cols) {
        uint32_t fit = 0, no = d->L + 1;  // cols in [fit, no)
        for (cols = d->L; no - fit > 1; cols = fit + (no - fit) / 2) {
            if (cols <= 1 || peel_ws_bytes(g, cols) <= budget) fit = cols;
            else no = cols;
        }
        cols = fit;
    }
    if (cols < 1) cols = 1;
    // the (column, node) index must stay below 2^32
    while (cols > 1 && (uint64_t)cols * d->n >= (1ull << 32)) cols--;
    return cols;
}

uint64_t peel_ws_bytes(const PeelGraph& g, uint32_t ncols, bool late) {
    const PeelSegSpec sp{g, 0, ncols, nullptr};
    return run_bytes(&sp, 1, late);
}

// The job of a plan in the workspace; the segment table goes to the device on
// s when there is more than one segment.
static fc_status carve(PeelPlan& p, void* ws, size_t ws_bytes, cudaStream_t s, PeelJob* j) {
    if (p.total > ws_bytes) return FC_ERR_INVALID;
    if (p.nx >= (1ull << 32) || p.qc_cap >= (1ull << 32) || p.hub_cap >= (1ull << 31))
        return FC_ERR_TOO_LARGE;
    char* const w = (char*)(((uintptr_t)ws + 255) & ~(uintptr_t)255);
    for (size_t i = 0; i < p.segs.size(); i++) {
        p.segs[i].deg = w + p.o_deg[i];
        p.segs[i].cnt = w + p.o_cnt[i];
    }
    *j = PeelJob{};
    j->seg0 = p.segs[0];
    j->nseg = (uint32_t)p.segs.size();
    j->nx = (uint32_t)p.nx;
    j->G = p.G;
    j->M = (uint32_t*)(w + p.o_M);
    for (int i = 0; i < 3; i++) j->P[i] = (uint32_t*)(w + p.o_P) + (uint64_t)i * p.nx;
    j->alive[0] = (uint32_t*)(w + p.o_alive);
    j->alive[1] = j->alive[0] + p.nx;
    j->qs = (uint32_t*)(w + p.o_qs);
    j->qc = (u64*)(w + p.o_qc);
    j->qs_cap = (uint32_t)p.nx;
    j->qc_cap = (uint32_t)p.qc_cap;
    if (p.hub_cap && !(p.late && p.lp.fresh)) {
        j->hub_idx = (uint32_t*)(w + p.o_hub);
        j->hub_ex = (int*)(w + p.o_ex);
        j->hub_cap = (uint32_t)p.hub_cap;
        j->hub_stride = (uint32_t)p.hub_stride;
        j->hub_pad = p.hub_pad();
    }
    j->ctl = (PeelCtl*)(w + p.o_ctl);
    j->max_level = p.max_level;
    j->stop_alive = p.late ? (uint32_t)p.lp.nodes : 0u;
    // a late field must hold any degree left: at most the nodes, each in one layer
    if (j->stop_alive > FIELD_MAX && p.hub_cap) j->stop_alive = FIELD_MAX;
    if (j->nseg > 1) {
        j->segs = (const SegP*)(w + p.o_segs);
        j->seg_xbase = (const uint32_t*)(w + p.o_xb);
        FC_TRY(to_device(w + p.o_segs, p.segs.data(), p.segs.size() * sizeof(SegP), s));
        FC_TRY(to_device(w + p.o_xb, p.xb.data(), p.xb.size() * 4, s));
    }
    return FC_OK;
}

// The masks and the control block start all zero (they are contiguous).
static fc_status reset_job(const PeelJob& j, bool pack, cudaStream_t s) {
    char* const from = pack ? (char*)j.P[0] : (char*)j.ctl;
    FC_CUDA_TRY(cudaMemsetAsync(from, 0, (size_t)((char*)(j.ctl + 1) - from), s));
    return FC_OK;
}

// A run that needs longer queues than the late form's is done again without it,
// as part of the same run.
struct Again {
    bool needed = false;
    uint64_t t_start = 0;  // when the run began
};

// Launches the prepared job and reads its control block back.
static fc_status run_job(PeelJob& j, const PeelPlan& p, uint32_t threads, cudaStream_t s, PeelStats* st,
                         bool instrument, uint32_t col0, uint32_t ncols, bool* use_graph,
                         Again* again) {
    const bool pack = p.pack;
    char* const lw =
        p.split ? (char*)p.late_ws : (char*)j.ctl - p.o_ctl + p.o_late;  // late.cu's scratch
    // the launches of the run
    auto go = [&]() -> fc_status {
        FC_TRY(reset_job(j, pack, s));
        if (!(p.late && p.lp.fresh)) FC_TRY(launch(j, pack, threads, s));
        return p.late ? late_launch(j, p.lp, lw, s) : FC_OK;
    };
    if (!j.small_row) j.small_row = env_u32("FC_PEEL_SMALL_ROW", SMALL_ROW_DEFAULT);
    j.timeout_ns = (uint64_t)env_u32("FC_BARRIER_TIMEOUT_MS", 10000) * 1000000ull;
    j.deadline_ns = (uint64_t)env_u32("FC_PEEL_DEADLINE_MS", 60000) * 1000000ull;
    j.trace = nullptr;
    j.trace_levels = 0;
    const bool tracing = instrument && env_u32("FC_PEEL_TRACE", 0) != 0;
    const uint64_t trace_bytes = 8ull * TRACE_W * ((uint64_t)j.max_level + 2);
    if (tracing) {
        j.trace_levels = j.max_level + 2;
        FC_TRY(dev_alloc((void**)&j.trace, trace_bytes, s));
        FC_CUDA_TRY(cudaMemsetAsync(j.trace, 0, trace_bytes, s));
    }
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (instrument) {
        FC_CUDA_TRY(cudaEventCreate(&e0));
        FC_CUDA_TRY(cudaEventCreate(&e1));
        count_alloc(2);
    }
    // the run: clear the masks and the control block, then the launch --
    // captured as one CUDA graph when asked (and when the driver captures a
    // cooperative launch), else issued directly
    bool graphed = false;
    if (use_graph && *use_graph) {
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        bool ok = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
        if (ok) {
            const fc_status r = go();
            ok = cudaStreamEndCapture(s, &graph) == cudaSuccess && r == FC_OK;
        }
        if (ok) ok = cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
        if (ok) {
            if (instrument) FC_CUDA_TRY(cudaEventRecord(e0, s));
            ok = cudaGraphLaunch(exec, s) == cudaSuccess;
            graphed = ok;
        }
        cudaGetLastError();  // a refused capture falls back to direct launches
        if (graph && !graphed) cudaGraphDestroy(graph);
        if (exec && !graphed) cudaGraphExecDestroy(exec);
        if (graphed) {
            if (instrument) FC_CUDA_TRY(cudaEventRecord(e1, s));
            FC_CUDA_TRY(cudaStreamSynchronize(s));
            cudaGraphExecDestroy(exec);
            cudaGraphDestroy(graph);
        }
    }
    if (!graphed) {
        if (instrument) FC_CUDA_TRY(cudaEventRecord(e0, s));
        FC_TRY(go());
        if (instrument) FC_CUDA_TRY(cudaEventRecord(e1, s));
    }
    if (use_graph) *use_graph = graphed;
    count_launch();
    PeelCtl out;
    FC_TRY(to_host(&out, j.ctl, sizeof(out), s));
    LateCtl lo[2] = {};
    if (p.late) {
        FC_TRY(to_host(lo, lw + p.lp.o_ctl, sizeof(lo), s));
        for (const LateCtl& c : lo)
            if (!out.err.v) {
                out.err.v = c.err.v;
                again->needed = c.err.v == PEEL_ERR_QUEUE;
            }
        again->t_start = lo[0].t_start;
        if (tracing)
            fprintf(stderr, "late-trace nodes %u entries %u first level %u levels %u\n", lo[0].m,
                    lo[0].entries, lo[0].first_level, lo[0].levels + lo[1].levels);
    }
    float ms = 0;
    if (instrument) {
        cudaEventElapsedTime(&ms, e0, e1);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    }
    if (st) {
        // times and items of all its launches (a repetition's after the first try's)
        st->ms += ms;
        st->levels = out.levels + lo[0].levels + lo[1].levels;
        st->subrounds += (uint32_t)(out.items + lo[0].queued + lo[1].queued);
        st->err = out.err.v;
        for (int i = 0; i < 2; i++)
            st->phase_ms[i] += (out.ph_ns[i] + lo[0].ph_ns[i] + lo[1].ph_ns[i]) * 1e-6;
    }
    if (tracing) {
        // one line per level: scan us, expansion us, rounds, queue items, alive nodes
        std::vector<unsigned long long> tr((size_t)TRACE_W * j.trace_levels);
        cudaMemcpy(tr.data(), j.trace, trace_bytes, cudaMemcpyDeviceToHost);
        dev_free(j.trace, s);
        for (uint32_t l = 0; l < j.trace_levels; l++) {
            const unsigned long long* r = tr.data() + (size_t)TRACE_W * l;
            if (r[0] || r[1])
                fprintf(stderr,
                        "peel-trace cols %u+%u level %u scan_us %.1f expand_us %.1f rounds %llu"
                        " items %llu alive %llu\n",
                        col0, ncols, l, r[0] * 1e-3, r[1] * 1e-3, r[2], r[3], r[4]);
        }
    }
    if (out.err.v) {
        if (env_u32("FC_DEBUG", 0))
            fprintf(stderr, "peel: error %u at level %u of %u (bad item %u, check %u), %u segments\n",
                    out.err.v, out.err_level, j.max_level, out.bad_item, out.bad_where, j.nseg);
        return FC_ERR_ITER_LIMIT;
    }
    return FC_OK;
}

static fc_status run_from(uint64_t t_start, const PeelGraph& g, uint32_t col0, uint32_t ncols,
                          uint32_t* table, void* ws, size_t ws_bytes, cudaStream_t s, PeelStats* st,
                          bool instrument, bool late, void* late_ws) {
    const PeelSegSpec sp{g, col0, ncols, table};
    PeelPlan p;
    plan_peel(&sp, 1, &p, late, late_ws != nullptr);
    p.late_ws = late_ws;
    PeelJob j;
    FC_TRY(carve(p, ws, ws_bytes, s, &j));
    j.t_start = t_start;
    Again again;
    const fc_status rc = run_job(j, p, default_threads(), s, st, instrument, col0, ncols, nullptr,
                                 &again);
    if (!again.needed) return rc;
    return run_from(again.t_start, g, col0, ncols, table, ws, ws_bytes, s, st, instrument, false,
                    nullptr);
}

fc_status peel_run(const PeelGraph& g, uint32_t col0, uint32_t ncols, uint32_t* table, void* ws,
                   size_t ws_bytes, cudaStream_t s, PeelStats* st, bool instrument, bool late,
                   void* late_ws) {
    return run_from(0, g, col0, ncols, table, ws, ws_bytes, s, st, instrument, late, late_ws);
}

uint64_t peel_batch_ws_bytes(const std::vector<PeelSegSpec>& specs, bool late) {
    return run_bytes(specs.data(), specs.size(), late);
}

bool peel_batch_peels(const std::vector<PeelSegSpec>& specs, bool late) {
    PeelPlan p;
    plan_peel(specs.data(), specs.size(), &p, late);
    return !(p.late && p.lp.fresh);
}

void peel_defaults(uint32_t* threads, uint32_t* small_row) {
    *threads = default_threads();
    *small_row = env_u32("FC_PEEL_SMALL_ROW", SMALL_ROW_DEFAULT);
}

static fc_status batch_from(uint64_t t_start, const std::vector<PeelSegSpec>& specs, void* ws,
                            size_t ws_bytes, cudaStream_t s, PeelStats* st, uint32_t threads,
                            uint32_t small_row, bool* use_graph, uint32_t max_sms, bool late) {
    if (specs.empty()) return FC_OK;
    PeelPlan p;
    plan_peel(specs.data(), specs.size(), &p, late);
    PeelJob j;
    FC_TRY(carve(p, ws, ws_bytes, s, &j));
    j.small_row = small_row;
    j.max_sms = max_sms;
    j.t_start = t_start;
    if (!threads) threads = default_threads();
    // the segment table must be on the device before a captured launch runs
    if (use_graph && *use_graph) FC_CUDA_TRY(cudaStreamSynchronize(s));
    Again again;
    const bool want_graph = use_graph && *use_graph;
    const fc_status rc =
        run_job(j, p, threads, s, st, true, specs[0].col0, specs[0].ncols, use_graph, &again);
    if (!again.needed) return rc;
    if (use_graph) *use_graph = want_graph;
    return batch_from(again.t_start, specs, ws, ws_bytes, s, st, threads, small_row, use_graph,
                      max_sms, false);
}

fc_status peel_batch(const std::vector<PeelSegSpec>& specs, void* ws, size_t ws_bytes,
                     cudaStream_t s, PeelStats* st, uint32_t threads, uint32_t small_row,
                     bool* use_graph, uint32_t max_sms, bool late) {
    return batch_from(0, specs, ws, ws_bytes, s, st, threads, small_row, use_graph, max_sms, late);
}

void peel_preload() {
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, k_peel<512, false, false>);
    cudaFuncGetAttributes(&a, k_peel<512, false, true>);
    cudaFuncGetAttributes(&a, k_peel<512, true, false>);
    cudaFuncGetAttributes(&a, k_peel<512, true, true>);
    cudaFuncGetAttributes(&a, k_peel<1024, false, false>);
    cudaFuncGetAttributes(&a, k_peel<1024, false, true>);
    cudaFuncGetAttributes(&a, k_peel<1024, true, false>);
    cudaFuncGetAttributes(&a, k_peel<1024, true, true>);
    whole_preload();
    late_preload();
    cudaGetLastError();
}

fc_status peel_columns(DeviceGraph* d, uint32_t col0, uint32_t ncols, cudaStream_t s,
                       PeelStats* st, bool late) {
    PeelGraph g{d->n, d->L, d->entries, d->node_ptr, d->adj, d->deg0, d->max_deg + 1, d->big_id,
                d->ptab};
    if (fits_whole(g, ncols)) {
        FC_TRY(ensure_ws(d, whole_ws_bytes(ncols), s));
        return whole_run(g, col0, ncols, d->table, d->ws, s, st);
    }
    // The late form's scratch after a peel is an allocation of its own: in one
    // with the peel's it fits none of the pool's free blocks after an upload,
    // and the pool maps memory anew for it in each step of a program that
    // uploads, peels and releases (2.44M nodes x 4 layers: 1.9 ms of a peel of
    // 14.7 ms, and 1.8 ms of the next upload).
    const PeelSegSpec sp{g, col0, ncols, d->table};
    PeelPlan p, q;
    plan_peel(&sp, 1, &p, false);
    plan_peel(&sp, 1, &q, late, true);
    const uint64_t late_bytes = q.split ? q.lp.total : 0;
    fc_status rc = ensure_ws(d, std::max(p.total, q.total), s);
    if (rc == FC_OK && d->late_bytes < late_bytes) {
        dev_free(d->late_ws, s);
        d->late_ws = nullptr;
        d->late_bytes = 0;
        rc = dev_alloc(&d->late_ws, late_bytes, s);
        if (rc == FC_OK) d->late_bytes = late_bytes;
    }
    if (rc == FC_ERR_OOM && late) {  // no room for the late form's scratch
        cudaGetLastError();
        late = false;
        rc = ensure_ws(d, p.total, s);
    }
    FC_TRY(rc);
    return peel_run(g, col0, ncols, d->table, d->ws, d->ws_bytes, s, st, true, late,
                    late && late_bytes ? d->late_ws : nullptr);
}

}  // namespace fc
