// What the peel (peel.cu) and the form that takes its last levels over
// (late.cu) share: the control block, the segments and the packed fields.
#pragma once

#include "device.h"

namespace fc {

// PEEL_ERR_BARRIER: a barrier made no progress for the timeout.  PEEL_ERR_LIMIT: more
// levels than the largest degree allows.  PEEL_ERR_QUEUE: a queue overflowed.
// PEEL_ERR_DEADLINE: the whole run took longer than its deadline.  PEEL_ERR_ITEM: a
// queued item named no node of the launch (recorded and skipped).
enum : uint32_t {
    PEEL_OK = 0, PEEL_ERR_BARRIER = 1, PEEL_ERR_LIMIT = 2, PEEL_ERR_QUEUE = 3,
    PEEL_ERR_DEADLINE = 4, PEEL_ERR_ITEM = 5
};

// Columns of one segment: four per 64-bit word in at most seven words, so
// that bit 31 of a node's mask is free for HUB.
constexpr uint32_t MAX_COLS = 28;
constexpr uint32_t COLS_MASK = (1u << MAX_COLS) - 1u;
// A node with a layer degree above 65,535: what its 16-bit fields cannot hold
// sits in counters beside them (absorb).
constexpr uint32_t HUB = 0x80000000u;
constexpr uint32_t FIELD_MAX = 0xFFFFu;
// a count of layers is a 16-bit field too: graphs with more layers are peeled
// one column per segment, unpacked
constexpr uint32_t MAX_PACKED_LAYERS = 32767;

// rows longer than the job's small_row entries are expanded as CHUNK-entry
// work items
constexpr uint32_t SMALL_ROW_DEFAULT = 64;
constexpr uint32_t CHUNK = 256;

// A counter alone on its 128-byte line.
struct alignas(128) Hot {
    uint32_t v;
};

struct alignas(128) Hot64 {
    unsigned long long v;
};

struct PeelCtl {
    Hot arrive;         // blocks that reached the grid barriers so far
    Hot tail[3][2];     // [step mod 3][short, chunk]: items queued for the step
    Hot alive_cnt[3];   // [scan mod 3] survivors
    Hot err;
    uint64_t ph_ns[2];  // time in scans, in expansions
    uint32_t levels, items, err_level, nhub;
    uint32_t bad_item, bad_where;  // what PEEL_ERR_ITEM saw
    uint64_t t_start;   // when the run began (the deadline counts from there)
    // the run stopped: the nodes alive after level stop_level are in list
    // `stop_list`, stop_alive entries (some of them removed since its scan)
    uint32_t stopped, stop_level, stop_list, stop_alive;
};

// One segment: a graph's group of columns, as the kernel reads it.
struct SegP {
    uint32_t xbase;            // first x of the segment
    uint32_t n, L, col0;
    FastDiv divL;
    const uint32_t* node_ptr;
    const uint32_t* adj;
    const uint32_t* deg0;
    void* deg;                 // n * L * Q words: degrees inside the alive sets
    void* cnt;                 // n * Q words: layers with degree >= K+1
    uint32_t* t;               // table + col0 * n
    const uint32_t* big_id;    // ordered long rows (device.h), or null
    const uint32_t* ptab;
    uint32_t ncols, Q;         // Q: words per (node, layer)
};

struct PeelJob {
    SegP seg0;                     // the only segment when the launch has one
    const SegP* segs;              // nseg segments (device), when more than one
    const uint32_t* seg_xbase;     // nseg + 1 (device): segment starts, then nx
    uint32_t nseg, nx;
    uint32_t G;                    // lanes per node in SCAN: the largest Q
    uint32_t* M;                   // nx: columns in which x is not yet expanded, and HUB
    uint32_t* P[3];                // nx each: columns removed for the step (packed form)
    uint32_t* alive[2];            // nx each
    uint32_t* qs;                  // short-row items
    unsigned long long* qc;        // chunk items
    uint32_t qs_cap, qc_cap;       // per step; three steps' worth when packed
    uint32_t* hub_idx;             // nx: index of a HUB node's counters, or null
    int* hub_ex;                   // hub_cap * hub_stride
    uint32_t hub_cap, hub_stride, hub_pad;
    PeelCtl* ctl;
    uint32_t max_level;
    uint32_t small_row;   // longest row queued as one item; longer rows go in chunks
    uint64_t timeout_ns;  // longest wait at a barrier
    uint64_t deadline_ns; // longest whole run, all its launches together
    uint64_t t_start;     // when it began, for a repetition; else 0 (this launch begins it)
    // optional per-level trace: {scan ns, expand ns, rounds, items, alive}
    unsigned long long* trace;
    uint32_t trace_levels;
    uint32_t max_sms;     // host side: SMs the grid may cover (0 = every SM)
    uint32_t stop_alive;  // stop once a level starts with this many nodes or fewer
};
constexpr uint32_t TRACE_W = 5;

// ---- memory-model helpers -------------------------------------------------

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_add_release(uint32_t* p, uint32_t v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// whether a run that began at t_start is past its deadline
__device__ __forceinline__ bool past_deadline(uint64_t t_start, uint64_t deadline_ns) {
    return (int64_t)(global_ns() - t_start) > (int64_t)deadline_ns;
}
// A word that another thread may be writing in the same step, where the old
// value will do as well as the new one: the nodes' masks, which an expansion
// tests while their owners clear columns.  (Plain accesses would race.)
__device__ __forceinline__ uint32_t ld_either(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void st_either(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ---- packed fields ----------------------------------------------------------

typedef unsigned long long u64;

// bit i of m4 (i < 4) as a 1 in field i
__device__ __forceinline__ u64 spread4(uint32_t m4) {
    return ((u64)m4 * 0x0000200040008001ull) & 0x0001000100010001ull;
}
// a 1 in field i as bit i
__device__ __forceinline__ uint32_t gather4(u64 f) {
    return (uint32_t)(f | (f >> 15) | (f >> 30) | (f >> 45)) & 15u;
}
__device__ __forceinline__ u64 all4(uint32_t v) { return (u64)v * 0x0001000100010001ull; }
// a 1 in every field of z that is zero
__device__ __forceinline__ u64 zero4(u64 z) {
    const u64 low = 0x7FFF7FFF7FFF7FFFull;
    return (~(((z & low) + low) | z | low)) >> 15;
}
// a 1 in every field of a that is >= the field of t (t in all fields)
__device__ __forceinline__ u64 geq4(u64 a, uint32_t t2) {
    const uint32_t lo = __vsetgeu2((uint32_t)a, t2), hi = __vsetgeu2((uint32_t)(a >> 32), t2);
    return ((u64)hi << 32) | lo;
}

// ---- segments ---------------------------------------------------------------

template <bool MULTI>
__device__ __forceinline__ uint32_t seg_of(const PeelJob& j, uint32_t x) {
    if (!MULTI) return 0;
    uint32_t lo = 0, hi = j.nseg;  // seg_xbase[lo] <= x < seg_xbase[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(j.seg_xbase + mid) <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

template <class T>
__device__ __forceinline__ T* ldg_ptr(T* const* p) {
    return (T*)__ldg((const unsigned long long*)p);
}

template <bool MULTI>
__device__ __forceinline__ SegP seg_load(const PeelJob& j, uint32_t s) {
    if (!MULTI) return j.seg0;
    SegP g;
    const SegP* p = j.segs + s;
    g.xbase = __ldg(&p->xbase);
    g.n = __ldg(&p->n);
    g.L = __ldg(&p->L);
    g.col0 = __ldg(&p->col0);
    g.divL.d = __ldg(&p->divL.d);
    g.divL.m = __ldg(&p->divL.m);
    g.divL.s1 = __ldg(&p->divL.s1);
    g.divL.s2 = __ldg(&p->divL.s2);
    g.node_ptr = ldg_ptr(&p->node_ptr);
    g.adj = ldg_ptr(&p->adj);
    g.deg0 = ldg_ptr(&p->deg0);
    g.deg = (void*)__ldg((const unsigned long long*)&p->deg);
    g.cnt = (void*)__ldg((const unsigned long long*)&p->cnt);
    g.t = ldg_ptr(&p->t);
    g.big_id = ldg_ptr(&p->big_id);
    g.ptab = ldg_ptr(&p->ptab);
    g.ncols = __ldg(&p->ncols);
    g.Q = __ldg(&p->Q);
    return g;
}

// ---- the late form (late.cu) -----------------------------------------------

// row entries of one item
constexpr uint32_t LATE_CHUNK = 128;
// the layers that an entry can name
constexpr uint32_t LATE_MAX_LAYERS = 512;

struct LateCtl {
    // [step mod 3] items queued in the step (low half) and blocks that have
    // ended it (high half): one load tells a waiting block both
    Hot64 step[3];
    Hot alive_cnt[3];   // [scan mod 3] survivors
    Hot err;
    uint32_t m, first_level, list, nfill, levels;  // where it starts: nodes, level, list
    uint32_t entries, words;  // row entries and degree words reserved
    uint64_t t_start;   // when the run began
    uint64_t ph_ns[2];  // time in scans, in expansions
    uint64_t queued;    // items
};

// Where the scratch of one run lies.
struct LatePlan {
    uint64_t nodes = 0, entries = 0, q_cap = 0, plane = 0, total = 0;
    uint32_t G = 1;
    bool fresh = false;
    uint64_t o_ctl = 0, o_row = 0, o_meta = 0, o_adj = 0, o_deg = 0, o_cnt = 0, o_M = 0, o_x = 0,
             o_id = 0, o_seg = 0, o_alive = 0, o_fill = 0, o_q = 0;
    void init(uint64_t nx, uint64_t nodes, uint64_t words, uint64_t entries, uint64_t items,
              uint32_t G, bool fresh);
};

bool late_takes(const PeelSegSpec* specs, size_t count);
// The kernels that finish a packed peel that stopped (or did not run:
// p.fresh), with its scratch at w; nothing waits on the host.
fc_status late_launch(const PeelJob& pj, const LatePlan& p, char* w, cudaStream_t s);
void late_preload();

// ---- small graphs (whole.cu) -----------------------------------------------

// whether the graph fits one block's or one cluster's shared memory per column
bool fits_whole(const PeelGraph& g, uint32_t ncols);
uint64_t whole_ws_bytes(uint32_t ncols);
fc_status whole_run(const PeelGraph& g, uint32_t col0, uint32_t ncols, uint32_t* table, void* ws,
                    cudaStream_t s, PeelStats* st);
void whole_preload();

}  // namespace fc
