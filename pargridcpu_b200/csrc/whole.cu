// Graphs small enough for the shared memory of one block, or of one
// thread-block cluster per column: every column peels the whole graph there,
// with the rules of peel.cu and no grid barrier.
#include <cooperative_groups.h>

#include <cstdlib>
#include <mutex>
#include <vector>

#include "device.h"
#include "peel_common.h"

namespace cg = cooperative_groups;

namespace fc {

// Warp-wide inclusive scan.
__device__ __forceinline__ uint32_t wh_incl_scan(uint32_t v) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (uint32_t)o) v += y;
    }
    return v;
}

// ---- the whole graph per column on one block ----------------------------------
//
// A graph whose nodes fit one block's shared memory is not worth a grid
// barrier: every column peels it on one block, with the same rules -- degrees,
// counts, alive flags, lists and queue in shared memory, rounds separated by
// __syncthreads.  Every loop is bounded (levels by the level cap, rounds by
// the nodes); no block waits on another.

constexpr uint32_t WH_THREADS = 1024;
constexpr uint32_t WH_SMEM = 220u * 1024u;  // dynamic shared memory of k_whole

// shared bytes per node: degrees (L halves), count (a half), alive flag, two
// alive lists and the queue (16-bit ids)
static uint32_t wh_node_bytes(uint32_t L) { return 2 * L + 9; }
static uint32_t wh_capacity(uint32_t L) {
    const uint64_t fixed = 8ull * WH_THREADS + 256;  // batch prefixes and row starts + alignment
    const uint64_t cap = (WH_SMEM - fixed) / wh_node_bytes(L);
    return cap > 65535 ? 65535u : (uint32_t)cap;
}

// Block-wide exclusive scan of the 1024 threads' values; returns the total.
__device__ __forceinline__ uint32_t wh_block_scan(uint32_t v, uint32_t* excl, uint32_t* s_warp) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t in = wh_incl_scan(v);
    __syncthreads();
    if (lane == 31) s_warp[w] = in;
    __syncthreads();
    if (w == 0) {
        const uint32_t x = s_warp[lane], y = wh_incl_scan(x);
        s_warp[lane] = y - x;  // exclusive
        if (lane == 31) s_warp[32] = y;
    }
    __syncthreads();
    *excl = s_warp[w] + in - v;
    const uint32_t total = s_warp[32];
    __syncthreads();
    return total;
}

__device__ __forceinline__ uint32_t wh_get16(const uint32_t* w, uint32_t i) {
    return (w[i >> 1] >> ((i & 1) * 16)) & 0xFFFFu;
}
// decrements half i of w; returns its old value.  A half is only decremented
// while it is at least 1 (every decrement stands for a neighbour it counts),
// so no borrow reaches the other half.
__device__ __forceinline__ uint32_t wh_dec16(uint32_t* w, uint32_t i) {
    const uint32_t sh = (i & 1) * 16;
    return (atomicSub(w + (i >> 1), 1u << sh) >> sh) & 0xFFFFu;
}

// One block per column: the levels 0, 1, ... of the column until no node is
// left (or the level cap, an error).
__global__ void __launch_bounds__(WH_THREADS) k_whole(
    const uint32_t* __restrict__ rp, const uint32_t* __restrict__ adj,
    const uint32_t* __restrict__ deg0, uint32_t m, uint32_t L, FastDiv divL,
    uint32_t* __restrict__ t, uint32_t col0, uint32_t max_level, uint32_t* __restrict__ levels,
    uint32_t* __restrict__ err) {
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ uint32_t s_warp[33];
    __shared__ uint32_t s_nalive, s_next, s_tail;
    const uint32_t c = blockIdx.x;
    const uint32_t lmd = col0 + c + 1;
    uint32_t* tc = t + (uint64_t)c * m;
    // shared layout: degrees | counts | batch prefixes | batch row starts |
    // alive | lists | queue
    uint32_t* dw = sm;                                   // (m * L + 1) / 2 words
    uint32_t* cw = dw + ((uint64_t)m * L + 1) / 2;       // (m + 1) / 2 words
    uint32_t* pre = cw + (m + 1) / 2;                    // WH_THREADS words
    uint32_t* rs = pre + WH_THREADS;                     // WH_THREADS words
    uint8_t* alive = (uint8_t*)(rs + WH_THREADS);        // m bytes
    uint16_t* list0 = (uint16_t*)(((uintptr_t)(alive + m) + 3) & ~(uintptr_t)3);
    uint16_t* list1 = list0 + m;
    uint16_t* queue = list1 + m;
    for (uint32_t i = threadIdx.x; i < ((uint64_t)m * L + 1) / 2; i += blockDim.x) dw[i] = 0;
    for (uint32_t i = threadIdx.x; i < (m + 1) / 2; i += blockDim.x) cw[i] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < m * L; i += blockDim.x)
        atomicOr(dw + (i >> 1), (deg0[i] & 0xFFFFu) << ((i & 1) * 16));
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
        alive[i] = 1;
        list0[i] = (uint16_t)i;
    }
    if (threadIdx.x == 0) s_nalive = m;
    __syncthreads();
    uint16_t* cur = list0;
    uint16_t* nxt = list1;
    uint32_t k = 0;
    for (;;) {
        const uint32_t na = s_nalive;
        if (na == 0) break;
        if (k > max_level) {
            if (threadIdx.x == 0) atomicExch(err, 2u);
            break;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s_next = 0;
            s_tail = 0;
        }
        __syncthreads();
        // SCAN(k)
        for (uint32_t i = threadIdx.x; i < na; i += blockDim.x) {
            const uint32_t x = cur[i];
            if (!alive[x]) continue;
            uint32_t cnt = 0;
            for (uint32_t l = 0; l < L; l++) cnt += wh_get16(dw, x * L + l) >= k + 1;
            if (cnt < lmd) {
                alive[x] = 0;
                tc[x] = k;
                queue[atomicAdd(&s_tail, 1u)] = (uint16_t)x;
            } else {
                atomicOr(cw + (x >> 1), cnt << ((x & 1) * 16));  // the half was 0
                nxt[atomicAdd(&s_next, 1u)] = (uint16_t)x;
            }
        }
        __syncthreads();
        // rounds over the queue, each round's rows flattened over the block in
        // batches of WH_THREADS items
        uint32_t qb = 0;
        for (uint32_t round = 0; round <= m; round++) {
            const uint32_t qe = s_tail;
            __syncthreads();
            if (qb >= qe) break;
            for (uint32_t b0 = qb; b0 < qe; b0 += WH_THREADS) {
                const uint32_t nb = min(WH_THREADS, qe - b0);
                uint32_t len = 0, start = 0;
                if (threadIdx.x < nb) {
                    const uint32_t x = queue[b0 + threadIdx.x];
                    start = rp[x];
                    len = rp[x + 1] - start;
                }
                uint32_t ex;
                const uint32_t total = wh_block_scan(len, &ex, s_warp);
                pre[threadIdx.x] = ex;
                rs[threadIdx.x] = start;
                __syncthreads();
                // four entries per thread at a time, their loads first
                uint32_t lo0 = 0;  // this thread's entries only move forward
                for (uint32_t e0 = threadIdx.x; e0 < total; e0 += 4 * blockDim.x) {
                    uint32_t slot[4];
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const uint32_t e = e0 + r * blockDim.x;
                        slot[r] = NO_BIG_ROW;
                        if (e < total) {
                            uint32_t lo = lo0, hi = nb - 1;  // last item whose prefix is <= e
                            while (lo < hi) {
                                const uint32_t mid = (lo + hi + 1) >> 1;
                                if (pre[mid] <= e) lo = mid;
                                else hi = mid - 1;
                            }
                            lo0 = lo;
                            slot[r] = adj[rs[lo] + (e - pre[lo])];
                        }
                    }
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        if (slot[r] == NO_BIG_ROW) continue;
                        const uint32_t u = divL.div(slot[r]);
                        if (u >= m || !alive[u]) continue;
                        const uint32_t old = wh_dec16(dw, slot[r]);
                        if (old == k + 1 && wh_dec16(cw, u) == lmd) {
                            alive[u] = 0;
                            tc[u] = k;
                            queue[atomicAdd(&s_tail, 1u)] = (uint16_t)u;
                        }
                    }
                }
                __syncthreads();
            }
            qb = qe;
        }
        // counts are rebuilt by the next SCAN: clear the kept ones
        for (uint32_t i = threadIdx.x; i < (m + 1) / 2; i += blockDim.x) cw[i] = 0;
        if (threadIdx.x == 0) s_nalive = s_next;
        uint16_t* tmp = cur;
        cur = nxt;
        nxt = tmp;
        k++;
        __syncthreads();
    }
    if (threadIdx.x == 0) levels[c] = k;
}

// ---- the whole graph per column on a thread-block cluster ----------------------
//
// The same levels as k_whole, with the graph's nodes spread over the CS blocks
// of one cluster (CS a power of two, at most 16): node i lives on block
// i % CS, at index i / CS of that block's degrees, count, alive flag and
// lists, and every block reaches the others' shared memory directly
// (distributed shared memory).  A level is a SCAN round, in which each block
// scans its own nodes, then expansion rounds: in each, every block expands
// the rows of its own nodes queued in the round before and its slice of
// every long row on block 0's list.  A removal its threads cause goes to
// that list when the node's row is long, else to one of the block's local
// halves, whose rows the block expands at once in further local iterations
// (separated by block barriers) until its threads cause no removal; only a
// removal that finds the local half full is queued on the removed node's
// owner for the next round.  Rounds are separated by cluster barriers.
// Block 0 holds, per round (three of them in rotation), the cluster-wide
// counts of nodes queued and of nodes a scan kept, and the long-row list;
// every block reads them right after the round's barrier, so all blocks take
// the same decisions.  The queue of round r+1 is the other half of a
// two-half queue, so a block never reads a slot another block may still be
// writing.  Every loop is bounded as in k_whole, and no block leaves while
// another may still reach its shared memory.
// Rows longer than CL_SPLIT entries are expanded by every block, a slice each.
constexpr uint32_t CL_SPLIT = 2048;
// The count half of a node that is not kept in the current level: decrements
// of a removed node's count (at most L, one per layer degree passing k + 1)
// leave it far above any lmd, and never borrow (L is at most 96 here: a
// block holds at least 1024 nodes at 2L + 11 shared bytes each, beside its
// fixed arrays; for larger L the cluster form is not used).
constexpr uint32_t CL_DEAD = 0x8000u;
constexpr uint32_t CL_DEAD2 = 0x80008000u;
// A kept node's count half is its count (bits 0-13) and, in bit 14, whether
// its row is long; a removed node's never matches lmd in bits 0-13.
constexpr uint32_t CL_BIG = 0x4000u;
constexpr uint32_t CL_CNT = 0x3FFFu;
// Long rows listed in one round, per cluster (more are expanded like short
// rows, by the block that found them removed or by their owners)
constexpr uint32_t CL_BIG_MAX = 256;
// Capacity of each of a block's two local halves: rows found removed by the
// block's own threads, expanded by the block before the round ends
constexpr uint32_t CL_LQ = 2048;
// set in block 0's count of a round by a block whose local iterations ran out
constexpr uint32_t CL_FAIL = 0x80000000u;

// Block 0's counters of round rho + 1 (pushes, kept nodes) and its long-row
// list of round rho + 2 start empty; called at the start of round rho, when
// every block has read what they held three rounds before.
__device__ __forceinline__ void cl_reset(uint32_t* cnt, uint32_t* kept, uint32_t* bign,
                                          uint32_t rho) {
    cnt[(rho + 1) % 3] = 0;
    kept[(rho + 1) % 3] = 0;
    bign[(rho + 2) % 3] = 0;
}

// adds the calling threads of a warp to a (remote) counter with one atomic
__device__ __forceinline__ void cl_count(uint32_t* p) {
    const uint32_t am = __activemask();
    if ((threadIdx.x & 31) == (uint32_t)(__ffs(am) - 1)) atomicAdd(p, (uint32_t)__popc(am));
}

// Block-wide exclusive scan of 32 warps' values with one barrier: each warp
// scans the warp totals itself.  Two calls need a barrier between them.
__device__ __forceinline__ uint32_t cl_block_scan(uint32_t v, uint32_t* excl, uint32_t* s_warp) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t in = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, in, d);
        if (lane >= (uint32_t)d) in += t;
    }
    if (lane == 31) s_warp[w] = in;
    __syncthreads();
    const uint32_t x = s_warp[lane];
    uint32_t y = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, y, d);
        if (lane >= (uint32_t)d) y += t;
    }
    *excl = __shfl_sync(0xffffffffu, y - x, w) + in - v;
    return __shfl_sync(0xffffffffu, y, 31);
}

// appends column-local node u to block 0's list of long rows for a round
__device__ __forceinline__ bool cl_push_big(uint32_t* big, uint32_t* bign, uint32_t slot,
                                             uint32_t u) {
    const uint32_t pos = atomicAdd(bign + slot, 1u);
    if (pos >= CL_BIG_MAX) return false;
    big[slot * CL_BIG_MAX + pos] = u;
    return true;
}

__device__ __forceinline__ uint32_t cl_dec16(uint32_t* w, uint32_t i) {
    const uint32_t sh = (i & 1) * 16;
    return (atomicSub(w + (i >> 1), 1u << sh) >> sh) & 0xFFFFu;
}

// shared bytes per node a block owns: degrees (L halves), count (a half),
// alive flag, two lists and two queue halves (16-bit indices); besides them
// the batch prefixes and row starts and the two local halves
static uint32_t cl_node_bytes(uint32_t L) { return 2 * L + 11; }
static uint32_t cl_block_capacity(uint32_t L) {
    const uint64_t fixed = 8ull * WH_THREADS + 4ull * CL_LQ + 256;
    uint64_t cap = (WH_SMEM - fixed) / cl_node_bytes(L);
    if (cap > 65535) cap = 65535;
    return cap >= 1024 ? (uint32_t)cap : 0u;
}
static uint64_t cl_smem_bytes(uint32_t mo, uint32_t L) {
    return 4ull * (((uint64_t)mo * L + 1) / 2 + (mo + 1) / 2 + 2ull * WH_THREADS) + mo + 4 +
           8ull * mo + 4ull * CL_LQ + 16;
}

__global__ void __launch_bounds__(WH_THREADS) k_whole_cl(
    const uint32_t* __restrict__ rp, const uint32_t* __restrict__ adj,
    const uint32_t* __restrict__ deg0, uint32_t m, uint32_t L, FastDiv divL,
    uint32_t* __restrict__ t, uint32_t col0, uint32_t max_level, uint32_t* __restrict__ levels,
    uint32_t* __restrict__ err) {
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ uint32_t s_warp[33];
    __shared__ uint32_t s_next, s_tail[2], s_lt[2];
    __shared__ uint32_t s_cnt[3], s_kept[3];  // block 0's are the cluster's
    __shared__ uint32_t s_big[3][CL_BIG_MAX], s_bign[3];  // block 0's are the cluster's
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t CS = cluster.num_blocks();
    const uint32_t r = cluster.block_rank();
    const uint32_t lg = 31 - __clz(CS);  // CS = 1 << lg
    const uint32_t c = blockIdx.x / CS;
    const uint32_t lmd = col0 + c + 1;
    const uint32_t mo_max = (m + CS - 1) / CS;               // the same layout on every block
    const uint32_t mo = r < m ? (m - r + CS - 1) / CS : 0u;  // survivors r, r + CS, ...
    uint32_t* tc = t + (uint64_t)c * m;
    uint32_t* dw = sm;                                       // (mo_max * L + 1) / 2 words
    uint32_t* cw = dw + ((uint64_t)mo_max * L + 1) / 2;      // (mo_max + 1) / 2 words
    uint32_t* pre = cw + (mo_max + 1) / 2;                   // WH_THREADS words
    uint32_t* rs = pre + WH_THREADS;                         // WH_THREADS words
    uint8_t* alive = (uint8_t*)(rs + WH_THREADS);            // mo_max bytes
    uint16_t* list0 = (uint16_t*)(((uintptr_t)(alive + mo_max) + 3) & ~(uintptr_t)3);
    uint16_t* list1 = list0 + mo_max;
    uint16_t* qh[2] = {list1 + mo_max, list1 + 2 * mo_max};  // the two queue halves
    uint16_t* lq[2] = {list1 + 3 * mo_max, list1 + 3 * mo_max + CL_LQ};  // the local halves
    for (uint32_t i = threadIdx.x; i < ((uint64_t)mo_max * L + 1) / 2; i += blockDim.x) dw[i] = 0;
    for (uint32_t i = threadIdx.x; i < (mo_max + 1) / 2; i += blockDim.x) cw[i] = CL_DEAD2;
    if (threadIdx.x < 3) {
        s_cnt[threadIdx.x] = 0;
        s_kept[threadIdx.x] = 0;
        s_bign[threadIdx.x] = 0;
    }
    if (threadIdx.x == 0) s_tail[0] = s_tail[1] = s_lt[0] = s_lt[1] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < mo * L; i += blockDim.x) {
        const uint32_t idx = i / L, l = i - idx * L;
        const uint32_t u = (idx << lg) + r;
        atomicOr(dw + (i >> 1), (deg0[(uint64_t)u * L + l] & 0xFFFFu) << ((i & 1) * 16));
    }
    // alive: 1, or 2 for a node whose row is longer than split (expanded by
    // every block of the cluster, a slice each)
    for (uint32_t i = threadIdx.x; i < mo; i += blockDim.x) {
        const uint32_t u = (i << lg) + r;
        alive[i] = rp[u + 1] - rp[u] > CL_SPLIT ? 2 : 1;
        list0[i] = (uint16_t)i;
    }
    uint32_t* const r0_cnt = cluster.map_shared_rank(s_cnt, 0);
    uint32_t* const r0_kept = cluster.map_shared_rank(s_kept, 0);
    uint32_t* const r0_big = cluster.map_shared_rank(&s_big[0][0], 0);
    uint32_t* const r0_bign = cluster.map_shared_rank(s_bign, 0);
    cluster.sync();  // every block initialised before any reaches another
    uint16_t* cur = list0;
    uint16_t* nxt = list1;
    uint32_t na = mo, k = 0, rho = 0;
    bool failed = false;
    for (;;) {
        if (k > max_level) {  // k is the same on every block
            failed = true;
            break;
        }
        // SCAN round rho: removals queue locally in half (rho + 1) & 1
        const uint32_t qn = (rho + 1) & 1;
        if (threadIdx.x == 0) {
            s_next = 0;
            s_tail[0] = s_tail[1] = 0;  // no block queues remotely during a scan round
            if (r == 0) cl_reset(s_cnt, s_kept, s_bign, rho);
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < na; i += blockDim.x) {
            const uint32_t x = cur[i];
            const uint32_t ax = alive[x];
            if (!ax) continue;
            uint32_t cnt = 0;
            for (uint32_t l = 0; l < L; l++) cnt += wh_get16(dw, x * L + l) >= k + 1;
            if (cnt < lmd) {
                alive[x] = 0;
                tc[(x << lg) + r] = k;
                if (!(ax == 2 && cl_push_big(r0_big, r0_bign, (rho + 1) % 3, (x << lg) + r)))
                    qh[qn][atomicAdd(&s_tail[qn], 1u)] = (uint16_t)x;
                cl_count(r0_cnt + rho % 3);
            } else {
                // CL_DEAD -> cnt, with the long-row flag
                const uint32_t v = cnt | (ax == 2 ? CL_BIG : 0u);
                atomicSub(cw + (x >> 1), (CL_DEAD - v) << ((x & 1) * 16));
                nxt[atomicAdd(&s_next, 1u)] = (uint16_t)x;
                cl_count(r0_kept + rho % 3);
            }
        }
        cluster.sync();  // every block's counts are in block 0, every queue is final
        const uint32_t kept = r0_kept[rho % 3];
        const uint32_t scanned = r0_cnt[rho % 3];
        uint32_t nbig = min(r0_bign[(rho + 1) % 3], CL_BIG_MAX);  // the next round's long rows
        // with no survivor left in the column the rows of this scan's
        // removals name no node that could still change
        uint32_t pushes = kept ? scanned : 0u;
        rho++;
        // DRAIN rounds while the last round queued anything for the cluster
        // (bounded: every node is queued at most once per level)
        for (uint32_t round = 0; pushes && round <= m; round++) {
            const uint32_t qc = rho & 1, qp = (rho + 1) & 1;
            const uint32_t* const bl = r0_big + (rho % 3) * CL_BIG_MAX;
            if (threadIdx.x == 0 && r == 0) cl_reset(s_cnt, s_kept, s_bign, rho);
            // Local iterations: the first expands this block's queued rows and
            // its slice of every long row, each later one the rows that the
            // block's own threads found removed in the one before (of any
            // owner), until they find none.  A row found removed goes to the
            // cluster's list when it is long, else to the local half while it
            // has room, else to its owner's queue; the list and the queues are
            // expanded in the next round (block 0 holds their counts).
            uint32_t lcnt = 0;
            bool ldone = false;
            for (uint32_t li = 0; li <= m; li++) {
                const uint32_t hw = (li + 1) & 1;  // the local half this iteration fills
                const uint32_t qe = li ? lcnt : s_tail[qc];
                const uint32_t items = li ? lcnt : qe + nbig;
                const uint16_t* const lr = lq[li & 1];  // read by iterations >= 1
                for (uint32_t b0 = 0; b0 < items; b0 += WH_THREADS) {
                    if (b0) __syncthreads();  // the last batch's pre and rs are read
                    const uint32_t nb = min(WH_THREADS, items - b0);
                    uint32_t len = 0, start = 0;
                    const uint32_t it = b0 + threadIdx.x;
                    if (it < qe) {
                        const uint32_t lid =
                            li ? (uint32_t)lr[it] : ((uint32_t)qh[qc][it] << lg) + r;
                        start = rp[lid];
                        len = rp[lid + 1] - start;
                        tc[lid] = k;  // again for a scan removal: the same value
                    } else if (it < items) {
                        const uint32_t u = bl[it - qe];
                        const uint32_t s0 = rp[u], l0 = rp[u + 1] - s0;
                        const uint32_t e0 = (uint32_t)((uint64_t)l0 * r / CS);
                        start = s0 + e0;
                        len = (uint32_t)((uint64_t)l0 * (r + 1) / CS) - e0;
                        if ((u & (CS - 1)) == r) tc[u] = k;  // its owner
                    }
                    uint32_t ex;
                    const uint32_t total = cl_block_scan(len, &ex, s_warp);
                    // every thread has read the half's length (before the
                    // scan's barrier): it takes a later iteration's (round's)
                    if (b0 == 0 && threadIdx.x == 0) {
                        if (li) s_lt[li & 1] = 0;
                        else s_tail[qc] = 0;
                    }
                    pre[threadIdx.x] = ex;
                    rs[threadIdx.x] = start;
                    __syncthreads();
                    uint32_t lo0 = 0;
                    for (uint32_t e0 = threadIdx.x; e0 < total; e0 += 4 * blockDim.x) {
                        uint32_t slot[4];
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const uint32_t e = e0 + q * blockDim.x;
                            slot[q] = NO_BIG_ROW;
                            if (e < total) {
                                uint32_t lo = lo0, hi = nb - 1;
                                while (lo < hi) {
                                    const uint32_t mid = (lo + hi + 1) >> 1;
                                    if (pre[mid] <= e) lo = mid;
                                    else hi = mid - 1;
                                }
                                lo0 = lo;
                                slot[q] = adj[rs[lo] + (e - pre[lo])];
                            }
                        }
                        // the degree decrements first, independent of one
                        // another; removed neighbours are decremented too (a
                        // half counts the alive neighbours, so it never drops
                        // below 0), and their count halves, CL_DEAD less at
                        // most L crossings, never equal lmd
                        uint32_t ow[4], ui[4], old[4];
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            old[q] = 0;  // never k + 1
                            ow[q] = ui[q] = 0;
                            if (slot[q] == NO_BIG_ROW) continue;
                            const uint32_t u = divL.div(slot[q]);
                            if (u >= m) continue;
                            const uint32_t l = slot[q] - u * L;
                            ow[q] = u & (CS - 1);
                            ui[q] = u >> lg;
                            old[q] = cl_dec16(cluster.map_shared_rank(dw, ow[q]), ui[q] * L + l);
                        }
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            if (old[q] != k + 1) continue;
                            const uint32_t oc = cl_dec16(cluster.map_shared_rank(cw, ow[q]), ui[q]);
                            if ((oc & CL_CNT) != lmd) continue;
                            // removed: its row is expanded by this block, by
                            // its owner or, when long, by every block (the
                            // table entry is written then)
                            cluster.map_shared_rank(alive, ow[q])[ui[q]] = 0;
                            const uint32_t u2 = (ui[q] << lg) | ow[q];
                            // (the list's own count tells the cluster)
                            if ((oc & CL_BIG) && cl_push_big(r0_big, r0_bign, (rho + 1) % 3, u2))
                                continue;
                            const uint32_t pos = atomicAdd(&s_lt[hw], 1u);
                            if (pos < CL_LQ) {
                                lq[hw][pos] = (uint16_t)u2;
                            } else {
                                uint32_t* const t_ow = cluster.map_shared_rank(s_tail, ow[q]);
                                const uint32_t p2 = atomicAdd(t_ow + qp, 1u);
                                cluster.map_shared_rank(qh[qp], ow[q])[p2] = (uint16_t)ui[q];
                                cl_count(r0_cnt + rho % 3);
                            }
                        }
                    }
                }
                __syncthreads();  // this iteration's local pushes are in place
                lcnt = min(s_lt[hw], CL_LQ);
                if (lcnt == 0) {
                    ldone = true;
                    break;
                }
            }
            // (cannot happen: every node is found removed at most once a level)
            if (!ldone && threadIdx.x == 0) atomicOr(r0_cnt + rho % 3, CL_FAIL);
            cluster.sync();  // every push is counted in block 0 and queued
            const uint32_t cnt = r0_cnt[rho % 3];
            nbig = min(r0_bign[(rho + 1) % 3], CL_BIG_MAX);
            pushes = (cnt & ~CL_FAIL) + nbig;
            if (cnt & CL_FAIL) {  // the same on every block
                pushes = 1;
                break;
            }
            rho++;
        }
        if (pushes) {  // the round bound ended the level with rows unexpanded
            failed = true;  // (the cluster-wide count: every block breaks)
            break;
        }
        // counts are rebuilt by the next scan: every half back to CL_DEAD
        for (uint32_t i = threadIdx.x; i < (mo_max + 1) / 2; i += blockDim.x) cw[i] = CL_DEAD2;
        na = s_next;
        uint16_t* tmp = cur;
        cur = nxt;
        nxt = tmp;
        k++;
        __syncthreads();
        if (kept == 0) break;  // the cluster-wide count: the same on every block
    }
    if (failed && r == 0 && threadIdx.x == 0) atomicExch(err, 2u);
    if (r == 0 && threadIdx.x == 0) levels[c] = k;
    cluster.sync();  // no block leaves while another may still reach its shared memory
}


// ---- host ---------------------------------------------------------------------

static uint32_t env_u32(const char* name, uint32_t dflt) {
    const char* s = getenv(name);
    return s && *s ? (uint32_t)strtoul(s, nullptr, 10) : dflt;
}

static cudaLaunchConfig_t cluster_config(uint32_t ncols, uint32_t cs, size_t smem,
                                         cudaLaunchAttribute* at) {
    cudaLaunchConfig_t cfg = {};
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = cs;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    cfg.gridDim = dim3(ncols * cs);
    cfg.blockDim = dim3(WH_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// Clusters of cs blocks with the largest shared memory that the device runs
// at once (0: it cannot place one).  Asked once per device.
static uint32_t clusters_at_once(uint32_t cs) {
    static std::mutex mu;
    static int cached[64][5];  // by log2(cs), plus one
    int dev = 0, lg = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    while ((1u << lg) < cs) lg++;
    std::lock_guard<std::mutex> lk(mu);
    if (cached[dev][lg]) return (uint32_t)cached[dev][lg] - 1;
    int n = 0;
    if (cudaFuncSetAttribute(k_whole_cl, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)WH_SMEM) == cudaSuccess &&
        cudaFuncSetAttribute(k_whole_cl, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
            cudaSuccess) {
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t cfg = cluster_config(1, cs, WH_SMEM, &at);
        if (cudaOccupancyMaxActiveClusters(&n, k_whole_cl, &cfg) != cudaSuccess) n = 0;
    }
    cudaGetLastError();
    cached[dev][lg] = n + 1;
    return (uint32_t)n;
}

// Blocks per column for a graph of n nodes: 1 when it fits a block, 16, 8 or 4
// when it fits such a cluster, 0 when it fits neither.  More blocks finish a
// column sooner, but fewer columns then run at once: 45,003 nodes, 13 columns
// take 2.09 ms on clusters of 16 (two waves), 1.57 on clusters of 8 (one wave)
// and 2.9 on the whole device, a level after another for all columns; with 24
// columns 16 blocks need three waves, 3.34 ms, and the whole device 2.76.
// 60,000 nodes x 20: 17.2 ms against 13.4.  Hence at most two waves, and the
// costs, which are one wave's times.
static uint32_t whole_blocks(uint32_t n, uint32_t L, uint32_t ncols) {
    if (!n || !env_u32("FC_PEEL_ENDGAME", 1) || !env_u32("FC_PEEL_WHOLE", 1)) return 0;
    if (n <= wh_capacity(L)) return 1;
    if (n > 65536) return 0;
    const uint32_t force = env_u32("FC_PEEL_CLUSTER", 0);
    uint32_t best = 0, best_cost = 0;
    const uint32_t sizes[3] = {16, 8, 4}, cost[3] = {100, 115, 150};
    for (int i = 0; i < 3; i++) {
        const uint32_t cs = sizes[i];
        if (force && cs != force) continue;
        if (n > cs * cl_block_capacity(L)) continue;
        const uint32_t at_once = clusters_at_once(cs);
        if (!at_once) continue;
        const uint32_t waves = (ncols + at_once - 1) / at_once;
        if (waves > 2 && !force) continue;
        const uint32_t c = waves * cost[i];
        if (!best || c < best_cost) {
            best = cs;
            best_cost = c;
        }
    }
    return best;
}

// The scratch of the whole-graph path: an error flag and each column's levels.
uint64_t whole_ws_bytes(uint32_t ncols) { return 4ull * ncols + 512; }

bool fits_whole(const PeelGraph& g, uint32_t ncols) { return whole_blocks(g.n, g.L, ncols) != 0; }

fc_status whole_run(const PeelGraph& g, uint32_t col0, uint32_t ncols, uint32_t* table,
                           void* ws, cudaStream_t s, PeelStats* st) {
    const uint32_t n = g.n, L = g.L;
    const uint32_t cs = whole_blocks(n, L, ncols);
    const uint64_t smem =
        cs > 1 ? cl_smem_bytes((n + cs - 1) / cs, L)
               : 4ull * (((uint64_t)n * L + 1) / 2 + (n + 1) / 2 + 2ull * WH_THREADS) + n + 4 +
                     6ull * n + 16;
    static const cudaError_t attr_rc = cudaFuncSetAttribute(
        k_whole, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WH_SMEM);
    if (!cs || attr_rc != cudaSuccess || smem > WH_SMEM) return FC_ERR_DEVICE;
    struct Events {  // destroyed on every return
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        ~Events() {
            if (e0) cudaEventDestroy(e0);
            if (e1) cudaEventDestroy(e1);
        }
    } ev;
    FC_CUDA_TRY(cudaEventCreate(&ev.e0));
    FC_CUDA_TRY(cudaEventCreate(&ev.e1));
    count_alloc(2);
    FC_CUDA_TRY(cudaEventRecord(ev.e0, s));
    uint32_t* const out = (uint32_t*)ws;  // the error flag, then each column's levels
    FC_CUDA_TRY(cudaMemsetAsync(out, 0, 4ull * (ncols + 1), s));
    FastDiv divL;
    divL.init(L);
    uint32_t* const tc = table + (uint64_t)col0 * n;
    if (cs > 1) {
        cudaLaunchAttribute at;
        cudaLaunchConfig_t cfg = cluster_config(ncols, cs, (size_t)smem, &at);
        cfg.stream = s;
        FC_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_whole_cl, g.node_ptr, g.adj, g.deg0, n, L, divL, tc,
                                       col0, g.max_level, out + 1, out));
    } else {
        k_whole<<<ncols, WH_THREADS, (size_t)smem, s>>>(g.node_ptr, g.adj, g.deg0, n, L, divL, tc,
                                                        col0, g.max_level, out + 1, out);
    }
    FC_CUDA_TRY(cudaGetLastError());
    count_launch();
    FC_CUDA_TRY(cudaEventRecord(ev.e1, s));
    std::vector<uint32_t> lv(ncols + 1);
    FC_TRY(to_host(lv.data(), out, 4ull * (ncols + 1), s));
    float ms = 0;
    cudaEventElapsedTime(&ms, ev.e0, ev.e1);
    if (st) st->ms += ms;
    if (lv[0]) return lv[0] == 2 ? FC_ERR_ITER_LIMIT : FC_ERR_DEVICE;
    if (st) {
        uint32_t m = 0;
        for (uint32_t c = 0; c < ncols; c++) m = lv[c + 1] > m ? lv[c + 1] : m;
        st->levels += m;
    }
    return FC_OK;
}

void whole_preload() {
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, k_whole);
    cudaFuncGetAttributes(&a, k_whole_cl);
    cudaGetLastError();
}

}  // namespace fc
