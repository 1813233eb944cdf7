// Densest-subgraph search over every non-empty fcgrid cell, from the core
// table, in one pass over the edges per group of lambda columns.
//
// A directed entry (v -> u, layer l) lies inside C_{k,lambda} iff
// min(core_lambda(v), core_lambda(u)) >= k.  So one histogram per lambda,
//     H[lambda][l][key] = #{entries (v,u,l) : min(core_lambda(v), core_lambda(u)) = key},
// gives by suffix sums over key every cell's
//     e2_l(k,lambda) = sum over v in C_{k,lambda} of deg_C(v,l)
// -- the `num_edge` the reference accumulates per cell (Core/FCPathLevelLeft.cpp:
// 60-64) -- and the node histogram gives |C_{k,lambda}|.  Each cell is then
// scored with the reference's expression (:66-90):
//     degree_l = (float)e2_l * 1.0f / 2;  sorted descending;
//     d_l = degree_(l) * 1.0f / |C| * 1.0 * pow(l, beta)   (FP64)
// keeping the best l (ties to the larger l), and the cells are folded in the
// reference's tree preorder (lambda-major, k ascending) with its float running
// maximum (Core/FCTree.cpp:69-82, main.cpp:406).  pow(l, beta) comes from the
// host's libm, as in the reference; every other step is IEEE FP32/FP64
// arithmetic in the same order, so densities are bit-identical.
#include <thrust/iterator/counting_iterator.h>

#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "device.h"

namespace fc {

struct DensState {
    uint32_t L = 0;
    std::vector<uint32_t> kmax;        // per lambda (index lambda-1)
    std::vector<uint64_t> hbase;       // per lambda: offset of H[lambda] (L*(kmax+1) words)
    std::vector<uint64_t> nbase;       // per lambda: offset of the node histogram
    std::vector<uint64_t> cbase;       // per lambda: first cell index
    uint64_t hwords = 0, nwords = 0, ncells = 0;
    uint32_t* H = nullptr;             // hwords: edge histogram -> suffix sums e2
    uint32_t* N = nullptr;             // nwords: node histogram -> suffix sums |C|
    uint4* rows = nullptr;             // the table as rows of 16-bit cores (k_core_rows)
    uint64_t* d_hbase = nullptr;       // device copies of the bases (L each)
    uint64_t* d_nbase = nullptr;
    uint32_t* d_kmax = nullptr;
    fc_cell* cells = nullptr;          // ncells
    double* powl = nullptr;            // L
    fc_densest_result* d_res = nullptr;
    uint32_t* cell_lk = nullptr;       // 2 * ncells: lambda index, then k, per cell
    std::vector<uint32_t> cell_host;
    uint64_t H_cap = 0, N_cap = 0, cells_cap = 0, cell_lk_cap = 0, hbase_cap = 0, nbase_cap = 0;
    bool hist_valid = false;
    uint32_t lo = 0, hi = 0;           // the lambda columns (0-based) the histograms cover
};

template <class T>
static fc_status grow(T*& p, uint64_t& cap, uint64_t need, cudaStream_t st) {
    if (p && cap >= need) return FC_OK;
    dev_free(p, st);
    p = nullptr;
    cap = 0;
    uint64_t c = need + need / 4 + 16;
    FC_TRY(dev_alloc((void**)&p, c * sizeof(T), st));
    cap = c;
    return FC_OK;
}

void free_densest_state(DeviceGraph* d, cudaStream_t st) {
    DensState* s = (DensState*)d->dens;
    if (!s) return;
    // called with the graph's work finished (release_device waits for it, or
    // its caller knows that it has completed)
    for (void* p : {(void*)s->H, (void*)s->N, (void*)s->rows, (void*)s->d_hbase,
                    (void*)s->d_nbase, (void*)s->d_kmax, (void*)s->cells, (void*)s->powl,
                    (void*)s->d_res, (void*)s->cell_lk})
        dev_free(p, st);
    delete s;
    d->dens = nullptr;
}

// ---- kernels -------------------------------------------------------------

__global__ void k_colmax(const uint32_t* __restrict__ table, uint32_t n, uint32_t L,
                         uint32_t* __restrict__ kmax) {
    // grid.y = lambda
    const uint32_t lam = blockIdx.y;
    const uint32_t* col = table + (uint64_t)lam * n;
    uint32_t m = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        m = max(m, col[v]);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(kmax + lam, m);
}

uint64_t core_rows_bytes(uint64_t n, uint64_t L) { return n * (L > 4 ? (L + 7) / 8 * 16 : 8); }

// A word of a core row: eight columns, or four where there are no more (2.5M
// nodes x 4 layers: 0.2 ms less than with eight).
template <bool WIDE>
struct CoreWord {
    static __device__ __forceinline__ uint4 load(const uint4* rows, uint64_t i) { return rows[i]; }
    static __device__ __forceinline__ void store(uint4* rows, uint64_t i, uint4 w) { rows[i] = w; }
};
template <>
struct CoreWord<false> {
    static __device__ __forceinline__ uint4 load(const uint4* rows, uint64_t i) {
        const uint2 w = ((const uint2*)rows)[i];
        return make_uint4(w.x, w.y, 0, 0);
    }
    static __device__ __forceinline__ void store(uint4* rows, uint64_t i, uint4 w) {
        ((uint2*)rows)[i] = make_uint2(w.x, w.y);
    }
};

// The table as rows of 16-bit cores, a node's columns side by side, padded to
// octets of eight (one word).  16 bits hold every core: rows have no
// repeated entries, so a core of k takes k+1 nodes with k entries each, and a
// graph has fewer than 2^32 entries.  Columns outside [lo, hi) are not read.
template <bool WIDE>
__global__ void k_core_rows(const uint32_t* __restrict__ table, uint32_t n, uint32_t lo, uint32_t hi,
                            uint32_t octets, uint4* __restrict__ rows) {
    const uint32_t o = blockIdx.y;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        uint32_t c[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; i++) {
            const uint32_t lam = o * 8 + i;
            c[i] = lam >= lo && lam < hi ? table[(uint64_t)lam * n + v] : 0u;
        }
        CoreWord<WIDE>::store(rows, (uint64_t)v * octets + o,
                              make_uint4(c[0] | c[1] << 16, c[2] | c[3] << 16,
                                         c[4] | c[5] << 16, c[6] | c[7] << 16));
    }
}

__global__ void k_node_hist(const uint32_t* __restrict__ table, uint32_t n,
                            const uint64_t* __restrict__ nbase, const uint32_t* __restrict__ kmax,
                            uint32_t* __restrict__ N) {
    extern __shared__ uint32_t sh[];
    const uint32_t lam = blockIdx.y;
    const uint32_t bins = kmax[lam] + 1;
    const bool use_sh = bins <= 12288;
    if (use_sh)
        for (uint32_t i = threadIdx.x; i < bins; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    const uint32_t* col = table + (uint64_t)lam * n;
    uint32_t* out = N + nbase[lam];
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        uint32_t c = col[v];
        if (use_sh) atomicAdd(sh + c, 1u);
        else atomicAdd(out + c, 1u);
    }
    __syncthreads();
    if (use_sh)
        for (uint32_t i = threadIdx.x; i < bins; i += blockDim.x)
            if (sh[i]) atomicAdd(out + i, sh[i]);
}

// The edge histogram of groups of lambda columns.
//
// An edge {v, u} of layer l counts 2 in bin (l, min(core(v), core(u))) of each
// column.  It is counted where the minimum is: entry (v, u, l) adds 2 to bin
// (l, core(v)) when core(u) > core(v), 1 when they are equal (the entry
// (u, v, l) adds the other 1) and 0 otherwise.  A run of entries of one (v, l)
// then goes to one bin per column, so its counts are added up in registers and
// each bin gets one atomic a run -- with a bin that depends on u every entry
// needs its own, and the lanes of a warp, on one row, collide on the bin of
// core(v).
//
// A warp takes a contiguous slice of the entries, 32 at a time, one a lane.
// Eight columns are compared at once, as 16-bit halves; their counts are
// bytes (32 entries add 64 at most), summed over a run's lanes by shuffles,
// and the run's first lane adds them to the bins.  The bins of a group lie in
// shared memory: as 32-bit words (mode 1), or as 16-bit halves when no block
// can count 65,536 (mode 2); a single column whose bins do not fit has them in
// global memory (mode 0).  All groups are one launch (blockIdx.y): a graph
// whose entries do not fill the device once still fills it with groups.
//
// Bound by instruction issue (about 60 a warp and octet) and the gather of
// the neighbours' rows.  Against an atomic per entry and column, groups one
// after another: a pass over 220 nodes x 360 layers 2.93 -> 1.93 ms, 180,001 x
// 17 (73M entries) 21.2 -> 19.5 ms, 2.6M x 24 (96M entries) 34.7 -> 32.8 ms.
constexpr uint32_t EH_THREADS = 1024;
constexpr uint32_t EH_BINS = 55 * 1024;    // 32-bit words of shared memory for bins
constexpr uint32_t EH_MAX_COLS = 64;       // columns of a group
constexpr uint32_t EH_MAX_GROUPS = 64;     // groups of a launch
struct EdgeGroup {
    uint32_t lam0, nl, bins, mode;
};
struct EdgeGroups {
    EdgeGroup g[EH_MAX_GROUPS];
};

// what entries with cores u add against v, per 16-bit half: 2 above, 1 equal,
// 0 below (v1: v - 1; halves with v = 0 are not used)
__device__ __forceinline__ uint32_t eh_count2(uint32_t u, uint32_t v1) {
    return __vminu2(__vmaxu2(u, v1) - v1, 0x00020002u);
}
__device__ __forceinline__ uint32_t eh_less1(uint32_t v) {
    return __vmaxu2(v, 0x00010001u) - 0x00010001u;
}

template <bool WIDE>
__global__ void __launch_bounds__(EH_THREADS)
k_edge_hist(const uint32_t* __restrict__ node_ptr, const uint32_t* __restrict__ adj, uint32_t n,
            uint32_t L, uint64_t entries, FastDiv divL, const uint4* __restrict__ rows,
            uint32_t octets, const __grid_constant__ EdgeGroups groups,
            const uint64_t* __restrict__ hbase, const uint32_t* __restrict__ kmax,
            uint32_t* __restrict__ H) {
    extern __shared__ uint32_t sh[];
    __shared__ uint32_t soff[EH_MAX_COLS];  // per column of the group: offset of its bins
    __shared__ uint32_t skm1[EH_MAX_COLS];  // kmax + 1
    __shared__ uint64_t shb[EH_MAX_COLS];   // the column's base in H
    const EdgeGroup gr = groups.g[blockIdx.y];
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t mode = gr.mode;
    if (threadIdx.x < gr.nl) {
        skm1[threadIdx.x] = kmax[gr.lam0 + threadIdx.x] + 1;
        shb[threadIdx.x] = hbase[gr.lam0 + threadIdx.x];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t o = 0;
        for (uint32_t i = 0; i < gr.nl; i++) {
            soff[i] = o;
            o += L * skm1[i];
        }
    }
    if (mode) {
        const uint32_t words = mode == 2 ? (gr.bins + 1) / 2 : gr.bins;
        for (uint32_t i = threadIdx.x; i < words; i += EH_THREADS) sh[i] = 0;
    }
    __syncthreads();
    const uint64_t nwarps = (uint64_t)gridDim.x * (EH_THREADS / 32);
    const uint64_t gw = (uint64_t)blockIdx.x * (EH_THREADS / 32) + (threadIdx.x >> 5);
    const uint64_t per = ((entries + nwarps - 1) / nwarps + 31) & ~31ull;
    const uint64_t e0 = min(entries, gw * per), e1 = min(entries, e0 + per);
    const uint32_t o0 = gr.lam0 / 8, o1 = (gr.lam0 + gr.nl + 7) / 8;
    if (e0 < e1) {  // warp-uniform
        uint32_t r0 = 0, hi = n;  // the row of the slice's first entry
        while (hi - r0 > 1) {
            const uint32_t mid = (r0 + hi) >> 1;
            if (node_ptr[mid] <= e0) r0 = mid;
            else hi = mid;
        }
        uint32_t slot = e0 + lane < e1 ? adj[e0 + lane] : 0u;
        for (uint64_t b0 = e0; b0 < e1; b0 += 32) {
            const bool on = b0 + lane < e1;
            const uint32_t e = on ? (uint32_t)b0 + lane : (uint32_t)e1 - 1;
            const uint32_t u = divL.div(slot), l = slot - u * L;
            slot = b0 + 32 + lane < e1 ? adj[b0 + 32 + lane] : 0u;
            // the entry's row: r0 and the row starts up to e (empty rows may
            // make them more than a warp's worth)
            uint32_t v = r0;
            for (uint32_t base = r0;; base += 32) {
                const uint32_t start = node_ptr[min(base + 1 + lane, n)];
                uint32_t c = 0;
#pragma unroll
                for (uint32_t s = 16; s; s >>= 1)
                    if (__shfl_sync(0xffffffffu, start, c + s - 1) <= e) c += s;
                if (__shfl_sync(0xffffffffu, start, c) <= e) c++;
                if (v == base) v += c;
                if (!__any_sync(0xffffffffu, v == base + 32)) break;
            }
            r0 = __shfl_sync(0xffffffffu, v, 31);
            // runs of one (row, layer); `end`: the lane after the run's last
            const uint32_t pv = __shfl_up_sync(0xffffffffu, v, 1);
            const uint32_t pl = __shfl_up_sync(0xffffffffu, l, 1);
            const bool head = lane == 0 || pv != v || pl != l;
            const uint32_t heads = __ballot_sync(0xffffffffu, head);
            const uint32_t after = heads & (0xfffffffeu << lane);
            const uint32_t end = after ? __ffs(after) - 1 : 32u;
            const uint32_t longest = __reduce_max_sync(0xffffffffu, head ? end - lane : 0u);
            for (uint32_t o = o0; o < o1; o++) {
                const uint4 a = CoreWord<WIDE>::load(rows, (uint64_t)v * octets + o);
                const bool some = (a.x | a.y | a.z | a.w) != 0u;
                if (!__any_sync(0xffffffffu, some)) continue;
                uint32_t s0 = 0, s1 = 0;  // counts of columns 0-3 and 4-7, a byte each
                if (on && some) {
                    const uint4 b = CoreWord<WIDE>::load(rows, (uint64_t)u * octets + o);
                    s0 = __byte_perm(eh_count2(b.x, eh_less1(a.x)), eh_count2(b.y, eh_less1(a.y)),
                                     0x6420);
                    s1 = __byte_perm(eh_count2(b.z, eh_less1(a.z)), eh_count2(b.w, eh_less1(a.w)),
                                     0x6420);
                }
                for (uint32_t d = 1; d < longest; d <<= 1) {
                    const uint32_t y0 = __shfl_down_sync(0xffffffffu, s0, d);
                    const uint32_t y1 = __shfl_down_sync(0xffffffffu, s1, d);
                    if (lane + d < end) {
                        s0 += y0;
                        s1 += y1;
                    }
                }
                if (head && some) {
                    const uint32_t key2[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                    for (uint32_t c = 0; c < 8; c++) {
                        const uint32_t cnt = ((c < 4 ? s0 : s1) >> (8 * (c & 3))) & 0xFFu;
                        const uint32_t key = (key2[c >> 1] >> (16 * (c & 1))) & 0xFFFFu;
                        const uint32_t i = o * 8 + c - gr.lam0;  // wraps below the group
                        if (cnt && key && i < gr.nl) {
                            const uint32_t at = soff[i] + l * skm1[i] + key;
                            if (mode == 1) atomicAdd(sh + at, cnt);
                            else if (mode == 2) atomicAdd(sh + (at >> 1), cnt << ((at & 1) * 16));
                            else atomicAdd(H + shb[i] + (uint64_t)l * skm1[i] + key, cnt);
                        }
                    }
                }
            }
        }
    }
    __syncthreads();
    if (!mode) return;
    for (uint32_t i = 0; i < gr.nl; i++) {
        const uint32_t bins = L * skm1[i];
        uint32_t* g = H + shb[i];
        for (uint32_t w = threadIdx.x; w < bins; w += EH_THREADS) {
            const uint32_t b = soff[i] + w;
            const uint32_t x = mode == 1 ? sh[b] : (sh[b >> 1] >> ((b & 1) * 16)) & 0xFFFFu;
            if (x) atomicAdd(g + w, x);
        }
    }
}

// Suffix sums over key, per (lambda, layer) row of H and per lambda of N, a
// warp per row: 32 keys at a time from the top, summed by shuffles (a thread
// per row pays a memory round trip per key).
// uint32 arithmetic wraps exactly as the reference's `uint num_edge`.
__global__ void k_suffix(uint32_t L, uint32_t lo, uint32_t hi, const uint64_t* __restrict__ hbase,
                         const uint64_t* __restrict__ nbase, const uint32_t* __restrict__ kmax,
                         uint32_t* __restrict__ H, uint32_t* __restrict__ N) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nrows = (uint64_t)(hi - lo) * (L + 1);
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrows; r += nwarps) {
        const uint32_t lam = lo + (uint32_t)(r / (L + 1)), l = (uint32_t)(r % (L + 1));
        const uint32_t km1 = kmax[lam] + 1;
        uint32_t* row = l < L ? H + hbase[lam] + (uint64_t)l * km1 : N + nbase[lam];
        uint32_t acc = 0;
        for (uint32_t done = 0; done < km1; done += 32) {
            const bool on = done + lane < km1;
            const uint32_t k = on ? km1 - 1 - done - lane : 0u;
            uint32_t x = on ? row[k] : 0u;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            x += acc;
            if (on) row[k] = x;
            acc = __shfl_sync(0xffffffffu, x, 31);
        }
    }
}

// One block per cell (lambda, k), k >= 1: sort the cell's L layer counts
// descending (bitonic sort in shared memory), evaluate every l, keep the best.
__global__ void k_cells(uint32_t L, uint32_t P /* pow2 >= L */, const uint64_t* __restrict__ hbase,
                        const uint64_t* __restrict__ nbase, const uint32_t* __restrict__ kmax,
                        const uint32_t* __restrict__ H, const uint32_t* __restrict__ N,
                        const double* __restrict__ powl, const uint32_t* __restrict__ cell_lam,
                        const uint32_t* __restrict__ cell_k, fc_cell* __restrict__ cells) {
    extern __shared__ uint32_t sv[];  // P values
    __shared__ double bestd[32];
    __shared__ uint32_t bestl[32];
    const uint32_t ci = blockIdx.x;
    const uint32_t lam = cell_lam[ci], k = cell_k[ci];
    const uint32_t km1 = kmax[lam] + 1;
    const uint32_t len = N[nbase[lam] + k];
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x)
        sv[i] = i < L ? H[hbase[lam] + (uint64_t)i * km1 + k] : 0u;
    __syncthreads();
    // bitonic sort, descending
    for (uint32_t size = 2; size <= P; size <<= 1) {
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
                uint32_t p = i ^ stride;
                if (p > i) {
                    bool desc = (i & size) == 0;
                    uint32_t a = sv[i], b = sv[p];
                    if (desc ? (a < b) : (a > b)) {
                        sv[i] = b;
                        sv[p] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
    double my_d = -1.0;
    uint32_t my_l = 0;
    for (uint32_t i = threadIdx.x; i < L; i += blockDim.x) {
        float f = __uint2float_rn(sv[i]) * 1.0f / 2;
        double degree = (double)f;
        double mad = (degree * 1.0f) / (double)len * 1.0;
        double d = mad * powl[i];
        if (d >= my_d) {  // later i in this thread's sequence wins ties
            my_d = d;
            my_l = i + 1;
        }
    }
    // block argmax, ties to the larger l
    for (int o = 16; o >= 1; o >>= 1) {
        double od = __shfl_down_sync(0xffffffffu, my_d, o);
        uint32_t ol = __shfl_down_sync(0xffffffffu, my_l, o);
        if (od > my_d || (od == my_d && ol > my_l)) {
            my_d = od;
            my_l = ol;
        }
    }
    const uint32_t w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        bestd[w] = my_d;
        bestl[w] = my_l;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double bd = -1.0;
        uint32_t bl = 0;
        for (uint32_t i = 0; i < (blockDim.x + 31) / 32; i++)
            if (bestd[i] > bd || (bestd[i] == bd && bestl[i] > bl)) {
                bd = bestd[i];
                bl = bestl[i];
            }
        // the reference starts from 0.0 and keeps l on `d >= best`
        fc_cell c;
        c.k = k;
        c.lmd = lam + 1;
        c.length = len;
        c.lstar = bl;
        c.density = bd < 0.0 ? 0.0 : bd;
        cells[ci] = c;
    }
}

// The reference's preorder fold with a float running maximum: cell i wins, and
// the maximum becomes (float)d_i, when d_i >= the maximum so far.
//
// The maximum after cell i is the largest (float)d_j, j <= i: rounding is
// monotone and keeps floats, so a cell that wins raises it to its own float (or
// leaves it), and one that does not is below it, its float too.  With F the
// largest of all and p the first cell of float F, p wins (its float is above
// the maximum before it), and after p exactly the cells with d_i >= F do; no
// cell before p has d_i >= F.  So the last winner is the last cell with
// d_i >= F, or p when there is none.  With no cell above 0, F is the initial 0
// and the same holds.  One block: F, then both candidates.
__global__ void k_fold(const fc_cell* __restrict__ cells, uint64_t ncells, double beta,
                       fc_densest_result* out) {
    __shared__ uint32_t s_max;  // floats >= 0 order like their bits
    __shared__ unsigned long long s_first, s_last;  // p; the last cell with d >= F, plus 1
    if (threadIdx.x == 0) {
        s_max = 0;
        s_first = ~0ull;
        s_last = 0;
    }
    __syncthreads();
    uint32_t m = 0;
    for (uint64_t i = threadIdx.x; i < ncells; i += blockDim.x)
        m = max(m, __float_as_uint((float)cells[i].density));
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_max, m);
    __syncthreads();
    const float F = __uint_as_float(s_max);
    unsigned long long first = ~0ull, last = 0;
    for (uint64_t i = threadIdx.x; i < ncells; i += blockDim.x) {
        const double d = cells[i].density;
        if (first == ~0ull && (float)d == F) first = i;
        if (d >= (double)F) last = i + 1;
    }
    if (first != ~0ull) atomicMin(&s_first, first);
    if (last) atomicMax(&s_last, last);
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint64_t win = s_last ? s_last - 1 : s_first;
        fc_densest_result r;
        r.beta = beta;
        r.density = 0.0;
        r.k = r.lmd = r.length = r.lstar = 0;
        if (win != ~0ull) {
            const fc_cell c = cells[win];
            r.density = c.density;
            r.k = c.k;
            r.lmd = c.lmd;
            r.length = c.length;
            r.lstar = c.lstar;
        }
        r.max_density_f = F;
        r.n_cells = (uint32_t)ncells;
        *out = r;
    }
}

// ---- host --------------------------------------------------------------------

static int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// Histograms for the resident table (beta-independent), over the lambda
// columns [lo, hi): the other columns count as empty (kmax 0, no cells), and
// no kernel reads them, since they may not have been computed.
static fc_status build_hist(DeviceGraph* d, cudaStream_t st, uint32_t lo, uint32_t hi,
                            const std::function<fc_status()>* after_maxima = nullptr) {
    DensState* s = (DensState*)d->dens;
    if (s && s->hist_valid && s->lo == lo && s->hi == hi) return FC_OK;
    if (!s) {
        s = new DensState();
        d->dens = s;
    }
    const uint32_t n = d->n, L = d->L;
    s->L = L;
    // per-lambda maxima
    if (!s->d_kmax) FC_TRY(dev_alloc((void**)&s->d_kmax, (L + 1) * 4, st));
    FC_CUDA_TRY(cudaMemsetAsync(s->d_kmax, 0, (L + 1) * 4, st));
    // blocks per column: enough to fill the SMs, at least 2048 nodes each
    const uint32_t per_col = std::max<uint32_t>(
        1u, std::min<uint32_t>((n + 2047) / 2048,
                               8u * (uint32_t)sm_count() / std::max<uint32_t>(1u, hi - lo)));
    dim3 g(per_col, hi - lo);
    k_colmax<<<g, 256, 0, st>>>(d->table + (uint64_t)lo * n, n, L, s->d_kmax + lo);
    count_launch();
    FC_CUDA_TRY(cudaGetLastError());
    s->kmax.assign(L, 0);
    FC_TRY(to_host(s->kmax.data(), s->d_kmax, L * 4, st));
    if (after_maxima) FC_TRY((*after_maxima)());
    d->kmax = s->kmax;
    for (uint32_t l = 0; l < L; l++)
        if (s->kmax[l] > d->max_deg || s->kmax[l] > 0xFFFFu)
            return FC_ERR_DEVICE;  // not a valid core table
    s->hbase.assign(L, 0);
    s->nbase.assign(L, 0);
    s->cbase.assign(L, 0);
    uint64_t hw = 0, nw = 0, nc = 0;
    for (uint32_t l = 0; l < L; l++) {
        s->hbase[l] = hw;
        s->nbase[l] = nw;
        s->cbase[l] = nc;
        hw += (uint64_t)L * (s->kmax[l] + 1);
        nw += s->kmax[l] + 1;
        nc += s->kmax[l];
    }
    // grow-only buffers: a recomputation of the same graph allocates nothing
    s->hwords = hw;
    s->nwords = nw;
    s->ncells = nc;
    FC_TRY(grow(s->H, s->H_cap, hw + 1, st));
    FC_TRY(grow(s->N, s->N_cap, nw + 1, st));
    FC_TRY(grow(s->cells, s->cells_cap, nc + 1, st));
    FC_TRY(grow(s->cell_lk, s->cell_lk_cap, 2 * nc + 2, st));
    FC_TRY(grow(s->d_hbase, s->hbase_cap, L + 1, st));
    FC_TRY(grow(s->d_nbase, s->nbase_cap, L + 1, st));
    const uint32_t octets = (L + 7) / 8;
    if (!s->rows) FC_TRY(dev_alloc((void**)&s->rows, core_rows_bytes(n, L) + 16, st));
    FC_TRY(to_device(s->d_hbase, s->hbase.data(), L * 8, st));
    FC_TRY(to_device(s->d_nbase, s->nbase.data(), L * 8, st));
    // cell list (lambda index, k) in the reference's order, for k_cells
    s->cell_host.resize(2 * nc + 2);
    {
        uint64_t i = 0;
        for (uint32_t l = 0; l < L; l++)
            for (uint32_t k = 1; k <= s->kmax[l]; k++, i++) {
                s->cell_host[i] = l;
                s->cell_host[nc + i] = k;
            }
    }
    if (nc)
        FC_TRY(to_device(s->cell_lk, s->cell_host.data(), 2 * nc * 4, st));
    FC_CUDA_TRY(cudaMemsetAsync(s->H, 0, hw * 4 + 4, st));
    FC_CUDA_TRY(cudaMemsetAsync(s->N, 0, nw * 4 + 4, st));
    if (n && L) {
        dim3 tg(std::max<uint32_t>(1u, std::min<uint32_t>((n + 255) / 256, 8u * sm_count())), octets);
        const bool wide = L > 4;
        auto* const core_rows = wide ? k_core_rows<true> : k_core_rows<false>;
        core_rows<<<tg, 256, 0, st>>>(d->table, n, lo, hi, octets, s->rows);
        FC_CUDA_TRY(cudaGetLastError());
        dim3 ng(per_col, hi - lo);
        k_node_hist<<<ng, 256, 12288 * 4, st>>>(d->table + (uint64_t)lo * n, n, s->d_nbase + lo,
                                               s->d_kmax + lo, s->N);
        count_launch(2);
        FC_CUDA_TRY(cudaGetLastError());
        // once per process (thread-safe static initialisation)
        static const cudaError_t attr_rc[2] = {
            cudaFuncSetAttribute(k_edge_hist<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 EH_BINS * 4),
            cudaFuncSetAttribute(k_edge_hist<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 EH_BINS * 4)};
        FC_CUDA_TRY(attr_rc[wide]);
        auto* const edge_hist = wide ? k_edge_hist<true> : k_edge_hist<false>;
        FastDiv divL;
        divL.init(L);
        // Blocks: one per 4096 entries, at most two per SM (they share an SM
        // where the bins leave room for two: 180,001 nodes x 17 layers 0.4 ms
        // less than one).  With many groups the groups fill the device, and a
        // block clears and flushes its group's bins: then one per 16,384
        // entries (220 nodes x 360 layers, 610K entries: 1.94 ms a pass with
        // 16,384 and 2.00 with 4096; one group of 280K entries: 0.38 and 0.36).
        const uint64_t most = 2ull * sm_count();
        const uint64_t few = std::max<uint64_t>(
            1, std::min<uint64_t>(most, (d->entries + 16383) / 16384));
        const uint64_t many = std::max<uint64_t>(
            1, std::min<uint64_t>(most, (d->entries + 4095) / 4096));
        // 16-bit bins when no block can count 65,536 in one bin (each entry
        // adds at most 2): twice the columns per pass over the entries
        const uint64_t warps = few * (EH_THREADS / 32);
        const bool half =
            2 * ((d->entries + warps - 1) / warps + 31) * (EH_THREADS / 32) < 65536;
        const uint32_t budget = half ? 2 * EH_BINS : EH_BINS;  // bins
        EdgeGroups groups;
        uint32_t ng_e = 0, lam = lo;
        size_t shb = 0;
        while (lam < hi && d->entries) {
            uint64_t bins = 0;
            uint32_t nl = 0;
            while (lam + nl < hi && nl < EH_MAX_COLS) {
                const uint64_t w = (uint64_t)L * (s->kmax[lam + nl] + 1);
                if (nl > 0 && bins + w > budget) break;
                bins += w;
                nl++;
            }
            EdgeGroup& gr = groups.g[ng_e++];
            gr.lam0 = lam;
            gr.nl = nl;
            gr.bins = (uint32_t)std::min<uint64_t>(bins, budget + 1);
            gr.mode = bins > budget ? 0 : half ? 2 : 1;
            if (gr.mode) shb = std::max(shb, 4 * (size_t)(half ? (bins + 1) / 2 : bins));
            lam += nl;
            if (ng_e == EH_MAX_GROUPS || lam >= hi) {
                const uint32_t blocks =
                    (uint32_t)std::max(few, std::min(many, most / ng_e));
                edge_hist<<<dim3(blocks, ng_e), EH_THREADS, shb, st>>>(
                    d->node_ptr, d->adj, n, L, d->entries, divL, s->rows, octets, groups,
                    s->d_hbase, s->d_kmax, s->H);
                count_launch();
                FC_CUDA_TRY(cudaGetLastError());
                ng_e = 0;
                shb = 0;
            }
        }
        const uint64_t srows = (uint64_t)(hi - lo) * (L + 1);
        k_suffix<<<(uint32_t)std::min<uint64_t>((srows + 7) / 8, 8u * sm_count()), 256, 0, st>>>(
            L, lo, hi, s->d_hbase, s->d_nbase, s->d_kmax, s->H, s->N);
        count_launch();
        FC_CUDA_TRY(cudaGetLastError());
    }
    s->hist_valid = true;
    s->lo = lo;
    s->hi = hi;
    return FC_OK;
}

static fc_status score_cells(DeviceGraph* d, double beta, cudaStream_t st) {
    DensState* s = (DensState*)d->dens;
    const uint32_t L = d->L;
    if (!s->powl) FC_TRY(dev_alloc((void**)&s->powl, L * 8 + 8, st));
    std::vector<double> pw(L);
    for (uint32_t l = 0; l < L; l++) pw[l] = pow((double)(l + 1), beta);  // pow((l+1), beta)
    FC_TRY(to_device(s->powl, pw.data(), L * 8, st));
    if (!s->ncells) return FC_OK;
    uint32_t P = 1;
    while (P < L) P <<= 1;
    uint32_t threads = P < 32 ? 32 : (P > 1024 ? 1024 : P);
    size_t shb = (size_t)P * 4;
    if (shb > 48 * 1024) FC_CUDA_TRY(cudaFuncSetAttribute(k_cells, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shb));
    k_cells<<<(uint32_t)s->ncells, threads, shb, st>>>(L, P, s->d_hbase, s->d_nbase, s->d_kmax, s->H,
                                                      s->N, s->powl, s->cell_lk,
                                                      s->cell_lk + s->ncells, s->cells);
    count_launch();
    FC_CUDA_TRY(cudaGetLastError());
    return FC_OK;
}

fc_status densest(fc_graph* g, const double* betas, uint32_t nb, fc_densest_result* res,
                  cudaStream_t st, const std::function<fc_status()>* after_maxima) {
    FC_TRY(coreindex(g, nullptr, false, st));
    DeviceGraph* d = g->dev;
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
    cudaEvent_t e0 = ev.e0, e1 = ev.e1;
    FC_CUDA_TRY(cudaEventRecord(e0, st));
    FC_TRY(build_hist(d, st, 0, d->L, after_maxima));
    DensState* s = (DensState*)d->dens;
    if (!s->d_res) FC_TRY(dev_alloc((void**)&s->d_res, sizeof(fc_densest_result), st));
    for (uint32_t b = 0; b < nb; b++) {
        FC_TRY(score_cells(d, betas[b], st));
        k_fold<<<1, 1024, 0, st>>>(s->cells, s->ncells, betas[b], s->d_res);
        count_launch();
        FC_CUDA_TRY(cudaGetLastError());
        FC_TRY(to_host(res + b, s->d_res, sizeof(fc_densest_result), st));
    }
    FC_CUDA_TRY(cudaEventRecord(e1, st));
    FC_CUDA_TRY(cudaStreamSynchronize(st));
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    d->stats.densest_ms = ms;
    return FC_OK;
}

fc_status cells(fc_graph* g, double beta, fc_cell* out, uint32_t cap, uint32_t* count,
                cudaStream_t st) {
    FC_TRY(coreindex(g, nullptr, false, st));
    DeviceGraph* d = g->dev;
    FC_TRY(build_hist(d, st, 0, d->L));
    DensState* s = (DensState*)d->dens;
    FC_TRY(score_cells(d, beta, st));
    uint64_t nc = s->ncells;
    if (count) *count = (uint32_t)nc;
    uint64_t w = nc < cap ? nc : cap;
    if (w && out) FC_TRY(to_host(out, s->cells, w * sizeof(fc_cell), st));
    FC_CUDA_TRY(cudaStreamSynchronize(st));
    return FC_OK;
}

// The cells of the lambda columns [lo, hi) (0-based), computing those
// columns first when they are not resident.
fc_status cells_range(fc_graph* g, uint32_t lo, uint32_t hi, double beta, fc_cell* out, uint32_t cap,
                      uint32_t* count, cudaStream_t st) {
    FC_TRY(coreindex_range(g, lo, hi, nullptr, false, st));
    DeviceGraph* d = g->dev;
    FC_TRY(build_hist(d, st, lo, hi));
    DensState* s = (DensState*)d->dens;
    FC_TRY(score_cells(d, beta, st));
    const uint64_t nc = s->ncells;
    if (count) *count = (uint32_t)nc;
    const uint64_t w = nc < cap ? nc : cap;
    if (w && out) FC_TRY(to_host(out, s->cells, w * sizeof(fc_cell), st));
    FC_CUDA_TRY(cudaStreamSynchronize(st));
    d->home = nullptr;
    return FC_OK;
}

fc_status densest_members(fc_graph* g, const fc_densest_result* r, uint32_t* nodes,
                          uint32_t* layers, cudaStream_t st) {
    if (!r || r->k == 0) return FC_OK;
    FC_TRY(coreindex(g, nullptr, false, st));
    DeviceGraph* d = g->dev;
    FC_TRY(build_hist(d, st, 0, d->L));
    DensState* s = (DensState*)d->dens;
    const uint32_t n = d->n, L = d->L, lam = r->lmd - 1;
    if (r->lmd < 1 || r->lmd > L || r->k > s->kmax[lam]) return FC_ERR_INVALID;
    if (nodes) {
        std::vector<uint32_t> col(n);
        FC_TRY(to_host(col.data(), d->table + (uint64_t)lam * n, (uint64_t)n * 4, st));
        uint32_t j = 0;
        for (uint32_t v = 0; v < n; v++)
            if (col[v] >= r->k) nodes[j++] = v;
    }
    if (layers) {
        // the cell's layer counts; the first lstar of the descending order
        // (ties by layer index) -- for beta >= 0 lstar never splits a tie
        const uint32_t km1 = s->kmax[lam] + 1;
        std::vector<uint32_t> e(L);
        for (uint32_t l = 0; l < L; l++)
            FC_TRY(to_host(&e[l], s->H + s->hbase[lam] + (uint64_t)l * km1 + r->k, 4, st));
        std::vector<uint32_t> idx(L);
        for (uint32_t l = 0; l < L; l++) idx[l] = l;
        std::stable_sort(idx.begin(), idx.end(), [&](uint32_t a, uint32_t b) { return e[a] > e[b]; });
        std::vector<uint32_t> pick(idx.begin(), idx.begin() + r->lstar);
        std::sort(pick.begin(), pick.end());
        for (uint32_t i = 0; i < r->lstar; i++) layers[i] = pick[i];
    }
    return FC_OK;
}

void invalidate_densest(DeviceGraph* d) {
    invalidate_cell_index(d);
    DensState* s = (DensState*)d->dens;
    if (s) s->hist_valid = false;
}

// C_{k,lambda} = {v : core_lambda(v) >= k} in ascending ids, by an
// order-preserving stream compaction of the lambda column on the device (the
// query of -m kpe -k -lmd, main.cpp:197-225 and FCTree::saveCoreToLocal,
// Core/FCTree.cpp:138-153).
struct InCell {
    const uint32_t* col;
    uint32_t k;
    __host__ __device__ __forceinline__ bool operator()(uint32_t v) const { return col[v] >= k; }
};

fc_status cell_members(fc_graph* g, uint32_t k, uint32_t lmd, uint32_t* nodes, uint32_t cap,
                       uint32_t* count, cudaStream_t st) {
    if (lmd < 1 || lmd > g->L) return FC_ERR_INVALID;
    FC_TRY(coreindex(g, nullptr, false, st));
    DeviceGraph* d = g->dev;
    const uint32_t n = d->n;
    uint32_t* out = nullptr;
    uint32_t* num = nullptr;
    void* tmp = nullptr;
    size_t tb = 0;
    const InCell pred{d->table + (uint64_t)(lmd - 1) * n, k};
    thrust::counting_iterator<uint32_t> ids(0);
    FC_CUDA_TRY(cub::DeviceSelect::If(nullptr, tb, ids, out, num, (int)n, pred, st));
    fc_status rc = dev_alloc((void**)&out, (uint64_t)n * 4 + 4, st);
    if (rc == FC_OK) rc = dev_alloc((void**)&num, 8, st);
    if (rc == FC_OK) rc = dev_alloc(&tmp, tb + 16, st);
    uint32_t total = 0;
    if (rc == FC_OK) {
        const cudaError_t e = cub::DeviceSelect::If(tmp, tb, ids, out, num, (int)n, pred, st);
        count_launch(1);
        if (e != cudaSuccess) {
            set_last_cuda_error(e, "DeviceSelect::If", __FILE__, __LINE__);
            rc = FC_ERR_DEVICE;
        }
    }
    if (rc == FC_OK) rc = to_host(&total, num, 4, st);
    if (rc == FC_OK && nodes && total)
        rc = to_host(nodes, out, (size_t)std::min(total, cap) * 4, st);
    dev_free(tmp, st);
    dev_free(num, st);
    dev_free(out, st);
    if (count) *count = total;
    return rc;
}

void densest_preload() {
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, k_colmax);
    cudaFuncGetAttributes(&a, k_core_rows<false>);
    cudaFuncGetAttributes(&a, k_core_rows<true>);
    cudaFuncGetAttributes(&a, k_node_hist);
    cudaFuncGetAttributes(&a, k_edge_hist<false>);
    cudaFuncGetAttributes(&a, k_edge_hist<true>);
    cudaFuncGetAttributes(&a, k_suffix);
    cudaFuncGetAttributes(&a, k_cells);
    cudaFuncGetAttributes(&a, k_fold);
    cudaGetLastError();
}

}  // namespace fc
