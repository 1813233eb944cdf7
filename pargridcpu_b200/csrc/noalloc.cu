// fc_coreindex_fixed_scratch: the core-index peel for callers that cannot
// allocate device memory.
//
// Some callers must not call cudaMalloc (or anything that does): an
// application whose memory manager reserved the whole device up front and
// hands out nothing more, or a latency-bound loop that cannot afford a device
// allocation, which may synchronise the device and stall every stream.  This
// entry point takes the graph and the output table in device memory the
// caller already owns and runs the same peel kernel as fc_coreindex with its
// scratch carved from one fixed array in this file, FC_FIXED_SCRATCH_BYTES
// (64 MiB), which every GPU that loads this module holds until the process
// exits.  It allocates nothing itself.
//
// Set-up: the first call on a device looks the array's device address up
// with that device current (cudaGetSymbolAddress); make that first call before
// any stream capture.  All calls share the one array and it keeps the last
// call's contents: each call clears what must start empty (queues, control
// block) before its kernel runs, and calls that overlap on the GPU -- on two
// streams, or from two host threads -- race on it.
//
// The caller's CSR is checked before the peel reads it: node_ptr must start
// at 0, never decrease and end at `entries`, and every slot must name one of
// the n*L degree counters.  Those are the properties the peel's indexing
// rests on; a violation ends the call with FC_ERR_INVALID.  Rows may repeat a
// neighbour (the library's own never do).  Where such a row has a degree past
// 16 bits, the peel runs on 32-bit degrees: the packed one relies on as many
// nodes as a degree counts.  So the check also lists the nodes with such a
// degree, and a second one looks for repeats in their rows.
#include <algorithm>
#include <mutex>

#include "device.h"

namespace fc {

constexpr size_t FIXED_SCRATCH_BYTES = 64ull << 20;
// the peel's part; the last 256 bytes hold what the input checks find
constexpr size_t PEEL_SCRATCH_BYTES = FIXED_SCRATCH_BYTES - 256;

// The scratch itself.  In host code this name is a host-side stand-in, not a
// device address: kernels are given the address from cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_fixed_scratch[FIXED_SCRATCH_BYTES];

static std::mutex g_fixed_mu;
static void* g_fixed_addr[64];  // per device

// Device address of the fixed scratch on the current device (looked up once).
static fc_status fixed_scratch(void** out) {
    int dev = 0;
    FC_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return FC_ERR_DEVICE;
    std::lock_guard<std::mutex> lk(g_fixed_mu);
    if (!g_fixed_addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_fixed_scratch);
        if (e != cudaSuccess || !p) {
            set_last_cuda_error(e, "cudaGetSymbolAddress(g_fixed_scratch)", __FILE__, __LINE__);
            return FC_ERR_DEVICE;
        }
        g_fixed_addr[dev] = p;
    }
    *out = g_fixed_addr[dev];
    return FC_OK;
}

struct Found {
    uint32_t bad;      // the CSR cannot be indexed safely
    uint32_t hubs;     // (node, layer)s of degree past 16 bits
    uint32_t repeats;  // a neighbour named twice in a layer by one of their nodes
};
// hubs listed at most (a graph of the array's size has fewer than 2^32 entries)
constexpr uint32_t HUBS_MOST = 65536;

// Bounded input check (grid-stride, no waits): f->bad when node_ptr does not
// start at 0, decreases or does not end at `entries`, or a slot is not below
// nL; the nodes with a degree past 16 bits go to `hubs`.
__global__ void k_check_csr(const uint32_t* __restrict__ node_ptr, uint32_t n,
                            const uint32_t* __restrict__ adj, uint64_t entries, uint64_t nL,
                            FastDiv divL, const uint32_t* __restrict__ deg0,
                            uint32_t* __restrict__ hubs, Found* __restrict__ f) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    uint32_t b = 0;
    if (t == 0 && (node_ptr[0] != 0 || node_ptr[n] != entries)) b = 1;
    for (uint64_t v = t; v < n; v += stride)
        if (node_ptr[v + 1] < node_ptr[v]) b = 1;
    for (uint64_t e = t; e < entries; e += stride)
        if (adj[e] >= nL) b = 1;
    for (uint64_t i = t; i < nL; i += stride)
        if (deg0[i] > 0xFFFFu) {
            const uint32_t h = atomicAdd(&f->hubs, 1u);
            if (h < HUBS_MOST) hubs[h] = divL.div((uint32_t)i);
        }
    if (__any_sync(0xffffffffu, b) && (threadIdx.x & 31) == 0) atomicOr(&f->bad, 1u);
}

// A block per listed node (grid-stride): its row's slots in a bitmap of nL
// bits, `words` words a block.  Bounded by the row; runs on a checked CSR.
// Where hubs repeat no neighbour the columns stay packed: 89,966 nodes x 4
// layers with a degree of 70,001 take 1.96 ms so, and 2.78 on 32-bit degrees.
__global__ void k_check_repeats(const uint32_t* __restrict__ node_ptr,
                                const uint32_t* __restrict__ adj, const uint32_t* __restrict__ hubs,
                                uint32_t count, uint32_t* __restrict__ bits, uint32_t words,
                                Found* __restrict__ f) {
    uint32_t* const mine = bits + (uint64_t)blockIdx.x * words;
    for (uint32_t h = blockIdx.x; h < count; h += gridDim.x) {
        for (uint32_t w = threadIdx.x; w < words; w += blockDim.x) mine[w] = 0;
        __syncthreads();
        const uint32_t v = hubs[h];
        uint32_t twice = 0;
        for (uint32_t e = node_ptr[v] + threadIdx.x; e < node_ptr[v + 1]; e += blockDim.x) {
            const uint32_t s = adj[e], bit = 1u << (s & 31);
            twice |= atomicOr(mine + (s >> 5), bit) & bit;
        }
        if (twice) atomicOr(&f->repeats, 1u);
        __syncthreads();
    }
}

}  // namespace fc

using namespace fc;

extern "C" fc_status fc_coreindex_fixed_scratch(uint32_t n, uint32_t n_layers, uint64_t entries,
                                                const uint32_t* node_ptr, const uint32_t* adj,
                                                const uint32_t* deg0, uint32_t* table,
                                                void* stream) {
    if (!cuda_available()) return FC_ERR_NO_DEVICE;
    if (n == 0 || n_layers == 0) return FC_OK;
    if (!node_ptr || !deg0 || !table || (entries && !adj)) return FC_ERR_INVALID;
    if ((uint64_t)n * n_layers >= (1ull << 32) || entries >= (1ull << 32)) return FC_ERR_TOO_LARGE;
    // the most columns per launch whose scratch fits the fixed array; a graph
    // whose single column does not fit is rejected before any device work
    uint32_t cols = n_layers;
    // core <= largest degree <= n - 1 bounds the level count
    PeelGraph g{n, n_layers, entries, node_ptr, adj, deg0, n + 1};
    // (with the form for a peel's last levels when all columns fit with it)
    bool late = peel_ws_bytes(g, cols, true) <= PEEL_SCRATCH_BYTES;
    while (!late && cols > 0 && peel_ws_bytes(g, cols) > PEEL_SCRATCH_BYTES) cols--;
    if (cols == 0) return FC_ERR_TOO_LARGE;
    void* ws = nullptr;
    FC_TRY(fixed_scratch(&ws));
    cudaStream_t s = (cudaStream_t)stream;
    {
        // (the peel's scratch is free until it runs)
        Found* const f = (Found*)((char*)ws + PEEL_SCRATCH_BYTES);
        uint32_t* const hubs = (uint32_t*)ws;
        uint32_t* const bits = hubs + HUBS_MOST;
        FC_CUDA_TRY(cudaMemsetAsync(f, 0, sizeof(Found), s));
        FastDiv divL;
        divL.init(n_layers);
        int dev = 0, sms = 0;
        FC_CUDA_TRY(cudaGetDevice(&dev));
        FC_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        k_check_csr<<<sms * 4, 256, 0, s>>>(node_ptr, n, adj, entries, (uint64_t)n * n_layers, divL,
                                           deg0, hubs, f);
        count_launch();
        FC_CUDA_TRY(cudaGetLastError());
        Found found{};
        FC_TRY(to_host(&found, f, sizeof(found), s));
        if (found.bad) return FC_ERR_INVALID;
        if (found.hubs) {
            const uint32_t words = (uint32_t)(((uint64_t)n * n_layers + 31) / 32);
            const uint64_t fit = (PEEL_SCRATCH_BYTES / 4 - HUBS_MOST) / words;
            const uint32_t blocks = (uint32_t)std::min<uint64_t>(fit, std::min<uint64_t>(sms, found.hubs));
            g.repeats = true;
            if (found.hubs <= HUBS_MOST && blocks) {
                k_check_repeats<<<blocks, 1024, 0, s>>>(node_ptr, adj, hubs, found.hubs, bits, words, f);
                count_launch();
                FC_CUDA_TRY(cudaGetLastError());
                FC_TRY(to_host(&found, f, sizeof(found), s));
                g.repeats = found.repeats != 0;
            }
        }
    }
    if (g.repeats) {  // (a column alone, which fits, never has more than 32 bits a degree)
        late = false;
        cols = n_layers;
        while (cols > 1 && peel_ws_bytes(g, cols) > PEEL_SCRATCH_BYTES) cols--;
    }
    for (uint32_t c0 = 0; c0 < n_layers; c0 += cols) {
        const uint32_t nc = n_layers - c0 < cols ? n_layers - c0 : cols;
        PeelStats st;
        FC_TRY(peel_run(g, c0, nc, table, ws, PEEL_SCRATCH_BYTES, s, &st, false, late));
    }
    return FC_OK;
}
