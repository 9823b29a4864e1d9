// batch.cu -- many cell graphs solved as one.
//
// Graphs of a batch are independent, so their disjoint union is one cut
// problem: pack them end to end (local vertex and neighbor ids become global
// ids), build and solve the union once, and split the results.  Compaction
// keeps tet order, so each graph's free nodes form one contiguous range and
// per-graph flows are sums over that range:
//   raw_g  = sum over free v in g of max(term_v, 0) - excess_v
//            (a preflow conserves flow per graph: what entered from the
//            source and is not left as excess went into the sink; positive
//            terminals never change during the solve)
//   base_g = sum over free v in g of min(src_v, snk_v)
#include <cuda_runtime.h>
#include <stdint.h>

#include "gpupr_internal.cuh"

namespace gpupr {
namespace {

constexpr int TPB = 256;

__device__ __forceinline__ uint32_t graph_of(uint64_t i, const unsigned long long* off, uint32_t G)
{
    uint32_t lo = 0, hi = G;   // largest g with off[g] <= i
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (off[mid] <= i) lo = mid;
        else hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(TPB) k_batch_pack(uint64_t N, uint32_t G,
                                                    const unsigned long long* __restrict__ tet_off,
                                                    const unsigned long long* __restrict__ vert_off,
                                                    const int4* __restrict__ tets_l,
                                                    const int4* __restrict__ nbrs_l,
                                                    int4* __restrict__ tets_g, int4* __restrict__ nbrs_g)
{
    for (uint64_t i = (uint64_t)blockIdx.x * TPB + threadIdx.x; i < N; i += (uint64_t)gridDim.x * TPB) {
        const uint32_t g = graph_of(i, tet_off, G);
        const long long tb = (long long)tet_off[g], vb = (long long)vert_off[g];
        const long long ng = (long long)tet_off[g + 1] - tb;
        const long long nvg = (long long)vert_off[g + 1] - vb;
        const int4 t = __ldg(tets_l + i);
        const int4 b = __ldg(nbrs_l + i);
        // out-of-graph local ids become -2^31 (caught later as invalid vertex /
        // out-of-range neighbor) instead of aliasing into another graph
        auto vmap = [&](int x) -> int { return (x >= 0 && x < nvg) ? (int)(x + vb) : (int)0x80000000; };
        auto nmap = [&](int x) -> int {
            if (x < 0) return x;
            return x < ng ? (int)(x + tb) : 0x7FFFFFFF;
        };
        tets_g[i] = make_int4(vmap(t.x), vmap(t.y), vmap(t.z), vmap(t.w));
        nbrs_g[i] = make_int4(nmap(b.x), nmap(b.y), nmap(b.z), nmap(b.w));
    }
}

// Where each graph's free nodes begin: free_old ascends, so the first reduced
// id of graph g is the number of entries below the graph's first tet.  One
// binary search a graph reads a few hundred bytes; counting the map's
// non-negative entries took a block a graph over 4 bytes a tet (64 graphs of
// 50k-4M tets: 1990 us, now 16).
__global__ void __launch_bounds__(TPB) k_batch_free_offsets(uint32_t G, uint32_t F,
                                                            const unsigned long long* __restrict__ tet_off,
                                                            const uint32_t* __restrict__ free_old,
                                                            unsigned long long* __restrict__ free_off,
                                                            uint32_t* __restrict__ seg_off)
{
    const uint32_t g = blockIdx.x * TPB + threadIdx.x;
    if (g > G) return;
    const unsigned long long first = tet_off[g];
    uint32_t lo = 0, hi = F;   // free_old[< lo] < first <= free_old[>= hi]
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (__ldg(free_old + mid) < first) lo = mid + 1;
        else hi = mid;
    }
    free_off[g] = lo;
    seg_off[g] = lo;
}

constexpr uint32_t FLOW_GROUP = 128;   // nodes a warp loads at once, four a lane

// Bound by the loads of 16 bytes a node.  Each warp sums a strip of nodes
// whatever graph they are in, so a batch of uneven graphs fills the chip: a
// block a graph left the time to the largest one (the same 64 graphs:
// 4700 us, now 137, near the rate of a plain copy).  A group inside one graph
// is added to the warp's running sums, which go out once a strip and graph; a
// group over a boundary adds node by node.  Integer sums: the order does not
// matter.
__global__ void __launch_bounds__(TPB) k_batch_flows(uint32_t G, uint32_t n, uint32_t strip,
                                                     const unsigned long long* __restrict__ free_off,
                                                     const int32_t* __restrict__ term,
                                                     const long long* __restrict__ excess,
                                                     const uint32_t* __restrict__ base_node,
                                                     unsigned long long* __restrict__ raw,
                                                     unsigned long long* __restrict__ base)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t start = ((uint64_t)blockIdx.x * (TPB / 32) + (threadIdx.x >> 5)) * strip;
    if (start >= n) return;
    const uint64_t stop = start + strip < n ? start + strip : n;
    uint32_t g = graph_of(start, free_off, G);
    unsigned long long end = free_off[g + 1];
    unsigned long long r = 0, b = 0;
    auto flush = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            r += __shfl_down_sync(0xffffffffu, r, o);
            b += __shfl_down_sync(0xffffffffu, b, o);
        }
        if (lane == 0) {
            if (r) atomicAdd(raw + g, r);
            if (b) atomicAdd(base + g, b);
        }
        r = b = 0;
    };
    for (uint64_t p = start; p < stop; p += FLOW_GROUP) {
        long long e[4];
        int32_t t[4];
        uint32_t c[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t q = p + (uint32_t)k * 32u + lane;
            const bool in = q < stop;
            e[k] = in ? excess[q] : 0ll;
            t[k] = in ? __ldg(term + q) : 0;
            c[k] = in ? __ldg(base_node + q) : 0u;
        }
        const uint64_t last = p + FLOW_GROUP < stop ? p + FLOW_GROUP : stop;
        if (last <= end) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                r += (unsigned long long)((t[k] > 0 ? (long long)t[k] : 0ll) - e[k]);
                b += c[k];
            }
            continue;
        }
        flush();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t q = p + (uint32_t)k * 32u + lane;
            if (q >= stop) continue;
            const uint32_t gq = graph_of(q, free_off, G);
            const unsigned long long v = (unsigned long long)((t[k] > 0 ? (long long)t[k] : 0ll) - e[k]);
            if (v) atomicAdd(raw + gq, v);
            if (c[k]) atomicAdd(base + gq, (unsigned long long)c[k]);
        }
        if (last < stop) {
            g = graph_of(last, free_off, G);
            end = free_off[g + 1];
        }
    }
    flush();
}

}  // namespace

void batch_pack(uint64_t N, uint32_t G, const unsigned long long* d_tet_off,
                const unsigned long long* d_vert_off, const int32_t* d_tets_local,
                const int32_t* d_nbrs_local, int32_t* d_tets, int32_t* d_nbrs, cudaStream_t s,
                uint64_t* launches)
{
    if (!N) return;
    const uint64_t want = (N + TPB - 1) / TPB;
    const uint64_t cap = (uint64_t)sm_count() * 16u;
    k_batch_pack<<<(unsigned)(want < cap ? want : cap), TPB, 0, s>>>(
        N, G, d_tet_off, d_vert_off, reinterpret_cast<const int4*>(d_tets_local),
        reinterpret_cast<const int4*>(d_nbrs_local), reinterpret_cast<int4*>(d_tets),
        reinterpret_cast<int4*>(d_nbrs));
    GPUPR_CUDA(cudaGetLastError());
    *launches += 1;
}

void batch_free_offsets(uint32_t G, uint32_t F, const unsigned long long* d_tet_off,
                        const uint32_t* d_free_old, unsigned long long* d_free_off,
                        uint32_t* d_seg_off, cudaStream_t s, uint64_t* launches)
{
    k_batch_free_offsets<<<(G + TPB) / TPB, TPB, 0, s>>>(G, F, d_tet_off, d_free_old, d_free_off,
                                                         d_seg_off);
    GPUPR_CUDA(cudaGetLastError());
    *launches += 1;
}

void batch_flows(uint32_t G, uint32_t n, const unsigned long long* d_free_off, const int32_t* d_term,
                 const long long* d_excess, const uint32_t* d_base_node, long long* d_raw,
                 unsigned long long* d_base, cudaStream_t s, uint64_t* launches)
{
    if (!G) return;
    GPUPR_CUDA(cudaMemsetAsync(d_raw, 0, G * 8u, s));
    GPUPR_CUDA(cudaMemsetAsync(d_base, 0, G * 8u, s));
    if (!n) return;
    // strips of one group until every warp slot of the chip has one, then
    // longer ones up to 16 groups: fewer atomics on the graphs' sums
    const uint64_t slots = (uint64_t)sm_count() * 64u * FLOW_GROUP;
    const uint64_t want = (n + slots - 1) / slots;
    const uint32_t strip = FLOW_GROUP * (uint32_t)(want > 16u ? 16u : want);
    const uint64_t per_block = (uint64_t)strip * (TPB / 32);
    k_batch_flows<<<(unsigned)((n + per_block - 1) / per_block), TPB, 0, s>>>(
        G, n, strip, d_free_off, d_term, d_excess, d_base_node,
        reinterpret_cast<unsigned long long*>(d_raw), d_base);
    GPUPR_CUDA(cudaGetLastError());
    *launches += 1;
}

}  // namespace gpupr
