// audit.cu -- edge-degree watertight audit of a triangle mesh on the GPU.
//
// Replaces is_watertight (native/core/wtivo_core.cpp:402-464).  A closed
// 2-manifold triangle mesh has every undirected edge in exactly two faces;
// the audit reports the number of "bad edge groups": distinct undirected
// edges whose face count is not 2.
//
// The reference writes 3F 64-bit edge keys (min << 32 | max), sorts them on
// host threads and counts runs of equal keys.  Here no sort is needed: every
// edge is counted in a device hash table (open addressing), and the bad groups
// are summed while the counts change: an edge is bad when its first face
// comes, good with the second, bad again with the third.  The number is the
// same: a run of equal keys in the sorted array is exactly one table entry, and
// its length is the entry's count.
//
// One 8-byte slot per edge: the edge as min * 2^31 + max (vertex ids are
// below 2^31, so 62 bits) and, in the top two bits, its face count
// saturating at 3 (1, 2, or "3 or more": the rule only asks whether the count
// is 2).  A slot is claimed with a 64-bit CAS that writes the edge with
// count 1 and raised with CAS; a used slot is never 0 (its count is at least
// 1), so 0 marks an empty slot.  Key and count share one 32-byte sector, so
// an edge update touches one sector of the table, not two.
//
// An edge is looked for first in the 64-byte window of its lower vertex, so
// the table is walked in the order of the mesh: a mesh's vertices and faces are
// numbered along its surface, and a vertex is the lower end of three edges on
// average.  With a slot from a mixed hash of the whole edge instead, every update was
// a random sector of a table larger than L2.  An edge asks three slots there,
// then those of its higher vertex's window, and scatters only then: asking all
// eight of the lower vertex's first, the spokes of a fan, whose centre's window
// fills at once, queued at that one line (5M faces: 1370 us).  An edge that two
// faces next to each other share, as in a strip or a fan, is counted once, by
// two, when their threads are neighbours in a warp.
//
// The whole call on B200, 5M faces, with a hash of the whole edge and a pass over
// the table afterwards / eight slots of the lower vertex's window / now: grid-numbered
// torus 490 / 258 / 228 us, the same with random ids 490 / 327 / 268, sphere 636 /
// 407 / 412, fan around one vertex 582 / 1430 / 485, fans of 1000 faces 577 / 945 /
// 263, triangles that share nothing 677 / 410 / 444 (shuffled 676 / 437 / 466), faces
// over 2.5M random ids 678 / 668 / 617; 200k faces of the torus 70 / 43 / 46.  Without
// the sharing between neighbours: torus 272, with random ids 455, fan 415, fans of
// 1000 333.  Three slots of the second window instead of eight: torus 228,
// triangles that share nothing 490.  Bound by the rate of 64-bit CAS on the meshes,
// by random sectors on the rest.  Reading the window through L1 helped neither (old
// lines there cost CASes that fail), nor did loading four slots at once (random ids
// 1100-1300 us).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "gpupr_internal.cuh"

namespace gpupr {
namespace {

constexpr int ATPB = 256;
constexpr unsigned long long EDGE_MASK = (1ull << 62) - 1ull;   // the edge's 62 bits
constexpr unsigned long long COUNT_ONE = 1ull << 62;            // count field, bits 62-63

// 64-bit mixer and increment of SplitMix64 (Steele, Lea, Flood, "Fast
// splittable pseudorandom number generators", OOPSLA 2014): neighboring edge
// keys, and successive probes of one, land in unrelated slots.
__device__ __forceinline__ unsigned long long mix64(unsigned long long x)
{
    x ^= x >> 30;
    x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 27;
    x *= 0x94d049bb133111ebull;
    x ^= x >> 31;
    return x;
}

constexpr uint32_t WINDOW = 8u;     // slots of a vertex's window (64 bytes)
constexpr uint32_t WINDOW_LOW = 3u; // of them asked in the lower vertex's window

// Puts c faces (1 or 2) of the edge into `slot`, which held v when it was read:
// true when the slot is or became the edge's, false when it holds another edge.
// bad gets the change of the number of bad edges (those whose count is not 2).
__device__ __forceinline__ bool count_in_slot(unsigned long long* slot, unsigned long long v,
                                              unsigned long long edge, uint32_t c, int* bad)
{
    if (v == 0ull) {
        v = atomicCAS(slot, 0ull, edge | (unsigned long long)c * COUNT_ONE);
        if (v == 0ull) {
            *bad += c == 1u;
            return true;
        }
    }
    if ((v & EDGE_MASK) != edge) return false;
    // raise the count, saturating at 3 (the slot's edge never changes)
    while ((v >> 62) != 3ull) {
        const unsigned long long n = min((v >> 62) + c, 3ull);
        const unsigned long long w = atomicCAS(slot, v, edge | n * COUNT_ONE);
        if (w == v) {
            *bad += (int)(n == 3ull) - (int)((v >> 62) == 1ull);
            return true;
        }
        v = w;
    }
    return true;
}

constexpr uint64_t SCATTER = 64u;   // scattered probes after the windows'

// Counts c faces of an edge: its probe sequence is three slots of the window of
// its lower vertex, the window of its higher one, then (vertices of many edges, or
// ids that share a window) scattered slots, a new hash for each, then the whole
// table in order.  Neighbouring windows fill up together, so stepping on from a
// full one would walk a long run of full windows (1M faces over 500k random ids:
// 1.5 s); scattered probes meet a used slot at most three times in four.  Slots
// are never emptied, so every face of an edge walks the same sequence to the same
// slot, and a table with a free slot always ends it (at most 3/4 get used; a full
// table is reported).
__device__ __forceinline__ void count_edge(unsigned long long edge, uint32_t c, unsigned long long* table,
                                           uint64_t cap, uint32_t nwin, int* bad, int* err)
{
    const unsigned long long mix = mix64(edge);
    unsigned long long* win = table + (size_t)((uint32_t)(edge >> 31) % nwin) * WINDOW;
    for (uint32_t p = 0; p < WINDOW_LOW; ++p) {
        unsigned long long* slot = win + (((uint32_t)mix + p) & (WINDOW - 1u));
        if (count_in_slot(slot, __ldcg(slot), edge, c, bad)) return;
    }
    win = table + (size_t)((uint32_t)(edge & 0x7fffffffull) % nwin) * WINDOW;
#pragma unroll 1
    for (uint32_t p = 0; p < WINDOW; ++p) {
        unsigned long long* slot = win + (((uint32_t)mix + p) & (WINDOW - 1u));
        if (count_in_slot(slot, __ldcg(slot), edge, c, bad)) return;
    }
    for (uint64_t p = 0; p < SCATTER; ++p) {
        unsigned long long* slot = table + __umul64hi(mix64(mix + (p + 1u) * 0x9e3779b97f4a7c15ull), cap);
        if (count_in_slot(slot, __ldcg(slot), edge, c, bad)) return;
    }
    for (uint64_t slot = 0; slot < cap; ++slot)
        if (count_in_slot(table + slot, __ldcg(table + slot), edge, c, bad)) return;
    atomicOr(err, 2);
}

__device__ __forceinline__ unsigned long long edge_of(int a, int b)
{
    return ((unsigned long long)(uint32_t)min(a, b) << 31) | (uint32_t)max(a, b);
}

// How often this lane counts each of its edges: once, or twice where the next
// lane has the edge too, or not at all where the lane before counts it for both.
// Of a run of lanes with the same edge only the first pair shares it, so each
// instance is counted by exactly one lane.
__device__ __forceinline__ void share_edges(const unsigned long long (&e)[3], uint32_t (&c)[3])
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t to[3] = {0, 0, 0};   // bit of the next lane's edge that equals edge k
    uint32_t seen = 0;            // those bits together
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const unsigned long long o = __shfl_down_sync(0xffffffffu, e[j], 1);
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (lane != 31u && o == e[k] && !to[k] && !(seen & (1u << j))) {
                to[k] = 1u << j;
                seen |= 1u << j;
            }
    }
    uint32_t before = __shfl_up_sync(0xffffffffu, seen, 1);   // this lane's edges that the lane before has
    if (lane == 0u) before = 0u;
    uint32_t take = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const bool both = to[k] && !(before & (1u << k));
        c[k] = both ? 2u : 1u;
        if (both) take |= to[k];
    }
    const uint32_t taken = __shfl_up_sync(0xffffffffu, take, 1);
#pragma unroll
    for (int k = 0; k < 3; ++k)
        if (lane != 0u && (taken & (1u << k))) c[k] = 0u;
}

// wtivo_core.cpp:420-446: the three undirected edges of every face, and the
// number of distinct edges whose face count is not 2.  Full SMs (32 registers):
// with 40, random ids took twice as long.
__global__ void __launch_bounds__(ATPB) k_edge_count(const int32_t* __restrict__ faces, uint64_t nf,
                                                     unsigned long long* table, uint64_t cap, uint32_t nwin,
                                                     unsigned long long* bad, int* err)
{
    __shared__ int s[ATPB / 32];
    int b = 0;
    // whole warps: share_edges needs all lanes
    for (uint64_t first = (uint64_t)blockIdx.x * ATPB; first < nf; first += (uint64_t)gridDim.x * ATPB) {
        const uint64_t i = first + threadIdx.x;
        int32_t v0 = -1, v1 = 0, v2 = 0;
        if (i < nf) {
            v0 = __ldg(faces + 3u * i);
            v1 = __ldg(faces + 3u * i + 1u);
            v2 = __ldg(faces + 3u * i + 2u);
            if ((v0 | v1 | v2) < 0) atomicOr(err, 1);   // :424 "negative vertex index"
        }
        const bool face = (v0 | v1 | v2) >= 0;
        // lanes without a face hold what no edge is, and another in the next lane
        const unsigned long long none = ~0ull - (threadIdx.x & 1u);
        const unsigned long long e[3] = {face ? edge_of(v0, v1) : none, face ? edge_of(v1, v2) : none,
                                         face ? edge_of(v2, v0) : none};
        uint32_t c[3];
        share_edges(e, c);
        // one copy of the probe code: three take more registers than there are
        uint32_t left = face ? c[0] | c[1] << 2 | c[2] << 4 : 0u;
        unsigned long long edge = e[0], next = e[1], last = e[2];
#pragma unroll 1
        while (left) {
            if (left & 3u) count_edge(edge, left & 3u, table, cap, nwin, &b, err);
            left >>= 2;
            edge = next;
            next = last;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b += __shfl_down_sync(0xffffffffu, b, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long t = 0;
        for (int w = 0; w < ATPB / 32; ++w) t += s[w];
        if (t) atomicAdd(bad, (unsigned long long)t);   // modulo 2^64: the sum is not negative
    }
}

}  // namespace

void edge_audit(const int32_t* d_faces, uint64_t nf, cudaStream_t s, uint64_t* bad_groups,
                uint64_t* table_bytes, uint64_t* launches)
{
    *bad_groups = 0;
    *table_bytes = 0;
    if (!nf) return;
    if (nf > (1ull << 40)) throw Error{GPUPR_ERR_INVALID_ARGUMENT, "too many faces"};
    // four slots per face: a closed mesh has half as many vertices as faces, so
    // each gets a window of its own, and 3F distinct edges still fit
    const uint64_t cap = std::max<uint64_t>(1024u, (4u * nf + WINDOW - 1u) / WINDOW * WINDOW);
    const uint32_t nwin = (uint32_t)std::min<uint64_t>(cap / WINDOW, 1ull << 31);
    DevBuf<unsigned long long> table(cap + 2u, s);   // the result and the error flag behind the slots
    unsigned long long* d_bad = table.p + cap;
    int* d_err = reinterpret_cast<int*>(d_bad + 1);
    GPUPR_CUDA(cudaMemsetAsync(table.p, 0, (cap + 2u) * 8u, s));
    const unsigned gf = (unsigned)std::min<uint64_t>((nf + ATPB - 1) / ATPB, (uint64_t)sm_count() * 16u);
    k_edge_count<<<gf, ATPB, 0, s>>>(d_faces, nf, table.p, cap, nwin, d_bad, d_err);
    GPUPR_CUDA(cudaGetLastError());
    if (launches) *launches += 1;
    unsigned long long hb = 0;
    int he = 0;
    unsigned long long h[2] = {0, 0};
    GPUPR_CUDA(cudaMemcpyAsync(h, d_bad, 16u, cudaMemcpyDeviceToHost, s));
    GPUPR_CUDA(cudaStreamSynchronize(s));
    hb = h[0];
    he = (int)h[1];
    if (he & 1) throw Error{GPUPR_ERR_INVALID_ARGUMENT, "negative vertex index"};
    if (he) throw Error{GPUPR_ERR_INVARIANT, "edge table full"};
    *bad_groups = hb;
    *table_bytes = cap * 8u;
}

}  // namespace gpupr
