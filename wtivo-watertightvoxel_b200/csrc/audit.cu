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
// a random sector of a table larger than L2.  Measured on B200, 5.24M-face
// torus: counting 350 -> 212 us, now bound by the rate of 64-bit CAS (69G/s), and
// no pass over the table afterwards (43 us); the whole call 495 -> 263 us.
// 5M unrelated triangles 685 -> 404 us, 5M faces over 2.5M random ids 688 -> 686
// us; only a fan of millions of faces around one vertex, whose full window every
// face asks first, got slower (5M faces: 580 -> 1450 us).  Reading the window
// through L1 first helped neither (319 us on the torus, 1920 us on the fan: old
// lines there cost CASes that fail).
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

constexpr uint32_t WINDOW = 8u;   // slots of a vertex's window (64 bytes)

// What one face more does to the number of bad edges when a count goes from
// c to c + 1 (0 -> 1: one more, 1 -> 2: one less, 2 -> 3: one more).
__device__ __forceinline__ int bad_step(unsigned long long c) { return c == 1ull ? -1 : 1; }

// Puts one face of the edge into `slot`, which held v when it was read: true
// when the slot is or became the edge's (bad then holds the change of the
// number of bad edges), false when it holds another edge.
__device__ __forceinline__ bool count_in_slot(unsigned long long* slot, unsigned long long v,
                                              unsigned long long edge, int* bad)
{
    if (v == 0ull) {
        v = atomicCAS(slot, 0ull, edge | COUNT_ONE);
        if (v == 0ull) {
            *bad += 1;
            return true;
        }
    }
    if ((v & EDGE_MASK) != edge) return false;
    // raise the count, saturating at 3 (the slot's edge never changes)
    while ((v >> 62) != 3ull) {
        const unsigned long long w = atomicCAS(slot, v, v + COUNT_ONE);
        if (w == v) {
            *bad += bad_step(v >> 62);
            return true;
        }
        v = w;
    }
    return true;
}

constexpr uint64_t SCATTER = 64u;   // scattered probes after the window's

// Counts one edge: its probe sequence is the window of its lower vertex, then
// (a vertex of many edges, or ids that share a window) scattered slots, a new
// hash for each, then the whole table in order.  Neighbouring windows fill up
// together, so stepping on from a full one would walk a long run of full
// windows (1M faces over 500k random ids: 1.5 s); scattered probes meet a used
// slot at most three times in four.  Slots are never emptied, so every face of
// an edge walks the same sequence to the same slot, and a table with a free
// slot always ends it (at most 3/4 get used; a full table is reported).
__device__ __forceinline__ void count_edge(uint32_t lo, uint32_t hi, unsigned long long* table, uint64_t cap,
                                           uint32_t nwin, int* bad, int* err)
{
    const unsigned long long edge = ((unsigned long long)lo << 31) | hi;
    unsigned long long* win = table + (size_t)(lo % nwin) * WINDOW;
    const unsigned long long mix = mix64(edge);
    for (uint32_t p = 0; p < WINDOW; ++p) {
        unsigned long long* slot = win + (((uint32_t)mix + p) & (WINDOW - 1u));
        if (count_in_slot(slot, __ldcg(slot), edge, bad)) return;
    }
    for (uint64_t p = 0; p < SCATTER; ++p) {
        unsigned long long* slot = table + __umul64hi(mix64(mix + (p + 1u) * 0x9e3779b97f4a7c15ull), cap);
        if (count_in_slot(slot, __ldcg(slot), edge, bad)) return;
    }
    for (uint64_t slot = 0; slot < cap; ++slot)
        if (count_in_slot(table + slot, __ldcg(table + slot), edge, bad)) return;
    atomicOr(err, 2);
}

// wtivo_core.cpp:420-446: the three undirected edges of every face, and the
// number of distinct edges whose face count is not 2
__global__ void __launch_bounds__(ATPB) k_edge_count(const int32_t* __restrict__ faces, uint64_t nf,
                                                     unsigned long long* table, uint64_t cap, uint32_t nwin,
                                                     unsigned long long* bad, int* err)
{
    __shared__ int s[ATPB / 32];
    int b = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * ATPB + threadIdx.x; i < nf;
         i += (uint64_t)gridDim.x * ATPB) {
        const int32_t v0 = __ldg(faces + 3u * i), v1 = __ldg(faces + 3u * i + 1u),
                      v2 = __ldg(faces + 3u * i + 2u);
        if (v0 < 0 || v1 < 0 || v2 < 0) {   // :424 "negative vertex index"
            atomicOr(err, 1);
            continue;
        }
        const uint32_t ua = (uint32_t)v0, ub = (uint32_t)v1, uc = (uint32_t)v2;
        count_edge(min(ua, ub), max(ua, ub), table, cap, nwin, &b, err);
        count_edge(min(ub, uc), max(ub, uc), table, cap, nwin, &b, err);
        count_edge(min(uc, ua), max(uc, ua), table, cap, nwin, &b, err);
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
