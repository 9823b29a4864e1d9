// labels.cu -- tet-centroid labels from a sparse unsigned distance grid.
//
// Replaces SparseUDF.sample_tet_labels (native/vdb/wtivo_vdb.cpp:1519-1584),
// the producer of the graph cut's initial labels: each tet's centroid is
// mapped into the unit query box, sampled from the narrow-band UDF with
// trilinear (box) interpolation, and labelled 0 (inside the band: source)
// when the sample is at most the threshold, else 1.  The reference runs this
// on host threads against an OpenVDB tree; here one GPU thread per tet reads
// a brick grid (8^3-voxel bricks behind a dense brick table) kept in HBM, so
// the labels are produced where the cut consumes them.
//
// Arithmetic follows the reference step by step in IEEE double (no FMA
// contraction: explicit __d*_rn operations), the index transform of an
// OpenVDB linear transform (world * (1 / voxel_size)), and OpenVDB 12.0.1's
// BoxSampler (openvdb/tools/Interpolation.h): the 8 voxels around
// floor(index), lerped along z, then y, then x, each lerp a + float((b-a)*w)
// with float values and a double weight.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "gpupr_internal.cuh"

namespace gpupr {
namespace {

constexpr int LTPB = 256;

struct GridView {
    double inv_h;
    int32_t origin[3];
    int32_t dims[3];
    float background;
    bool finite_bg;
    const int32_t* __restrict__ table;
    const float* __restrict__ values;
};

// The 8 voxels around the base voxel (i, j, k) of a box sample, in the order
// d[4x + 2y + z]; coordinates relative to the grid's origin.  Per axis the two
// voxels lie in one brick or in two neighbouring ones, so the brick and voxel
// offsets are sums of per-axis terms, and every lane does the same eight
// lookups (a path of its own for samples inside one brick, two in three, is
// executed next to the other one by nearly every warp).  False when all 8 are
// background because they lie in one inactive brick or outside.
template <class I>
__device__ __forceinline__ bool box_voxels(const GridView& g, I i, I j, I k, float (&d)[8])
{
    const I q[3] = {i, j, k};
    const I stride[3] = {(I)g.dims[1] * (I)g.dims[2], (I)g.dims[2], (I)1};
    I cell[3][2];
    int vox[3][2];
    bool in[3][2];
    bool one = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int vs = a == 0 ? 64 : a == 1 ? 8 : 1;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const I c = (q[a] + e) >> 3;   // floor: -1 below the origin
            in[a][e] = c >= 0 && c < g.dims[a];
            cell[a][e] = c * stride[a];
            vox[a][e] = (int)((q[a] + e) & 7) * vs;
        }
        one = one && vox[a][0] != 7 * vs;
    }
    int32_t b0 = -1;
    if (in[0][0] && in[1][0] && in[2][0]) b0 = __ldg(g.table + (cell[0][0] + cell[1][0] + cell[2][0]));
#pragma unroll
    for (int c = 0; c < 8; ++c) d[c] = g.background;
    if (one && b0 < 0) return false;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int x = c >> 2, y = (c >> 1) & 1, z = c & 1;
        int32_t b = b0;
        if (c != 0 && !one) {
            b = -1;
            if (in[0][x] && in[1][y] && in[2][z]) b = __ldg(g.table + (cell[0][x] + cell[1][y] + cell[2][z]));
        }
        if (b >= 0) d[c] = __ldg(g.values + ((size_t)b * 512u + (unsigned)(vox[0][x] + vox[1][y] + vox[2][z])));
    }
    return true;
}

// one lerp of the box sampler: a + float((b - a) * w)
__device__ __forceinline__ float box_lerp(float a, float b, double w)
{
    const float diff = __fsub_rn(b, a);
    return __fadd_rn(a, __double2float_rn(__dmul_rn((double)diff, w)));
}

// floor of an index coordinate, and the same relative to the grid's origin,
// clamped to just outside the grid's n bricks (all of it is background there).
// 32-bit: the conversion saturates, and the caller keeps the grid's ends away
// from the ends of the range.  A NaN coordinate goes anywhere: its weight is NaN,
// and so is the sample whatever the voxels hold.
__device__ __forceinline__ void floor_index(double x, int32_t origin, int32_t n, double& f, int& i)
{
    f = floor(x);
    const int v = __double2int_rz(f);
    i = min(max(v, origin - 16), origin + n * 8 + 8) - origin;
}
__device__ __forceinline__ void floor_index(double x, int32_t origin, int32_t n, double& f, long long& i)
{
    f = floor(x);
    i = (long long)fmin(fmax(f - (double)origin, -16.0), (double)n * 8.0 + 8.0);
}

// One thread per tet.  Bound by the instructions it issues (71% of the issue
// slots, 384 of them a tet: three exact divisions, the box lookups, seven lerps
// with their conversions), not by memory (21% of the copy rate).  24M tets around
// a knot, 580 -> 427 us for the call: 32-bit voxel coordinates from saturating
// conversions, one path for all lookups, background samples without lerps, one
// range check a tet, the next tet's row loaded ahead.
// I: the type of voxel coordinates relative to the grid's origin
template <class I>
__global__ void __launch_bounds__(LTPB) k_sample_labels(GridView g, const double* __restrict__ V,
                                                        uint32_t nv, const int4* __restrict__ tets,
                                                        uint64_t nt, double3 bmin, double3 span,
                                                        double scale, double padding,
                                                        double threshold, uint8_t* labels,
                                                        float* udf, int* err)
{
    const uint64_t step = (uint64_t)gridDim.x * LTPB;
    uint64_t i = (uint64_t)blockIdx.x * LTPB + threadIdx.x;
    int4 next = i < nt ? __ldg(tets + i) : make_int4(0, 0, 0, 0);
    for (; i < nt; i += step) {
        const int4 t = next;
        if (i + step < nt) next = __ldg(tets + i + step);   // in flight while this tet is sampled
        const uint32_t q[4] = {(uint32_t)t.x, (uint32_t)t.y, (uint32_t)t.z, (uint32_t)t.w};
        if (q[0] >= nv || q[1] >= nv || q[2] >= nv || q[3] >= nv) {   // negative ids are 2^31 and up
            atomicOr(err, 1);
            continue;
        }
        double cx = 0.0, cy = 0.0, cz = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {   // wtivo_vdb.cpp:1563-1570
            const double* p = V + 3u * (size_t)q[k];
            cx = __dadd_rn(cx, __ldg(p));
            cy = __dadd_rn(cy, __ldg(p + 1));
            cz = __dadd_rn(cz, __ldg(p + 2));
        }
        cx = __dmul_rn(cx, 0.25);
        cy = __dmul_rn(cy, 0.25);
        cz = __dmul_rn(cz, 0.25);
        // :1572-1574, then the grid's index transform
        const double nx = __dadd_rn(__dmul_rn(__ddiv_rn(__dsub_rn(cx, bmin.x), span.x), scale), padding);
        const double ny = __dadd_rn(__dmul_rn(__ddiv_rn(__dsub_rn(cy, bmin.y), span.y), scale), padding);
        const double nz = __dadd_rn(__dmul_rn(__ddiv_rn(__dsub_rn(cz, bmin.z), span.z), scale), padding);
        const double x = __dmul_rn(nx, g.inv_h), y = __dmul_rn(ny, g.inv_h), z = __dmul_rn(nz, g.inv_h);
        double fx, fy, fz;
        I ix, iy, iz;
        floor_index(x, g.origin[0], g.dims[0], fx, ix);
        floor_index(y, g.origin[1], g.dims[1], fy, iy);
        floor_index(z, g.origin[2], g.dims[2], fz, iz);
        const double u = __dsub_rn(x, fx), v = __dsub_rn(y, fy), w = __dsub_rn(z, fz);
        float d[8];
        float val;
        // equal finite samples lerp to themselves (+0 for -0) unless a weight
        // is NaN: most of space is background and skips the seven lerps
        if (box_voxels<I>(g, ix, iy, iz, d) || !g.finite_bg || !(u + v + w < 3.0)) {
            val = box_lerp(box_lerp(box_lerp(d[0], d[1], w), box_lerp(d[2], d[3], w), v),
                           box_lerp(box_lerp(d[4], d[5], w), box_lerp(d[6], d[7], w), v), u);
        } else {
            val = g.background + 0.0f;
        }
        labels[i] = ((double)val <= threshold) ? 0u : 1u;   // :1576
        if (udf) udf[i] = val;
    }
}

}  // namespace

void sample_tet_labels(const BrickGridDesc& grid, const double* d_vertices, uint64_t nv,
                       const int32_t* d_tets, uint64_t nt, const double* bmin, const double* bmax,
                       double padding, double threshold, uint8_t* d_labels, float* d_udf,
                       cudaStream_t s, uint64_t* launches)
{
    const double sx = bmax[0] - bmin[0], sy = bmax[1] - bmin[1], sz = bmax[2] - bmin[2];
    if (!(sx > 0 && sy > 0 && sz > 0))   // :1546-1547
        throw Error{GPUPR_ERR_INVALID_ARGUMENT, "SparseUDF.sample_tet_labels: degenerate bbox"};
    if (!nt) return;
    GridView g;
    g.inv_h = 1.0 / grid.voxel_size;
    for (int k = 0; k < 3; ++k) {
        g.origin[k] = grid.origin[k];
        g.dims[k] = grid.dims[k];
    }
    g.background = grid.background;
    g.finite_bg = std::isfinite(grid.background);
    g.table = grid.d_table;
    g.values = grid.d_values;
    DevBuf<int> err(1, s);
    GPUPR_CUDA(cudaMemsetAsync(err.p, 0, sizeof(int), s));
    const unsigned blocks = (unsigned)std::min<uint64_t>((nt + LTPB - 1) / LTPB, (uint64_t)sm_count() * 16u);
    // 32-bit coordinates while every voxel of the grid and a few bricks around
    // it has them and the table has fewer than 2^30 cells
    const double cells = ((double)g.dims[0] + 4) * ((double)g.dims[1] + 4) * ((double)g.dims[2] + 4);
    bool small = cells < 1073741824.0;
    for (int k = 0; k < 3; ++k)
        small = small && (double)g.origin[k] > -2147480000.0 &&
                (double)g.origin[k] + 8.0 * (double)g.dims[k] < 2147480000.0;
    const uint32_t nv32 = (uint32_t)std::min<uint64_t>(nv, 1ull << 31);   // ids are int32
    auto kernel = small ? k_sample_labels<int> : k_sample_labels<long long>;
    kernel<<<blocks, LTPB, 0, s>>>(g, d_vertices, nv32, reinterpret_cast<const int4*>(d_tets), nt,
                                   make_double3(bmin[0], bmin[1], bmin[2]), make_double3(sx, sy, sz),
                                   1.0 - 2.0 * padding, padding, threshold, d_labels, d_udf, err.p);
    GPUPR_CUDA(cudaGetLastError());
    if (launches) *launches += 1;
    int he = 0;
    GPUPR_CUDA(cudaMemcpyAsync(&he, err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    GPUPR_CUDA(cudaStreamSynchronize(s));
    if (he) throw Error{GPUPR_ERR_INVALID_ARGUMENT, "SparseUDF.sample_tet_labels: tet index out of range"};
}

}  // namespace gpupr
