// Conservative fields on the GPU: boundary rasterisation, component labelling,
// witness fill, clearance dilation, the analytic box container, and the
// blocked-field stamp/unstamp with occupancy extraction.
//
// Reference (engine/pack_geometry/src): rasterize_boundary + run_raster_cursor
// (validation_kernel.cpp:3248-3340, 3668-3762) tag a cell 2 when the closed
// cell's interval box and a triangle's vertex intervals are not SAT-disjoint;
// fill_components (conservative_fields.cpp:257-360) gives every 6-connected
// component of non-2 cells the decision of its first cell in scan order
// (0 void, 1 material, 3 uncertain); dilate_and_crop (:436-504) marks every
// requested cell reached by a seed through the clearance stencil;
// BlockedField::add/remove/blocked (:1666-1886) keep per-cell copy counts and
// report mask || count.  The rasterised tags are an OR over faces, so one warp
// per face with benign same-value writes reproduces them exactly; component
// roots are the minimum linear index (= first in scan order) by union-find.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <optional>
#include <thread>
#include <vector>

#include "context.hpp"
#include "fields.hpp"
#include "host_chunks.hpp"
#include "interval.cuh"

namespace spk {

namespace {

int blocks_for(long long n, int threads)
{
    const long long want = (n + threads - 1) / threads;
    return static_cast<int>(std::min<long long>(std::max<long long>(want, 1), 148LL * 32));
}

// ---- vertex intervals ---------------------------------------------------------

// The vertex intervals of posed meshes (place(), validation_kernel.cpp:
// 805-943) on the device, for rotations that are not cardinal: each
// coordinate is transformed_interval_at, the code the host runs.
struct PoseIntervals {
    Interval rotation[3][3];
    double translation[3];
};

// Per pose: the vertices' bounds as maxima, -lowest low and highest high per
// axis, then the same at translation zero (oriented_bounds,
// physical_bounds.cpp:347), and whether an interval was not valid.
struct PoseBounds {
    double most[12];
    int invalid, oriented_invalid;
    double lo(int a) const { return -most[a]; }
    double hi(int a) const { return most[3 + a]; }
    double oriented_hi(int a) const { return most[9 + a]; }
};

constexpr int kVertexThreads = 128;
constexpr int kVertexBlocks = 64;  // per pose at most

// blockIdx.y: the pose (poses, or the single one).  Each block covers a
// stretch of the vertices; the pose's last block to finish combines the
// blocks' bounds, a lane per value.  `done` holds a zero per pose.
__global__ void __launch_bounds__(kVertexThreads) vertex_intervals_kernel(
    const double* __restrict__ vertices, int count, const PoseIntervals single,
    const PoseIntervals* __restrict__ poses, int oriented, IVec3* __restrict__ vint, PoseBounds* partial,
    unsigned int* done, PoseBounds* __restrict__ out)
{
    __shared__ double warp_most[kVertexThreads / 32][12];
    __shared__ PoseIntervals pose;
    __shared__ int invalid, oriented_invalid;
    const int item = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int values = oriented ? 12 : 6;
    if (threadIdx.x == 0) {
        pose = poses ? poses[item] : single;
        invalid = oriented_invalid = 0;
    }
    __syncthreads();
    const double zero[3] = { 0.0, 0.0, 0.0 };
    double most[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        most[k] = -INFINITY;
    }
    for (int i = blockIdx.x * kVertexThreads + threadIdx.x; i < count; i += gridDim.x * kVertexThreads) {
        const double point[3] = { vertices[3 * i], vertices[3 * i + 1], vertices[3 * i + 2] };
        IVec3 v;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            v.v[a] = transformed_interval_at(point, pose.translation, pose.rotation, a);
            if (!v.v[a].valid) {
                invalid = 1;
            }
            most[a] = f_max(most[a], -v.v[a].low);
            most[3 + a] = f_max(most[3 + a], v.v[a].high);
            if (oriented) {
                const Interval o = transformed_interval_at(point, zero, pose.rotation, a);
                if (!o.valid) {
                    oriented_invalid = 1;
                }
                most[6 + a] = f_max(most[6 + a], -o.low);
                most[9 + a] = f_max(most[9 + a], o.high);
            }
        }
        vint[static_cast<long long>(item) * count + i] = v;
    }
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        if (k < values) {
            for (int o = 16; o > 0; o >>= 1) {
                most[k] = f_max(most[k], __shfl_xor_sync(0xffffffffu, most[k], o));
            }
            if (lane == 0) {
                warp_most[warp][k] = most[k];
            }
        }
    }
    __syncthreads();
    if (warp != 0) {
        return;
    }
    PoseBounds* mine = partial + item * gridDim.x + blockIdx.x;
    if (lane < values) {
        double m = warp_most[0][lane];
        for (int k = 1; k < kVertexThreads / 32; ++k) {
            m = f_max(m, warp_most[k][lane]);
        }
        mine->most[lane] = m;
    }
    if (lane == 0) {
        mine->invalid = invalid;
        mine->oriented_invalid = oriented_invalid;
    }
    __threadfence();
    __syncwarp();
    unsigned int before = 0;
    if (lane == 0) {
        before = atomicAdd(&done[item], 1u);
    }
    if (__shfl_sync(0xffffffffu, before, 0) != gridDim.x - 1) {
        return;
    }
    __threadfence();
    const PoseBounds* all = partial + item * gridDim.x;
    double m = -INFINITY;
    int bad = 0;
    if (lane < values) {
#pragma unroll 8
        for (unsigned int k = 0; k < gridDim.x; ++k) {
            m = f_max(m, __ldcg(&all[k].most[lane]));
        }
    }
    else if (lane >= 30) {
#pragma unroll 8
        for (unsigned int k = 0; k < gridDim.x; ++k) {
            bad |= lane == 30 ? __ldcg(&all[k].invalid) : __ldcg(&all[k].oriented_invalid);
        }
    }
    if (lane < values) {
        out[item].most[lane] = m;
    }
    else if (lane == 30) {
        out[item].invalid = bad;
    }
    else if (lane == 31) {
        out[item].oriented_invalid = bad;
    }
}

// ---- boundary raster -----------------------------------------------------------

// One posed mesh of a raster batch: its window and where its cells start.
// Its vertex intervals follow the batch's order.
struct RasterItem {
    FieldWindow w;
    long long cells_at;
};

// Per-face candidate cell range: face_ranges (validation_kernel.cpp:3248-3340
// cursor bounds) with the host's binary64 path, floor((v - origin) / pitch)
// when the quotient lies farther than |q| 2^-48 + 2^-60 from every integer.
// Nearer to an integer n the host takes the floor of a long double quotient,
// which is n - 1 or n; here the range takes n - 1 for its low end and n for
// its high end instead.  The range is then at most one cell wider than the
// host's, and a cell it adds lies outside the face's padded interval bounds,
// where the SAT's first three axes separate it: the raster is the same.
// Quotients of magnitude 2^50 or more, or not finite, return false (the host
// path then runs).
__device__ __forceinline__ bool range_end(double bound, double origin, double pitch, bool low, long long& out)
{
    const double q = f_div(f_sub(bound, origin), pitch);
    if (!(fabs(q) < 0x1p50)) {
        out = 0;
        return false;
    }
    const double fl = floor(q);
    const double margin = f_add(f_mul(fabs(q), 0x1p-48), 0x1p-60);
    if (f_sub(q, fl) > margin && f_sub(f_add(fl, 1.0), q) > margin) {
        out = static_cast<long long>(fl);
    }
    else {
        const long long n = static_cast<long long>(rint(q));
        out = low ? n - 1 : n;
    }
    return true;
}

constexpr int kRasterWarps = 4;
constexpr int kRasterFaces = 16;  // per block at most

// A face's interval data, an axis per lane, and the interval test of one cell
// against it.  Kept out of line: their registers would halve the filter's
// occupancy.
__device__ __noinline__ void face_interval_data(const IVec3* a, const IVec3* b, const IVec3* c, int lane, FaceSat& sat)
{
    const IVec3 tri[3] = { *a, *b, *c };
    if (lane < 10) {
        face_sat_axis(tri, lane, sat);
    }
    else if (lane == 10) {
        face_sat_bounds(tri, sat);
    }
}
__device__ __noinline__ bool interval_cell_meets(const FaceSat& sat, const FieldWindow& w, long long x, long long y,
                                                 long long z, int* error)
{
    const std::int64_t index[3] = { x, y, z };
    IVec3 box;
    if (!grid_cell_interval(w.origin, w.pitch, index, box)) {
        atomicOr(error, 1);
        return false;
    }
    return !face_sat_disjoint(sat, box);
}

// The clipped cells of a face.
struct FaceCells {
    long long first[3];
    unsigned int extent[3];
    unsigned int total;  // 0: none
};

// `per_block` faces per block (and a split of their cells per blockIdx.y).  A
// thread per face works out its cells and its plain binary64 filter
// (FaceFilter); then a warp per face tests the cells, one per lane.  Only where
// a cell stays uncertain does the warp compute the face's interval data (FaceSat)
// and run the interval test, so the fields are those of the interval test on
// every cell.  The interval test on every cell of every face's range was bound
// by issue: 138 us for 8,192 faces; with the filter worked out by every lane of
// a face's warp 31 us, by one thread per face 18 us (5,120 faces of more cells
// 22 and 19 us, 12 faces whose every cell stays uncertain 42 and 15 us, most of
// that by the branch-free interval operations).
__global__ void __launch_bounds__(32 * kRasterWarps, 6) raster_kernel(
    const RasterItem single, const RasterItem* __restrict__ items, const std::uint32_t* __restrict__ tris,
    const IVec3* __restrict__ vint, int vertex_count, int faces, int per_block,
    const geo::FaceRange* __restrict__ given, std::uint8_t* __restrict__ all_cells, int* __restrict__ error)
{
    __shared__ FaceSat sats[kRasterWarps];
    __shared__ FaceFilter filters[kRasterFaces];  // read by broadcast
    __shared__ FaceCells ranges[kRasterFaces];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int face0 = blockIdx.x * per_block, here = min(per_block, faces - face0);
    const int at = blockIdx.z;
    const FieldWindow& w = items ? items[at].w : single.w;
    std::uint8_t* cells = all_cells + (items ? items[at].cells_at : single.cells_at);
    const IVec3* points = vint + static_cast<long long>(at) * vertex_count;
    if (static_cast<int>(threadIdx.x) < here) {
        const int face = face0 + threadIdx.x;
        IVec3 tri[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            tri[k] = points[tris[3 * face + k]];
        }
        double reach = 0.0;
        FaceCells r;
        bool fine = true, outside = given && given[face].outside;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double lo = f_min(f_min(tri[0].v[a].low, tri[1].v[a].low), tri[2].v[a].low);
            const double hi = f_max(f_max(tri[0].v[a].high, tri[1].v[a].high), tri[2].v[a].high);
            reach = f_max(reach, fabs(w.origin[a]));
            long long from, to;
            if (given) {
                from = given[face].first[a];
                to = given[face].last[a];
            }
            else {
                fine = range_end(lo, w.origin[a], w.pitch, true, from) && fine;
                fine = range_end(hi, w.origin[a], w.pitch, false, to) && fine;
                --from;
                ++to;
            }
            from = max(from, w.first[a]);
            to = min(to, w.first[a] + static_cast<long long>(w.shape[a] - 1));
            outside = outside || to < from;
            r.first[a] = from;
            r.extent[a] = static_cast<unsigned int>(to - from + 1);
        }
        if (!fine) {
            atomicOr(error, 4);
        }
        r.total = fine && !outside ? r.extent[0] * r.extent[1] * r.extent[2] : 0u;  // within the window: below 2^31
        ranges[threadIdx.x] = r;
        FaceFilter mine;
        face_filter(tri, reach + 8.0 * w.pitch, mine);
        filters[threadIdx.x] = mine;
    }
    __syncthreads();
    for (int f = warp; f < here; f += kRasterWarps) {
        const FaceCells& r = ranges[f];
        const FaceFilter& filter = filters[f];
        const long long base = (r.first[0] - w.first[0]) +
                               static_cast<long long>(w.shape[0]) *
                                   ((r.first[1] - w.first[1]) +
                                    static_cast<long long>(w.shape[1]) * (r.first[2] - w.first[2]));
        bool sat_ready = false;
        __syncwarp();  // the previous face's interval data is read
        for (unsigned int c0 = blockIdx.y * 32; c0 < r.total; c0 += gridDim.y * 32) {
            const unsigned int c = c0 + lane;
            const unsigned int row = c / r.extent[0], x = c - row * r.extent[0];
            const unsigned int z = row / r.extent[1], y = row - z * r.extent[1];
            const long long flat =
                base + x + static_cast<long long>(w.shape[0]) * (y + static_cast<long long>(w.shape[1]) * z);
            FaceCell cell = FaceCell::disjoint;
            if (c < r.total && cells[flat] != 2) {
                const double h = 0.5 * w.pitch;
                const double centre[3] = { w.origin[0] + w.pitch * (static_cast<double>(r.first[0] + x) + 0.5),
                                           w.origin[1] + w.pitch * (static_cast<double>(r.first[1] + y) + 0.5),
                                           w.origin[2] + w.pitch * (static_cast<double>(r.first[2] + z) + 0.5) };
                cell = given ? FaceCell::uncertain : face_filter_cell(filter, centre, h);
            }
            if (__any_sync(0xffffffffu, cell == FaceCell::uncertain)) {
                if (!sat_ready) {
                    const std::uint32_t* t = tris + 3 * (face0 + f);
                    face_interval_data(points + t[0], points + t[1], points + t[2], lane, sats[warp]);
                    sat_ready = true;
                    __syncwarp();
                }
                if (cell == FaceCell::uncertain &&
                    interval_cell_meets(sats[warp], w, r.first[0] + x, r.first[1] + y, r.first[2] + z, error)) {
                    cell = FaceCell::meets;
                }
            }
            if (cell == FaceCell::meets) {
                cells[flat] = 2;
            }
        }
    }
}

// ---- components -----------------------------------------------------------------

__device__ int find_root(const int* __restrict__ parent, int i)
{
    for (int guard = 0; guard < (1 << 26); ++guard) {
        const int p = parent[i];
        if (p == i) {
            return i;
        }
        i = p;
    }
    return i;
}

// Labels start as the first cell of each run of non-boundary cells along x
// (-1 at boundary cells): one warp per row.  A component's root is its lowest
// cell, and a run's lowest cell is its first, so runs join as wholes.
// blockIdx.y: the item; labels are cell numbers within it.
__global__ void __launch_bounds__(256) ccl_runs_kernel(const RasterItem single, const RasterItem* __restrict__ items,
                                                       const std::uint8_t* __restrict__ all_cells,
                                                       int* __restrict__ all_parents)
{
    const RasterItem& it = items ? items[blockIdx.y] : single;
    const std::uint8_t* cells = all_cells + it.cells_at;
    int* parent = all_parents + it.cells_at;
    const int lane = threadIdx.x & 31, sx = it.w.shape[0];
    const long long rows = static_cast<long long>(it.w.shape[1]) * it.w.shape[2];
    for (long long row = blockIdx.x * 8LL + (threadIdx.x >> 5); row < rows; row += gridDim.x * 8LL) {
        const int base = static_cast<int>(row * sx);
        int start = 0;  // first cell of the run that reaches into this stretch
        for (int x0 = 0; x0 < sx; x0 += 32) {
            const int x = x0 + lane;
            const bool wall = x < sx && cells[base + x] == 2;
            const unsigned walls = __ballot_sync(0xffffffffu, wall);
            if (x < sx) {
                const unsigned before = walls & ((1u << lane) - 1u);
                const int run = before ? x0 + 32 - __clz(before) : start;
                parent[base + x] = wall ? -1 : base + run;
            }
            start = walls ? x0 + 32 - __clz(walls) : start;
        }
    }
}

__device__ void unite(int* parent, int a, int b, int* error)
{
    for (int guard = 0; guard < (1 << 24); ++guard) {
        a = find_root(parent, a);
        b = find_root(parent, b);
        if (a == b) {
            return;
        }
        if (a < b) {
            const int t = a;
            a = b;
            b = t;
        }
        const int old = atomicMin(&parent[a], b);
        if (old == a) {
            return;
        }
        a = old;
    }
    atomicOr(error, 2);  // bounded retries exhausted: reported, never spun forever
}

// Joins runs that touch along y and z, once per pair of overlapping runs: at
// the first cell of the overlap.
__global__ void ccl_union_kernel(const RasterItem single, const RasterItem* __restrict__ items,
                                 const std::uint8_t* __restrict__ all_cells, int* __restrict__ all_parents,
                                 int* __restrict__ error)
{
    const RasterItem& it = items ? items[blockIdx.y] : single;
    const std::uint8_t* cells = all_cells + it.cells_at;
    int* parent = all_parents + it.cells_at;
    const int sx = it.w.shape[0], sy = it.w.shape[1], sz = it.w.shape[2];
    const int n = sx * sy * sz, plane = sx * sy;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (cells[i] == 2) {
            continue;
        }
        const int x = i % sx, r = i / sx, y = r % sy;
        const bool begins = x == 0 || cells[i - 1] == 2;
        if (y > 0 && cells[i - sx] != 2 && (begins || cells[i - sx - 1] == 2)) {
            unite(parent, i, i - sx, error);
        }
        if (i >= plane && cells[i - plane] != 2 && (begins || cells[i - plane - 1] == 2)) {
            unite(parent, i, i - plane, error);
        }
    }
}

// Every cell's label becomes its root; roots are listed as cell numbers of the
// whole batch.
__global__ void ccl_compress_kernel(const RasterItem single, const RasterItem* __restrict__ items,
                                    int* __restrict__ all_parents, int* __restrict__ roots,
                                    unsigned int* __restrict__ root_count, unsigned int root_capacity)
{
    const RasterItem& it = items ? items[blockIdx.y] : single;
    int* parent = all_parents + it.cells_at;
    const int n = it.w.shape[0] * it.w.shape[1] * it.w.shape[2];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (parent[i] < 0) {
            continue;
        }
        const int root = find_root(parent, i);
        parent[i] = root;
        if (root == i) {
            const unsigned int slot = atomicAdd(root_count, 1u);
            if (slot < root_capacity) {
                roots[slot] = static_cast<int>(it.cells_at + root);
            }
        }
    }
}

__global__ void scatter_decisions_kernel(const int* __restrict__ roots, const std::uint8_t* __restrict__ values,
                                         int count, std::uint8_t* __restrict__ root_value)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) {
        root_value[roots[i]] = values[i];
    }
}

// The decisions of a batch's few roots, passed by value.
constexpr int kFewRoots = 32;
struct FewRoots {
    int root[kFewRoots];
    std::uint8_t value[kFewRoots];
    int count;  // -1: the decisions are in root_value, by root cell
};

__global__ void fill_kernel(const RasterItem single, const RasterItem* __restrict__ items,
                            std::uint8_t* __restrict__ all_cells, const int* __restrict__ all_parents,
                            const std::uint8_t* __restrict__ root_value, const FewRoots few, int normalize)
{
    const RasterItem& it = items ? items[blockIdx.y] : single;
    std::uint8_t* cells = all_cells + it.cells_at;
    const int* parent = all_parents + it.cells_at;
    const int n = it.w.shape[0] * it.w.shape[1] * it.w.shape[2];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        std::uint8_t v = cells[i];
        if (v != 2) {
            const int root = static_cast<int>(it.cells_at + parent[i]);
            if (few.count < 0) {
                v = root_value[root];
            }
            else {
                for (int k = 0; k < few.count; ++k) {
                    v = few.root[k] == root ? few.value[k] : v;
                }
            }
        }
        cells[i] = normalize ? (v != 0 ? 1 : 0) : v;
    }
}

// A sub-box [lo, lo + extent) of a window (cell offsets from its first
// cell); the box kernels visit its cells only.
struct CellBox {
    int lo[3];
    int extent[3];
};

__device__ __forceinline__ long long box_cells(const CellBox& b)
{
    return static_cast<long long>(b.extent[0]) * b.extent[1] * b.extent[2];
}

// Offset (x, y, z) from the window's first cell of the box's cell i.
__device__ __forceinline__ void box_cell(const CellBox& b, long long i, int (&c)[3])
{
    c[0] = b.lo[0] + static_cast<int>(i % b.extent[0]);
    c[1] = b.lo[1] + static_cast<int>((i / b.extent[0]) % b.extent[1]);
    c[2] = b.lo[2] + static_cast<int>(i / (static_cast<long long>(b.extent[0]) * b.extent[1]));
}

// The offsets of a small stencil, passed by value: a copy to the device would
// cost more than the dilation.
constexpr int kFewOffsets = 343;  // 7^3: clearances of up to three cells
struct FewOffsets {
    signed char at[kFewOffsets][3];
};

// out[t] over `req` = OR over stencil deltas d of seed(raw[t - d]) inside `raw`;
// with counts, the cells are added to them as well.
__global__ void dilate_kernel(const std::uint8_t* __restrict__ raw, FieldWindow rw,
                              const __grid_constant__ FewOffsets few, const int* __restrict__ stencil,
                              int stencil_count, int invert, std::uint8_t* __restrict__ out, FieldWindow req,
                              CellBox box, const StampCounts stamp)
{
    const long long n = box_cells(box);
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        int c[3];
        box_cell(box, i, c);
        const long long t[3] = { req.first[0] + c[0], req.first[1] + c[1], req.first[2] + c[2] };
        const long long at = c[0] + static_cast<long long>(req.shape[0]) * (c[1] + static_cast<long long>(req.shape[1]) * c[2]);
        std::uint8_t value = 0;
        for (int s = 0; s < stencil_count && !value; ++s) {
            const long long sx = t[0] - (stencil ? stencil[3 * s] : few.at[s][0]) - rw.first[0];
            const long long sy = t[1] - (stencil ? stencil[3 * s + 1] : few.at[s][1]) - rw.first[1];
            const long long sz = t[2] - (stencil ? stencil[3 * s + 2] : few.at[s][2]) - rw.first[2];
            if (sx < 0 || sy < 0 || sz < 0 || sx >= rw.shape[0] || sy >= rw.shape[1] || sz >= rw.shape[2]) {
                continue;
            }
            const std::uint8_t v = raw[sx + rw.shape[0] * (sy + static_cast<long long>(rw.shape[1]) * sz)];
            value = invert ? (v != 1) : (v != 0);
        }
        out[at] = value;
        if (stamp.counts && value) {
            stamp.counts[at] += stamp.direction > 0 ? 1u : static_cast<std::uint32_t>(-1);
        }
    }
}

__global__ void box_mask_kernel(const std::uint8_t* __restrict__ ax, const std::uint8_t* __restrict__ ay,
                                const std::uint8_t* __restrict__ az, int sx, int sy, int sz,
                                std::uint8_t* __restrict__ mask)
{
    const long long n = static_cast<long long>(sx) * sy * sz;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int x = static_cast<int>(i % sx);
        const long long r = i / sx;
        const int y = static_cast<int>(r % sy);
        const int z = static_cast<int>(r / sy);
        mask[i] = (ax[x] && ay[y] && az[z]) ? 0 : 1;
    }
}

__global__ void occupancy_box_kernel(const std::uint8_t* __restrict__ mask, const std::uint32_t* __restrict__ counts,
                                     std::uint8_t* __restrict__ occ, int sx, int sy, CellBox box)
{
    const long long n = box_cells(box);
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        int c[3];
        box_cell(box, i, c);
        const long long at = c[0] + static_cast<long long>(sx) * (c[1] + static_cast<long long>(sy) * c[2]);
        occ[at] = (mask[at] != 0 || counts[at] != 0) ? 1 : 0;
    }
}

__global__ void occupancy_kernel(const std::uint8_t* __restrict__ mask, const std::uint32_t* __restrict__ counts,
                                 std::uint8_t* __restrict__ occ, long long n)
{
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        occ[i] = (mask[i] != 0 || counts[i] != 0) ? 1 : 0;
    }
}

}  // namespace

namespace {

// Everything a raster batch needs: posed meshes (vertex intervals in d_vint,
// [item][vertex]), their windows, and where each item's cells start.
struct RasterBatch {
    const geo::Mesh* mesh;
    const geo::Placed* placed;
    const FieldWindow* windows;
    int count;
    const long long* cells_at;  // count + 1 entries
    const std::uint32_t* d_tris;
    const IVec3* d_vint;
};

// Raster, components, witnesses and fill of a batch into d_cells.  host_ranges
// (one item): the faces' cell ranges come from the host.
int raster_batch(spk_context* ctx, const RasterBatch& b, std::uint8_t* d_cells, bool normalize, bool host_ranges)
{
    cudaStream_t st = ctx->stream;
    const long long total = b.cells_at[b.count];
    if (total >= (1LL << 31)) {
        return kCellLimit;
    }
    const int F = static_cast<int>(b.mesh->triangles.size()), V = static_cast<int>(b.mesh->vertices.size());
    int status = kOk;
    const auto root_capacity = static_cast<unsigned int>(ctx->cap_bytes ? std::min(total, 1LL << 20) : 1LL << 20);
    constexpr unsigned int kEarlyRoots = 240;  // read back with the flags
    auto* d_parent = static_cast<int*>(device_buffer(ctx, "field.parent", total * sizeof(int), status));
    // [0] errors, [1] roots found, from [16] on the roots.
    auto* d_misc = static_cast<int*>(device_buffer(
        ctx, "field.misc", (16 + std::max(root_capacity, kEarlyRoots)) * 4ULL, status));
    auto* h_misc = static_cast<int*>(host_buffer(ctx, "field.misc", (16 + kEarlyRoots) * 4ULL, status));
    RasterItem single {};
    RasterItem* d_items = nullptr;
    if (!d_parent || !d_misc || !h_misc) {
        return status;
    }
    long long largest = 1, rows = 1;
    if (b.count == 1) {
        single = { b.windows[0], b.cells_at[0] };
    }
    else {
        auto* h_items =
            static_cast<RasterItem*>(host_buffer(ctx, "field.items", b.count * sizeof(RasterItem), status));
        d_items = static_cast<RasterItem*>(device_buffer(ctx, "field.items", b.count * sizeof(RasterItem), status));
        if (!h_items || !d_items) {
            return status;
        }
        for (int i = 0; i < b.count; ++i) {
            h_items[i] = { b.windows[i], b.cells_at[i] };
        }
        cudaMemcpyAsync(d_items, h_items, b.count * sizeof(RasterItem), cudaMemcpyHostToDevice, st);
    }
    for (int i = 0; i < b.count; ++i) {
        const auto& w = b.windows[i];
        largest = std::max(largest, static_cast<long long>(w.shape[0]) * w.shape[1] * w.shape[2]);
        rows = std::max(rows, static_cast<long long>(w.shape[1]) * w.shape[2]);
    }
    cudaMemsetAsync(d_cells, 0, total, st);
    cudaMemsetAsync(d_misc, 0, 64, st);
    const geo::FaceRange* d_ranges = nullptr;
    if (F > 0 && host_ranges) {
        // The host reads the vertex intervals back and takes the floors of
        // long double quotients.
        geo::Window gw;
        for (int a = 0; a < 3; ++a) {
            gw.first[a] = b.windows[0].first[a];
            gw.shape[a] = b.windows[0].shape[a];
        }
        geo::Placed source = b.placed[0];
        source.intervals.resize(V);
        if (cudaMemcpyAsync(source.intervals.data(), b.d_vint, V * sizeof(IVec3), cudaMemcpyDeviceToHost, st) !=
                cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            cudaGetLastError();
            return kCuda;
        }
        std::vector<geo::FaceRange> ranges;
        if (!geo::face_ranges(source, gw, b.windows[0].origin, b.windows[0].pitch, ranges)) {
            return kFieldIndexOverflow;
        }
        auto* d = static_cast<geo::FaceRange*>(device_buffer(ctx, "field.ranges", F * sizeof(geo::FaceRange), status));
        if (!d) {
            return status;
        }
        cudaMemcpyAsync(d, ranges.data(), F * sizeof(geo::FaceRange), cudaMemcpyHostToDevice, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) {  // the host vector ends with this scope
            cudaGetLastError();
            return kCuda;
        }
        d_ranges = d;
    }
    const auto items = static_cast<unsigned>(b.count);
    if (F > 0) {
        // Few faces: their cells are split over several warps each.
        const int splits = static_cast<int>(std::min<long long>(64, std::max<long long>(1, 4736LL / F / b.count)));
        // Blocks of 16 faces, of fewer where that leaves SMs without three; a
        // warp per face where faces are few and their cells many.
        int per_block = splits > 1 ? kRasterWarps : kRasterFaces;
        while (per_block > kRasterWarps &&
               static_cast<long long>((F + per_block - 1) / per_block) * splits * b.count < 3 * 148) {
            per_block /= 2;
        }
        raster_kernel<<<dim3((F + per_block - 1) / per_block, splits, items), 32 * kRasterWarps, 0, st>>>(
            single, d_items, b.d_tris, b.d_vint, V, F, per_block, d_ranges, d_cells, d_misc);
        ctx->launches++;
    }
    const int threads = 256;
    const auto share = [&](long long n) {  // blocks per item
        return static_cast<unsigned>(std::max<long long>(1, std::min<long long>(n, 148LL * 32 / b.count)));
    };
    const dim3 by_row(share((rows + 7) / 8), items), by_cell(share((largest + threads - 1) / threads), items);
    ccl_runs_kernel<<<by_row, 256, 0, st>>>(single, d_items, d_cells, d_parent);
    ccl_union_kernel<<<by_cell, threads, 0, st>>>(single, d_items, d_cells, d_parent, d_misc);
    ccl_compress_kernel<<<by_cell, threads, 0, st>>>(single, d_items, d_parent, d_misc + 16,
                                                     reinterpret_cast<unsigned int*>(d_misc + 1), root_capacity);
    ctx->launches += 3;
    cudaMemcpyAsync(h_misc, d_misc, (16 + kEarlyRoots) * 4ULL, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return kCuda;
    }
    if (h_misc[0] & 4) {
        // A quotient the device's binary64 path does not cover: the host's
        // face ranges decide, item by item.
        for (int i = 0; i < b.count; ++i) {
            const long long cells_at[2] = { 0, b.cells_at[i + 1] - b.cells_at[i] };
            const RasterBatch one { b.mesh,   b.placed + i, b.windows + i, 1, cells_at,
                                    b.d_tris, b.d_vint + static_cast<long long>(i) * V };
            if ((status = raster_batch(ctx, one, d_cells + b.cells_at[i], normalize, true))) {
                return status;
            }
        }
        return kOk;
    }
    if (h_misc[0] & 1) {
        return kFieldIndexOverflow;
    }
    if (h_misc[0] & 2) {
        return kKernelWait;
    }
    const auto roots = static_cast<unsigned int>(h_misc[1]);
    if (roots > root_capacity) {
        return kCellLimit;
    }
    std::vector<int> h_roots(h_misc + 16, h_misc + 16 + std::min(roots, kEarlyRoots));
    if (roots > kEarlyRoots) {
        h_roots.resize(roots);
        cudaMemcpyAsync(h_roots.data(), d_misc + 16, roots * 4ULL, cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) {
            cudaGetLastError();
            return kCuda;
        }
    }
    std::vector<std::uint8_t> values(roots);
    std::atomic<bool> overflow { false };
    const std::size_t parts = roots < 16 ? 1 : std::min<std::size_t>(8, std::max(1U, std::thread::hardware_concurrency()));
    run_chunks(roots, parts, [&](std::size_t, std::size_t begin, std::size_t end) {
        for (std::size_t k = begin; k < end; ++k) {
            const int item =
                static_cast<int>(std::upper_bound(b.cells_at, b.cells_at + b.count, h_roots[k]) - b.cells_at) - 1;
            const FieldWindow& w = b.windows[item];
            const long long i = h_roots[k] - b.cells_at[item];
            const std::int64_t index[3] = { w.first[0] + i % w.shape[0], w.first[1] + (i / w.shape[0]) % w.shape[1],
                                             w.first[2] + i / (static_cast<long long>(w.shape[0]) * w.shape[1]) };
            geo::Bounds witness;
            if (!geo::outward_grid_cell(w.origin, w.pitch, index, witness)) {
                overflow = true;
                return;
            }
            const auto decision = geo::classify_material_witness(b.placed[item], witness);
            values[k] = decision == geo::Decision::indeterminate ? 3 : decision == geo::Decision::yes ? 1 : 0;
        }
    });
    if (overflow) {
        return kFieldIndexOverflow;
    }
    FewRoots few {};
    std::uint8_t* d_rootv = nullptr;
    few.count = roots <= static_cast<unsigned>(kFewRoots) ? static_cast<int>(roots) : -1;
    for (int k = 0; k < few.count; ++k) {
        few.root[k] = h_roots[k];
        few.value[k] = values[k];
    }
    if (few.count < 0) {
        auto* h_values = static_cast<std::uint8_t*>(host_buffer(ctx, "field.values", roots, status));
        auto* d_values = static_cast<std::uint8_t*>(device_buffer(ctx, "field.values", roots, status));
        d_rootv = static_cast<std::uint8_t*>(device_buffer(ctx, "field.rootv", total, status));
        if (!h_values || !d_values || !d_rootv) {
            return status;
        }
        std::memcpy(h_values, values.data(), roots);
        cudaMemcpyAsync(d_values, h_values, roots, cudaMemcpyHostToDevice, st);
        scatter_decisions_kernel<<<(roots + 255) / 256, 256, 0, st>>>(d_misc + 16, d_values, static_cast<int>(roots),
                                                                      d_rootv);
        ctx->launches++;
    }
    fill_kernel<<<by_cell, threads, 0, st>>>(single, d_items, d_cells, d_parent, d_rootv, few, normalize ? 1 : 0);
    ctx->launches++;
    return cudaGetLastError() == cudaSuccess ? kOk : kCuda;
}

long long window_cells(const FieldWindow& w)
{
    return static_cast<long long>(w.shape[0]) * w.shape[1] * w.shape[2];
}

// The poses' vertex intervals (into d_vint, [pose][vertex]) and bounds on the
// device, for poses whose rotation is not cardinal; eligible[i] tells which.
// Waits for the bounds.
int device_intervals(spk_context* ctx, const geo::Mesh& mesh, const double* d_vertices, const geo::Vec3& translation,
                     const geo::Quat* q, int count, bool oriented, IVec3* d_vint, std::vector<PoseBounds>& bounds)
{
    cudaStream_t st = ctx->stream;
    const int V = static_cast<int>(mesh.vertices.size());
    const int blocks = std::max(1, std::min(kVertexBlocks, (V + kVertexThreads - 1) / kVertexThreads));
    int status = kOk;
    const std::size_t n = static_cast<std::size_t>(count);
    auto* d_bounds = static_cast<char*>(
        device_buffer(ctx, "field.pose_bounds", n * (blocks + 1) * sizeof(PoseBounds) + n * 4, status));
    auto* h_bounds = static_cast<PoseBounds*>(host_buffer(ctx, "field.pose_bounds", n * sizeof(PoseBounds), status));
    PoseIntervals single {};
    PoseIntervals* d_poses = nullptr;
    if (!d_bounds || !h_bounds) {
        return status;
    }
    const auto make = [&](const geo::Quat& quat, PoseIntervals& pose) {
        geo::rotation_intervals(quat, pose.rotation);
        for (int a = 0; a < 3; ++a) {
            pose.translation[a] = translation[a];
        }
    };
    if (count == 1) {
        make(q[0], single);
    }
    else {
        auto* h_poses = static_cast<PoseIntervals*>(host_buffer(ctx, "field.poses", n * sizeof(PoseIntervals), status));
        d_poses = static_cast<PoseIntervals*>(device_buffer(ctx, "field.poses", n * sizeof(PoseIntervals), status));
        if (!h_poses || !d_poses) {
            return status;
        }
        for (int i = 0; i < count; ++i) {
            make(q[i], h_poses[i]);
        }
        cudaMemcpyAsync(d_poses, h_poses, n * sizeof(PoseIntervals), cudaMemcpyHostToDevice, st);
    }
    auto* d_out = reinterpret_cast<PoseBounds*>(d_bounds);
    auto* d_done = reinterpret_cast<unsigned int*>(d_bounds + n * (blocks + 1) * sizeof(PoseBounds));
    cudaMemsetAsync(d_done, 0, n * 4, st);
    vertex_intervals_kernel<<<dim3(blocks, count), kVertexThreads, 0, st>>>(d_vertices, V, single, d_poses,
                                                                           oriented ? 1 : 0, d_vint, d_out + n, d_done,
                                                                           d_out);
    ctx->launches++;
    cudaMemcpyAsync(h_bounds, d_out, n * sizeof(PoseBounds), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return kCuda;
    }
    bounds.assign(h_bounds, h_bounds + n);
    return kOk;
}

// Whether the device computes a pose's intervals: the host's place() handles
// cardinal rotations and poses that are not finite.
bool device_pose(const geo::Vec3& translation, const geo::Quat& q, std::optional<geo::RotationTransform>& transform)
{
    if (!geo::finite_pose(translation, q)) {
        return false;
    }
    transform = geo::rotation_transform(q);
    return transform && !transform->exact_cardinal;
}

geo::Placed device_placed(const geo::Prepared& prepared, const geo::Vec3& translation, const geo::Quat& q,
                          const geo::RotationTransform& transform, const PoseBounds& b)
{
    geo::Placed out {};
    out.prepared = &prepared;
    out.translation = translation;
    out.q = q;
    out.is_cardinal = false;
    for (int a = 0; a < 3; ++a) {
        out.source_axis[a] = transform.source_axis[a];
        out.sign[a] = transform.sign[a];
        out.conservative.min[a] = b.lo(a);
        out.conservative.max[a] = b.hi(a);
    }
    out.finite = true;
    out.world_exact = false;
    return out;
}

}  // namespace

int raster_fill(spk_context* ctx, const geo::Placed& placed, const FieldWindow& w, std::uint8_t* d_cells, bool normalize,
                const std::uint32_t* d_tris_kept, bool device_intervals)
{
    const auto& mesh = *placed.prepared->mesh;
    const std::size_t F = mesh.triangles.size(), V = mesh.vertices.size();
    int status = kOk;
    auto* d_tris = d_tris_kept ? const_cast<std::uint32_t*>(d_tris_kept)
                               : static_cast<std::uint32_t*>(device_buffer(ctx, "field.tris", F * 12, status));
    auto* d_vint = static_cast<IVec3*>(device_buffer(ctx, "field.vint", V * sizeof(IVec3), status));
    if (!d_tris || !d_vint) {
        return status;
    }
    if (!d_tris_kept) {
        cudaMemcpyAsync(d_tris, mesh.triangles.data(), F * 12, cudaMemcpyHostToDevice, ctx->stream);
    }
    if (!device_intervals) {
        // The vertex intervals go through pinned memory (the previous call's
        // copy finished at its synchronisation).
        auto* h_vint = static_cast<IVec3*>(host_buffer(ctx, "field.vint", V * sizeof(IVec3), status));
        if (!h_vint) {
            return status;
        }
        std::memcpy(h_vint, placed.intervals.data(), V * sizeof(IVec3));
        cudaMemcpyAsync(d_vint, h_vint, V * sizeof(IVec3), cudaMemcpyHostToDevice, ctx->stream);
    }
    const long long cells_at[2] = { 0, window_cells(w) };
    return raster_batch(ctx, { &mesh, &placed, &w, 1, cells_at, d_tris, d_vint }, d_cells, normalize, false);
}

int place_on_device(spk_context* ctx, const geo::Prepared& prepared, const double* d_vertices,
                    const geo::Vec3& translation, const geo::Quat& q, geo::Placed& out, bool& done)
{
    done = false;
    std::optional<geo::RotationTransform> transform;
    const auto& mesh = *prepared.mesh;
    if (mesh.vertices.empty() || !device_pose(translation, q, transform)) {
        return kOk;  // the host's place() decides
    }
    int status = kOk;
    auto* d_vint = static_cast<IVec3*>(device_buffer(ctx, "field.vint", mesh.vertices.size() * sizeof(IVec3), status));
    if (!d_vint) {
        return status;
    }
    std::vector<PoseBounds> bounds;
    if ((status = device_intervals(ctx, mesh, d_vertices, translation, &q, 1, false, d_vint, bounds))) {
        return status;
    }
    if (bounds[0].invalid) {
        return kOk;  // the host's place() decides (it returns false)
    }
    out = device_placed(prepared, translation, q, *transform, bounds[0]);
    done = true;
    return kOk;
}

int object_fields(spk_context* ctx, const geo::Prepared& prepared, const std::uint32_t* d_tris,
                  const double* d_vertices, const double* origin, double pitch, const geo::Quat* q, int count,
                  ObjectFields& out)
{
    const auto& mesh = *prepared.mesh;
    const int V = static_cast<int>(mesh.vertices.size());
    const geo::Vec3 translation { origin[0], origin[1], origin[2] };
    cudaStream_t st = ctx->stream;
    int status = kOk;
    out.windows.clear();
    out.max_z.clear();
    out.cells_at.assign(1, 0);
    auto* d_vint = static_cast<IVec3*>(
        device_buffer(ctx, "field.vint", static_cast<std::size_t>(count) * V * sizeof(IVec3), status));
    if (!d_vint) {
        return status;
    }
    std::vector<PoseBounds> bounds;
    if ((status = device_intervals(ctx, mesh, d_vertices, translation, q, count, true, d_vint, bounds))) {
        return status;
    }
    std::vector<geo::Placed> placed;
    std::vector<FieldWindow> windows;
    std::vector<int> on_host;
    int taken = 0;
    for (; taken < count; ++taken) {
        const int i = taken;
        geo::Placed pose;
        geo::Window window;
        double max_z = 0;
        bool host = false;
        if (!geo::canonical_unit(q[i])) {
            return kFieldInput;
        }
        std::optional<geo::RotationTransform> transform;
        if (device_pose(translation, q[i], transform) && !bounds[i].invalid && !bounds[i].oriented_invalid) {
            pose = device_placed(prepared, translation, q[i], *transform, bounds[i]);
            max_z = bounds[i].oriented_hi(2);
        }
        else {
            geo::Bounds oriented;
            if (!geo::place(prepared, translation, q[i], pose) || !geo::oriented_bounds(mesh, q[i], oriented)) {
                return kFieldInput;
            }
            max_z = oriented.max[2];
            host = true;
        }
        if (!geo::object_window(pose, origin, pitch, window)) {
            return kFieldIndexOverflow;
        }
        const FieldWindow w = make_window(window, origin, pitch);
        const long long end = out.cells_at[i] + window_cells(w);
        if (i > 0 && end > kBatchCells) {
            break;
        }
        if (host) {
            on_host.push_back(i);
        }
        placed.push_back(std::move(pose));
        windows.push_back(w);
        out.windows.push_back(window);
        out.max_z.push_back(max_z);
        out.cells_at.push_back(end);
    }
    for (int i : on_host) {
        cudaMemcpyAsync(d_vint + static_cast<long long>(i) * V, placed[i].intervals.data(), V * sizeof(IVec3),
                        cudaMemcpyHostToDevice, st);
    }
    out.d_cells = static_cast<std::uint8_t*>(device_buffer(ctx, "obj.cells", out.cells_at[taken], status));
    if (!out.d_cells) {
        return status;
    }
    return raster_batch(ctx, { &mesh, placed.data(), windows.data(), taken, out.cells_at.data(), d_tris, d_vint },
                        out.d_cells, true, false);
}

int dilate_crop(spk_context* ctx, const std::uint8_t* d_raw, const FieldWindow& raw, std::uint64_t halo,
                double clearance, bool invert, std::uint8_t* d_out, const FieldWindow& req, const int* box_lo,
                const int* box_hi, const StampCounts& stamp)
{
    const auto stencil = geo::make_stencil(halo, req.pitch, clearance);
    int status = kOk;
    FewOffsets few {};
    int* d_stencil = nullptr;
    if (halo <= 127 && stencil.size() <= static_cast<std::size_t>(kFewOffsets)) {
        for (std::size_t i = 0; i < stencil.size(); ++i) {
            for (int a = 0; a < 3; ++a) {
                few.at[i][a] = static_cast<signed char>(stencil[i][a]);
            }
        }
    }
    else {
        std::vector<int> flat(3 * stencil.size());
        for (std::size_t i = 0; i < stencil.size(); ++i) {
            for (int a = 0; a < 3; ++a) {
                flat[3 * i + a] = static_cast<int>(stencil[i][a]);
            }
        }
        d_stencil = static_cast<int*>(device_buffer(ctx, "field.stencil", flat.size() * 4, status));
        if (!d_stencil) {
            return status;
        }
        cudaMemcpyAsync(d_stencil, flat.data(), flat.size() * 4, cudaMemcpyHostToDevice, ctx->stream);
    }
    const long long n = static_cast<long long>(req.shape[0]) * req.shape[1] * req.shape[2];
    CellBox box {};
    for (int a = 0; a < 3; ++a) {
        box.lo[a] = box_lo ? box_lo[a] : 0;
        box.extent[a] = (box_hi ? box_hi[a] : req.shape[a]) - box.lo[a];
        if (box.extent[a] <= 0) {
            box.extent[a] = 0;
        }
    }
    const long long m = static_cast<long long>(box.extent[0]) * box.extent[1] * box.extent[2];
    if (m < n && !stamp.counts) {
        cudaMemsetAsync(d_out, 0, n, ctx->stream);  // no stencil offset reaches the raw window from outside the box
    }
    if (m > 0) {
        dilate_kernel<<<blocks_for(m, 256), 256, 0, ctx->stream>>>(d_raw, raw, few, d_stencil,
                                                                   static_cast<int>(stencil.size()), invert ? 1 : 0,
                                                                   d_out, req, box, stamp);
        ctx->launches++;
    }
    return cudaGetLastError() == cudaSuccess ? kOk : kCuda;
}

int box_mask(spk_context* ctx, const double* dims, double clearance, const FieldWindow& w, std::uint8_t* d_mask)
{
    std::vector<std::uint8_t> axes[3];
    for (int a = 0; a < 3; ++a) {
        axes[a].resize(w.shape[a]);
        for (std::uint32_t k = 0; k < w.shape[a]; ++k) {
            std::int64_t index[3] = { w.first[0], w.first[1], w.first[2] };
            index[a] = w.first[a] + k;
            IVec3 cell;
            if (!grid_cell_interval(w.origin, w.pitch, index, cell)) {
                return kFieldIndexOverflow;
            }
            axes[a][k] = geo::analytic_box_axis_inside(w.origin[a], w.pitch, index[a], dims[a], clearance, cell, a) ? 1
                                                                                                                   : 0;
        }
    }
    int status = kOk;
    auto* d_axes = static_cast<std::uint8_t*>(
        device_buffer(ctx, "field.axes", static_cast<std::size_t>(w.shape[0]) + w.shape[1] + w.shape[2], status));
    if (!d_axes) {
        return status;
    }
    cudaMemcpyAsync(d_axes, axes[0].data(), w.shape[0], cudaMemcpyHostToDevice, ctx->stream);
    cudaMemcpyAsync(d_axes + w.shape[0], axes[1].data(), w.shape[1], cudaMemcpyHostToDevice, ctx->stream);
    cudaMemcpyAsync(d_axes + w.shape[0] + w.shape[1], axes[2].data(), w.shape[2], cudaMemcpyHostToDevice, ctx->stream);
    const long long n = static_cast<long long>(w.shape[0]) * w.shape[1] * w.shape[2];
    box_mask_kernel<<<blocks_for(n, 256), 256, 0, ctx->stream>>>(d_axes, d_axes + w.shape[0],
                                                                 d_axes + w.shape[0] + w.shape[1], w.shape[0],
                                                                 w.shape[1], w.shape[2], d_mask);
    ctx->launches++;
    return cudaGetLastError() == cudaSuccess ? kOk : kCuda;
}

int occupancy_box(spk_context* ctx, const std::uint8_t* d_mask, const std::uint32_t* d_counts, std::uint8_t* d_occ,
                  const int* shape, const int* lo, const int* hi)
{
    CellBox box {};
    for (int a = 0; a < 3; ++a) {
        box.lo[a] = lo[a];
        box.extent[a] = hi[a] > lo[a] ? hi[a] - lo[a] : 0;
    }
    const long long m = static_cast<long long>(box.extent[0]) * box.extent[1] * box.extent[2];
    if (m > 0) {
        occupancy_box_kernel<<<blocks_for(m, 256), 256, 0, ctx->stream>>>(d_mask, d_counts, d_occ, shape[0], shape[1],
                                                                          box);
        ctx->launches++;
    }
    return cudaGetLastError() == cudaSuccess ? kOk : kCuda;
}

int occupancy(spk_context* ctx, const std::uint8_t* d_mask, const std::uint32_t* d_counts, std::uint8_t* d_occ,
              long long n)
{
    occupancy_kernel<<<blocks_for(n, 256), 256, 0, ctx->stream>>>(d_mask, d_counts, d_occ, n);
    ctx->launches++;
    return cudaGetLastError() == cudaSuccess ? kOk : kCuda;
}

}  // namespace spk
