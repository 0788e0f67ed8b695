// Spectral page pipeline kernels and host orchestration (see pipeline.hpp).
//
// Per environment (once per layout): Z = B + iP (B the u8 occupancy, P the
// FP32 proximity), transformed along x and y plane by plane.
// Per oriented kernel (once per run): the kernel transformed along x and y,
// kept for its K2 non-empty z planes ("partial spectrum").
// Per page request, over z slabs of the environment (passes.hpp):
//   pass A  - per (kx, ky) column: the slab's environment column and the
//             kernel column transformed along z, multiplied, inverted;
//   pass B1 - inverse along y, legal rows kept;
//   pass B2 - inverse along x and the fused epilogue: real part = overlap
//             count, imaginary part = proximity sum, candidates' keys
//             (orderable approximate score, legal linear index z-major) below
//             a per-request pruning bound;
//   merge   - per request, the smallest keys in order;
//   exact   - per selected key, exact u8 overlap recount and the exact,
//             correctly rounded FP64 proximity sum.
// The host then scores exactly, orders by (score, z, y, x), applies the
// cursor and certifies that no excluded candidate could enter the page; an
// uncertified page is recomputed in threshold mode (every candidate whose
// approximate score is within the error bound of the page's last entry).
//
// The score rises with z and falls with the proximity sum, which the kernel's
// shape bounds (KernelSlot::most_proximity).  Where the goal allows it, planes
// are therefore visited upwards in rounds, from the first plane with room for
// the kernel, until the bound of the planes above lies past what is wanted.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <tuple>
#include <vector>

#include "context.hpp"
#include "edt.cuh"
#include "keys.cuh"
#include "pipeline.hpp"
#include "superacc.cuh"

namespace spk {

namespace {

constexpr std::int32_t kInf = INT32_MAX;
constexpr unsigned kFull = 0xffffffffu;

int launch_blocks(long long n, int threads)
{
    const long long want = (n + threads - 1) / threads;
    return static_cast<int>(std::min<long long>(std::max<long long>(want, 1), 148LL * 32));
}

// ---- kernel depth --------------------------------------------------------------
//
// Squared distance of every kernel cell to the nearest cell that is not the
// kernel's (cells outside its window among them), by one pass per axis.  A
// cell's search runs outwards and stops at the best distance so far, so it
// costs the depth, not the line.

// blockIdx.y: the item of a batch.
__global__ void depth_pass_kernel(const KernelItem* __restrict__ items, const std::uint8_t* __restrict__ all_cells,
                                  const std::int32_t* __restrict__ all_in, std::int32_t* __restrict__ all_out, int axis)
{
    const KernelItem& it = items[blockIdx.y];
    const std::uint8_t* cells = all_cells + it.cells_at;
    const std::int32_t* in = all_in + it.cells_at;
    std::int32_t* out = all_out + it.cells_at;
    const int n = it.K[0] * it.K[1] * it.K[2];
    const int length = it.K[axis];
    const int stride = axis == 0 ? 1 : axis == 1 ? it.K[0] : it.K[0] * it.K[1];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int at = (i / stride) % length;
        // Axis 0 starts from the cells: 0 at a cell that is not the kernel's.
        std::int32_t best = axis == 0 ? (cells[i] ? kInf : 0) : in[i];
        for (int r = 1; r * r < best; ++r) {
            for (int side = 0; side < 2; ++side) {
                const int q = side ? at + r : at - r;
                std::int32_t v = 0;
                if (q >= 0 && q < length) {
                    const int c = i + (side ? r : -r) * stride;
                    v = axis == 0 ? (cells[c] ? kInf : 0) : in[c];
                }
                if (v != kInf) {
                    best = min(best, v + r * r);
                }
            }
        }
        out[i] = best;
    }
}

// One block per plane of the batch: the sum of table[depth^2] over its kernel
// cells and the largest depth^2.
__global__ void __launch_bounds__(256) depth_plane_kernel(const KernelItem* __restrict__ items,
                                                         const int* __restrict__ plane_item,
                                                         const std::int32_t* __restrict__ depth2,
                                                         const double* __restrict__ table, RowStats* __restrict__ out)
{
    __shared__ double warp_sum[8];
    __shared__ std::int32_t warp_max[8];
    const KernelItem& it = items[plane_item[blockIdx.x]];
    const int plane_cells = it.K[0] * it.K[1];
    const std::int32_t* plane =
        depth2 + it.cells_at + static_cast<long long>(plane_cells) * (static_cast<int>(blockIdx.x) - it.first_plane);
    double sum = 0;
    std::int32_t most = 0;
    for (int i = threadIdx.x; i < plane_cells; i += blockDim.x) {
        const std::int32_t v = plane[i];
        if (v > 0) {
            sum += table[v];
            most = max(most, v);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(kFull, sum, o);
        most = max(most, __shfl_xor_sync(kFull, most, o));
    }
    if ((threadIdx.x & 31) == 0) {
        warp_sum[threadIdx.x >> 5] = sum;
        warp_max[threadIdx.x >> 5] = most;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        RowStats r { 0.0, 0, 0 };
        for (int w = 0; w < 8; ++w) {
            r.norm += warp_sum[w];
            r.max_d2 = max(r.max_d2, warp_max[w]);
        }
        out[blockIdx.x] = r;
    }
}

// The environment-relative offsets of each item's cells that are set, in
// ones[cells_at ...], and their number (in any order: every use sums over them
// exactly).
__global__ void ones_kernel(const KernelItem* __restrict__ items, const std::uint8_t* __restrict__ all_cells, int E0,
                            int E1, std::int32_t* __restrict__ ones, unsigned int* __restrict__ counts)
{
    const KernelItem& it = items[blockIdx.y];
    const int n = it.K[0] * it.K[1] * it.K[2], lane = threadIdx.x & 31;
    for (int i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + threadIdx.x;
        const bool one = i < n && all_cells[it.cells_at + i];
        const unsigned mask = __ballot_sync(kFull, one);
        unsigned int at = 0;
        if (lane == 0 && mask) {
            at = atomicAdd(&counts[blockIdx.y], static_cast<unsigned int>(__popc(mask)));
        }
        at = __shfl_sync(kFull, at, 0) + __popc(mask & ((1u << lane) - 1u));
        if (one) {
            const int x = i % it.K[0], r = i / it.K[0], y = r % it.K[1], z = r / it.K[1];
            ones[it.cells_at + at] = x + E0 * (y + E1 * z);
        }
    }
}

// ---- merge -----------------------------------------------------------------------

// Per request: no bound, no residual, no keys.
__global__ void page_init_kernel(unsigned long long* __restrict__ tau, unsigned long long* __restrict__ resid,
                                 unsigned long long* __restrict__ count, int requests, int* __restrict__ range_error)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < requests) {
        tau[r] = kEmptyKey;
        resid[r] = 0;
        count[r] = 0;
    }
    if (r == 0) {
        *range_error = 0;
    }
}

// Bitonic sort of n <= capacity keys in shared memory (padded with kEmptyKey
// to a power of two); the block then holds them in ascending order in s[].
__device__ unsigned int block_sort(const unsigned long long* __restrict__ src, unsigned int n,
                                   unsigned long long* s)
{
    unsigned int size = 1;
    while (size < n) {
        size <<= 1;
    }
    for (unsigned int i = threadIdx.x; i < size; i += blockDim.x) {
        s[i] = i < n ? src[i] : kEmptyKey;
    }
    __syncthreads();
    for (unsigned int k = 2; k <= size; k <<= 1) {
        for (unsigned int j = k >> 1; j > 0; j >>= 1) {
            for (unsigned int i = threadIdx.x; i < size; i += blockDim.x) {
                const unsigned int p = i ^ j;
                if (p > i) {
                    const bool up = (i & k) == 0;
                    const unsigned long long x = s[i], y = s[p];
                    if ((x > y) == up) {
                        s[i] = y;
                        s[p] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
    return size;
}

// First stage of the merge: chunk c (kKeyCapacity keys) of request r keeps its
// `per` smallest keys in partial[(r * chunks + c) * per ...].
__global__ void merge_chunk_kernel(const unsigned long long* __restrict__ keys, unsigned int cap,
                                   const unsigned long long* __restrict__ counts, const int* __restrict__ lanes,
                                   int per, unsigned long long* __restrict__ partial)
{
    __shared__ unsigned long long sorted[kKeyCapacity];
    const int c = blockIdx.x, r = lanes[blockIdx.y], chunks = gridDim.x;
    const unsigned int n_r = min(static_cast<unsigned int>(counts[r]), cap);
    const unsigned int begin = static_cast<unsigned int>(c) * kKeyCapacity;
    const unsigned int n = begin < n_r ? min(kKeyCapacity, n_r - begin) : 0u;
    unsigned long long* out = partial + (static_cast<long long>(r) * chunks + c) * per;
    if (n == 0) {
        for (int i = threadIdx.x; i < per; i += blockDim.x) {
            out[i] = kEmptyKey;
        }
        return;
    }
    const unsigned int size = block_sort(keys + static_cast<long long>(r) * cap + begin, n, sorted);
    for (int i = threadIdx.x; i < per; i += blockDim.x) {
        out[i] = static_cast<unsigned int>(i) < size ? sorted[i] : kEmptyKey;
    }
}

// Second stage of the merge: request r's `lists` sorted lists of
// `per` keys each (the first stage's chunk winners) merged into their `per`
// smallest, ascending, by one warp-pair per request: thread c holds the head
// of list c, and each round the smallest head (keys are distinct, empty
// slots are kEmptyKey) is written out and its list advances.  The result is
// the first `per` keys of the sorted union, as a full sort would give.
__global__ void __launch_bounds__(64) merge_lists_kernel(const unsigned long long* __restrict__ partial,
                                                        const int* __restrict__ lanes, int lists, int per,
                                                        unsigned long long* __restrict__ selected)
{
    __shared__ unsigned long long warp_min[2];
    const int r = lanes[blockIdx.x], c = threadIdx.x, lane = c & 31, warp = c >> 5;
    const unsigned long long* list = partial + (static_cast<long long>(r) * lists + c) * per;
    int head = 0;
    unsigned long long value = c < lists ? list[0] : kEmptyKey;
    for (int i = 0; i < per; ++i) {
        unsigned long long m = value;
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(kFull, m, o);
            m = other < m ? other : m;
        }
        if (lane == 0) {
            warp_min[warp] = m;
        }
        __syncthreads();
        const unsigned long long best = warp_min[0] < warp_min[1] ? warp_min[0] : warp_min[1];
        __syncthreads();
        if (c == 0) {
            selected[static_cast<long long>(r) * per + i] = best;
        }
        if (value == best && best != kEmptyKey) {
            ++head;
            value = head < per ? list[head] : kEmptyKey;
        }
    }
}

// ---- merge of few ---------------------------------------------------------------------

// Ascending bitonic sort of a warp's keys; `first` = 2 sorts any keys, 32 a
// bitonic sequence.
__device__ __forceinline__ unsigned long long warp_sort(unsigned long long v, int first)
{
    const int lane = threadIdx.x & 31;
    for (int k = first; k <= 32; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            const unsigned long long o = __shfl_xor_sync(kFull, v, j);
            const bool low = (lane & j) == 0, up = (lane & k) == 0;
            v = (low == up) == (o < v) ? o : v;
        }
    }
    return v;
}
// The 32 smallest of two ascending sets: the pairwise minima of one and the
// other reversed, a bitonic sequence.
__device__ __forceinline__ unsigned long long warp_merge(unsigned long long a, unsigned long long b)
{
    const unsigned long long r = __shfl_sync(kFull, b, 31 - (threadIdx.x & 31));
    return warp_sort(r < a ? r : a, 32);
}

// The `per` <= 32 smallest keys of each request, ascending: a block per
// request; every warp keeps the 32 smallest of its share in registers, sorting
// in only batches that can change them, and the warps' sets are merged in
// pairs.  The result is that of the two-stage merge, which sorts whole chunks
// for longer lists (96 requests: 18 and 7 us for its kernels, 5.3 us this way).
constexpr int kFewKeys = 32;
constexpr int kHeadThreads = 1024;
__global__ void __launch_bounds__(kHeadThreads) merge_heads_kernel(const unsigned long long* __restrict__ keys,
                                                                  unsigned int cap,
                                                                  const unsigned long long* __restrict__ counts,
                                                                  const int* __restrict__ lanes, int per,
                                                                  unsigned long long* __restrict__ selected)
{
    __shared__ unsigned long long sets[kHeadThreads / 32][32];
    const int r = lanes[blockIdx.x], lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned int n = min(static_cast<unsigned int>(counts[r]), cap);
    const unsigned long long* from = keys + static_cast<long long>(r) * cap;
    unsigned long long best = kEmptyKey;
#pragma unroll 4
    for (unsigned int i0 = warp * 32; i0 < n; i0 += kHeadThreads) {
        const unsigned long long v = i0 + lane < n ? from[i0 + lane] : kEmptyKey;
        const unsigned long long most = __shfl_sync(kFull, best, 31);
        if (__any_sync(kFull, v < most)) {
            best = warp_merge(best, warp_sort(v, 2));
        }
    }
    for (int half = kHeadThreads / 64; half > 0; half >>= 1) {
        if (warp >= half && warp < 2 * half) {
            sets[warp][lane] = best;
        }
        __syncthreads();
        if (warp < half) {
            best = warp_merge(best, sets[warp + half][lane]);
        }
    }
    if (warp == 0 && lane < per) {
        selected[static_cast<long long>(r) * per + lane] = best;
    }
}

// ---- exact rescoring ----------------------------------------------------------------

struct ExactJob {
    const std::int32_t* ones;
    int ones_count;
    int legal_x, legal_y;
};

// Squared distances below this are counted per value (the rest, cells more
// than 64 cells from everything, are added one by one).
constexpr int kExactBins = 4096;
// Fixed point of the counted sum: exp(-sqrt(4095) / 2) > 2^-47, so the last
// bit of every counted term is at or above 2^-99, and counts below 2^27 keep
// the sum under 2^127 of those units.
constexpr int kExactLowBit = -99;
constexpr int kExactThreads = 512;
constexpr int kExactUnroll = 8;

// One block per selected key (the first `count` of each request in `lanes`,
// or of every request): exact overlap recount and exact proximity sum.
// Proximity is a function of the integer squared distance, so the sum over
// the item's cells is sum over v of count[v] table[v]: the cells are counted
// in shared memory (one load and one shared atomic per cell) and only the
// few hundred distinct values are multiplied out, exactly, in 128-bit fixed
// point.  Bound by the latency of the dependent loads (offset, then cell), so
// eight cells are in flight per thread.  Adding every cell's value to a
// 23-limb accumulator per thread put those limbs in local memory: 190 us a
// launch on a 128^3 window at 0.5 mm pitch, 43 us this way; 90 and 15 us on a
// 66^3 window with a 2,800-cell cuboid (means over greedy fills).  Only cells at
// distance 0 are occupied, so no other cell's occupancy is read (1,536 keys of
// 80,000 cells: 132 us with it, 100 us without).
__global__ void __launch_bounds__(kExactThreads) exact_kernel(
    const unsigned long long* __restrict__ selected, const ExactJob* __restrict__ jobs,
    const int* __restrict__ lanes, int per_request, int count,
    const std::uint8_t* __restrict__ occ, const std::int32_t* __restrict__ d2, const double* __restrict__ table,
    int E0, int E1, long long* __restrict__ out_count, double* __restrict__ out_p, int* __restrict__ range_error)
{
    __shared__ unsigned int hist[kExactBins];
    __shared__ unsigned long long far[kSuperLimbs];
    __shared__ unsigned int far_cells, bad;
    __shared__ unsigned long long s_hi[kExactThreads / 32], s_lo[kExactThreads / 32];
    __shared__ unsigned long long s_overlap[kExactThreads / 32];
    const int request = lanes ? lanes[blockIdx.x / count] : static_cast<int>(blockIdx.x / count);
    const int at = request * per_request + static_cast<int>(blockIdx.x % count);
    const unsigned long long key = selected[at];
    if (key == kEmptyKey) {
        if (threadIdx.x == 0) {
            out_count[at] = -1;
            out_p[at] = 0.0;
        }
        return;
    }
    for (int i = threadIdx.x; i < kExactBins; i += kExactThreads) {
        hist[i] = 0;
    }
    if (threadIdx.x < kSuperLimbs) {
        far[threadIdx.x] = 0;
    }
    if (threadIdx.x == 0) {
        far_cells = 0;
        bad = 0;
    }
    const ExactJob job = jobs[request];
    const unsigned int index = static_cast<unsigned int>(key & 0xffffffffULL);
    const long long sx = index % job.legal_x;
    const long long rest = index / job.legal_x;
    const long long sy = rest % job.legal_y;
    const long long sz = rest / job.legal_y;
    const long long base = sx + E0 * (sy + static_cast<long long>(E1) * sz);
    unsigned long long overlap = 0;
    __syncthreads();
    const std::int32_t* at_base = d2 + base;
    const std::uint8_t* occ_base = occ + base;
    for (int i0 = threadIdx.x; i0 < job.ones_count; i0 += kExactUnroll * kExactThreads) {
        // Independent loads first: a cell costs two dependent L2 reads, and one
        // cell per iteration left the block waiting on them.
        std::int32_t v[kExactUnroll], cell[kExactUnroll];
#pragma unroll
        for (int u = 0; u < kExactUnroll; ++u) {
            const int i = i0 + u * kExactThreads;
            cell[u] = i < job.ones_count ? job.ones[i] : -1;
        }
#pragma unroll
        for (int u = 0; u < kExactUnroll; ++u) {
            v[u] = cell[u] >= 0 ? at_base[cell[u]] : kInf;
        }
#pragma unroll
        for (int u = 0; u < kExactUnroll; ++u) {
            if (v[u] == 0) {
                overlap += occ_base[cell[u]];  // only occupied cells are at distance 0
            }
            if (static_cast<std::uint32_t>(v[u]) < static_cast<std::uint32_t>(kExactBins)) {
                atomicAdd(&hist[v[u]], 1u);
            }
            else if (v[u] != kInf) {
                SuperAcc one;
                super_clear(one);
                if (super_add(one, table[v[u]])) {
                    for (int l = 0; l < kSuperLimbs; ++l) {
                        if (one.limb[l]) {
                            atomicAdd(&far[l], static_cast<unsigned long long>(one.limb[l]));
                        }
                    }
                    atomicAdd(&far_cells, 1u);
                }
                else {
                    bad = 1;
                }
            }
        }
    }
    __syncthreads();
    unsigned __int128 sum = 0;
    for (int v = threadIdx.x; v < kExactBins; v += kExactThreads) {
        const unsigned int c = hist[v];
        if (c) {
            const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(table[v]));
            const unsigned long long mant = (bits & ((1ULL << 52) - 1)) | (1ULL << 52);
            const int shift = static_cast<int>(bits >> 52) - 1075 - kExactLowBit;
            sum += (static_cast<unsigned __int128>(mant) * c) << shift;
        }
    }
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        overlap += __shfl_xor_sync(kFull, overlap, o);
        const unsigned long long lo = __shfl_xor_sync(kFull, static_cast<unsigned long long>(sum), o);
        const unsigned long long hi = __shfl_xor_sync(kFull, static_cast<unsigned long long>(sum >> 64), o);
        sum += (static_cast<unsigned __int128>(hi) << 64) | lo;
    }
    if (lane == 0) {
        s_overlap[warp] = overlap;
        s_hi[warp] = static_cast<unsigned long long>(sum >> 64);
        s_lo[warp] = static_cast<unsigned long long>(sum);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned __int128 total = 0;
        long long cells = 0;
        for (int w = 0; w < kExactThreads / 32; ++w) {
            cells += static_cast<long long>(s_overlap[w]);
            total += (static_cast<unsigned __int128>(s_hi[w]) << 64) | s_lo[w];
        }
        const auto hi = static_cast<unsigned long long>(total >> 64), lo = static_cast<unsigned long long>(total);
        out_count[at] = cells;
        if (!far_cells) {
            out_p[at] = round_u128(hi, lo, kExactLowBit);
        }
        else {
            SuperAcc acc;
            for (int l = 0; l < kSuperLimbs; ++l) {
                acc.limb[l] = static_cast<long long>(far[l]);
            }
            super_add_at(acc, lo, kExactLowBit - kSuperLowBit);
            super_add_at(acc, hi, kExactLowBit - kSuperLowBit + 64);
            out_p[at] = super_round(acc);
        }
        if (bad) {
            atomicOr(range_error, 1);
        }
    }
}

double decode_key_score(unsigned long long key)
{
    const unsigned int k = static_cast<unsigned int>(key >> 32);
    const unsigned int u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    float f;
    std::memcpy(&f, &u, 4);
    return static_cast<double>(f);
}

bool rank_less(const Candidate& l, const Candidate& r)
{
    if (l.score != r.score) {
        return l.score < r.score;
    }
    if (l.orientation != r.orientation) {
        return l.orientation < r.orientation;
    }
    return std::tie(l.t[2], l.t[1], l.t[0]) < std::tie(r.t[2], r.t[1], r.t[0]);
}

}  // namespace

Pipeline::Pipeline(spk_context* ctx, const char* name) : ctx_(ctx), name_(name)
{
    const char* fixed = std::getenv("SPK_FFT_LENGTHS");
    pow2_ = fixed && std::strcmp(fixed, "pow2") == 0;
    debug_ = std::getenv("SPK_DEBUG_PAGES") != nullptr;
}

Pipeline::~Pipeline()
{
    if (side_) {
        cudaStreamSynchronize(side_);
        cudaEventDestroy(ev_in_);
        cudaEventDestroy(ev_done_);
        cudaStreamDestroy(side_);
    }
    for (const auto& b : blocks_) {
        give_block(ctx_, b.ptr, b.bytes);
    }
}

// A window of E cells takes the smallest supported length L >= E per axis:
// legal translations never wrap on it, and the register plans' cost per point
// differs too little between neighbouring lengths to pay for more points.
// SPK_FFT_LENGTHS=pow2 allows powers of two only.
int Pipeline::choose_lengths(const std::uint32_t* env_shape)
{
    int count = 0;
    const int* lengths = axis_lengths(count);
    for (int a = 0; a < 3; ++a) {
        L_[a] = 0;
        for (int i = 0; i < count && !L_[a]; ++i) {
            const bool allowed = !pow2_ || is_pow2(static_cast<std::uint64_t>(lengths[i]));
            if (allowed && lengths[i] >= static_cast<int>(std::min<std::uint32_t>(env_shape[a], INT32_MAX))) {
                L_[a] = lengths[i];
            }
        }
        if (!L_[a]) {
            return kUnsupportedLength;
        }
    }
    return kOk;
}

int Pipeline::set_geometry(const std::int64_t* env_first, const std::uint32_t* env_shape, const double* origin,
                           double pitch, double container_min_z, double container_height)
{
    for (int a = 0; a != 3; ++a) {
        if (env_shape[a] == 0) {
            return kInvalidArgument;
        }
        E_[a] = static_cast<int>(env_shape[a]);
        env_first_[a] = env_first[a];
        origin_[a] = origin[a];
    }
    if (int status = choose_lengths(env_shape)) {
        return status;
    }
    pitch_ = pitch;
    cmin_z_ = container_min_z;
    height_ = container_height;
    const long long cells = static_cast<long long>(E_[0]) * E_[1] * E_[2];
    const long long grid = static_cast<long long>(L_[0]) * L_[1] * E_[2];
    const std::size_t row_blocks = static_cast<std::size_t>((E_[1] + kRowsPerBlock - 1) / kRowsPerBlock) * E_[2];
    int status = kOk;
    occ_ = static_cast<std::uint8_t*>(device_buffer(ctx_, name_ + ".occ", cells, status));
    d2_ = static_cast<std::int32_t*>(device_buffer(ctx_, name_ + ".d2", cells * sizeof(std::int32_t), status));
    env_ = static_cast<float2*>(device_buffer(ctx_, name_ + ".env", grid * sizeof(float2), status));
    stats_ = static_cast<RowStats*>(device_buffer(ctx_, name_ + ".stats", row_blocks * sizeof(RowStats), status));
    const long long tiles = static_cast<long long>((E_[0] + kEdtTile - 1) / kEdtTile) *
                            ((E_[1] + kEdtTile - 1) / kEdtTile) * ((E_[2] + kEdtTile - 1) / kEdtTile);
    tile_max_ =
        static_cast<std::int32_t*>(device_buffer(ctx_, name_ + ".tile_max", tiles * sizeof(std::int32_t), status));
    if (!occ_ || !d2_ || !env_ || !stats_ || !tile_max_) {
        return status;
    }
    const std::uint32_t shape[3] = { env_shape[0], env_shape[1], env_shape[2] };
    if (!proximity_shape_supported(shape)) {
        return kProximityShape;
    }
    return table(status) ? kOk : status;
}

const double* Pipeline::table(int& status) const
{
    const std::uint32_t shape[3] = { static_cast<std::uint32_t>(E_[0]), static_cast<std::uint32_t>(E_[1]),
                                     static_cast<std::uint32_t>(E_[2]) };
    // A kernel cell lies at most as deep as half its window's shortest side and
    // one, within the window's largest distance except in a window of one cell,
    // whose kernel is one cell deep.
    return proximity_table(ctx_, std::max(max_squared_distance(shape), 1), status);
}

int Pipeline::set_occupancy(const std::uint8_t* d_occupancy)
{
    cudaStream_t st = ctx_->stream;
    const long long cells = static_cast<long long>(E_[0]) * E_[1] * E_[2];
    if (d_occupancy != occ_) {
        cudaMemcpyAsync(occ_, d_occupancy, cells, cudaMemcpyDeviceToDevice, st);
    }
    const std::uint32_t shape[3] = { static_cast<std::uint32_t>(E_[0]), static_cast<std::uint32_t>(E_[1]),
                                     static_cast<std::uint32_t>(E_[2]) };
    int status = edt_squared(ctx_, occ_, d2_, shape, st);
    if (status || (status = edt_tile_max(ctx_, d2_, shape, tile_max_, st))) {
        return status;
    }
    return update_spectrum(nullptr);
}

int Pipeline::add_occupied(const std::uint8_t* d_occupancy, const std::uint8_t* d_sites, const EdtBox& sites)
{
    cudaStream_t st = ctx_->stream;
    const long long cells = static_cast<long long>(E_[0]) * E_[1] * E_[2];
    if (d_occupancy != occ_) {
        cudaMemcpyAsync(occ_, d_occupancy, cells, cudaMemcpyDeviceToDevice, st);
    }
    const std::uint32_t shape[3] = { static_cast<std::uint32_t>(E_[0]), static_cast<std::uint32_t>(E_[1]),
                                     static_cast<std::uint32_t>(E_[2]) };
    const EdtBox* d_region = nullptr;
    int status = edt_add_sites(ctx_, d_sites, sites, d2_, tile_max_, shape, st, &d_region);
    if (status || !d_region) {
        return status;  // no new site inside the window: nothing changed
    }
    return update_spectrum(d_region);
}

int Pipeline::update_spectrum(const EdtBox* d_region)
{
    cudaStream_t st = ctx_->stream;
    int status = kOk;
    const auto* tw0 = twiddle_table<float>(ctx_, L_[0], status);
    const auto* tw1 = twiddle_table<float>(ctx_, L_[1], status);
    const double* proximity = table(status);
    if (!tw0 || !tw1 || !proximity) {
        return status;
    }
    if (launch_env_rows(L_[0], L_[1], env_, E_, occ_, d2_, proximity, tw0, stats_, d_region, st) != cudaSuccess ||
        launch_forward_y(L_[0], L_[1], env_, E_[1], E_[2], tw1, d_region, st) != cudaSuccess) {
        cudaGetLastError();
        return kCuda;
    }
    ctx_->launches += 2;
    // The plane statistics come back to pinned memory; the host reads them
    // (finish_stats) only when a page needs them, so nothing here waits.
    const std::size_t bytes =
        sizeof(RowStats) * static_cast<std::size_t>((E_[1] + kRowsPerBlock - 1) / kRowsPerBlock) * E_[2];
    auto* host = static_cast<RowStats*>(host_buffer(ctx_, name_ + ".stats", bytes, status));
    if (!host) {
        return status;
    }
    cudaMemcpyAsync(host, stats_, bytes, cudaMemcpyDeviceToHost, st);
    stats_host_ = host;
    stats_stream_ = st;
    stats_pending_ = true;
    return cudaGetLastError() == cudaSuccess ? kOk : kCuda;
}

int Pipeline::finish_stats()
{
    if (!stats_pending_) {
        return kOk;
    }
    if (cudaStreamSynchronize(stats_stream_) != cudaSuccess) {
        cudaGetLastError();
        return kCuda;
    }
    const int row_blocks = (E_[1] + kRowsPerBlock - 1) / kRowsPerBlock;
    plane_max_.assign(E_[2], 0);
    double most = 0;
    for (int z = 0; z < E_[2]; ++z) {
        double norm = 0;
        for (int b = 0; b < row_blocks; ++b) {
            const RowStats& r = stats_host_[static_cast<std::size_t>(z) * row_blocks + b];
            norm += r.norm;
            plane_max_[z] = std::max(plane_max_[z], r.max_d2);
        }
        most = std::max(most, norm);
    }
    plane_rms_ = std::sqrt(most / (static_cast<double>(L_[0]) * L_[1]));
    stats_pending_ = false;
    return kOk;
}

int Pipeline::refresh_begin(const std::uint8_t* d_occupancy, const std::uint8_t* d_sites, const EdtBox* sites)
{
    refresh_order();
    if (!side_) {
        if (cudaStreamCreateWithFlags(&side_, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&ev_in_, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&ev_done_, cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            return kCuda;
        }
    }
    cudaStream_t main = ctx_->stream;
    cudaEventRecord(ev_in_, main);
    cudaStreamWaitEvent(side_, ev_in_, 0);
    // Every launch of the update goes to the side stream while it is queued.
    ctx_->stream = side_;
    const int status = d_sites ? add_occupied(d_occupancy, d_sites, *sites) : set_occupancy(d_occupancy);
    cudaEventRecord(ev_done_, side_);
    ctx_->stream = main;
    pending_ = true;
    return status;
}

void Pipeline::refresh_order()
{
    if (pending_) {
        cudaStreamWaitEvent(ctx_->stream, ev_done_, 0);
        pending_ = false;
    }
}

int Pipeline::add_kernel(std::uint64_t orientation, const std::int64_t* first, const std::uint32_t* shape,
                         const std::uint8_t* cells, double max_z, std::uint64_t& slot_out)
{
    geo::Window w;
    std::uint64_t n = 1;
    for (int a = 0; a != 3; ++a) {
        w.first[a] = first[a];
        w.shape[a] = shape[a];
        n *= shape[a];
    }
    int status = kOk;
    auto* d_cells = static_cast<std::uint8_t*>(device_buffer(ctx_, "pipe.kcells", n, status));
    if (!d_cells) {
        return status;
    }
    cudaMemcpyAsync(d_cells, cells, n, cudaMemcpyHostToDevice, ctx_->stream);
    const long long cells_at[2] = { 0, static_cast<long long>(n) };
    slot_out = slots_.size();
    return add_kernels(orientation, { w }, d_cells, cells_at, &max_z);
}

int Pipeline::add_kernels(std::uint64_t first_orientation, const std::vector<geo::Window>& windows,
                          const std::uint8_t* d_cells, const long long* cells_at, const double* max_z)
{
    cudaStream_t st = ctx_->stream;
    const int count = static_cast<int>(windows.size());
    int status = kOk;
    std::vector<KernelSlot> slots(count);
    // The kernels that fit the window get device data; K <= E <= L holds for them.
    std::vector<int> fit;
    std::vector<KernelItem> items;
    std::vector<int> plane_item;
    int rows = 1;
    long long most_cells = 1;
    for (int i = 0; i < count; ++i) {
        KernelSlot& s = slots[i];
        s.orientation = first_orientation + i;
        s.max_z = max_z[i];
        for (int a = 0; a != 3; ++a) {
            s.K[a] = static_cast<int>(windows[i].shape[a]);
            s.first[a] = windows[i].first[a];
            s.legal[a] = E_[a] >= s.K[a] ? E_[a] - s.K[a] + 1 : 0;
        }
        if (!s.legal[0] || !s.legal[1] || !s.legal[2]) {
            continue;
        }
        KernelItem it { cells_at[i], { s.K[0], s.K[1], s.K[2] }, static_cast<int>(plane_item.size()) };
        plane_item.insert(plane_item.end(), s.K[2], static_cast<int>(fit.size()));
        rows = std::max(rows, s.K[1]);
        most_cells = std::max(most_cells, static_cast<long long>(s.K[0]) * s.K[1] * s.K[2]);
        fit.push_back(i);
        items.push_back(it);
        s.t65_host.resize(s.legal[2]);
        for (int zi = 0; zi < s.legal[2]; ++zi) {
            const std::int64_t tz = env_first_[2] - s.first[2] + zi;
            const double world_z = origin_[2] + pitch_ * static_cast<double>(tz);
            const double top = (world_z + s.max_z - cmin_z_) / height_;
            s.t65_host[zi] = .65 * top;
        }
    }
    const std::size_t total = static_cast<std::size_t>(cells_at[count]);
    std::vector<std::uint8_t> host_cells(total);
    const std::size_t planes = plane_item.size();
    unsigned int* h_counts = nullptr;
    RowStats* h_planes = nullptr;
    if (!fit.empty()) {
        // One block for the batch: partial spectra, offset lists (room for
        // every cell), and the legal planes' .65 top.
        const std::size_t plane_bytes = static_cast<std::size_t>(L_[0]) * L_[1] * sizeof(float2);
        const std::size_t partial_bytes = plane_bytes * planes;
        const std::size_t ones_bytes = (total * sizeof(std::int32_t) + 255) / 256 * 256;
        std::size_t t65_count = 0;
        for (int i : fit) {
            t65_count += slots[i].t65_host.size();
        }
        // Tables of the batch, up in one copy: items, planes' items, .65 top.
        const std::size_t items_bytes = items.size() * sizeof(KernelItem);
        const std::size_t table_bytes = (items_bytes + planes * sizeof(int) + 7) / 8 * 8;
        auto* h_table = static_cast<char*>(
            host_buffer(ctx_, "pipe.kernel_table", table_bytes + t65_count * sizeof(double), status));
        auto* d_table = static_cast<char*>(device_buffer(ctx_, "pipe.kernel_table", table_bytes, status));
        // The passes of the depths alternate between a buffer and the raster's
        // labels, which are done with.
        const std::size_t depth_bytes = total * sizeof(std::int32_t);
        auto* depth = static_cast<std::int32_t*>(device_buffer(ctx_, "pipe.depth", depth_bytes, status));
        auto* other = static_cast<std::int32_t*>(device_buffer(ctx_, "field.parent", depth_bytes, status));
        // Results: plane statistics, then counts.
        const std::size_t result_bytes = planes * sizeof(RowStats) + fit.size() * sizeof(unsigned int);
        auto* d_result = static_cast<char*>(device_buffer(ctx_, "pipe.kernel_result", result_bytes, status));
        auto* h_result = static_cast<char*>(host_buffer(ctx_, "pipe.kernel_result", result_bytes, status));
        const auto* tw0 = twiddle_table<float>(ctx_, L_[0], status);
        const auto* tw1 = twiddle_table<float>(ctx_, L_[1], status);
        const double* proximity = table(status);
        if (!h_table || !d_table || !depth || !other || !d_result || !h_result || !tw0 || !tw1 || !proximity) {
            return status;
        }
        Block block { nullptr, partial_bytes + ones_bytes + t65_count * sizeof(double) };
        block.ptr = take_block(ctx_, block.bytes, status);
        if (!block.ptr) {
            return status;
        }
        blocks_.push_back(block);
        auto* partial = static_cast<float2*>(block.ptr);
        auto* ones = reinterpret_cast<std::int32_t*>(static_cast<char*>(block.ptr) + partial_bytes);
        auto* t65 = reinterpret_cast<double*>(reinterpret_cast<char*>(ones) + ones_bytes);
        std::memcpy(h_table, items.data(), items_bytes);
        std::memcpy(h_table + items_bytes, plane_item.data(), planes * sizeof(int));
        auto* h_t65 = reinterpret_cast<double*>(h_table + table_bytes);
        std::size_t at = 0;
        for (std::size_t f = 0; f < fit.size(); ++f) {
            KernelSlot& s = slots[fit[f]];
            s.partial = partial + static_cast<std::size_t>(items[f].first_plane) * L_[0] * L_[1];
            s.ones = ones + items[f].cells_at;
            s.t65 = t65 + at;
            std::copy(s.t65_host.begin(), s.t65_host.end(), h_t65 + at);
            at += s.t65_host.size();
        }
        cudaMemcpyAsync(d_table, h_table, table_bytes, cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(t65, h_t65, t65_count * sizeof(double), cudaMemcpyHostToDevice, st);
        const auto* d_items = reinterpret_cast<const KernelItem*>(d_table);
        const auto* d_plane_item = reinterpret_cast<const int*>(d_table + items_bytes);
        auto* d_planes = reinterpret_cast<RowStats*>(d_result);
        auto* d_counts = reinterpret_cast<unsigned int*>(d_result + planes * sizeof(RowStats));
        cudaMemsetAsync(d_counts, 0, fit.size() * sizeof(unsigned int), st);
        const auto n = static_cast<unsigned>(fit.size());
        const dim3 grid(static_cast<unsigned>(std::max<long long>(
                            1, std::min<long long>((most_cells + 127) / 128, 148LL * 32 / n + 1))),
                        n);
        ones_kernel<<<grid, 128, 0, st>>>(d_items, d_cells, E_[0], E_[1], ones, d_counts);
        if (launch_kernel_rows(L_[0], L_[1], partial, d_items, d_plane_item, static_cast<int>(planes), rows, d_cells,
                               tw0, st) != cudaSuccess ||
            launch_forward_y(L_[0], L_[1], partial, rows, static_cast<int>(planes), tw1, nullptr, st) != cudaSuccess) {
            cudaGetLastError();
            return kCuda;
        }
        depth_pass_kernel<<<grid, 128, 0, st>>>(d_items, d_cells, nullptr, depth, 0);
        depth_pass_kernel<<<grid, 128, 0, st>>>(d_items, d_cells, depth, other, 1);
        depth_pass_kernel<<<grid, 128, 0, st>>>(d_items, d_cells, other, depth, 2);
        depth_plane_kernel<<<static_cast<unsigned>(planes), 256, 0, st>>>(d_items, d_plane_item, depth, proximity,
                                                                         d_planes);
        ctx_->launches += 7;
        cudaMemcpyAsync(h_result, d_result, result_bytes, cudaMemcpyDeviceToHost, st);
        h_planes = reinterpret_cast<RowStats*>(h_result);
        h_counts = reinterpret_cast<unsigned int*>(h_result + planes * sizeof(RowStats));
    }
    cudaMemcpyAsync(host_cells.data(), d_cells, total, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return kCuda;
    }
    for (int i = 0; i < count; ++i) {
        slots[i].host_cells.assign(host_cells.begin() + cells_at[i], host_cells.begin() + cells_at[i + 1]);
    }
    for (std::size_t f = 0; f < fit.size(); ++f) {
        KernelSlot& s = slots[fit[f]];
        s.occupied = h_counts[f];
        double sum = 0;
        s.depth2.resize(s.K[2]);
        for (int z = 0; z < s.K[2]; ++z) {
            const RowStats& r = h_planes[items[f].first_plane + z];
            sum += r.norm;
            s.depth2[z] = r.max_d2;
        }
        s.most_proximity = sum * (1.0 + 1e-9);  // far above the rounding of either sum
    }
    for (auto& s : slots) {
        slots_.push_back(std::move(s));
    }
    return kOk;
}

double Pipeline::epsilon_p(const KernelSlot& s) const
{
    // Error bound of the FP32 proximity sum (and of the overlap count beside
    // it): 2^-14 log2(N) rms(Z) sqrt(occ), with the largest plane's rms, which
    // bounds that of any slab; checked at run time against every exactly
    // rescored candidate.
    const double n = static_cast<double>(L_[0]) * L_[1] * L_[2];
    return std::ldexp(1.0, -14) * std::log2(n) * plane_rms_ * std::sqrt(static_cast<double>(s.occupied));
}

double Pipeline::approx_epsilon(const KernelSlot& s) const
{
    return .35 * epsilon_p(s) / static_cast<double>(s.occupied);
}

double Pipeline::score(const KernelSlot& s, const std::int64_t* t, double p) const
{
    // spectral_pipeline.cpp:1794-1800, evaluated in the same order.
    const double mean_proximity = p / static_cast<double>(s.occupied);
    const double world_z = origin_[2] + pitch_ * static_cast<double>(t[2]);
    const double top = (world_z + s.max_z - cmin_z_) / height_;
    return .65 * top - .35 * mean_proximity;
}

void Pipeline::feasible_planes(const KernelSlot& s, int& zb, int& zt) const
{
    const auto fits = [&](int z) {
        for (int k = 0; k < s.K[2]; ++k) {
            if (plane_max_[z + k] < s.depth2[k]) {
                return false;
            }
        }
        return true;
    };
    zb = 0;
    zt = s.legal[2];
    while (zb < zt && !fits(zb)) {
        ++zb;
    }
    while (zt > zb && !fits(zt - 1)) {
        --zt;
    }
}

// Cost of a slab's transforms along z per orientation and column: its points,
// weighted by the plans' measured cost per point (longer lines hold more
// registers and so fewer warps).
double slab_cost(int LZ)
{
    return LZ * (LZ <= 64 ? 1.0 : LZ <= 128 ? 1.2 : LZ == 192 ? 1.4 : LZ <= 256 ? 1.25 : 2.0);
}

// Slab intermediates of a launch at most.  Whole batches measured fastest at
// every window size, in L2 or not: a launch of two or three orientations (64
// MB) loses more to its tail and to the environment column's transform than the
// intermediate's trip through HBM costs (32 orientations of a 256^3 window, one
// slab: passes A, B1 and B2 1.11 ms at 64 MB, 0.80 ms in batches of 16; a
// 128^3 window 0.75 and 0.63 ms).
constexpr std::size_t kInterBytes = 2ULL << 30;

int Pipeline::run_planes(const std::vector<PlaneWork>& work, PassMode mode, bool bound_known)
{
    cudaStream_t st = ctx_->stream;
    int status = kOk;
    const std::size_t plane_cells = static_cast<std::size_t>(L_[0]) * L_[1];
    const auto* tw0 = twiddle_table<float>(ctx_, L_[0], status);
    const auto* tw1 = twiddle_table<float>(ctx_, L_[1], status);
    if (!tw0 || !tw1) {
        return status;
    }
    // Kernels of like depth share launches.
    std::vector<int> order(work.size()), next(work.size());
    for (std::size_t i = 0; i < order.size(); ++i) {
        order[i] = static_cast<int>(i);
        next[i] = work[i].z0;
    }
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return work[a].slot->K[2] < work[b].slot->K[2]; });
    int length_count = 0;
    const int* lengths = slab_lengths(length_count);
    const bool earlier = bound_known;
    for (std::size_t i0 = 0; i0 < order.size(); i0 += kPassBatch) {
        const int n = static_cast<int>(std::min<std::size_t>(kPassBatch, order.size() - i0));
        for (bound_known = earlier;; bound_known = true) {
            // The next slab starts at the lowest plane any orientation of the
            // group still wants; its length is the one that finishes the group
            // at the lowest cost.  An orientation of K2 planes gets LZ - K2 + 1
            // planes of it.
            int lo = INT32_MAX;
            for (int i = 0; i < n; ++i) {
                const int w = order[i0 + i];
                lo = next[w] < work[w].z1 ? std::min(lo, next[w]) : lo;
            }
            if (lo == INT32_MAX) {
                break;
            }
            int LZ = 0;
            double least = INFINITY;
            for (int l = 0; l < length_count; ++l) {
                if (pow2_ && !is_pow2(static_cast<std::uint64_t>(lengths[l]))) {
                    continue;
                }
                int slabs = 0;
                for (int i = 0; i < n; ++i) {
                    const PlaneWork& w = work[order[i0 + i]];
                    const int W = lengths[l] - w.slot->K[2] + 1, left = w.z1 - std::max(next[order[i0 + i]], lo);
                    if (left > 0) {
                        slabs = W < 1 ? INT32_MAX : std::max(slabs, (left + W - 1) / W);
                    }
                }
                if (slabs != INT32_MAX && slabs * slab_cost(lengths[l]) < least) {
                    least = slabs * slab_cost(lengths[l]);
                    LZ = lengths[l];
                }
            }
            const auto* twz = LZ ? twiddle_table<float>(ctx_, LZ, status) : nullptr;
            if (!twz) {
                return LZ ? status : kUnsupportedLength;
            }
            int W = 1;  // the most planes one of them visits
            for (int i = 0; i < n; ++i) {
                const PlaneWork& w = work[order[i0 + i]];
                W = std::max(W, std::min(w.z1, lo + LZ - w.slot->K[2] + 1) - std::max(next[order[i0 + i]], lo));
            }
            const std::size_t bytes = plane_cells * W * sizeof(float2);
            int per_launch = static_cast<int>(
                std::min<std::size_t>(std::max<std::size_t>(kInterBytes / bytes, 1), static_cast<std::size_t>(n)));
            if (ctx_->cap_bytes) {  // half of what is left: placements need theirs
                per_launch = static_cast<int>(std::max<std::uint64_t>(
                    1, std::min<std::uint64_t>(per_launch, room_for(ctx_, "pipe.inter") / 2 / bytes)));
            }
            float2* inter = nullptr;
            while (!inter) {  // under a device-memory cap, fewer orientations per launch
                inter = static_cast<float2*>(device_buffer(ctx_, "pipe.inter", bytes * per_launch, status));
                if (!inter && per_launch == 1) {
                    return status;
                }
                per_launch = inter ? per_launch : per_launch / 2;
            }
            status = kOk;
            int i = 0;
            while (i < n) {
                PassBatch batch {};
                batch.L0 = L_[0];
                batch.L1 = L_[1];
                batch.z0 = lo;
                batch.E2 = E_[2];
                batch.bound_known = bound_known;
                batch.scale = static_cast<float>(1.0 / (static_cast<double>(plane_cells) * LZ));
                const int groups = (L_[0] + 15) / 16;
                int blocks1 = 0;
                double bytes_a = 8.0 * plane_cells * std::min(LZ, E_[2] - lo), bytes1 = 0, bytes2 = 0;
                int rows_blocks[kPassBatch];
                for (; i < n && batch.count < per_launch; ++i) {
                    const PlaneWork& w = work[order[i0 + i]];
                    const KernelSlot& s = *w.slot;
                    const int z0 = next[order[i0 + i]], z1 = std::min(w.z1, lo + LZ - s.K[2] + 1);
                    if (z0 >= z1) {
                        continue;
                    }
                    next[order[i0 + i]] = z1;
                    PassSlot& p = batch.slot[batch.count];
                    p.partial = s.partial;
                    p.inter = inter + static_cast<std::size_t>(batch.count) * plane_cells * W;
                    p.t65 = s.t65 + z0;
                    p.keys = w.keys;
                    p.count = w.count;
                    p.tau = w.tau;
                    p.resid = w.resid;
                    p.inv_occ = 1.0 / static_cast<double>(s.occupied);
                    p.cursor_floor = w.cursor_floor;
                    p.threshold = w.threshold;
                    p.prune = w.prune;
                    p.target = w.target;
                    p.cap = w.cap;
                    p.key_base = static_cast<unsigned int>(s.legal[0]) * s.legal[1] * z0;
                    p.K2 = s.K[2];
                    p.skip = z0 - lo;
                    p.planes = z1 - z0;
                    p.legal_x = s.legal[0];
                    p.legal_y = s.legal[1];
                    p.first_b1 = blocks1;
                    blocks1 += groups * p.planes;
                    const long long rows = static_cast<long long>(p.legal_y) * p.planes;
                    rows_blocks[batch.count] = static_cast<int>((rows + kRowsPerBlock - 1) / kRowsPerBlock);
                    bytes_a += 8.0 * plane_cells * (p.K2 + p.planes);
                    bytes1 += 8.0 * plane_cells * p.planes + 8.0 * L_[0] * rows;
                    bytes2 += 8.0 * L_[0] * rows;
                    ++batch.count;
                }
                if (!batch.count) {
                    break;
                }
                // Pass B2 visits the orientations round-robin (PassBatch).
                batch.min_blocks = *std::min_element(rows_blocks, rows_blocks + batch.count);
                batch.interleaved = batch.count * batch.min_blocks;
                int blocks2 = batch.interleaved;
                for (int g = 0; g < batch.count; ++g) {
                    batch.slot[g].first_b2 = blocks2;
                    blocks2 += rows_blocks[g] - batch.min_blocks;
                }
                auto ev = pass_begin(ctx_);
                cudaError_t err = launch_pass_a(LZ, env_, batch, twz, st);
                pass_end(ctx_, 0, ev, bytes_a);
                ev = pass_begin(ctx_);
                err = err == cudaSuccess ? launch_pass_b1(batch, blocks1, tw1, st) : err;
                pass_end(ctx_, 1, ev, bytes1);
                ev = pass_begin(ctx_);
                err = err == cudaSuccess ? launch_pass_b2(mode, batch, blocks2, tw0, st) : err;
                pass_end(ctx_, 2, ev, bytes2);
                ctx_->launches += 3;
                if (err != cudaSuccess) {
                    cudaGetLastError();
                    return kCuda;
                }
            }
        }
    }
    return kOk;
}

int Pipeline::pages(const std::vector<PageRequest>& requests, std::vector<PageOutcome>& out, PageGoal goal)
{
    refresh_order();
    if (int status = finish_stats()) {
        return status;
    }
    std::vector<std::size_t> ordinary;
    for (std::size_t r = 0; r < requests.size(); ++r) {
        if (!requests[r].low_overlap) {
            ordinary.push_back(r);
        }
    }
    if (ordinary.size() == requests.size()) {
        return ordinary_pages(requests, out, goal);
    }
    out.assign(requests.size(), {});
    if (!ordinary.empty()) {
        std::vector<PageRequest> sub;
        for (std::size_t r : ordinary) {
            sub.push_back(requests[r]);
        }
        std::vector<PageOutcome> sub_out;
        if (int status = ordinary_pages(sub, sub_out, goal)) {
            return status;
        }
        for (std::size_t i = 0; i < ordinary.size(); ++i) {
            out[ordinary[i]] = std::move(sub_out[i]);
        }
    }
    for (std::size_t r = 0; r < requests.size(); ++r) {
        if (requests[r].low_overlap) {
            if (int status = low_overlap_page(requests[r], out[r])) {
                return status;
            }
        }
    }
    return kOk;
}

// A low-overlap page (spectral_pipeline.cpp:1758-1824, mode low_overlap):
// the 32 legal translations after the cursor that are smallest by
// (rounded overlap count, score, z, y, x), over every legal translation, with
// no recount (direct_zero_overlap stays false).  A histogram pass counts the
// translations per rounded overlap; then, from the cursor's count upward,
// each count with translations contributes its certified ordinary-style page
// (candidates: overlap == that count) until 32 entries are gathered.  Counts
// of kOverlapBins - 1 and above share the last bin; a page that would need
// them fails with SPK_SCRATCH_LIMIT.
int Pipeline::low_overlap_page(const PageRequest& req, PageOutcome& out)
{
    out = {};
    const auto& s = slots_[req.slot];
    if (!s.legal[0] || !s.legal[1] || !s.legal[2]) {
        out.certified = true;
        return kOk;
    }
    if (!s.occupied) {
        out.status = kEmptyKernel;
        return kOk;
    }
    constexpr unsigned int kOverlapBins = 4096;
    cudaStream_t st = ctx_->stream;
    int status = kOk;
    auto* hist = static_cast<unsigned int*>(device_buffer(ctx_, "pipe.overlap_hist", kOverlapBins * 4, status));
    auto* meta = static_cast<unsigned long long*>(device_buffer(ctx_, "pipe.overlap_meta", 24, status));
    if (!hist || !meta) {
        return status;
    }
    cudaMemsetAsync(hist, 0, kOverlapBins * 4, st);
    cudaMemsetAsync(meta, 0, 24, st);
    const PlaneWork work { &s, 0, s.legal[2], reinterpret_cast<unsigned long long*>(hist),
                           reinterpret_cast<unsigned int*>(meta + 2), kOverlapBins, meta, meta + 1, 0.f, 0.0, -INFINITY,
                           INFINITY };
    if ((status = run_planes({ work }, PassMode::histogram, false))) {
        return status;
    }
    std::vector<unsigned int> h(kOverlapBins);
    unsigned long long h_meta[3] {};
    cudaMemcpyAsync(h.data(), hist, kOverlapBins * 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(h_meta, meta, 24, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return kCuda;
    }
    std::uint32_t rbits = static_cast<std::uint32_t>(h_meta[1]);
    float rf;
    std::memcpy(&rf, &rbits, 4);
    out.max_integer_residual = rf;
    if (rf >= 0.25f) {
        out.status = kNumeric;  // correlation.cpp:521-528 residual guard
        return kOk;
    }
    // The cursor's overlap is a rounded count held as a double.
    const std::uint32_t first =
        req.has_cursor ? static_cast<std::uint32_t>(std::max(0.0, std::nearbyint(req.cursor.binary_overlap))) : 0u;
    for (std::uint32_t c = first; c < kOverlapBins && out.page.size() < static_cast<std::size_t>(kPageSize); ++c) {
        if (h[c] == 0) {
            continue;
        }
        if (c == kOverlapBins - 1) {
            out.status = kScratchLimit;  // the counts beyond the histogram are not resolved
            return kOk;
        }
        PageRequest bin = req;
        bin.low_overlap = false;
        bin.overlap = c;
        bin.has_cursor = req.has_cursor && c == first;
        std::vector<PageOutcome> bin_out;
        if ((status = ordinary_pages({ bin }, bin_out, PageGoal {}))) {
            return status;
        }
        if (bin_out[0].status) {
            out.status = bin_out[0].status;
            return kOk;
        }
        out.rescored += bin_out[0].rescored;
        out.max_score_error = std::max(out.max_score_error, bin_out[0].max_score_error);
        for (auto& candidate : bin_out[0].page) {
            if (out.page.size() == static_cast<std::size_t>(kPageSize)) {
                break;
            }
            candidate.direct_zero = false;
            out.page.push_back(candidate);
        }
    }
    out.certified = true;
    out.exact_floor = INFINITY;
    return kOk;
}

int Pipeline::ordinary_pages(const std::vector<PageRequest>& requests, std::vector<PageOutcome>& out, PageGoal goal)
{
    const int R = static_cast<int>(requests.size());
    out.assign(R, {});
    if (R == 0) {
        return kOk;
    }
    cudaStream_t st = ctx_->stream;
    int status = kOk;
    // Per request: the planes left to visit and what is known of them.
    struct Lane {
        const KernelSlot* s {};
        double eps {}, floor {};
        double prune_key { INFINITY }, prune_exact { INFINITY };
        int z {}, end {};  // legal planes [z, end) are still to be visited
    };
    std::vector<Lane> lanes(R);
    std::vector<int> runnable;
    int deepest = 1, most_planes = 1;
    long long most_blocks = 1;
    for (int r = 0; r < R; ++r) {
        const auto& s = slots_[requests[r].slot];
        Lane& l = lanes[r];
        l.s = &s;
        if (!s.legal[0] || !s.legal[1] || !s.legal[2]) {
            out[r].certified = true;  // kernel wider than the environment: complete, empty page
            continue;
        }
        if (!s.occupied) {
            out[r].status = kEmptyKernel;
            continue;
        }
        l.eps = approx_epsilon(s) + std::ldexp(1.0, -22);
        l.floor = requests[r].has_cursor ? requests[r].cursor.score - l.eps : -INFINITY;
        l.end = s.legal[2];
        // Planes are pruned only where the FP32 bound keeps every count's
        // residual inside the guard: one beyond it must be seen wherever it is,
        // and the planes that were visited say nothing about the others.
        if (goal.prune && requests[r].overlap == 0 && epsilon_p(s) < 0.25) {
            const double occ = static_cast<double>(s.occupied);
            feasible_planes(s, l.z, l.end);
            l.prune_exact = .35 * s.most_proximity / occ + 1e-12;
            // Keys carry the FP32 error and are rounded down to FP32.
            l.prune_key = .35 * (s.most_proximity + 2 * epsilon_p(s)) / occ + 4e-7;
        }
        deepest = std::max(deepest, s.K[2]);
        most_planes = std::max(most_planes, s.legal[2]);
        most_blocks = std::max(most_blocks, (static_cast<long long>(s.legal[1]) * s.legal[2] + 15) / 16);
        runnable.push_back(r);
    }
    if (runnable.empty()) {
        return kOk;
    }
    // Each pass-B2 block emits the keys of its histogram bins up to the one
    // where 64 accumulate (about 64), below the pruning bound, so 64 keys per
    // block cover a request; only heavy exact ties could exceed that, and an
    // overflowing page is then left uncertified and widened.
    const int exact = goal.full ? kExactPerOrientation : kHeadCandidates;
    const int per = exact + 1;
    unsigned int chunks = static_cast<unsigned int>(std::min<long long>(
        kMaxKeyChunks, std::max<long long>(1, (most_blocks * 64 + kKeyCapacity - 1) / kKeyCapacity)));
    // One result block, read back in one copy: bound, residual and key count
    // per request, then per candidate its key, exact count and exact sum, then
    // the range flag.
    const std::size_t words = static_cast<std::size_t>(R) * (3 + 3 * per) + 1;
    auto* result = static_cast<unsigned long long*>(device_buffer(ctx_, "pipe.result", words * 8, status));
    auto* host = static_cast<unsigned long long*>(host_buffer(ctx_, "pipe.result", words * 8, status));
    const std::size_t job_bytes = R * sizeof(ExactJob);
    auto* d_jobs = static_cast<char*>(device_buffer(ctx_, "pipe.jobs", job_bytes + R * sizeof(int), status));
    auto* h_jobs = static_cast<char*>(host_buffer(ctx_, "pipe.jobs", job_bytes + R * sizeof(int), status));
    const double* proximity = table(status);
    if (!result || !host || !d_jobs || !h_jobs || !proximity) {
        return status;
    }
    if (ctx_->cap_bytes) {
        // One orientation's intermediate comes first (run_planes takes room for
        // more where there is some), then keys in up to a quarter of what is left:
        // a shorter range, which may overflow.
        if (!device_buffer(ctx_, "pipe.inter", sizeof(float2) * L_[0] * L_[1] * most_planes, status)) {
            return status;
        }
        const std::uint64_t chunk_bytes = static_cast<std::uint64_t>(R) * (kKeyCapacity + per) * 8;
        while (chunks > 1 && chunks * chunk_bytes > room_for(ctx_, "pipe.keys") / 4) {
            chunks /= 2;
        }
    }
    // The first stage's winners (the heads' merge has one stage).
    unsigned long long* partial = nullptr;
    if (per > kFewKeys && !(partial = static_cast<unsigned long long*>(device_buffer(
                                ctx_, "pipe.partial", static_cast<std::size_t>(R) * chunks * per * 8, status)))) {
        return status;
    }
    unsigned long long* keys = nullptr;
    while (!keys) {  // where memory is short, a shorter range as well
        keys = static_cast<unsigned long long*>(
            device_buffer(ctx_, "pipe.keys", static_cast<std::size_t>(R) * chunks * kKeyCapacity * 8, status));
        if (!keys && chunks == 1) {
            return status;
        }
        chunks = keys ? chunks : chunks / 2;
    }
    status = kOk;
    const unsigned int cap = chunks * kKeyCapacity;
    unsigned long long* tau = result;
    unsigned long long* resid = tau + R;
    unsigned long long* count = resid + R;
    unsigned long long* selected = count + R;
    auto* counts_out = reinterpret_cast<long long*>(selected + static_cast<std::size_t>(R) * per);
    auto* p_out = reinterpret_cast<double*>(counts_out + static_cast<std::size_t>(R) * per);
    auto* range_error = reinterpret_cast<int*>(p_out + static_cast<std::size_t>(R) * per);
    auto* jobs = reinterpret_cast<ExactJob*>(d_jobs);
    auto* d_lanes = reinterpret_cast<int*>(d_jobs + job_bytes);
    for (int r = 0; r < R; ++r) {
        const KernelSlot& s = *lanes[r].s;
        const ExactJob job { s.ones, static_cast<int>(s.occupied), std::max(s.legal[0], 1), std::max(s.legal[1], 1) };
        std::memcpy(h_jobs + r * sizeof(ExactJob), &job, sizeof(job));
    }
    page_init_kernel<<<(R + 127) / 128, 128, 0, st>>>(tau, resid, count, R, range_error);
    ctx_->launches++;
    // First round: the planes of one slab from the lowest plane wanted, in the
    // shortest slab that leaves enough of them beside the deepest kernel: for
    // whole pages half its depth and 16, for the heads, which the lowest few
    // planes mostly hold, a quarter and 12; or every plane where one slab for all
    // costs little more.  Later rounds visit twice as many planes as the one
    // before.  Planes that heads need, and a step's time by the planes visited
    // first: 24 cuboids on a 66^3 window 2 to 5 of 50 (47 planes 297 us, 15 planes
    // 278 us); 32 blobs of 25 planes on a 256^3 window 28 to 31 of 231 (40 planes; 8
    // would take three rounds).  Requests that are not pruned visit every plane
    // in the first round.
    int step = INT32_MAX;
    if (goal.prune) {
        int n = 0, range = 0;
        const int* lengths = slab_lengths(n);
        for (int r : runnable) {
            range = std::max(range, lanes[r].end - lanes[r].z);
        }
        int shortest = 0;
        for (int i = 0; i < n && step == INT32_MAX; ++i) {
            const int W = lengths[i] - deepest + 1;
            if (W >= (goal.full ? std::max(16, deepest / 2) : std::max(12, deepest / 4))) {
                step = W;
                shortest = lengths[i];
            }
        }
        for (int i = 0; i < n; ++i) {
            if (lengths[i] - deepest + 1 >= range && slab_cost(lengths[i]) <= 1.5 * slab_cost(shortest)) {
                step = INT32_MAX;
            }
        }
    }
    std::vector<int> active = runnable;
    bool first = true;
    while (!active.empty()) {
        int from = INT32_MAX;
        for (int r : active) {
            from = std::min(from, lanes[r].z < lanes[r].end ? lanes[r].z : INT32_MAX);
        }
        const int to = from > INT32_MAX - step ? INT32_MAX : from + step;
        std::vector<PlaneWork> work;
        for (int r : active) {
            Lane& l = lanes[r];
            const int z1 = std::isinf(l.prune_key) ? l.end : std::min(l.end, to);
            if (l.z < z1) {
                work.push_back({ l.s, l.z, z1, keys + static_cast<std::size_t>(r) * cap,
                                 reinterpret_cast<unsigned int*>(count + r), cap, tau + r, resid + r,
                                 static_cast<float>(requests[r].overlap), 0.0, l.floor, l.prune_key });
                l.z = z1;
            }
        }
        if ((status = run_planes(work, PassMode::select, !first))) {
            return status;
        }
        std::memcpy(h_jobs + job_bytes, active.data(), active.size() * sizeof(int));
        cudaMemcpyAsync(d_jobs + (first ? 0 : job_bytes), h_jobs + (first ? 0 : job_bytes),
                        (first ? job_bytes : 0) + active.size() * sizeof(int), cudaMemcpyHostToDevice, st);
        first = false;
        const int n = static_cast<int>(active.size());
        auto ev = pass_begin(ctx_);
        if (per <= kFewKeys) {
            merge_heads_kernel<<<n, kHeadThreads, 0, st>>>(keys, cap, count, d_lanes, per, selected);
        }
        else {
            merge_chunk_kernel<<<dim3(chunks, n), 1024, 0, st>>>(keys, cap, count, d_lanes, per, partial);
            static_assert(kMaxKeyChunks <= 64, "merge_lists_kernel holds one list head per thread of 64");
            merge_lists_kernel<<<n, 64, 0, st>>>(partial, d_lanes, static_cast<int>(chunks), per, selected);
            ctx_->launches++;
        }
        exact_kernel<<<n * exact, kExactThreads, 0, st>>>(selected, jobs, d_lanes, per, exact, occ_, d2_, proximity,
                                                          E_[0], E_[1], counts_out, p_out, range_error);
        pass_end(ctx_, 3, ev);
        ctx_->launches += 2;
        cudaMemcpyAsync(host, result, words * 8, cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) {
            cudaGetLastError();
            return kCuda;
        }
        if (static_cast<std::uint32_t>(host[words - 1])) {
            return kNumericRange;
        }
        const auto* h_sel = host + 3 * static_cast<std::size_t>(R);
        const auto* h_count = reinterpret_cast<const long long*>(h_sel + static_cast<std::size_t>(R) * per);
        const auto* h_p = reinterpret_cast<const double*>(h_count + static_cast<std::size_t>(R) * per);
        std::vector<int> again;
        for (int r : active) {
            const auto& req = requests[r];
            const Lane& l = lanes[r];
            const KernelSlot& s = *l.s;
            PageOutcome& o = out[r];
            o = {};
            const auto rbits = static_cast<std::uint32_t>(host[R + r]);
            float rf;
            std::memcpy(&rf, &rbits, 4);
            o.max_integer_residual = rf;
            if (rf >= 0.25f) {
                o.status = kNumeric;  // correlation.cpp:521-528 residual guard
                continue;
            }
            const auto n_r = static_cast<unsigned int>(host[2 * R + r]);
            const unsigned long long tau_r = host[r];
            std::vector<Candidate> all;
            double max_error = 0;
            const std::int64_t legal_first[3] = { env_first_[0] - s.first[0], env_first_[1] - s.first[1],
                                                  env_first_[2] - s.first[2] };
            const int m = static_cast<int>(std::min<unsigned int>(n_r, exact));
            for (int i = 0; i < m; ++i) {
                const unsigned long long key = h_sel[static_cast<std::size_t>(r) * per + i];
                const long long overlap = h_count[static_cast<std::size_t>(r) * per + i];
                const double p = h_p[static_cast<std::size_t>(r) * per + i];
                const unsigned int index = static_cast<unsigned int>(key & 0xffffffffULL);
                Candidate c {};
                c.t[0] = legal_first[0] + index % s.legal[0];
                c.t[1] = legal_first[1] + (index / s.legal[0]) % s.legal[1];
                c.t[2] = legal_first[2] + index / (static_cast<unsigned int>(s.legal[0]) * s.legal[1]);
                c.orientation = s.orientation;
                c.score = score(s, c.t, p);
                c.binary_overlap = static_cast<double>(overlap);
                c.direct_zero = overlap == 0;
                const double approx = decode_key_score(key);
                max_error = std::max(max_error, std::fabs(approx - c.score));
                ++o.rescored;
                if (overlap != static_cast<long long>(req.overlap)) {
                    continue;  // the reference's FFT rounding never admits these
                }
                if (req.has_cursor && !rank_less(req.cursor, c)) {
                    continue;
                }
                all.push_back(c);
            }
            o.max_score_error = max_error;
            if (max_error > l.eps) {
                o.status = kNumeric;  // the FP32 bound did not hold: fail closed
                continue;
            }
            std::sort(all.begin(), all.end(), rank_less);
            if (all.size() > static_cast<std::size_t>(kPageSize)) {
                all.resize(kPageSize);
            }
            unsigned long long excluded = kEmptyKey;
            if (n_r > cap) {
                excluded = 0;  // overflowed: nothing can be certified
            }
            else {
                if (n_r > static_cast<unsigned int>(exact)) {
                    excluded = h_sel[static_cast<std::size_t>(r) * per + exact];
                }
                excluded = std::min(excluded, tau_r);
            }
            // Every score left out so far is above this, and every score of
            // the planes not yet visited above `above`.
            const double visited = excluded == kEmptyKey ? INFINITY
                                   : excluded == 0      ? -INFINITY
                                                        : decode_key_score(excluded) - l.eps;
            const double above = l.z < l.end ? s.t65_host[l.z] - l.prune_exact : INFINITY;
            o.exact_floor = std::min(visited, above);
            o.certified = o.exact_floor == INFINITY ||
                          (all.size() == static_cast<std::size_t>(kPageSize) && o.exact_floor > all.back().score);
            o.page = std::move(all);
            // Starting bound for a threshold pass over a page that is not full:
            // the lowest excluded approximate score, or the last rescored one.
            double start = m > 0 ? decode_key_score(h_sel[static_cast<std::size_t>(r) * per + m - 1]) : -INFINITY;
            if (excluded != kEmptyKey && excluded != 0) {
                start = std::max(start, decode_key_score(excluded));
            }
            o.excluded_score = start;
            if (debug_) {
                std::fprintf(stderr, "page r=%d n=%u tau=%llx m=%d planes=%d/%d page=%zu certified=%d eps=%g err=%g\n", r,
                             n_r, tau_r, m, l.z, l.end, o.page.size(), o.certified ? 1 : 0, l.eps, max_error);
            }
            // A whole page needs the planes above while its last entry, or a
            // missing one, could come from there.
            if (l.z < l.end && goal.full &&
                (o.page.size() < static_cast<std::size_t>(kPageSize) || above <= o.page.back().score)) {
                again.push_back(r);
            }
        }
        if (!goal.full) {
            // The merge needs an orientation's planes above only while a
            // candidate there could precede the best exact head so far.
            double best = INFINITY;
            for (int r : runnable) {
                const PageOutcome& o = out[r];
                if (!o.status && !o.page.empty() && o.page.front().score <= o.exact_floor) {
                    best = std::min(best, o.page.front().score);
                }
            }
            for (int r : runnable) {
                const Lane& l = lanes[r];
                if (!out[r].status && l.z < l.end && l.s->t65_host[l.z] - l.prune_exact <= best) {
                    again.push_back(r);
                }
            }
        }
        active = std::move(again);
        step = step > INT32_MAX / 2 ? INT32_MAX : 2 * step;
    }
    for (int r : runnable) {
        if (!out[r].status) {
            ++stat_pages;
            stat_first_certified += out[r].certified ? 1 : 0;
        }
        stat_rescored += out[r].rescored;
    }
    // Threshold passes for every uncertified page (each recomputes that
    // orientation): collect every candidate whose approximate score is <= T,
    // rescore all of them exactly, and widen T until the page is certified.
    for (int r = 0; r < R && goal.full; ++r) {
        auto& o = out[r];
        if (o.status || o.certified) {
            continue;
        }
        const auto& req = requests[r];
        const Lane& l = lanes[r];
        const KernelSlot& s = *l.s;
        const std::int64_t legal_first[3] = { env_first_[0] - s.first[0], env_first_[1] - s.first[1],
                                              env_first_[2] - s.first[2] };
        // Everything left out of a threshold pass has approximate score > T, so
        // exact score > T - eps; T = S32 + 2 eps certifies a page whose 32nd
        // entry did not get worse.
        double threshold = o.page.size() == static_cast<std::size_t>(kPageSize) ? o.page.back().score + 2 * l.eps
                                                                                : o.excluded_score + 2 * l.eps;
        double widen = std::max(4 * l.eps, 1e-6);
        unsigned int tcap = kKeyCapacity;
        auto* meta = static_cast<unsigned long long*>(device_buffer(ctx_, "pipe.tmeta", 24, status));
        if (!meta) {
            return status;
        }
        for (int attempt = 0; attempt < 24 && !o.certified; ++attempt) {
            auto* tkeys = static_cast<unsigned long long*>(device_buffer(ctx_, "pipe.tkeys", tcap * 8ULL, status));
            if (!tkeys) {
                return status;
            }
            cudaMemsetAsync(meta, 0, 24, st);
            const PlaneWork work { &s, 0, s.legal[2], tkeys, reinterpret_cast<unsigned int*>(meta + 2), tcap, meta,
                                   meta + 1, static_cast<float>(req.overlap), threshold, l.floor, INFINITY };
            if ((status = run_planes({ work }, PassMode::threshold, false))) {
                return status;
            }
            ++stat_threshold_passes;
            unsigned long long h[3];
            cudaMemcpyAsync(h, meta, 24, cudaMemcpyDeviceToHost, st);
            if (cudaStreamSynchronize(st) != cudaSuccess) {
                return kCuda;
            }
            const unsigned int n = static_cast<unsigned int>(h[2] & 0xffffffffULL);
            const unsigned long long total = h[0];
            if (n > tcap) {
                tcap = n + 1024;
                --attempt;
                continue;
            }
            std::vector<Candidate> all;
            if (n) {
                auto* tcount = static_cast<long long*>(device_buffer(ctx_, "pipe.tcount", n * 8ULL, status));
                auto* tp = static_cast<double*>(device_buffer(ctx_, "pipe.tp", n * 8ULL, status));
                if (!tcount || !tp) {
                    return status;
                }
                exact_kernel<<<n, kExactThreads, 0, st>>>(tkeys, jobs + r, nullptr, static_cast<int>(n),
                                                          static_cast<int>(n), occ_, d2_, proximity, E_[0], E_[1],
                                                          tcount, tp, range_error);
                ctx_->launches++;
                std::vector<unsigned long long> hk(n);
                std::vector<long long> cnt(n);
                std::vector<double> pv(n);
                cudaMemcpyAsync(hk.data(), tkeys, n * 8ULL, cudaMemcpyDeviceToHost, st);
                cudaMemcpyAsync(cnt.data(), tcount, n * 8ULL, cudaMemcpyDeviceToHost, st);
                cudaMemcpyAsync(pv.data(), tp, n * 8ULL, cudaMemcpyDeviceToHost, st);
                if (cudaStreamSynchronize(st) != cudaSuccess) {
                    return kCuda;
                }
                for (unsigned int i = 0; i < n; ++i) {
                    const unsigned int index = static_cast<unsigned int>(hk[i] & 0xffffffffULL);
                    Candidate c {};
                    c.t[0] = legal_first[0] + index % s.legal[0];
                    c.t[1] = legal_first[1] + (index / s.legal[0]) % s.legal[1];
                    c.t[2] = legal_first[2] + index / (static_cast<unsigned int>(s.legal[0]) * s.legal[1]);
                    c.orientation = s.orientation;
                    c.score = score(s, c.t, pv[i]);
                    c.binary_overlap = static_cast<double>(cnt[i]);
                    c.direct_zero = cnt[i] == 0;
                    o.max_score_error = std::max(o.max_score_error, std::fabs(decode_key_score(hk[i]) - c.score));
                    ++o.rescored;
                    if (cnt[i] != static_cast<long long>(req.overlap) || (req.has_cursor && !rank_less(req.cursor, c))) {
                        continue;
                    }
                    all.push_back(c);
                }
            }
            if (o.max_score_error > l.eps) {
                o.status = kNumeric;
                break;
            }
            std::sort(all.begin(), all.end(), rank_less);
            if (all.size() > static_cast<std::size_t>(kPageSize)) {
                all.resize(kPageSize);
            }
            const bool complete = n == total;
            const bool full_page = all.size() == static_cast<std::size_t>(kPageSize);
            o.page = std::move(all);
            o.threshold_pass = true;
            if (complete || (full_page && o.page.back().score < threshold - l.eps)) {
                o.certified = true;
                o.exact_floor = complete ? INFINITY : threshold - l.eps;
                break;
            }
            if (debug_) {
                std::fprintf(stderr, "threshold r=%d T=%.17g n=%u total=%llu page=%zu\n", r, threshold, n, total,
                             o.page.size());
            }
            threshold = full_page ? std::max(o.page.back().score + 2 * l.eps, threshold + widen) : threshold + widen;
            widen *= 4;
        }
        if (!o.certified && !o.status) {
            o.status = kScratchLimit;
        }
    }
    return kOk;
}

}  // namespace spk
