// Column passes along y: pass B1 (inverse, over a slab's valid planes, legal
// rows kept) and the forward transform of environment and kernel planes.  Both
// in place, 16 adjacent columns per block, bound by memory (L2 for a slab's
// intermediate, HBM for a 256^2 environment's planes).
#include "fft_plan.cuh"
#include "keys.cuh"
#include "passes.hpp"

namespace spk {

namespace {

template <int L1>
constexpr std::size_t column_smem()
{
    return sizeof(ColumnRoots<Plan<L1>>) + static_cast<std::size_t>(L1) * kColumns * sizeof(float2);
}

// Resident blocks the registers are limited for: 1024 threads per SM keep
// enough loads in flight (92 registers and two blocks of 256 cost pass B1 a
// fifth); lines of more than 24 values per thread would spill.
template <int L1>
constexpr int kColumnBlocks = Plan<L1>::R1 > 24 ? 1 : 1024 / (kColumns * Plan<L1>::T);

// ROW: the row length L0 where it equals L1 (strides are then immediate
// offsets, which frees registers and issue slots), else 0.
template <int L1, int ROW>
__global__ void __launch_bounds__(kColumns* Plan<L1>::T, kColumnBlocks<L1>)
    pass_b1_kernel(const __grid_constant__ PassBatch batch, const float2* __restrict__ roots)
{
    using P = Plan<L1>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto& w = *reinterpret_cast<ColumnRoots<P>*>(smem_raw);
    float2* buf = reinterpret_cast<float2*>(smem_raw + sizeof(ColumnRoots<P>));
    int g = 0;
    while (g + 1 < batch.count && batch.slot[g + 1].first_b1 <= static_cast<int>(blockIdx.x)) {
        ++g;
    }
    const PassSlot& s = batch.slot[g];
    const int local = static_cast<int>(blockIdx.x) - s.first_b1;
    const int L0 = ROW ? ROW : batch.L0;
    const int groups = (L0 + kColumns - 1) / kColumns;
    const int plane = local / groups;
    if (batch.bound_known && plane_pruned(s.t65[plane], s.prune, *s.tau)) {
        return;  // uniform: nothing writes the bound during this launch
    }
    const int j = threadIdx.x % kColumns, t = threadIdx.x / kColumns;
    const int kx = (local - plane * groups) * kColumns + j;
    const bool inside = kx < L0;
    const unsigned row = static_cast<unsigned>(L0);  // 32-bit offsets within a plane
    // Columns past the row load its last one, which they do not store.
    float2* data = s.inter + static_cast<long long>(plane) * (L1 * L0) + min(kx, L0 - 1);
    // The loads go out before the root table's round trip.
    float2 a[P::R1], b[P::I2][P::R2];
#pragma unroll
    for (int i = 0; i < P::I2; ++i) {
        const int k = t + P::T * i;
        const float2* from = data + (P::has_b(k) ? k : 0) * row;
#pragma unroll
        for (int n = 0; n < P::R2; ++n) {
            b[i][n] = from[P::R1 * n * row];
        }
    }
    load_roots(w, roots);
    __syncthreads();
    column_inverse<P>(b, a, buf, w, j, t);
    if (inside && P::has_a(t)) {
        float2* to = data + t * row;
        const int left = s.legal_y - t;
#pragma unroll
        for (int n = 0; n < P::R1; ++n) {
            if (P::R2 * n < left) {
                to[P::R2 * n * row] = a[n];
            }
        }
    }
}

template <int L1, int ROW>
__global__ void __launch_bounds__(kColumns* Plan<L1>::T, kColumnBlocks<L1>)
    forward_y_kernel(float2* __restrict__ planes, int row_length, int rows, const float2* __restrict__ roots,
                     const EdtBox* __restrict__ region)
{
    using P = Plan<L1>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto& w = *reinterpret_cast<ColumnRoots<P>*>(smem_raw);
    float2* buf = reinterpret_cast<float2*>(smem_raw + sizeof(ColumnRoots<P>));
    const int L0 = ROW ? ROW : row_length;
    const int groups = (L0 + kColumns - 1) / kColumns;
    const int plane = static_cast<int>(blockIdx.x) / groups;
    if (region && (plane < region->lo[2] || plane >= region->hi[2])) {
        return;
    }
    const int j = threadIdx.x % kColumns, t = threadIdx.x / kColumns;
    const int kx = (static_cast<int>(blockIdx.x) - plane * groups) * kColumns + j;
    const bool inside = kx < L0;
    const unsigned row = static_cast<unsigned>(L0);
    float2* data = planes + static_cast<long long>(plane) * (L1 * L0) + kx;
    float2 a[P::R1], b[P::I2][P::R2];
#pragma unroll
    for (int n = 0; n < P::R1; ++n) {
        const int y = P::R2 * n + t;
        a[n] = inside && P::has_a(t) && y < rows ? data[y * row] : make_float2(0.f, 0.f);
    }
    load_roots(w, roots);
    __syncthreads();
    column_forward<P>(a, b, buf, w, j, t);
#pragma unroll
    for (int i = 0; i < P::I2; ++i) {
        const int k = t + P::T * i;
        if (inside && P::has_b(k)) {
#pragma unroll
            for (int n = 0; n < P::R2; ++n) {
                data[k * row + P::R1 * n * row] = b[i][n];
            }
        }
    }
}

template <int L1>
void configure()
{
    static std::once_flag configured[64];
    once_per_device(configured, [] {
        constexpr int smem = static_cast<int>(column_smem<L1>());
        cudaFuncSetAttribute(pass_b1_kernel<L1, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaFuncSetAttribute(pass_b1_kernel<L1, L1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaFuncSetAttribute(forward_y_kernel<L1, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaFuncSetAttribute(forward_y_kernel<L1, L1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    });
}

}  // namespace

cudaError_t launch_pass_b1(const PassBatch& batch, int blocks, const float2* roots, cudaStream_t stream)
{
    switch (batch.L1) {
#define SPK_CASE(L)                                                                                               \
    case L: {                                                                                                     \
        configure<L>();                                                                                           \
        const auto kernel = batch.L0 == L ? pass_b1_kernel<L, L> : pass_b1_kernel<L, 0>;                          \
        kernel<<<blocks, kColumns * Plan<L>::T, column_smem<L>(), stream>>>(batch, roots);                        \
        break;                                                                                                    \
    }
        SPK_AXIS_LENGTHS(SPK_CASE)
#undef SPK_CASE
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_forward_y(int L0, int L1, float2* data, int rows, int planes, const float2* roots,
                             const EdtBox* region, cudaStream_t stream)
{
    const int blocks = planes * ((L0 + kColumns - 1) / kColumns);
    switch (L1) {
#define SPK_CASE(L)                                                                                               \
    case L: {                                                                                                     \
        configure<L>();                                                                                           \
        const auto kernel = L0 == L ? forward_y_kernel<L, L> : forward_y_kernel<L, 0>;                            \
        kernel<<<blocks, kColumns * Plan<L>::T, column_smem<L>(), stream>>>(data, L0, rows, roots, region);       \
        break;                                                                                                    \
    }
        SPK_AXIS_LENGTHS(SPK_CASE)
#undef SPK_CASE
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace spk
