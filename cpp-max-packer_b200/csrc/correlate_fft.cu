// Transform passes of the FP64 full-range correlations.
//
// The packed field Z = E + iK lives on the grid L >= E + K - 1 as [z][y][x].
// Five passes, each a register transform L = r1 x r2 with one exchange through
// shared memory per direction:
//   rows_forward     reads the inputs, x transform; only rows holding input
//   columns<fwd>     y transform of the planes holding input
//   pairs            z transform of a column (kx, ky) and of its mirror
//                    (-kx, -ky), the product E^ conj K^ that needs both, and
//                    the z transform back
//   columns<inv>     y transform back
//   rows_extract     x transform back and the output checks
// The field is read and written in place, so a correlation moves it four times
// (the first three passes touch only the planes and rows that the inputs
// fill).  W is Hermitian: the mirror column's z transform back is the
// conjugate of the first one's and is not computed again.
//
// At 256^3 with inputs of half that extent (268 MB of field) the passes take 51,
// 55, 116, 72 and 93 us and move 1.4 GB in all; the FP64 pipe and memory share
// the time (six staged passes with separate packing, product and extraction
// kernels: 1,820 us).  The radices are chosen at run time (18 of them cover
// every 2^a 3^b 5^c <= 512 as a pair), one switch per phase, because 50 lengths
// x 3 axes as template instances would be 300 kernels for the same traffic.
// Radix classes keep the registers of long lines (r1 up to 32) away from the
// others.
#include <algorithm>
#include <mutex>

#include "context.hpp"
#include "correlate_checks.cuh"
#include "fft_plan.cuh"

namespace spk {
namespace {

using C = double2;

// Adjacent lines per block: 128 contiguous bytes.
constexpr int kLines = 128 / static_cast<int>(sizeof(C));

// Radix classes: r1 <= 16, <= 20, <= 32.
template <int CLASS>
constexpr int kMaxThreads = kLines * (CLASS == 0 ? 16 : CLASS == 1 ? 20 : 32);
// Blocks per SM that the registers of a class are held to.
template <int CLASS>
constexpr int kMinBlocks = CLASS == 0 ? 4 : CLASS == 1 ? 3 : 1;
template <int CLASS>
constexpr int kMinPairBlocks = CLASS == 0 ? 3 : CLASS == 1 ? 2 : 1;

template <int N>
using Int = std::integral_constant<int, N>;

// f(Int<r>) for the first radix of a plan.
template <int CLASS, class F>
__device__ __forceinline__ void with_r1(int r, F&& f)
{
    if constexpr (CLASS == 2) {
        switch (r) {
        case 24: return f(Int<24> {});
        case 25: return f(Int<25> {});
        case 27: return f(Int<27> {});
        default: return f(Int<32> {});
        }
    }
    else if constexpr (CLASS == 1) {
        if (r == 18) {
            return f(Int<18> {});
        }
        return f(Int<20> {});
    }
    else {
        switch (r) {
        case 2: return f(Int<2> {});
        case 3: return f(Int<3> {});
        case 4: return f(Int<4> {});
        case 5: return f(Int<5> {});
        case 6: return f(Int<6> {});
        case 8: return f(Int<8> {});
        case 9: return f(Int<9> {});
        case 10: return f(Int<10> {});
        case 12: return f(Int<12> {});
        case 15: return f(Int<15> {});
        default: return f(Int<16> {});
        }
    }
}
// And for the second.
template <int CLASS, class F>
__device__ __forceinline__ void with_r2(int r, F&& f)
{
    if constexpr (CLASS > 0) {
        switch (r) {
        case 5: return f(Int<5> {});
        case 9: return f(Int<9> {});
        case 10: return f(Int<10> {});
        case 12: return f(Int<12> {});
        case 15: return f(Int<15> {});
        case 16: return f(Int<16> {});
        case 18: return f(Int<18> {});
        default: return f(Int<20> {});
        }
    }
    else {
        switch (r) {
        case 1: return f(Int<1> {});
        case 2: return f(Int<2> {});
        case 3: return f(Int<3> {});
        case 4: return f(Int<4> {});
        case 5: return f(Int<5> {});
        case 6: return f(Int<6> {});
        case 8: return f(Int<8> {});
        case 9: return f(Int<9> {});
        case 10: return f(Int<10> {});
        case 12: return f(Int<12> {});
        case 15: return f(Int<15> {});
        default: return f(Int<16> {});
        }
    }
}

__device__ __forceinline__ void stage_roots(C* to, const C* __restrict__ from, int L)
{
    for (int i = threadIdx.x; i < L; i += blockDim.x) {
        to[i] = from[i];
    }
}

// A line's exchange buffer in the row passes: [k][t] with an odd pitch, so
// that neither the writes (lanes along t) nor the reads (lanes along k)
// conflict.
__host__ __device__ __forceinline__ int row_pitch(AxisPlan p) { return p.r2 | 1; }

// First phase of a row transform: thread `t` < r2 of a line loads its values
// r2 n + t, n < r1, with `load`, and leaves them in the exchange buffer.
template <bool INV, int CLASS, class LOAD>
__device__ __forceinline__ void row_first(AxisPlan p, C* line, const C* roots, int t, bool holds, LOAD&& load)
{
    if (holds && t < p.r2) {
        with_r1<CLASS>(p.r1, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            C a[R];
#pragma unroll
            for (int n = 0; n < R; ++n) {
                a[n] = load(p.r2 * n + t);
            }
            dft<R, INV>(a);
            const int pitch = row_pitch(p);
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const C w = roots[t * k];
                line[k * pitch + t] = k == 0 ? a[k] : INV ? cmulconj(a[k], w) : cmul(a[k], w);
            }
        });
    }
}
// Second phase: thread `k` < r1 gives the values k + r1 n, n < r2, to `store`.
template <bool INV, int CLASS, class STORE>
__device__ __forceinline__ void row_second(AxisPlan p, const C* line, int k, bool holds, STORE&& store)
{
    if (holds && k < p.r1) {
        with_r2<CLASS>(p.r2, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            C b[R];
            const C* from = line + k * row_pitch(p);
#pragma unroll
            for (int n = 0; n < R; ++n) {
                b[n] = from[n];
            }
            dft<R, INV>(b);
#pragma unroll
            for (int n = 0; n < R; ++n) {
                store(k + p.r1 * n, b[n]);
            }
        });
    }
}

template <typename E, int CLASS>
__global__ void __launch_bounds__(kMaxThreads<CLASS>, kMinBlocks<CLASS>)
    rows_forward_kernel(C* __restrict__ z, AxisPlan p, int Ly, int rows_y, int rows,
                        const C* __restrict__ table, CorrelationShape s, const E* __restrict__ env,
                        const std::uint8_t* __restrict__ ker)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* roots = reinterpret_cast<C*>(smem_raw);
    const int j = threadIdx.x / p.r1, t = threadIdx.x - j * p.r1;
    C* line = roots + p.L + j * p.r1 * row_pitch(p);
    const int row = blockIdx.x * kLines + j;
    const bool holds = j < kLines && row < rows;
    const int zz = row / rows_y, y = row - zz * rows_y;
    stage_roots(roots, table, p.L);
    __syncthreads();
    const int ex = y < s.env[1] && zz < s.env[2] ? s.env[0] : 0;
    const int kx = y < s.ker[1] && zz < s.ker[2] ? s.ker[0] : 0;
    const E* e = env + static_cast<long long>(s.env[0]) * (y + static_cast<long long>(s.env[1]) * zz);
    const std::uint8_t* k = ker + static_cast<long long>(s.ker[0]) * (y + static_cast<long long>(s.ker[1]) * zz);
    row_first<false, CLASS>(p, line, roots, t, holds, [&](int x) {
        return cmake<C>(x < ex ? static_cast<double>(e[x]) : 0.0, x < kx ? static_cast<double>(k[x]) : 0.0);
    });
    __syncthreads();
    C* to = z + static_cast<long long>(p.L) * (y + static_cast<long long>(Ly) * zz);
    row_second<false, CLASS>(p, line, t, holds, [&](int x, C v) { to[x] = v; });
}

// y transform of 128-byte groups of columns: grid (groups of x, planes).
// Forward: plane blockIdx.y, rows `fill` and up are zero.  Inverse: the planes
// that outputs read, which begin at `first` and wrap.
template <bool INV, int CLASS>
__global__ void __launch_bounds__(kMaxThreads<CLASS>, kMinBlocks<CLASS>)
    columns_kernel(C* __restrict__ z, int Lx, AxisPlan p, int Lz, int first, int fill,
                   const C* __restrict__ table)
{
    constexpr int G = kLines;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* roots = reinterpret_cast<C*>(smem_raw);
    C* buf = roots + (p.L + G - 1) / G * G;
    const int j = threadIdx.x % G, t = threadIdx.x / G;
    const int x = blockIdx.x * G + j;
    const bool holds = x < Lx;
    C* column = z + static_cast<long long>(wrap(first + static_cast<int>(blockIdx.y), Lz)) * Lx * p.L + x;
    stage_roots(roots, table, p.L);
    __syncthreads();
    if (holds && t < p.r2) {
        with_r1<CLASS>(p.r1, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            C a[R];
#pragma unroll
            for (int n = 0; n < R; ++n) {
                const int y = p.r2 * n + t;
                a[n] = y < fill ? column[y * Lx] : cmake<C>(0, 0);
            }
            dft<R, INV>(a);
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const C w = roots[t * k];
                buf[(k * p.r2 + t) * G + j] = k == 0 ? a[k] : INV ? cmulconj(a[k], w) : cmul(a[k], w);
            }
        });
    }
    __syncthreads();
    if (holds && t < p.r1) {
        with_r2<CLASS>(p.r2, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            C b[R];
#pragma unroll
            for (int n = 0; n < R; ++n) {
                b[n] = buf[(t * R + n) * G + j];
            }
            dft<R, INV>(b);
#pragma unroll
            for (int n = 0; n < R; ++n) {
                column[(t + p.r1 * n) * Lx] = b[n];
            }
        });
    }
}

// z transform, product and transform back of the columns (kx, ky), 2 kx <= Lx,
// with their mirrors: grid (groups of kx, ky).  Where kx is its own mirror,
// the pair belongs to the smaller ky: every column is read and written by one
// thread group only.
template <int CLASS>
__global__ void __launch_bounds__(kMaxThreads<CLASS>, kMinPairBlocks<CLASS>)
    pairs_kernel(C* __restrict__ z, int Lx, int Ly, AxisPlan p, int fill, const C* __restrict__ table,
                 double scale)
{
    constexpr int G = kLines;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* roots = reinterpret_cast<C*>(smem_raw);
    C* buf = roots + (p.L + G - 1) / G * G;
    C* mirror_buf = buf + p.L * G;
    const int j = threadIdx.x % G, t = threadIdx.x / G;
    const int kx = blockIdx.x * G + j, ky = blockIdx.y;
    const int mx = kx == 0 ? 0 : Lx - kx, my = ky == 0 ? 0 : Ly - ky;
    const bool holds = 2 * kx <= Lx && !(kx == mx && ky > my);
    const bool self = kx == mx && ky == my;
    const int plane = Lx * Ly;
    C* column = z + ky * Lx + kx;
    C* mirror = z + my * Lx + mx;
    stage_roots(roots, table, p.L);
    __syncthreads();
    if (holds && t < p.r2) {
        with_r1<CLASS>(p.r1, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
#pragma unroll 1
            for (int side = 0; side < 2; ++side) {
                const C* from = side ? mirror : column;
                C* to = side ? mirror_buf : buf;
                C a[R];
#pragma unroll
                for (int n = 0; n < R; ++n) {
                    const int zz = p.r2 * n + t;
                    a[n] = zz < fill ? from[zz * plane] : cmake<C>(0, 0);
                }
                dft<R, false>(a);
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    to[(k * p.r2 + t) * G + j] = k == 0 ? a[k] : cmul(a[k], roots[t * k]);
                }
            }
        });
    }
    __syncthreads();
    if (holds && t < p.r1) {
        with_r2<CLASS>(p.r2, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            C b[R], m[R];
            // Value n of thread t is kz = t + r1 n; its mirror is value
            // r2 - 1 - n of thread r1 - t, or (r2 - n) % r2 of thread 0.
            const int tm = t == 0 ? 0 : p.r1 - t;
#pragma unroll
            for (int n = 0; n < R; ++n) {
                b[n] = buf[(t * R + n) * G + j];
                m[n] = mirror_buf[(tm * R + n) * G + j];
            }
            dft<R, false>(b);
            dft<R, false>(m);
#pragma unroll
            for (int n = 0; n < R; ++n) {
                // W = E^ conj K^ with E^ = (Z(k) + conj Z(-k))/2, K^ = (Z(k) - conj Z(-k))/(2i).
                const C va = b[n];
                const C vm = cconj(t == 0 ? m[(R - n) % R] : m[R - 1 - n]);
                const C e = cscale(cadd(va, vm), 0.5);
                const C d = csub(va, vm);  // = 2i K^
                b[n] = cscale(cmulconj(e, cmake<C>(d.y * 0.5, -d.x * 0.5)), scale);
            }
            dft<R, true>(b);
#pragma unroll
            for (int n = 0; n < R; ++n) {
                buf[(t * R + n) * G + j] = n == 0 ? b[n] : cmulconj(b[n], roots[t * n]);
            }
        });
    }
    __syncthreads();
    if (holds && t < p.r2) {
        with_r1<CLASS>(p.r1, [&](auto radix) {
            constexpr int R = decltype(radix)::value;
            C a[R];
#pragma unroll
            for (int k = 0; k < R; ++k) {
                a[k] = buf[(k * p.r2 + t) * G + j];
            }
            dft<R, true>(a);
#pragma unroll
            for (int n = 0; n < R; ++n) {
                column[(p.r2 * n + t) * plane] = a[n];
            }
            if (!self) {
#pragma unroll
                for (int n = 0; n < R; ++n) {
                    mirror[(p.r2 * n + t) * plane] = cconj(a[n]);
                }
            }
        });
    }
}

// x transform back of the output rows and their checks.  A block takes `per`
// consecutive groups of rows, so that blocks are in index order.
template <int CLASS>
__global__ void __launch_bounds__(kMaxThreads<CLASS>, kMinBlocks<CLASS>)
    rows_extract_kernel(const C* __restrict__ z, AxisPlan p, int Ly, int Lz,
                        const C* __restrict__ table, CorrelationShape s, int binary, double rel,
                        const InputStats* __restrict__ input, int per, double* __restrict__ out,
                        ExtractStats* __restrict__ stats, OutputFlags* __restrict__ flags)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* roots = reinterpret_cast<C*>(smem_raw);
    const int j = threadIdx.x / p.r1, t = threadIdx.x - j * p.r1;
    C* line = roots + p.L + j * p.r1 * row_pitch(p);
    const unsigned int rows = static_cast<unsigned int>(s.out[1]) * s.out[2];
    const int ox = s.out[0];
    stage_roots(roots, table, p.L);
    CellChecks checks(*input, binary != 0, rel);
    for (int i = 0; i < per; ++i) {
        const unsigned int row = (blockIdx.x * static_cast<unsigned int>(per) + i) * kLines + j;
        const bool holds = j < kLines && row < rows;
        const int y = static_cast<int>(row % s.out[1]), zz = static_cast<int>(row / s.out[1]);
        const C* from = z + static_cast<long long>(p.L) *
                                (wrap(y - (s.ker[1] - 1), Ly) +
                                 static_cast<long long>(Ly) * wrap(zz - (s.ker[2] - 1), Lz));
        __syncthreads();  // roots are there; the exchange buffers are free
        row_first<true, CLASS>(p, line, roots, t, holds, [&](int x) { return from[x]; });
        __syncthreads();
        const long long first = static_cast<long long>(row) * ox;
        row_second<true, CLASS>(p, line, t, holds, [&](int position, C v) {
            const int x = wrap(position + s.ker[0] - 1, p.L);
            if (x >= ox) {
                return;
            }
            const long long at = first + x;
            out[at] = checks.take(at, v.x, v.y);
        });
    }
    checks.finish(stats, flags);
}

// Threads of a block: one per line and radix r1 item, whole warps.
int block_threads(AxisPlan p)
{
    return (kLines * p.r1 + 31) / 32 * 32;
}
std::size_t row_bytes(AxisPlan p)
{
    // Whole warps: threads past the last line point behind it but touch nothing.
    return sizeof(C) * (p.L + kLines * static_cast<std::size_t>(p.r1) * row_pitch(p));
}
std::size_t column_bytes(AxisPlan p, int buffers)
{
    const int G = kLines;
    return sizeof(C) * ((p.L + G - 1) / G * G + static_cast<std::size_t>(buffers) * p.L * G);
}

// Launches `kernel` with its dynamic shared memory allowed.
template <auto KERNEL, class... A>
int launch(dim3 grid, int threads, std::size_t bytes, cudaStream_t stream, A... args)
{
    static std::once_flag once[64];
    once_per_device(once, [] {
        cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    });
    KERNEL<<<grid, threads, bytes, stream>>>(args...);
    return cudaGetLastError() == cudaSuccess ? kOk : kCuda;
}
// f(Int<class>) for a plan.
template <class F>
int with_class(AxisPlan p, F&& f)
{
    return p.r1 <= 16 ? f(Int<0> {}) : p.r1 <= 20 ? f(Int<1> {}) : f(Int<2> {});
}

}  // namespace

template <typename E>
int CorrelationPasses::forward(const E* env, const std::uint8_t* ker) const
{
    const int fill_y = std::max(shape.env[1], shape.ker[1]), fill_z = std::max(shape.env[2], shape.ker[2]);
    const int rows = fill_y * fill_z, G = kLines;
    const AxisPlan &px = plan[0], &py = plan[1];
    int status = with_class(px, [&](auto c) {
        return launch<rows_forward_kernel<E, decltype(c)::value>>(dim3((rows + G - 1) / G), block_threads(px),
                                                                  row_bytes(px), stream, z, px, py.L, fill_y, rows,
                                                                  roots[0], shape, env, ker);
    });
    if (status == kOk) {
        status = with_class(py, [&](auto c) {
            return launch<columns_kernel<false, decltype(c)::value>>(dim3((px.L + G - 1) / G, fill_z),
                                                                     block_threads(py), column_bytes(py, 1), stream, z,
                                                                     px.L, py, plan[2].L, 0, fill_y, roots[1]);
        });
    }
    return status;
}

int CorrelationPasses::multiply() const
{
    const int fill_z = std::max(shape.env[2], shape.ker[2]), G = kLines;
    const AxisPlan &px = plan[0], &py = plan[1], &pz = plan[2];
    const double scale = 1.0 / (static_cast<double>(px.L) * py.L * pz.L);
    int status = with_class(pz, [&](auto c) {
        return launch<pairs_kernel<decltype(c)::value>>(dim3((px.L / 2 + G) / G, py.L), block_threads(pz),
                                                        column_bytes(pz, 2), stream, z, px.L, py.L, pz, fill_z,
                                                        roots[2], scale);
    });
    if (status == kOk) {
        status = with_class(py, [&](auto c) {
            return launch<columns_kernel<true, decltype(c)::value>>(
                dim3((px.L + G - 1) / G, shape.out[2]), block_threads(py), column_bytes(py, 1), stream, z, px.L, py,
                pz.L, 1 - shape.ker[2], py.L, roots[1]);
        });
    }
    return status;
}

int CorrelationPasses::extract_blocks() const
{
    const long long groups = (static_cast<long long>(shape.out[1]) * shape.out[2] + kLines - 1) / kLines;
    const long long per = (groups + 148 * 8 - 1) / (148 * 8);
    return static_cast<int>((groups + per - 1) / per);
}

int CorrelationPasses::extract(const InputStats* input, bool binary, double rel, double* out, ExtractStats* stats,
                               int blocks, OutputFlags* flags) const
{
    const AxisPlan& px = plan[0];
    const long long groups = (static_cast<long long>(shape.out[1]) * shape.out[2] + kLines - 1) / kLines;
    const int per = static_cast<int>((groups + blocks - 1) / blocks);
    return with_class(px, [&](auto c) {
        return launch<rows_extract_kernel<decltype(c)::value>>(
            dim3(blocks), block_threads(px), row_bytes(px), stream, z, px, plan[1].L, plan[2].L, roots[0], shape,
            binary ? 1 : 0, rel, input, per, out, stats, flags);
    });
}

template int CorrelationPasses::forward<double>(const double*, const std::uint8_t*) const;
template int CorrelationPasses::forward<std::uint8_t>(const std::uint8_t*, const std::uint8_t*) const;

AxisPlan axis_plan(int L)
{
    constexpr int radices[] = { 1, 2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 20, 24, 25, 27, 32 };
    for (const int r1 : radices) {
        for (const int r2 : radices) {
            if (r1 >= r2 && r1 * r2 == L) {
                return { L, r1, r2 };
            }
        }
    }
    return { L, 0, 0 };
}

}  // namespace spk
