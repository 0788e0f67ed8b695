// Full-range FFT cross-correlation: the GPU replacement of
// compute::correlate_binary_cpu / correlate_proximity_cpu
// (reference engine/pack_compute/src/correlation.cpp:238-655).
//
// Math: out(t) = sum_i E[i + t] * K[i] for every t in the (E+K-1)^3 range,
// t_first = env_first - kernel_first - (K-1)  (correlation.cpp:281-304).
// The environment and kernel are packed as one complex field Z = E + iK on a
// grid L >= E+K-1 per axis (no wrap for any output), one forward 3D FFT gives
// both spectra through Hermitian symmetry, W = E^ conj(K^) is formed, and one
// inverse 3D FFT (scaled 1/N) yields the correlation in the real part; the
// imaginary part must stay below the reference's tolerance.  The last pass
// applies the reference's per-cell checks (correlation.cpp:494-540); input
// validity and masses (:316-365) and the 8 direct probes (:542-577) are reduced
// on the device beside it, from the copies of the inputs that the transform
// reads.

#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <chrono>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <limits>
#include <vector>

#include "context.hpp"
#include "correlate_fft.hpp"
#include "host_copy.hpp"

namespace spk {

std::int64_t monotonic_ns()
{
    return std::chrono::duration_cast<std::chrono::nanoseconds>(std::chrono::steady_clock::now().time_since_epoch())
        .count();
}

namespace {

constexpr std::uint64_t kExactInteger = 1ULL << 53;

// ---- input checks and masses -------------------------------------------------

// A sum with its rounding error carried along (Knuth's two-sum): partial sums
// of any grouping agree to the last bits of the result.
struct Compensated2 {
    double value, error;
};
__device__ __forceinline__ Compensated2 comp_add(Compensated2 a, double v)
{
    const double s = a.value + v, t = s - a.value;
    return { s, a.error + ((a.value - (s - t)) + (v - t)) };
}
__device__ __forceinline__ Compensated2 comp_merge(Compensated2 a, Compensated2 b)
{
    const Compensated2 s = comp_add(a, b.value);
    return { s.value, s.error + b.error };
}
// Over the block's threads; thread 0 gets the sum.
template <int THREADS>
__device__ __forceinline__ Compensated2 comp_block(Compensated2 c)
{
    __shared__ Compensated2 warps[THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) {
        const Compensated2 other { __shfl_down_sync(0xffffffffu, c.value, o), __shfl_down_sync(0xffffffffu, c.error, o) };
        c = comp_merge(c, other);
    }
    __syncthreads();  // an earlier use of `warps` is read
    if ((threadIdx.x & 31) == 0) {
        warps[threadIdx.x >> 5] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < THREADS / 32; ++w) {
            c = comp_merge(c, warps[w]);
        }
    }
    return c;
}

constexpr int kValidateThreads = 256;

// Validity and masses of the inputs: blocks leave partial masses, the last one
// to finish adds them in order.  `stats` starts as zeros.
template <typename E>
__global__ void __launch_bounds__(kValidateThreads) validate_kernel(const E* __restrict__ env, long long env_count,
                                                                   const std::uint8_t* __restrict__ ker,
                                                                   long long ker_count, Compensated2* partial,
                                                                   unsigned int* done, InputStats* stats)
{
    constexpr bool binary = std::is_same_v<E, std::uint8_t>;
    const long long start = blockIdx.x * static_cast<long long>(kValidateThreads) + threadIdx.x;
    const long long step = static_cast<long long>(gridDim.x) * kValidateThreads;
    Compensated2 mass { 0.0, 0.0 };
    unsigned int env_ones = 0, ker_ones = 0;  // per thread: far below 2^32
    bool bad_env = false, bad_ker = false;
#pragma unroll 4
    for (long long i = start; i < env_count; i += step) {
        const E v = env[i];
        if constexpr (binary) {
            env_ones += v;
            bad_env = bad_env || v > 1;
        }
        else {
            bad_env = bad_env || !(v >= 0.0 && v <= 1.0);
            mass = comp_add(mass, v);
        }
    }
#pragma unroll 4
    for (long long i = start; i < ker_count; i += step) {
        const std::uint8_t v = ker[i];
        ker_ones += v;
        bad_ker = bad_ker || v > 1;
    }
    const unsigned long long e = __reduce_add_sync(0xffffffffu, env_ones), k = __reduce_add_sync(0xffffffffu, ker_ones);
    const bool any_env = __any_sync(0xffffffffu, bad_env), any_ker = __any_sync(0xffffffffu, bad_ker);
    if ((threadIdx.x & 31) == 0) {
        if (e) {
            atomicAdd(&stats->env_ones, e);
        }
        if (k) {
            atomicAdd(&stats->ker_ones, k);
        }
        if (any_env) {
            atomicOr(&stats->bad_environment, 1u);
        }
        if (any_ker) {
            atomicOr(&stats->bad_kernel, 1u);
        }
    }
    if constexpr (!binary) {
        __shared__ bool last;
        mass = comp_block<kValidateThreads>(mass);
        if (threadIdx.x == 0) {
            partial[blockIdx.x] = mass;
            __threadfence();
            last = atomicAdd(done, 1u) == gridDim.x - 1;
            __threadfence();
        }
        __syncthreads();
        if (!last) {
            return;
        }
        Compensated2 sum { 0.0, 0.0 };
        for (unsigned int b = threadIdx.x; b < gridDim.x; b += kValidateThreads) {
            sum = comp_merge(sum, { __ldcg(&partial[b].value), __ldcg(&partial[b].error) });
        }
        sum = comp_block<kValidateThreads>(sum);
        if (threadIdx.x == 0) {
            stats->mass = sum.value + sum.error;
        }
    }
}

// ---- direct probes ------------------------------------------------------------------

// The deterministic direct checks (correlation.cpp:549-577): output indices
// in the reference's order, the extracted value there and the direct sum.
struct Probes {
    unsigned long long index[8];
    double value[8];
    double expected[8];
    double mass;  // of all unrounded outputs
};

constexpr int kProbeThreads = 512;
constexpr int kProbeSplit = 16;

// kProbeSplit blocks per probe: the direct sum at one output index
// (direct_probe, correlation.cpp:153-218), rows dealt out to the warps; the last
// block of a probe adds up the parts in order.  (One block per probe: 137 us
// for 10^6-term probes, 8 SMs busy.)  Probe 3 looks where the largest output is,
// which its blocks find from the extraction's per-block maxima (the lowest index
// of equal ones); the first block also adds up the outputs' mass.
template <typename E>
__global__ void __launch_bounds__(kProbeThreads) probe_kernel(CorrelationShape s, const E* __restrict__ env,
                                                             const std::uint8_t* __restrict__ ker,
                                                             const double* __restrict__ out,
                                                             const ExtractStats* __restrict__ stats, int blocks,
                                                             Compensated2* __restrict__ partial, unsigned int* done,
                                                             Probes* __restrict__ probes)
{
    constexpr bool binary = std::is_same_v<E, std::uint8_t>;
    __shared__ double best_abs[kProbeThreads];
    __shared__ int best_block[kProbeThreads];
    const unsigned long long count =
        static_cast<unsigned long long>(s.out[0]) * s.out[1] * static_cast<unsigned long long>(s.out[2]);
    const int p = blockIdx.x;
    unsigned long long at = 0;
    if (p == 3) {
        double best = -1.0;
        int block = 0;
        for (int b = threadIdx.x; b < blocks; b += kProbeThreads) {
            if (stats[b].max_abs > best || (stats[b].max_abs == best && stats[b].max_index < stats[block].max_index)) {
                best = stats[b].max_abs;
                block = b;
            }
        }
        best_abs[threadIdx.x] = best;
        best_block[threadIdx.x] = block;
        __syncthreads();
        for (int half = kProbeThreads / 2; half > 0; half >>= 1) {
            if (threadIdx.x < half) {
                const double a = best_abs[threadIdx.x + half];
                const int b = best_block[threadIdx.x + half];
                if (a > best_abs[threadIdx.x] ||
                    (a == best_abs[threadIdx.x] && stats[b].max_index < stats[best_block[threadIdx.x]].max_index)) {
                    best_abs[threadIdx.x] = a;
                    best_block[threadIdx.x] = b;
                }
            }
            __syncthreads();
        }
        at = static_cast<unsigned long long>(stats[best_block[0]].max_index);
    }
    else {
        at = p == 0   ? 0
             : p == 1 ? count - 1
             : p == 2 ? count / 2
             : p == 4 ? count / 4
             : p == 5 ? count / 3
             : p == 6 ? count / 3 * 2
                      : count / 4 * 3;
    }
    const int x = static_cast<int>(at % s.out[0]);
    const unsigned long long yz = at / s.out[0];
    const int shift[3] = { x - (s.ker[0] - 1), static_cast<int>(yz % s.out[1]) - (s.ker[1] - 1),
                           static_cast<int>(yz / s.out[1]) - (s.ker[2] - 1) };
    // The kernel cells whose environment cell exists.
    int lo[3], extent[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = max(0, -shift[a]);
        extent[a] = max(0, min(s.ker[a], s.env[a] - shift[a]) - lo[a]);
    }
    const unsigned int rows = static_cast<unsigned int>(extent[1]) * extent[2];
    unsigned long long ones = 0;
    Compensated2 sum { 0.0, 0.0 };
    const int lane = threadIdx.x & 31;
    for (unsigned int row = blockIdx.y * (kProbeThreads / 32) + (threadIdx.x >> 5); row < rows;
         row += kProbeSplit * (kProbeThreads / 32)) {
        const int ky = lo[1] + static_cast<int>(row % extent[1]), kz = lo[2] + static_cast<int>(row / extent[1]);
        const E* e = env + shift[0] + static_cast<long long>(s.env[0]) *
                                          ((ky + shift[1]) + static_cast<long long>(s.env[1]) * (kz + shift[2]));
        const std::uint8_t* k = ker + static_cast<long long>(s.ker[0]) * (ky + static_cast<long long>(s.ker[1]) * kz);
#pragma unroll 4
        for (int kx = lo[0] + lane; kx < lo[0] + extent[0]; kx += 32) {
            if constexpr (binary) {
                ones += static_cast<unsigned int>(e[kx]) * k[kx];
            }
            else {
                sum = comp_add(sum, e[kx] * k[kx]);
            }
        }
    }
    if constexpr (binary) {
        sum.value = static_cast<double>(ones);  // exact: below 2^53, and so is the sum
    }
    sum = comp_block<kProbeThreads>(sum);
    if (threadIdx.x == 0) {
        partial += p * kProbeSplit;
        partial[blockIdx.y] = sum;
        __threadfence();
        if (atomicAdd(&done[p], 1u) == kProbeSplit - 1) {
            __threadfence();
            sum = { 0.0, 0.0 };
#pragma unroll
            for (int b = 0; b < kProbeSplit; ++b) {
                sum = comp_merge(sum, { __ldcg(&partial[b].value), __ldcg(&partial[b].error) });
            }
            probes->index[p] = at;
            probes->value[p] = out[at];
            probes->expected[p] = sum.value + sum.error;
        }
    }
    if (p == 0 && blockIdx.y == 0) {
        Compensated2 mass { 0.0, 0.0 };
        for (int b = threadIdx.x; b < blocks; b += kProbeThreads) {
            mass = comp_add(mass, stats[b].mass);
        }
        mass = comp_block<kProbeThreads>(mass);
        if (threadIdx.x == 0) {
            probes->mass = mass.value + mass.error;
        }
    }
}

// Translation mask over a caller's box of absolute translations, from the
// rounded full-range counts: inside the range, 1 where the count is zero
// (want_zero) or non-zero (otherwise); outside the range, 0.  These are the
// free and blocked rules of gap_fill.cpp:404-420 and :443-446.  dx..dz are the
// box's first translation minus the range's first, clamped on the host so
// that dx + x cannot overflow.
__global__ void mask_kernel(const double* __restrict__ counts, long long ox, long long oy, long long oz, long long dx,
                            long long dy, long long dz, long long bx, long long by, long long bz, int want_zero,
                            std::uint8_t* __restrict__ mask)
{
    const long long n = bx * by * bz;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long x = dx + i % bx;
        const long long r = i / bx;
        const long long y = dy + r % by;
        const long long z = dz + r / by;
        std::uint8_t m = 0;
        if (x >= 0 && y >= 0 && z >= 0 && x < ox && y < oy && z < oz) {
            const bool zero = counts[x + ox * (y + oy * z)] == 0.0;
            m = (zero == (want_zero != 0)) ? 1 : 0;
        }
        mask[i] = m;
    }
}

// Inputs up to this size go out in one copy, results up to this size come back
// with the checks' outcome.  (Pinned memory comes in chunks of 2 MB that cost a
// millisecond or more; buffers of this size mostly share one.)
constexpr std::size_t kEarlyResult = 512 << 10;

// A request to threshold on the device: the mask is written to host memory
// and the FP64 counts stay on the device.
struct MaskRequest {
    std::int64_t first[3];
    std::uint32_t shape[3];
    bool want_zero;
    std::uint8_t* mask;
    std::uint64_t capacity;
};

struct Compensated {
    double value {}, correction {};
    void add(double v)
    {
        const double adjusted = v - correction;
        const double next = value + adjusted;
        correction = (next - value) - adjusted;
        value = next;
    }
};

bool checked_mul(std::uint64_t a, std::uint64_t b, std::uint64_t& r)
{
    if (a && b > UINT64_MAX / a) {
        return false;
    }
    r = a * b;
    return true;
}

// Terms of the direct sum at output index `index`: the kernel cells whose
// environment cell exists.
std::uint64_t probe_terms(const spk_correlation_spec& spec, const std::uint32_t* oshape, std::uint64_t index)
{
    const std::uint64_t at[3] = { index % oshape[0], index / oshape[0] % oshape[1], index / oshape[0] / oshape[1] };
    std::uint64_t terms = 1;
    for (int a = 0; a < 3; ++a) {
        const std::int64_t shift =
            static_cast<std::int64_t>(at[a]) - (static_cast<std::int64_t>(spec.kernel_shape[a]) - 1);
        const std::int64_t lo = std::max<std::int64_t>(0, -shift);
        const std::int64_t hi = std::min<std::int64_t>(spec.kernel_shape[a],
                                                       static_cast<std::int64_t>(spec.environment_shape[a]) - shift);
        terms *= static_cast<std::uint64_t>(std::max<std::int64_t>(0, hi - lo));
    }
    return terms;
}

int grid_blocks(long long n, int threads)
{
    const long long want = (n + threads - 1) / threads;
    return static_cast<int>(std::min<long long>(std::max<long long>(want, 1), 148LL * 16));
}

template <typename T, typename E>
int correlate(spk_context* ctx, const spk_correlation_spec* spec_ptr, const E* environment, const std::uint8_t* kernel,
              const spk_correlation_limits* limits_ptr, const spk_control* control, double* out_values,
              std::uint64_t out_capacity, spk_correlation_result* result, bool half_spectra = false,
              const MaskRequest* mask_request = nullptr)
{
    constexpr bool binary = std::is_same_v<E, std::uint8_t>;
    if (!ctx || !spec_ptr || !environment || !kernel || !result) {
        return kInvalidArgument;
    }
    const auto& spec = *spec_ptr;
    spk_correlation_limits limits { 512ULL << 20, 0, 16'777'216, 200'000'000 };
    if (limits_ptr) {
        limits = *limits_ptr;
    }
    std::memset(result, 0, sizeof(*result));
    ctx->message = "";
    // The reference admits its own call metadata before anything else
    // (correlation.cpp:255-259); here that is the result record.
    if (limits.reserved_bytes > limits.max_working_bytes ||
        limits.max_working_bytes - limits.reserved_bytes < sizeof(spk_correlation_result)) {
        return fail(ctx, kMemoryLimit, "Correlation metadata exceeds its memory limit.");
    }
    if (int s = poll(control)) {
        return fail(ctx, s, "Correlation interrupted.");
    }
    std::uint64_t env_count = 1, ker_count = 1, padded_count = 1;
    std::uint32_t padded[3];
    for (int a = 0; a != 3; ++a) {
        if (spec.environment_shape[a] == 0 || spec.kernel_shape[a] == 0 ||
            !checked_mul(env_count, spec.environment_shape[a], env_count) ||
            !checked_mul(ker_count, spec.kernel_shape[a], ker_count)) {
            return fail(ctx, kShapeOverflow, "Correlation extents must be positive and representable.");
        }
        const std::uint64_t length = std::uint64_t { spec.environment_shape[a] } + spec.kernel_shape[a] - 1;
        if (length > UINT32_MAX || !checked_mul(padded_count, length, padded_count)) {
            return fail(ctx, kShapeOverflow, "Padded correlation shape overflowed.");
        }
        padded[a] = static_cast<std::uint32_t>(length);
        const std::int64_t ef = spec.environment_first[a], kf = spec.kernel_first[a];
        if ((kf > 0 && ef < INT64_MIN + kf) || (kf < 0 && ef > INT64_MAX + kf)) {
            return fail(ctx, kIndexOverflow, "The first output translation is not representable.");
        }
        const std::int64_t diff = ef - kf;
        const std::int64_t k1 = static_cast<std::int64_t>(spec.kernel_shape[a]) - 1;
        if (diff < INT64_MIN + k1) {
            return fail(ctx, kIndexOverflow, "The first output translation is not representable.");
        }
        result->translation_first[a] = diff - k1;
        if (result->translation_first[a] > INT64_MAX - static_cast<std::int64_t>(length - 1)) {
            return fail(ctx, kIndexOverflow, "The last output translation is not representable.");
        }
        result->shape[a] = padded[a];
    }
    // Input validity and masses (correlation.cpp:316-365) are checked on the
    // device with the rest of the work; a call that fails a later check than
    // those gets them from the host first, so that the first failure in the
    // reference's order is the one reported.
    const auto host_inputs = [&]() -> int {
        std::uint64_t env_ones = 0, ker_ones = 0;
        Compensated env_mass_sum;
        for (std::uint64_t i = 0; i != env_count; ++i) {
            const double value = static_cast<double>(environment[i]);
            if (!std::isfinite(value) || value < 0.0 || value > 1.0) {
                return fail(ctx, kInvalidEnvironment, "Environment cells must be finite values in [0,1].");
            }
            if constexpr (binary) {
                env_ones += environment[i];
            }
            else {
                env_mass_sum.add(value);
            }
        }
        for (std::uint64_t i = 0; i != ker_count; ++i) {
            if (kernel[i] > 1) {
                return fail(ctx, kInvalidKernel, "Kernel cells must be binary.");
            }
            ker_ones += kernel[i];
        }
        if constexpr (binary) {
            std::uint64_t product;
            if (!checked_mul(env_ones, ker_ones, product) || product > kExactInteger) {
                return fail(ctx, kNumericRange, "Binary correlation mass is not exactly representable.");
            }
        }
        else if (!std::isfinite(env_mass_sum.value) ||
                 !std::isfinite(env_mass_sum.value * static_cast<double>(ker_ones))) {
            return fail(ctx, kNumericRange, "Proximity correlation mass is not representable.");
        }
        return kOk;
    };
    if (padded_count > limits.max_padded_cells) {
        if (int s = host_inputs()) {
            return s;
        }
        result->padded_cells = padded_count;
        return fail(ctx, kPaddedCellLimit, "Padded field exceeds its cell limit.");
    }
    // FP64 takes the register passes.  In FP32 and FP16 the last bits of a
    // transform decide which calls pass the checks (a total mass within 0.25),
    // and are the values' own: these keep the staged transforms' arithmetic.
    constexpr bool staged = sizeof(T) == 4;
    CorrelationPasses passes {};  // FP64
    StagedCorrelation stages {};   // FP32, FP16
    CorrelationShape shape {};
    int L[3];
    for (int a = 0; a != 3; ++a) {
        const std::uint32_t length = transform_length(padded[a]);
        if (length == 0) {
            if (int s = host_inputs()) {
                return s;
            }
            result->padded_cells = padded_count;
            std::copy(L, L + a, result->padded_shape);
            return fail(ctx, kUnsupportedLength, "Padded extent exceeds the device FFT's longest axis.");
        }
        L[a] = static_cast<int>(length);
        shape.env[a] = static_cast<int>(spec.environment_shape[a]);
        shape.ker[a] = static_cast<int>(spec.kernel_shape[a]);
        shape.out[a] = static_cast<int>(padded[a]);
        if constexpr (staged) {
            stages.L[a] = L[a];
        }
        else {
            passes.plan[a] = axis_plan(L[a]);
        }
    }
    passes.shape = shape;
    stages.shape = shape;
    const std::uint64_t grid = static_cast<std::uint64_t>(L[0]) * L[1] * L[2];
    using C = cplx_t<T>;
    const std::uint64_t grid_bytes = grid * sizeof(C);
    const std::uint64_t out_bytes = padded_count * sizeof(double);
    int extract_blocks;
    if constexpr (staged) {
        extract_blocks = stages.blocks();
    }
    else {
        extract_blocks = passes.extract_blocks();
    }
    const auto finish_shape = [&] {
        result->padded_cells = padded_count;
        for (int a = 0; a != 3; ++a) {
            result->padded_shape[a] = static_cast<std::uint32_t>(L[a]);
        }
    };
    const std::uint64_t half_bytes = half_spectra ? grid * 4 : 0;
    std::uint64_t mask_count = 0;
    if (mask_request) {
        mask_count = 1;
        for (int a = 0; a != 3; ++a) {
            if (!checked_mul(mask_count, mask_request->shape[a], mask_count)) {
                if (int s = host_inputs()) {
                    return s;
                }
                finish_shape();
                return fail(ctx, kShapeOverflow, "Mask box size is not representable.");
            }
        }
    }
    const std::uint64_t working = limits.reserved_bytes + 2 * grid_bytes + half_bytes + out_bytes +
                                  env_count * sizeof(E) + ker_count +
                                  grid_blocks(static_cast<long long>(padded_count), 256) *
                                      sizeof(ExtractStats) +
                                  64 + mask_count;
    if (working > limits.max_working_bytes) {
        if (int s = host_inputs()) {
            return s;
        }
        finish_shape();
        return fail(ctx, kMemoryLimit, "Correlation buffers and FFT workspace exceed their memory limit.");
    }
    if (mask_request ? (mask_request->capacity < mask_count || (mask_count && !mask_request->mask))
                     : (out_capacity < padded_count || !out_values)) {
        if (int s = host_inputs()) {
            return s;
        }
        finish_shape();
        result->working_bytes_peak = working;
        return kInvalidArgument;
    }
    int status = kOk;
    // Small results, read back in one copy: input statistics, output flags,
    // probes.
    struct Readback {
        InputStats input;
        OutputFlags flags;
        Probes probes;
        unsigned int done, probe_done[8];
    };
    const int validate_blocks = grid_blocks(static_cast<long long>(env_count), 4 * kValidateThreads);
    auto* z = static_cast<C*>(device_buffer(ctx, "corr.z", grid_bytes, status));
    // The register passes work in place; what a call is admitted by stays the
    // published estimate of two grids.
    auto* w = staged ? static_cast<C*>(device_buffer(ctx, "corr.w", grid_bytes, status)) : z;
    const std::size_t result_bytes = mask_request ? mask_count : out_bytes;
    // The inputs side by side, and the small results in front of the large one:
    // small calls then copy once each way.
    const std::size_t ker_at = env_count * sizeof(E);
    constexpr std::size_t out_at = (sizeof(Readback) + 255) / 256 * 256;
    auto* d_in = static_cast<std::uint8_t*>(device_buffer(ctx, "corr.in", ker_at + ker_count, status));
    auto* d_back = static_cast<Readback*>(device_buffer(ctx, "corr.out", out_at + out_bytes, status, out_at));
    // The checks' sums (up to 100 KB) lie outside the cap: the host holds no
    // others, and a call that fits without them is not refused for them.
    const std::size_t stats_bytes = extract_blocks * sizeof(ExtractStats);
    const std::size_t partial_bytes = (validate_blocks + 8 * kProbeSplit) * sizeof(Compensated2);
    auto* d_stats = static_cast<ExtractStats*>(device_buffer(ctx, "corr.stats", stats_bytes, status, stats_bytes));
    auto* d_partial =
        static_cast<Compensated2*>(device_buffer(ctx, "corr.partial", partial_bytes, status, partial_bytes));
    const bool small_in = ker_at + ker_count <= kEarlyResult;
    const std::size_t early_bytes = result_bytes <= kEarlyResult ? result_bytes : 0;
    auto* back = static_cast<Readback*>(host_buffer(ctx, "corr.back", out_at + early_bytes, status));
    auto* in = small_in ? static_cast<std::uint8_t*>(host_buffer(ctx, "corr.in", ker_at + ker_count, status)) : nullptr;
    if (!z || !w || !d_in || !d_stats || !d_partial || !d_back || !back || (small_in && !in)) {
        return status;
    }
    auto* d_env = reinterpret_cast<E*>(d_in);
    std::uint8_t* d_ker = d_in + ker_at;
    auto* d_out = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(d_back) + out_at);
    cudaStream_t st = ctx->stream;
    // A call that stops early waits for what it has launched: the pinned
    // copies of its inputs are the context's.
    const auto stop = [&](int s) {
        cudaStreamSynchronize(st);
        return s;
    };
    if (small_in) {
        std::memcpy(in, environment, env_count * sizeof(E));
        std::memcpy(in + ker_at, kernel, ker_count);
        cudaMemcpyAsync(d_in, in, ker_at + ker_count, cudaMemcpyHostToDevice, st);
    }
    else if ((status = copy_to_device(ctx, d_env, environment, env_count * sizeof(E))) ||
             (status = copy_to_device(ctx, d_ker, kernel, ker_count))) {
        return stop(status);
    }
    cudaMemsetAsync(d_back, 0, sizeof(Readback), st);
    validate_kernel<E><<<validate_blocks, kValidateThreads, 0, st>>>(
        d_env, static_cast<long long>(env_count), d_ker, static_cast<long long>(ker_count), d_partial, &d_back->done,
        &d_back->input);
    ctx->launches++;
    const int threads = 256;
    // FP64 keeps the reference's 1e-10 proximity tolerance; FP32 states its
    // own bound, 2^-13 relative to the output scale (2^-8 with FP16 spectra).
    const double rel = sizeof(T) == 8 ? 1e-10 : half_spectra ? 1.0 / 256.0 : 1.0 / 8192.0;
    if constexpr (staged) {
        for (int a = 0; a != 3; ++a) {
            stages.roots[a] = twiddle_table<T>(ctx, L[a], status);
            if (!stages.roots[a]) {
                return stop(status);
            }
        }
        stages.z = z;
        stages.w = w;
        stages.stream = st;
        if ((status = stages.forward(d_env, d_ker))) {
            return stop(status);
        }
        if (int s = poll(control)) {
            return stop(s);
        }
        __half2* zh = nullptr;
        int shift = 0;
        if (half_spectra) {
            // |Z(k)| <= sum |e| + sum |k|: a power-of-two scale puts that bound at 2^15 or below.
            // The masses come back first: this scale is the host's to choose.
            cudaMemcpyAsync(&back->input, &d_back->input, sizeof(InputStats), cudaMemcpyDeviceToHost, st);
            if (cudaStreamSynchronize(st) != cudaSuccess) {
                cudaGetLastError();
                return stop(kCuda);
            }
            const double bound = (binary ? static_cast<double>(back->input.env_ones) : back->input.mass) +
                                 static_cast<double>(back->input.ker_ones);
            shift = bound > 0 ? 15 - static_cast<int>(std::ceil(std::log2(bound))) : 0;
            zh = static_cast<__half2*>(device_buffer(ctx, "corr.zh", half_bytes, status));
            if (!zh || (status = stages.to_half(zh, shift))) {
                return stop(status);
            }
            ctx->launches++;
        }
        if ((status = stages.back(zh, shift, &d_back->input, binary, rel, d_out, d_stats, &d_back->flags))) {
            return stop(status);
        }
        if (int s = poll(control)) {
            return stop(s);
        }
        ctx->launches += 6;
    }
    else {
        for (int a = 0; a != 3; ++a) {
            passes.roots[a] = twiddle_table<T>(ctx, L[a], status);
            if (!passes.roots[a]) {
                return stop(status);
            }
        }
        passes.z = z;
        passes.stream = st;
        if ((status = passes.forward(d_env, d_ker))) {
            return stop(status);
        }
        if (int s = poll(control)) {
            return stop(s);
        }
        if ((status = passes.multiply())) {
            return stop(status);
        }
        if (int s = poll(control)) {
            return stop(s);
        }
        if ((status = passes.extract(&d_back->input, binary, rel, d_out, d_stats, extract_blocks, &d_back->flags))) {
            return stop(status);
        }
        ctx->launches += 4;
    }
    probe_kernel<E><<<dim3(8, kProbeSplit), kProbeThreads, 0, st>>>(shape, d_env, d_ker, d_out, d_stats,
                                                                    extract_blocks, d_partial + validate_blocks,
                                                                    d_back->probe_done, &d_back->probes);
    ctx->launches += 2;
    std::uint8_t* d_mask = nullptr;
    if (mask_request && mask_count) {
        // Box offset from the range's first translation, per axis.  A box
        // more than 2^33 away lies wholly outside the < 2^32-wide range, so
        // the offset is clamped there and dx + x stays far from overflow.
        long long delta[3];
        for (int a = 0; a != 3; ++a) {
            long long d;
            if (__builtin_sub_overflow(mask_request->first[a], result->translation_first[a], &d)) {
                d = mask_request->first[a] < 0 ? -(1LL << 33) : (1LL << 33);
            }
            delta[a] = std::max(-(1LL << 33), std::min(1LL << 33, d));
        }
        d_mask = static_cast<std::uint8_t*>(device_buffer(ctx, "corr.mask", mask_count, status));
        if (!d_mask) {
            return stop(status);
        }
        mask_kernel<<<grid_blocks(static_cast<long long>(mask_count), threads), threads, 0, st>>>(
            d_out, padded[0], padded[1], padded[2], delta[0], delta[1], delta[2], mask_request->shape[0],
            mask_request->shape[1], mask_request->shape[2], mask_request->want_zero ? 1 : 0, d_mask);
        ctx->launches++;
    }
    // The result goes out once the checks have passed: a small one comes back
    // with them, a large one is copied after.
    const void* d_result = mask_request ? static_cast<const void*>(d_mask) : d_out;
    void* destination = mask_request ? static_cast<void*>(mask_request->mask) : out_values;
    const bool early = early_bytes > 0;
    auto* early_at = reinterpret_cast<unsigned char*>(back) + out_at;
    cudaMemcpyAsync(back, d_back, early && !mask_request ? out_at + result_bytes : sizeof(Readback),
                    cudaMemcpyDeviceToHost, st);
    if (early && mask_request) {
        cudaMemcpyAsync(early_at, d_result, result_bytes, cudaMemcpyDeviceToHost, st);
    }
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return kCuda;
    }
    const InputStats& input = back->input;
    if (input.bad_environment) {
        return fail(ctx, kInvalidEnvironment, "Environment cells must be finite values in [0,1].");
    }
    if (input.bad_kernel) {
        return fail(ctx, kInvalidKernel, "Kernel cells must be binary.");
    }
    double expected_mass;
    if constexpr (binary) {
        std::uint64_t product;
        if (!checked_mul(input.env_ones, input.ker_ones, product) || product > kExactInteger) {
            return fail(ctx, kNumericRange, "Binary correlation mass is not exactly representable.");
        }
        expected_mass = static_cast<double>(product);
    }
    else {
        expected_mass = input.mass * static_cast<double>(input.ker_ones);
        if (!std::isfinite(input.mass) || !std::isfinite(expected_mass)) {
            return fail(ctx, kNumericRange, "Proximity correlation mass is not representable.");
        }
    }
    finish_shape();
    result->working_bytes_peak = working;
    const double maximum_output = output_bounds(input, binary, rel).maximum;
    const unsigned long long first_failure[2] = { ~back->flags.inverted_failure[0], ~back->flags.inverted_failure[1] };
    if (first_failure[0] != ~0ULL || first_failure[1] != ~0ULL) {
        if (first_failure[0] <= first_failure[1]) {
            return fail(ctx, kNumeric, "FFT produced a nonfinite or non-real value.");
        }
        return fail(ctx, kNumeric, binary ? "Binary FFT output failed its integer or range check."
                                          : "Proximity FFT output failed its range check.");
    }
    double max_residual = 0;
    std::memcpy(&max_residual, &back->flags.max_residual_bits, 8);
    const Probes& probes = back->probes;
    const double mass_residual = std::fabs(probes.mass - expected_mass);
    const double mass_tolerance = binary ? 0.25 : rel * std::max(1.0, std::fabs(expected_mass));
    if (!std::isfinite(mass_residual) || (binary ? mass_residual >= mass_tolerance : mass_residual > mass_tolerance)) {
        return fail(ctx, kNumeric, "FFT output failed its total-mass check.");
    }
    // Deterministic direct checks (correlation.cpp:549-577), in the
    // reference's order, an index repeated on a small output once.
    double max_probe_error = 0;
    std::uint64_t terms = 0;
    for (int p = 0; p != 8; ++p) {
        if (std::find(probes.index, probes.index + p, probes.index[p]) != probes.index + p) {
            continue;
        }
        const std::uint64_t more = probe_terms(spec, padded, probes.index[p]);
        if (more > limits.max_direct_terms - terms) {
            result->direct_terms = limits.max_direct_terms;
            if (int s = poll(control)) {
                return fail(ctx, s, "Correlation interrupted.");
            }
            return fail(ctx, kDirectTermLimit, "Deterministic direct checks exhausted their work limit.");
        }
        terms += more;
        const double expected = probes.expected[p];
        const double error = std::fabs(probes.value[p] - expected);
        max_probe_error = std::max(max_probe_error, error);
        // FP64 keeps the reference's per-probe relative tolerance; FP32 and
        // FP16 state their bounds relative to the output scale.
        const double tolerance =
            binary ? 0.25 : rel * std::max(1.0, sizeof(T) == 8 ? std::fabs(expected) : maximum_output);
        if (!std::isfinite(error) || (binary ? error >= tolerance : error > tolerance)) {
            result->direct_terms = terms;
            return fail(ctx, kNumeric, "FFT output failed a deterministic direct check.");
        }
    }
    result->direct_terms = terms;
    result->max_integer_residual = max_residual;
    result->mass_residual = mass_residual;
    result->max_probe_error = max_probe_error;
    if (early) {
        std::memcpy(destination, early_at, result_bytes);
    }
    else if (result_bytes && (status = copy_to_host(ctx, destination, d_result, result_bytes))) {
        return status;
    }
    if (int s = poll(control)) {
        return fail(ctx, s, "Correlation interrupted.");
    }
    return kOk;
}

}  // namespace
}  // namespace spk

using namespace spk;

extern "C" {

int spk_estimate_correlation(const spk_correlation_spec* spec, uint32_t precision, spk_correlation_estimate* out)
{
    if (!spec || !out) {
        return kInvalidArgument;
    }
    std::memset(out, 0, sizeof(*out));
    std::uint64_t padded_cells = 1, grid = 1;
    for (int a = 0; a != 3; ++a) {
        const std::uint64_t length = std::uint64_t { spec->environment_shape[a] } + spec->kernel_shape[a] - 1;
        if (!spec->environment_shape[a] || !spec->kernel_shape[a] || length > UINT32_MAX ||
            !checked_mul(padded_cells, length, padded_cells)) {
            return kShapeOverflow;
        }
        const std::uint32_t L = transform_length(length);
        if (L == 0) {
            return kUnsupportedLength;
        }
        out->padded_shape[a] = L;
        grid *= L;
    }
    out->padded_cells = padded_cells;
    out->working_bytes = 2 * grid * (precision == SPK_FP64 ? 16 : 8) + (precision == SPK_FP16 ? 4 * grid : 0) +
                         padded_cells * 8;
    return kOk;
}

int spk_correlate_binary(spk_context* ctx, const spk_correlation_spec* spec, const uint8_t* environment,
                         const uint8_t* kernel, const spk_correlation_limits* limits, const spk_control* control,
                         uint32_t precision, double* out_values, uint64_t out_capacity, spk_correlation_result* result)
{
    try {
        if (ctx) {
            ctx->message = "";
        }
        if (ctx && cudaSetDevice(ctx->device) != cudaSuccess) {
            return finish(ctx, kCuda);
        }
        if (precision > SPK_FP16) {
            return finish(ctx, kInvalidArgument);
        }
        return finish(ctx, precision == SPK_FP64
                               ? correlate<double, std::uint8_t>(ctx, spec, environment, kernel, limits, control,
                                                                 out_values, out_capacity, result)
                               : correlate<float, std::uint8_t>(ctx, spec, environment, kernel, limits, control,
                                                                out_values, out_capacity, result,
                                                                precision == SPK_FP16));
    }
    catch (...) {
        return ctx ? fail(ctx, kAllocation, "Correlation allocation failed.") : kAllocation;
    }
}

int spk_correlate_binary_mask(spk_context* ctx, const spk_correlation_spec* spec, const uint8_t* environment,
                              const uint8_t* kernel, const spk_correlation_limits* limits, const spk_control* control,
                              uint32_t precision, const int64_t box_first[3], const uint32_t box_shape[3],
                              uint32_t select, uint8_t* mask, uint64_t mask_capacity, spk_correlation_result* result)
{
    try {
        if (ctx) {
            ctx->message = "";
        }
        if (ctx && cudaSetDevice(ctx->device) != cudaSuccess) {
            return finish(ctx, kCuda);
        }
        if (precision > SPK_FP16 || select > SPK_MASK_NONZERO || !box_first || !box_shape) {
            return finish(ctx, kInvalidArgument);
        }
        MaskRequest request {};
        for (int a = 0; a != 3; ++a) {
            request.first[a] = box_first[a];
            request.shape[a] = box_shape[a];
        }
        request.want_zero = select == SPK_MASK_ZERO;
        request.mask = mask;
        request.capacity = mask_capacity;
        return finish(ctx, precision == SPK_FP64
                               ? correlate<double, std::uint8_t>(ctx, spec, environment, kernel, limits, control,
                                                                 nullptr, 0, result, false, &request)
                               : correlate<float, std::uint8_t>(ctx, spec, environment, kernel, limits, control,
                                                                nullptr, 0, result, precision == SPK_FP16,
                                                                &request));
    }
    catch (...) {
        return ctx ? fail(ctx, kAllocation, "Correlation allocation failed.") : kAllocation;
    }
}

int spk_correlate_proximity(spk_context* ctx, const spk_correlation_spec* spec, const double* environment,
                            const uint8_t* kernel, const spk_correlation_limits* limits, const spk_control* control,
                            uint32_t precision, double* out_values, uint64_t out_capacity,
                            spk_correlation_result* result)
{
    try {
        if (ctx) {
            ctx->message = "";
        }
        if (ctx && cudaSetDevice(ctx->device) != cudaSuccess) {
            return finish(ctx, kCuda);
        }
        if (precision > SPK_FP16) {
            return finish(ctx, kInvalidArgument);
        }
        return finish(ctx, precision == SPK_FP64
                               ? correlate<double, double>(ctx, spec, environment, kernel, limits, control,
                                                           out_values, out_capacity, result)
                               : correlate<float, double>(ctx, spec, environment, kernel, limits, control, out_values,
                                                          out_capacity, result, precision == SPK_FP16));
    }
    catch (...) {
        return ctx ? fail(ctx, kAllocation, "Correlation allocation failed.") : kAllocation;
    }
}

}  // extern "C"
