// Spectral page pipeline: legal-translation correlation of one environment
// (occupancy + proximity) against many oriented kernels, fused threshold,
// approximate score and top-k, then exact integer recount and exact FP64
// proximity sums for the selected candidates.
//
// Reference behaviour restated (engine/pack_solver/src/spectral_pipeline.cpp):
//   legal translations  first = env.first - kernel.first, extent E-K+1   :1618-1648
//   score = .65 * (world_z + max_z - c_min_z) / H - .35 * prox / occ      :1794-1800
//   ordinary pages keep round(binary) == 0, rank by (score, o, z, y, x),
//   32 entries after an exclusive cursor                                  :1706-1824
//   direct_zero_overlap = exact u8 recount of each page candidate         :1825-1857
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/spk_b200.h"
#include "common.cuh"
#include "edt.cuh"
#include "geometry.hpp"
#include "passes.hpp"

struct spk_context;

namespace spk {

constexpr int kPageSize = 32;
constexpr int kExactPerOrientation = 64;
constexpr unsigned kKeyCapacity = 4096;   // keys per sorted chunk
constexpr unsigned kMaxKeyChunks = 64;    // chunks of a request's key range at most

struct Candidate {
    std::int64_t t[3];
    double score;
    bool direct_zero;
    std::uint64_t orientation;
    double binary_overlap;
};

// One oriented kernel on the device, prepared for a fixed environment shape.
struct KernelSlot {
    std::uint64_t orientation {};
    int K[3] {};
    std::int64_t first[3] {};
    std::uint64_t occupied {};
    double max_z {};
    float2* partial {};           // [z < K2][ky < L1][kx < L0], x and y transformed
    std::int32_t* ones {};        // environment-relative offsets of kernel ones
    double* t65 {};               // .65 * top(z) for each legal z
    std::vector<double> t65_host;
    int legal[3] {};              // E - K + 1 per axis (0 when the kernel does not fit)
    // Each kernel cell's depth is its distance to the nearest cell that is not
    // the kernel's.  Where a copy fits, every kernel cell is free, so the
    // nearest occupied cell is at least that far: the proximity sum is at most
    // most_proximity, and plane z of the kernel needs an environment plane
    // with a squared distance of at least depth2[z].
    double most_proximity {};
    std::vector<std::int32_t> depth2;
    std::vector<std::uint8_t> host_cells;
};

struct PageRequest {
    std::uint64_t slot {};
    bool has_cursor {};
    Candidate cursor {};
    // Candidates are the legal translations whose overlap count is this
    // (0: ordinary pages; low-overlap pages use one count at a time).
    std::uint32_t overlap {};
    // A low-overlap page (spectral_pipeline.hpp:45, CandidatePageMode::low_overlap).
    bool low_overlap {};
};

struct PageOutcome {
    int status {};
    std::vector<Candidate> page;
    bool certified {};
    bool threshold_pass {};
    double max_integer_residual {};
    double max_score_error {};
    double excluded_score {};  // lowest approximate score of an unrescored candidate
    // Every candidate left out of the rescored set has an exact score above
    // this bound; page entries scoring <= it are exact and correctly placed.
    double exact_floor { INFINITY };
    std::uint64_t rescored {};
};

// What a page call must certify.
struct PageGoal {
    // true: whole pages (threshold passes where needed).  false: the first
    // kHeadCandidates candidates of each orientation with their exact_floor,
    // as far as the merge over orientations can need them.
    bool full { true };
    // Planes that cannot hold a candidate of the page may be skipped (their
    // cells then take no part in the reported residual).
    bool prune { false };
};
constexpr int kHeadCandidates = 16;

class Pipeline {
public:
    // `name` prefixes the context's buffers that hold this pipeline's state
    // between calls: pipelines that live side by side need different ones.
    Pipeline(spk_context* ctx, const char* name);
    ~Pipeline();

    // Environment window (global first + shape) and lattice/container terms.
    int set_geometry(const std::int64_t* env_first, const std::uint32_t* env_shape, const double* origin,
                     double pitch, double container_min_z, double container_height);
    // Device occupancy (u8, E^3): runs the exact EDT and the environment spectrum.
    int set_occupancy(const std::uint8_t* d_occupancy);
    // The same after the only change since the last call is that the cells
    // d_sites != 0 (all inside `sites`, window coordinates) became occupied:
    // the EDT is updated in place over the region they can affect, and only
    // that region's planes are transformed again.
    int add_occupied(const std::uint8_t* d_occupancy, const std::uint8_t* d_sites, const EdtBox& sites);
    // The same updates queued on the pipeline's own stream, after the work
    // already on the context's stream (d_sites null: set_occupancy), so that
    // the context's stream can run other work (the proposal) meanwhile.
    // refresh_order() makes the context's stream wait for it; pages() does
    // so itself.  Until then nothing the update writes may be read, and
    // nothing it reads (the occupancy, the sites) rewritten.
    int refresh_begin(const std::uint8_t* d_occupancy, const std::uint8_t* d_sites, const EdtBox* sites);
    void refresh_order();
    // Adds an oriented kernel field (host cells, X-fastest); returns the slot.
    int add_kernel(std::uint64_t orientation, const std::int64_t* first, const std::uint32_t* shape,
                   const std::uint8_t* cells, double max_z, std::uint64_t& slot);
    // Adds a batch of kernels whose cells (u8, X-fastest) are on the device,
    // item i at d_cells + cells_at[i], as orientations first_orientation + i;
    // their slots follow the ones there are.  Waits for the stream.
    int add_kernels(std::uint64_t first_orientation, const std::vector<geo::Window>& windows,
                    const std::uint8_t* d_cells, const long long* cells_at, const double* max_z);
    int pages(const std::vector<PageRequest>& requests, std::vector<PageOutcome>& out, PageGoal goal);

    const std::uint8_t* occupancy() const { return occ_; }
    const std::int32_t* d2() const { return d2_; }
    const int* env_shape() const { return E_; }
    const int* fft_shape() const { return L_; }
    std::size_t kernels() const { return slots_.size(); }
    const KernelSlot& slot(std::size_t i) const { return slots_[i]; }
    double epsilon_p(const KernelSlot& s) const;

private:
    // One orientation's legal planes [z0, z1) to visit, and where its
    // candidates go.
    struct PlaneWork {
        const KernelSlot* slot;
        int z0, z1;
        unsigned long long* keys;
        unsigned int* count;
        unsigned int cap;
        unsigned long long* tau;
        unsigned long long* resid;
        float target;
        double threshold, cursor_floor, prune;
    };
    // bound_known: the work's bounds may come from planes visited before.
    int run_planes(const std::vector<PlaneWork>& work, PassMode mode, bool bound_known);
    int ordinary_pages(const std::vector<PageRequest>& requests, std::vector<PageOutcome>& out, PageGoal goal);
    int low_overlap_page(const PageRequest& request, PageOutcome& out);
    // Legal planes [zb, zt) outside which no translation of the kernel is free.
    void feasible_planes(const KernelSlot& s, int& zb, int& zt) const;
    // Environment rows and columns (x and y) of the region's planes, or of all.
    int update_spectrum(const EdtBox* d_region);
    // The plane statistics of the last update, once the device has them.
    int finish_stats();
    // Transform lengths per axis for the window; sets L_.
    int choose_lengths(const std::uint32_t* env_shape);
    // The proximity table, which other calls on the context may have moved.
    const double* table(int& status) const;
    double score(const KernelSlot& s, const std::int64_t* t, double p) const;
    double approx_epsilon(const KernelSlot& s) const;

    spk_context* ctx_;
    const std::string name_;
    int E_[3] {};
    int L_[3] {};  // x and y transform lengths; z: the length a whole column would take
    bool pow2_ {};   // SPK_FFT_LENGTHS=pow2
    bool debug_ {};  // SPK_DEBUG_PAGES
    std::int64_t env_first_[3] {};
    double origin_[3] {};
    double pitch_ {};
    double cmin_z_ {};
    double height_ {};
    std::uint8_t* occ_ {};
    std::int32_t* d2_ {};
    std::int32_t* tile_max_ {};  // largest d2 per kEdtTile^3 tile (incremental EDT)
    float2* env_ {};             // [z < E2][ky < L1][kx < L0]: Z = B + iP, x and y transformed
    RowStats* stats_ {};             // device, one entry per row block
    const RowStats* stats_host_ {};  // pinned copy of the last update
    cudaStream_t stats_stream_ {};
    bool stats_pending_ {};
    double plane_rms_ {};                  // largest sqrt(mean |Z|^2) of a plane over the transform grid
    std::vector<std::int32_t> plane_max_;  // largest d2 per environment plane
    cudaStream_t side_ {};  // refresh_begin's stream
    cudaEvent_t ev_in_ {}, ev_done_ {};
    bool pending_ {};
    std::vector<KernelSlot> slots_;
    struct Block {
        void* ptr;
        std::size_t bytes;
    };
    std::vector<Block> blocks_;  // the slots' device data

public:
    // Work counters since the last reset: first-pass pages, threshold passes,
    // candidates rescored exactly, pages certified by the first pass.
    std::uint64_t stat_pages {}, stat_threshold_passes {}, stat_rescored {}, stat_first_certified {};
};

}  // namespace spk
