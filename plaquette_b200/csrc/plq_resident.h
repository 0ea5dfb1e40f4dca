// plq_resident.h -- one launch for all the sweeps and samples of a call
// (plq_resident.cu).
#pragma once
#include <cuda_runtime.h>

#include "plq_device.cuh"

namespace plq {

enum class ResidentKind { kNone, kSites, kLinks32, kLinks64, kWords, kRanks, kGeneric };

struct ResidentArgs {
    LocalArgs p;             // the chain's pass arguments; sweep32 and pass_offset of the first sweep
    int64_t n_vars;
    uint64_t samples, sweeps;  // samples, and the sweeps before each
    uint8_t *snapshots;      // samples x n_vars bytes in the host's order, or null
    long long *primaries;    // samples x n_primaries, zero before the launch, or null
    int n_primaries;
    unsigned long long arrived;  // arrivals at the grid barrier before this launch
    void *packed;            // the plan's packed_bytes of scratch, then (PCG stream) kResidentTotals words
    uint32_t *totals;
    // filled by launch_resident
    uint32_t units, chunks;  // of a pass: words, rows or ranks; CTAs' shares of them
    uint32_t words_per_row, wpr_m;
    int32_t wpr_l, groups_l;
    uint32_t groups, groups_m;  // threads per word or row (packed kinds)
    int n_keys, words_per_thread, cluster;
};

constexpr size_t kResidentTotals = 2 * 1024;

// The launch shape, fixed at a chain's creation.
struct ResidentPlan {
    ResidentKind kind = ResidentKind::kNone;
    uint32_t units = 0, chunks = 0, words_per_row = 0;
    uint32_t groups = 1, most_groups = 1;
    int per_thread = 1, block = 0;
    unsigned grid = 0;
    bool cluster = false;
    int share = 0;  // plq_resident.cu's Share
    bool stream_draws = false;  // a packed kind on the PCG stream
    int barriers_per_pass = 1;
    size_t shared_bytes = 0;
    size_t packed_bytes = 0;  // scratch of the packed kinds
};

// How a chain without look-back passes would run resident (kNone: not at all).
ResidentKind resident_kind(int model, int q, int d, const int32_t *L, int updater, int rng, bool words);
cudaError_t resident_plan(ResidentKind kind, const Geom &g, bool stream_draws, bool heat_bath, int sm_count,
                          ResidentPlan &p);
// Barriers of a launch of `samples` times `sweeps` sweeps.
uint64_t resident_barriers(const ResidentPlan &p, int passes, uint64_t samples, uint64_t sweeps, bool sampling);
cudaError_t launch_resident(const ResidentPlan &p, ResidentArgs a, cudaStream_t stream);

}  // namespace plq
