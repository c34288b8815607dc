// Host-side launch interface of the per-step kernels and the device network builder.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "dtb_device.cuh"

namespace dtb {

// Windows of the population-window push over a batch.
struct LocalPlan {
    const uint32_t* win_prefix;   // device [n_nets + 1] cumulative windows
    uint32_t windows;
    uint32_t dense_min;           // spikes from which a step takes the windows
    uint32_t always;              // 1: every population with a spike takes its windows
    uint32_t unit_target;         // work units wanted in a busy step (a few per SM)
    uint32_t flush_reds;          // reductions a window neuron costs to flush: 1 (float), 2 (fixed)
    uint32_t* scratch;            // device [local_scratch_words(windows)], see local_prep
    uint32_t* live;               // device [pops] every network's NetView::pop_live, network by network in one array, so that
    uint32_t pops;                // one flat loop empties them (64 quiet networks: 0.7 us a step; a turn per network took 13 us)
};
inline size_t local_scratch_words(size_t windows) { return 2 * windows + 4; }
constexpr uint32_t kUnitsPerSm = 4;

// Events (spikes x mean out-degree) from which a step takes the windows.  Scattered rows run at
// 6.0 to 6.5 ps per event; the windows cost about 3.5 ps and 40 to 60 us of preparation, unit
// start-up and uneven ends.  Measured, windows against scatter: 86 / 41 us at 6.0e6 events (250k
// neurons, BF16, fixed), 84 / 82 us at 1.3e7, 110 / 118 us at 1.9e7 (200k, FP32, float),
// 158 / 217 us at 3.2e7.  All four are single networks; a batch uses the same line, and whether its
// windows, spread over the members, pay over a run is the tuner's to find.
constexpr uint64_t kDenseEvents = 16000000;
// Networks whose every synapse together stays below kDenseEvents never take windows, and the
// register-staged forms are within 5 % of each other on them (8.1 to 8.6 us on the 10,000-neuron
// block): the tuner's reads, a synchronisation each, and the eager steps around them would cost
// more than it could choose (10,000 neurons, 100 steps: 1325 us tuned, 1298 us untouched).
inline bool worth_tuning(uint64_t edges) { return edges >= kDenseEvents; }
inline uint32_t dense_min_spikes(uint64_t edges, uint64_t neurons) {
    const uint64_t c = edges ? kDenseEvents * neurons / edges : 1u;
    return static_cast<uint32_t>(c < 1 ? 1 : c > 0x7fffffffu ? 0x7fffffffu : c);
}

// One launch group: a batch of networks advanced together.
struct LaunchBatch {
    const NetView* nets;          // device array [n_nets]
    const uint32_t* lif_prefix;   // device [n_nets + 1] cumulative LIF tiles (1024 neurons)
    const uint32_t* tile_net;     // device [lif tiles] network of every LIF tile (batches), or null
    const uint32_t* pull_prefix;  // device [n_nets + 1] cumulative pull tiles (256 neurons)
    const uint32_t* vbase;        // device [n_nets + 1] cumulative padded neuron counts
    uint32_t n_nets;
    uint32_t lif_tiles_total;
    uint32_t pull_tiles_total;
    uint32_t pull_degree;         // mean in-edges of a neuron
    uint32_t push_ctas;
    uint32_t lif_ctas;            // persistent grid of the LIF kernel
    uint32_t lif_chunk;           // consecutive tiles a LIF CTA steps before striding (0 or 1: one)
    LocalPlan local;              // population-window push (windows 0: none)
    uint32_t sm_count;
    SpikeList spikes;
};

cudaError_t launch_lif(const LaunchBatch& b, int jmode, uint32_t flags, int prop_mode, cudaStream_t s);
// Push kernel variants chosen by the autotuner.
enum PushKind : int { PUSH_REG = 0, PUSH_TMA = 1, PUSH_LOCAL = 2 };
struct PushCfg {
    int kind;    // PUSH_REG: register-staged loads, param = synapses in flight per lane (4, 8, 16)
                 // PUSH_TMA: bulk-copy staged rows, param = synapses per stage (256, 512)
                 // PUSH_LOCAL: in busy steps own-population synapses are summed per window in shared
                 //   memory and the rest scattered; quiet steps scatter whole rows
    int param;
    int lpr = 32;  // PUSH_REG: lanes per row (32, 16, 8; sub-warp rows use 8 in flight per lane)
};

// The variant of a network (or batch) that is not tuned, or not yet: a warp per row, or a quarter
// warp for rows that would leave most of a warp idle.  Eight synapses in flight by 32 against by 8
// lanes: 32.1 / 30.1 us a step with 15 synapses a row (1M neurons, 1.1 % of them spiking), 37.1 /
// 34.9 with 10 (1.5M), 45.8 / 43.5 with 5 (2M), 24.6 / 24.6 with 30 (500,000) and 18.5 / 18.5 with
// 50 (300,000).
constexpr uint64_t kShortRow = 24;
inline PushCfg default_push(uint64_t edges, uint64_t neurons) { return PushCfg{PUSH_REG, 8, edges < kShortRow * neurons ? 8 : 32}; }

// Every variant the autotuner times.
constexpr int kPushCandidates = 12;
// PUSH_LOCAL params: 8 (and 8 with 16 lanes per cross-population row) give every warp to the
// windows first; the others start some of each CTA's warps on the cross-population rows at once
constexpr int kLocalConcurrent = 2008;   // 24 warps on the windows, 8 on the cross-population rows
constexpr int kLocalConcurrent2 = 2016;  // 16 and 16
constexpr int kLocalConcurrentHalf = 3008;  // as 2008 with half-warp rows in the windows (short spans)
extern const PushCfg kPushCands[kPushCandidates];
// Sets kernel attributes and returns the persistent grid (max resident CTAs).
// `acc` is the AccMode of the launch (float, exact or fixed-point accumulators).
cudaError_t push_prepare(int acc, int weight_type, const PushCfg& cfg, int sm_count, uint32_t* ctas);
cudaError_t launch_push(const LaunchBatch& b, int acc, int weight_type, const PushCfg& cfg, uint32_t ctas,
                        cudaStream_t s);
cudaError_t launch_pull(const LaunchBatch& b, int gather, int weight_type, uint32_t flags, int prop_mode, cudaStream_t s);
cudaError_t launch_fold_finish(const LaunchBatch& b, int acc, cudaStream_t s);
// Per-population sums of the end-of-step synaptic currents (after the push of
// the step; with exact or fixed accumulators J still lacks the step's sums).
cudaError_t launch_stat_isyn(const LaunchBatch& b, int acc, int sm_count, cudaStream_t s);
cudaError_t launch_gather_finish(const LaunchBatch& b, int weight_type, cudaStream_t s);

// Population-local push tables (rows must be sorted by postsynaptic neuron;
// *unsorted is set otherwise).  Pass 1 (woff == nullptr): per-neuron own-
// population in-degree into own_cnt, per-population max |w| (float bits) into
// maxw_bits; pass 2: own_seg and woff from pop_loc.
cudaError_t build_local_offsets(const unsigned long long* out_ptr, const uint32_t* out_col, const void* out_w, int wt,
                                const uint32_t* pop_off, uint32_t n_pops, uint32_t n, const uint4* pop_loc,
                                uint32_t* own_cnt, uint32_t* maxw_bits, uint2* own_seg, uint32_t* woff,
                                uint32_t* unsorted, cudaStream_t s);

// ---- device network generator (dtb_generate.cu)
struct GenSpec {
    uint32_t n, n_pops, in_degree, dyadic;
    unsigned long long seed;
    const uint32_t* pop_off;          // device [n_pops + 1]
    const uint32_t* pop_exc;          // device [n_pops]
    const unsigned long long* cdf;    // device [n_pops * n_pops]
};

// Builds the requested CSRs on the device.  out_* / in_* may be null when not
// wanted.  Temporary device memory is allocated and released inside.
cudaError_t build_structured(const GenSpec& g, int weight_type,
                             unsigned long long* out_ptr, uint32_t* out_col, void* out_w,
                             unsigned long long* in_ptr, uint32_t* in_col, void* in_w,
                             uint32_t* out_deg, cudaStream_t s);

// Host mirror of one generated edge (used by the host builder for small networks
// and by the tests through the oracle).
void host_gen_edge(uint32_t n_pops, const uint32_t* pop_off, const uint32_t* pop_exc,
                   const unsigned long long* cdf, unsigned long long seed, uint32_t dyadic,
                   uint32_t post, uint32_t pop_of_post, uint32_t k,
                   uint32_t* pre, uint32_t* kind, float* w0, float* w1);

}  // namespace dtb
