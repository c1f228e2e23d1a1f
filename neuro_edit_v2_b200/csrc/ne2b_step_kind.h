// ne2b_step_kind.h — the step kernels by kind (internal).  Each of the four
// kinds (int32 or f32 ring) x (with or without the AdEx path) is compiled in
// its own translation unit (ne2b_step_k*.cu) so the kernel instances build in
// parallel; ne2b_kernels.cu dispatches to them.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ne2b_layout.h"

// Tile shapes compiled in: (threads per block, neurons per thread).
#define NE2B_SHAPES(X) \
    X(64, 1) X(64, 2) X(64, 4) X(128, 1) X(128, 2) X(128, 4) X(128, 8) X(256, 1) X(256, 2) X(256, 4) X(256, 8) \
    X(512, 1) X(512, 2) X(512, 4)
// Shapes with an instance of the warp-specialised single-net kernel
// (step_kernel_ws: the tile warps plus separate delivery warps).
#define NE2B_WS_SHAPES(X) \
    X(128, 1) X(128, 2) X(128, 4) X(128, 8) X(256, 1) X(256, 2) X(256, 4) X(256, 8) X(512, 1) X(512, 2) X(512, 4)

namespace ne2b {

bool pdl_enabled();  // programmatic dependent launch of the streaming kernels (ne2b_kernels.cu)

// 32-bit words of the delivery phase's shared lists (SmemLists).
template <int BLOCK, int NPT>
__host__ __device__ constexpr uint32_t smem_lists_words() {
    return 2 * BLOCK * NPT + 1 + 2 * (BLOCK / 32) + 2;
}

// Resident kernel shared memory: [delivery lists][flag u32], 16-byte aligned,
// then the owned state [v M f32][u M f32][s M f32][tk M u16][pidx M u16].
template <int BLOCK, int NPT>
__host__ __device__ constexpr uint32_t resident_head_bytes() {
    return (uint32_t)((smem_lists_words<BLOCK, NPT>() + 1) * 4 + 15) / 16 * 16;
}

// Custom-tau currents that a warp stages at once, and a block's buffer of them
// (behind the resident kernel's state where there is room).
constexpr uint32_t kXChunk = 256;
__host__ __device__ constexpr uint32_t xsyn_buffer_bytes(uint32_t block) { return block / 32u * kXChunk * 4u; }

// Streaming kernel instances: one net with any features, one net without the
// optional ones (external current, stimulus, records, windows, custom-tau
// synapses, f32 trace, watches), many nets (batches, the server), and many
// nets without records, custom-tau synapses, f32 trace or watches.
constexpr uint32_t kDeferBlock = 128;  // threads and neurons of a tile of step_kernel_defer
// Its instances: without the optional features, with them, and with custom-tau
// synapses as well.
enum DeferVariant : int { kDeferPlain = 0, kDeferFull = 1, kDeferXs = 2 };
enum StepVariant : int { kStepSingle = 0, kStepMulti = 1, kStepPlain = 2, kStepMultiLean = 3 };
// Added to kStepSingle or kStepPlain: the warp-specialised instance
// (separate delivery warps; engines of one net, NE2B_WS_SHAPES only).
constexpr int kStepWS = 0x10;
// Added to kStepSingle or kStepMulti: some net has custom-tau synapses.
constexpr int kStepXs = 0x20;

constexpr size_t kClSmemMax = 200 * 1024;  // dynamic shared memory of a cluster kernel block, at most
constexpr uint32_t kClMaxThreads = 1024;  // threads of a cluster kernel block, at most

// A cluster kernel block: threads, whether its range takes several passes of
// them (state in shared memory), and whether every hop is 1.
struct ClusterShape {
    uint32_t threads;
    bool loop, one;
};
// Its shared memory: three sets of spike counters, the lists (u16 per neuron and
// step), then (loop) the state (16 bytes per neuron).
inline uint32_t cluster_smem(uint32_t m, uint32_t hop, const ClusterShape &s) {
    return (s.one ? 0u : 3u * kMaxHop * 4u + m * hop * 2u) + (s.loop ? m * 16u : 0u);
}

template <bool INT, bool ADEX>
struct StepKind {
    static int defer_occupancy(int variant);
    static cudaError_t launch_defer(int variant, const EngineDev *eng, uint32_t n_deliver, uint32_t k_step, uint32_t grid, cudaStream_t st);
    static cudaError_t launch_defer_flush(const EngineDev *eng, uint32_t n_deliver, uint32_t steps, cudaStream_t st);
    // cluster kernel: `clusters` clusters of `blocks` blocks; `full` = with
    // records, the f32 trace and watches (custom-tau nets do not run on it)
    static int cluster_fit(bool full, uint32_t blocks, const ClusterShape &cs, size_t smem);
    static cudaError_t launch_cluster(bool full, uint32_t blocks, uint32_t clusters, const ClusterShape &cs,
                                      size_t smem, const EngineDev *eng, const ClusterNet *plan, uint32_t steps,
                                      cudaStream_t st);
    static int occupancy(uint32_t block, uint32_t npt, int variant);
    static cudaError_t launch(uint32_t block, uint32_t npt, int variant, const EngineDev *eng, uint32_t k_step,
                              uint32_t grid, cudaStream_t st);
    static int resident_occupancy(uint32_t block, uint32_t npt, size_t smem);
    static cudaError_t launch_resident(uint32_t block, uint32_t npt, const EngineDev *eng, uint32_t k0,
                                       uint32_t nsteps, uint32_t grid, size_t smem, cudaStream_t st);
};
extern template struct StepKind<false, false>;
extern template struct StepKind<false, true>;
extern template struct StepKind<true, false>;
extern template struct StepKind<true, true>;

}  // namespace ne2b
