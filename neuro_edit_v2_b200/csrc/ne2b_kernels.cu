// ne2b_kernels.cu — the helper kernels (advance, reset, trace and window
// readouts) and the host launchers; the step kernels themselves are in
// ne2b_step.cuh, instantiated per kind in ne2b_step_k*.cu.
#include <cuda_runtime.h>
#include <stdint.h>

#include "ne2b_kernels.h"
#include "ne2b_step.cuh"

namespace ne2b {

// Advance every active net by `steps` after a launch group (t and t % D).
__global__ void advance_kernel(NetDev *nets, uint32_t n_nets, uint32_t steps) {
    pdl_enter();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_nets) return;
    NetDev &nd = nets[j];
    if (!(nd.flags & kNetActive)) return;
    unsigned long long t = nd.t + steps;
    if (t > nd.t_end) t = nd.t_end;
    set_step(nd, t);
}

// reset_state for one net (cpu.rs:158-183): state rows from v0/u0, zeros.
__global__ void reset_neurons_kernel(NetDev nd) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nd.n_pad) return;
    nd.v[i] = nd.v0[i];
    nd.u[i] = nd.u0[i];
    nd.s[i] = 0.0f;
    nd.tk[i] = kTraceZero;
    nd.pn_total[i] = 0ull;
    if (nd.wcount) nd.wcount[i] = 0u;
}

// Backend::trace (lib.rs:137): trace_tab[tk], 0 for kTraceZero.
__global__ void trace_kernel(const uint16_t *tk, const float *tab, uint32_t n, float *out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint16_t k = tk[i];
    out[i] = k == kTraceZero ? 0.0f : tab[k];
}

// spike_counts over the last `rows` record rows (cpu.rs:424-458): a block
// takes 32 record words (1024 neurons); warp w adds rows w, w + 32, ... with
// each lane holding one word, whose 32 bits it adds into a 32-bit counter per
// bit kept as eight planes of byte counters (a mask and an add for every four
// bits), emptied into the block's totals in shared memory every 252 rows.
// Bound by the record's bytes from L2.  (A thread per neuron, one 64-bit
// modulo and one shared word per row, took 0.2 ms more for 500 rows of 100k
// neurons.)
__global__ void __launch_bounds__(1024) window_count_kernel(const uint32_t *__restrict__ rec_bits, uint32_t rec_rows,
                                                            uint32_t n_pad, uint32_t n, uint32_t first, uint32_t rows,
                                                            uint32_t *__restrict__ out) {
    __shared__ uint32_t total[32][33];  // [word][bit]
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t words32 = n_pad >> 5, word = blockIdx.x * 32u + lane;
    total[warp][lane] = 0u;
    __syncthreads();
    // plane p, byte b counts bit p + 8 b
    uint32_t plane[8] = {};
    uint32_t held = 0;
    auto empty = [&]() {
#pragma unroll
        for (uint32_t p = 0; p < 8u; ++p) {
#pragma unroll
            for (uint32_t b = 0; b < 4u; ++b) {
                const uint32_t c = (plane[p] >> (8u * b)) & 0xffu;
                if (c) atomicAdd(&total[lane][p + 8u * b], c);
            }
            plane[p] = 0u;
        }
        held = 0;
    };
    for (uint32_t r0 = warp; r0 < rows; r0 += 32u * 4u) {
        uint32_t v[4];
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
            const uint32_t r = r0 + 32u * q;
            uint32_t row = first + r;  // first < rec_rows, r < rows <= rec_rows
            if (row >= rec_rows) row -= rec_rows;
            v[q] = r < rows && word < words32 ? rec_bits[(size_t)row * words32 + word] : 0u;
        }
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q)
#pragma unroll
            for (uint32_t p = 0; p < 8u; ++p) plane[p] += (v[q] >> p) & 0x01010101u;
        if ((held += 4u) > 251u) empty();
    }
    empty();
    __syncthreads();
    // one neuron per thread, in order
    const uint32_t i = blockIdx.x * 1024u + threadIdx.x;
    if (i < n) out[i] = total[warp][lane];
}

// pn_total saturated to u32 (cpu.rs:432-436).
__global__ void pn_total_kernel(const unsigned long long *pn, uint32_t n, uint32_t *out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long c = pn[i];
    out[i] = c > 0xffffffffull ? 0xffffffffu : (uint32_t)c;
}

// A warp per row: does it hold a synapse of delay 1?
__global__ void urgent_kernel(NetDev nd, uint32_t *bits, uint32_t *count) {
    const uint32_t lane = threadIdx.x & 31u, nw = gridDim.x * (blockDim.x >> 5);
    for (uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < nd.n; i += nw) {
        const uint32_t lo = nd.rowptr[i], hi = nd.rowptr[i + 1];
        bool one = false;
        for (uint32_t j = lo + lane; j < hi; j += 32u)
            one |= ((nd.flags & kNetDelayWide) ? (uint32_t)nd.delay16[j] : nd.syn[j].td >> kSynTgtBits) == 1u;
        if (__any_sync(0xffffffffu, one) && lane == 0u) {
            atomicOr(bits + (i >> 5), 1u << (i & 31u));
            atomicAdd(count, 1u);
        }
    }
}

// Self-test of the bounded grid barrier: every block but `absent` arrives,
// so the others give up after `limit_ns`, set the error flag and return
// (a wait that cannot end, ended by its limit, with no fault).
__global__ void barrier_selftest_kernel(unsigned int *counter, unsigned int *err, uint32_t absent,
                                        unsigned long long limit_ns) {
    __shared__ unsigned int s_flag;
    if (blockIdx.x == absent) return;
    grid_barrier(counter, gridDim.x, err, &s_flag, limit_ns);
}

// ------------------------------------------------------------- launchers
bool shape_supported(uint32_t block, uint32_t npt) {
#define X(B, P) if (block == B && npt == P) return true;
    NE2B_SHAPES(X)
#undef X
    return false;
}

bool ws_shape_supported(uint32_t block, uint32_t npt) {
#define X(B, P) if (block == B && npt == P) return true;
    NE2B_WS_SHAPES(X)
#undef X
    return false;
}

void shape_list(uint32_t *blocks, uint32_t *npts, uint32_t *count) {
    uint32_t c = 0;
#define X(B, P) blocks[c] = B; npts[c] = P; ++c;
    NE2B_SHAPES(X)
#undef X
    *count = c;
}

static bool g_pdl = true;
void set_pdl(bool on) { g_pdl = on; }
bool pdl_enabled() { return g_pdl; }

// Kernel variants: INT (int32 fixed-point ring) x ADEX (AdEx rows present;
// an all-Izhikevich engine runs the instance without the AdEx path).
#define NE2B_KIND(int_ring, adex, call)                                  \
    ((int_ring) ? ((adex) ? StepKind<true, true>::call : StepKind<true, false>::call) \
                : ((adex) ? StepKind<false, true>::call : StepKind<false, false>::call))

int step_occupancy(bool int_ring, bool adex, int variant, uint32_t block, uint32_t npt) {
    return NE2B_KIND(int_ring, adex, occupancy(block, npt, variant));
}

cudaError_t launch_step(bool int_ring, bool adex, int variant, uint32_t block, uint32_t npt, const EngineDev *eng,
                        uint32_t k_step, uint32_t grid, cudaStream_t st) {
    return NE2B_KIND(int_ring, adex, launch(block, npt, variant, eng, k_step, grid, st));
}

uint32_t resident_head(uint32_t block, uint32_t npt) {
#define X(B, P) if (block == B && npt == P) return resident_head_bytes<B, P>();
    NE2B_SHAPES(X)
#undef X
    return 0;
}

int resident_occupancy(bool int_ring, bool adex, uint32_t block, uint32_t npt, size_t smem) {
    return NE2B_KIND(int_ring, adex, resident_occupancy(block, npt, smem));
}

cudaError_t launch_resident(bool int_ring, bool adex, uint32_t block, uint32_t npt, const EngineDev *eng,
                            uint32_t k0, uint32_t nsteps, uint32_t grid, size_t smem, cudaStream_t st) {
    return NE2B_KIND(int_ring, adex, launch_resident(block, npt, eng, k0, nsteps, grid, smem, st));
}

int defer_occupancy(bool int_ring, bool adex, int variant) {
    return NE2B_KIND(int_ring, adex, defer_occupancy(variant));
}

cudaError_t launch_defer(bool int_ring, bool adex, int variant, const EngineDev *eng, uint32_t n_deliver,
                         uint32_t k_step, uint32_t grid, cudaStream_t st) {
    return NE2B_KIND(int_ring, adex, launch_defer(variant, eng, n_deliver, k_step, grid, st));
}

cudaError_t launch_defer_flush(bool int_ring, bool adex, const EngineDev *eng, uint32_t n_deliver, uint32_t steps,
                               cudaStream_t st) {
    return NE2B_KIND(int_ring, adex, launch_defer_flush(eng, n_deliver, steps, st));
}

cudaError_t launch_urgent(const NetDev &nd, uint32_t *bits, uint32_t *count, cudaStream_t st) {
    if (nd.n == 0) return cudaSuccess;
    const uint32_t blocks = (nd.n + 7u) / 8u;
    urgent_kernel<<<blocks < 148u * 32u ? blocks : 148u * 32u, 256, 0, st>>>(nd, bits, count);
    return cudaGetLastError();
}

int cluster_fit(bool int_ring, bool adex, bool full, uint32_t blocks, const ClusterShape &cs, size_t smem) {
    return NE2B_KIND(int_ring, adex, cluster_fit(full, blocks, cs, smem));
}

cudaError_t launch_cluster(bool int_ring, bool adex, bool full, uint32_t blocks, uint32_t clusters,
                           const ClusterShape &cs, size_t smem, const EngineDev *eng, const ClusterNet *plan, uint32_t steps, cudaStream_t st) {
    return NE2B_KIND(int_ring, adex, launch_cluster(full, blocks, clusters, cs, smem, eng, plan, steps, st));
}

cudaError_t launch_barrier_selftest(unsigned int *counter, unsigned int *err, uint32_t blocks, uint32_t absent,
                                    unsigned long long limit_ns, cudaStream_t st) {
    void *args[] = {(void *)&counter, (void *)&err, (void *)&absent, (void *)&limit_ns};
    return cudaLaunchCooperativeKernel((const void *)barrier_selftest_kernel, dim3(blocks), dim3(32), args, 0, st);
}

cudaError_t launch_advance(NetDev *nets, uint32_t n_nets, uint32_t steps, cudaStream_t st) {
    if (n_nets == 0) return cudaSuccess;
    return launch_pdl(advance_kernel, (n_nets + 127) / 128, 128, st, true, nets, n_nets, steps);
}

cudaError_t launch_reset_neurons(const NetDev &nd, cudaStream_t st) {
    if (nd.n_pad == 0) return cudaSuccess;
    reset_neurons_kernel<<<(nd.n_pad + 255) / 256, 256, 0, st>>>(nd);
    return cudaGetLastError();
}

cudaError_t launch_trace(const uint16_t *tk, const float *tab, uint32_t n, float *out, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    trace_kernel<<<(n + 255) / 256, 256, 0, st>>>(tk, tab, n, out);
    return cudaGetLastError();
}

cudaError_t launch_window_count(const uint32_t *rec_bits, uint32_t rec_rows, uint32_t n_pad, uint32_t n,
                                unsigned long long t, uint32_t rows, uint32_t *out, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    // the oldest row of the window
    const uint32_t first = (uint32_t)((t - rows) % rec_rows);
    window_count_kernel<<<(n + 1023) / 1024, 1024, 0, st>>>(rec_bits, rec_rows, n_pad, n, first, rows, out);
    return cudaGetLastError();
}

cudaError_t launch_pn_total(const unsigned long long *pn, uint32_t n, uint32_t *out, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    pn_total_kernel<<<(n + 255) / 256, 256, 0, st>>>(pn, n, out);
    return cudaGetLastError();
}

}  // namespace ne2b
