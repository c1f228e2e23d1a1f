// ne2b_cluster.cuh — the cluster kernel: one thread-block cluster per net,
// many steps per launch (included by ne2b_step.cuh's translation units).
//
// A net of up to a few tens of thousands of neurons runs on one cluster of
// 1 to 16 blocks.  Each block owns a contiguous range of the net's neurons
// whose state stays in its registers for the whole launch, or, past a neuron
// per thread, in its shared memory (16 bytes per neuron); the steps are separated by the hardware's
// cluster barrier, which costs a fraction of a kernel boundary or of a
// software grid barrier.  Nets of an engine share nothing, so the clusters
// of a batch or of the server run on without waiting for one another.
//
// A net whose shortest synaptic delay is B steps needs a barrier only every
// B steps (a hop): a spike of step t lands in slot t + d, d >= B, so every
// slot of steps [T, T + B) is complete when step T starts.  Each neuron then
// runs B steps at once from registers, its ring words loaded ahead, and the
// spikes of the B steps are listed in shared memory and delivered together
// after a block barrier.  With B = 1 (ONE) each warp delivers its own spikes
// at once.  The nets that run here have kRingSpare ring slots beyond their
// longest delay, so no delivery of a hop lands in a slot that the hop reads.
//
// What orders the ring between blocks (ne2b_layout.h, release_due):
//   add -> read   an add of hop h is read in a later hop: the warp that added
//                 releases at the barrier between them;
//   read, clear -> add   a slot read and cleared at step t is added to again
//                 at step t + kRingSpare + 1 at the earliest: every warp
//                 releases often enough that one of its releases lies between.
// Every warp acquires at every barrier.  The spike lists of a block are
// written before, and read after, a block barrier; they are written again
// after the cluster barrier, at which the warps that read them (they deliver)
// release.  The hop's counters take turns among three sets: a set is cleared
// one block barrier after its last read and one before its next use.
//
// The arithmetic per neuron is process_tile's, in its order (ne2b_step.cuh).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ne2b_device.cuh"
#include "ne2b_step_kind.h"

namespace ne2b {

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_blocks() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// All threads of the cluster (of the block when it is alone).  Every warp
// acquires; a relaxed arrival orders nothing that the warp did before it.
// 0.16 us for 16 blocks of 512 threads when no warp releases, 0.3 when all do,
// 0.6 with ring writes in flight.
__device__ __forceinline__ void cluster_barrier(uint32_t blocks, bool release) {
    if (blocks == 1u) {
        __syncthreads();
        return;
    }
    if (release) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    else asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A spiking neuron's CSR row into ring slot (ts + delay) % D, strided by the
// `lanes` lanes of a group (this one is `gl`), four synapses per lane and
// pass, their loads in flight before the adds; a lane past the row's end
// repeats its first synapse's load and skips the add.
template <bool INT>
__device__ __forceinline__ void deliver_row(const NetDev &nd, uint32_t rlo, uint32_t len, uint32_t ts, uint32_t gl,
                                            uint32_t lanes, uint64_t pol) {
    constexpr int U = 4;
    const uint32_t D = nd.D, n_pad = nd.n_pad, flags = nd.flags;
    const bool wide = flags & kNetDelayWide;
    const SynRec *__restrict__ csr = nd.syn + rlo;
    uint32_t *__restrict__ ringw = (uint32_t *)nd.ring;
    for (uint32_t f = gl; f < len; f += lanes * U) {
        uint2 r[U];
#pragma unroll
        for (int q = 0; q < U; ++q)
            r[q] = *reinterpret_cast<const uint2 *>(csr + (f + lanes * q < len ? f + lanes * q : f));
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const uint32_t j = f + lanes * q;
            if (j >= len) continue;
            const uint32_t d = wide ? (uint32_t)nd.delay16[rlo + j] : r[q].x >> kSynTgtBits;
            uint32_t slot = ts + d;
            if (slot >= D) slot -= D;
            const uint32_t tg = wide ? r[q].x : r[q].x & kSynTgtMask;
            ring_add<INT>(ringw + (size_t)slot * n_pad + tg, r[q].y, pol);
        }
    }
}

__device__ __forceinline__ uint32_t add_mod(uint32_t a, uint32_t b, uint32_t m) {  // a < m, b <= m
    const uint32_t r = a + b;
    return r >= m ? r - m : r;
}

// FULL: record rows, the f32 trace or watches are used by some net of the
// engine; else their code is compiled out.
// A block with a thread for each neuron keeps their state in registers for
// the whole launch; with LOOP its range is larger, the threads take it in
// passes, and the state waits in shared memory between the passes of a hop.
// ONE: every net of the launch has hop 1.
template <bool INT, bool ADEX, bool FULL, bool LOOP, bool ONE>
__global__ void __launch_bounds__(kClMaxThreads) cluster_kernel(const EngineDev *__restrict__ eng,
                                                               const ClusterNet *__restrict__ plan, uint32_t steps) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(16) NetDev s_nd;
    __shared__ __align__(16) ParamRow s_ptab[kSmemParamRows];
    const uint32_t T = blockDim.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t C = cluster_blocks(), rank = cluster_rank();
    const ClusterNet cn = plan[blockIdx.x / C];
    for (uint32_t w = threadIdx.x; w < sizeof(NetDev) / 16; w += T)
        reinterpret_cast<uint4 *>(&s_nd)[w] = reinterpret_cast<const uint4 *>(eng->nets + cn.net)[w];
    const uint32_t np = eng->n_params;
    if (np <= kSmemParamRows)
        for (uint32_t w = threadIdx.x; w < np * (sizeof(ParamRow) / 16); w += T)
            reinterpret_cast<uint4 *>(s_ptab)[w] = reinterpret_cast<const uint4 *>(eng->ptab)[w];
    const ParamRow *ptab = np <= kSmemParamRows ? s_ptab : eng->ptab;
    __syncthreads();
    const NetDev &nd = s_nd;
    const uint32_t flags = nd.flags;
    const uint64_t t0 = nd.t;
    if (!(flags & kNetActive) || t0 >= nd.t_end) return;  // uniform across the cluster
    if (nd.t_end - t0 < steps) steps = (uint32_t)(nd.t_end - t0);
    const uint32_t n = nd.n, n_pad = nd.n_pad, D = nd.D, m = cn.m, B = ONE ? 1u : nd.hop;
    const uint32_t start = min(rank * m, n_pad), cnt = min(m, n_pad - start);  // multiples of 32

    // the hop's spikes: three sets of [step] counters, then [step][m] local
    // neurons (u16); then (LOOP) the state
    uint32_t *sets = reinterpret_cast<uint32_t *>(smem);
    uint16_t *slist = reinterpret_cast<uint16_t *>(sets + (ONE ? 0u : 3u * kMaxHop));
    float *sv = reinterpret_cast<float *>(slist + (ONE ? 0u : m * B));
    float *su = sv + m, *ss = su + m;
    uint16_t *slast = reinterpret_cast<uint16_t *>(ss + m), *spi = slast + m;
    if (!ONE) {
        for (uint32_t w = threadIdx.x; w < 3u * kMaxHop; w += T) sets[w] = 0u;
        __syncthreads();
    }

    // last: 1 + the launch's step of the neuron's last spike, 0 before any;
    // the trace's step count follows from it when the launch ends
    float v = 0.0f, u = 0.0f, s = 0.0f;
    uint32_t last = 0u, pi = 0u;
    if (!LOOP) {
        if (threadIdx.x < cnt) {
            const uint32_t i = start + threadIdx.x;
            v = nd.v[i];
            u = nd.u[i];
            s = nd.s[i];
            pi = nd.pidx[i];
        }
    } else {
        for (uint32_t o = threadIdx.x; o < cnt; o += T) {
            const uint32_t i = start + o;
            sv[o] = nd.v[i];
            su[o] = nd.u[i];
            ss[o] = nd.s[i];
            slast[o] = 0;
            spi[o] = nd.pidx[i];
        }
    }

    uint32_t *__restrict__ ringw = (uint32_t *)nd.ring;
    const float dt = nd.dt, decay_s = nd.decay_s;
    const float kick = nd.kick, gauss_k = nd.gauss_k;
    const bool kicks = nd.pkick > 0.0f, gauss = gauss_k != 0.0f;
    const uint32_t kick_last = nd.kick_last;
    const bool has_ext = flags & kNetHasExt, windows = flags & kNetWindows;
    const bool record = FULL && (flags & kNetRecord);
    const bool has_stim = nd.stim_ptr && cnt > 0 && start < n && nd.stim_ptr[start] < nd.stim_ptr[min(start + cnt, n)];
    uint32_t tm = nd.tmod, rrow = nd.rphase;
    uint64_t nbase = nd.noise_step;
    // the window that the coming steps belong to, and its steps left
    uint32_t wleft = !windows ? ~0u : nd.wphase == 0u ? 1u : nd.win_steps - nd.wphase + 1u;
    uint32_t widx = nd.wphase == 0u ? nd.widx0 - 1u : nd.widx0;
    uint32_t nspk = 0;  // this warp's spikes (warp-uniform)

    // what a thread needs of its neuron besides its state; constant over
    // the launch (LOOP: over the pass)
    bool act = false;  // whole warps: cnt is a multiple of 32
    float ext = 0.0f, gain = 1.0f, p[ADEX ? 10 : 4];
    uint32_t slo = 0u, shi = 0u;
    auto load_consts = [&](uint32_t o0) {
        const uint32_t i = start + o0 + threadIdx.x;
        act = o0 + warp * 32u < cnt;
        ext = has_ext && act ? nd.ext[i] : 0.0f;
        slo = shi = 0u;
        if (has_stim && act && i < n) {
            slo = nd.stim_ptr[i];
            shi = nd.stim_ptr[i + 1];
        }
        const ParamRow &pr = ptab[pi & ~kParamAdexBit];
        const float4 p0 = *reinterpret_cast<const float4 *>(&pr.p[0]);
        p[0] = p0.x; p[1] = p0.y; p[2] = p0.z; p[3] = p0.w;
        if (ADEX) {
            const float4 p1 = *reinterpret_cast<const float4 *>(&pr.p[4]);
            const float2 p2 = *reinterpret_cast<const float2 *>(&pr.p[8]);
            p[ADEX ? 4 : 0] = p1.x; p[ADEX ? 5 : 0] = p1.y;
            p[ADEX ? 6 : 0] = p1.z; p[ADEX ? 7 : 0] = p1.w;
            p[ADEX ? 8 : 0] = p2.x; p[ADEX ? 9 : 0] = p2.y;
            gain = (pi & kParamAdexBit) ? p[0] : 1.0f;  // model/mod.rs:104-106, adex.rs:189-191
        }
    };
    if (!LOOP) load_consts(0u);
    const uint64_t pol = ring_policy();
    // lanes that share a row in a hop's delivery: a group covers an average
    // row in one pass of four synapses per lane
    uint32_t glanes = 32u;
    if (!ONE) {
        const uint32_t e_avg = n ? nd.rowptr[n] / n : 0u;
        glanes = e_avg <= 32u ? 8u : e_avg <= 64u ? 16u : 32u;
    }

    uint32_t set = 0u, since = 0u;  // this hop's counters; steps since every warp released
    for (uint32_t s0 = 0; s0 < steps;) {
        const uint32_t nb = ONE ? 1u : min(min(B, steps - s0), wleft);  // a window ends with a hop
        uint32_t *scnt = sets + set * kMaxHop;
        bool wrote = false;  // this warp added to the ring
        for (uint32_t o0 = 0; o0 < (LOOP ? cnt : 1u); o0 += T) {
            const uint32_t o = o0 + threadIdx.x, i = start + o;
            if (LOOP) {
                if (o0 + warp * 32u < cnt) {
                    v = sv[o];
                    u = su[o];
                    s = ss[o];
                    last = slast[o];
                    pi = spi[o];
                }
                load_consts(o0);
            }
            // ring words are loaded two steps ahead (the loop is not
            // unrolled: a launch of a few steps is bound by fetching its
            // instructions)
            auto fetch = [&](uint32_t b) -> uint32_t {
                if (!act || b >= nb) return 0u;
                return __ldcg(ringw + (size_t)(ONE ? tm : add_mod(tm, b, D)) * n_pad + i);
            };
            uint32_t w0 = fetch(0u), w1 = fetch(1u);
            uint32_t slot = tm, row = rrow;
            uint64_t nbase_b = nbase;
#pragma unroll 1
            for (uint32_t b = 0; b < nb; ++b) {
                const float arr = INT ? __fmul_rn(__int2float_rn((int)w0), 0x1p-12f)  // rt_get, kernels.rs:60
                                      : __uint_as_float(w0);
                if (w0 != 0u) ringw[(size_t)slot * n_pad + i] = 0u;
                w0 = w1;
                w1 = fetch(b + 2u);
                const float sc = __fadd_rn(s, arr);
                float I = __fadd_rn(sc, ext);
                if (slo < shi) {
                    const long long rel = (long long)(t0 + s0 + b) - nd.stim_t0;
                    if (rel >= 0 && rel < (long long)nd.stim_len) {
                        const float *in = nd.stim_buf + (size_t)rel * nd.n_inputs;
                        for (uint32_t x = slo; x < shi; ++x)
                            I = __fadd_rn(I, __fmul_rn(nd.stim_w[x], in[nd.stim_in[x]]));
                    }
                }
                if (kicks && noise_fires(noise_base_at(i, nbase_b), kick_last)) I = __fadd_rn(I, __fmul_rn(kick, gain));
                if (gauss) I = __fadd_rn(I, __fmul_rn(gauss_numer(i, nbase_b), __fmul_rn(gauss_k, gain)));
                bool sp = (ADEX && (pi & kParamAdexBit)) ? adex_step(p, v, u, I, dt) : izh_step(p, v, u, I, dt);
                sp = sp && act && i < n;
                s = __fmul_rn(sc, decay_s);
                if (FULL && act && i < n) {
                    if (flags & kNetTraceF32) {  // a readout tau too long for the step table
                        const float tr = nd.trace_f[i];
                        const float tn = sp ? 1.0f : __fmul_rn(tr, nd.decay_t);
                        if (__float_as_uint(tn) != __float_as_uint(tr)) nd.trace_f[i] = tn;
                    }
                    const uint32_t w = (flags & kNetWatch) ? nd.watch_idx[i] : kNoWatch;
                    if (w != kNoWatch) {  // state after the step, cpu.rs:311-324
                        const size_t pos = (size_t)((t0 + s0 + b) & (kWatchCap - 1u));
                        nd.watch_ring[(size_t)w * kWatchCap + pos] = v;
                        nd.watch_ring[((size_t)nd.watch_n + w) * kWatchCap + pos] = u;
                    }
                }
                const uint32_t word = __ballot_sync(0xffffffffu, sp);
                if (record && lane == 0 && act) nd.rec_bits[(size_t)row * (n_pad >> 5) + (i >> 5)] = word;
                if (word) {
                    nspk += __popc(word);
                    uint32_t lo = 0, hi = 0;
                    if (ONE && sp) {
                        lo = nd.rowptr[i];
                        hi = nd.rowptr[i + 1];
                    }
                    if (sp) {
                        last = s0 + b + 1u;
                        atomicAdd(nd.pn_total + i, 1ull);  // no return: nothing waits for it
                        if (windows) nd.wcount[i] += 1u;
                        if (FULL && (flags & kNetGridWatch)) {  // cpu.rs:293-304
                            const uint64_t t = t0 + s0 + b;
                            const uint32_t t32 = t < 0xFFFFFFFEull ? (uint32_t)t : 0xFFFFFFFEu;
                            for (uint32_t g = 0; g < nd.gw_n; ++g) {
                                const int32_t x = nd.gw_map[(size_t)g * n_pad + i];
                                if (x >= 0) nd.gw_ls[nd.gw_off[g] + (uint32_t)x] = t32;
                            }
                        }
                    }
                    if (ONE) {  // deliver this warp's spikes now, a row at a time
                        wrote = true;
                        for (uint32_t bits = word; bits; bits &= bits - 1u) {
                            const int l = __ffs(bits) - 1;
                            const uint32_t rlo = __shfl_sync(0xffffffffu, lo, l);
                            const uint32_t len = __shfl_sync(0xffffffffu, hi, l) - rlo;
                            deliver_row<INT>(nd, rlo, len, tm, lane, 32u, pol);
                        }
                    } else {
                        uint32_t pos = 0;
                        if (lane == 0) pos = atomicAdd(scnt + b, (uint32_t)__popc(word));
                        pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(word & ((1u << lane) - 1u));
                        if (sp) slist[b * m + pos] = (uint16_t)(o0 + threadIdx.x);
                    }
                }
                if (++slot == D) slot = 0;
                if (record && ++row == nd.rec_rows) row = 0;
                nbase_b += kNoiseStepMul;
            }
            if (LOOP && act) {
                sv[o] = v;
                su[o] = u;
                ss[o] = s;
                slast[o] = (uint16_t)last;
            }
            if (windows && wleft == nb && act && i < n) {  // the window ends
                const uint32_t c = nd.wcount[i];
                if (widx < nd.max_windows) nd.win_out[(size_t)widx * n_pad + i] = (uint16_t)(c > 65535u ? 65535u : c);
                if (c) nd.wcount[i] = 0u;
            }
        }
        nbase += (uint64_t)nb * kNoiseStepMul;
        if (record) {
            rrow += nb;
            while (rrow >= nd.rec_rows) rrow -= nd.rec_rows;
        }
        if (windows && (wleft -= nb) == 0u) {
            wleft = nd.win_steps;
            ++widx;
        }
        if (!ONE) {
            __syncthreads();  // the block's lists are complete
            const uint32_t after = set == 0u ? 2u : set - 1u;  // the set of the hop after next
            if (threadIdx.x < kMaxHop) sets[after * kMaxHop + threadIdx.x] = 0u;
            set = set == 2u ? 0u : set + 1u;
            // the block's spikes of the hop, one per group of lanes
            uint32_t total = 0;
            for (uint32_t b = 0; b < nb; ++b) total += scnt[b];
            const uint32_t gl = threadIdx.x & (glanes - 1u);
            for (uint32_t r = threadIdx.x / glanes; r < total; r += T / glanes) {
                uint32_t b = 0, k = r;
                while (k >= scnt[b]) k -= scnt[b++];
                const uint32_t i = start + slist[b * m + k];
                const uint32_t rlo = nd.rowptr[i], len = nd.rowptr[i + 1] - rlo;
                deliver_row<INT>(nd, rlo, len, add_mod(tm, b, D), gl, glanes, pol);
                wrote = true;
            }
            wrote = __any_sync(0xffffffffu, wrote);
        }
        since += nb;
        const bool due = release_due(since, B);
        cluster_barrier(C, wrote || due);  // the deliveries have landed before the next hop reads
        if (due) since = 0u;
        tm = add_mod(tm, nb, D);
        s0 += nb;
    }

    // the trace after k steps without a spike is entry k of the step table
    // (saturating at its last entry), counted from the last spike of the
    // launch or from the count before it
    const uint32_t tlast = nd.trace_last;
    auto trace_steps = [&](uint32_t i, uint32_t spiked) -> uint16_t {
        if (spiked) return (uint16_t)min(steps - spiked, tlast);
        const uint32_t k = nd.tk[i];
        return (uint16_t)(k == kTraceZero ? k : min(k + steps, tlast));
    };
    const bool table = !(FULL && (flags & kNetTraceF32));
    if (!LOOP) {
        const uint32_t i = start + threadIdx.x;
        if (threadIdx.x < cnt) {
            nd.v[i] = v;
            nd.u[i] = u;
            nd.s[i] = s;
            if (table) nd.tk[i] = trace_steps(i, last);
        }
    } else {
        for (uint32_t o = threadIdx.x; o < cnt; o += T) {
            const uint32_t i = start + o;
            nd.v[i] = sv[o];
            nd.u[i] = su[o];
            nd.s[i] = ss[o];
            if (table) nd.tk[i] = trace_steps(i, slast[o]);
        }
    }
    if (lane == 0 && nspk) atomicAdd(&eng->counters[cn.net].spikes_total, (unsigned long long)nspk);
    // every block of the cluster copied the descriptor before the barriers
    // above, so its step may move on now
    if (rank == 0 && threadIdx.x == 0) set_step(eng->nets[cn.net], t0 + steps);
}

}  // namespace ne2b
