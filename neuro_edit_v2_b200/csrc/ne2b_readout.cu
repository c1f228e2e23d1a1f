// ne2b_readout.cu — readout training on the GPU, from features that are
// already on the device (a batch's per-window spike counts) or that the
// caller passes: the multi-class ridge of sim/src/readout.rs:190-252
// (`fit_ridge_multi`), solved in the dual, and the binary ridge of
// readout.rs:103-141 (`fit_ridge`), solved in the primal.
//
// fit_ridge_multi:
//   1. column means mu (f64, rows summed in order) and the centred design
//      Xc = x - mu (f64);
//   2. the Gram matrix G = Xc Xc^T + lambda I, each entry summed exactly as
//      the reference does (four accumulators by column mod 4, the tail
//      apart, then tail + ((a0 + a1) + a2) + a3);
//   3. Cholesky G = U^T U in place of the upper triangle, in panels of 32
//      rows: every entry meets its subtractions in the same order k = 0, 1,
//      ... as the reference's left-looking loop;
//   4. U^T z = y and U a = z per class on the host (T^2 work).  The second
//      sums ascend from the entry computed last, as the reference's do, so
//      each class is one chain of T^2 / 2 dependent subtractions, which a
//      CPU core runs three times faster than a GPU thread; four classes go
//      side by side;
//   5. w = Xc^T a on the device (rows summed in order), bias on the host.
//
// fit_ridge: the normal matrix of [X 1 y], each entry summed over the rows
// in order as the reference accumulates it (the products with 1 are exact,
// so the bias column and the right-hand side are sums of the same kind),
// lambda on the diagonal and off the bias again ((s + lambda) - lambda, as
// there), the same Cholesky, and the solve on the host; a matrix that is not
// positive definite is refactored with 1e-3 + lambda more on the diagonal
// (from a copy kept on the device), then gives zeros.
//
// Every f64 operation is an explicit round-to-nearest intrinsic, so nothing
// is contracted into an FMA: the weights equal the reference's bit for bit.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <exception>
#include <vector>

#include "ne2b_engine.h"
#include "ne2b_handles.h"
#include "ne2b_solve.h"
#include "ne2b_workspace.h"

#define NE2B_CUDA(call)                                      \
    do {                                                     \
        cudaError_t _e = (call);                             \
        if (_e != cudaSuccess) return cuda_error(_e, #call); \
    } while (0)
#define NE2B_TRY(call)                 \
    do {                               \
        ne2b_status _s = (call);       \
        if (_s != NE2B_OK) return _s;  \
    } while (0)

namespace ne2b {
namespace {

constexpr uint32_t kTile = 32;    // 32 x 32 entries per block, 8 x 8 threads of 4 x 4
constexpr uint32_t kChunk = 32;   // terms staged per pass (a multiple of 4)
constexpr uint32_t kPitch = kTile + 2;  // doubles per staged term: rows stay 16-byte aligned
constexpr uint32_t kPanel = 32;   // Cholesky rows per panel
constexpr uint32_t kUpdTile = 64; // trailing update: 64 x 64 entries per block, 16 x 16 threads of 4 x 4

// linear block id -> (bi, bj), bi <= bj
__device__ __forceinline__ void triangle_tile(uint32_t id, uint32_t &bi, uint32_t &bj) {
    bj = (uint32_t)((sqrt(8.0 * id + 1.0) - 1.0) / 2.0);
    while ((bj + 1) * (bj + 2) / 2 <= id) ++bj;
    while (bj * (bj + 1) / 2 > id) --bj;
    bi = id - bj * (bj + 1) / 2;
}

// A thread's four rows (or columns) of a W-wide tile: 2 k, 2 k + 1, W / 2 + 2 k
// and W / 2 + 2 k + 1, so that neighbouring threads' 16-byte loads are neighbours in
// shared memory (four consecutive ones would collide on every other bank).
template <uint32_t W>
__device__ __forceinline__ uint32_t spread4(uint32_t k, uint32_t e) { return (e >> 1) * (W / 2u) + 2u * k + (e & 1u); }
template <uint32_t W>
__device__ __forceinline__ void load_spread4(const double *row, uint32_t k, double (&v)[4]) {  // row 16-byte aligned
    const double2 a = *reinterpret_cast<const double2 *>(row + 2u * k);
    const double2 b = *reinterpret_cast<const double2 *>(row + W / 2u + 2u * k);
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
}
__device__ __forceinline__ void load4(const double *p, double (&v)[4]) {  // p 16-byte aligned
    const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
}

// 32 columns per block: all four warps stage 128 rows while the first adds
// the 128 before them in order (24 us at 1000 x 4320; T serial loads by F
// threads took 66 us).
__global__ void __launch_bounds__(128) col_mean_kernel(const float *__restrict__ x, uint32_t t, uint32_t f,
                                                       double *__restrict__ mu) {
    constexpr uint32_t R = 128;
    __shared__ float sx[2][R][32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t c = blockIdx.x * 32u + lane;
    auto stage = [&](uint32_t r0, uint32_t buf) {
        float v[R / 4u];
#pragma unroll
        for (uint32_t e = 0; e < R / 4u; ++e) {
            const uint32_t r = r0 + 4u * e + warp;
            v[e] = r < t && c < f ? x[(size_t)r * f + c] : 0.0f;
        }
#pragma unroll
        for (uint32_t e = 0; e < R / 4u; ++e) sx[buf][4u * e + warp][lane] = v[e];
    };
    double s = 0.0;
    stage(0u, 0u);
    __syncthreads();
    for (uint32_t r0 = 0, buf = 0; r0 < t; r0 += R, buf ^= 1u) {
        if (warp == 0u) {
            const uint32_t rn = min(R, t - r0);
#pragma unroll 8
            for (uint32_t r = 0; r < rn; ++r) s = __dadd_rn(s, (double)sx[buf][r][lane]);
        }
        if (r0 + R < t) stage(r0 + R, buf ^ 1u);
        __syncthreads();
    }
    if (warp == 0u && c < f) mu[c] = __ddiv_rn(s, (double)t);
}

__global__ void center_kernel(const float *__restrict__ x, uint64_t n, uint32_t f, const double *__restrict__ mu,
                              double *__restrict__ xc) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        xc[i] = __dsub_rn((double)x[i], mu[i % f]);
}

__device__ __forceinline__ void copy_async8(double *smem, const double *g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
                 : "memory");
}

__device__ __forceinline__ void copy_async16(double *smem, const double *g) {  // both 16-byte aligned
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
                 : "memory");
}

// Upper-triangle tiles of G = Xc Xc^T; the diagonal gets lambda.  Bound by
// the f64 pipe (T^2 F multiplies and adds, never fused): each thread owns
// 4 x 4 entries, so one column's 8 operands from shared memory feed 32
// operations, and the next 32 columns arrive by cp.async meanwhile.  Blocks
// of two warps keep the tiles small: 528 of them at T = 1000, spread evenly.
// Measured at 1000 x 4320: 457 us, 9.4e12
// operations per second (2 x 2 entries per thread, 256 threads: 1076 us).
__global__ void __launch_bounds__(64) gram_kernel(const double *__restrict__ xc, uint32_t t, uint32_t f,
                                                  double lambda, double *__restrict__ g) {
    __shared__ __align__(16) double sa[2][kChunk][kPitch], sb[2][kChunk][kPitch];
    uint32_t bi, bj;
    triangle_tile(blockIdx.x, bi, bj);
    const uint32_t i0 = bi * kTile, j0 = bj * kTile;
    const uint32_t tx = threadIdx.x & 7u, ty = threadIdx.x >> 3, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t f4 = f / 4u * 4u;
    auto stage = [&](uint32_t k0, uint32_t buf) {
        if (k0 + lane < f4)
            for (uint32_t r = warp; r < kTile; r += 2u) {
                copy_async8(&sa[buf][lane][r], xc + (size_t)min(i0 + r, t - 1u) * f + k0 + lane);
                copy_async8(&sb[buf][lane][r], xc + (size_t)min(j0 + r, t - 1u) * f + k0 + lane);
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double acc[4][4][4] = {};
    stage(0u, 0u);
    for (uint32_t k0 = 0, buf = 0; k0 < f4; k0 += kChunk, buf ^= 1u) {
        stage(k0 + kChunk, buf ^ 1u);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const uint32_t kn = min(kChunk, f4 - k0);
        for (uint32_t c = 0; c < kn; c += 4u)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                double av[4], bv[4];
                load_spread4<kTile>(sa[buf][c + q], ty, av);
                load_spread4<kTile>(sb[buf][c + q], tx, bv);
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b < 4; ++b) acc[a][b][q] = __dadd_rn(acc[a][b][q], __dmul_rn(av[a], bv[b]));
            }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const uint32_t i = i0 + spread4<kTile>(ty, a), j = j0 + spread4<kTile>(tx, b);
            if (i >= t || j >= t || j < i) continue;
            double tail = 0.0;
            for (uint32_t c = f4; c < f; ++c)
                tail = __dadd_rn(tail, __dmul_rn(xc[(size_t)j * f + c], xc[(size_t)i * f + c]));
            const double *q = acc[a][b];
            double s = __dadd_rn(tail, __dadd_rn(__dadd_rn(__dadd_rn(q[0], q[1]), q[2]), q[3]));
            if (i == j) s = __dadd_rn(s, lambda);
            g[(size_t)i * t + j] = s;
        }
}

// Rows [p, p + kPanel) of U.  Warp 0 of every block factors the panel's
// diagonal block (lane i holds column i) while the other warps' threads
// divide and update one column to the right of it each, a row behind: they
// take row j - 1 from shared memory as warp 0 works on row j.  A latency
// chain of 32 square roots and divisions; in the place of two launches per
// row it serves 32 rows at once: 15.5 us a panel at 1000 rows, with the
// update 0.82 ms in all, against 7.8 ms.  The loop over j is rolled (the registers
// move up one place per j) so that a launch's code, which runs once, is
// short.  The factored diagonal block goes to dblk, because other blocks may
// still be reading the original; the trailing update puts it in place (the
// last panel, one block, does so itself).  A non-positive pivot (the matrix is
// not positive definite) raises bad[1], which only the update tests; the
// update passes it on to bad[0], which only the next panel tests.  So no
// launch tests a flag that it may be setting, and all threads find the same.
constexpr uint32_t kPanelCols = 96;  // columns right of the panel per block
__global__ void __launch_bounds__(32 + kPanelCols) chol_panel_kernel(double *g, uint32_t n, uint32_t p,
                                                                     double *__restrict__ dblk, unsigned int *bad) {
    __shared__ double sd[kPanel][2u * kPanel];  // sd[j][k] = U[p + j][p + k], k >= j; read up to k = j + 31
    if (bad[0]) return;  // an earlier panel failed
    const uint32_t nb = min(kPanel, n - p), lane = threadIdx.x & 31u;
    const bool diag = threadIdx.x < 32u;
    // columns to the right exist only past a full panel
    const uint32_t i = diag ? p + lane : p + kPanel + blockIdx.x * kPanelCols + threadIdx.x - 32u;
    const bool active = diag ? lane < nb : i < n;
    double c[kPanel];  // c[k]: row j + k of column i
#pragma unroll
    for (uint32_t j = 0; j < kPanel; ++j) {
        c[j] = active && j < nb && p + j <= i ? g[(size_t)(p + j) * n + i] : 1.0;
        if (diag) sd[j][kPanel + lane] = 0.0;
    }
    bool stop = false;
#pragma unroll 1
    for (uint32_t s = 0; s <= kPanel; ++s) {
        const uint32_t j = diag ? s : s - 1u;  // this warp's row
        if (j < kPanel) {
            double l;
            if (diag) {
                const double d = __shfl_sync(0xffffffffu, c[0], j);
                stop |= j < nb && d <= 0.0;  // the reference's test (readout.rs:155): a NaN pivot carries on
                const double ljj = __dsqrt_rn(d);
                l = lane == j ? ljj : __ddiv_rn(c[0], ljj);
                sd[j][lane] = l;
                __syncwarp();
            } else {
                l = __ddiv_rn(c[0], sd[j][j]);
            }
            if (!diag) {
                if (active) g[(size_t)(p + j) * n + i] = l;
            } else if (blockIdx.x == 0u && active && j < nb && lane >= j) {
                if (p + kPanel < n) dblk[j * kPanel + lane] = l;
                else g[(size_t)(p + j) * n + i] = l;
            }
#pragma unroll
            for (uint32_t k = 1; k < kPanel; ++k)  // row j + k loses U[j][j + k] U[j][i]
                c[k - 1] = __dsub_rn(c[k], __dmul_rn(l, sd[j][j + k]));
        }
        __syncthreads();
    }
    if (diag && stop && blockIdx.x == 0u && lane == 0u) bad[1] = 1u;
}

// The trailing upper triangle past a full panel: G[k][i] -= U[p + j][k]
// U[p + j][i] for j = 0..31 in order, from registers (one read and one write
// of the matrix per 32 rows).
__global__ void __launch_bounds__(256) chol_update_kernel(double *g, uint32_t n, uint32_t p,
                                                          const double *__restrict__ dblk, unsigned int *bad) {
    __shared__ __align__(16) double sk[kPanel][kUpdTile], si[kPanel][kUpdTile];
    if (bad[1]) {
        if (blockIdx.x == 0u && threadIdx.x == 0u) bad[0] = 1u;
        return;
    }
    if (blockIdx.x == 0u)  // the panel's diagonal block, which nothing here reads
        for (uint32_t e = threadIdx.x; e < kPanel * kPanel; e += 256u)
            if (e % kPanel >= e / kPanel) g[(size_t)(p + e / kPanel) * n + p + e % kPanel] = dblk[e];
    uint32_t bk, bi;
    triangle_tile(blockIdx.x, bk, bi);
    const uint32_t q0 = p + kPanel, k0 = q0 + bk * kUpdTile, i0 = q0 + bi * kUpdTile;
    for (uint32_t e = threadIdx.x; e < kPanel * kUpdTile; e += 256u) {
        const uint32_t j = e / kUpdTile, c = e % kUpdTile;
        sk[j][c] = g[(size_t)(p + j) * n + min(k0 + c, n - 1u)];
        si[j][c] = g[(size_t)(p + j) * n + min(i0 + c, n - 1u)];
    }
    const uint32_t tx = threadIdx.x & 15u, ty = threadIdx.x >> 4;
    double acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const uint32_t k = k0 + spread4<kUpdTile>(ty, a), i = i0 + spread4<kUpdTile>(tx, b);
            acc[a][b] = k < n && i < n ? g[(size_t)k * n + i] : 0.0;
        }
    __syncthreads();
#pragma unroll 4
    for (uint32_t j = 0; j < kPanel; ++j) {
        double kv[4], iv[4];
        load_spread4<kUpdTile>(sk[j], ty, kv);
        load_spread4<kUpdTile>(si[j], tx, iv);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a][b] = __dsub_rn(acc[a][b], __dmul_rn(iv[b], kv[a]));
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const uint32_t k = k0 + spread4<kUpdTile>(ty, a), i = i0 + spread4<kUpdTile>(tx, b);
            if (k < n && i < n && k <= i) g[(size_t)k * n + i] = acc[a][b];
        }
}

// w[c][q] = sum over rows r (in order) of a[c][r] xc[r][q]: a thread takes
// one column for four classes, the next 16 rows' loads in flight while this
// 16 are added, the dual weights broadcast from shared memory (74 us for 4
// classes at 1000 x 4320; a thread per column and class: 122 us).
__global__ void __launch_bounds__(32) weights_kernel(const double *__restrict__ xc, const double *__restrict__ a,
                                                     uint32_t t, uint32_t f, uint32_t k, double *__restrict__ w) {
    constexpr uint32_t R = 16;
    __shared__ __align__(16) double sa[R][4];
    const uint32_t q = blockIdx.x * 32u + threadIdx.x, c0 = blockIdx.y * 4u, qq = min(q, f - 1u);
    double v[R], nx[R], av[2], s[4] = {};
    // two of the 16 x 4 dual weights per thread: row lane / 2, classes 2 (lane % 2) and the next
    const uint32_t ar = threadIdx.x >> 1, ac = (threadIdx.x & 1u) * 2u;
    auto fetch = [&](uint32_t r0, double (&d)[R]) {
#pragma unroll
        for (uint32_t e = 0; e < R; ++e) d[e] = r0 + e < t ? xc[(size_t)(r0 + e) * f + qq] : 0.0;
#pragma unroll
        for (uint32_t e = 0; e < 2u; ++e)
            av[e] = r0 + ar < t ? a[(size_t)min(c0 + ac + e, k - 1u) * t + r0 + ar] : 0.0;
    };
    fetch(0u, v);
    for (uint32_t r0 = 0; r0 < t; r0 += R) {
        sa[ar][ac] = av[0];
        sa[ar][ac + 1u] = av[1];
        __syncwarp();
        fetch(r0 + R, nx);
#pragma unroll
        for (uint32_t e = 0; e < R; ++e) {
            double a4[4];
            load4(sa[e], a4);
            if (r0 + e < t)
#pragma unroll
                for (int c = 0; c < 4; ++c) s[c] = __dadd_rn(s[c], __dmul_rn(a4[c], v[e]));
            v[e] = nx[e];
        }
        __syncwarp();
    }
#pragma unroll
    for (uint32_t c = 0; c < 4u; ++c)
        if (q < f && c0 + c < k) w[(size_t)(c0 + c) * f + q] = s[c];
}

// The columns [x 1 y] as f64, rows of `pitch` doubles (even: 16-byte aligned;
// zeros past y).
__global__ void augment_kernel(const float *__restrict__ x, const float *__restrict__ y, uint32_t t, uint32_t f,
                               uint32_t pitch, double *__restrict__ xa) {
    const uint32_t r = blockIdx.y;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < pitch; c += gridDim.x * blockDim.x)
        xa[(size_t)r * pitch + c] = c < f ? (double)x[(size_t)r * f + c] : c == f ? 1.0 : c == f + 1u ? (double)y[r] : 0.0;
}

// Upper-triangle tiles of the normal matrix of the columns [x 1 y], each
// entry summed over the rows in order: a (F + 1 wide) and, from the last
// column, the right-hand side.  4 x 4 entries per thread and cp.async as in
// gram_kernel; the conversion to f64 is done once beforehand (on the way to
// shared memory it took as long as the sums).  `more`: the sums go on from
// those of earlier rows.  166 us at 1200 x 1080 with the
// conversion, against 249 + 315 us with 2 x 2 entries per thread and a thread
// per column for the bias and right-hand side.
__global__ void __launch_bounds__(64) normal_kernel(const double *__restrict__ xa, uint32_t t, uint32_t f,
                                                    uint32_t pitch, bool more, double *__restrict__ a,
                                                    double *__restrict__ rhs) {
    __shared__ __align__(16) double si[2][kChunk][kTile], sj[2][kChunk][kTile];
    uint32_t bi, bj;
    triangle_tile(blockIdx.x, bi, bj);
    const uint32_t i0 = bi * kTile, j0 = bj * kTile, nf = f + 1u;
    const uint32_t tx = threadIdx.x & 7u, ty = threadIdx.x >> 3;
    auto stage = [&](uint32_t r0, uint32_t buf) {
        for (uint32_t e = threadIdx.x; e < kChunk * kTile / 2u; e += 64u) {
            const uint32_t r = e / (kTile / 2u), c = e % (kTile / 2u) * 2u;
            if (r0 + r >= t) break;  // e ascends with r
            const double *row = xa + (size_t)(r0 + r) * pitch;
            copy_async16(&si[buf][r][c], row + min(i0 + c, pitch - 2u));
            copy_async16(&sj[buf][r][c], row + min(j0 + c, pitch - 2u));
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto entry = [&](int p, int q) -> double * {  // where the sum of this thread's entry (p, q) is kept
        const uint32_t i = i0 + spread4<kTile>(ty, p), j = j0 + spread4<kTile>(tx, q);
        if (i > f || i > j || j > nf) return nullptr;
        return j < nf ? a + (size_t)i * nf + j : rhs + i;
    };
    double acc[4][4] = {};
    if (more)  // the rows before these, summed by an earlier launch
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (const double *e = entry(p, q)) acc[p][q] = *e;
    stage(0u, 0u);
    for (uint32_t r0 = 0, buf = 0; r0 < t; r0 += kChunk, buf ^= 1u) {
        stage(r0 + kChunk, buf ^ 1u);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const uint32_t rn = min(kChunk, t - r0);
#pragma unroll 4
        for (uint32_t r = 0; r < rn; ++r) {
            double iv[4], jv[4];
            load_spread4<kTile>(si[buf][r], ty, iv);
            load_spread4<kTile>(sj[buf][r], tx, jv);
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[p][q] = __dadd_rn(acc[p][q], __dmul_rn(iv[p], jv[q]));
        }
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (double *e = entry(p, q)) *e = acc[p][q];
}

// a[i][i] += add for every i; with `unbias`, a[f][f] then loses lambda again.
__global__ void diag_kernel(double *a, uint32_t n, double add, bool unbias, double lambda) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v = __dadd_rn(a[(size_t)i * n + i], add);
    if (unbias && i + 1u == n) v = __dsub_rn(v, lambda);
    a[(size_t)i * n + i] = v;
}

// trial r's features: window counts [windows][n] of one net (u16 -> f32)
__global__ void gather_counts_kernel(const uint16_t *const *__restrict__ win, uint32_t n, uint32_t n_pad,
                                     uint32_t windows, float *__restrict__ x) {
    const uint32_t r = blockIdx.y;
    const uint32_t f = windows * n;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < f; q += gridDim.x * blockDim.x) {
        const uint32_t wdx = q / n, i = q - wdx * n;
        x[(size_t)r * f + q] = (float)win[r][(size_t)wdx * n_pad + i];
    }
}

// A fit's device memory; `device`: of the workspaces kept for that device, or
// (kEnginePool) of the default pool, as an engine's other arrays.
constexpr int kEnginePool = -1;
struct DevBuf {
    std::vector<void *> ps;
    cudaStream_t st;
    int device;
    DevBuf(cudaStream_t s, int dev) : st(s), device(dev) {}
    ~DevBuf() {
        for (void *p : ps) cudaFreeAsync(p, st);
        cudaStreamSynchronize(st);
    }
    template <class T>
    ne2b_status get(T **p, size_t count) {
        void *q = nullptr;
        const size_t bytes = sizeof(T) * (count ? count : 1);
        const cudaError_t e = device == kEnginePool ? device_alloc(&q, bytes, st) : workspace_alloc(&q, bytes, device, st);
        if (e != cudaSuccess) return cuda_error(e, "cudaMallocAsync (readout)");
        ps.push_back(q);
        *p = (T *)q;
        return NE2B_OK;
    }
};

// G = U^T U in place of the upper triangle; true when G is positive definite.
// dblk: scratch, 32 x 32; bad: two flags.
ne2b_status cholesky(double *g, uint32_t n, double *dblk, unsigned int *bad, cudaStream_t st, bool *pd) {
    NE2B_CUDA(cudaMemsetAsync(bad, 0, 2 * sizeof(unsigned int), st));
    for (uint32_t p = 0; p < n; p += kPanel) {
        const uint32_t right = n - std::min(n, p + kPanel);  // columns right of the panel
        chol_panel_kernel<<<std::max(1u, (right + kPanelCols - 1u) / kPanelCols), 32 + kPanelCols, 0, st>>>(g, n, p, dblk, bad);
        const uint32_t nt = (right + kUpdTile - 1u) / kUpdTile;
        if (nt) chol_update_kernel<<<nt * (nt + 1u) / 2u, 256, 0, st>>>(g, n, p, dblk, bad);
    }
    NE2B_CUDA(cudaGetLastError());
    unsigned int bad_h = 0;
    NE2B_CUDA(cudaMemcpyAsync(&bad_h, bad + 1, sizeof bad_h, cudaMemcpyDeviceToHost, st));
    NE2B_CUDA(cudaStreamSynchronize(st));
    *pd = bad_h == 0;
    return NE2B_OK;
}

// fit_ridge on a device design x[T x F] and host targets y[T].
ne2b_status fit_binary_on_device(const float *x, uint32_t t, uint32_t f, const float *y_host, float lambda,
                                 int device, cudaStream_t st, double *w_out) {
    const uint32_t nf = f + 1u;
    DevBuf buf(st, device);
    double *a = nullptr, *a0 = nullptr, *b = nullptr;
    float *y = nullptr;
    unsigned int *bad = nullptr;
    NE2B_TRY(buf.get(&a, (size_t)nf * nf));
    NE2B_TRY(buf.get(&a0, (size_t)nf * nf));
    NE2B_TRY(buf.get(&b, nf));
    NE2B_TRY(buf.get(&y, t));
    NE2B_TRY(buf.get(&bad, 2));
    double *dblk = nullptr;
    NE2B_TRY(buf.get(&dblk, (size_t)kPanel * kPanel));
    NE2B_CUDA(cudaMemcpyAsync(y, y_host, sizeof(float) * t, cudaMemcpyHostToDevice, st));
    const uint32_t nt = (nf + 1u + kTile - 1u) / kTile;  // columns x, 1 and y
    const uint32_t pitch = (nf + 2u) / 2u * 2u;
    // the f64 copy of at most 2 GB of rows at a time, summed on
    const uint32_t rows = std::min(t, (uint32_t)std::max<uint64_t>(64u, (2ull << 30) / (8ull * pitch)));
    double *xa = nullptr;
    NE2B_TRY(buf.get(&xa, (size_t)rows * pitch));
    for (uint32_t r0 = 0; r0 < t; r0 += rows) {
        const uint32_t nr = std::min(rows, t - r0);
        for (uint32_t g0 = 0; g0 < nr; g0 += 65535u)  // rows along grid y
            augment_kernel<<<dim3(std::min(64u, (pitch + 255u) / 256u), std::min(65535u, nr - g0)), 256, 0, st>>>(
                x + (size_t)(r0 + g0) * f, y + r0 + g0, nr - g0, f, pitch, xa + (size_t)g0 * pitch);
        normal_kernel<<<nt * (nt + 1) / 2, 64, 0, st>>>(xa, nr, f, pitch, r0 > 0u, a, b);
    }
    const double lam = (double)lambda;
    diag_kernel<<<(nf + 255) / 256, 256, 0, st>>>(a, nf, lam, true, lam);
    NE2B_CUDA(cudaMemcpyAsync(a0, a, sizeof(double) * nf * nf, cudaMemcpyDeviceToDevice, st));
    bool pd = false;
    NE2B_TRY(cholesky(a, nf, dblk, bad, st, &pd));
    if (!pd) {  // readout.rs:131-139: more regularisation, once
        NE2B_CUDA(cudaMemcpyAsync(a, a0, sizeof(double) * nf * nf, cudaMemcpyDeviceToDevice, st));
        diag_kernel<<<(nf + 255) / 256, 256, 0, st>>>(a, nf, 1e-3 + lam, false, 0.0);
        NE2B_TRY(cholesky(a, nf, dblk, bad, st, &pd));
    }
    if (!pd) {
        for (uint32_t i = 0; i < nf; ++i) w_out[i] = 0.0;
        return NE2B_OK;
    }
    HostWorkspace host;
    double *u = (double *)host.get(sizeof(double) * ((size_t)nf * nf + nf));
    if (!u) return set_error(NE2B_ENOMEM, "host allocation failed");
    double *bh = u + (size_t)nf * nf;
    NE2B_CUDA(cudaMemcpyAsync(u, a, sizeof(double) * nf * nf, cudaMemcpyDeviceToHost, st));
    NE2B_CUDA(cudaMemcpyAsync(bh, b, sizeof(double) * nf, cudaMemcpyDeviceToHost, st));
    NE2B_CUDA(cudaStreamSynchronize(st));
    host_solve1(u, bh, nf, w_out);
    return NE2B_OK;
}

ne2b_status check_labels(const uint32_t *labels, uint32_t t, uint32_t f, uint32_t k) {
    if (t < 2 || k < 2 || f == 0)
        return set_error(NE2B_EINVAL, "fit_ridge_multi: need T >= 2, K >= 2, F >= 1 (T=%u F=%u K=%u)", t, f, k);
    if (t > 32768) return set_error(NE2B_UNSUPPORTED, "fit_ridge_multi: at most 32768 rows (T=%u)", t);
    for (uint32_t r = 0; r < t; ++r)
        if (labels[r] >= k) return set_error(NE2B_EINVAL, "fit_ridge_multi: label %u outside 0..%u", labels[r], k);
    return NE2B_OK;
}

// The fit on a device design x[T x F] (f32) on stream `st`.
ne2b_status fit_on_device(const float *x, uint32_t t, uint32_t f, const uint32_t *labels, uint32_t k, double lambda,
                          int device, cudaStream_t st, double *w_out) {
    DevBuf buf(st, device);
    double *mu = nullptr, *xc = nullptr, *g = nullptr, *a = nullptr, *w = nullptr;
    unsigned int *bad = nullptr;
    NE2B_TRY(buf.get(&mu, f));
    NE2B_TRY(buf.get(&xc, (size_t)t * f));
    NE2B_TRY(buf.get(&g, (size_t)t * t));
    NE2B_TRY(buf.get(&a, (size_t)t * k));
    NE2B_TRY(buf.get(&w, (size_t)f * k));
    NE2B_TRY(buf.get(&bad, 2));
    double *dblk = nullptr;
    NE2B_TRY(buf.get(&dblk, (size_t)kPanel * kPanel));
    col_mean_kernel<<<(f + 31) / 32, 128, 0, st>>>(x, t, f, mu);
    const uint64_t n = (uint64_t)t * f;
    center_kernel<<<(unsigned)std::min<uint64_t>((n + 255) / 256, 148ull * 64), 256, 0, st>>>(x, n, f, mu, xc);
    const uint32_t nt = (t + kTile - 1) / kTile;
    gram_kernel<<<nt * (nt + 1) / 2, 64, 0, st>>>(xc, t, f, lambda, g);
    bool pd = false;
    NE2B_TRY(cholesky(g, t, dblk, bad, st, &pd));
    // the triangular solves on the host, in the reference's order, four
    // classes side by side
    std::vector<double> mu_h(f), ybar(k, 0.0), ah((size_t)t * k, 0.0);
    NE2B_CUDA(cudaMemcpyAsync(mu_h.data(), mu, sizeof(double) * f, cudaMemcpyDeviceToHost, st));
    for (uint32_t r = 0; r < t; ++r) ybar[labels[r]] += 1.0 / (double)t;
    if (pd) {
        HostWorkspace host;
        double *u = (double *)host.get(sizeof(double) * (size_t)t * t);
        if (!u) return set_error(NE2B_ENOMEM, "host allocation failed");
        NE2B_CUDA(cudaMemcpyAsync(u, g, sizeof(double) * (size_t)t * t, cudaMemcpyDeviceToHost, st));
        NE2B_CUDA(cudaStreamSynchronize(st));
        constexpr uint32_t kSide = 4;
        std::vector<double> yc((size_t)t * kSide), ac((size_t)t * kSide);
        for (uint32_t c0 = 0; c0 < k; c0 += kSide) {
            for (uint32_t i = 0; i < t; ++i)
                for (uint32_t c = 0; c < kSide; ++c)
                    yc[(size_t)i * kSide + c] =
                        c0 + c < k ? (labels[i] == c0 + c ? 1.0 : 0.0) - ybar[c0 + c] : 0.0;
            host_solve4(u, yc.data(), t, ac.data());
            for (uint32_t c = 0; c < kSide && c0 + c < k; ++c)
                for (uint32_t i = 0; i < t; ++i) ah[(size_t)(c0 + c) * t + i] = ac[(size_t)i * kSide + c];
        }
    }
    NE2B_CUDA(cudaMemcpyAsync(a, ah.data(), sizeof(double) * ah.size(), cudaMemcpyHostToDevice, st));
    weights_kernel<<<dim3((f + 31) / 32, (k + 3) / 4), 32, 0, st>>>(xc, a, t, f, k, w);
    NE2B_CUDA(cudaGetLastError());
    std::vector<double> wh((size_t)f * k);
    NE2B_CUDA(cudaMemcpyAsync(wh.data(), w, sizeof(double) * wh.size(), cudaMemcpyDeviceToHost, st));
    NE2B_CUDA(cudaStreamSynchronize(st));
    for (uint32_t c = 0; c < k; ++c) {
        double *wc = w_out + (size_t)c * (f + 1);
        memcpy(wc, wh.data() + (size_t)c * f, sizeof(double) * f);
        double dot = 0.0;
        for (uint32_t q = 0; q < f; ++q) dot += wc[q] * mu_h[q];
        wc[f] = ybar[c] - dot;
    }
    return NE2B_OK;
}

}  // namespace
}  // namespace ne2b

using ne2b::cuda_error;
using ne2b::set_error;

extern "C" {

ne2b_status ne2b_fit_ridge_multi(const float *x, uint32_t t, uint32_t f, const uint32_t *labels, uint32_t k,
                                 double lambda, int device, double *w) {
    if (!x || !labels || !w) return set_error(NE2B_EINVAL, "ne2b_fit_ridge_multi: null argument");
    const ne2b_status cs = ne2b::check_labels(labels, t, f, k);
    if (cs != NE2B_OK) return cs;
    try {
        cudaError_t e = cudaSetDevice(device);
        if (e != cudaSuccess) return ne2b::cuda_error(e, "cudaSetDevice");
        cudaPointerAttributes attr{};
        const bool on_device = cudaPointerGetAttributes(&attr, x) == cudaSuccess && attr.type == cudaMemoryTypeDevice;
        cudaGetLastError();  // a host pointer may leave a benign error behind
        cudaStream_t st = nullptr;
        e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
        if (e != cudaSuccess) return ne2b::cuda_error(e, "cudaStreamCreate");
        ne2b_status r = NE2B_OK;
        {
            ne2b::DevBuf buf(st, device);
            const float *xd = x;
            if (!on_device) {
                float *p = nullptr;
                r = buf.get(&p, (size_t)t * f);
                if (r == NE2B_OK)
                    r = ne2b::cuda_error(cudaMemcpyAsync(p, x, sizeof(float) * (size_t)t * f, cudaMemcpyHostToDevice, st),
                                         "design upload");
                xd = p;
            }
            if (r == NE2B_OK) r = ne2b::fit_on_device(xd, t, f, labels, k, lambda, device, st, w);
        }
        cudaStreamDestroy(st);
        return r;
    } catch (const std::bad_alloc &) {
        return set_error(NE2B_ENOMEM, "host allocation failed");
    }
}

ne2b_status ne2b_release_workspaces(void) {
    try {
        ne2b::release_workspaces();
        return NE2B_OK;
    } catch (const std::exception &e) {
        return set_error(NE2B_ENOMEM, "ne2b_release_workspaces: %s", e.what());
    }
}

}  // extern "C"

// A batch's window counts as a [t x windows*n] design on its stream.
static ne2b_status gather_batch(ne2b_batch *b, const uint32_t *nets, uint32_t t, uint32_t windows,
                                ne2b::DevBuf &buf, float **x, uint32_t *f_out) {
    if (t == 0 || windows == 0) return set_error(NE2B_EINVAL, "batch readout: no trials or no windows");
    std::vector<const uint16_t *> win(t);
    uint32_t n = 0, n_pad = 0;
    for (uint32_t r = 0; r < t; ++r) {
        if (nets[r] >= b->slots.size()) return set_error(NE2B_EINVAL, "net %u out of range", nets[r]);
        ne2b::NetHost *h = b->eng.net(b->slots[nets[r]]);
        if (!h) return set_error(NE2B_EINVAL, "net %u has no network", nets[r]);
        if (r == 0) {
            n = h->n;
            n_pad = h->n_pad;
        } else if (h->n != n) {
            return set_error(NE2B_EINVAL, "the trials' nets differ in size (%u and %u neurons)", n, h->n);
        }
        const uint64_t done = h->dev.win_steps ? h->t / h->dev.win_steps : 0;
        if (!h->dev.win_out || done < windows || windows > h->dev.max_windows)
            return set_error(NE2B_EINVAL, "net %u has %llu of the %u windows asked for", nets[r],
                             (unsigned long long)done, windows);
        win[r] = h->dev.win_out;
    }
    const uint64_t f64 = (uint64_t)windows * n;
    if (f64 == 0 || f64 > 0xffffffffull) return set_error(NE2B_UNSUPPORTED, "%llu features", (unsigned long long)f64);
    const uint32_t f = (uint32_t)f64;
    cudaStream_t st = b->eng.stream();  // after the batch's queued steps
    const uint16_t **wd = nullptr;
    NE2B_TRY(buf.get(&wd, t));
    NE2B_TRY(buf.get(x, (size_t)t * f));
    NE2B_CUDA(cudaMemcpyAsync(wd, win.data(), sizeof(void *) * t, cudaMemcpyHostToDevice, st));
    ne2b::gather_counts_kernel<<<dim3((f + 255) / 256 < 1024 ? (f + 255) / 256 : 1024, t), 256, 0, st>>>(
        wd, n, n_pad, windows, *x);
    NE2B_CUDA(cudaGetLastError());
    *f_out = f;
    return NE2B_OK;
}

extern "C" {

ne2b_status ne2b_batch_fit_ridge_multi(ne2b_batch *b, const uint32_t *nets, uint32_t t, uint32_t windows,
                                       const uint32_t *labels, uint32_t k, double lambda, uint32_t *n_features,
                                       double *w) {
    if (!b || !nets || !labels || !w) return set_error(NE2B_EINVAL, "ne2b_batch_fit_ridge_multi: null argument");
    try {
        ne2b::DevBuf buf(b->eng.stream(), ne2b::kEnginePool);
        float *x = nullptr;
        uint32_t f = 0;
        NE2B_TRY(gather_batch(b, nets, t, windows, buf, &x, &f));
        const ne2b_status cs = ne2b::check_labels(labels, t, f, k);
        if (cs != NE2B_OK) return cs;
        if (n_features) *n_features = f;
        return ne2b::fit_on_device(x, t, f, labels, k, lambda, ne2b::kEnginePool, b->eng.stream(), w);
    } catch (const std::bad_alloc &) {
        return set_error(NE2B_ENOMEM, "host allocation failed");
    }
}

ne2b_status ne2b_fit_ridge(const float *x, uint32_t t, uint32_t f, const float *y, float lambda, int device,
                           double *w) {
    if (!x || !y || !w) return set_error(NE2B_EINVAL, "ne2b_fit_ridge: null argument");
    if (t == 0 || f == 0) return set_error(NE2B_EINVAL, "fit_ridge: need T >= 1, F >= 1 (T=%u F=%u)", t, f);
    if (f >= 32768) return set_error(NE2B_UNSUPPORTED, "fit_ridge: at most 32767 features (F=%u)", f);
    try {
        cudaError_t e = cudaSetDevice(device);
        if (e != cudaSuccess) return ne2b::cuda_error(e, "cudaSetDevice");
        cudaPointerAttributes attr{};
        const bool on_device = cudaPointerGetAttributes(&attr, x) == cudaSuccess && attr.type == cudaMemoryTypeDevice;
        cudaGetLastError();
        cudaStream_t st = nullptr;
        e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
        if (e != cudaSuccess) return ne2b::cuda_error(e, "cudaStreamCreate");
        ne2b_status r = NE2B_OK;
        {
            ne2b::DevBuf buf(st, device);
            const float *xd = x;
            if (!on_device) {
                float *p = nullptr;
                r = buf.get(&p, (size_t)t * f);
                if (r == NE2B_OK)
                    r = ne2b::cuda_error(cudaMemcpyAsync(p, x, sizeof(float) * (size_t)t * f, cudaMemcpyHostToDevice, st),
                                         "design upload");
                xd = p;
            }
            if (r == NE2B_OK) r = ne2b::fit_binary_on_device(xd, t, f, y, lambda, device, st, w);
        }
        cudaStreamDestroy(st);
        return r;
    } catch (const std::bad_alloc &) {
        return set_error(NE2B_ENOMEM, "host allocation failed");
    }
}

ne2b_status ne2b_batch_fit_ridge(ne2b_batch *b, const uint32_t *nets, uint32_t t, uint32_t windows, const float *y,
                                 float lambda, uint32_t *n_features, double *w) {
    if (!b || !nets || !y || !w) return set_error(NE2B_EINVAL, "ne2b_batch_fit_ridge: null argument");
    try {
        ne2b::DevBuf buf(b->eng.stream(), ne2b::kEnginePool);
        float *x = nullptr;
        uint32_t f = 0;
        NE2B_TRY(gather_batch(b, nets, t, windows, buf, &x, &f));
        if (f >= 32768) return set_error(NE2B_UNSUPPORTED, "fit_ridge: at most 32767 features (F=%u)", f);
        if (n_features) *n_features = f;
        return ne2b::fit_binary_on_device(x, t, f, y, lambda, ne2b::kEnginePool, b->eng.stream(), w);
    } catch (const std::bad_alloc &) {
        return set_error(NE2B_ENOMEM, "host allocation failed");
    }
}

}  // extern "C"
