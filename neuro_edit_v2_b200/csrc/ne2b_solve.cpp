// ne2b_solve.cpp — see ne2b_solve.h.  Compiled without contraction, so every
// product and difference is rounded on its own, as the reference's.
//
// The first solve runs over U's rows: z_q leaves every later sum at once,
// which still meets q = 0, 1, ... in order, so it runs in vectors.  In the
// second, value i subtracts the terms of i + 1, i + 2, ... ascending, and
// value i + 1 is the one found last: one chain of n^2 / 2 dependent
// subtractions, four cycles each, which four right-hand sides share.
#include "ne2b_solve.h"

#include <string.h>

#include <vector>

namespace ne2b {
namespace {

typedef double v4 __attribute__((vector_size(32)));

v4 load(const double *p) {
    v4 v;
    memcpy(&v, p, sizeof v);
    return v;
}
void store(double *p, const v4 &v) { memcpy(p, &v, sizeof v); }

}  // namespace

void host_solve1(const double *u, const double *b, uint32_t n, double *w) {
    std::vector<double> z(b, b + n);
    for (uint32_t q = 0; q < n; ++q) {
        const double *row = u + (size_t)q * n;
        const double zq = z[q] /= row[q];
        const v4 zv = {zq, zq, zq, zq};
        uint32_t i = q + 1;
        for (; i + 4 <= n; i += 4) store(&z[i], load(&z[i]) - load(row + i) * zv);
        for (; i < n; ++i) z[i] -= row[i] * zq;
    }
    for (uint32_t i = n; i-- > 0;) {
        const double *row = u + (size_t)i * n;
        double s = z[i];
        for (uint32_t q = i + 1; q < n; ++q) s -= row[q] * w[q];
        w[i] = s / row[i];
    }
}

void host_solve4(const double *u, const double *b, uint32_t n, double *w) {
    std::vector<double> z(b, b + (size_t)n * 4);
    for (uint32_t q = 0; q < n; ++q) {
        const double *row = u + (size_t)q * n;
        double *zp = z.data() + (size_t)q * 4;
        const v4 zq = load(zp) / row[q];
        store(zp, zq);
        zp += 4;
        for (uint32_t i = q + 1; i < n; ++i, zp += 4) store(zp, load(zp) - row[i] * zq);
    }
    for (uint32_t i = n; i-- > 0;) {
        const double *row = u + (size_t)i * n;
        v4 s = load(z.data() + (size_t)i * 4);
        const double *wq = w + (size_t)(i + 1) * 4;
        for (uint32_t q = i + 1; q < n; ++q, wq += 4) s = s - row[q] * load(wq);
        store(w + (size_t)i * 4, s / row[i]);
    }
}

}  // namespace ne2b
