// ne2b_solve.h — the triangular solves of the readout fits, on the host
// (ne2b_solve.cpp).
#pragma once
#include <stdint.h>

namespace ne2b {

// U^T z = b, U w = z with U the upper triangle of u [n][n], for one
// right-hand side b[n] -> w[n], or four side by side, b[n][4] -> w[n][4].
// Each value's sums run in the reference's order (sim/src/readout.rs:170-186).
void host_solve1(const double *u, const double *b, uint32_t n, double *w);
void host_solve4(const double *u, const double *b, uint32_t n, double *w);

}  // namespace ne2b
