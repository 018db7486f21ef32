// The Bloch-space psi layout on the device (qspace.cu builds the tables).
#pragma once

#include "common.cuh"

namespace tdscha {

// alpha1 blocks from psi (Wigner change of variables per pair element).
// pcoef layout per pair element: [0] -(w1-w2)^2 vm, [1] -(w1+w2)^2 vm,
// [2] w2X sqrt(-chi-/2), [3] w2X sqrt(chi+/2), [4] sqrt(-chi-/2), [5] -sqrt(chi+/2)
__device__ __forceinline__ long q_store(int p, int i, int j, int nb, int full, const long *off) {
    if (full) return off[p] + (long)i * nb + j;
    // upper triangle rows from the diagonal, i <= j
    return off[p] + (long)i * nb - (long)i * (i - 1) / 2 + (j - i);
}

// Element (i, j) of pair p's alpha1
__device__ __forceinline__ double2 q_alpha1(const double2 *__restrict__ psi,
                                            const int *__restrict__ pair_q,
                                            const long *__restrict__ off_a,
                                            const long *__restrict__ off_b,
                                            const double *__restrict__ pcoef, int p, int i, int j,
                                            int nb) {
    const int full = pair_q[2 * p] < pair_q[2 * p + 1];
    // the lower triangle of a Hermitian block is the conjugate of the upper one
    const bool lower = !full && i > j;
    const int r = lower ? j : i, s = lower ? i : j;
    double2 a = psi[q_store(p, r, s, nb, full, off_a)], b = psi[q_store(p, r, s, nb, full, off_b)];
    if (lower) {
        a.y = -a.y;
        b.y = -b.y;
    }
    const double *c = pcoef + (((long)p * nb + i) * nb + j) * 6;
    return make_double2(c[2] * a.x - c[3] * b.x, c[2] * a.y - c[3] * b.y);
}

}  // namespace tdscha
