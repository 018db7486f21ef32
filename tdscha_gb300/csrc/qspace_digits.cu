// Bloch-space averages in float64 by exact digit products on the tensor cores
// (perturb_digits.cu explains the arithmetic, qspace.cu the averages).
//
// A q-point's n_b complex bands are 2 n_b <= 64 real columns (Re, Im, Re, Im ...),
// one tile of the digit contraction.  Two of them carry the work that the float64
// pipe did at 0.7 of its 1.25 TFLOP/s:
//
//   u_q = A_q x_partner(q)     rows tile x real form of A_q (2 n_b x 2 n_b; several
//                              q-points side by side in one 64 x 64 tile where that
//                              leaves enough tiles); the epilogue takes
//                              sum conj(x) u and sum conj(u) g
//   d2v_p = sum_r A1 conj(f2) + A2 conj(u2), with A1 = -w_cross u1 and
//           A2 = -(w_cross f1 + w_diag u1): the real products of the 4 n_b columns
//           [A1 | A2] of pair p with those [f2 | u2] of its second q-point (one or
//           two tiles of 64), combined to complex at the end.  Half of them, A1 with
//           u2 and A2 with f2, are not needed and cost nothing: they fill a tile
//           that would be empty.
//
// Scales as in perturb_digits.cu: a column's is the largest weighted exponent of its
// elements; a configuration has one for y and one for u of each q-point, the exponent above its largest
// element there.  The rows of [f2 | u2] are without it and those of A1 and A2 carry it.
//
// Measured (averages, one call): 4x4x4 grid, 12 bands, N=10000 2479 -> 526 us
// (row dots 224, W 134, d2v 143 in a launch list).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "digits.cuh"
#include "qspace.cuh"

namespace tdscha {

// x, g = f_psi y, u = f_Y x and y as real columns, [q][row tile][2 nb][128 rows]
struct QDigitStore {
    int nr = 0, nbq = 1;          // real columns of a q-point, tiles of [y | u]
    int G = 1, ngrp = 1;          // q-points of a tile of xa, such tiles
    long nrt = 0, Rp = 0, nkb = 0;
    int flush = kFlushMin, nsm = 1;
    void *slab = nullptr, *pslab = nullptr;
    double *x = nullptr, *g = nullptr, *u = nullptr, *y = nullptr, *qp = nullptr;
    __half *xa = nullptr, *xb = nullptr, *yb = nullptr;
    int *ec = nullptr, *er = nullptr, *ecb = nullptr, *et = nullptr, *cofs = nullptr,
        *wtop = nullptr;
    int *failed = nullptr;        // whether a bounded wait gave up in this call
    int *err = nullptr;           // its code, until it has been reported (pinned host memory)
    int2 *erb = nullptr;          // a row's scales in y and in u, [q][Rp]
    int *rowfar = nullptr, anyfar = 0;
    double *rowc = nullptr;       // 8 doubles a row
    // per perturbation
    uint32_t abytes = 0;          // of a digit of a W block: rows up to a multiple of eight
    int n_pairs = 0, per = 1, nfc = 1, kbps = 1, ns = 1;
    __half *wa = nullptr;
    int *ew = nullptr, *bmap = nullptr;
    double *gpart = nullptr, *fpart = nullptr;
    long long budget = kDefaultBudget;
};

// ------------------------------------------------- once per ensemble
// 128 rows of one q-point from the image rows (R x L complex) to columns
__global__ void __launch_bounds__(256) k_qd_cols(const double *__restrict__ Xr,
                                                 const double *__restrict__ Yr,
                                                 const double *__restrict__ fY,
                                                 const double *__restrict__ fpsi, int L, int nb,
                                                 long R, double *__restrict__ x,
                                                 double *__restrict__ g, double *__restrict__ u,
                                                 double *__restrict__ y) {
    __shared__ double sx[32][65], sy[32][65];
    const long rt = blockIdx.x;
    const int q = blockIdx.y, nr = 2 * nb;
    const long base = ((long)q * gridDim.x + rt) * nr * 128;
    for (int part = 0; part < 4; ++part) {
        for (int t = threadIdx.x; t < 32 * nr; t += blockDim.x) {
            const int k = t / nr, c = t % nr;
            const long r = rt * 128 + part * 32 + k, o = (r * L + q * nb) * 2 + c;
            sx[k][c] = r < R ? Xr[o] : 0.0;
            sy[k][c] = r < R ? Yr[o] : 0.0;
        }
        __syncthreads();
        for (int t = threadIdx.x; t < 32 * nr; t += blockDim.x) {
            const int k = t & 31, c = t >> 5;
            const long o = base + c * 128L + part * 32 + k;
            const double xv = sx[k][c], yv = sy[k][c];
            const int m = q * nb + (c >> 1);
            x[o] = xv;
            y[o] = yv;
            g[o] = fpsi[m] * yv;
            u[o] = fY[m] * xv;
        }
        __syncthreads();
    }
}

// Scales of the columns, their largest weighted exponents (dg_weight_exp): of x in ec, of y
// and u as the tiles [y | u] have them in ecb.  A column without an element (the imaginary
// parts at Gamma, masked modes) has kZeroExp, which leaves it out of the rows' scales of A_q
// and of W's bounds.
__global__ void __launch_bounds__(128) k_qd_colscale(const double *__restrict__ x,
                                                     const double *__restrict__ y,
                                                     const double *__restrict__ u,
                                                     const double *__restrict__ rho, int S, int rtop,
                                                     long R, long nrt, int nr, int nbq, int G,
                                                     int *__restrict__ ec, int *__restrict__ ecb) {
    __shared__ int sh[4][3];
    const int c = blockIdx.x, q = blockIdx.y;
    int e[3] = {INT_MIN, INT_MIN, INT_MIN};
    for (long rt = 0; rt < nrt; ++rt) {
        const long o = (((long)q * nrt + rt) * nr + c) * 128 + threadIdx.x, r = rt * 128 + threadIdx.x;
        if (r >= R) break;
        const int less = dg_weight_exp(rho[(unsigned)r / (unsigned)S], rtop);
        const double v[3] = {x[o], y[o], u[o]};
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (v[k] != 0) e[k] = max(e[k], exp_above(v[k]) + less);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        e[k] = __reduce_max_sync(0xffffffffu, e[k]);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5][k] = e[k];
    }
    __syncthreads();
    if (threadIdx.x >= 3) return;
    const int k = threadIdx.x;
    int top = max(max(sh[0][k], sh[1][k]), max(sh[2][k], sh[3][k]));
    if (top < INT_MIN / 4) top = kZeroExp;
    if (k == 0) ec[q / G * 64 + q % G * nr + c] = top;
    else ecb[(long)q * nbq * kGN + (k == 1 ? c : nbq == 1 ? nr + c : kGN + c)] = top;
}

// erb[q][r]: exponents above |y| 2^-ecb and |u| 2^-ecb of a row; rowfar[r]: one is above 0
__global__ void __launch_bounds__(128) k_qd_rowscale(const double *__restrict__ y,
                                                     const double *__restrict__ u,
                                                     const int *__restrict__ ecb, int nr, int nbq,
                                                     int2 *__restrict__ erb, int *__restrict__ rowfar,
                                                     int *__restrict__ anyfar) {
    const int q = blockIdx.y, *e = ecb + (long)q * nbq * kGN;
    const long t = (long)q * gridDim.x + blockIdx.x;
    int ey = INT_MIN, eu = INT_MIN;
#pragma unroll 4
    for (int c = 0; c < nr; ++c) {
        const double a = y[(t * nr + c) * 128 + threadIdx.x], b = u[(t * nr + c) * 128 + threadIdx.x];
        if (a != 0) ey = max(ey, exp_above(a) - e[c]);
        if (b != 0) eu = max(eu, exp_above(b) - e[nbq == 1 ? nr + c : kGN + c]);
    }
    // An ordinary row stays at the columns' scales: with its own, up to 2^3 larger, its first
    // digits would be, and accumulations shorter (4x4x2 grid, 5 bands, N=5000 140 us a call
    // with them, 132 so; in real space, with more columns to a row, own scales cost nothing).
    auto scale = [](int e) { return e == INT_MIN ? kZeroExp : e <= 0 && e >= -3 ? 0 : e; };
    const int2 e2 = make_int2(scale(ey), scale(eu));
    erb[t * 128 + threadIdx.x] = e2;
    if (max(e2.x, e2.y) > 0) rowfar[blockIdx.x * 128L + threadIdx.x] = *anyfar = 1;
}

// er[group][r]: exponent above the largest |x| 2^-ec of a row
__global__ void __launch_bounds__(128) k_qd_rowexp(const double *__restrict__ x,
                                                   const int *__restrict__ ec, int nr, int G,
                                                   int n_q, int *__restrict__ er) {
    const int nc = min(G, n_q - (int)blockIdx.y * G) * nr;
    int e = INT_MIN;
    for (int m = 0; m < nc; ++m) {
        const int q = blockIdx.y * G + m / nr;
        const double v = x[(((long)q * gridDim.x + blockIdx.x) * nr + m % nr) * 128 + threadIdx.x];
        // (what a column of kZeroExp has is in rows of weight 0)
        if (v != 0 && ec[blockIdx.y * 64 + m] != kZeroExp)
            e = max(e, exp_above(v) - ec[blockIdx.y * 64 + m]);
    }
    er[(blockIdx.x + (long)blockIdx.y * gridDim.x) * 128 + threadIdx.x] = e == INT_MIN ? kZeroExp : e;
}

// xa: [group][row tile][digit 7][128 x 64], thread = (row, eight columns)
__global__ void __launch_bounds__(256) k_qd_xa(const double *__restrict__ x,
                                               const int *__restrict__ ec,
                                               const int *__restrict__ er, int nr, int G, int n_q,
                                               __half *__restrict__ xa) {
    const long t = blockIdx.x + (long)blockIdx.y * gridDim.x;
    const int row = threadIdx.x & 127, nc = min(G, n_q - (int)blockIdx.y * G) * nr;
    uint8_t *out = reinterpret_cast<uint8_t *>(xa) + t * kRes * (long)kGA;
    for (int c = threadIdx.x >> 7; c < 8; c += 2) {
        long long v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int m = c * 8 + k, q = blockIdx.y * G + m / nr;
            const int e = m < nc ? ec[blockIdx.y * 64 + m] : kZeroExp;
            v[k] = e == kZeroExp
                       ? 0
                       : fixed_point(x[(((long)q * gridDim.x + blockIdx.x) * nr + m % nr) * 128 + row],
                                     55 - e - er[t * 128 + row]);
        }
        uint4 w[kRes];
        digits8<kRes>(v, w);
#pragma unroll
        for (int d = 0; d < kRes; ++d)
            *reinterpret_cast<uint4 *>(out + d * kGA + sw_place(row, c)) = w[d];
    }
}

// xb: [q][tile of [y | u]][K block 64 rows][digit 7][64 x 64], thread = (column,
// eight rows), and the digits' norms
__global__ void __launch_bounds__(256) k_qd_xb(const double *__restrict__ y,
                                               const double *__restrict__ u,
                                               const int *__restrict__ ecb,
                                               const int2 *__restrict__ erb, int nr, int nbq,
                                               long nrt, long nkb, __half *__restrict__ xb,
                                               float *__restrict__ nrm) {
    const long kb = blockIdx.x, t = blockIdx.y;                   // t = q nbq + tile
    const int q = (int)(t / nbq), j = (int)(t % nbq), c = threadIdx.x & 7;
    uint8_t *out = reinterpret_cast<uint8_t *>(xb) + (t * nkb + kb) * kRes * (long)kGB;
    const long r0 = kb * kGK + c * 8;
    for (int col = threadIdx.x >> 3; col < kGN; col += 32) {
        const double *src = nullptr;
        if (nbq == 1) {
            if (col < nr) src = y;
            else if (col < 2 * nr) src = u;
        } else if (col < nr) {
            src = j == 0 ? y : u;
        }
        const int cc = nbq == 1 && col >= nr ? col - nr : col;
        const bool of_y = src == y;
        const int e = ecb[t * kGN + col];
        const int2 *es = erb + q * nrt * 128 + r0;
        if (src) src += (((long)q * nrt + (r0 >> 7)) * nr + cc) * 128 + (r0 & 127);
        long long v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            v[k] = src ? fixed_point(src[k], 55 - e - (of_y ? es[k].x : es[k].y)) : 0;
        uint4 w[kRes];
        digits8<kRes>(v, w);
#pragma unroll
        for (int d = 0; d < kRes; ++d)
            *reinterpret_cast<uint4 *>(out + d * kGB + sw_place(col, c)) = w[d];
        digit_norms(w, c, nrm + (t * nkb + kb) * kRes * kGN, kGN, col);
    }
}

// ------------------------------------------------- once per call
// Digits of the real form of A_q, q = partner(k), in the tile of x_k: block (row, k),
// one warp.  A_q = alpha_p, or alpha_p^H for the second member of the pair; row 2 n is
// (Re, -Im) and row 2 n + 1 (Im, Re) of complex row n.  The K axis carries the scales of
// x's columns; outside x_k's the row is zero.  cofs: where x_q's column begins, and
// whether q is its own partner, the first or the second of two.
struct QAlpha {                    // alpha1 itself, or the psi that it follows from
    const double2 *alpha, *psi;
    const int *pair_q;
    const long *off;
    const double *pcoef;
    int n_pairs;
};
__global__ void __launch_bounds__(32) k_qd_alpha(const QAlpha src, const int *__restrict__ qpair,
                                                 const int *__restrict__ qrole,
                                                 const int *__restrict__ qpartner,
                                                 const int *__restrict__ ec, int nb, int G, int nrt,
                                                 __half *__restrict__ yb, int *__restrict__ et,
                                                 int *__restrict__ cofs,
                                                 int *__restrict__ wtop, int *__restrict__ failed) {
    __shared__ long long s[64];
    const int nr = 2 * nb, lane = threadIdx.x, grp = blockIdx.y / G, k0 = blockIdx.y % G * nr;
    const int q = qpartner[blockIdx.y], row = k0 + blockIdx.x, n = blockIdx.x >> 1;
    const int *e2 = ec + grp * 64 + k0;
    pdl_enter();
    s[lane] = s[lane + 32] = 0;
    __syncwarp();
    double v0 = 0, v1 = 0;                 // the two columns of band lane
    if (lane < nb) {
        const int p = qpair[q], role = qrole[q], i = role ? lane : n, j = role ? n : lane;
        double2 a = src.alpha ? src.alpha[((long)p * nb + i) * nb + j]
                              : q_alpha1(src.psi, src.pair_q, src.off, src.off + src.n_pairs, src.pcoef,
                                         p, i, j, nb);
        if (role) a.y = -a.y;
        v0 = blockIdx.x & 1 ? a.y : a.x;
        v1 = blockIdx.x & 1 ? a.x : -a.y;
    }
    int e = INT_MIN;
    if (v0 != 0) e = isfinite(v0) ? exp_above(v0) + e2[2 * lane] : kBadExp;
    if (v1 != 0) e = max(e, isfinite(v1) ? exp_above(v1) + e2[2 * lane + 1] : kBadExp);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    if (e == INT_MIN) e = 0;
    if (lane < nb && e < kBadExp / 2) {
        s[k0 + 2 * lane] = fixed_point(v0, 62 + e2[2 * lane] - e);
        s[k0 + 2 * lane + 1] = fixed_point(v1, 62 + e2[2 * lane + 1] - e);
    }
    __syncwarp();
    if (lane < 8) {
        long long v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = s[lane * 8 + k];
        uint4 w[kCall];
        digits8<kCall>(v, w);
        uint8_t *out = reinterpret_cast<uint8_t *>(yb) + (long)grp * kCall * kGB;
#pragma unroll
        for (int d = 0; d < kCall; ++d)
            *reinterpret_cast<uint4 *>(out + d * kGB + sw_place(row, lane)) = w[d];
    }
    if (blockIdx.x == 0 && blockIdx.y == 0 && lane >= 30) wtop[lane - 30] = INT_MIN;
    if (blockIdx.x == 0 && blockIdx.y == 0 && lane == 29) *failed = 0;
    // (there are no more pairs than q-points)
    if (blockIdx.x == 0 && (int)blockIdx.y < src.n_pairs && lane < 3) wtop[4 + 4 * blockIdx.y + lane] = INT_MIN;
    if (lane == 0) {
        et[grp * 64 + row] = e;
        cofs[grp * 64 + row] =
            4 * (q * nrt * nr + (int)blockIdx.x) + (qpartner[q] == q ? 0 : 1 + qrole[q]);
    }
}

// Row weights (k_q_rows of qspace.cu): 64 rows a block, four threads a row, each a
// quarter of the sums (with one thread a row its loads took 13 us at 2000 rows).
// Rows past the end get zeros.  wtop: the largest exponents of w_cross and w_diag over the
// rows whose own scales are at most 1 everywhere; and of each pair (q1, q2), from 4 + 4 pair
// on, over the others (rowfar), of w_cross with the row's scales in u of q1 and y of q2, of
// w_cross with those in y of q1 and u of q2, and of w_diag with those in u of both.  An
// ensemble without such rows takes the form without (kFar; with it 2 to 4 us of 85 with 36
// pairs).  kBadExp of one that is not finite.
template <bool kFar>
__global__ void __launch_bounds__(256) k_qd_rows(const double *__restrict__ qp, int ngrp,
                                                 const double *__restrict__ u,
                                                 const double *__restrict__ y,
                                                 const double2 *__restrict__ R1,
                                                 const double *__restrict__ rho, int S, long R,
                                                 long nrt, int nb, int iq_pert, int apply_d4,
                                                 const int2 *__restrict__ erb,
                                                 const int *__restrict__ rowfar,
                                                 const int *__restrict__ pair_q, int n_pairs,
                                                 double2 *__restrict__ rowc,
                                                 int *__restrict__ wtop) {
    __shared__ double sum[8][4][64];
    __shared__ int we[2][kFar ? 64 : 1];      // exponents of w_cross, w_diag of the rows far out
    const int part = threadIdx.x >> 6, i = threadIdx.x & 63;
    const long r = blockIdx.x * 64L + i;
    pdl_enter();
    double s[8] = {};              // total, bfw, sum u conj(R1), sum y conj(R1)
    if (r < R) {
        const double *o = qp + 4 * part * R + r;
#pragma unroll 4
        for (int g = part; g < ngrp; g += 4, o += 16 * R)
#pragma unroll
            for (int k = 0; k < 4; ++k) s[k] += o[k * R];
        const long base = (((long)iq_pert * nrt + (r >> 7)) * 2 * nb) * 128 + (r & 127);
#pragma unroll 2
        for (int n = part; n < nb; n += 4) {
            const double2 a = R1 ? R1[n] : make_double2(0, 0);
            const double ur = u[base + n * 256], ui = u[base + n * 256 + 128];
            const double yr = y[base + n * 256], yi = y[base + n * 256 + 128];
            s[4] = fma(ur, a.x, fma(ui, a.y, s[4]));
            s[5] = fma(ui, a.x, fma(-ur, a.y, s[5]));
            s[6] = fma(yr, a.x, fma(yi, a.y, s[6]));
            s[7] = fma(yi, a.x, fma(-yr, a.y, s[7]));
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) sum[k][part][i] = s[k];
    __syncthreads();
    if (!kFar && threadIdx.x >= 64) return;
    if (threadIdx.x < 64) {
        const int far = kFar ? rowfar[r] : 0;
        double2 w[4] = {};
        if (r < R) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
                s[k] = (sum[k][0][i] + sum[k][1][i]) + (sum[k][2][i] + sum[k][3][i]);
            const double rw = rho[(unsigned)r / (unsigned)S], d4 = apply_d4 ? 1.0 : 0.0;
            const double t3 = rw / 3.0, t8 = -d4 * rw / 8.0, t4 = -d4 * rw / 4.0;
            w[0] = make_double2(s[0] * (-0.5 * t3), s[1] * (-0.5 * t3));
            w[1] = make_double2(s[2] * -t3, s[3] * -t3);
            w[2] = make_double2(fma(s[4], t3, s[0] * t8), fma(s[5], t3, s[1] * t8));
            w[3] = make_double2(fma(s[6], t3, s[2] * t4), fma(s[7], t3, s[3] * t4));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) rowc[4 * r + k] = w[k];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const unsigned long long a =
                max((unsigned long long)__double_as_longlong(w[2 + k].x) & 0x7fffffffffffffffULL,
                    (unsigned long long)__double_as_longlong(w[2 + k].y) & 0x7fffffffffffffffULL);
            const int e = a >= 0x7ff0000000000000ULL ? kBadExp
                          : a ? exp_above(__longlong_as_double((long long)a)) : INT_MIN;
            if (kFar) we[k][i] = far ? e : INT_MIN;
            const int m = __reduce_max_sync(0xffffffffu, far ? INT_MIN : e);
            if ((threadIdx.x & 31) == 0) atomicMax(wtop + k, m);
        }
    }
    if (!kFar) return;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int p = threadIdx.x >> 5; p < n_pairs; p += 8) {
        const int2 *s1 = erb + pair_q[2 * p] * nrt * 128 + blockIdx.x * 64L,
                   *s2 = erb + pair_q[2 * p + 1] * nrt * 128 + blockIdx.x * 64L;
        int top[3] = {INT_MIN, INT_MIN, INT_MIN};
#pragma unroll
        for (int h = 0; h < 64; h += 32) {
            const int c = we[0][h + lane], d = we[1][h + lane];
            const int2 a = s1[h + lane], b = s2[h + lane];
            auto with = [](int e, int x) { return e == INT_MIN || e == kBadExp ? e : e + x; };
            top[0] = max(top[0], with(c, a.y + b.x));
            top[1] = max(top[1], with(c, a.x + b.y));
            top[2] = max(top[2], with(d, a.y + b.y));
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int e = __reduce_max_sync(0xffffffffu, top[k]);
            if (lane == k) atomicMax(wtop + 4 + 4 * p + k, e);
        }
    }
}

// Digits of the rows [A1 | A2] of pair blockIdx.y over a group of K blocks: thread =
// (band, eight rows), which makes four rows of digits; with few bands several K blocks
// side by side.  The scales are bounds from those of the weights and of the columns; a
// row's own scale goes into the shift that cuts the digits.  blockIdx.y == n_pairs: the
// partial f of the group's rows.
__global__ void __launch_bounds__(128) k_qd_wbuild(
    const double *__restrict__ u, const double *__restrict__ y, const double2 *__restrict__ rowc,
    const int *__restrict__ wtop, const int *__restrict__ ecb, const int2 *__restrict__ erb,
    const int *__restrict__ pair_q, int n_pairs, int nb, int nbq, int iq_pert, long nrt, long nkb,
    int per, uint32_t abytes, __half *__restrict__ wa,
    int *__restrict__ ew, double2 *__restrict__ fpart) {
    __shared__ double2 fs[16];
    const int c = threadIdx.x & 7, m = threadIdx.x >> 3, nr = 2 * nb, p = blockIdx.y;
    const int wide = max(1, 16 / nb);            // K blocks side by side
    const long kb0 = blockIdx.x * (long)per, kb1 = min(nkb, kb0 + per);
    const bool force = p == n_pairs;
    // (what does not change between calls is read ahead)
    const int q1 = force ? iq_pert : pair_q[2 * p];
    const int2 *es2 = erb + (force ? 0 : pair_q[2 * p + 1]) * nrt * 128;
    pdl_enter();
    if (force) {
        for (int n0 = 0; n0 < nb; n0 += 16) {
            const int n = n0 + (nb < 16 ? m % nb : m);
            double fr = 0, fi = 0;
            if (n < nb && m < nb * wide)
                for (long kb = kb0 + (nb < 16 ? m / nb : 0); kb < kb1; kb += wide) {
                    const long r0 = kb * kGK + c * 8;
                    const long o = (((long)q1 * nrt + (r0 >> 7)) * nr + 2 * n) * 128 + (r0 & 127);
#pragma unroll 4
                    for (int k = 0; k < 8; ++k) {
                        const double2 a = rowc[4 * (r0 + k)], b = rowc[4 * (r0 + k) + 1];
                        const double yr = y[o + k], yi = y[o + 128 + k], ur = u[o + k],
                                     ui = u[o + 128 + k];
                        fr = fma(a.x, yr, fma(-a.y, yi, fma(b.x, ur, fma(-b.y, ui, fr))));
                        fi = fma(a.x, yi, fma(a.y, yr, fma(b.x, ui, fma(b.y, ur, fi))));
                    }
                }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                fr += __shfl_xor_sync(0xffffffffu, fr, o);
                fi += __shfl_xor_sync(0xffffffffu, fi, o);
            }
            if (c == 0) fs[m] = make_double2(fr, fi);
            __syncthreads();
            if ((int)threadIdx.x < min(16, nb - n0)) {
                double2 v = fs[threadIdx.x];
                for (int k = 1; k < wide && nb < 16; ++k) {
                    v.x += fs[k * nb + threadIdx.x].x;
                    v.y += fs[k * nb + threadIdx.x].y;
                }
                fpart[blockIdx.x * (long)nb + n0 + threadIdx.x] = v;
            }
            __syncthreads();
        }
        return;
    }
    const int *wt = wtop + 4 + 4 * p;
    const int w0 = max(wtop[0], wt[0]), w1 = max(wtop[0], wt[1]), w2 = max(wtop[1], wt[2]);
    uint8_t *out = reinterpret_cast<uint8_t *>(wa) + p * nkb * kCall * (long)abytes;
    for (int n0 = 0; n0 < nb; n0 += 16) {
        const int n = n0 + (nb < 16 ? m % nb : m);
        if (n >= nb || m >= nb * wide) break;
        const int *ey = ecb + (long)q1 * nbq * kGN + 2 * n, *eu = ey + (nbq == 1 ? nr : kGN);
        const int ym = max(ey[0], ey[1]), um = max(eu[0], eu[1]);
        // real and imaginary part: two products each, and two of them in A2
        auto bound = [](int a, int e) { return a == INT_MIN ? INT_MIN : a + e; };
        const int b1 = bound(w0, um), b2 = max(bound(w1, ym), bound(w2, um));
        const bool bad1 = w0 == kBadExp, bad2 = w1 == kBadExp || w2 == kBadExp;
        const int e1 = bad1 ? kBadExp : b1 == INT_MIN ? 0 : b1 + 1;
        const int e2 = bad2 ? kBadExp : b2 == INT_MIN ? 0 : b2 + 2;
        if (blockIdx.x == 0 && c == 0) {
            ew[p * kGM + 2 * n] = ew[p * kGM + 2 * n + 1] = e1;
            ew[p * kGM + nr + 2 * n] = ew[p * kGM + nr + 2 * n + 1] = e2;
        }
        for (long kb = kb0 + (nb < 16 ? m / nb : 0); kb < kb1; kb += wide) {
            const long r0 = kb * kGK + c * 8;
            const long o = (((long)q1 * nrt + (r0 >> 7)) * nr + 2 * n) * 128 + (r0 & 127);
            const double2 *ur = reinterpret_cast<const double2 *>(u + o),
                          *yr = reinterpret_cast<const double2 *>(y + o);
            long long a1r[8], a1i[8], a2r[8], a2i[8];
            // A1 = -wc u, A2 = -(wc y + wd u)
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                const double2 vur = ur[k / 2], vui = ur[64 + k / 2], vyr = yr[k / 2], vyi = yr[64 + k / 2];
                const int4 es = *reinterpret_cast<const int4 *>(es2 + r0 + k);    // of two rows
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double pu = h ? vur.y : vur.x, pv = h ? vui.y : vui.x;
                    const double py = h ? vyr.y : vyr.x, pz = h ? vyi.y : vyi.x;
                    const double2 wc = rowc[4 * (r0 + k + h) + 2], wd = rowc[4 * (r0 + k + h) + 3];
                    const int sy = h ? es.z : es.x, su = h ? es.w : es.y;
                    const double xr = fma(wc.y, pv, -wc.x * pu), xi = fma(-wc.x, pv, -wc.y * pu);
                    const double zr = fma(wd.y, pv, fma(-wd.x, pu, fma(wc.y, pz, -wc.x * py)));
                    const double zi = fma(-wd.x, pv, fma(-wd.y, pu, fma(-wc.x, pz, -wc.y * py)));
                    a1r[k + h] = bad1 ? 0 : fixed_point(xr, 62 - e1 + sy);
                    a1i[k + h] = bad1 ? 0 : fixed_point(xi, 62 - e1 + sy);
                    a2r[k + h] = bad2 ? 0 : fixed_point(zr, 62 - e2 + su);
                    a2i[k + h] = bad2 ? 0 : fixed_point(zi, 62 - e2 + su);
                }
            }
            uint8_t *blk = out + kb * kCall * (long)abytes;
            auto put = [&](const long long(&v)[8], int row) {
                uint4 w[kCall];
                digits8<kCall>(v, w);
#pragma unroll
                for (int d = 0; d < kCall; ++d)
                    *reinterpret_cast<uint4 *>(blk + d * abytes + sw_place(row, c)) = w[d];
            };
            put(a1r, 2 * n);
            put(a1i, 2 * n + 1);
            put(a2r, nr + 2 * n);
            put(a2i, nr + 2 * n + 1);
        }
    }
}

// The real products of the tiles to complex blocks, and f: H[row][col] of pair p and
// split s at gpart[((s n_pairs + p) 128 + row) ld + col].  Eight lanes an element, each
// every eighth split.  After a wait that gave up the results are NaN: calls that do not
// return to the host report it that way (and in tdscha_qctx_sync).
__global__ void __launch_bounds__(128) k_qd_final(const double *__restrict__ gpart, int ns, int nb,
                                                  int n_pairs, int nbq,
                                                  const double2 *__restrict__ fpart, int nff,
                                                  double inv_norm, const int *__restrict__ failed,
                                                  double2 *__restrict__ f, double2 *__restrict__ d2v) {
    const int nr = 2 * nb, ld = nbq * kGN, uc = nbq == 1 ? nr : kGN;
    const long n = (long)n_pairs * nb * nb, e = blockIdx.x * 16L + (threadIdx.x >> 3);
    const int k0 = threadIdx.x & 7;
    pdl_enter();
    double re = 0, im = 0;
    double2 *out = nullptr;
    if (e < n) {
        const int p = (int)(e / (nb * nb)), m = (int)(e - (long)p * nb * nb), i = m / nb, j = m % nb;
        const long step = (long)n_pairs * kGM * ld;
        const double *h = gpart + k0 * step + (long)p * kGM * ld;
#pragma unroll 2
        for (int s = k0; s < ns; s += 8, h += 8 * step) {
            const double2 a0 = *reinterpret_cast<const double2 *>(h + (2L * i) * ld + 2 * j),
                          a1 = *reinterpret_cast<const double2 *>(h + (2L * i + 1) * ld + 2 * j),
                          b0 = *reinterpret_cast<const double2 *>(h + (nr + 2L * i) * ld + uc + 2 * j),
                          b1 = *reinterpret_cast<const double2 *>(h + (nr + 2L * i + 1) * ld + uc + 2 * j);
            re += (a0.x + a1.y) + (b0.x + b1.y);
            im += (a1.x - a0.y) + (b1.x - b0.y);
        }
        out = d2v + e;
    } else if (e < n + nb) {
        for (int k = k0; k < nff; k += 8) {
            const double2 v = fpart[(long)k * nb + (e - n)];
            re += v.x;
            im += v.y;
        }
        out = f + (e - n);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if (*failed) inv_norm = __longlong_as_double(0x7ff8000000000000LL);
    if (out && k0 == 0) *out = make_double2(re * inv_norm, im * inv_norm);
}

// ------------------------------------------------------------- host side
static size_t pad1k(size_t b) { return (b + 1023) & ~size_t(1023); }

void qdigits_release(tdscha_qctx *c) {
    if (!c->qd) return;
    cached_free(c->qd->slab);
    cached_free(c->qd->pslab);
    flag_free(c->qd->err);
    delete c->qd;
    c->qd = nullptr;
}

struct QPart {
    void **p;
    size_t bytes;
};
static size_t place(const std::vector<QPart> &parts, void *slab) {
    size_t at = 0;
    for (const QPart &q : parts) {
        if (slab) *q.p = reinterpret_cast<uint8_t *>(slab) + at;
        at += pad1k(q.bytes);
    }
    return at;
}

// The resident digit operands of a context; leaves c->qd null (the float64 kernels
// of qspace.cu serve it) where they do not fit or with TDSCHA_FP64_DIGITS=0.
static int qdigits_prepare(tdscha_qctx *c) {
    if (c->qd) return TDSCHA_OK;
    if (const char *e = getenv("TDSCHA_FP64_DIGITS"))
        if (atoi(e) == 0) return TDSCHA_OK;
    QDigitStore *x = new QDigitStore();
    const int n_q = c->n_q, nb = c->nb, nr = 2 * nb;
    x->nr = nr;
    x->nbq = 2 * nr <= kGN ? 1 : 2;
    x->nrt = (c->R + kGM - 1) / kGM;
    x->Rp = x->nrt * kGM;
    x->nkb = x->Rp / kGK;
    if (const char *b = getenv("TDSCHA_WAIT_BUDGET_CYCLES")) x->budget = atoll(b);
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&x->nsm, cudaDevAttrMultiProcessorCount, dev);
    // as many q-points to a tile as there are tiles to keep every SM busy
    x->G = (int)std::max<long>(1, std::min<long>(kGK / nr, n_q * x->nrt / x->nsm));
    x->ngrp = ceil_div(n_q, x->G);
    const size_t col = sizeof(double) * (size_t)n_q * nr * x->Rp, rows = (size_t)n_q * x->Rp;
    float *nrm = nullptr, *fl = nullptr;
    const std::vector<QPart> parts = {
        {(void **)&x->x, col}, {(void **)&x->g, col}, {(void **)&x->u, col}, {(void **)&x->y, col},
        {(void **)&x->xa, (size_t)x->ngrp * x->Rp * kGK * 2 * kRes},
        {(void **)&x->xb, rows * x->nbq * kGN * 2 * kRes},
        {(void **)&x->qp, sizeof(double) * 4 * x->ngrp * (size_t)c->R},
        {(void **)&x->rowc, sizeof(double) * 8 * x->Rp},
        {(void **)&x->er, sizeof(int) * x->ngrp * x->Rp},
        {(void **)&nrm, sizeof(float) * kRes * (size_t)n_q * x->nbq * kGN * x->nkb},
        {(void **)&x->erb, sizeof(int2) * rows},
        {(void **)&x->wtop, sizeof(int) * 4 * (n_q + 1)},
        // zero from the start: flags, exponents of padding columns, rows of padding bands
        {(void **)&x->rowfar, sizeof(int) * x->Rp},
        {(void **)&x->ec, sizeof(int) * x->ngrp * 64},
        {(void **)&x->ecb, sizeof(int) * (size_t)n_q * x->nbq * kGN},
        {(void **)&x->et, sizeof(int) * x->ngrp * 64},
        {(void **)&x->cofs, sizeof(int) * x->ngrp * 64},
        {(void **)&fl, sizeof(float) * (kFlushes * kRes + 1)},
        {(void **)&x->yb, (size_t)x->ngrp * kCall * kGB},
    };
    const size_t total = place(parts, nullptr);
    x->err = flag_alloc();
    if (!x->err || !memory_to_spare(total) || cached_malloc(&x->slab, total) != cudaSuccess) {
        cudaGetLastError();
        flag_free(x->err);
        delete x;
        return TDSCHA_OK;
    }
    c->qd = x;
    place(parts, x->slab);
    uint8_t *z = reinterpret_cast<uint8_t *>(x->rowfar);
    TDS_CUDA(cudaMemsetAsync(z, 0, (uint8_t *)x->slab + total - z, 0));
    const dim3 gt((unsigned)x->nrt, n_q);
    k_qd_cols<<<gt, 256>>>((const double *)c->Xr, (const double *)c->Yr, c->fY, c->fpsi, c->L, nb,
                           c->R, x->x, x->g, x->u, x->y);
    TDS_CHECK_LAUNCH();
    k_qd_colscale<<<dim3(nr, n_q), 128>>>(x->x, x->y, x->u, c->rho, c->S, c->rho_top, c->R, x->nrt, nr,
                                          x->nbq, x->G, x->ec, x->ecb);
    TDS_CHECK_LAUNCH();
    k_qd_rowscale<<<gt, 128>>>(x->y, x->u, x->ecb, nr, x->nbq, x->erb, x->rowfar,
                               reinterpret_cast<int *>(fl) + kFlushes * kRes);
    TDS_CHECK_LAUNCH();
    const dim3 gg((unsigned)x->nrt, x->ngrp);
    k_qd_rowexp<<<gg, 128>>>(x->x, x->ec, nr, x->G, n_q, x->er);
    TDS_CHECK_LAUNCH();
    k_qd_xa<<<gg, 256>>>(x->x, x->ec, x->er, nr, x->G, n_q, x->xa);
    TDS_CHECK_LAUNCH();
    k_qd_xb<<<dim3((unsigned)x->nkb, n_q * x->nbq), 256>>>(x->y, x->u, x->ecb, x->erb, nr, x->nbq,
                                                           x->nrt, x->nkb, x->xb, nrm);
    TDS_CHECK_LAUNCH();
    TDS_CUDA(dg_windows(nrm, n_q * x->nbq, kGN, (int)x->nkb, fl, 0));
    float h_fl[kFlushes * kRes + 1];
    TDS_CUDA(cudaMemcpy(h_fl, fl, sizeof(h_fl), cudaMemcpyDeviceToHost));
    x->flush = digits_flush(h_fl);
    std::memcpy(&x->anyfar, h_fl + kFlushes * kRes, sizeof(int));
    TDS_CUDA((dg_setup<DG_QDOTS, true>()));
    TDS_CUDA((dg_setup<DG_PARTS, true>()));
    return TDSCHA_OK;
}

// The operands and the buffers of the layout's pairs, for a context in float64
int qdigits_set_pert(tdscha_qctx *c) {
    if (c->precision == TDSCHA_PREC_MIXED) return TDSCHA_OK;
    TDS_TRY(qdigits_prepare(c));
    QDigitStore *x = c->qd;
    if (!x) return TDSCHA_OK;
    std::vector<int> pq(2 * (size_t)c->n_pairs);
    TDS_CUDA(cudaMemcpy(pq.data(), c->pair_q, sizeof(int) * pq.size(), cudaMemcpyDeviceToHost));
    x->n_pairs = c->n_pairs;
    x->abytes = (uint32_t)(2 * x->nr + 7) / 8 * 1024;
    x->kbps = dg_blocks_per_split(x->nkb, x->flush, x->n_pairs, x->nbq, x->nsm);
    x->ns = ceil_div(x->nkb, x->kbps);
    // about 16 W blocks per SM, at most 16 passes over K blocks each
    const int wide = std::max(1, 16 / c->nb);
    x->per = wide * (int)std::max<long>(1, std::min<long>(16, x->nkb * x->n_pairs / (x->nsm * 16L * wide)));
    x->nfc = ceil_div(x->nkb, x->per);
    std::vector<int> bmap(x->n_pairs);
    for (int p = 0; p < x->n_pairs; ++p) bmap[p] = pq[2 * p + 1] * x->nbq;
    const std::vector<QPart> parts = {
        {(void **)&x->failed, sizeof(int)},
        {(void **)&x->gpart, sizeof(double) * (size_t)x->ns * x->n_pairs * kGM * x->nbq * kGN},
        {(void **)&x->fpart, sizeof(double) * 2 * x->nfc * c->nb},
        {(void **)&x->ew, sizeof(int) * x->n_pairs * kGM},
        {(void **)&x->bmap, sizeof(int) * x->n_pairs},
        {(void **)&x->wa, (size_t)x->n_pairs * x->nkb * kCall * x->abytes},
    };
    cudaDeviceSynchronize();
    cached_free(x->pslab);
    x->pslab = nullptr;
    const size_t total = place(parts, nullptr);
    if (!memory_to_spare(total) || cached_malloc(&x->pslab, total) != cudaSuccess) {
        cudaGetLastError();
        x->pslab = nullptr;
        x->n_pairs = 0;         // this perturbation on the CUDA cores
        return TDSCHA_OK;
    }
    place(parts, x->pslab);
    TDS_CUDA(cudaMemcpy(x->bmap, bmap.data(), sizeof(int) * x->n_pairs, cudaMemcpyHostToDevice));
    TDS_CUDA(cudaMemset(x->wa, 0, (size_t)x->n_pairs * x->nkb * kCall * x->abytes));
    TDS_CUDA(cudaStreamSynchronize(0));     // runs may be on streams that do not wait for this one
    return TDSCHA_OK;
}

bool qdigits_ready(const tdscha_qctx *c) { return c->qd && c->qd->n_pairs > 0; }

int qdigits_path(const tdscha_qctx *c) {
    if (c->n_pairs == 0 || c->precision == TDSCHA_PREC_MIXED) return TDSCHA_FP64_PENDING;
    return qdigits_ready(c) ? TDSCHA_FP64_TENSOR_CORES : TDSCHA_FP64_CUDA_CORES;
}

// After the stream has been waited for
int qdigits_check_error(tdscha_qctx *c) {
    if (!c->qd || !*(volatile int *)c->qd->err) return TDSCHA_OK;
    const int v = *(volatile int *)c->qd->err;
    *(volatile int *)c->qd->err = 0;
    set_error("tensor-core pipeline: a bounded wait expired (code %d)", v);
    return TDSCHA_ERR_TIMEOUT;
}

// The averages of c->R1, c->alpha, or of psi's, into c->f, c->d2v.
int qdigits_perturb(tdscha_qctx *c, int apply_d4, const double *psi, cudaStream_t st) {
    QDigitStore *x = c->qd;
    const int n_q = c->n_q, nb = c->nb, live = x->G * x->nr;
    const double2 *ps = reinterpret_cast<const double2 *>(psi);
    const QAlpha src{ps ? nullptr : c->alpha, ps, c->pair_q, c->q_off, c->pcoef, c->n_pairs};
    const double2 *R1 = !ps ? c->R1 : c->ignore_v3 ? nullptr : ps;
    double2 *rowc = reinterpret_cast<double2 *>(x->rowc), *fpart = reinterpret_cast<double2 *>(x->fpart);
    TDS_CUDA(launch_pdl(k_qd_alpha, dim3(x->nr, n_q), 32, 0, st, src, (const int *)c->qpair,
                        (const int *)c->qrole, (const int *)c->qpartner, (const int *)x->ec, nb, x->G,
                        (int)x->nrt, x->yb, x->et, x->cofs, x->wtop, x->failed));
    DgArgs a{};
    a.a = x->xa;
    a.b = x->yb;
    a.nkb = a.kbps = a.flush = 1;
    a.kk = ceil_div(live, 16);
    a.hc = dg_part_cols(live);
    a.win = 1;
    a.abytes = kGA;
    a.nat = (int)x->nrt;
    a.nbt = x->ngrp;
    a.nitems = (long)x->nrt * x->ngrp;
    a.cofs = x->cofs;
    a.nr = x->nr;
    a.err = x->err;
    a.failed = x->failed;
    a.budget = x->budget;
    a.dt = x->x;
    a.gt = x->g;
    a.et = x->et;
    a.er = x->er;
    a.qp = x->qp;
    a.R = c->R;
    a.M = live;
    TDS_CUDA((dg_launch<DG_QDOTS, true>(a, x->nsm, st)));
    TDS_CUDA(launch_pdl(x->anyfar ? k_qd_rows<true> : k_qd_rows<false>, (unsigned)x->nkb, 256, 0, st, (const double *)x->qp, x->ngrp,
                        (const double *)x->u, (const double *)x->y, R1, (const double *)c->rho, c->S,
                        c->R, x->nrt, nb, c->iq_pert, apply_d4, (const int2 *)x->erb,
                        (const int *)x->rowfar, (const int *)c->pair_q, x->n_pairs, rowc, x->wtop));
    TDS_CUDA(launch_pdl(k_qd_wbuild, dim3(x->nfc, x->n_pairs + 1), 128, 0, st, (const double *)x->u,
                        (const double *)x->y, (const double2 *)rowc,
                        (const int *)x->wtop, (const int *)x->ecb, (const int2 *)x->erb,
                        (const int *)c->pair_q, x->n_pairs, nb, x->nbq, c->iq_pert, x->nrt, x->nkb, x->per, x->abytes, x->wa, x->ew, fpart));
    DgArgs b{};
    b.a = x->wa;
    b.b = x->xb;
    b.nkb = (int)x->nkb;
    b.kbps = x->kbps;
    b.flush = x->flush;
    b.kk = kGK / 16;
    b.hc = dg_part_cols(x->nbq == 1 ? 2 * x->nr : x->nr);
    b.win = 1;
    b.abytes = x->abytes;
    b.nat = x->n_pairs;
    b.nbt = x->nbq;
    b.nitems = (long)x->n_pairs * x->nbq * x->ns;
    b.bmap = x->bmap;
    b.Mp = x->nbq * kGN;
    b.M = x->nbq * kGN;
    b.err = x->err;
    b.failed = x->failed;
    b.budget = x->budget;
    b.ec = x->ecb;
    b.ew = x->ew;
    b.gpart = x->gpart;
    b.rmod = kGM;
    b.rlive = 2 * x->nr;
    b.rows_b = (long)x->n_pairs * kGM;
    TDS_CUDA((dg_launch<DG_PARTS, true>(b, x->nsm, st)));
    const long n = (long)x->n_pairs * nb * nb + nb;
    TDS_CUDA(launch_pdl(k_qd_final, ceil_div(n, 16), 128, 0, st, (const double *)x->gpart, x->ns, nb,
                        x->n_pairs, x->nbq, (const double2 *)fpart, x->nfc,
                        1.0 / (c->sum_rho * c->S), (const int *)x->failed, c->f, c->d2v));
    return TDSCHA_OK;
}

}  // namespace tdscha
