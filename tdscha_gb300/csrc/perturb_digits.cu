// Float64 perturbation averages by exact digit products on the tensor cores.
//
// The two contractions of perturb_fp64.cu carry float64 operands that GB300's
// CUDA cores multiply at about 1.2 TFLOP/s.  Here every operand is written as
// a sum of 8-bit digits of one fixed-point scale per row (the splitting of
// Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 95 (2012); on tensor
// cores Mukunoki, Ozaki, Ogita and Imamura, ISC 2020),
//
//   x = 2^E sum_i d_i 2^(-7-8i),   d_i whole, |d_i| <= 128,
//
// held as fp16, which represents every digit exactly.  A product of two digits
// is a whole number of at most 2^14 and a sum of 1024 of them at most 2^24, so
// the fp32 accumulators of tcgen05.mma hold the digit sums without rounding.
// The products d_i d_j of one order o = i + j share a scale and an accumulator;
// the epilogue adds the orders as 64-bit integers and rounds once, to float64.
//
// Digits: 7 of the resident operand (55 bits under the largest element of its
// row), 8 of the operand made per call (62 bits), products of order 0..7 (35 of
// 56).  Before the sums an element of the resident operand is rounded by up to 2^-56
// of its row's largest, one of the per-call operand by 2^-63.  Left out are the products
// of order 8 and above: six pairs of digits, up to 2^14 in units of 2^-77 each, 2^-60.4 of
// the product of the two rows' largest elements for every element of the sum.  Both are
// relative to the largest elements of the rows, not to the result; the float64
// sums this replaces round every partial sum at 2^-53 of itself.
//
// Length of an accumulation: three K blocks (192 elements) keep orders 0..4 exact
// for any input (5 * 192 products of 2^14 stay below 2^24).  The digits of real
// numbers are far from their limits, so the longest accumulation is chosen per
// ensemble by a bound that holds for every perturbation: by Cauchy and Schwarz the
// order-o sum is at most sum_i |d_i| 128 sqrt(K) with |d_i| the largest 2-norm of
// digit i over any K consecutive elements of any row, measured when the operands are
// made (k_dg_windows, digits_flush).  Gaussian displacements allow five to seven blocks.
// Orders 5..7 could round, by 2^-53 of the row maxima's product or less, only where the
// digits of two rows agree in sign and size over a whole accumulation.
//
// Error (2-norm, against 113-bit arithmetic) of f and d2v, these kernels | those
// of perturb_fp64.cu: M=573 N=2000 6.5e-16 6.9e-16 | 1.3e-15 1.2e-15; with Y1 over
// six decades 7.8e-16 7.6e-16 | 1.4e-15 1.2e-15; M=192 N=3000 1.4e-15 1.5e-15 |
// 1.7e-15 1.6e-15; M=24 N=400 48 images 1.2e-15 5.4e-16 | 3.1e-15 5.6e-16.
// One call: M=573 N=50000 57.1 -> 1.71 ms; M=189 N=10000 48 images 62.8 -> 2.09 ms;
// M=97 N=4999 554 -> 66 us; M=21 N=1000 245 -> 34 us.
//
// Scales: a mode's is the largest exponent of its elements, each less what its
// configuration's weight is below the largest weight (dg_weight_exp); a configuration's is
// the exponent above its largest element in those units.  Both are powers of two, and stage
// B's X is without the configuration's: W carries it instead.  So a configuration that the
// weights take out, or nearly so, costs the others nothing, however far out it lies, and
// loses itself at most as many bits as its weight is smaller (a configuration's scale is
// never further above 1 than that).  With the columns' maxima over all configurations as the
// only scales one outlier of weight 0, 1e6 times the others, took 20 bits from all of them:
// errors of d2v of 2e-11 (and 2e-9 at 1e8).  The mean exponent of a mode's elements as its
// scale leaves a mode of rounding noise over many decades, as symmetry makes them, to set
// the scales of the configurations.
//
// Form of the contractions, with g = y / f_Y (= f_psi y) so that both operands
// of the second stage come from x and g alone (u = f_Y x, y = f_Y g):
//
//   stage A   v = X Y1          q = x.v  p = g.v  s = x.(f_Y R1)  t = g.(f_Y R1)
//   rows      alpha = rho (s/3 - q/8)   beta = rho (t/3 - p/4)
//   W         w = alpha g + beta/2 x    f_avg = f_Y sum(-rho q/6 g - rho p/3 x)
//   stage B   H = W^T X         G[a][b] = f_Y,a f_Y,b H[b][a]
//
// Layouts (the kernels copy whole blocks, already in the 128-byte swizzle that
// the tensor core reads, with untiled bulk copies):
//   xa  rows of X      [row tile 128][K block 64 modes][digit 7][128 x 64]
//   xb  columns of X   [mode tile 64][K block 64 rows ][digit 7][ 64 x 64]
//   yb  rows of Y1_j   [image, mode tile 64][K block 64 modes][digit 8][64 x 64]
//   wa  columns of W_j [tile 128 of (image, mode)][K block 64 rows][digit 8][128 x 64]
//   dt, gt  x and g, float64, [row tile 128][mode][128 rows]
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>

#include "digits.cuh"

namespace tdscha {

// alpha, beta / 2 and the force weights (of g and of x) of the images' rows:
// abcc[(4 image + k) Rp + row]

// ------------------------------------------------- once per ensemble
// ec[m], ec[Mp + m]: largest weighted exponents of column m of D and of F (before: kNone)
constexpr int kNone = (int)0x80808080u;
__global__ void __launch_bounds__(128) k_dg_colexp(const double *__restrict__ D,
                                                   const double *__restrict__ F,
                                                   const double *__restrict__ rho, int rho_div, int rtop,
                                                   long R, int M, int Mp, long per,
                                                   int *__restrict__ ec) {
    __shared__ int less[128];      // what 128 rows' elements count for beside their exponents
    const int m = blockIdx.x * 128 + threadIdx.x;
    const double *a = (blockIdx.z ? F : D) + min(m, M - 1);
    const long r0 = blockIdx.y * per, r1 = min(R, r0 + per);
    int e = INT_MIN;
    for (long c0 = r0; c0 < r1; c0 += 128) {
        const int n = (int)min(128L, r1 - c0);
        const long r = c0 + threadIdx.x;
        __syncthreads();
        if (r < r1) {
            less[threadIdx.x] = dg_weight_exp(rho[rho_div == 1 ? r : r / rho_div], rtop);
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < n; ++k) {
            const double x = a[(c0 + k) * M];
            const int v = exp_above(x) + less[k];
            e = max(e, x != 0 ? v : INT_MIN);
        }
    }
    if (m < M && e > INT_MIN / 4) atomicMax(ec + blockIdx.z * Mp + m, e);
}

// From there: g's scales from y's, and 0 of a column without an element; eb has kZeroExp
// there, for what is scaled with it: Y1's rows and the bounds of W
__global__ void k_dg_colend(const double *__restrict__ fY, int M, int Mp, int *__restrict__ ec,
                            int *__restrict__ eb) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= 2 * Mp) return;
    const int e = ec[m], k = m % Mp, s = m >= Mp && k < M ? e - exp_above(fY[k]) : e;
    ec[m] = e == kNone ? 0 : s;
    eb[m] = e == kNone ? kZeroExp : s;
}

// dt, gt: 128 rows x 32 modes per block through shared memory.  Rows and modes
// past the end are zero.  g = y / f_Y by the reciprocal and one residual step
// (a division costs about ten float64 operations), so that f_Y g is y to one
// rounding; with f_psi y the rounding of f_psi would stand in every row alike.
__global__ void k_dg_cols(const double *__restrict__ D, const double *__restrict__ F,
                          const double *__restrict__ fY, long R, int M, int Mp,
                          double *__restrict__ dt, double *__restrict__ gt) {
    __shared__ double td[32][33], tg[32][33];
    const long rt = blockIdx.x;
    const int m0 = blockIdx.y * 32, tx = threadIdx.x, ty = threadIdx.y;
    const double fy = m0 + tx < M ? fY[m0 + tx] : 1.0, rf = 1.0 / fy;
    for (int part = 0; part < 4; ++part) {
        for (int k = ty; k < 32; k += 8) {
            const long r = rt * 128 + part * 32 + k;
            const int m = m0 + tx;
            const bool in = r < R && m < M;
            td[k][tx] = in ? D[r * M + m] : 0.0;
            const double y = in ? F[r * M + m] : 0.0, g = y * rf;
            tg[k][tx] = fma(fma(-g, fy, y), rf, g);
        }
        __syncthreads();
        for (int k = ty; k < 32; k += 8) {
            const long o = (rt * Mp + m0 + k) * 128 + part * 32 + tx;
            dt[o] = td[tx][k];
            gt[o] = tg[tx][k];
        }
        __syncthreads();
    }
}

// er[r], er[Rp + r]: exponents above the maxima over the modes of |x| 2^-ec and |g| 2^-ec
// (kZeroExp for a row of zeros)
__global__ void k_dg_rowexp(const double *__restrict__ dt, const double *__restrict__ gt,
                            const int *__restrict__ ec, int M, int Mp, int *__restrict__ er) {
    __shared__ int sh[8][128];
    const long rt = blockIdx.x;
    const int row = threadIdx.x, g = threadIdx.y, *e0 = ec + blockIdx.y * Mp;
    const double *a = (blockIdx.y ? gt : dt) + rt * Mp * 128 + row;
    int e = INT_MIN;
#pragma unroll 4
    for (int m = g; m < M; m += 8) {
        const double d = a[m * 128L];
        if (d != 0) e = max(e, exp_above(d) - e0[m]);
    }
    sh[g][row] = e;
    __syncthreads();
    if (g == 0) {
        for (int k = 1; k < 8; ++k) e = max(e, sh[k][row]);
        er[(blockIdx.y * (long)gridDim.x + rt) * 128 + row] = e == INT_MIN ? kZeroExp : e;
    }
}

// xa: thread = (row, eight modes); xb: thread = (mode, eight rows)
__global__ void __launch_bounds__(256) k_dg_xa(const double *__restrict__ D,
                                               const int *__restrict__ ec,
                                               const int *__restrict__ er, long R, int M, int nkb,
                                               __half *__restrict__ xa, float *__restrict__ nrm) {
    const long rt = blockIdx.x;
    const int kb = blockIdx.y, c = threadIdx.x & 7;
    uint8_t *out = reinterpret_cast<uint8_t *>(xa) + (rt * nkb + kb) * (long)kRes * kGA;
    for (int row = threadIdx.x >> 3; row < kGM; row += 32) {
        const long r = rt * kGM + row;
        long long q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int m = kb * kGK + c * 8 + k;
            const double d = (r < R && m < M) ? D[r * M + m] : 0.0;
            q[k] = fixed_point(d, m < M && r < R ? 55 - ec[m] - er[r] : 0);
        }
        uint4 w[kRes];
        digits8<kRes>(q, w);
#pragma unroll
        for (int d = 0; d < kRes; ++d)
            *reinterpret_cast<uint4 *>(out + d * kGA + sw_place(row, c)) = w[d];
        digit_norms(w, c, nrm + (rt * nkb + kb) * kRes * kGM, kGM, row);
    }
}

// The same from the column layout (g): thread = (row, eight modes)
__global__ void __launch_bounds__(256) k_dg_ga(const double *__restrict__ gt,
                                               const int *__restrict__ ec,
                                               const int *__restrict__ er, int M, int Mp, int nkb,
                                               __half *__restrict__ ga) {
    const long rt = blockIdx.x;
    const int kb = blockIdx.y, row = threadIdx.x & 127;
    uint8_t *out = reinterpret_cast<uint8_t *>(ga) + (rt * nkb + kb) * (long)kRes * kGA;
    for (int c = threadIdx.x >> 7; c < 8; c += 2) {
        long long q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int m = kb * kGK + c * 8 + k;
            q[k] = m < M ? fixed_point(gt[(rt * Mp + m) * 128 + row], 55 - ec[m] - er[rt * kGM + row]) : 0;
        }
        uint4 w[kRes];
        digits8<kRes>(q, w);
#pragma unroll
        for (int d = 0; d < kRes; ++d)
            *reinterpret_cast<uint4 *>(out + d * kGA + sw_place(row, c)) = w[d];
    }
}

__global__ void __launch_bounds__(256) k_dg_xb(const double *__restrict__ dt,
                                               const int *__restrict__ ec,
                                               const int *__restrict__ er, int Mp, long nkb,
                                               __half *__restrict__ xb, float *__restrict__ nrm) {
    const long kb = blockIdx.x;
    const int at = blockIdx.y, c = threadIdx.x & 7;
    uint8_t *out = reinterpret_cast<uint8_t *>(xb) + (at * nkb + kb) * kRes * (long)kGB;
    for (int row = threadIdx.x >> 3; row < kGN; row += 32) {
        const int a = at * kGN + row;
        const double *src = dt + ((kb >> 1) * Mp + a) * 128 + (kb & 1) * 64 + 8 * c;
        long long q[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const double2 v = dg_two(src + 2 * j);
            const int2 e = *reinterpret_cast<const int2 *>(er + kb * kGK + 8 * c + 2 * j);
            q[2 * j] = fixed_point(v.x, 55 - ec[a] - e.x);
            q[2 * j + 1] = fixed_point(v.y, 55 - ec[a] - e.y);
        }
        uint4 w[kRes];
        digits8<kRes>(q, w);
#pragma unroll
        for (int d = 0; d < kRes; ++d)
            *reinterpret_cast<uint4 *>(out + d * kGB + sw_place(row, c)) = w[d];
        digit_norms(w, c, nrm + (at * nkb + kb) * kRes * kGN, kGN, row);
    }
}

// ------------------------------------------------- once per call
// Where a call's Y1 and R1 come from: matrices, or psi unpacked on the way
// (Modules/DynamicalLanczos.py:2773-2948, :3009-3053, :3369-3430), so that no
// Y1 is written and read again.  Image i of a source starts i strides further on.
enum { DG_MATRIX = 0,     // symmetric as it is
       DG_AVERAGE,        // (Y1 + Y1^T) / 2
       DG_PSI,            // plain layout
       DG_PSI_T,          // transposed layout, per-pair factors ca, cb
       DG_PSI_WIGNER,     // ca a' - cb b'
       DG_STATIC };       // -2 Upsilon W Upsilon, Upsilon = ca
struct DgSource {
    int kind;
    const double *Y, *R;
    long ystride, rstride;
    const double *S;          // the vector of s, or null: f_Y R
    const double *ca, *cb;
    long H;
    int no_r;                 // R1 = 0
};
// images 0 .. n - 2 are sources 0 .. n - 2, the others follow source n - 1
struct DgSources {
    DgSource s[2];
    int n;
};

__device__ __forceinline__ double dg_y1(const DgSource &c, const double *__restrict__ Y, int M,
                                        int n, int m) {
    if (c.kind == DG_MATRIX) return Y[(long)n * M + m];
    if (c.kind == DG_AVERAGE)
        return n == m ? Y[(long)n * M + n] : 0.5 * (Y[(long)n * M + m] + Y[(long)m * M + n]);
    const int i = min(n, m), j = max(n, m);
    const long k = (long)i * M - (long)i * (i - 1) / 2 + (j - i);
    const double y = Y[M + k];
    if (c.kind == DG_PSI) return y;
    if (c.kind == DG_PSI_T) return y * c.ca[k] + Y[M + c.H + k] * c.cb[k];
    if (c.kind == DG_PSI_WIGNER) return c.ca[k] * y - c.cb[k] * Y[M + c.H + k];
    // both orders of the product, as the average of the matrix and its transpose
    const double a = -2 * ((y * c.ca[n]) * c.ca[m]), b = -2 * ((y * c.ca[m]) * c.ca[n]);
    return n == m ? a : 0.5 * (a + b);
}

// Row n of image blockIdx.y of Y1 (symmetric): digits of y 2^(eb - et) with et
// the exponent above the row's maximum, and the two vectors of the row scalars.
// Also clears the image's maxima of alpha, beta and the force weights.  With many
// images rows M and M + 1 are those two vectors, digits of rows `image` of the tiles vb.
// failed: the call's failure flag, cleared by its first pass (null in the others).
__global__ void __launch_bounds__(128) k_dg_y1(const DgSources src, const double *__restrict__ fY,
                                               const int *__restrict__ ecol, int M, int Mp,
                                               __half *__restrict__ yb, int *__restrict__ et,
                                               double *__restrict__ vs, double *__restrict__ vt,
                                               __half *__restrict__ vb, int *__restrict__ etv,
                                               unsigned long long *__restrict__ absmax,
                                               int *__restrict__ failed) {
    pdl_enter();
    extern __shared__ double yrow[];     // M
    __shared__ int sh[4];
    const int n = blockIdx.x, is = min((int)blockIdx.y, src.n - 1);
    const long img = blockIdx.y, rel = img - is;
    const DgSource &c = src.s[is];
    const double *Y = c.Y + rel * c.ystride;
    auto vec = [&](int m, bool of_s) {
        const double r = c.no_r ? 0.0 : c.R[rel * c.rstride + m];
        return of_s && c.S ? c.S[rel * c.rstride + m] : fY[m] * r;
    };
    const int v2 = n - M;             // 0, 1: s and t
    const int *ec = ecol + (v2 == 1 ? Mp : 0);
    int e = INT_MIN;
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        const double v = v2 >= 0 ? vec(m, v2 == 0) : dg_y1(c, Y, M, n, m);
        yrow[m] = v;
        if (v != 0) e = max(e, isfinite(v) ? exp_above(v) + ec[m] : kBadExp);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = e;
    __syncthreads();
    e = max(max(sh[0], sh[1]), max(sh[2], sh[3]));
    if (e == INT_MIN) e = 0;
    const bool bad = e >= kBadExp / 2;
    const int nkb = Mp / kGK, row = v2 >= 0 ? (int)img : n % kGN;
    uint8_t *out = v2 >= 0 ? reinterpret_cast<uint8_t *>(vb) + v2 * (long)nkb * kCall * kGB
                           : reinterpret_cast<uint8_t *>(yb) +
                                 (img * (Mp / kGN) + n / kGN) * nkb * (long)kCall * kGB;
    for (int ch = threadIdx.x; ch < Mp / 8; ch += blockDim.x) {
        const int kb = ch >> 3, c8 = ch & 7;
        long long q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int m = ch * 8 + k;
            q[k] = (m < M && !bad) ? fixed_point(yrow[m], 62 + ec[m] - e) : 0;
        }
        uint4 w[kCall];
        digits8<kCall>(q, w);
#pragma unroll
        for (int d = 0; d < kCall; ++d)
            *reinterpret_cast<uint4 *>(out + (kb * (long)kCall + d) * kGB + sw_place(row, c8)) = w[d];
    }
    if (threadIdx.x == 0 && v2 >= 0) {
        etv[v2 * kGN + img] = e;
    } else if (threadIdx.x == 0) {
        et[img * Mp + n] = e;
        vs[img * Mp + n] = vec(n, true);
        vt[img * Mp + n] = vec(n, false);
        if (n == 0)
            for (int k = 0; k < 4; ++k) absmax[4 * img + k] = 0ULL;
        if (n == 0 && img == 0 && failed) *failed = 0;
    }
}

// Row scalars of the image blockIdx.y from the stage A partials (s and t of many images
// from st, [2 Rp][images]), those of W times the row's scale of x, which the row of xb
// does without; max |alpha| and max |beta / 2| with the scales of g's and x's row, and with
// many images the same of the force weights.  Rows past the end get zeros.
template <bool kMany>
__global__ void __launch_bounds__(128) k_dg_rows(const double *__restrict__ qp,
                                                 const double *__restrict__ st, int nct, long R,
                                                 long Rp, int rho_div,
                                                 const double *__restrict__ rho,
                                                 const int *__restrict__ er,
                                                 const int *__restrict__ erg, int apply_d4,
                                                 double *__restrict__ abcc,
                                                 unsigned long long *__restrict__ absmax) {
    pdl_enter();
    constexpr int kMax = kMany ? 4 : 2;
    __shared__ unsigned long long red[kMax][4];
    const long img = blockIdx.y, r = blockIdx.x * 128L + threadIdx.x;
    double w[4] = {0, 0, 0, 0}, top[4] = {0, 0, 0, 0};
    if (r < R) {
        double q = 0, p = 0, s = 0, t = 0;
        const double *o = qp + img * nct * 4 * R + r;
        for (int ct = 0; ct < nct; ++ct, o += 4 * R) {
            q += o[0];
            p += o[R];
            if (!kMany) {
                s += o[2 * R];
                t += o[3 * R];
            }
        }
        if (kMany) {
            s = st[r * gridDim.y + img];
            t = st[(Rp + r) * gridDim.y + img];
        }
        const double f = pow2(er[r]), fg = pow2(erg[r]), rw = rho[r / rho_div];
        q *= f;
        p *= f;
        // rho / 3 by the reciprocal and one residual step: a warp's float64 operation
        // takes 64 cycles, a division ten of them
        constexpr double third = 1.0 / 3.0;
        const double y = rw * third, t3 = fma(fma(-y, 3.0, rw), third, y), h3 = 0.5 * t3,
                     t8 = apply_d4 ? 0.125 * rw : 0.0;
        w[0] = fma(s, t3, -q * t8) * f;       // rho (s / 3 - q / 8)
        w[1] = fma(t, h3, -p * t8) * f;       // rho (t / 3 - p / 4) / 2
        w[2] = -q * h3;
        w[3] = -p * t3;
        top[0] = w[0] * fg;
        top[1] = w[1] * f;
        if (kMany) {
            w[2] = top[2] = w[2] * fg;
            w[3] = top[3] = w[3] * f;
        }
    }
    if (r < Rp) {
        double *o = abcc + 4 * img * Rp + r;
        o[0] = w[0];
        o[Rp] = w[1];
        o[2 * Rp] = w[2];
        o[3 * Rp] = w[3];
    }
#pragma unroll
    for (int k = 0; k < kMax; ++k) {
        unsigned long long a = (unsigned long long)__double_as_longlong(top[k]) & 0x7fffffffffffffffULL;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a = max(a, __shfl_xor_sync(0xffffffffu, a, o));
        if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = a;
    }
    __syncthreads();
    if (threadIdx.x < kMax) {
        unsigned long long a = red[threadIdx.x][0];
        for (int k = 1; k < 4; ++k) a = max(a, red[threadIdx.x][k]);
        atomicMax(absmax + 4 * img + threadIdx.x, a);
    }
}

// Exponent above |w| of a mode of an image, kBadExp where that is not finite: am, the
// image's maxima of the rows' weights with their scales, times the scales of the mode in
// g and x (an element is below its row's and its column's scale).  Whole numbers only: every
// row of a W block asks for it (24 vectors at M=60, N=5000: 248 us with four float64
// operations each, 237 so).
__device__ __forceinline__ int dg_wexp(const unsigned long long *__restrict__ am, int ex, int eg) {
    constexpr unsigned long long kInf = 0x7ff0000000000000ULL;
    const unsigned long long a = am[0], b = am[1];
    if (a >= kInf || b >= kInf) return kBadExp;
    if (!(a | b)) return 0;
    const int ea = a ? exp_above(__longlong_as_double((long long)a)) + eg : INT_MIN,
              eb = b ? exp_above(__longlong_as_double((long long)b)) + ex : INT_MIN;
    return max(ea, eb) + 1;             // of the sum of both
}

// Digits of eight numbers as row `row` of the A block blk, chunk c
__device__ __forceinline__ void dg_put(const long long (&q)[8], uint8_t *blk, int row, int c) {
    uint4 w[kCall];
    digits8<kCall>(q, w);
    blk += sw_place(row, c);
#pragma unroll
    for (int d = 0; d < kCall; ++d) *reinterpret_cast<uint4 *>(blk + d * kGA) = w[d];
}

// W digits: block = (group of K blocks, tile of 128 rows (image, mode)); thread
// = (mode, eight rows of the ensemble) for 32 modes at a time, so that a warp
// writes whole 128-byte rows of every digit.  The force partials
// fpart[(img nfc + group) M + b] ride along.
__global__ void __launch_bounds__(256) k_dg_wbuild(
    const double *__restrict__ dt, const double *__restrict__ gt,
    const double *__restrict__ abcc, const unsigned long long *__restrict__ absmax,
    const int *__restrict__ eb, const double *__restrict__ fY, int M, int Mp, long Rp, int nimg,
    long nkb, int per,
    __half *__restrict__ wa, int *__restrict__ ew, double *__restrict__ fpart) {
    pdl_enter();
    const int c = threadIdx.x & 7;
    const long wt = blockIdx.y, kb0 = blockIdx.x * (long)per, kb1 = min(nkb, kb0 + per);
    uint8_t *out = reinterpret_cast<uint8_t *>(wa) + wt * nkb * kCall * (long)kGA;
    for (int row = blockIdx.z * 32 + (threadIdx.x >> 3); row < kGM; row += 32 * gridDim.z) {
        const long grow = wt * kGM + row;
        const int img = (int)(grow / Mp), b = (int)(grow % Mp);
        // (the eight lanes of a mode take the same branch; padding rows of wa
        // are zero from the start)
        const bool live = img < nimg && b < M;
        double f1 = 0, f2 = 0;
        if (live) {
            const int e = dg_wexp(absmax + 4 * img, eb[b], eb[Mp + b]);
            const bool bad = e == kBadExp;
            const int K = 62 - e;
            if (blockIdx.x == 0 && c == 0) ew[grow] = e;
            for (long kb = kb0; kb < kb1; ++kb) {
                const long o = ((kb >> 1) * Mp + b) * 128 + (kb & 1) * 64 + 8 * c;
                const double *pa = abcc + 4L * img * Rp + kb * kGK + 8 * c;
                long long q[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const double2 d = dg_two(dt + o + 2 * j), g = dg_two(gt + o + 2 * j);
                    const double *pr = pa + 2 * j;
                    const double2 sa = dg_two(pr), sb = dg_two(pr + Rp), c1 = dg_two(pr + 2 * Rp),
                                  c2 = dg_two(pr + 3 * Rp);
                    const double w0 = fma(sa.x, g.x, sb.x * d.x),
                                 w1 = fma(sa.y, g.y, sb.y * d.y);
                    q[2 * j] = bad ? 0 : fixed_point(w0, K);
                    q[2 * j + 1] = bad ? 0 : fixed_point(w1, K);
                    f1 = fma(c1.x, g.x, f1);
                    f2 = fma(c2.x, d.x, f2);
                    f1 = fma(c1.y, g.y, f1);
                    f2 = fma(c2.y, d.y, f2);
                }
                dg_put(q, out + kb * kCall * (long)kGA, row, c);
            }
        }
        double facc = f1 + f2;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) facc += __shfl_xor_sync(0xffffffffu, facc, o);
        if (live && c == 0) fpart[((long)img * gridDim.x + blockIdx.x) * M + b] = facc * fY[b];
    }
}

// The same for many images: block = (K block, 32 modes, kWImages images); x and g of a
// thread's rows stay in registers while the images go by.  The forces are products of
// their own with the rows that the blocks blockIdx.y == modes / 32 build in wf: digits
// of the weights of x (rows 0 .. 63: images) and of g (rows 64 .. 127); as two float64
// products an element they were half of this kernel's work.  M=189, N=10000, 48 images:
// 781 us with the forces and every image its own pass over x and g, 364 so.
constexpr int kWImages = 8;
__global__ void __launch_bounds__(256) k_dg_wimages(
    const double *__restrict__ dt, const double *__restrict__ gt,
    const double *__restrict__ abcc, const unsigned long long *__restrict__ absmax,
    const int *__restrict__ eb, int M, int Mp, long Rp, int nimg, long nkb,
    __half *__restrict__ wa, int *__restrict__ ew,
    __half *__restrict__ wf, int *__restrict__ ewf) {
    pdl_enter();
    const int c = threadIdx.x & 7, slot = threadIdx.x >> 3, i0 = blockIdx.z * kWImages,
              i1 = min(nimg, i0 + kWImages);
    const long kb = blockIdx.x;
    if (blockIdx.y == gridDim.y - 1) {
        // (an image in both halves of the tile)
        const int img = i0 + slot / 2, row = img + (slot & 1 ? 64 : 0), k = slot & 1 ? 2 : 3;
        if (img >= i1) return;
        const double top = __longlong_as_double((long long)absmax[4 * img + k]);
        const int e = !isfinite(top) ? kBadExp : top > 0 ? exp_above(top) : 0;
        if (kb == 0 && c == 0) ewf[row] = e;
        const double *src = abcc + (4L * img + k) * Rp + kb * kGK + 8 * c;
        long long q[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const double2 v = dg_two(src + 2 * j);
            q[2 * j] = e == kBadExp ? 0 : fixed_point(v.x, 62 - e);
            q[2 * j + 1] = e == kBadExp ? 0 : fixed_point(v.y, 62 - e);
        }
        dg_put(q, reinterpret_cast<uint8_t *>(wf) + kb * kCall * (long)kGA, row, c);
        return;
    }
    __shared__ int sexp[kWImages][32];
    const int b0 = blockIdx.y * 32, b = b0 + slot;
    for (int t = threadIdx.x; t < (i1 - i0) * 32; t += blockDim.x) {
        const int img = i0 + (t >> 5), m = b0 + (t & 31);
        int e = 0;
        if (m < M)
            e = dg_wexp(absmax + 4 * img, eb[m], eb[Mp + m]);
        sexp[t >> 5][t & 31] = e;
        if (kb == 0 && m < M) ew[(long)img * Mp + m] = e;
    }
    __syncthreads();
    if (b >= M) return;
    const long o = ((kb >> 1) * Mp + b) * 128 + (kb & 1) * 64 + 8 * c;
    double2 d[4], g[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        d[j] = dg_two(dt + o + 2 * j);
        g[j] = dg_two(gt + o + 2 * j);
    }
#pragma unroll 1
    for (int img = i0; img < i1; ++img) {
        const int e = sexp[img - i0][slot];
        const double *pa = abcc + 4L * img * Rp + kb * kGK + 8 * c;
        long long q[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const double2 sa = dg_two(pa + 2 * j), sb = dg_two(pa + Rp + 2 * j);
            const double w0 = fma(sa.x, g[j].x, sb.x * d[j].x), w1 = fma(sa.y, g[j].y, sb.y * d[j].y);
            q[2 * j] = e == kBadExp ? 0 : fixed_point(w0, 62 - e);
            q[2 * j + 1] = e == kBadExp ? 0 : fixed_point(w1, 62 - e);
        }
        const long grow = (long)img * Mp + b;
        dg_put(q, reinterpret_cast<uint8_t *>(wa) + ((grow >> 7) * nkb + kb) * kCall * (long)kGA,
               (int)(grow & 127), c);
    }
}

// fpart[img][m] from the products gf[split][128][2 Mp] of the force weights' rows with
// [x | g]
__global__ void __launch_bounds__(128) k_dg_force(const double *__restrict__ gf, int ns, int M, int Mp,
                                                  const double *__restrict__ fY,
                                                  double *__restrict__ fpart) {
    pdl_enter();
    const int m = blockIdx.x * 128 + threadIdx.x, img = blockIdx.y;
    if (m >= M) return;
    const double *p = gf + (long)img * 2 * Mp + m, *q = p + (long)64 * 2 * Mp + Mp;
    double a = 0;
#pragma unroll 4
    for (int s = 0; s < ns; ++s, p += (long)kGM * 2 * Mp, q += (long)kGM * 2 * Mp) a += *p + *q;
    fpart[(long)img * M + m] = a * fY[m];
}

// sum_s p[s * stride] in split order, eight loads in flight
__device__ __forceinline__ double dg_split_sum(const double *__restrict__ p, int n, long stride) {
    double acc = 0;
    int s = 0;
    for (; s + 8 <= n; s += 8) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = p[(s + u) * stride];
#pragma unroll
        for (int u = 0; u < 8; ++u) acc += v[u];
    }
    for (; s < n; ++s) acc += p[s * stride];
    return acc;
}

// d2v = -f_Y,a f_Y,b (H + H^T) / norm and f = sum fpart / norm of the image blockIdx.y (no
// symmetry images): one block per 8-row slab of a pair (A, B), A <= B, of
// 32 x 32 tiles, each element summed over the splits once.  kRows = 2 and four groups
// of threads, each with every fourth split, where slabs of 8 rows would leave SMs idle:
// an addition takes a warp 64 cycles and the loads wait for one another (32 splits of
// M=48: 11.4 us with the slabs of 8, 6.9 so).  After a wait that gave up the results are
// NaN: calls on device pointers report it that way (and in tdscha_ctx_sync).
template <int kRows, int kGroups>
__global__ void __launch_bounds__(32 * kRows * kGroups) k_dg_final(
    const double *__restrict__ gpart, int nsplit, long stride, int M, int Mp,
    const double *__restrict__ fpart, int nfc, const double *__restrict__ fY, double inv,
    const int *__restrict__ failed, double *__restrict__ f, double *__restrict__ d2v) {
    pdl_enter();
    gpart += blockIdx.y * (long)Mp * Mp;
    fpart += blockIdx.y * (long)nfc * M;
    f += blockIdx.y * (long)M;
    d2v += blockIdx.y * (long)M * M;
    constexpr int kSlabs = 32 / kRows;
    constexpr int kThreads = 32 * kRows;
    const double kNaN = __longlong_as_double(0x7ff8000000000000LL);
    __shared__ double tr[kGroups][32][kRows + 1], red[kGroups][kRows][33];
    const int nt = (M + 31) / 32, slab = blockIdx.x % kSlabs;
    const int group = threadIdx.x / kThreads, t = threadIdx.x % kThreads;
    int A = 0, rem = blockIdx.x / kSlabs;
    while (rem >= nt - A) {
        rem -= nt - A;
        ++A;
    }
    const int B = A + rem, a0 = A * 32 + slab * kRows, b0 = B * 32;
    const int tx = t & 31, ty = t >> 5;
    const int mine = (nsplit - group + kGroups - 1) / kGroups;
    gpart += group * stride;
    {
        const int ao = t % kRows, bo = t / kRows;
        const int b = b0 + bo, a = a0 + ao;
        tr[group][bo][ao] =
            (a < M && b < M) ? dg_split_sum(gpart + (long)b * Mp + a, mine, kGroups * stride) : 0.0;
    }
    const int a = a0 + ty, b = b0 + tx;
    const bool in = a < M && b < M;
    double h = in ? dg_split_sum(gpart + (long)a * Mp + b, mine, kGroups * stride) : 0.0;
    if (kGroups > 1) red[group][ty][tx] = h;
    __syncthreads();
    if (group == 0 && in) {
        for (int k = 1; k < kGroups; ++k) h += red[k][ty][tx];
        for (int k = 0; k < kGroups; ++k) h += tr[k][tx][ty];
        // (the flag beside these: read ahead of the sums it made them 10 us longer at M=24,
        // N=50000, and 3 us between them and here)
        const bool bad = *failed;
        double v = -(h * fY[a]) * fY[b] * inv;
        if (bad) v = kNaN;
        d2v[(long)a * M + b] = v;
        if (A != B) d2v[(long)b * M + a] = v;
    }
    if (A == 0 && slab == 0) {
        const int e = b0 + tx;
        double acc = 0;
        if (e < M)
            for (int ch = group * kRows + ty; ch < nfc; ch += kGroups * kRows) acc += fpart[(long)ch * M + e];
        __syncthreads();
        red[group][ty][tx] = acc;
        __syncthreads();
        if (threadIdx.x < 32 && e < M) {
            acc = 0;
            for (int k = 0; k < kGroups * kRows; ++k) acc += red[k / kRows][k % kRows][tx];
            f[e] = *failed ? kNaN : acc * inv;
        }
    }
}

// ------------------------------------------------------------- host side
struct DigitStore {
    int Mp = 0, nkbM = 0, nct = 0, nsm = 1;
    long Rp = 0, nkbR = 0;
    int cap = 1;                 // images that the per-call buffers hold
    int per = 1, nfc = 1;        // K blocks of one W block, force partials an image
    // s, t and the forces as digit products of their own (many symmetry images): g's
    // digits behind x's in xa and xb.  (Its exponents are always behind x's in er and ec.)
    bool many = false;
    int kbF = 1, nsF = 1;
    double *st = nullptr, *gf = nullptr;
    __half *vb = nullptr, *wf = nullptr;
    int *etv = nullptr, *ewf = nullptr, *bmap = nullptr;
    int flushA = kFlushMin, flushB = kFlushMin;   // K blocks per accumulation of the stages
    void *slab = nullptr;
    double *dt = nullptr, *gt = nullptr, *vs = nullptr, *vt = nullptr, *qp = nullptr,
           *gpart = nullptr, *fpart = nullptr, *fo = nullptr, *d2vo = nullptr;
    double *abcc = nullptr;
    unsigned long long *absmax = nullptr;
    __half *xa = nullptr, *xb = nullptr, *yb = nullptr, *wa = nullptr;
    int *ec = nullptr, *eb = nullptr, *er = nullptr, *et = nullptr, *ew = nullptr;
    int *err = nullptr;          // bounded-wait failure code (pinned host memory)
    int *failed = nullptr;       // whether one gave up in this call
    long long budget = kDefaultBudget;
};

void digits_release(tdscha_ctx *c) {
    if (!c->dg) return;
    cached_free(c->dg->slab);
    delete c->dg;
    c->dg = nullptr;
}

// Builds the digit operands of the context's rows D, F.  Leaves c->dg null (the
// float64 kernels of perturb_fp64.cu serve the context) where the buffers
// would not fit beside the caller's own, or with TDSCHA_FP64_DIGITS=0.
int digits_prepare(tdscha_ctx *c) {
    if (const char *e = getenv("TDSCHA_FP64_DIGITS"))
        if (atoi(e) == 0) return TDSCHA_OK;
    const int M = c->M;
    const long R = c->Nrows;
    if (sizeof(double) * M > 200 * 1024) return TDSCHA_OK;   // k_dg_y1 keeps a row on chip
    DigitStore *x = new DigitStore();
    x->Mp = ceil_div(M, kGN) * kGN;
    x->nkbM = x->nct = x->Mp / kGK;
    const long nrt = (R + kGM - 1) / kGM;
    x->Rp = nrt * kGM;
    x->nkbR = x->Rp / kGK;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&x->nsm, cudaDevAttrMultiProcessorCount, dev);
    x->nsm = std::max(1, x->nsm);
    if (const char *b = getenv("TDSCHA_WAIT_BUDGET_CYCLES")) x->budget = atoll(b);
    const int Mp = x->Mp;
    const size_t elems = (size_t)Mp * x->Rp;
    // Images of one pass: the context's symmetry images within 6 GB of W digits; or,
    // without images, perturbations given together (the two of a bi-Lanczos step,
    // static vectors), two within 6 GB and up to 32 within 256 MB.
    const size_t per_img = elems * 2 * kCall;
    const size_t most = std::max<size_t>(1, (size_t(6) << 30) / per_img);
    if (c->J > 1)
        x->cap = (int)std::min<size_t>(std::min(c->J, 64), most);
    else
        x->cap = (int)std::max(std::min<size_t>(2, most),
                               std::min<size_t>(32, (size_t(256) << 20) / per_img));
    const int cap = x->cap, nat = ceil_div((long)cap * Mp, kGM);
    // From 8 images on (one tile of 64 takes them, 128 rows the forces' weights), where
    // the four float64 products an element that it saves, 6.2 us a million, are worth
    // three more launches: M=60, N=300, 48 images (0.9 million) 153 us with it and 119
    // without; M=189, N=10000, 48 images (92 million) 2106 and 2632.
    x->many = cap >= 8 && c->J > 1 && (double)cap * M * R >= 4e6;
    x->kbF = dg_blocks_per_split(x->nkbR, kFlushMin, 1, 2 * x->nct, x->nsm);
    x->nsF = ceil_div(x->nkbR, x->kbF);
    const size_t two = x->many ? 2 : 1, one = x->many ? 1 : 0;
    // about eight W blocks per SM, at most 16 K blocks each
    x->per = (int)std::max<long>(1, std::min<long>(16, x->nkbR * nat / (152L * 8)));
    x->nfc = ceil_div(x->nkbR, x->per);
    size_t gbytes = 0;
    for (x->flushB = kFlushMax; ; --x->flushB) {      // ends at kFlushMin, its value until measured
        for (int n = 1; n <= cap; ++n) {
            const int na = ceil_div((long)n * Mp, kGM), kb = dg_blocks_per_split(x->nkbR, x->flushB, na, x->nct, x->nsm);
            gbytes = std::max(gbytes, (size_t)ceil_div(x->nkbR, kb) * na * kGM * Mp * sizeof(double));
        }
        if (x->flushB == kFlushMin) break;
    }
    float *fl = nullptr;         // largest digit norms of xa and of xb
    struct Part {
        void **p;
        size_t bytes;
        bool zero;
    };
    const size_t d = sizeof(double), i4 = sizeof(int), u8 = sizeof(unsigned long long);
    std::vector<Part> parts = {
        {(void **)&x->dt, d * elems, false},
        {(void **)&x->gt, d * elems, false},
        {(void **)&x->xa, two * 2 * kRes * elems, false},
        {(void **)&x->xb, two * 2 * kRes * elems, false},
        {(void **)&x->er, 2 * i4 * x->Rp, false},
        {(void **)&x->st, one * d * 2 * cap * x->Rp, false},
        {(void **)&x->gf, one * d * x->nsF * kGM * 2 * Mp, false},
        {(void **)&x->bmap, one * i4 * 2 * nrt, false},
        // (the column parts of small tiles are at most as many as there are SMs)
        {(void **)&x->qp, d * 4 * std::max((size_t)x->nct * cap, (size_t)(x->nsm / nrt)) * R, false},
        {(void **)&x->abcc, d * 4 * (size_t)cap * x->Rp, false},
        {(void **)&x->failed, i4, false},
        {(void **)&x->gpart, gbytes, false},
        {(void **)&x->fpart, d * (size_t)cap * x->nfc * M, false},
        {(void **)&x->fo, c->J == 1 ? d * cap * M : 0, false},
        {(void **)&x->d2vo, c->J == 1 ? d * (size_t)cap * M * M : 0, false},
        {(void **)&x->ec, 2 * i4 * Mp, false},
        {(void **)&x->eb, 2 * i4 * Mp, false},
        // zero from the start: maxima, and the rows of padding modes
        {(void **)&x->absmax, u8 * 4 * cap, true},
        {(void **)&x->etv, one * i4 * 2 * kGN, true},
        {(void **)&x->ewf, one * i4 * kGM, true},
        {(void **)&x->vb, one * 2 * (size_t)x->nkbM * kCall * kGB, true},
        {(void **)&x->wf, one * (size_t)x->nkbR * kCall * kGA, true},
        {(void **)&x->vs, d * cap * Mp, true},
        {(void **)&x->vt, d * cap * Mp, true},
        {(void **)&x->et, i4 * cap * Mp, true},
        {(void **)&x->ew, i4 * (size_t)nat * kGM, true},
        {(void **)&fl, sizeof(float) * 2 * kFlushes * kRes, true},
        {(void **)&x->yb, 2 * kCall * (size_t)cap * Mp * Mp, true},
        {(void **)&x->wa, 2 * kCall * (size_t)nat * kGM * x->Rp, true},
    };
    size_t total = 0, zero0 = 0;
    for (auto &p : parts) {
        if (p.zero && !zero0) zero0 = total;
        total += (p.bytes + 1023) & ~size_t(1023);
    }
    if (!memory_to_spare(total) || cached_malloc(&x->slab, total) != cudaSuccess) {
        cudaGetLastError();
        delete x;
        return TDSCHA_OK;
    }
    c->dg = x;
    uint8_t *at = reinterpret_cast<uint8_t *>(x->slab);
    for (auto &p : parts) {
        *p.p = at;
        at += (p.bytes + 1023) & ~size_t(1023);
    }
    x->err = reinterpret_cast<int *>(c->host_pinned);
    *x->err = 0;
    TDS_CUDA(cudaMemsetAsync((uint8_t *)x->slab + zero0, 0, total - zero0, 0));
    // rows a block walks one after the other: 8 in a small ensemble, 128 in a large one, more
    // where the grid's second dimension (65535) would not hold the blocks
    const long walk = std::max<long>(std::min<long>(128, std::max<long>(8, R / 400)),
                                     (R + 65534) / 65535);
    int *ecg = x->ec + Mp, *erg = x->er + x->Rp;
    TDS_CUDA(cudaMemsetAsync(x->ec, kNone & 0xff, i4 * 2 * Mp, 0));
    k_dg_colexp<<<dim3(ceil_div(M, 128), ceil_div(R, walk), 2), 128>>>(
        c->D, c->F, c->rho, c->rho_div, c->rho_top, R, M, Mp, walk, x->ec);
    TDS_CHECK_LAUNCH();
    k_dg_colend<<<ceil_div(2 * Mp, 128), 128>>>(c->fY, M, Mp, x->ec, x->eb);
    TDS_CHECK_LAUNCH();
    k_dg_cols<<<dim3((unsigned)nrt, Mp / 32), dim3(32, 8)>>>(c->D, c->F, c->fY, R, M, Mp, x->dt,
                                                              x->gt);
    TDS_CHECK_LAUNCH();
    k_dg_rowexp<<<dim3((unsigned)nrt, 2), dim3(128, 8)>>>(x->dt, x->gt, x->ec, M, Mp, x->er);
    TDS_CHECK_LAUNCH();
    // the digit norms pass through the W digits' space, which is zeroed again
    float *nrm = reinterpret_cast<float *>(x->wa);
    k_dg_xa<<<dim3((unsigned)nrt, x->nkbM), 256>>>(c->D, x->ec, x->er, R, M, x->nkbM, x->xa, nrm);
    TDS_CHECK_LAUNCH();
    TDS_CUDA(dg_windows(nrm, (int)nrt, kGM, x->nkbM, fl, 0));
    k_dg_xb<<<dim3((unsigned)x->nkbR, x->nct), 256>>>(x->dt, x->ec, x->er, Mp, x->nkbR, x->xb, nrm);
    TDS_CHECK_LAUNCH();
    TDS_CUDA(dg_windows(nrm, x->nct, kGN, (int)x->nkbR, fl + kFlushes * kRes, 0));
    if (x->many) {
        __half *ga = x->xa + kRes * elems, *gb = x->xb + kRes * elems;
        k_dg_ga<<<dim3((unsigned)nrt, x->nkbM), 256>>>(x->gt, ecg, erg, M, Mp, x->nkbM, ga);
        TDS_CHECK_LAUNCH();
        k_dg_xb<<<dim3((unsigned)x->nkbR, x->nct), 256>>>(x->gt, ecg, erg, Mp, x->nkbR, gb, nrm);
        TDS_CHECK_LAUNCH();
        std::vector<int> bm(2 * nrt, 0);
        std::fill(bm.begin() + nrt, bm.end(), 1);
        TDS_CUDA(cudaMemcpy(x->bmap, bm.data(), i4 * 2 * nrt, cudaMemcpyHostToDevice));
        TDS_CUDA((dg_setup<DG_STORE, false>()));
    }
    TDS_CUDA(cudaMemsetAsync(nrm, 0, sizeof(float) * kRes * (elems / kGK), 0));
    float h_fl[2 * kFlushes * kRes];
    TDS_CUDA(cudaMemcpy(h_fl, fl, sizeof(h_fl), cudaMemcpyDeviceToHost));
    x->flushA = digits_flush(h_fl);
    x->flushB = digits_flush(h_fl + kFlushes * kRes);
    TDS_CUDA(cudaFuncSetAttribute(k_dg_y1, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    TDS_CUDA((dg_setup<DG_DOTS, false>()));
    TDS_CUDA((dg_setup<DG_DOTS, true>()));
    TDS_CUDA((dg_setup<DG_PARTS, false>()));
    TDS_CUDA((dg_setup<DG_PARTS, true>()));
    return TDSCHA_OK;
}

// Outside of stream captures, where nothing may be allocated (a call in one takes the CUDA
// cores and leaves the digits to a later call)
int digits_first_use(tdscha_ctx *c, cudaStream_t st) {
    if (!c->dg_pending) return TDSCHA_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    TDS_CUDA(cudaStreamIsCapturing(st, &cap));
    if (cap != cudaStreamCaptureStatusNone) return TDSCHA_OK;
    c->dg_pending = false;
    return digits_prepare(c);
}

int digits_check_error(tdscha_ctx *c) {
    if (!c->dg || !*(volatile int *)c->dg->err) return TDSCHA_OK;
    const int v = *(volatile int *)c->dg->err;
    *(volatile int *)c->dg->err = 0;
    set_error("tensor-core pipeline: a bounded wait expired (code %d)", v);
    return TDSCHA_ERR_TIMEOUT;
}

// Stages A and B for nimg perturbations: split-K partials of every image's H in
// x->gpart, force partials in x->fpart.  first: the call's first pass.
static int digits_contract(tdscha_ctx *c, int nimg, const DgSources &src, int apply_d4,
                           bool first, int *nsplit, cudaStream_t st) {
    DigitStore *x = c->dg;
    const int M = c->M, Mp = x->Mp;
    const long R = c->Nrows;
    {
        ProfScope ps(c, 5, st);
        TDS_CUDA(launch_pdl(k_dg_y1, dim3(x->many ? M + 2 : M, nimg), 128, sizeof(double) * M, st,
                            src, (const double *)c->fY, (const int *)x->eb, M, Mp, x->yb, x->et,
                            x->vs, x->vt, x->vb, x->etv, x->absmax, first ? x->failed : nullptr));
        if (x->many) {
            // s and t of all images: [x; g] times their vectors
            DgArgs g{};
            g.a = x->xa;
            g.b = x->vb;
            g.nkb = g.kbps = x->nkbM;
            g.flush = kFlushMin;
            g.nat = (int)(2 * x->Rp / kGM);
            g.nbt = 1;
            g.nitems = g.nat;
            g.bmap = x->bmap;
            g.err = x->err;
            g.failed = x->failed;
            g.budget = x->budget;
            g.et = x->etv;
            g.er = x->er;
            g.R = 2 * x->Rp;
            g.M = nimg;
            g.out = x->st;
            TDS_CUDA((dg_launch<DG_STORE, false>(g, x->nsm, st)));
        }
    }
    DgArgs ga{};
    ga.a = x->xa;
    ga.b = x->yb;
    ga.nkb = ga.kbps = x->nkbM;
    ga.flush = x->flushA;
    ga.kk = ceil_div(M, 16);             // (read where M <= 64)
    // At most 64 modes: where that leaves SMs, two or four work items end a tile, each a
    // part of its columns (and do all of its products): with one, 16 row tiles at M=48
    // spend 16 000 cycles on the float64 operations of the row dots: 23.3 us at M=48,
    // N=2000, 13.0 so.
    int win = 1;
    ga.hc = M <= 32 ? 8 : 16;
    while (M <= kGN && ga.hc > 4 && 2 * ga.hc < M && 2 * win * nimg * (x->Rp / kGM) <= x->nsm) {
        win *= 2;
        ga.hc /= 2;
    }
    if (win == 1) ga.hc = dg_part_cols(M);
    ga.win = win;
    ga.abytes = kGA;
    ga.nat = (int)(x->Rp / kGM);
    ga.nbt = nimg * x->nct * win;
    ga.nitems = (long)ga.nat * ga.nbt;
    ga.Mp = Mp;
    ga.err = x->err;
    ga.failed = x->failed;
    ga.budget = x->budget;
    ga.dt = x->dt;
    ga.gt = x->gt;
    ga.vs = x->many ? nullptr : x->vs;
    ga.vt = x->vt;
    ga.et = x->et;
    ga.qp = x->qp;
    ga.R = R;
    ga.nct = x->nct;
    ga.M = M;
    {
        ProfScope ps(c, 0, st);
        TDS_CUDA((M <= kGK ? dg_launch<DG_DOTS, true>(ga, x->nsm, st)
                           : dg_launch<DG_DOTS, false>(ga, x->nsm, st)));
    }
    {
        ProfScope ps(c, 1, st);
        TDS_CUDA(launch_pdl(x->many ? k_dg_rows<true> : k_dg_rows<false>, dim3((unsigned)(x->Rp / 128), nimg), 128, 0, st,
                            (const double *)x->qp, (const double *)x->st,
                            x->nct * win, R, x->Rp, c->rho_div,
                            (const double *)c->rho, (const int *)x->er,
                            (const int *)x->er + x->Rp, apply_d4, x->abcc, x->absmax));
    }
    const int nat = ceil_div((long)nimg * Mp, kGM);
    {
        ProfScope ps(c, 2, st);
        if (x->many)
            TDS_CUDA(launch_pdl(k_dg_wimages, dim3(x->nkbR, Mp / 32 + 1, ceil_div(nimg, kWImages)), 256,
                                0, st, (const double *)x->dt, (const double *)x->gt,
                                (const double *)x->abcc, (const unsigned long long *)x->absmax,
                                (const int *)x->eb, M, Mp, x->Rp, nimg, x->nkbR,
                                x->wa, x->ew, x->wf, x->ewf));
        else
            // (few blocks: a group of 32 modes each)
            TDS_CUDA(launch_pdl(k_dg_wbuild, dim3(x->nfc, nat, x->nfc * nat <= 2 * x->nsm ? 4 : 1),
                                256, 0, st, (const double *)x->dt,
                                (const double *)x->gt, (const double *)x->abcc,
                                (const unsigned long long *)x->absmax,
                                (const int *)x->eb, (const double *)c->fY, M, Mp, x->Rp, nimg,
                                x->nkbR, x->per, x->wa, x->ew, x->fpart));
    }
    DgArgs gb{};
    gb.a = x->wa;
    gb.b = x->xb;
    gb.nkb = (int)x->nkbR;
    gb.kbps = dg_blocks_per_split(x->nkbR, x->flushB, nat, x->nct, x->nsm);
    gb.flush = x->flushB;
    gb.kk = kGK / 16;
    gb.hc = dg_part_cols(M);
    gb.win = 1;
    gb.abytes = kGA;
    gb.nat = nat;
    gb.nbt = x->nct;
    *nsplit = ceil_div(x->nkbR, gb.kbps);
    gb.nitems = (long)nat * x->nct * *nsplit;
    gb.Mp = Mp;
    gb.err = x->err;
    gb.failed = x->failed;
    gb.budget = x->budget;
    gb.ec = x->ec;
    gb.ew = x->ew;
    gb.gpart = x->gpart;
    gb.M = M;
    gb.rmod = Mp;
    gb.rlive = M;
    gb.rows_b = (long)nimg * Mp;
    ProfScope ps(c, 3, st);
    TDS_CUDA((M <= 32 ? dg_launch<DG_PARTS, true>(gb, x->nsm, st)
                      : dg_launch<DG_PARTS, false>(gb, x->nsm, st)));
    if (x->many) {
        // the forces: the weights' rows times [x | g]
        DgArgs g = gb;
        g.a = x->wf;
        g.kbps = x->kbF;
        g.flush = kFlushMin;
        g.nat = 1;
        g.nbt = 2 * x->nct;
        g.nitems = (long)g.nbt * x->nsF;
        g.Mp = g.M = 2 * Mp;
        g.ew = x->ewf;
        g.gpart = x->gf;
        g.rmod = kGM;
        g.rlive = kGM;
        g.rows_b = kGM;
        TDS_CUDA((dg_launch<DG_PARTS, false>(g, x->nsm, st)));
        TDS_CUDA(launch_pdl(k_dg_force, dim3(ceil_div(M, 128), nimg), 128, 0, st,
                            (const double *)x->gf, x->nsF, M, Mp, (const double *)c->fY, x->fpart));
    }
    return TDSCHA_OK;
}

static DgSource dg_matrix(int kind, const double *Y, const double *R, long ystride) {
    return DgSource{kind, Y, R, ystride, 0, nullptr, nullptr, nullptr, 0, 0};
}

// The averages of nimg <= cap perturbations, one context image each (J = 1), into
// f (M each) and d2v (M x M each).
static int digits_averages(tdscha_ctx *c, int nimg, const DgSources &src, int apply_d4, double *f,
                           double *d2v, cudaStream_t st) {
    DigitStore *x = c->dg;
    const int M = c->M, Mp = x->Mp;
    int ns = 0;
    TDS_TRY(digits_contract(c, nimg, src, apply_d4, true, &ns, st));
    ProfScope ps(c, 4, st);
    const int nt = ceil_div(M, 32), nat = ceil_div((long)nimg * Mp, kGM);
    const int pairs = nt * (nt + 1) / 2;
    const bool small = 4 * pairs * nimg < x->nsm;
    TDS_CUDA(launch_pdl(small ? k_dg_final<2, 4> : k_dg_final<8, 1>,
                        dim3((small ? 16 : 4) * pairs, nimg), 256, 0, st, (const double *)x->gpart, ns,
                        (long)nat * kGM * Mp, M, Mp, (const double *)x->fpart, x->nfc,
                        (const double *)c->fY, 1.0 / (c->sum_rho * c->S), (const int *)x->failed, f,
                        d2v));
    return TDSCHA_OK;
}

bool digits_single(const tdscha_ctx *c) { return c->dg && c->J == 1; }
int digits_batch(const tdscha_ctx *c) { return digits_single(c) ? c->dg->cap : 0; }

// The averages of c->Y1 (symmetric), c->R1 into c->f, c->d2v.
int perturb_digits(tdscha_ctx *c, int apply_d4, cudaStream_t st) {
    DigitStore *x = c->dg;
    const int M = c->M, Mp = x->Mp, J = c->J;
    if (J == 1)
        return digits_averages(c, 1, {{dg_matrix(DG_MATRIX, c->Y1, c->R1, 0)}, 1}, apply_d4, c->f,
                               c->d2v, st);
    TDS_TRY(psi_perturbation64(c, st));
    const long MM = (long)M * M;
    for (int j0 = 0; j0 < J; j0 += x->cap) {
        const int nj = std::min(x->cap, J - j0);
        int ns = 0;
        DgSource s = dg_matrix(DG_MATRIX, c->Y1all + j0 * MM, c->vsv + (long)(J + j0) * M, MM);
        s.rstride = M;
        s.S = c->vsv + (long)j0 * M;
        TDS_TRY(digits_contract(c, nj, {{s}, 1}, apply_d4, j0 == 0, &ns, st));
        const int nat = ceil_div((long)nj * Mp, kGM);
        TDS_TRY(psi_hsum64(c, x->gpart, ns, (long)nat * kGM * Mp, (long)Mp * Mp, Mp, x->fpart,
                           x->many ? 1 : x->nfc, c->fY, j0, nj, st));
    }
    return psi_reduce64(c, x->failed, st);
}

int digits_from_matrix(tdscha_ctx *c, int apply_d4, const double *R1, const double *Y1, double *f,
                       double *d2v, cudaStream_t st) {
    return digits_averages(c, 1, {{dg_matrix(DG_AVERAGE, Y1, R1, 0)}, 1}, apply_d4, f, d2v, st);
}

static DgSource dg_psi(const tdscha_ctx *c, const double *psi, const double *ca, const double *cb) {
    const int kind = c->use_wigner ? DG_PSI_WIGNER : ca ? DG_PSI_T : DG_PSI;
    return DgSource{kind, psi, psi, 0, 0, nullptr, ca, cb, c->H, c->ignore_v3};
}

int digits_from_psi(tdscha_ctx *c, int apply_d4, const double *psi, const double *ca,
                    const double *cb, cudaStream_t st) {
    return digits_averages(c, 1, {{dg_psi(c, psi, ca, cb)}, 1}, apply_d4, c->f, c->d2v, st);
}

int digits_from_pair(tdscha_ctx *c, int apply_d4, const double *q, const double *p,
                     const double *ca, const double *cb, double **f, double **d2v,
                     cudaStream_t st) {
    *f = c->dg->fo;
    *d2v = c->dg->d2vo;
    return digits_averages(c, 2, {{dg_psi(c, q, nullptr, nullptr), dg_psi(c, p, ca, cb)}, 2},
                           apply_d4, *f, *d2v, st);
}

int digits_from_static(tdscha_ctx *c, int apply_d4, int nvec, const double *psi, double **f,
                       double **d2v, cudaStream_t st) {
    const long Ps = c->M + c->H;
    *f = c->dg->fo;
    *d2v = c->dg->d2vo;
    const DgSource s{DG_STATIC, psi, psi, Ps, Ps, nullptr, c->Yw, nullptr, c->H, 0};
    return digits_averages(c, nvec, {{s}, 1}, apply_d4, *f, *d2v, st);
}

}  // namespace tdscha
