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
// 56).  What is left out is below 2^-64 of the product of the two row maxima;
// the float64 sums this replaces round every partial sum at 2^-53.
//
// Length of an accumulation: three K blocks (192 elements) keep orders 0..4 exact
// for any input (5 * 192 products of 2^14 stay below 2^24).  The digits of real
// numbers are far from their limits, so the longest accumulation is chosen per
// ensemble by a bound that holds for every perturbation: by Cauchy and Schwarz the
// order-o sum is at most sum_i |d_i| 128 sqrt(K) with |d_i| the largest 2-norm of
// digit i over K elements of any row, measured when the context is made
// (digits_flush).  Gaussian displacements allow five to seven blocks.  Orders 5..7
// could round, by 2^-53 of the row maxima's product or less, only where the
// digits of two rows agree in sign and size over a whole accumulation.
//
// Error (2-norm, against 113-bit arithmetic) of f and d2v, these kernels | those
// of perturb_fp64.cu: M=573 N=2000 6.9e-16 7.0e-16 | 1.3e-15 1.2e-15; with Y1 over
// six decades 7.9e-16 7.7e-16 | 1.4e-15 1.2e-15; M=192 N=3000 1.5e-15 1.5e-15 |
// 1.7e-15 1.6e-15; M=24 N=400 48 images 1.3e-15 5.3e-16 | 3.1e-15 5.6e-16.
// One call: M=573 N=50000 57.1 -> 1.77 ms; M=189 N=10000 48 images 62.8 -> 2.68 ms;
// M=97 N=4999 554 -> 86 us; M=21 N=1000 245 -> 61 us.
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

// alpha, beta / 2 and the force weights of one (image, row)
struct __align__(32) RowScalars {
    double a, b, c1, c2;
};

// ------------------------------------------------- once per ensemble
// Column maxima of |x| and |g|.
__global__ void k_dg_colmax(const double *__restrict__ D, const double *__restrict__ F,
                            const double *__restrict__ fY, long R, int M, long rows_per_block,
                            unsigned long long *__restrict__ dmax,
                            unsigned long long *__restrict__ gmax) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    const long rb = blockIdx.y * rows_per_block, re = min(R, rb + rows_per_block);
    double a = 0, b = 0;
    for (long r = rb; r < re; ++r) {
        a = fmax(a, fabs(D[r * M + m]));
        b = fmax(b, fabs(F[r * M + m]));
    }
    atomic_max_abs(dmax + m, a);
    atomic_max_abs(gmax + m, b / fY[m]);
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

// ec[m]: exponent above the column's maximum; 0 for a zero or padding column
__global__ void k_dg_colexp(const unsigned long long *__restrict__ dmax, int M, int Mp,
                            int *__restrict__ ec) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= Mp) return;
    const double d = m < M ? __longlong_as_double((long long)dmax[m]) : 0.0;
    ec[m] = d > 0 ? exp_above(d) : 0;
}

// er[r]: exponent above the maximum over the modes of |x| 2^-ec (0 for a zero row)
__global__ void k_dg_rowexp(const double *__restrict__ dt, const int *__restrict__ ec, int M,
                            int Mp, int *__restrict__ er) {
    __shared__ int sh[8][128];
    const long rt = blockIdx.x;
    const int row = threadIdx.x, g = threadIdx.y;
    int e = INT_MIN;
    for (int m = g; m < M; m += 8) {
        const double d = dt[(rt * Mp + m) * 128 + row];
        if (d != 0) e = max(e, exp_above(d) - ec[m]);
    }
    sh[g][row] = e;
    __syncthreads();
    if (g == 0) {
        for (int k = 1; k < 8; ++k) e = max(e, sh[k][row]);
        er[rt * 128 + row] = e == INT_MIN ? 0 : e;
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

__global__ void __launch_bounds__(256) k_dg_xb(const double *__restrict__ dt,
                                               const int *__restrict__ ec, int Mp, long nkb,
                                               __half *__restrict__ xb, float *__restrict__ nrm) {
    const long kb = blockIdx.x;
    const int at = blockIdx.y, c = threadIdx.x & 7;
    uint8_t *out = reinterpret_cast<uint8_t *>(xb) + (at * nkb + kb) * kRes * (long)kGB;
    const long r0 = kb * kGK + c * 8;
    for (int row = threadIdx.x >> 3; row < kGN; row += 32) {
        const int a = at * kGN + row;
        const double *src = dt + ((r0 >> 7) * Mp + a) * 128 + (r0 & 127);
        long long q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) q[k] = fixed_point(src[k], 55 - ec[a]);
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

// Row n of image blockIdx.y of Y1 (symmetric): digits of y 2^(ec - et) with et
// the exponent above the row's maximum, and the two vectors of the row scalars.
// Also clears the image's maxima of alpha and beta.
__global__ void __launch_bounds__(128) k_dg_y1(const DgSources src, const double *__restrict__ fY,
                                               const int *__restrict__ ec, int M, int Mp,
                                               __half *__restrict__ yb, int *__restrict__ et,
                                               double *__restrict__ vs, double *__restrict__ vt,
                                               unsigned long long *__restrict__ absmax) {
    pdl_enter();
    extern __shared__ double yrow[];     // M
    __shared__ int sh[4];
    const int n = blockIdx.x, is = min((int)blockIdx.y, src.n - 1);
    const long img = blockIdx.y, rel = img - is;
    const DgSource &c = src.s[is];
    const double *Y = c.Y + rel * c.ystride;
    int e = INT_MIN;
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        const double v = dg_y1(c, Y, M, n, m);
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
    const int nkb = Mp / kGK, row = n % kGN;
    uint8_t *out = reinterpret_cast<uint8_t *>(yb) + (img * (Mp / kGN) + n / kGN) * nkb * (long)kCall * kGB;
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
    if (threadIdx.x == 0) {
        et[img * Mp + n] = e;
        const double r = c.no_r ? 0.0 : c.R[rel * c.rstride + n];
        vs[img * Mp + n] = c.S ? c.S[rel * c.rstride + n] : fY[n] * r;
        vt[img * Mp + n] = fY[n] * r;
        if (n == 0) absmax[2 * img] = absmax[2 * img + 1] = 0ULL;
    }
}

// Row scalars of the image blockIdx.y from the stage A partials; max |alpha|
// and max |beta / 2| of the image.  Rows past the end get zeros.
__global__ void __launch_bounds__(128) k_dg_rows(const double *__restrict__ qp, int nct, long R,
                                                 long Rp, int rho_div,
                                                 const double *__restrict__ rho,
                                                 const int *__restrict__ er, int apply_d4,
                                                 RowScalars *__restrict__ abcc,
                                                 unsigned long long *__restrict__ absmax) {
    pdl_enter();
    __shared__ unsigned long long red[2][4];
    const long img = blockIdx.y, r = blockIdx.x * 128L + threadIdx.x;
    RowScalars v = {0, 0, 0, 0};
    if (r < R) {
        double q = 0, p = 0, s = 0, t = 0;
        const double *o = qp + img * nct * 4 * R + r;
        for (int ct = 0; ct < nct; ++ct, o += 4 * R) {
            q += o[0];
            p += o[R];
            s += o[2 * R];
            t += o[3 * R];
        }
        const double f = pow2(er[r]), rw = rho[r / rho_div], d4 = apply_d4 ? 1.0 : 0.0;
        q *= f;
        p *= f;
        v.a = rw * (s / 3 - d4 * q / 8);
        v.b = 0.5 * (rw * (t / 3 - d4 * p / 4));
        v.c1 = -rw * q / 6;
        v.c2 = -rw * p / 3;
    }
    if (r < Rp) abcc[img * Rp + r] = v;
    unsigned long long a = (unsigned long long)__double_as_longlong(v.a) & 0x7fffffffffffffffULL;
    unsigned long long b = (unsigned long long)__double_as_longlong(v.b) & 0x7fffffffffffffffULL;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = max(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = a;
        red[1][threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 4; ++k) {
            a = max(a, red[0][k]);
            b = max(b, red[1][k]);
        }
        atomicMax(absmax + 2 * img, a);
        atomicMax(absmax + 2 * img + 1, b);
    }
}

// W digits: block = (group of K blocks, tile of 128 rows (image, mode)); thread
// = (mode, eight rows of the ensemble) for 32 modes at a time, so that a warp
// reads 512 contiguous bytes of x and g a mode and writes whole 128-byte rows of
// every digit.  The scale of a mode is the exponent above
// max|alpha| max|g| + max|beta/2| max|x|.  The force partials
// fpart[(img nfc + group) M + b] ride along.
__global__ void __launch_bounds__(256) k_dg_wbuild(
    const double *__restrict__ dt, const double *__restrict__ gt,
    const RowScalars *__restrict__ abcc, const unsigned long long *__restrict__ absmax,
    const unsigned long long *__restrict__ dmax, const unsigned long long *__restrict__ gmax,
    const double *__restrict__ fY, int M, int Mp, long Rp, int nimg, long nkb, int per,
    __half *__restrict__ wa, int *__restrict__ ew, double *__restrict__ fpart) {
    pdl_enter();
    const int c = threadIdx.x & 7;
    const long wt = blockIdx.y, kb0 = blockIdx.x * (long)per, kb1 = min(nkb, kb0 + per);
    uint8_t *out = reinterpret_cast<uint8_t *>(wa) + wt * nkb * kCall * (long)kGA;
    for (int row = threadIdx.x >> 3; row < kGM; row += 32) {
        const long grow = wt * kGM + row;
        const int img = (int)(grow / Mp), b = (int)(grow % Mp);
        // (the eight lanes of a mode take the same branch; padding rows of wa
        // are zero from the start)
        const bool live = img < nimg && b < M;
        double facc = 0;
        if (live) {
            const double am = __longlong_as_double((long long)absmax[2 * img]),
                         bm = __longlong_as_double((long long)absmax[2 * img + 1]),
                         dm = __longlong_as_double((long long)dmax[b]),
                         gm = __longlong_as_double((long long)gmax[b]);
            // a little above the bound: w itself is rounded
            const double bound = (am * gm + bm * dm) * (1.0 + 0x1p-40);
            const bool bad = !isfinite(bound);
            const int e = bad ? kBadExp : bound > 0 ? exp_above(bound) : 0;
            const int K = 62 - e;
            if (blockIdx.x == 0 && c == 0) ew[grow] = e;
            for (long kb = kb0; kb < kb1; ++kb) {
                const long r0 = kb * kGK + c * 8;
                const long o = ((r0 >> 7) * Mp + b) * 128 + (r0 & 127);
                const double2 *d2 = reinterpret_cast<const double2 *>(dt + o);
                const double2 *g2 = reinterpret_cast<const double2 *>(gt + o);
                const RowScalars *ab = abcc + img * Rp + r0;
                long long q[8];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const double2 d = d2[k], g = g2[k];
                    const RowScalars s0 = ab[2 * k], s1 = ab[2 * k + 1];
                    const double w0 = fma(s0.a, g.x, s0.b * d.x), w1 = fma(s1.a, g.y, s1.b * d.y);
                    q[2 * k] = bad ? 0 : fixed_point(w0, K);
                    q[2 * k + 1] = bad ? 0 : fixed_point(w1, K);
                    facc = fma(s0.c1, g.x, facc);
                    facc = fma(s0.c2, d.x, facc);
                    facc = fma(s1.c1, g.y, facc);
                    facc = fma(s1.c2, d.y, facc);
                }
                uint4 w[kCall];
                digits8<kCall>(q, w);
                uint8_t *blk = out + kb * kCall * (long)kGA + sw_place(row, c);
#pragma unroll
                for (int d = 0; d < kCall; ++d) *reinterpret_cast<uint4 *>(blk + d * kGA) = w[d];
            }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) facc += __shfl_xor_sync(0xffffffffu, facc, o);
        if (live && c == 0) fpart[((long)img * gridDim.x + blockIdx.x) * M + b] = facc * fY[b];
    }
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
// 32 x 32 tiles, each element summed over the splits once.
__global__ void __launch_bounds__(256) k_dg_final(const double *__restrict__ gpart, int nsplit,
                                                  long stride, int M, int Mp,
                                                  const double *__restrict__ fpart, int nfc,
                                                  const double *__restrict__ fY, double norm,
                                                  double *__restrict__ f,
                                                  double *__restrict__ d2v) {
    pdl_enter();
    gpart += blockIdx.y * (long)Mp * Mp;
    fpart += blockIdx.y * (long)nfc * M;
    f += blockIdx.y * (long)M;
    d2v += blockIdx.y * (long)M * M;
    __shared__ double tr[32][9], red[8][33];
    const int nt = (M + 31) / 32, slab = blockIdx.x & 3;
    int A = 0, rem = blockIdx.x >> 2;
    while (rem >= nt - A) {
        rem -= nt - A;
        ++A;
    }
    const int B = A + rem, a0 = A * 32 + slab * 8, b0 = B * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const double inv = 1.0 / norm;
    {
        const int ao = threadIdx.x & 7, bo = threadIdx.x >> 3;
        const int b = b0 + bo, a = a0 + ao;
        tr[bo][ao] = (a < M && b < M) ? dg_split_sum(gpart + (long)b * Mp + a, nsplit, stride) : 0.0;
    }
    __syncthreads();
    {
        const int a = a0 + ty, b = b0 + tx;
        if (a < M && b < M) {
            const double h = dg_split_sum(gpart + (long)a * Mp + b, nsplit, stride) + tr[tx][ty];
            const double v = -(h * fY[a]) * fY[b] * inv;
            d2v[(long)a * M + b] = v;
            if (A != B) d2v[(long)b * M + a] = v;
        }
    }
    if (A == 0 && slab == 0) {
        const int e = b0 + tx;
        double acc = 0;
        if (e < M)
            for (int ch = ty; ch < nfc; ch += 8) acc += fpart[(long)ch * M + e];
        red[ty][tx] = acc;
        __syncthreads();
        if (ty == 0 && e < M) {
            for (int k = 1; k < 8; ++k) acc += red[k][tx];
            f[e] = acc * inv;
        }
    }
}

// ------------------------------------------------------------- host side
struct DigitStore {
    int Mp = 0, nkbM = 0, nct = 0, nsm = 1;
    long Rp = 0, nkbR = 0;
    int cap = 1;                 // images that the per-call buffers hold
    int per = 1, nfc = 1;        // K blocks of one W block, force partials an image
    int flushA = kFlushMin, flushB = kFlushMin;   // K blocks per accumulation of the stages
    void *slab = nullptr;
    double *dt = nullptr, *gt = nullptr, *vs = nullptr, *vt = nullptr, *qp = nullptr,
           *gpart = nullptr, *fpart = nullptr, *fo = nullptr, *d2vo = nullptr;
    RowScalars *abcc = nullptr;
    unsigned long long *dmax = nullptr, *gmax = nullptr, *absmax = nullptr;
    __half *xa = nullptr, *xb = nullptr, *yb = nullptr, *wa = nullptr;
    int *ec = nullptr, *er = nullptr, *et = nullptr, *ew = nullptr;
    int *err = nullptr;          // bounded-wait failure code (pinned host memory)
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
        x->cap = (int)std::min<size_t>(c->J, most);
    else
        x->cap = (int)std::max(std::min<size_t>(2, most),
                               std::min<size_t>(32, (size_t(256) << 20) / per_img));
    const int cap = x->cap, nat = ceil_div((long)cap * Mp, kGM);
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
        {(void **)&x->xa, 2 * kRes * elems, false},
        {(void **)&x->xb, 2 * kRes * elems, false},
        {(void **)&x->er, i4 * x->Rp, false},
        {(void **)&x->qp, d * 4 * x->nct * (size_t)cap * R, false},
        {(void **)&x->abcc, sizeof(RowScalars) * (size_t)cap * x->Rp, false},
        {(void **)&x->gpart, gbytes, false},
        {(void **)&x->fpart, d * (size_t)cap * x->nfc * M, false},
        {(void **)&x->fo, c->J == 1 ? d * cap * M : 0, false},
        {(void **)&x->d2vo, c->J == 1 ? d * (size_t)cap * M * M : 0, false},
        {(void **)&x->ec, i4 * Mp, false},
        // zero from the start: maxima, and the rows of padding modes
        {(void **)&x->dmax, u8 * Mp, true},
        {(void **)&x->gmax, u8 * Mp, true},
        {(void **)&x->absmax, u8 * 2 * cap, true},
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
    // a quarter of the free memory at most (asked for only where it can matter)
    if (total > (size_t(4) << 30)) {
        size_t fr = 0, all = 0;
        if (cudaMemGetInfo(&fr, &all) != cudaSuccess || total > fr / 4) {
            cudaGetLastError();
            delete x;
            return TDSCHA_OK;
        }
    }
    if (cached_malloc(&x->slab, total) != cudaSuccess) {
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
    // rows a block walks one after the other: 8 in a small ensemble, at most 128
    const long walk = std::min<long>(128, std::max<long>(8, R / 400));
    k_dg_colmax<<<dim3(ceil_div(M, 128), ceil_div(R, walk)), 128>>>(c->D, c->F, c->fY, R, M, walk,
                                                                    x->dmax, x->gmax);
    TDS_CHECK_LAUNCH();
    k_dg_colexp<<<ceil_div(Mp, 128), 128>>>(x->dmax, M, Mp, x->ec);
    TDS_CHECK_LAUNCH();
    k_dg_cols<<<dim3((unsigned)nrt, Mp / 32), dim3(32, 8)>>>(c->D, c->F, c->fY, R, M, Mp, x->dt,
                                                              x->gt);
    TDS_CHECK_LAUNCH();
    k_dg_rowexp<<<(unsigned)nrt, dim3(128, 8)>>>(x->dt, x->ec, M, Mp, x->er);
    TDS_CHECK_LAUNCH();
    // the digit norms pass through the W digits' space, which is zeroed again
    float *nrm = reinterpret_cast<float *>(x->wa);
    k_dg_xa<<<dim3((unsigned)nrt, x->nkbM), 256>>>(c->D, x->ec, x->er, R, M, x->nkbM, x->xa, nrm);
    TDS_CHECK_LAUNCH();
    k_dg_windows<<<dim3((unsigned)nrt, kFlushes), kGM>>>(nrm, x->nkbM, fl);
    TDS_CHECK_LAUNCH();
    k_dg_xb<<<dim3((unsigned)x->nkbR, x->nct), 256>>>(x->dt, x->ec, Mp, x->nkbR, x->xb, nrm);
    TDS_CHECK_LAUNCH();
    k_dg_windows<<<dim3(x->nct, kFlushes), kGN>>>(nrm, (int)x->nkbR, fl + kFlushes * kRes);
    TDS_CHECK_LAUNCH();
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

int digits_check_error(tdscha_ctx *c) {
    if (!c->dg || !*(volatile int *)c->dg->err) return TDSCHA_OK;
    const int v = *(volatile int *)c->dg->err;
    *(volatile int *)c->dg->err = 0;
    set_error("tensor-core pipeline: a bounded wait expired (code %d)", v);
    return TDSCHA_ERR_TIMEOUT;
}

// Stages A and B for nimg perturbations: split-K partials of every image's H in
// x->gpart, force partials in x->fpart.
static int digits_contract(tdscha_ctx *c, int nimg, const DgSources &src, int apply_d4,
                           int *nsplit, cudaStream_t st) {
    DigitStore *x = c->dg;
    const int M = c->M, Mp = x->Mp;
    const long R = c->Nrows;
    {
        ProfScope ps(c, 5, st);
        TDS_CUDA(launch_pdl(k_dg_y1, dim3(M, nimg), 128, sizeof(double) * M, st, src,
                            (const double *)c->fY, (const int *)x->ec, M, Mp, x->yb, x->et, x->vs,
                            x->vt, x->absmax));
    }
    DgArgs ga{};
    ga.a = x->xa;
    ga.b = x->yb;
    ga.nkb = ga.kbps = x->nkbM;
    ga.flush = x->flushA;
    ga.kk = ceil_div(M, 16);             // (read where M <= 64)
    ga.hc = M <= 32 ? 8 : 16;
    ga.abytes = kGA;
    ga.nat = (int)(x->Rp / kGM);
    ga.nbt = nimg * x->nct;
    ga.nitems = (long)ga.nat * ga.nbt;
    ga.Mp = Mp;
    ga.err = x->err;
    ga.budget = x->budget;
    ga.dt = x->dt;
    ga.gt = x->gt;
    ga.vs = x->vs;
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
        TDS_CUDA(launch_pdl(k_dg_rows, dim3((unsigned)(x->Rp / 128), nimg), 128, 0, st,
                            (const double *)x->qp, x->nct, R, x->Rp, c->rho_div,
                            (const double *)c->rho, (const int *)x->er, apply_d4, x->abcc,
                            x->absmax));
    }
    const int nat = ceil_div((long)nimg * Mp, kGM);
    {
        ProfScope ps(c, 2, st);
        TDS_CUDA(launch_pdl(k_dg_wbuild, dim3(x->nfc, nat), 256, 0, st, (const double *)x->dt,
                            (const double *)x->gt, (const RowScalars *)x->abcc,
                            (const unsigned long long *)x->absmax,
                            (const unsigned long long *)x->dmax,
                            (const unsigned long long *)x->gmax, (const double *)c->fY, M, Mp,
                            x->Rp, nimg, x->nkbR, x->per, x->wa, x->ew, x->fpart));
    }
    DgArgs gb{};
    gb.a = x->wa;
    gb.b = x->xb;
    gb.nkb = (int)x->nkbR;
    gb.kbps = dg_blocks_per_split(x->nkbR, x->flushB, nat, x->nct, x->nsm);
    gb.flush = x->flushB;
    gb.kk = kGK / 16;
    gb.hc = M <= 32 ? 8 : 16;
    gb.abytes = kGA;
    gb.nat = nat;
    gb.nbt = x->nct;
    *nsplit = ceil_div(x->nkbR, gb.kbps);
    gb.nitems = (long)nat * x->nct * *nsplit;
    gb.Mp = Mp;
    gb.err = x->err;
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
    TDS_TRY(digits_contract(c, nimg, src, apply_d4, &ns, st));
    ProfScope ps(c, 4, st);
    const int nt = ceil_div(M, 32), nat = ceil_div((long)nimg * Mp, kGM);
    TDS_CUDA(launch_pdl(k_dg_final, dim3(4 * (nt * (nt + 1) / 2), nimg), 256, 0, st,
                        (const double *)x->gpart, ns, (long)nat * kGM * Mp, M, Mp,
                        (const double *)x->fpart, x->nfc, (const double *)c->fY,
                        c->sum_rho * c->S, f, d2v));
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
        TDS_TRY(digits_contract(c, nj, {{s}, 1}, apply_d4, &ns, st));
        const int nat = ceil_div((long)nj * Mp, kGM);
        TDS_TRY(psi_hsum64(c, x->gpart, ns, (long)nat * kGM * Mp, (long)Mp * Mp, Mp, x->fpart,
                           x->nfc, c->fY, j0, nj, st));
    }
    return psi_reduce64(c, st);
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
