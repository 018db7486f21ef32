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
// the float64 sums this replaces round every partial sum at 2^-53.  An
// accumulation covers three K blocks (192 elements): 5 * 192 products of
// 2^14 stay below 2^24, which keeps orders 0..4 exact for any input; orders
// 5..7 could only round if every digit were at its limit, at 2^-64 of the sum.
//
// Error (2-norm, against 113-bit arithmetic) of f and d2v, these kernels | those
// of perturb_fp64.cu: M=573 N=2000 6.9e-16 7.0e-16 | 1.3e-15 1.2e-15; with Y1 over
// six decades 7.9e-16 7.7e-16 | 1.4e-15 1.2e-15; M=192 N=3000 1.5e-15 1.5e-15 |
// 1.7e-15 1.6e-15; M=24 N=400 48 images 1.3e-15 5.3e-16 | 3.1e-15 5.6e-16.
// One call: M=573 N=50000 57.1 -> 2.55 ms; M=189 N=10000 48 images 62.8 -> 3.69 ms;
// M=97 N=4999 554 -> 99 us; M=21 N=1000 245 -> 73 us.
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

#include "common.cuh"
#include "tcgen05.cuh"

namespace tdscha {

constexpr int kGM = 128;        // rows of an A tile: TMEM lanes
constexpr int kGN = 64;         // rows of a B tile: columns of each order's accumulator
constexpr int kGK = 64;         // K block: one 128-byte swizzle row of fp16
constexpr int kRes = 7;         // digits of the resident operand
constexpr int kCall = 8;        // digits of the operand made per call
constexpr int kOrders = 8;      // orders kept: 8 x 64 accumulator columns fill the TMEM
constexpr int kFlush = 3;       // K blocks per exact accumulation
constexpr int kUnit = -69;      // one unit of the order-7 accumulator: 2^(-7-6-56)
constexpr int kBadExp = 1 << 20;   // exponent of a row with a non-finite element
constexpr uint32_t kGA = kGM * kGK * 2;   // bytes of one digit of an A block
constexpr uint32_t kGB = kGN * kGK * 2;   // and of a B block

// alpha, beta / 2 and the force weights of one (image, row)
struct __align__(32) RowScalars {
    double a, b, c1, c2;
};

// ------------------------------------------------------------ digit splitting
// Smallest E with |x| < 2^E (x finite; 0 and subnormal numbers give -1021).
__device__ __forceinline__ int exp_above(double x) {
    const int e = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
    return max(e, 1) - 1022;
}

// x / 2^(E - frac) rounded to the nearest whole number, |x| < 2^E, K = frac - E.
// Integer operations only: float64 runs at two operations per cycle per SM.
__device__ __forceinline__ long long fixed_point(double x, int K) {
    const long long b = __double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7ff);
    long long m = b & 0xfffffffffffffLL;
    if (e) m |= 1LL << 52;
    const int s = max(e, 1) - 1075 + K;
    const int n = min(-s, 62);
    long long q = s >= 0 ? m << (s & 63) : (m + (1LL << ((n - 1) & 63))) >> (n & 63);
    return b < 0 ? -q : q;
}

// Digits of eight numbers q in units of the last digit, kD of them, as fp16 in
// the order of the numbers (16 bytes a digit).  Adding 128 to every byte turns
// the balanced digits into unsigned bytes; 0x6400 | byte is the fp16 number
// 1024 + byte, and 1152 less is the digit.  The top digit of the 7-digit form
// reaches +128 and takes nine bits.
template <int kD>
__device__ __forceinline__ void digits8(const long long (&q)[8], uint4 (&out)[kD]) {
    uint32_t lo[8], hi[8];
    constexpr unsigned long long kBias = kD == 8 ? 0x8080808080808080ULL : 0x0080808080808080ULL;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const unsigned long long t = (unsigned long long)q[k] + kBias;
        lo[k] = (uint32_t)t;
        hi[k] = (uint32_t)(t >> 32);
    }
    const __half2 off = __half2half2(__ushort_as_half((unsigned short)0xE480));   // -1152
#pragma unroll
    for (int d = 0; d < kD; ++d) {
        const int byte = kD - 1 - d;
        uint32_t w[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const uint32_t a = byte < 4 ? lo[2 * p] : hi[2 * p];
            const uint32_t c = byte < 4 ? lo[2 * p + 1] : hi[2 * p + 1];
            uint32_t v;
            if (kD == 7 && d == 0) {
                // bits 48.. hold the top digit with its bias of 128: 0..256
                v = __byte_perm(a, c, 0x7632) | 0x64006400u;
            } else {
                const uint32_t k = (uint32_t)(byte & 3);
                v = __byte_perm(a, c, k | (k << 4) | ((4 + k) << 8) | ((4 + k) << 12));
                v = (v & 0x00ff00ffu) | 0x64006400u;
            }
            const __half2 h = __hadd2(*reinterpret_cast<const __half2 *>(&v), off);
            w[p] = *reinterpret_cast<const uint32_t *>(&h);
        }
        out[d] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Place of the 16 bytes (row, elements 8 c .. 8 c + 7) inside a [rows x 64] fp16
// block in the 128-byte swizzle, in bytes.
__device__ __forceinline__ uint32_t sw_place(int row, int c) {
    return (uint32_t)row * 128u + (uint32_t)((c ^ (row & 7)) << 4);
}

// (hi 2^32 + lo) 2^e rounded to float64, |hi| < 2^62.  Whole-number operations:
// a conversion of a 64-bit integer occupies the float64 pipe.
__device__ __forceinline__ double fixed_to_double(long long hi, long long lo, int e) {
    const long long h = hi + (lo >> 32);      // floor: what remains is in [0, 2^32)
    const uint32_t l = (uint32_t)lo;
    const bool neg = h < 0;
    unsigned long long mh = neg ? ~(unsigned long long)h + (l == 0u) : (unsigned long long)h;
    const uint32_t ml = neg ? 0u - l : l;
    // the leading 64 bits of the magnitude
    int z;
    unsigned long long top;
    if (mh) {
        z = __clzll((long long)mh);
        top = (mh << z) | (((unsigned long long)ml << 32) >> (64 - z));     // z >= 1
    } else {
        if (ml == 0u) return e >= kBadExp / 2 ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
        z = 64 + __clz((int)ml);
        top = (unsigned long long)ml << (z - 32);
    }
    const unsigned long long m = (top >> 11) + ((top >> 10) & 1ULL);   // 2^52 <= m <= 2^53
    const int E = 1074 + 43 - z + e;          // one less than the exponent field: m adds one
    if (E >= 2046) return __longlong_as_double(e >= kBadExp / 2 ? 0x7ff8000000000000LL
                                               : neg ? 0xfff0000000000000ULL : 0x7ff0000000000000LL);
    if (E < 0) return 0.0;
    const unsigned long long bits = ((unsigned long long)E << 52) + m;
    return __longlong_as_double((long long)(bits | (neg ? 1ULL << 63 : 0ULL)));
}

// 2^e for the exponents of finite float64 rows
__device__ __forceinline__ double pow2(int e) { return ldexp(1.0, e); }

// ------------------------------------------------- once per ensemble
__device__ __forceinline__ void atomic_max_abs(unsigned long long *addr, double v) {
    // absolute values order like their bit patterns (NaN above infinity)
    atomicMax(addr, (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffULL);
}

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
                                               __half *__restrict__ xa) {
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
    }
}

__global__ void __launch_bounds__(256) k_dg_xb(const double *__restrict__ dt,
                                               const int *__restrict__ ec, int Mp, long nkb,
                                               __half *__restrict__ xb) {
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
    }
}

// ------------------------------------------------- once per call
// Row n of image blockIdx.y of Y1 (symmetric): digits of y 2^(ec - et) with et
// the exponent above the row's maximum, and the two vectors of the row scalars.
// Also clears the image's maxima of alpha and beta.
__global__ void __launch_bounds__(128) k_dg_y1(const double *__restrict__ Y1,
                                               const double *__restrict__ svec,
                                               const double *__restrict__ tvec, int s_times_fy,
                                               const double *__restrict__ fY,
                                               const int *__restrict__ ec, int M, int Mp,
                                               __half *__restrict__ yb, int *__restrict__ et,
                                               double *__restrict__ vs, double *__restrict__ vt,
                                               unsigned long long *__restrict__ absmax) {
    pdl_enter();
    __shared__ int sh[4];
    const int n = blockIdx.x;
    const long img = blockIdx.y;
    const double *y = Y1 + (img * M + n) * M;
    int e = INT_MIN;
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        const double v = y[m];
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
        const int kb = ch >> 3, c = ch & 7;
        long long q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int m = ch * 8 + k;
            q[k] = (m < M && !bad) ? fixed_point(y[m], 62 + ec[m] - e) : 0;
        }
        uint4 w[kCall];
        digits8<kCall>(q, w);
#pragma unroll
        for (int d = 0; d < kCall; ++d)
            *reinterpret_cast<uint4 *>(out + (kb * (long)kCall + d) * kGB + sw_place(row, c)) = w[d];
    }
    if (threadIdx.x == 0) {
        et[img * Mp + n] = e;
        const double s = svec[img * M + n];
        vs[img * Mp + n] = s_times_fy ? fY[n] * s : s;
        vt[img * Mp + n] = fY[n] * tvec[img * M + n];
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

// -------------------------------------------------------- the contraction
// Persistent, one CTA per SM, 320 threads, one 128 x 64 output tile at a time;
// its accumulators, eight orders of 64 columns, fill the TMEM.
//   warp 8  copies: B blocks (all digits of 64 rows) into two buffers, A digits
//           (128 rows each) into a ring
//   warp 9  MMA issue: A digit i against the B digits 0 .. 7 - i at once, which
//           lie behind one another in shared memory as their accumulators do in
//           TMEM, so one instruction covers up to four orders (N = 256).  i
//           runs downwards: the light high orders come first.
//   warps 0-7  every three K blocks the accumulators are read, order 7 first,
//           and added to two 64-bit integers an element (warp w: lanes 32 (w % 4),
//           columns 32 (w / 4) of every order).  Each order has its own
//           release, so the MMAs of the next blocks start on order 7 while the
//           lower ones are still read.  At the end of a tile the sums become
//           float64: row dots (stage A) or a partial tile (stage B).
// Bounded waits and the abort flag as in perturb_mixed.cu.
struct DgArgs {
    const __half *a, *b;
    int nkb;               // K blocks of an operand row
    int kbps;              // K blocks per work item (stage A: nkb)
    int nat, nbt;          // A and B tiles
    long nitems;
    int Mp;
    int *err;
    long long budget;
    // stage A
    const double *dt, *gt, *vs, *vt;
    const int *et;
    double *qp;            // [image][column tile][4][R]
    long R;
    int nct;               // column tiles of one image
    // stage B
    const double *fY;
    const int *ec, *ew;
    double *gpart;         // [split][A rows][Mp]
    int M;
    long rows_b;           // rows (image, mode) in use
};

template <bool kStageA>
struct DgShape {
    static constexpr int SA = kStageA ? kRes : kCall, SB = kStageA ? kCall : kRes;
    static constexpr int slots = kStageA ? 5 : 6;     // A ring: with the B buffers 208 KB
    static constexpr uint32_t bbytes = SB * kGB;
    static constexpr int bars = 2 * slots + 4 + 1 + kOrders + 1;
    static constexpr size_t ring = 2 * (size_t)bbytes + slots * (size_t)kGA;
    static constexpr size_t smem = 1024 + ring + 2 * 4 * 128 * sizeof(double) +
                                   2 * kGN * (2 * sizeof(double) + sizeof(int)) + 8 * bars + 16;
};
static_assert(DgShape<true>::smem <= 232448 && DgShape<false>::smem <= 232448,
              "shared memory above the per-block limit");

// Named barrier 1 over the 256 epilogue threads; true if `pred` was set in any.
__device__ __forceinline__ bool dg_sync_or(bool pred) {
    uint32_t out;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, 1, 256, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(out)
        : "r"((uint32_t)pred)
        : "memory");
    return out != 0;
}

template <bool kStageA>
__global__ void __launch_bounds__(320, 1) k_dg_gemm(const DgArgs args) {
    using Sh = DgShape<kStageA>;
    constexpr int SA = Sh::SA, SB = Sh::SB, slots = Sh::slots;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *ring = smem + 2 * Sh::bbytes;
    double *red = reinterpret_cast<double *>(smem + Sh::ring);        // [2][4][128]
    double *colv = red + 2 * 4 * 128;                                  // [2][2][64]
    int *cole = reinterpret_cast<int *>(colv + 2 * 2 * kGN);           // [2][64]
    uint64_t *bars = reinterpret_cast<uint64_t *>(cole + 2 * kGN);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + Sh::bars);
    volatile int *abort = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const uint32_t afull = smem_u32(bars), aempty = afull + 8 * slots, bfull = aempty + 8 * slots,
                   bempty = bfull + 16, tfull = bempty + 16, tempty = tfull + 8,
                   done = tempty + 8 * kOrders;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long budget = args.budget;
    const long G = gridDim.x;
    const long nloc = args.nitems > (long)blockIdx.x ? (args.nitems - 1 - blockIdx.x) / G + 1 : 0;
    const int tiles = args.nat * args.nbt;

    if (threadIdx.x == 0) {
        for (int s = 0; s < slots; ++s) {
            mbar_init(afull + 8 * s, 1);
            mbar_init(aempty + 8 * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(bfull + 8 * s, 1);
            mbar_init(bempty + 8 * s, 1);
        }
        mbar_init(tfull, 1);
        for (int o = 0; o < kOrders; ++o) mbar_init(tempty + 8 * o, 8);
        mbar_init(done, 1);
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 9) tmem_alloc<512>(smem_u32(tmem_slot));
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_enter();
    int fail_code = 0;

    // work item i of this CTA: neighbouring CTAs take neighbouring B tiles of
    // one A tile (stage A) or of one split (stage B) and share it in L2
    auto item = [&](long i, int &at, int &bt, int &kb0, int &nkb) {
        const long w = blockIdx.x + i * G;
        const int split = (int)(w / tiles), tile = (int)(w % tiles);
        at = tile / args.nbt;
        bt = tile % args.nbt;
        kb0 = split * args.kbps;
        nkb = min(args.kbps, args.nkb - kb0);
    };

    if (warp == 8) {
        if (lane == 0) {
            long ga = 0, gb = 0;
            for (long i = 0; i < nloc && !fail_code; ++i) {
                int at, bt, kb0, nkb;
                item(i, at, bt, kb0, nkb);
                const uint8_t *pa = reinterpret_cast<const uint8_t *>(args.a) +
                                    ((long)at * args.nkb + kb0) * SA * (long)kGA;
                const uint8_t *pb = reinterpret_cast<const uint8_t *>(args.b) +
                                    ((long)bt * args.nkb + kb0) * SB * (long)kGB;
                for (int kb = 0; kb < nkb && !fail_code; ++kb) {
                    const int sb = (int)(gb & 1);
                    if (gb >= 2 && !mbar_wait_ab(bempty + 8 * sb, ((uint32_t)(gb >> 1) & 1) ^ 1,
                                                 budget, abort)) {
                        fail_code = 1;
                        break;
                    }
                    mbar_expect_tx(bfull + 8 * sb, Sh::bbytes);
#pragma unroll
                    for (int d = 0; d < SB; ++d)
                        bulk_load(smem_u32(smem + sb * Sh::bbytes + d * kGB), pb + d * kGB, kGB,
                                  bfull + 8 * sb);
                    pb += SB * (long)kGB;
                    ++gb;
                    for (int d = SA - 1; d >= 0; --d, ++ga) {
                        const int s = (int)(ga % slots);
                        const uint32_t n = (uint32_t)(ga / slots);
                        if (ga >= slots && !mbar_wait_ab(aempty + 8 * s, (n & 1) ^ 1, budget, abort)) {
                            fail_code = 1;
                            break;
                        }
                        mbar_expect_tx(afull + 8 * s, kGA);
                        bulk_load(smem_u32(ring + s * kGA), pa + d * (long)kGA, kGA, afull + 8 * s);
                    }
                    pa += SA * (long)kGA;
                }
            }
            if (fail_code) {
                *abort = 1;
                // every issued copy must land before the CTA exits
                for (long g = ga > slots ? ga - slots : 0; g < ga; ++g)
                    mbar_wait(afull + 8 * (int)(g % slots), (uint32_t)(g / slots) & 1, kDefaultBudget);
                for (long g = gb > 2 ? gb - 2 : 0; g < gb; ++g)
                    mbar_wait(bfull + 8 * (int)(g & 1), (uint32_t)(g >> 1) & 1, kDefaultBudget);
            }
        }
    } else if (warp == 9) {
        if (lane == 0) {
            long ga = 0, gb = 0, nch = 0;    // A digits, B blocks, accumulations so far
            for (long i = 0; i < nloc && !fail_code; ++i) {
                int at, bt, kb0, nkb;
                item(i, at, bt, kb0, nkb);
                for (int kb = 0; kb < nkb && !fail_code; ++kb, ++gb) {
                    const bool first = kb % kFlush == 0;
                    const int sb = (int)(gb & 1);
                    if (!mbar_wait_ab(bfull + 8 * sb, (uint32_t)(gb >> 1) & 1, budget, abort)) {
                        fail_code = 2;
                        break;
                    }
                    const uint32_t bbase = smem_u32(smem + sb * Sh::bbytes);
#pragma unroll
                    for (int d = SA - 1; d >= 0; --d) {
                        constexpr int kTop = SA - 1;
                        const int cnt = SB < kOrders - d ? SB : kOrders - d;   // orders d .. d + cnt - 1
                        const int s = (int)(ga % slots);
                        bool ok = mbar_wait_ab(afull + 8 * s, (uint32_t)(ga / slots) & 1, budget, abort);
                        if (first && nch > 0) {
                            // the orders that this digit writes first: d, and at the
                            // top digit all of its orders
                            const uint32_t par = (uint32_t)(nch - 1) & 1;
                            for (int o = d; o < (d == kTop ? d + cnt : d + 1); ++o)
                                ok = ok && mbar_wait_ab(tempty + 8 * o, par, budget, abort);
                        }
                        if (!ok) {
                            fail_code = 2;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t abase = smem_u32(ring + s * kGA);
#pragma unroll
                        for (int kk = 0; kk < kGK / 16; ++kk) {
                            const uint64_t da = sdesc_sw128(abase + kk * 32);
                            const uint32_t col = tmem + kGN * d;
                            auto span = [&](int j0, int n, uint32_t acc) {
                                mma_f16(col + kGN * j0, da, sdesc_sw128(bbase + j0 * kGB + kk * 32),
                                        idesc_f16(kGM, kGN * n), acc);
                            };
                            const int n1 = cnt > 4 ? (cnt + 1) / 2 : cnt;
                            if (first && kk == 0 && d < kTop) {
                                // order d starts here, the higher ones go on
                                span(0, 1, 0u);
                                if (cnt > 5) {
                                    span(1, 4, 1u);
                                    span(5, cnt - 5, 1u);
                                } else if (cnt > 1) {
                                    span(1, cnt - 1, 1u);
                                }
                            } else {
                                const uint32_t acc = (kk == 0 && first) ? 0u : 1u;
                                span(0, n1, acc);
                                if (cnt > n1) span(n1, cnt - n1, acc);
                            }
                        }
                        mma_commit(aempty + 8 * s);
                        ++ga;
                    }
                    if (fail_code) break;
                    mma_commit(bempty + 8 * sb);
                    if (kb % kFlush == kFlush - 1 || kb == nkb - 1) {
                        mma_commit(tfull);
                        ++nch;
                    }
                }
            }
            if (fail_code) *abort = 1;
            mma_commit(done);
        }
    } else {
        const int quad = warp & 3, half = warp >> 2;
        const int row = quad * 32 + lane;
        const uint32_t base = tmem + ((uint32_t)(quad * 32) << 16) + 32 * half;
        long nch = 0;
        for (long i = 0; i < nloc; ++i) {
            int at, bt, kb0, nkb;
            item(i, at, bt, kb0, nkb);
            double *cv = colv + (i & 1) * 2 * kGN;
            int *ce = cole + (i & 1) * kGN;
            if (threadIdx.x < kGN) {
                const long c = (long)bt * kGN + threadIdx.x;
                if (kStageA) {
                    cv[threadIdx.x] = args.vs[c];
                    cv[kGN + threadIdx.x] = args.vt[c];
                    ce[threadIdx.x] = args.et[c] + kUnit;
                } else {
                    cv[threadIdx.x] = c < args.M ? args.fY[c] : 0.0;
                    ce[threadIdx.x] = args.ec[c] + kUnit;
                }
            }
            long long hi[32], lo[32];
#pragma unroll
            for (int e = 0; e < 32; ++e) hi[e] = lo[e] = 0;
            const int nacc = (nkb + kFlush - 1) / kFlush;
            for (int c = 0; c < nacc; ++c, ++nch) {
                const bool ok = mbar_wait_ab(tfull, (uint32_t)nch & 1, budget, abort);
                __syncwarp();
                if (dg_sync_or(!ok)) {     // also publishes cv and ce
                    fail_code = 3;
                    break;
                }
                tc_fence_after();
#pragma unroll
                for (int o = kOrders - 1; o >= 0; --o) {
                    const int k = 8 * ((kOrders - 1 - o) & 3);
#pragma unroll
                    for (int e0 = 0; e0 < 32; e0 += 16) {
                        uint32_t v[16];
                        tmem_ld16(base + kGN * o + e0, v);
                        tmem_wait_ld();
                        if (e0) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(tempty + 8 * o);
                        }
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            const long long t = (long long)__float2int_rn(__uint_as_float(v[e]));
                            if (o >= 4)
                                lo[e0 + e] += t * (1LL << k);
                            else
                                hi[e0 + e] += t * (1LL << k);
                        }
                    }
                }
            }
            if (fail_code) break;
            const int c0 = half * 32;
            if (kStageA) {
                const long tile = ((long)at * args.Mp + (long)(bt % args.nct) * kGN + c0) * 128 + row;
                const double *pd = args.dt + tile, *pg = args.gt + tile;
                double q = 0, p = 0, s = 0, t = 0;
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    const double d = pd[e * 128], g = pg[e * 128];
                    const double v = fixed_to_double(hi[e], lo[e], ce[c0 + e]);
                    q = fma(d, v, q);
                    p = fma(g, v, p);
                    s = fma(cv[c0 + e], d, s);
                    t = fma(cv[kGN + c0 + e], g, t);
                }
                double *rb = red + (i & 1) * 4 * 128 + row;
                if (half) {
                    rb[0] = q;
                    rb[128] = p;
                    rb[256] = s;
                    rb[384] = t;
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
                const long r = (long)at * kGM + row;
                if (!half && r < args.R) {
                    double *o = args.qp + (long)bt * 4 * args.R + r;
                    o[0] = q + rb[0];
                    o[args.R] = p + rb[128];
                    o[2 * args.R] = s + rb[256];
                    o[3 * args.R] = t + rb[384];
                }
            } else {
                const long grow = (long)at * kGM + row;
                const int b = (int)(grow % args.Mp);
                const bool live = grow < args.rows_b && b < args.M;
                if (live) {
                    const long w = blockIdx.x + i * G;
                    const double fb = args.fY[b];
                    const int eb = args.ew[grow];
                    double *o = args.gpart + ((w / tiles) * args.nat * kGM + grow) * args.Mp +
                                (long)bt * kGN + c0;
#pragma unroll
                    for (int e = 0; e < 32; e += 2) {
                        double2 x;
                        x.x = fixed_to_double(hi[e], lo[e], ce[c0 + e] + eb) * (fb * cv[c0 + e]);
                        x.y = fixed_to_double(hi[e + 1], lo[e + 1], ce[c0 + e + 1] + eb) *
                              (fb * cv[c0 + e + 1]);
                        *reinterpret_cast<double2 *>(o + e) = x;
                    }
                }
            }
        }
        if (fail_code) *abort = 1;
    }
    if (fail_code && lane == 0) *(volatile int *)args.err = 10 + fail_code;
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        mbar_wait(done, 0, kDefaultBudget);
        __syncwarp();
        tc_fence_after();
        tmem_dealloc<512>(tmem);
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

// d2v = -(G + G^T) / norm and f = sum fpart / norm of the image blockIdx.y (no
// symmetry images): one block per 8-row slab of a pair (A, B), A <= B, of
// 32 x 32 tiles, each element summed over the splits once.
__global__ void __launch_bounds__(256) k_dg_final(const double *__restrict__ gpart, int nsplit,
                                                  long stride, int M, int Mp,
                                                  const double *__restrict__ fpart, int nfc,
                                                  double norm, double *__restrict__ f,
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
            const double v = -(dg_split_sum(gpart + (long)a * Mp + b, nsplit, stride) + tr[tx][ty]) * inv;
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
    void *slab = nullptr;
    double *dt = nullptr, *gt = nullptr, *vs = nullptr, *vt = nullptr, *qp = nullptr,
           *gpart = nullptr, *fpart = nullptr;
    RowScalars *abcc = nullptr;
    unsigned long long *dmax = nullptr, *gmax = nullptr, *absmax = nullptr;
    __half *xa = nullptr, *xb = nullptr, *yb = nullptr, *wa = nullptr;
    int *ec = nullptr, *er = nullptr, *et = nullptr, *ew = nullptr;
    int *err = nullptr;          // bounded-wait failure code (pinned host memory)
    long long budget = kDefaultBudget;
};

// K blocks per split of stage B for `nat` W tiles: the fewest waves of 152 SMs
// weighted with what a wave costs: 4900 cycles a K block (35 products of 128 x 64
// x 64 at 4096 a cycle, and a tenth), 8000 to fill the ring and to write the
// tile; and the partial tiles written and read again (both at about 3 KB a cycle).
static int dg_blocks_per_split(const DigitStore *x, int nat) {
    const long tiles = (long)nat * x->nct, nkb = x->nkbR;
    const double part = 16.0 * nat * kGM * x->Mp / 3000.0;
    double best = 1e300;
    int kb_best = (int)nkb;
    for (long n = 1; n <= std::min<long>(nkb, 96); ++n) {
        long kb = (nkb + n - 1) / n;
        // whole accumulations where a split has several
        if (kb > kFlush) kb = (kb + kFlush - 1) / kFlush * kFlush;
        const long ns = (nkb + kb - 1) / kb;
        if (kb > 16384) continue;             // 64-bit sums of the orders
        const double cost = (double)((tiles * ns + x->nsm - 1) / x->nsm) * (kb * 4900.0 + 8000.0) +
                            part * ns;
        if (cost < best * 0.999) {
            best = cost;
            kb_best = (int)kb;
        }
    }
    return kb_best;
}

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
    // images of one pass over W: all of them within 6 GB of W digits
    x->cap = (int)std::max<size_t>(1, std::min<size_t>(c->J, (size_t(6) << 30) / (elems * 2 * kCall)));
    const int cap = x->cap, nat = ceil_div((long)cap * Mp, kGM);
    // about eight W blocks per SM, at most 16 K blocks each
    x->per = (int)std::max<long>(1, std::min<long>(16, x->nkbR * nat / (152L * 8)));
    x->nfc = ceil_div(x->nkbR, x->per);
    size_t gbytes = 0;
    for (int n = 1; n <= cap; ++n) {
        const int na = ceil_div((long)n * Mp, kGM), kb = dg_blocks_per_split(x, na);
        gbytes = std::max(gbytes, (size_t)ceil_div(x->nkbR, kb) * na * kGM * Mp * sizeof(double));
    }
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
        {(void **)&x->ec, i4 * Mp, false},
        // zero from the start: maxima, and the rows of padding modes
        {(void **)&x->dmax, u8 * Mp, true},
        {(void **)&x->gmax, u8 * Mp, true},
        {(void **)&x->absmax, u8 * 2 * cap, true},
        {(void **)&x->vs, d * cap * Mp, true},
        {(void **)&x->vt, d * cap * Mp, true},
        {(void **)&x->et, i4 * cap * Mp, true},
        {(void **)&x->ew, i4 * (size_t)nat * kGM, true},
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
    k_dg_colmax<<<dim3(ceil_div(M, 128), ceil_div(R, 128)), 128>>>(c->D, c->F, c->fY, R, M, 128,
                                                                    x->dmax, x->gmax);
    TDS_CHECK_LAUNCH();
    k_dg_colexp<<<ceil_div(Mp, 128), 128>>>(x->dmax, M, Mp, x->ec);
    TDS_CHECK_LAUNCH();
    k_dg_cols<<<dim3((unsigned)nrt, Mp / 32), dim3(32, 8)>>>(c->D, c->F, c->fY, R, M, Mp, x->dt,
                                                              x->gt);
    TDS_CHECK_LAUNCH();
    k_dg_rowexp<<<(unsigned)nrt, dim3(128, 8)>>>(x->dt, x->ec, M, Mp, x->er);
    TDS_CHECK_LAUNCH();
    k_dg_xa<<<dim3((unsigned)nrt, x->nkbM), 256>>>(c->D, x->ec, x->er, R, M, x->nkbM, x->xa);
    TDS_CHECK_LAUNCH();
    k_dg_xb<<<dim3((unsigned)x->nkbR, x->nct), 256>>>(x->dt, x->ec, Mp, x->nkbR, x->xb);
    TDS_CHECK_LAUNCH();
    TDS_CUDA(cudaFuncSetAttribute(k_dg_gemm<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)DgShape<true>::smem));
    TDS_CUDA(cudaFuncSetAttribute(k_dg_gemm<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)DgShape<false>::smem));
    return TDSCHA_OK;
}

int digits_check_error(tdscha_ctx *c) {
    if (!c->dg || !*(volatile int *)c->dg->err) return TDSCHA_OK;
    const int v = *(volatile int *)c->dg->err;
    *(volatile int *)c->dg->err = 0;
    set_error("tensor-core pipeline: a bounded wait expired (code %d)", v);
    return TDSCHA_ERR_TIMEOUT;
}

// Stages A and B for nimg symmetric matrices Y1 (M x M each) with their two row
// vectors (M each): split-K partials of every image's H in x->gpart, force
// partials in x->fpart.
static int digits_contract(tdscha_ctx *c, int nimg, const double *Y1, const double *svec,
                           const double *tvec, int s_times_fy, int apply_d4, int *nsplit,
                           cudaStream_t st) {
    DigitStore *x = c->dg;
    const int M = c->M, Mp = x->Mp;
    const long R = c->Nrows;
    {
        ProfScope ps(c, 5, st);
        TDS_CUDA(launch_pdl(k_dg_y1, dim3(M, nimg), 128, 0, st, Y1, svec, tvec, s_times_fy, c->fY,
                            x->ec, M, Mp, x->yb, x->et, x->vs, x->vt, x->absmax));
    }
    DgArgs ga{};
    ga.a = x->xa;
    ga.b = x->yb;
    ga.nkb = ga.kbps = x->nkbM;
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
    {
        ProfScope ps(c, 0, st);
        TDS_CUDA(launch_pdl(k_dg_gemm<true>, (int)std::min<long>(ga.nitems, x->nsm), 320,
                            DgShape<true>::smem, st, ga));
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
    gb.kbps = dg_blocks_per_split(x, nat);
    gb.nat = nat;
    gb.nbt = x->nct;
    *nsplit = ceil_div(x->nkbR, gb.kbps);
    gb.nitems = (long)nat * x->nct * *nsplit;
    gb.Mp = Mp;
    gb.err = x->err;
    gb.budget = x->budget;
    gb.fY = c->fY;
    gb.ec = x->ec;
    gb.ew = x->ew;
    gb.gpart = x->gpart;
    gb.M = M;
    gb.rows_b = (long)nimg * Mp;
    ProfScope ps(c, 3, st);
    TDS_CUDA(launch_pdl(k_dg_gemm<false>, (int)std::min<long>(gb.nitems, x->nsm), 320,
                        DgShape<false>::smem, st, gb));
    return TDSCHA_OK;
}

// The averages of c->Y1 (symmetric), c->R1 into c->f, c->d2v.
int perturb_digits(tdscha_ctx *c, int apply_d4, cudaStream_t st) {
    DigitStore *x = c->dg;
    const int M = c->M, Mp = x->Mp, J = c->J;
    int ns = 0;
    if (J == 1) {
        TDS_TRY(digits_contract(c, 1, c->Y1, c->R1, c->R1, 1, apply_d4, &ns, st));
        ProfScope ps(c, 4, st);
        const int nt = ceil_div(M, 32), nat = ceil_div((long)Mp, kGM);
        TDS_CUDA(launch_pdl(k_dg_final, dim3(4 * (nt * (nt + 1) / 2), 1), 256, 0, st,
                            (const double *)x->gpart, ns, (long)nat * kGM * Mp, M, Mp,
                            (const double *)x->fpart, x->nfc, c->sum_rho * c->S, c->f, c->d2v));
        return TDSCHA_OK;
    }
    TDS_TRY(psi_perturbation64(c, st));
    for (int j0 = 0; j0 < J; j0 += x->cap) {
        const int nj = std::min(x->cap, J - j0);
        TDS_TRY(digits_contract(c, nj, c->Y1all + (size_t)j0 * M * M, c->vsv + (size_t)j0 * M,
                                c->vsv + (size_t)(J + j0) * M, 0, apply_d4, &ns, st));
        const int nat = ceil_div((long)nj * Mp, kGM);
        TDS_TRY(psi_hsum64(c, x->gpart, ns, (long)nat * kGM * Mp, (long)Mp * Mp, Mp, x->fpart,
                           x->nfc, j0, nj, st));
    }
    return psi_reduce64(c, st);
}

}  // namespace tdscha
