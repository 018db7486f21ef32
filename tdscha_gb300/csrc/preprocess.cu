// Ensemble preprocessing and the gamma-only translation projection.
//
// * Mode projection (Modules/DynamicalLanczos.py:392-452): with u the
//   displacements and f the forces minus the SSCHA forces, both N x n_cart,
//     X = (u * u_scale * sqrt(m)) . pols,   Y = ((f * f_scale - f_mean) / sqrt(m)) . pols
// * Bloch projection (Modules/QSpaceLanczos.py:221-296): per q-point,
//     X_q = (u_q * u_scale * sqrt(m)) . conj(pols_q),
//     Y_q = ((f_q - f_mean_q) * f_scale / sqrt(m)) . conj(pols_q)
//   with f_mean_q non-zero at Gamma only.
// * gamma_only projection of the averages (DynamicalLanczos.py:3173-3191):
//     f   <- P_t f,  P_t = mean_R pols^T P_R pols
//     d2v <- pols^T [ mean_R Perm_R(pols d2v pols^T) ] pols
//   Perm_R(D)[r][s] = D[perm_R[r]][perm_R[s]] (Cartesian index permutations).
// The mode projection of an ensemble, N x n_cart x M, runs as exact digit products
// on the tensor cores (perturb_digits.cu explains them); the others, O(M^3) per
// application or small, in float64 (complex double2 for the Bloch projection) on
// the CUDA cores.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "digits.cuh"

namespace tdscha {

struct RealOps {
    using T = double;
    __device__ static T zero() { return 0.0; }
    __device__ static T fma_(T a, T b, T c) { return fma(a, b, c); }
};
struct CplxConjBOps {   // acc + a conj(b)
    using T = double2;
    __device__ static T zero() { return make_double2(0, 0); }
    __device__ static T fma_(T a, T b, T c) {
        c.x = fma(a.x, b.x, c.x);
        c.x = fma(a.y, b.y, c.x);
        c.y = fma(a.y, b.x, c.y);
        c.y = fma(-a.x, b.y, c.y);
        return c;
    }
};

// C (rows x cols) = A . B, A(i, k) = A[i*sai + k*sak], B(k, j) = B[k*sbk + j*sbj],
// C row-major with leading dimension ldc.  64 x 64 tiles, 16-deep k slices,
// 256 threads, 4 x 4 outputs per thread; batched over blockIdx.z with the
// given per-batch strides.
template <class Ops>
__global__ void __launch_bounds__(256) k_gemm64(const typename Ops::T *__restrict__ A,
                                                const typename Ops::T *__restrict__ B,
                                                typename Ops::T *__restrict__ C, int rows,
                                                int cols, int K, long sai, long sak, long sbk,
                                                long sbj, long ldc, long bsA, long bsB,
                                                long bsC) {
    using T = typename Ops::T;
    __shared__ T As[16][64 + 1];
    __shared__ T Bs[16][64 + 1];
    A += blockIdx.z * bsA;
    B += blockIdx.z * bsB;
    C += blockIdx.z * bsC;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int i0 = blockIdx.y * 64, j0 = blockIdx.x * 64;
    T acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = Ops::zero();
    for (int k0 = 0; k0 < K; k0 += 16) {
        for (int t = threadIdx.x; t < 16 * 64; t += 256) {
            int kk = t % 16, ii = t / 16;
            int i = i0 + ii, k = k0 + kk;
            As[kk][ii] = (i < rows && k < K) ? A[i * sai + k * sak] : Ops::zero();
            int jj = t % 64, kb = t / 64;
            int j = j0 + jj, k2 = k0 + kb;
            Bs[kb][jj] = (j < cols && k2 < K) ? B[k2 * sbk + j * sbj] : Ops::zero();
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            T a[4], b[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                a[q] = As[kk][ty + 16 * q];
                b[q] = Bs[kk][tx + 16 * q];
            }
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[p][q] = Ops::fma_(a[p], b[q], acc[p][q]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            int i = i0 + ty + 16 * p, j = j0 + tx + 16 * q;
            if (i < rows && j < cols) C[i * ldc + j] = acc[p][q];
        }
}

template <class Ops>
static int gemm(const typename Ops::T *A, const typename Ops::T *B, typename Ops::T *C, int rows,
                int cols, int K, long sai, long sak, long sbk, long sbj, long ldc,
                cudaStream_t st, int batch = 1, long bsA = 0, long bsB = 0, long bsC = 0) {
    dim3 grid(ceil_div(cols, 64), ceil_div(rows, 64), batch);
    k_gemm64<Ops><<<grid, 256, 0, st>>>(A, B, C, rows, cols, K, sai, sak, sbk, sbj, ldc, bsA, bsB,
                                        bsC);
    TDS_CHECK_LAUNCH();
    return TDSCHA_OK;
}

// a'[i][k] = (a[i][k] * s - sub[k]) * mul[k] on row-major n x K data (T = double or double2)
__global__ void k_prologue(const double *__restrict__ a, long n, int K, int width, double s,
                           const double *__restrict__ sub, const double *__restrict__ mul,
                           double *__restrict__ out) {
    // width = 1 (real) or 2 (interleaved complex); sub has width entries per k
    long total = n * K * width;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
        int k = (int)((e / width) % K), c = (int)(e % width);
        double v = a[e] * s;
        if (sub) v -= sub[k * width + c];
        out[e] = v * mul[k];
    }
}

// Scales of the columns of a' = (a s - sub) mul, taken into mul2 = mul 2^-ec.  A row's scale
// is the exponent above its largest |a'| 2^-ec, so any ec keeps the digits in range; what
// counts is that it makes the columns alike.  Every row is a result of its own here, so ec is
// the mean of the largest exponents of 16 groups of up to 32 rows spread over all: an outlier
// moves it by its group's share only, and a column of rounding noise over many decades counts
// by its largest elements.  Columns without an element in these rows are searched through;
// one without any gets kZeroExp, which leaves it out of B's scales.
// Block: 8 columns, 128 rows at a time: a warp's float64 operation takes 64 cycles, so the
// 512 rows are spread over many warps of many blocks.
__global__ void __launch_bounds__(1024) k_dg_colscale(const double *__restrict__ a, long rows, int K,
                                                      double s, const double *__restrict__ sub,
                                                      const double *__restrict__ mul,
                                                      double *__restrict__ mul2, int *__restrict__ ec) {
    pdl_enter();
    __shared__ int sh[32][8];
    const int cc = threadIdx.x & 7, slot = threadIdx.x >> 3, warp = threadIdx.x >> 5,
              k = blockIdx.x * 8 + cc;
    const bool in = k < K;
    const double m = in && sub ? -sub[k] : 0.0;
    auto exponent = [&](double v) {
        if (sub) v = fma(v, s, m);
        return v != 0 && isfinite(v) ? exp_above(v) : INT_MIN;
    };
    // over the 32 threads of a warp that have a column in common
    auto warp_max = [](int e) {
        e = max(e, __shfl_xor_sync(0xffffffffu, e, 8));
        return max(e, __shfl_xor_sync(0xffffffffu, e, 16));
    };
    const int group = slot >> 3;                  // two warps
    const long r0 = rows * group / 16, r1 = min(r0 + 32, rows * (group + 1) / 16);
    int e = INT_MIN;
    double v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long r = r0 + (slot & 7) + 8 * i;
        // (NaN counts as nothing, also with a mean taken off)
        v[i] = in && r < r1 ? a[r * K + k] : __longlong_as_double(0x7ff8000000000000LL);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) e = max(e, exponent(v[i]));
    e = warp_max(e);
    if ((threadIdx.x & 31) < 8) sh[warp][cc] = e;
    __syncthreads();
    int sum = 0, n = 0;
    for (int q = 0; q < 32; q += 2) {
        e = max(sh[q][cc], sh[q + 1][cc]);
        if (e != INT_MIN) {
            sum += e;
            ++n;
        }
    }
    if (__syncthreads_or(in && n == 0 && rows > 512)) {
        e = INT_MIN;
        if (in)
#pragma unroll 8
            for (long r = slot; r < rows; r += 128) e = max(e, exponent(a[r * K + k]));
        e = warp_max(e);
        if ((threadIdx.x & 31) < 8) sh[warp][cc] = e;
        __syncthreads();
        if (n == 0) {
            for (int q = 0; q < 32; ++q) e = max(e, sh[q][cc]);
            if (e != INT_MIN) {
                sum = e;
                n = 1;
            }
        }
    }
    if (!in || slot) return;
    const double f = mul[k];
    int out = kZeroExp;
    if (n) {
        // (rounded, ties upwards; with a mean taken off, s is in what was looked at.  Within
        // what mul2 can hold.)
        const int t = 2 * sum + n, ef = exp_above(f);
        out = (t - (t < 0 ? 2 * n - 1 : 0)) / (2 * n) + ef - 1 + (sub ? 0 : exp_above(s) - 1);
        out = min(max(out, ef - 1000), ef + 1000);
    }
    ec[k] = out;
    mul2[k] = n ? ldexp(f, -out) : 0.0;
}

// Digits of the rows a' 2^-ec of k_prologue (real data), one warp per row, and the
// exponent above each row's maximum.  Rows past n (of the last tile) are zero.
__device__ __forceinline__ void dg_slice_rows(const double *__restrict__ a, long n, int K, int nkb, double s,
                                              const double *__restrict__ sub,
                                              const double *__restrict__ mul, __half *__restrict__ out,
                                              int *__restrict__ er) {
    const long r = blockIdx.x * 8L + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    const double *p = a + r * K;
    auto value = [&](int k) {
        double v = p[k] * s;
        if (sub) v -= sub[k];
        return v * mul[k];
    };
    int e = INT_MIN;
    if (r < n)
        for (int k = lane; k < K; k += 32) {
            const double v = value(k);
            if (v != 0) e = max(e, isfinite(v) ? exp_above(v) : kBadExp);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    if (e == INT_MIN) e = 0;
    const bool bad = e >= kBadExp / 2 || r >= n;
    if (lane == 0) er[r] = e;
    uint8_t *blk = reinterpret_cast<uint8_t *>(out) + (r / kGM) * nkb * kRes * (long)kGA;
    const int row = (int)(r % kGM);
    for (int ch = lane; ch < nkb * 8; ch += 32) {
        long long q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int m = ch * 8 + k;
            q[k] = m < K && !bad ? fixed_point(value(m), 55 - e) : 0;
        }
        uint4 w[kRes];
        digits8<kRes>(q, w);
#pragma unroll
        for (int d = 0; d < kRes; ++d)
            *reinterpret_cast<uint4 *>(blk + ((ch >> 3) * (long)kRes + d) * kGA +
                                       sw_place(row, ch & 7)) = w[d];
    }
}

// Digits of column c of b 2^ec (K x n), or of a column of padding, by a block
__device__ __forceinline__ void dg_slice_col(int c, const double *__restrict__ b,
                                             const int *__restrict__ ec, int K, int n, int nkb,
                                             __half *__restrict__ out, int *__restrict__ et) {
    __shared__ int sh[8];
    int e = INT_MIN;
    if (c < n)
        for (int k = threadIdx.x; k < K; k += blockDim.x) {
            const double v = b[(long)k * n + c];
            if (v != 0) e = max(e, isfinite(v) ? exp_above(v) + ec[k] : kBadExp);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = e;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; ++k) e = max(e, sh[k]);
    if (e == INT_MIN) e = 0;
    const bool bad = e >= kBadExp / 2 || c >= n;
    if (threadIdx.x == 0) et[c] = e;
    uint8_t *blk = reinterpret_cast<uint8_t *>(out) + (c / kGN) * nkb * (long)kCall * kGB;
    for (int ch = threadIdx.x; ch < nkb * 8; ch += blockDim.x) {
        long long q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int m = ch * 8 + k;
            q[k] = m < K && !bad ? fixed_point(b[(long)m * n + c], 62 + ec[m] - e) : 0;
        }
        uint4 w[kCall];
        digits8<kCall>(q, w);
#pragma unroll
        for (int d = 0; d < kCall; ++d)
            *reinterpret_cast<uint4 *>(blk + ((ch >> 3) * (long)kCall + d) * kGB +
                                       sw_place(c % kGN, ch & 7)) = w[d];
    }
}

// Both in one launch: eight rows a block, then the columns (up to a multiple of 64, or none)
__global__ void __launch_bounds__(256) k_dg_slice(const double *__restrict__ a, long rows, int row_blocks,
                                                  int K, int nkb, double s,
                                                  const double *__restrict__ sub,
                                                  const double *__restrict__ mul,
                                                  __half *__restrict__ outa, int *__restrict__ er,
                                                  const double *__restrict__ b,
                                                  const int *__restrict__ ec, int n,
                                                  __half *__restrict__ outb, int *__restrict__ et) {
    pdl_enter();
    if ((int)blockIdx.x < row_blocks)
        dg_slice_rows(a, rows, K, nkb, s, sub, mul, outa, er);
    else
        dg_slice_col(blockIdx.x - row_blocks, b, ec, K, n, nkb, outb, et);
}

// C (rows x n) = A' B by digit products: A' the rows of k_prologue, B K x n.  The
// digits of 2^16 rows at a time (14 bytes an element) beside those of B.  The columns of A'
// (coordinates) have scales of their own, which B's rows carry: atoms of unequal mass have
// displacements and forces of unequal size, and a mode of the smaller ones keeps its bits.
struct DigitProduct {
    void *slab = nullptr;
    __half *a = nullptr, *b = nullptr;
    int *er = nullptr, *et = nullptr, *ec = nullptr, *err = nullptr;
    double *mul2 = nullptr;
    int K = 0, n = 0, nkb = 0, nbt = 0, nsm = 1;
    long chunk = 0;
    long long budget = kDefaultBudget;
    ~DigitProduct() { cached_free(slab); }

    // false: the digits do not fit (the caller takes the CUDA-core product)
    bool init(long rows, int K_, int n_) {
        if (const char *e = getenv("TDSCHA_FP64_DIGITS"))
            if (atoi(e) == 0) return false;
        if (const char *e = getenv("TDSCHA_WAIT_BUDGET_CYCLES")) budget = atoll(e);
        K = K_;
        n = n_;
        nkb = ceil_div(K, kGK);
        nbt = ceil_div(n, kGN);
        chunk = std::min<long>(65536, (rows + kGM - 1) / kGM * kGM);
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        auto pad = [](size_t x) { return (x + 1023) & ~size_t(1023); };
        const size_t ba = (size_t)chunk * nkb * kGK * 2 * kRes, bb = (size_t)nbt * nkb * kCall * kGB,
                     be = pad(sizeof(int) * chunk), bt = pad(sizeof(int) * nbt * kGN),
                     bc = pad(sizeof(int) * K), bm = pad(sizeof(double) * K);
        if (cached_malloc(&slab, ba + bb + be + bt + bc + bm + 1024) != cudaSuccess) {
            cudaGetLastError();
            slab = nullptr;
            return false;
        }
        uint8_t *p = reinterpret_cast<uint8_t *>(slab);
        a = reinterpret_cast<__half *>(p);
        b = reinterpret_cast<__half *>(p + ba);
        er = reinterpret_cast<int *>(p + ba + bb);
        et = reinterpret_cast<int *>(p + ba + bb + be);
        ec = reinterpret_cast<int *>(p + ba + bb + be + bt);
        mul2 = reinterpret_cast<double *>(p + ba + bb + be + bt + bc);
        err = reinterpret_cast<int *>(p + ba + bb + be + bt + bc + bm);
        return true;
    }

    int begin() {
        TDS_CUDA(cudaMemsetAsync(err, 0, sizeof(int), 0));
        TDS_CUDA((dg_setup<DG_STORE, false>()));
        return TDSCHA_OK;
    }

    int product(const double *A, long rows, double s, const double *sub, const double *mul,
                const double *B, double *C) {
        const cudaStream_t st = 0;
        TDS_CUDA(launch_pdl(k_dg_colscale, ceil_div(K, 8), 1024, 0, st, A, rows, K, s, sub, mul, mul2, ec));
        for (long r0 = 0; r0 < rows; r0 += chunk) {
            const long nr = std::min(chunk, rows - r0), nrp = (nr + kGM - 1) / kGM * kGM;
            const int rb = (int)(nrp / 8);
            TDS_CUDA(launch_pdl(k_dg_slice, rb + (r0 ? 0 : nbt * kGN), 256, 0, st, A + r0 * K, nr, rb, K, nkb, s,
                                sub, (const double *)mul2, a, er, B, (const int *)ec, n, b, et));
            DgArgs g{};
            g.a = a;
            g.b = b;
            g.nkb = g.kbps = nkb;
            g.flush = kFlushMin;
            g.nat = (int)(nrp / kGM);
            g.nbt = nbt;
            g.nitems = (long)g.nat * nbt;
            g.err = err;
            g.budget = budget;
            g.et = et;
            g.er = er;
            g.R = nr;
            g.M = n;
            g.out = C + r0 * n;
            TDS_CUDA((dg_launch<DG_STORE, false>(g, nsm, st)));
        }
        return TDSCHA_OK;
    }

    int status() {
        int v = 0;
        TDS_CUDA(cudaMemcpy(&v, err, sizeof(int), cudaMemcpyDeviceToHost));
        if (!v) return TDSCHA_OK;
        set_error("tensor-core pipeline: a bounded wait expired (code %d)", v);
        return TDSCHA_ERR_TIMEOUT;
    }
};

// Perm-average: out[r][s] = mean_R D[perm_R[r]][perm_R[s]]
__global__ void k_perm_average(const double *__restrict__ D, const int *__restrict__ perms,
                               int n_trans, int n, double *__restrict__ out) {
    long total = (long)n * n;
    const double inv = 1.0 / n_trans;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
        int r = (int)(e / n), s = (int)(e % n);
        double acc = 0;
        for (int t = 0; t < n_trans; ++t) {
            const int *p = perms + (long)t * n;
            acc += D[(long)p[r] * n + p[s]];
        }
        out[e] = acc * inv;
    }
}

// Q[r][mu] = mean_R pols[perm_R[r]][mu]
__global__ void k_perm_rows(const double *__restrict__ pols, const int *__restrict__ perms,
                            int n_trans, int n, int M, double *__restrict__ Q) {
    long total = (long)n * M;
    const double inv = 1.0 / n_trans;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
        int r = (int)(e / M), mu = (int)(e % M);
        double acc = 0;
        for (int t = 0; t < n_trans; ++t) acc += pols[(long)perms[(long)t * n + r] * M + mu];
        Q[e] = acc * inv;
    }
}

// y = P x (M x M, row-major)
__global__ void k_matvec(const double *__restrict__ P, const double *__restrict__ x, int M,
                         double *__restrict__ y) {
    int i = blockIdx.x;
    __shared__ double sh[32];
    double acc = 0;
    for (int k = threadIdx.x; k < M; k += blockDim.x) acc = fma(P[(long)i * M + k], x[k], acc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
        y[i] = s;
    }
}

// gamma_only projection of ctx->f and ctx->d2v in place (device, stream ordered)
int apply_translation_projection(tdscha_ctx *c, cudaStream_t st) {
    const int M = c->M, n = c->tr_ncart;
    // f <- P_t f
    k_matvec<<<M, 128, 0, st>>>(c->tr_proj, c->f, M, c->tr_f);
    TDS_CHECK_LAUNCH();
    TDS_CUDA(cudaMemcpyAsync(c->f, c->tr_f, sizeof(double) * M, cudaMemcpyDeviceToDevice, st));
    // T1 = pols . d2v (n x M); D = T1 . pols^T (n x n)
    TDS_TRY(gemm<RealOps>(c->tr_pols, c->d2v, c->tr_w1, n, M, M, M, 1, M, 1, M, st));
    TDS_TRY(gemm<RealOps>(c->tr_w1, c->tr_pols, c->tr_w2, n, n, M, M, 1, 1, M, n, st));
    int nb = std::max(1, std::min(ceil_div((long)n * n, 256), 152 * 8));
    k_perm_average<<<nb, 256, 0, st>>>(c->tr_w2, c->tr_perms, c->tr_ntrans, n, c->tr_w3);
    TDS_CHECK_LAUNCH();
    // T2 = pols^T . Davg (M x n); d2v = T2 . pols (M x M)
    TDS_TRY(gemm<RealOps>(c->tr_pols, c->tr_w3, c->tr_w1, M, n, n, 1, M, n, 1, n, st));
    TDS_TRY(gemm<RealOps>(c->tr_w1, c->tr_pols, c->d2v, M, M, n, n, 1, M, 1, M, st));
    return TDSCHA_OK;
}

void free_translations(tdscha_ctx *c) {
    double *bufs[] = {c->tr_pols, c->tr_proj, c->tr_w1, c->tr_w2, c->tr_w3, c->tr_f};
    for (double *b : bufs)
        if (b) cudaFree(b);
    if (c->tr_perms) cudaFree(c->tr_perms);
    c->tr_pols = c->tr_proj = c->tr_w1 = c->tr_w2 = c->tr_w3 = c->tr_f = nullptr;
    c->tr_perms = nullptr;
    c->tr_ntrans = 0;
    c->tr_ncart = 0;
}

}  // namespace tdscha

using namespace tdscha;

extern "C" int tdscha_project_modes(int N, int n_cart, int M, const double *u, const double *f,
                                    const double *f_mean, const double *masses,
                                    const double *pols, double u_scale, double f_scale,
                                    double *X_out, double *Y_out) {
    set_error("");
    if (N <= 0 || n_cart <= 0 || M <= 0 || !u || !f || !masses || !pols || !X_out || !Y_out) {
        set_error("project_modes: bad arguments");
        return TDSCHA_ERR_ARG;
    }
    std::vector<double> sq(n_cart), isq(n_cart), sub;
    for (int k = 0; k < n_cart; ++k) {
        if (!(masses[k] > 0)) { set_error("project_modes: masses must be positive"); return TDSCHA_ERR_ARG; }
        sq[k] = std::sqrt(masses[k]);
        isq[k] = 1.0 / sq[k];
    }
    if (f_mean) {
        sub.resize(n_cart);
        for (int k = 0; k < n_cart; ++k) sub[k] = f_mean[k] * f_scale;
    }
    size_t nu = (size_t)N * n_cart, nx = (size_t)N * M;
    double *d_in = nullptr, *d_tmp = nullptr, *d_pols = nullptr, *d_out = nullptr, *d_vec = nullptr;
    // blocks of the process-wide cache: five cudaMalloc and cudaFree of an
    // ensemble's size cost as much as the product
    auto done = [&](int rc) {
        if (rc != TDSCHA_OK) cudaDeviceSynchronize();
        double *b[] = {d_in, d_tmp, d_pols, d_out, d_vec};
        for (double *p : b) cached_free(p);
        return rc;
    };
#define PCU(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) { set_error("%s: %s", #x, cudaGetErrorString(_e)); return done(TDSCHA_ERR_CUDA); } } while (0)
    DigitProduct dg;
    const bool digits = dg.init(N, n_cart, M);
    PCU(cached_malloc(&d_in, sizeof(double) * nu));
    if (!digits) PCU(cached_malloc(&d_tmp, sizeof(double) * nu));
    PCU(cached_malloc(&d_pols, sizeof(double) * (size_t)n_cart * M));
    PCU(cached_malloc(&d_out, sizeof(double) * nx));
    PCU(cached_malloc(&d_vec, sizeof(double) * 3 * n_cart));
    PCU(cudaMemcpy(d_pols, pols, sizeof(double) * (size_t)n_cart * M, cudaMemcpyHostToDevice));
    PCU(cudaMemcpy(d_vec, sq.data(), sizeof(double) * n_cart, cudaMemcpyHostToDevice));
    PCU(cudaMemcpy(d_vec + n_cart, isq.data(), sizeof(double) * n_cart, cudaMemcpyHostToDevice));
    if (f_mean) PCU(cudaMemcpy(d_vec + 2 * n_cart, sub.data(), sizeof(double) * n_cart, cudaMemcpyHostToDevice));
    int nb = std::max(1, std::min(ceil_div((long)nu, 256), 152 * 8)), rc = TDSCHA_OK;
    if (digits && (rc = dg.begin()) != TDSCHA_OK) return done(rc);
    for (int pass = 0; pass < 2; ++pass) {
        PCU(cudaMemcpy(d_in, pass == 0 ? u : f, sizeof(double) * nu, cudaMemcpyHostToDevice));
        const double scale = pass == 0 ? u_scale : f_scale;
        const double *sub = pass == 1 && f_mean ? d_vec + 2 * n_cart : nullptr;
        const double *mul = pass == 0 ? d_vec : d_vec + n_cart;
        if (digits) {
            rc = dg.product(d_in, N, scale, sub, mul, d_pols, d_out);
        } else {
            k_prologue<<<nb, 256>>>(d_in, N, n_cart, 1, scale, sub, mul, d_tmp);
            PCU(cudaGetLastError());
            rc = gemm<RealOps>(d_tmp, d_pols, d_out, N, M, n_cart, n_cart, 1, M, 1, M, 0);
        }
        if (rc != TDSCHA_OK) return done(rc);
        PCU(cudaMemcpy(pass == 0 ? X_out : Y_out, d_out, sizeof(double) * nx, cudaMemcpyDeviceToHost));
    }
    if (digits && (rc = dg.status()) != TDSCHA_OK) return done(rc);
#undef PCU
    return done(TDSCHA_OK);
}

extern "C" int tdscha_project_bloch(int n_q, int N, int n_cart, int nb, const double *u_q,
                                    const double *f_q, const double *f_mean_gamma,
                                    const double *masses, const double *pols_q, double u_scale,
                                    double f_scale, double *X_q, double *Y_q) {
    set_error("");
    if (n_q <= 0 || N <= 0 || n_cart <= 0 || nb <= 0 || !u_q || !f_q || !masses || !pols_q || !X_q || !Y_q) {
        set_error("project_bloch: bad arguments");
        return TDSCHA_ERR_ARG;
    }
    // layouts: u_q, f_q (n_q, N, n_cart) complex; pols_q (n_q, n_cart, nb) complex;
    // X_q, Y_q (n_q, N, nb) complex; f_mean_gamma (n_cart) complex or NULL
    std::vector<double> sq(n_cart), isq(n_cart);
    for (int k = 0; k < n_cart; ++k) {
        if (!(masses[k] > 0)) { set_error("project_bloch: masses must be positive"); return TDSCHA_ERR_ARG; }
        sq[k] = std::sqrt(masses[k]);
        isq[k] = 1.0 / sq[k];
    }
    size_t nu = (size_t)n_q * N * n_cart, nx = (size_t)n_q * N * nb, npol = (size_t)n_q * n_cart * nb;
    double2 *d_in = nullptr, *d_tmp = nullptr, *d_pols = nullptr, *d_out = nullptr;
    double *d_vec = nullptr;
    auto done = [&](int rc) {
        void *b[] = {d_in, d_tmp, d_pols, d_out, d_vec};
        for (void *p : b) if (p) cudaFree(p);
        return rc;
    };
#define PCU(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) { set_error("%s: %s", #x, cudaGetErrorString(_e)); return done(TDSCHA_ERR_CUDA); } } while (0)
    PCU(cudaMalloc(&d_in, sizeof(double2) * nu));
    PCU(cudaMalloc(&d_tmp, sizeof(double2) * nu));
    PCU(cudaMalloc(&d_pols, sizeof(double2) * npol));
    PCU(cudaMalloc(&d_out, sizeof(double2) * nx));
    PCU(cudaMalloc(&d_vec, sizeof(double) * 4 * n_cart));
    PCU(cudaMemcpy(d_pols, pols_q, sizeof(double2) * npol, cudaMemcpyHostToDevice));
    PCU(cudaMemcpy(d_vec, sq.data(), sizeof(double) * n_cart, cudaMemcpyHostToDevice));
    PCU(cudaMemcpy(d_vec + n_cart, isq.data(), sizeof(double) * n_cart, cudaMemcpyHostToDevice));
    if (f_mean_gamma) PCU(cudaMemcpy(d_vec + 2 * n_cart, f_mean_gamma, sizeof(double) * 2 * n_cart, cudaMemcpyHostToDevice));
    int nbk = std::max(1, std::min(ceil_div((long)nu * 2, 256), 152 * 8));
    for (int pass = 0; pass < 2; ++pass) {
        PCU(cudaMemcpy(d_in, pass == 0 ? u_q : f_q, sizeof(double2) * nu, cudaMemcpyHostToDevice));
        if (pass == 0) {
            k_prologue<<<nbk, 256>>>((const double *)d_in, (long)n_q * N, n_cart, 2, u_scale, nullptr,
                                     d_vec, (double *)d_tmp);
        } else {
            // (f - f_mean) * f_scale / sqrt(m): the mean is subtracted at Gamma (q index 0) only
            k_prologue<<<nbk, 256>>>((const double *)d_in, (long)n_q * N, n_cart, 2, 1.0, nullptr,
                                     d_vec + n_cart, (double *)d_tmp);
            if (f_mean_gamma) {
                // Gamma rows: redo with the mean subtracted, scale folded as (f - g) / sqrt(m)
                k_prologue<<<nbk, 256>>>((const double *)d_in, (long)N, n_cart, 2, 1.0, d_vec + 2 * n_cart,
                                         d_vec + n_cart, (double *)d_tmp);
            }
        }
        PCU(cudaGetLastError());
        int rc = gemm<CplxConjBOps>(d_tmp, d_pols, d_out, N, nb, n_cart, n_cart, 1, nb, 1, nb, 0, n_q,
                                    (long)N * n_cart, (long)n_cart * nb, (long)N * nb);
        if (rc != TDSCHA_OK) return done(rc);
        PCU(cudaMemcpy(pass == 0 ? X_q : Y_q, d_out, sizeof(double2) * nx, cudaMemcpyDeviceToHost));
        if (pass == 1 && f_scale != 1.0) {
            for (size_t e = 0; e < 2 * nx; ++e) Y_q[e] *= f_scale;
        }
    }
#undef PCU
    return done(TDSCHA_OK);
}

extern "C" int tdscha_ctx_set_translations(tdscha_ctx *ctx, int n_cart, const double *pols,
                                           int n_trans, const int *perms) {
    set_error("");
    if (!ctx) { set_error("ctx_set_translations: null context"); return TDSCHA_ERR_ARG; }
    cudaDeviceSynchronize();
    free_translations(ctx);
    if (n_trans == 0) return TDSCHA_OK;
    const int M = ctx->M;
    if (n_cart < M || n_trans < 0 || !pols || !perms) { set_error("ctx_set_translations: bad arguments"); return TDSCHA_ERR_ARG; }
    for (long e = 0; e < (long)n_trans * n_cart; ++e)
        if (perms[e] < 0 || perms[e] >= n_cart) { set_error("ctx_set_translations: permutation index out of range"); return TDSCHA_ERR_ARG; }
    const int n = n_cart;
    ctx->tr_ncart = n;
    ctx->tr_ntrans = n_trans;
    TDS_CUDA(cudaMalloc(&ctx->tr_pols, sizeof(double) * (size_t)n * M));
    TDS_CUDA(cudaMalloc(&ctx->tr_perms, sizeof(int) * (size_t)n_trans * n));
    TDS_CUDA(cudaMalloc(&ctx->tr_proj, sizeof(double) * (size_t)M * M));
    TDS_CUDA(cudaMalloc(&ctx->tr_w1, sizeof(double) * (size_t)n * std::max(n, M)));
    TDS_CUDA(cudaMalloc(&ctx->tr_w2, sizeof(double) * (size_t)n * n));
    TDS_CUDA(cudaMalloc(&ctx->tr_w3, sizeof(double) * (size_t)n * n));
    TDS_CUDA(cudaMalloc(&ctx->tr_f, sizeof(double) * M));
    TDS_CUDA(cudaMemcpy(ctx->tr_pols, pols, sizeof(double) * (size_t)n * M, cudaMemcpyHostToDevice));
    TDS_CUDA(cudaMemcpy(ctx->tr_perms, perms, sizeof(int) * (size_t)n_trans * n, cudaMemcpyHostToDevice));
    // P_t = pols^T (mean_R P_R pols) (the reference's trans_projector, :764-785)
    int nb = std::max(1, std::min(ceil_div((long)n * M, 256), 152 * 8));
    k_perm_rows<<<nb, 256>>>(ctx->tr_pols, ctx->tr_perms, n_trans, n, M, ctx->tr_w2);
    TDS_CUDA(cudaGetLastError());
    TDS_TRY(gemm<RealOps>(ctx->tr_pols, ctx->tr_w2, ctx->tr_proj, M, M, n, 1, M, M, 1, M, 0));
    TDS_CUDA(cudaDeviceSynchronize());
    return TDSCHA_OK;
}
