// Exact digit products: splitting float64 numbers into digits, the tensor-core
// contraction over digit operands, and the way back to float64.  perturb_digits.cu
// explains the arithmetic.
#pragma once

#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "tcgen05.cuh"

namespace tdscha {

constexpr int kGM = 128;        // rows of an A tile: TMEM lanes
constexpr int kGN = 64;         // rows of a B tile: columns of each order's accumulator
constexpr int kGK = 64;         // K block: one 128-byte swizzle row of fp16
constexpr int kRes = 7;         // digits of the resident operand
constexpr int kCall = 8;        // digits of the operand made per call
constexpr int kOrders = 8;      // orders kept: 8 x 64 accumulator columns fill the TMEM
constexpr int kFlushMin = 3;    // K blocks per accumulation, exact for any input
constexpr int kFlushMax = 9;
constexpr int kFlushes = kFlushMax - kFlushMin + 1;
constexpr int kUnit = -69;      // one unit of the order-7 accumulator: 2^(-7-6-56)
constexpr int kBadExp = 1 << 20;   // exponent of a row with a non-finite element
constexpr int kZeroExp = -8192;    // of a row of zeros: 2^kZeroExp counts as 0
constexpr uint32_t kGA = kGM * kGK * 2;   // bytes of one digit of an A block
constexpr uint32_t kGB = kGN * kGK * 2;   // and of a B block

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

__device__ __forceinline__ double2 dg_two(const double *p) {
    return *reinterpret_cast<const double2 *>(p);
}

// (hi 2^32 + lo) 2^e as float64, |hi| < 2^62, rounded to nearest to within 2^-60
// of itself or one unit of lo.  About 25 whole-number operations: a conversion of
// a 64-bit integer, like every float64 operation, runs at two per cycle per SM.
__device__ __forceinline__ double fixed_to_double(long long hi, long long lo, int e) {
    const long long h = hi + (lo >> 32);      // what remains of lo is in [0, 2^32)
    const uint32_t sgn = (uint32_t)(h >> 63);
    // magnitude, three words (of a negative number one unit too small)
    const uint32_t w2 = (uint32_t)((unsigned long long)h >> 32) ^ sgn, w1 = (uint32_t)h ^ sgn,
                   w0 = (uint32_t)lo ^ sgn;
    const bool k0 = w2 != 0u, k1 = w1 != 0u;
    const uint32_t a = k0 ? w2 : k1 ? w1 : w0, b = k0 ? w1 : k1 ? w0 : 0u, c = k0 ? w0 : 0u;
    const int z = __clz((int)a);
    // the leading 64 bits, then 53 of them
    const uint32_t th = __funnelshift_l(b, a, z), tl = __funnelshift_l(c, b, z);
    const uint64_t m = (((uint64_t)th << 32 | tl) >> 11) + ((tl >> 10) & 1u);
    // one less than the exponent field: the leading bit of m adds one
    const int E = 1074 + 43 + e - z - (k0 ? 0 : k1 ? 32 : 64);
    uint64_t bits = ((uint64_t)(uint32_t)E << 52) + m;
    if (a == 0u || (uint32_t)E >= 2046u) {
        bits = 0u;
        if (e >= kBadExp / 2)
            bits = 0x7ff8000000000000ULL;
        else if (a != 0u && E >= 2046)
            bits = 0x7ff0000000000000ULL;
    }
    return __longlong_as_double((long long)(bits | ((uint64_t)(sgn & 0x80000000u) << 32)));
}

// 2^e for the exponents of finite float64 rows (0 below the normal numbers)
__device__ __forceinline__ double pow2(int e) {
    return __longlong_as_double((long long)(e < -1022 ? 0 : min(e + 1023, 2047)) << 52);
}

// What a configuration's elements count for in the scales of their columns beside their
// exponents: what its weight is below the largest one (exponent rtop), if that is much.
// With every weight counted, ordinary configurations would lie outside by a bit or two.
__device__ __forceinline__ int dg_weight_exp(double rho, int rtop) {
    const int e = exp_above(rho) - rtop;
    return rho == 0 ? INT_MIN / 2 : e < -8 ? e : 0;
}

// Sums of the squares of each digit over the 64 elements of a block's row, from
// the eight lanes that hold it: nrm[digit * rows + row].
__device__ __forceinline__ void digit_norms(const uint4 (&w)[kRes], int c, float *__restrict__ nrm,
                                            int rows, int row) {
#pragma unroll
    for (int d = 0; d < kRes; ++d) {
        const uint32_t v[4] = {w[d].x, w[d].y, w[d].z, w[d].w};
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&v[k]));
            s = fmaf(f.x, f.x, fmaf(f.y, f.y, s));
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (c == 0) nrm[d * rows + row] = s;
    }
}

// out[L - 3][digit]: largest norm (squared) of any row over any L = 3 + blockIdx.y blocks
// that follow one another (a split of the contraction may start at any block);
// nrm[tile][block][digit][rows], thread = row, kWindowStarts first blocks a block.  The sums
// are whole numbers up to 9 2^20, exact in fp32.
constexpr int kWindowStarts = 32;
static __global__ void k_dg_windows(const float *__restrict__ nrm, int nkb, float *__restrict__ out) {
    const int L = kFlushMin + blockIdx.y, s0 = blockIdx.z * kWindowStarts,
              s1 = min(s0 + kWindowStarts, max(1, nkb - L + 1));
    if (s0 >= s1) return;
    const long step = (long)kRes * blockDim.x;
    const float *p = nrm + (blockIdx.x * (long)nkb + s0) * step + threadIdx.x, *q = p;
    float s[kRes] = {}, mx[kRes];
    for (int k = s0; k < min(nkb, s0 + L); ++k, q += step)
#pragma unroll
        for (int d = 0; d < kRes; ++d) s[d] += q[d * blockDim.x];
#pragma unroll
    for (int d = 0; d < kRes; ++d) mx[d] = s[d];
#pragma unroll 4
    for (int k = s0 + 1; k < s1; ++k, p += step, q += step)
#pragma unroll
        for (int d = 0; d < kRes; ++d) {
            s[d] += q[d * blockDim.x] - p[d * blockDim.x];
            mx[d] = fmaxf(mx[d], s[d]);
        }
#pragma unroll
    for (int d = 0; d < kRes; ++d) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx[d] = fmaxf(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        // non-negative floats order like their bit patterns
        if ((threadIdx.x & 31) == 0)
            atomicMax(reinterpret_cast<int *>(out + blockIdx.y * kRes + d), __float_as_int(mx[d]));
    }
}

// (nkb <= 65535 kWindowStarts, over a hundred million rows)
inline cudaError_t dg_windows(const float *nrm, int tiles, int rows, int nkb, float *out, cudaStream_t st) {
    k_dg_windows<<<dim3(tiles, kFlushes, ceil_div(nkb, kWindowStarts)), rows, 0, st>>>(nrm, nkb, out);
    return cudaGetLastError();
}

// The longest accumulation (K blocks) that keeps orders 0..4 below 2^24 for any
// per-call operand: mx[L - 3][i] is the largest squared norm of digit i over L
// blocks.  The other operand's digits are at most 64 (the first) and 128.
inline int digits_flush(const float *mx) {
    for (int L = kFlushMax; L > kFlushMin; --L) {
        bool fits = true;
        for (int o = 0; o <= 4 && fits; ++o) {
            double sum = 0;
            for (int i = 0; i <= o; ++i)
                sum += std::sqrt((double)mx[(L - kFlushMin) * kRes + i] * kGK * L) *
                       (i == o ? 64.0 : 128.0);
            fits = sum <= 16777216.0;
        }
        if (fits) return L;
    }
    return kFlushMin;
}

// K blocks per split of a split-K contraction (of nkb blocks, accumulations of
// `flush`) with `nat` A and `nbt` B tiles on `nsm` SMs: the fewest waves weighted
// with what a wave costs: 4900 cycles a K block (35 products of 128 x 64 x 64 at
// 4096 a cycle, and a tenth), 8000 to fill the ring and to write the tile; and the
// partial tiles written and read again (both at about 3 KB a cycle).
inline int dg_blocks_per_split(long nkb, int flush, int nat, int nbt, int nsm) {
    const long tiles = (long)nat * nbt;
    const double part = 16.0 * tiles * kGM * kGN / 3000.0;
    double best = 1e300;
    int kb_best = (int)nkb;
    for (long n = 1; n <= std::min<long>(nkb, 96); ++n) {
        long kb = (nkb + n - 1) / n;
        // whole accumulations where a split has several
        if (kb > flush) kb = (kb + flush - 1) / flush * flush;
        const long ns = (nkb + kb - 1) / kb;
        if (kb > 16384) continue;             // 64-bit sums of the orders
        const double cost = (double)((tiles * ns + nsm - 1) / nsm) * (kb * 4900.0 + 8000.0) + part * ns;
        if (cost < best * 0.999) {
            best = cost;
            kb_best = (int)kb;
        }
    }
    return kb_best;
}

// -------------------------------------------------------- the contraction
// Persistent, one CTA per SM, one 128 x 64 output tile at a time; its accumulators,
// eight orders of 64 columns, fill the TMEM.
//   warps 0-15  every `flush` K blocks the accumulators are read, order 7 first, and
//           added to two 64-bit integers an element (warp w: lanes 32 (w % 4), columns
//           16 (w / 4) of every order).  Each order has its own release, so the MMAs of
//           the next blocks start on order 7 while the lower ones are still read.  At
//           the end of a tile the sums become float64: row dots, a partial tile or a
//           product.
//   warp 16  copies: B blocks (all digits of 64 rows) into two buffers, A digits
//           (128 rows each) into a ring
//   warp 17  MMA issue: A digit i against the B digits 0 .. 7 - i at once, which
//           lie behind one another in shared memory as their accumulators do in
//           TMEM, so one instruction covers up to four orders (N = 256).  i
//           runs downwards: the light high orders come first.
//   warps 20-23  (row dots of the real-space stage A) s and t
// Bounded waits and the abort flag as in perturb_mixed.cu.
//
// What it takes at M=573, N=50000 (1.95 GHz): stage A 673 us, stage B 759 us; the
// 35 products alone are 0.93 and 1.04 million cycles an SM, 480 and 530 us.  The
// same loop on one thread (`if (lane == 0)`) took 794 and 928 us, with 64-bit
// divisions for the ring slots 1165 and 1098.  Reading an accumulation back takes
// the sixteen epilogue warps 6300 cycles, of which the next products wait for about
// 2900 (eight warps of 32 columns: 8000); the end of a tile with row dots 12 000 to
// 15 000: two float64 products an element, and as many for s and t beside them.  With
// 48 images at M=189, N=10000 stage A (783 us) is bound by that and the reading back,
// 20 000 cycles a tile against 13 400 of products.  The copies (176 KB a K block) take
// 3700 cycles of a block's 4500 and do not show.
// What becomes of a tile: row dots (stage A), split-K partials (stage B), the
// product itself, or the complex row dots of Bloch space (qspace_digits.cu)
enum { DG_DOTS = 0, DG_PARTS, DG_STORE, DG_QDOTS };

struct DgArgs {
    const __half *a, *b;
    int nkb;               // K blocks of an operand row
    int kbps;              // K blocks per work item (stage A: nkb)
    int flush;             // K blocks per accumulation
    int nat, nbt;          // A and B tiles
    // tiles that are partly empty:
    int kk;                // 16-element steps of a K block
    int hc;                // columns of an epilogue warp: 16, or 12, 8, 4 of narrower tiles
    int win;               // work items that share a tile: each ends its own 4 hc columns
    uint32_t abytes;       // bytes of one digit of an A block: kGA, or 1024 for every eight
                           // rows of tiles with fewer (the others stay zero in shared memory)
    // B tile of work item (at, bt): bt, or bmap[at] + bt.  The A tile is at (Bloch-space
    // dots: bt nat + at)
    const int *bmap;
    long nitems;
    int Mp;
    int *err;              // failure code, for the host
    int *failed;           // set with it, for the kernels that end the call (or null)
    long long budget;
    // stage A
    const double *dt, *gt, *vs, *vt;
    const int *et;
    double *qp;            // [image][column tile][4][R]
    long R;
    int nct;               // column tiles of one image
    const int *cofs;       // Bloch-space dots: 4 o + kind of a tile column, whose x and g
    int nr;                // begin at column (of 128 rows) o + nr x row tile of dt and gt
    // stage B
    const int *ec, *ew;
    double *gpart;         // [split][A rows][Mp]: H[b][a]
    int M;                 // columns in use (of an image)
    int rmod, rlive;       // of the A rows, those with row % rmod < rlive ...
    long rows_b;           // ... and row < rows_b are in use
    // product: out[R][M], row exponents er (also of the Bloch-space dots, by A tile)
    const int *er;
    double *out;
};

// hc where `cols` of a tile's columns are in use: a quarter of them, in fours (Bloch-space
// averages with 12 bands, 48 columns of a tile: 538 us with three warps of 16, 530 so)
inline int dg_part_cols(int cols) { return std::min(16, (cols + 15) / 16 * 4); }

constexpr int kEpi = 16;           // epilogue warps

template <int kMode>
struct DgShape {
    static constexpr bool wide = kMode == DG_PARTS;    // 8 digits of A, 7 of B
    static constexpr int SA = wide ? kCall : kRes, SB = wide ? kRes : kCall;
    static constexpr int slots = wide ? 6 : 5;         // A ring: with the B buffers 208 KB
    static constexpr uint32_t bbytes = SB * kGB;
    static constexpr int bars = 2 * slots + 4 + 1 + kOrders + 1;
    static constexpr size_t ring = 2 * (size_t)bbytes + slots * (size_t)kGA;
    // registers: 61440 at launch, of which the epilogue takes the larger share
    static constexpr int threads = 32 * (kEpi + (kMode == DG_DOTS ? 8 : 4));
    static constexpr int regs = 61440 / threads, epi = kMode == DG_DOTS ? 96 : 104,
                         rest = kMode == DG_DOTS ? 48 : 64;
    static_assert(32 * kEpi * epi + (threads - 32 * kEpi) * rest == threads * regs, "register shares");
    static constexpr int sums = kMode == DG_QDOTS ? 4 : 2;      // of a row
    static constexpr size_t smem = 1024 + ring + 3 * sums * 128 * sizeof(double) +
                                   4 * kGN * sizeof(int) + 8 * bars + 16;
};
static_assert(DgShape<DG_QDOTS>::smem <= 232448 && DgShape<DG_PARTS>::smem <= 232448,
              "shared memory above the per-block limit");

// Named barrier 1 over the 512 epilogue threads; true if `pred` was set in any.
__device__ __forceinline__ bool dg_sync_or(bool pred) {
    uint32_t out;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, 1, 512, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(out)
        : "r"((uint32_t)pred)
        : "memory");
    return out != 0;
}

// kPart: tiles that are partly empty (kk, hc, abytes), the sizes of a full tile are
// constants otherwise (read from the arguments they cost the M=573 call 3%)
template <int kMode, bool kPart>
__global__ void __launch_bounds__(DgShape<kMode>::threads, 1) k_dg_gemm(const DgArgs args) {
    const int hc = kPart ? args.hc : 16, win = kPart ? args.win : 1;
    const uint32_t abytes = kPart ? args.abytes : kGA;
    using Sh = DgShape<kMode>;
    constexpr int SA = Sh::SA, SB = Sh::SB, slots = Sh::slots;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *ring = smem + 2 * Sh::bbytes;
    double *red = reinterpret_cast<double *>(smem + Sh::ring);   // [sum][3][128]
    int *cole = reinterpret_cast<int *>(red + 3 * Sh::sums * 128);   // [2][64], offsets [2][64]
    uint64_t *bars = reinterpret_cast<uint64_t *>(cole + 4 * kGN);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + Sh::bars);
    volatile int *abort = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const uint32_t afull = smem_u32(bars), aempty = afull + 8 * slots, bfull = aempty + 8 * slots,
                   bempty = bfull + 16, tfull = bempty + 16, tempty = tfull + 8,
                   done = tempty + 8 * kOrders;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long budget = args.budget;

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
        for (int o = 0; o < kOrders; ++o) mbar_init(tempty + 8 * o, kEpi);
        mbar_init(done, 1);
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (kPart && abytes < kGA) {
        for (uint32_t o = 16 * threadIdx.x; o < slots * kGA; o += 16 * Sh::threads)
            *reinterpret_cast<uint4 *>(ring + o) = make_uint4(0, 0, 0, 0);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == kEpi + 1) tmem_alloc<512>(smem_u32(tmem_slot));
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_enter();
    int fail_code = 0;

    // Work items blockIdx.x, blockIdx.x + gridDim.x, ...: neighbouring CTAs take
    // neighbouring B tiles of one A tile (stage A) or of one split (stage B) and
    // share it in L2.  Stepped, not divided: 64-bit divisions between two blocks
    // held the issue thread up for longer than its MMAs run.
    struct Item {
        int at, bt, split, left;
        int step_at, step_bt, step_split, nat, nbt;
        __device__ Item(const DgArgs &a) {
            const int w = (int)blockIdx.x, g = (int)gridDim.x;
            nat = a.nat;
            nbt = a.nbt;
            bt = w % nbt;
            at = w / nbt % nat;
            split = w / nbt / nat;
            step_bt = g % nbt;
            step_at = g / nbt % nat;
            step_split = g / nbt / nat;
            left = a.nitems > w ? (int)((a.nitems - 1 - w) / g) + 1 : 0;
        }
        __device__ void next() {
            bt += step_bt;
            at += step_at;
            split += step_split;
            if (bt >= nbt) {
                bt -= nbt;
                ++at;
            }
            if (at >= nat) {
                at -= nat;
                ++split;
            }
            --left;
        }
    };
    auto a_tile = [&](const Item &w) { return kMode == DG_QDOTS ? w.bt * args.nat + w.at : w.at; };
    auto b_tile = [&](const Item &w) { return args.bmap ? args.bmap[w.at] + w.bt : kPart ? w.bt / win : w.bt; };
    // a ring's slot and the parity of its use
    struct Cursor {
        int s = 0;
        uint32_t ph = 0;
        __device__ void next(int n) {
            if (++s == n) {
                s = 0;
                ph ^= 1;
            }
        }
    };

    if (warp >= kEpi) {
    regs_dec<Sh::rest>();
    if (warp == kEpi) {
        if (lane == 0) {
            Cursor ca, cb;
            long ga = 0, gb = 0;             // copies issued
            for (Item w(args); w.left > 0 && !fail_code; w.next()) {
                const int kb0 = w.split * args.kbps, nkb = min(args.kbps, args.nkb - kb0);
                const uint8_t *pa = reinterpret_cast<const uint8_t *>(args.a) +
                                    ((long)a_tile(w) * args.nkb + kb0) * SA * (long)abytes;
                const uint8_t *pb = reinterpret_cast<const uint8_t *>(args.b) +
                                    ((long)b_tile(w) * args.nkb + kb0) * SB * (long)kGB;
                for (int kb = 0; kb < nkb && !fail_code; ++kb) {
                    if (gb >= 2 && !mbar_wait_ab(bempty + 8 * cb.s, cb.ph ^ 1, budget, abort)) {
                        fail_code = 1;
                        break;
                    }
                    mbar_expect_tx(bfull + 8 * cb.s, Sh::bbytes);
#pragma unroll
                    for (int d = 0; d < SB; ++d)
                        bulk_load(smem_u32(smem + cb.s * Sh::bbytes + d * kGB), pb + d * kGB, kGB,
                                  bfull + 8 * cb.s);
                    pb += SB * (long)kGB;
                    cb.next(2);
                    ++gb;
                    for (int d = SA - 1; d >= 0; --d, ++ga) {
                        if (ga >= slots && !mbar_wait_ab(aempty + 8 * ca.s, ca.ph ^ 1, budget, abort)) {
                            fail_code = 1;
                            break;
                        }
                        mbar_expect_tx(afull + 8 * ca.s, abytes);
                        bulk_load(smem_u32(ring + ca.s * kGA), pa + d * (long)abytes,
                                  abytes, afull + 8 * ca.s);
                        ca.next(slots);
                    }
                    pa += SA * (long)abytes;
                }
            }
            if (fail_code) *abort = 1;
            // every issued copy must land before the CTA exits, also where it is another
            // role that has given up
            for (long g = ga > slots ? ga - slots : 0; g < ga; ++g)
                mbar_wait(afull + 8 * (int)(g % slots), (uint32_t)(g / slots) & 1, kDefaultBudget);
            for (long g = gb > 2 ? gb - 2 : 0; g < gb; ++g)
                mbar_wait(bfull + 8 * (int)(g & 1), (uint32_t)(g >> 1) & 1, kDefaultBudget);
        }
    } else if (warp == kEpi + 1) {
        {
            // the whole warp runs the loop, one lane issues
            const uint32_t one = elect_one();
            Cursor ca, cb;
            uint32_t nch = 0;                // accumulations so far
            // the next A digit, the next B block were seen to have landed
            bool ready = false, readyb = false;
            for (Item w(args); w.left > 0 && !fail_code; w.next()) {
                const int kb0 = w.split * args.kbps, nkb = min(args.kbps, args.nkb - kb0);
                int in = 0;                  // K blocks in this accumulation
                for (int kb = 0; kb < nkb && !fail_code; ++kb) {
                    const bool first = in == 0;
                    const int sb = cb.s;
                    if (!readyb && !mbar_all(bfull + 8 * sb, cb.ph, budget, abort)) {
                        fail_code = 2;
                        break;
                    }
                    cb.next(2);
                    const uint64_t db0 = sdesc_sw128(smem_u32(smem + sb * Sh::bbytes));
#pragma unroll
                    for (int d = SA - 1; d >= 0; --d) {
                        constexpr int kTop = SA - 1;
                        const int cnt = min(SB, kOrders - d);       // orders d .. d + cnt - 1
                        const int s = ca.s;
                        bool ok = ready || mbar_all(afull + 8 * s, ca.ph, budget, abort);
                        if (first && nch > 0) {
                            // the orders that this digit writes first: d, and at the
                            // top digit all of its orders
                            const uint32_t par = (nch - 1) & 1;
                            for (int o = d; o < (d == kTop ? d + cnt : d + 1); ++o)
                                ok = mbar_all(tempty + 8 * o, par, budget, abort) && ok;
                        }
                        if (!ok) {
                            fail_code = 2;
                            break;
                        }
                        ca.next(slots);
                        // the next digit's barrier is read while this digit's MMAs
                        // go out (a wait between two digits idled the tensor core
                        // for about 100 cycles)
                        ready = __all_sync(0xffffffffu, mbar_test(afull + 8 * ca.s, ca.ph));
                        if (d == 0) readyb = __all_sync(0xffffffffu, mbar_test(bfull + 8 * cb.s, cb.ph));
                        if (first) tc_fence_after();
                        const uint64_t da0 = sdesc_sw128(smem_u32(ring + s * kGA));
                        const uint32_t col = tmem + kGN * d;
                        // at most four orders (N = 256) an instruction
                        const int n1 = cnt > 4 ? (cnt + 1) / 2 : cnt;
#pragma unroll
                        for (int kk = 0; kk < kGK / 16; ++kk) {
                            if (kPart && kk >= args.kk) break;
                            // descriptor addresses count 16 bytes; the digits of B
                            // lie kGB apart
                            auto span = [&](int j0, int n, uint32_t acc) {
                                mma_f16_one(one, col + kGN * j0, da0 + 2 * kk,
                                        db0 + j0 * (kGB / 16) + 2 * kk, idesc_f16(kGM, kGN * n), acc);
                            };
                            if (kk == 0 && first) {
                                // order d starts here, the higher ones go on; at the
                                // top digit (at most two orders) all of them start
                                if (d == kTop) {
                                    span(0, cnt, 0u);
                                } else {
                                    span(0, 1, 0u);
                                    span(1, min(4, cnt - 1), 1u);
                                    if (cnt > 5) span(5, cnt - 5, 1u);
                                }
                            } else {
                                span(0, n1, 1u);
                                if (cnt > n1) span(n1, cnt - n1, 1u);
                            }
                        }
                        mma_commit_one(one, aempty + 8 * s);
                    }
                    if (fail_code) break;
                    mma_commit_one(one, bempty + 8 * sb);
                    if (++in == args.flush || kb == nkb - 1) {
                        mma_commit_one(one, tfull);
                        ++nch;
                        in = 0;
                    }
                }
            }
            if (fail_code) *abort = 1;
            mma_commit_one(one, done);
        }
    } else if (warp >= kEpi + 4) {
        if (kMode == DG_DOTS) {
            // thread = row: its partial s and t over the tile's 64 modes, beside
            // the matrix work (in the epilogue these two products an element kept
            // the float64 pipe for longer than the tile's MMAs run)
            const int row = (warp - kEpi - 4) * 32 + lane;
            // (left out where s and t come from a product of their own)
            for (Item w(args); args.vs && w.left > 0; w.next()) {
                const int at = w.at, bt = w.bt, tb = kPart ? bt / win : bt;
                const int cw = 4 * hc, w0 = kPart ? bt % win * cw : 0;
                const long tile = ((long)at * args.Mp + (long)(tb % args.nct) * kGN + w0) * 128 + row;
                const double *pd = args.dt + tile, *pg = args.gt + tile;
                const double *vs = args.vs + (long)tb * kGN + w0, *vt = args.vt + (long)tb * kGN + w0;
                double s = 0, t = 0;
#pragma unroll 1
                for (int c = 0; c < cw; c += 8) {
                    double d[8], g[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        d[e] = pd[(c + e) * 128];
                        g[e] = pg[(c + e) * 128];
                    }
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        s = fma(vs[c + e], d[e], s);
                        t = fma(vt[c + e], g[e], t);
                    }
                }
                const long r = (long)at * kGM + row;
                if (r < args.R) {
                    double *o = args.qp + (long)bt * 4 * args.R + r;
                    o[2 * args.R] = s;
                    o[3 * args.R] = t;
                }
            }
        }
    }
    } else {
        regs_inc<Sh::epi>();
        const int quad = warp & 3, part = warp >> 2;   // part: columns c0 .. c0 + hc - 1
        const int row = quad * 32 + lane;
        const bool full = hc > 8;
        const uint32_t base = tmem + ((uint32_t)(quad * 32) << 16);
        uint32_t nch = 0;
        bool bad = false;            // a wait of this warp gave up
        int i = 0;
        for (Item w(args); w.left > 0; w.next(), ++i) {
            const int at = w.at, bt = w.bt, tb = kPart ? bt / win : bt;
            const int c0 = (kPart ? bt % win * 4 * hc : 0) + part * hc;
            const int nkb = min(args.kbps, args.nkb - w.split * args.kbps);
            int *ce = cole + (i & 1) * kGN;
            if (threadIdx.x < kGN) {
                const long c = (long)b_tile(w) * kGN + threadIdx.x;
                ce[threadIdx.x] = (kMode == DG_PARTS ? args.ec[c] : args.et[c]) + kUnit;
                if (kMode == DG_QDOTS) ce[2 * kGN + threadIdx.x] = args.cofs[c] + 4 * at * args.nr;
            }
            const int nacc = (nkb + args.flush - 1) / args.flush;
            // An accumulator |a| <= 2^22 becomes a whole number by adding 1.5 2^23:
            // the bits of the sum are kMagic + a.  Their weighted sums are taken
            // modulo 2^64 from minus what the kMagic terms add up to.  (Conversions
            // run at an eighth of this rate and took as long as an accumulation's
            // read may take.)
            constexpr uint32_t kMagic = 0x4B400000u;
            long long hi[16], lo[16];
            const long long start = -(long long)nacc * (long long)((uint64_t)kMagic * 0x01010101u);
#pragma unroll
            for (int e = 0; e < 16; ++e) hi[e] = lo[e] = start;
            for (int c = 0; c < nacc; ++c, ++nch) {
                if (!bad && !mbar_all(tfull, nch & 1, budget, abort)) {
                    bad = true;
                    *abort = 1;
                }
                if (bad) continue;
                tc_fence_after();
                // Rolled: a small call runs this code once.
                uint32_t v[16];
                auto add = [&](uint32_t w, long long *acc, int e0, auto count) {
                    constexpr int n = decltype(count)::value;
                    uint32_t over = 0, b[n];
#pragma unroll
                    for (int e = 0; e < n; ++e) {
                        b[e] = __float_as_uint(__uint_as_float(v[e0 + e]) + 12582912.f);
                        over |= b[e] ^ 0x4B000000u;
                    }
                    if (__any_sync(0xffffffffu, over >> 23)) {
#pragma unroll
                        for (int e = 0; e < n; ++e)
                            b[e] = kMagic + (uint32_t)__float2int_rn(__uint_as_float(v[e0 + e]));
                    }
#pragma unroll
                    for (int e = 0; e < n; ++e) acc[e0 + e] += (long long)((uint64_t)b[e] * w);
                };
                using Eight = std::integral_constant<int, 8>;
                using Four = std::integral_constant<int, 4>;
                auto order = [&](int o, uint32_t w, long long(&acc)[16]) {
                    const uint32_t from = base + c0 + kGN * o;
                    if (full) tmem_ld16(from, v);
                    else if (hc > 4) tmem_ld8(from, v);
                    else tmem_ld4(from, v);
                    tmem_wait_ld();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tempty + 8 * o);
                    if (kPart && hc == 4) {
                        add(w, acc, 0, Four());
                    } else {
                        add(w, acc, 0, Eight());
                        if (full) add(w, acc, 8, Eight());
                    }
                };
#pragma unroll 1
                for (int k = 0; k < 4; ++k) order(7 - k, 1u << (8 * k), lo);
#pragma unroll 1
                for (int k = 0; k < 4; ++k) order(3 - k, 1u << (8 * k), hi);
            }
            // the other warps' column scales and failures
            if (dg_sync_or(bad)) {
                fail_code = 3;
                break;
            }
            if (kMode == DG_DOTS) {
                const long tile = ((long)at * args.Mp + (long)(tb % args.nct) * kGN + c0) * 128 + row;
                const double *pd = args.dt + tile, *pg = args.gt + tile;
                // four modes' x and g on the way while the four before are used
                double q = 0, p = 0, d[4], g[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    d[e] = pd[e * 128];
                    g[e] = pg[e * 128];
                }
                // the rest is padding
                const int ncol = min(hc, args.M - (tb % args.nct) * kGN - c0);
#pragma unroll
                for (int e0 = 0; e0 < 16; e0 += 4) {
                    if (e0 >= ncol) break;
                    double v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        v[e] = fixed_to_double(hi[e0 + e], lo[e0 + e], ce[c0 + e0 + e]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        q = fma(d[e], v[e], q);
                        p = fma(g[e], v[e], p);
                        // (never past this warp's columns: the last part of a shared
                        // tile ends with the tile, and the last tile with the array)
                        if (e0 + 4 < ncol) {
                            d[e] = pd[(e0 + 4 + e) * 128];
                            g[e] = pg[(e0 + 4 + e) * 128];
                        }
                    }
                }
                double *rb = red + row;
                if (part) {
                    rb[(part - 1) * 128] = q;
                    rb[(part + 2) * 128] = p;
                }
                asm volatile("bar.sync 1, 512;" ::: "memory");
                const long r = (long)at * kGM + row;
                if (!part && r < args.R) {
                    double *o = args.qp + (long)bt * 4 * args.R + r;
                    o[0] = (q + rb[0]) + (rb[128] + rb[256]);
                    o[args.R] = (p + rb[384]) + (rb[512] + rb[640]);
                }
            } else if (kMode == DG_QDOTS) {
                // columns 2 n, 2 n + 1 are Re and Im of a band of u: sum conj(x) u and
                // sum conj(u) g.  Of the former the second member of a pair (kind 2) has
                // the conjugate of the first's (kind 1): twice that one's real part.
                const int *co = ce + 2 * kGN + c0;
                const double *px = args.dt + row, *pg = args.gt + row;
                const int ncol = min(hc, args.M - c0);
                double tr = 0, ti = 0, t2 = 0, br = 0, bi = 0, x[4], g[4];
                auto load = [&](int e0) {
#pragma unroll
                    for (int e = 0; e < 4; e += 2) {
                        const long o = (co[e0 + e] >> 2) * 128L;
                        x[e] = px[o];
                        x[e + 1] = px[o + 128];
                        g[e] = pg[o];
                        g[e + 1] = pg[o + 128];
                    }
                };
                load(0);
#pragma unroll
                for (int e0 = 0; e0 < 16; e0 += 4) {
                    if (e0 >= ncol) break;
                    double v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        v[e] = fixed_to_double(hi[e0 + e], lo[e0 + e], ce[c0 + e0 + e]);
#pragma unroll
                    for (int e = 0; e < 4; e += 2) {
                        const int kind = co[e0 + e] & 3;
                        if (kind == 0) {
                            tr = fma(x[e], v[e], tr);
                            tr = fma(x[e + 1], v[e + 1], tr);
                            ti = fma(x[e], v[e + 1], ti);
                            ti = fma(-x[e + 1], v[e], ti);
                        } else if (kind == 1) {
                            t2 = fma(x[e], v[e], t2);
                            t2 = fma(x[e + 1], v[e + 1], t2);
                        }
                        br = fma(g[e], v[e], br);
                        br = fma(g[e + 1], v[e + 1], br);
                        bi = fma(g[e + 1], v[e], bi);
                        bi = fma(-g[e], v[e + 1], bi);
                    }
                    if (e0 < 12) load(e0 + 4);
                }
                tr = fma(2.0, t2, tr);
                double *rb = red + row;
                if (part) {
                    double *o = rb + (part - 1) * 128;
                    o[0] = tr;
                    o[384] = ti;
                    o[768] = br;
                    o[1152] = bi;
                }
                asm volatile("bar.sync 1, 512;" ::: "memory");
                const long r = (long)at * kGM + row;
                if (!part && r < args.R) {
                    const double f = pow2(args.er[(long)a_tile(w) * kGM + row]);
                    double *o = args.qp + (long)bt * 4 * args.R + r;
                    auto all = [&](double s, int k) {
                        return ((s + rb[384 * k]) + (rb[384 * k + 128] + rb[384 * k + 256])) * f;
                    };
                    o[0] = all(tr, 0);
                    o[args.R] = all(ti, 1);
                    o[2 * args.R] = all(br, 2);
                    o[3 * args.R] = all(bi, 3);
                }
            } else if (kMode == DG_STORE) {
                const long r = (long)at * kGM + row;
                if (r < args.R) {
                    const int er = args.er[r], ncol = min(hc, args.M - bt * kGN - c0);
                    double *o = args.out + r * args.M + (long)bt * kGN + c0;
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        if (e >= ncol) break;
                        o[e] = fixed_to_double(hi[e], lo[e], ce[c0 + e] + er);
                    }
                }
            } else {
                const long grow = (long)at * kGM + row;
                const bool live = grow < args.rows_b && (int)(grow % args.rmod) < args.rlive;
                if (live) {
                    const int eb = args.ew[grow];
                    double *o = args.gpart + ((long)w.split * args.nat * kGM + grow) * args.Mp +
                                (long)bt * kGN + c0;
                    const int ncol = min(hc, args.M - bt * kGN - c0);
#pragma unroll
                    for (int e = 0; e < 16; e += 2) {
                        if (e >= ncol) break;
                        double2 x;
                        x.x = fixed_to_double(hi[e], lo[e], ce[c0 + e] + eb);
                        x.y = fixed_to_double(hi[e + 1], lo[e + 1], ce[c0 + e + 1] + eb);
                        *reinterpret_cast<double2 *>(o + e) = x;
                    }
                }
            }
        }
        if (fail_code) *abort = 1;
    }
    if (fail_code && lane == 0) {
        *(volatile int *)args.err = 10 + fail_code;
        if (args.failed) *(volatile int *)args.failed = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kEpi + 1) {
        mbar_wait(done, 0, kDefaultBudget);
        __syncwarp();
        tc_fence_after();
        tmem_dealloc<512>(tmem);
    }
}

template <int kMode, bool kPart>
inline cudaError_t dg_setup() {
    return cudaFuncSetAttribute(k_dg_gemm<kMode, kPart>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)DgShape<kMode>::smem);
}

// kk, hc and abytes of tiles that are partly empty, of full ones otherwise
template <int kMode, bool kPart>
inline cudaError_t dg_launch(const DgArgs &a, int nsm, cudaStream_t st) {
    return launch_pdl(k_dg_gemm<kMode, kPart>, (int)std::min<long>(a.nitems, nsm),
                      DgShape<kMode>::threads, DgShape<kMode>::smem, st, a);
}

}  // namespace tdscha
