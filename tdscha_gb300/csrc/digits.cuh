// Exact digit products: splitting float64 numbers into digits, the tensor-core
// contraction over digit operands, and the way back to float64.  perturb_digits.cu
// explains the arithmetic.
#pragma once

#include <algorithm>
#include <climits>

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

// 2^e for the exponents of finite float64 rows
__device__ __forceinline__ double pow2(int e) { return ldexp(1.0, e); }

// -------------------------------------------------------- the contraction
// Persistent, one CTA per SM, 512 threads, one 128 x 64 output tile at a time;
// its accumulators, eight orders of 64 columns, fill the TMEM.
//   warp 8  copies: B blocks (all digits of 64 rows) into two buffers, A digits
//           (128 rows each) into a ring
//   warp 9  MMA issue: A digit i against the B digits 0 .. 7 - i at once, which
//           lie behind one another in shared memory as their accumulators do in
//           TMEM, so one instruction covers up to four orders (N = 256).  i
//           runs downwards: the light high orders come first.
//   warps 12-15  (stage A) s and t
//   warps 0-7  every three K blocks the accumulators are read, order 7 first,
//           and added to two 64-bit integers an element (warp w: lanes 32 (w % 4),
//           columns 32 (w / 4) of every order).  Each order has its own
//           release, so the MMAs of the next blocks start on order 7 while the
//           lower ones are still read.  At the end of a tile the sums become
//           float64: row dots (stage A) or a partial tile (stage B).
// Bounded waits and the abort flag as in perturb_mixed.cu.
//
// What it takes at M=573, N=50000 (1.95 GHz): stage A 700 us, stage B 774 us; the
// 35 products alone are 0.93 and 1.04 million cycles an SM, 480 and 530 us.  The
// same loop on one thread (`if (lane == 0)`) took 794 and 928 us, with 64-bit
// divisions for the ring slots 1165 and 1098.  Reading an accumulation back takes
// the epilogue 8000 cycles, of which 1200 stand before the next MMAs; a tile's end
// 12000 (stage A: two float64 products an element on the float64 pipe).  With 48
// images stage A (976 us at M=189, N=10000) is bound by that pipe and the epilogue.
// The copies (176 KB a K block) take 3700 cycles of a block's 4500 and do not show.
// What becomes of a tile: row dots (stage A), split-K partials (stage B), or the
// product itself
enum { DG_DOTS = 0, DG_PARTS, DG_STORE };

struct DgArgs {
    const __half *a, *b;
    int nkb;               // K blocks of an operand row
    int kbps;              // K blocks per work item (stage A: nkb)
    int flush;             // K blocks per accumulation
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
    const int *ec, *ew;
    double *gpart;         // [split][A rows][Mp]: H[b][a]
    int M;                 // columns in use (of an image)
    long rows_b;           // rows (image, mode) in use
    // product: out[R][M], row exponents er
    const int *er;
    double *out;
};

// 512 threads of 128 registers; the epilogue's two warpgroups take 192 of each
// thread, the other two 64: 256 * 192 + 256 * 64 = 512 * 128.
constexpr int kGThreads = 512, kGRegsEpi = 192, kGRegsRest = 64;
static_assert(256 * kGRegsEpi + 256 * kGRegsRest == kGThreads * 128, "register shares");

template <int kMode>
struct DgShape {
    static constexpr bool wide = kMode == DG_PARTS;    // 8 digits of A, 7 of B
    static constexpr int SA = wide ? kCall : kRes, SB = wide ? kRes : kCall;
    static constexpr int slots = wide ? 6 : 5;         // A ring: with the B buffers 208 KB
    static constexpr uint32_t bbytes = SB * kGB;
    static constexpr int bars = 2 * slots + 4 + 1 + kOrders + 1;
    static constexpr size_t ring = 2 * (size_t)bbytes + slots * (size_t)kGA;
    static constexpr size_t smem = 1024 + ring + 2 * 2 * 128 * sizeof(double) +
                                   2 * kGN * sizeof(int) + 8 * bars + 16;
};
static_assert(DgShape<DG_DOTS>::smem <= 232448 && DgShape<DG_PARTS>::smem <= 232448,
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

template <int kMode>
__global__ void __launch_bounds__(kGThreads, 1) k_dg_gemm(const DgArgs args) {
    using Sh = DgShape<kMode>;
    constexpr int SA = Sh::SA, SB = Sh::SB, slots = Sh::slots;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *ring = smem + 2 * Sh::bbytes;
    double *red = reinterpret_cast<double *>(smem + Sh::ring);        // [2][2][128]
    int *cole = reinterpret_cast<int *>(red + 2 * 2 * 128);            // [2][64]
    uint64_t *bars = reinterpret_cast<uint64_t *>(cole + 2 * kGN);
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

    if (warp >= 8) {
    regs_dec<kGRegsRest>();
    if (warp == 8) {
        if (lane == 0) {
            Cursor ca, cb;
            long ga = 0, gb = 0;             // copies issued
            for (Item w(args); w.left > 0 && !fail_code; w.next()) {
                const int kb0 = w.split * args.kbps, nkb = min(args.kbps, args.nkb - kb0);
                const uint8_t *pa = reinterpret_cast<const uint8_t *>(args.a) +
                                    ((long)w.at * args.nkb + kb0) * SA * (long)kGA;
                const uint8_t *pb = reinterpret_cast<const uint8_t *>(args.b) +
                                    ((long)w.bt * args.nkb + kb0) * SB * (long)kGB;
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
                        mbar_expect_tx(afull + 8 * ca.s, kGA);
                        bulk_load(smem_u32(ring + ca.s * kGA), pa + d * (long)kGA, kGA,
                                  afull + 8 * ca.s);
                        ca.next(slots);
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
    } else if (warp >= 12) {
        if (kMode == DG_DOTS) {
            // thread = row: its partial s and t over the tile's 64 modes, beside
            // the matrix work (in the epilogue these two products an element kept
            // the float64 pipe for longer than the tile's MMAs run)
            const int row = (warp - 12) * 32 + lane;
            for (Item w(args); w.left > 0; w.next()) {
                const int at = w.at, bt = w.bt;
                const long tile = ((long)at * args.Mp + (long)(bt % args.nct) * kGN) * 128 + row;
                const double *pd = args.dt + tile, *pg = args.gt + tile;
                const double *vs = args.vs + (long)bt * kGN, *vt = args.vt + (long)bt * kGN;
                double s = 0, t = 0;
#pragma unroll 1
                for (int c = 0; c < kGN; c += 8) {
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
        regs_inc<kGRegsEpi>();
        const int quad = warp & 3, half = warp >> 2;
        const int row = quad * 32 + lane;
        const uint32_t base = tmem + ((uint32_t)(quad * 32) << 16) + 32 * half;
        uint32_t nch = 0;
        bool bad = false;            // a wait of this warp gave up
        int i = 0;
        for (Item w(args); w.left > 0; w.next(), ++i) {
            const int at = w.at, bt = w.bt;
            const int nkb = min(args.kbps, args.nkb - w.split * args.kbps);
            int *ce = cole + (i & 1) * kGN;
            if (threadIdx.x < kGN) {
                const long c = (long)bt * kGN + threadIdx.x;
                ce[threadIdx.x] = (kMode == DG_PARTS ? args.ec[c] : args.et[c]) + kUnit;
            }
            const int nacc = (nkb + args.flush - 1) / args.flush;
            // An accumulator |a| <= 2^22 becomes a whole number by adding 1.5 2^23:
            // the bits of the sum are kMagic + a.  Their weighted sums are taken
            // modulo 2^64 from minus what the kMagic terms add up to.  (Conversions
            // run at an eighth of this rate and took as long as an accumulation's
            // read may take.)
            constexpr uint32_t kMagic = 0x4B400000u;
            long long hi[32], lo[32];
            const long long start = -(long long)nacc * (long long)((uint64_t)kMagic * 0x01010101u);
#pragma unroll
            for (int e = 0; e < 32; ++e) hi[e] = lo[e] = start;
            for (int c = 0; c < nacc; ++c, ++nch) {
                if (!bad && !mbar_all(tfull, nch & 1, budget, abort)) {
                    bad = true;
                    *abort = 1;
                }
                if (bad) continue;
                tc_fence_after();
                // Half an order (16 columns) at a time, the next half's read on its
                // way while one is added.  Rolled: a small call runs this code once.
                uint32_t v[2][16];
                tmem_ld16(base + kGN * (kOrders - 1), v[0]);
                auto add = [&](const uint32_t(&x)[16], uint32_t w, long long *acc) {
                    uint32_t b[16], over = 0;
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        b[e] = __float_as_uint(__uint_as_float(x[e]) + 12582912.f);
                        over |= b[e] ^ 0x4B000000u;
                    }
                    if (__any_sync(0xffffffffu, over >> 23)) {
#pragma unroll
                        for (int e = 0; e < 16; ++e)
                            b[e] = kMagic + (uint32_t)__float2int_rn(__uint_as_float(x[e]));
                    }
#pragma unroll
                    for (int e = 0; e < 16; ++e) acc[e] += (long long)((uint64_t)b[e] * w);
                };
                auto order = [&](int o, uint32_t w, long long(&acc)[32]) {
                    tmem_wait_ld();
                    tmem_ld16(base + kGN * o + 16, v[1]);
                    add(v[0], w, acc);
                    tmem_wait_ld();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tempty + 8 * o);
                    if (o > 0) tmem_ld16(base + kGN * (o - 1), v[0]);
                    add(v[1], w, acc + 16);
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
            const int c0 = half * 32;
            if (kMode == DG_DOTS) {
                const long tile = ((long)at * args.Mp + (long)(bt % args.nct) * kGN + c0) * 128 + row;
                const double *pd = args.dt + tile, *pg = args.gt + tile;
                // eight modes' x and g on the way while the eight before are used
                double q = 0, p = 0, d[8], g[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    d[e] = pd[e * 128];
                    g[e] = pg[e * 128];
                }
                const int ncol = args.M - (bt % args.nct) * kGN - c0;    // the rest is padding
#pragma unroll
                for (int e0 = 0; e0 < 32; e0 += 8) {
                    if (e0 >= ncol) break;
                    double v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        v[e] = fixed_to_double(hi[e0 + e], lo[e0 + e], ce[c0 + e0 + e]);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        q = fma(d[e], v[e], q);
                        p = fma(g[e], v[e], p);
                        if (e0 < 24) {
                            d[e] = pd[(e0 + 8 + e) * 128];
                            g[e] = pg[(e0 + 8 + e) * 128];
                        }
                    }
                }
                double *rb = red + (i & 1) * 2 * 128 + row;
                if (half) {
                    rb[0] = q;
                    rb[128] = p;
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
                const long r = (long)at * kGM + row;
                if (!half && r < args.R) {
                    double *o = args.qp + (long)bt * 4 * args.R + r;
                    o[0] = q + rb[0];
                    o[args.R] = p + rb[128];
                }
            } else if (kMode == DG_STORE) {
                const long r = (long)at * kGM + row;
                if (r < args.R) {
                    const int er = args.er[r], ncol = args.M - bt * kGN - c0;
                    double *o = args.out + r * args.M + (long)bt * kGN + c0;
#pragma unroll
                    for (int e = 0; e < 32; ++e) {
                        if (e >= ncol) break;
                        o[e] = fixed_to_double(hi[e], lo[e], ce[c0 + e] + er);
                    }
                }
            } else {
                const long grow = (long)at * kGM + row;
                const int b = (int)(grow % args.Mp);
                const bool live = grow < args.rows_b && b < args.M;
                if (live) {
                    const int eb = args.ew[grow];
                    double *o = args.gpart + ((long)w.split * args.nat * kGM + grow) * args.Mp +
                                (long)bt * kGN + c0;
                    const int ncol = args.M - bt * kGN - c0;
#pragma unroll
                    for (int e = 0; e < 32; e += 2) {
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

}  // namespace tdscha
