// gemm_pairs.cu — exact FP64 products of slice pairs on the INT8 tensor cores.
//
// A slice is an integer q (at most 26 bits) times a power of two, so the exact
// product of a slice pair over k is an integer below 2^53 (the rho rule) times
// a power of two, whatever computes it.  q is cut into D signed digits; the
// products of digit d of A and digit e of B belong to digit level L = d + e,
// and V = sum_L 2^(radix (2D-2-L)) W_L with W_L the INT32 sums of level L.
//
// What bounds it: the tensor pipe (D^2 digit products per pair), the operand
// traffic per product, and the FP64 work that turns 2D - 1 INT32 sums per
// output and pair into one term of the ordered sum.  So:
//   * 8-bit digits (22-bit slices in 3 digits; 7-bit digits take 4): 9 instead
//     of 16 products per pair.
//   * All 2D - 1 levels of a pair are accumulated in one pass over k, each in its
//     own tensor-memory accumulator (5 x 96 or 7 x 64 columns), so the D + D
//     digit planes of a 128-wide k step serve all D^2 products: 84 KB per
//     nine 128 x 96 products, where one level at a time reads 2 planes a product.
//   * The accumulators are handed over level by level: the last k step of a pair
//     completes level 0 first, and the first k step of the next pair starts with
//     level 0, so the epilogue's reads run under the MMAs of both.
//     A 128 x 96 x 32 MMA takes 56 cycles (7 KB of operands through the 128 B a
//     clock shared-memory port; 48 of math), so a k step is 2016 cycles at best.
//   * FP64 work stands still while MMAs stream, so the epilogue combines levels
//     as integers (the kernel's epilogue says more).
//   * The tiles' pairs are cut into equal shares, tiles included (pp_share).
//   * Where a tile's lines have no slice at a level (the counts are those of the
//     worst line of the whole operand), its pairs are skipped: they add zero.
// Product kernel, before (one digit level at a time, 7-bit digits) and now, one
// B200: 1024^3 plain, 16 pairs, 1076 -> 145 us; 3001 x 1999 x 2500 plain, 20 pairs,
// 4.08 -> 1.69 ms (and 0.15 for the sum, now inside); 2048^3
// <float,double,double>, 9 pairs, 1.73 (0.10) -> 0.57 ms: 2.2, 3.0 and 2.6
// POP/s of digit products, against 3.6 that the power limit leaves N = 96
// MMAs.  Split to digit planes (count, FP64 slices, digits in three passes
// before), 3001 lines of 2500: 374 -> 54 us.
#include <cuda.h>

#include "gemm_pairs.h"
#include "ozb_device.cuh"
#include "sum.cuh"
#include "tc05.cuh"

namespace ozb {

uint64_t i8_test_wait_ns();  // gemm_i8.cu: the limit of every bounded wait
int i8_test_hold_copies();
int make_map_planes(CUtensorMap *map, const int8_t *base, uint64_t k_pad, uint64_t lines, uint64_t planes,
                    uint32_t box_lines);  // gemm_i8.cu

PairDigits pair_digits(int bits, int k) {
    // largest |q| a D-digit balanced form of radix 2^r holds: (2^(r-1) - 1) (1 + 2^r + ... + 2^(r(D-1)))
    for (int radix = 8; radix >= 7; radix--)
        for (int D = 3; D <= 4; D++) {
            int64_t hold = 0;
            for (int d = 0; d < D; d++) hold = (hold << radix) + (((int64_t)1 << (radix - 1)) - 1);
            if (((int64_t)1 << bits) <= hold && ((int64_t)D * k << (2 * radix - 2)) <= 2147483647LL)
                return PairDigits{D, radix};
        }
    return PairDigits{0, 8};
}

// ---------------------------------------------------------------------------
// Split.  One CTA per line with the line in registers (C chunks of 8
// consecutive elements per thread): the levels' chain of maxima, the slices
// and their digits in one read of the line.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t abs_bits(double v) {  // |v| as an ordered integer, 0 for NaN (the reference's max ignores it)
    const uint64_t b = dbits(v) & 0x7fffffffffffffffULL;
    return b > 0x7ff0000000000000ULL ? 0 : b;
}
__device__ __forceinline__ uint32_t abs_bits(float v) {
    const uint32_t b = (uint32_t)__float_as_int(v) & 0x7fffffffu;
    return b > 0x7f800000u ? 0 : b;
}
__device__ __forceinline__ uint32_t warp_max(uint32_t v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ uint64_t warp_max(uint64_t v) {
    const uint32_t hi = (uint32_t)(v >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
    const uint32_t ml = __reduce_max_sync(0xffffffffu, hi == mh ? (uint32_t)v : 0u);
    return ((uint64_t)mh << 32) | ml;
}
template <typename B>
__device__ __forceinline__ B block_max_bits(B v, B *red) {  // red: two sets of 32, used in turn by the caller
    v = warp_max(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (l == 0) red[w] = v;
    __syncthreads();
    return warp_max(l < nw ? red[l] : (B)0);
}

// The digits of 8 slices, packed per digit plane: byte d of q + bias is digit
// (D-1-d) offset by 2^(radix-1).
template <int D>
__device__ __forceinline__ void digits8(const int (&q)[8], int radix, uint2 (&out)[D]) {
    const uint32_t half = 1u << (radix - 1), mask = (1u << radix) - 1;
    uint32_t bias = 0;
#pragma unroll
    for (int d = 0; d < D; d++) bias = (bias << radix) + half;
    uint32_t w[D][2];
#pragma unroll
    for (int d = 0; d < D; d++) w[d][0] = w[d][1] = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t t = (uint32_t)q[i] + bias;
#pragma unroll
        for (int d = 0; d < D; d++)
            w[d][i >> 2] |= (((t >> (radix * (D - 1 - d))) & mask)) << (8 * (i & 3));
    }
#pragma unroll
    for (int d = 0; d < D; d++) {  // offset digits back to signed bytes
        const uint32_t h4 = half * 0x01010101u;
        out[d] = make_uint2(__vsub4(w[d][0], h4), __vsub4(w[d][1], h4));
    }
}

template <typename T>
struct SplitRange;
template <>
struct SplitRange<double> {
    using Bits = uint64_t;
    static constexpr int kMant = 53, kEmin = -1021, kEmax = 1023;
    static __device__ __forceinline__ double val(uint64_t b) { return __longlong_as_double((long long)b); }
    static __device__ __forceinline__ int tau(double v) { return tau_rule(v); }
};
template <>
struct SplitRange<float> {
    using Bits = uint32_t;
    static constexpr int kMant = 24, kEmin = -125, kEmax = 127;
    static __device__ __forceinline__ float val(uint32_t b) { return __int_as_float((int)b); }
    static __device__ __forceinline__ int tau(float v) { return tau_rule_f32(v); }
};

// A level's constants from the largest remainder: tau, sigma = 0.75 2^(rho + tau),
// whether a slice's integer can be read off the bits of r + sigma (sigma
// normal), and whether sigma overflows.
template <typename T>
struct SplitLevel {
    T sigma;
    int tau, sh;
    bool fast, over;
    __device__ __forceinline__ SplitLevel(typename SplitRange<T>::Bits mb, int rho) {
        using R = SplitRange<T>;
        tau = R::tau(R::val(mb));
        sigma = (T)(0.75 * (double)(T)pow2(rho + tau));
        fast = rho + tau >= R::kEmin && rho + tau <= R::kEmax;
        over = rho + tau > R::kEmax;
        sh = R::kMant - rho - tau;
    }
};

// One level of one element: the slice's integer q; r becomes the remainder.
__device__ __forceinline__ int cut_level(double &r, const SplitLevel<double> &lv) {
    const double t = r + lv.sigma, sl = t - lv.sigma;
    r = r - sl;
    return lv.fast ? __double2loint(t) : (int)scale2(sl, lv.sh);  // t = sigma + q ulp, sigma's low word 0
}
__device__ __forceinline__ int cut_level(float &r, const SplitLevel<float> &lv) {
    const float t = __fadd_rn(r, lv.sigma), sl = __fsub_rn(t, lv.sigma);
    r = __fsub_rn(r, sl);
    return lv.fast ? __float_as_int(t) - __float_as_int(lv.sigma) : (int)scale2((double)sl, lv.sh);
}

template <int D>
__device__ __forceinline__ void store_digits8(const int (&q)[8], int radix, int8_t *dig, size_t plane0, int nl,
                                              int line, int k_pad, int i0) {
    uint2 w[D];
    digits8<D>(q, radix, w);
#pragma unroll
    for (int d = 0; d < D; d++) *reinterpret_cast<uint2 *>(dig + ((plane0 + d) * nl + line) * k_pad + i0) = w[d];
}

// A line's end (one thread): no slices above level cnt - 1, the tile's level
// count, and the first level that left a zero remainder.
__device__ __forceinline__ void split_line_done(int line, int nl, int z, int cnt, int lcap, bool bad, int tile_lines,
                                                short *exps, int *tile_lev, int *zmax) {
    for (int s = cnt; s < lcap; s++) exps[(size_t)s * nl + line] = bad ? kExpNaN : kExpZero;
    atomicMax(&tile_lev[line / tile_lines], cnt < lcap ? cnt : lcap);
    atomicMax(zmax, z);
}

template <typename T, int D, int C>
__global__ void __launch_bounds__(512) k_pair_split(int k, int k_pad, int nl, const T *__restrict__ X, int ldx, int rho,
                                                    int maxS, int lcap, int radix, int tile_lines,
                                                    int8_t *__restrict__ dig, short *__restrict__ exps,
                                                    int *__restrict__ tile_lev, int *__restrict__ zmax) {
    using B = typename SplitRange<T>::Bits;
    __shared__ B red[2][32];
    const int line = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
    const T *x = X + (size_t)line * ldx;
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    T r[C][8];
    B mb = 0;
    bool bad = false;
#pragma unroll
    for (int c = 0; c < C; c++) {
        const int i0 = (c * nt + tid) * 8;
        if (vec && i0 + 8 <= k) {
            constexpr int kPer = 16 / (int)sizeof(T);
            using V = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
#pragma unroll
            for (int j = 0; j < 8 / kPer; j++) {
                const V v = *reinterpret_cast<const V *>(x + i0 + j * kPer);
                r[c][j * kPer] = v.x;
                r[c][j * kPer + 1] = v.y;
                if constexpr (sizeof(T) == 4) {
                    r[c][j * kPer + 2] = v.z;
                    r[c][j * kPer + 3] = v.w;
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) r[c][i] = i0 + i < k ? x[i0 + i] : (T)0;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const B a = abs_bits(r[c][i]);
            mb = a > mb ? a : mb;
            bad |= !isfinite(r[c][i]);
        }
    }
    bad = __syncthreads_or(bad);
    mb = block_max_bits<B>(mb, red[0]);
    int z = maxS - 1, cnt = maxS;
    for (int s = 0; s < maxS; s++) {
        const SplitLevel<T> lv(mb, rho);
        B nm = 0;
#pragma unroll
        for (int c = 0; c < C; c++) {
            const int i0 = (c * nt + tid) * 8;
            int q[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                q[i] = cut_level(r[c][i], lv);
                const B a = abs_bits(r[c][i]);
                nm = a > nm ? a : nm;
            }
            if (s < lcap && i0 < k_pad) store_digits8<D>(q, radix, dig, (size_t)s * D, nl, line, k_pad, i0);
        }
        if (tid == 0 && s < lcap) exps[(size_t)s * nl + line] = bad || lv.over ? kExpNaN : (short)lv.tau;
        mb = block_max_bits<B>(nm, red[(s + 1) & 1]);
        if (mb == 0) {
            z = s < maxS - 1 ? s : maxS - 1;
            cnt = s + 1;
            break;
        }
    }
    if (tid == 0) split_line_done(line, nl, z, cnt, lcap, bad, tile_lines, exps, tile_lev, zmax);
}

// Lines longer than the register kernel holds: the same levels with the
// remainders in global memory (rem: k_pad values per line).
template <typename T, int D>
__global__ void __launch_bounds__(512) k_pair_split_long(int k, int k_pad, int nl, const T *__restrict__ X, int ldx,
                                                         int rho, int maxS, int lcap, int radix, int tile_lines,
                                                         int8_t *__restrict__ dig, short *__restrict__ exps,
                                                         int *__restrict__ tile_lev, int *__restrict__ zmax,
                                                         T *__restrict__ rem) {
    using B = typename SplitRange<T>::Bits;
    __shared__ B red[2][32];
    const int line = blockIdx.x, tid = threadIdx.x;
    const T *x = X + (size_t)line * ldx;
    T *rm = rem + (size_t)line * k_pad;
    B mb = 0;
    bool bad = false;
    for (int i = tid; i < k; i += blockDim.x) {
        const T v = x[i];
        const B a = abs_bits(v);
        mb = a > mb ? a : mb;
        bad |= !isfinite(v);
    }
    bad = __syncthreads_or(bad);
    mb = block_max_bits<B>(mb, red[0]);
    int z = maxS - 1, cnt = maxS;
    for (int s = 0; s < maxS; s++) {
        const SplitLevel<T> lv(mb, rho);
        B nm = 0;
        for (int i0 = tid * 8; i0 < k_pad; i0 += blockDim.x * 8) {
            int q[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                T r = s == 0 ? (i0 + i < k ? x[i0 + i] : (T)0) : rm[i0 + i];
                q[i] = cut_level(r, lv);
                rm[i0 + i] = r;
                const B a = abs_bits(r);
                nm = a > nm ? a : nm;
            }
            if (s < lcap) store_digits8<D>(q, radix, dig, (size_t)s * D, nl, line, k_pad, i0);
        }
        if (tid == 0 && s < lcap) exps[(size_t)s * nl + line] = bad || lv.over ? kExpNaN : (short)lv.tau;
        mb = block_max_bits<B>(nm, red[(s + 1) & 1]);
        if (mb == 0) {
            z = s < maxS - 1 ? s : maxS - 1;
            cnt = s + 1;
            break;
        }
    }
    if (tid == 0) split_line_done(line, nl, z, cnt, lcap, bad, tile_lines, exps, tile_lev, zmax);
}

template <typename T, int D>
static int launch_split(cuozblasHandle_t *h, int k, int k_pad, const T *X, int ldx, int rho, int maxS, int radix,
                        int tile_lines, const PairOperand &op, int *zmax_dev) {
    cudaStream_t s = state(h)->stream;
    if (k_pad > kPairSplitMaxK) {
        Arena ar(h);
        const uint64_t mk = ar.mark();
        T *rem = ar.take<T>((uint64_t)op.nl * k_pad);
        if (!ar.ok) return CUOZBLAS_STATUS_WORKSPACE;
        counted(h);
        k_pair_split_long<T, D><<<op.nl, 512, 0, s>>>(k, k_pad, op.nl, X, ldx, rho, maxS, op.levels, radix, tile_lines,
                                                      op.dig, op.exps, op.tile_lev, zmax_dev, rem);
        OZB_CHECK(cudaGetLastError());
        ar.release(mk);
        return CUOZBLAS_STATUS_SUCCESS;
    }
    counted(h);
    // 8 C elements per thread; the fewest threads that hold the line keep more lines per SM in flight
    auto go = [&](auto kern, int C) {
        const int threads = (k_pad + 8 * C - 1) / (8 * C);
        kern<<<op.nl, (threads + 31) / 32 * 32, 0, s>>>(k, k_pad, op.nl, X, ldx, rho, maxS, op.levels, radix, tile_lines,
                                                       op.dig, op.exps, op.tile_lev, zmax_dev);
    };
    if (k_pad <= 2048)
        go(k_pair_split<T, D, 1>, 1);
    else if (k_pad <= 8192)
        go(k_pair_split<T, D, 2>, 2);
    else
        go(k_pair_split<T, D, 4>, 4);
    OZB_CHECK(cudaGetLastError());
    return CUOZBLAS_STATUS_SUCCESS;
}

template <typename T>
int pair_split(cuozblasHandle_t *h, int k, int k_pad, const T *X, int ldx, int rho, int maxS, const PairDigits &pd,
               int tile_lines, const PairOperand &op, int *zmax_dev) {
    if (op.nl == 0 || k_pad == 0) return CUOZBLAS_STATUS_SUCCESS;
    const int tiles = (op.nl + tile_lines - 1) / tile_lines;
    OZB_CHECK(cudaMemsetAsync(op.tile_lev, 0, sizeof(int) * tiles, state(h)->stream));
    return pd.D == 3 ? launch_split<T, 3>(h, k, k_pad, X, ldx, rho, maxS, pd.radix, tile_lines, op, zmax_dev)
                     : launch_split<T, 4>(h, k, k_pad, X, ldx, rho, maxS, pd.radix, tile_lines, op, zmax_dev);
}
template int pair_split<double>(cuozblasHandle_t *, int, int, const double *, int, int, int, const PairDigits &, int,
                                const PairOperand &, int *);
template int pair_split<float>(cuozblasHandle_t *, int, int, const float *, int, int, int, const PairDigits &, int,
                               const PairOperand &, int *);

// ---------------------------------------------------------------------------
// Product kernel.  Persistent, one CTA per SM: warp 0 lane 0 loads digit
// stages (digit d of A and of B for one k step) by TMA into a ring, warps 1
// and 2 issue the MMAs, warps 4-11 read the accumulators.  Every wait is bounded.
// ---------------------------------------------------------------------------
constexpr int kPpThreads = 384;
constexpr uint32_t kPpRegLo = 40, kPpRegHi = 232;  // 4 x 40 + 8 x 232 = 12 x 168 registers at launch

template <int D>
struct PpShape {
    static constexpr int BN = D == 3 ? 96 : 64;
    static constexpr int LV = 2 * D - 1;                // 5 x 96 = 480 or 7 x 64 = 448 tensor-memory columns
    static constexpr int TILE_A = 128 * 128, TILE_B = BN * 128, STAGE = TILE_A + TILE_B;
    static constexpr int ST = D == 3 ? 7 : 8;
    static constexpr int SMEM = ST * STAGE + 1024 /*align*/ + 512 /*barriers*/ + 8 * (BN / 2) * 4 /*column exponents*/;
    static constexpr int CW = BN / 2;                   // columns per epilogue warp
};

struct PpParams {
    int m, n, ldc, nkb, tiles_m, tiles_n, strip;
    int col0, cn;        // the launch's columns: cn from col0 (a tile boundary); tiles_n and lb count from col0
    int nA, nB, maxlevel, np, bias, radix;
    const int *la, *lb;  // levels in use per tile, or null
    const short *ea, *eb;
    double alpha, beta;
    void *C;
    double *pbuf;        // kPairStore: the pair buffer; else the partial sums handed from one CTA to the next
    unsigned *handed;    // per CTA and epilogue warp: its partial sums are in pbuf (zeroed before the launch)
    int *err;
};

// The pairs of a tile with LA x LB levels in use, in summation order.
struct PairCursor {
    int LA, LB, top, ik, ia, hi;
    __device__ __forceinline__ PairCursor(int la, int lb, int maxlevel) : LA(la), LB(lb), ik(-1), ia(0), hi(-1) {
        top = LA + LB - 2 < maxlevel ? LA + LB - 2 : maxlevel;
    }
    __device__ __forceinline__ bool next(int &a, int &b) {
        if (++ia > hi) {
            if (++ik > top) return false;
            ia = ik - (LB - 1) > 0 ? ik - (LB - 1) : 0;
            hi = ik < LA - 1 ? ik : LA - 1;
        }
        a = ia;
        b = ik - ia;
        return true;
    }
};
// How many there are.
__device__ __forceinline__ int pair_count(int LA, int LB, int maxlevel) {
    int n = 0;
    const int top = LA + LB - 2 < maxlevel ? LA + LB - 2 : maxlevel;
    for (int ik = 0; ik <= top; ik++) n += min(ik, LA - 1) - max(0, ik - (LB - 1)) + 1;
    return n;
}
__device__ __forceinline__ void pair_at(int p, int nA, int nB, int &a, int &b) {
    for (int ik = 0;; ik++) {
        const int lo = ik - (nB - 1) > 0 ? ik - (nB - 1) : 0, hi = ik < nA - 1 ? ik : nA - 1, c = hi - lo + 1;
        if (p < c) {
            a = lo + p;
            b = ik - a;
            return;
        }
        p -= c;
    }
}

// The CTA's share of a fused launch.  All (tile, pair) units in tile order are
// cut into one equal range per CTA, so the last wave is full; a tile cut in two
// is summed in order all the same: the CTA that holds its first pairs runs them
// first and hands its partial sums on, the CTA that holds the rest runs them
// last.  With ranges of at least a tile's pairs no tile meets three CTAs;
// otherwise (and in launches of at most one tile per CTA) whole tiles are dealt
// round robin.  first_tile / skip: where the range begins, last_tile / head:
// where it ends (head pairs of last_tile; 0: it ends with a tile).
struct PpShare {
    int split, first_tile, skip, last_tile, head;
};
enum { kWhole = 0, kHead = 1, kTail = 2 };  // what a CTA runs of a tile

__device__ __forceinline__ void pp_coords(const PpParams &p, int tile, int &tm, int &tn) {
    // strips of tile rows, column-major inside a strip
    const int per = p.strip * p.tiles_n, s = tile / per, w = tile - s * per;
    const int rows = min(p.strip, p.tiles_m - s * p.strip);
    tm = s * p.strip + w % rows;
    tn = w / rows;
}
__device__ __forceinline__ void pp_levels(const PpParams &p, int tm, int tn, int &LA, int &LB) {
    LA = p.la ? min(__ldg(p.la + tm), p.nA) : p.nA;
    LB = p.lb ? min(__ldg(p.lb + tn), p.nB) : p.nB;
}

// Computed by the whole CTA before the roles part (scratch: one int per thread).
__device__ __forceinline__ void pp_share(const PpParams &p, int *scratch, PpShare *out) {
    const int ntiles = p.tiles_m * p.tiles_n, nt = blockDim.x, tid = threadIdx.x;
    const int per = (ntiles + nt - 1) / nt, lo = min(ntiles, tid * per), hi = min(ntiles, lo + per);
    auto count = [&](int tile) {
        int tm, tn, LA, LB;
        pp_coords(p, tile, tm, tn);
        pp_levels(p, tm, tn, LA, LB);
        return pair_count(LA, LB, p.maxlevel);
    };
    int sum = 0, most = 0;
    for (int t = lo; t < hi; t++) {
        const int c = count(t);
        sum += c;
        most = max(most, c);
    }
    scratch[tid] = sum;
    most = __reduce_max_sync(0xffffffffu, most);
    __syncthreads();
    if (tid == 0) {
        int run = 0;
        for (int i = 0; i < nt; i++) {
            const int v = scratch[i];
            scratch[i] = run;
            run += v;
        }
        scratch[nt] = run;
        scratch[nt + 1] = 0;
        out->split = 0;
    }
    __syncthreads();
    if ((tid & 31) == 0) atomicMax(&scratch[nt + 1], most);
    __syncthreads();
    const int64_t total = scratch[nt];
    const int u0 = (int)(total * blockIdx.x / gridDim.x), u1 = (int)(total * (blockIdx.x + 1) / gridDim.x);
    if (total / gridDim.x < scratch[nt + 1] || gridDim.x == 1) return;
    int at = scratch[tid];
    for (int t = lo; t < hi; t++) {
        const int c = count(t);
        if (u0 >= at && u0 < at + c) {
            out->first_tile = t;
            out->skip = u0 - at;
        }
        if (u1 >= at && u1 < at + c) {
            out->last_tile = t;
            out->head = u1 - at;
        }
        at += c;
    }
    if (tid == 0) {
        out->split = 1;
        if (u1 == total) {
            out->last_tile = ntiles;
            out->head = 0;
        }
    }
}

// Calls begin(kind), unit(tm, tn, ia, ib, pair) for the pairs in order and
// end(tm, tn, kind) for every (part of a) tile of the CTA; false stops.
// FUSED: the CTA's share; else (pair, tile) units dealt round robin, pair by
// pair, so the CTAs that run together share the planes of one pair.
template <bool FUSED, typename B, typename U, typename E>
__device__ __forceinline__ void pp_units(const PpParams &p, const PpShare *sh, B begin, U unit, E end) {
    const int ntiles = p.tiles_m * p.tiles_n;
    int tm, tn, a, b;
    if (FUSED) {
        const bool split = sh->split != 0;
        const int first = sh->first_tile, last = sh->last_tile, skip = sh->skip, head = sh->head;
        // split: step 0 the head of last_tile, then the whole tiles, then the tail of first_tile
        const int whole0 = skip > 0 ? first + 1 : first, wholes = last - whole0;
        const int steps = split ? wholes + 2 : (ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
        for (int st = 0; st < steps; st++) {
            int tile, kind = kWhole;
            if (!split) {
                tile = blockIdx.x + st * gridDim.x;
            } else if (st == 0) {
                if (head == 0) continue;
                tile = last;
                kind = kHead;
            } else if (st <= wholes) {
                tile = whole0 + st - 1;
            } else {
                if (skip == 0) continue;
                tile = first;
                kind = kTail;
            }
            pp_coords(p, tile, tm, tn);
            int LA, LB;
            pp_levels(p, tm, tn, LA, LB);
            PairCursor cur(LA, LB, p.maxlevel);
            if (!begin(kind)) return;
            for (int q = 0; cur.next(a, b); q++) {
                if (kind == kTail && q < skip) continue;
                if (kind == kHead && q >= head) break;
                if (!unit(tm, tn, a, b, q)) return;
            }
            if (!end(tm, tn, kind)) return;
        }
    } else {
        const int64_t total = (int64_t)ntiles * p.np;
        for (int64_t u = blockIdx.x; u < total; u += gridDim.x) {
            const int pr = (int)(u / ntiles);
            pp_coords(p, (int)(u - (int64_t)pr * ntiles), tm, tn);
            pair_at(pr, p.nA, p.nB, a, b);
            if ((p.la && a >= __ldg(p.la + tm)) || (p.lb && b >= __ldg(p.lb + tn))) continue;  // the pair is zero here
            if (!unit(tm, tn, a, b, pr)) return;
        }
    }
}

__device__ __forceinline__ double exp_scale(int e) {  // 2^e, or the line's 0 / NaN
    return e == kExpZero ? 0.0 : (e == kExpNaN ? __longlong_as_double(0x7ff8000000000000LL) : pow2(e));
}

// |v| < 2^53 as a double in two FP64 additions: 2^84 + 2^63 + hi 2^32 and
// 2^52 + lo built from their bits, minus the constants (every step exact).
__device__ __forceinline__ double i2d(long long v) {
    const int hi = (int)(v >> 32), lo = (int)v;
    return (__hiloint2double(0x45300000, (int)((uint32_t)hi ^ 0x80000000u)) - 0x1.00000801p84) +
           __hiloint2double(0x43300000, lo);
}
// The exact pair product V 2^e of a pair-buffer entry, 0 or NaN where either
// line's exponent says so, rounded once if it is subnormal.  Not inlined: the
// callers' common case is one test away, and inlined this ran predicated.
__device__ __noinline__ double pair_value(long long v, int bias, int ea, int eb) {
    const bool spa = ea == kExpZero || ea == kExpNaN, spb = eb == kExpZero || eb == kExpNaN;
    const double d = i2d(v);
    if (spa || spb) return d * (spa ? exp_scale(ea) : 1.0) * (spb ? exp_scale(eb) : 1.0);
    const int e = bias + ea + eb;
    return e >= -1022 && e <= 969 ? d * pow2(e) : scale2(d, e);
}

// The <float,double,double> sum's term of c32, the product rounded to float:
// (float)scalbn(c32, tauA + tauB).
__device__ __noinline__ double pair_term_sd(double c32, int ea, int eb) {
    const bool spa = ea == kExpZero || ea == kExpNaN, spb = eb == kExpZero || eb == kExpNaN;
    if (spa || spb) return c32 * (spa ? exp_scale(ea) : 1.0) * (spb ? exp_scale(eb) : 1.0);
    return (double)__double2float_rn(scale2(c32, ea + eb));
}

// a[c] for a run-time c without indexing the register array.
template <int N>
__device__ __forceinline__ long long pick(const long long (&a)[N], int c) {
    long long v = 0;
#pragma unroll
    for (int j = 0; j < N; j++)
        if (j == c) v = a[j];
    return v;
}

// MMA issuer PAR (0, 1): the digit levels of that parity, in their own
// accumulators.  The whole warp walks the units and waits, one elected lane's
// predicate issues: a branch on the lane index costs 80 cycles an MMA (the
// compiler cannot tell that one thread issues), the predicated form 50; the
// waits and commits of a k step add 1300 cycles, which two issuers overlap.
template <int D, bool FUSED, int PAR>
__device__ __forceinline__ void pp_issue(const PpParams &p, const PpShare *sh, uint8_t *smem, uint64_t *full, uint64_t *empty,
                                         uint64_t *acc_full, uint64_t *acc_empty, uint64_t *drain, uint32_t tmem_base,
                                         volatile int *abort_flag, uint64_t wait_ns) {
    using S = PpShape<D>;
    const uint32_t idesc = tc::idesc_i8(128, S::BN);
    const bool lead = tc::elect_one();
    const uint64_t desc0 = tc::smem_desc_k_sw128(tc::smem_u32(smem));  // + 16-byte units within the ring
    uint32_t base = 0, bphase = 0;  // ring slot of the k step's first digit stage, and its phase
    uint32_t units = 0;
    bool ok = true, issued = false;
    pp_units<FUSED>(
        p, sh, [](int) { return true; },
        [&](int, int, int, int, int) {
            for (int kb = 0; kb < p.nkb; kb++) {
                uint32_t sl[D], ph[D];
                uint64_t ad[D];
#pragma unroll
                for (int d = 0; d < D; d++) {
                    sl[d] = base + d;
                    ph[d] = bphase;
                    if (sl[d] >= (uint32_t)S::ST) {
                        sl[d] -= S::ST;
                        ph[d] ^= 1u;
                    }
                    ad[d] = desc0 + sl[d] * (uint32_t)(S::STAGE / 16);
                }
#pragma unroll
                for (int L = PAR; L < S::LV; L += 2) {
                    bool w = true;
                    if (kb == 0 && units > 0)
                        w = tc::mbar_wait(&acc_empty[L], (units - 1) & 1u, abort_flag, p.err, 2, wait_ns);
                    // the digit stages that come into use with this level
#pragma unroll
                    for (int d = (L - 1 > 0 ? L - 1 : 0); d <= L; d++)
                        if (d < D) w = w && tc::mbar_wait(&full[sl[d < D ? d : 0]], ph[d < D ? d : 0], abort_flag, p.err, 2, wait_ns);
                    if (!__all_sync(0xffffffffu, w)) {
                        ok = false;
                        return false;
                    }
                    tc::fence_after_sync();
                    const uint32_t tmem_d = tmem_base + (uint32_t)(L * S::BN);
                    uint32_t accumulate = kb > 0;
#pragma unroll
                    for (int d = 0; d < D; d++) {
                        const int e = L - d;
                        if (e < 0 || e >= D) continue;
#pragma unroll
                        for (int kk = 0; kk < 4; kk++) {
                            tc::mma_i8_if(lead, tmem_d, ad[d] + 2 * kk, ad[e] + S::TILE_A / 16 + 2 * kk, idesc,
                                          accumulate);
                            accumulate = 1;
                        }
                    }
                    issued = true;
                    // stage d serves levels d .. d + D - 1: released after this issuer's last of them
#pragma unroll
                    for (int d = 0; d < D; d++)
                        if (L <= d + D - 1 && L + 2 > d + D - 1) tc::mma_commit_if(lead, &empty[sl[d]]);
                    if (kb == p.nkb - 1) tc::mma_commit_if(lead, &acc_full[L]);
                }
                base += D;
                if (base >= (uint32_t)S::ST) {
                    base -= S::ST;
                    bphase ^= 1u;
                }
            }
            units++;
            return true;
        },
        [](int, int, int) { return true; });
    if (!ok && issued) {  // drain MMAs still in flight before tensor memory is released
        tc::mma_commit_if(lead, drain);
        const uint64_t t0 = tc::globaltimer();
        while (!tc::mbar_try_wait(drain, 0) && tc::globaltimer() - t0 < 100000000ull) {
        }
    }
}

template <int D, int EPI>
__global__ void __launch_bounds__(kPpThreads, 1)
    k_pair_products(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ PpParams p, uint64_t wait_ns, int hold_copies) {
    using S = PpShape<D>;
    constexpr bool FUSED = EPI != kPairStore;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full = (uint64_t *)(smem + S::ST * S::STAGE), *empty = full + S::ST;
    uint64_t *acc_full = empty + S::ST, *acc_empty = acc_full + S::LV, *drain = acc_empty + S::LV;
    int *sbs = (int *)(smem + S::ST * S::STAGE + 512);
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    __shared__ PpShare share;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::ST; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 2);
        }
        for (int l = 0; l < S::LV; l++) {
            tc::mbar_init(&acc_full[l], 1);
            tc::mbar_init(&acc_empty[l], 256);
        }
        tc::mbar_init(drain, 1);
        tc::mbar_init(drain + 1, 1);
        abort_flag = 0;
        tc::fence_mbar_init();
        tc::prefetch_tmap(&tmA);
        tc::prefetch_tmap(&tmB);
    }
    if (warp == 1) tc::tmem_alloc(&tmem_slot, 512);
    if (FUSED) pp_share(p, (int *)smem, &share);  // the ring is free until the roles begin
    tc::fence_proxy_async();                      // and its first copies come after these writes
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = tmem_slot;

    if (warp < 4) {
        tc::reg_dealloc<kPpRegLo>();
        if (warp == 0 && lane == 0) {
            // ---------------------------------------------------------------- producer
            uint32_t slot = 0, phase = 0, issued = 0, issued_phase = 0;
            bool ok = hold_copies == 0;
            if (ok)
                pp_units<FUSED>(
                    p, &share, [](int) { return true; },
                    [&](int tm, int tn, int ia, int ib, int) {
                        for (int kb = 0; kb < p.nkb; kb++)
#pragma unroll
                            for (int d = 0; d < D; d++) {
                                if (!tc::mbar_wait(&empty[slot], phase ^ 1u, &abort_flag, p.err, 1, wait_ns)) {
                                    ok = false;
                                    return false;
                                }
                                uint8_t *sa = smem + slot * S::STAGE;
                                tc::mbar_arrive_expect_tx(&full[slot], S::STAGE);
                                tc::tma_load_3d(sa, &tmA, &full[slot], kb * 128, tm * 128, ia * D + d);
                                tc::tma_load_3d(sa + S::TILE_A, &tmB, &full[slot], kb * 128, p.col0 + tn * S::BN,
                                                ib * D + d);
                                issued |= 1u << slot;
                                issued_phase = (issued_phase & ~(1u << slot)) | (phase << slot);
                                if (++slot == S::ST) {
                                    slot = 0;
                                    phase ^= 1u;
                                }
                            }
                        return true;
                    },
                    [](int, int, int) { return true; });
            if (!ok) tc::drain_copies(full, S::ST, issued, issued_phase);
        } else if (warp == 1) {
            pp_issue<D, FUSED, 0>(p, &share, smem, full, empty, acc_full, acc_empty, drain, tmem_base, &abort_flag, wait_ns);
        } else if (warp == 2) {
            pp_issue<D, FUSED, 1>(p, &share, smem, full, empty, acc_full, acc_empty, drain + 1, tmem_base, &abort_flag, wait_ns);
        }
    } else {
        tc::reg_alloc<kPpRegHi>();
        // ---------------------------------------------------------------- epilogue
        // FP64 instructions make next to no progress while MMAs stream (measured: 48
        // columns' conversions and FMAs 720 cycles alone, 3900 beside N = 96 MMAs, which
        // they do not slow), integer ones run beside them.  So the levels are combined
        // as 64-bit integers, and the three FP64 operations per output that the ordered
        // sum needs run between the read of the last accumulator and its release: the
        // MMAs then wait for that accumulator, which opens the window they run in.
        constexpr int CW = S::CW, LV = S::LV;
        const int q = warp & 3, half = (warp - 4) >> 2;
        const int row = q * 32 + lane;
        const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16) + half * CW;
        int *sb = sbs + (warp - 4) * CW;  // this warp's column exponents, shifted to the exponent field
        constexpr int kShift = EPI == kPairSd ? 23 : 20, kOne = EPI == kPairSd ? 127 : 1023;
        constexpr int kLo = EPI == kPairSd ? -126 : -1022, kHi = EPI == kPairSd ? 73 : 969;
        constexpr int kColZero = -0x7f000000;  // plus any row term below: negative, clamped to a zero scale
        uint32_t units = 0;
        long long acc[CW];
        typename std::conditional<EPI == kPairSd, float, double>::type t[FUSED ? CW : 1];
#pragma unroll
        for (int c = 0; c < (FUSED ? CW : 1); c++) t[c] = 0;
        pp_units<FUSED>(
            p, &share,
            [&](int kind) {
                if (FUSED && kind == kTail) {  // go on from the previous CTA's sums (it ran its part first)
                    bool ok = true;
                    if (lane == 0) {
                        const unsigned *f = p.handed + (blockIdx.x - 1) * 8 + (warp - 4);
                        const uint64_t t0 = tc::globaltimer();
                        unsigned v;
                        for (;;) {
                            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
                            if (v != 0) break;
                            if (abort_flag || tc::globaltimer() - t0 > wait_ns) {
                                abort_flag = 1;
                                atomicExch(p.err, 4);
                                ok = false;
                                break;
                            }
                        }
                    }
                    if (!__all_sync(0xffffffffu, ok)) return false;
                    __syncwarp();
                    const auto *from = reinterpret_cast<decltype(&t[0])>(p.pbuf) +
                                       (size_t)(blockIdx.x - 1) * (128 * S::BN) + (size_t)(half * CW) * 128 + row;
#pragma unroll
                    for (int c = 0; c < (FUSED ? CW : 1); c++) t[c] = __ldcg(from + c * 128);
                }
                return true;
            },
            [&](int tm, int tn, int ia, int ib, int pr) {
                const int gr = tm * 128 + row, gc0 = p.col0 + tn * S::BN + half * CW;
                // the scales do not depend on the MMAs: loaded before the waits
                int ea = 0;
                bool fast = false;
                const short *ebr = nullptr;
                if (FUSED) {
                    ea = gr < p.m ? (int)p.ea[(size_t)ia * p.m + gr] : 0;
                    ebr = p.eb + (size_t)ib * p.n + gc0;
                    int ebmin = 0x7fffffff, ebmax = -0x7fffffff;
                    bool nan = false;
                    __syncwarp();
#pragma unroll
                    for (int c = lane; c < CW; c += 32) {
                        const int e = gc0 + c < p.n ? (int)ebr[c] : 0;
                        sb[c] = e == kExpZero ? kColZero : (int)((uint32_t)e << kShift);
                        nan |= e == kExpNaN;
                        if (e != kExpZero) {
                            ebmin = min(ebmin, e);
                            ebmax = max(ebmax, e);
                        }
                    }
                    ebmin = __reduce_min_sync(0xffffffffu, ebmin);
                    ebmax = __reduce_max_sync(0xffffffffu, ebmax);
                    nan = __any_sync(0xffffffffu, nan);
                    // V 2^(bias + ea + eb) is an exact normal number for every column
                    fast = !nan && ea != kExpNaN && ea != kExpZero && p.bias + ea >= kLo && p.bias + ea <= kHi &&
                           (ebmin > ebmax || (p.bias + ea + ebmin >= kLo && p.bias + ea + ebmax <= kHi));
                    __syncwarp();
                }
#pragma unroll
                for (int L = 0; L < LV; L++) {
                    // the lanes agree before the warp-wide loads
                    if (!__all_sync(0xffffffffu,
                                    tc::mbar_wait(&acc_full[L], units & 1u, &abort_flag, p.err, 3, wait_ns)))
                        return false;
                    tc::fence_after_sync();
                    const int sh = p.radix * (LV - 1 - L);
#pragma unroll
                    for (int c0 = 0; c0 < CW; c0 += 16) {
                        uint32_t v[16];
                        tc::tmem_ld_32x32b_x16(lane_base + L * S::BN + c0, v);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int c = 0; c < 16; c++) {
                            const long long w = (long long)(int)v[c];
                            if (L == 0)
                                acc[c0 + c] = w << sh;
                            else if (LV - 1 - L > 3)  // weights that leave 32 bits
                                acc[c0 + c] += w << sh;
                            else
                                acc[c0 + c] += w * (long long)(1 << sh);
                        }
                    }
                    tc::fence_before_sync();
                    if (!FUSED || L < LV - 1) tc::mbar_arrive(&acc_empty[L]);
                }
                units++;
                if constexpr (EPI == kPairStore) {
                    if (gr < p.m) {
                        long long *o = reinterpret_cast<long long *>(p.pbuf) + ((size_t)pr * p.cn + (gc0 - p.col0)) * p.m +
                                       gr;
                        const int nc = min(CW, p.col0 + p.cn - gc0);
#pragma unroll
                        for (int c = 0; c < CW; c++)
                            if (c < nc) o[(size_t)c * p.m] = acc[c];
                    }
                } else {
                    if (fast) {
                        // the product is exact, so one fma rounds as the addition of the product
                        const int rowhi = (p.bias + ea + kOne) * (1 << kShift);
#pragma unroll
                        for (int c = 0; c < CW; c++) {
                            const int sc = max(rowhi + sb[c], 0);
                            if constexpr (EPI == kPairSd)
                                t[c] = fmaf(__ll2float_rn(acc[c]), __int_as_float(sc), t[c]);
                            else
                                t[c] = fma(i2d(acc[c]), __hiloint2double(sc, 0), t[c]);
                        }
                    } else if (ea != kExpZero) {  // exponents at the ends of the range, NaN lines
#pragma unroll 1
                        for (int c = 0; c < CW; c++) {
                            const int e = gc0 + c < p.n ? (int)ebr[c] : 0;
                            double add;
                            if constexpr (EPI == kPairSd)
                                add = pair_term_sd((double)__ll2float_rn(pick(acc, c)) * pow2(p.bias), ea, e);
                            else
                                add = pair_value(pick(acc, c), p.bias, ea, e);
#pragma unroll
                            for (int j = 0; j < CW; j++)
                                if (j == c) {
                                    if constexpr (EPI == kPairSd)
                                        t[j] = __fadd_rn(t[j], (float)add);
                                    else
                                        t[j] = __dadd_rn(t[j], add);
                                }
                        }
                    }
                    tc::mbar_arrive(&acc_empty[LV - 1]);
                }
                return true;
            },
            [&](int tm, int tn, int kind) {
                if (FUSED && kind == kHead) {
                    auto *to = reinterpret_cast<decltype(&t[0])>(p.pbuf) + (size_t)blockIdx.x * (128 * S::BN) +
                               (size_t)(half * CW) * 128 + row;
#pragma unroll
                    for (int c = 0; c < (FUSED ? CW : 1); c++) {
                        __stcg(to + c * 128, t[c]);
                        t[c] = 0;
                    }
                    __syncwarp();
                    if (lane == 0) {
                        __threadfence();
                        asm volatile("st.release.gpu.global.u32 [%0], 1;" ::"l"(p.handed + blockIdx.x * 8 + (warp - 4))
                                     : "memory");
                    }
                } else if (FUSED) {
                    const int gr = tm * 128 + row, gc0 = p.col0 + tn * S::BN + half * CW;
                    if (gr < p.m) {
#pragma unroll
                        for (int c = 0; c < CW; c++) {
                            if (gc0 + c < p.n) {
                                const size_t at = (size_t)(gc0 + c) * p.ldc + gr;
                                if constexpr (EPI == kPairSd) {
                                    float *cp = reinterpret_cast<float *>(p.C) + at;
                                    *cp = __double2float_rn(fma((double)(float)p.alpha, (double)t[c],
                                                                (double)__fmul_rn((float)p.beta, *cp)));
                                } else {
                                    double *cp = reinterpret_cast<double *>(p.C) + at;
                                    *cp = fma(p.alpha, (double)t[c], p.beta * *cp);
                                }
                            }
                        }
                    }
#pragma unroll
                    for (int c = 0; c < (FUSED ? CW : 1); c++) t[c] = 0;
                }
                return true;
            });
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem_base, 512);
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static int transpose_t(cuozblasHandle_t *h, int rows, int cols, const double *A, int lda, double *out, int ldo) {
    return transpose(h, rows, cols, A, lda, out, ldo);
}
static int transpose_t(cuozblasHandle_t *h, int rows, int cols, const float *A, int lda, float *out, int ldo) {
    return transpose_f32(h, rows, cols, A, lda, out, ldo);
}

// The two ways to the ordered sum, in microseconds as measured: a pair's 128 k
// take 1.35 (D = 3), its hand-over 2 (1.5 more with the sum in the epilogue).
static double pair_us(int k_pad, int D) { return (double)(k_pad / 128) * 0.15 * D * D + 2.0; }

// In the epilogue: every CTA runs an equal share, but no tile meets three CTAs
// (pp_share), so a CTA runs at least a tile's pairs.
static double pair_fused_us(int m, int n, int k_pad, int np, int D) {
    const int64_t tiles = (int64_t)((m + 127) / 128) * ((n + pair_tile_b(D) - 1) / pair_tile_b(D));
    const int64_t share = (tiles * np + sm_count() - 1) / sm_count();
    return (double)(share > np ? share : np) * (pair_us(k_pad, D) + 1.5);
}

// Through a pair buffer: the pairs of a tile spread over the CTAs, then the
// sum.  A buffer beyond L2 is written back while it is read; in column blocks of
// at most 64 MB it stays on chip, at the price of a last wave and two launches
// per block.
struct PairStorePlan {
    int blocks;
    double us;
};
static PairStorePlan pair_store_plan(int m, int n, int k_pad, int np, int D) {
    const int bn = pair_tile_b(D), tn = (n + bn - 1) / bn, tm = (m + 127) / 128;
    PairStorePlan best{1, 1e30};
    for (int blocks = 1; blocks <= 8 && blocks <= tn; blocks++) {
        const int cols = (tn + blocks - 1) / blocks;  // tile columns per block
        const int count = (tn + cols - 1) / cols;
        const double mb = 8e-6 * np * (double)m * (cols * bn < n ? cols * bn : n);
        double us = 0.0;
        for (int b = 0; b < count; b++) {
            const int64_t units = (int64_t)tm * (b + 1 < count ? cols : tn - cols * (count - 1)) * np;
            us += (double)((units + sm_count() - 1) / sm_count()) * pair_us(k_pad, D) + 7.0;
        }
        us += count * mb / (mb <= 64.0 ? 5.0 : 3.5);  // MB / (TB/s) = us
        if (us < best.us) best = PairStorePlan{count, us};
    }
    return best;
}

int pair_products(cuozblasHandle_t *h, const PairDigits &pd, const PairOperand &A, const PairOperand &B,
                  const PairCall &c) {
    State *st = state(h);
    PpParams p;
    p.m = c.m;
    p.n = c.n;
    p.ldc = c.ldc;
    p.nkb = c.k_pad / 128;
    const int bn = pair_tile_b(pd.D);
    p.tiles_m = (c.m + 127) / 128;
    p.col0 = c.col0;
    p.cn = c.cn > 0 ? c.cn : c.n;
    p.tiles_n = (p.cn + bn - 1) / bn;
    p.strip = p.tiles_m < 12 ? p.tiles_m : 12;
    p.nA = c.nA;
    p.nB = c.nB;
    p.maxlevel = c.maxlevel;
    p.np = 0;
    for_each_pair(c.nA, c.nB, c.maxlevel, [&](int, int) { p.np++; });
    p.bias = c.bias;
    p.radix = pd.radix;
    p.la = A.tile_lev;
    p.lb = B.tile_lev ? B.tile_lev + c.col0 / bn : nullptr;
    p.ea = A.exps;
    p.eb = B.exps;
    p.alpha = c.alpha;
    p.beta = c.beta;
    p.C = c.C;
    p.pbuf = c.pbuf;
    p.err = st->d_ints + kPairErrInt;  // cleared by the caller's reset of the counters
    CUtensorMap tmA, tmB;
    OZB_TRY(make_map_planes(&tmA, A.dig, c.k_pad, c.m, (uint64_t)c.nA * pd.D, 128));
    OZB_TRY(make_map_planes(&tmB, B.dig, c.k_pad, c.n, (uint64_t)c.nB * pd.D, bn));
    const int64_t units = (int64_t)p.tiles_m * p.tiles_n * (c.epi == kPairStore ? p.np : 1);
    const int grid = (int)(units < sm_count() ? units : sm_count());
    p.handed = nullptr;
    if (c.epi != kPairStore) {
        p.pbuf = c.pbuf;
        p.handed = reinterpret_cast<unsigned *>(c.pbuf + (size_t)sm_count() * 128 * bn);
        OZB_CHECK(cudaMemsetAsync(p.handed, 0, sizeof(unsigned) * 8 * sm_count(), st->stream));
    }
    // the fused CTAs wait for one another: a cooperative launch
    auto go = [&](auto kern, int smem, std::atomic<uint64_t> &done) -> cudaError_t {
        cudaError_t e = smem_optin((const void *)kern, smem, done);
        if (e != cudaSuccess) return e;
        counted(h);
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(kPpThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st->stream;
        cfg.attrs = &at;
        cfg.numAttrs = c.epi == kPairStore ? 0 : 1;
        return cudaLaunchKernelEx(&cfg, kern, tmA, tmB, p, i8_test_wait_ns(), i8_test_hold_copies());
    };
    static std::atomic<uint64_t> done[6];
    if (pd.D == 3) {
        constexpr int sm = PpShape<3>::SMEM;
        if (c.epi == kPairStore) OZB_CHECK(go(k_pair_products<3, kPairStore>, sm, done[0]));
        if (c.epi == kPairFsum) OZB_CHECK(go(k_pair_products<3, kPairFsum>, sm, done[1]));
        if (c.epi == kPairSd) OZB_CHECK(go(k_pair_products<3, kPairSd>, sm, done[2]));
    } else {
        constexpr int sm = PpShape<4>::SMEM;
        if (c.epi == kPairStore) OZB_CHECK(go(k_pair_products<4, kPairStore>, sm, done[3]));
        if (c.epi == kPairFsum) OZB_CHECK(go(k_pair_products<4, kPairFsum>, sm, done[4]));
        if (c.epi == kPairSd) OZB_CHECK(go(k_pair_products<4, kPairSd>, sm, done[5]));
    }
    return CUOZBLAS_STATUS_SUCCESS;
}

int pair_status(cuozblasHandle_t *h) {
    State *st = state(h);
    OZB_CHECK(cudaMemcpyAsync(st->h_ints, st->d_ints + kPairErrInt, sizeof(int), cudaMemcpyDeviceToHost, st->stream));
    OZB_CHECK(cudaStreamSynchronize(st->stream));
    if (st->h_ints[0] != 0) {
        fprintf(stderr, "cuozblas: INT8 pair-product kernel wait timed out (code %d)\n", st->h_ints[0]);
        return CUOZBLAS_STATUS_DEVICE_TIMEOUT;
    }
    return CUOZBLAS_STATUS_SUCCESS;
}

// The ordered sum of a pair buffer pbuf[p][col][row] of exact integer products V
// (columns col0 .. col0 + cn): FSum in pair order, or NearSum (which overwrites
// the buffer); FLOATS: the <float,double,double> sum, t += (float)scalbn((float)P,
// tauA + tauB).  One thread per output row and kPsCols columns, the loads of
// kPsIn pairs in flight.  A block lists, per column, each pair's A level and
// its part of the exponent, so that a term takes two shared loads and about
// fifteen instructions (with the list found per term and both forms of it
// inlined a term took 74, and the code did not fit the instruction cache).
// Entries of pairs that the product kernel skipped hold anything: the lines'
// marks at those levels make them zeros.  *err: a wait of the product kernel ran
// out, so the buffer is not complete and C stays as it is (a warp without a part
// in the lists reads the word: by every thread into a register, or by the first
// warp, it cost 3 us of the 278 of a call at 1024^3).
constexpr int kPsRows = 256, kPsCols = 2, kPsIn = 16;
constexpr int kPsLevels = 12, kPsPairs = 144;  // held in shared memory; k_pair_sum_any beyond

template <bool FLOATS>
__device__ __noinline__ double pair_term(long long v, int bias, int a, int b) {
    return FLOATS ? pair_term_sd((double)__ll2float_rn(v) * pow2(bias), a, b) : pair_value(v, bias, a, b);
}

template <bool FLOATS>
__device__ __forceinline__ void pair_out(void *Cv, size_t at, double alpha, double beta, double t, float tf) {
    if (FLOATS) {
        float *cp = reinterpret_cast<float *>(Cv) + at;
        *cp = __double2float_rn(fma((double)(float)alpha, (double)tf, (double)__fmul_rn((float)beta, *cp)));
    } else {
        double *cp = reinterpret_cast<double *>(Cv) + at;
        *cp = fma(alpha, t, beta * *cp);
    }
}

template <bool FLOATS>
__global__ void __launch_bounds__(kPsRows, 4)
    k_pair_sum(int m, int n, int col0, int cn, int nA, int nB, int np, const double *__restrict__ pbuf,
               const short *__restrict__ ea, const short *__restrict__ eb, int bias, double alpha, double beta,
               void *__restrict__ Cv, int ldc, const int *__restrict__ err) {
    __shared__ int failed;
    __shared__ short sA[kPsLevels][kPsRows];
    __shared__ int2 sP[kPsCols][kPsPairs];  // A level, B level's tau
    const int rb = (m + kPsRows - 1) / kPsRows, tr = threadIdx.x;
    const int row = (int)(blockIdx.x % rb) * kPsRows + tr, c0 = col0 + (int)(blockIdx.x / rb) * kPsCols;
    const int nc = min(kPsCols, col0 + cn - c0);
    if (row < m)
        for (int s = 0; s < nA; s++) sA[s][tr] = ea[(size_t)s * m + row];
    if (tr == kPsRows - 1) failed = *err;  // beside the first warps' lists
    for (int i = tr; i < np * nc; i += kPsRows) {
        const int q = i / nc, c = i - q * nc;
        int ia, ib;
        pair_at(q, nA, nB, ia, ib);
        sP[c][q] = make_int2(ia, eb[(size_t)ib * n + c0 + c]);
    }
    __syncthreads();
    if (row >= m) return;
    const size_t count = (size_t)m * cn;
    for (int c = 0; c < nc; c++) {
        const double *pe = pbuf + (size_t)(c0 + c - col0) * m + row;
        double t = 0.0;
        float tf = 0.f;
        for (int q0 = 0; q0 < np; q0 += kPsIn) {
            long long v[kPsIn];
#pragma unroll
            for (int j = 0; j < kPsIn; j++) v[j] = __double_as_longlong(pe[(size_t)min(q0 + j, np - 1) * count]);
#pragma unroll
            for (int j = 0; j < kPsIn; j++) asm volatile("" : "+l"(v[j]));  // all loaded here, not each at its use
#pragma unroll
            for (int j = 0; j < kPsIn; j++) {
                if (q0 + j < np) {  // uniform
                    const int2 pr = sP[c][q0 + j];
                    const int a = sA[pr.x][tr], e = bias + a + pr.y;
                    // V 2^e is exact when e is well inside the range: one fma rounds as the addition.  The
                    // line marks lie far outside, so one test sends them to the general form.
                    if (FLOATS) {
                        if (e >= -126 && e <= 73)  // float(V) has at most 24 bits
                            tf = fmaf(__ll2float_rn(v[j]), __int_as_float((e + 127) << 23), tf);
                        else
                            tf = __fadd_rn(tf, (float)pair_term<true>(v[j], bias, a, pr.y));
                    } else {
                        if (e >= -1022 && e <= 969)
                            t = fma(i2d(v[j]), __hiloint2double((e + 1023) << 20, 0), t);
                        else
                            t = __dadd_rn(t, pair_term<false>(v[j], bias, a, pr.y));
                    }
                }
            }
        }
        if (failed == 0) pair_out<FLOATS>(Cv, (size_t)(c0 + c) * ldc + row, alpha, beta, t, tf);
    }
}

// The same without the shared lists (any counts), and NearSum.
template <bool FLOATS>
__global__ void __launch_bounds__(256)
    k_pair_sum_any(int m, int n, int col0, int cn, int nA, int nB, int maxlevel, int np, double *__restrict__ pbuf,
                   const short *__restrict__ ea, const short *__restrict__ eb, int bias, int sum_mode, double alpha,
                   double beta, void *__restrict__ Cv, int ldc, const int *__restrict__ err) {
    const int failed = *err;
    const int rb = (m + 255) / 256;
    const int row = (int)(blockIdx.x % rb) * 256 + threadIdx.x, col = col0 + (int)(blockIdx.x / rb);
    if (row >= m) return;
    const size_t count = (size_t)m * cn;
    double *pe = pbuf + (size_t)(col - col0) * m + row;
    double t = 0.0;
    float tf = 0.f;
    int p = 0;
    for_each_pair(nA, nB, maxlevel, [&](int ia, int ib) {
        double *v = pe + (size_t)p++ * count;
        const double term =
            pair_term<FLOATS>(__double_as_longlong(*v), bias, ea[(size_t)ia * m + row], eb[(size_t)ib * n + col]);
        if (FLOATS)
            tf = __fadd_rn(tf, (float)term);
        else if (sum_mode == 1)
            *v = term;
        else
            t = __dadd_rn(t, term);
    });
    if (!FLOATS && sum_mode == 1) t = nearsum(np, pe, (int64_t)count);
    if (failed == 0) pair_out<FLOATS>(Cv, (size_t)col * ldc + row, alpha, beta, t, tf);
}

// C = alpha op(A) op(B) + beta C with m, n > 1 in the plain form (T = double)
// or <float,double,double> (T = float): split, exact pair products, ordered
// sum.  *done stays false when the form does not apply (digits, arena): the
// caller's slice path then runs.
template <typename T>
int gemm_pairs_core(cuozblasHandle_t *h, char ta, char tb, int m, int n, int k, double alpha, const T *A, int lda,
                    const T *B, int ldb, double beta, T *C, int ldc, int fastMode, int rho, bool *done) {
    constexpr bool kFloats = sizeof(T) == 4;
    constexpr int kMant = SplitRange<T>::kMant;
    State *st = state(h);
    *done = false;
    const PairDigits pd = pair_digits(kMant - rho, k);
    if (pd.D == 0 || k == 0) return CUOZBLAS_STATUS_SUCCESS;
    const int maxS = h->nSplitMax > 0 ? h->nSplitMax : kMaxSplitDefault;
    const int k_pad = (k + 127) / 128 * 128;
    const int tile[2] = {kPairTileA, pair_tile_b(pd.D)};
    const uint64_t mark0 = Arena(h).mark();
    int zmax[2] = {0, 0}, ns[2] = {0, 0};
    PairOperand op[2];
    // Planes for 8 levels; data whose lines span more is split again with planes for all of them.
    int levels[2] = {maxS < 8 ? maxS : 8, maxS < 8 ? maxS : 8};
    for (int attempt = 0;; attempt++) {
        Arena ar(h);
        ar.release(mark0);
        for (int o = 0; o < 2; o++) {
            op[o].nl = o == 0 ? m : n;
            op[o].levels = levels[o];
            op[o].dig = ar.take<int8_t>((uint64_t)levels[o] * pd.D * op[o].nl * k_pad);
            op[o].exps = ar.take<short>((uint64_t)levels[o] * op[o].nl);
            op[o].tile_lev = ar.take<int>((op[o].nl + tile[o] - 1) / tile[o]);
        }
        if (!ar.ok) {
            ar.release(mark0);
            return CUOZBLAS_STATUS_SUCCESS;
        }
        const uint64_t mark1 = ar.mark();
        phases_begin(h);
        OZB_CHECK(cudaMemsetAsync(st->d_ints, 0, (kPairErrInt + 1) * sizeof(int), st->stream));
        for (int o = 0; o < 2; o++) {
            const bool strided = o == 0 ? !is_trans(ta) : is_trans(tb);
            const T *X = o == 0 ? A : B;
            int ldx = o == 0 ? lda : ldb;
            if (strided) {  // element (line l, i) at X[i * ldx + l]
                const int ldt = (k + 1) / 2 * 2;
                T *tmp = ar.take<T>((uint64_t)op[o].nl * ldt);
                if (!ar.ok) {
                    ar.release(mark0);
                    return CUOZBLAS_STATUS_SUCCESS;
                }
                OZB_TRY(transpose_t(h, op[o].nl, k, X, ldx, tmp, ldt));
                X = tmp;
                ldx = ldt;
            }
            const int r = pair_split(h, k, k_pad, X, ldx, rho, maxS, pd, tile[o], op[o], st->d_ints + o);
            if (r == CUOZBLAS_STATUS_WORKSPACE) {
                ar.release(mark0);
                return CUOZBLAS_STATUS_SUCCESS;
            }
            OZB_TRY(r);
            ar.release(mark1);
            ev_record(h, o + 1);
        }
        OZB_CHECK(cudaMemcpyAsync(st->h_ints, st->d_ints, 2 * sizeof(int), cudaMemcpyDeviceToHost, st->stream));
        OZB_CHECK(cudaStreamSynchronize(st->stream));
        bool again = false;
        for (int o = 0; o < 2; o++) {
            const int c = (st->h_ints[o] < 1 ? 1 : st->h_ints[o]) + 1;
            ns[o] = c < maxS ? c : maxS;
            zmax[o] = st->h_ints[o] + 1 < maxS ? st->h_ints[o] + 1 : maxS;  // levels with a slice
            if (zmax[o] > levels[o]) {
                levels[o] = zmax[o];
                again = true;
            }
        }
        if (!again || attempt > 0) break;
    }
    const int nA = ns[0], nB = ns[1];
    int maxlevel = (nA - 1) + (nB - 1);
    {
        const int mn = nA - 1 < nB - 1 ? nA - 1 : nB - 1;
        maxlevel = (maxlevel - fastMode) > mn ? (maxlevel - fastMode) : mn;  // src/cpu/ozblas_gemm.cpp:163-164
    }
    int np = 0;
    for_each_pair(nA, nB, maxlevel, [&](int, int) { np++; });
    h->nSplitA = (float)nA;
    h->nSplitB = (float)nB;
    h->nSplitC = (float)np;
    h->mbk = m;
    h->nbk = n;
    // Levels without a slice anywhere (the count includes one when level 0 is
    // exact) add zeros: their pairs are left out.
    PairCall c;
    c.m = m;
    c.n = n;
    c.k_pad = k_pad;
    c.nA = nA < zmax[0] ? nA : zmax[0];
    c.nB = nB < zmax[1] ? nB : zmax[1];
    c.maxlevel = maxlevel < c.nA + c.nB - 2 ? maxlevel : c.nA + c.nB - 2;
    c.bias = 2 * (rho - kMant);
    c.alpha = alpha;
    c.beta = beta;
    c.C = C;
    c.ldc = ldc;
    int npu = 0;
    for_each_pair(c.nA, c.nB, c.maxlevel, [&](int, int) { npu++; });
    Arena ar(h);
    const bool near = !kFloats && h->sumMode == 1;
    c.epi = kFloats ? kPairSd : kPairFsum;
    const PairStorePlan sp = pair_store_plan(m, n, k_pad, npu, pd.D);
    if (near || sp.us < pair_fused_us(m, n, k_pad, npu, pd.D)) {
        // in column blocks: as many as the plan asks for, or as the arena does.  A block is whole tiles:
        // the plan's rounded up, or what the arena holds rounded down.
        const uint64_t avail = h->workSizeBytes - ((ar.mark() + 255) / 256 * 256);
        int64_t cols = (n + sp.blocks - 1) / sp.blocks;
        const int64_t most = (int64_t)(avail / (sizeof(double) * (uint64_t)npu * (uint64_t)m));
        if (cols < n) cols = (cols + tile[1] - 1) / tile[1] * tile[1];
        if (cols > most) cols = most / tile[1] * tile[1];
        if (cols > 0) {
            c.cn = (int)cols;
            c.pbuf = ar.take<double>((uint64_t)npu * m * cols);
            c.epi = kPairStore;
        } else if (near) {  // the slice path blocks the columns further
            ar.release(mark0);
            return CUOZBLAS_STATUS_SUCCESS;
        }
        if (!ar.ok) {
            ar.release(mark0);
            return CUOZBLAS_STATUS_SUCCESS;
        }
    }
    if (c.epi == kPairStore) {
        const int cols = c.cn;
        for (int c0 = 0; c0 < n; c0 += cols) {
            c.col0 = c0;
            c.cn = n - c0 < cols ? n - c0 : cols;
            OZB_TRY(pair_products(h, pd, op[0], op[1], c));
            if (c0 + cols >= n) ev_record(h, 3);
            counted(h);
            if (!near && c.nA <= kPsLevels && npu <= kPsPairs)
                k_pair_sum<kFloats><<<(unsigned)((int64_t)((m + kPsRows - 1) / kPsRows) * ((c.cn + kPsCols - 1) / kPsCols)),
                                      kPsRows, 0, st->stream>>>(m, n, c0, c.cn, c.nA, c.nB, npu, c.pbuf, op[0].exps,
                                                                op[1].exps, c.bias, alpha, beta, C, ldc,
                                                                st->d_ints + kPairErrInt);
            else
                k_pair_sum_any<kFloats><<<(unsigned)((int64_t)((m + 255) / 256) * c.cn), 256, 0, st->stream>>>(
                    m, n, c0, c.cn, c.nA, c.nB, c.maxlevel, npu, c.pbuf, op[0].exps, op[1].exps, c.bias, h->sumMode,
                    alpha, beta, C, ldc, st->d_ints + kPairErrInt);
            OZB_CHECK(cudaGetLastError());
        }
    } else {
        c.pbuf = ar.take<double>(pair_handover_doubles(pd.D));
        if (!ar.ok) {
            ar.release(mark0);
            return CUOZBLAS_STATUS_SUCCESS;
        }
        OZB_TRY(pair_products(h, pd, op[0], op[1], c));
        ev_record(h, 3);  // the ordered sum runs inside the product kernel
    }
    ev_record(h, 4);
    *done = true;
    return pair_status(h);
}
template int gemm_pairs_core<double>(cuozblasHandle_t *, char, char, int, int, int, double, const double *, int,
                                     const double *, int, double, double *, int, int, int, bool *);
template int gemm_pairs_core<float>(cuozblasHandle_t *, char, char, int, int, int, double, const float *, int,
                                    const float *, int, double, float *, int, int, int, bool *);

}  // namespace ozb
