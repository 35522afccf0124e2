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
//     What is left is the shared-memory port: a 128 x 96 x 32 MMA reads 7 KB (57
//     cycles at 128 B a clock, against 48 of math), and the TMA writes share it.
//   * Where a tile's lines have no slice at a level (the counts are those of the
//     worst line of the whole operand), its pairs are skipped: they add zero.
// Product kernel, before (one digit level at a time, pair buffer, 7-bit digits)
// and now, one B200: 1024^3 plain, 16 pairs, 1076 -> 268 us; 3001 x 1999 x 2500
// plain, 20 pairs, 4.08 (and 0.15 for the sum) -> 2.33 ms; 2048^3
// <float,double,double>, 9 pairs, 1.73 (0.10) -> 0.81 ms.  Split to digit
// planes (count, FP64 slices, digits in three passes before), 3001 lines of
// 2500: 374 -> 54 us.
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
// stages (digit d of A and of B for one k step) by TMA into a ring, warp 1
// issues the MMAs, warps 4-11 read the accumulators.  Every wait is bounded.
// ---------------------------------------------------------------------------
constexpr int kPpThreads = 384;
constexpr uint32_t kPpRegLo = 40, kPpRegHi = 232;  // 4 x 40 + 8 x 232 = 12 x 168 registers at launch

template <int D>
struct PpShape {
    static constexpr int BN = D == 3 ? 96 : 64;
    static constexpr int LV = 2 * D - 1;                // 5 x 96 = 480 or 7 x 64 = 448 tensor-memory columns
    static constexpr int TILE_A = 128 * 128, TILE_B = BN * 128, STAGE = TILE_A + TILE_B;
    static constexpr int ST = D == 3 ? 7 : 8;
    static constexpr int SMEM = ST * STAGE + 1024 /*align*/ + 512 /*barriers*/ + 8 * (BN / 2) * 8 /*column scales*/;
    static constexpr int CW = BN / 2;                   // columns per epilogue warp
};

struct PpParams {
    int m, n, ldc, nkb, tiles_m, tiles_n, strip;
    int nA, nB, maxlevel, np, bias, radix;
    const int *la, *lb;  // levels in use per tile, or null
    const short *ea, *eb;
    double alpha, beta;
    void *C;
    double *pbuf;
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

// Calls unit(tm, tn, ia, ib, pair) for the CTA's units in order, and
// tile_end(tm, tn) after the last unit of a tile; both return false to stop.
// FUSED: all pairs of tiles blockIdx.x, + gridDim.x, ...; else (pair, tile)
// units dealt round robin, pair by pair, so the CTAs that run together share
// the planes of one pair.
template <bool FUSED, typename U, typename E>
__device__ __forceinline__ void pp_units(const PpParams &p, U unit, E tile_end) {
    const int ntiles = p.tiles_m * p.tiles_n;
    auto coords = [&](int tile, int &tm, int &tn) {  // strips of tile rows, column-major inside a strip
        const int per = p.strip * p.tiles_n, s = tile / per, w = tile - s * per;
        const int rows = min(p.strip, p.tiles_m - s * p.strip);
        tm = s * p.strip + w % rows;
        tn = w / rows;
    };
    int tm, tn, a, b;
    if (FUSED) {
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            coords(tile, tm, tn);
            PairCursor cur(p.la ? min(__ldg(p.la + tm), p.nA) : p.nA, p.lb ? min(__ldg(p.lb + tn), p.nB) : p.nB, p.maxlevel);
            int q = 0;
            while (cur.next(a, b))
                if (!unit(tm, tn, a, b, q++)) return;
            if (!tile_end(tm, tn)) return;
        }
    } else {
        const int64_t total = (int64_t)ntiles * p.np;
        for (int64_t u = blockIdx.x; u < total; u += gridDim.x) {
            const int pr = (int)(u / ntiles);
            coords((int)(u - (int64_t)pr * ntiles), tm, tn);
            pair_at(pr, p.nA, p.nB, a, b);
            if ((p.la && a >= __ldg(p.la + tm)) || (p.lb && b >= __ldg(p.lb + tn))) continue;  // the pair is zero here
            if (!unit(tm, tn, a, b, pr) || !tile_end(tm, tn)) return;
        }
    }
}

__device__ __forceinline__ double exp_scale(int e) {  // 2^e, or the line's 0 / NaN
    return e == kExpZero ? 0.0 : (e == kExpNaN ? __longlong_as_double(0x7ff8000000000000LL) : pow2(e));
}

// INT32 -> FP64 without the conversion unit (a quarter of the FP64 rate):
// 2^52 + 2^31 + w built from its bits, minus the constant (exact).
__device__ __forceinline__ double i2d(uint32_t w) {
    return __hiloint2double(0x43300000, (int)(w ^ 0x80000000u)) - 4503601774854144.0;
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
    double *sbs = (double *)(smem + S::ST * S::STAGE + 512);
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::ST; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int l = 0; l < S::LV; l++) {
            tc::mbar_init(&acc_full[l], 1);
            tc::mbar_init(&acc_empty[l], 256);
        }
        tc::mbar_init(drain, 1);
        abort_flag = 0;
        tc::fence_mbar_init();
        tc::prefetch_tmap(&tmA);
        tc::prefetch_tmap(&tmB);
    }
    if (warp == 1) tc::tmem_alloc(&tmem_slot, 512);
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
                    p,
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
                                tc::tma_load_3d(sa + S::TILE_A, &tmB, &full[slot], kb * 128, tn * S::BN, ib * D + d);
                                issued |= 1u << slot;
                                issued_phase = (issued_phase & ~(1u << slot)) | (phase << slot);
                                if (++slot == S::ST) {
                                    slot = 0;
                                    phase ^= 1u;
                                }
                            }
                        return true;
                    },
                    [](int, int) { return true; });
            if (!ok) tc::drain_copies(full, S::ST, issued, issued_phase);
        } else if (warp == 1) {
            // ---------------------------------------------------------------- MMA issuer
            // The whole warp walks the units and waits; one elected lane issues.  (A
            // branch on the lane index instead costs 80 cycles an MMA against 57: the
            // compiler then cannot tell that a single thread issues.)
            const uint32_t idesc = tc::idesc_i8(128, S::BN);
            uint32_t base = 0, bphase = 0;  // ring slot of the k step's first digit stage, and its phase
            uint32_t units = 0;
            bool ok = true, issued = false;
            pp_units<FUSED>(
                p,
                [&](int, int, int, int, int) {
                    for (int kb = 0; kb < p.nkb; kb++) {
                        uint32_t sl[D], ph[D];
#pragma unroll
                        for (int d = 0; d < D; d++) {
                            sl[d] = base + d;
                            ph[d] = bphase;
                            if (sl[d] >= (uint32_t)S::ST) {
                                sl[d] -= S::ST;
                                ph[d] ^= 1u;
                            }
                        }
#pragma unroll
                        for (int L = 0; L < S::LV; L++) {
                            bool w = true;
                            if (kb == 0 && units > 0)
                                w = tc::mbar_wait(&acc_empty[L], (units - 1) & 1u, &abort_flag, p.err, 2, wait_ns);
                            if (L < D)  // levels 0 .. D - 1 bring in one digit stage each
                                w = w && tc::mbar_wait(&full[sl[L < D ? L : 0]], ph[L < D ? L : 0], &abort_flag, p.err, 2,
                                                       wait_ns);
                            if (!__all_sync(0xffffffffu, w)) {
                                ok = false;
                                return false;
                            }
                            tc::fence_after_sync();
                            if (tc::elect_one()) {
                                const uint32_t tmem_d = tmem_base + (uint32_t)(L * S::BN);
                                uint32_t accumulate = kb > 0;
#pragma unroll
                                for (int d = 0; d < D; d++) {
                                    const int e = L - d;
                                    if (e < 0 || e >= D) continue;
                                    const uint64_t ad = tc::smem_desc_k_sw128(tc::smem_u32(smem + sl[d] * S::STAGE));
                                    const uint64_t bd =
                                        tc::smem_desc_k_sw128(tc::smem_u32(smem + sl[e] * S::STAGE + S::TILE_A));
#pragma unroll
                                    for (int kk = 0; kk < 4; kk++) {
                                        tc::mma_i8(tmem_d, ad + 2 * kk, bd + 2 * kk, idesc, accumulate);
                                        accumulate = 1;
                                    }
                                }
                                // stage L - D + 1 serves levels up to L
                                if (L >= D - 1) tc::mma_commit(&empty[sl[L >= D - 1 ? L - (D - 1) : 0]]);
                                if (kb == p.nkb - 1) tc::mma_commit(&acc_full[L]);
                            }
                            __syncwarp();
                            issued = true;
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
                [](int, int) { return true; });
            if (!ok && issued) {  // drain MMAs still in flight before tensor memory is released
                if (tc::elect_one()) tc::mma_commit(drain);
                const uint64_t t0 = tc::globaltimer();
                while (!tc::mbar_try_wait(drain, 0) && tc::globaltimer() - t0 < 100000000ull) {
                }
            }
        }
    } else {
        tc::reg_alloc<kPpRegHi>();
        // ---------------------------------------------------------------- epilogue
        constexpr int CW = S::CW;
        const int q = warp & 3, half = (warp - 4) >> 2;
        const int row = q * 32 + lane;
        const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16) + half * CW;
        double *sb = sbs + (warp - 4) * CW;  // this warp's column scales
        const double rad = p.radix == 8 ? 256.0 : 128.0;
        uint32_t units = 0;
        double acc[CW];
        typename std::conditional<EPI == kPairSd, float, double>::type t[FUSED ? CW : 1];
#pragma unroll
        for (int c = 0; c < (FUSED ? CW : 1); c++) t[c] = 0;
        pp_units<FUSED>(
            p,
            [&](int tm, int tn, int ia, int ib, int pr) {
                const int gr = tm * 128 + row, gc0 = tn * S::BN + half * CW;
                // the scales do not depend on the MMAs: loaded before the waits
                int ea = p.ea && gr < p.m ? (int)p.ea[(size_t)ia * p.m + gr] : 0;
                int ebmin = 0x7fffffff, ebmax = -0x7fffffff;
                __syncwarp();
#pragma unroll
                for (int c = lane; c < CW; c += 32) {
                    const int e = p.eb && gc0 + c < p.n ? (int)p.eb[(size_t)ib * p.n + gc0 + c] : 0;
                    sb[c] = exp_scale(e);
                    if (e != kExpZero && e != kExpNaN) {
                        ebmin = min(ebmin, e);
                        ebmax = max(ebmax, e);
                    }
                }
                ebmin = __reduce_min_sync(0xffffffffu, ebmin);
                ebmax = __reduce_max_sync(0xffffffffu, ebmax);
                const bool special = ea == kExpZero || ea == kExpNaN;
                // V * 2^(bias + ea) and its product with 2^eb are exact normal numbers for every column
                constexpr int kLo = EPI == kPairSd ? -126 : -1022, kHi = EPI == kPairSd ? 73 : 969;
                const bool fast = special || ebmin > ebmax ||
                                  (p.bias + ea >= kLo && p.bias + ea <= kHi && p.bias + ea + ebmin >= kLo &&
                                   p.bias + ea + ebmax <= kHi && ebmin >= kLo && ebmax <= kHi + 53);
                const double sa = special ? exp_scale(ea) : pow2(p.bias + ea);
#pragma unroll
                for (int L = 0; L < S::LV; L++) {
                    // the lanes agree before the warp-wide loads
                    if (!__all_sync(0xffffffffu,
                                    tc::mbar_wait(&acc_full[L], units & 1u, &abort_flag, p.err, 3, wait_ns)))
                        return false;
                    tc::fence_after_sync();
#pragma unroll
                    for (int c0 = 0; c0 < CW; c0 += 16) {
                        uint32_t v[16];
                        tc::tmem_ld_32x32b_x16(lane_base + L * S::BN + c0, v);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int c = 0; c < 16; c++) acc[c0 + c] = L == 0 ? i2d(v[c]) : fma(acc[c0 + c], rad, i2d(v[c]));
                    }
                    tc::fence_before_sync();
                    tc::mbar_arrive(&acc_empty[L]);
                }
                units++;
                __syncwarp();
                if constexpr (EPI == kPairStore) {
                    if (gr < p.m) {
                        double *o = p.pbuf + ((size_t)pr * p.n + gc0) * p.m + gr;
                        const int nc = min(CW, p.n - gc0);
                        const short *ebr = p.eb ? p.eb + (size_t)ib * p.n + gc0 : nullptr;
#pragma unroll
                        for (int c = 0; c < CW; c++)
                            if (c < nc) {
                                if (fast) {
                                    o[(size_t)c * p.m] = (acc[c] * sa) * sb[c];
                                } else {
                                    const int e = ebr ? (int)ebr[c] : 0;
                                    o[(size_t)c * p.m] = e == kExpZero || e == kExpNaN ? acc[c] * exp_scale(e)
                                                                                       : scale2(acc[c], p.bias + ea + e);
                                }
                            }
                    }
                } else if constexpr (EPI == kPairFsum) {
                    // the product is exact, so one fma rounds as the addition of the product
                    if (fast) {
#pragma unroll
                        for (int c = 0; c < CW; c++) t[c] = fma(acc[c] * sa, sb[c], t[c]);
                    } else {
                        const short *ebr = p.eb + (size_t)ib * p.n;
#pragma unroll
                        for (int c = 0; c < CW; c++) {
                            const int e = gc0 + c < p.n ? (int)ebr[gc0 + c] : 0;
                            t[c] = __dadd_rn(t[c], e == kExpZero || e == kExpNaN ? acc[c] * exp_scale(e)
                                                                                : scale2(acc[c], p.bias + ea + e));
                        }
                    }
                } else {
                    const float saf = (float)sa;
                    if (fast) {
#pragma unroll
                        for (int c = 0; c < CW; c++)
                            t[c] = fmaf(__double2float_rn(acc[c]) * saf, (float)sb[c], t[c]);
                    } else {
                        const short *ebr = p.eb + (size_t)ib * p.n;
#pragma unroll
                        for (int c = 0; c < CW; c++) {
                            const int e = gc0 + c < p.n ? (int)ebr[gc0 + c] : 0;
                            const double c32 = (double)__double2float_rn(acc[c] * pow2(p.bias));
                            t[c] = __fadd_rn(t[c], __double2float_rn(e == kExpZero || e == kExpNaN ? c32 * exp_scale(e)
                                                                                                  : scale2(c32, ea + e)));
                        }
                    }
                }
                return true;
            },
            [&](int tm, int tn) {
                if (FUSED) {
                    const int gr = tm * 128 + row, gc0 = tn * S::BN + half * CW;
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

bool pair_fuse_sum(int m, int n, int k_pad, int np, int D) {
    const int64_t tiles = (int64_t)((m + 127) / 128) * ((n + pair_tile_b(D) - 1) / pair_tile_b(D));
    const int sms = sm_count();
    // microseconds: a pair's MMAs over 128 k (D^2 products of 4 MMAs at about 56 cycles) and its
    // hand-over, against the pair buffer written and read back at about 3 TB/s
    const double pair_us = (double)(k_pad / 128) * D * D * 4 * 56e-3 / 1.9 + 1.0;
    const double fused = (double)((tiles + sms - 1) / sms) * np * pair_us;
    const double split = (double)((tiles * np + sms - 1) / sms) * pair_us + 16.0 * np * (double)m * n / 3e6 + 4.0;
    return fused <= split;
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
    p.tiles_n = (c.n + bn - 1) / bn;
    p.strip = p.tiles_m < 12 ? p.tiles_m : 12;
    p.nA = c.nA;
    p.nB = c.nB;
    p.maxlevel = c.maxlevel;
    p.np = 0;
    for_each_pair(c.nA, c.nB, c.maxlevel, [&](int, int) { p.np++; });
    p.bias = c.bias;
    p.radix = pd.radix;
    p.la = A.tile_lev;
    p.lb = B.tile_lev;
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
    auto go = [&](auto kern, int smem, std::atomic<uint64_t> &done) -> cudaError_t {
        const cudaError_t e = smem_optin((const void *)kern, smem, done);
        if (e != cudaSuccess) return e;
        counted(h);
        kern<<<grid, kPpThreads, smem, st->stream>>>(tmA, tmB, p, i8_test_wait_ns(), i8_test_hold_copies());
        return cudaGetLastError();
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

// The ordered sum of a pair buffer pbuf[p][col][row] of exact products: FSum
// in pair order, or NearSum (which overwrites the buffer); FLOATS: the
// <float,double,double> sum, t += (float)scalbn((float)P, tauA + tauB).  One
// thread per output, the loads of 4 pairs in flight; pairs that the product
// kernel skipped (levels not in use in the tile) are skipped here too.
template <bool FLOATS>
__global__ void __launch_bounds__(256) k_pair_sum(int m, int n, int nA, int nB, int maxlevel, int np,
                                                  double *__restrict__ pbuf, const int *__restrict__ la,
                                                  const int *__restrict__ lb, int tile_b,
                                                  const short *__restrict__ ea, const short *__restrict__ eb,
                                                  int sum_mode, double alpha, double beta, void *__restrict__ Cv,
                                                  int ldc) {
    const int rb = (m + 255) / 256, col = blockIdx.x / rb, row = (blockIdx.x - col * rb) * 256 + threadIdx.x;
    if (row >= m) return;
    const size_t count = (size_t)m * n;
    double *pe = pbuf + (size_t)col * m + row;
    const size_t at = (size_t)col * ldc + row;
    if (!FLOATS && sum_mode == 1) {
        double *cp = reinterpret_cast<double *>(Cv) + at;
        *cp = fma(alpha, nearsum(np, pe, (int64_t)count), beta * *cp);
        return;
    }
    const int LA = la ? min(la[row / kPairTileA], nA) : nA, LB = lb ? min(lb[col / tile_b], nB) : nB;
    double t = 0.0;
    float tf = 0.f;
    int p = 0;
    for (int ik = 0; ik <= maxlevel; ik++) {
        const int lo = max(0, ik - (nB - 1)), hi = min(ik, nA - 1);
        const int from = max(lo, ik - (LB - 1)), to = min(hi, LA - 1);  // the pairs in use
#pragma unroll 4
        for (int ia = from; ia <= to; ia++) {
            const double v = __ldcs(pe + (size_t)(p + ia - lo) * count);
            if (FLOATS) {
                const int a = ea[(size_t)ia * m + row], b = eb[(size_t)(ik - ia) * n + col];
                const double c32 = (double)__double2float_rn(v);
                const bool special = a == kExpZero || a == kExpNaN || b == kExpZero || b == kExpNaN;
                tf = __fadd_rn(tf, __double2float_rn(special ? c32 * (a == kExpZero || a == kExpNaN ? exp_scale(a) : 1.0) *
                                                                   (b == kExpZero || b == kExpNaN ? exp_scale(b) : 1.0)
                                                             : scale2(c32, a + b)));
            } else {
                t += v;
            }
        }
        p += hi - lo + 1;
    }
    if (FLOATS) {
        float *cp = reinterpret_cast<float *>(Cv) + at;
        *cp = __double2float_rn(fma((double)(float)alpha, (double)tf, (double)__fmul_rn((float)beta, *cp)));
    } else {
        double *cp = reinterpret_cast<double *>(Cv) + at;
        *cp = fma(alpha, t, beta * *cp);
    }
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
        ev_record(h, 0);
        st->plain_timers = true;
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
    if (near || !pair_fuse_sum(m, n, k_pad, npu, pd.D)) {
        c.pbuf = ar.take<double>((uint64_t)npu * m * n);
        if (ar.ok)
            c.epi = kPairStore;
        else if (near) {  // the slice path blocks the columns
            ar.release(mark0);
            return CUOZBLAS_STATUS_SUCCESS;
        }
    }
    if (c.epi == kPairStore) {
        PairOperand a = op[0], b = op[1];
        if (near) a.tile_lev = b.tile_lev = nullptr;  // NearSum reads every term
        if (kFloats) a.exps = b.exps = nullptr;       // the float sum scales after rounding
        OZB_TRY(pair_products(h, pd, a, b, c));
        ev_record(h, 3);
        counted(h);
        k_pair_sum<kFloats><<<(unsigned)((int64_t)((m + 255) / 256) * n), 256, 0, st->stream>>>(
            m, n, c.nA, c.nB, c.maxlevel, npu, c.pbuf, a.tile_lev, b.tile_lev, tile[1], op[0].exps, op[1].exps,
            h->sumMode, alpha, beta, C, ldc);
        OZB_CHECK(cudaGetLastError());
    } else {
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
