// gemv_t.cu — the plain GEMV with contiguous lines (y = A^T x) without slices
// in memory, and the one-launch split of a short vector.
//
// The reference splits every line of A level by level, x likewise, forms the
// exact products of all slice pairs of a line and sums them in pair order
// (src/cpu/ozblas_gemm.cpp with n = 1, called by ozblas_gemv.cpp:22-26).  With
// the slices materialised a line is read, its slices written and read again:
// 8 (2 nA + 2) bytes an element.  Here a line is read twice:
//   pass 1  its largest element and lowest set bit, which under the predicted
//           chain tau_{s+1} = tau_s + rho - 54 (chain.cuh) fix every level;
//   pass 2  each element is cut in registers and multiplied with x's slices
//           (read through L1); the largest remainder of every level is kept
//           until it proves the prediction.
// A line whose prediction is not proven is done again with its exact chain
// (one pass per level).  The pair products are exact, so their order is free;
// the ordered sum over the pairs follows, per line.  What bounds it is the FP64
// pipe: per element 3 L + L nB operations for L levels of the line against
// nB slices of x (28 for 4 x 4), 18 T a second on the chip.
// Lines with more than kGtLevels levels or with Inf / NaN are listed and done by
// a block each, level by level (k_gemv_t_deep).  Exponents near the ends of the
// range, and x with Inf / NaN or more than kGtLevels slices, leave the call to
// the slice path (nothing is written; x's slices are kept for it).
//
// 6001 x 3001 (phi = 1, 5 x 4 levels), one B200: the materialised path 853 us a
// call (split 309, products 466, x's split 19), this one 206 (statistics 35,
// products 129, x's split 9.5).  The products run at a fifth of the FP64 pipe:
// 16 warps per SM (the accumulators take the registers) and the loads of x's
// slices between their steps.
#include "chain.cuh"
#include "ozb_device.cuh"
#include "ozb_internal.h"
#include "sum.cuh"

namespace ozb {

constexpr int kGtLevels = 6;
constexpr int kGtThreads = 256;
constexpr int kGtStages = 8;  // steps of a line's elements in flight per warp (a step: 64 elements)

struct VecSplitInfo {
    int ns;     // the reference's slice count
    int nz;     // slices that can be nonzero
    int tau0;   // tau of level 0
    int glast;  // exponent of the last nonzero slice's grid
    int bad;    // Inf / NaN or a sigma beyond the range: the slices are not meaningful here
};

// ---------------------------------------------------------------------------
// The split of a vector of at most 16384 elements without a grid-wide barrier
// per level (k_split_vector's cooperative launch, split.cu: 17-21 us at 8192):
// every CTA holds the whole vector in registers and follows the chain by
// itself, and writes its share of the slices (one CTA's stores alone take
// 2 us a level).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mag_bits(double v) {  // |v| in order; 0 for NaN, which the reference's max skips
    const uint64_t b = dbits(v) & 0x7fffffffffffffffULL;
    return b > 0x7ff0000000000000ULL ? 0 : b;
}

// The block's largest |v| over C values per thread (NaN skipped): by high
// words, the low words only where the rule for tau or a zero depends on them:
// in normal numbers just above a power of two, in subnormal ones (whose leading
// bit may be any bit of the high word) always.
template <int C>
__device__ __forceinline__ double block_max_abs(const double (&v)[C], unsigned *red) {  // red: 2 x 32, used in turn
    unsigned hm = 0;
#pragma unroll
    for (int c = 0; c < C; c++) {
        const unsigned h = abs_hiword(v[c]);
        hm = max(hm, h > 0x7ff00000u ? 0u : h);
    }
    hm = __reduce_max_sync(0xffffffffu, hm);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (l == 0) red[w] = hm;
    __syncthreads();
    hm = __reduce_max_sync(0xffffffffu, l < nw ? red[l] : 0u);
    unsigned lm = 1;
    if ((hm & 0xfffffu) == 0 || hm < 0x100000u) {  // uniform: at a power of two, or subnormal, or zero
        lm = 0;
#pragma unroll
        for (int c = 0; c < C; c++)
            if (abs_hiword(v[c]) == hm && mag_bits(v[c]) != 0) lm = max(lm, (unsigned)__double2loint(v[c]));
        lm = __reduce_max_sync(0xffffffffu, lm);
        __syncthreads();
        if (l == 0) red[w] = lm;
        __syncthreads();
        lm = __reduce_max_sync(0xffffffffu, l < nw ? red[l] : 0u);
    }
    return __hiloint2double((int)hm, (int)lm);
}

template <int C>
__global__ void __launch_bounds__(1024) k_split_vector_one(int n, const double *__restrict__ x, int rho, int maxS,
                                                           double *__restrict__ out, int ldo,
                                                           VecSplitInfo *__restrict__ info) {
    __shared__ unsigned red[2][32];
    const int tid = threadIdx.x, nt = blockDim.x;
    double r[C];
    bool bad = false;
#pragma unroll
    for (int c = 0; c < C; c++) {
        const int i = c * nt + tid;
        r[c] = i < n ? x[i] : 0.0;
        bad |= !isfinite(r[c]);
    }
    bad = __syncthreads_or(bad);
    double mx = block_max_abs(r, red[0]);
    int s = 0, tau0 = 0, glast = 0, nz = 0;
    for (; s < maxS; s++) {
        if (s >= 2 && mx == 0.0) break;
        const int tau = tau_rule(mx);
        const double sigma = 0.75 * pow2(rho + tau);
        if (rho + tau > 1023) bad = true;
        if (s == 0) tau0 = tau;
        if (mx != 0.0) {
            glast = rho + tau - 53;
            nz = s + 1;
        }
#pragma unroll
        for (int c = 0; c < C; c++) {
            const int i = c * nt + tid;
            const double sl = (r[c] + sigma) - sigma;
            r[c] = r[c] - sl;
            if (c % (int)gridDim.x == (int)blockIdx.x && i < ldo) out[(size_t)s * ldo + i] = i < n ? sl : 0.0;
        }
        mx = block_max_abs(r, red[(s + 1) & 1]);
    }
    if (tid == 0 && blockIdx.x == 0) *info = VecSplitInfo{s, nz, tau0, glast, bad ? 1 : 0};
}

constexpr int kSplitOneMax = kSplitVectorSmallMax;

static int split_vector_one(cuozblasHandle_t *h, int n, const double *x, int rho, int maxS, double *out, int ldo,
                            VecSplitInfo *info) {
    cudaStream_t s = state(h)->stream;
    counted(h);
    const int len = ldo > n ? ldo : n;
    if (len <= 2048)
        k_split_vector_one<2><<<2, 1024, 0, s>>>(n, x, rho, maxS, out, ldo, info);
    else if (len <= 8192)
        k_split_vector_one<8><<<8, 1024, 0, s>>>(n, x, rho, maxS, out, ldo, info);
    else
        k_split_vector_one<16><<<16, 1024, 0, s>>>(n, x, rho, maxS, out, ldo, info);
    OZB_CHECK(cudaGetLastError());
    return CUOZBLAS_STATUS_SUCCESS;
}

// The same for a caller that needs the count on the host.
int split_vector_small(cuozblasHandle_t *h, int n, const double *x, int rho, int maxS, double *out, int ldo, int *ns) {
    State *st = state(h);
    VecSplitInfo *info = reinterpret_cast<VecSplitInfo *>(st->d_ints + 16);
    OZB_TRY(split_vector_one(h, n, x, rho, maxS, out, ldo, info));
    OZB_CHECK(cudaMemcpyAsync(st->h_ints, info, sizeof(int), cudaMemcpyDeviceToHost, st->stream));
    OZB_CHECK(cudaStreamSynchronize(st->stream));
    *ns = st->h_ints[0];
    return CUOZBLAS_STATUS_SUCCESS;
}

// ---------------------------------------------------------------------------
// The lines.  WPR warps per line (8 / WPR lines per CTA).
// ---------------------------------------------------------------------------
struct GemvTStatus {  // zeroed before the launch
    int declined;     // some line (or x) needs the slice path: y is not written
    int zmax;         // the largest first all-zero level of a line
    int ndeep;        // lines listed for k_gemv_t_deep
};

struct GtPlan {
    double sig[kGtLevels];
    int L, z, bad;  // L above kGtLevels: a deep line
};

// A (part of a) line's statistics from the first pass: the largest |v| (+inf
// where it holds Inf or NaN) and the lowest set-bit exponent (4000: all zero).
struct GtStat {
    double mx;
    int lb, pad;
};

// The levels of a line from tau_0 and its lowest set bit, under the predicted chain.
__device__ __forceinline__ GtPlan gt_predict(int tau0, int lb, int rho, int maxS, int glast) {
    GtPlan p;
    const int d = 54 - rho, G0 = rho + tau0 - 53;
    const int num = lb >= 4000 ? 0 : G0 - lb;
    p.z = num <= 0 ? 0 : (num + d - 1) / d;
    p.L = p.z + 1 < maxS ? p.z + 1 : maxS;
    // every sigma and grid normal, every slice product on a representable grid
    p.bad = rho + tau0 > 1000 || G0 - p.z * d < -1000 || G0 - (p.L - 1) * d + glast < -1060;
#pragma unroll
    for (int s = 0; s < kGtLevels; s++) p.sig[s] = 0.75 * pow2(rho + tau0 - s * d);
    return p;
}

// Pass 1: one warp per (line, part of it), ended after its first loads when x
// leaves the call to the slice path.
__global__ void __launch_bounds__(256) k_gemv_t_stats(int nl, int k, const double *__restrict__ A, int lda, int parts,
                                                      const VecSplitInfo *__restrict__ info, GtStat *__restrict__ out) {
    const int w = (int)(((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    const int row = w / parts, part = w % parts;
    if (row >= nl) return;
    const double *a = A + (size_t)row * lda;
    const int xbad = info->bad, xnz = info->nz;
    LazyStats rs;
    constexpr int kIn = 8;
    const int step = 32 * parts;
    int i = part * 32 + lane;
    for (; i - lane + (kIn - 1) * step + 31 < k; i += kIn * step) {
        double v[kIn];
#pragma unroll
        for (int u = 0; u < kIn; u++) v[u] = __ldg(a + i + u * step);
        if (xbad || xnz > kGtLevels) return;  // uniform
#pragma unroll
        for (int u = 0; u < kIn; u++) lazy_elem(rs, v[u]);
        lazy_sync(rs);
    }
    for (; i - lane < k; i += step) lazy_elem(rs, i < k ? __ldg(a + i) : 0.0);
    const uint64_t b = dbits(rs.mx);
    const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(b >> 32));
    const uint32_t lo = __reduce_max_sync(0xffffffffu, (uint32_t)(b >> 32) == hi ? (uint32_t)b : 0u);
    const unsigned hmx = __reduce_max_sync(0xffffffffu, rs.hmax);
    const int lb = __reduce_min_sync(0xffffffffu, rs.lb);
    if (lane == 0)
        out[w] = GtStat{hmx >= 0x7ff00000u ? __longlong_as_double(0x7ff0000000000000LL) : __hiloint2double((int)hi, (int)lo),
                        lb, 0};
}

// E elements at once: their slices (levels 0..L-1) against x's, interleaved.
// STEP: level by level, with hm[s] the largest high word of the remainder
// after level s.  Otherwise two levels from one base, half the depth for the
// same operations (chain.cuh; holds on the predicted chain for rho >= 29).
template <int L, int NB, int E, bool STEP>
__device__ __forceinline__ void gt_elements(double (&r)[E], const double (&xb)[E][NB], const double (&sig)[kGtLevels],
                                            double (&P)[kGtLevels][NB], unsigned (&hm)[kGtLevels]) {
    constexpr int G = STEP ? 1 : 2;
#pragma unroll
    for (int s = 0; s < L; s += G) {
        double s0[E], s1[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
            s0[e] = (r[e] + sig[s]) - sig[s];
            if (G == 2 && s + 1 < L) {
                const double rn = (r[e] + sig[s + 1]) - sig[s + 1];
                s1[e] = rn - s0[e];
                r[e] = r[e] - rn;
            } else {
                r[e] = r[e] - s0[e];
            }
            if (STEP) hm[s] = max(hm[s], abs_hiword(r[e]));
        }
#pragma unroll
        for (int e = 0; e < E; e++)
#pragma unroll
            for (int b = 0; b < NB; b++) {
                P[s][b] = fma(s0[e], xb[e][b], P[s][b]);
                if (G == 2 && s + 1 < L) P[s + 1][b] = fma(s1[e], xb[e][b], P[s + 1][b]);
            }
    }
}
template <int NB, int E, bool STEP>
__device__ __forceinline__ void gt_elements(int L, double (&r)[E], const double (&xb)[E][NB],
                                            const double (&sig)[kGtLevels], double (&P)[kGtLevels][NB],
                                            unsigned (&hm)[kGtLevels]) {
    switch (L) {  // uniform over a line
        case 0: break;
        case 1: gt_elements<1, NB, E, STEP>(r, xb, sig, P, hm); break;
        case 2: gt_elements<2, NB, E, STEP>(r, xb, sig, P, hm); break;
        case 3: gt_elements<3, NB, E, STEP>(r, xb, sig, P, hm); break;
        case 4: gt_elements<4, NB, E, STEP>(r, xb, sig, P, hm); break;
        case 5: gt_elements<5, NB, E, STEP>(r, xb, sig, P, hm); break;
        default: gt_elements<6, NB, E, STEP>(r, xb, sig, P, hm); break;
    }
}

template <int WPR>
__device__ __forceinline__ void gt_bar(int group) {  // the warps of one line
    if (WPR == 1)
        __syncwarp();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(32 * WPR) : "memory");
}

// The ordered sum of a line's pairs from its warps' partial products.
template <int WPR, int NB>
__device__ __forceinline__ void gt_line_sum(double (&P)[kGtLevels][NB], int L, int nB, int sum_mode, double *ps,
                                            int warp, int lane, int group, double *out) {
    double *mine = ps + warp * (kGtLevels * kGtLevels);
#pragma unroll
    for (int s = 0; s < kGtLevels; s++)
        if (s < L) {
#pragma unroll
            for (int b = 0; b < NB; b++) {
                double v = P[s][b];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) mine[s * kGtLevels + b] = v;
            }
        }
    gt_bar<WPR>(group);
    if ((warp & (WPR - 1)) == 0) {
        // lane = index of a pair in summation order
        double *terms = ps + (size_t)(8 * kGtLevels * kGtLevels) + warp * 64;
        int np = 0;
        for_each_pair(L, nB, L + nB - 2, [&](int ia, int ib) {
            if ((np & 31) == lane) {
                double v = 0.0;
                for (int w = 0; w < WPR; w++) v += mine[w * (kGtLevels * kGtLevels) + ia * kGtLevels + ib];
                terms[np] = v;
            }
            np++;
        });
        __syncwarp();
        if (lane == 0) {
            double t = 0.0;
            if (sum_mode == 1)
                t = nearsum(np, terms, 1);
            else
                for (int i = 0; i < np; i++) t += terms[i];
            *out = t;
        }
    }
}

struct GtShared {
    double am[kGtStages][8][64];  // per warp: its elements, each read back by the lane that copied it
    double ps[8 * kGtLevels * kGtLevels + 8 * 64];
    uint64_t smx[8];
    unsigned shm[8][kGtLevels];
};

template <int WPR, int NB>
__device__ __forceinline__ void gt_lines(int nl, int k, const double *__restrict__ A, int lda,
                                         const double *__restrict__ xs, int ldx, const VecSplitInfo &xi, int rho,
                                         int maxS, int sum_mode, int parts, const GtStat *__restrict__ stats,
                                         double *__restrict__ yt, GemvTStatus *st, int *__restrict__ deep_lines,
                                         GtShared &sh) {
    auto &ps = sh.ps;
    auto &smx = sh.smx;
    auto &shm = sh.shm;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = warp / WPR, sub = warp % WPR, w0 = group * WPR;
    const int row = blockIdx.x * (8 / WPR) + group;
    const bool live = row < nl;
    const double *a = A + (size_t)(live ? row : nl - 1) * lda;
    const int nB = xi.nz;

    // step `it` of this warp: elements (it WPR + sub) 64 + 2 lane, + 1.  x's slices
    // come from L1, where the warps that run side by side share them.
    const int nsteps = ((k + 63) / 64 - sub + WPR - 1) / WPR;
    const int last_full = nsteps - (((nsteps - 1) * WPR + sub) * 64 + 64 > k ? 1 : 0);  // steps below it lie within the line
    double *ring = &sh.am[0][warp][2 * lane];
    constexpr int kRing = 8 * 64;
    const double *aj = a + sub * 64 + 2 * lane;  // of the next step to issue
    int slot = 0;
    auto issue = [&](int it) {
        if (it < last_full) {
            cp_async8(ring + slot * kRing, aj);
            cp_async8(ring + slot * kRing + 1, aj + 1);
        } else if (it < nsteps) {
            const int j = (it * WPR + sub) * 64 + 2 * lane;
            cp_async8_zfill(ring + slot * kRing, j < k ? aj : a, j < k ? 8u : 0u);
            cp_async8_zfill(ring + slot * kRing + 1, j + 1 < k ? aj + 1 : a, j + 1 < k ? 8u : 0u);
        }
        cp_async_commit();
        aj += 64 * WPR;
        slot = slot == kGtStages - 1 ? 0 : slot + 1;
    };
#pragma unroll
    for (int g = 0; g < kGtStages - 1; g++) issue(g);

    // the line's statistics
    double mx = 0.0;
    int lb = 4000;
    for (int w = 0; w < parts; w++) {
        const GtStat g = stats[(size_t)(live ? row : nl - 1) * parts + w];
        mx = fmax(mx, g.mx);
        lb = min(lb, g.lb);
    }
    const bool nonfinite = !(mx <= 1.7976931348623157e308);
    const int tau0 = nonfinite ? 0 : tau_rule(mx);
    GtPlan pl = gt_predict(tau0, lb, rho, maxS, xi.glast);
    bool deep = nonfinite || pl.L > kGtLevels;
    bool bad = !deep && (pl.bad || tau0 + xi.tau0 + ceil_log2_int((uint32_t)k) > 1000);
    if (bad || deep) pl.L = 0;
    const int step = 32 * WPR;

    // ---- pass 2 ----
    double P[kGtLevels][NB];
    unsigned hm[kGtLevels];
#pragma unroll
    for (int s = 0; s < kGtLevels; s++) {
        hm[s] = 0;
#pragma unroll
        for (int b = 0; b < NB; b++) P[s][b] = 0.0;
    }
    // tau_rule of a value of at most 2^t is t when its high word is above that
    // of 2^(t-1): level s is proven by a remainder above thr(s)
    auto thr = [&](int s) { return (unsigned)(dbits(pow2(tau0 - (s + 1) * (54 - rho) - 1)) >> 32); };
    bool track = true;  // per warp, until its own elements prove every level
    const double *xj = xs + sub * 64 + 2 * lane;  // slices are padded with zeros to whole steps
    int rd = 0;
    for (int it = 0; it < nsteps; it++, xj += 64 * WPR) {
        double xb[2][NB];
#pragma unroll
        for (int b = 0; b < NB; b++) {
            const double2 v = b < nB ? __ldg(reinterpret_cast<const double2 *>(xj + (size_t)b * ldx))
                                     : make_double2(0.0, 0.0);
            xb[0][b] = v.x;
            xb[1][b] = v.y;
        }
        cp_async_wait<kGtStages - 2>();
        const double2 av = *reinterpret_cast<const double2 *>(ring + rd * kRing);
        rd = rd == kGtStages - 1 ? 0 : rd + 1;
        double r[2] = {av.x, av.y};
        issue(it + kGtStages - 1);
        if (track) {
            gt_elements<NB, 2, true>(pl.L, r, xb, pl.sig, P, hm);
            if ((it & 7) == 0) {
                bool open = false;
#pragma unroll
                for (int s = 0; s + 1 < kGtLevels; s++)
                    if (s + 1 < pl.L) open |= !__any_sync(0xffffffffu, hm[s] > thr(s));
                track = open || rho < 29;
            }
        } else {
            gt_elements<NB, 2, false>(pl.L, r, xb, pl.sig, P, hm);
        }
    }
    cp_async_wait<0>();

    // ---- proof: the first level that leaves nothing, and that every level before it leaves a remainder whose tau
    // is the predicted one
#pragma unroll
    for (int s = 0; s < kGtLevels; s++) {
        const unsigned h = __reduce_max_sync(0xffffffffu, hm[s]);
        if (lane == 0) shm[warp][s] = h;
    }
    gt_bar<WPR>(group);
    bool proven = true, ended = false;
#pragma unroll
    for (int s = 0; s + 1 < kGtLevels; s++)
        if (s + 1 < pl.L && !ended) {
            unsigned h = 0;
            for (int w = 0; w < WPR; w++) h = max(h, shm[w0 + w][s]);
            if (h == 0) {  // exact zeros from here on: grids are normal, so no remainder hides below the high word
                pl.z = s;
                ended = true;
            } else {
                proven = proven && h > thr(s);
            }
        }
    if (!bad && !deep && !proven) {  // the exact chain, one pass per level, and the products again (x's slices from L2)
        int z = maxS - 1, L = maxS;
        for (int s = 1;; s++) {
            uint64_t m = 0;
            for (int j = sub * 32 + lane; j < k; j += step) {
                double r = __ldg(a + j);
#pragma unroll
                for (int q = 0; q < kGtLevels; q++)
                    if (q < s) r = r - ((r + pl.sig[q]) - pl.sig[q]);
                const uint64_t b = mag_bits(r);
                m = b > m ? b : m;
            }
            const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(m >> 32));
            const uint32_t lo = __reduce_max_sync(0xffffffffu, (uint32_t)(m >> 32) == hi ? (uint32_t)m : 0u);
            gt_bar<WPR>(group);
            if (lane == 0) smx[warp] = ((uint64_t)hi << 32) | lo;
            gt_bar<WPR>(group);
            uint64_t mm = 0;
            for (int w = 0; w < WPR; w++) mm = smx[w0 + w] > mm ? smx[w0 + w] : mm;
            if (mm == 0) {
                z = s - 1 < maxS - 1 ? s - 1 : maxS - 1;
                L = s;
                break;
            }
            if (s == maxS) break;
            const int tau = tau_rule(__longlong_as_double((long long)mm));
            deep = s == kGtLevels;
            bad = !deep && (rho + tau - 53 < -1000 || rho + tau - 53 + xi.glast < -1060);
            if (bad || deep) break;
#pragma unroll
            for (int q = 0; q < kGtLevels; q++)
                if (q == s) pl.sig[q] = 0.75 * pow2(rho + tau);
        }
        pl.z = z;
        pl.L = bad || deep ? 0 : L;
#pragma unroll
        for (int s = 0; s < kGtLevels; s++)
#pragma unroll
            for (int b = 0; b < NB; b++) P[s][b] = 0.0;
        for (int j = sub * 32 + lane; j < k; j += step) {
            double xb[1][NB], r[1] = {__ldg(a + j)};
#pragma unroll
            for (int b = 0; b < NB; b++) xb[0][b] = b < nB ? xs[(size_t)b * ldx + j] : 0.0;
            gt_elements<NB, 1, true>(pl.L, r, xb, pl.sig, P, hm);
        }
    }
    double t = 0.0;
    gt_line_sum<WPR, NB>(P, pl.L, nB, sum_mode, ps, warp, lane, group, &t);
    if (live && sub == 0 && lane == 0) {
        const int z = pl.z < maxS - 1 ? pl.z : maxS - 1;
        if (deep)
            deep_lines[atomicAdd(&st->ndeep, 1)] = row;
        else if (bad)
            atomicOr(&st->declined, 1);
        else {
            __stcg(yt + row, t);
            if (z > __ldcg(&st->zmax)) atomicMax(&st->zmax, z);
        }
    }
}

template <int WPR>
__global__ void __launch_bounds__(kGtThreads, 2)
    k_gemv_t(int nl, int k, const double *__restrict__ A, int lda, const double *__restrict__ xs, int ldx,
             const VecSplitInfo *__restrict__ info, int rho, int maxS, int sum_mode, int parts,
             const GtStat *__restrict__ stats, double *__restrict__ yt, GemvTStatus *st, int *__restrict__ deep_lines) {
    const VecSplitInfo xi = *info;
    __shared__ __align__(16) GtShared sh;
    if (xi.bad || xi.nz > kGtLevels) {  // uniform over the grid
        if (blockIdx.x == 0 && threadIdx.x == 0) st->declined = 1;
        return;
    }
    if (xi.nz <= 4)
        gt_lines<WPR, 4>(nl, k, A, lda, xs, ldx, xi, rho, maxS, sum_mode, parts, stats, yt, st, deep_lines, sh);
    else
        gt_lines<WPR, 6>(nl, k, A, lda, xs, ldx, xi, rho, maxS, sum_mode, parts, stats, yt, st, deep_lines, sh);
}

// A deep line: a block follows its true chain, the remainders in shared memory
// (k doubles), and adds each level's products as it is cut.  What binds it is the
// chain: a cut, a block maximum and nB block sums a level, some 2 us.  2000 lines
// of 3000, one of them such: the call 156 us, all of them 351 (by the slice path
// alone 627 and 680, after a declined pass over the lines 704 and 747).
__global__ void __launch_bounds__(kGtThreads) k_gemv_t_deep(int k, const double *__restrict__ A, int lda,
                                                            const double *__restrict__ xs, int ldx,
                                                            const VecSplitInfo *__restrict__ info, int rho, int maxS,
                                                            int sum_mode, const int *__restrict__ deep_lines,
                                                            double *__restrict__ yt, GemvTStatus *st) {
    extern __shared__ double rem[];
    __shared__ double red[kGtThreads / 32], part[kGtLevels][kGtThreads / 32];
    __shared__ double P[kMaxSplitDefault * kGtLevels], terms[kMaxSplitDefault * kGtLevels];
    const VecSplitInfo xi = *info;
    const int t = threadIdx.x, line = deep_lines[blockIdx.x], nB = xi.nz;
    const double *a = A + (size_t)line * lda;
    double mx = 0.0;
    bool nonfinite = false;
    for (int i = t; i < k; i += kGtThreads) {
        const double v = a[i];
        rem[i] = v;
        mx = ref_max(mx, fabs(v));
        nonfinite |= !isfinite(v);
    }
    nonfinite = __syncthreads_or(nonfinite);
    mx = block_max_nonneg(mx, red);
    // (no slice of x would make NaN of it)
    bool bad = (nonfinite && nB == 0) || tau_rule(mx) + xi.tau0 + ceil_log2_int((uint32_t)k) > 1000;
    int L = maxS, z = maxS - 1;
    for (int s = 0; s < maxS && !bad; s++) {  // uniform
        const int tau = tau_rule(mx);
        bad = rho + tau > 1000 || rho + tau - 53 < -1000 || rho + tau - 53 + xi.glast < -1060;
        if (bad) break;
        const double sigma = 0.75 * pow2(rho + tau);
        double acc[kGtLevels], nm = 0.0;
#pragma unroll
        for (int b = 0; b < kGtLevels; b++) acc[b] = 0.0;
        for (int i = t; i < k; i += kGtThreads) {
            double r = rem[i];
            const double sl = (r + sigma) - sigma;
            r = r - sl;
            rem[i] = r;
            nm = ref_max(nm, fabs(r));
#pragma unroll
            for (int b = 0; b < kGtLevels; b++)
                if (b < nB) acc[b] = fma(sl, xs[(size_t)b * ldx + i], acc[b]);
        }
#pragma unroll
        for (int b = 0; b < kGtLevels; b++) {
            for (int o = 16; o > 0; o >>= 1) acc[b] += __shfl_xor_sync(0xffffffffu, acc[b], o);
            if ((t & 31) == 0) part[b][t >> 5] = acc[b];
        }
        mx = block_max_nonneg(nm, red);  // synchronises: the parts are written
        if (t < kGtLevels) {
            double v = 0.0;
            for (int w = 0; w < kGtThreads / 32; w++) v += part[t][w];
            P[s * kGtLevels + t] = v;
        }
        if (mx == 0.0) {
            L = s + 1;
            z = s;
            break;
        }
        __syncthreads();  // before the parts are written again
    }
    __syncthreads();
    if (t != 0) return;
    if (bad) {
        atomicOr(&st->declined, 1);
        return;
    }
    int np = 0;
    for_each_pair(L, nB, L + nB - 2, [&](int ia, int ib) { terms[np++] = P[ia * kGtLevels + ib]; });
    double sum = 0.0;
    if (sum_mode == 1)
        sum = nearsum(np, terms, 1);
    else
        for (int i = 0; i < np; i++) sum += terms[i];
    yt[line] = sum;
    atomicMax(&st->zmax, z);
}

// y, once it is known that every line has its sum (the first `ndeep` deep ones done).
__global__ void k_gemv_t_write(int nl, const double *__restrict__ yt, const GemvTStatus *__restrict__ st, int ndeep,
                               double alpha, double beta, double *__restrict__ y) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < nl && !st->declined && st->ndeep == ndeep) y[r] = fma(alpha, yt[r], beta * y[r]);
}

// y = alpha A^T x + beta y over nl lines of length k (line l at A + l lda),
// splitEpsMode 0 and the full pair set.  *done false (y untouched) when the
// slice path must run: then xs has x's slices where they were formed and the
// arena has room beside them (they stay allocated), else null.
int gemv_t_fused(cuozblasHandle_t *h, int nl, int k, const double *A, int lda, const double *x, double alpha,
                 double beta, double *y, bool *done, int *nA, int *nB, VecSlices *kept) {
    State *st = state(h);
    *done = false;
    *kept = VecSlices{};
    if (k < 1 || nl < 1 || k > kSplitOneMax) return CUOZBLAS_STATUS_SUCCESS;
    const int maxS = h->nSplitMax > 0 ? h->nSplitMax : kMaxSplitDefault;
    const int rho = rho_rule(k, 0);
    const int ldx = (k + 63) / 64 * 64;  // whole steps, zero padded
    Arena ar(h);
    const uint64_t mk = ar.mark();
    double *xs = ar.take<double>((uint64_t)maxS * ldx);
    const uint64_t mk_xs = ar.mark();
    double *yt = ar.take<double>(nl);
    int *deep_lines = ar.take<int>(nl);
    // parts of a line in pass 1: enough warps to keep the memory busy
    int parts = 1;
    while (parts < 8 && (int64_t)nl * parts < 48 * sm_count() && k > 512 * parts) parts *= 2;
    GtStat *stats = ar.take<GtStat>((uint64_t)nl * parts);
    struct Block {
        GemvTStatus st;
        VecSplitInfo info;
    } *blk = ar.take<Block>(1);
    if (!ar.ok) {
        ar.release(mk);
        return CUOZBLAS_STATUS_SUCCESS;
    }
    span_begin(h);
    OZB_CHECK(cudaMemsetAsync(blk, 0, sizeof(Block), st->stream));
    OZB_TRY(split_vector_one(h, k, x, rho, maxS, xs, ldx, &blk->info));
    counted(h);
    k_gemv_t_stats<<<(unsigned)(((int64_t)nl * parts * 32 + 255) / 256), 256, 0, st->stream>>>(nl, k, A, lda, parts,
                                                                                               &blk->info, stats);
    OZB_CHECK(cudaGetLastError());
    // Warps per line: the fewest rounds of the 16 resident warps per SM over (line part + its reductions).
    int wpr = 1;
    int64_t best = INT64_MAX;
    for (int w = 1; w <= 8; w *= 2) {
        const int64_t rounds = ((int64_t)nl * w + 16 * sm_count() - 1) / (16 * sm_count());
        const int64_t cost = rounds * ((k + w - 1) / w + 400);
        if (cost < best) {
            best = cost;
            wpr = w;
        }
    }
    const int rows = 8 / wpr, grid = (nl + rows - 1) / rows;
    counted(h);
    auto go = [&](auto kern) {
        kern<<<grid, kGtThreads, 0, st->stream>>>(nl, k, A, lda, xs, ldx, &blk->info, rho, maxS, h->sumMode, parts, stats,
                                                  yt, &blk->st, deep_lines);
    };
    wpr == 1 ? go(k_gemv_t<1>) : wpr == 2 ? go(k_gemv_t<2>) : wpr == 4 ? go(k_gemv_t<4>) : go(k_gemv_t<8>);
    OZB_CHECK(cudaGetLastError());
    Block *hb = reinterpret_cast<Block *>(st->h_ints);
    for (int ndeep = 0;; ndeep = hb->st.ndeep) {
        if (ndeep > 0) {
            static std::atomic<uint64_t> attr{0};
            OZB_CHECK(smem_optin((const void *)k_gemv_t_deep, kSplitOneMax * (int)sizeof(double), attr));
            counted(h);
            k_gemv_t_deep<<<ndeep, kGtThreads, k * sizeof(double), st->stream>>>(
                k, A, lda, xs, ldx, &blk->info, rho, maxS, h->sumMode, deep_lines, yt, &blk->st);
            OZB_CHECK(cudaGetLastError());
        }
        counted(h);
        k_gemv_t_write<<<(nl + 255) / 256, 256, 0, st->stream>>>(nl, yt, &blk->st, ndeep, alpha, beta, y);
        OZB_CHECK(cudaGetLastError());
        span_end(h);
        OZB_CHECK(cudaMemcpyAsync(hb, blk, sizeof(Block), cudaMemcpyDeviceToHost, st->stream));
        OZB_CHECK(cudaStreamSynchronize(st->stream));
        if (hb->st.declined || hb->st.ndeep == ndeep) break;
    }
    ar.release(mk);
    if (hb->st.declined) {
        // x's slices for the slice path, if that has all the room it can need above them
        const uint64_t most = sizeof(double) * ((uint64_t)maxS * nl * (k + 1) + 2 * (uint64_t)maxS * maxS * nl) + (1u << 20);
        if (mk_xs + most <= h->workSizeBytes) {
            ar.take<double>((uint64_t)maxS * ldx);
            *kept = VecSlices{xs, ldx, hb->info.ns};
        }
        return CUOZBLAS_STATUS_SUCCESS;
    }
    const int c = (hb->st.zmax < 1 ? 1 : hb->st.zmax) + 1;
    *nA = c < maxS ? c : maxS;
    *nB = hb->info.ns;
    *done = true;
    return CUOZBLAS_STATUS_SUCCESS;
}

}  // namespace ozb
