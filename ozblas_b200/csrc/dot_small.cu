// dot_small.cu — the plain-form DOT / NRM2 of a few thousand elements in one
// launch.
//
// Such a call is all latency: with the two-pass DOT (dot_fused.cu) it is a
// memset, two kernels of a block each and a copy back, 43 us from the first to
// the last of them for 1000 elements, of which the kernels take 14.  Here one
// block does the whole of it and leaves the status in mapped host memory, so
// the host launches once and waits once.  The elements stay in registers, so
// the tau chain is followed level by level with a block maximum (as
// src/cpu/ozblas_split.cpp:62-103 does) instead of predicted and proven:
// vectors whose chain is not the predicted one, a third of the short ones,
// stay on this path too.  Then every element is cut again along the known
// sigmas and the slice-pair products add up exactly in 64 registers; the
// block's sums go through a halving butterfly (62 exchanges per lane, 320
// with a butterfly per product).
//
// Up to kDotSmallMax elements the block's own work (about a microsecond per
// 1000 elements) stays below the launches it saves.  Whatever one launch
// cannot hold (more than 8 levels, Inf / NaN, sigmas or products near the ends
// of the range) is left to the general paths, which took it before.
#include <cstring>

#include "fused.h"
#include "ozb_internal.h"
#include "sum.cuh"

namespace ozb {

constexpr int kDsThreads = 256, kDotSmallMax = 4096;

__device__ __forceinline__ uint64_t ds_abs_bits(double v) { return dbits(v) & 0x7fffffffffffffffULL; }

// Largest |v| of the block, as bits (finite values: ordered as integers).
__device__ __forceinline__ uint64_t ds_warp_max(uint64_t b) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(b >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(b >> 32) == hi ? (unsigned)b : 0u);
    return (uint64_t)hi << 32 | lo;
}

template <int C, int T>
__device__ __forceinline__ void ds_products(int n, const double *__restrict__ x, const double *__restrict__ y,
                                            const double (*sig)[kDotLevels], double (&P)[kDotLevels * kDotLevels]) {
#pragma unroll 1
    for (int c = 0; c < C; c++) {
        const int i = c * kDsThreads + threadIdx.x;
        if (i >= n) break;
        double a = x[i], b = y[i], qa[T + 1], qb[T + 1];
#pragma unroll
        for (int s = 0; s <= T; s++) {
            const double sa = sig[0][s], sb = sig[1][s];
            qa[s] = __dsub_rn(__dadd_rn(a, sa), sa);
            a = __dsub_rn(a, qa[s]);
            qb[s] = __dsub_rn(__dadd_rn(b, sb), sb);
            b = __dsub_rn(b, qb[s]);
        }
#pragma unroll
        for (int ia = 0; ia <= T; ia++)
#pragma unroll
            for (int ib = 0; ib <= T; ib++) P[ia * kDotLevels + ib] = fma(qa[ia], qb[ib], P[ia * kDotLevels + ib]);
    }
}

// One exchange of the halving butterfly: v[0..2H) of two lanes O apart become
// the pair's sums, the lower H in the lane with bit O clear.
template <int H, int O>
__device__ __forceinline__ void ds_halve(double *v) {
    const bool up = (threadIdx.x & O) != 0;
#pragma unroll
    for (int i = 0; i < H; i++) {
        const double keep = up ? v[i + H] : v[i], send = up ? v[i] : v[i + H];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
    }
}

template <int C>
__global__ void __launch_bounds__(kDsThreads, 1) k_dot_small(int n, const double *__restrict__ x,
                                                             const double *__restrict__ y, int rho, int maxS,
                                                             int sum_mode, volatile DotStatus *out) {
    __shared__ uint64_t mxs[2][2][kDsThreads / 32];  // by level parity, vector, warp
    __shared__ double sig[2][kDotLevels], red[kDsThreads / 32][kDotLevels * kDotLevels];
    __shared__ double Pv[kDotLevels * kDotLevels], tmp[kDotLevels * kDotLevels];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    double rx[C], ry[C];
    uint64_t bx = 0, by = 0;
#pragma unroll
    for (int c = 0; c < C; c++) {
        const int i = c * kDsThreads + t;
        rx[c] = i < n ? x[i] : 0.0;
        ry[c] = i < n ? y[i] : 0.0;
    }
#pragma unroll
    for (int c = 0; c < C; c++) {
        bx = max(bx, ds_abs_bits(rx[c]));
        by = max(by, ds_abs_bits(ry[c]));
    }
    // the two chains (every thread follows them: no branch depends on the thread)
    int ns[2] = {0, 0}, glast[2] = {0, 0}, tau0[2] = {0, 0};
    bool ok = true, open[2] = {true, true};
#pragma unroll 1
    for (int s = 0;; s++) {
        const uint64_t wx = ds_warp_max(bx), wy = ds_warp_max(by);
        if (lane == 0) {
            mxs[s & 1][0][w] = wx;
            mxs[s & 1][1][w] = wy;
        }
        __syncthreads();
        double mx[2];
#pragma unroll
        for (int v = 0; v < 2; v++) {
            uint64_t m = 0;
#pragma unroll
            for (int j = 0; j < kDsThreads / 32; j++) m = max(m, mxs[s & 1][v][j]);
            mx[v] = __longlong_as_double((long long)m);
            if (m >= 0x7ff0000000000000ULL) ok = false;  // Inf or NaN (a NaN only ever has larger bits)
            // levels 0 and 1 always run, later ones while a remainder is left
            if (s >= maxS || (s >= 2 && m == 0)) open[v] = false;
        }
        if (!ok || (!open[0] && !open[1])) break;
        if (s == kDotLevels) {  // more levels than are held
            ok = false;
            break;
        }
        double sg[2];
#pragma unroll
        for (int v = 0; v < 2; v++) {
            const int tau = tau_rule(mx[v]);
            sg[v] = open[v] ? 0.75 * pow2(rho + tau) : 0.0;
            if (open[v]) {
                ns[v] = s + 1;
                if (s == 0) tau0[v] = tau;
                if (mx[v] != 0.0) {
                    glast[v] = rho + tau - 53;
                    if (rho + tau > 1000 || glast[v] < -1000) ok = false;
                }
            }
            if (t == 0) sig[v][s] = sg[v];
        }
        bx = by = 0;
#pragma unroll
        for (int c = 0; c < C; c++) {
            rx[c] = __dsub_rn(rx[c], __dsub_rn(__dadd_rn(rx[c], sg[0]), sg[0]));
            ry[c] = __dsub_rn(ry[c], __dsub_rn(__dadd_rn(ry[c], sg[1]), sg[1]));
            bx = max(bx, ds_abs_bits(rx[c]));
            by = max(by, ds_abs_bits(ry[c]));
        }
    }
    // every slice product and sum on a representable grid
    if (glast[0] + glast[1] < -1060 || tau0[0] + tau0[1] > 960) ok = false;
    if (!ok) {  // uniform: the general paths
        if (t == 0) out->status = 0;
        return;
    }
    __syncthreads();  // sig
    double P[kDotLevels * kDotLevels];
#pragma unroll
    for (int i = 0; i < kDotLevels * kDotLevels; i++) P[i] = 0.0;
    switch (max(ns[0], ns[1])) {  // uniform
        case 1: ds_products<C, 0>(n, x, y, sig, P); break;
        case 2: ds_products<C, 1>(n, x, y, sig, P); break;
        case 3: ds_products<C, 2>(n, x, y, sig, P); break;
        case 4: ds_products<C, 3>(n, x, y, sig, P); break;
        case 5: ds_products<C, 4>(n, x, y, sig, P); break;
        case 6: ds_products<C, 5>(n, x, y, sig, P); break;
        case 7: ds_products<C, 6>(n, x, y, sig, P); break;
        default: ds_products<C, 7>(n, x, y, sig, P); break;
    }
    __syncwarp();
    ds_halve<32, 16>(P);
    ds_halve<16, 8>(P);
    ds_halve<8, 4>(P);
    ds_halve<4, 2>(P);
    ds_halve<2, 1>(P);  // lane l: products 2 l and 2 l + 1
    red[w][2 * lane] = P[0];
    red[w][2 * lane + 1] = P[1];
    __syncthreads();
    if (t < kDotLevels * kDotLevels) {
        double v = 0.0;
#pragma unroll
        for (int j = 0; j < kDsThreads / 32; j++) v += red[j][t];
        Pv[t] = v;
    }
    __syncthreads();
    if (t != 0) return;
    const int nA = ns[0], nB = ns[1], maxlevel = nA + nB - 2;  // DOT: fastMode is ignored (src/cpu/ozblas_gemm.cpp:26-29)
    double sum = 0.0;
    if (sum_mode == 1) {
        int np = 0;
        for_each_pair(nA, nB, maxlevel, [&](int ia, int ib) { tmp[np++] = Pv[ia * kDotLevels + ib]; });
        sum = nearsum(np, tmp, 1);
    } else {
        for_each_pair(nA, nB, maxlevel, [&](int ia, int ib) { sum += Pv[ia * kDotLevels + ib]; });
    }
    out->ns0 = nA;
    out->ns1 = nB;
    out->result = fma(1.0, sum, 0.0 * 0.0);  // alpha = 1, beta = 0 as the DOT driver passes them
    out->status = 1;
}

// Returns SUCCESS with *done = true and the result in *ret, or *done = false
// for the caller's other paths.
int dot_small(cuozblasHandle_t *h, int n, const double *x, const double *y, double *ret, bool *done, int *nA,
              int *nB) {
    State *st = state(h);
    *done = false;
    if (n < 1 || n > kDotSmallMax || st->env.dot_tree || st->env.dot_two_pass)
        return CUOZBLAS_STATUS_SUCCESS;
    if (h->sumMode == 0) {  // the smallest workspace an FSum DOT is accepted with (dot_fused.cu)
        Arena ar(h);
        const uint64_t mk = ar.mark();
        ar.take<DotScratch>(1);
        if (!ar.ok) return CUOZBLAS_STATUS_WORKSPACE;
        ar.release(mk);
    }
    const int maxS = h->nSplitMax > 0 ? h->nSplitMax : kMaxSplitDefault;
    const int rho = rho_rule(n, h->splitEpsMode);
    DotStatus res{};
    memcpy(st->h_mail, &res, sizeof(res));
    volatile DotStatus *out = reinterpret_cast<volatile DotStatus *>(st->d_mail);
    span_begin(h);
    counted(h);
    if (n <= 4 * kDsThreads)
        k_dot_small<4><<<1, kDsThreads, 0, st->stream>>>(n, x, y, rho, maxS, h->sumMode, out);
    else
        k_dot_small<16><<<1, kDsThreads, 0, st->stream>>>(n, x, y, rho, maxS, h->sumMode, out);
    OZB_CHECK(cudaGetLastError());
    span_end(h);
    OZB_CHECK(cudaStreamSynchronize(st->stream));
    memcpy(&res, st->h_mail, sizeof(res));
    if (res.status == 1) {
        *done = true;
        *nA = res.ns0;
        *nB = res.ns1;
        *ret = res.result;
    }
    return CUOZBLAS_STATUS_SUCCESS;
}

}  // namespace ozb
