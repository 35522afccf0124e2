// split.cu — error-free extraction of FP64 slices (the "plain" Ozaki split).
//
// Arithmetic of every level (src/cpu/ozblas_split.cpp:137-178 dense,
// :62-103 vector, :779-815 sparse):
//   tau   = ceil(log2(max|r|))            (tau_rule: glibc's rounding)
//   sigma = 0.75 * 2^(rho+tau) * shift    (sparse: / shift)
//   slice = (r + sigma) - sigma;  r -= slice;  new max = max|r|
// Termination (src/cpu/ozblas_split.cpp:272-289): level 0 always runs;
// levels 1.. run until one leaves every remainder zero (that level counts)
// or maxS levels exist.  With z = the first level whose remainder is zero
// for a line, the count is min(maxS, max(1, max_lines z) + 1).
#include <cooperative_groups.h>

#include <type_traits>

#include "ozb_device.cuh"
#include "ozb_internal.h"

namespace cg = cooperative_groups;

namespace ozb {

constexpr int kSplitThreads = 256;
constexpr int kSplitSmemMaxK = 26 * 1024;  // doubles kept on chip per line (208 KB)

// How a slice is stored.  Plain form: the FP64 slice itself.  Mixed form
// <double, float, float> (src/cpu/ozblas_split.cpp:181-221): scalbn(slice,
// -tau) in FP32, exact because a slice has at most 53 - rho <= 12 significant
// bits on the grid 2^(rho + tau - 53), with tau kept per line and level.
template <typename SL>
__device__ __forceinline__ SL slice_store(double sl, int tau);
template <>
__device__ __forceinline__ double slice_store<double>(double sl, int) {
    return sl;
}
template <>
__device__ __forceinline__ float slice_store<float>(double sl, int tau) {
    return (float)scalbn(sl, -tau);
}

// One CTA per line.  COUNT: atomicMax(*zmax, z_line).  WRITE: ns slices
// (and, for FP32 slices, tau of every level at exps[level * nl + line]).
// `rem` is either dynamic shared memory (k <= kSplitSmemMaxK) or a global
// scratch line of k doubles per CTA.
template <bool WRITE, typename SL = double>
__global__ void __launch_bounds__(kSplitThreads) k_split_lines(int k, int nl, const double *__restrict__ X, int ldx,
                                                               int rho, int levels, SL *__restrict__ out, int ldo,
                                                               short *__restrict__ exps,
                                                               double *__restrict__ gscratch,
                                                               int *__restrict__ zmax) {
    extern __shared__ double smem[];
    __shared__ double red[kSplitThreads / 32];
    const int line = blockIdx.x;
    if (line >= nl) return;
    double *rem = gscratch ? gscratch + (size_t)line * k : smem;
    const double *x = X + (size_t)line * ldx;
    double mx = 0.0;
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
        const double v = x[i];
        rem[i] = v;
        mx = ref_max(mx, fabs(v));
    }
    mx = block_max_nonneg(mx, red);
    int z = levels;  // COUNT: first level leaving a zero remainder (levels = maxS-1 cap)
    for (int s = 0; s < levels; s++) {
        const int tau = tau_rule(mx);
        const double sigma = 0.75 * pow2(rho + tau);  // dense_sigma(rho, mx, 1)
        double nm = 0.0;
        SL *o = WRITE ? out + ((size_t)s * nl + line) * ldo : nullptr;
        if (WRITE && exps && threadIdx.x == 0) exps[(size_t)s * nl + line] = (short)tau;
        for (int i = threadIdx.x; i < k; i += blockDim.x) {
            double r = rem[i];
            const double sl = (r + sigma) - sigma;
            r = r - sl;
            rem[i] = r;
            nm = ref_max(nm, fabs(r));
            if (WRITE) o[i] = slice_store<SL>(sl, tau);
        }
        if (WRITE)
            for (int i = k + threadIdx.x; i < ldo; i += blockDim.x) o[i] = (SL)0;
        mx = block_max_nonneg(nm, red);
        if (!WRITE && mx == 0.0) {
            z = s;
            break;
        }
    }
    if (!WRITE && threadIdx.x == 0) atomicMax(zmax, z);
}

template <typename SL>
static int launch_split_lines(cuozblasHandle_t *h, bool write, int k, int nl, const double *X, int ldx, int rho,
                              int levels, SL *out, int ldo, short *exps, int *zmax_dev) {
    State *st = state(h);
    double *gscratch = nullptr;
    size_t smem = 0;
    Arena ar(h);
    const uint64_t mk = ar.mark();
    if (k > kSplitSmemMaxK) {
        gscratch = ar.take<double>((uint64_t)k * nl);
        if (!ar.ok) return CUOZBLAS_STATUS_WORKSPACE;
    } else {
        smem = sizeof(double) * (size_t)(k > 0 ? k : 1);
    }
    if (write) {
        OZB_CHECK(cudaFuncSetAttribute(k_split_lines<true, SL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(kSplitSmemMaxK * sizeof(double))));
        counted(h);
        k_split_lines<true, SL><<<nl, kSplitThreads, smem, st->stream>>>(k, nl, X, ldx, rho, levels, out, ldo, exps,
                                                                         gscratch, nullptr);
    } else {
        OZB_CHECK(cudaFuncSetAttribute(k_split_lines<false, double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(kSplitSmemMaxK * sizeof(double))));
        counted(h);
        k_split_lines<false, double><<<nl, kSplitThreads, smem, st->stream>>>(k, nl, X, ldx, rho, levels, nullptr, 0,
                                                                      nullptr, gscratch, zmax_dev);
    }
    OZB_CHECK(cudaGetLastError());
    ar.release(mk);
    return CUOZBLAS_STATUS_SUCCESS;
}

int split_lines_count(cuozblasHandle_t *h, int k, int nl, const double *X, int ldx, int rho, int maxS, int *ns) {
    State *st = state(h);
    if (maxS <= 1 || nl == 0) {
        *ns = (nl == 0) ? (maxS < 2 ? maxS : 2) : 1;
        if (maxS <= 1) *ns = 1;
        return CUOZBLAS_STATUS_SUCCESS;
    }
    OZB_CHECK(cudaMemsetAsync(st->d_ints, 0, sizeof(int), st->stream));
    OZB_TRY(launch_split_lines<double>(h, false, k, nl, X, ldx, rho, maxS - 1, nullptr, 0, nullptr, st->d_ints));
    OZB_CHECK(cudaMemcpyAsync(st->h_ints, st->d_ints, sizeof(int), cudaMemcpyDeviceToHost, st->stream));
    OZB_CHECK(cudaStreamSynchronize(st->stream));
    int zmax = st->h_ints[0];
    int c = (zmax < 1 ? 1 : zmax) + 1;
    *ns = c < maxS ? c : maxS;
    return CUOZBLAS_STATUS_SUCCESS;
}

int split_lines_write(cuozblasHandle_t *h, int k, int nl, const double *X, int ldx, int rho, int ns, double *out,
                      int ldo) {
    if (nl == 0 || ns == 0) return CUOZBLAS_STATUS_SUCCESS;
    return launch_split_lines<double>(h, true, k, nl, X, ldx, rho, ns, out, ldo, nullptr, nullptr);
}

int split_lines_write_f32(cuozblasHandle_t *h, int k, int nl, const double *X, int ldx, int rho, int ns, float *out,
                          int ldo, short *exps) {
    if (nl == 0 || ns == 0) return CUOZBLAS_STATUS_SUCCESS;
    return launch_split_lines<float>(h, true, k, nl, X, ldx, rho, ns, out, ldo, exps, nullptr);
}

// ---------------------------------------------------------------------------
// Transpose (column-major rows x cols -> cols x rows), 32x32 tiles.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void transpose_tile(int rows, int cols, const T *__restrict__ A, int lda,
                                               T *__restrict__ out, int ldo) {
    __shared__ T t[32][33];
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int r = r0 + threadIdx.x, c = c0 + j;
        t[j][threadIdx.x] = (r < rows && c < cols) ? A[(size_t)c * lda + r] : (T)0;
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int c = c0 + threadIdx.x, r = r0 + j;
        if (r < rows && c < cols) out[(size_t)r * ldo + c] = t[threadIdx.x][j];
    }
}

__global__ void k_transpose(int rows, int cols, const double *__restrict__ A, int lda, double *__restrict__ out,
                            int ldo) {
    transpose_tile<double>(rows, cols, A, lda, out, ldo);
}

__global__ void k_transpose_f32(int rows, int cols, const float *__restrict__ A, int lda, float *__restrict__ out,
                                int ldo) {
    transpose_tile<float>(rows, cols, A, lda, out, ldo);
}

int transpose(cuozblasHandle_t *h, int rows, int cols, const double *A, int lda, double *out, int ldo) {
    if (rows == 0 || cols == 0) return CUOZBLAS_STATUS_SUCCESS;
    dim3 grid((rows + 31) / 32, (cols + 31) / 32), block(32, 8);
    counted(h);
    k_transpose<<<grid, block, 0, state(h)->stream>>>(rows, cols, A, lda, out, ldo);
    OZB_CHECK(cudaGetLastError());
    return CUOZBLAS_STATUS_SUCCESS;
}

int transpose_f32(cuozblasHandle_t *h, int rows, int cols, const float *A, int lda, float *out, int ldo) {
    if (rows == 0 || cols == 0) return CUOZBLAS_STATUS_SUCCESS;
    dim3 grid((rows + 31) / 32, (cols + 31) / 32), block(32, 8);
    counted(h);
    k_transpose_f32<<<grid, block, 0, state(h)->stream>>>(rows, cols, A, lda, out, ldo);
    OZB_CHECK(cudaGetLastError());
    return CUOZBLAS_STATUS_SUCCESS;
}

// ---------------------------------------------------------------------------
// Float data, FP64 slices: the mixed form <float, double, double>
// (src/cpu/ozblas_split.cpp:181-221 with TYPE1 = float).  The arithmetic is
// the reference's float arithmetic: tau = ceil((float)log2((double)max))
// (tau_rule_f32), sigma = (float)(0.75 * (float)2^(rho+tau) * shift),
// slice = (r + sigma) - sigma and r -= slice in float, and the slice stored
// as the double scalbn(slice, -tau) with tau at exps[level * nl + line].
// rho may be negative (k < 32).  One CTA per line, as k_split_lines; `rem`
// holds floats.  COUNT: atomicMax(*zmax, z_line).  WRITE: ns slices.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float sd_sigma(int rho, int tau) {
    const float p = (float)pow2(rho + tau);  // (float)scalbn(1., rho + tau)
    return (float)(0.75 * (double)p);
}

template <bool WRITE>
__global__ void __launch_bounds__(kSplitThreads) k_split_lines_sd(int k, int nl, const float *__restrict__ X, int ldx,
                                                                  int rho, int levels, double *__restrict__ out,
                                                                  int ldo, short *__restrict__ exps,
                                                                  float *__restrict__ gscratch,
                                                                  int *__restrict__ zmax) {
    extern __shared__ float fsmem[];
    __shared__ double red[kSplitThreads / 32];
    const int line = blockIdx.x;
    if (line >= nl) return;
    float *rem = gscratch ? gscratch + (size_t)line * k : fsmem;
    const float *x = X + (size_t)line * ldx;
    float mx = 0.f;
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
        const float v = x[i];
        rem[i] = v;
        const float av = fabsf(v);
        mx = (mx < av) ? av : mx;
    }
    mx = (float)block_max_nonneg((double)mx, red);  // exact: a max of floats
    int z = levels;
    for (int s = 0; s < levels; s++) {
        const int tau = tau_rule_f32(mx);
        const float sigma = sd_sigma(rho, tau);
        float nm = 0.f;
        double *o = WRITE ? out + ((size_t)s * nl + line) * ldo : nullptr;
        if (WRITE && threadIdx.x == 0) exps[(size_t)s * nl + line] = (short)tau;
        for (int i = threadIdx.x; i < k; i += blockDim.x) {
            float r = rem[i];
            const float sl = __fsub_rn(__fadd_rn(r, sigma), sigma);
            r = __fsub_rn(r, sl);
            rem[i] = r;
            const float ar = fabsf(r);
            nm = (nm < ar) ? ar : nm;
            if (WRITE) o[i] = scalbn((double)sl, -tau);  // exact, and exactly a float
        }
        if (WRITE)
            for (int i = k + threadIdx.x; i < ldo; i += blockDim.x) o[i] = 0.0;
        mx = (float)block_max_nonneg((double)nm, red);
        if (!WRITE && mx == 0.f) {
            z = s;
            break;
        }
    }
    if (!WRITE && threadIdx.x == 0) atomicMax(zmax, z);
}

static int launch_split_lines_sd(cuozblasHandle_t *h, bool write, int k, int nl, const float *X, int ldx, int rho,
                                 int levels, double *out, int ldo, short *exps, int *zmax_dev) {
    State *st = state(h);
    float *gscratch = nullptr;
    size_t smem = 0;
    Arena ar(h);
    const uint64_t mk = ar.mark();
    if (k > 2 * kSplitSmemMaxK) {
        gscratch = ar.take<float>((uint64_t)k * nl);
        if (!ar.ok) return CUOZBLAS_STATUS_WORKSPACE;
    } else {
        smem = sizeof(float) * (size_t)(k > 0 ? k : 1);
    }
    const int maxsmem = (int)(2 * kSplitSmemMaxK * sizeof(float));
    if (write) {
        OZB_CHECK(cudaFuncSetAttribute(k_split_lines_sd<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxsmem));
        counted(h);
        k_split_lines_sd<true><<<nl, kSplitThreads, smem, st->stream>>>(k, nl, X, ldx, rho, levels, out, ldo, exps,
                                                                         gscratch, nullptr);
    } else {
        OZB_CHECK(cudaFuncSetAttribute(k_split_lines_sd<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxsmem));
        counted(h);
        k_split_lines_sd<false><<<nl, kSplitThreads, smem, st->stream>>>(k, nl, X, ldx, rho, levels, nullptr, 0,
                                                                          nullptr, gscratch, zmax_dev);
    }
    OZB_CHECK(cudaGetLastError());
    ar.release(mk);
    return CUOZBLAS_STATUS_SUCCESS;
}

int split_lines_count_sd(cuozblasHandle_t *h, int k, int nl, const float *X, int ldx, int rho, int maxS, int *ns) {
    State *st = state(h);
    if (maxS <= 1 || nl == 0) {
        *ns = (nl == 0) ? (maxS < 2 ? maxS : 2) : 1;
        if (maxS <= 1) *ns = 1;
        return CUOZBLAS_STATUS_SUCCESS;
    }
    OZB_CHECK(cudaMemsetAsync(st->d_ints, 0, sizeof(int), st->stream));
    OZB_TRY(launch_split_lines_sd(h, false, k, nl, X, ldx, rho, maxS - 1, nullptr, 0, nullptr, st->d_ints));
    OZB_CHECK(cudaMemcpyAsync(st->h_ints, st->d_ints, sizeof(int), cudaMemcpyDeviceToHost, st->stream));
    OZB_CHECK(cudaStreamSynchronize(st->stream));
    const int zmax = st->h_ints[0];
    const int c = (zmax < 1 ? 1 : zmax) + 1;
    *ns = c < maxS ? c : maxS;
    return CUOZBLAS_STATUS_SUCCESS;
}

int split_lines_write_sd(cuozblasHandle_t *h, int k, int nl, const float *X, int ldx, int rho, int ns, double *out,
                         int ldo, short *exps) {
    if (nl == 0 || ns == 0) return CUOZBLAS_STATUS_SUCCESS;
    return launch_split_lines_sd(h, true, k, nl, X, ldx, rho, ns, out, ldo, exps, nullptr);
}

// ---------------------------------------------------------------------------
// Vector split: one global tau chain (src/cpu/ozblas_split.cpp:62-103 and the
// driver :254-289 with n = 1).  One cooperative launch runs every level; the
// grid syncs after each level's max reduction.  rem: n doubles of scratch.
// slot[s] = max|remainder| entering level s (slot[0] = max|x|); *ns_out is
// written by block 0, and for FP32 slices exps[s] = tau of level s.
// ---------------------------------------------------------------------------
template <typename SL>
__global__ void __launch_bounds__(256) k_split_vector(int n, const double *__restrict__ x, int rho, int maxS,
                                                      SL *__restrict__ out, int ldo, short *__restrict__ exps,
                                                      double *__restrict__ rem, double *__restrict__ slot,
                                                      int *__restrict__ ns_out) {
    cg::grid_group grid = cg::this_grid();
    __shared__ double red[8];
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    double m = 0.0;
    for (size_t i = tid; i < (size_t)n; i += stride) m = ref_max(m, fabs(x[i]));
    m = block_max_nonneg(m, red);
    if (threadIdx.x == 0) atomic_max_nonneg(&slot[0], m);
    grid.sync();
    int s = 0;
    for (; s < maxS; s++) {
        const double mx = slot[s];
        if (s >= 2 && slot[s] == 0.0) break;  // previous level left nothing: the count is s
        const int tau = tau_rule(mx);
        const double sigma = 0.75 * pow2(rho + tau);  // dense_sigma(rho, mx, 1)
        const double *src = (s == 0) ? x : rem;
        SL *o = out + (size_t)s * ldo;
        if (exps && tid == 0) exps[s] = (short)tau;
        double nm = 0.0;
        for (size_t i = tid; i < (size_t)n; i += stride) {
            double r = src[i];
            const double sl = (r + sigma) - sigma;
            r = r - sl;
            rem[i] = r;
            o[i] = slice_store<SL>(sl, tau);
            nm = ref_max(nm, fabs(r));
        }
        for (size_t i = (size_t)n + tid; i < (size_t)ldo; i += stride) o[i] = (SL)0;
        nm = block_max_nonneg(nm, red);
        if (threadIdx.x == 0) atomic_max_nonneg(&slot[s + 1], nm);
        grid.sync();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *ns_out = s;
}

template <typename SL>
static int split_vector_t(cuozblasHandle_t *h, int n, const double *x, int rho, int maxS, SL *out, int ldo,
                          short *exps, int *ns) {
    State *st = state(h);
    Arena ar(h);
    const uint64_t mk = ar.mark();
    double *rem = ar.take<double>(n > 0 ? n : 1);
    double *slot = ar.take<double>(kMaxSplitDefault + 2);
    if (!ar.ok) return CUOZBLAS_STATUS_WORKSPACE;
    OZB_CHECK(cudaMemsetAsync(slot, 0, sizeof(double) * (kMaxSplitDefault + 2), st->stream));
    int dev = 0, nsm = 0, per = 0;
    OZB_CHECK(cudaGetDevice(&dev));
    OZB_CHECK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    OZB_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_split_vector<SL>, 256, 0));
    int blocks = nsm * (per < 4 ? per : 4);
    const int need = (n + 255) / 256;
    if (blocks > need) blocks = need > 0 ? need : 1;
    int *ns_dev = st->d_ints;
    void *args[] = {&n, &x, &rho, &maxS, &out, &ldo, &exps, &rem, &slot, &ns_dev};
    counted(h);
    OZB_CHECK(cudaLaunchCooperativeKernel((void *)k_split_vector<SL>, dim3(blocks), dim3(256), args, 0, st->stream));
    OZB_CHECK(cudaMemcpyAsync(st->h_ints, ns_dev, sizeof(int), cudaMemcpyDeviceToHost, st->stream));
    OZB_CHECK(cudaStreamSynchronize(st->stream));
    *ns = st->h_ints[0];
    ar.release(mk);
    return CUOZBLAS_STATUS_SUCCESS;
}

int split_vector(cuozblasHandle_t *h, int n, const double *x, int rho, int maxS, double *out, int ldo, int *ns) {
    if (n <= kSplitVectorSmallMax && ldo <= kSplitVectorSmallMax)
        return split_vector_small(h, n, x, rho, maxS, out, ldo, ns);
    return split_vector_t<double>(h, n, x, rho, maxS, out, ldo, nullptr, ns);
}

int split_vector_f32(cuozblasHandle_t *h, int n, const double *x, int rho, int maxS, float *out, int ldo, short *exps,
                     int *ns) {
    return split_vector_t<float>(h, n, x, rho, maxS, out, ldo, exps, ns);
}

// ---------------------------------------------------------------------------
// CSR row split (src/cpu/ozblas_split.cpp:779-815, driver :875-928): rho from
// the row's nnz; sigma divided by shift.  The count pass leaves the largest
// z in *zmax, the write pass writes `levels` slices of nnz.
//
// W lanes hold a row and kCsrHeld entries each in registers, W so that this
// covers twice the mean row length: the level's sigma is computed by every lane
// of a row, so wider rows only repeat it.  The counts are folded per block: one
// atomic per row on the one counter was the bound (10^6 rows of 7 with it and a
// warp per row: 675 us, of which the 56 MB of values account for 9; 8 lanes per
// row 94, 4 lanes 55; the writing pass 385 -> 63).
//
// Longer rows keep their remainders in `rem` (nnz doubles).  Its own lanes walk a
// row of up to kCsrWalk entries each.  Beyond that a row stands out (at most one
// in 8 does): the block lists those and its warps share them at the end, up to
// csr_block_row entries.  The rest is left to k_split_csr_long, which the count
// pass asks for when it meets one: a launch and a host wait more, 25 us a pass.
// 10^6 rows of 3 with 1000 of 600, cuozblasDcsrmvSplitA: 0.45 ms (1.2 in their two
// lanes, 1.5 in k_split_csr_long, 4.0 with a warp for every row).
// ---------------------------------------------------------------------------
constexpr int kCsrHeld = 4;   // entries of a row per lane in registers
constexpr int kCsrWalk = 16;  // entries per lane that the row's own lanes walk (W < 32)
constexpr int kCsrList = 512;
__host__ __device__ constexpr int csr_block_row(int lanes) { return lanes < 32 ? 1024 : 8192; }

// The split of the row of n entries from lo by W lanes of a warp (`mask`; this
// one is `sub`), the remainders in memory, the loads of four steps in flight.
// Returns the first level that leaves nothing.
template <bool WRITE, int W>
__device__ __forceinline__ int split_row_rem(int lo, int n, int sub, unsigned mask, const double *__restrict__ val,
                                             int epsmode, int shift, int levels, double *__restrict__ rem,
                                             double *__restrict__ out, int64_t ldo) {
    constexpr int U = 4;
    val += lo;
    rem += lo;
    if (WRITE) out += lo;
    double mx = 0.0;
    for (int i = sub; i < n; i += W) mx = ref_max(mx, fabs(val[i]));
    for (int o = W / 2; o > 0; o >>= 1) mx = ref_max(mx, __shfl_xor_sync(mask, mx, o));
    const int rho = rho_rule(n, epsmode);
    for (int s = 0; s < levels; s++) {
        const double sigma = shift_sigma(0.75 * pow2(rho + tau_rule(mx)), shift);
        const double *from = s == 0 ? val : rem;
        double nm = 0.0;
        for (int i0 = sub; i0 < n; i0 += U * W) {
            double v[U];
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = i0 + u * W < n ? from[i0 + u * W] : 0.0;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 + u * W;
                if (i < n) {
                    const double sl = (v[u] + sigma) - sigma;
                    const double r = v[u] - sl;
                    rem[i] = r;
                    nm = ref_max(nm, fabs(r));
                    if (WRITE) out[(size_t)s * ldo + i] = sl;
                }
            }
        }
        for (int o = W / 2; o > 0; o >>= 1) nm = ref_max(nm, __shfl_xor_sync(mask, nm, o));
        mx = nm;
        if (!WRITE && mx == 0.0) return s;
    }
    return levels;
}

template <bool WRITE, int W>
__global__ void __launch_bounds__(256) k_split_csr(int m, const double *__restrict__ val,
                                                   const int *__restrict__ rowptr, int epsmode, int shift,
                                                   int levels, double *__restrict__ rem, double *__restrict__ out,
                                                   int64_t ldo, int *__restrict__ zmax, int *__restrict__ longer) {
    __shared__ int zsh[8], list[kCsrList], nlist;
    const int lane = threadIdx.x & 31, sub = lane % W;
    const unsigned rows_lanes = W == 32 ? 0xffffffffu : ((1u << W) - 1u) << (lane - sub);  // this row's lanes
    const int64_t nrows = (int64_t)gridDim.x * (256 / W);
    int zbest = 0;
    if (W < 32) {
        if (threadIdx.x == 0) nlist = 0;
        __syncthreads();
    }
    // base: the warp's first row
    for (int64_t base = ((int64_t)blockIdx.x * 256 + (threadIdx.x & ~31)) / W; base < m; base += nrows) {
        const int64_t row = base + lane / W;
        const int lo = row < m ? rowptr[row] : 0, hi = row < m ? rowptr[row + 1] : 0;
        const int len = hi - lo;  // uniform over the row's lanes; an empty row has z = 0
        if (len > 0 && len <= kCsrHeld * W) {
            double r[kCsrHeld], mx = 0.0;
#pragma unroll
            for (int e = 0; e < kCsrHeld; e++) {
                const int i = lo + e * W + sub;
                r[e] = i < hi ? val[i] : 0.0;
                mx = ref_max(mx, fabs(r[e]));
            }
            for (int o = W / 2; o > 0; o >>= 1) mx = ref_max(mx, __shfl_xor_sync(rows_lanes, mx, o));
            int z = levels;
            const int rho = rho_rule(len, epsmode);
            for (int s = 0; s < levels; s++) {
                const double sigma = shift_sigma(0.75 * pow2(rho + tau_rule(mx)), shift);
                double nm = 0.0;
#pragma unroll
                for (int e = 0; e < kCsrHeld; e++) {
                    const int i = lo + e * W + sub;
                    if (i < hi) {
                        const double sl = (r[e] + sigma) - sigma;
                        r[e] = r[e] - sl;
                        nm = ref_max(nm, fabs(r[e]));
                        if (WRITE) out[(size_t)s * ldo + i] = sl;
                    }
                }
                for (int o = W / 2; o > 0; o >>= 1) nm = ref_max(nm, __shfl_xor_sync(rows_lanes, nm, o));
                mx = nm;
                if (!WRITE && mx == 0.0) {
                    z = s;
                    break;
                }
            }
            zbest = z > zbest ? z : zbest;
        } else if (len > csr_block_row(W)) {
            if (!WRITE && sub == 0) *longer = 1;
        } else if (len > 0) {
            bool own = W == 32 || len <= kCsrWalk * W;
            if (!own) {
                int at = sub == 0 ? atomicAdd(&nlist, 1) : 0;
                at = __shfl_sync(rows_lanes, at, lane - sub);
                own = at >= kCsrList;  // no room
                if (!own && sub == 0) list[at] = (int)row;
            }
            if (own) {
                const int z = split_row_rem<WRITE, W>(lo, len, sub, rows_lanes, val, epsmode, shift, levels, rem, out, ldo);
                zbest = z > zbest ? z : zbest;
            }
        }
    }
    if (W < 32) {
        __syncthreads();
        const int n = nlist < kCsrList ? nlist : kCsrList;
        for (int k = threadIdx.x >> 5; k < n; k += 8) {
            const int lo = rowptr[list[k]], len = rowptr[list[k] + 1] - lo;
            const int z = split_row_rem<WRITE, 32>(lo, len, lane, 0xffffffffu, val, epsmode, shift, levels, rem, out, ldo);
            zbest = z > zbest ? z : zbest;
        }
    }
    if (!WRITE) {
        const int zw = __reduce_max_sync(0xffffffffu, zbest);
        if (lane == 0) zsh[threadIdx.x >> 5] = zw;
        __syncthreads();
        if (threadIdx.x == 0) {
            int zb = 0;
            for (int w = 0; w < 8; w++) zb = zsh[w] > zb ? zsh[w] : zb;
            if (zb > 0) atomicMax(zmax, zb);
        }
    }
}

// The rows of more than `over` entries, a block per row.  Row r belongs to block
// r % gridDim.x, so long rows that stand together are spread over the chip; a
// block finds its own 1024 at a time.  cuozblasDcsrmvSplitA (a count per shift and
// the write) of 10^6 rows of 3 with one of 10^5: 1.65 ms (in a row's own two lanes
// 347, with a warp for every row 13.7); with 1000 of 5000 side by side 1.6 (15.8,
// 6.5); without such rows 0.75 (8.2).
constexpr int kCsrLongThreads = 1024;

template <bool WRITE>
__global__ void __launch_bounds__(kCsrLongThreads) k_split_csr_long(int m, int over, const double *__restrict__ val,
                                                                    const int *__restrict__ rowptr, int epsmode,
                                                                    int shift, int levels, double *__restrict__ rem,
                                                                    double *__restrict__ out, int64_t ldo,
                                                                    int *__restrict__ zmax) {
    __shared__ int list[kCsrLongThreads], nlist;
    __shared__ double red[kCsrLongThreads / 32];
    const int t = threadIdx.x;
    int zbest = 0;
    for (int64_t r0 = blockIdx.x; r0 < m; r0 += (int64_t)gridDim.x * kCsrLongThreads) {
        __syncthreads();
        if (t == 0) nlist = 0;
        __syncthreads();
        const int64_t row = r0 + (int64_t)gridDim.x * t;
        if (row < m && rowptr[row + 1] - rowptr[row] > over) list[atomicAdd(&nlist, 1)] = (int)row;
        __syncthreads();
        for (int k = 0; k < nlist; k++) {
            const int lo = rowptr[list[k]];
            const int64_t n = rowptr[list[k] + 1] - lo;
            double *r = rem + lo;
            double mx = 0.0;
            for (int64_t i = t; i < n; i += kCsrLongThreads) mx = ref_max(mx, fabs(val[lo + i]));
            mx = block_max_nonneg(mx, red);
            int z = levels;
            const int rho = rho_rule((int)n, epsmode);
            for (int s = 0; s < levels; s++) {
                const double sigma = shift_sigma(0.75 * pow2(rho + tau_rule(mx)), shift);
                const double *from = s == 0 ? val + lo : r;
                double nm = 0.0;
                for (int64_t i = t; i < n; i += kCsrLongThreads) {
                    double v = from[i];
                    const double sl = (v + sigma) - sigma;
                    v = v - sl;
                    r[i] = v;
                    nm = ref_max(nm, fabs(v));
                    if (WRITE) out[(size_t)s * ldo + lo + i] = sl;
                }
                mx = block_max_nonneg(nm, red);
                if (!WRITE && mx == 0.0) {  // uniform
                    z = s;
                    break;
                }
            }
            zbest = z > zbest ? z : zbest;
        }
    }
    if (!WRITE && t == 0 && zbest > 0) atomicMax(zmax, zbest);
}

// Lanes per row (see above).
static int split_csr_lanes(int m, int nnz) {
    const int64_t mean = m > 0 ? ((int64_t)nnz + m - 1) / m : 0;
    return mean <= 4 ? 2 : mean <= 8 ? 4 : mean <= 16 ? 8 : mean <= 32 ? 16 : 32;
}

template <bool WRITE>
static int split_csr_launch(cuozblasHandle_t *h, int m, int lanes, const double *val, const int *rowptr, int epsmode,
                            int shift, int levels, double *rem, double *out, int64_t ldo, int *zmax, int *longer) {
    if (m <= 0) return CUOZBLAS_STATUS_SUCCESS;
    cudaStream_t s = state(h)->stream;
    auto go = [&](auto width) {
        constexpr int W = decltype(width)::value;
        // one resident wave, so that the counts fold; a few waves of one row per warp as they come
        const int64_t need = ((int64_t)m + 256 / W - 1) / (256 / W), cap = (int64_t)sm_count() * 8;
        k_split_csr<WRITE, W><<<(int)(need < (W < 32 ? cap : 8 * cap) ? need : cap), 256, 0, s>>>(m, val, rowptr, epsmode, shift, levels,
                                                                             rem, out, ldo, zmax, longer);
    };
    counted(h);
    switch (lanes) {
        case 2: go(std::integral_constant<int, 2>{}); break;
        case 4: go(std::integral_constant<int, 4>{}); break;
        case 8: go(std::integral_constant<int, 8>{}); break;
        case 16: go(std::integral_constant<int, 16>{}); break;
        default: go(std::integral_constant<int, 32>{}); break;
    }
    OZB_CHECK(cudaGetLastError());
    return CUOZBLAS_STATUS_SUCCESS;
}

template <bool WRITE>
static int split_csr_long_launch(cuozblasHandle_t *h, int m, int lanes, const double *val, const int *rowptr,
                                 int epsmode, int shift, int levels, double *rem, double *out, int64_t ldo, int *zmax) {
    if (m <= 0) return CUOZBLAS_STATUS_SUCCESS;
    const int cap = sm_count() * 2;
    counted(h);
    k_split_csr_long<WRITE><<<m < cap ? m : cap, kCsrLongThreads, 0, state(h)->stream>>>(
        m, csr_block_row(lanes), val, rowptr, epsmode, shift, levels, rem, out, ldo, zmax);
    OZB_CHECK(cudaGetLastError());
    return CUOZBLAS_STATUS_SUCCESS;
}

int split_csr_count(cuozblasHandle_t *h, int m, const double *val, const int *rowptr, int epsmode, int shift,
                    int maxS, int *ns, CsrSplitRows *rows) {
    State *st = state(h);
    *rows = CsrSplitRows{};  // not looked at
    if (maxS <= 1) {
        *ns = 1;
        return CUOZBLAS_STATUS_SUCCESS;
    }
    int nnz = 0;
    OZB_CHECK(cudaMemcpyAsync(st->h_ints, rowptr + m, sizeof(int), cudaMemcpyDeviceToHost, st->stream));
    OZB_CHECK(cudaStreamSynchronize(st->stream));
    nnz = st->h_ints[0];
    rows->lanes = split_csr_lanes(m, nnz);
    Arena ar(h);
    const uint64_t mk = ar.mark();
    double *rem = ar.take<double>(nnz > 0 ? nnz : 1);
    if (!ar.ok) return CUOZBLAS_STATUS_WORKSPACE;
    int *res = st->d_ints;  // the largest z, whether a row was left out as too long
    OZB_CHECK(cudaMemsetAsync(res, 0, 2 * sizeof(int), st->stream));
    OZB_TRY(split_csr_launch<false>(h, m, rows->lanes, val, rowptr, epsmode, shift, maxS - 1, rem, nullptr, 0, res,
                                    res + 1));
    OZB_CHECK(cudaMemcpyAsync(st->h_ints, res, 2 * sizeof(int), cudaMemcpyDeviceToHost, st->stream));
    OZB_CHECK(cudaStreamSynchronize(st->stream));
    rows->longer = st->h_ints[1] != 0;
    if (rows->longer) {
        OZB_TRY(split_csr_long_launch<false>(h, m, rows->lanes, val, rowptr, epsmode, shift, maxS - 1, rem, nullptr, 0,
                                             res));
        OZB_CHECK(cudaMemcpyAsync(st->h_ints, res, sizeof(int), cudaMemcpyDeviceToHost, st->stream));
        OZB_CHECK(cudaStreamSynchronize(st->stream));
    }
    const int zmax = st->h_ints[0];
    const int c = (zmax < 1 ? 1 : zmax) + 1;
    *ns = c < maxS ? c : maxS;
    ar.release(mk);
    return CUOZBLAS_STATUS_SUCCESS;
}

int split_csr_write(cuozblasHandle_t *h, int m, int nnz, const double *val, const int *rowptr, int epsmode,
                    int shift, int ns, double *out, int64_t ld, const CsrSplitRows &rows) {
    const int lanes = rows.lanes > 0 ? rows.lanes : split_csr_lanes(m, nnz);
    Arena ar(h);
    const uint64_t mk = ar.mark();
    double *rem = ar.take<double>(nnz > 0 ? nnz : 1);
    if (!ar.ok) return CUOZBLAS_STATUS_WORKSPACE;
    OZB_TRY(split_csr_launch<true>(h, m, lanes, val, rowptr, epsmode, shift, ns, rem, out, ld, nullptr, nullptr));
    if (rows.longer)
        OZB_TRY(split_csr_long_launch<true>(h, m, lanes, val, rowptr, epsmode, shift, ns, rem, out, ld, nullptr));
    ar.release(mk);
    return CUOZBLAS_STATUS_SUCCESS;
}

}  // namespace ozb
