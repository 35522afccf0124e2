// gemm_pairs.h — exact slice-pair products on the INT8 tensor cores, shared by
// the forms whose slices are integers times a power of two: the plain form,
// <float,double,double> and the quad form.
#pragma once
#include <stdint.h>

#include "ozb_internal.h"

namespace ozb {

// A slice is q 2^g with an integer |q| <= 2^bits.  q is cut into `D` signed
// digits of radix 2^radix, most significant first: q = sum_d digit_d
// 2^(radix (D-1-d)), digit in [-2^(radix-1), 2^(radix-1)).
struct PairDigits {
    int D = 0;      // 3 or 4 (0: no form fits, see pair_digits)
    int radix = 8;  // 8, or 7 where k products of 8-bit digits would leave INT32
};

// The digit form for slices of `bits` bits and products over k terms: every
// accumulator sums at most D k products of at most 2^(2 radix - 2).
PairDigits pair_digits(int bits, int k);

// The digit planes of one operand: plane (level s, digit d) is nl lines of
// k_pad bytes at dig + ((s D + d) nl) k_pad; exps[s * nl + line] the level's
// tau, kExpZero where the line has no slice at that level (its digits are then
// unwritten), kExpNaN where the line holds Inf or NaN or its split overflows.
struct PairOperand {
    int8_t *dig = nullptr;
    short *exps = nullptr;
    int *tile_lev = nullptr;  // levels in use per tile of the product kernel (null: all)
    int nl = 0, levels = 0;   // lines, levels the planes hold
};
constexpr short kExpZero = -32768, kExpNaN = -32767;  // both far below any exponent, also in a sum

// Where the pair products go.
enum PairEpi {
    kPairStore = 0,  // pbuf[pair][col][row] = sum q q as a 64-bit integer (|.| < 2^53)
    kPairFsum = 1,   // C = fma(alpha, t, beta C), t the FP64 sum of the products in pair order
    kPairSd = 2,     // the <float,double,double> sum: each product rounded to float, scaled, added in float
};

// Lines per tile of the two operands for a digit form (the sizes of tile_lev).
constexpr int kPairTileA = 128;
inline int pair_tile_b(int D) { return D == 3 ? 96 : 64; }

// k up to this is split on chip by pair_split.
constexpr int kPairSplitMaxK = 16384;

// Split nl contiguous lines of length k (line l at X + l * ldx) into digit
// planes for at most `levels` levels (op.levels); counts every level up to maxS.  The
// count of levels the reference would use (min(maxS, max(1, z) + 1)) goes to
// *ns_dev as max z; op's buffers are the caller's.  T: double (plain form) or
// float (<float,double,double>, slices scaled by 2^-tau: same digits).
template <typename T>
int pair_split(cuozblasHandle_t *h, int k, int k_pad, const T *X, int ldx, int rho, int maxS, const PairDigits &pd,
               int tile_lines, const PairOperand &op, int *zmax_dev);

// The products of every pair (ia, ib), ia + ib <= maxlevel, ia < nA, ib < nB.
// A bounded wait that runs out sets the handle's error word (kPairErrInt): a sum
// over the pair buffer must leave C alone then (kPairFsum and kPairSd have stored
// the tiles that were complete), and pair_status reports it.
struct PairCall {
    int m, n, k_pad, nA, nB, maxlevel;
    int bias = 0;  // a pair product is 2^(bias + tauA + tauB) sum q q (kPairStore: for the sum that reads pbuf)
    PairEpi epi;
    double alpha = 1.0, beta = 0.0;
    void *C = nullptr;
    int ldc = 0;
    double *pbuf = nullptr;  // kPairStore: np m cn entries, else pair_handover_doubles
    int col0 = 0, cn = 0;    // kPairStore: the columns of this launch, from a tile boundary (cn = 0: all)
};
// Partial sums that one CTA of a fused launch hands to the next, and their flags.
inline uint64_t pair_handover_doubles(int D) { return (uint64_t)sm_count() * (128 * pair_tile_b(D) + 4); }
int pair_products(cuozblasHandle_t *h, const PairDigits &pd, const PairOperand &A, const PairOperand &B,
                  const PairCall &c);
constexpr int kPairErrInt = 2;  // the kernel's error word among the handle's device ints (zeroed by the caller)
// Waits for the stream and reports a wait that ran out in the product kernel.
int pair_status(cuozblasHandle_t *h);

// The whole product (gemm_pairs.cu); rho the split's, *done false when the
// form does not apply and the caller's slice path must run.
template <typename T>
int gemm_pairs_core(cuozblasHandle_t *h, char ta, char tb, int m, int n, int k, double alpha, const T *A, int lda,
                    const T *B, int ldb, double beta, T *C, int ldc, int fastMode, int rho, bool *done);

}  // namespace ozb
