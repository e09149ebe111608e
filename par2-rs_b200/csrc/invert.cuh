// invert.cuh -- device Gauss-Jordan over GF(2^16).
#pragma once
#include "common.cuh"

namespace p2g {

// Scratch of one inversion: the augmented matrix and a status word.
struct GjWork {
    DevBuf &M;
    DevBuf &status;
};

// Inverts the m x m matrix given either as PAR2 constants of the missing
// slices and recovery exponents (A[row][col] = cmiss[col]^exps[row]) or, when
// d_A is non-null, as a dense row-major device matrix.  d_inv receives A^-1
// (row-major m x m).  h_exps (optional) is a host copy of the exponents: when
// they are a permutation of consecutive values, the closed-form Vandermonde
// inverse replaces the elimination.  Singularity is reported by gj_status.
// beside: it runs beside other work, on few SMs and in few launches if it can.
int gj_invert(p2g_ctx *ctx, GjWork &w, int m, const uint16_t *d_cmiss, const uint32_t *d_exps,
              const uint32_t *h_exps, const uint16_t *d_A, uint16_t *d_inv, bool beside = false);

// Inverses that the closed form makes in one CTA each, in one launch: m
// consecutive exponents from s on, in any order (small_inverse says whether and
// finds s; `alone`: whether it is also the faster way for a single one); x are the
// missing slices' constants, ld the row stride of inv and *status becomes 1 where
// the matrix is singular, else 0.
struct SmallInverse {
    const uint16_t *x;
    const uint32_t *exps;
    uint16_t *inv;
    int *status;
    uint32_t s;
    int m, ld;
};
bool small_inverse(const uint32_t *h_exps, int m, uint32_t *s, bool alone = false);
int small_inverses(p2g_ctx *ctx, const SmallInverse *d_items, int n);

// Whether an inversion of m rows runs in one CTA, without the multiply-accumulate
// kernels and their scratch: it can then run beside them, on another stream.
bool gj_one_cta(int m);

// Waits for the inversion and reads its status (1 = singular).
int gj_status(p2g_ctx *ctx, GjWork &w, int *singular);

}  // namespace p2g
