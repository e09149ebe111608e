// tensor.cuh -- host launchers of the tensor-core multiply-accumulate.
#pragma once
#include "common.cuh"
#include "prep.cuh"

namespace p2g {

constexpr int kTensorM = 128;      // symbols per accumulator tile (two tiles per CTA)
constexpr int kTensorMaxN = 208;   // outputs per block, at most
constexpr int kTensorStage = 256;  // inputs per pipeline stage

// Output blocks of a problem and the rows of each (a multiple of 16).
inline int tensor_blocks(int nout) { return (nout + kTensorMaxN - 1) / kTensorMaxN; }
inline int tensor_rows(int nout)
{
    const int nblk = tensor_blocks(nout);
    return ((nout + nblk - 1) / nblk + 15) / 16 * 16;
}
inline int tensor_stages(int nin) { return (nin + kTensorStage - 1) / kTensorStage; }
// 32-input words of the coefficient operand: whole products of K = 64
inline int tensor_words(int nin) { return (nin + 63) / 64 * 2; }

// Bytes of the coefficient operand of an nin x nout problem.
size_t tensor_coef_bytes(int nin, int nout);
// Bytes of the symbol operand for `tiles` tiles of 128 symbols of nin inputs.
size_t tensor_form_bytes(int nin, size_t tiles);

// The coefficient operand.
int tensor_coefs(cudaStream_t st, const CoefSource &c, const uint16_t *glog, const uint16_t *gexp,
                 int nin, int nout, void *coef);

// SM clocks that a problem takes (an estimate), and the parts its work is split
// into for that (folded with atomic XOR).
double tensor_clocks(int sms, int nin, int nout, size_t S, int *split);
inline int tensor_splits(int sms, int nin, int nout, size_t S)
{
    int split = 1;
    tensor_clocks(sms, nin, nout, S, &split);
    return split;
}

// dst[o] (^)= sum over inputs [i0, i0 + nin) of coeff(i, o) * src[i - i0] over
// slices of S bytes; coef is the operand of a whole problem of nin_total
// inputs and i0 a multiple of 64.
struct TensorRun {
    const uint8_t *const *src;  // device array of nin slice pointers (16-byte aligned)
    uint8_t *const *dst;        // device array of nout slice pointers
    int nin_total, i0, nin, nout;
    size_t S;
    const void *coef;
    void *forms;  // tensor_form_bytes(nin, tiles) bytes for the tiles of one launch
    int mode;     // 0 stores, 1 XORs
    int split;    // parts of the work; above 1 they are XORed atomically into dst
    int *err;     // device-visible word, set when a bounded wait gave up
    uint32_t tries;  // of a thread's waits (kWaitTries)
};
inline size_t tensor_tiles(size_t S) { return (S / 2 + kTensorM - 1) / kTensorM; }
// The forms of tiles [t0, t0 + n), the coefficient operand (r.coef, of the whole
// problem) where `todo` is given, and the outputs' start; then the products of the
// same tiles.
int tensor_prepare(cudaStream_t st, const TensorRun &r, size_t t0, size_t n, const CoefSource *todo,
                   const uint16_t *glog, const uint16_t *gexp, const OutputPrep &z);
int tensor_products(cudaStream_t st, const TensorRun &r, size_t t0, size_t n);

// ---- batches: the same three kernels over many problems -------------------

// What the products kernel reads of a problem (device-resident in a batch).
struct TensorArgs {
    const uint32_t *forms;  // [tile pair][30][8 * stage][256]
    const uint4 *coef;      // [nblk][60][cwords][rows]
    uint8_t *const *dst;
    size_t S;
    size_t byte0;     // first byte of the chunk
    int tiles;        // tiles of the chunk
    int steps;        // of 64 inputs
    int cwords, cw0;  // words of the coefficients, and this run's first
    int rows, nblk, nout, mode;
    int split;  // parts of the 60 products (above 1: partial results are XORed atomically)
    int *err;
    uint32_t tries;
};
// One CTA's work: a tile pair, an output block and a part of the products.
struct TensorItem {
    int prob, pair, nb, part;
};
// `first`: the problem's first CTA of the batched launch (forms: tile pairs x
// 64-input groups; coefficients: 32 rows x 4 words).
struct TensorFormProb {
    const uint8_t *const *src;
    uint32_t *forms;
    size_t S;
    int nin;
    unsigned long long first;
};
struct TensorCoefProb {
    const uint16_t *coeff;  // matrix, or null: consts[i]^exps[o]
    const uint16_t *consts;
    const uint32_t *exps;
    uint4 *coef;
    int nin, nout;
    unsigned long long first;
};
inline unsigned long long tensor_form_ctas(int nin, size_t S)
{
    return static_cast<unsigned long long>((tensor_tiles(S) + 1) / 2) * ((nin + 63) / 64);
}
inline unsigned long long tensor_coef_ctas(int nin, int nout)
{
    return static_cast<unsigned long long>((tensor_rows(nout) * tensor_blocks(nout) + 31) / 32) *
           ((tensor_words(nin) + 3) / 4);
}
// SM clocks per tile pair of a problem that runs among others: the products of
// all its output blocks, and the forms.
double tensor_pair_clocks(int nin, int nout);
// SM clocks of one item that takes `products` of the 60.
double tensor_item_clocks(int nin, int nout, int products);

int tensor_batch_forms(cudaStream_t st, const TensorFormProb *d, int np, unsigned long long ctas);
int tensor_batch_coefs(cudaStream_t st, const uint16_t *glog, const uint16_t *gexp,
                       const TensorCoefProb *d, int np, unsigned long long ctas);
// One CTA per item, in the order given (longest first); `rows` the largest of
// the problems'.  A CTA that starts once *abort is set does nothing.
int tensor_batch(cudaStream_t st, const TensorArgs *probs, const TensorItem *items, int nitems, int rows,
                 const volatile int *abort);

}  // namespace p2g
