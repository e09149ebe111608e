// tensor.cu -- GF(2^16) region multiply-accumulate on the tensor cores.
//
// The same operation as muladd.cu (par2-rs galois/simd/x86/avx2.rs:686-821,
// par2_rs.rs:816-870),
//
//     dst[o][x] (^)= XOR_i  coeff(i, o) * src[i][x]      (GF(2^16), 0x1100B)
//
// as 60 matrix products of bits (bilinear.cuh): with the 60 linear forms of
// every coefficient and of every symbol,
//
//     P_e[x][o] = sum_i  phi_e(src[i][x]) * phi_e(coeff(i, o)),   e = 0..59
//     dst[o][x] ^= XOR_e  (P_e[x][o] odd ? w_e : 0).
//
// The bits are 4-bit floating-point numbers of value 0 or 1 and the sums run
// in the 32-bit accumulators of tcgen05.mma (kind::mxf4, block scales of powers
// of two); they are whole multiples of the scale, so they are exact and their
// parity is the GF(2) sum.  One symbol times one coefficient takes 60
// multiply-adds, of which an SM does 16384 per clock; the table kernels spend
// 4 bytes of shared-memory reads on it, of which an SM does 128 per clock.
//
//   * forms_of_pair reads the slices once and writes the 30 forms that all 60
//     phi_e are sums of (1, 2 or 4 of them) as bits, 32 inputs to a word.
//   * coef_block writes the coefficients' 60 forms as the 4-bit B operand.
//   * tensor_muladd: a CTA owns 256 symbols (two accumulator tiles of 128
//     rows) and up to 208 outputs (columns).  For each e it runs over all
//     inputs in stages of 256: four warps per tile turn the form words of 128
//     symbols into the 4-bit A operand in tensor memory, one warp per tile
//     issues the products, and eight warps per tile then read the accumulators
//     and add w_e where they are odd, while the other tile's products run.
//     A in tensor memory leaves shared memory to B alone, read twice (once per
//     tile) for one copy from L2 -- from shared memory, A's writes and reads
//     would hold the products to 75 % of their rate.
//
// The accumulators are not cleared between products: they start at 2^23 and
// keep counting, so that what is read after e is the parity of the sum over
// 0..e, which only changes the constants (w_e ^ w_{e+1} instead of w_e).  With
// a scale of 2^7 the sums' units are bit 7 of the accumulators' low byte, where
// one byte permute spreads them over an output's 16 bits; the low 16 bits are
// all that is read (packed in pairs by the load).  Before the sums reach 2^24
// the accumulators are set back: every 65535 / inputs products.
//
// Bounds, on one B200 at 1.9 GHz, 2048 inputs of 1 MiB: 205 outputs 3.8 ms
// (the products' issue rate alone 2.8 ms: one product takes 104 clocks at 208
// columns; the paired table kernel 31.4 ms); 13 outputs 2.0 ms (1.3 ms: no
// product takes less than 48 clocks; the small tables 4.2 ms).  What remains
// is latency: with one stage of A per tile at 208 columns its refill is only
// partly hidden by the other tile's products, and a tile stands still while its
// accumulators are read.  The symbol forms: 1.0 ms for 2 GiB, 6.4 of 6.55 TB/s.
//
// The place of an input in an operand word: bit j of a form word (input j of
// 32) becomes nibble j / 4 of word j % 4 of the 16-byte group.  The A side
// masks the bits where they stand (0x1 = 0.5, 0x2 = 1, 0x4 = 2, and the
// fourth moved to 0x4), the B side holds the reciprocals (2, 1, 0.5, 0.5).
#include <algorithm>

#include "bilinear.cuh"
#include "bitslice.cuh"
#include "tensor.cuh"

namespace p2g {

namespace {

constexpr int kStageWords = kTensorStage / 32;  // form words of one symbol per stage
constexpr int kStageSteps = kTensorStage / 64;  // products of K = 64 per stage
constexpr int kRingB = 4, kRingF = 3;           // shared-memory stages: B operand, forms
constexpr int kMaxRingA = 4;                    // tensor-memory stages of A per tile (1 to 4)
constexpr int kPairM = 2 * kTensorM;                    // symbols of a tile pair
constexpr int kFormBytes = kStageWords * kPairM * 4;    // one form of one stage and tile pair
constexpr int kSlotF = 4 * kFormBytes;                  // a product takes up to 4 forms
constexpr int kStageCols = kStageWords * 4;             // tensor-memory columns of a stage of A
constexpr int kThreads = 896;  // warpgroups: control, a generator and two epilogues per tile
// Tensor-memory columns 496-503: block scales of B, 1; 504-511: of A, 2^7, so
// that the sums' units are bit 7 of the accumulators' low bytes.
constexpr int kScaleB = 496, kScaleA = 504;
constexpr int kBatch = 2;       // 16-column groups of accumulators read at a time
constexpr int kSmemBars = 512;

// Byte 0 of forms[e]: the first form of product e, byte 1: the second (or the
// first again), byte 2: how many forms phi_e is the sum of.
struct ProdTab {
    uint32_t forms[kProds];
    uint32_t w[kProds];
};
constexpr ProdTab make_prod_tab()
{
    ProdTab t{};
    for (int e = 0; e < kProds; ++e) {
        t.forms[e] = kBilinear.idx[e][0] | static_cast<uint32_t>(kBilinear.idx[e][1]) << 8 |
                     static_cast<uint32_t>(kBilinear.nf[e]) << 16;
        t.w[e] = kBilinear.w[e];
    }
    return t;
}
__constant__ ProdTab c_prod = make_prod_tab();

// ---- PTX -----------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
// Waits for a barrier phase.  The loop is inside the asm block (branches that
// the compiler sees cost ten to twenty clocks each, also when not taken) and
// bounded: `left`, a thread's failing tries, serves all of its waits, so that once
// it is used up each later wait is one try.  A thread that finds it 0 skips its
// copies, products and arrivals (what it would announce may not be there).  Its
// warp then leaves its role, all lanes together, by which it says so (false).
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t phase, uint32_t &left)
{
    asm volatile("{\n.reg .pred p, q;\n"
                 "WAIT:\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 "@p bra DONE;\nsetp.ne.u32 q, %0, 0;\n@q sub.u32 %0, %0, 1;\n@q bra WAIT;\n"
                 "DONE:\n}"
                 : "+r"(left)
                 : "r"(bar), "r"(phase)
                 : "memory");
}
// Whether a phase has completed, without waiting.  Asked for some time before
// the wait, so that the answer's latency passes behind other work.
__device__ __forceinline__ uint32_t bar_test(uint32_t bar, uint32_t phase)
{
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 "selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(bar), "r"(phase)
                 : "memory");
    return done;
}
// The wait that follows a test: no more than a predicate if it was done.
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t phase, uint32_t &left, uint32_t done)
{
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %3, 0;\n@p bra DONE;\n"
                 "WAIT:\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 "@p bra DONE;\nsetp.ne.u32 q, %0, 0;\n@q sub.u32 %0, %0, 1;\n@q bra WAIT;\n"
                 "DONE:\n}"
                 : "+r"(left)
                 : "r"(bar), "r"(phase), "r"(done)
                 : "memory");
}
// Whether no lane of the warp has given up.
__device__ __forceinline__ bool all_left(uint32_t left) { return __all_sync(0xffffffffu, left != 0); }
// global -> shared copy of `bytes` (a multiple of 16, both sides aligned)
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}
// D[128 x N] += A[128 x 64] * B[N x 64]^T, A in tensor memory, 4-bit floats
__device__ __forceinline__ void tc_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t sa, uint32_t sb)
{
    asm volatile("{\n.reg .pred p;\nsetp.eq.u32 p, 0, 0;\n"
                 "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X "
                 "[%0], [%1], %2, %3, [%4], [%5], p;\n}" ::"r"(d),
                 "r"(a), "l"(b), "r"(idesc), "r"(sa), "r"(sb)
                 : "memory");
}
// K-major operand without swizzle: 8 x 16-byte core matrices of 128
// contiguous bytes, `lbo` bytes apart along K and 128 along the rows.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo)
{
    return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | static_cast<uint64_t>(lbo >> 4) << 16 |
           static_cast<uint64_t>(128 >> 4) << 32 | 1ull << 46;
}
__device__ __forceinline__ void tmem_st4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a),
                 "r"(b), "r"(c), "r"(d)
                 : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
                 "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]),
                 "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st()
{
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// Bit 7 of each 16-bit half over the whole half (the permute's sign mode).
__device__ __forceinline__ uint32_t spread_bit7(uint32_t v)
{
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, 0xAA88;" : "=r"(r) : "r"(v));
    return r;
}
// 16 columns, their low 16 bits packed in pairs
__device__ __forceinline__ void tmem_ld16_packed(uint32_t addr, uint32_t (&v)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.pack::16b.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                   "=r"(v[7])
                 : "r"(addr)
                 : "memory");
}
// The loaded registers pass through the wait, so no use moves above it.
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&v)[kBatch][8])
{
#define P2G_R8(c) "+r"(v[c][0]), "+r"(v[c][1]), "+r"(v[c][2]), "+r"(v[c][3]), "+r"(v[c][4]), "+r"(v[c][5]), \
                  "+r"(v[c][6]), "+r"(v[c][7])
    static_assert(kBatch == 2, "registers of the wait");
    asm volatile("tcgen05.wait::ld.sync.aligned;" : P2G_R8(0), P2G_R8(1)::"memory");
#undef P2G_R8
}

// ---- the operands' forms ---------------------------------------------------

template <int F>
__device__ __forceinline__ uint32_t form_word(const uint32_t *x)
{
    constexpr uint32_t m = kBilinear.form[F];
    uint32_t v = 0;
#pragma unroll
    for (int b = 0; b < 16; ++b)
        if ((m >> b) & 1u)
            v ^= x[b];
    return v;
}

// 32 x 32 bit transpose: afterwards bit i of x[j] is what bit j of x[i] was.
// The 16- and 8-bit block swaps are byte permutes.
__device__ __forceinline__ void transpose32(uint32_t (&x)[32])
{
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const uint32_t a = x[j], b = x[j + 16];
        x[j] = __byte_perm(a, b, 0x5410);
        x[j + 16] = __byte_perm(a, b, 0x7632);
    }
#pragma unroll
    for (int j0 = 0; j0 < 32; j0 += 16)
#pragma unroll
        for (int j = j0; j < j0 + 8; ++j) {
            const uint32_t a = x[j], b = x[j + 8];
            x[j] = __byte_perm(a, b, 0x6240);
            x[j + 8] = __byte_perm(a, b, 0x7351);
        }
#define P2G_SWAP(j, h, m)                                   \
    {                                                       \
        uint32_t t_ = ((x[j] >> (h)) ^ x[(j) + (h)]) & (m); \
        x[(j) + (h)] ^= t_;                                 \
        x[j] ^= t_ << (h);                                  \
    }
#pragma unroll
    for (int j0 = 0; j0 < 32; j0 += 8)
#pragma unroll
        for (int j = j0; j < j0 + 4; ++j)
            P2G_SWAP(j, 4, 0x0F0F0F0Fu);
#pragma unroll
    for (int j0 = 0; j0 < 32; j0 += 4)
#pragma unroll
        for (int j = j0; j < j0 + 2; ++j)
            P2G_SWAP(j, 2, 0x33333333u);
#pragma unroll
    for (int j0 = 0; j0 < 32; j0 += 2)
        P2G_SWAP(j0, 1, 0x55555555u);
#undef P2G_SWAP
}

template <int F>
__device__ __forceinline__ void store_forms(const uint32_t *lo, const uint32_t *hi, uint32_t *out, size_t stride)
{
    if constexpr (F < kForms) {
        *reinterpret_cast<uint2 *>(out + F * stride) = make_uint2(form_word<F>(lo), form_word<F>(hi));
        store_forms<F + 1>(lo, hi, out, stride);
    }
}

// Slices -> forms[tile pair][form][word][symbol of the pair]: one thread takes
// two neighbouring symbols (one 32-bit word) of 32 inputs, transposes the 32 x
// 32 bits and writes the 30 forms of each symbol; a CTA takes a pair's 256
// symbols of 2 words.  Bound by HBM (read 1, write 1.9 times the slices).
__device__ __forceinline__ void forms_of_pair(const uint8_t *const *__restrict__ src, int nin, size_t S,
                                              size_t byte0, uint32_t *__restrict__ forms, int pair, int word2)
{
    const int kw = word2 * 2 + (threadIdx.x >> 7), x2 = threadIdx.x & 127;
    const size_t off = byte0 + (static_cast<size_t>(pair) * kTensorM + x2) * 4;
    if (off >= S || kw * 32 >= nin)
        return;
    uint32_t x[32];
    if (off + 4 <= S) {
#pragma unroll
        for (int i = 0; i < 32; ++i)
            x[i] = kw * 32 + i < nin
                       ? __ldg(reinterpret_cast<const uint32_t *>(src[kw * 32 + i] + off))
                       : 0u;
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i)
            x[i] = kw * 32 + i < nin
                       ? __ldg(reinterpret_cast<const uint16_t *>(src[kw * 32 + i] + off))
                       : 0u;
    }
    transpose32(x);
    const int stages = (nin + kTensorStage - 1) / kTensorStage;
    const size_t plane = static_cast<size_t>(stages) * (kFormBytes / 4);
    uint32_t *out = forms + static_cast<size_t>(pair) * kForms * plane + kw * kPairM + x2 * 2;
    store_forms<0>(x, x + 16, out, plane);
}

// the problem that CTA `id` of a batched launch works for
template <class P>
__device__ __forceinline__ int problem_of(const P *probs, int np, unsigned long long id)
{
    int lo = 0, hi = np - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (probs[mid].first <= id)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(256) batch_symbol_forms(const TensorFormProb *__restrict__ probs, int np)
{
    const TensorFormProb p = probs[problem_of(probs, np, blockIdx.x)];
    const unsigned local = static_cast<unsigned>(blockIdx.x - p.first);
    const unsigned pairs = static_cast<unsigned>((p.S / 2 + kPairM - 1) / kPairM);
    forms_of_pair(p.src, p.nin, p.S, 0, p.forms, local % pairs, local / pairs);
}

// the 4-bit B operand group of 32 inputs' bits (see the head of this file)
__device__ __forceinline__ uint4 expand_b(uint32_t v)
{
    return make_uint4((v << 2) & 0x44444444u, v & 0x22222222u, (v >> 2) & 0x11111111u,
                      (v >> 3) & 0x11111111u);
}

// products of place G: the 5 values (3 products each), then the 5 residues (9)
template <int G>
__device__ __forceinline__ void store_coef(const uint32_t *x, uint4 *out, size_t stride, int g)
{
    if constexpr (G < 10) {
        if (g == G) {
            if constexpr (G < 5) {
                const uint32_t u = form_word<2 * G>(x), v = form_word<2 * G + 1>(x);
                out[(3 * G) * stride] = expand_b(u);
                out[(3 * G + 1) * stride] = expand_b(v);
                out[(3 * G + 2) * stride] = expand_b(u ^ v);
            } else {
                constexpr int F = 10 + 4 * (G - 5), E = 15 + 9 * (G - 5);
                const uint32_t a = form_word<F>(x), b = form_word<F + 1>(x);
                const uint32_t d = form_word<F + 2>(x), c = form_word<F + 3>(x);
                out[(E + 0) * stride] = expand_b(a);
                out[(E + 1) * stride] = expand_b(b);
                out[(E + 2) * stride] = expand_b(a ^ b);
                out[(E + 3) * stride] = expand_b(c);
                out[(E + 4) * stride] = expand_b(d);
                out[(E + 5) * stride] = expand_b(c ^ d);
                out[(E + 6) * stride] = expand_b(a ^ c);
                out[(E + 7) * stride] = expand_b(b ^ d);
                out[(E + 8) * stride] = expand_b(a ^ b ^ c ^ d);
            }
        } else {
            store_coef<G + 1>(x, out, stride, g);
        }
    }
}

// coef[block][e][word][row] (16 bytes: 32 inputs of one output).  A block of
// 256 threads takes 32 rows (of all output blocks' rows, padding included) of 4
// words: its threads find 16 coefficients each, 128 of them transpose 32
// coefficients' bits, and then a warp takes a word's products of one of the ten
// places at a time.  (With one thread for all of an output's coefficients and
// one place, the ten of a word found them all ten times: 32000 inputs and 1600
// outputs took 1.36 ms; now they and the forms of 64 KiB slices, 0.96 ms alone,
// take 1.31 in one launch.)
constexpr int kCoefWords = 4;
__device__ __forceinline__ void coef_block(const TensorCoefProb &p, const uint16_t *__restrict__ glog,
                                           const uint16_t *__restrict__ gexp, unsigned block)
{
    __shared__ uint32_t bits[kCoefWords][16][32];
    const int nblk = (p.nout + kTensorMaxN - 1) / kTensorMaxN, per = (p.nout + nblk - 1) / nblk;
    const int rows = (per + 15) / 16 * 16, all = rows * nblk, words = (p.nin + 63) / 64 * 2;
    const unsigned groups = (all + 31) / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ro = static_cast<int>(block % groups) * 32 + lane, kw0 = static_cast<int>(block / groups) * kCoefWords;
    const int nb = ro / rows, row = ro % rows;
    // blocks of equal size: block nb holds outputs [nb * per, ...)
    const int o = nb * per + row;
    const bool live = ro < all && row < per && o < p.nout;
    const CoefSource c = {p.coeff, p.consts, p.exps};
    {
        const int w = warp & 3, j0 = (warp >> 2) * 8, in0 = (kw0 + w) * 32;
#pragma unroll 4
        for (int j = j0; j < j0 + 8; ++j) {
            uint32_t x = 0;
            if (live && in0 + j < p.nin)
                x = coefficient(c, p.nin, in0 + j, o, glog, gexp);
            if (live && in0 + j + 16 < p.nin)
                x |= coefficient(c, p.nin, in0 + j + 16, o, glog, gexp) << 16;
            bits[w][j][lane] = x;
        }
    }
    __syncthreads();
    if (warp < kCoefWords) {
        uint32_t x[16];
#pragma unroll
        for (int j = 0; j < 16; ++j)
            x[j] = bits[warp][j][lane];
        transpose16x2(x);
#pragma unroll
        for (int j = 0; j < 16; ++j)
            bits[warp][j][lane] = x[j];
    }
    __syncthreads();
    const size_t stride = static_cast<size_t>(words) * rows;
    for (int job = warp; job < 10 * kCoefWords; job += 8) {
        const int w = job / 10, kw = kw0 + w;
        if (ro >= all || kw >= words)
            continue;
        uint32_t x[16];
#pragma unroll
        for (int j = 0; j < 16; ++j)
            x[j] = bits[w][j][lane];
        store_coef<0>(x, p.coef + (static_cast<size_t>(nb) * kProds * words + kw) * rows + row, stride, job % 10);
    }
}

__global__ void __launch_bounds__(256)
    coef_forms(const TensorCoefProb p, const uint16_t *__restrict__ glog, const uint16_t *__restrict__ gexp)
{
    coef_block(p, glog, gexp, blockIdx.x);
}

__global__ void __launch_bounds__(256)
    batch_coef_forms(const TensorCoefProb *__restrict__ probs, int np, const uint16_t *__restrict__ glog,
                     const uint16_t *__restrict__ gexp)
{
    const TensorCoefProb p = probs[problem_of(probs, np, blockIdx.x)];
    coef_block(p, glog, gexp, static_cast<unsigned>(blockIdx.x - p.first));
}

// Both operands, and the outputs that partial results are XORed into, in one
// launch: blocks for the coefficients, then the symbols (pairs x 64 inputs), then
// the outputs.
__global__ void __launch_bounds__(256)
    prepare_tensor(const TensorCoefProb p, const uint16_t *__restrict__ glog, const uint16_t *__restrict__ gexp,
                   unsigned coef_blocks, const uint8_t *const *__restrict__ src, int nin, size_t S, size_t byte0,
                   uint32_t *__restrict__ forms, unsigned pairs, unsigned form_blocks, const OutputPrep z)
{
    let_next_start();
    unsigned b = blockIdx.x;
    if (b < coef_blocks) {
        coef_block(p, glog, gexp, b);
        return;
    }
    b -= coef_blocks;
    if (b < form_blocks)
        forms_of_pair(src, nin, S, byte0, forms, b % pairs, b / pairs);
    else
        output_block(z, b - form_blocks);
}

// ---- the products ----------------------------------------------------------

// Shared-memory layout: barriers, form rings, B ring.
constexpr int oF = 2 * kRingB, oA = oF + 2 * kRingF, oD = oA + 4 * kMaxRingA;
static_assert((oD + 8) * 8 <= kSmemBars, "barrier block");
__device__ __forceinline__ constexpr uint32_t full_b(int s) { return s * 8; }
__device__ __forceinline__ constexpr uint32_t empty_b(int s) { return (kRingB + s) * 8; }
__device__ __forceinline__ constexpr uint32_t full_f(int s) { return (oF + s) * 8; }
__device__ __forceinline__ constexpr uint32_t empty_f(int s) { return (oF + kRingF + s) * 8; }
__device__ __forceinline__ constexpr uint32_t full_a(int t, int s) { return (oA + t * kMaxRingA + s) * 8; }
__device__ __forceinline__ constexpr uint32_t empty_a(int t, int s) { return (oA + (2 + t) * kMaxRingA + s) * 8; }
__device__ __forceinline__ constexpr uint32_t full_d(int t, int buf) { return (oD + 2 * t + buf) * 8; }
__device__ __forceinline__ constexpr uint32_t empty_d(int t, int buf) { return (oD + 4 + 2 * t + buf) * 8; }
constexpr uint32_t kOffF = kSmemBars, kOffB = kOffF + kRingF * kSlotF;

// What the roles of a CTA share.
struct CtaWork {
    uint32_t smem;  // shared-memory address of the dynamic block
    uint32_t tmem;
    int N, slotB, ringA, nt, pair, nb, ns;
    int dbuf;    // 1: each tile has two sets of accumulators, used in turn
    int last;    // products of K = 64 in the last stage (1 to 4)
    int e0, e1;  // products of the multiplication
};

// ---- products of tile T: one warp runs the loop (so that its addresses stay
// in uniform registers), one elected lane issues
template <int T>
__device__ __forceinline__ bool issue_products(const TensorArgs &a, const CtaWork &c)
{
    const bool one = elect_one();
    const uint32_t idesc = (1u << 7) | (1u << 10) | (static_cast<uint32_t>(c.N >> 3) << 17) | (1u << 23) |
                           (8u << 24);
    const uint32_t sa = c.tmem + kScaleA, sb = c.tmem + kScaleB;
    const uint32_t d0 = c.tmem + T * c.N;
    const uint32_t colA = c.tmem + ((2 * c.N) << c.dbuf) + T * c.ringA * kStageCols;
    const uint64_t desc0 = smem_desc(c.smem + kOffB, c.N * 16);
    const uint32_t stepB = c.slotB >> 4, step = 2 * c.N;  // in 16-byte units
    const uint32_t endA = c.ringA * 8;
    uint32_t offB = 0, offA = 0, pa = 0, pb = 0, pd = 0;
    uint64_t b = desc0;
    uint32_t left = a.tries;
    auto advance = [&] {
        b += stepB;
        offB += 8;
        const bool wrap = offB == kRingB * 8;
        offB = wrap ? 0 : offB;
        b = wrap ? desc0 : b;
        pb ^= wrap;
        offA += 8;
        const bool wrapA = offA == endA;
        offA = wrapA ? 0 : offA;
        pa ^= wrapA;
    };
    uint32_t buf = 0;  // 8 * accumulator set
    for (int e = c.e0; e < c.e1; ++e) {
        bar_wait(c.smem + empty_d(T, 0) + buf, pd, left);
        const uint32_t d = d0 + (buf >> 2) * c.N;
        for (int n = 1; n < c.ns; ++n) {
            {
                const uint32_t db = bar_test(c.smem + full_b(0) + offB, pb);
                const uint32_t da = bar_test(c.smem + full_a(T, 0) + offA, pa);
                bar_wait(c.smem + full_b(0) + offB, pb, left, db);
                bar_wait(c.smem + full_a(T, 0) + offA, pa, left, da);
            }
            tc_fence_after();
            if (one && left != 0) {
                const uint32_t col = colA + offA * (kStageCols / 8);
                tc_mma(d, col, b, idesc, sa, sb);
                tc_mma(d, col + 8, b + step, idesc, sa, sb);
                tc_mma(d, col + 16, b + 2 * step, idesc, sa, sb);
                tc_mma(d, col + 24, b + 3 * step, idesc, sa, sb);
                tc_commit(c.smem + empty_a(T, 0) + offA);
                tc_commit(c.smem + empty_b(0) + offB);
            }
            __syncwarp();
            advance();
        }
        bar_wait(c.smem + full_b(0) + offB, pb, left);
        bar_wait(c.smem + full_a(T, 0) + offA, pa, left);
        tc_fence_after();
        if (one && left != 0) {
            const uint32_t col = colA + offA * (kStageCols / 8);
#pragma unroll 1
            for (int q = 0; q < c.last; ++q)
                tc_mma(d, col + 8 * q, b + q * step, idesc, sa, sb);
            tc_commit(c.smem + empty_a(T, 0) + offA);
            tc_commit(c.smem + empty_b(0) + offB);
            tc_commit(c.smem + full_d(T, 0) + buf);
        }
        __syncwarp();
        advance();
        pd ^= buf == static_cast<uint32_t>(c.dbuf) * 8;
        buf ^= c.dbuf * 8;
    }
    return all_left(left);
}

// ---- copies of the B stages
__device__ __forceinline__ bool copy_b(const TensorArgs &a, const CtaWork &c)
{
    const bool one = elect_one();
    const uint4 *cb = a.coef + (static_cast<size_t>(c.nb) * kProds * a.cwords + a.cw0) * c.N;
    const uint32_t last_bytes = c.last * 2 * c.N * 16;
    const uint32_t ring = c.smem + kOffB;
    uint32_t off = 0, ph = 1, dst = ring;
    uint32_t left = a.tries;
    for (int e = c.e0; e < c.e1; ++e) {
        const uint4 *src = cb + static_cast<size_t>(e) * a.cwords * c.N;
        // (unrolled, the kernel's code outgrows 128 KB, and verifications that run beside
        // a batch's products take 4 % longer: 1.96 ms against 1.89)
#pragma unroll 1
        for (int n = 0; n < c.ns; ++n) {
            bar_wait(c.smem + empty_b(0) + off, ph, left);
            if (one && left != 0) {
                const uint32_t bytes = n == c.ns - 1 ? last_bytes : c.slotB;
                bar_expect(c.smem + full_b(0) + off, bytes);
                bulk_copy(dst, src, bytes, c.smem + full_b(0) + off);
            }
            __syncwarp();
            src += kStageWords * c.N;
            off += 8;
            dst += c.slotB;
            const bool wrap = off == kRingB * 8;
            off = wrap ? 0 : off;
            dst = wrap ? ring : dst;
            ph ^= wrap;
        }
    }
    return all_left(left);
}

// ---- copies of the tile pair's form words: a slot holds four stages of one
// form, two of two or one of four
__device__ __forceinline__ bool copy_forms(const TensorArgs &a, const CtaWork &c)
{
    const bool one = elect_one();
    const uint32_t plane = c.ns * kFormBytes;  // bytes of one form of one pair
    const uint8_t *ft = reinterpret_cast<const uint8_t *>(a.forms) + static_cast<size_t>(c.pair) * kForms * plane;
    uint32_t off = 0, d = c.smem + kOffF, ph = 1, left = a.tries;
    uint32_t next = c_prod.forms[c.e0];
    for (int e = c.e0; e < c.e1; ++e) {
        const uint32_t t = next;
        next = c_prod.forms[min(e + 1, kProds - 1)];
        const uint32_t nf = (t >> 16) & 0xFF, step = (4u >> (nf >> 1)) * kFormBytes;
        const uint8_t *f0 = ft + static_cast<size_t>(t & 0xFF) * plane;
        const uint8_t *f1 = ft + static_cast<size_t>((t >> 8) & 0xFF) * plane;
        for (uint32_t at = 0; at < plane; at += step) {
            const uint32_t bytes = min(step, plane - at);
            bar_wait(c.smem + empty_f(0) + off, ph, left);
            if (one && left != 0) {
                const uint32_t bar = c.smem + full_f(0) + off;
                bar_expect(bar, nf * bytes);
                bulk_copy(d, f0 + at, bytes, bar);
                if (nf >= 2)
                    bulk_copy(d + step, f1 + at, bytes, bar);
                if (nf == 4) {
                    // the four forms of a residue are neighbours
                    bulk_copy(d + 2 * step, f0 + at + 2 * static_cast<size_t>(plane), bytes, bar);
                    bulk_copy(d + 3 * step, f0 + at + 3 * static_cast<size_t>(plane), bytes, bar);
                }
            }
            __syncwarp();
            off += 8;
            d += kSlotF;
            const bool wrap = off == kRingF * 8;
            off = wrap ? 0 : off;
            d = wrap ? c.smem + kOffF : d;
            ph ^= wrap;
        }
    }
    return all_left(left);
}

// ---- the A operand of a tile: row = lane of tensor memory = symbol
struct GenState {
    uint32_t lanes, fullA, emptyA, offA, endA, pa;  // A slots
    uint32_t ring, fullF, emptyF, sf, pf;            // form slots
    uint32_t left;
    int ns;
    bool first;  // lane 0
};
// All stages of a product whose phi_e is the sum of NF forms.
template <int NF>
__device__ __forceinline__ void generate_product(GenState &g)
{
    constexpr int kPer = 4 / NF;  // stages per slot
    for (int n = 0; n < g.ns; n += kPer) {
        bar_wait(g.fullF + g.sf * 8, g.pf, g.left);
        const uint32_t F = g.ring + g.sf * kSlotF;
#pragma unroll
        for (int s = 0; s < kPer; ++s) {
            if (s == 0 || n + s < g.ns) {
                const uint32_t doneA = bar_test(g.emptyA + g.offA, g.pa);
                uint32_t w[kStageWords];
#pragma unroll
                for (int j = 0; j < kStageWords; ++j) {
                    w[j] = lds32(F + s * kFormBytes + j * kPairM * 4);
#pragma unroll
                    for (int k = 1; k < NF; ++k)
                        w[j] ^= lds32(F + (k * kPer + s) * kFormBytes + j * kPairM * 4);
                }
                uint32_t v[kStageWords / 4][16];
#pragma unroll
                for (int j = 0; j < kStageWords; ++j) {
                    uint32_t *o = v[j >> 2] + 4 * (j & 3);
                    o[0] = w[j] & 0x11111111u;
                    o[1] = w[j] & 0x22222222u;
                    o[2] = w[j] & 0x44444444u;
                    o[3] = (w[j] >> 1) & 0x44444444u;
                }
                bar_wait(g.emptyA + g.offA, g.pa, g.left, doneA);
                tc_fence_after();
                const uint32_t col = g.lanes + g.offA * (kStageCols / 8);
#pragma unroll
                for (int h = 0; h < kStageWords / 4; ++h)
                    tmem_st16(col + h * 16, v[h]);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (g.first && g.left != 0)
                    bar_arrive(g.fullA + g.offA);
                g.offA += 8;
                const bool wrapA = g.offA == g.endA;
                g.offA = wrapA ? 0 : g.offA;
                g.pa ^= wrapA;
            }
        }
        if (g.first && g.left != 0)
            bar_arrive(g.emptyF + g.sf * 8);
        const bool wrap = ++g.sf == kRingF;
        g.sf = wrap ? 0 : g.sf;
        g.pf ^= wrap;
    }
}
__device__ __forceinline__ bool generate_a(const TensorArgs &a, const CtaWork &c, int t, int warp, int lane)
{
    GenState g;
    g.lanes = c.tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + ((2 * c.N) << c.dbuf) +
              t * c.ringA * kStageCols;
    g.fullA = c.smem + full_a(t, 0);
    g.emptyA = c.smem + empty_a(t, 0);
    g.offA = 0;
    g.endA = c.ringA * 8;
    g.pa = 1;
    g.ring = c.smem + kOffF + (t * kTensorM + (warp & 3) * 32 + lane) * 4;
    g.fullF = c.smem + full_f(0);
    g.emptyF = c.smem + empty_f(0);
    g.sf = 0;
    g.pf = 0;
    g.left = a.tries;
    g.ns = c.ns;
    g.first = lane == 0;
    uint32_t next = c_prod.forms[c.e0];
    for (int e = c.e0; e < c.e1; ++e) {
        const uint32_t nf = (next >> 16) & 0xFF;
        next = c_prod.forms[min(e + 1, kProds - 1)];
        if (nf == 1)
            generate_product<1>(g);
        else if (nf == 2)
            generate_product<2>(g);
        else
            generate_product<4>(g);
        if (!all_left(g.left))
            return false;
    }
    return true;
}

// Stores (mode 0), XORs (1) or atomically XORs (2) up to four symbols at an
// 8-byte aligned address with `room` bytes of the slice left (room > 0, even).
// Nothing beyond the slice is touched: a last odd symbol is folded with a
// 16-bit compare-and-swap.
__device__ __forceinline__ void store_symbols(uint8_t *p, size_t room, uint2 v, int mode)
{
    if (room >= 8) {
        if (mode == 2) {
            atomicXor(reinterpret_cast<uint32_t *>(p), v.x);
            atomicXor(reinterpret_cast<uint32_t *>(p) + 1, v.y);
            return;
        }
        uint2 *q = reinterpret_cast<uint2 *>(p);
        if (mode == 1) {
            const uint2 o = *q;
            v.x ^= o.x;
            v.y ^= o.y;
        }
        *q = v;
        return;
    }
    for (int i = 0; i < static_cast<int>(room) / 2; ++i) {
        unsigned short *q = reinterpret_cast<unsigned short *>(p) + i;
        const unsigned short s = static_cast<unsigned short>((i < 2 ? v.x : v.y) >> (16 * (i & 1)));
        if (mode == 2) {
            unsigned short seen = *reinterpret_cast<volatile unsigned short *>(q), was;
            do {
                was = seen;
                seen = atomicCAS(q, was, static_cast<unsigned short>(was ^ s));
            } while (seen != was);
        } else {
            *q = mode == 1 ? static_cast<unsigned short>(*q ^ s) : s;
        }
    }
}

// ---- accumulators of tile t to outputs, by one of its two warpgroups: G
// groups of 16 columns from column col0 (compiled for each G, since a test per
// group costs as much as its work)
template <int G>
__device__ __forceinline__ bool read_products(const TensorArgs &a, const CtaWork &c, uint8_t *smem, int t, int half,
                                              int col0, int warp, int lane)
{
    const uint32_t d = c.tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + t * c.N + col0;
    // The accumulators start at 2^23 and count units of 2^7; they are set back
    // before their sum reaches 2^24, every `span` products.
    const int nbuf = 1 + c.dbuf;
    const int span = max(1, 65535 / (((c.ns - 1) * 4 + c.last) * 64));
    auto reset = [&](uint32_t col) {
        for (int q = 0; q < 16 * G; q += 4)
            tmem_st4(col + q, 0x4B000000u, 0x4B000000u, 0x4B000000u, 0x4B000000u);
        tmem_wait_st();
    };
    reset(d);
    if (c.dbuf)
        reset(d + 2 * c.N);
    tc_fence_before();
    __syncwarp();
    if (lane == 0) {
        bar_arrive(c.smem + empty_d(t, 0));
        if (c.dbuf)
            bar_arrive(c.smem + empty_d(t, 1));
    }
    // acc[q][j]: columns 16q + 2j (low half) and 16q + 2j + 1
    uint32_t acc[G][8];
#pragma unroll
    for (int q = 0; q < G; ++q)
#pragma unroll
        for (int j = 0; j < 8; ++j)
            acc[q][j] = 0;
    uint32_t pd = 0, left = a.tries, buf = 0;
    bool whole = true;
    int run = 1;  // products since the accumulators of this set were set, this one included
    for (int e = c.e0; e < c.e1; ++e) {
        // parities of sums over all products since then (see the head of this
        // file); a set's next product is nbuf further on
        const bool end = run == span || e + nbuf >= c.e1;
        const uint32_t w = (end ? c_prod.w[e] : c_prod.w[e] ^ c_prod.w[e + nbuf]) * 0x10001u;
        const uint32_t col = d + (buf >> 2) * c.N;
        bar_wait(c.smem + full_d(t, 0) + buf, pd, left);
        tc_fence_after();
#pragma unroll
        for (int q0 = 0; q0 < G; q0 += kBatch) {
            uint32_t v[kBatch][8];
#pragma unroll
            for (int q = 0; q < kBatch; ++q)
                if (q0 + q < G)
                    tmem_ld16_packed(col + (q0 + q) * 16, v[q]);
            tmem_wait_ld(v);
            if (q0 + kBatch >= G) {
                // all columns read
                if (end)
                    reset(col);
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    bar_arrive(c.smem + empty_d(t, 0) + buf);
            }
#pragma unroll
            for (int q = 0; q < kBatch; ++q)
                if (q0 + q < G)
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        // bit 7 of each half spread over the half
                        acc[q0 + q][j] ^= spread_bit7(v[q][j]) & w;
        }
        if (buf == static_cast<uint32_t>(c.dbuf) * 8) {
            pd ^= 1;
            run = run == span ? 1 : run + 1;
        }
        buf ^= c.dbuf * 8;
        if (!all_left(left)) {
            // stores nothing, but still meets the others below
            whole = false;
            break;
        }
    }
    // The sums go through shared memory (the form ring is idle once both tiles'
    // last products have ended: all epilogue warps meet here), [column pair][row], so that a warp writes whole
    // 256-byte rows of the outputs: a lane takes four symbols of a column pair.
    asm volatile("bar.sync 9, %0;" ::"r"(c.nt * (c.N > 16 ? 256 : 128)) : "memory");
    uint32_t *ex = reinterpret_cast<uint32_t *>(smem + kOffF + (2 * t + half) * (kRingF * kSlotF / 4));
    const int row = (warp & 3) * 32 + lane;
    const int per = (a.nout + a.nblk - 1) / a.nblk;
    const int nrows = min(per, a.nout - c.nb * per);
    const size_t off = a.byte0 + (static_cast<size_t>(2 * c.pair + t) * kTensorM + lane * 4) * 2;
    const size_t end = whole ? a.S : 0;
    const int mode = a.split > 1 ? 2 : a.mode;
    constexpr int kHalf = 4;  // column groups per exchange
    static_assert(kHalf * 8 * kTensorM * 4 <= kRingF * kSlotF / 4, "exchange fits a quarter of the form ring");
#pragma unroll
    for (int q0 = 0; q0 < G; q0 += kHalf) {
        asm volatile("bar.sync %0, 128;" ::"r"(1 + 2 * t + half) : "memory");
#pragma unroll
        for (int q = 0; q < kHalf; ++q)
            if (q0 + q < G)
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    ex[(q * 8 + j) * kTensorM + row] = acc[q0 + q][j];
        asm volatile("bar.sync %0, 128;" ::"r"(1 + 2 * t + half) : "memory");
        constexpr int kMost = kHalf * 8;
        const int pairs = G - q0 < kHalf ? (G - q0) * 8 : kMost;
#pragma unroll 1
        for (int p = warp & 3; p < pairs; p += 4) {
            const uint4 x = *reinterpret_cast<const uint4 *>(ex + p * kTensorM + lane * 4);
#pragma unroll 1
            for (int hi = 0; hi < 2; ++hi) {
                const int o = col0 + (q0 * 8 + p) * 2 + hi;
                if (o >= nrows || off >= end)
                    continue;
                const uint32_t sel = hi ? 0x7632u : 0x5410u;
                store_symbols(a.dst[c.nb * per + o] + off, a.S - off,
                              make_uint2(__byte_perm(x.x, x.y, sel), __byte_perm(x.z, x.w, sel)), mode);
            }
        }
    }
    return whole;
}

// BATCH: CTA i works on items[i] of its problem (args unused).
template <bool BATCH>
__global__ void __launch_bounds__(kThreads, 1)
    tensor_muladd(const TensorArgs args, const TensorArgs *__restrict__ probs,
                  const TensorItem *__restrict__ items, const volatile int *abort)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint32_t tmem_base;
    __shared__ int aborted;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wg = warp >> 2;
    const uint32_t bars = smem_u32(smem);

    // this CTA's tile pair, output block and products
    TensorItem it;
    if constexpr (BATCH)
        it = items[blockIdx.x];
    const TensorArgs a = BATCH ? probs[it.prob] : args;
    if constexpr (!BATCH) {
        const int pairs = (a.tiles + 1) >> 1;
        int id = blockIdx.x;
        it.nb = id % a.nblk;
        id /= a.nblk;
        it.pair = id % pairs;
        it.part = id / pairs;
    }
    CtaWork c;
    c.nb = it.nb;
    c.pair = it.pair;
    const int part = it.part;
    c.nt = min(2, a.tiles - 2 * c.pair);
    c.ns = (a.steps + kStageSteps - 1) / kStageSteps;
    c.last = a.steps - kStageSteps * (c.ns - 1);
    c.e0 = kProds * part / a.split;
    c.e1 = kProds * (part + 1) / a.split;
    c.N = a.rows;
    c.slotB = a.rows * kStageWords * 16;
    // two sets of accumulators per tile where two stages of A fit beside them
    c.dbuf = a.rows <= 80;
    c.ringA = min(kMaxRingA, (kScaleB - ((2 * a.rows) << c.dbuf)) / (2 * kStageCols));
    c.smem = bars;

    if (threadIdx.x == 0) {
        aborted = BATCH && *abort != 0;
        for (int s = 0; s < kRingB; ++s) {
            bar_init(bars + full_b(s), 1);
            bar_init(bars + empty_b(s), c.nt);
        }
        for (int s = 0; s < kRingF; ++s) {
            bar_init(bars + full_f(s), 1);
            bar_init(bars + empty_f(s), 4 * c.nt);
        }
        for (int t = 0; t < 2; ++t) {
            for (int s = 0; s < kMaxRingA; ++s) {
                bar_init(bars + full_a(t, s), 4);
                bar_init(bars + empty_a(t, s), 1);
            }
            for (int buf = 0; buf < 2; ++buf) {
                bar_init(bars + full_d(t, buf), 1);
                bar_init(bars + empty_d(t, buf), a.rows > 16 ? 8 : 4);
            }
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                         smem_u32(&tmem_base))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    c.tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    // the block scales (powers of two, biased by 127)
    if (wg == 1) {
        const uint32_t sc = c.tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        for (int q = 0; q < 8; q += 4) {
            tmem_st4(sc + kScaleB + q, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
            tmem_st4(sc + kScaleA + q, 0x86868686u, 0x86868686u, 0x86868686u, 0x86868686u);
        }
        tmem_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    if (BATCH && aborted) {
        if (warp == 2)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(c.tmem));
        return;
    }
    if constexpr (!BATCH)
        wait_for_previous();
    bool whole = true;  // this warp's role ended as it should
    // Registers: 896 threads x 72 = 64512 at launch; 128 x (56 + 2 x 64 + 4 x
    // 80) = 64512 after the split.
    if (wg == 0) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 0)
            whole = copy_b(a, c);
        else if (warp == 1)
            whole = issue_products<0>(a, c);
        else if (warp == 2)
            whole = copy_forms(a, c);
        else if (c.nt == 2)
            whole = issue_products<1>(a, c);
        __syncwarp();
    } else if (wg <= 2) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        if (wg - 1 < c.nt)
            whole = generate_a(a, c, wg - 1, warp, lane);
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 80;");
        const int t = (wg - 3) >> 1, half = (wg - 3) & 1, low = ((c.N >> 4) + 1) / 2;
        if (t < c.nt)
            switch (half ? (c.N >> 4) - low : low) {
#define P2G_GROUPS(g)                                       \
    case g:                                                 \
        whole = read_products<g>(a, c, smem, t, half, half * low * 16, warp, lane); \
        break;
                P2G_GROUPS(1) P2G_GROUPS(2) P2G_GROUPS(3) P2G_GROUPS(4) P2G_GROUPS(5) P2G_GROUPS(6)
                P2G_GROUPS(7)
#undef P2G_GROUPS
            }
    }
    if (!whole) {
        // a wait gave up: 2 ms for copies and products in flight (each takes
        // microseconds) to end before the CTA gives its memory back
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000ll) {
        }
        *static_cast<volatile int *>(a.err) = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 2)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(c.tmem));
}

size_t tensor_smem(int rows) { return kOffB + static_cast<size_t>(kRingB) * rows * kStageWords * 16; }

// clocks of one product of a CTA's two tiles (see tensor_clocks)
double product_clocks(int nin, int nout)
{
    const double N = tensor_rows(nout);
    return 700.0 + 4.0 * N + tensor_stages(nin) * std::max(470.0, 4.37 * N);
}

}  // namespace

size_t tensor_coef_bytes(int nin, int nout)
{
    return static_cast<size_t>(tensor_blocks(nout)) * tensor_rows(nout) * kProds * tensor_words(nin) * 16;
}

size_t tensor_form_bytes(int nin, size_t tiles)
{
    return (tiles + 1) / 2 * static_cast<size_t>(tensor_stages(nin)) * kForms * kFormBytes;
}

int tensor_coefs(cudaStream_t st, const CoefSource &c, const uint16_t *glog, const uint16_t *gexp,
                 int nin, int nout, void *coef)
{
    if (nin <= 0 || nout <= 0)
        return P2G_OK;
    const TensorCoefProb p{c.coeff, c.consts, c.exps, static_cast<uint4 *>(coef), nin, nout, 0};
    coef_forms<<<static_cast<unsigned>(tensor_coef_ctas(nin, nout)), 256, 0, st>>>(p, glog, gexp);
    P2G_CUDA(cudaGetLastError());
    return P2G_OK;
}

// SM clocks of a problem's two launches, and the parts of the 60 products (CTAs
// per tile pair and output block) that make them fewest.  Per product a CTA
// takes about 700 + 4 N clocks (the accumulators' read-out, which the other
// tile's products hide in part) and max(470, 4.37 N) per 256 inputs -- measured
// with 256 and 2048 inputs: 1250 and 4600 at N = 16, 2440 and 8800 at N = 208 --
// and some 9000 to start and end; folding costs a launch that zeroes the
// outputs and the atomics of 256 x N symbols.  The forms take 67 clocks per
// input and tile pair (the HBM rate).
double tensor_clocks(int sms, int nin, int nout, size_t S, int *split)
{
    const long long pairs = static_cast<long long>((S / 2 + 2 * kTensorM - 1) / (2 * kTensorM));
    const long long ctas = pairs * tensor_blocks(nout);
    const double N = tensor_rows(nout);
    const double product = product_clocks(nin, nout);
    double best = 0;
    for (int sp : {1, 2, 3, 4, 5, 6, 10, 12, 15, 20, 30}) {
        const long long waves = (ctas * sp + sms - 1) / sms;
        const double c = waves * (kProds / sp * product + 9000.0 + (sp > 1 ? 20.0 * N : 0.0)) + (sp > 1 ? 5000.0 : 0.0);
        if (sp == 1 || c < best * 0.97) {
            best = c;
            *split = sp;
        }
    }
    return best + 8000.0 + 67.0 * static_cast<double>(pairs) * nin / sms;
}

double tensor_pair_clocks(int nin, int nout)
{
    return tensor_blocks(nout) * tensor_item_clocks(nin, nout, kProds) + 67.0 * nin;
}

double tensor_item_clocks(int nin, int nout, int products)
{
    return products * product_clocks(nin, nout) + 9000.0;
}

int tensor_batch_forms(cudaStream_t st, const TensorFormProb *d, int np, unsigned long long ctas)
{
    if (!ctas)
        return P2G_OK;
    batch_symbol_forms<<<static_cast<unsigned>(ctas), 256, 0, st>>>(d, np);
    P2G_CUDA(cudaGetLastError());
    return P2G_OK;
}

int tensor_batch_coefs(cudaStream_t st, const uint16_t *glog, const uint16_t *gexp,
                       const TensorCoefProb *d, int np, unsigned long long ctas)
{
    if (!ctas)
        return P2G_OK;
    batch_coef_forms<<<static_cast<unsigned>(ctas), 256, 0, st>>>(d, np, glog, gexp);
    P2G_CUDA(cudaGetLastError());
    return P2G_OK;
}

int tensor_batch(cudaStream_t st, const TensorArgs *probs, const TensorItem *items, int nitems, int rows,
                 const volatile int *abort)
{
    if (nitems <= 0)
        return P2G_OK;
    const size_t smem = tensor_smem(rows);
    P2G_CUDA(cudaFuncSetAttribute(tensor_muladd<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem)));
    tensor_muladd<true><<<static_cast<unsigned>(nitems), kThreads, smem, st>>>(TensorArgs{}, probs, items, abort);
    P2G_CUDA(cudaGetLastError());
    return P2G_OK;
}

int tensor_prepare(cudaStream_t st, const TensorRun &r, size_t t0, size_t n, const CoefSource *todo,
                   const uint16_t *glog, const uint16_t *gexp, const OutputPrep &z)
{
    const size_t byte0 = t0 * kTensorM * 2;
    TensorCoefProb p{};
    unsigned long long coef_blocks = 0;
    if (todo) {
        p = TensorCoefProb{todo->coeff, todo->consts, todo->exps,
                           static_cast<uint4 *>(const_cast<void *>(r.coef)), r.nin_total, r.nout, 0};
        coef_blocks = tensor_coef_ctas(r.nin_total, r.nout);
    }
    const unsigned long long pairs = (n + 1) / 2, form_blocks = pairs * ((r.nin + 63) / 64),
                             grid = coef_blocks + form_blocks + z.blocks;
    if (grid > 0x7fffffffull) {
        set_error("tensor multiply-accumulate: grid too large");
        return P2G_ERANGE;
    }
    prepare_tensor<<<static_cast<unsigned>(grid), 256, 0, st>>>(
        p, glog, gexp, static_cast<unsigned>(coef_blocks), r.src, r.nin, std::min(r.S, byte0 + n * kTensorM * 2),
        byte0, static_cast<uint32_t *>(r.forms), static_cast<unsigned>(pairs), static_cast<unsigned>(form_blocks), z);
    P2G_CUDA(cudaGetLastError());
    return P2G_OK;
}

int tensor_products(cudaStream_t st, const TensorRun &r, size_t t0, size_t n)
{
    const int rows = tensor_rows(r.nout), nblk = tensor_blocks(r.nout);
    const size_t smem = tensor_smem(rows);
    P2G_CUDA(cudaFuncSetAttribute(tensor_muladd<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem)));
    TensorArgs a;
    a.forms = static_cast<const uint32_t *>(r.forms);
    a.coef = static_cast<const uint4 *>(r.coef);
    a.dst = r.dst;
    a.S = r.S;
    a.byte0 = t0 * kTensorM * 2;
    a.tiles = static_cast<int>(n);
    a.steps = (r.nin + 63) / 64;
    a.cwords = tensor_words(r.nin_total);
    a.cw0 = r.i0 / 32;
    a.rows = rows;
    a.nblk = nblk;
    a.nout = r.nout;
    a.mode = r.mode;
    a.split = std::max(1, std::min(r.split, kProds));
    a.err = r.err;
    a.tries = r.tries;
    const long long grid = static_cast<long long>((n + 1) / 2) * nblk * a.split;
    if (grid > 0x7fffffffLL) {
        set_error("tensor multiply-accumulate: grid too large");
        return P2G_ERANGE;
    }
    P2G_CUDA(launch_linked(tensor_muladd<false>, static_cast<unsigned>(grid), kThreads, smem, st, true, a, nullptr,
                           nullptr, nullptr));
    return P2G_OK;
}

}  // namespace p2g
