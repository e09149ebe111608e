// prep.cuh -- what a multiply-accumulate's preparing launch does besides the
// operands: its outputs' start, in blocks of the same grid.
#pragma once
#include <algorithm>

#include <stddef.h>
#include <stdint.h>

namespace p2g {

// Coefficient (i, o) is coeff[o][i], or consts[i]^exps[o] when coeff is null.
struct CoefSource {
    const uint16_t *coeff = nullptr, *consts = nullptr;
    const uint32_t *exps = nullptr;
};

// The outputs: zeroed where partial results are XORed in; and, if *status is
// set by the time the launch runs, put aside -- the device array of their
// addresses gets the addresses `alt` instead, so that nothing is written to them.
struct OutputPrep {
    uint8_t **dst = nullptr;
    size_t S = 0;
    int n = 0, per = 0;                   // outputs; zeroing blocks of each
    unsigned zero_blocks = 0, blocks = 0;  // of 256 threads
    const int *status = nullptr;
    uint8_t *const *alt = nullptr;
};
inline OutputPrep output_prep(uint8_t *const *dst, int n, size_t S, bool zero, const int *status = nullptr,
                              uint8_t *const *alt = nullptr)
{
    OutputPrep z;
    z.dst = const_cast<uint8_t **>(dst);
    z.S = S;
    z.n = n;
    z.per = static_cast<int>(std::min<size_t>((S + 4095) / 4096, 1024));
    z.zero_blocks = zero ? static_cast<unsigned>(z.per) * static_cast<unsigned>(n) : 0;
    z.blocks = z.zero_blocks + (status ? 1 : 0);
    z.status = status;
    z.alt = alt;
    return z;
}

#ifdef __CUDACC__
// Block b of the z.blocks (256 threads each).
__device__ __forceinline__ void output_block(const OutputPrep &z, unsigned b)
{
    const bool aside = z.status && *z.status != 0;
    if (b >= z.zero_blocks) {
        for (int i = threadIdx.x; aside && i < z.n; i += 256)
            z.dst[i] = z.alt[i];
        return;
    }
    if (aside)
        return;
    uint8_t *d = z.dst[b / z.per];
    for (size_t x = (static_cast<size_t>(b % z.per) * 256 + threadIdx.x) * 16; x < z.S;
         x += static_cast<size_t>(z.per) * 4096) {
        if (x + 16 <= z.S)
            *reinterpret_cast<uint4 *>(d + x) = make_uint4(0, 0, 0, 0);
        else
            for (size_t y = x; y < z.S; y += 2)
                *reinterpret_cast<uint16_t *>(d + y) = 0;
    }
}

// c_i^e by the log / antilog tables: (log c * e) mod 65535 (galois/core.rs:242-258)
__device__ __forceinline__ uint32_t coefficient(const CoefSource &c, int nin, int i, int o,
                                                const uint16_t *__restrict__ glog,
                                                const uint16_t *__restrict__ gexp)
{
    if (c.coeff)
        return c.coeff[static_cast<size_t>(o) * nin + i];
    const uint32_t base = c.consts[i], e = c.exps[o];
    if (e == 0)
        return 1;
    if (base == 0)
        return 0;
    return gexp[static_cast<uint32_t>((static_cast<uint64_t>(glog[base]) * e) % 65535u)];
}
#endif

}  // namespace p2g
