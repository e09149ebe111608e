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

// Zeroes nout outputs of S bytes (for partial results that are XORed in).
struct ZeroOutputs {
    uint8_t *const *dst = nullptr;
    size_t S = 0;
    int per = 0;  // blocks of 256 threads per output
    unsigned blocks = 0;
};
inline ZeroOutputs zero_blocks(uint8_t *const *dst, int nout, size_t S)
{
    ZeroOutputs z;
    z.dst = dst;
    z.S = S;
    z.per = static_cast<int>(std::min<size_t>((S + 4095) / 4096, 1024));
    z.blocks = static_cast<unsigned>(z.per) * static_cast<unsigned>(nout);
    return z;
}

#ifdef __CUDACC__
// Block b of the z.blocks (256 threads each).
__device__ __forceinline__ void zero_block(const ZeroOutputs &z, unsigned b)
{
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
