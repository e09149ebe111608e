// prep.cuh -- what a multiply-accumulate's preparing launch does besides the
// operands: its outputs' start, in blocks of the same grid.
#pragma once
#include <algorithm>

#include <cuda_runtime.h>
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
// A preparing launch lets the next one start its CTAs once its own all run; the
// next one waits for its end (and its writes) before it reads or writes anything
// that others do.  (Neither does anything in launches that are not so linked.)
// What it hides: the launch's latency and the tensor kernel's setup of tensor
// memory, 2-5 us a call (20 x 4 KiB, 2 outputs 28.1 -> 26.0 us; 256 x 64 KiB,
// 13 outputs 70.9 -> 67.3; 777 x 150002, 61 outputs 265 -> 260).
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

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

// Launches a kernel that calls wait_for_previous; `linked`: right after its
// preparing launch.
template <class... P, class... A>
inline cudaError_t launch_linked(void (*fn)(P...), unsigned grid, int threads, size_t smem, cudaStream_t st, bool linked,
                                 A... args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = linked ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, fn, static_cast<P>(args)...);
}

}  // namespace p2g
