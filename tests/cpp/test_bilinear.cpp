// Checks the 60-product form of GF(2^16) multiplication (bilinear.cuh)
// against shift-and-add multiplication, on every pair of basis elements and
// on random elements.
#include <stdio.h>

#include <random>

#include "../../par2-rs_b200/csrc/bilinear.cuh"

using namespace p2g;

static uint32_t by_products(uint32_t a, uint32_t b)
{
    uint32_t r = 0;
    for (int e = 0; e < kProds; ++e) {
        int fa = 0, fb = 0;
        for (int k = 0; k < kBilinear.nf[e]; ++k) {
            fa ^= bl_parity(kBilinear.form[kBilinear.idx[e][k]] & a);
            fb ^= bl_parity(kBilinear.form[kBilinear.idx[e][k]] & b);
        }
        if (fa & fb)
            r ^= kBilinear.w[e];
    }
    return r;
}

int main()
{
    int checked = 0;
    for (int i = 0; i < 16; ++i)
        for (int j = 0; j < 16; ++j, ++checked)
            if (by_products(1u << i, 1u << j) != bl_mul(1u << i, 1u << j)) {
                printf("basis pair %d %d differs\n", i, j);
                return 1;
            }
    std::mt19937 rng(7);
    for (int k = 0; k < 20000; ++k, ++checked) {
        const uint32_t a = rng() & 0xFFFF, b = k < 8 ? k : rng() & 0xFFFF;
        if (by_products(a, b) != bl_mul(a, b)) {
            printf("%u * %u differs\n", a, b);
            return 1;
        }
    }
    printf("ok %d\n", checked);
    return 0;
}
