// bilinear.cuh -- multiplication in GF(2^16) as 60 products of single bits.
//
// A product a * b of two field elements is bilinear over GF(2), so it can be
// written a * b = XOR_e  phi_e(a) & phi_e(b)  ? w_e : 0 with linear forms
// phi_e (each the parity of some of the element's bits) and constants w_e.
// The obvious choice (every bit of a with every bit of b) takes 256 terms.
// Here it takes 60: over a matrix product sum_i c_oi * s_ix the forms of the
// coefficients and of the symbols are taken once, the 60 matrix products over
// GF(2) run on the tensor cores, and w_e is applied to their results.
//
// Construction.  GF(2^16) = GF(4)[y] / (p(y)) with deg p = 8: an element is a
// polynomial of 8 coefficients in GF(4), the product of two has 15.  By the
// Chinese remainder theorem (evaluation and interpolation, Toom-Cook's
// method with places of degree 1 and 2) those 15 follow from the values at
// the 5 places of degree 1 of the line over GF(4) -- 0, 1, omega, omega^2 and
// infinity -- and the residues modulo 5 of its 6 irreducible monic quadratics:
// 5 + 5 * 2 = 15.  A value takes one product in GF(4), a residue three
// (Karatsuba: low, high, low + high); a product in GF(4) takes three products
// of bits (the same way): (5 + 5 * 3) * 3 = 60.  All forms are sums of the 30
// bits of the 5 values and 5 residues, "the forms" below.
//
// The element theta that stands for y is free; it was searched for the least
// number of bits in the 30 forms (185 of 480).
#pragma once
#include <stdint.h>

namespace p2g {

constexpr int kForms = 30;  // linear forms stored per symbol
constexpr int kProds = 60;  // products of bits per multiplication

struct Bilinear {
    uint16_t form[kForms];   // form f is the parity of (form[f] & element)
    uint32_t sum[kProds];    // product e's phi_e is the sum of the forms in sum[e]
    uint8_t nf[kProds];      // how many forms that is: 1, 2 or 4
    uint8_t idx[kProds][4];  // ... and which
    uint16_t w[kProds];      // what product e adds to the result
    bool ok;                 // theta generates the field and the w exist
};

constexpr uint32_t bl_mul(uint32_t a, uint32_t b)
{
    uint32_t r = 0;
    for (; b; b >>= 1) {
        if (b & 1)
            r ^= a;
        a <<= 1;
        if (a & 0x10000u)
            a ^= 0x1100Bu;
    }
    return r;
}

constexpr int bl_parity(uint32_t v)
{
    int p = 0;
    for (; v; v &= v - 1)
        p ^= 1;
    return p;
}

// GF(4): bit 0 + bit 1 * omega, omega^2 = omega + 1
constexpr uint32_t bl_mul4(uint32_t a, uint32_t b)
{
    const uint32_t l = a & b & 1, h = (a >> 1) & (b >> 1);
    const uint32_t m = ((a & 1) & (b >> 1)) ^ ((a >> 1) & (b & 1));
    return (l ^ h) | ((m ^ h) << 1);
}

constexpr Bilinear make_bilinear()
{
    Bilinear B{};
    constexpr uint32_t theta = 10590;
    uint32_t omega = 1;  // 2^21845, of order 3
    for (int bit = 14; bit >= 0; --bit) {
        omega = bl_mul(omega, omega);
        if ((21845 >> bit) & 1)
            omega = bl_mul(omega, 2);
    }
    // element -> the bits of its 8 coefficients in GF(4): invert the basis
    // theta^j, omega theta^j (row r: bit r of each basis element)
    uint32_t M[16] = {};
    uint32_t t = 1;
    for (int j = 0; j < 8; ++j) {
        const uint32_t col[2] = {t, bl_mul(omega, t)};
        for (int h = 0; h < 2; ++h)
            for (int r = 0; r < 16; ++r)
                M[r] |= ((col[h] >> r) & 1u) << (2 * j + h);
        t = bl_mul(t, theta);
    }
    for (int r = 0; r < 16; ++r)
        M[r] |= 1u << (16 + r);
    B.ok = true;
    for (int c = 0; c < 16; ++c) {
        int p = c;
        while (p < 16 && !((M[p] >> c) & 1u))
            ++p;
        if (p == 16) {
            B.ok = false;
            return B;
        }
        const uint32_t x = M[p];
        M[p] = M[c];
        M[c] = x;
        for (int r = 0; r < 16; ++r)
            if (r != c && ((M[r] >> c) & 1u))
                M[r] ^= M[c];
    }
    // adds m * (coefficient j) to the pair of masks (v0, v1)
    auto add = [&M](uint32_t v[2], int j, uint32_t m) {
        const uint32_t s0 = M[2 * j] >> 16, s1 = M[2 * j + 1] >> 16;
        if (m & 1) {
            v[0] ^= s0;
            v[1] ^= s1;
        }
        if (m & 2) {
            v[0] ^= s1;
            v[1] ^= s0 ^ s1;
        }
    };
    int nform = 0, ne = 0;
    // the values at 0, 1, omega, omega^2 and infinity
    for (uint32_t a = 0; a < 5; ++a) {
        uint32_t v[2] = {0, 0};
        if (a == 4) {
            add(v, 7, 1);
        } else {
            uint32_t pw = 1;
            for (int j = 0; j < 8; ++j) {
                add(v, j, pw);
                pw = bl_mul4(pw, a);
            }
        }
        B.form[nform] = static_cast<uint16_t>(v[0]);
        B.form[nform + 1] = static_cast<uint16_t>(v[1]);
        const uint32_t u = 1u << nform;
        B.sum[ne++] = u;
        B.sum[ne++] = u << 1;
        B.sum[ne++] = u * 3;
        nform += 2;
    }
    // the residues modulo y^2 + p y + q, for 5 of the 6 irreducible ones
    // (the omitted one has the heaviest forms)
    int nq = 0;
    for (uint32_t p = 0; p < 4; ++p)
        for (uint32_t q = 0; q < 4; ++q) {
            bool root = false;
            for (uint32_t x = 0; x < 4; ++x)
                root = root || (bl_mul4(x, x) ^ bl_mul4(p, x) ^ q) == 0;
            if (root || nq++ == 3)
                continue;
            uint32_t lo[2] = {0, 0}, hi[2] = {0, 0};
            uint32_t A = 1, H = 0;  // y^j = A + H y
            for (int j = 0; j < 8; ++j) {
                add(lo, j, A);
                add(hi, j, H);
                const uint32_t nA = bl_mul4(H, q), nH = A ^ bl_mul4(H, p);
                A = nA;
                H = nH;
            }
            B.form[nform] = static_cast<uint16_t>(lo[0]);
            B.form[nform + 1] = static_cast<uint16_t>(lo[1]);
            B.form[nform + 2] = static_cast<uint16_t>(hi[1]);
            B.form[nform + 3] = static_cast<uint16_t>(hi[0]);
            // low, high, low + high; each as bit 0, bit 1, bit 0 + bit 1 (the
            // order of the forms makes all but one of the pairs neighbours)
            const uint32_t u = 1u << nform;
            const uint32_t s[9] = {u * 1, u * 2, u * 3, u * 8, u * 4, u * 12, u * 9, u * 6, u * 15};
            for (int k = 0; k < 9; ++k)
                B.sum[ne++] = s[k];
            nform += 4;
        }
    uint32_t phi[kProds] = {};  // product e's form as a mask of element bits
    for (int e = 0; e < kProds; ++e) {
        for (int f = 0; f < kForms; ++f)
            if ((B.sum[e] >> f) & 1u) {
                B.idx[e][B.nf[e]++] = static_cast<uint8_t>(f);
                phi[e] ^= B.form[f];
            }
        for (int k = B.nf[e]; k < 4; ++k)
            B.idx[e][k] = B.idx[e][0];
    }
    // the w: x^(i + j) = XOR of w_e over the e with both phi_e(x^i) and
    // phi_e(x^j) set, for all i <= j (136 equations, rank 60)
    uint64_t row[136] = {};
    uint32_t rhs[136] = {};
    int n = 0;
    for (int i = 0; i < 16; ++i)
        for (int j = i; j < 16; ++j) {
            for (int e = 0; e < kProds; ++e)
                if (((phi[e] >> i) & 1u) && ((phi[e] >> j) & 1u))
                    row[n] |= 1ull << e;
            rhs[n++] = bl_mul(1u << i, 1u << j);
        }
    int rank = 0;
    int lead[kProds] = {};
    for (int e = 0; e < kProds; ++e) {
        int p = rank;
        while (p < n && !((row[p] >> e) & 1ull))
            ++p;
        if (p == n) {
            lead[e] = -1;  // free: w_e = 0
            continue;
        }
        const uint64_t x = row[p];
        row[p] = row[rank];
        row[rank] = x;
        const uint32_t y = rhs[p];
        rhs[p] = rhs[rank];
        rhs[rank] = y;
        for (int r = 0; r < n; ++r)
            if (r != rank && ((row[r] >> e) & 1ull)) {
                row[r] ^= row[rank];
                rhs[r] ^= rhs[rank];
            }
        lead[e] = rank++;
    }
    for (int r = rank; r < n; ++r)
        if (rhs[r])
            B.ok = false;
    for (int e = 0; e < kProds; ++e)
        B.w[e] = lead[e] < 0 ? 0 : static_cast<uint16_t>(rhs[lead[e]]);
    return B;
}

constexpr Bilinear kBilinear = make_bilinear();
static_assert(kBilinear.ok, "the 60 products reproduce GF(2^16)");

}  // namespace p2g
