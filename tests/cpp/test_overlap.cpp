// Checks the overlap test of slice tables (overlap.hpp) against a comparison of
// every pair of ranges.
#include <stdio.h>

#include <random>

#include "../../par2-rs_b200/csrc/overlap.hpp"

using namespace p2g;

int main()
{
    std::mt19937 rng(11);
    int checked = 0, hits = 0;
    auto at = [](size_t x) { return reinterpret_cast<const uint8_t *>(uintptr_t(1000) + x); };
    for (int round = 0; round < 20000; ++round) {
        // from dense (nearly all overlap) to sparse, equal and differing lengths
        const size_t space = 4u << (rng() % 12), len = 1 + rng() % 24;
        const int n = 1 + rng() % 12;
        ByteRanges set;
        std::vector<std::pair<size_t, size_t>> all;
        std::vector<const uint8_t *> a, b;
        for (int i = 0; i < n; ++i) {
            const size_t p = rng() % space, q = round % 2 ? len : rng() % 24;
            set.add(at(p), q);
            all.push_back({p, q});
            b.push_back(at(p));
        }
        bool any = false;
        for (int i = 0; i < 8; ++i, ++checked) {
            const size_t p = rng() % space, q = round % 2 ? len : rng() % 24;
            bool want = false;
            for (const auto &x : all)
                want = want || (x.second && q && p < x.first + x.second && x.first < p + q);
            if (set.overlaps(at(p), q) != want) {
                printf("[%zu, +%zu) differs\n", p, q);
                return 1;
            }
            hits += want;
            any = any || want;
            a.push_back(at(p));
        }
        if (round % 2 && slices_overlap(a, b, len) != any) {
            printf("tables differ\n");
            return 1;
        }
    }
    printf("ok %d %d\n", checked, hits);
    return 0;
}
