/* Host check of the search by rank (vt_search.h, has_children_rank) against
 * the builder's search over ranges, on random levels: every father whose
 * children hold a set code.  Prints fathers checked and found; exits 1 on a
 * difference. */
#include <cstdio>
#include <random>
#include <vector>

#include "vt_search.h"

int main() {
    std::mt19937_64 g(7);
    long long fathers = 0, found = 0, missed = 0;
    for (int rep = 0; rep < 3000; rep++) {
        const int l = 1 + rep % 4;
        const uint64_t n = 1ull << (3 * l), base = n;
        std::vector<char> set(n);
        const double p = std::uniform_real_distribution<>(0, 1)(g), stay = std::uniform_real_distribution<>(0, 1)(g);
        bool on = false;
        for (uint64_t i = 0; i < n; i++) {
            if (std::uniform_real_distribution<>(0, 1)(g) > stay) on = std::uniform_real_distribution<>(0, 1)(g) < p * p;
            set[i] = on;
        }
        std::vector<uint64_t> e;
        std::vector<int64_t> rank(n);
        std::vector<char> start(n);
        for (uint64_t i = 0; i < n; i++) {
            start[i] = set[i] && (i == 0 || !set[i - 1]);
            rank[i] = (i ? rank[i - 1] : 0) + start[i];
            if (start[i]) e.push_back(base + i);
            if (set[i] && (i + 1 == n || !set[i + 1])) e.push_back(base + i);
        }
        for (uint64_t f = 0; f < n / 8; f++) {
            unsigned byte = 0, st = 0;
            for (int k = 0; k < 8; k++) { byte |= (unsigned)set[8 * f + k] << k; st |= (unsigned)start[8 * f + k] << k; }
            if (!byte) continue;
            const bool want = vtsearch::search_children_host(e.data(), (int64_t)e.size(), (base >> 3) + f) > 0;
            const bool got = vtsearch::has_children_rank((int64_t)e.size(), byte, st, f ? rank[8 * f - 1] : 0);
            fathers++; found += want; missed += !want;
            if (want != got) { printf("level %d father %llu: %d, by rank %d\n", l, (unsigned long long)f, want, got); return 1; }
        }
    }
    printf("%lld %lld %lld\n", fathers, found, missed);
    return 0;
}
