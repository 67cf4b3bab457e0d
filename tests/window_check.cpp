/* Host check of window_blocks (vt_search.h) on random levels: the blocks it
 * names for a window of the range array hold every word of it, and over all
 * windows of a level every block is named once, and once more where a window
 * ends in it.  Prints levels, windows, blocks named; exits 1 otherwise. */
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

#include "vt_search.h"

int main() {
    std::mt19937_64 g(3);
    long long levels = 0, windows = 0, named = 0;
    for (int rep = 0; rep < 4000; rep++) {
        const int64_t bits = 64 + (int64_t)(g() % 4000), per = 1 + (int64_t)(g() % 90), blocks = (bits + per - 1) / per;
        const double stay = std::uniform_real_distribution<>(0, 1)(g), p = std::uniform_real_distribution<>(0, 1)(g);
        std::vector<char> set(bits);
        bool on = false;
        for (int64_t i = 0; i < bits; i++) {
            if (std::uniform_real_distribution<>(0, 1)(g) > stay * stay) on = std::uniform_real_distribution<>(0, 1)(g) < p;
            set[i] = on;
        }
        std::vector<unsigned long long> block(blocks);
        std::vector<int64_t> at;                                   /* block of each word of the range array */
        unsigned long long runs = 0;
        for (int64_t i = 0; i < bits; i++) {
            if (i % per == 0) block[i / per] = runs;
            if (set[i] && (i == 0 || !set[i - 1])) { at.push_back(i / per); runs++; }
            if (set[i] && (i + 1 == bits || !set[i + 1])) at.push_back(i / per);
        }
        const unsigned long long words = at.size(), window = 2 * (1 + g() % 40);
        std::vector<int> times(blocks, 0), inside(blocks, 0);
        for (unsigned long long k0 = 0; k0 < words; k0 += window) {
            const unsigned long long k1 = std::min(words, k0 + window);
            int64_t b0, b1;
            vtsearch::window_blocks(block.data(), blocks, runs, k0, k1, &b0, &b1);
            for (unsigned long long k = k0; k < k1; k++)
                if (at[k] < b0 || at[k] >= b1) { printf("word %llu of block %lld not in [%lld, %lld)\n", k, (long long)at[k], (long long)b0, (long long)b1); return 1; }
            if (b0 < 0 || b1 > blocks) return 1;
            for (int64_t b = b0; b < b1; b++) times[b]++;
            for (int64_t b = at[k0]; b <= at[k1 - 1]; b++) inside[b]++;
            windows++; named += b1 - b0;
        }
        for (int64_t b = 0; b < blocks; b++)
            if (times[b] > std::max(inside[b], 1) + 1) { printf("block %lld named %d times, needed %d\n", (long long)b, times[b], inside[b]); return 1; }
        levels++;
    }
    printf("%lld %lld %lld\n", levels, windows, named);
    return 0;
}
