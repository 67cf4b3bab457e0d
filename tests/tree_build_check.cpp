/* Host check of build_tree64 (tree64_build.h): the same tree as from looking
 * at each of a node's 64 cells, in how much of the time.  Prints trees
 * compared, nodes, and the two times of one large tree in microseconds;
 * exits 1 on a difference. */
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <random>
#include <vector>

#include "tree64.cuh"
#include "tree64_build.h"

using namespace vt;

static std::vector<uint4> cell_by_cell(const std::vector<uint2>& bin, int Lo) {
    std::vector<uint4> out;
    std::vector<unsigned int> cur(1, 0u), next;
    auto child = [&](unsigned int n, int k) { return bin[n].x + __builtin_popcount(bin[n].y & ((1u << k) - 1u)); };
    for (int K = (Lo + 1) / 2 - 1; K >= 0; K--) {
        const bool top2 = (Lo & 1) && K == (Lo + 1) / 2 - 1;
        const size_t base = out.size() + cur.size();
        next.clear();
        for (unsigned int n : cur) {
            uint64_t mask = 0;
            unsigned int cells[64];
            for (int x = 0; x < 4; x++)
                for (int y = 0; y < 4; y++)
                    for (int z = 0; z < 4; z++) {
                        const int o = (x >> 1) * 4 + (y >> 1) * 2 + (z >> 1), k = (x & 1) * 4 + (y & 1) * 2 + (z & 1);
                        if (top2 ? o > 0 : !((bin[n].y >> o) & 1u)) continue;
                        const unsigned int c = top2 ? n : child(n, o);
                        if (!((bin[c].y >> k) & 1u)) continue;
                        mask |= 1ull << (x * 16 + y * 4 + z);
                        cells[x * 16 + y * 4 + z] = K > 0 ? child(c, k) : 0u;
                    }
            out.push_back(make_uint4((unsigned int)mask, (unsigned int)(mask >> 32), (unsigned int)(base + next.size()), 0));
            if (K > 0)
                for (uint64_t m = mask; m; m &= m - 1) next.push_back(cells[__builtin_ctzll(m)]);
        }
        cur.swap(next);
    }
    return out;
}

static std::vector<uint2> tree(std::mt19937& g, int Lo, double p) {
    std::vector<uint2> bin;
    size_t cur = 1;
    for (int l = 0; l < Lo; l++) {
        const size_t base = bin.size() + cur;
        size_t run = 0;
        for (size_t i = 0; i < cur; i++) {
            unsigned m = 0;
            for (int k = 0; k < 8; k++)
                if (std::uniform_real_distribution<>(0, 1)(g) < p) m |= 1u << k;
            bin.push_back(make_uint2((unsigned)(base + run), m));
            run += __builtin_popcount(m);
        }
        cur = run;
    }
    return bin;
}

int main() {
    std::mt19937 g(5);
    long long trees = 0, nodes = 0;
    for (int rep = 0; rep < 60; rep++)
        for (int Lo = 1; Lo <= 7; Lo++) {
            const std::vector<uint2> bin = tree(g, Lo, Lo > 5 ? 0.4 : rep % 4 * 0.33);
            const std::vector<uint4> a = cell_by_cell(bin, Lo), b = build_tree64(bin, Lo);
            bool same = a.size() == b.size();
            for (size_t i = 0; same && i < a.size(); i++)
                same = a[i].x == b[i].x && a[i].y == b[i].y && a[i].z == b[i].z && a[i].w == b[i].w;
            if (!same) { printf("Lo %d: %zu and %zu nodes\n", Lo, a.size(), b.size()); return 1; }
            trees++; nodes += (long long)a.size();
        }
    const std::vector<uint2> bin = tree(g, 9, 0.5);
    double best[2] = {1e30, 1e30};
    for (int rep = 0; rep < 9; rep++)
        for (int k = 0; k < 2; k++) {
            const auto t = std::chrono::steady_clock::now();
            const size_t n = (k ? build_tree64(bin, 9) : cell_by_cell(bin, 9)).size();
            const double us = std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t).count();
            if (n) best[k] = std::min(best[k], us);
        }
    printf("%lld %lld %.0f %.0f\n", trees, nodes, best[0], best[1]);
    return 0;
}
