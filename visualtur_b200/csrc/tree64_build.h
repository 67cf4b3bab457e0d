/*
 * tree64_build.h -- the 64-ary candidate tree (tree64.cuh) from the
 * flattened binary octree (host).
 */
#pragma once
#include <stdint.h>

#include <vector>

#include <cuda_runtime.h>

namespace vt {

/* Two levels of the flattened binary nodes per 64-ary node (tree64.cuh).
 * `bin` holds a node's first child index and mask, level after level; with
 * an odd Lo the top 64-ary node has the root as its only octant. */
inline std::vector<uint4> build_tree64(const std::vector<uint2>& bin, int Lo) {
    std::vector<uint4> out;
    std::vector<unsigned int> cur(1, 0u), next;
    auto child = [&](unsigned int n, int k) { return bin[n].x + __builtin_popcount(bin[n].y & ((1u << k) - 1u)); };
    for (int K = (Lo + 1) / 2 - 1; K >= 0; K--) {
        const bool top2 = (Lo & 1) && K == (Lo + 1) / 2 - 1;
        const size_t base = out.size() + cur.size();
        next.clear();
        for (unsigned int n : cur) {
            uint64_t mask = 0;
            unsigned int cells[64];   /* binary index of the set cells, where they have children */
            for (int o = 0; o < (top2 ? 1 : 8); o++) {
                if (!top2 && !((bin[n].y >> o) & 1u)) continue;
                const unsigned int c = top2 ? n : child(n, o);
                for (int k = 0; k < 8; k++) {
                    if (!((bin[c].y >> k) & 1u)) continue;
                    const int x = ((o >> 2) & 1) * 2 + ((k >> 2) & 1), y = ((o >> 1) & 1) * 2 + ((k >> 1) & 1),
                              z = (o & 1) * 2 + (k & 1), bit = x * 16 + y * 4 + z;
                    mask |= 1ull << bit;
                    cells[bit] = K > 0 ? child(c, k) : 0u;
                }
            }
            uint4 r;
            r.x = (unsigned int)mask; r.y = (unsigned int)(mask >> 32);
            r.z = (unsigned int)(base + next.size()); r.w = 0;
            out.push_back(r);
            if (K > 0)
                for (uint64_t m = mask; m; m &= m - 1) next.push_back(cells[__builtin_ctzll(m)]);
        }
        cur.swap(next);
    }
    return out;
}

}  // namespace vt
