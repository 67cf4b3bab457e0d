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

/* Whether every ray from `o` ends its walk at once (WALK_TIE): from the top
 * node down, the walk looks at the cells that touch t = 0, and where o lies
 * on planes of two axes or more of a node's cells, the products of these
 * planes coincide at 0.  A cell without anything in it is left without a
 * look inside, so such planes below it do not count.  set(level, x, y, z):
 * whether the binary octree has that node. */
template <class Set>
inline bool ties_at_start(float3 o, int nLevels, int Lo, Set set) {
    const float N = (float)(1 << nLevels), p[3] = {o.x, o.y, o.z};
    for (int a = 0; a < 3; a++)
        if (!(p[a] >= 0.0f && p[a] <= N)) return false;
    for (int k = (Lo + 1) / 2 - 1; k >= 0; k--) {
        const int sh = nLevels - Lo + 2 * k, cells = 1 << (nLevels - sh);
        int lo[3], hi[3], planes = 0;
        for (int a = 0; a < 3; a++) {
            hi[a] = (int)p[a] >> sh;
            const bool on = p[a] == (float)(hi[a] << sh);
            planes += on;
            lo[a] = on && hi[a] > 0 ? hi[a] - 1 : hi[a];
            if (hi[a] >= cells) hi[a] = cells - 1;
        }
        if (planes >= 2) return true;
        bool any = false;
        for (int x = lo[0]; x <= hi[0]; x++)
            for (int y = lo[1]; y <= hi[1]; y++)
                for (int z = lo[2]; z <= hi[2]; z++) any = any || set(nLevels - sh, x, y, z);
        if (!any) return false;
    }
    return false;
}

}  // namespace vt
