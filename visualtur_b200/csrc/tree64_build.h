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
 * an odd Lo the top 64-ary node has the root as its only octant.  Part of
 * opening a renderer: a node's mask is put together from its octants' eight
 * bits at a time, and only set cells are visited (80 000 binary nodes
 * on one core: 4.4 ms looking at each of the 64 cells, 0.56 ms so; the large
 * levels also go to several cores). */
inline std::vector<uint4> build_tree64(const std::vector<uint2>& bin, int Lo) {
    std::vector<uint4> out;
    std::vector<unsigned int> cur(1, 0u), next;
    for (int K = (Lo + 1) / 2 - 1; K >= 0; K--) {
        const unsigned int octants = (Lo & 1) && K == (Lo + 1) / 2 - 1 ? 1u : 0u;   /* the root alone */
        const long long n = (long long)cur.size();
        const size_t at = out.size();
        out.resize(at + cur.size());
        uint4* const rec = out.data() + at;
        const unsigned int* const from = cur.data();
        /* binary node of octant o of node i */
        auto octant = [&](long long i, int o) {
            const uint2 b = bin[from[i]];
            return octants ? from[i] : b.x + (unsigned int)__builtin_popcount(b.y & ((1u << o) - 1u));
        };
#pragma omp parallel for schedule(static) if (n > 4096)
        for (long long i = 0; i < n; i++) {
            uint64_t mask = 0;
            for (unsigned int m = octants ? octants : bin[from[i]].y & 255u; m; m &= m - 1) {
                const int o = __builtin_ctz(m);
                const uint64_t c = bin[octant(i, o)].y & 255u;
                mask |= ((c & 3) | (c & 0xC) << 2 | (c & 0x30) << 12 | (c & 0xC0) << 14)
                        << ((o & 4) * 8 + (o & 2) * 4 + (o & 1) * 2);
            }
            rec[i].x = (unsigned int)mask; rec[i].y = (unsigned int)(mask >> 32); rec[i].z = rec[i].w = 0;
        }
        size_t children = 0;
        for (long long i = 0; i < n; i++) {
            rec[i].z = (unsigned int)(out.size() + children);
            if (K > 0) children += (size_t)__builtin_popcount(rec[i].x) + (size_t)__builtin_popcount(rec[i].y);
        }
        if (K == 0) break;
        next.resize(children);
        unsigned int* const to = next.data();
        const size_t base = out.size();
#pragma omp parallel for schedule(static) if (n > 4096)
        for (long long i = 0; i < n; i++) {
            unsigned int* t = to + (rec[i].z - base);
            for (uint64_t m = (uint64_t)rec[i].y << 32 | rec[i].x; m; m &= m - 1) {
                const int bit = __builtin_ctzll(m), x = bit >> 4, y = (bit >> 2) & 3, z = bit & 3;
                const uint2 c = bin[octant(i, (x & 2) * 2 + (y & 2) + (z >> 1))];
                const int k = (x & 1) * 4 + (y & 1) * 2 + (z & 1);
                *t++ = c.x + (unsigned int)__builtin_popcount(c.y & ((1u << k) - 1u));
            }
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
