/* Host check of ties_at_start (tree64_build.h) on random trees: from the
 * points it names every ray's walk (tree64.cuh) ends with WALK_TIE before
 * its first candidate ahead, from others few do.  Prints, for named and for
 * other points: points, rays, rays that tied; exits 1 where a ray from a
 * named point did not. */
#include <cstdio>
#include <random>
#include <vector>

#include "tree64.cuh"
#include "tree64_build.h"

using namespace vt;

int main() {
    std::mt19937 g(99);
    auto U = [&](double a, double b) { return (float)std::uniform_real_distribution<>(a, b)(g); };
    long long named[3] = {0, 0, 0}, other[3] = {0, 0, 0};
    for (int Lo = 1; Lo <= 6; Lo++) {
        for (int rep = 0; rep < 60; rep++) {
            const int nLevels = Lo + rep % 4;
            const double p = rep % 2 ? 1.0 : 0.5;
            /* nodes level by level, as the flattened octree has them */
            std::vector<uint2> bin;
            std::vector<std::vector<char> > has(Lo + 1);
            std::vector<int> xyz = {0, 0, 0}, next;
            has[0].assign(1, 1);
            for (int l = 0; l < Lo; l++) {
                const size_t cur = xyz.size() / 3, base = bin.size() + cur;
                const int e = 1 << (l + 1);
                has[l + 1].assign((size_t)e * e * e, 0);
                next.clear();
                for (size_t i = 0; i < cur; i++) {
                    uint2 n;
                    n.x = (unsigned)(base + next.size() / 3); n.y = 0;
                    for (int k = 0; k < 8; k++) {
                        if (std::uniform_real_distribution<>(0, 1)(g) >= p) continue;
                        n.y |= 1u << k;
                        const int c[3] = {2 * xyz[3 * i] + ((k >> 2) & 1), 2 * xyz[3 * i + 1] + ((k >> 1) & 1), 2 * xyz[3 * i + 2] + (k & 1)};
                        has[l + 1][((size_t)c[0] * e + c[1]) * e + c[2]] = 1;
                        next.insert(next.end(), c, c + 3);
                    }
                    bin.push_back(n);
                }
                xyz.swap(next);
            }
            const std::vector<uint4> t64 = build_tree64(bin, Lo);
            const Tree64 T = {t64.data(), nLevels, Lo};
            const float N = (float)(1 << nLevels);
            auto set = [&](int l, int x, int y, int z) { return has[l][((((size_t)x << l) + y) << l) + z] != 0; };
            for (int i = 0; i < 40; i++) {
                float3 o = f3(U(0, N), U(0, N), U(0, N));
                const int s = (int)(g() % (unsigned)(nLevels + 1)), axes = (int)(g() % 4);   /* planes on some axes */
                float* c[3] = {&o.x, &o.y, &o.z};
                for (int a = 0; a < axes; a++) *c[(a + i) % 3] = (float)((int)*c[(a + i) % 3] >> s << s);
                const bool name = ties_at_start(o, nLevels, Lo, set);
                long long* n = name ? named : other;
                n[0]++;
                for (int q = 0; q < 20; q++) {
                    const float3 d = normalize(f3(U(-1, 1), U(-1, 1), U(-1, 1)));
                    RayInv r;
                    r.o = o; r.dx = 1 / d.x; r.dy = 1 / d.y; r.dz = 1 / d.z;
                    Walk w;
                    PathNode path[VT_TREE64_LEVELS];
                    int res = walk_root<1>(T, r, w, path);
                    bool fresh = true, ahead = false;
                    while (res == WALK_CANDIDATE) {
                        float tf = 0.0f;
                        int budget = 1 << 20;
                        unsigned entered = 0;
                        res = walk_next<1>(T, r, w, path, fresh, budget, &tf, &entered);
                        fresh = false;
                        ahead = ahead || (res == WALK_CANDIDATE && tf > 0.0f);
                        if (ahead) break;
                    }
                    /* a point on the volume's faces has no cell on the far side; rays leaving it there end */
                    const bool tied = res == WALK_TIE;
                    n[1]++; n[2] += tied;
                    if (name && !tied && o.x > 0 && o.y > 0 && o.z > 0 && o.x < N && o.y < N && o.z < N && p == 1.0) {
                        printf("Lo %d nLevels %d o %g %g %g: a ray walks on\n", Lo, nLevels, o.x, o.y, o.z);
                        return 1;
                    }
                }
            }
        }
    }
    printf("named %lld %lld %lld\nother %lld %lld %lld\n", named[0], named[1], named[2], other[0], other[1], other[2]);
    return 0;
}
