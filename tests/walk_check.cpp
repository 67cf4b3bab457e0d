/* Host check of the 64-ary walk (tree64.cuh) against the depth-first search
 * of the reference (8 slab tests per node, siblings sorted by (tnear, tfar),
 * src/Octree.cu:375-532, 620-760) on random trees.  Prints one line per ray
 * family: rays, candidates, rays the walk handed back; exits 1 on a
 * difference. */
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <random>
#include <vector>

#include "tree64.cuh"
#include "tree64_build.h"

using namespace vt;

struct Cand { int x, y, z; float tn, tf; };

struct Tree {
    int Lo, nLevels;
    std::vector<uint2> bin;
    std::vector<uint4> t64;
};

static Tree make_tree(std::mt19937& g, int Lo, int nLevels, double p) {
    Tree t;
    t.Lo = Lo; t.nLevels = nLevels;
    size_t cur = 1;
    for (int l = 0; l < Lo; l++) {
        const size_t base = t.bin.size() + cur;
        size_t run = 0;
        for (size_t i = 0; i < cur; i++) {
            unsigned m = 0;
            for (int k = 0; k < 8; k++)
                if (std::uniform_real_distribution<>(0, 1)(g) < p) m |= 1u << k;
            uint2 n;
            n.x = (unsigned)(base + run); n.y = m;
            t.bin.push_back(n);
            run += __builtin_popcount(m);
        }
        cur = run;
    }
    t.t64 = build_tree64(t.bin, Lo);
    return t;
}

static void literal(const Tree& t, const RayInv& r, unsigned node, int level, int x, int y, int z,
                    std::vector<Cand>& out) {
    struct C { int x, y, z; unsigned idx; float tn, tf; } c[8];
    int n = 0;
    const uint2 nd = t.bin[node];
    const int e = 1 << (t.nLevels - level - 1);
    for (int k = 0; k < 8; k++) {
        if (!((nd.y >> k) & 1)) continue;
        C q;
        q.x = 2 * x + ((k >> 2) & 1); q.y = 2 * y + ((k >> 1) & 1); q.z = 2 * z + (k & 1);
        q.idx = nd.x + __builtin_popcount(nd.y & ((1u << k) - 1));
        if (slab(r, q.x * e, q.y * e, q.z * e, (q.x + 1) * e, (q.y + 1) * e, (q.z + 1) * e, &q.tn, &q.tf) && q.tf >= 0.0f)
            c[n++] = q;
    }
    for (int i = n; i > 1; i--)
        for (int q = 1; q < i; q++)
            if (c[q - 1].tn > c[q].tn || (c[q - 1].tn == c[q].tn && c[q - 1].tf > c[q].tf)) std::swap(c[q - 1], c[q]);
    for (int i = 0; i < n; i++) {
        if (level + 1 == t.Lo) out.push_back({c[i].x, c[i].y, c[i].z, c[i].tn, c[i].tf});
        else literal(t, r, c[i].idx, level + 1, c[i].x, c[i].y, c[i].z, out);
    }
}

/* walk with small budgets and, now and then, a resume from the candidate's
 * coordinates alone; returns the last result */
static int walk(const Tree& t, const RayInv& r, std::mt19937& g, std::vector<Cand>& out) {
    Tree64 T = {t.t64.data(), t.nLevels, t.Lo};
    Walk w;
    PathNode path[VT_TREE64_LEVELS];
    int s = walk_root<1>(T, r, w, path);
    if (s != WALK_CANDIDATE) return s;
    bool fresh = true;
    for (;;) {
        float tf;
        unsigned entered = 0;
        int budget = (int)(g() % 5);
        s = walk_next<1>(T, r, w, path, fresh, budget, &tf, &entered);
        fresh = true;
        if (s == WALK_MORE) continue;
        if (s != WALK_CANDIDATE) return s;
        int x, y, z;
        walk_cell(T, r, w, x, y, z);
        const Cand c = {x, y, z, w.tc < 0.0f ? 0.0f : w.tc, tf};
        if (g() % 4 == 0) {
            Walk v;
            walk_at<1>(T, r, x, y, z, v, path);
            if (v.tc != w.tc || v.tx != w.tx || v.ty != w.ty || v.tz != w.tz || v.T1 != w.T1 || v.mlo != w.mlo ||
                v.mhi != w.mhi || v.first != w.first || v.px != w.px || v.py != w.py || v.pz != w.pz || v.Tn != w.Tn || v.idx != w.idx) {
                printf("resume differs\n");
                exit(1);
            }
            w = v;
            if (g() % 2) continue;   /* found again */
        }
        out.push_back(c);
        fresh = false;
    }
}

int main() {
    std::mt19937 g(12345);
    auto U = [&](double a, double b) { return (float)std::uniform_real_distribution<>(a, b)(g); };
    const char* names[] = {"outside", "inside", "integer_origin", "axis", "diagonal", "plane", "behind", "far"};
    for (int fam = 0; fam < 8; fam++) {
        long long rays = 0, cands = 0, ties = 0;
        for (int Lo = 1; Lo <= 7; Lo++) {
            for (int rep = 0; rep < 6; rep++) {
                const int nLevels = Lo + rep % 4;
                const Tree t = make_tree(g, Lo, nLevels, Lo > 5 ? 0.35 : rep % 2 ? 0.5 : 0.9);
                const float N = (float)(1 << nLevels);
                for (int i = 0; i < 400; i++) {
                    float3 o = f3(U(-2 * N, 3 * N), U(-2 * N, 3 * N), U(-2 * N, 3 * N)), to = f3(U(0, N), U(0, N), U(0, N));
                    if (fam == 1) o = f3(U(0, N), U(0, N), U(0, N));
                    if (fam == 2) o = f3((float)(int)U(0, N + 1), (float)(int)U(-N, 2 * N), U(0, N));
                    if (fam == 7) o = f3(U(-40, 41) * N, U(-40, 41) * N, U(-40, 41) * N);
                    float3 d = normalize(sub(to, o));
                    if (fam == 3) { o = f3(U(-N, 2 * N), (float)(int)U(0, N + 1), U(0, N)); d = f3(i & 1 ? 1.0f : -1.0f, 0.0f, i & 2 ? 0.0f : -0.0f); }
                    if (fam == 4) {
                        o = f3((float)((int)U(-N, N)), (float)((int)U(-N, N)), (float)((int)U(-N, N)));
                        d = normalize(f3(1.0f, i & 1 ? 1.0f : -1.0f, i & 2 ? 1.0f : 0.5f));
                    }
                    if (fam == 5) { o.x = (float)(1 << (nLevels - 1)); d = normalize(f3(i & 1 ? 0.0f : 0.25f, d.y, d.z)); }
                    if (fam == 6) d = mul(d, -1.0f);
                    RayInv r;
                    r.o = o; r.dx = 1 / d.x; r.dy = 1 / d.y; r.dz = 1 / d.z;
                    std::vector<Cand> a, b;
                    float tn, tf;
                    if (slab(r, 0, 0, 0, 1 << nLevels, 1 << nLevels, 1 << nLevels, &tn, &tf)) literal(t, r, 0, 0, 0, 0, 0, a);
                    const int s = walk(t, r, g, b);
                    rays++; cands += a.size(); ties += s == WALK_TIE;
                    bool same = s == WALK_TIE ? b.size() <= a.size() : s == WALK_END && b.size() == a.size();
                    for (size_t k = 0; same && k < b.size(); k++)
                        same = a[k].x == b[k].x && a[k].y == b[k].y && a[k].z == b[k].z && a[k].tn == b[k].tn && a[k].tf == b[k].tf;
                    if (!same) {
                        printf("%s: Lo %d nLevels %d o %.9g %.9g %.9g d %.9g %.9g %.9g: literal %zu walk %zu end %d\n", names[fam], Lo,
                               nLevels, o.x, o.y, o.z, d.x, d.y, d.z, a.size(), b.size(), s);
                        for (size_t k = 0; k < a.size() || k < b.size(); k++) {
                            if (k < a.size()) printf("  L %d %d %d %.9g %.9g", a[k].x, a[k].y, a[k].z, a[k].tn, a[k].tf);
                            if (k < b.size()) printf("  W %d %d %d %.9g %.9g", b[k].x, b[k].y, b[k].z, b[k].tn, b[k].tf);
                            printf("\n");
                        }
                        return 1;
                    }
                }
            }
        }
        printf("%s %lld %lld %lld\n", names[fam], rays, cands, ties);
    }
    return 0;
}
