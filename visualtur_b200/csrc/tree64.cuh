/*
 * tree64.cuh -- a ray's walk over the 64-ary candidate tree.
 *
 * Two binary octree levels make one node of 4 x 4 x 4 cells: a 64-bit mask
 * (bit x*16 + y*4 + z) and the index of the first child, children of a node
 * being contiguous in bit order.  Cells of the last level are the candidate
 * nodes of octreeLevel; with an odd octreeLevel the top node covers twice
 * the volume's edge and has cells in its low half only.
 *
 * The walk steps from cell to cell along the ray and yields the candidates
 * the reference's depth-first search yields (src/Octree.cu:620-760), in its
 * order.  That search accepts a node when, per axis, its entry and exit
 * products (plane - o) * (1 / dir) leave a non-empty interval that ends at
 * t >= 0, and sorts siblings by (tnear, tfar).  Products are monotone in the
 * plane, so a candidate's ancestors accept whenever the candidate does, and
 * while all products met on the way are finite and pairwise distinct the
 * accepted candidates are the cells the ray passes through one after the
 * other, with tnear and tfar the products of the planes it enters and leaves
 * by.  Any coincidence or non-finite product ends the walk with WALK_TIE
 * before a candidate it could affect; the caller then takes the literal
 * search, passing over the candidates already taken.
 */
#pragma once
#include <string.h>

#include "vt_math.cuh"

namespace vt {

/* walk results */
enum { WALK_CANDIDATE = 0, WALK_END = 1, WALK_TIE = 2, WALK_MORE = 3 };

#define VT_TREE64_LEVELS 6      /* ceil(VT_MAX_OCTREE_LEVEL / 2) */

struct Tree64 {
    const uint4* nodes;         /* x, y: cell mask (low, high word); z: first child */
    int nLevels, Lo;            /* candidate cells: 2^Lo per axis, of edge 2^(nLevels - Lo) */
};

struct Walk {
    float px, py, pz;           /* planes the ray would leave the current cell by (voxel coordinates) */
    float tx, ty, tz;           /* their products */
    float tc, Tn, T1;           /* product at which it entered the cell; leaves the node; leaves the volume */
    int sh;                     /* cell edge 1 << sh voxels */
    int idx;                    /* cell in its node: bit of the mask */
    unsigned int mlo, mhi, first;   /* the node */
};

/* a node on the walk's path: its mask, first child and exit product */
typedef uint4 PathNode;

VT_HD float bits_float(int b) {
#ifdef __CUDA_ARCH__
    return __int_as_float(b);
#else
    float f;
    memcpy(&f, &b, 4);
    return f;
#endif
}
VT_HD int float_bits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_int(f);
#else
    int b;
    memcpy(&b, &f, 4);
    return b;
#endif
}
VT_HD int popc32(unsigned int v) {
#ifdef __CUDA_ARCH__
    return __popc(v);
#else
    return __builtin_popcount(v);
#endif
}
/* whole numbers 0 <= v < 2^23 between int and float by the bits of 2^23 + v */
VT_HD float to_float(int v) { return bits_float(0x4B000000 + v) - 8388608.0f; }
VT_HD int to_int(float v) { return float_bits(v + 8388608.0f) - 0x4B000000; }

/* the operations of the reference's slab test */
VT_HD float plane_t(float p, float o, float inv) { return (p - o) * inv; }

VT_HD bool cell_set(const Walk& w) { return (((w.idx & 32) ? w.mhi : w.mlo) >> (w.idx & 31)) & 1u; }
VT_HD unsigned int child_index(const Walk& w) {
    const unsigned int below = (1u << (w.idx & 31)) - 1u;
    return w.first + ((w.idx & 32) ? popc32(w.mlo) + popc32(w.mhi & below) : popc32(w.mlo & below));
}
VT_HD PathNode path_node(const Walk& w) { return make_uint4(w.mlo, w.mhi, w.first, (unsigned int)float_bits(w.Tn)); }
VT_HD void load_node(const Tree64& T, unsigned int n, Walk& w) {
#ifdef __CUDA_ARCH__
    const uint4 v = __ldg(T.nodes + n);
#else
    const uint4 v = T.nodes[n];
#endif
    w.mlo = v.x; w.mhi = v.y; w.first = v.z;
}

/* One axis of entering a node of edge 4 q (two: 2 q) at product tc, sq = q
 * with the ray's sign.  p, t: the plane the ray would leave the node by on
 * this axis and its product; they become those of the cell.  Returns the
 * number of cells behind it.  A plane is passed when its product lies before
 * tc; one that equals it becomes the cell's exit plane, and the walk's next
 * look at the cell (which must end after tc) finds the tie. */
VT_HD int enter_axis(float sq, float o, float inv, float tc, float& p, float& t, bool two) {
    float b = p, bt = t;          /* far plane of the half the ray is in */
    bool far = !two;              /* it is the second half */
    if (!two) {
        const float pm = p - 2 * sq, tm = plane_t(pm, o, inv);
        far = tm < tc;
        if (!far) { b = pm; bt = tm; }
    }
    const float pq = b - sq, tq = plane_t(pq, o, inv);
    const bool passed = tq < tc;
    p = passed ? b : pq; t = passed ? bt : tq;
    return (far ? 2 : 0) + (passed ? 1 : 0);
}

VT_HD bool finite_f(float v) { return v - v == 0.0f; }

/* entry and exit products of the whole volume; false when one is not finite */
VT_HD bool root_span(const Tree64& T, const RayInv& r, Walk& w) {
    const float N = (float)(1 << T.nLevels);
    const float ax = (0.0f - r.o.x) * r.dx, bx = (N - r.o.x) * r.dx;
    const float ay = (0.0f - r.o.y) * r.dy, by = (N - r.o.y) * r.dy;
    const float az = (0.0f - r.o.z) * r.dz, bz = (N - r.o.z) * r.dz;
    const bool sx = r.dx >= 0, sy = r.dy >= 0, sz = r.dz >= 0;
    w.px = sx ? N : 0.0f; w.py = sy ? N : 0.0f; w.pz = sz ? N : 0.0f;
    w.tx = sx ? bx : ax; w.ty = sy ? by : ay; w.tz = sz ? bz : az;
    w.tc = fmaxf(fmaxf(sx ? ax : bx, sy ? ay : by), sz ? az : bz);
    w.T1 = fminf(fminf(w.tx, w.ty), w.tz);
    return finite_f(ax) && finite_f(bx) && finite_f(ay) && finite_f(by) && finite_f(az) && finite_f(bz);
}

/* the mask bits of the axes the ray runs down on (flips a cell counted along
 * the ray into its mask bit, within a node of `two` or four cells an axis) */
VT_HD int flip_bits(const RayInv& r, bool two) {
    return ((r.dx >= 0 ? 0 : 48) | (r.dy >= 0 ? 0 : 12) | (r.dz >= 0 ? 0 : 3)) & (two ? 21 : 63);
}
/* into node n (cells of edge 1 << w.sh) at product w.tc */
template <int STRIDE>
VT_HD void enter_node(const Tree64& T, const RayInv& r, Walk& w, PathNode* path, unsigned int n, bool two = false) {
    const int shS = T.nLevels - T.Lo;
    load_node(T, n, w);
    path[((w.sh - shS) >> 1) * STRIDE] = path_node(w);
    const float q = to_float(1 << w.sh);
    const int nx = enter_axis(r.dx >= 0 ? q : -q, r.o.x, r.dx, w.tc, w.px, w.tx, two);
    const int ny = enter_axis(r.dy >= 0 ? q : -q, r.o.y, r.dy, w.tc, w.py, w.ty, two);
    const int nz = enter_axis(r.dz >= 0 ? q : -q, r.o.z, r.dz, w.tc, w.pz, w.tz, two);
    w.idx = ((nx << 4) | (ny << 2) | nz) ^ flip_bits(r, two);
}

/* Puts the ray into the volume's first cell.  WALK_CANDIDATE: there;
 * WALK_END: it misses the volume (or the volume lies behind it). */
template <int STRIDE>
VT_HD int walk_root(const Tree64& T, const RayInv& r, Walk& w, PathNode* path) {
    if (!root_span(T, r, w)) return WALK_TIE;
    if (w.tc > w.T1 || w.T1 < 0.0f) return WALK_END;
    if (w.tc == w.T1) return WALK_TIE;
    w.Tn = w.T1;
    w.sh = T.nLevels - T.Lo + 2 * (((T.Lo + 1) >> 1) - 1);
    enter_node<STRIDE>(T, r, w, path, 0, T.Lo & 1);
    return WALK_CANDIDATE;
}

/* low corner of the current cell on an axis */
VT_HD int cell_low(float p, float inv, int sh) { return to_int(p) - (inv >= 0 ? 1 << sh : 0); }

/* the current candidate cell's coordinates, in candidate cells */
VT_HD void walk_cell(const Tree64& T, const RayInv& r, const Walk& w, int& x, int& y, int& z) {
    const int shS = T.nLevels - T.Lo;
    x = cell_low(w.px, r.dx, w.sh) >> shS; y = cell_low(w.py, r.dy, w.sh) >> shS; z = cell_low(w.pz, r.dz, w.sh) >> shS;
}

/* Puts the ray back into candidate cell (x,y,z), as it was when the walk
 * yielded it. */
template <int STRIDE>
VT_HD void walk_at(const Tree64& T, const RayInv& r, int x, int y, int z, Walk& w, PathNode* path) {
    const int shS = T.nLevels - T.Lo;
    const bool sx = r.dx >= 0, sy = r.dy >= 0, sz = r.dz >= 0;
    root_span(T, r, w);
    w.Tn = w.T1;
    unsigned int n = 0;
    float ex = 0, ey = 0, ez = 0;
    for (int k = ((T.Lo + 1) >> 1) - 1; k >= 0; k--) {
        load_node(T, n, w);
        path[k * STRIDE] = path_node(w);
        w.sh = shS + 2 * k;
        const int cx = x >> (2 * k), cy = y >> (2 * k), cz = z >> (2 * k);
        w.idx = ((cx & 3) << 4) | ((cy & 3) << 2) | (cz & 3);
        w.px = to_float((cx + sx) << w.sh); w.py = to_float((cy + sy) << w.sh); w.pz = to_float((cz + sz) << w.sh);
        ex = to_float((cx + !sx) << w.sh); ey = to_float((cy + !sy) << w.sh); ez = to_float((cz + !sz) << w.sh);
        w.tx = plane_t(w.px, r.o.x, r.dx); w.ty = plane_t(w.py, r.o.y, r.dy); w.tz = plane_t(w.pz, r.o.z, r.dz);
        if (k > 0) { n = child_index(w); w.Tn = fminf(fminf(w.tx, w.ty), w.tz); }
    }
    w.tc = fmaxf(fmaxf(plane_t(ex, r.o.x, r.dx), plane_t(ey, r.o.y, r.dy)), plane_t(ez, r.o.z, r.dz));
}

/* Walks to the next candidate cell (walk_cell): w.tc its entry product, *tf
 * its exit product.  fresh = false: the current cell has been dealt with.
 * Enters at most `budget` nodes (counted down, and up in *entered); with
 * none left it stops at the cell it would enter, WALK_MORE (fresh again).
 *
 * The inner loop steps through a node's cells by the products alone: it
 * leaves the node where the next product is the node's own exit product,
 * and two planes crossed at once show as a step that does not advance.  It
 * runs until it must leave or enter a node: a warp pays for a turn of the
 * outer loop whatever few lanes need it, so the more cheap steps before one
 * the better (at most 1, 2, 3, 4 steps a turn: 1047, 793, 708, 654 us on a
 * 1920x1080 frame, unbounded 584), and a node left for a set cell is
 * followed by entering that cell in the same turn (612 -> 584 us).
 */
template <int STRIDE>
VT_HD int walk_next(const Tree64& T, const RayInv& r, Walk& w, PathNode* path, bool fresh, int& budget, float* tf,
                    unsigned int* entered) {
    const int shS = T.nLevels - T.Lo;
    const bool sx = r.dx >= 0, sy = r.dy >= 0, sz = r.dz >= 0;
    int res = -1;
    do {
        float m = fminf(fminf(w.tx, w.ty), w.tz);
        bool set = fresh && m >= 0.0f && cell_set(w);
        const float q = to_float(1 << w.sh);
        while (!set && m < w.Tn && m > w.tc) {
            const bool ax = w.tx == m, ay = !ax && w.ty == m, az = !ax && !ay;   /* one axis a step */
            w.tc = m;
            if (ax) { w.px += sx ? q : -q; w.tx = plane_t(w.px, r.o.x, r.dx); w.idx += sx ? 16 : -16; }
            if (ay) { w.py += sy ? q : -q; w.ty = plane_t(w.py, r.o.y, r.dy); w.idx += sy ? 4 : -4; }
            if (az) { w.pz += sz ? q : -q; w.tz = plane_t(w.pz, r.o.z, r.dz); w.idx += sz ? 1 : -1; }
            m = fminf(fminf(w.tx, w.ty), w.tz);
            set = m >= 0.0f && cell_set(w);
        }
        fresh = true;
        if (!(m > w.tc)) {
            res = WALK_TIE;
        } else if (!set || m == 0.0f) {
            /* two planes at once: seen here where the next step would not
             * show it, on leaving the node, and at t = 0, where the cells
             * before and behind sort alike (their tnear is clamped to 0) */
            const bool ax = w.tx == m, ay = w.ty == m, az = w.tz == m;
            if ((ax && ay) || (ax && az) || (ay && az)) {
                res = WALK_TIE;
            } else if (!set) {
                if (m >= w.T1) {
                    res = WALK_END;
                } else {
                    /* out of the node: up to the one in which the plane separates two cells */
                    const int P = to_int(ax ? w.px : ay ? w.py : w.pz);
                    int X = cell_low(w.px, r.dx, w.sh), Y = cell_low(w.py, r.dy, w.sh), Z = cell_low(w.pz, r.dz, w.sh);
#ifdef __CUDA_ARCH__
                    const int b = 31 - __clz(P & -P);
#else
                    const int b = __builtin_ctz(P);
#endif
                    w.sh = shS + ((b - shS) & ~1);
                    const int Q = 1 << w.sh;
                    X = (ax ? (sx ? P : P - Q) : X) & -Q;
                    Y = (ay ? (sy ? P : P - Q) : Y) & -Q;
                    Z = (az ? (sz ? P : P - Q) : Z) & -Q;
                    const PathNode e = path[((w.sh - shS) >> 1) * STRIDE];
                    w.mlo = e.x; w.mhi = e.y; w.first = e.z;
                    w.Tn = bits_float((int)e.w);
                    w.idx = (((X >> w.sh) & 3) << 4) | (((Y >> w.sh) & 3) << 2) | ((Z >> w.sh) & 3);
                    w.px = to_float(sx ? X + Q : X); w.py = to_float(sy ? Y + Q : Y); w.pz = to_float(sz ? Z + Q : Z);
                    w.tx = plane_t(w.px, r.o.x, r.dx); w.ty = plane_t(w.py, r.o.y, r.dy); w.tz = plane_t(w.pz, r.o.z, r.dz);
                    w.tc = m;
                    /* a set cell is entered in this same turn (one that ends at 0 gets the look above first) */
                    m = fminf(fminf(w.tx, w.ty), w.tz);
                    set = m > 0.0f && m > w.tc && cell_set(w);
                }
            }
        }
        if (res < 0 && set) {
            if (w.sh == shS) {
                *tf = m;
                res = WALK_CANDIDATE;
            } else if (budget-- <= 0) {
                res = WALK_MORE;
            } else {
                (*entered)++;
                const unsigned int n = child_index(w);
                w.sh -= 2;
                w.Tn = m;
                enter_node<STRIDE>(T, r, w, path, n);
            }
        }
    } while (res < 0);
    return res;
}

}  // namespace vt
