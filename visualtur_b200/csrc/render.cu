/*
 * render.cu -- ray-casting kernels of libvt.so (sm_100a).
 *
 * k_trace fuses the reference's three per-iteration phases -- octree
 * traversal (cuda_getFirtsVoxel, src/Octree.cu:620-739), cache lookup
 * (lruCache::updateCube, src/lruCache.cu:168-296) and march + shade
 * (cuda_rayCaster, src/rayCaster.cu:139-265) -- into one kernel: each ray
 * walks from candidate node to candidate node, marches every one whose brick
 * is resident, and either finishes or, at an absent brick, suspends with the
 * cell it has come to.  The result equals the reference's
 * iterate-until-PAINTED loop: candidates are marched in its depth-first
 * order and the first hit is shaded.  The instantiations with SKIP = true
 * let a ray set absent-brick candidates aside and march later ones in the
 * same pass (see run_ray); the first hit in that order still decides the
 * pixel.
 *
 * Octree: the same tree twice, from a flattened node array with 8-bit child
 * masks that hold the result of the reference's range search (computed once
 * per octree load).  k_trace walks it two levels at a time (tree64.cuh);
 * rays that meet coinciding planes, and the wavefront passes, search the
 * binary nodes depth first and suspend with their stack.
 */
#include "vt_kernels.h"
#include "vt_math.cuh"

namespace vt {

/* ---- samplers ---------------------------------------------------------- */
/* Small integers and floats without the conversion unit: the bits of
 * 2^23 + k are 0x4B000000 + k for an integer 0 <= k < 2^23.  Conversions
 * issue at a quarter of the rate of an add (16 lanes a clock per SM), and a
 * trilinear sample needs three of them for its tap indices and eight more
 * for uint8 voxels.  Against converting: 96^2 resident frame 121 -> 108 us,
 * 512^2 192 -> 174 us, 1277x719 uint8 with bisection 724 -> 679 us,
 * 1920x1080 float32 836 -> 816 us (same pixels). */
#define VT_2P23 8388608.0f
#define VT_2P23_BITS 0x4B000000

/* Trilinear sampler over one brick (slab mode) or the padded volume
 * (dense mode).  ox,oy,oz: integer origin of the index space (the
 * reference's minBox = brick min corner - cubeInc); h: largest first tap
 * on each axis so both taps stay inside the buffer (the clamp is never
 * active for finite positions with cubeInc >= 3). */
struct Samp {
    const void* base; int sx, sy; float ox, oy, oz, h;
};

/* voxel p[i]; a uint8 voxel becomes a float by its bits, exactly */
template <int VTYPE, bool SHM>
__device__ __forceinline__ float ldv(const void* p, int i) {
    if (VTYPE == 0) return SHM ? ((const float*)p)[i] : __ldg((const float*)p + i);
    const unsigned int b = SHM ? ((const unsigned char*)p)[i] : __ldg((const unsigned char*)p + i);
    return __uint_as_float(VT_2P23_BITS | b) - VT_2P23;
}

/* p = integral part + fraction, both with p's sign (modff) */
__device__ __forceinline__ float split_pos(float p, float* r) {
    *r = truncf(p);
    return copysignf(p - *r, p);
}

/* the clamped first tap as VT_2P23_BITS + index: r - o is an integer, exact
 * wherever the clamp leaves it; NaN gives 0 (as cvt.rzi does) */
__device__ __forceinline__ int tap_bits(float r, float o, float h) {
    return __float_as_int(fminf(fmaxf(r - o, 0.0f), h) + VT_2P23);
}

/* getElementInterpolate (src/rayCaster.cu:86-106). */
template <int VTYPE, bool SLAB = false, bool SHM = false>
__device__ __forceinline__ float interp(const Samp& s, float3 p) {
    float rx, ry, rz;
    const float px = split_pos(p.x, &rx), py = split_pos(p.y, &ry), pz = split_pos(p.z, &rz);
    const int x0 = tap_bits(rx, s.ox, s.h), y0 = tap_bits(ry, s.oy, s.h), z0 = tap_bits(rz, s.oz, s.h);
    const int es = VTYPE == 0 ? 4 : 1;
    const char* p00;
    if (SLAB) {
        /* a brick holds < 2^31 voxels: 32-bit index arithmetic, the three
         * VT_2P23_BITS terms taken off modulo 2^32 */
        const unsigned int b = (unsigned int)x0 * (unsigned int)s.sx + (unsigned int)y0 * (unsigned int)s.sy +
                               (unsigned int)z0 - (unsigned int)VT_2P23_BITS * (unsigned int)(s.sx + s.sy + 1);
        p00 = (const char*)s.base + (size_t)b * es;
    } else {
        const int yz = (y0 - VT_2P23_BITS) * s.sy + (z0 - VT_2P23_BITS);
        p00 = (const char*)s.base + ((long long)(x0 - VT_2P23_BITS) * s.sx + yz) * es;
    }
    const char* p01 = p00 + (size_t)(unsigned int)s.sy * es;
    const char* p10 = p00 + (size_t)(unsigned int)s.sx * es;
    const char* p11 = p10 + (size_t)(unsigned int)s.sy * es;
    const float v000 = ldv<VTYPE, SHM>(p00, 0), v001 = ldv<VTYPE, SHM>(p00, 1);
    const float v010 = ldv<VTYPE, SHM>(p01, 0), v011 = ldv<VTYPE, SHM>(p01, 1);
    const float v100 = ldv<VTYPE, SHM>(p10, 0), v101 = ldv<VTYPE, SHM>(p10, 1);
    const float v110 = ldv<VTYPE, SHM>(p11, 0), v111 = ldv<VTYPE, SHM>(p11, 1);
    float qx = 1.0f - px, qy = 1.0f - py, qz = 1.0f - pz;
    float c00 = v000 * qx + v100 * px;
    float c01 = v001 * qx + v101 * px;
    float c10 = v010 * qx + v110 * px;
    float c11 = v011 * qx + v111 * px;
    float c0 = c00 * qy + c10 * py;
    float c1 = c01 * qy + c11 * py;
    return c0 * qz + c1 * pz;
}

/* getNormal (src/rayCaster.cu:131-137). */
template <int VTYPE, bool SLAB, bool SHM = false>
__device__ __forceinline__ float3 normal_at(const Samp& s, float3 p) {
    /* six taps through one call site: shading runs once per hit ray, and
     * the smaller kernel keeps the traversal loop in the instruction cache */
    float v[6];
#pragma unroll 1
    for (int t = 0; t < 6; t++) {
        const float d = (t & 1) ? 1.0f : -1.0f;
        float3 q = p;
        if (t < 2) q.x = p.x + d;
        else if (t < 4) q.y = p.y + d;
        else q.z = p.z + d;
        v[t] = interp<VTYPE, SLAB, SHM>(s, q);
    }
    return normalize(f3((v[0] - v[1]) / 2.0f, (v[2] - v[3]) / 2.0f, (v[4] - v[5]) / 2.0f));
}

/* The march of cuda_rayCaster (src/rayCaster.cu:166-237): samples at
 * Xnear, Xnear += 0.5*dir, for steps 0..maxStep, to the first sign change of
 * iso - value (equality counts).  U samples are fetched per round: their
 * positions accumulate in the reference's order, their taps are issued
 * together, and the crossing test then runs sample by sample -- fetches
 * past the crossing are discarded (indices stay clamped to the brick) and
 * are not counted.  A crossing leaves the sample before it in C. */
struct Crossing {
    float3 P;        /* last sample before the crossing; the crossing sample is P + 0.5*dir */
    float ant, sig;  /* their values */
};
template <int VTYPE, bool SLAB, int U, bool SHM = false>
__device__ __forceinline__ bool march(const Samp& s, float3 origin, float3 ray, float tnear, int maxStep, float iso,
                                      Crossing& C, unsigned int* nsamp) {
    const float3 vStep = mul(ray, 0.5f);
    if (maxStep < 0) return false;
    C.P = add(origin, mul(ray, tnear));
    C.ant = interp<VTYPE, SLAB, SHM>(s, C.P);
    unsigned int ns = 1;
    bool hit = false;
    for (int steps = 1; steps <= maxStep && !hit; steps += U) {
        float3 X[U];
        float v[U];
#pragma unroll
        for (int u = 0; u < U; u++) X[u] = add(u == 0 ? C.P : X[u - 1], vStep);
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = interp<VTYPE, SLAB, SHM>(s, X[u]);
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (hit || steps + u > maxStep) break;
            C.sig = v[u];
            ns++;
            if ((((iso - C.ant) < 0.0f) && ((iso - C.sig) < 0.0f)) ||
                (((iso - C.ant) > 0.0f) && ((iso - C.sig) > 0.0f))) {
                C.ant = C.sig;
                C.P = X[u];
            } else {
                hit = true;
            }
        }
    }
    *nsamp += ns;
    return hit;
}

/* The crossing refined to the hit point (src/rayCaster.cu:227-228): one
 * linear step.  refine > 0 first bisects the bracketing pair that many
 * times: the midpoint replaces the end whose iso - value has the same
 * strict sign as its own (the crossing test's "no crossing" condition), so
 * the pair keeps bracketing the crossing.  Each midpoint is one more
 * trilinear sample. */
template <int VTYPE, bool SLAB, bool SHM>
__device__ __forceinline__ float3 refine_hit(const Samp& s, float3 ray, const Crossing& C, float iso, int refine,
                                             unsigned int* nsamp) {
    float3 P = C.P, Q = add(C.P, mul(ray, 0.5f));
    float ant = C.ant, sig = C.sig;
    for (int k = 0; k < refine; k++) {
        float3 M = mul(add(P, Q), 0.5f);
        float vm = interp<VTYPE, SLAB, SHM>(s, M);
        if ((((iso - ant) < 0.0f) && ((iso - vm) < 0.0f)) || (((iso - ant) > 0.0f) && ((iso - vm) > 0.0f))) {
            P = M; ant = vm;
        } else {
            Q = M; sig = vm;
        }
    }
    *nsamp += refine;
    float a = (iso - ant) / (sig - ant);
    return add(mul(P, 1.0f - a), mul(Q, a));
}

/* Stack entry: (node index in its level << code_bits) | Morton code. */
struct Stk {
    unsigned long long e[VT_STACK];
    unsigned long long sk[VT_SKIP_MAX];   /* passed-over candidates, DFS order */
};

/* stack entry helpers (layout in vt_kernels.h) */
__device__ __forceinline__ unsigned long long make_entry(unsigned int idx, int level, unsigned int x, unsigned int y,
                                                         unsigned int z) {
    return ((unsigned long long)idx << VT_E_INDEX_SHIFT) | ((unsigned long long)level << VT_E_LEVEL_SHIFT) |
           ((unsigned long long)x << (2 * VT_E_COORD_BITS)) | ((unsigned long long)y << VT_E_COORD_BITS) | z;
}
__device__ __forceinline__ int e_level(unsigned long long e) { return (int)((e >> VT_E_LEVEL_SHIFT) & 15u); }
__device__ __forceinline__ unsigned int e_index(unsigned long long e) { return (unsigned int)(e >> VT_E_INDEX_SHIFT); }
__device__ __forceinline__ unsigned int e_x(unsigned long long e) { return (unsigned int)(e >> (2 * VT_E_COORD_BITS)) & 0x7FFu; }
__device__ __forceinline__ unsigned int e_y(unsigned long long e) { return (unsigned int)(e >> VT_E_COORD_BITS) & 0x7FFu; }
__device__ __forceinline__ unsigned int e_z(unsigned long long e) { return (unsigned int)e & 0x7FFu; }

/* sampler for the brick at brick coordinates (bx,by,bz), in device slot `slot` */
template <int VTYPE, bool SLAB>
__device__ __forceinline__ void brick_sampler(const TraceArgs& A, unsigned int bx, unsigned int by, unsigned int bz,
                                              int slot, Samp& s) {
    const DevBricks& B = A.br;
    if (SLAB) {
        const int sh = A.oct.nLevels - A.oct.Lc;
        s.ox = (float)((int)(bx << sh) - B.inc); s.oy = (float)((int)(by << sh) - B.inc);
        s.oz = (float)((int)(bz << sh) - B.inc);
        s.base = (const char*)B.slab + (size_t)slot * (size_t)B.brickVol * (VTYPE == 0 ? 4 : 1);
        s.sx = B.D * B.D; s.sy = B.D;
        s.h = (float)(B.D - 2);
    } else {
        /* dense: index space = the padded volume, global voxel g at g + P.
         * Equals the brick-relative index of the reference whenever every
         * tap lies inside the brick and its apron (cubeInc >= 3). */
        s.ox = s.oy = s.oz = (float)-B.P;
        s.base = B.vol;
        s.sx = (int)B.vsx; s.sy = (int)B.vsy;
        s.h = (float)(B.ve - 2);
    }
}

/* One ray in flight. */
struct Ray {
    RayInv r;
    int lastSlot;          /* slot whose stamp this ray wrote last */
    float3 dir;
    int top;
    int view, i, j;
    unsigned int g;        /* padded global ray index */
    float4 rgba;
    unsigned long long node, brick;
    float t;
    float3 n;
    bool hit;
    int nskip;             /* candidates passed over (brick absent), in st.sk */
    bool tent;             /* the pixel holds a hit found past them */
    bool resumeSkips;      /* the passed-over candidates come first (a resumed ray) */
    unsigned int taken;    /* candidates the 64-ary walk has already dealt with */
};

/* RAY_TENTATIVE: a hit past passed-over candidates (the pixel is written,
 * the ray suspends until they are decided); RAY_DONE_WRITTEN: they all
 * missed, the pixel written earlier stands. */
enum { RAY_RUNNING = 0, RAY_DONE = 1, RAY_SUSPENDED = 2, RAY_TENTATIVE = 3, RAY_DONE_WRITTEN = 4 };
enum { CAND_MISSING = 0, CAND_EMPTY = 1, CAND_HIT = 2 };

/* Requests page `pidx` once per pass.  A demand request (a ray waits on
 * the brick) moves the page from absent (-1) or speculatively requested
 * (-3) to -2; a speculative one (lookahead) from -1 to -3 and is tagged in
 * the list, so the host loads it only into a slot this frame has not used.
 * Past the list's capacity the page goes back to absent and the request
 * waits for the next pass (the rays that need it suspend and ask again),
 * as the reference's per-pass admission cap defers NOCACHED rays
 * (src/lruCache.cu:184-192). */
__device__ __forceinline__ void request_brick(const TraceArgs& A, unsigned int pidx, bool spec = false) {
    const int mark = spec ? VT_PAGE_SPECULATIVE : VT_PAGE_REQUESTED;
    int old = atomicCAS(&A.br.page[pidx], -1, mark);
    if (old == VT_PAGE_SPECULATIVE && !spec)
        old = atomicCAS(&A.br.page[pidx], VT_PAGE_SPECULATIVE, VT_PAGE_REQUESTED) == VT_PAGE_SPECULATIVE ? -1 : old;
    if (old == -1) {
        unsigned int q = atomicAdd(A.ctl.n_req, 1u);
        if (q < A.ctl.req_cap) {
            A.ctl.req[q] = pidx | (spec ? VT_REQ_SPECULATIVE : 0ull);
        } else {
            atomicCAS(&A.br.page[pidx], mark, -1);
            atomicAdd(&A.ctl.counters[VT_C_REQDEFER], 1ull);
        }
    }
}

/* Expands the inner node `ent` (_cuda_searchChildrenValidAndHit2,
 * src/Octree.cu:375-532, with membership from the flattened child mask):
 * children hit by the ray with tfar >= 0 are sorted by (tnear, tfar)
 * (src/Octree.cu:665-706) and pushed far to near. */
__device__ __forceinline__ bool expand(const TraceArgs& A, const RayInv& r, Stk& st, int& top,
                                       unsigned long long ent, unsigned int* cnt, bool sortChildren) {
    const DevOctree& O = A.oct;
    const int nLevels = O.nLevels, Lo = O.Lo;
    const int level = e_level(ent);
    const unsigned int px_ = e_x(ent), py_ = e_y(ent), pz_ = e_z(ent);
    const uint2 nd = O.nodes[e_index(ent)];
    const int cl = level + 1;
    const int cd = 1 << (nLevels - cl);
    const int mx = (int)(px_ << (nLevels - level)), my = (int)(py_ << (nLevels - level)), mz = (int)(pz_ << (nLevels - level));
    /* the children's faces lie on 3 planes per axis: the slab products of
     * all 8 children are these 9 values (the same float operations the
     * reference performs per child, src/Octree.cu:258-330) */
    const float x0 = ((float)mx - r.o.x) * r.dx, x1 = ((float)(mx + cd) - r.o.x) * r.dx,
                x2 = ((float)(mx + 2 * cd) - r.o.x) * r.dx;
    const float y0 = ((float)my - r.o.y) * r.dy, y1 = ((float)(my + cd) - r.o.y) * r.dy,
                y2 = ((float)(my + 2 * cd) - r.o.y) * r.dy;
    const float z0 = ((float)mz - r.o.z) * r.dz, z1 = ((float)(mz + cd) - r.o.z) * r.dz,
                z2 = ((float)(mz + 2 * cd) - r.o.z) * r.dz;
    /* entry / exit parameter of the low (0) and high (1) half on each axis,
     * ordered by the direction's sign as the reference's slab test orders
     * them (src/Octree.cu:268-300) */
    const bool sx = r.dx >= 0, sy = r.dy >= 0, sz = r.dz >= 0;
    const float ex0 = sx ? x0 : x1, fx0 = sx ? x1 : x0, ex1 = sx ? x1 : x2, fx1 = sx ? x2 : x1;
    const float ey0 = sy ? y0 : y1, fy0 = sy ? y1 : y0, ey1 = sy ? y1 : y2, fy1 = sy ? y2 : y1;
    const float ez0 = sz ? z0 : z1, fz0 = sz ? z1 : z0, ez1 = sz ? z1 : z2, fz1 = sz ? z2 : z1;
    const unsigned int m = nd.y;
    /* Fast path (parametric traversal).  Inside the node the ray's
     * parameter runs from T0 to T1 and changes half on axis a where it
     * crosses the mid-plane, at t = a1.  When T0, T1, the three crossings
     * and 0 are finite and pairwise distinct, the children the slab tests
     * accept are exactly the segments between consecutive events whose end
     * is >= 0; their tnear values are the segment starts, distinct after
     * the clamp to 0, so (tnear, tfar) order is segment order.  The
     * segments, filtered by membership, are pushed directly; any
     * coincidence, infinity or NaN takes the literal path below. */
    if (sortChildren) {
        const float T0 = fmaxf(fmaxf(sx ? x0 : x2, sy ? y0 : y2), sz ? z0 : z2);
        const float T1 = fminf(fminf(sx ? x2 : x0, sy ? y2 : y0), sz ? z2 : z0);
        bool ok = isfinite(x0) && isfinite(x1) && isfinite(x2) && isfinite(y0) && isfinite(y1) && isfinite(y2) &&
                  isfinite(z0) && isfinite(z1) && isfinite(z2) && T0 < T1;
        ok = ok && T0 != x1 && T0 != y1 && T0 != z1 && T0 != 0.0f && T1 != x1 && T1 != y1 && T1 != z1 &&
             T1 != 0.0f && x1 != y1 && x1 != z1 && y1 != z1 && x1 != 0.0f && y1 != 0.0f && z1 != 0.0f;
        if (ok) {
            /* half of each axis at entry: the sign-ordered first half while
             * the crossing lies ahead */
            const int kx = (x1 > T0) ? (sx ? 0 : 1) : (sx ? 1 : 0);
            const int ky = (y1 > T0) ? (sy ? 0 : 1) : (sy ? 1 : 0);
            const int kz = (z1 > T0) ? (sz ? 0 : 1) : (sz ? 1 : 0);
            /* crossings inside (T0, T1), sorted with the child-index bit each flips */
            const float INF = __int_as_float(0x7f800000);
            float c0 = (x1 > T0 && x1 < T1) ? x1 : INF, c1 = (y1 > T0 && y1 < T1) ? y1 : INF,
                  c2 = (z1 > T0 && z1 < T1) ? z1 : INF;
            int b0 = 4, b1 = 2, b2 = 1;
            if (c1 < c0) { float t = c0; c0 = c1; c1 = t; int b = b0; b0 = b1; b1 = b; }
            if (c2 < c1) { float t = c1; c1 = c2; c2 = t; int b = b1; b1 = b2; b2 = b; }
            if (c1 < c0) { float t = c0; c0 = c1; c1 = t; int b = b0; b0 = b1; b1 = b; }
            const int n1 = c0 < INF, n2 = c1 < INF, n3 = c2 < INF;
            const int ch0 = (kx << 2) | (ky << 1) | kz, ch1 = ch0 ^ b0, ch2 = ch1 ^ b1, ch3 = ch2 ^ b2;
            const bool a0 = (n1 ? c0 : T1) >= 0.0f && ((m >> ch0) & 1u);
            const bool a1 = n1 && (n2 ? c1 : T1) >= 0.0f && ((m >> ch1) & 1u);
            const bool a2 = n2 && (n3 ? c2 : T1) >= 0.0f && ((m >> ch2) & 1u);
            const bool a3 = n3 && T1 >= 0.0f && ((m >> ch3) & 1u);
            const int nvf = (int)a0 + (int)a1 + (int)a2 + (int)a3;
            if (top + nvf >= VT_STACK) {
                atomicOr(A.ctl.err, VT_KERR_STACK);
                top = -1;
                return false;
            }
            /* near to far: the first accepted segment ends on top */
            int q = top + nvf;
            const int chs[4] = {ch0, ch1, ch2, ch3};
            const bool acc[4] = {a0, a1, a2, a3};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (acc[i]) {
                    const int k = chs[i];
                    const unsigned int cidx = cl < Lo ? nd.x + __popc(m & ((1u << k) - 1u)) : 0u;
                    st.e[q--] = make_entry(cidx, cl, (px_ << 1) | ((k >> 2) & 1), (py_ << 1) | ((k >> 1) & 1),
                                           (pz_ << 1) | (k & 1));
                }
            }
            top += nvf;
            if ((unsigned int)(top + 1) > cnt[VT_C_MAXSTACK]) cnt[VT_C_MAXSTACK] = top + 1;
            return true;
        }
    }
    unsigned long long cent[8];
    float ctn[8], ctf[8];
    int nv = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        if ((m >> k) & 1u) {
            const int kx = (k >> 2) & 1, ky = (k >> 1) & 1, kz = k & 1;
            float a, b;
            if (slab_t(kx ? ex1 : ex0, kx ? fx1 : fx0, ky ? ey1 : ey0, ky ? fy1 : fy0, kz ? ez1 : ez0, kz ? fz1 : fz0,
                       &a, &b) &&
                b >= 0.0f) {
                unsigned int cidx = cl < Lo ? nd.x + __popc(m & ((1u << k) - 1u)) : 0u;
                cent[nv] = make_entry(cidx, cl, (px_ << 1) | kx, (py_ << 1) | ky, (pz_ << 1) | kz);
                ctn[nv] = a; ctf[nv] = b;
                nv++;
            }
        }
    }
    if (sortChildren) {
        if (nv == 2) {
            /* one pass of the bubble sort decides two children */
            if (ctn[0] > ctn[1] || (ctn[0] == ctn[1] && ctf[0] > ctf[1])) {
                unsigned long long te = cent[0]; cent[0] = cent[1]; cent[1] = te;
            }
        } else if (nv > 2) {
            int n = nv;
            while (n != 0) {
                int newn = 0;
                for (int q = 1; q < nv; q++) {
                    if (ctn[q - 1] > ctn[q] || (ctn[q - 1] == ctn[q] && ctf[q - 1] > ctf[q])) {
                        unsigned long long te = cent[q]; cent[q] = cent[q - 1]; cent[q - 1] = te;
                        float tt = ctn[q]; ctn[q] = ctn[q - 1]; ctn[q - 1] = tt;
                        tt = ctf[q]; ctf[q] = ctf[q - 1]; ctf[q - 1] = tt;
                        newn = q;
                    }
                }
                n = newn;
            }
        }
    }
    if (top + nv >= VT_STACK) {
        if (sortChildren) atomicOr(A.ctl.err, VT_KERR_STACK);   /* lookahead walks only stop */
        top = -1;
        return false;
    }
    for (int q = nv - 1; q >= 0; q--) st.e[++top] = cent[q];
    if ((unsigned int)(top + 1) > cnt[VT_C_MAXSTACK]) cnt[VT_C_MAXSTACK] = top + 1;
    return true;
}

/* Shading of a hit at X (src/rayCaster.cu:238-250): the normal from
 * central differences, |n . l| against the light, the colour ramp over y;
 * the ray's hit fields for the pixel and the diagnostics. */
template <int VTYPE, bool SLAB, bool SHM>
__device__ __forceinline__ void shade_hit(const TraceArgs& A, Ray& R, const Samp& s, float3 X, unsigned int x,
                                          unsigned int y, unsigned int z, unsigned int bx, unsigned int by,
                                          unsigned int bz, unsigned int* cnt) {
    float3 n = normal_at<VTYPE, SLAB, SHM>(s, X);
    cnt[VT_C_NSAMPLES] += 6;
    float3 l = normalize(sub(X, A.light));
    float dif = fabsf(n.x * l.x + n.y * l.y + n.z * l.z);
    float a = X.y / 256.0f;
    R.rgba = make_float4((1 - a) * dif, a * dif, 0.0f * dif, 1.0f);
    R.hit = true; R.n = n;
    if (A.out.node) R.node = node_code(x, y, z, A.oct.Lo);
    if (A.out.brick) R.brick = node_code(bx, by, bz, A.oct.Lc);
    R.t = dot(sub(X, R.r.o), R.dir);
}

/* Candidate `ent` (a node at octreeLevel): brick lookup
 * (lruCache::updateCube, src/lruCache.cu:177-291), then march and shade
 * (src/rayCaster.cu:139-265).  CAND_MISSING when the brick is absent (it is
 * requested), CAND_HIT with R's hit fields set, else CAND_EMPTY. */
template <int VTYPE, bool SLAB, int U>
__device__ __forceinline__ int candidate(const TraceArgs& A, Ray& R, unsigned long long ent, unsigned int* cnt) {
    const DevOctree& O = A.oct;
    const int nLevels = O.nLevels, Lo = O.Lo, Lc = O.Lc;
    const int dimO = 1 << (nLevels - Lo);
    const unsigned int x = e_x(ent), y = e_y(ent), z = e_z(ent);
    const unsigned int bx = x >> (Lo - Lc), by = y >> (Lo - Lc), bz = z >> (Lo - Lc);
    const unsigned int pidx = (bx << (2 * Lc)) | (by << Lc) | bz;
    const int slot = SLAB ? A.br.page[pidx] : 0;
    if (SLAB && slot < 0) {
        if (slot == -1 || slot == VT_PAGE_SPECULATIVE) request_brick(A, pidx);
        cnt[VT_C_DEVMISSES]++;
        return CAND_MISSING;
    }
    cnt[VT_C_CANDIDATES]++;
    if (SLAB) {
        cnt[VT_C_DEVHITS]++;
        if (slot != R.lastSlot) { A.br.stamp[slot] = A.br.pass; R.lastSlot = slot; }   /* once per brick run */
    }
    if (A.ctl.touched) {
        const int d = A.ctl.touch_shift / 3;   /* Lo - trace level */
        unsigned long long tn = (spread3(x >> d) << 2) | (spread3(y >> d) << 1) | spread3(z >> d);
        atomicOr(&A.ctl.touched[tn >> 5], 1u << (tn & 31));
    }
    const int mbx = (int)(x << (nLevels - Lo)), mby = (int)(y << (nLevels - Lo)), mbz = (int)(z << (nLevels - Lo));
    float tn, tf;
    if (!slab(R.r, mbx, mby, mbz, mbx + dimO, mby + dimO, mbz + dimO, &tn, &tf)) return CAND_EMPTY;
    Samp s;
    brick_sampler<VTYPE, SLAB>(A, bx, by, bz, slot, s);
    Crossing C;
    if (!march<VTYPE, SLAB, U>(s, R.r.o, R.dir, tn, max_steps(tn, tf), A.iso, C, &cnt[VT_C_SAMPLES]))
        return CAND_EMPTY;
    const float3 X = refine_hit<VTYPE, SLAB, false>(s, R.dir, C, A.iso, A.refine, &cnt[VT_C_SAMPLES]);
    shade_hit<VTYPE, SLAB, false>(A, R, s, X, x, y, z, bx, by, bz, cnt);
    return CAND_HIT;
}

/* Takes one ray's DFS to its end (src/Octree.cu:620-720 interleaved with
 * src/rayCaster.cu:139-265): inner nodes are expanded until a candidate is
 * on top, then the candidate is marched.  Returns RAY_DONE when the ray is
 * shaded or exhausted, RAY_SUSPENDED when it must wait for absent bricks.
 *
 * Passing over absent bricks (A.ctl.skip > 0): a candidate whose brick is
 * absent is requested and set aside, and the DFS goes on to later
 * candidates, up to A.ctl.skip of them a pass.  The first hit still wins in
 * DFS order: a hit found past set-aside candidates is tentative (written,
 * RAY_TENTATIVE), the rest of the DFS is dropped, and the next pass marches
 * the set-aside candidates first, in order; the first of them that hits
 * replaces it, and if none does it stands.  So a ray whose candidates lie
 * in several absent bricks asks for all of them in one pass instead of one
 * per pass, and the image is the one of the in-order traversal. */
template <int VTYPE, bool SLAB, int U, bool SKIP>
__device__ int run_ray(const TraceArgs& A, Ray& R, Stk& st, unsigned int* cnt) {
    const int Lo = A.oct.Lo;
    if (SKIP) {
        while (R.resumeSkips) {
            if (R.nskip == 0) {
                R.resumeSkips = false;
                if (R.tent) return RAY_DONE_WRITTEN;
                break;
            }
            const int c = candidate<VTYPE, SLAB, U>(A, R, st.sk[0], cnt);
            if (c == CAND_MISSING) return RAY_SUSPENDED;
            for (int k = 1; k < R.nskip; k++) st.sk[k - 1] = st.sk[k];
            R.nskip--;
            if (c == CAND_HIT) { R.nskip = 0; R.resumeSkips = false; return RAY_DONE; }
        }
    }
    const int K = SKIP ? A.ctl.skip : 0;
    for (;;) {
        unsigned long long ent;
        for (;;) {
            if (R.top < 0) return (SKIP && R.nskip > 0) ? RAY_SUSPENDED : RAY_DONE;   /* exhausted: background */
            ent = st.e[R.top];
            if (e_level(ent) == Lo) break;
            R.top--;
            cnt[VT_C_EXPANSIONS]++;
            if (!expand(A, R.r, st, R.top, ent, cnt, true)) return RAY_DONE;
        }
        if (R.taken) { R.taken--; R.top--; continue; }
        const int c = candidate<VTYPE, SLAB, U>(A, R, ent, cnt);
        if (c == CAND_MISSING) {
            if (SKIP && R.nskip < K) { st.sk[R.nskip++] = ent; R.top--; continue; }
            return RAY_SUSPENDED;   /* the candidate stays on the stack */
        }
        R.top--;
        if (c == CAND_HIT) {
            if (!SKIP || R.nskip == 0) return RAY_DONE;
            R.top = -1;             /* later candidates cannot matter */
            R.tent = true;
            return RAY_TENTATIVE;
        }
    }
}

/* Speculative requests: walks a copy of a suspended ray's DFS (without
 * marching) and requests up to `lookahead` further absent bricks. */
template <int VTYPE>
__device__ void lookahead_requests(const TraceArgs& A, Ray R, Stk& st, unsigned int* cnt) {
    const DevOctree& O = A.oct;
    const int Lo = O.Lo, Lc = O.Lc;
    int want = A.ctl.lookahead, pops = 0;
    unsigned int last = 0xFFFFFFFFu;
    while (R.top >= 0 && want > 0 && pops++ < 256) {
        unsigned long long ent = st.e[R.top--];
        if (e_level(ent) == Lo) {
            const unsigned int pidx = ((e_x(ent) >> (Lo - Lc)) << (2 * Lc)) | ((e_y(ent) >> (Lo - Lc)) << Lc) |
                                      (e_z(ent) >> (Lo - Lc));
            if (pidx != last && A.br.page[pidx] == -1) { request_brick(A, pidx, true); want--; }
            last = pidx;
            continue;
        }
        unsigned int scratch[VT_C_COUNT];
        scratch[VT_C_MAXSTACK] = cnt[VT_C_MAXSTACK];
        if (!expand(A, R.r, st, R.top, ent, scratch, false)) break;   /* order only affects which bricks get asked */
    }
}

/* padded global ray index -> view and pixel (tile order); the divisions by
 * shifts and a product where the host found them exact */
__device__ __forceinline__ bool decode_ray(const TraceArgs& A, const DevView* sv, unsigned int g, int& v, int& i, int& j) {
    v = 0;
    for (int b = VT_MAX_VIEWS / 2; b; b >>= 1)   /* last view whose base is <= g */
        if (v + b < A.views.n && sv[v + b].rayBase <= g) v += b;
    const unsigned int local = g - sv[v].rayBase, tilesX = sv[v].tilesX, inv = sv[v].tilesXInv;
    const unsigned int rays = (unsigned int)(A.tile_w * A.tile_h);
    const bool pow2 = A.tile_shift >= 0;
    const unsigned int tile = pow2 ? local >> A.tile_shift : local / rays, lt = local - tile * rays;
    const unsigned int ti = inv ? __umulhi(tile, inv) : tile / tilesX, tj = tile - ti * tilesX;
    const unsigned int li = pow2 ? lt >> A.tile_w_shift : lt / (unsigned int)A.tile_w;
    i = (int)(ti * A.tile_h + li);
    j = (int)(tj * A.tile_w + (lt - li * A.tile_w));
    return i < sv[v].cam.H && j < sv[v].cam.W;
}

/* ray g's camera ray; false for tile padding */
__device__ __forceinline__ bool ray_of(const TraceArgs& A, const DevView* sv, unsigned int g, int& view, int& i, int& j,
                                       float3& dir, RayInv& r) {
    if (!decode_ray(A, sv, g, view, i, j)) return false;
    const DevCamera& C = sv[view].cam;
    dir = ray_dir(C.look, C.up, C.right, C.dist, C.h, C.w, C.ih, C.iw, i, j);
    r.o = C.pos; r.dx = 1 / dir.x; r.dy = 1 / dir.y; r.dz = 1 / dir.z;
    return true;
}

/* Sets up ray rec.ray for the literal search: from the root (fresh rays,
 * depth 0), from its saved stack, or, suspended by the 64-ary walk, from
 * the root passing over the candidates it has taken.  Returns RAY_RUNNING
 * when the ray has traversal to do, RAY_DONE when it is background already
 * (root miss), -1 for tile padding. */
template <bool SKIP>
__device__ int start_ray(const TraceArgs& A, const DevView* sv, const SuspRec& rec, Ray& R, Stk& st) {
    R.g = rec.ray;
    if (!ray_of(A, sv, R.g, R.view, R.i, R.j, R.dir, R.r)) return -1;
    R.rgba = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    R.hit = false; R.node = 0; R.brick = 0; R.t = -1.0f; R.n = f3(0, 0, 0);
    R.top = -1;
    R.lastSlot = -1;
    R.nskip = 0; R.tent = false; R.resumeSkips = false; R.taken = 0;
    if (rec.depth & VT_SUSP_WALK) {
        R.taken = rec.depth >> VT_SUSP_TAKEN_SHIFT;
    } else if (rec.depth > 0) {
        int nsk = 0;
        if (SKIP) {
            nsk = (int)((rec.depth >> 8) & 7u);
            R.nskip = nsk;
            R.tent = (rec.depth >> 11) & 1u;
            R.resumeSkips = nsk > 0 || R.tent;
            for (int e = 0; e < nsk; e++) st.sk[e] = A.ctl.pool_in[rec.off + e];
        }
        R.top = (int)(rec.depth & 255u) - 1;
        for (int e = 0; e <= R.top; e++) st.e[e] = A.ctl.pool_in[rec.off + nsk + e];
        return RAY_RUNNING;
    }
    const int N = 1 << A.oct.nLevels;
    float tn, tf;
    /* root test (src/Octree.cu:729) */
    if (A.oct.rootValid && slab(R.r, 0, 0, 0, N, N, N, &tn, &tf)) { R.top = 0; st.e[0] = make_entry(0, 0, 0, 0, 0); return RAY_RUNNING; }
    return RAY_DONE;   /* background */
}

/* count = false: a tentative hit (past set-aside candidates) is written
 * uncounted; the hit is counted once, when the pixel is final */
__device__ __forceinline__ void write_ray(const TraceArgs& A, const DevView* sv, const Ray& R, unsigned int* cnt,
                                          bool count = true) {
    const DevView& V = sv[R.view];
    const size_t id = (size_t)R.i * V.cam.W + R.j;
    if (R.hit && count) cnt[VT_C_HITS]++;
    if (V.rgba) V.rgba[id] = R.rgba;
    if (V.rgb8) {
        V.rgb8[3 * id] = to_u8(R.rgba.x);
        V.rgb8[3 * id + 1] = to_u8(R.rgba.y);
        V.rgb8[3 * id + 2] = to_u8(R.rgba.z);
    }
    if (R.view == 0) {
        if (A.out.node) A.out.node[id] = R.node;
        if (A.out.brick) A.out.brick[id] = R.brick;
        if (A.out.t) A.out.t[id] = R.t;
        if (A.out.n) { A.out.n[3 * id] = R.n.x; A.out.n[3 * id + 1] = R.n.y; A.out.n[3 * id + 2] = R.n.z; }
    }
}

template <int VTYPE, bool SLAB, bool SKIP>
__device__ __forceinline__ void suspend_ray(const TraceArgs& A, Ray& R, Stk& st, unsigned int* cnt) {
    cnt[VT_C_SUSPENDED]++;
    unsigned int q = atomicAdd(A.ctl.n_out, 1u);
    if (q >= A.ctl.out_cap) { atomicOr(A.ctl.err, VT_KERR_SUSPEND_FULL); return; }
    const unsigned int depth = (unsigned int)(R.top + 1), nsk = SKIP ? (unsigned int)R.nskip : 0u;
    unsigned long long off = atomicAdd(A.ctl.pool_used, (unsigned long long)(depth + nsk));
    SuspRec rec;
    rec.ray = R.g;
    if (off + depth + nsk <= A.ctl.pool_cap) {
        for (unsigned int e = 0; e < nsk; e++) A.ctl.pool_out[off + e] = st.sk[e];
        for (unsigned int e = 0; e < depth; e++) A.ctl.pool_out[off + nsk + e] = st.e[e];
        rec.depth = depth | (nsk << 8) | ((SKIP && R.tent ? 1u : 0u) << 11); rec.off = off;
    } else {
        /* pool full: the ray restarts from the root and finds the same first
         * hit; a tentative pixel is rewritten then, and counted once */
        rec.depth = 0; rec.off = 0;
    }
    A.ctl.out[q] = rec;
    if (SLAB && A.ctl.lookahead > 0) lookahead_requests<VTYPE>(A, R, st, cnt);
}

__device__ __forceinline__ void flush_counters(const TraceArgs& A, unsigned int* cnt) {
#pragma unroll
    for (int c = 0; c < VT_C_COUNT; c++) {
        unsigned int v = cnt[c];
        if (c == VT_C_MAXSTACK) {
            for (int off = 16; off; off >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, off));
            if ((threadIdx.x & 31) == 0 && v) atomicMax(&A.ctl.counters[c], (unsigned long long)v);
        } else {
            for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if ((threadIdx.x & 31) == 0 && v) atomicAdd(&A.ctl.counters[c], (unsigned long long)v);
        }
    }
}

/* The literal depth-first search for one ray, to its end.  sk: set-aside
 * candidates of a ray handed over by the walk.  False for tile padding. */
template <int VTYPE, bool SLAB, int U, bool SKIP>
__device__ __forceinline__ bool search_ray(const TraceArgs& A, const DevView* sv, const SuspRec& rec, int nskip,
                                           const unsigned long long* sk, unsigned int* cnt) {
    Stk st;
    Ray R;
    int s = start_ray<SKIP>(A, sv, rec, R, st);
    if (s < 0) return false;
    if (SKIP && nskip > 0) {
        R.nskip = nskip;
        for (int e = 0; e < nskip; e++) st.sk[e] = sk[e];
    }
    if (s == RAY_RUNNING) s = run_ray<VTYPE, SLAB, U, SKIP>(A, R, st, cnt);
    if (s == RAY_DONE) write_ray(A, sv, R, cnt);
    else if (SKIP && s == RAY_TENTATIVE) {
        write_ray(A, sv, R, cnt, false);
        suspend_ray<VTYPE, SLAB, SKIP>(A, R, st, cnt);
    } else if (s == RAY_SUSPENDED) suspend_ray<VTYPE, SLAB, SKIP>(A, R, st, cnt);
    else if (SKIP && s == RAY_DONE_WRITTEN) cnt[VT_C_HITS]++;   /* the tentative hit stands */
    return true;
}

/* The literal search in k_trace: rays whose 64-ary walk met coinciding or
 * non-finite plane products, and rays resumed with a saved stack.  Rare, so
 * it is kept out of line: its stack and its registers cost the others
 * nothing (inlined, a 1920x1080 frame without such rays 602 -> 648 us).
 * s_cnt: the CTA's counters in shared memory (each ray adding to the ones in
 * global memory, a frame of such rays took 8.45 ms instead of 1.33 ms). */
template <int VTYPE, bool SLAB, int U, bool SKIP>
__device__ __noinline__ void literal_ray(const TraceArgs& A, const DevView* sv, SuspRec rec, int nskip,
                                         const unsigned long long* sk, unsigned int* s_cnt) {
    unsigned int cnt[VT_C_COUNT];
#pragma unroll
    for (int c = 0; c < VT_C_COUNT; c++) cnt[c] = 0;
    search_ray<VTYPE, SLAB, U, SKIP>(A, sv, rec, nskip, sk, cnt);
#pragma unroll
    for (int c = 0; c < VT_C_COUNT; c++) {
        if (!cnt[c]) continue;
        if (c == VT_C_MAXSTACK) atomicMax(&s_cnt[c], cnt[c]);
        else atomicAdd(&s_cnt[c], cnt[c]);
    }
}

#define VT_TRACE_THREADS 32
#define VT_TRACE_CTAS 24

/* One ray of k_trace in flight. */
struct Trip {
    RayInv r;
    float3 dir;
    Walk w;
    int cx, cy, cz;            /* candidate last looked at */
    unsigned int g;            /* padded global ray index */
    int view, i, j;
    bool fresh;                /* the walk's current cell is still to be looked at */
    unsigned int taken;        /* candidates dealt with so far */
    unsigned int pidx; int slot;   /* brick of the last resident candidate (its page cannot change in a pass) */
    Crossing C;                /* a hit's crossing (refined and shaded when the ray is finished) */
    /* set-aside candidates (SKIP) */
    int nskip;
    bool tent, resumeSkips;    /* as Ray's */
    bool ended;                /* the walk is over; only set-aside candidates are left */
};
/* how a ray left the advance loop (besides RAY_*) */
enum { TRIP_MISS = 5, TRIP_LITERAL = 6 };

/* Candidate (R.cx, R.cy, R.cz), whose cell the ray crosses from product tn
 * to tf: brick lookup (lruCache::updateCube, src/lruCache.cu:177-291) and
 * march (src/rayCaster.cu:139-237).  CAND_MISSING when the brick is absent
 * (it is requested), CAND_HIT with the crossing in R.C. */
template <int VTYPE, bool SLAB, int U>
__device__ __forceinline__ int try_candidate(const TraceArgs& A, Trip& R, float tn, float tf, unsigned int* cnt) {
    const int Lo = A.oct.Lo, Lc = A.oct.Lc;
    const unsigned int bx = (unsigned)R.cx >> (Lo - Lc), by = (unsigned)R.cy >> (Lo - Lc), bz = (unsigned)R.cz >> (Lo - Lc);
    const unsigned int pidx = (bx << (2 * Lc)) | (by << Lc) | bz;
    if (SLAB && pidx != R.pidx) {
        const int slot = A.br.page[pidx];
        if (slot < 0) {
            if (slot == -1 || slot == VT_PAGE_SPECULATIVE) request_brick(A, pidx);
            cnt[VT_C_DEVMISSES]++;
            return CAND_MISSING;
        }
        R.pidx = pidx; R.slot = slot;
        A.br.stamp[slot] = A.br.pass;
    }
    cnt[VT_C_CANDIDATES]++;
    if (A.ctl.touched) {
        const int d = A.ctl.touch_shift / 3;   /* Lo - trace level */
        const unsigned long long n = (spread3((unsigned)R.cx >> d) << 2) | (spread3((unsigned)R.cy >> d) << 1) |
                                     spread3((unsigned)R.cz >> d);
        atomicOr(&A.ctl.touched[n >> 5], 1u << (n & 31));
    }
    Samp s;
    brick_sampler<VTYPE, SLAB>(A, bx, by, bz, R.slot, s);
    return march<VTYPE, SLAB, U>(s, R.r.o, R.dir, tn, max_steps(tn, tf), A.iso, R.C, &cnt[VT_C_SAMPLES]) ? CAND_HIT
                                                                                                        : CAND_EMPTY;
}

/* Sets up ray rec.ray: RAY_RUNNING (walk to do), TRIP_MISS (background),
 * TRIP_LITERAL, or -1 for tile padding. */
template <bool SKIP>
__device__ __forceinline__ int start_trip(const TraceArgs& A, const DevView* sv, const SuspRec& rec, Trip& R,
                                          PathNode* path, unsigned long long* sk) {
    R.g = rec.ray;
    R.pidx = 0xFFFFFFFFu; R.slot = 0;
    R.fresh = true; R.taken = 0;
    R.nskip = 0; R.tent = false; R.resumeSkips = false; R.ended = false;
    if (rec.depth && !(rec.depth & VT_SUSP_WALK)) return TRIP_LITERAL;   /* a saved stack */
    if (!ray_of(A, sv, R.g, R.view, R.i, R.j, R.dir, R.r)) return -1;
    if (rec.depth) {
        R.taken = rec.depth >> VT_SUSP_TAKEN_SHIFT;
        int nsk = 0;
        if (SKIP) {
            nsk = (int)((rec.depth >> 8) & 7u);
            R.nskip = nsk;
            R.tent = (rec.depth >> 11) & 1u;
            R.resumeSkips = nsk > 0 || R.tent;
            for (int e = 0; e < nsk; e++) sk[e] = A.ctl.pool_in[rec.off + e];
        }
        if (rec.depth & 255u) {
            const unsigned long long c = A.ctl.pool_in[rec.off + nsk];
            walk_at<VT_TRACE_THREADS>(A.oct.t64, R.r, (int)e_x(c), (int)e_y(c), (int)e_z(c), R.w, path);
        } else {
            R.ended = true;
        }
        return RAY_RUNNING;
    }
    if (!A.oct.rootValid) return TRIP_MISS;
    const int s = walk_root<VT_TRACE_THREADS>(A.oct.t64, R.r, R.w, path);
    return s == WALK_CANDIDATE ? RAY_RUNNING : s == WALK_END ? TRIP_MISS : TRIP_LITERAL;
}

/* Takes a running ray to its end: walk to the next candidate, march it,
 * until a hit, an absent brick or the end of the walk.  Set-aside candidates
 * as in run_ray. */
template <int VTYPE, bool SLAB, int U, bool SKIP>
__device__ __forceinline__ int advance_trip(const TraceArgs& A, Trip& R, PathNode* path, unsigned long long* sk,
                                            unsigned int* cnt) {
    if (SKIP) {
        while (R.resumeSkips) {
            if (R.nskip == 0) {
                R.resumeSkips = false;
                if (R.tent) return RAY_DONE_WRITTEN;
                if (R.ended) return TRIP_MISS;
                break;
            }
            R.cx = (int)e_x(sk[0]); R.cy = (int)e_y(sk[0]); R.cz = (int)e_z(sk[0]);
            const int sh = A.oct.nLevels - A.oct.Lo;
            float tn, tf;
            slab(R.r, R.cx << sh, R.cy << sh, R.cz << sh, (R.cx + 1) << sh, (R.cy + 1) << sh, (R.cz + 1) << sh, &tn, &tf);
            const int c = try_candidate<VTYPE, SLAB, U>(A, R, tn, tf, cnt);
            if (c == CAND_MISSING) return RAY_SUSPENDED;
            for (int k = 1; k < R.nskip; k++) sk[k - 1] = sk[k];
            R.nskip--;
            if (c == CAND_HIT) { R.nskip = 0; return RAY_DONE; }
        }
    }
    const int K = SKIP ? A.ctl.skip : 0;
    for (;;) {
        int budget = 0x7FFFFFFF;
        float tf;
        const int s = walk_next<VT_TRACE_THREADS>(A.oct.t64, R.r, R.w, path, R.fresh, budget, &tf, &cnt[VT_C_EXPANSIONS]);
        if (s == WALK_TIE) return TRIP_LITERAL;
        if (s == WALK_END) {
            if (SKIP && R.nskip > 0) { R.ended = true; return RAY_SUSPENDED; }
            return TRIP_MISS;
        }
        walk_cell(A.oct.t64, R.r, R.w, R.cx, R.cy, R.cz);
        const int c = try_candidate<VTYPE, SLAB, U>(A, R, R.w.tc < 0.0f ? 0.0f : R.w.tc, tf, cnt);
        if (c == CAND_MISSING) {
            if (!SKIP || R.nskip >= K) return RAY_SUSPENDED;   /* the candidate is the one to resume at */
            sk[R.nskip++] = make_entry(0, A.oct.Lo, R.cx, R.cy, R.cz);
        }
        R.taken++;
        R.fresh = false;
        if (c == CAND_HIT) return (!SKIP || R.nskip == 0) ? (int)RAY_DONE : (int)RAY_TENTATIVE;
    }
}

/* Speculative requests: walks on from a suspended ray's candidate (without
 * marching) and requests up to `lookahead` further absent bricks. */
__device__ __forceinline__ void lookahead_walk(const TraceArgs& A, Trip& R, PathNode* path) {
    const int Lo = A.oct.Lo, Lc = A.oct.Lc;
    int want = A.ctl.lookahead, budget = 256;
    unsigned int last = 0xFFFFFFFFu, entered = 0;
    bool fresh = true;
    while (want > 0 && budget-- > 0) {
        float tf;
        if (walk_next<VT_TRACE_THREADS>(A.oct.t64, R.r, R.w, path, fresh, budget, &tf, &entered) != WALK_CANDIDATE) break;
        walk_cell(A.oct.t64, R.r, R.w, R.cx, R.cy, R.cz);
        const unsigned int pidx = (((unsigned)R.cx >> (Lo - Lc)) << (2 * Lc)) | (((unsigned)R.cy >> (Lo - Lc)) << Lc) |
                                  ((unsigned)R.cz >> (Lo - Lc));
        if (pidx != last && A.br.page[pidx] == -1) { request_brick(A, pidx, true); want--; }
        last = pidx;
        fresh = false;
    }
}

template <bool SLAB, bool SKIP>
__device__ __forceinline__ void suspend_trip(const TraceArgs& A, Trip& R, PathNode* path,
                                             const unsigned long long* sk, unsigned int* cnt) {
    cnt[VT_C_SUSPENDED]++;
    unsigned int q = atomicAdd(A.ctl.n_out, 1u);
    if (q >= A.ctl.out_cap) { atomicOr(A.ctl.err, VT_KERR_SUSPEND_FULL); return; }
    const bool more = !SKIP || !(R.tent || R.ended);   /* a candidate to resume the walk at */
    const unsigned int depth = more ? 1u : 0u, nsk = SKIP ? (unsigned int)R.nskip : 0u;
    unsigned long long off = atomicAdd(A.ctl.pool_used, (unsigned long long)(depth + nsk));
    SuspRec rec;
    rec.ray = R.g;
    if (off + depth + nsk <= A.ctl.pool_cap) {
        for (unsigned int e = 0; e < nsk; e++) A.ctl.pool_out[off + e] = sk[e];
        if (more) {
            /* the walk's own cell: R.cx.. is a set-aside candidate where that one's brick is absent once more */
            int x, y, z;
            walk_cell(A.oct.t64, R.r, R.w, x, y, z);
            A.ctl.pool_out[off + nsk] = make_entry(0, A.oct.Lo, x, y, z);
        }
        rec.depth = depth | (nsk << 8) | ((SKIP && R.tent ? 1u : 0u) << 11) | VT_SUSP_WALK |
                    (R.taken << VT_SUSP_TAKEN_SHIFT);
        rec.off = off;
    } else {
        /* pool full: as suspend_ray */
        rec.depth = 0; rec.off = 0;
    }
    A.ctl.out[q] = rec;
    if (SLAB && more && A.ctl.lookahead > 0) lookahead_walk(A, R, path);
}

/* A ray that left advance_trip: shades a hit (all lanes of a warp that have
 * one together) and writes the pixel, suspends the ray, or hands it to the
 * literal search. */
template <int VTYPE, bool SLAB, int U, bool SKIP>
__device__ __forceinline__ void finish_trip(const TraceArgs& A, const DevView* sv, Trip& R, PathNode* path,
                                            const unsigned long long* sk, int s, unsigned int* cnt) {
    if (s == RAY_DONE || s == RAY_TENTATIVE || s == TRIP_MISS) {
        Ray P;
        P.rgba = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        P.hit = false; P.node = 0; P.brick = 0; P.t = -1.0f; P.n = f3(0, 0, 0);
        P.view = R.view; P.i = R.i; P.j = R.j;
        if (s != TRIP_MISS) {
            const unsigned int x = R.cx, y = R.cy, z = R.cz, d = A.oct.Lo - A.oct.Lc;
            Samp sm;
            brick_sampler<VTYPE, SLAB>(A, x >> d, y >> d, z >> d, R.slot, sm);
            P.r.o = R.r.o; P.dir = R.dir;
            const float3 X = refine_hit<VTYPE, SLAB, false>(sm, R.dir, R.C, A.iso, A.refine, &cnt[VT_C_SAMPLES]);
            shade_hit<VTYPE, SLAB, false>(A, P, sm, X, x, y, z, x >> d, y >> d, z >> d, cnt);
        }
        write_ray(A, sv, P, cnt, s != RAY_TENTATIVE);
    }
    if (s == RAY_TENTATIVE) R.tent = true;
    if (s == RAY_SUSPENDED || (SKIP && s == RAY_TENTATIVE)) suspend_trip<SLAB, SKIP>(A, R, path, sk, cnt);
    else if (SKIP && s == RAY_DONE_WRITTEN) cnt[VT_C_HITS]++;   /* the tentative hit stands */
}

/* record of a ray for the literal search: as it came in (a saved stack), or
 * from the root past the candidates taken */
__device__ __forceinline__ SuspRec literal_rec(const SuspRec& in, const Trip& R) {
    SuspRec rec = in;
    if (!in.depth || (in.depth & VT_SUSP_WALK)) rec.depth = VT_SUSP_WALK | (R.taken << VT_SUSP_TAKEN_SHIFT);
    return rec;
}

/* adds a warp's counters to the CTA's */
__device__ __forceinline__ void warp_counters(unsigned int* s_cnt, const unsigned int* cnt) {
#pragma unroll
    for (int c = 0; c < VT_C_COUNT; c++) {
        const unsigned int v = c == VT_C_MAXSTACK ? __reduce_max_sync(0xffffffffu, cnt[c]) : __reduce_add_sync(0xffffffffu, cnt[c]);
        if ((threadIdx.x & 31) == 0 && v) {
            if (c == VT_C_MAXSTACK) atomicMax(&s_cnt[c], v);
            else atomicAdd(&s_cnt[c], v);
        }
    }
}

/* One ray per lane, `group` rays a warp (a tile of the screen); a warp's rays
 * walk, march and, at the end, shade together.  Bound by instruction issue
 * and divergence (1920x1080 frame of the 512^3 blobs, warm: two thirds of
 * the issue slots, 15 of 32 lanes per instruction) and, on small frames, by
 * the latency of the slowest warp; of an average warp's time the walk takes
 * 57 %, the march 26 %, set-up and shading the rest.  One warp a CTA, so
 * that a warp's place is free for the next tile when its own rays are done
 * (CTAs of 128, 64, 32 threads: 3.48, 3.37, 3.35 ms for 16 mixed views, 563,
 * 557, 557 us for that frame), 24 of them per SM (80 registers; 20, 24, 28,
 * 32 warps: 594, 574, 580, 601 us).  Against the binary depth-first search
 * it replaced: 767 -> 557 us there, 4.18 -> 3.35 ms for the views, 769 -> 390
 * us for a 1277x719 uint8 frame with bisection, 94 -> 40 us for a 96x96
 * frame. */
template <int VTYPE, bool SLAB, int U, bool SKIP>
__global__ void __launch_bounds__(VT_TRACE_THREADS, VT_TRACE_CTAS) k_trace(const __grid_constant__ TraceArgs A) {
    __shared__ PathNode s_path[VT_TREE64_LEVELS * VT_TRACE_THREADS];   /* per thread: the node entered at each level */
    __shared__ unsigned int s_cnt[VT_C_COUNT];
    PathNode* const path = s_path + threadIdx.x;
    if (threadIdx.x < VT_C_COUNT) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    const DevView* const sv = A.views.v;
    const unsigned int nItems =
        A.ctl.in ? (A.ctl.n_in_dev ? min(*A.ctl.n_in_dev, A.ctl.n_in) : A.ctl.n_in) : A.views.totalRays;
    const unsigned int lane = threadIdx.x & 31;
    const unsigned int w = (unsigned int)(blockIdx.x * (VT_TRACE_THREADS / 32) + (threadIdx.x >> 5)) * A.group + lane;
    unsigned int cnt[VT_C_COUNT];
#pragma unroll
    for (int c = 0; c < VT_C_COUNT; c++) cnt[c] = 0;
    unsigned long long sk[VT_SKIP_MAX];
    Trip R;
    SuspRec rec;
    int s = -1;
    if (lane < A.group && w < nItems) {
        if (A.ctl.in) rec = A.ctl.in[w];
        else { rec.ray = w; rec.depth = 0; }
        s = start_trip<SKIP>(A, sv, rec, R, path, sk);
        if (s >= 0 && !A.ctl.in) cnt[VT_C_RAYS]++;
        if (s == RAY_RUNNING) s = advance_trip<VTYPE, SLAB, U, SKIP>(A, R, path, sk, cnt);
    }
    __syncwarp();
    if (s >= 0) finish_trip<VTYPE, SLAB, U, SKIP>(A, sv, R, path, sk, s, cnt);
    if (s == TRIP_LITERAL) literal_ray<VTYPE, SLAB, U, SKIP>(A, sv, literal_rec(rec, R), R.nskip, sk, s_cnt);
    __syncwarp();
    warp_counters(s_cnt, cnt);
    __syncthreads();
    if (threadIdx.x < VT_C_COUNT) {
        const int c = threadIdx.x;
        unsigned int v = s_cnt[c];
        if (SLAB && c == VT_C_DEVHITS) v = s_cnt[VT_C_CANDIDATES];
        if (c == VT_C_MAXSTACK) v = max(v, s_cnt[VT_C_CANDIDATES] ? (unsigned int)(A.oct.Lo + 1) >> 1 : 0u);
        if (v && c == VT_C_MAXSTACK) atomicMax(&A.ctl.counters[c], (unsigned long long)v);
        else if (v) atomicAdd(&A.ctl.counters[c], (unsigned long long)v);
    }
}

/* The literal search, one ray per thread: frames whose rays all need it
 * (TraceArgs::literal) and the rays left over after wavefront rounds.  Eight
 * 128-thread CTAs per SM: it is bound by latency, and in k_trace, with 24
 * warps an SM, the same frames take a fifth longer (1920x1080 from a lattice
 * point of the 512^3 blobs 1699 -> 1292 us, of the 401x290x333 uint8 fractal
 * 1328 -> 1035 us; the 64-ary walk next to these points: 717 and 377 us). */
template <int VTYPE, bool SLAB, bool SKIP>
__global__ void __launch_bounds__(128, 8) k_literal(const __grid_constant__ TraceArgs A) {
    unsigned int cnt[VT_C_COUNT];
#pragma unroll
    for (int c = 0; c < VT_C_COUNT; c++) cnt[c] = 0;
    const unsigned int nItems =
        A.ctl.in ? (A.ctl.n_in_dev ? min(*A.ctl.n_in_dev, A.ctl.n_in) : A.ctl.n_in) : A.views.totalRays;
    const unsigned int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w < nItems) {
        SuspRec rec;
        if (A.ctl.in) rec = A.ctl.in[w];
        else { rec.ray = w; rec.depth = 0; }
        if (search_ray<VTYPE, SLAB, 1, SKIP>(A, A.views.v, rec, 0, nullptr, cnt) && !A.ctl.in) cnt[VT_C_RAYS]++;
    }
    __syncwarp();
    flush_counters(A, cnt);
}

/* ---- wavefront passes ------------------------------------------------- */
/* Traversal round: each input ray (a fresh ray of the pass, a ray resumed
 * from the last pass, or a ray whose candidate missed in the last round)
 * walks its DFS (the same expansions as run_ray) to its next candidate.  An
 * absent brick suspends the ray as in the one-kernel pass; a resident one
 * pops the candidate, saves the ray's remaining stack as a wait record and
 * queues a march item, counted into its slot's bin (the first item of a
 * slot lists the slot as touched).  Where the wait pool is full the ray
 * marches the candidate itself, as the one-kernel pass does. */
template <int VTYPE>
__global__ void __launch_bounds__(128, 8) k_wf_traverse(TraceArgs A, WaveRound W) {
    __shared__ DevView sv[VT_MAX_VIEWS];
    for (int k = threadIdx.x; k < A.views.n; k += blockDim.x) sv[k] = A.views.v[k];
    __syncthreads();
    unsigned int cnt[VT_C_COUNT];
#pragma unroll
    for (int c = 0; c < VT_C_COUNT; c++) cnt[c] = 0;
    const unsigned int nItems =
        A.ctl.in ? (A.ctl.n_in_dev ? min(*A.ctl.n_in_dev, A.ctl.n_in) : A.ctl.n_in) : A.views.totalRays;
    const DevOctree& O = A.oct;
    const int Lo = O.Lo, Lc = O.Lc, nLevels = O.nLevels, dimO = 1 << (nLevels - Lo);
    Stk st;
    Ray R;
    for (unsigned int w = blockIdx.x * blockDim.x + threadIdx.x; w < nItems; w += gridDim.x * blockDim.x) {
        SuspRec rec0;
        if (A.ctl.in) rec0 = A.ctl.in[w];
        else { rec0.ray = w; rec0.depth = 0; }
        const int s0 = start_ray<false>(A, sv, rec0, R, st);
        if (s0 < 0) continue;
        if (!A.ctl.in) cnt[VT_C_RAYS]++;
        if (s0 == RAY_DONE) { write_ray(A, sv, R, cnt); continue; }
        for (;;) {
            bool stop = false;
            for (;;) {   /* expand until a candidate is on top */
                if (R.top < 0) { stop = true; break; }
                const unsigned long long e = st.e[R.top];
                if (e_level(e) == Lo) break;
                R.top--;
                cnt[VT_C_EXPANSIONS]++;
                if (!expand(A, R.r, st, R.top, e, cnt, true)) { stop = true; break; }
            }
            if (stop) { write_ray(A, sv, R, cnt); break; }   /* exhausted (or stack overflow, flagged) */
            if (R.taken) { R.taken--; R.top--; continue; }
            const unsigned long long ent = st.e[R.top];
            const unsigned int x = e_x(ent), y = e_y(ent), z = e_z(ent);
            const unsigned int bx = x >> (Lo - Lc), by = y >> (Lo - Lc), bz = z >> (Lo - Lc);
            const unsigned int pidx = (bx << (2 * Lc)) | (by << Lc) | bz;
            const int slot = A.br.page[pidx];
            if (slot < 0) {
                if (slot == -1 || slot == VT_PAGE_SPECULATIVE) request_brick(A, pidx);
                cnt[VT_C_DEVMISSES]++;
                suspend_ray<VTYPE, true, false>(A, R, st, cnt);   /* the candidate stays on the stack */
                break;
            }
            cnt[VT_C_CANDIDATES]++;
            cnt[VT_C_DEVHITS]++;
            if (slot != R.lastSlot) { A.br.stamp[slot] = A.br.pass; R.lastSlot = slot; }
            const int mbx = (int)(x << (nLevels - Lo)), mby = (int)(y << (nLevels - Lo)), mbz = (int)(z << (nLevels - Lo));
            float tn, tf;
            R.top--;
            if (!slab(R.r, mbx, mby, mbz, mbx + dimO, mby + dimO, mbz + dimO, &tn, &tf)) continue;   /* empty */
            const unsigned int depth = (unsigned int)(R.top + 1);
            const unsigned int q = atomicAdd(W.n_wait, 1u);
            const unsigned long long off = atomicAdd(W.pool_wait_used, (unsigned long long)depth);
            if (q < W.wait_cap && off + depth <= W.pool_wait_cap) {
                for (unsigned int e = 0; e < depth; e++) W.pool_wait[off + e] = st.e[e];
                SuspRec rec;
                rec.ray = R.g; rec.depth = depth; rec.off = off;
                W.wait[q] = rec;
                const unsigned int i = atomicAdd(W.n_items, 1u);
                if (i >= W.items_cap) { atomicOr(A.ctl.err, VT_KERR_WAVE); break; }   /* cannot happen: one item a ray */
                const unsigned int rank = atomicAdd(&W.binCount[slot], 1u);
                if (rank == 0) W.touched[atomicAdd(W.n_touched, 1u)] = (unsigned int)slot;
                MarchItem it;
                it.entry = ent; it.rec = q; it.slot = slot; it.tn = tn; it.maxStep = max_steps(tn, tf);
                it.g = R.g; it.rank = rank; it.dx = R.dir.x; it.dy = R.dir.y; it.dz = R.dir.z; it.pad = 0;
                W.items[i] = it;
                break;
            }
            /* no room to wait: march here */
            Samp sm;
            brick_sampler<VTYPE, true>(A, bx, by, bz, slot, sm);
            Crossing C;
            if (march<VTYPE, true, 1>(sm, R.r.o, R.dir, tn, max_steps(tn, tf), A.iso, C,
                                      &cnt[VT_C_SAMPLES])) {
                const float3 X = refine_hit<VTYPE, true, false>(sm, R.dir, C, A.iso, A.refine, &cnt[VT_C_SAMPLES]);
                shade_hit<VTYPE, true, false>(A, R, sm, X, x, y, z, bx, by, bz, cnt);
                write_ray(A, sv, R, cnt);
                break;
            }
        }
    }
    flush_counters(A, cnt);
}

/* Bin offsets: an exclusive prefix sum of the touched slots' counts (one
 * CTA; a few tens of thousands of slots per round). */
__global__ void __launch_bounds__(1024) k_wf_scan(WaveRound W) {
    __shared__ unsigned int part[1024];
    const unsigned int nT = *W.n_touched;
    const unsigned int per = (nT + 1023u) / 1024u;
    const unsigned int b = threadIdx.x * per, e = min(nT, b + per);
    unsigned int sum = 0;
    for (unsigned int i = b; i < e; i++) sum += W.binCount[W.touched[i]];
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const unsigned int v = (int)threadIdx.x >= o ? part[threadIdx.x - o] : 0u;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    unsigned int base = threadIdx.x ? part[threadIdx.x - 1] : 0u;
    for (unsigned int i = b; i < e; i++) {
        const unsigned int sl = W.touched[i];
        W.binStart[sl] = base;
        base += W.binCount[sl];
    }
}

/* Items into slot order. */
__global__ void k_wf_scatter(WaveRound W) {
    const unsigned int n = min(*W.n_items, W.items_cap);
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const MarchItem it = W.items[i];
        const unsigned int d = W.binStart[it.slot] + it.rank;
        if (d < W.items_cap) W.sorted[d] = it;
    }
}

/* March round: one touched slot at a time per CTA.  One thread stages the
 * slot's brick (edge + 2 inc voxels a side, contiguous) into shared memory
 * with a single bulk copy (cp.async.bulk, the tensor memory accelerator's
 * non-tensor form) completing on an mbarrier; every thread then marches
 * items of that slot from shared memory (src/rayCaster.cu:166-250, the same
 * arithmetic as the one-kernel pass).  A hit shades and writes the pixel; a
 * miss sends the ray's wait record on to the next traversal round, or, with
 * nothing left on its stack, writes the background.  Waits are bounded: past
 * the limit the CTA flags VT_KERR_STAGE and stops. */
template <int VTYPE>
__global__ void __launch_bounds__(128) k_wf_march(TraceArgs A, WaveRound W, unsigned int slotBytes) {
    __shared__ DevView sv[VT_MAX_VIEWS];
    __shared__ __align__(8) unsigned long long mbar;
    extern __shared__ __align__(128) unsigned char wf_brick[];
    for (int k = threadIdx.x; k < A.views.n; k += blockDim.x) sv[k] = A.views.v[k];
    const uint32_t mb = (uint32_t)__cvta_generic_to_shared(&mbar);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(mb), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    __syncthreads();
    unsigned int cnt[VT_C_COUNT];
#pragma unroll
    for (int c = 0; c < VT_C_COUNT; c++) cnt[c] = 0;
    const DevOctree& O = A.oct;
    const int Lo = O.Lo, Lc = O.Lc, sh = O.nLevels - O.Lc;
    const DevBricks& B = A.br;
    const unsigned int nT = *W.n_touched;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(wf_brick);
    uint32_t phase = 0;
    for (unsigned int t = blockIdx.x; t < nT; t += gridDim.x) {
        const unsigned int slot = W.touched[t];
        const unsigned int count = W.binCount[slot], start = W.binStart[slot];
        if (threadIdx.x == 0) {
            /* the last slot's reads (generic proxy) before this copy's writes (async proxy) */
            asm volatile("fence.proxy.async.shared::cta;");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(mb), "r"(slotBytes) : "memory");
            const char* src = (const char*)B.slab + (size_t)slot * slotBytes;
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         :: "r"(dst), "l"(src), "r"(slotBytes), "r"(mb) : "memory");
        }
        uint32_t done = 0;
        for (long long it = 0; it < (1ll << 22) && !done; it++) {
            asm volatile("{\n\t.reg .pred P1;\n\t"
                         "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
                         "selp.b32 %0, 1, 0, P1;\n\t}"
                         : "=r"(done) : "r"(mb), "r"(phase) : "memory");
        }
        phase ^= 1u;
        if (__syncthreads_or(!done)) {
            if (threadIdx.x == 0) atomicOr(A.ctl.err, VT_KERR_STAGE);
            break;
        }
        for (unsigned int k = threadIdx.x; k < count && start + k < W.items_cap; k += blockDim.x) {
            const MarchItem it = W.sorted[start + k];
            Ray R;
            decode_ray(A, sv, it.g, R.view, R.i, R.j);
            R.g = it.g;
            R.dir = f3(it.dx, it.dy, it.dz);
            R.r.o = sv[R.view].cam.pos;
            R.hit = false;
            const unsigned int x = e_x(it.entry), y = e_y(it.entry), z = e_z(it.entry);
            const unsigned int bx = x >> (Lo - Lc), by = y >> (Lo - Lc), bz = z >> (Lo - Lc);
            Samp sm;
            sm.base = wf_brick;
            sm.sx = B.D * B.D; sm.sy = B.D;
            sm.ox = (float)((int)(bx << sh) - B.inc); sm.oy = (float)((int)(by << sh) - B.inc);
            sm.oz = (float)((int)(bz << sh) - B.inc);
            sm.h = (float)(B.D - 2);
            Crossing C;
            if (march<VTYPE, true, 1, true>(sm, R.r.o, R.dir, it.tn, it.maxStep, A.iso, C, &cnt[VT_C_SAMPLES])) {
                const float3 X = refine_hit<VTYPE, true, true>(sm, R.dir, C, A.iso, A.refine, &cnt[VT_C_SAMPLES]);
                shade_hit<VTYPE, true, true>(A, R, sm, X, x, y, z, bx, by, bz, cnt);
                write_ray(A, sv, R, cnt);
            } else {
                const SuspRec rec = W.wait[it.rec];
                if (rec.depth == 0) {   /* nothing left on its stack: background */
                    R.rgba = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
                    R.node = 0; R.brick = 0; R.t = -1.0f; R.n = f3(0, 0, 0);
                    write_ray(A, sv, R, cnt);
                } else {
                    W.next[atomicAdd(W.n_next, 1u)] = rec;
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) W.binCount[slot] = 0;   /* the bins start empty next round */
    }
    flush_counters(A, cnt);
}

/* cuda_updateRays (src/Camera.cu:39-74) */
__global__ void k_rays(DevCamera C, float* dirs) {
    long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)C.W * C.H) return;
    int i = (int)(id / C.W), j = (int)(id % C.W);
    float3 d = ray_dir(C.look, C.up, C.right, C.dist, C.h, C.w, C.ih, C.iw, i, j);
    dirs[3 * id] = d.x; dirs[3 * id + 1] = d.y; dirs[3 * id + 2] = d.z;
}

/* cuda_rayCasterCube (src/rayCaster.cu:267-357) */
__device__ __forceinline__ float cube_get(const float* c, int D, long long total, int x, int y, int z) {
    long long i = (long long)z + (long long)y * D + (long long)x * D * D;
    if (i < 0 || i >= total) return 0.0f;   /* outside the allocation */
    return __ldg(c + i);
}
/* Trilinear sample; where all eight taps lie inside the brick (the float
 * test is false for NaN), one address and seven offsets, else the
 * reference's linear addressing tap by tap.  h: largest first tap of the
 * short way (negative: never, a brick of 2^31 voxels or more). */
__device__ __forceinline__ float cube_interp(const float* c, int D, long long total, float h, int3 mb, float3 p) {
    float rx, ry, rz;
    const float px = split_pos(p.x, &rx), py = split_pos(p.y, &ry), pz = split_pos(p.z, &rz);
    const float fx = rx - (float)mb.x, fy = ry - (float)mb.y, fz = rz - (float)mb.z;
    float v000, v001, v010, v011, v100, v101, v110, v111;
    if (fminf(fminf(fx, fy), fz) >= 0.0f && fmaxf(fmaxf(fx, fy), fz) <= h && fx == fx && fy == fy && fz == fz) {
        const int b = (__float_as_int(fx + VT_2P23) - VT_2P23_BITS) * D * D + (__float_as_int(fy + VT_2P23) - VT_2P23_BITS) * D +
                      (__float_as_int(fz + VT_2P23) - VT_2P23_BITS);
        const float *p00 = c + b, *p01 = p00 + D, *p10 = p00 + D * D, *p11 = p10 + D;
        v000 = __ldg(p00); v001 = __ldg(p00 + 1); v010 = __ldg(p01); v011 = __ldg(p01 + 1);
        v100 = __ldg(p10); v101 = __ldg(p10 + 1); v110 = __ldg(p11); v111 = __ldg(p11 + 1);
    } else {
        const int x0 = f2i(fx), y0 = f2i(fy), z0 = f2i(fz), x1 = x0 + 1, y1 = y0 + 1, z1 = z0 + 1;
        v000 = cube_get(c, D, total, x0, y0, z0); v001 = cube_get(c, D, total, x0, y0, z1);
        v010 = cube_get(c, D, total, x0, y1, z0); v011 = cube_get(c, D, total, x0, y1, z1);
        v100 = cube_get(c, D, total, x1, y0, z0); v101 = cube_get(c, D, total, x1, y0, z1);
        v110 = cube_get(c, D, total, x1, y1, z0); v111 = cube_get(c, D, total, x1, y1, z1);
    }
    float c00 = v000 * (1.0f - px) + v100 * px;
    float c01 = v001 * (1.0f - px) + v101 * px;
    float c10 = v010 * (1.0f - px) + v110 * px;
    float c11 = v011 * (1.0f - px) + v111 * px;
    float c0 = c00 * (1.0f - py) + c10 * py;
    float c1 = c01 * (1.0f - py) + c11 * py;
    return c0 * (1.0f - pz) + c1 * pz;
}
/* One ray per thread, an 8 x 4 tile of pixels per warp.  Bound by the
 * samples' instructions and divergence; one address per sample and square
 * tiles instead of 64-bit addresses with two tests a tap and rows of pixels:
 * 512 x 512 pixels of a 32^3 brick 55 -> 31 us a call. */
__global__ void k_cube(DevCamera C, const float* cube, int3 pmin, int3 cdim, int3 cinc, float iso,
                       float3 light, float4* rgba) {
    const int lane = threadIdx.x & 31;
    const unsigned int tilesX = (unsigned int)(C.W + 7) / 8;
    const unsigned int tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const long long i = (long long)(tile / tilesX) * 4 + (lane >> 3);
    const int j = (int)(tile % tilesX * 8) + (lane & 7);
    if (i >= C.H || j >= C.W) return;
    const long long tid = i * C.W + j;
    float3 ray = ray_dir(C.look, C.up, C.right, C.dist, C.h, C.w, C.ih, C.iw, (int)i, j);
    RayInv r; r.o = C.pos; r.dx = 1 / ray.x; r.dy = 1 / ray.y; r.dz = 1 / ray.z;
    int3 mb = pmin;
    const int D = cdim.x + 2 * cinc.x;
    const long long total = (long long)(cdim.x + 2 * cinc.x) * (cdim.y + 2 * cinc.y) * (cdim.z + 2 * cinc.z);
    /* taps up to D - 1 on every axis stay inside a brick that is D on every axis */
    const bool cubic = cdim.y + 2 * cinc.y == D && cdim.z + 2 * cinc.z == D && total < (1ll << 31);
    const float h = cubic ? (float)(D - 2) : -1.0f;
    float tn, tf;
    bool hit = false;
    float3 Xnew = f3(0, 0, 0);
    if (slab(r, mb.x, mb.y, mb.z, mb.x + cdim.x, mb.y + cdim.y, mb.z + cdim.z, &tn, &tf)) {
        mb.x -= cinc.x; mb.y -= cinc.y; mb.z -= cinc.z;
        float3 Xnear = add(C.pos, mul(ray, tn));
        float3 Xfar = Xnear;
        Xnew = Xnear;
        bool primera = true;
        float ant = 0.0f, sig = 0.0f;
        float steps = 0;
        float3 vStep = mul(ray, 0.5f);
        float maxStep = (tf - tn) * 2.0f;   /* (tfar-tnear)/0.5, an exact doubling */
        while (steps <= maxStep) {
            if (primera) {
                primera = false;
                ant = cube_interp(cube, D, total, h, mb, Xnear);
                Xfar = Xnear;
            } else {
                sig = cube_interp(cube, D, total, h, mb, Xnear);
                if ((((iso - ant) < 0.0f) && ((iso - sig) < 0.0f)) ||
                    (((iso - ant) > 0.0f) && ((iso - sig) > 0.0f))) {
                    ant = sig;
                    Xfar = Xnear;
                } else {
                    float a = (iso - ant) / (sig - ant);
                    Xnew = add(mul(Xfar, 1.0f - a), mul(Xnear, a));
                    hit = true;
                    steps = maxStep;
                }
            }
            Xnear = add(Xnear, vStep);
            steps++;
        }
    }
    float4 out = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    if (hit) {
        float gx = (cube_interp(cube, D, total, h, mb, f3(Xnew.x - 1.0f, Xnew.y, Xnew.z)) -
                    cube_interp(cube, D, total, h, mb, f3(Xnew.x + 1.0f, Xnew.y, Xnew.z))) / 2.0f;
        float gy = (cube_interp(cube, D, total, h, mb, f3(Xnew.x, Xnew.y - 1.0f, Xnew.z)) -
                    cube_interp(cube, D, total, h, mb, f3(Xnew.x, Xnew.y + 1.0f, Xnew.z))) / 2.0f;
        float gz = (cube_interp(cube, D, total, h, mb, f3(Xnew.x, Xnew.y, Xnew.z - 1.0f)) -
                    cube_interp(cube, D, total, h, mb, f3(Xnew.x, Xnew.y, Xnew.z + 1.0f))) / 2.0f;
        float3 n = normalize(f3(gx, gy, gz));
        float3 l = normalize(sub(Xnew, light));
        float dif = fabsf(dot(n, l));
        float a = Xnew.y / (float)cdim.y;
        out = make_float4((1 - a) * dif, a * dif, 0.0f * dif, 1.0f);
    }
    rgba[tid] = out;
}

/* Copies a host-visible (mapped) volume into the zero-padded device copy. */
template <int VTYPE>
__global__ void k_fill_dense(void* dst, const void* src, long long nx, long long ny, long long nz, int P,
                             long long ey, long long ez) {
    long long row = blockIdx.x;   /* one (x,y) row per block */
    long long x = row / ny, y = row % ny;
    long long dbase = ((x + P) * ey + (y + P)) * ez + P;
    long long sbase = (x * ny + y) * nz;
    for (long long z = threadIdx.x; z < nz; z += blockDim.x) {
        if (VTYPE == 0) ((float*)dst)[dbase + z] = ((const float*)src)[sbase + z];
        else ((unsigned char*)dst)[dbase + z] = ((const unsigned char*)src)[sbase + z];
    }
}

/* Learned prefetch: one thread per leaf brick (page index); its coarse
 * node at `level` is the brick's coordinates shifted by levelCubes - level,
 * Morton-ordered like the trace log's bits.  Absent pages of predicted
 * nodes go to -3 (requested speculatively) and into the list; past the
 * list's capacity a page goes back to absent. */
__global__ void k_predict_requests(int* page, const unsigned int* leafPages, int nLeaf, const float* probs, int ncams,
                                   int level, int Lc, float thr, unsigned int* list, unsigned int* count,
                                   unsigned int cap) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nLeaf) return;
    const unsigned int p = leafPages[i];
    const unsigned int m = (1u << Lc) - 1u, sh = (unsigned int)(Lc - level);
    const unsigned int bx = p >> (2 * Lc), by = (p >> Lc) & m, bz = p & m;
    const unsigned long long node = (spread3(bx >> sh) << 2) | (spread3(by >> sh) << 1) | spread3(bz >> sh);
    const long long nodes = 1ll << (3 * level);
    float pm = 0.0f;
    for (int c = 0; c < ncams; c++) pm = fmaxf(pm, __ldg(probs + (long long)c * nodes + (long long)node));
    if (!(pm > thr) || page[p] != -1) return;
    if (atomicCAS(&page[p], -1, VT_PAGE_SPECULATIVE) != -1) return;
    const unsigned int q = atomicAdd(count, 1u);
    if (q < cap) list[q] = p;
    else atomicCAS(&page[p], VT_PAGE_SPECULATIVE, -1);
}

}  // namespace vt

using namespace vt;

cudaError_t vt_launch_predict_requests(int* page, const unsigned int* leafPages, int nLeaf, const float* probs,
                                       int ncams, int level, int Lc, float thr, unsigned int* list,
                                       unsigned int* count, unsigned int cap, cudaStream_t s) {
    if (nLeaf <= 0) return cudaSuccess;
    k_predict_requests<<<(nLeaf + 255) / 256, 256, 0, s>>>(page, leafPages, nLeaf, probs, ncams, level, Lc, thr, list,
                                                          count, cap);
    return cudaGetLastError();
}

cudaError_t vt_launch_trace(const TraceArgs& a0, bool slabMode, cudaStream_t s) {
    const unsigned int items = a0.ctl.in ? a0.ctl.n_in : a0.views.totalRays;
    if (items == 0) return cudaSuccess;
    if (a0.views.n < 1 || a0.views.n > VT_MAX_VIEWS) return cudaErrorInvalidValue;
    TraceArgs a = a0;
    /* a full warp a tile, unless that leaves the GPU short of warps: then
     * fewer rays a warp, which diverge less.  A warp's time is the sum of its
     * lanes' separate turns, so on a 96x96 frame (288 full warps for 3552
     * places) pass 0 took 74, 75, 70, 68, 63, 62 us with 32, 16, 8, 4, 2, 1
     * rays a warp; the rule takes 2 there.  Later passes have no more rays
     * than earlier ones, so records of k_trace's walk never come to
     * k_literal, which reads saved stacks only. */
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const unsigned int places = (unsigned int)sms * VT_TRACE_CTAS * (VT_TRACE_THREADS / 32);
    a.group = 32;
    while (a.group > 1 && items / a.group < places) a.group >>= 1;
    const unsigned long long warps = (items + (unsigned long long)a.group - 1) / a.group;
    const unsigned int blocks = (unsigned int)((warps + VT_TRACE_THREADS / 32 - 1) / (VT_TRACE_THREADS / 32));
    /* setting absent bricks aside is compiled into its own kernels, so the
     * in-order traversal keeps its registers; it needs bricks (slab mode)
     * and is off while a trace is logged */
    const bool skip = slabMode && a.ctl.skip > 0 && !a.ctl.touched;
    if (a.literal && a.group == 32) {   /* few rays are better off spread over k_trace's warps */
        const unsigned int b = (unsigned int)((items + 127ull) / 128);
#define VT_LITERAL(V) \
    { if (slabMode && skip) k_literal<V, true, true><<<b, 128, 0, s>>>(a); \
      else if (slabMode) k_literal<V, true, false><<<b, 128, 0, s>>>(a); \
      else k_literal<V, false, false><<<b, 128, 0, s>>>(a); }
        if (a.br.vtype == 0) VT_LITERAL(0) else VT_LITERAL(1)
#undef VT_LITERAL
        return cudaGetLastError();
    }
#define VT_LAUNCH_U(V, S, K)                                                     \
    switch (a.unroll) {                                                          \
        case 2: k_trace<V, S, 2, K><<<blocks, VT_TRACE_THREADS, 0, s>>>(a); break; \
        case 4: k_trace<V, S, 4, K><<<blocks, VT_TRACE_THREADS, 0, s>>>(a); break; \
        case 8: k_trace<V, S, 8, K><<<blocks, VT_TRACE_THREADS, 0, s>>>(a); break; \
        default: k_trace<V, S, 1, K><<<blocks, VT_TRACE_THREADS, 0, s>>>(a); break; \
    }
#define VT_LAUNCH(V, S) { if (S && skip) VT_LAUNCH_U(V, S, S) else VT_LAUNCH_U(V, S, false) }
    if (a.br.vtype == 0) { if (slabMode) VT_LAUNCH(0, true) else VT_LAUNCH(0, false) }
    else { if (slabMode) VT_LAUNCH(1, true) else VT_LAUNCH(1, false) }
#undef VT_LAUNCH_U
#undef VT_LAUNCH
    return cudaGetLastError();
}

cudaError_t vt_launch_wave_round(const TraceArgs& a, const WaveRound& w, int blocksPerSM, size_t slotBytes,
                                 cudaStream_t s) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const unsigned int grid = (unsigned int)(sms * (blocksPerSM > 0 ? blocksPerSM : 8));
    if (slotBytes % 16 != 0 || slotBytes > 200 * 1024) return cudaErrorInvalidValue;
    /* per launch (a cheap host call): the attribute belongs to the current device */
    const int v = a.br.vtype == 0 ? 0 : 1;
    cudaError_t e = v == 0 ? cudaFuncSetAttribute(k_wf_march<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024)
                           : cudaFuncSetAttribute(k_wf_march<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    if (v == 0) k_wf_traverse<0><<<grid, 128, 0, s>>>(a, w);
    else k_wf_traverse<1><<<grid, 128, 0, s>>>(a, w);
    k_wf_scan<<<1, 1024, 0, s>>>(w);
    k_wf_scatter<<<(unsigned int)(sms * 4), 256, 0, s>>>(w);
    if (v == 0) k_wf_march<0><<<(unsigned int)(sms * 4), 128, slotBytes, s>>>(a, w, (unsigned int)slotBytes);
    else k_wf_march<1><<<(unsigned int)(sms * 4), 128, slotBytes, s>>>(a, w, (unsigned int)slotBytes);
    return cudaGetLastError();
}

cudaError_t vt_launch_rays(const DevCamera& c, float* dirs, cudaStream_t s) {
    long long n = (long long)c.W * c.H;
    if (n == 0) return cudaSuccess;
    k_rays<<<(unsigned int)((n + 255) / 256), 256, 0, s>>>(c, dirs);
    return cudaGetLastError();
}

cudaError_t vt_launch_cube(const DevCamera& c, const float* cube, int3 minBox, int3 cubeDim,
                           int3 cubeInc, float iso, float3 light, float4* rgba, cudaStream_t s) {
    long long n = (long long)c.W * c.H;
    if (n == 0) return cudaSuccess;
    const long long tiles = (long long)((c.W + 7) / 8) * ((c.H + 3) / 4);
    if (tiles > 0xFFFFFFFFll) return cudaErrorInvalidValue;
    k_cube<<<(unsigned int)((tiles + 3) / 4), 128, 0, s>>>(c, cube, minBox, cubeDim, cubeInc, iso, light, rgba);
    return cudaGetLastError();
}

cudaError_t vt_launch_fill_dense(void* dst, int vtype, const void* src, long long nx, long long ny,
                                 long long nz, int P, long long ey, long long ez, cudaStream_t s) {
    long long rows = nx * ny;
    if (rows == 0) return cudaSuccess;
    if (rows > 2147483647LL) return cudaErrorInvalidValue;
    if (vtype == 0) k_fill_dense<0><<<(unsigned int)rows, 256, 0, s>>>(dst, src, nx, ny, nz, P, ey, ez);
    else k_fill_dense<1><<<(unsigned int)rows, 256, 0, s>>>(dst, src, nx, ny, nz, P, ey, ez);
    return cudaGetLastError();
}
