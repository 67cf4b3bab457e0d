/*
 * builder.cu -- GPU octree builder writing the reference's octree file
 * (OctreeM, src/CreateOctree.cu:300-573, writeToFile :342-371).
 *
 * Reference semantics, restated level by level:
 *   nLevels  = ceil(log2(max extent)) computed as the reference does in
 *              float (:316-319); dimension = 2^nLevels;
 *   leaf     = every cell code of level nLevels (inclusive range, :452),
 *              valid when the 8 zero-padded corner voxels straddle iso with
 *              the test ((v-iso)<0) != ((v0-iso)<0) (:497-501);
 *   inner l  = every code of level l except the last (`while(inicio!=fin)`,
 *              :550) whose children the builder's range search finds in
 *              level l+1 (:553, searchChildren :247-284);
 *   root     = {1,1} when level 1 has children of node 1 (:532-540);
 *   a level  = its valid codes as sorted inclusive runs [s,e] (insert /
 *              completeLevel, :79-128).
 * The GPU version keeps each level as a bitmask over its Morton codes and
 * counts run starts with a prefix sum; a parent's range search follows from
 * the count before its children and their bits alone (vt_search.h,
 * has_children_rank), so no level waits for the ranges of the one below and
 * the host is asked for nothing until all levels are done.  The ranges are
 * then made and copied back window by window, and written (octree_write.h).
 * Output is byte-identical to the reference's volumeToOctree.
 */
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <memory>
#include <new>

#include "../../include/vt.h"
#include "octree_write.h"
#include "vt_math.cuh"
#include "vt_runtime.h"
#include "vt_search.h"

namespace vtb {

#define CKB(call)                                                                              \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess) { st = vtrt::fail(VT_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); goto done; } \
    } while (0)

/* Leaf cells of one 8 x 8 x 64 box (x, y, z) per CTA turn (src/CreateOctree.cu:471-517):
 * bit b of word w = cell with Morton offset 32w + b.  Each voxel row of the
 * box and its far faces (9 x 9 rows of 65) becomes sign bits by ballots, a
 * row of cells is then an AND and an OR of four rows and their shifts (all
 * eight corners alike or not), and 128 threads gather the words, 2 x 4 x 4
 * cells each.  Bound by memory: a voxel is read 1.3 times, by whole 128-byte
 * lines.  Against one thread per word reading eight corners per cell: 512^3
 * float32 1003 -> 283 us, 201 x 333 x 129 uint8 (in its 512^3 cube)
 * 994 -> 33 us. */
#define LB_X 8
#define LB_Y 8
#define LB_Z 64
template <int VTYPE>
__global__ void __launch_bounds__(256) k_leaf(const void* v, long long dx, long long dy, long long dz, float iso,
                                              uint32_t* bits, int N, long long nby, long long nbz, long long boxes) {
    __shared__ unsigned long long row[LB_X + 1][LB_Y + 1];
    __shared__ unsigned char ext[LB_X + 1][LB_Y + 1];          /* the sign behind the row's end */
    __shared__ unsigned long long cells[LB_X][LB_Y];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool zero = (0.0f - iso) < 0;                        /* zero padding */
    for (long long box = blockIdx.x; box < boxes; box += gridDim.x) {
        const long long z0 = box % nbz * LB_Z, y0 = box / nbz % nby * LB_Y, x0 = box / nbz / nby * LB_X;
        for (int r = warp; r < (LB_X + 1) * (LB_Y + 1); r += 8) {
            const int rx = r / (LB_Y + 1), ry = r % (LB_Y + 1);
            const long long x = x0 + rx, y = y0 + ry;
            bool s0 = zero, s1 = zero, s2 = zero;
            if (x < dx && y < dy) {
                const long long i = (x * dy + y) * dz + z0;
                const long long left = dz - z0;                /* voxels of the row from z0 on */
                if (VTYPE == 0) {
                    const float* p = (const float*)v + i;
                    float a = 0.0f, b = 0.0f, c = 0.0f;
                    if (lane < left) a = __ldg(p + lane);
                    if (lane + 32 < left) b = __ldg(p + lane + 32);
                    if (lane == 0 && left > LB_Z) c = __ldg(p + LB_Z);
                    s0 = (a - iso) < 0; s1 = (b - iso) < 0; s2 = (c - iso) < 0;
                } else {
                    const unsigned char* p = (const unsigned char*)v + i;
                    unsigned int a = 0, b = 0, c = 0;
                    if (lane < left) a = __ldg(p + lane);
                    if (lane + 32 < left) b = __ldg(p + lane + 32);
                    if (lane == 0 && left > LB_Z) c = __ldg(p + LB_Z);
                    s0 = ((float)a - iso) < 0; s1 = ((float)b - iso) < 0; s2 = ((float)c - iso) < 0;
                }
            }
            const unsigned int lo = __ballot_sync(0xffffffffu, s0), hi = __ballot_sync(0xffffffffu, s1);
            if (lane == 0) { row[rx][ry] = (unsigned long long)hi << 32 | lo; ext[rx][ry] = s2; }
        }
        __syncthreads();
        if (tid < LB_X * LB_Y) {
            const int cx = tid / LB_Y, cy = tid % LB_Y;
            unsigned long long all = ~0ull, any = 0;
            unsigned long long allE = 1, anyE = 0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const unsigned long long m = row[cx + (k >> 1)][cy + (k & 1)], e = ext[cx + (k >> 1)][cy + (k & 1)];
                all &= m; any |= m; allE &= e; anyE |= e;
            }
            cells[cx][cy] = (any | (any >> 1 | anyE << 63)) & ~(all & (all >> 1 | allE << 63));
        }
        __syncthreads();
        if (tid < (LB_X / 2) * (LB_Y / 4) * (LB_Z / 4)) {
            /* 16 consecutive words make an 8^3 block: x1, z2, y2, x2 of the cell from the low bit up */
            const int X = ((tid & 1) << 1) | ((tid & 8) >> 1), Z = ((tid & 2) << 1) | ((tid >> 4) << 3), Y = tid & 4;
            if (x0 + X < N && y0 + Y < N && z0 + Z < N) {
                uint32_t m = 0;
#pragma unroll
                for (int x = 0; x < 2; x++)
#pragma unroll
                    for (int y = 0; y < 4; y++) {
                        const uint32_t q = (uint32_t)(cells[X + x][Y + y] >> Z) & 15u;   /* four cells in z */
                        m |= ((q & 3u) | (q & 12u) << 6) << (4 * x + 2 * (y & 1) + 16 * (y >> 1));
                    }
                const uint64_t off = (vt::spread3((uint32_t)(x0 + X)) << 2) | (vt::spread3((uint32_t)(y0 + Y)) << 1) |
                                     vt::spread3((uint32_t)(z0 + Z));
                bits[off >> 5] = m;
            }
        }
        __syncthreads();
    }
}

/* one level on the device */
struct Level {
    uint32_t* bits;                 /* its codes as a bitmask (Morton offset i = bit i) */
    uint32_t* offs;                 /* per word: run starts before it in its block of CB_WORDS words */
    unsigned long long* block;      /* per block: run starts, then (k_scan) run starts before it */
    unsigned long long* total;      /* run starts */
    long long words, blocks;
};
#define CB_WORDS 2048

/* runs that start before word w */
__device__ __forceinline__ unsigned long long starts_before(const Level& L, long long w) {
    return L.block[w / CB_WORDS] + L.offs[w];
}
/* the run starts / ends among word w's bits */
__device__ __forceinline__ uint32_t run_starts(const Level& L, long long w, uint32_t m) {
    return m & ~((m << 1) | (w > 0 ? L.bits[w - 1] >> 31 : 0u));
}
__device__ __forceinline__ uint32_t run_ends(const Level& L, long long w, uint32_t m) {
    return m & ~((m >> 1) | (w + 1 < L.words ? L.bits[w + 1] << 31 : 0u));
}

/* inner level: parent p exists when it has a set child byte, is not the
 * level's last code, and the builder's search over the child level finds a
 * child.  One parent per lane, a word per warp. */
__global__ void __launch_bounds__(256) k_inner(const Level C, uint32_t* bits, long long words, long long parents) {
    const int64_t n = 2 * (int64_t)*C.total;
    const int lane = threadIdx.x & 31;
    for (long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < words;
         w += ((long long)gridDim.x * blockDim.x) >> 5) {
        const long long p = w * 32 + lane;
        bool set = false;
        if (p < parents - 1) {
            const long long cw = p >> 2;
            const uint32_t m = C.bits[cw];
            const int sh = 8 * (int)(p & 3);
            const uint32_t byte = (m >> sh) & 0xFFu;
            if (byte) {
                const uint32_t st = run_starts(C, cw, m);
                set = vtsearch::has_children_rank(n, byte, (st >> sh) & 0xFFu,
                                                  (int64_t)starts_before(C, cw) + __popc(st & ((1u << sh) - 1u)));
            }
        }
        const uint32_t b = __ballot_sync(0xffffffffu, set);
        if (lane == 0) bits[w] = b;
    }
}

/* run starts per word (exclusive within its block) and per block; eight
 * words a thread */
__global__ void __launch_bounds__(256) k_count(const Level L) {
    __shared__ uint32_t warpSum[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long blk = blockIdx.x; blk < L.blocks; blk += gridDim.x) {
        const long long w0 = blk * CB_WORDS + threadIdx.x * 8;
        uint32_t c[8], sum = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            c[k] = sum;
            if (w0 + k < L.words) sum += __popc(run_starts(L, w0 + k, L.bits[w0 + k]));
        }
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) warpSum[warp] = inc;
        __syncthreads();
        uint32_t base = inc - sum, all = 0;
        for (int k = 0; k < 8; k++) { if (k < warp) base += warpSum[k]; all += warpSum[k]; }
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (w0 + k < L.words) L.offs[w0 + k] = base + c[k];
        if (threadIdx.x == 0) L.block[blk] = all;
        __syncthreads();
    }
}

/* block counts -> exclusive offsets, and the level's total (one CTA) */
__global__ void __launch_bounds__(1024) k_scan(const Level L) {
    __shared__ unsigned long long warpSum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long carry = 0;
    for (long long b0 = 0; b0 < L.blocks; b0 += 1024) {
        const long long b = b0 + threadIdx.x;
        const unsigned long long v = b < L.blocks ? L.block[b] : 0ull;
        unsigned long long inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) warpSum[warp] = inc;
        __syncthreads();
        unsigned long long before = carry, all = 0;
        for (int k = 0; k < 32; k++) { if (k < warp) before += warpSum[k]; all += warpSum[k]; }
        if (b < L.blocks) L.block[b] = before + inc - v;
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *L.total = carry;
}

/* words [k0, k1) of the level's inclusive ranges [s, e], in order: the run an
 * end belongs to is the last one that starts at or before it.  Only the blocks
 * that meet the window are read: a level of many windows is read once or
 * twice in all, not once a window (512^3 of noise, 91 windows: 5.8 -> 2.8 ms
 * in this kernel; 1024^3, 730 windows: 1.92 -> 1.58 s for the call). */
__global__ void __launch_bounds__(256) k_ranges(const Level L, uint64_t base, unsigned long long k0, unsigned long long k1,
                                                uint64_t* out) {
    __shared__ int64_t range[2];
    if (threadIdx.x == 0) vtsearch::window_blocks(L.block, L.blocks, *L.total, k0, k1, &range[0], &range[1]);
    __syncthreads();
    for (long long blk = range[0] + blockIdx.x; blk < range[1]; blk += gridDim.x) {
        for (long long w = blk * CB_WORDS + threadIdx.x; w < L.words && w < (blk + 1) * CB_WORDS; w += blockDim.x) {
            const uint32_t m = L.bits[w];
            if (!m) continue;
            const uint32_t starts = run_starts(L, w, m), ends = run_ends(L, w, m);
            const unsigned long long before = starts_before(L, w);
            unsigned long long k = 2 * before;
            for (uint32_t s = starts; s; s &= s - 1, k += 2)
                if (k >= k0 && k < k1) out[k - k0] = base + (uint64_t)w * 32 + (__ffs(s) - 1);
            for (uint32_t e = ends; e; e &= e - 1) {
                const int b = __ffs(e) - 1;
                k = 2 * (before + __popc(starts & (0xFFFFFFFFu >> (31 - b)))) - 1;
                if (k >= k0 && k < k1) out[k - k0] = base + (uint64_t)w * 32 + b;
            }
        }
    }
}
#define RANGE_WINDOW (1ll << 19)   /* words made and copied at a time (4 MB) */

static unsigned int grid_for(long long threads, int block) {
    const long long g = (threads + block - 1) / block;
    return (unsigned int)(g < 148 * 32 ? (g < 1 ? 1 : g) : 148 * 32);
}

}  // namespace vtb

using namespace vtb;

extern "C" vt_status vt_octree_build_device(const void* dev_vol, int vtype, const int64_t dims[3], float iso,
                                            const char* out_path, void* stream) {
    vtrt::clear_error();
    if (!dev_vol || !dims || !out_path) return vtrt::fail(VT_ERR_INVALID, "vt_octree_build_device: null argument");
    cudaStream_t s = (cudaStream_t)stream;
    vt_status st = VT_OK;
    /* nLevels exactly as the reference computes it (src/CreateOctree.cu:308-319) */
    int rd[3] = {(int)dims[0], (int)dims[1], (int)dims[2]};
    int dimension;
    if (rd[0] > rd[1] && rd[0] > rd[2]) dimension = rd[0];
    else if (rd[1] > rd[2]) dimension = rd[1];
    else dimension = rd[2];
    float aux = logf((float)dimension) / logf(2.0);
    float aux2 = aux - floorf(aux);
    int nLevels = aux2 > 0.0 ? (int)(aux + 1) : (int)aux;
    dimension = (int)pow(2, nLevels);
    if (nLevels < 1 || nLevels > 13) return vtrt::fail(VT_ERR_UNSUPPORTED, "volume extent gives %d levels", nLevels);
    /* one device allocation: every level's bits and counts, and the window */
    Level L[14];
    unsigned long long total[15];
    unsigned char* ws = nullptr;
    uint64_t* window = nullptr;
    std::unique_ptr<uint64_t[]> host;
    size_t bytes = 256;
    for (int pass = 0; pass < 2; pass++) {
        bytes = 256;   /* the totals */
        for (int l = 1; l <= nLevels; l++) {
            L[l].words = ((1ll << (3 * l)) + 31) / 32;
            L[l].blocks = (L[l].words + CB_WORDS - 1) / CB_WORDS;
            const size_t w4 = ((size_t)L[l].words * 4 + 255) & ~(size_t)255;
            L[l].bits = (uint32_t*)(ws + bytes); bytes += w4;
            L[l].offs = (uint32_t*)(ws + bytes); bytes += w4;
            L[l].block = (unsigned long long*)(ws + bytes); bytes += ((size_t)L[l].blocks * 8 + 255) & ~(size_t)255;
            L[l].total = (unsigned long long*)ws + l;
        }
        window = (uint64_t*)(ws + bytes); bytes += (size_t)RANGE_WINDOW * 8;
        if (pass == 0) CKB(cudaMalloc(&ws, bytes));
    }
    {
        /* cells outside the volume have no corner inside it: their words stay 0 */
        CKB(cudaMemsetAsync(L[nLevels].bits, 0, (size_t)L[nLevels].words * 4, s));
        const long long nbx = (dims[0] + LB_X - 1) / LB_X, nby = (dims[1] + LB_Y - 1) / LB_Y, nbz = (dims[2] + LB_Z - 1) / LB_Z;
        const long long boxes = nbx * nby * nbz;
        const unsigned int grid = (unsigned int)(boxes < 148 * 64 ? (boxes < 1 ? 1 : boxes) : 148 * 64);
        if (vtype == VT_U8) k_leaf<1><<<grid, 256, 0, s>>>(dev_vol, dims[0], dims[1], dims[2], iso, L[nLevels].bits, dimension, nby, nbz, boxes);
        else k_leaf<0><<<grid, 256, 0, s>>>(dev_vol, dims[0], dims[1], dims[2], iso, L[nLevels].bits, dimension, nby, nbz, boxes);
        CKB(cudaGetLastError());
    }
    for (int l = nLevels; l >= 1; l--) {
        if (l < nLevels)
            k_inner<<<grid_for(L[l].words * 32, 256), 256, 0, s>>>(L[l + 1], L[l].bits, L[l].words, 1ll << (3 * l));
        k_count<<<grid_for(L[l].blocks * 256, 256), 256, 0, s>>>(L[l]);
        k_scan<<<1, 1024, 0, s>>>(L[l]);
        CKB(cudaGetLastError());
    }
    CKB(cudaMemcpyAsync(total, ws, (size_t)(nLevels + 1) * 8, cudaMemcpyDeviceToHost, s));
    CKB(cudaMemcpyAsync(&total[14], L[1].bits, 4, cudaMemcpyDeviceToHost, s));
    CKB(cudaStreamSynchronize(s));
    for (int l = nLevels; l >= 1; l--)
        if (2 * total[l] > 0x7FFFFFFFull) { st = vtrt::fail(VT_ERR_UNSUPPORTED, "level with %llu ranges exceeds the file format", total[l]); goto done; }
    host.reset(new (std::nothrow) uint64_t[RANGE_WINDOW]);
    if (!host) { st = vtrt::fail(VT_ERR_NOMEM, "octree build: host window"); goto done; }
    {
        vtoct::Levels file;
        file.iso = iso; file.dimension = dimension; file.nLevels = nLevels; file.bits1 = (uint32_t)total[14];
        for (int a = 0; a < 3; a++) file.realDim[a] = rd[a];
        for (int l = 1; l <= nLevels; l++) file.runs[l] = total[l];
        /* as much of level l from word k0 on, and of the following levels, as the window holds */
        auto fetch = [&](int l, size_t k0, size_t* n) -> const uint64_t* {
            long long fill = 0, next = (long long)k0;
            for (; l >= 1 && fill < RANGE_WINDOW; l--, next = 0) {
                const long long k1 = std::min((long long)(2 * total[l]), next + RANGE_WINDOW - fill);
                if (k1 > next)
                    k_ranges<<<grid_for(L[l].blocks * 256, 256), 256, 0, s>>>(L[l], 1ull << (3 * l), (unsigned long long)next,
                                                                              (unsigned long long)k1, window + fill);
                fill += k1 - next;
            }
            cudaError_t e = cudaGetLastError();
            if (e == cudaSuccess) e = cudaMemcpyAsync(host.get(), window, (size_t)fill * 8, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) { st = vtrt::fail(VT_ERR_CUDA, "octree build, ranges: %s", cudaGetErrorString(e)); return nullptr; }
            *n = (size_t)fill;
            return host.get();
        };
        switch (vtoct::write_octree(out_path, file, fetch)) {
            case vtoct::WRITE_OPEN: st = vtrt::fail(VT_ERR_IO, "unable to write %s", out_path); break;
            case vtoct::WRITE_SHORT: st = vtrt::fail(VT_ERR_IO, "short write to %s", out_path); break;
            default: break;   /* written, or fetch's own status */
        }
    }
done:
    cudaFree(ws);
    return st;
}

extern "C" vt_status vt_octree_build(const vt_volume* v, float iso, const char* out_path, void* stream) {
    vtrt::clear_error();
    if (!v || !out_path) return vtrt::fail(VT_ERR_INVALID, "vt_octree_build: null argument");
    if (!v->data) return vtrt::fail(VT_ERR_UNSUPPORTED, "vt_octree_build: the volume is read through a function");
    size_t bytes = v->voxels() * v->esize();
    void* d = nullptr;
    cudaError_t e = cudaMalloc(&d, bytes);
    if (e != cudaSuccess) return vtrt::fail(VT_ERR_NOMEM, "octree build: %s", cudaGetErrorString(e));
    e = cudaMemcpy(d, v->data, bytes, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) { cudaFree(d); return vtrt::fail(VT_ERR_CUDA, "octree build upload: %s", cudaGetErrorString(e)); }
    vt_status st = vt_octree_build_device(d, v->vtype, v->dims, iso, out_path, stream);
    cudaFree(d);
    return st;
}
