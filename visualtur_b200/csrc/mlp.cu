/*
 * mlp.cu -- the brick-prefetch network of libvt.so (no reference
 * counterpart): pose features (12) -> 512 -> 512 -> 4096 sigmoid, one
 * output per coarse octree node, trained with binary cross-entropy on
 * traces of the nodes each frame marched.
 *
 * Weights are stored in BF16 with FP32 master copies updated by Adam.  The
 * forward and backward GEMMs run on the tensor cores (tcgen05.mma, BF16 x
 * BF16 -> FP32 in tensor memory); activations and gradients are rounded to
 * BF16 once, by the epilogue that makes them, and everything around a GEMM
 * (bias, ReLU, sigmoid, cross-entropy gradient, column sums, Adam) runs in
 * an epilogue, in FP32.  A register-tiled SIMT kernel (FP32 activations x
 * BF16 weights, FMA) does the same contractions where
 * vt_mlp_use_tensor_cores switches the tensor cores off.
 */
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "../../include/vt.h"
#include "vt_runtime.h"

namespace vtm {

#define CKM(call)                                                                             \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess) return vtrt::fail(VT_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

template <class T> __device__ __forceinline__ float ld(const T* p, long long i);
template <> __device__ __forceinline__ float ld<float>(const float* p, long long i) { return p[i]; }
template <> __device__ __forceinline__ float ld<__nv_bfloat16>(const __nv_bfloat16* p, long long i) {
    return __bfloat162float(p[i]);
}

enum { ACT_NONE = 0, ACT_RELU = 1, ACT_SIGMOID = 2 };

/* C[m,n] = act(sum_k A[m,k] B[k,n] + bias[n]), with
 * element (m,k) of A at A[m*am + k*ak] and (k,n) of B at B[k*bk + n*bn], so
 * transposed operands are just other strides.  64x64 tile per 256-thread
 * CTA, 4x4 outputs per thread, K staged through shared memory in 16s.  Four
 * CTAs an SM are asked for so that the compiler spends 64 registers: left to
 * itself it takes 40, and a training step of the 12-512-512-4096 network at
 * batch 256 1027 instead of 985 us. */
template <class TA, class TB>
__global__ void __launch_bounds__(256, 4) k_gemm(const TA* A, long long am, long long ak, const TB* B, long long bk,
                                              long long bn, float* C, long long cm, int M, int N, int K,
                                              const float* bias, int act) {
    __shared__ float As[16][64 + 1];
    __shared__ float Bs[16][64 + 1];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += 16) {
        for (int e = threadIdx.x; e < 16 * 64; e += 256) {
            int kk = e / 64, mm = e % 64;
            int m = m0 + mm, k = k0 + kk;
            As[kk][mm] = (m < M && k < K) ? ld<TA>(A, (long long)m * am + (long long)k * ak) : 0.0f;
            int n = n0 + mm;
            Bs[kk][mm] = (n < N && k < K) ? ld<TB>(B, (long long)k * bk + (long long)n * bn) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; kk++) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) { a[i] = As[kk][ty * 4 + i]; b[i] = Bs[kk][tx * 4 + i]; }
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            float v = acc[i][j] + (bias ? bias[n] : 0.0f);
            if (act == ACT_RELU) v = fmaxf(v, 0.0f);
            else if (act == ACT_SIGMOID) v = 1.0f / (1.0f + expf(-v));
            C[(long long)m * cm + n] = v;
        }
    }
}

/* dZ = (p - y) / batch for sigmoid + BCE; loss partial sums */
__global__ void k_bce_grad(const float* P, const float* Y, float* dZ, long long n, float invB, float* loss) {
    float l = 0.0f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float p = P[i], y = Y[i];
        dZ[i] = (p - y) * invB;
        float pc = fminf(fmaxf(p, 1e-7f), 1.0f - 1e-7f);
        l -= y * logf(pc) + (1.0f - y) * logf(1.0f - pc);
    }
    for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, l * invB);
}
/* dX *= (X > 0) for ReLU layers (X = post-activation values) */
__global__ void k_relu_mask(float* d, const float* a, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        if (a[i] <= 0.0f) d[i] = 0.0f;
}
/* db[n] = sum_m dZ[m,n] */
__global__ void k_colsum(const float* dZ, int M, int N, float* db) {
    int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    float s = 0.0f;
    for (int m = 0; m < M; m++) s += dZ[(long long)m * N + n];
    db[n] = s;
}
/* one Adam step of a parameter (FP32 master, moments) */
struct Adam { float lr, b1, b2, eps, c1, c2; };
__device__ __forceinline__ float adam_step(const Adam& o, float w, float g, float& m, float& v) {
    m = o.b1 * m + (1.0f - o.b1) * g;
    v = o.b2 * v + (1.0f - o.b2) * g * g;
    return w - o.lr * (m / o.c1) / (sqrtf(v / o.c2) + o.eps);
}
/* Adam on FP32 masters, refresh the BF16 copy (rows of N at ldb) */
__global__ void k_adam(float* w, __nv_bfloat16* wb, const float* g, float* m, float* v, long long n, int N, int ldb,
                       Adam o) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float mi = m[i], vi = v[i];
        const float wi = adam_step(o, w[i], g[i], mi, vi);
        m[i] = mi; v[i] = vi;
        w[i] = wi;
        if (wb) wb[N == ldb ? i : i / N * ldb + i % N] = __float2bfloat16_rn(wi);
    }
}
__global__ void k_to_bf16(const float* w, __nv_bfloat16* wb, long long n, int N, int ldb) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        wb[N == ldb ? i : i / N * ldb + i % N] = __float2bfloat16_rn(w[i]);
}

/* ------------------------------------------------------------------------ */
/* Tensor-core GEMM (tcgen05, sm_100a)                                       */
/* ------------------------------------------------------------------------ */
/* C[m,n] = sum_k A[m,k] B[k,n] with a fused epilogue.  One 256-thread CTA
 * per 128 x 64 output tile (and range of K).  Per 64-deep K step the tiles
 * land in one of S shared-memory stages by 16-byte cp.async (zero-filled
 * outside the matrices), in the tensor core's unswizzled core-matrix order:
 * 128-byte core matrices of eight 16-byte rows, (128 or 64) / 8 of them side
 * by side per eight k.  A row of a core matrix is eight k of one m or n
 * where the operand is K-major, eight m or n of one k where it is MN-major
 * (the operand's unit stride), so neither is transposed on the way.  One
 * thread issues four tcgen05.mma (M 128, N 64, K 16) a step into a
 * 64-column tensor-memory accumulator and commits them to the stage's
 * mbarrier, which is waited for (bounded: past the limit the kernel records
 * it in the network's err, frees its tensor memory and returns) before the stage is
 * filled again.  The accumulator then goes through shared memory so that
 * the epilogue's reads and writes are coalesced.
 *
 * Bound by latency: 8 to 296 CTAs of 1 to 8 K steps each.  The tile is for
 * grid size (a 256 x 512 layer still makes 16 tiles); where tiles are few and
 * K is deep (the 4096-deep gradient to the last hidden layer) K is split
 * over CTAs and k_dgrad_finish adds the parts in order.  Against a kernel
 * that staged scalar by scalar, one K step at a time, in 128 x 128 tiles: a
 * training step of the 12-512-512-4096 network at batch 256 1310 -> 102 us
 * (that kernel's 4096-deep gradient alone, on 8 CTAs, about 1 ms), a forward
 * pass of 8 poses 161 -> 20 us; of that, dependent launches and up to eight
 * K steps in flight 124 -> 102 and 29 -> 20 us. */
#define G_THREADS 256
#define G_M 128
#define G_N 64
#define G_K 64
#define G_STAGE_BYTES ((G_M + G_N) * G_K * 2)

/* Programmatic dependent launch: the kernels of a pass let the next one start
 * (its set-up overlaps this one's work and end) and wait for the one before
 * ahead of their first access to global memory; the wait ends when that
 * grid, and so every grid before it, is complete. */
__device__ __forceinline__ void grid_wait() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

/* tensor-core shared-memory matrix descriptor, no swizzle: lbo between the
 * core matrices of successive eight k, sbo between those of successive
 * eight m or n */
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

/* operand forms: BF16 with 16-byte aligned rows, or FP32 of any alignment
 * (the network's input) */
enum { OP_BF16_K = 0, OP_BF16_MN = 1, OP_F32_K = 2, OP_F32_MN = 3 };

/* one operand tile (R rows of m or n, G_K deep) into shared memory at dst:
 * rows r0.. of `rows`, k from k0 to kEnd.  lanes take neighbouring 16-byte
 * chunks of a row in pairs (K-major) or fours (MN-major) and eight or
 * sixteen rows, which keeps both the 32-byte sectors of global memory and
 * the banks of shared memory full. */
template <int OP, int R>
__device__ __forceinline__ void load_tile(uint32_t dst, const void* src, long long ld, int r0, int rows, int k0, int kEnd) {
    const bool f32 = OP == OP_F32_K || OP == OP_F32_MN;
    uint32_t q[f32 ? R * 8 / G_THREADS : 1][4];
#pragma unroll
    for (int pass = f32 ? 0 : 1; pass < 2; pass++) {   /* FP32: every chunk is read before the first is stored */
#pragma unroll
        for (int e = 0; e < R * 8 / G_THREADS; e++) {
            const int i = e * G_THREADS + threadIdx.x;
            int off, row, col, n;   /* shared offset; matrix row and column of the chunk; its valid elements */
            if (OP == OP_BF16_K || OP == OP_F32_K) {
                const int kc = (i & 1) + 2 * (i / (2 * R)), r = (i >> 1) % R;
                off = (kc * (R / 8) + (r >> 3)) * 128 + (r & 7) * 16;
                row = r0 + r; col = k0 + kc * 8;
                n = row < rows ? min(max(kEnd - col, 0), 8) : 0;
            } else {
                const int rest = i >> 5, mb = (i & 3) + 4 * (rest % (R / 32)), kb = rest / (R / 32), kl = (i >> 2) & 7;
                off = (kb * (R / 8) + mb) * 128 + kl * 16;
                row = k0 + kb * 8 + kl; col = r0 + mb * 8;
                n = row < kEnd ? min(max(rows - col, 0), 8) : 0;
            }
            if (!f32) {
                const __nv_bfloat16* p = (const __nv_bfloat16*)src + (n ? (long long)row * ld + col : 0);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst + off), "l"(p), "r"(n * 2) : "memory");
            } else if (pass == 0) {
                const float* p = (const float*)src + (n ? (long long)row * ld + col : 0);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const __nv_bfloat162 h =
                        __floats2bfloat162_rn(2 * j < n ? p[2 * j] : 0.0f, 2 * j + 1 < n ? p[2 * j + 1] : 0.0f);
                    q[f32 ? e : 0][j] = *(const uint32_t*)&h;
                }
            } else {
                const uint32_t* v = q[f32 ? e : 0];
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                             :: "r"(dst + off), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
            }
        }
    }
}

/* epilogues */
enum {
    EPI_HIDDEN = 0,   /* relu(acc + bias): BF16 copy (the next operand) and, if C, FP32 */
    EPI_OUT = 1,      /* sigmoid(acc + bias) into C; with targets Y also the BF16 gradient (p - y) / batch, the loss
                         and the gradient's column sums over the tile's rows */
    EPI_PART = 2,     /* the accumulator into part `blockIdx.z` of C */
    EPI_GRAD = 3      /* a weight gradient, into C */
};
struct GemmArgs {
    const void* A; long long lda;
    const __nv_bfloat16* B; long long ldb;
    int M, N, K, kPer;                  /* kPer: K of one part (blockIdx.z) */
    const float* bias;
    float* C; long long ldc;
    __nv_bfloat16* Cb; long long ldcb;
    const float* Y; float invB; float* loss; float* colsum;
    __nv_bfloat16* Xb; int ldx;         /* OP_F32_K: a BF16 copy of A, for the backward pass */
};
/* up to three products in one launch: grid.x holds the tiles of one after
 * those of the other, from tile first[i] on */
struct GemmGroup { GemmArgs g[3]; unsigned int first[3]; unsigned int* err; };

template <int OPA, int OPB, int EPI, int S>
__global__ void __launch_bounds__(G_THREADS) k_gemm_tc(const __grid_constant__ GemmGroup P) {
    extern __shared__ __align__(1024) unsigned char g_smem[];
    __shared__ __align__(8) unsigned long long mbar[S];
    __shared__ uint32_t tslot;
    __shared__ float s_sum[G_THREADS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const GemmArgs& G = P.g[(blockIdx.x >= P.first[1]) + (blockIdx.x >= P.first[2])];
    const unsigned int tile = blockIdx.x - P.first[(blockIdx.x >= P.first[1]) + (blockIdx.x >= P.first[2])];
    const unsigned int nTiles = (G.N + G_N - 1) / G_N;
    const int tm = tile / nTiles, m0 = tm * G_M, n0 = (tile % nTiles) * G_N;
    const int kBeg = blockIdx.z * G.kPer, kEnd = min(G.K, kBeg + G.kPer);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&tslot)), "r"(G_N));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int i = 0; i < S; i++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&mbar[i])), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tslot;
    /* the launch before this one may still run until here */
    grid_wait();
    if (EPI == EPI_HIDDEN && G.loss && tile == 0 && tid == 0) *G.loss = 0.0f;
    if (OPA == OP_F32_K && G.Xb)   /* dealt out over the row block's tiles */
        for (int e = (tile % nTiles) * G_THREADS + tid; e < G_M * G.K; e += nTiles * G_THREADS) {
            const int r = e / G.K, k = e % G.K;
            if (m0 + r < G.M)
                G.Xb[(long long)(m0 + r) * G.ldx + k] =
                    __float2bfloat16_rn(((const float*)G.A)[(long long)(m0 + r) * G.lda + k]);
        }

    /* kind::f16 instruction descriptor: FP32 accumulator, BF16 A and B, their
     * majors (0: K, 1: M or N), N / 8 and M / 16 */
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((OPA & 1) ? 1u << 15 : 0u) | ((OPB & 1) ? 1u << 16 : 0u) |
                           ((uint32_t)(G_N >> 3) << 17) | ((uint32_t)(G_M >> 4) << 24);
    const uint32_t base = smem_u32(g_smem);
    const int nk = (kEnd - kBeg + G_K - 1) / G_K;

    auto fill = [&](int t) {   /* K step t into its stage (an empty group past the end keeps the count) */
        if (t < nk) {
            const uint32_t st = base + (t % S) * G_STAGE_BYTES;
            load_tile<OPA, G_M>(st, G.A, G.lda, m0, G.M, kBeg + t * G_K, kEnd);
            load_tile<OPB, G_N>(st + G_M * G_K * 2, G.B, G.ldb, n0, G.N, kBeg + t * G_K, kEnd);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto wait_mma = [&](int t) -> bool {   /* the MMAs of K step t have read their stage */
        const uint32_t mb = smem_u32(&mbar[t % S]), parity = (uint32_t)(t / S) & 1u;
        uint32_t done = 0;
        for (long long it = 0; it < (1ll << 22) && !done; it++) {
            asm volatile("{\n\t.reg .pred P1;\n\t"
                         "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
                         "selp.b32 %0, 1, 0, P1;\n\t}"
                         : "=r"(done) : "r"(mb), "r"(parity) : "memory");
        }
        if (!done) atomicOr(P.err, 1u);
        return done != 0;
    };
#pragma unroll 1
    for (int t = 0; t < S - 1; t++) fill(t);
    bool ok = true;
#pragma unroll 1
    for (int t = 0; t < nk; t++) {
        asm volatile("cp.async.wait_group %0;" :: "n"(S - 2) : "memory");
        /* the tensor core reads shared memory through the async proxy */
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t a = base + (t % S) * G_STAGE_BYTES, b = a + G_M * G_K * 2;
#pragma unroll
            for (int j = 0; j < G_K / 16; j++) {
                const uint64_t da = tc_desc(a + j * 2 * (G_M / 8) * 128, (G_M / 8) * 128, 128);
                const uint64_t db = tc_desc(b + j * 2 * (G_N / 8) * 128, (G_N / 8) * 128, 128);
                const uint32_t accum = (t > 0 || j > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                    :: "r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(accum), "r"(0), "r"(0), "r"(0), "r"(0));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         :: "r"(smem_u32(&mbar[t % S])));
        }
        /* the next step to load takes the stage of the step before, once its MMAs are through */
        if (t > 0 && t + S - 1 < nk) ok = wait_mma(t - 1) && ok;
        fill(t + S - 1);
    }
    if (nk > 0) ok = wait_mma(nk - 1) && ok;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    ok = __syncthreads_and(ok);   /* also: every thread is done with the stages */
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (ok) {
        /* accumulator -> shared: warp w reads rows 32 (w % 4).., columns 32 (w / 4).. */
        float* const sC = (float*)g_smem;
        const int ldS = G_N + 1, srow = (warp & 3) * 32 + lane;
        {
            const int c0 = (warp >> 2) * 32;
            uint32_t v[32];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                  "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                  "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                : "r"(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0));
            asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
            for (int j = 0; j < 32; j++) sC[srow * ldS + c0 + j] = __uint_as_float(v[j]);
        }
        __syncthreads();
        /* a thread owns one column of the tile and every fourth row */
        const int c = tid & (G_N - 1), n = n0 + c, rows = min(G_M, G.M - m0);
        float loss = 0.0f, sum = 0.0f;
        if (n < G.N) {
            const float bias = (EPI == EPI_HIDDEN || EPI == EPI_OUT) ? G.bias[n] : 0.0f;
            /* sixteen rows at a time, what they read before what they write:
             * the compiler cannot tell the arrays apart */
#pragma unroll 1
            for (int r0 = tid >> 6; r0 < rows; r0 += 64) {
                float y16[16];
                if (EPI == EPI_OUT && G.Y) {
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        if (r0 + 4 * j < rows) y16[j] = G.Y[(long long)(m0 + r0 + 4 * j) * G.N + n];
                }
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const int r = r0 + 4 * j;
                    if (r >= rows) continue;
                    const float acc = sC[r * ldS + c];
                    const long long m = m0 + r;
                    if (EPI == EPI_HIDDEN) {
                        const float x = fmaxf(acc + bias, 0.0f);
                        G.Cb[m * G.ldcb + n] = __float2bfloat16_rn(x);
                        if (G.C) G.C[m * G.ldc + n] = x;
                    } else if (EPI == EPI_OUT) {
                        const float x = acc + bias, p = 1.0f / (1.0f + expf(-x));
                        if (G.C) G.C[m * G.ldc + n] = p;
                        if (G.Y) {
                            const float y = y16[j], d = (p - y) * G.invB;
                            G.Cb[m * G.ldcb + n] = __float2bfloat16_rn(d);
                            sum += d;
                            const float pc = fminf(fmaxf(p, 1e-7f), 1.0f - 1e-7f);
                            loss -= y * logf(pc) + (1.0f - y) * logf(1.0f - pc);
                        }
                    } else if (EPI == EPI_PART) {
                        G.C[((long long)blockIdx.z * G.M + m) * G.N + n] = acc;
                    } else {
                        G.C[m * G.ldc + n] = acc;
                    }
                }
            }
        }
        if (EPI == EPI_OUT && G.Y) {
            s_sum[tid] = sum;
            for (int o = 16; o; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
            if (lane == 0) atomicAdd(G.loss, loss * G.invB);
            __syncthreads();
            if (tid < G_N && n < G.N) 
                G.colsum[(long long)tm * G.N + n] = (s_sum[tid] + s_sum[tid + 64]) + (s_sum[tid + 128] + s_sum[tid + 192]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(G_N));
}

/* Gradient to a hidden layer from its K parts: added in order, masked by the
 * layer's ReLU, as BF16 (the next operand) and column sums of 16 rows each
 * (cs[row block][n], the bias gradient's parts). */
__global__ void __launch_bounds__(256) k_dgrad_finish(const float* __restrict__ part, int parts,
                                                      const float* __restrict__ act, int M, int N,
                                                      __nv_bfloat16* __restrict__ dz, int ldz, float* __restrict__ cs) {
    __shared__ float s[4][64];
    /* column and row blocks in one grid dimension: the other ones end at 65535 */
    const unsigned int cols = (unsigned int)(N + 63) / 64, rb = blockIdx.x / cols;
    const int c = threadIdx.x & 63, q = threadIdx.x >> 6, n = (int)(blockIdx.x - rb * cols) * 64 + c;
    grid_wait();
    float sum = 0.0f;
    if (n < N) {
        float d[4] = {}, a[4] = {};
        const int m0 = (int)rb * 16 + q * 4;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (m0 + j < M) a[j] = act[(long long)(m0 + j) * N + n];
#pragma unroll 4
        for (int z = 0; z < parts; z++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (m0 + j < M) d[j] += part[((long long)z * M + m0 + j) * N + n];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (m0 + j >= M) break;
            if (a[j] <= 0.0f) d[j] = 0.0f;
            dz[(long long)(m0 + j) * ldz + n] = __float2bfloat16_rn(d[j]);
            sum += d[j];
        }
    }
    s[q][c] = sum;
    __syncthreads();
    if (q == 0 && n < N) cs[(long long)rb * N + n] = (s[0][c] + s[1][c]) + (s[2][c] + s[3][c]);
}

/* The parameters of the three layers after a backward pass: bias gradients
 * added up from their parts, then (step) one Adam step of everything, four
 * weights a thread.  Bound by memory: 30 bytes a weight (16 read, 14 written),
 * mostly in L2 (the 2.37 M weights of the 12-512-512-4096 network: 71 MB).  As
 * the epilogue of the weight-gradient GEMM, 8 warps an SM at most, the same
 * step took 37 us for the last layer and 53 us for the middle one. */
struct UpdateArgs {
    float *w[3], *m[3], *v[3]; const float* g[3]; __nv_bfloat16* wb[3]; int rows[3], N[3], ldb[3];
    float *b[3], *bm[3], *bv[3], *gb[3]; const float* part[3]; int parts[3];
    unsigned int first[7];   /* blocks: weights of layer 0, 1, 2, biases of layer 0, 1, 2 */
    Adam adam; int step;
    const unsigned int* err;   /* set: a product of this pass is incomplete, no step */
};
__global__ void __launch_bounds__(256) k_update(const __grid_constant__ UpdateArgs U) {
    int k = 0;
    while (k < 5 && blockIdx.x >= U.first[k + 1]) k++;
    grid_wait();
    if (U.step && *U.err) return;
    const long long i0 = (long long)(blockIdx.x - U.first[k]) * 256 + threadIdx.x;
    if (k >= 3) {
        const int l = k - 3, i = (int)i0, N = U.N[l];
        if (i >= N) return;
        float g = 0.0f;
        for (int z = 0; z < U.parts[l]; z++) g += U.part[l][(long long)z * N + i];
        if (!U.step) { U.gb[l][i] = g; return; }
        float m = U.bm[l][i], v = U.bv[l][i];
        U.b[l][i] = adam_step(U.adam, U.b[l][i], g, m, v);
        U.bm[l][i] = m; U.bv[l][i] = v;
        return;
    }
    const long long n = (long long)U.rows[k] * U.N[k], i = 4 * i0;
    if (i >= n) return;
    float w[4], m[4], v[4], g[4];
    const bool vec = i + 4 <= n;
    if (vec) {
        *(float4*)w = *(const float4*)(U.w[k] + i); *(float4*)m = *(const float4*)(U.m[k] + i);
        *(float4*)v = *(const float4*)(U.v[k] + i); *(float4*)g = *(const float4*)(U.g[k] + i);
    } else {
        for (int j = 0; j < 4 && i + j < n; j++) { w[j] = U.w[k][i + j]; m[j] = U.m[k][i + j]; v[j] = U.v[k][i + j]; g[j] = U.g[k][i + j]; }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) w[j] = adam_step(U.adam, w[j], g[j], m[j], v[j]);
    if (vec) {
        *(float4*)(U.w[k] + i) = *(const float4*)w; *(float4*)(U.m[k] + i) = *(const float4*)m;
        *(float4*)(U.v[k] + i) = *(const float4*)v;
    }
    const unsigned int N = U.N[k];
    unsigned int row = (unsigned int)((unsigned long long)i / N), col = (unsigned int)(i - (long long)row * N);
    for (int j = 0; j < 4 && i + j < n; j++) {
        if (!vec) { U.w[k][i + j] = w[j]; U.m[k][i + j] = m[j]; U.v[k][i + j] = v[j]; }
        U.wb[k][(long long)row * U.ldb[k] + col] = __float2bfloat16_rn(w[j]);
        if (++col == N) { col = 0; row++; }
    }
}

static unsigned int g1(long long n) { long long b = (n + 255) / 256; return (unsigned int)(b > 4096 ? 4096 : (b < 1 ? 1 : b)); }

/* a launch that may start before the one ahead of it in the stream is done
 * (its kernel calls grid_wait) */
template <class... P, class... A>
static cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c;
    memset(&c, 0, sizeof(c));
    c.gridDim = grid; c.blockDim = dim3(threads); c.dynamicSmemBytes = smem; c.stream = s;
    c.attrs = &at; c.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, kernel, P(args)...);
    if (e != cudaSuccess) cudaGetLastError();   /* reported here: not left for the caller's next check */
    return e;
}

/* n products of one kind (n > 1: parts = 1) */
template <int OPA, int OPB, int EPI>
static cudaError_t gemm_tc(const GemmArgs* g, int n, int parts, unsigned int* err, cudaStream_t s) {
    /* the weight gradients make two CTAs an SM of four K steps at a usual
     * batch; the rest one CTA of up to eight, all of them in flight at once */
    constexpr int S = EPI == EPI_GRAD ? 4 : 8;
    /* per launch (a cheap host call): the attribute belongs to the current device */
    cudaError_t e = cudaFuncSetAttribute(k_gemm_tc<OPA, OPB, EPI, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         S * G_STAGE_BYTES);
    if (e != cudaSuccess) return e;
    GemmGroup P;
    memset(&P, 0, sizeof(P));
    P.err = err;
    unsigned int tiles = 0;
    int stages = 0;
    for (int i = 0; i < 3; i++) {
        P.first[i] = i < n ? tiles : 0xFFFFFFFFu;
        if (i >= n) continue;
        P.g[i] = g[i];
        stages = std::max(stages, (g[i].kPer + G_K - 1) / G_K);
        tiles += (unsigned int)((g[i].N + G_N - 1) / G_N) * (unsigned int)((g[i].M + G_M - 1) / G_M);
    }
    /* a product of fewer K steps uses as many stages: with a narrow network
     * and a large batch several CTAs then share an SM (4-8-8-8, 1 048 576
     * rows: 1025 -> 340 us a forward pass) */
    const size_t smem = std::max((size_t)std::min(stages, S) * G_STAGE_BYTES, (size_t)G_M * (G_N + 1) * 4);
    return launch_pdl(k_gemm_tc<OPA, OPB, EPI, S>, dim3(tiles, 1, parts), G_THREADS, smem, s, P);
}
/* K parts of a product with few tiles: enough to give every SM one, each at
 * least two K steps deep */
static int k_parts(int M, int N, int K, int* kPer) {
    const int tiles = ((M + G_M - 1) / G_M) * ((N + G_N - 1) / G_N), steps = (K + G_K - 1) / G_K;
    int parts = 148 / tiles;
    if (parts > steps / 2) parts = steps / 2;
    if (parts < 1) parts = 1;
    *kPer = (steps + parts - 1) / parts * G_K;
    return (K + *kPer - 1) / *kPer;
}

/* the SIMT GEMM */
template <class TA, class TB>
static cudaError_t gemm(const TA* A, long long am, long long ak, const TB* B, long long bk, long long bn, float* C,
                        long long cm, int M, int N, int K, const float* bias, int act, cudaStream_t s) {
    dim3 grid((N + 63) / 64, (M + 63) / 64);
    k_gemm<TA, TB><<<grid, 256, 0, s>>>(A, am, ak, B, bk, bn, C, cm, M, N, K, bias, act);
    return cudaGetLastError();
}

}  // namespace vtm

using namespace vtm;

struct vt_mlp {
    int L = 3;
    int dims[4];                          /* in, h1, h2, out */
    int ld[4];                            /* row length of BF16 matrices over dims[l]: a multiple of 8 (16-byte rows) */
    float* w[3] = {}; float* b[3] = {};   /* FP32 masters, w[l]: dims[l] x dims[l+1] */
    __nv_bfloat16* wb[3] = {};            /* BF16 copies, rows of ld[l+1] */
    float* gw[3] = {}; float* gb[3] = {};
    float* mw[3] = {}; float* vw[3] = {}; float* mb[3] = {}; float* vb[3] = {};
    float* loss = nullptr;
    unsigned int* err = nullptr;          /* device word: a bounded tensor-core wait of this network gave up */
    /* SIMT path: FP32 activations (act[0] = input copy) and gradients */
    float* act[4] = {};
    float* dact[4] = {};
    int cap = 0;                          /* batch capacity of these buffers */
    /* tensor-core path: BF16 operands (h: hidden activations, dz: gradients of
     * dims[1..3]; xb: the input), FP32 hidden activations, K parts, column-sum parts */
    __nv_bfloat16* xb = nullptr; __nv_bfloat16* h[3] = {}; __nv_bfloat16* dz[4] = {};
    float* ha[3] = {}; float* part = nullptr; float* cs[4] = {};
    int capF = 0, capB = 0;               /* batch capacity: forward buffers, training buffers */
    long long step = 0;
    bool tc = true;                       /* GEMMs on the tensor cores (tcgen05); false: SIMT FMA */
};

/* A bounded tensor-core wait of this network gave up since the last report:
 * reported by the calls that synchronise (a training step that returns its
 * loss, gradients, reading and setting the weights); until then no training
 * step changes the parameters. */
static vt_status mma_status(vt_mlp* m) {
    unsigned int e = 0;
    if (cudaMemcpy(&e, m->err, sizeof(e), cudaMemcpyDeviceToHost) != cudaSuccess) return vtrt::fail(VT_ERR_CUDA, "MLP status read");
    if (e) {
        cudaMemset(m->err, 0, sizeof(e));
        return vtrt::fail(VT_ERR_TIMEOUT, "a tensor-core GEMM did not complete within its wait bound");
    }
    return VT_OK;
}

static vt_status mlp_buffers(vt_mlp* m, int batch) {
    if (batch <= m->cap) return VT_OK;
    m->cap = 0;
    for (int l = 0; l < 4; l++) { cudaFree(m->act[l]); cudaFree(m->dact[l]); m->act[l] = m->dact[l] = nullptr; }
    for (int l = 0; l < 4; l++) {
        CKM(cudaMalloc(&m->act[l], (size_t)batch * m->dims[l] * 4));
        CKM(cudaMalloc(&m->dact[l], (size_t)batch * m->dims[l] * 4));
    }
    m->cap = batch;
    return VT_OK;
}

/* buffers of the tensor-core path: a forward pass's, and a backward pass's */
static vt_status tc_buffers(vt_mlp* m, int batch, bool train) {
    const int* d = m->dims;
    if (batch > m->capF) {
        m->capF = 0;
        for (int l = 1; l < 3; l++) { cudaFree(m->h[l]); m->h[l] = nullptr; }
        for (int l = 1; l < 3; l++) CKM(cudaMalloc(&m->h[l], (size_t)batch * m->ld[l] * 2));
        m->capF = batch;
    }
    if (train && batch > m->capB) {
        m->capB = 0;
        for (int l = 1; l < 4; l++) { cudaFree(m->dz[l]); cudaFree(m->cs[l]); m->dz[l] = nullptr; m->cs[l] = nullptr; }
        for (int l = 1; l < 3; l++) { cudaFree(m->ha[l]); m->ha[l] = nullptr; }
        cudaFree(m->part); cudaFree(m->xb); m->part = nullptr; m->xb = nullptr;
        CKM(cudaMalloc(&m->xb, (size_t)batch * m->ld[0] * 2));
        size_t part = 0;
        for (int l = 1; l < 4; l++) {
            CKM(cudaMalloc(&m->dz[l], (size_t)batch * m->ld[l] * 2));
            const size_t blocks = l == 3 ? (size_t)(batch + G_M - 1) / G_M : (size_t)(batch + 15) / 16;
            CKM(cudaMalloc(&m->cs[l], blocks * d[l] * 4));
            if (l == 3) break;
            CKM(cudaMalloc(&m->ha[l], (size_t)batch * d[l] * 4));
            /* k_parts' tiles and parts multiply to 148 at most, where there is
             * more than one part: room for any batch up to this one */
            const size_t rows = (size_t)148 * G_M / ((d[l] + G_N - 1) / G_N);
            const size_t need = (rows > (size_t)batch ? rows : (size_t)batch) * d[l];
            if (need > part) part = need;
        }
        CKM(cudaMalloc(&m->part, part * 4));
        m->capB = batch;
    }
    return VT_OK;
}

extern "C" vt_status vt_mlp_create(int in, int h1, int h2, int out, uint64_t seed, vt_mlp** res) {
    vtrt::clear_error();
    if (!res || in <= 0 || h1 <= 0 || h2 <= 0 || out <= 0) return vtrt::fail(VT_ERR_INVALID, "bad MLP shape");
    vt_mlp* m = new vt_mlp();
    int d[4] = {in, h1, h2, out};
    memcpy(m->dims, d, sizeof(d));
    for (int l = 0; l < 4; l++) m->ld[l] = (d[l] + 7) & ~7;
    /* He initialisation (normal, std sqrt(2/fan_in)) from splitmix64 + Box-Muller; biases 0 */
    uint64_t k = vtrt::splitmix64(seed ^ 0x4D4C50ull);
    for (int l = 0; l < 3; l++) {
        long long n = (long long)d[l] * d[l + 1];
        std::vector<float> w(n);
        float sd = sqrtf(2.0f / (float)d[l]);
        for (long long i = 0; i < n; i++) {
            double u1 = ((vtrt::splitmix64(k++) >> 11) + 1.0) * (1.0 / 9007199254740993.0);
            double u2 = (vtrt::splitmix64(k++) >> 11) * (1.0 / 9007199254740992.0);
            w[i] = (float)(sd * std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2));
        }
        vt_status st = VT_OK;
        cudaError_t e = cudaSuccess;
        size_t nb = (size_t)d[l + 1] * 4;
        if ((e = cudaMalloc(&m->w[l], n * 4)) != cudaSuccess || (e = cudaMalloc(&m->wb[l], (size_t)d[l] * m->ld[l + 1] * 2)) != cudaSuccess ||
            (e = cudaMalloc(&m->b[l], nb)) != cudaSuccess || (e = cudaMalloc(&m->gw[l], n * 4)) != cudaSuccess ||
            (e = cudaMalloc(&m->gb[l], nb)) != cudaSuccess || (e = cudaMalloc(&m->mw[l], n * 4)) != cudaSuccess ||
            (e = cudaMalloc(&m->vw[l], n * 4)) != cudaSuccess || (e = cudaMalloc(&m->mb[l], nb)) != cudaSuccess ||
            (e = cudaMalloc(&m->vb[l], nb)) != cudaSuccess) {
            st = vtrt::fail(VT_ERR_NOMEM, "MLP alloc: %s", cudaGetErrorString(e));
        }
        if (st == VT_OK) {
            cudaMemcpy(m->w[l], w.data(), n * 4, cudaMemcpyHostToDevice);
            cudaMemset(m->b[l], 0, nb);
            cudaMemset(m->mw[l], 0, n * 4); cudaMemset(m->vw[l], 0, n * 4);
            cudaMemset(m->mb[l], 0, nb); cudaMemset(m->vb[l], 0, nb);
            k_to_bf16<<<g1(n), 256>>>(m->w[l], m->wb[l], n, d[l + 1], m->ld[l + 1]);
            if ((e = cudaDeviceSynchronize()) != cudaSuccess) st = vtrt::fail(VT_ERR_CUDA, "MLP init: %s", cudaGetErrorString(e));
        }
        if (st != VT_OK) { vt_mlp_free(m); return st; }
    }
    if (cudaMalloc(&m->loss, 8) != cudaSuccess) { vt_mlp_free(m); return vtrt::fail(VT_ERR_NOMEM, "MLP loss"); }
    m->err = (unsigned int*)m->loss + 1;
    if (cudaMemset(m->loss, 0, 8) != cudaSuccess) { vt_mlp_free(m); return vtrt::fail(VT_ERR_CUDA, "MLP init"); }
    *res = m;
    return VT_OK;
}

extern "C" void vt_mlp_free(vt_mlp* m) {
    if (!m) return;
    for (int l = 0; l < 3; l++) {
        cudaFree(m->w[l]); cudaFree(m->wb[l]); cudaFree(m->b[l]); cudaFree(m->gw[l]); cudaFree(m->gb[l]);
        cudaFree(m->mw[l]); cudaFree(m->vw[l]); cudaFree(m->mb[l]); cudaFree(m->vb[l]);
    }
    for (int l = 0; l < 4; l++) { cudaFree(m->act[l]); cudaFree(m->dact[l]); cudaFree(m->dz[l]); cudaFree(m->cs[l]); }
    for (int l = 0; l < 3; l++) { cudaFree(m->h[l]); cudaFree(m->ha[l]); }
    cudaFree(m->part); cudaFree(m->xb); cudaFree(m->loss);
    delete m;
}

/* forward pass on the tensor cores: `batch` rows of x (batch x in, FP32) to
 * probabilities p (NULL: none kept) through the hidden operands h1, h2; with
 * targets y also the training pass's buffers */
static vt_status forward_tc(vt_mlp* m, const float* x, int batch, float* p, __nv_bfloat16* h1, __nv_bfloat16* h2,
                            const float* y, cudaStream_t s) {
    const int* d = m->dims;
    GemmArgs g;
    memset(&g, 0, sizeof(g));
    g.M = batch;
    g.A = x; g.lda = d[0]; g.B = m->wb[0]; g.ldb = m->ld[1]; g.N = d[1]; g.K = g.kPer = d[0]; g.bias = m->b[0];
    g.Cb = h1; g.ldcb = m->ld[1]; g.C = y ? m->ha[1] : nullptr; g.ldc = d[1];
    g.loss = y ? m->loss : nullptr;   /* cleared */
    g.Xb = y ? m->xb : nullptr; g.ldx = m->ld[0];
    CKM((gemm_tc<OP_F32_K, OP_BF16_MN, EPI_HIDDEN>(&g, 1, 1, m->err, s)));
    g.loss = nullptr;
    g.A = h1; g.lda = m->ld[1]; g.B = m->wb[1]; g.ldb = m->ld[2]; g.N = d[2]; g.K = g.kPer = d[1]; g.bias = m->b[1];
    g.Cb = h2; g.ldcb = m->ld[2]; g.C = y ? m->ha[2] : nullptr; g.ldc = d[2];
    CKM((gemm_tc<OP_BF16_K, OP_BF16_MN, EPI_HIDDEN>(&g, 1, 1, m->err, s)));
    g.A = h2; g.lda = m->ld[2]; g.B = m->wb[2]; g.ldb = m->ld[3]; g.N = d[3]; g.K = g.kPer = d[2]; g.bias = m->b[2];
    g.C = p; g.ldc = d[3];
    g.Y = y; g.invB = 1.0f / batch; g.loss = m->loss; g.Cb = m->dz[3]; g.ldcb = m->ld[3]; g.colsum = m->cs[3];
    CKM((gemm_tc<OP_BF16_K, OP_BF16_MN, EPI_OUT>(&g, 1, 1, m->err, s)));
    return VT_OK;
}

/* training pass on the tensor cores: forward, the gradients to the hidden
 * layers, the three weight gradients in one launch, the update (adam NULL:
 * gradients into gw/gb only) */
static vt_status train_tc(vt_mlp* m, const float* x, const float* y, int batch, const Adam* adam, cudaStream_t s) {
    vt_status st = tc_buffers(m, batch, true);
    if (st != VT_OK) return st;
    if ((st = forward_tc(m, x, batch, nullptr, m->h[1], m->h[2], y, s)) != VT_OK) return st;
    const int* d = m->dims;
    for (int l = 2; l > 0; l--) {
        GemmArgs g;
        memset(&g, 0, sizeof(g));
        g.A = m->dz[l + 1]; g.lda = m->ld[l + 1]; g.B = m->wb[l]; g.ldb = m->ld[l + 1];
        g.M = batch; g.N = d[l]; g.K = d[l + 1];
        g.C = m->part;
        const int parts = k_parts(g.M, g.N, g.K, &g.kPer);
        CKM((gemm_tc<OP_BF16_K, OP_BF16_K, EPI_PART>(&g, 1, parts, m->err, s)));
        CKM(launch_pdl(k_dgrad_finish, dim3(((unsigned int)d[l] + 63) / 64 * (((unsigned int)batch + 15) / 16)), 256, 0, s,
                       m->part, parts, m->ha[l], batch, d[l], m->dz[l], m->ld[l], m->cs[l]));
    }
    GemmArgs g[3];
    UpdateArgs u;
    memset(g, 0, sizeof(g));
    memset(&u, 0, sizeof(u));
    unsigned int blocks = 0;
    for (int l = 2, i = 0; l >= 0; l--, i++) {   /* the largest first */
        g[i].A = l ? m->h[l] : m->xb; g[i].lda = m->ld[l]; g[i].B = m->dz[l + 1]; g[i].ldb = m->ld[l + 1];
        g[i].M = d[l]; g[i].N = d[l + 1]; g[i].K = g[i].kPer = batch;
        g[i].C = m->gw[l]; g[i].ldc = d[l + 1];
    }
    CKM((gemm_tc<OP_BF16_MN, OP_BF16_MN, EPI_GRAD>(g, 3, 1, m->err, s)));
    for (int l = 0; l < 3; l++) {
        u.w[l] = m->w[l]; u.m[l] = m->mw[l]; u.v[l] = m->vw[l]; u.g[l] = m->gw[l]; u.wb[l] = m->wb[l];
        u.rows[l] = d[l]; u.N[l] = d[l + 1]; u.ldb[l] = m->ld[l + 1];
        u.b[l] = m->b[l]; u.bm[l] = m->mb[l]; u.bv[l] = m->vb[l]; u.gb[l] = m->gb[l];
        u.part[l] = m->cs[l + 1]; u.parts[l] = l == 2 ? (batch + G_M - 1) / G_M : (batch + 15) / 16;
        u.first[l] = blocks;
        if (adam) blocks += (unsigned int)(((long long)d[l] * d[l + 1] + 1023) / 1024);
    }
    for (int l = 0; l < 3; l++) {
        u.first[3 + l] = blocks;
        blocks += (unsigned int)(d[l + 1] + 255) / 256;
    }
    if (adam) { u.adam = *adam; u.step = 1; }
    u.err = m->err;
    CKM(launch_pdl(k_update, dim3(blocks), 256, 0, s, u));
    return VT_OK;
}

/* the same passes on the SIMT pipes */
static vt_status forward_simt(vt_mlp* m, const float* x, int batch, cudaStream_t s) {
    vt_status st = mlp_buffers(m, batch);
    if (st != VT_OK) return st;
    const int* d = m->dims;
    CKM(cudaMemcpyAsync(m->act[0], x, (size_t)batch * d[0] * 4, cudaMemcpyDeviceToDevice, s));
    for (int l = 0; l < 3; l++)
        CKM((gemm<float, __nv_bfloat16>(m->act[l], d[l], 1, m->wb[l], m->ld[l + 1], 1, m->act[l + 1], d[l + 1], batch,
                                       d[l + 1], d[l], m->b[l], l < 2 ? ACT_RELU : ACT_SIGMOID, s)));
    return VT_OK;
}

extern "C" vt_status vt_mlp_forward(vt_mlp* m, const float* dev_x, int batch, float* dev_p, void* stream) {
    vtrt::clear_error();
    if (!m || !dev_x || !dev_p || batch <= 0) return vtrt::fail(VT_ERR_INVALID, "vt_mlp_forward: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    vt_status st;
    if (m->tc) {
        if ((st = tc_buffers(m, batch, false)) != VT_OK) return st;
        return forward_tc(m, dev_x, batch, dev_p, m->h[1], m->h[2], nullptr, s);
    }
    if ((st = forward_simt(m, dev_x, batch, s)) != VT_OK) return st;
    CKM(cudaMemcpyAsync(dev_p, m->act[3], (size_t)batch * m->dims[3] * 4, cudaMemcpyDeviceToDevice, s));
    return VT_OK;
}

/* gradients of the mean BCE over the batch into gw/gb; loss into m->loss */
static vt_status backward_simt(vt_mlp* m, const float* y, int batch, cudaStream_t s) {
    const int* d = m->dims;
    long long no = (long long)batch * d[3];
    CKM(cudaMemsetAsync(m->loss, 0, 4, s));
    k_bce_grad<<<g1(no), 256, 0, s>>>(m->act[3], y, m->dact[3], no, 1.0f / batch, m->loss);
    for (int l = 2; l >= 0; l--) {
        /* gW[l] = act[l]^T dact[l+1]   (d[l] x d[l+1]) */
        CKM((gemm<float, float>(m->act[l], 1, d[l], m->dact[l + 1], d[l + 1], 1, m->gw[l], d[l + 1], d[l], d[l + 1],
                               batch, nullptr, ACT_NONE, s)));
        k_colsum<<<(d[l + 1] + 255) / 256, 256, 0, s>>>(m->dact[l + 1], batch, d[l + 1], m->gb[l]);
        if (l > 0) {
            /* dact[l] = dact[l+1] W[l]^T, masked by ReLU */
            CKM((gemm<float, __nv_bfloat16>(m->dact[l + 1], d[l + 1], 1, m->wb[l], 1, m->ld[l + 1], m->dact[l], d[l], batch,
                                           d[l], d[l + 1], nullptr, ACT_NONE, s)));
            k_relu_mask<<<g1((long long)batch * d[l]), 256, 0, s>>>(m->dact[l], m->act[l], (long long)batch * d[l]);
        }
    }
    CKM(cudaGetLastError());
    return VT_OK;
}

extern "C" vt_status vt_mlp_train_step(vt_mlp* m, const float* dev_x, const float* dev_y, int batch, float lr,
                                       float* loss, void* stream) {
    vtrt::clear_error();
    if (!m || !dev_x || !dev_y || batch <= 0) return vtrt::fail(VT_ERR_INVALID, "vt_mlp_train_step: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    const float b1 = 0.9f, b2 = 0.999f;
    const Adam o = {lr, b1, b2, 1e-8f, 1.0f - powf(b1, (float)(m->step + 1)), 1.0f - powf(b2, (float)(m->step + 1))};
    vt_status st;
    if (m->tc) {
        if ((st = train_tc(m, dev_x, dev_y, batch, &o, s)) != VT_OK) return st;
    } else {
        if ((st = forward_simt(m, dev_x, batch, s)) != VT_OK) return st;
        if ((st = backward_simt(m, dev_y, batch, s)) != VT_OK) return st;
        for (int l = 0; l < 3; l++) {
            const int N = m->dims[l + 1];
            long long n = (long long)m->dims[l] * N;
            k_adam<<<g1(n), 256, 0, s>>>(m->w[l], m->wb[l], m->gw[l], m->mw[l], m->vw[l], n, N, m->ld[l + 1], o);
            k_adam<<<g1(N), 256, 0, s>>>(m->b[l], nullptr, m->gb[l], m->mb[l], m->vb[l], N, N, N, o);
        }
        CKM(cudaGetLastError());
    }
    m->step++;
    if (loss) {
        CKM(cudaMemcpyAsync(loss, m->loss, 4, cudaMemcpyDeviceToHost, s));
        CKM(cudaStreamSynchronize(s));
        return mma_status(m);
    }
    return VT_OK;
}

/* gradients only (no update), for checking against a CPU implementation:
 * host buffers laid out as the weights (layer by layer: W then b) */
extern "C" vt_status vt_mlp_gradients(vt_mlp* m, const float* dev_x, const float* dev_y, int batch, float* host_grads,
                                      float* loss) {
    vtrt::clear_error();
    if (!m || !dev_x || !dev_y || !host_grads || batch <= 0) return vtrt::fail(VT_ERR_INVALID, "bad arguments");
    vt_status st;
    if (m->tc) {
        if ((st = train_tc(m, dev_x, dev_y, batch, nullptr, 0)) != VT_OK) return st;
    } else {
        if ((st = forward_simt(m, dev_x, batch, 0)) != VT_OK) return st;
        if ((st = backward_simt(m, dev_y, batch, 0)) != VT_OK) return st;
    }
    CKM(cudaDeviceSynchronize());
    size_t o = 0;
    for (int l = 0; l < 3; l++) {
        size_t n = (size_t)m->dims[l] * m->dims[l + 1];
        CKM(cudaMemcpy(host_grads + o, m->gw[l], n * 4, cudaMemcpyDeviceToHost)); o += n;
        CKM(cudaMemcpy(host_grads + o, m->gb[l], (size_t)m->dims[l + 1] * 4, cudaMemcpyDeviceToHost)); o += m->dims[l + 1];
    }
    if (loss) CKM(cudaMemcpy(loss, m->loss, 4, cudaMemcpyDeviceToHost));
    return mma_status(m);
}

extern "C" vt_status vt_debug_mlp_timeout(vt_mlp* m) {
    vtrt::clear_error();
    if (!m) return vtrt::fail(VT_ERR_INVALID, "null argument");
    const unsigned int e = 1;
    CKM(cudaDeviceSynchronize());
    CKM(cudaMemcpy(m->err, &e, sizeof(e), cudaMemcpyHostToDevice));
    return VT_OK;
}

extern "C" vt_status vt_mlp_use_tensor_cores(vt_mlp* m, int on) {
    vtrt::clear_error();
    if (!m) return vtrt::fail(VT_ERR_INVALID, "null argument");
    m->tc = on != 0;
    return VT_OK;
}

extern "C" vt_status vt_mlp_info(const vt_mlp* m, int dims[4]) {
    vtrt::clear_error();
    if (!m || !dims) return vtrt::fail(VT_ERR_INVALID, "null argument");
    memcpy(dims, m->dims, sizeof(m->dims));
    return VT_OK;
}

/* FP32 master weights (layer by layer: W [in x out] then b [out]) */
extern "C" vt_status vt_mlp_get_weights(vt_mlp* m, float* host, int64_t* n) {
    vtrt::clear_error();
    if (!m || !n) return vtrt::fail(VT_ERR_INVALID, "null argument");
    int64_t total = 0;
    for (int l = 0; l < 3; l++) total += (int64_t)m->dims[l] * m->dims[l + 1] + m->dims[l + 1];
    int64_t cap = *n;
    *n = total;
    if (!host) return VT_OK;
    if (cap < total) return vtrt::fail(VT_ERR_INVALID, "need %lld floats", (long long)total);
    CKM(cudaDeviceSynchronize());
    const vt_status st = mma_status(m);
    if (st != VT_OK) return st;
    size_t o = 0;
    for (int l = 0; l < 3; l++) {
        size_t nw = (size_t)m->dims[l] * m->dims[l + 1];
        CKM(cudaMemcpy(host + o, m->w[l], nw * 4, cudaMemcpyDeviceToHost)); o += nw;
        CKM(cudaMemcpy(host + o, m->b[l], (size_t)m->dims[l + 1] * 4, cudaMemcpyDeviceToHost)); o += m->dims[l + 1];
    }
    return VT_OK;
}

extern "C" vt_status vt_mlp_set_weights(vt_mlp* m, const float* host, int64_t n) {
    vtrt::clear_error();
    if (!m || !host) return vtrt::fail(VT_ERR_INVALID, "null argument");
    int64_t total = 0;
    for (int l = 0; l < 3; l++) total += (int64_t)m->dims[l] * m->dims[l + 1] + m->dims[l + 1];
    if (n != total) return vtrt::fail(VT_ERR_INVALID, "expected %lld floats", (long long)total);
    size_t o = 0;
    for (int l = 0; l < 3; l++) {
        size_t nw = (size_t)m->dims[l] * m->dims[l + 1];
        CKM(cudaMemcpy(m->w[l], host + o, nw * 4, cudaMemcpyHostToDevice)); o += nw;
        CKM(cudaMemcpy(m->b[l], host + o, (size_t)m->dims[l + 1] * 4, cudaMemcpyHostToDevice)); o += m->dims[l + 1];
        k_to_bf16<<<g1((long long)nw), 256>>>(m->w[l], m->wb[l], (long long)nw, m->dims[l + 1], m->ld[l + 1]);
    }
    CKM(cudaDeviceSynchronize());
    return mma_status(m);
}

/* ------------------------------------------------------------------------ */
/* Allocation-free inference                                                */
/* ------------------------------------------------------------------------ */
/* Some callers cannot allocate GPU memory at the point where they run the
 * prefetch network: a render loop inside a host application that owns the
 * device's memory (its own pool, a fixed budget), or a frame thread that
 * must not call cudaMalloc because it synchronises the device and can stall
 * the frame.  vt_mlp_forward_noalloc serves them: its two hidden-layer
 * activations live in this fixed, file-scope device array instead of the
 * handle's lazily allocated buffers.  Every GPU that loads libvt.so holds
 * the array (1 MiB) until the process exits. */
#define VT_MLP_NOALLOC_FLOATS (1 << 18)
static __device__ __align__(256) float g_mlp_noalloc_scratch[VT_MLP_NOALLOC_FLOATS];

#include <mutex>
static std::mutex g_noalloc_mu;
static float* g_noalloc_dev[256];   /* per device: address of the array, looked up once */

extern "C" vt_status vt_mlp_forward_noalloc(vt_mlp* m, const float* dev_x, int batch, float* dev_p, void* stream) {
    vtrt::clear_error();
    if (!m || !dev_x || !dev_p || batch <= 0) return vtrt::fail(VT_ERR_INVALID, "vt_mlp_forward_noalloc: bad arguments");
    const int* d = m->dims;
    long long need = (long long)batch * (d[1] + d[2]);
    if (need > VT_MLP_NOALLOC_FLOATS)
        return vtrt::fail(VT_ERR_INVALID,
                          "vt_mlp_forward_noalloc: batch %d x (%d + %d) hidden units = %lld floats exceeds the "
                          "static scratch of %d floats", batch, d[1], d[2], need, VT_MLP_NOALLOC_FLOATS);
    int dev = 0;
    CKM(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 256) return vtrt::fail(VT_ERR_UNSUPPORTED, "device ordinal %d", dev);
    float* scratch = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (g_noalloc_dev[dev]) {
            /* an address looked up before a cudaDeviceReset belongs to the
             * destroyed context: the runtime no longer knows it as device
             * memory of this device, so it is looked up again (a host query,
             * no allocation) */
            cudaPointerAttributes pa;
            if (cudaPointerGetAttributes(&pa, g_noalloc_dev[dev]) != cudaSuccess || pa.type != cudaMemoryTypeDevice ||
                pa.device != dev) {
                cudaGetLastError();
                g_noalloc_dev[dev] = nullptr;
            }
        }
        if (!g_noalloc_dev[dev]) {
            /* host code only sees a stand-in for the array: its device address
             * comes from the runtime, once per device (and context), with
             * that device current */
            void* p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_mlp_noalloc_scratch);
            if (e != cudaSuccess)
                return vtrt::fail(VT_ERR_CUDA, "cudaGetSymbolAddress(g_mlp_noalloc_scratch): %s", cudaGetErrorString(e));
            g_noalloc_dev[dev] = (float*)p;
        }
        scratch = g_noalloc_dev[dev];
    }
    cudaStream_t s = (cudaStream_t)stream;
    /* every activation element is written before it is read, so the array's
     * leftovers from the previous call need no clearing */
    if (m->tc) {
        /* BF16 rows of whole 16-byte chunks: with layers narrower than 8 they
         * can take more than the bound above allows for, so by row blocks */
        const int per = m->ld[1] + m->ld[2], rows = 2 * VT_MLP_NOALLOC_FLOATS / per;
        for (int r = 0; r < batch; r += rows) {
            const int nb = batch - r < rows ? batch - r : rows;
            __nv_bfloat16* h1 = (__nv_bfloat16*)scratch;
            vt_status st = forward_tc(m, dev_x + (size_t)r * d[0], nb, dev_p + (size_t)r * d[3], h1,
                                      h1 + (size_t)nb * m->ld[1], nullptr, s);
            if (st != VT_OK) return st;
        }
        return VT_OK;
    }
    float* h1 = scratch;
    float* h2 = scratch + (size_t)batch * d[1];
    CKM((gemm<float, __nv_bfloat16>(dev_x, d[0], 1, m->wb[0], m->ld[1], 1, h1, d[1], batch, d[1], d[0], m->b[0], ACT_RELU, s)));
    CKM((gemm<float, __nv_bfloat16>(h1, d[1], 1, m->wb[1], m->ld[2], 1, h2, d[2], batch, d[2], d[1], m->b[1], ACT_RELU, s)));
    CKM((gemm<float, __nv_bfloat16>(h2, d[2], 1, m->wb[2], m->ld[3], 1, dev_p, d[3], batch, d[3], d[2], m->b[2],
                                    ACT_SIGMOID, s)));
    return VT_OK;
}
