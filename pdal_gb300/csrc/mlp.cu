/*
 * mlp.cu -- training and inference of the warm-start MLP (include/pdal_learn.h)
 * with the library's own CUDA kernels (sm_103a).
 *
 * The network is three layers of width 256.  Training runs in FP32 on
 * register-tiled SIMT GEMMs with the bias, ReLU, loss, ReLU gradient and Adam
 * update in their epilogues.  BF16 inference runs its three products on the
 * tensor cores (mma.sync m16n8k16, FP32 accumulation, k_gemm_bf16_tc), each
 * layer writing the next one's BF16 operand.  All reductions run in a fixed
 * order, so a training run and a prediction are reproducible bit for bit.
 */
#include "../../include/pdal_learn.h"
#include "common.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <numeric>
#include <random>
#include <string>
#include <vector>

namespace pdal {
namespace {

thread_local std::string g_mlp_error;

constexpr int GT = 256;

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
/* 16 bytes, the first `bytes` of them from src and zeros behind */
__device__ __forceinline__ void cp_async16(void *dst, const void *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(bytes) : "memory");
}
/* four bytes, zeros when !in */
__device__ __forceinline__ void cp_async4(void *dst, const void *src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(in ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

/* ---- FP32 products ---------------------------------------------------- */
/*
 * C[M][N] = sum_k A(m, k) B(k, n): every element one chain of FP32 fused
 * multiply-adds in k order, whatever the tile.  The operands' elements are
 *   A(m, k)  A[row(m) * lda + k], or with TA A[row(k) * lda + m]
 *   B(k, n)  B[k * ldb + n],      or with TB B[n * ldb + k]
 * where row(i) = rows ? rows[i] : i picks the rows of a mini-batch in place.
 *
 * The network's products are small and long (layer 1 at a batch of 128: 128 x
 * 256 outputs of 3,280 terms), so what bounds them is how many SMs have a
 * tile and how far ahead of the chain the loads run: tiles of 64, 32 or 16
 * squared, the largest that gives every SM one, fed by a ring of stages of 32
 * or 64 terms (cp.async, 16 bytes where an operand's rows are aligned and run
 * along its stage's rows, else 4: the output layer's rows have odd lengths).
 * A is kept [m][k] in shared memory (one 128-bit load per row and four
 * terms), or [k][m] with TA.
 * Measured (3,280 -> 256 -> 256 -> 1,681, batch 128): a training step 98 us,
 * against 1,070 us with 64 x 64 tiles only, whose layer 1 ran in 8 blocks, and
 * separate gather, bias, ReLU, loss, column-sum and Adam passes.  Layer 1 takes
 * 34 us of it and is bound by the issue of one warp per scheduler along its
 * 3,280-term chains; splitting the sums over clusters was 7 us a step slower
 * end to end and changes the rounding, which Adam's first steps amplify.
 */
struct GemmOp {
    int M, N, K;
    const float *A, *B;
    long long lda, ldb;
    const int *rows;
};

template <int BT, bool TA>
struct Tile {
    static constexpr int TK = BT == 16 ? 64 : 32;
    static constexpr int RM = BT == 64 ? 4 : BT == 32 ? 2 : 1; /* a thread's rows and columns */
    static constexpr int RN = BT == 64 ? 4 : 2;
    static constexpr int NT = BT * BT / (RM * RN);
    static constexpr int STAGES = BT == 64 ? 3 : 4;
    static constexpr int LA = TA ? BT + 4 : TK + 4, NA = TA ? TK : BT; /* A's row length and rows */
    static constexpr int LB = BT + 4;
    struct Stage {
        float a[NA][LA];
        float b[TK][LB];
    };
    static constexpr size_t BYTES = sizeof(Stage) * STAGES;
};

/* The thread's RM x RN outputs of the tile at (m0, n0); elements outside the
 * matrices count as zeros.  With `colsum`, thread n < BT also adds the B
 * elements of column n in k order. */
template <int BT, bool TA, bool TB>
__device__ __forceinline__ void tile_sum(const GemmOp &g, int m0, int n0, unsigned char *smem,
                                         float (&acc)[Tile<BT, TA>::RM][Tile<BT, TA>::RN], float *colsum) {
    using T = Tile<BT, TA>;
    constexpr int TK = T::TK, RM = T::RM, RN = T::RN, NT = T::NT, ST = T::STAGES;
    auto *st = reinterpret_cast<typename T::Stage *>(smem);
    const int tid = threadIdx.x, tx = tid % (BT / RN), ty = tid / (BT / RN);
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = 0.f;
    const int steps = (g.K + TK - 1) / TK;
    constexpr int LD = BT * TK / NT; /* elements of each operand a thread copies per stage */
    static_assert(LD % 4 == 0 && NT % (TK / 4) == 0 && NT % (BT / 4) == 0, "whole vectors, one column per thread");
    /* neighbouring threads take neighbouring addresses; whole 16-byte vectors
     * where every row starts on one */
    const bool va = g.lda % 4 == 0 && ((uintptr_t)g.A & 15) == 0;
    const bool vb = !TB && g.ldb % 4 == 0 && ((uintptr_t)g.B & 15) == 0;
    constexpr int FA = TA ? BT : TK; /* A's contiguous index and the others */
    /* without TA the rows a thread copies are the same in every stage: found
     * once, so that no copy waits for a row number */
    const float *arow[TA ? 1 : LD];
    if (!TA) {
#pragma unroll
        for (int q = 0; q < LD; ++q) {
            const int e = va ? 4 * (tid + (q < LD / 4 ? q : 0) * NT) : tid + q * NT, m = m0 + e / FA;
            arow[TA ? 0 : q] =
                m < g.M ? g.A + (long long)(g.rows ? g.rows[m] : m) * g.lda + e % FA : nullptr;
        }
    }
    auto copy = [&](int step) {
        typename T::Stage &s = st[step % ST];
        const int k0 = step * TK;
        if (va) {
#pragma unroll
            for (int q = 0; q < LD / 4; ++q) {
                const int e = 4 * (tid + q * NT), f = e % FA, r = e / FA;
                const int m = m0 + f, k = k0 + (TA ? r : f);
                int bytes = max(0, min(16, 4 * (TA ? g.M - m : g.K - k)));
                if (TA ? k >= g.K : !arow[TA ? 0 : q]) bytes = 0;
                const float *src = g.A;
                if (bytes) src = TA ? g.A + (long long)(g.rows ? g.rows[k] : k) * g.lda + m : arow[TA ? 0 : q] + k0;
                cp_async16(&s.a[r][f], src, bytes);
            }
        } else {
#pragma unroll
            for (int q = 0; q < LD; ++q) {
                const int e = tid + q * NT, f = e % FA, r = e / FA;
                const int m = m0 + f, k = k0 + (TA ? r : f);
                const bool in = k < g.K && (TA ? m < g.M : arow[TA ? 0 : q] != nullptr);
                const float *src = g.A;
                if (in) src = TA ? g.A + (long long)(g.rows ? g.rows[k] : k) * g.lda + m : arow[TA ? 0 : q] + k0;
                cp_async4(&s.a[r][f], src, in);
            }
        }
        if (vb) {
#pragma unroll
            for (int q = 0; q < LD / 4; ++q) {
                const int e = 4 * (tid + q * NT), n = n0 + e % BT, k = k0 + e / BT;
                const int bytes = k < g.K ? max(0, min(16, 4 * (g.N - n))) : 0;
                cp_async16(&s.b[e / BT][e % BT], bytes ? g.B + (long long)k * g.ldb + n : g.B, bytes);
            }
        } else {
#pragma unroll
            for (int q = 0; q < LD; ++q) {
                const int e = tid + q * NT;
                const int nn = TB ? e / TK : e % BT, kb = TB ? e % TK : e / BT, n = n0 + nn, k = k0 + kb;
                const bool in = n < g.N && k < g.K;
                cp_async4(&s.b[kb][nn],
                          in ? g.B + (TB ? (long long)n * g.ldb + k : (long long)k * g.ldb + n) : g.B, in);
            }
        }
    };
#pragma unroll
    for (int q = 0; q < ST - 1; ++q) {
        if (q < steps) copy(q);
        cp_async_commit();
    }
    for (int t = 0; t < steps; ++t) {
        cp_async_wait<ST - 2>();
        __syncthreads(); /* stage t has landed, stage t - 1 is free */
        if (t + ST - 1 < steps) copy(t + ST - 1);
        cp_async_commit();
        const typename T::Stage &s = st[t % ST];
        /* four terms at a time, the next four loaded before these are used */
        float a[2][RM][4], b[2][4][RN];
        auto fetch = [&](int kk, float (&fa)[RM][4], float (&fb)[4][RN]) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (RN == 4) {
                    const float4 v = *reinterpret_cast<const float4 *>(&s.b[kk + q][tx * RN]);
                    fb[q][0] = v.x;
                    fb[q][1] = v.y;
                    fb[q][RN - 2] = v.z;
                    fb[q][RN - 1] = v.w;
                } else {
                    const float2 v = *reinterpret_cast<const float2 *>(&s.b[kk + q][tx * RN]);
                    fb[q][0] = v.x;
                    fb[q][1] = v.y;
                }
            }
            if (TA) {
                static_assert(!TA || RM == 4, "one 128-bit load per term");
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 v = *reinterpret_cast<const float4 *>(&s.a[TA ? kk + q : 0][TA ? ty * RM : 0]);
                    fa[0][q] = v.x;
                    fa[RM > 1 ? 1 : 0][q] = v.y;
                    fa[RM > 2 ? 2 : 0][q] = v.z;
                    fa[RM > 3 ? 3 : 0][q] = v.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    const float4 v = *reinterpret_cast<const float4 *>(&s.a[TA ? 0 : ty * RM + i][TA ? 0 : kk]);
                    fa[i][0] = v.x;
                    fa[i][1] = v.y;
                    fa[i][2] = v.z;
                    fa[i][3] = v.w;
                }
            }
        };
        fetch(0, a[0], b[0]);
#pragma unroll
        for (int kk = 0; kk < TK; kk += 4) {
            const int c = (kk >> 2) & 1;
            if (kk + 4 < TK) fetch(kk + 4, a[c ^ 1], b[c ^ 1]);
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int i = 0; i < RM; ++i)
#pragma unroll
                    for (int j = 0; j < RN; ++j) acc[i][j] = fmaf(a[c][i][q], b[c][q][j], acc[i][j]);
        }
        if (colsum && tid < BT)
#pragma unroll
            for (int kk = 0; kk < TK; ++kk) *colsum += s.b[kk][tid];
    }
    cp_async_wait<0>();
}

/* what becomes of a finished element v of C */
enum class Finish {
    bias_relu, /* C = max(v + bias, 0) */
    bias,      /* C = v + bias */
    mask,      /* C = H > 0 ? v : 0 (the ReLU's gradient) */
    mse        /* P = v + bias: C = scale * (P - Y), the block's sum of (P - Y)^2 in FP64 */
};
struct GemmOut {
    float *C;
    const float *bias, *H, *Y;
    const int *rows; /* rows of Y */
    float scale;
    double *loss; /* one per block */
};

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <int BT, bool TB, Finish F>
__global__ void __launch_bounds__(Tile<BT, false>::NT) k_gemm(GemmOp g, GemmOut o) {
    using T = Tile<BT, false>;
    extern __shared__ __align__(16) unsigned char gemm_smem[];
    __shared__ double sb[T::NT / 32];
    pdl_wait();
    const int m0 = blockIdx.y * BT, n0 = blockIdx.x * BT;
    float acc[T::RM][T::RN];
    tile_sum<BT, false, TB>(g, m0, n0, gemm_smem, acc, nullptr);
    const int tx = threadIdx.x % (BT / T::RN), ty = threadIdx.x / (BT / T::RN);
    double loss = 0.0;
#pragma unroll
    for (int i = 0; i < T::RM; ++i)
#pragma unroll
        for (int j = 0; j < T::RN; ++j) {
            const int m = m0 + ty * T::RM + i, n = n0 + tx * T::RN + j;
            if (m >= g.M || n >= g.N) continue;
            const float v = acc[i][j];
            float *c = o.C + (size_t)m * g.N + n;
            if (F == Finish::bias_relu) {
                *c = fmaxf(v + o.bias[n], 0.f);
            } else if (F == Finish::bias) {
                *c = v + o.bias[n];
            } else if (F == Finish::mask) {
                *c = o.H[(size_t)m * g.N + n] > 0.f ? v : 0.f;
            } else {
                const float d = (v + o.bias[n]) - o.Y[(size_t)(o.rows ? o.rows[m] : m) * g.N + n];
                if (o.C) *c = o.scale * d;
                loss += (double)d * (double)d;
            }
        }
    if (F == Finish::mse) {
        for (int q = 16; q > 0; q >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, q);
        if ((threadIdx.x & 31) == 0) sb[threadIdx.x >> 5] = loss;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < T::NT / 32; ++w) t += sb[w];
            o.loss[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = t;
        }
    }
}

/* The weight gradients dW = A^T dZ and bias gradients (the column sums of dZ,
 * in row order) of the three layers in one launch; each element is stored, or
 * goes straight into its Adam update, so that a training step writes no
 * gradient.  The last block adds the batch's loss to `loss_sum`. */
struct LayerGrad {
    GemmOp g; /* M x N = the weight's shape, K = rows of the batch */
    size_t w, b; /* offsets of the weight and the bias in the parameter vector */
    int tiles_n, first; /* tiles along N, first block */
};
struct AdamArgs {
    float *p, *m, *v, *grad; /* grad: store the gradient instead of updating */
    float lr, b1, b2, eps, bc1, bc2;
};
struct WeightArgs {
    LayerGrad l[3];
    AdamArgs adam;
    const double *loss;
    int nloss;
    double inv_count, *loss_sum;
};

__global__ void __launch_bounds__(GT, 3) k_weights(WeightArgs W) {
    using T = Tile<64, true>;
    static_assert(T::NT == GT, "one thread shape for the tiles and the loss");
    extern __shared__ __align__(16) unsigned char gemm_smem[];
    pdl_wait();
    if (blockIdx.x + 1 == gridDim.x) {
        __shared__ double sb[GT / 32];
        double t = 0.0;
        for (int i = threadIdx.x; i < W.nloss; i += GT) t += W.loss[i];
        for (int q = 16; q > 0; q >>= 1) t += __shfl_xor_sync(0xffffffffu, t, q);
        if ((threadIdx.x & 31) == 0) sb[threadIdx.x >> 5] = t;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int w = 0; w < GT / 32; ++w) s += sb[w];
            *W.loss_sum += s * W.inv_count;
        }
        return;
    }
    const int li = (int)blockIdx.x >= W.l[2].first ? 2 : (int)blockIdx.x >= W.l[1].first ? 1 : 0;
    const LayerGrad &l = W.l[li];
    const int t = blockIdx.x - l.first, m0 = t / l.tiles_n * 64, n0 = t % l.tiles_n * 64;
    float acc[T::RM][T::RN], col = 0.f;
    tile_sum<64, true, false>(l.g, m0, n0, gemm_smem, acc, m0 == 0 ? &col : nullptr);
    const AdamArgs &A = W.adam;
    auto update = [&](size_t at, float g, float p, float m, float v) {
        const float mi = A.b1 * m + (1.f - A.b1) * g;
        const float vi = A.b2 * v + (1.f - A.b2) * g * g;
        A.m[at] = mi;
        A.v[at] = vi;
        A.p[at] = p - A.lr * (mi / A.bc1) / (sqrtf(vi / A.bc2) + A.eps);
    };
    /* through shared memory, so that a warp updates neighbouring elements */
    float(*out)[64] = reinterpret_cast<float(*)[64]>(gemm_smem);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4 *>(&out[ty * 4 + i][tx * 4]) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    __syncthreads();
    const int n = n0 + (threadIdx.x & 63);
    if (n >= l.g.N) return;
    /* eight elements' moments loaded before any is used */
    constexpr int U = 8;
    for (int r0 = threadIdx.x >> 6; r0 < 64; r0 += 4 * U) {
        float p[U], m[U], v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t at = l.w + (size_t)(m0 + r0 + 4 * u) * l.g.N + n;
            if (!A.grad && m0 + r0 + 4 * u < l.g.M) {
                p[u] = A.p[at];
                m[u] = A.m[at];
                v[u] = A.v[at];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = r0 + 4 * u;
            if (m0 + r >= l.g.M) continue;
            const size_t at = l.w + (size_t)(m0 + r) * l.g.N + n;
            if (A.grad)
                A.grad[at] = out[r][n - n0];
            else
                update(at, out[r][n - n0], p[u], m[u], v[u]);
        }
    }
    if (m0 == 0 && threadIdx.x < 64) {
        const size_t at = l.b + n;
        if (A.grad)
            A.grad[at] = col;
        else
            update(at, col, A.p[at], A.m[at], A.v[at]);
    }
}

/* ---- BF16 inference on the tensor cores ------------------------------ */

/* C = A B with A [M][K] and B [K][N] in BF16 (row-major, leading dimensions
 * lda, ldb) and FP32 accumulation in mma.sync m16n8k16 tensor-core
 * instructions.  Block tile 64 x 64 x 32 (four warps of 32 x 32), operands
 * staged in shared memory by cp.async in two buffers and fed to the tensor
 * cores by ldmatrix (B transposed on the fly, so both operands stay in their
 * row-major storage).  Split-K: block z sums k in [z*kchunk, (z+1)*kchunk)
 * into slice z of `part` ([gridDim.z][M][N]); k_tc_finish adds the slices in
 * order, so the result does not depend on the split's timing. */
constexpr int TCM = 64, TCN = 64, TCK = 32, TCT = 128;

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_addr(p)));
}
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
struct TcSmem {
    __nv_bfloat16 a[2][TCM][TCK + 8]; /* rows of 80 bytes: ldmatrix rows fall in distinct banks */
    __nv_bfloat16 b[2][TCK][TCN + 8]; /* rows of 144 bytes */
};

/* Stages the 64 x 32 tile of A at (m0, k) and the 32 x 64 tile of B at
 * (k, n0); 16-byte copies where a whole aligned chunk is inside the matrix,
 * element by element (zero outside) elsewhere. */
__device__ __forceinline__ void tc_stage(TcSmem &sm, int buf, int M, int N, int kend, int m0, int n0, int k,
                                         const __nv_bfloat16 *__restrict__ A, long long lda,
                                         const __nv_bfloat16 *__restrict__ B, long long ldb, bool avec, bool bvec) {
    const __nv_bfloat16 zero = __float2bfloat16(0.f);
    for (int idx = threadIdx.x; idx < TCM * TCK / 8; idx += TCT) {
        const int r = idx / (TCK / 8), c = (idx % (TCK / 8)) * 8;
        const int gm = m0 + r, gk = k + c;
        __nv_bfloat16 *dst = &sm.a[buf][r][c];
        if (avec && gm < M && gk + 8 <= kend) {
            cp_async16(dst, A + (size_t)gm * lda + gk);
        } else {
            for (int q = 0; q < 8; ++q) dst[q] = (gm < M && gk + q < kend) ? A[(size_t)gm * lda + gk + q] : zero;
        }
    }
    for (int idx = threadIdx.x; idx < TCK * TCN / 8; idx += TCT) {
        const int r = idx / (TCN / 8), c = (idx % (TCN / 8)) * 8;
        const int gk = k + r, gn = n0 + c;
        __nv_bfloat16 *dst = &sm.b[buf][r][c];
        if (bvec && gk < kend && gn + 8 <= N) {
            cp_async16(dst, B + (size_t)gk * ldb + gn);
        } else {
            for (int q = 0; q < 8; ++q) dst[q] = (gk < kend && gn + q < N) ? B[(size_t)gk * ldb + gn + q] : zero;
        }
    }
}

__global__ void __launch_bounds__(TCT) k_gemm_bf16_tc(int M, int N, int K, int kchunk,
                                                      const __nv_bfloat16 *__restrict__ A, long long lda,
                                                      const __nv_bfloat16 *__restrict__ B, long long ldb,
                                                      float *part) {
    __shared__ __align__(128) TcSmem sm;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int m0 = blockIdx.y * TCM, n0 = blockIdx.x * TCN;
    const int kbeg = blockIdx.z * kchunk, kend = min(K, kbeg + kchunk);
    /* 16-byte copies need 16-byte aligned rows */
    const bool avec = (lda % 8) == 0 && ((uintptr_t)A % 16) == 0;
    const bool bvec = (ldb % 8) == 0 && ((uintptr_t)B % 16) == 0;
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
    const int ntiles = kend > kbeg ? (kend - kbeg + TCK - 1) / TCK : 0;
    if (ntiles > 0) tc_stage(sm, 0, M, N, kend, m0, n0, kbeg, A, lda, B, ldb, avec, bvec);
    cp_async_commit();
    for (int t = 0; t < ntiles; ++t) {
        const int buf = t & 1;
        if (t + 1 < ntiles) tc_stage(sm, buf ^ 1, M, N, kend, m0, n0, kbeg + (t + 1) * TCK, A, lda, B, ldb, avec, bvec);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
#pragma unroll
        for (int ks = 0; ks < TCK; ks += 16) {
            uint32_t af[2][4], bfr[2][4];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi) ldsm_x4(af[mi], &sm.a[buf][wm + mi * 16 + (lane & 15)][ks + (lane >> 4) * 8]);
#pragma unroll
            for (int nj = 0; nj < 2; ++nj)
                ldsm_x4_trans(bfr[nj], &sm.b[buf][ks + (lane & 15)][wn + nj * 16 + (lane >> 4) * 8]);
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int nt = 0; nt < 4; ++nt)
                    mma_bf16_16816(acc[mi][nt], af[mi], bfr[nt >> 1][(nt & 1) * 2], bfr[nt >> 1][(nt & 1) * 2 + 1]);
        }
        __syncthreads();
    }
    cp_async_wait<0>();
    float *out = part + (size_t)blockIdx.z * M * N;
    const int g = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = m0 + wm + mi * 16 + g + (q >> 1) * 8, c = n0 + wn + nt * 8 + tq * 2 + (q & 1);
                if (r < M && c < N) out[(size_t)r * N + c] = acc[mi][nt][q];
            }
}

/* C[m][n] = sum over slices z (in order) of part[z][m][n], + bias[n], ReLU;
 * written in FP32 to C and, when Cb is given, in BF16 to Cb (the next
 * layer's input) */
__global__ void k_tc_finish(const float *__restrict__ part, int Z, int M, int N, const float *__restrict__ bias,
                            int relu, float *C, __nv_bfloat16 *Cb) {
    const size_t total = (size_t)M * N;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        float v = 0.f;
        for (int z = 0; z < Z; ++z) v += part[(size_t)z * total + t];
        if (bias) v += bias[t % N];
        if (relu) v = fmaxf(v, 0.f);
        if (C) C[t] = v;
        if (Cb) Cb[t] = __float2bfloat16(v);
    }
}

__global__ void k_to_bf16(const float *__restrict__ src, __nv_bfloat16 *dst, size_t count) {
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += (size_t)gridDim.x * blockDim.x)
        dst[t] = __float2bfloat16(src[t]);
}

/* ---- the transportation family on the device --------------------------- */

/* standardised network input of B instances (FP64 arithmetic, rounded once
 * to FP32) */
__global__ void k_tr_features(int B, int S, int D, const double *__restrict__ c, const double *__restrict__ cap,
                              const double *__restrict__ b, const double *__restrict__ xm,
                              const double *__restrict__ xs, float *X) {
    const long long n = (long long)S * D, m = S + D, in = 2 * n + m;
    const long long total = (long long)B * in;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long r = t / in, f = t % in;
        double v;
        if (f < n)
            v = c[r * n + f] / 100.0;
        else if (f < 2 * n)
            v = cap[r * n + f - n] / 200.0;
        else
            v = b[r * m + f - 2 * n] / 100.0;
        X[t] = (float)(__dsub_rn(v, xm[f]) / xs[f]);
    }
}

/* t = T * ys + ym (two roundings, no fused multiply-add), then the warm
 * start it encodes */
__global__ void k_tr_decode(int B, int S, int D, const float *__restrict__ T, const double *__restrict__ ym,
                            const double *__restrict__ ys, const double *__restrict__ cap, double *x, double *y,
                            double *sigma) {
    const long long n = (long long)S * D, m = S + D, out = n + m + 1;
    const long long total = (long long)B * out;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long r = t / out, f = t % out;
        const double v = __dadd_rn(__dmul_rn((double)T[t], ys[f]), ym[f]);
        if (f < n)
            x[r * n + f] = fmin(fmax(v, 0.0), 1.0) * cap[r * n + f];
        else if (f < n + m)
            y[r * m + f - n] = v * 100.0;
        else
            sigma[r] = exp(v);
    }
}

__device__ __forceinline__ double tr_block_sum(double v, double *sb) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) sb[w] = v;
    __syncthreads();
    double t = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += sb[i];
    return t;
}

/* relative KKT error of (x, y) per instance, one block each (cold: x = y = 0) */
__global__ void __launch_bounds__(GT) k_tr_kkt(int S, int D, const double *__restrict__ x,
                                               const double *__restrict__ y, const double *__restrict__ c,
                                               const double *__restrict__ cap, const double *__restrict__ b,
                                               int cold, double *kkt) {
    __shared__ double sb[GT / 32];
    const long long n = (long long)S * D, m = S + D, r = blockIdx.x;
    const double *xr = x ? x + r * n : nullptr, *yr = y ? y + r * m : nullptr;
    const double *cr = c + r * n, *ur = cap + r * n, *br = b + r * m;
    double pobj = 0.0, dterm = 0.0, res2 = 0.0, b2 = 0.0, by = 0.0;
    for (long long a = threadIdx.x; a < n; a += blockDim.x) {
        const double xa = cold ? 0.0 : fmin(fmax(xr[a], 0.0), ur[a]);
        const int i = (int)(a / D), j = (int)(a % D);
        const double rc = cold ? cr[a] : cr[a] - yr[i] - yr[S + j];
        pobj += cr[a] * xa;
        dterm += fmin(rc, 0.0) * ur[a];
    }
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        double s = 0.0;
        if (!cold) {
            if (i < S)
                for (int j = 0; j < D; ++j) s += fmin(fmax(xr[(long long)i * D + j], 0.0), ur[(long long)i * D + j]);
            else
                for (int q = 0; q < S; ++q) {
                    const long long a = (long long)q * D + (i - S);
                    s += fmin(fmax(xr[a], 0.0), ur[a]);
                }
        }
        const double ri = s - br[i];
        res2 += ri * ri;
        b2 += br[i] * br[i];
        by += cold ? 0.0 : br[i] * yr[i];
    }
    pobj = tr_block_sum(pobj, sb);
    dterm = tr_block_sum(dterm, sb);
    res2 = tr_block_sum(res2, sb);
    b2 = tr_block_sum(b2, sb);
    by = tr_block_sum(by, sb);
    if (threadIdx.x == 0) {
        const double dobj = by + dterm;
        const double rel_p = sqrt(res2) / (1.0 + sqrt(b2));
        const double gap = fabs(pobj - dobj) / (1.0 + fabs(pobj) + fabs(dobj));
        kkt[r] = fmax(rel_p, gap);
    }
}

int grid1(size_t count) { return (int)std::min<size_t>((count + GT - 1) / GT, 152 * 16); }

/* a launch that is prepared while the kernel before it finishes (every kernel
 * of the network's products begins with griddepcontrol.wait) */
template <typename... K, typename... A>
void launch(void (*kern)(K...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
    if (smem > 48 * 1024)
        PDAL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    PDAL_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
}

/* returns the number of blocks (the losses of Finish::mse) */
template <int BT, bool TB, Finish F>
int gemm_tiles(cudaStream_t s, const GemmOp &g, const GemmOut &o) {
    using T = Tile<BT, false>;
    const dim3 grid((g.N + BT - 1) / BT, (g.M + BT - 1) / BT);
    launch(k_gemm<BT, TB, F>, grid, T::NT, T::BYTES, s, g, o);
    return (int)(grid.x * grid.y);
}
template <bool TB, Finish F>
int gemm(cudaStream_t s, int sms, const GemmOp &g, const GemmOut &o) {
    if (g.M <= 0 || g.N <= 0) return 0;
    auto tiles = [&](long long bt) { return ((g.N + bt - 1) / bt) * ((g.M + bt - 1) / bt); };
    if (tiles(64) >= sms) return gemm_tiles<64, TB, F>(s, g, o);
    if (tiles(32) >= sms) return gemm_tiles<32, TB, F>(s, g, o);
    return gemm_tiles<16, TB, F>(s, g, o);
}

template <typename T>
struct DevBuf;

/* the tensor-core product of one BF16 layer: split-K when the output tiles
 * alone would not fill two waves of the GPU's SMs */
void gemm_tc(cudaStream_t s, int M, int N, int K, const __nv_bfloat16 *A, long long lda, const __nv_bfloat16 *B,
             long long ldb, float *C, __nv_bfloat16 *Cb, const float *bias, bool relu, DevBuf<float> &part);

template <typename T>
struct DevBuf {
    T *p = nullptr;
    size_t n = 0;
    void ensure(size_t count) {
        if (count <= n) return;
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
        PDAL_CUDA(cudaMalloc(&p, sizeof(T) * std::max<size_t>(count, 1)));
        n = count;
    }
    ~DevBuf() {
        if (p) cudaFree(p);
    }
};

void gemm_tc(cudaStream_t s, int M, int N, int K, const __nv_bfloat16 *A, long long lda, const __nv_bfloat16 *B,
             long long ldb, float *C, __nv_bfloat16 *Cb, const float *bias, bool relu, DevBuf<float> &part) {
    if (M <= 0 || N <= 0) return;
    int dev = 0, sms = 0;
    PDAL_CUDA(cudaGetDevice(&dev));
    PDAL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const long long tiles = (long long)((N + TCN - 1) / TCN) * ((M + TCM - 1) / TCM);
    int Z = 1;
    if (tiles < 2LL * sms) Z = (int)std::min<long long>((2LL * sms + tiles - 1) / tiles, std::max(1, K / 512));
    int kchunk = (K + Z - 1) / Z;
    kchunk = (kchunk + TCK - 1) / TCK * TCK;
    Z = std::max(1, (K + kchunk - 1) / kchunk);
    part.ensure((size_t)Z * M * N);
    dim3 grid((N + TCN - 1) / TCN, (M + TCM - 1) / TCM, Z);
    k_gemm_bf16_tc<<<grid, TCT, 0, s>>>(M, N, K, kchunk, A, lda, B, ldb, part.p);
    k_tc_finish<<<grid1((size_t)M * N), GT, 0, s>>>(part.p, Z, M, N, bias, relu ? 1 : 0, C, Cb);
}

} // namespace

struct Mlp {
    int in, h, out, device;
    size_t oW1, ob1, oW2, ob2, oW3, ob3, np;
    cudaStream_t s = nullptr;
    DevBuf<float> P, G, Ma, Va;
    DevBuf<float> Xb, Yb, H1, H2, Yp, dY, dH1, dH2;
    DevBuf<int> idx;
    DevBuf<double> part; /* loss sums of the blocks, then the epoch's loss */
    int sms = 0;
    DevBuf<float> Xd, Yd;
    DevBuf<__nv_bfloat16> Pb, Xbb, H1b, H2b;
    DevBuf<double> warm[9]; /* instances, results and statistics of a warm-start call */
    DevBuf<float> Tp; /* split-K slices of the tensor-core products */
    int ndata = 0;
    long long adam_t = 0;

    Mlp(int in_, int h_, int out_, unsigned seed, int dev) : in(in_), h(h_), out(out_), device(dev) {
        if (device >= 0) PDAL_CUDA(cudaSetDevice(device));
        int current = 0;
        PDAL_CUDA(cudaGetDevice(&current));
        PDAL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, current));
        oW1 = 0;
        ob1 = oW1 + (size_t)in * h;
        oW2 = ob1 + h;
        ob2 = oW2 + (size_t)h * h;
        oW3 = ob2 + h;
        ob3 = oW3 + (size_t)h * out;
        np = ob3 + out;
        PDAL_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        P.ensure(np);
        G.ensure(np);
        Ma.ensure(np);
        Va.ensure(np);
        std::vector<float> init(np, 0.f);
        std::mt19937 gen(seed);
        auto fill = [&](size_t off, size_t count, int fan_in) {
            const float a = std::sqrt(6.0f / (float)fan_in);
            std::uniform_real_distribution<float> U(-a, a);
            for (size_t i = 0; i < count; ++i) init[off + i] = U(gen);
        };
        fill(oW1, (size_t)in * h, in);
        fill(oW2, (size_t)h * h, h);
        fill(oW3, (size_t)h * out, h);
        set_params(init.data());
    }
    /* Copies run on the handle's stream, which no other stream orders: what the
     * legacy stream holds of other work neither delays them past the products
     * that read them nor waits for these. */
    void put(float *dst, const float *src, size_t count) {
        PDAL_CUDA(cudaMemcpyAsync(dst, src, count * 4, cudaMemcpyHostToDevice, s));
    }
    void get(float *dst, const float *src, size_t count) {
        PDAL_CUDA(cudaMemcpyAsync(dst, src, count * 4, cudaMemcpyDeviceToHost, s));
        PDAL_CUDA(cudaStreamSynchronize(s));
    }
    /* new parameters, the moments of their updates zero */
    void set_params(const float *params) {
        put(P.p, params, np);
        PDAL_CUDA(cudaStreamSynchronize(s));
        PDAL_CUDA(cudaMemsetAsync(Ma.p, 0, np * 4, s));
        PDAL_CUDA(cudaMemsetAsync(Va.p, 0, np * 4, s));
        adam_t = 0;
    }
    ~Mlp() {
        if (s) cudaStreamDestroy(s);
    }

    /* activations of B rows; with `train` also the gradients */
    void buffers(int B, bool train) {
        H1.ensure((size_t)B * h);
        H2.ensure((size_t)B * h);
        if (!train) {
            Yp.ensure((size_t)B * out);
            return;
        }
        dY.ensure((size_t)B * out);
        dH1.ensure((size_t)B * h);
        dH2.ensure((size_t)B * h);
        part.ensure((size_t)((out + 15) / 16) * ((B + 15) / 16) + 1);
    }
    double *loss_sum() const { return part.p + part.n - 1; }

    /* inference of B rows of X (device, FP32) into Yp: FP32 SIMT, or BF16
     * operands on the tensor cores (the weights' BF16 copy made by
     * prepare_bf16) */
    void prepare_bf16(int chunk) {
        Pb.ensure(np);
        Xbb.ensure((size_t)chunk * in);
        H1b.ensure((size_t)chunk * h);
        H2b.ensure((size_t)chunk * h);
        k_to_bf16<<<grid1(np), GT, 0, s>>>(P.p, Pb.p, np);
    }
    void infer(int B, const float *X, bool bf16) {
        if (!bf16) {
            forward(B, X);
            return;
        }
        const __nv_bfloat16 *W1 = Pb.p + oW1, *W2 = Pb.p + oW2, *W3 = Pb.p + oW3;
        const float *b1 = P.p + ob1, *b2 = P.p + ob2, *b3 = P.p + ob3;
        k_to_bf16<<<grid1((size_t)B * in), GT, 0, s>>>(X, Xbb.p, (size_t)B * in);
        /* each layer's BF16 output is the next layer's tensor-core operand */
        gemm_tc(s, B, h, in, Xbb.p, in, W1, h, nullptr, H1b.p, b1, true, Tp);
        gemm_tc(s, B, h, h, H1b.p, h, W2, h, nullptr, H2b.p, b2, true, Tp);
        gemm_tc(s, B, out, h, H2b.p, h, W3, out, Yp.p, nullptr, b3, false, Tp);
    }

    /* the two hidden layers of B rows of X (device; row i is rows[i]) */
    void hidden(int B, const float *X, const int *rows) {
        GemmOut o{};
        o.C = H1.p;
        o.bias = P.p + ob1;
        gemm<false, Finish::bias_relu>(s, sms, GemmOp{B, h, in, X, P.p + oW1, in, h, rows}, o);
        o.C = H2.p;
        o.bias = P.p + ob2;
        gemm<false, Finish::bias_relu>(s, sms, GemmOp{B, h, h, H1.p, P.p + oW2, h, h, nullptr}, o);
    }
    /* forward of B rows of X (device) into Yp */
    void forward(int B, const float *X) {
        hidden(B, X, nullptr);
        GemmOut o{};
        o.C = Yp.p;
        o.bias = P.p + ob3;
        gemm<false, Finish::bias>(s, sms, GemmOp{B, out, h, H2.p, P.p + oW3, h, out, nullptr}, o);
    }

    /* One batch: rows[0..B) (or the first B) of X and Y, their mean squared
     * error added to loss_sum(), the gradient into A.grad or the Adam update.
     * Without `back` the loss alone. */
    void step(int B, const float *X, const float *Y, const int *rows, const AdamArgs &A, bool back) {
        const size_t cnt = (size_t)B * out;
        hidden(B, X, rows);
        GemmOut o{};
        o.C = back ? dY.p : nullptr;
        o.bias = P.p + ob3;
        o.Y = Y;
        o.rows = rows;
        o.scale = 2.0f / (float)cnt;
        o.loss = part.p;
        WeightArgs W{};
        W.nloss = gemm<false, Finish::mse>(s, sms, GemmOp{B, out, h, H2.p, P.p + oW3, h, out, nullptr}, o);
        W.loss = part.p;
        W.inv_count = 1.0 / (double)cnt;
        W.loss_sum = loss_sum();
        W.adam = A;
        int blocks = 0;
        if (back) {
            GemmOut d{};
            d.C = dH2.p;
            d.H = H2.p;
            gemm<true, Finish::mask>(s, sms, GemmOp{B, h, out, dY.p, P.p + oW3, out, out, nullptr}, d);
            d.C = dH1.p;
            d.H = H1.p;
            gemm<true, Finish::mask>(s, sms, GemmOp{B, h, h, dH2.p, P.p + oW2, h, h, nullptr}, d);
            /* the largest first */
            const GemmOp g[3] = {{in, h, B, X, dH1.p, in, h, rows},
                                 {h, out, B, H2.p, dY.p, h, out, nullptr},
                                 {h, h, B, H1.p, dH2.p, h, h, nullptr}};
            const size_t ow[3] = {oW1, oW3, oW2}, ob[3] = {ob1, ob3, ob2};
            for (int q = 0; q < 3; ++q) {
                const int tn = (g[q].N + 63) / 64, tm = (g[q].M + 63) / 64;
                W.l[q] = LayerGrad{g[q], ow[q], ob[q], tn, blocks};
                blocks += tn * tm;
            }
        }
        launch(k_weights, dim3(blocks + 1), GT, Tile<64, true>::BYTES, s, W);
    }
    double read_loss() {
        double t = 0.0;
        PDAL_CUDA(cudaMemcpyAsync(&t, loss_sum(), sizeof(double), cudaMemcpyDeviceToHost, s));
        PDAL_CUDA(cudaStreamSynchronize(s));
        PDAL_CUDA(cudaGetLastError());
        return t;
    }
    void clear_loss() { PDAL_CUDA(cudaMemsetAsync(loss_sum(), 0, sizeof(double), s)); }
};

} // namespace pdal

struct pdal_mlp {
    pdal::Mlp *m;
};

namespace {
int fail(const std::string &msg) {
    pdal::g_mlp_error = msg;
    fprintf(stderr, "[pdal_learn] %s\n", msg.c_str());
    return -1;
}
} // namespace

extern "C" {

pdal_mlp_t *pdal_mlp_create(int in, int hidden, int out, unsigned seed, int device) {
    if (in <= 0 || hidden <= 0 || out <= 0) {
        fail("pdal_mlp_create: dimensions must be positive");
        return nullptr;
    }
    try {
        pdal_mlp_t *h = new pdal_mlp_t;
        h->m = new pdal::Mlp(in, hidden, out, seed, device);
        return h;
    } catch (const std::exception &e) {
        fail(e.what());
        return nullptr;
    }
}

void pdal_mlp_free(pdal_mlp_t *h) {
    if (!h) return;
    delete h->m;
    delete h;
}

long long pdal_mlp_num_params(const pdal_mlp_t *h) { return h ? (long long)h->m->np : -1; }

int pdal_mlp_get_params(const pdal_mlp_t *h, float *params) {
    if (!h || !params) return fail("pdal_mlp_get_params: NULL argument");
    try {
        h->m->get(params, h->m->P.p, h->m->np);
        return 0;
    } catch (const std::exception &e) {
        return fail(e.what());
    }
}

int pdal_mlp_set_params(pdal_mlp_t *h, const float *params) {
    if (!h || !params) return fail("pdal_mlp_set_params: NULL argument");
    try {
        h->m->set_params(params);
        return 0;
    } catch (const std::exception &e) {
        return fail(e.what());
    }
}

int pdal_mlp_set_data(pdal_mlp_t *h, int n, const float *X, const float *Y) {
    if (!h || n <= 0 || !X || !Y) return fail("pdal_mlp_set_data: invalid arguments");
    try {
        pdal::Mlp &m = *h->m;
        m.Xd.ensure((size_t)n * m.in);
        m.Yd.ensure((size_t)n * m.out);
        m.put(m.Xd.p, X, (size_t)n * m.in);
        m.put(m.Yd.p, Y, (size_t)n * m.out);
        PDAL_CUDA(cudaStreamSynchronize(m.s));
        m.ndata = n;
        return 0;
    } catch (const std::exception &e) {
        return fail(e.what());
    }
}

double pdal_mlp_train(pdal_mlp_t *h, int epochs, int batch, float lr, unsigned seed) {
    if (!h || epochs <= 0 || batch <= 0 || h->m->ndata <= 0) return fail("pdal_mlp_train: invalid arguments");
    try {
        pdal::Mlp &m = *h->m;
        const int n = m.ndata;
        const int B = std::min(batch, n);
        m.buffers(B, true);
        m.idx.ensure(n);
        std::vector<int> perm(n);
        std::iota(perm.begin(), perm.end(), 0);
        std::mt19937 gen(seed);
        double last = 0.0;
        pdal::AdamArgs A{m.P.p, m.Ma.p, m.Va.p, nullptr, lr, 0.9f, 0.999f, 1e-8f, 0.f, 0.f};
        for (int ep = 0; ep < epochs; ++ep) {
            std::shuffle(perm.begin(), perm.end(), gen);
            PDAL_CUDA(cudaMemcpyAsync(m.idx.p, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, m.s));
            m.clear_loss();
            int batches = 0;
            for (int b0 = 0; b0 + B <= n; b0 += B) {
                ++batches;
                ++m.adam_t;
                A.bc1 = 1.f - std::pow(A.b1, (float)m.adam_t);
                A.bc2 = 1.f - std::pow(A.b2, (float)m.adam_t);
                m.step(B, m.Xd.p, m.Yd.p, m.idx.p + b0, A, true);
            }
            if (ep + 1 == epochs) last = batches ? m.read_loss() / batches : 0.0;
        }
        return last;
    } catch (const std::exception &e) {
        return fail(e.what());
    }
}

double pdal_mlp_loss_grad(pdal_mlp_t *h, int n, const float *X, const float *Y, float *grad) {
    if (!h || n <= 0 || !X || !Y) return fail("pdal_mlp_loss_grad: invalid arguments");
    try {
        pdal::Mlp &m = *h->m;
        m.buffers(n, true);
        m.Xb.ensure((size_t)n * m.in);
        m.Yb.ensure((size_t)n * m.out);
        PDAL_CUDA(cudaMemcpyAsync(m.Xb.p, X, (size_t)n * m.in * 4, cudaMemcpyHostToDevice, m.s));
        PDAL_CUDA(cudaMemcpyAsync(m.Yb.p, Y, (size_t)n * m.out * 4, cudaMemcpyHostToDevice, m.s));
        m.clear_loss();
        pdal::AdamArgs A{};
        A.grad = m.G.p;
        m.step(n, m.Xb.p, m.Yb.p, nullptr, A, grad != nullptr);
        const double loss = m.read_loss();
        if (grad) m.get(grad, m.G.p, m.np);
        return loss;
    } catch (const std::exception &e) {
        return fail(e.what());
    }
}

int pdal_mlp_predict(pdal_mlp_t *h, int n, const float *X, float *Y, int bf16) {
    if (!h || n <= 0 || !X || !Y) return fail("pdal_mlp_predict: invalid arguments");
    try {
        pdal::Mlp &m = *h->m;
        const int chunk = std::min(n, 1024);
        m.buffers(chunk, false);
        m.Xb.ensure((size_t)chunk * m.in);
        if (bf16) m.prepare_bf16(chunk);
        for (int r0 = 0; r0 < n; r0 += chunk) {
            const int B = std::min(chunk, n - r0);
            PDAL_CUDA(cudaMemcpyAsync(m.Xb.p, X + (size_t)r0 * m.in, (size_t)B * m.in * 4, cudaMemcpyHostToDevice,
                                      m.s));
            m.infer(B, m.Xb.p, bf16 != 0);
            PDAL_CUDA(cudaMemcpyAsync(Y + (size_t)r0 * m.out, m.Yp.p, (size_t)B * m.out * 4, cudaMemcpyDeviceToHost,
                                      m.s));
        }
        PDAL_CUDA(cudaStreamSynchronize(m.s));
        PDAL_CUDA(cudaGetLastError());
        return 0;
    } catch (const std::exception &e) {
        return fail(e.what());
    }
}

int pdal_transport_warm_start(pdal_mlp_t *h, int S, int D, int count, const double *costs, const double *caps,
                              const double *rhs, const double *xm, const double *xs, const double *ym,
                              const double *ys, int bf16, double *x, double *y, double *sigma, double *kkt_pred,
                              double *kkt_cold) {
    if (!h || S <= 0 || D <= 0 || count <= 0 || !costs || !caps || !rhs || !xm || !xs || !ym || !ys || !x || !y ||
        !sigma || !kkt_pred || !kkt_cold)
        return fail("pdal_transport_warm_start: invalid arguments");
    try {
        pdal::Mlp &m = *h->m;
        const long long n = (long long)S * D, mm = S + D;
        if (m.in != 2 * n + mm || m.out != n + mm + 1)
            return fail("pdal_transport_warm_start: the network's sizes do not match the S x D family");
        const int chunk = std::min(count, 1024);
        m.buffers(chunk, false);
        m.Xb.ensure((size_t)chunk * m.in);
        if (bf16) m.prepare_bf16(chunk);
        auto &[dc, du, db, dx, dy, ds, dk0, dk1, st] = m.warm;
        dc.ensure((size_t)chunk * n);
        du.ensure((size_t)chunk * n);
        db.ensure((size_t)chunk * mm);
        dx.ensure((size_t)chunk * n);
        dy.ensure((size_t)chunk * mm);
        ds.ensure(chunk);
        dk0.ensure(chunk);
        dk1.ensure(chunk);
        st.ensure((size_t)2 * m.in + 2 * m.out);
        double *dxm = st.p, *dxs = st.p + m.in, *dym = st.p + 2 * m.in, *dys = st.p + 2 * m.in + m.out;
        PDAL_CUDA(cudaMemcpyAsync(dxm, xm, sizeof(double) * m.in, cudaMemcpyHostToDevice, m.s));
        PDAL_CUDA(cudaMemcpyAsync(dxs, xs, sizeof(double) * m.in, cudaMemcpyHostToDevice, m.s));
        PDAL_CUDA(cudaMemcpyAsync(dym, ym, sizeof(double) * m.out, cudaMemcpyHostToDevice, m.s));
        PDAL_CUDA(cudaMemcpyAsync(dys, ys, sizeof(double) * m.out, cudaMemcpyHostToDevice, m.s));
        for (int r0 = 0; r0 < count; r0 += chunk) {
            const int B = std::min(chunk, count - r0);
            PDAL_CUDA(cudaMemcpyAsync(dc.p, costs + (size_t)r0 * n, sizeof(double) * B * n, cudaMemcpyHostToDevice,
                                      m.s));
            PDAL_CUDA(cudaMemcpyAsync(du.p, caps + (size_t)r0 * n, sizeof(double) * B * n, cudaMemcpyHostToDevice,
                                      m.s));
            PDAL_CUDA(cudaMemcpyAsync(db.p, rhs + (size_t)r0 * mm, sizeof(double) * B * mm, cudaMemcpyHostToDevice,
                                      m.s));
            pdal::k_tr_features<<<pdal::grid1((size_t)B * m.in), pdal::GT, 0, m.s>>>(B, S, D, dc.p, du.p, db.p, dxm,
                                                                                    dxs, m.Xb.p);
            m.infer(B, m.Xb.p, bf16 != 0);
            pdal::k_tr_decode<<<pdal::grid1((size_t)B * m.out), pdal::GT, 0, m.s>>>(B, S, D, m.Yp.p, dym, dys, du.p,
                                                                                   dx.p, dy.p, ds.p);
            pdal::k_tr_kkt<<<B, pdal::GT, 0, m.s>>>(S, D, dx.p, dy.p, dc.p, du.p, db.p, 0, dk0.p);
            pdal::k_tr_kkt<<<B, pdal::GT, 0, m.s>>>(S, D, nullptr, nullptr, dc.p, du.p, db.p, 1, dk1.p);
            PDAL_CUDA(cudaGetLastError());
            PDAL_CUDA(cudaMemcpyAsync(x + (size_t)r0 * n, dx.p, sizeof(double) * B * n, cudaMemcpyDeviceToHost, m.s));
            PDAL_CUDA(cudaMemcpyAsync(y + (size_t)r0 * mm, dy.p, sizeof(double) * B * mm, cudaMemcpyDeviceToHost,
                                      m.s));
            PDAL_CUDA(cudaMemcpyAsync(sigma + r0, ds.p, sizeof(double) * B, cudaMemcpyDeviceToHost, m.s));
            PDAL_CUDA(cudaMemcpyAsync(kkt_pred + r0, dk0.p, sizeof(double) * B, cudaMemcpyDeviceToHost, m.s));
            PDAL_CUDA(cudaMemcpyAsync(kkt_cold + r0, dk1.p, sizeof(double) * B, cudaMemcpyDeviceToHost, m.s));
            /* the chunk's device buffers are reused by the next chunk */
            PDAL_CUDA(cudaStreamSynchronize(m.s));
        }
        return 0;
    } catch (const std::exception &e) {
        return fail(e.what());
    }
}

const char *pdal_mlp_last_error(void) { return pdal::g_mlp_error.c_str(); }

} // extern "C"
