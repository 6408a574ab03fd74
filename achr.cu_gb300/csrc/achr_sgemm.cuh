// FP32 matrix products and the inverse of an SPD matrix on sm_103a, for the
// direction preconditioner (achr_precond.cu).
//
// Products.  C (M x N) = A B with both operands given as rows of the
// contraction index: A[k * lda + m], B[k * ldb + n] (or, with ?K = true, with
// k contiguous: A[m * lda + k]).  Every element is one chain of FMAs over k in
// order, whatever the tile.  What bounds it is FP32 issue and the shared-memory
// reads that feed it (GB300 has no full-precision FP32 tensor path): T x T per
// thread as packed fma.rn.f32x2 pairs along N.  Measured with 128 x 128 tiles
// and 8 x 8 per thread: 57 TFLOP/s at 8192 x 8192 x 1024 (53 with scalar FMAs, 46
// with A held doubled in shared memory instead of paired in registers); the 64 x
// 64 tiles with 4 x 4 scalars per thread that this replaces ran at a third of
// that.  The next k-block travels through registers while this one is
// multiplied.  The tile shrinks until the GPU is filled (gemm_tile); where the
// caller allows it, a long contraction is split over grid.z instead, into
// partial results that a second kernel adds in order.
#pragma once
#include <cuda_runtime.h>

#include <stdint.h>

#include <algorithm>

namespace achr {
namespace {

constexpr int kGK = 16;
constexpr int kResTile = 128;  // rows of C per partial sum of GEMM_RESIDUE

// What becomes of the tile.
enum GemmOut {
    GEMM_PLAIN,    // C = alpha acc + beta D (+ 1 on the diagonal)
    GEMM_PART,     // part[z] = acc
    GEMM_RESIDUE,  // C = scale[n] X[n * ldx + m] - acc, Ct = C^T, and sums over the tile's m of C X and C C for each n
};

struct GemmArgs {
    int M, N, K, k_split;  // k_split: contraction length per grid.z
    const float *A, *B;
    long long lda, ldb;
    int va, vb;  // 1: 16-byte loads (aligned base, leading dimension a multiple of 4)
    float *C;
    long long ldc;
    float alpha, beta;
    const float *D;  // like C, or NULL
    int unit_diag;
    float *Ct;
    long long ldct;
    const float *X, *scale;
    long long ldx;
    float *sxv, *svv;  // (M tiles) x N
};

__device__ __forceinline__ void fma2(unsigned long long &c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long twice(float v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    return make_float2(__uint_as_float((unsigned)v), __uint_as_float((unsigned)(v >> 32)));
}

// Four consecutive values of a row (n valid ones from p), zeros beyond.
__device__ __forceinline__ float4 load4(const float *p, int n, bool vec) {
    if (n >= 4 && vec) return __ldg(reinterpret_cast<const float4 *>(p));
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (n > 0) v.x = __ldg(p);
    if (n > 1) v.y = __ldg(p + 1);
    if (n > 2) v.z = __ldg(p + 2);
    if (n > 3) v.w = __ldg(p + 3);
    return v;
}

// BT x BT of C per CTA, T x T per thread.
template <GemmOut OUT, bool AK, bool BK, int BT, int T>
__global__ void __launch_bounds__((BT / T) * (BT / T), BT == 128 ? 2 : BT == 64 ? 3 : 8) gemm_kernel(const GemmArgs g) {
    constexpr int kThreads = (BT / T) * (BT / T), WX = BT / T / 8, H = T / 4;
    __shared__ __align__(16) float As[2][kGK][BT], Bs[2][kGK][BT];
    // a warp covers 4 x 8 threads, so its A reads have four addresses and its B reads eight
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (warp % WX) * 8 + (lane & 7), ty = (warp / WX) * 4 + (lane >> 3);
    const int m0 = blockIdx.y * BT, n0 = blockIdx.x * BT;
    const int kb = blockIdx.z * g.k_split, ke = min(g.K, kb + g.k_split);
    constexpr int kLoads = kGK * BT / 4 / kThreads;  // float4 per thread of either operand's block
    float4 ra[kLoads], rb[kLoads];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            const int t = tid + u * kThreads;
            if (AK) {  // row m, four k
                const int m = m0 + t / (kGK / 4), k = k0 + 4 * (t % (kGK / 4));
                ra[u] = load4(g.A + (long long)m * g.lda + k, m < g.M ? ke - k : 0, g.va);
            } else {
                const int k = k0 + t / (BT / 4), m = m0 + 4 * (t % (BT / 4));
                ra[u] = load4(g.A + (long long)k * g.lda + m, k < ke ? g.M - m : 0, g.va);
            }
            if (BK) {
                const int n = n0 + t / (kGK / 4), k = k0 + 4 * (t % (kGK / 4));
                rb[u] = load4(g.B + (long long)n * g.ldb + k, n < g.N ? ke - k : 0, g.vb);
            } else {
                const int k = k0 + t / (BT / 4), n = n0 + 4 * (t % (BT / 4));
                rb[u] = load4(g.B + (long long)k * g.ldb + n, k < ke ? g.N - n : 0, g.vb);
            }
        }
    };
    auto store = [&](int s) {
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            const int t = tid + u * kThreads;
            if (AK) {
                const int m = t / (kGK / 4), k = 4 * (t % (kGK / 4));
                As[s][k][m] = ra[u].x;
                As[s][k + 1][m] = ra[u].y;
                As[s][k + 2][m] = ra[u].z;
                As[s][k + 3][m] = ra[u].w;
            } else {
                *reinterpret_cast<float4 *>(&As[s][t / (BT / 4)][4 * (t % (BT / 4))]) = ra[u];
            }
            if (BK) {
                const int n = t / (kGK / 4), k = 4 * (t % (kGK / 4));
                Bs[s][k][n] = rb[u].x;
                Bs[s][k + 1][n] = rb[u].y;
                Bs[s][k + 2][n] = rb[u].z;
                Bs[s][k + 3][n] = rb[u].w;
            } else {
                *reinterpret_cast<float4 *>(&Bs[s][t / (BT / 4)][4 * (t % (BT / 4))]) = rb[u];
            }
        }
    };
    // rows and columns BT/H h + 4 t + {0..3}, h < H (t = ty, tx), columns as pairs
    unsigned long long acc[T][T / 2];
#pragma unroll
    for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T / 2; ++j) acc[i][j] = 0ull;
    fetch(kb);
    store(0);
    __syncthreads();
    int s = 0;
    for (int k0 = kb; k0 < ke; k0 += kGK, s ^= 1) {
        const bool more = k0 + kGK < ke;
        if (more) fetch(k0 + kGK);
#pragma unroll
        for (int k = 0; k < kGK; ++k) {
            float av[T];
            unsigned long long bv[T / 2];
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const float4 x = *reinterpret_cast<const float4 *>(&As[s][k][BT / H * h + 4 * ty]);
                const ulonglong2 p = *reinterpret_cast<const ulonglong2 *>(&Bs[s][k][BT / H * h + 4 * tx]);
                av[4 * h] = x.x;
                av[4 * h + 1] = x.y;
                av[4 * h + 2] = x.z;
                av[4 * h + 3] = x.w;
                bv[2 * h] = p.x;
                bv[2 * h + 1] = p.y;
            }
#pragma unroll
            for (int i = 0; i < T; ++i) {
                const unsigned long long a2 = twice(av[i]);
#pragma unroll
                for (int j = 0; j < T / 2; ++j) fma2(acc[i][j], a2, bv[j]);
            }
        }
        if (more) store(s ^ 1);
        __syncthreads();
    }
    float sx[T], sv[T];  // sums over this thread's rows, per column
    if (OUT == GEMM_RESIDUE) {
#pragma unroll
        for (int j = 0; j < T; ++j) sx[j] = sv[j] = 0.0f;
    }
#pragma unroll
    for (int i = 0; i < T; ++i) {
        const int m = m0 + BT / H * (i >> 2) + 4 * ty + (i & 3);
        if (m >= g.M) continue;
#pragma unroll
        for (int j = 0; j < T; ++j) {
            const int n = n0 + BT / H * (j >> 2) + 4 * tx + (j & 3);
            if (n >= g.N) continue;
            const float2 p = unpack2(acc[i][j >> 1]);
            const float v = (j & 1) ? p.y : p.x;
            const long long o = (long long)m * g.ldc + n;
            if (OUT == GEMM_PLAIN) {
                float c = g.alpha * v;
                if (g.D) c = fmaf(g.beta, g.D[o], c);
                g.C[o] = c + (g.unit_diag && m == n ? 1.0f : 0.0f);
            }
            if (OUT == GEMM_PART) g.C[(long long)blockIdx.z * g.M * g.ldc + o] = v;
            if (OUT == GEMM_RESIDUE) {
                const float x = __ldg(g.X + (long long)n * g.ldx + m);
                const float r = fmaf(__ldg(g.scale + n), x, -v);
                g.C[o] = r;
                g.Ct[(long long)n * g.ldct + m] = r;
                sx[j] = fmaf(x, r, sx[j]);
                sv[j] = fmaf(r, r, sv[j]);
            }
        }
    }
    if constexpr (OUT == GEMM_RESIDUE) {  // the tile's rows: BT/T threads (ty) per column, summed in order
        static_assert(BT == kResTile && BT / T <= kGK, "the partial sums fit the operands' first buffers");
        float *bx = &As[0][0][0], *bv = &Bs[0][0][0];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < T; ++j) {
            const int n = BT / H * (j >> 2) + 4 * tx + (j & 3);
            bx[ty * BT + n] = sx[j];
            bv[ty * BT + n] = sv[j];
        }
        __syncthreads();
        if (tid < BT && n0 + tid < g.N) {
            float x = 0.0f, v = 0.0f;
#pragma unroll
            for (int t = 0; t < BT / T; ++t) {
                x += bx[t * BT + tid];
                v += bv[t * BT + tid];
            }
            g.sxv[(long long)blockIdx.y * g.N + n0 + tid] = x;
            g.svv[(long long)blockIdx.y * g.N + n0 + tid] = v;
        }
    }
}

// C = alpha sum_z part[z] + beta D (+ 1 on the diagonal), the partial results added in order.
__global__ void gemm_reduce_kernel(int M, int N, int splits, const float *__restrict__ part, float alpha, float beta,
                                   const float *__restrict__ D, int unit_diag, float *__restrict__ C) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, cnt = (long long)M * N;
    if (t >= cnt) return;
    float v = 0.0f;
    for (int z = 0; z < splits; ++z) v += part[z * cnt + t];
    v *= alpha;
    if (D) v = fmaf(beta, D[t], v);
    if (unit_diag && t / N == t % N) v += 1.0f;
    C[t] = v;
}

inline int gemm_vec(const void *p, long long ld) { return ((uintptr_t)p & 15u) == 0 && ld % 4 == 0 ? 1 : 0; }

// Largest tile (128, 64, 32) that gives most SMs a CTA.
inline int gemm_tile(int M, int N) {
    for (int t : {128, 64})
        if ((long long)((M + t - 1) / t) * ((N + t - 1) / t) >= 128) return t;
    return 32;
}

// Splits of a contraction over K with 128 x 128 tiles: as many CTAs as fit (two per SM), at least 64 of K each.
inline int gemm_splits(int M, int N, int K) {
    const long long tiles = (long long)((M + 127) / 128) * ((N + 127) / 128);
    const long long want = (2 * 152) / std::max(tiles, 1ll), most = std::max(1, K / 64);
    return (int)std::max(1ll, std::min(std::min(want, most), 64ll));
}

template <GemmOut OUT, bool AK = false, bool BK = false>
cudaError_t gemm_launch(cudaStream_t st, GemmArgs g, int tile, int splits = 1) {
    if (g.M <= 0 || g.N <= 0) return cudaSuccess;
    g.va = gemm_vec(g.A, g.lda);
    g.vb = gemm_vec(g.B, g.ldb);
    g.k_split = ((g.K + splits - 1) / splits + kGK - 1) / kGK * kGK;
    dim3 grid((unsigned)((g.N + tile - 1) / tile), (unsigned)((g.M + tile - 1) / tile), (unsigned)splits);
    if (tile == 128) {
        gemm_kernel<OUT, AK, BK, 128, 8><<<grid, 256, 0, st>>>(g);
    } else if constexpr (OUT == GEMM_PLAIN) {
        if (tile == 64) gemm_kernel<OUT, AK, BK, 64, 4><<<grid, 256, 0, st>>>(g);
        else gemm_kernel<OUT, AK, BK, 32, 4><<<grid, 64, 0, st>>>(g);
    }
    return cudaGetLastError();
}

// C = alpha A B + beta D (+ I), C dense (leading dimension N).  With `part` (gemm_splits(M, N, K) x M
// x N floats) a contraction that is worth splitting is split.
template <bool AK = false, bool BK = false>
cudaError_t gemm(cudaStream_t st, int M, int N, int K, const float *A, long long lda, const float *B, long long ldb,
                 float *part, float alpha, float beta, const float *D, int unit_diag, float *C) {
    const int splits = part ? gemm_splits(M, N, K) : 1;
    GemmArgs g{};
    g.M = M;
    g.N = N;
    g.K = K;
    g.A = A;
    g.lda = lda;
    g.B = B;
    g.ldb = ldb;
    g.ldc = N;
    g.alpha = alpha;
    g.beta = beta;
    g.D = D;
    g.unit_diag = unit_diag;
    g.C = splits > 1 ? part : C;
    if (splits == 1) return gemm_launch<GEMM_PLAIN, AK, BK>(st, g, gemm_tile(M, N));
    if (cudaError_t e = gemm_launch<GEMM_PART, AK, BK>(st, g, 128, splits)) return e;
    const long long cnt = (long long)M * N;
    gemm_reduce_kernel<<<(unsigned)((cnt + 255) / 256), 256, 0, st>>>(M, N, splits, part, alpha, beta, D, unit_diag, C);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Inverse and log determinant of a symmetric positive definite matrix M (r x r)
// through its Cholesky factor: M = L L^T, X = L^-1, Minv = X^T X, every element
// summed over k in order.  A column at a time in one CTA (a barrier per column,
// the matrix in L2) this took 4.9 ms at r = 256.  Here the factorisation works
// on panels of 32 columns in shared memory (in L2 above kCholSmemMax), X is
// formed by a CTA per 32 columns, and Minv is a product: 0.18 ms (114 + 49 + 13 us).
constexpr int kNB = 32;
constexpr int kCholSmemMax = 304;  // rows of the factor that fit shared memory (packed lower triangle, and a panel)
constexpr int kNextBlock = (kNB / 4) * (kNB / 4 + 1) / 2;  // 4 x 4 elements of a diagonal block's triangle
constexpr int kInverseMax = 1024;  // rows the inverse's shared-memory layouts allow

// Element (i, j), j <= i, of the factor while it is formed: packed rows in shared memory, or the r x r
// matrix in global memory.
struct LowerPacked {
    float *p;
    __device__ __forceinline__ float &at(int i, int j) const { return p[(i * (i + 1)) / 2 + j]; }
};
struct LowerDense {
    float *p;
    int r;
    __device__ __forceinline__ float &at(int i, int j) const { return p[(long long)i * r + j]; }
};

// The panel's rows below its diagonal block once more, transposed (column k at panel + k * ld): the
// trailing update then reads four rows with one 16-byte load.  Row by row from the packed triangle
// it read single words with bank conflicts.  r = 256: 159 us before; 144 with this; 138 with the divisions
// below as three operations; 114 with the diagonal block's shuffles free of branches.
__host__ __device__ inline int chol_panel_ld(int r) { return r <= kNB ? 4 : (r - kNB + 3) / 4 * 4; }
inline size_t chol_panel_bytes(int r) { return sizeof(float) * (size_t)kNB * chol_panel_ld(r); }

// v / d from inv = 1 / d, both rounded to nearest: the quotient's remainder is exact, and one
// correction rounds it correctly (Markstein, IBM J. Res. Dev. 34, 1990) for a normal quotient.  The
// divisions below follow one another; this one is three dependent operations and no branch.
__device__ __forceinline__ float div_by(float v, float d, float inv) {
    const float q = v * inv;
    return fmaf(fmaf(-q, d, v), inv, q);
}

// diag: the diagonal block, transposed; dinv: 1 / its diagonal.
template <class Low>
__device__ __forceinline__ void chol_panels(int r, const Low L, int *bad, float (*diag)[kNB + 4], float *dinv,
                                            float *panel) {
    const int ldp = chol_panel_ld(r);
    const int tid = threadIdx.x, nt = blockDim.x;
    __syncthreads();
    for (int c0 = 0; c0 < r; c0 += kNB) {
        // Triangle from row c0 on, less the previous panel's part: 4 x 4 elements per thread and turn.
        // Warp 0 takes the diagonal block (the first 36 of them) and factors it, a chain of 32 square
        // roots and divisions, while the others update the rest.
        const int nb = min(kNB, r - c0);
        const int nq = c0 ? (r - c0 + 3) / 4 : 0, all = nq * (nq + 1) / 2, first = min(kNextBlock, all);
        for (int t = tid < 32 ? tid : first + tid - 32; t < (tid < 32 ? first : all); t += tid < 32 ? 32 : nt - 32) {
            int bi = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
            while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
            while (bi * (bi + 1) / 2 > t) --bi;
            const int i0 = c0 + 4 * bi, j0 = c0 + 4 * (t - bi * (bi + 1) / 2);
            float acc[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = i0 + i < r && j0 + j <= i0 + i ? L.at(i0 + i, j0 + j) : 0.0f;
            const float *pi = panel + i0 - c0, *pj = panel + j0 - c0;
#pragma unroll 8
            for (int k = 0; k < kNB; ++k) {
                const float4 a4 = *reinterpret_cast<const float4 *>(pi + k * ldp);
                const float4 b4 = *reinterpret_cast<const float4 *>(pj + k * ldp);
                const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(-a[i], b[j], acc[i][j]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (i0 + i < r && j0 + j <= i0 + i) L.at(i0 + i, j0 + j) = acc[i][j];
        }
        if (tid < 32) {  // lane i holds row i of the block
            __syncwarp();
            float row[kNB];
            bool failed = false;
#pragma unroll
            for (int j = 0; j < kNB; ++j) row[j] = tid < nb && j <= tid ? L.at(c0 + tid, c0 + j) : 0.0f;
#pragma unroll
            for (int k = 0; k < kNB; ++k) {
                float d = __shfl_sync(0xffffffffu, row[k], k);
                const bool ok = d > 0.0f;
                failed |= !ok && k < nb;
                d = ok ? d : 1.0f;  // (past a ragged block's end: row k is zero and stays so)
                const float piv = sqrtf(d);
                row[k] = tid == k ? piv : row[k] / piv;
                // (no branch around these: their shuffles are in flight together)
#pragma unroll
                for (int j = k + 1; j < kNB; ++j)
                    row[j] = fmaf(-row[k], __shfl_sync(0xffffffffu, row[k], j), row[j]);
            }
            if (failed && tid == 0) *bad = 1;
#pragma unroll
            for (int j = 0; j < kNB; ++j) {
                diag[j][tid] = row[j];
                if (tid < nb && j <= tid) L.at(c0 + tid, c0 + j) = row[j];
            }
            __syncwarp();
            dinv[tid] = 1.0f / diag[tid][tid];
        }
        __syncthreads();
        // rows below: a thread per row, its 32 elements in registers
        for (int i = c0 + nb + tid; i < r; i += nt) {
            float v[kNB];
#pragma unroll
            for (int j = 0; j < kNB; ++j) v[j] = L.at(i, c0 + j);
#pragma unroll
            for (int k = 0; k < kNB; ++k) {
                asm volatile("" ::: "memory");  // this column's 32 loads only (all 496 would not fit the registers)
                v[k] = div_by(v[k], diag[k][k], dinv[k]);
#pragma unroll
                for (int j = k + 1; j < kNB; ++j) v[j] = fmaf(-v[k], diag[k][j], v[j]);
            }
#pragma unroll
            for (int j = 0; j < kNB; ++j) {
                L.at(i, c0 + j) = v[j];
                panel[j * ldp + i - c0 - nb] = v[j];
            }
        }
        __syncthreads();
    }
}

// One CTA: Lw = the Cholesky factor of M (lower triangle, r x r) and *logdet of M; a non-positive
// pivot sets *bad.
template <bool SMEM>
__global__ void __launch_bounds__(512)
    chol_kernel(int r, const float *__restrict__ M, float *__restrict__ Lw, float *__restrict__ logdet,
                int *__restrict__ bad) {
    extern __shared__ __align__(16) float packed[];
    __shared__ __align__(16) float diag[kNB][kNB + 4];
    __shared__ float dinv[kNB], red[32];
    float *panel = packed + (SMEM ? (r * (r + 1) / 2 + 3) / 4 * 4 : 0);
    const int tid = threadIdx.x, nt = blockDim.x;
    if (SMEM) {
        const LowerPacked L{packed};
        for (int t = tid; t < r * r; t += nt) {
            const int i = t / r, j = t % r;
            if (j <= i) L.at(i, j) = M[t];
        }
        chol_panels(r, L, bad, diag, dinv, panel);
        for (int t = tid; t < r * r; t += nt) {
            const int i = t / r, j = t % r;
            if (j <= i) Lw[t] = L.at(i, j);
        }
    } else {
        const LowerDense L{Lw, r};
        for (int t = tid; t < r * r; t += nt) Lw[t] = M[t];
        chol_panels(r, L, bad, diag, dinv, panel);
    }
    __syncthreads();
    // log det M = 2 sum log L_kk, in the order of 1024 strided sums
    for (int v = tid; v < 1024; v += nt) {
        float x = 0.0f;
        for (int k = v; k < r; k += 1024) x += logf(Lw[(long long)k * r + k]);
        for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((v & 31) == 0) red[v >> 5] = x;
    }
    __syncthreads();
    if (tid == 0) {
        float t = 0.0f;
        for (int w = 0; w < 32; ++w) t += red[w];
        *logdet = 2.0f * t;
    }
}

// X = L^-1, 32 columns per CTA: rows in blocks of 32, each first with the earlier blocks' part of the
// sums (a thread per 4 columns of a row), then by forward substitution (a thread per column).  A CTA
// is one serial chain of blocks, so latency bounds it: its columns of X stay in shared memory, and the next 32 x 32 tile of L is requested before the present one is used
// (r = 256: 103 us with both read from L2 when needed, 49 now).
constexpr int kTriLd = kNB + 4;
__global__ void __launch_bounds__(256) tri_inverse_kernel(int r, const float *__restrict__ Lw, float *__restrict__ X) {
    extern __shared__ __align__(16) float packed[];
    float *const xs = packed;  // rows c0.. of the CTA's columns
    __shared__ __align__(16) float Ls[kNB][kTriLd], S[kNB][kTriLd];
    __shared__ float dinv[kNB];
    const int tid = threadIdx.x, c0 = blockIdx.x * kNB;
    const int row = tid >> 3, cq = 4 * (tid & 7), lr = tid >> 5, lc = tid & 31;
    float next[kNB / 8];
    auto request = [&](int i0, int k0) {
#pragma unroll
        for (int u = 0; u < kNB / 8; ++u) {
            const int i = i0 + lr + 8 * u, k = k0 + lc;
            next[u] = i < r && k < r ? __ldg(Lw + (long long)i * r + k) : 0.0f;
        }
    };
    for (int t = tid; t < c0 * kNB; t += 256)  // zeros above
        if (c0 + t % kNB < r) X[(long long)(t / kNB) * r + c0 + t % kNB] = 0.0f;
    request(c0, c0);
    for (int i0 = c0; i0 < r; i0 += kNB) {
        float acc[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = i0 + row == c0 + cq + q ? 1.0f : 0.0f;
        for (int k0 = c0; k0 <= i0; k0 += kNB) {
            __syncthreads();
#pragma unroll
            for (int u = 0; u < kNB / 8; ++u) Ls[lr + 8 * u][lc] = next[u];
            const float *xb = xs + (k0 - c0) * kTriLd;
            if (k0 < i0) request(i0, k0 + kNB);
            else request(i0 + kNB, c0);
            if (k0 == i0) *reinterpret_cast<float4 *>(&S[row][cq]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
            __syncthreads();
            if (k0 < i0) {
#pragma unroll
                for (int k = 0; k < kNB; k += 4) {
                    const float4 l4 = *reinterpret_cast<const float4 *>(&Ls[row][k]);
                    const float l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float4 x = *reinterpret_cast<const float4 *>(xb + (k + u) * kTriLd + cq);
                        acc[0] = fmaf(-l[u], x.x, acc[0]);
                        acc[1] = fmaf(-l[u], x.y, acc[1]);
                        acc[2] = fmaf(-l[u], x.z, acc[2]);
                        acc[3] = fmaf(-l[u], x.w, acc[3]);
                    }
                }
            } else if (tid < kNB) {
                dinv[tid] = 1.0f / Ls[tid][tid];
                __syncwarp();
                float x[kNB];
#pragma unroll
                for (int i = 0; i < kNB; ++i) {
                    asm volatile("" ::: "memory");  // (one row's loads at a time)
                    float v = S[i][tid];
#pragma unroll
                    for (int k = 0; k < i; ++k) v = fmaf(-Ls[i][k], x[k], v);
                    x[i] = i0 + i < r ? div_by(v, Ls[i][i], dinv[i]) : 0.0f;
                    xs[(i0 - c0 + i) * kTriLd + tid] = x[i];
                    if (i0 + i < r && c0 + tid < r) X[(long long)(i0 + i) * r + c0 + tid] = x[i];
                }
            }
        }
    }
}

// Minv = M^-1 and *logdet; Lw and X (r x r each) are scratch.
inline cudaError_t spd_inverse(cudaStream_t st, int r, const float *M, float *Lw, float *X, float *Minv, float *logdet,
                               int *bad) {
    cudaError_t e;
    if (r > kInverseMax) return cudaErrorInvalidValue;
    constexpr size_t kSmemMost = 216 * 1024;  // dynamic shared memory asked for at most
    const size_t tri = r <= kCholSmemMax ? sizeof(float) * (((size_t)r * (r + 1) / 2 + 3) / 4 * 4) : 0;
    const auto chol = r <= kCholSmemMax ? chol_kernel<true> : chol_kernel<false>;
    if ((e = cudaFuncSetAttribute(chol, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMost))) return e;
    chol<<<1, 512, tri + chol_panel_bytes(r), st>>>(r, M, Lw, logdet, bad);
    if ((e = cudaGetLastError())) return e;
    const int blocks = (r + kNB - 1) / kNB;
    if ((e = cudaFuncSetAttribute(tri_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMost)))
        return e;
    tri_inverse_kernel<<<(unsigned)blocks, 256, sizeof(float) * (size_t)blocks * kNB * kTriLd, st>>>(r, Lw, X);
    if ((e = cudaGetLastError())) return e;
    return gemm(st, r, r, r, X, r, X, r, nullptr, 1.0f, 0.0f, nullptr, 0, Minv);
}

}  // namespace
}  // namespace achr
