// Batched null-space reprojection of many chains on the tensor cores, and the
// periodic-reprojection sampling driver built on it.
//
// The reference reprojects one chain at a time, x <- N (N^T x), as two FP64
// GEMVs (reprojectPoint / reprojectPoint2, ACHRcu/ACHRCuda.cu:208-230,
// triggered at :338-343).  Here all chains of a block are reprojected at
// once with the same orthogonal projector written through S:
//
//     N N^T = I - S^T (S S^T)^+ S,   so   x <- x - S^T (B (S x)),  B = (S S^T)^+.
//
//   1. r = S x for every chain, FP64 sparse (exact to rounding; |r| is the
//      small infeasibility the chain has accumulated), split into BF16 hi + lo;
//   2. z = B r as one tensor-core GEMM over all chains, with B split the same
//      way and the three leading split products (Bh rh + Bh rl + Bl rh)
//      accumulated in FP32 (achr_tc_gemm.cu);
//   3. x <- clip(x - S^T z), the sparse sum in double-float on the FP32 pipes
//      (z itself is FP32) and the subtraction in FP64, the same clip the
//      reference applies after reprojecting (correctBounds, :193-206,
//      :347-350); the chain's centre accumulator follows the point.
//
// The low-precision GEMM only ever sees the residual, so its relative error
// (about 2^-16 times the condition number of S S^T on its range) multiplies
// |S x|, not |x|: one pass takes a residual of 1e-9 to ~1e-11 while the
// point moves by no more than the residual's preimage.  Applying N N^T to x
// itself in BF16 would move every coordinate by ~1e-5 |x| and leave |S x|
// near 1e-2 for fluxes of size 1000.
#include <cublas_v2.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cusolverDn.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "achr_ctx.h"
#include "achr_float.cuh"
#include "achr_pool.h"

extern "C" void achr_io_set_error(const char *msg);

namespace achr {

void reproj_free(ReprojState *r) { delete r; }

namespace {

constexpr int kRowChunk = 64;   // residual rows per staging tile (one 128-byte BF16 row per chain)
constexpr int kResWarps = 8;
constexpr int kStageStride = 72;  // BF16 entries per chain row of the staging tile (144 B: 16-byte aligned)
constexpr int kCorrWarps = 8;
constexpr int kCorrRows = 16;     // reactions per warp of the correction
constexpr int kLoads = 4;         // nonzeros requested before any is used
constexpr size_t kResSmem = (size_t)kResWarps * 2 * 32 * kStageStride * sizeof(__nv_bfloat16);
constexpr int kMaxChunk = 65536;  // chains per GEMM

achr_status set_err(achr_status st, const std::string &msg) {
    achr_io_set_error(msg.c_str());
    return st;
}

achr_status cuda_err(cudaError_t e, const char *what) {
    return set_err(ACHR_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

#define REPROJ_TRY(expr)                                      \
    do {                                                      \
        cudaError_t e_ = (expr);                              \
        if (e_ != cudaSuccess) return achr::cuda_err(e_, #expr); \
    } while (0)

__device__ __forceinline__ unsigned long long abs_bits64(double v) {
    return (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
}

// r = S x for 32 chains per block row (lane = chain, so every load of x is
// one coalesced 256-byte row segment) and 64-row chunks per warp.  With SPLIT
// the residuals go out as BF16 hi/lo rows of R (chain-major, K = metabolite
// contiguous, the layout the GEMM's TMA maps read), staged through shared
// memory so every chain row is written as 16-byte pieces.  Always: the
// largest |r| (as non-negative double bits) goes to *maxbits.
//
// Bound by the FP64 pipe: one DFMA per nonzero and chain (5063 x 7440, 16,384
// chains: 0.98 ms at the pipe's rate) and nothing else on it, the split being
// integer and FP32 work.  The blocks of one group of chains run together (the
// row chunks vary fastest), so the group's 1.9 MB of x stay in L2 for the four
// times its rows are read.
template <bool SPLIT>
__global__ void __launch_bounds__(kResWarps * 32)
    residual_kernel(int m, int kpad, int P, const double *__restrict__ X, long long ldx,
                    const int *__restrict__ rp, const int *__restrict__ ci, const double *__restrict__ rv,
                    __nv_bfloat16 *__restrict__ Rh, __nv_bfloat16 *__restrict__ Rl,
                    unsigned long long *maxbits, const unsigned long long *prev, unsigned long long tol_bits) {
    // A chunk whose previous round found it within tolerance was not corrected,
    // so its residual is unchanged: carry the value over and skip the pass.
    if (prev && *prev <= tol_bits) {
        if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *maxbits = *prev;
        return;
    }
    extern __shared__ __align__(16) unsigned short stage_raw[];  // [warp][hi, lo][chain][row]
    __shared__ unsigned long long wmax[kResWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned short *const sh = stage_raw + (size_t)warp * 2 * 32 * kStageStride, *const sl = sh + 32 * kStageStride;
    const int p0 = blockIdx.y * 32;
    const int p = p0 + lane;
    const bool live = p < P;
    const double *xp = X + (live ? p : P - 1);
    unsigned long long mx = 0;
    const int nchunks = kpad / kRowChunk;
    for (int c = blockIdx.x * kResWarps + warp; c < nchunks; c += gridDim.x * kResWarps) {
        for (int r = 0; r < kRowChunk; ++r) {
            const int i = c * kRowChunk + r;
            double acc = 0.0;
            if (i < m) {
                const int q1 = __ldg(rp + i + 1);
                for (int q = __ldg(rp + i); q < q1; q += kLoads) {
                    double v[kLoads], x[kLoads];
#pragma unroll
                    for (int u = 0; u < kLoads; ++u) {  // past the row: its last entry again, not used
                        const int qq = min(q + u, q1 - 1);
                        v[u] = __ldg(rv + qq);
                        x[u] = xp[(long long)__ldg(ci + qq) * ldx];
                    }
#pragma unroll
                    for (int u = 0; u < kLoads; ++u)
                        if (q + u < q1) acc = fma(v[u], x[u], acc);
                }
            }
            if (live) mx = max(mx, abs_bits64(acc));
            if (SPLIT) {
                // (a residual beyond BF16's range, infinite or NaN: hi is infinite, every z of the chain infinite
                // or NaN, and the correction, whose error terms subtract infinities, NaN)
                unsigned short h, l;
                split_bf16_bits(f64_to_f32_near_any(acc), h, l);
                sh[lane * kStageStride + r] = h;
                sl[lane * kStageStride + r] = l;
            }
        }
        if (SPLIT) {
            __syncwarp();
            for (int t = lane; t < 32 * (kRowChunk / 8); t += 32) {
                const int row = t / (kRowChunk / 8), part = t % (kRowChunk / 8);
                const int pp = p0 + row;
                if (pp < P) {
                    const size_t off = (size_t)pp * (size_t)kpad + (size_t)c * kRowChunk + (size_t)part * 8;
                    *reinterpret_cast<uint4 *>(Rh + off) =
                        *reinterpret_cast<const uint4 *>(&sh[row * kStageStride + part * 8]);
                    *reinterpret_cast<uint4 *>(Rl + off) =
                        *reinterpret_cast<const uint4 *>(&sl[row * kStageStride + part * 8]);
                }
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = max(mx, (unsigned long long)__shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) wmax[warp] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kResWarps; ++w) mx = max(mx, wmax[w]);
        if (mx) atomicMax(maxbits, mx);
    }
}

// x_j <- clip(x_j - sum_i S_ij z_i, lb_j, ub_j) for 32 chains per block row
// (lane = chain: loads of z and x are coalesced rows); the centre accumulator
// moves with the point.  The sum is formed in double-float on the FP32 pipes
// (error-free products and sums, about 48 bits: far below z's own FP32
// rounding), so the FP64 pipe does only dh + dl, x - d and the accumulator's
// two additions; the clip compares integers.  Summed and converted in FP64 it
// was the larger half of a round (3.4 ms of 6.6 at 5063 x 7440, 16,384 chains).
// The blocks of one group of chains run together, so the group's z stays in L2.
template <bool EXACT32>
__global__ void __launch_bounds__(kCorrWarps * 32)
    correct_kernel(int n, int P, double *__restrict__ X, long long ldx, double *__restrict__ Acc, long long lda,
                   const int *__restrict__ cp, const int *__restrict__ ri, const float *__restrict__ ch,
                   const float *__restrict__ cl, const float *__restrict__ Z, long long ldz,
                   const double2 *__restrict__ lbub, const unsigned long long *gate, unsigned long long tol_bits) {
    if (*gate <= tol_bits) return;  // this chunk's residual is already within tolerance
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = blockIdx.y * 32 + lane;
    if (p >= P) return;
    const float *zp = Z + p;
    for (int j = blockIdx.x * kCorrWarps + warp; j < n; j += gridDim.x * kCorrWarps) {
        float ah = 0.0f, al = 0.0f;
        const int q1 = __ldg(cp + j + 1);
        for (int q = __ldg(cp + j); q < q1; q += kLoads) {
            float vh[kLoads], vl[kLoads], z[kLoads];
#pragma unroll
            for (int u = 0; u < kLoads; ++u) {
                const int qq = min(q + u, q1 - 1);
                vh[u] = __ldg(ch + qq);
                if (!EXACT32) vl[u] = __ldg(cl + qq);
                z[u] = __ldg(zp + (long long)__ldg(ri + qq) * ldz);
            }
#pragma unroll
            for (int u = 0; u < kLoads; ++u)
                if (q + u < q1) {
                    float ph, pe, s, e;
                    two_prod(vh[u], z[u], ph, pe);
                    if (!EXACT32) pe = fmaf(vl[u], z[u], pe);
                    two_sum(ah, ph, s, e);
                    ah = s;
                    al = __fadd_rn(al, __fadd_rn(e, pe));
                }
        }
        double *xp = X + (long long)j * ldx + p;
        const double xo = *xp;
        double d;
        if (fabsf(ah) + fabsf(al) < INFINITY) d = f32_to_f64_exact(ah) + f32_to_f64_exact(al);
        else d = (double)ah + (double)al;  // NaN, or beyond FP32's range: NaN
        const double xc = xo - d;
        const double xn = abs_bits64(xc) > 0x7FF0000000000000ull ? xc : clip_exact(xc, lbub[j]);
        *xp = xn;
        if (Acc) Acc[(long long)j * lda + p] += xn - xo;
    }
}

// Column k of the eigenvector matrix scaled by 1 / lambda_k (kept columns only).
__global__ void scale_columns(int m, int r, const double *__restrict__ U, const double *__restrict__ lam,
                              double *__restrict__ V) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)m * r) return;
    const int k = (int)(t / m);
    V[t] = U[t] / lam[k];
}

// F = S V diag(1 / lambda) for the kept eigenvectors V (n x r, column-major, one block column each) of
// S^T S: F F^T = sum_k (S v_k)(S v_k)^T / lambda_k^2 = (S S^T)^+, S v_k being sqrt(lambda_k) times an
// eigenvector of S S^T.
__global__ void __launch_bounds__(256)
    row_space_kernel(int n, int m, const int *__restrict__ rp, const int *__restrict__ ci,
                     const double *__restrict__ rv, const double *__restrict__ V, const double *__restrict__ lam,
                     double *__restrict__ F) {
    const int k = blockIdx.x;
    const double *v = V + (size_t)k * (size_t)n;
    const double inv = 1.0 / lam[k];
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        double acc = 0.0;
        const int q1 = __ldg(rp + i + 1);
        for (int q = __ldg(rp + i); q < q1; ++q) acc = fma(__ldg(rv + q), __ldg(v + __ldg(ci + q)), acc);
        F[(size_t)k * (size_t)m + i] = acc * inv;
    }
}

// B (m x m, symmetric, column-major) -> row-major BF16 hi/lo with zero K padding.
__global__ void split_matrix(int m, int kpad, const double *__restrict__ B, __nv_bfloat16 *__restrict__ Bh,
                             __nv_bfloat16 *__restrict__ Bl) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)m * kpad) return;
    const int i = (int)(t / kpad), k = (int)(t % kpad);
    const double v = k < m ? B[(long long)k * m + i] : 0.0;  // B[i][k] = B[k][i]
    const __nv_bfloat16 hi = __double2bfloat16(v);
    Bh[t] = hi;
    Bl[t] = __double2bfloat16(v - (double)__bfloat162float(hi));
}

// (S S^T)^+ (column-major FP64) to FP32, rows and columns permuted to the
// device row order of the chain kernel's S.
__global__ void pinv32_kernel(int m, const int *__restrict__ order, const double *__restrict__ B,
                              float *__restrict__ out) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)m * m) return;
    const int i = (int)(t / m), k = (int)(t % m);
    out[t] = (float)B[(long long)order[k] * m + order[i]];  // B symmetric, column-major
}

// The operator.  `eig` (or NULL): the eigenvectors of S^T S that span the row space (device, n x rank) and
// their eigenvalues, which the null-space set-up has anyway; with them B is one sparse and one dense
// product (2766 x 3742: 50 ms instead of 290 ms for the eigen-decomposition of S S^T).
achr_status build_reproj(achr_ctx *ctx, ReprojState &R, bool want_pinv32, const RowSpace *eig) {
    const int m = ctx->m, n = ctx->n;
    R.m = m;
    R.n = n;
    R.kpad = (m + kRowChunk - 1) / kRowChunk * kRowChunk;
    REPROJ_TRY(cudaGetDevice(&R.device));
    // CSR (as stored) and CSC of S.
    const std::vector<int> &rp = ctx->h_rowptr, &ci = ctx->h_colidx;
    const std::vector<double> &rv = ctx->h_val;
    std::vector<int> cp((size_t)n + 1, 0), ri(ci.size());
    std::vector<double> cv(ci.size());
    for (int c : ci) cp[(size_t)c + 1]++;
    for (int j = 0; j < n; ++j) cp[(size_t)j + 1] += cp[(size_t)j];
    {
        std::vector<int> fill(cp.begin(), cp.end() - 1);
        for (int i = 0; i < m; ++i)
            for (int q = rp[(size_t)i]; q < rp[(size_t)i + 1]; ++q) {
                const int dst = fill[(size_t)ci[(size_t)q]]++;
                ri[(size_t)dst] = i;
                cv[(size_t)dst] = rv[(size_t)q];
            }
    }
    REPROJ_TRY(R.rp.upload(rp.data(), rp.size()));
    REPROJ_TRY(R.ci.upload(ci.data(), ci.size()));
    REPROJ_TRY(R.rv.upload(rv.data(), rv.size()));
    REPROJ_TRY(R.cp.upload(cp.data(), cp.size()));
    REPROJ_TRY(R.ri.upload(ri.data(), ri.size()));
    std::vector<float> ch(cv.size()), cl(cv.size());
    R.exact32 = true;
    for (size_t q = 0; q < cv.size(); ++q) {
        ch[q] = (float)cv[q];
        cl[q] = (float)(cv[q] - (double)ch[q]);
        R.exact32 = R.exact32 && cl[q] == 0.0f;
    }
    REPROJ_TRY(R.ch.upload(ch.data(), ch.size()));
    REPROJ_TRY(R.cl.upload(cl.data(), cl.size()));

    // B = (S S^T)^+, from `eig` or from the eigen-decomposition of S S^T, eigenvalues
    // below m * lambda_max * 2.2204e-16 dropped (the reference's null-space cutoff
    // rule, ACHRCuda.cu:478-487, applied to S S^T).
    DevBuf<double> B;
    cublasHandle_t cb = nullptr;
    cusolverDnHandle_t sh = nullptr;
    if (cublasCreate(&cb) != CUBLAS_STATUS_SUCCESS) return set_err(ACHR_ERR_CUDA, "cublasCreate failed");
    struct Guard {
        cublasHandle_t &cb;
        cusolverDnHandle_t &sh;
        ~Guard() {
            if (sh) cusolverDnDestroy(sh);
            if (cb) cublasDestroy(cb);
        }
    } guard{cb, sh};
    const double one = 1.0, zero = 0.0;
    REPROJ_TRY(B.alloc((size_t)m * m));
    if (eig) {
        const int r = (int)eig->lam.size();
        R.rank = r;
        R.lam_max = r > 0 ? *std::max_element(eig->lam.begin(), eig->lam.end()) : 0.0;
        R.lam_min = r > 0 ? *std::min_element(eig->lam.begin(), eig->lam.end()) : 0.0;
        if (r > 0) {
            DevBuf<double> F, lam;
            REPROJ_TRY(F.alloc((size_t)m * r));
            REPROJ_TRY(lam.upload(eig->lam.data(), (size_t)r));
            row_space_kernel<<<(unsigned)r, 256>>>(n, m, R.rp.p, R.ci.p, R.rv.p, eig->V, lam.p, F.p);
            REPROJ_TRY(cudaGetLastError());
            if (cublasDgemm(cb, CUBLAS_OP_N, CUBLAS_OP_T, m, m, r, &one, F.p, m, F.p, m, &zero, B.p, m) !=
                CUBLAS_STATUS_SUCCESS)
                return set_err(ACHR_ERR_CUDA, "cublasDgemm (pseudo-inverse) failed");
            REPROJ_TRY(cudaDeviceSynchronize());  // F is freed here
        } else {
            REPROJ_TRY(cudaMemset(B.p, 0, sizeof(double) * (size_t)m * m));
        }
    } else {
        std::vector<double> dS((size_t)m * n, 0.0);
        for (int i = 0; i < m; ++i)
            for (int q = rp[(size_t)i]; q < rp[(size_t)i + 1]; ++q) dS[(size_t)ci[(size_t)q] * m + i] = rv[(size_t)q];
        DevBuf<double> S, G, lam, V;
        DevBuf<int> info;
        REPROJ_TRY(S.upload(dS.data(), dS.size()));
        dS.clear();
        dS.shrink_to_fit();
        REPROJ_TRY(G.alloc((size_t)m * m));
        REPROJ_TRY(lam.alloc((size_t)m));
        REPROJ_TRY(info.alloc(1));
        if (cublasDgemm(cb, CUBLAS_OP_N, CUBLAS_OP_T, m, m, n, &one, S.p, m, S.p, m, &zero, G.p, m) !=
            CUBLAS_STATUS_SUCCESS)
            return set_err(ACHR_ERR_CUDA, "cublasDgemm (S S^T) failed");
        S.reset();
        if (cusolverDnCreate(&sh) != CUSOLVER_STATUS_SUCCESS) return set_err(ACHR_ERR_CUDA, "cusolverDnCreate failed");
        int lwork = 0;
        if (cusolverDnDsyevd_bufferSize(sh, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, m, G.p, m, lam.p, &lwork) !=
            CUSOLVER_STATUS_SUCCESS)
            return set_err(ACHR_ERR_NUMERIC, "syevd workspace query failed");
        {
            DevBuf<double> work;
            REPROJ_TRY(work.alloc((size_t)std::max(lwork, 1)));
            if (cusolverDnDsyevd(sh, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, m, G.p, m, lam.p, work.p, lwork,
                                 info.p) != CUSOLVER_STATUS_SUCCESS)
                return set_err(ACHR_ERR_NUMERIC, "cusolverDnDsyevd (S S^T) failed");
            int h_info = 0;
            REPROJ_TRY(cudaMemcpy(&h_info, info.p, sizeof(int), cudaMemcpyDeviceToHost));
            if (h_info != 0) return set_err(ACHR_ERR_NUMERIC, "syevd of S S^T did not converge");
        }
        std::vector<double> h_lam((size_t)m);
        REPROJ_TRY(cudaMemcpy(h_lam.data(), lam.p, sizeof(double) * m, cudaMemcpyDeviceToHost));
        const double lmax = h_lam.back();
        const double tol = (double)m * lmax * 2.2204e-16;
        int k0 = 0;
        while (k0 < m && !(h_lam[(size_t)k0] > tol)) ++k0;
        const int r = m - k0;
        R.rank = r;
        R.lam_max = lmax;
        R.lam_min = r > 0 ? h_lam[(size_t)k0] : 0.0;
        if (r > 0) {
            REPROJ_TRY(V.alloc((size_t)m * r));
            const long long cnt = (long long)m * r;
            scale_columns<<<(unsigned)((cnt + 255) / 256), 256>>>(m, r, G.p + (size_t)k0 * m, lam.p + k0, V.p);
            REPROJ_TRY(cudaGetLastError());
            if (cublasDgemm(cb, CUBLAS_OP_N, CUBLAS_OP_T, m, m, r, &one, V.p, m, G.p + (size_t)k0 * m, m, &zero, B.p,
                            m) != CUBLAS_STATUS_SUCCESS)
                return set_err(ACHR_ERR_CUDA, "cublasDgemm (pseudo-inverse) failed");
        } else {
            REPROJ_TRY(cudaMemset(B.p, 0, sizeof(double) * (size_t)m * m));
        }
    }
    REPROJ_TRY(R.Bh.alloc((size_t)m * R.kpad));
    REPROJ_TRY(R.Bl.alloc((size_t)m * R.kpad));
    const long long cnt = (long long)m * R.kpad;
    split_matrix<<<(unsigned)((cnt + 255) / 256), 256>>>(m, R.kpad, B.p, R.Bh.p, R.Bl.p);
    REPROJ_TRY(cudaGetLastError());
    if (want_pinv32) {
        DevBuf<int> ord;
        REPROJ_TRY(ord.upload(ctx->h_row_order.data(), ctx->h_row_order.size()));
        REPROJ_TRY(ctx->pinv32.alloc((size_t)m * m));
        const long long mm = (long long)m * m;
        pinv32_kernel<<<(unsigned)((mm + 255) / 256), 256>>>(m, ord.p, B.p, ctx->pinv32.p);
        REPROJ_TRY(cudaGetLastError());
        REPROJ_TRY(cudaDeviceSynchronize());
    }
    REPROJ_TRY(cudaDeviceSynchronize());
    return ACHR_OK;
}

}  // namespace

achr_status ensure_reproj(achr_ctx *ctx) {
    if (ctx->reproj) return ACHR_OK;
    std::unique_ptr<ReprojState> R(new (std::nothrow) ReprojState());
    if (!R) return set_err(ACHR_ERR_NOMEM, "allocation failed");
    const achr_status st = build_reproj(ctx, *R, false, nullptr);
    if (st == ACHR_OK) ctx->reproj = R.release();
    return st;
}

namespace {

achr_status ensure_chunk(ReprojState &R, int chunk) {
    if (chunk <= R.chunk_cap) return ACHR_OK;
    R.Rh.reset();
    R.Rl.reset();
    R.Z.reset();
    R.chunk_cap = 0;
    REPROJ_TRY(R.Rh.alloc((size_t)chunk * R.kpad));
    REPROJ_TRY(R.Rl.alloc((size_t)chunk * R.kpad));
    REPROJ_TRY(R.Z.alloc((size_t)R.m * chunk));
    R.chunk_cap = chunk;
    return ACHR_OK;
}

double bits_to_double(unsigned long long b) {
    double v;
    std::memcpy(&v, &b, sizeof v);
    return v;
}

dim3 residual_grid(int P, int kpad) {
    const int nchunks = kpad / kRowChunk;
    return dim3((unsigned)((nchunks + kResWarps - 1) / kResWarps), (unsigned)((P + 31) / 32));
}

}  // namespace

achr_status build_operator(achr_ctx *ctx, bool want_pinv32, const RowSpace *eig) {
    if (ctx->reproj && (!want_pinv32 || ctx->pinv32.p)) return ACHR_OK;
    if ((int)ctx->h_row_order.size() != ctx->m) return set_err(ACHR_ERR_INVALID, "row order missing");
    std::unique_ptr<ReprojState> R(new (std::nothrow) ReprojState());
    if (!R) return set_err(ACHR_ERR_NOMEM, "allocation failed");
    const achr_status st = build_reproj(ctx, *R, want_pinv32, eig);
    if (st != ACHR_OK) return st;
    reproj_free(ctx->reproj);
    ctx->reproj = R.release();
    return ACHR_OK;
}

}  // namespace achr

using achr::ReprojState;

extern "C" {

achr_status achr_gemm_bf16(int32_t M, int32_t N, int32_t K, int32_t nsplit, const void *A0, const void *A1,
                           int64_t lda, const void *B0, const void *B1, int64_t ldb, float *C, int64_t ldc,
                           void *stream) {
    achr::TcGemm g{M, N, K, nsplit, A0, A1, (long long)lda, B0, B1, (long long)ldb, C, (long long)ldc};
    if (const char *why = achr::tc_gemm_check(g)) return achr::set_err(ACHR_ERR_INVALID, why);
    achr::PoolBuf buf((cudaStream_t)stream);
    REPROJ_TRY(buf.alloc(sizeof(unsigned long long)));
    unsigned long long *err = reinterpret_cast<unsigned long long *>(buf.p);
    REPROJ_TRY(cudaMemsetAsync(err, 0, sizeof(unsigned long long), (cudaStream_t)stream));
    REPROJ_TRY(achr::launch_tc_gemm(g, err, (cudaStream_t)stream));
    unsigned long long h = 0;
    REPROJ_TRY(cudaMemcpyAsync(&h, err, sizeof h, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    REPROJ_TRY(cudaStreamSynchronize((cudaStream_t)stream));
    if (h) return achr::set_err(ACHR_ERR_TIMEOUT, "a tensor-core pipeline wait expired");
    return ACHR_OK;
}

achr_status achr_reproject_batch(achr_ctx *ctx, int32_t n_points, double *d_points, double *d_centre_acc, int64_t ld,
                                 int32_t max_rounds, void *stream_v, achr_reproj_stats *stats) {
    using namespace achr;
    if (!ctx || !d_points || n_points < 0 || max_rounds < 1 || max_rounds > 16 || ld < n_points)
        return set_err(ACHR_ERR_INVALID, "bad reprojection arguments");
    if (stats) std::memset(stats, 0, sizeof *stats);
    if (n_points == 0 || ctx->m == 0) return ACHR_OK;
    achr_status st = ensure_reproj(ctx);
    if (st != ACHR_OK) return st;
    ReprojState &R = *ctx->reproj;
    const int chunk = std::min(n_points, kMaxChunk);
    st = ensure_chunk(R, chunk);
    if (st != ACHR_OK) return st;
    const int nchunks = (n_points + chunk - 1) / chunk;
    REPROJ_TRY(cudaFuncSetAttribute(residual_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResSmem));
    const size_t nflags = 8 + (size_t)max_rounds * nchunks;
    if (R.flags.count < nflags) REPROJ_TRY(R.flags.alloc(nflags));
    cudaStream_t s = (cudaStream_t)stream_v;
    REPROJ_TRY(cudaMemsetAsync(R.flags.p, 0, nflags * sizeof(unsigned long long), s));
    double tol = ctx->opt.residual_tol;
    unsigned long long tol_bits;
    std::memcpy(&tol_bits, &tol, sizeof tol_bits);

    std::vector<cudaEvent_t> ev;  // destroyed on every return below
    struct EvGuard {
        std::vector<cudaEvent_t> &v;
        ~EvGuard() {
            for (cudaEvent_t e : v) cudaEventDestroy(e);
        }
    } ev_guard{ev};
    auto new_event = [&](cudaEvent_t &e) -> bool {
        if (cudaEventCreate(&e) != cudaSuccess) return false;
        ev.push_back(e);
        return true;
    };
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    if (stats) {
        if (!new_event(t0) || !new_event(t1)) return set_err(ACHR_ERR_CUDA, "cudaEventCreate failed");
        REPROJ_TRY(cudaEventRecord(t0, s));
    }
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> gemm_ev;
    std::vector<double> chunk_flops((size_t)nchunks, 0.0);
    // Round r, chunk c: residual + split, then (gated on that chunk's residual
    // exceeding residual_tol) the tensor-core GEMM and the correction.
    for (int r = 0; r < max_rounds; ++r) {
        for (int c = 0; c < nchunks; ++c) {
            const int c0 = c * chunk;
            const int pc = std::min(chunk, n_points - c0);
            double *X = d_points + c0;
            unsigned long long *slot = R.flags.p + 8 + (size_t)r * nchunks + c;
            const unsigned long long *prev = r > 0 ? slot - nchunks : nullptr;
            residual_kernel<true><<<residual_grid(pc, R.kpad), kResWarps * 32, kResSmem, s>>>(
                R.m, R.kpad, pc, X, ld, R.rp.p, R.ci.p, R.rv.p, R.Rh.p, R.Rl.p, slot, prev, tol_bits);
            REPROJ_TRY(cudaGetLastError());
            TcGemm g{R.m, pc, R.kpad, 3, R.Bh.p, R.Bl.p, (long long)R.kpad, R.Rh.p, R.Rl.p, (long long)R.kpad,
                     R.Z.p, (long long)pc};
            g.gate = slot;
            g.gate_max = tol_bits;
            if (const char *why = tc_gemm_check(g)) return set_err(ACHR_ERR_INVALID, why);
            cudaEvent_t g0 = nullptr, g1 = nullptr;
            if (stats) {
                if (!new_event(g0) || !new_event(g1)) return set_err(ACHR_ERR_CUDA, "cudaEventCreate failed");
                REPROJ_TRY(cudaEventRecord(g0, s));
            }
            REPROJ_TRY(launch_tc_gemm(g, R.flags.p + 2, s));
            if (stats) {
                REPROJ_TRY(cudaEventRecord(g1, s));
                gemm_ev.emplace_back(g0, g1);
            }
            chunk_flops[(size_t)c] = tc_gemm_flops(g);
            const dim3 cgrid((unsigned)((R.n + kCorrWarps * kCorrRows - 1) / (kCorrWarps * kCorrRows)),
                             (unsigned)((pc + 31) / 32));
            (R.exact32 ? correct_kernel<true> : correct_kernel<false>)<<<cgrid, kCorrWarps * 32, 0, s>>>(
                R.n, pc, X, ld, d_centre_acc ? d_centre_acc + c0 : nullptr, ld, R.cp.p, R.ri.p, R.ch.p, R.cl.p, R.Z.p,
                (long long)pc, ctx->lbub.p, slot, tol_bits);
            REPROJ_TRY(cudaGetLastError());
        }
    }
    if (stats) {
        for (int c0 = 0; c0 < n_points; c0 += chunk) {
            const int pc = std::min(chunk, n_points - c0);
            residual_kernel<false><<<residual_grid(pc, R.kpad), kResWarps * 32, 0, s>>>(
                R.m, R.kpad, pc, d_points + c0, ld, R.rp.p, R.ci.p, R.rv.p, nullptr, nullptr, R.flags.p + 1, nullptr,
                0ull);
            REPROJ_TRY(cudaGetLastError());
        }
        REPROJ_TRY(cudaEventRecord(t1, s));
    }
    std::vector<unsigned long long> h(nflags, 0);
    REPROJ_TRY(cudaMemcpyAsync(h.data(), R.flags.p, nflags * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    REPROJ_TRY(cudaStreamSynchronize(s));
    if (h[2]) return set_err(ACHR_ERR_TIMEOUT, "a tensor-core pipeline wait expired");
    if (stats) {
        float ms = 0.0f;
        double gms = 0.0, flops = 0.0;
        int rounds = 0;
        unsigned long long before = 0;
        for (int c = 0; c < nchunks; ++c) before = std::max(before, h[8 + (size_t)c]);
        for (int r = 0; r < max_rounds; ++r) {
            bool any = false;
            for (int c = 0; c < nchunks; ++c)
                if (h[8 + (size_t)r * nchunks + c] > tol_bits) {
                    any = true;
                    flops += chunk_flops[(size_t)c];
                    if (cudaEventElapsedTime(&ms, gemm_ev[(size_t)r * nchunks + c].first,
                                             gemm_ev[(size_t)r * nchunks + c].second) == cudaSuccess)
                        gms += ms;
                }
            rounds += any ? 1 : 0;
        }
        REPROJ_TRY(cudaEventElapsedTime(&ms, t0, t1));
        stats->residual_before = bits_to_double(before);
        stats->residual_after = bits_to_double(h[1]);
        stats->gemm_ms = gms;
        stats->total_ms = ms;
        stats->gemm_flops = flops;
        stats->rounds = rounds;
        stats->rank = R.rank;
        stats->lambda_min = R.lam_min;
        stats->lambda_max = R.lam_max;
    }
    return ACHR_OK;
}

achr_status achr_sample_periodic(achr_ctx *ctx, uint64_t seed, uint64_t chain_offset, int32_t n_points,
                                 int32_t n_steps, int32_t period, int32_t max_rounds, double *d_points,
                                 double *d_centre_acc, int64_t ld, void *stream, achr_stats *stats,
                                 achr_reproj_stats *rstats) {
    if (!ctx || !d_points || !d_centre_acc || n_points < 0 || n_steps < 0 || period <= 0 || max_rounds < 1 ||
        ld < n_points)
        return achr::set_err(ACHR_ERR_INVALID, "bad periodic-sampling arguments");
    if (stats) std::memset(stats, 0, sizeof *stats);
    if (rstats) std::memset(rstats, 0, sizeof *rstats);
    for (int t0 = 0; t0 < n_steps || (t0 == 0 && n_steps == 0); t0 += period) {
        const int seg = std::min(period, n_steps - t0);
        achr_stats s1;
        achr_status st = achr_sample_resume(ctx, seed, chain_offset, n_points, t0, seg, t0 > 0 ? 1 : 0, d_points,
                                            d_centre_acc, ld, stream, stats ? &s1 : nullptr);
        if (st != ACHR_OK) return st;
        if (stats) {
            stats->accepted += s1.accepted;
            stats->rejected += s1.rejected;
            stats->checks += s1.checks;
            stats->reprojections += s1.reprojections;
            stats->stuck_chains = std::max(stats->stuck_chains, s1.stuck_chains);
            stats->exact_evals += s1.exact_evals;
            stats->final_projections += s1.final_projections;
            stats->max_bound_violation = std::max(stats->max_bound_violation, s1.max_bound_violation);
            stats->max_residual = s1.max_residual;
            stats->kernel_ms += s1.kernel_ms;
        }
        if (n_steps == 0) break;
        achr_reproj_stats r1;
        st = achr_reproject_batch(ctx, n_points, d_points, d_centre_acc, ld, max_rounds, stream,
                                  rstats ? &r1 : nullptr);
        if (st != ACHR_OK) return st;
        if (rstats) {
            rstats->residual_before = std::max(rstats->residual_before, r1.residual_before);
            rstats->residual_after = std::max(rstats->residual_after, r1.residual_after);
            rstats->gemm_ms += r1.gemm_ms;
            rstats->total_ms += r1.total_ms;
            rstats->gemm_flops += r1.gemm_flops;
            rstats->rounds += r1.rounds;
            rstats->rank = r1.rank;
            rstats->lambda_min = r1.lambda_min;
            rstats->lambda_max = r1.lambda_max;
        }
        if (stats && rstats) stats->max_residual = r1.residual_after;  // the emitted points are the reprojected ones
    }
    return ACHR_OK;
}

}  // extern "C"
