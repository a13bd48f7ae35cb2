// Batched dense complex linear algebra in FP64 (interleaved complex128,
// column-major): GEMM, LU with partial pivoting, triangular solves.
//
// Every routine works on `batch` independent matrices `stride` elements
// apart, so a whole spectrum of wavelengths goes through each launch
// together: per-matrix latency (the column-by-column panel) is hidden by the
// other matrices in the batch.
#include "common.cuh"
#include "dense_f64.cuh"
#include "lu_panel.cuh"

namespace mnpb {

// ---------------------------------------------------------------------------
// GEMM: C = alpha A B + beta C, all no-transpose, on the FP64 tensor path
// (mma.sync m16n8k4, FP64 accumulation; there is no tcgen05 kind for FP64).
// Four warps per CTA, each a (BM/2) x (BN/2) block of real and imaginary
// accumulators; operands come through a ring of cp.async stages as they are
// stored (interleaved complex), so one 16-byte shared load feeds both parts.
// Shared strides: A columns are BM + 2 elements and B columns 12 elements
// apart, so that the eight lanes of a 128-bit load phase (2 rows x 4 k) hit
// eight different 16-byte bank groups.  Bound by the FP64 pipe (37 TFLOP/s):
// 2884 x 2884 x 2884 8.51 -> 6.54 ms (29.3 TFLOP/s), 41 x 1148 x 512 x 512
// 4.01 -> 3.00 ms (32.9) against the FMA kernel with one 64 x 64 tile shape
// this replaces.
// ---------------------------------------------------------------------------
namespace {
constexpr int GK = 8, GSTAGES = 4, GTHREADS = 128;
constexpr int GBS = GK + 4;   // B column stride in shared memory

__device__ __forceinline__ void cp16(uint32_t dst, const void *src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
                 "r"(ok ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void mma_f64(double (&d)[4], double a0, double a1, double b) {
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, "
                 "{%6}, {%0,%1,%2,%3};"
                 : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
                 : "d"(a0), "d"(a1), "d"(b));
}

template <int BM, int BN>
__global__ void __launch_bounds__(GTHREADS) zgemm_kernel(int m, int n, int k, cd alpha,
                                                         const cd *__restrict__ A, int64_t lda,
                                                         int64_t sA, const cd *__restrict__ B,
                                                         int64_t ldb, int64_t sB, cd beta,
                                                         cd *__restrict__ C, int64_t ldc,
                                                         int64_t sC) {
    constexpr int AS = BM + 2;               // A column (fixed k) stride
    constexpr int MI = BM / 32, NI = BN / 16;   // 16 x 8 fragments per warp
    extern __shared__ __align__(16) cd zsm[];
    cd *As = zsm;                            // [GSTAGES][GK][AS]
    cd *Bs = zsm + GSTAGES * GK * AS;        // [GSTAGES][BN][GBS]
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int wm = (wid & 1) * (BM / 2), wn = (wid >> 1) * (BN / 2);
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int64_t b = blockIdx.z;
    A += b * sA;
    B += b * sB;
    C += b * sC;
    double re[MI][NI][4], im[MI][NI][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) re[i][j][e] = im[i][j][e] = 0.0;
    const int nk = (k + GK - 1) / GK;
    auto load = [&](int kt) {
        if (kt < nk) {
            const int st = kt % GSTAGES, k0 = kt * GK;
            const uint32_t da = (uint32_t)__cvta_generic_to_shared(As + st * GK * AS);
            const uint32_t db = (uint32_t)__cvta_generic_to_shared(Bs + st * BN * GBS);
#pragma unroll
            for (int e = tid; e < BM * GK; e += GTHREADS) {
                const int r = e % BM, kk = e / BM;
                const bool ok = m0 + r < m && k0 + kk < k;
                cp16(da + (kk * AS + r) * 16, ok ? A + (int64_t)(k0 + kk) * lda + m0 + r : A, ok);
            }
#pragma unroll
            for (int e = tid; e < BN * GK; e += GTHREADS) {
                const int kk = e % GK, c = e / GK;
                const bool ok = n0 + c < n && k0 + kk < k;
                cp16(db + (c * GBS + kk) * 16, ok ? B + (int64_t)(n0 + c) * ldb + k0 + kk : B, ok);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int q = 0; q < GSTAGES - 1; ++q) load(q);
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GSTAGES - 2) : "memory");
        __syncthreads();                       // stage kt has landed; stage kt - 1 is free
        load(kt + GSTAGES - 1);
        const cd *as = As + (kt % GSTAGES) * GK * AS + wm + g;
        const cd *bs = Bs + (kt % GSTAGES) * BN * GBS + (wn + g) * GBS;
#pragma unroll
        for (int ks = 0; ks < GK; ks += 4) {
            cd av[MI][2], bv[NI];
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) av[i][h] = as[(ks + t) * AS + 16 * i + 8 * h];
#pragma unroll
            for (int j = 0; j < NI; ++j) bv[j] = bs[8 * j * GBS + ks + t];
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NI; ++j) {
                    mma_f64(re[i][j], av[i][0].x, av[i][1].x, bv[j].x);
                    mma_f64(im[i][j], av[i][0].x, av[i][1].x, bv[j].y);
                }
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NI; ++j) {
                    mma_f64(re[i][j], -av[i][0].y, -av[i][1].y, bv[j].y);
                    mma_f64(im[i][j], av[i][0].y, av[i][1].y, bv[j].x);
                }
        }
    }
    const bool beta0 = (beta.x == 0.0 && beta.y == 0.0);
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        cd cv[NI][4];
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int gr = m0 + wm + 16 * i + g + 8 * (e >> 1);
                const int gc = n0 + wn + 8 * j + 2 * t + (e & 1);
                cv[j][e] = (!beta0 && gr < m && gc < n) ? C[(int64_t)gc * ldc + gr]
                                                        : cmk(0.0, 0.0);
            }
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int gr = m0 + wm + 16 * i + g + 8 * (e >> 1);
                const int gc = n0 + wn + 8 * j + 2 * t + (e & 1);
                if (gr < m && gc < n)
                    C[(int64_t)gc * ldc + gr] =
                        cfma(beta, cv[j][e], cmul(alpha, cmk(re[i][j][e], im[i][j][e])));
            }
    }
}

// ---------------------------------------------------------------------------
// LU panel: columns [k0, k0+kb) over rows [k0, n), one CTA per matrix.
// Pivot = first row of maximal |re|+|im| (LAPACK izamax rule).
// ---------------------------------------------------------------------------
constexpr int PANEL_THREADS = 512;

__global__ void __launch_bounds__(PANEL_THREADS) panel_kernel(int n, int k0, int kb, cd *A,
                                                              int64_t lda, int64_t sA,
                                                              int32_t *ipiv, int64_t sP,
                                                              int32_t *info) {
    __shared__ double red_v[PANEL_THREADS / 32];
    __shared__ int red_i[PANEL_THREADS / 32];
    __shared__ cd prow[64];
    __shared__ int s_piv;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t b = blockIdx.x;
    A += b * sA;
    ipiv += b * sP;
    for (int jj = 0; jj < kb; ++jj) {
        const int c = k0 + jj;
        cd *col = A + (int64_t)c * lda;
        double best = -1.0;
        int bi = n;
        for (int r = c + tid; r < n; r += PANEL_THREADS) {
            double v = cabs1(col[r]);
            if (v > best) { best = v; bi = r; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            double ov = __shfl_xor_sync(0xffffffffu, best, o);
            int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) { red_v[wid] = best; red_i[wid] = bi; }
        __syncthreads();
        if (wid == 0) {
            best = (lane < PANEL_THREADS / 32) ? red_v[lane] : -1.0;
            bi = (lane < PANEL_THREADS / 32) ? red_i[lane] : n;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                double ov = __shfl_xor_sync(0xffffffffu, best, o);
                int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
            }
            if (lane == 0) {
                int p = bi;
                if (!(best > 0.0)) {       // zero column: no interchange, record singularity
                    p = c;
                    if (info && info[b] == 0) info[b] = c + 1;
                }
                s_piv = p;
                ipiv[c] = p;
            }
        }
        __syncthreads();
        const int p = s_piv;
        if (p != c) {
            for (int cc = tid; cc < kb; cc += PANEL_THREADS) {
                cd *cp = A + (int64_t)(k0 + cc) * lda;
                cd t = cp[c];
                cp[c] = cp[p];
                cp[p] = t;
            }
        }
        __syncthreads();
        const int rest = kb - jj;
        for (int cc = tid; cc < rest; cc += PANEL_THREADS) prow[cc] = A[(int64_t)(c + cc) * lda + c];
        __syncthreads();
        const cd piv = prow[0];
        const bool nz = (piv.x != 0.0 || piv.y != 0.0);
        const cd inv = nz ? crcp(piv) : cmk(0.0, 0.0);
        for (int r = c + 1 + tid; r < n; r += PANEL_THREADS) {
            cd l = col[r];
            if (nz) l = cmul(l, inv);
            col[r] = l;
            for (int cc = 1; cc < rest; ++cc) {
                cd *q = A + (int64_t)(c + cc) * lda + r;
                *q = cfms(l, prow[cc], *q);
            }
        }
        __syncthreads();
    }
}

// Row interchanges piv[c0..c1) applied to columns [j0, j1) (forward or
// backward order), one thread per column.
__global__ void laswp_kernel(cd *A, int64_t lda, int64_t sA, int j0, int j1, int jskip0,
                             int jskip1, const int32_t *ipiv, int64_t sP, int c0, int c1,
                             int forward) {
    const int64_t b = blockIdx.y;
    int j = j0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= j1) return;
    if (j >= jskip0 && j < jskip1) return;
    cd *col = A + b * sA + (int64_t)j * lda;
    const int32_t *pv = ipiv + b * sP;
    if (forward) {
        for (int c = c0; c < c1; ++c) {
            int p = pv[c];
            if (p != c) { cd t = col[c]; col[c] = col[p]; col[p] = t; }
        }
    } else {
        for (int c = c1 - 1; c >= c0; --c) {
            int p = pv[c];
            if (p != c) { cd t = col[c]; col[c] = col[p]; col[p] = t; }
        }
    }
}

// Column interchanges of X (rows [0, m)), c from n-1 down to 0: X <- X P.
__global__ void colswp_kernel(cd *X, int64_t ldx, int64_t sX, int m, const int32_t *ipiv,
                              int64_t sP, int n) {
    const int64_t b = blockIdx.y;
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= m) return;
    cd *x = X + b * sX + r;
    const int32_t *pv = ipiv + b * sP;
    for (int c = n - 1; c >= 0; --c) {
        int p = pv[c];
        if (p != c) {
            cd t = x[(int64_t)c * ldx];
            x[(int64_t)c * ldx] = x[(int64_t)p * ldx];
            x[(int64_t)p * ldx] = t;
        }
    }
}

// Small triangular solves on a kb x kb diagonal block (kb <= 32).
// mode 0: left lower unit     L x = b   (one thread per column of B)
// mode 1: left upper non-unit U x = b   (one thread per column of B)
// mode 2: right upper non-unit x U = b  (one thread per row of B)
// mode 3: right lower unit     x L = b  (one thread per row of B)
constexpr int TS = 32;

__global__ void __launch_bounds__(128) trsm_small_kernel(int mode, int kb, const cd *T,
                                                         int64_t ldt, int64_t sT, cd *B,
                                                         int64_t ldb, int64_t sB, int nvec) {
    __shared__ cd Ts[TS][TS + 1];
    const int64_t b = blockIdx.y;
    T += b * sT;
    B += b * sB;
    for (int e = threadIdx.x; e < TS * TS; e += blockDim.x) {
        int r = e % TS, c = e / TS;
        Ts[r][c] = (r < kb && c < kb) ? T[(int64_t)c * ldt + r] : cmk(r == c ? 1.0 : 0.0, 0.0);
    }
    __syncthreads();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nvec) return;
    cd x[TS];
    const bool left = (mode < 2);
    // element e of the vector: left -> B(e, v); right -> B(v, e)
#pragma unroll
    for (int e = 0; e < TS; ++e)
        x[e] = (e < kb) ? (left ? B[(int64_t)v * ldb + e] : B[(int64_t)e * ldb + v]) : cmk(0, 0);
    if (mode == 0) {
#pragma unroll
        for (int r = 1; r < TS; ++r)
#pragma unroll
            for (int c = 0; c < r; ++c) x[r] = cfms(Ts[r][c], x[c], x[r]);
    } else if (mode == 1) {
#pragma unroll
        for (int r = TS - 1; r >= 0; --r) {
#pragma unroll
            for (int c = r + 1; c < TS; ++c) x[r] = cfms(Ts[r][c], x[c], x[r]);
            x[r] = cdiv(x[r], Ts[r][r]);
        }
    } else if (mode == 2) {
#pragma unroll
        for (int c = 0; c < TS; ++c) {
#pragma unroll
            for (int r = 0; r < c; ++r) x[c] = cfms(x[r], Ts[r][c], x[c]);
            x[c] = cdiv(x[c], Ts[c][c]);
        }
    } else {
#pragma unroll
        for (int c = TS - 1; c >= 0; --c)
#pragma unroll
            for (int r = c + 1; r < TS; ++r) x[c] = cfms(x[r], Ts[r][c], x[c]);
    }
#pragma unroll
    for (int e = 0; e < TS; ++e)
        if (e < kb) {
            if (left) B[(int64_t)v * ldb + e] = x[e];
            else B[(int64_t)e * ldb + v] = x[e];
        }
}

__global__ void set_identity_kernel(cd *W, int64_t ldw, int64_t sW, int n) {
    const int64_t b = blockIdx.z;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int j = blockIdx.y;
    if (i >= n) return;
    W[b * sW + (int64_t)j * ldw + i] = cmk(i == j ? 1.0 : 0.0, 0.0);
}

}  // namespace

// ---------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------
template <int BM, int BN>
static int launch_zgemm(cudaStream_t s, int m, int n, int k, int batch, cd alpha, const cd *A,
                        int64_t lda, int64_t sA, const cd *B, int64_t ldb, int64_t sB, cd beta,
                        cd *C, int64_t ldc, int64_t sC) {
    const int smem = GSTAGES * (GK * (BM + 2) + BN * GBS) * (int)sizeof(cd);
    MNPB_TRY(smem_opt_in(zgemm_kernel<BM, BN>, smem, "zgemm_kernel"));
    dim3 grid(ceil_div(m, BM), ceil_div(n, BN), batch);
    zgemm_kernel<BM, BN><<<grid, GTHREADS, smem, s>>>(m, n, k, alpha, A, lda, sA, B, ldb, sB,
                                                      beta, C, ldc, sC);
    MNPB_LAUNCH_CHECK("zgemm_kernel");
    return MNPB_OK;
}

int zgemm(cudaStream_t s, int m, int n, int k, int batch, cd alpha, const cd *A, int64_t lda,
          int64_t sA, const cd *B, int64_t ldb, int64_t sB, cd beta, cd *C, int64_t ldc,
          int64_t sC) {
    if (m <= 0 || n <= 0 || batch <= 0) return MNPB_OK;
    ProfScope ps(s, PC_ZGEMM, 8.0 * m * n * (double)(k > 0 ? k : 0) * batch);
    // C = beta C for k <= 0
    // 64 x 64 tiles once two CTAs per SM have one; smaller tiles until then,
    // so that small updates and few right-hand sides spread over the SMs
    // (2800 x 32 x 32, 2 matrices: 20.7 -> 14.6 us; 2884 x 4 x 2884, which a
    // 64-column tile padded 16-fold: 795 -> 157 us)
    const int kk = k > 0 ? k : 0;
    const int64_t t64 = (int64_t)ceil_div(m, 64) * ceil_div(n, 64) * batch;
    const int64_t t32 = (int64_t)ceil_div(m, 64) * ceil_div(n, 32) * batch;
    if (t64 >= 2 * device_sms() && n > 32)
        return launch_zgemm<64, 64>(s, m, n, kk, batch, alpha, A, lda, sA, B, ldb, sB, beta, C,
                                    ldc, sC);
    if (t32 >= 2 * device_sms())
        return launch_zgemm<64, 32>(s, m, n, kk, batch, alpha, A, lda, sA, B, ldb, sB, beta, C,
                                    ldc, sC);
    return launch_zgemm<32, 32>(s, m, n, kk, batch, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc,
                                sC);
}

static int trsm_small(cudaStream_t s, int mode, int kb, const cd *T, int64_t ldt, int64_t sT,
                      cd *B, int64_t ldb, int64_t sB, int nvec, int batch) {
    if (nvec <= 0 || kb <= 0) return MNPB_OK;
    dim3 grid(ceil_div(nvec, 128), batch);
    ProfScope ps(s, PC_TRSM, 4.0 * kb * kb * (double)nvec * batch);
    trsm_small_kernel<<<grid, 128, 0, s>>>(mode, kb, T, ldt, sT, B, ldb, sB, nvec);
    MNPB_LAUNCH_CHECK("trsm_small_kernel");
    return MNPB_OK;
}

static int split_point(int n) {
    int h = n / 2;
    h = (h / TS) * TS;
    return h < TS ? TS : h;
}

// L X = B, L unit lower n x n; B n x m.
int trsm_llu(cudaStream_t s, int n, int m, int batch, const cd *L, int64_t ldl, int64_t sL,
             cd *B, int64_t ldb, int64_t sB) {
    if (n <= TS) return trsm_small(s, 0, n, L, ldl, sL, B, ldb, sB, m, batch);
    int n1 = split_point(n);
    MNPB_TRY(trsm_llu(s, n1, m, batch, L, ldl, sL, B, ldb, sB));
    MNPB_TRY(zgemm(s, n - n1, m, n1, batch, cmk(-1, 0), L + n1, ldl, sL, B, ldb, sB, cmk(1, 0),
                   B + n1, ldb, sB));
    return trsm_llu(s, n - n1, m, batch, L + n1 + (int64_t)n1 * ldl, ldl, sL, B + n1, ldb, sB);
}

// U X = B, U upper non-unit.
int trsm_lun(cudaStream_t s, int n, int m, int batch, const cd *U, int64_t ldu, int64_t sU,
             cd *B, int64_t ldb, int64_t sB) {
    if (n <= TS) return trsm_small(s, 1, n, U, ldu, sU, B, ldb, sB, m, batch);
    int n1 = split_point(n);
    MNPB_TRY(trsm_lun(s, n - n1, m, batch, U + n1 + (int64_t)n1 * ldu, ldu, sU, B + n1, ldb, sB));
    MNPB_TRY(zgemm(s, n1, m, n - n1, batch, cmk(-1, 0), U + (int64_t)n1 * ldu, ldu, sU, B + n1,
                   ldb, sB, cmk(1, 0), B, ldb, sB));
    return trsm_lun(s, n1, m, batch, U, ldu, sU, B, ldb, sB);
}

// X U = B, U upper non-unit n x n; X, B m x n.
int trsm_run(cudaStream_t s, int n, int m, int batch, const cd *U, int64_t ldu, int64_t sU,
             cd *B, int64_t ldb, int64_t sB) {
    if (n <= TS) return trsm_small(s, 2, n, U, ldu, sU, B, ldb, sB, m, batch);
    int n1 = split_point(n);
    MNPB_TRY(trsm_run(s, n1, m, batch, U, ldu, sU, B, ldb, sB));
    MNPB_TRY(zgemm(s, m, n - n1, n1, batch, cmk(-1, 0), B, ldb, sB, U + (int64_t)n1 * ldu, ldu,
                   sU, cmk(1, 0), B + (int64_t)n1 * ldb, ldb, sB));
    return trsm_run(s, n - n1, m, batch, U + n1 + (int64_t)n1 * ldu, ldu, sU,
                    B + (int64_t)n1 * ldb, ldb, sB);
}

// X L = B, L unit lower n x n; X, B m x n.
int trsm_rlu(cudaStream_t s, int n, int m, int batch, const cd *L, int64_t ldl, int64_t sL,
             cd *B, int64_t ldb, int64_t sB) {
    if (n <= TS) return trsm_small(s, 3, n, L, ldl, sL, B, ldb, sB, m, batch);
    int n1 = split_point(n);
    MNPB_TRY(trsm_rlu(s, n - n1, m, batch, L + n1 + (int64_t)n1 * ldl, ldl, sL,
                      B + (int64_t)n1 * ldb, ldb, sB));
    MNPB_TRY(zgemm(s, m, n1, n - n1, batch, cmk(-1, 0), B + (int64_t)n1 * ldb, ldb, sB, L + n1,
                   ldl, sL, cmk(1, 0), B, ldb, sB));
    return trsm_rlu(s, n1, m, batch, L, ldl, sL, B, ldb, sB);
}

int laswp(cudaStream_t s, cd *A, int64_t lda, int64_t sA, int ncols, int jskip0, int jskip1,
          const int32_t *ipiv, int64_t sP, int c0, int c1, bool forward, int batch) {
    if (ncols <= 0 || c1 <= c0) return MNPB_OK;
    dim3 grid(ceil_div(ncols, 128), batch);
    ProfScope ps(s, PC_SWAP, 0.0);
    laswp_kernel<<<grid, 128, 0, s>>>(A, lda, sA, 0, ncols, jskip0, jskip1, ipiv, sP, c0, c1,
                                      forward ? 1 : 0);
    MNPB_LAUNCH_CHECK("laswp_kernel");
    return MNPB_OK;
}

// Row interchanges piv[c0..c1) applied to the columns [j0, j1) only.
static int laswp_range(cudaStream_t s, cd *A, int64_t lda, int64_t sA, int j0, int j1,
                       const int32_t *ipiv, int64_t sP, int c0, int c1, int batch) {
    if (j1 <= j0 || c1 <= c0) return MNPB_OK;
    dim3 grid(ceil_div(j1 - j0, 128), batch);
    ProfScope ps(s, PC_SWAP, 0.0);
    laswp_kernel<<<grid, 128, 0, s>>>(A, lda, sA, j0, j1, 0, 0, ipiv, sP, c0, c1, 1);
    MNPB_LAUNCH_CHECK("laswp_kernel");
    return MNPB_OK;
}

// Columns of an LU leaf over m rows: what the cluster's registers hold (32, 16
// or 8 columns of 1, 2 or 4 rows a thread); beyond that the leaf in global
// memory takes 32.
static int leaf_width(int m) {
    int C, threads;
    if (lup::panel_shape(m, 1, C, threads)) return TS;
    if (lup::panel_shape(m, 2, C, threads)) return TS / 2;
    if (lup::panel_shape(m, 4, C, threads)) return TS / 4;
    return TS;
}

// Recursive LU: factor columns [off, off+w) over rows [off, n); absolute pivots.
static int rgetrf(cudaStream_t s, int n, int off, int w, int batch, cd *A, int64_t lda,
                  int64_t sA, int32_t *ipiv, int64_t sP, int32_t *info) {
    if (w <= leaf_width(n - off)) {
        ProfScope ps(s, PC_PANEL, 8.0 * w * w * (double)(n - off) * batch / 2);
        const lup::F64::Mat mat{A, lda, sA};
        int C, threads;
        if (lup::panel_shape(n - off, 1, C, threads))
            return lup::launch_panel<lup::F64, TS, 1>(s, n, off, w, mat, ipiv, sP, info, batch, C,
                                                      threads);
        if (lup::panel_shape(n - off, 2, C, threads))
            return lup::launch_panel<lup::F64, TS / 2, 2>(s, n, off, w, mat, ipiv, sP, info,
                                                          batch, C, threads);
        if (lup::panel_shape(n - off, 4, C, threads))
            return lup::launch_panel<lup::F64, TS / 4, 4>(s, n, off, w, mat, ipiv, sP, info,
                                                          batch, C, threads);
        panel_kernel<<<batch, PANEL_THREADS, 0, s>>>(n, off, w, A, lda, sA, ipiv, sP, info);
        MNPB_LAUNCH_CHECK("panel_kernel");
        return MNPB_OK;
    }
    const int w1 = w > TS ? split_point(w) : leaf_width(n - off);
    MNPB_TRY(rgetrf(s, n, off, w1, batch, A, lda, sA, ipiv, sP, info));
    MNPB_TRY(laswp_range(s, A, lda, sA, off + w1, off + w, ipiv, sP, off, off + w1, batch));
    cd *A11 = A + off + (int64_t)off * lda;
    cd *A12 = A + off + (int64_t)(off + w1) * lda;
    MNPB_TRY(trsm_llu(s, w1, w - w1, batch, A11, lda, sA, A12, lda, sA));
    MNPB_TRY(zgemm(s, n - off - w1, w - w1, w1, batch, cmk(-1, 0), A11 + w1, lda, sA, A12, lda,
                   sA, cmk(1, 0), A12 + w1, lda, sA));
    MNPB_TRY(rgetrf(s, n, off + w1, w - w1, batch, A, lda, sA, ipiv, sP, info));
    return laswp_range(s, A, lda, sA, off, off + w1, ipiv, sP, off + w1, off + w, batch);
}

int getrf(cudaStream_t s, int n, int batch, cd *A, int64_t lda, int64_t sA, int32_t *ipiv,
          int64_t sP, int32_t *info) {
    return rgetrf(s, n, 0, n, batch, A, lda, sA, ipiv, sP, info);
}

int getrs(cudaStream_t s, int n, int nrhs, int batch, const cd *LU, int64_t lda, int64_t sA,
          const int32_t *ipiv, int64_t sP, cd *B, int64_t ldb, int64_t sB) {
    MNPB_TRY(laswp(s, B, ldb, sB, nrhs, 0, 0, ipiv, sP, 0, n, true, batch));
    MNPB_TRY(trsm_llu(s, n, nrhs, batch, LU, lda, sA, B, ldb, sB));
    return trsm_lun(s, n, nrhs, batch, LU, lda, sA, B, ldb, sB);
}

// X A = B in place on B (m x n), A = P^T L U from getrf.
int right_solve(cudaStream_t s, int n, int m, int batch, const cd *LU, int64_t lda, int64_t sA,
                const int32_t *ipiv, int64_t sP, cd *B, int64_t ldb, int64_t sB) {
    MNPB_TRY(trsm_run(s, n, m, batch, LU, lda, sA, B, ldb, sB));
    MNPB_TRY(trsm_rlu(s, n, m, batch, LU, lda, sA, B, ldb, sB));
    dim3 grid(ceil_div(m, 128), batch);
    ProfScope ps(s, PC_SWAP, 0.0);
    colswp_kernel<<<grid, 128, 0, s>>>(B, ldb, sB, m, ipiv, sP, n);
    MNPB_LAUNCH_CHECK("colswp_kernel");
    return MNPB_OK;
}

int set_identity(cudaStream_t s, int n, int batch, cd *W, int64_t ldw, int64_t sW) {
    dim3 grid(ceil_div(n, 128), n, batch);
    set_identity_kernel<<<grid, 128, 0, s>>>(W, ldw, sW, n);
    MNPB_LAUNCH_CHECK("set_identity_kernel");
    return MNPB_OK;
}

}  // namespace mnpb

using namespace mnpb;

extern "C" int mnpb_zgemm(void *stream, int64_t m, int64_t n, int64_t k, int64_t batch,
                          double alpha_re, double alpha_im, const double *A, int64_t lda,
                          int64_t sA, const double *B, int64_t ldb, int64_t sB, double beta_re,
                          double beta_im, double *C, int64_t ldc, int64_t sC) {
    clear_error();
    MNPB_REQUIRE(m >= 0 && n >= 0 && k >= 0 && batch >= 0 && batch < 65536,
                 "zgemm: bad sizes");
    MNPB_REQUIRE(C && (k == 0 || (A && B)), "zgemm: null pointer");
    return zgemm(as_stream(stream), (int)m, (int)n, (int)k, (int)batch, cmk(alpha_re, alpha_im),
                 (const cd *)A, lda, sA, (const cd *)B, ldb, sB, cmk(beta_re, beta_im), (cd *)C,
                 ldc, sC);
}

extern "C" int mnpb_getrf_f64(void *stream, int64_t n, int64_t batch, double *A, int64_t ld,
                              int64_t stride, int32_t *piv, int64_t pstride, int32_t *info) {
    clear_error();
    MNPB_REQUIRE(n > 0 && batch > 0 && ld >= n && batch < 65536, "getrf: bad sizes");
    MNPB_REQUIRE(A && piv, "getrf: null pointer");
    return getrf(as_stream(stream), (int)n, (int)batch, (cd *)A, ld, stride, piv, pstride, info);
}

extern "C" int mnpb_getrs_f64(void *stream, int64_t n, int64_t batch, int64_t nrhs,
                              const double *LU, int64_t ld, int64_t stride, const int32_t *piv,
                              int64_t pstride, double *B, int64_t ldb, int64_t bstride) {
    clear_error();
    MNPB_REQUIRE(n > 0 && batch > 0 && nrhs > 0 && ld >= n && ldb >= n, "getrs: bad sizes");
    MNPB_REQUIRE(LU && piv && B, "getrs: null pointer");
    return getrs(as_stream(stream), (int)n, (int)nrhs, (int)batch, (const cd *)LU, ld, stride,
                 piv, pstride, (cd *)B, ldb, bstride);
}
