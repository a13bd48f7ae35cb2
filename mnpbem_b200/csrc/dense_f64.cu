// Batched dense complex linear algebra in FP64 (interleaved complex128,
// column-major): GEMM, LU with partial pivoting, triangular solves.
//
// Every routine works on `batch` independent matrices `stride` elements
// apart, so a whole spectrum of wavelengths goes through each launch
// together: per-matrix latency (the column-by-column panel) is hidden by the
// other matrices in the batch.
#include "common.cuh"
#include "dense_f64.cuh"
#include "fork.cuh"
#include "lu_panel.cuh"
#include "interchange.cuh"
#include "trsv_cluster.cuh"
#include "skinny.cuh"

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

template <int BM, int BN>
__global__ void __launch_bounds__(GTHREADS) zgemm_kernel(int m, int n, int k, cd alpha,
                                                         const cd *A, int64_t lda, int64_t sA,
                                                         const cd *B, int64_t ldb, int64_t sB,
                                                         cd beta, cd *C, int64_t ldc,
                                                         int64_t sC) {
    grid_wait();
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
constexpr int TS = 32;         // columns of an LU leaf

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

// Row interchanges of whole columns (all n steps) composed once per CTA, then
// column by column through shared memory: reads and writes are coalesced and
// independent, where laswp_kernel walks n dependent steps per column.
__global__ void __launch_bounds__(512) permute_rows_kernel(cd *A, int64_t lda, int64_t sA, int n,
                                                           int ncols, const int32_t *ipiv,
                                                           int64_t sP) {
    extern __shared__ __align__(16) int perm_sm[];
    cd *col = (cd *)perm_sm;
    int *w = perm_sm + 4 * n;
    const int64_t b = blockIdx.y;
    trc::compose(w, ipiv + b * sP, n);
    for (int j = blockIdx.x; j < ncols; j += gridDim.x) {
        cd *a = A + b * sA + (int64_t)j * lda;
        for (int i = threadIdx.x; i < n; i += blockDim.x) col[i] = a[i];
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) a[i] = col[w[i]];
        __syncthreads();
    }
}

// X <- X P: the interchanges' columns c and ipiv[c], c from n - 1 down to 0, on
// RS rows per CTA through shared memory.  The reverse order undoes the forward
// gather (row c <- src[c]), so column c goes to column src[c].
__global__ void __launch_bounds__(256) permute_cols_kernel(cd *X, int64_t ldx, int64_t sX, int m,
                                                           const int32_t *ipiv, int64_t sP,
                                                           int n, int RS) {
    extern __shared__ __align__(16) int perm_sm[];
    cd *buf = (cd *)perm_sm;                   // [n][RS]
    int *w = perm_sm + 4 * (int64_t)n * RS;
    const int64_t b = blockIdx.y;
    const int r0 = blockIdx.x * RS, nr = min(RS, m - r0);
    cd *x = X + b * sX + r0;
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(buf);
    for (int e = threadIdx.x; e < n * RS; e += blockDim.x) {
        const int r = e % RS, c = e / RS;
        cp16(d + e * 16, r < nr ? x + (int64_t)c * ldx + r : x, r < nr);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    trc::compose(w, ipiv + b * sP, n);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int e = threadIdx.x; e < n * RS; e += blockDim.x) {
        const int r = e % RS, c = e / RS;
        if (r < nr && w[c] != c) x[(int64_t)w[c] * ldx + r] = buf[e];
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

// ---------------------------------------------------------------------------
// Triangular solves on a diagonal block of up to SN = 128 rows, one CTA per
// strip of SV right-hand sides (32, or 16 while those strips are too few to
// give every SM one) held in shared memory.
// mode 0: left lower unit     L x = b   (vectors: columns of B)
// mode 1: left upper non-unit U x = b   (vectors: columns of B)
// mode 2: right upper non-unit x U = b  (vectors: rows of B)
// mode 3: right lower unit     x L = b  (vectors: rows of B)
// All four are one forward substitution with the triangle in the order of the
// solve: M(l, k) = op(T)(phys(l), phys(k)), op the transpose for the right
// solves, phys reversed for modes 1 and 3.  Per 32-row block: four lanes per
// vector (eight for 16) substitute the diagonal block, each with its own rows, then
// the blocks below subtract M(I, J) x_J on the tensor path, warp by warp a
// 16 x 16 piece; M's blocks stream through two cp.async buffers.  One launch
// replaces the 32-row leaves and the products between them (7 launches for
// 128 rows); bound by the chain of substitutions at one strip per SM, by the
// FP64 pipe beyond.  Measured with 32-row leaves -> strips: 284 right-hand
// sides of a 284 x 284 LU (2 matrices) 612 -> 257 us, 1365 of 1365 3.54 ->
// 1.90 ms, 2884 of 2884 13.2 -> 9.3 ms.
// Mode 0 can apply the row interchanges of an LU panel to its columns first
// (the panel's rows are the block's), which saves their launch and one pass
// over the block's rows; strips of columns < jsolve are only interchanged.
// ---------------------------------------------------------------------------
constexpr int SN = 128, STHREADS = 128;
constexpr int MST = 34;        // M's stride in shared memory (bank groups, see zgemm_kernel)

struct StripArgs {
    int mode, kb;              // triangle rows
    const cd *T;
    int64_t ldt, sT;
    cd *B;                     // modes 0, 1: kb x nvec; modes 2, 3: nvec x kb
    int64_t ldb, sB;
    int nvec;
    // interchanges (mode 0): pivots of the block's rows, absolute from `base`;
    // vectors [0, jsolve) are interchanged only; [skip0, skip1) are left out
    const int32_t *ipiv;
    int64_t sP;
    int base, jsolve, skip0, skip1;
};

template <int SV>
__global__ void __launch_bounds__(STHREADS) trsm_strip_kernel(StripArgs g) {
    grid_wait();
    constexpr int SST = SV + 2;                // X's stride
    constexpr int LV = STHREADS / SV, RL = 32 / LV;   // lanes per vector, rows per lane
    constexpr int NJ = SV / 16;                // 8-column fragments per warp
    extern __shared__ __align__(16) cd strip_sm[];
    cd *X = strip_sm;                          // [SN][SST], rows in solve order
    cd *M = strip_sm + SN * SST;               // [2][32][MST]: M(l, k) at [k][l]
    __shared__ cd dinv[32];
    __shared__ swp::Swaps sw;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int kb = g.kb, mode = g.mode;
    const bool fwd = mode == 0 || mode == 2, left = mode < 2, unit = mode == 0 || mode == 3;
    const int64_t b = blockIdx.y;
    const cd *T = g.T + b * g.sT;
    cd *B = g.B + b * g.sB;
    int v0 = blockIdx.x * SV;
    int vend = g.nvec;
    bool solve = true;
    if (g.ipiv) {
        // strips cover [0, skip0), then [skip1, nvec)
        const int ns = (g.skip0 + SV - 1) / SV;
        if ((int)blockIdx.x < ns) vend = g.skip0;
        else v0 = g.skip1 + (blockIdx.x - ns) * SV;
        solve = v0 >= g.jsolve;
    }
    const int nv = min(SV, vend - v0);
    auto phys = [&](int l) { return fwd ? l : kb - 1 - l; };
    const int nblk = (kb + 31) / 32;
    // M block (I, J) into buffer q
    auto stage = [&](int I, int J, int q) {
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(M + q * 32 * MST);
#pragma unroll
        for (int e = tid; e < 1024; e += STHREADS) {
            // consecutive threads along the contiguous direction of T
            const int u = e & 31, w = e >> 5;
            const int l = left ? u : w, k = left ? w : u;
            const int gl = 32 * I + l, gk = 32 * J + k;
            const bool ok = gl < kb && gk < kb;
            const int64_t o = !ok ? 0
                              : left ? (int64_t)phys(gk) * g.ldt + phys(gl)
                                     : (int64_t)phys(gl) * g.ldt + phys(gk);
            cp16(d + (k * MST + l) * 16, T + o, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const uint32_t xs = (uint32_t)__cvta_generic_to_shared(X);
    if (solve) stage(0, 0, 0);
    if (g.ipiv) {
        const int32_t *pv = g.ipiv + b * g.sP;
        swp::compose(sw, pv, g.base, kb);
        // gather the block's rows, and the rows below that the steps reached;
        // rows past kb and vectors past nv are zero
        for (int e = tid; e < nblk * 32 * SV; e += STHREADS) {
            const int c = e % (nblk * 32), v = e / (nblk * 32);
            const bool ok = c < kb && v < nv;
            cp16(xs + (c * SST + v) * 16, ok ? B + (int64_t)(v0 + v) * g.ldb + sw.out[c] : B, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        cd t[SN * SV / STHREADS];
#pragma unroll
        for (int q = 0; q < SN * SV / STHREADS; ++q) {
            const int e = tid + q * STHREADS, c = e % SN, v = e / SN;
            t[q] = (v < nv && c < kb && sw.tail[c] >= 0)
                       ? B[(int64_t)(v0 + v) * g.ldb + sw.tail[c]]
                       : cmk(0.0, 0.0);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                       // every row read: B may be written
#pragma unroll
        for (int q = 0; q < SN * SV / STHREADS; ++q) {
            const int e = tid + q * STHREADS, c = e % SN, v = e / SN;
            if (v < nv && c < kb && sw.tail[c] >= 0)
                B[(int64_t)(v0 + v) * g.ldb + sw.p[c]] = t[q];
        }
        if (!solve) {
            for (int e = tid; e < kb * nv; e += STHREADS) {
                const int c = e % kb, v = e / kb;
                B[(int64_t)(v0 + v) * g.ldb + c] = X[c * SST + v];
            }
            return;
        }
    } else {
        for (int e = tid; e < nblk * 32 * SV; e += STHREADS) {
            const int l = left ? e % (nblk * 32) : e / SV, v = left ? e / (nblk * 32) : e % SV;
            const bool ok = l < kb && v < nv;
            const cd *src = !ok    ? B
                            : left ? B + (int64_t)(v0 + v) * g.ldb + phys(l)
                                   : B + (int64_t)phys(l) * g.ldb + v0 + v;
            cp16(xs + (l * SST + v) * 16, src, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int q = 0;
    for (int J = 0; J < nblk; ++J) {
        for (int I = J; I < nblk; ++I) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();                   // block (I, J) staged; X rows of the last step
            const cd *m = M + q * 32 * MST;
            q ^= 1;
            // the other buffer was last read before this barrier
            if (I + 1 < nblk) stage(I + 1, J, q);
            else if (J + 1 < nblk) stage(J + 1, J + 1, q);
            if (I == J) {
                if (!unit && tid < 32)
                    dinv[tid] = 32 * J + tid < kb ? crcp(m[tid * MST + tid]) : cmk(0.0, 0.0);
                if (!unit) __syncthreads();
                const int v = wid * (32 / LV) + lane / LV, r = lane % LV;
                cd y[RL];
#pragma unroll
                for (int i = 0; i < RL; ++i) y[i] = X[(32 * J + LV * i + r) * SST + v];
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    const int ci = c / LV, cr = c % LV;
                    if (!unit && r == cr) y[ci] = cmul(y[ci], dinv[c]);
                    const int src = (lane & ~(LV - 1)) | cr;
                    const cd x = cmk(__shfl_sync(0xffffffffu, y[ci].x, src),
                                     __shfl_sync(0xffffffffu, y[ci].y, src));
                    if (r > cr) y[ci] = cfms(m[c * MST + LV * ci + r], x, y[ci]);
#pragma unroll
                    for (int i = ci + 1; i < RL; ++i)
                        y[i] = cfms(m[c * MST + LV * i + r], x, y[i]);
                }
#pragma unroll
                for (int i = 0; i < RL; ++i) X[(32 * J + LV * i + r) * SST + v] = y[i];
            } else {
                const int gr = lane >> 2, t = lane & 3;
                const int rl = (wid & 1) * 16, cv = (wid >> 1) * 8 * NJ;
                double re[NJ][4], im[NJ][4];
                cd *xo = X + (32 * I + rl) * SST + cv;
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const cd w = xo[(gr + 8 * (e >> 1)) * SST + 8 * j + 2 * t + (e & 1)];
                        re[j][e] = w.x;
                        im[j][e] = w.y;
                    }
#pragma unroll
                for (int ks = 0; ks < 32; ks += 4) {
                    const cd a0 = m[(ks + t) * MST + rl + gr], a1 = m[(ks + t) * MST + rl + gr + 8];
#pragma unroll
                    for (int j = 0; j < NJ; ++j) {
                        const cd x = X[(32 * J + ks + t) * SST + cv + 8 * j + gr];
                        mma_f64(re[j], -a0.x, -a1.x, x.x);
                        mma_f64(im[j], -a0.x, -a1.x, x.y);
                        mma_f64(re[j], a0.y, a1.y, x.y);
                        mma_f64(im[j], -a0.y, -a1.y, x.x);
                    }
                }
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        xo[(gr + 8 * (e >> 1)) * SST + 8 * j + 2 * t + (e & 1)] =
                            cmk(re[j][e], im[j][e]);
            }
        }
    }
    __syncthreads();
    for (int e = tid; e < kb * nv; e += STHREADS) {
        const int c = left ? e % kb : e / nv, v = left ? e / kb : e % nv;
        const cd x = X[(fwd ? c : kb - 1 - c) * SST + v];
        if (left) B[(int64_t)(v0 + v) * g.ldb + c] = x;
        else B[(int64_t)c * g.ldb + v0 + v] = x;
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
    return launch_chained("zgemm_kernel", zgemm_kernel<BM, BN>, grid, dim3(GTHREADS), smem, s, 1, m,
                          n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC);
}

int zgemm(cudaStream_t s, int m, int n, int k, int batch, cd alpha, const cd *A, int64_t lda,
          int64_t sA, const cd *B, int64_t ldb, int64_t sB, cd beta, cd *C, int64_t ldc,
          int64_t sC) {
    if (m <= 0 || n <= 0 || batch <= 0) return MNPB_OK;
    ProfScope ps(s, PC_ZGEMM, 8.0 * m * n * (double)(k > 0 ? k : 0) * batch);
    // C = beta C for k <= 0
    // 64 x 64 tiles once two CTAs per SM have one; smaller tiles until then, so that
    // small updates spread over the SMs (2800 x 32 x 32, 2 matrices: 20.7 -> 14.6 us).
    // Up to 16 columns go to the few-vector kernels (2884 x 4 x 2884, which a
    // 64-column tile padded 16-fold: 795 us, on 32 x 32 tiles 157, there 40)
    const int kk = k > 0 ? k : 0;
    if (n <= 16 && kk > 0)
        return skn::run<skn::F64>(s, m, n, kk, batch, alpha, {(cd *)A, lda, sA},
                                  {(cd *)B, ldb, sB}, beta, {C, ldc, sC});
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

template <int SV>
static int launch_strip_sv(cudaStream_t s, const StripArgs &g, int strips, int batch) {
    if (strips <= 0) return MNPB_OK;
    const int smem = (SN * (SV + 2) + 2 * 32 * MST) * (int)sizeof(cd);
    MNPB_TRY(smem_opt_in(trsm_strip_kernel<SV>, smem, "trsm_strip_kernel"));
    ProfScope ps(s, PC_TRSM, 4.0 * g.kb * g.kb * (double)g.nvec * batch);
    return launch_chained("trsm_strip_kernel", trsm_strip_kernel<SV>, dim3(strips, batch),
                          dim3(STHREADS), smem, s, 1, g);
}

// vectors [0, g.skip0) and [g.skip1, g.nvec)
static int launch_strip(cudaStream_t s, const StripArgs &g, int batch) {
    if (g.kb <= 0) return MNPB_OK;
    // 16 vectors per CTA while strips of 32 would leave SMs idle: half the work
    // per strip (one matrix of 284: LU 0.63 -> 0.56 ms, 2884 11.2 -> 10.4 ms)
    auto strips = [&](int sv) { return ceil_div(g.skip0, sv) + ceil_div(g.nvec - g.skip1, sv); };
    if ((int64_t)strips(32) * batch <= device_sms())
        return launch_strip_sv<16>(s, g, strips(16), batch);
    return launch_strip_sv<32>(s, g, strips(32), batch);
}

static int trsm_strip(cudaStream_t s, int mode, int kb, const cd *T, int64_t ldt, int64_t sT,
                      cd *B, int64_t ldb, int64_t sB, int nvec, int batch) {
    StripArgs g{mode, kb, T, ldt, sT, B, ldb, sB, nvec, nullptr, 0, 0, 0, 0, 0};
    return launch_strip(s, g, batch);
}

static int split_point(int n) {
    int h = n / 2;
    h = (h / SN) * SN;
    return h < SN ? SN : h;
}

// L X = B, L unit lower n x n; B n x m.
int trsm_llu(cudaStream_t s, int n, int m, int batch, const cd *L, int64_t ldl, int64_t sL,
             cd *B, int64_t ldb, int64_t sB) {
    if (n <= SN) return trsm_strip(s, 0, n, L, ldl, sL, B, ldb, sB, m, batch);
    int n1 = split_point(n);
    MNPB_TRY(trsm_llu(s, n1, m, batch, L, ldl, sL, B, ldb, sB));
    MNPB_TRY(zgemm(s, n - n1, m, n1, batch, cmk(-1, 0), L + n1, ldl, sL, B, ldb, sB, cmk(1, 0),
                   B + n1, ldb, sB));
    return trsm_llu(s, n - n1, m, batch, L + n1 + (int64_t)n1 * ldl, ldl, sL, B + n1, ldb, sB);
}

// U X = B, U upper non-unit.
int trsm_lun(cudaStream_t s, int n, int m, int batch, const cd *U, int64_t ldu, int64_t sU,
             cd *B, int64_t ldb, int64_t sB) {
    if (n <= SN) return trsm_strip(s, 1, n, U, ldu, sU, B, ldb, sB, m, batch);
    int n1 = split_point(n);
    MNPB_TRY(trsm_lun(s, n - n1, m, batch, U + n1 + (int64_t)n1 * ldu, ldu, sU, B + n1, ldb, sB));
    MNPB_TRY(zgemm(s, n1, m, n - n1, batch, cmk(-1, 0), U + (int64_t)n1 * ldu, ldu, sU, B + n1,
                   ldb, sB, cmk(1, 0), B, ldb, sB));
    return trsm_lun(s, n1, m, batch, U, ldu, sU, B, ldb, sB);
}

// X U = B, U upper non-unit n x n; X, B m x n.
int trsm_run(cudaStream_t s, int n, int m, int batch, const cd *U, int64_t ldu, int64_t sU,
             cd *B, int64_t ldb, int64_t sB) {
    if (n <= SN) return trsm_strip(s, 2, n, U, ldu, sU, B, ldb, sB, m, batch);
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
    if (n <= SN) return trsm_strip(s, 3, n, L, ldl, sL, B, ldb, sB, m, batch);
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
    ProfScope ps(s, PC_SWAP, 0.0);
    dim3 grid(ceil_div(ncols, 128), batch);
    laswp_kernel<<<grid, 128, 0, s>>>(A, lda, sA, 0, ncols, jskip0, jskip1, ipiv, sP, c0, c1,
                                      forward ? 1 : 0);
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

// One LU leaf: columns [off, off + w) over rows [off, n).
static int leaf(cudaStream_t s, int n, int off, int w, int batch, cd *A, int64_t lda, int64_t sA,
                int32_t *ipiv, int64_t sP, int32_t *info) {
    ProfScope ps(s, PC_PANEL, 8.0 * w * w * (double)(n - off) * batch / 2);
    const lup::F64::Mat mat{A, lda, sA};
    int C, threads;
    if (lup::panel_shape(n - off, 1, C, threads))
        return lup::launch_panel<lup::F64, TS, 1>(s, n, off, w, mat, ipiv, sP, info, batch, C,
                                                  threads);
    if (lup::panel_shape(n - off, 2, C, threads))
        return lup::launch_panel<lup::F64, TS / 2, 2>(s, n, off, w, mat, ipiv, sP, info, batch,
                                                      C, threads);
    if (lup::panel_shape(n - off, 4, C, threads))
        return lup::launch_panel<lup::F64, TS / 4, 4>(s, n, off, w, mat, ipiv, sP, info, batch,
                                                      C, threads);
    panel_kernel<<<batch, PANEL_THREADS, 0, s>>>(n, off, w, A, lda, sA, ipiv, sP, info);
    MNPB_LAUNCH_CHECK("panel_kernel");
    return MNPB_OK;
}

// Interchanges of the pivots of columns [off, off + w) on the columns
// [j0, off) and [r0, j1), r0 >= off + w, and L^-1 on the rows [off, off + w) of
// the latter.
static int swap_solve(cudaStream_t s, int off, int w, int j0, int r0, int j1, int batch, cd *A,
                      int64_t lda, int64_t sA, const int32_t *ipiv, int64_t sP) {
    if (j0 >= off && r0 >= j1) return MNPB_OK;
    const int skip0 = off - j0, skip1 = r0 - j0, nvec = j1 - j0;
    StripArgs g{0,    w,         A + off + (int64_t)off * lda, lda, sA,
                A + off + (int64_t)j0 * lda, lda, sA, nvec,
                ipiv + off, sP, off, skip1, skip0, skip1};
    return launch_strip(s, g, batch);
}

// The columns [j0, j1) of a block, leaf by leaf.
static int block_getrf(cudaStream_t s, int n, int j0, int j1, int batch, cd *A, int64_t lda,
                       int64_t sA, int32_t *ipiv, int64_t sP, int32_t *info) {
    for (int off = j0; off < j1;) {
        const int w = min(leaf_width(n - off), j1 - off), c1 = off + w;
        MNPB_TRY(leaf(s, n, off, w, batch, A, lda, sA, ipiv, sP, info));
        MNPB_TRY(swap_solve(s, off, w, j0, c1, j1, batch, A, lda, sA, ipiv, sP));
        MNPB_TRY(zgemm(s, n - c1, j1 - c1, w, batch, cmk(-1, 0), A + c1 + (int64_t)off * lda,
                       lda, sA, A + off + (int64_t)c1 * lda, lda, sA, cmk(1, 0),
                       A + c1 + (int64_t)c1 * lda, lda, sA));
        off = c1;
    }
    return MNPB_OK;
}

// A block's interchanges on the columns [0, j0) (left) and [r0, r1), and its
// update of the latter.
static int block_update(cudaStream_t s, int n, int j0, int j1, bool left, int r0, int r1,
                        int batch, cd *A, int64_t lda, int64_t sA, const int32_t *ipiv,
                        int64_t sP) {
    MNPB_TRY(swap_solve(s, j0, j1 - j0, left ? 0 : j0, r0, r1, batch, A, lda, sA, ipiv, sP));
    return zgemm(s, n - j1, r1 - r0, j1 - j0, batch, cmk(-1, 0), A + j1 + (int64_t)j0 * lda, lda,
                 sA, A + j0 + (int64_t)r0 * lda, lda, sA, cmk(1, 0), A + j1 + (int64_t)r0 * lda,
                 lda, sA);
}

// Right-looking LU in blocks of SN columns; inside a block, leaf by leaf.  A
// block costs its leaves, two launches per leaf inside the block, and two for
// the rest of the matrix, where halving the columns recursively took some 40
// per 128 columns: at one matrix the launches outnumber what they do.  The
// update's depth of 128 already runs at the GEMM's full rate.  One matrix of
// 2884: 17.6 -> 11.2 ms, 1365 6.1 -> 4.0 ms, 284 0.79 -> 0.63 ms (with the
// panels' reductions by redux.sync); 41 of 1148 14.5 -> 11.0 ms.
//
// While one wave holds the panels of all matrices, the chain panel, update of the
// next block, panel runs on a stream of its own (high priority: its launches need
// whole SMs) and the caller's stream has the updates of the columns beyond.  The
// chain at block k + 1 waits for the bulk of block k before it reads the columns
// of block k + 2, the bulk of block k for the panels of block k.  One stream ->
// two: 2884 x 1 / 2 / 16 10.2 / 12.8 / 47.9 -> 8.9 / 10.6 / 45.2 ms, 2044 x 4 8.8 ->
// 7.4, 1148 x 41 9.8 -> 9.1, 700 x 20 2.49 -> 2.21, 1365 x 1 3.68 -> 3.61; too little
// to overlap below (1148 x 1 2.89 -> 2.95, 700 x 1 1.62 -> 1.66, 500 x 3 the same).
// Where no second stream is to be had (more calls at once than the pool has, or the
// caller captures) the columns are cut the same way on one: a product's kernel and
// its order of summation follow from its columns, and the factors must not depend on
// what other threads do.
int getrf(cudaStream_t s, int n, int batch, cd *A, int64_t lda, int64_t sA, int32_t *ipiv,
          int64_t sP, int32_t *info) {
    int C, threads;
    if (n > 2 * SN && (int64_t)n * batch > 1280 && lup::panel_shape(n, 1, C, threads) &&
        (int64_t)C * batch <= device_sms()) {
        ForkLease lease(s);
        const Fork *f = lease.get();
        const cudaStream_t p = f ? f->p : s;      // no second stream: the same pieces in turn
        auto chain = [&]() -> int {
            for (int j0 = 0; j0 < n; j0 += SN) {
                const int j1 = min(n, j0 + SN), j2 = min(n, j1 + SN);
                MNPB_TRY(block_getrf(p, n, j0, j1, batch, A, lda, sA, ipiv, sP, info));
                if (f) {
                    // es: the bulk of the block before, which updated [j1, j2)
                    if (j0 > 0) MNPB_TRY(stream_after(p, s, f->es));
                    MNPB_TRY(stream_after(s, p, f->ep));
                }
                MNPB_TRY(block_update(p, n, j0, j1, false, j1, j2, batch, A, lda, sA, ipiv, sP));
                MNPB_TRY(block_update(s, n, j0, j1, true, j2, n, batch, A, lda, sA, ipiv, sP));
            }
            return MNPB_OK;
        };
        if (!f) return chain();
        MNPB_TRY(stream_after(p, s, f->es));
        const int rc = chain();
        const int rj = stream_after(s, p, f->ep);   // also after an error
        return rc != MNPB_OK ? rc : rj;
    }
    for (int j0 = 0; j0 < n; j0 += SN) {
        const int j1 = min(n, j0 + SN);
        MNPB_TRY(block_getrf(s, n, j0, j1, batch, A, lda, sA, ipiv, sP, info));
        MNPB_TRY(block_update(s, n, j0, j1, true, j1, n, batch, A, lda, sA, ipiv, sP));
    }
    return MNPB_OK;
}

// All n interchanges of an LU on the rows of B.
static int permute_rows(cudaStream_t s, cd *B, int64_t ldb, int64_t sB, int n, int ncols,
                        const int32_t *ipiv, int64_t sP, int batch) {
    const int64_t smem = 32 * (int64_t)n;          // a column and 4 n ints
    if (smem > 200 * 1024)
        return laswp(s, B, ldb, sB, ncols, 0, 0, ipiv, sP, 0, n, true, batch);
    MNPB_TRY(smem_opt_in(permute_rows_kernel, 200 * 1024, "permute_rows_kernel"));
    ProfScope ps(s, PC_SWAP, 0.0);
    const int per = max(1, 4 * device_sms() / batch);
    permute_rows_kernel<<<dim3(min(ncols, per), batch), 512, (size_t)smem, s>>>(B, ldb, sB, n,
                                                                              ncols, ipiv, sP);
    MNPB_LAUNCH_CHECK("permute_rows_kernel");
    return MNPB_OK;
}

// Forward then backward solve of up to 16 right-hand sides, a cluster per
// matrix and NC columns; the interchanges ride along with the forward solve.
template <int NC>
static int getrs_few(cudaStream_t s, int n, int nrhs, const trc::Groups &gr, const cd *LU,
                     int64_t lda, int64_t sA, const int32_t *ipiv, int64_t sP, cd *B, int64_t ldb,
                     int64_t sB, int C) {
    const trc::F64::Mat A{(cd *)LU, lda, sA}, X{B, ldb, sB};
    const bool ride = trc::Smem<trc::F64, NC>::composes(n);
    if (!ride)
        for (int g = 0; g < gr.groups; ++g)
            MNPB_TRY(laswp(s, B + g * gr.X, ldb, sB, nrhs, 0, 0, ipiv + g * gr.P, sP, 0, n, true,
                           gr.per));
    ProfScope ps(s, PC_TRSV, 16.0 * (double)n * n * gr.per * gr.groups);   // both triangles
    MNPB_TRY((trc::launch_trsv<trc::F64, NC>(s, true, true, n, nrhs, gr, A, nullptr, X,
                                             ride ? ipiv : nullptr, sP, C)));
    return trc::launch_trsv<trc::F64, NC>(s, false, false, n, nrhs, gr, A, nullptr, X, nullptr, 0,
                                          C);
}

// Clusters of the few-column solves of `batch` matrices: NC = 1 or 4 columns
// each, C CTAs; false if the columns are too many or do not fit.
static bool few_shape(int n, int nrhs, int64_t batch, int &NC, int &C) {
    if (nrhs > 16) return false;
    NC = nrhs == 1 ? 1 : 4;
    C = NC == 1 ? trc::cluster_size<trc::F64, 1>(n, batch)
                : trc::cluster_size<trc::F64, 4>(n, batch * ceil_div(nrhs, 4));
    return C > 0;
}

int getrs_pair(cudaStream_t s, int n, int nrhs, int batch, const cd *LU1, const cd *LU2,
               int64_t lda, int64_t sA, const int32_t *piv1, const int32_t *piv2, int64_t sP,
               cd *B1, cd *B2, int64_t ldb, int64_t sB) {
    int NC, C;
    if (!few_shape(n, nrhs, 2 * (int64_t)batch, NC, C)) {
        MNPB_TRY(getrs(s, n, nrhs, batch, LU1, lda, sA, piv1, sP, B1, ldb, sB));
        return getrs(s, n, nrhs, batch, LU2, lda, sA, piv2, sP, B2, ldb, sB);
    }
    const trc::Groups gr{batch, 2, LU2 - LU1, 0, B2 - B1, piv2 - piv1};
    return NC == 1 ? getrs_few<1>(s, n, nrhs, gr, LU1, lda, sA, piv1, sP, B1, ldb, sB, C)
                   : getrs_few<4>(s, n, nrhs, gr, LU1, lda, sA, piv1, sP, B1, ldb, sB, C);
}

int getrs(cudaStream_t s, int n, int nrhs, int batch, const cd *LU, int64_t lda, int64_t sA,
          const int32_t *ipiv, int64_t sP, cd *B, int64_t ldb, int64_t sB) {
    int NC, C;
    if (few_shape(n, nrhs, batch, NC, C)) {
        const trc::Groups gr{batch, 1, 0, 0, 0, 0};
        return NC == 1 ? getrs_few<1>(s, n, nrhs, gr, LU, lda, sA, ipiv, sP, B, ldb, sB, C)
                       : getrs_few<4>(s, n, nrhs, gr, LU, lda, sA, ipiv, sP, B, ldb, sB, C);
    }
    MNPB_TRY(permute_rows(s, B, ldb, sB, n, nrhs, ipiv, sP, batch));
    MNPB_TRY(trsm_llu(s, n, nrhs, batch, LU, lda, sA, B, ldb, sB));
    return trsm_lun(s, n, nrhs, batch, LU, lda, sA, B, ldb, sB);
}

// Column interchanges X <- X P of an m x n block.
static int permute_cols(cudaStream_t s, cd *X, int64_t ldx, int64_t sX, int m, int n,
                        const int32_t *ipiv, int64_t sP, int batch) {
    ProfScope ps(s, PC_SWAP, 0.0);
    const int RS = (int)min((int64_t)8, 200 * 1024 / (16 * (int64_t)n) - 1);
    if (RS < 2) {
        dim3 grid(ceil_div(m, 128), batch);
        colswp_kernel<<<grid, 128, 0, s>>>(X, ldx, sX, m, ipiv, sP, n);
        MNPB_LAUNCH_CHECK("colswp_kernel");
        return MNPB_OK;
    }
    MNPB_TRY(smem_opt_in(permute_cols_kernel, 200 * 1024, "permute_cols_kernel"));
    permute_cols_kernel<<<dim3(ceil_div(m, RS), batch), 256, (size_t)16 * n * (RS + 1), s>>>(
        X, ldx, sX, m, ipiv, sP, n, RS);
    MNPB_LAUNCH_CHECK("permute_cols_kernel");
    return MNPB_OK;
}

// Whether the right-hand sides of a solve are cut in halves (in_halves, fork.cuh):
// the strips of one, bound by their chains, run beside the products of the other,
// bound by the FP64 pipe.  The four LUs, two right solves and one inverse of a
// wavelength, n x batch: 2884 x 1 55.7 -> 53.8 ms, 2044 x 1 29.9 -> 28.6, 284 x 41
// 4.29 -> 4.04, 700 x 16 14.2 -> 13.8; nothing to gain below (508 x 2 and 284 x 1 the
// same).
static bool worth_halves(int n, int m, int batch) {
    return n > 2 * SN && (int64_t)m * batch > 1024;
}

// X A = B in place on B (m x n), A = P^T L U from getrf.
int right_solve(cudaStream_t s, int n, int m, int batch, const cd *LU, int64_t lda, int64_t sA,
                const int32_t *ipiv, int64_t sP, cd *B, int64_t ldb, int64_t sB) {
    const bool cut = worth_halves(n, m, batch);
    MNPB_TRY(in_halves(s, m, cut, [&](cudaStream_t st, int i0, int i1) -> int {
        MNPB_TRY(trsm_run(st, n, i1 - i0, batch, LU, lda, sA, B + i0, ldb, sB));
        return trsm_rlu(st, n, i1 - i0, batch, LU, lda, sA, B + i0, ldb, sB);
    }));
    return permute_cols(s, B, ldb, sB, m, n, ipiv, sP, batch);
}

// X <- L^-1 for X = identity on entry: above the diagonal X stays zero, so
// X11 = L11^-1, X21 = -L22^-1 (L21 X11), X22 = L22^-1: a third of the
// operations of a solve against n full columns.
static int trsm_llu_eye(cudaStream_t s, int n, int batch, const cd *L, int64_t ldl, int64_t sL,
                        cd *X, int64_t ldx, int64_t sX) {
    if (n <= SN) return trsm_strip(s, 0, n, L, ldl, sL, X, ldx, sX, n, batch);
    const int n1 = split_point(n);
    const cd *L22 = L + n1 + (int64_t)n1 * ldl;
    MNPB_TRY(trsm_llu_eye(s, n1, batch, L, ldl, sL, X, ldx, sX));
    MNPB_TRY(zgemm(s, n - n1, n1, n1, batch, cmk(-1, 0), L + n1, ldl, sL, X, ldx, sX, cmk(0, 0),
                   X + n1, ldx, sX));
    MNPB_TRY(trsm_llu(s, n - n1, n1, batch, L22, ldl, sL, X + n1, ldx, sX));
    return trsm_llu_eye(s, n - n1, batch, L22, ldl, sL, X + n1 + (int64_t)n1 * ldx, ldx, sX);
}

// X <- A^-1 = U^-1 L^-1 P from getrf's factors.
int getri(cudaStream_t s, int n, int batch, const cd *LU, int64_t lda, int64_t sA,
          const int32_t *ipiv, int64_t sP, cd *X, int64_t ldx, int64_t sX) {
    MNPB_TRY(set_identity(s, n, batch, X, ldx, sX));
    MNPB_TRY(trsm_llu_eye(s, n, batch, LU, lda, sA, X, ldx, sX));
    const bool cut = worth_halves(n, n, batch);
    MNPB_TRY(in_halves(s, n, cut, [&](cudaStream_t st, int j0, int j1) -> int {
        return trsm_lun(st, n, j1 - j0, batch, LU, lda, sA, X + (int64_t)j0 * ldx, ldx, sX);
    }));
    return permute_cols(s, X, ldx, sX, n, n, ipiv, sP, batch);
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
