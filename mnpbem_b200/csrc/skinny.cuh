// Matrix times a few vectors, Y = alpha A X + beta Y, A m x k, X k x n with
// n <= NC columns.
//
// Bound by reading A once.  A CTA covers 64 R rows; four k lanes of 64 threads
// each take every fourth column, U loads in flight per thread; X is staged in
// shared memory in chunks.  Where the row blocks of all matrices are too few
// to fill the GPU, a cluster of C CTAs splits k and the partial sums meet in
// the first CTA's shared memory, added in a fixed order.
//
// Measured, FP64: 2884 x 4 x 2884, one matrix, 157 us on 32 x 32 GEMM tiles,
// 40 us here (3.3 TB/s); the refinement's residual, one 2884 matrix 190 -> 33
// us, 27 matrices 0.68 -> 0.61 ms (5.9 TB/s), 12 columns of mixed sizes in one
// pass over the matrix instead of two.  FP32, 4 columns: one 2884 matrix 460 ->
// 23 us; 12 columns of mixed sizes 0.42 -> 0.12 ms.
#pragma once
#include "lu_panel.cuh"

namespace mnpb {
namespace skn {

constexpr int LANES = 4, ROWT = 64, THREADS = LANES * ROWT, KT = 64, MAXC = 8;
// a chunk is a whole number of unrolled steps, so a step never leaves it

struct F64 {
    typedef cd V;
    typedef lup::F64::Mat Mat;
    static constexpr int R = 1, U = 8;
    static __device__ __forceinline__ V zero() { return cmk(0.0, 0.0); }
    static __device__ __forceinline__ V add(V a, V b) { return cadd(a, b); }
    static __device__ __forceinline__ V fma(V a, V b, V c) { return cfma(a, b, c); }
    static __device__ __forceinline__ V load(const Mat &m, int64_t b, int64_t row, int64_t col) {
        return __ldg(m.A + b * m.sA + col * m.lda + row);
    }
    static __device__ __forceinline__ void rows(const Mat &m, int64_t b, int64_t row, int64_t col,
                                                V (&a)[R]) {
        a[0] = load(m, b, row, col);
    }
    static __device__ __forceinline__ void push(uint32_t addr, V v) { lup::F64::push(addr, v); }
    typedef cd Scale;
    static __device__ __forceinline__ void out(const Mat &m, int64_t b, int64_t row, int64_t col,
                                               Scale al, V v, Scale be) {
        cd *y = m.A + b * m.sA + col * m.lda + row;
        const cd w = cmul(al, v);
        *y = (be.x == 0.0 && be.y == 0.0) ? w : cfma(be, *y, w);
    }
};

template <typename T, int NC>
__global__ void __launch_bounds__(THREADS) kernel(int m, int n, int k, typename T::Scale alpha,
                                                  typename T::Mat A, typename T::Mat X,
                                                  typename T::Scale beta, typename T::Mat Y,
                                                  int C) {
    typedef typename T::V V;
    constexpr int R = T::R, ROWS = ROWT * R;
    static_assert(KT % (LANES * T::U) == 0, "chunk");
    extern __shared__ __align__(16) unsigned char skn_sm[];
    V *xs = (V *)skn_sm;                       // [KT][NC]
    V *part = xs + KT * NC;                    // [LANES][ROWS][NC], then [C][ROWS][NC] in CTA 0
    const int tid = threadIdx.x, rt = tid % ROWT, kl = tid / ROWT;
    const int64_t b = blockIdx.y;
    const int me = C > 1 ? (int)lup::cluster_rank() : 0;
    const int row = (blockIdx.x / C) * ROWS + rt * R;
    // this CTA's columns of A, whole chunks
    const int nch = (k + KT - 1) / KT, per = (nch + C - 1) / C;
    const int kbeg = min(k, me * per * KT), kend = min(k, (me + 1) * per * KT);
    V acc[R][NC];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[r][c] = T::zero();
    for (int k0 = kbeg; k0 < kend; k0 += KT) {
        __syncthreads();
        for (int e = tid; e < KT * NC; e += THREADS) {
            const int kk = e % KT, c = e / KT;
            xs[kk * NC + c] = (k0 + kk < k && c < n) ? T::load(X, b, k0 + kk, c) : T::zero();
        }
        __syncthreads();
        if (row < m) {
            const int kn = min(KT, kend - k0);
#pragma unroll 1
            for (int q = kl; q < kn; q += LANES * T::U) {
                V a[T::U][R];
#pragma unroll
                for (int u = 0; u < T::U; ++u) {
                    if (q + u * LANES < kn) {
                        T::rows(A, b, row, k0 + q + u * LANES, a[u]);
                    } else {
#pragma unroll
                        for (int r = 0; r < R; ++r) a[u][r] = T::zero();
                    }
                }
#pragma unroll
                for (int u = 0; u < T::U; ++u) {
                    const V *x = xs + (q + u * LANES) * NC;   // zero from kn on
#pragma unroll
                    for (int c = 0; c < NC; ++c)
#pragma unroll
                        for (int r = 0; r < R; ++r) acc[r][c] = T::fma(a[u][r], x[c], acc[r][c]);
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < NC; ++c) part[(kl * ROWS + rt * R + r) * NC + c] = acc[r][c];
    __syncthreads();
    if (C > 1) {
        // sum the k lanes, send to CTA 0
        V s[(ROWS * NC + THREADS - 1) / THREADS];
#pragma unroll
        for (int u = 0; u < (ROWS * NC + THREADS - 1) / THREADS; ++u) {
            const int e = tid + u * THREADS;
            if (e < ROWS * NC) {
                s[u] = part[e];
#pragma unroll
                for (int q = 1; q < LANES; ++q) s[u] = T::add(s[u], part[q * ROWS * NC + e]);
            }
        }
        lup::cluster_sync();                   // every CTA has taken its lane sums: part is free
#pragma unroll
        for (int u = 0; u < (ROWS * NC + THREADS - 1) / THREADS; ++u) {
            const int e = tid + u * THREADS;
            if (e < ROWS * NC) T::push(lup::map_rank(part + me * ROWS * NC + e, 0), s[u]);
        }
        lup::cluster_sync();
        if (me != 0) return;
    }
    const int np = C > 1 ? C : LANES;
    for (int e = tid; e < ROWS * NC; e += THREADS) {
        const int r = e % ROWS, c = e / ROWS;
        const int gr = (blockIdx.x / C) * ROWS + r;
        if (gr < m && c < n) {
            V s = part[r * NC + c];
            for (int q = 1; q < np; ++q) s = T::add(s, part[(q * ROWS + r) * NC + c]);
            T::out(Y, b, gr, c, alpha, s, beta);
        }
    }
}

// CTAs along k: as many as bring the grid to three CTAs per SM.
inline int split(int m, int k, int rows, int batch) {
    const int64_t blocks = (int64_t)ceil_div(m, rows) * batch;
    int C = 1;
    while (C < MAXC && blocks * 2 * C <= 3 * device_sms() && 2 * C * KT <= k) C *= 2;
    return C;
}

template <typename T, int NC>
int launch(cudaStream_t s, int m, int n, int k, int batch, typename T::Scale alpha,
           typename T::Mat A, typename T::Mat X, typename T::Scale beta, typename T::Mat Y) {
    constexpr int ROWS = ROWT * T::R;
    const int C = split(m, k, ROWS, batch);
    const int np = C > LANES ? C : LANES;
    const int smem = (KT * NC + np * ROWS * NC) * (int)sizeof(typename T::V);
    if (smem > 48 * 1024) MNPB_TRY(smem_opt_in(kernel<T, NC>, 220 * 1024, "skn::kernel"));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ceil_div(m, ROWS) * C), (unsigned)batch);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = C > 1 ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, kernel<T, NC>, m, n, k, alpha, A, X, beta, Y, C) !=
        cudaSuccess) {
        set_error("matrix times vectors: launch failed: %s",
                  cudaGetErrorString(cudaGetLastError()));
        return MNPB_ECUDA;
    }
    MNPB_LAUNCH_CHECK("skn::kernel");
    return MNPB_OK;
}

// n <= 16 columns.
template <typename T>
int run(cudaStream_t s, int m, int n, int k, int batch, typename T::Scale alpha,
        typename T::Mat A, typename T::Mat X, typename T::Scale beta, typename T::Mat Y) {
    if (n <= 1) return launch<T, 1>(s, m, n, k, batch, alpha, A, X, beta, Y);
    if (n <= 4) return launch<T, 4>(s, m, n, k, batch, alpha, A, X, beta, Y);
    if (n <= 8) return launch<T, 8>(s, m, n, k, batch, alpha, A, X, beta, Y);
    if (n <= 12) return launch<T, 12>(s, m, n, k, batch, alpha, A, X, beta, Y);
    return launch<T, 16>(s, m, n, k, batch, alpha, A, X, beta, Y);
}

}  // namespace skn
}  // namespace mnpb
