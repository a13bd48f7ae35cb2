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

#include <type_traits>

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
        return m.A[b * m.sA + col * m.lda + row];
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

// The lane sums of all CTAs of the cluster, part[lane][row][column], summed in
// a fixed order and stored by the first CTA.
template <typename T, int NC>
__device__ __forceinline__ void finish(int m, int n, typename T::Scale alpha,
                                       typename T::Scale beta, typename T::Mat Y,
                                       typename T::V *part, int C, int me, int64_t b) {
    typedef typename T::V V;
    constexpr int ROWS = ROWT * T::R;
    const int tid = threadIdx.x;
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

template <typename T, int NC>
__global__ void __launch_bounds__(THREADS) kernel(int m, int n, int k, typename T::Scale alpha,
                                                  typename T::Mat A, typename T::Mat X,
                                                  typename T::Scale beta, typename T::Mat Y,
                                                  int C) {
    typedef typename T::V V;
    constexpr int R = T::R, ROWS = ROWT * R;
    static_assert(KT % (LANES * T::U) == 0, "chunk");
    grid_wait();
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
    // finish() written out: with the call the loop above is compiled another way (FP64, 4
    // columns: 70 registers instead of 80), and 81 wavelengths of 2884 faces take 425
    // instead of 393 ms, 13 of six uneven particles 148.5 instead of 146.1
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

// FP64 products with more than four columns.  4 NC FMAs per 16-byte element of A
// take the FP64 pipe about as long as the memory, and in the kernel above every
// group of four also reads x from shared memory.  Here X becomes two real
// operands, [Re X | Im X] and [-Im X | Re X], for mma.sync m16n8k4: a warp's 32
// rows x 4 columns of A meet 2 NC real columns in NT tiles of eight, the parts of
// A being the two A operands as they are loaded.  Same rows, k lanes and chunks
// per CTA as above.  Bound by the latency of the loads at one or two CTAs per SM
// (12 columns 2.7 TB/s).  Against the kernel above: 8 x 2884 x 2884, 8 / 12 / 16
// columns 511 -> 273, 620 -> 401, 960 -> 513 us; 41 x 284, 12 columns 51 -> 42 us;
// with four columns or fewer that one is at 3.7 to 5.7 TB/s and stays.
template <int NC>
__global__ void __launch_bounds__(THREADS, NC <= 8 ? 2 : 1)
    mma_kernel(int m, int n, int k, cd alpha, F64::Mat A, F64::Mat X, cd beta, F64::Mat Y,
               int C) {
    // row stride 2 XS of x: 4 k rows x 4 columns of a load meet 16 banks of 8 bytes
    constexpr int NT = NC / 4, XS = 8 * NT + 2;
    constexpr int STEPS = KT / (4 * LANES);
    grid_wait();
    extern __shared__ __align__(16) unsigned char skn_sm[];
    double *xs = (double *)skn_sm;             // [2][KT][2 XS]: both operands of a k row
    cd *part = (cd *)(xs + 4 * KT * XS);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int g = lane >> 2, t = lane & 3, kl = wid % LANES, rw = wid / LANES * 32;
    const int64_t b = blockIdx.y;
    const int me = C > 1 ? (int)lup::cluster_rank() : 0;
    const int row = (blockIdx.x / C) * ROWT + rw + g;
    const int nch = (k + KT - 1) / KT, per = (nch + C - 1) / C;
    const int kbeg = min(k, me * per * KT), kend = min(k, (me + 1) * per * KT);
    double acc[2][NT][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;
    // x one chunk, A one chunk ahead of its use, through registers
    constexpr int XR = KT * NC / THREADS;
    cd xr[XR], a[STEPS][4];
    auto xload = [&](int k0) {
#pragma unroll
        for (int i = 0; i < XR; ++i) {
            const int e = tid + i * THREADS, kk = e % KT, c = e / KT;
            xr[i] = (k0 + kk < kend && c < n) ? F64::load(X, b, k0 + kk, c) : F64::zero();
        }
    };
    auto xstore = [&](int buf) {
#pragma unroll
        for (int i = 0; i < XR; ++i) {
            const int e = tid + i * THREADS, kk = e % KT, c = e / KT;
            double *x = xs + (buf * KT + kk) * 2 * XS + c;
            x[0] = xr[i].x;
            x[NC] = xr[i].y;
            x[XS] = -xr[i].y;
            x[XS + NC] = xr[i].x;
        }
    };
    auto aload = [&](cd (&v)[4], int col) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            v[i] = (col < kend && row + 8 * i < m) ? F64::load(A, b, row + 8 * i, col)
                                                   : F64::zero();
    };
    xload(kbeg);
    // this warp's 4-column steps kl, kl + LANES, ... of a chunk
#pragma unroll
    for (int u = 0; u < STEPS; ++u) aload(a[u], kbeg + 4 * (kl + u * LANES) + t);
    xstore(0);
    int buf = 0;
    for (int k0 = kbeg; k0 < kend; k0 += KT, buf ^= 1) {
        __syncthreads();                       // chunk k0 staged, the other buffer free
        if (k0 + KT < kend) xload(k0 + KT);
#pragma unroll
        for (int u = 0; u < STEPS; ++u) {
            const double *x = xs + (buf * KT + 4 * (kl + u * LANES) + t) * 2 * XS + g;
            double x1[NT], x2[NT];
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                x1[j] = x[8 * j];
                x2[j] = x[XS + 8 * j];
            }
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                mma_f64(acc[0][j], a[u][0].x, a[u][1].x, x1[j]);
                mma_f64(acc[1][j], a[u][2].x, a[u][3].x, x1[j]);
            }
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                mma_f64(acc[0][j], a[u][0].y, a[u][1].y, x2[j]);
                mma_f64(acc[1][j], a[u][2].y, a[u][3].y, x2[j]);
            }
            aload(a[u], k0 + KT + 4 * (kl + u * LANES) + t);
        }
        if (k0 + KT < kend) xstore(buf ^ 1);
    }
    __syncthreads();
    double *pd = (double *)part;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = rw + 16 * i + g + 8 * (e >> 1), q = 8 * j + 2 * t + (e & 1);
                pd[((kl * ROWT + r) * NC + (q < NC ? q : q - NC)) * 2 + (q < NC ? 0 : 1)] =
                    acc[i][j][e];
            }
    __syncthreads();
    finish<F64, NC>(m, n, alpha, beta, Y, part, C, me, b);
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
    // FP64 from 8 columns on: the tensor path
    constexpr bool MMA = std::is_same<T, F64>::value && NC >= 8;
    const int xs = MMA ? 4 * KT * (2 * NC + 2) * (int)sizeof(double)
                       : KT * NC * (int)sizeof(typename T::V);
    const int smem = xs + np * ROWS * NC * (int)sizeof(typename T::V);
    const auto f = [] {
        if constexpr (MMA)
            return mma_kernel<NC>;
        else
            return kernel<T, NC>;
    }();
    if (smem > 48 * 1024) MNPB_TRY(smem_opt_in(f, 220 * 1024, "skn::kernel"));
    const dim3 grid((unsigned)(ceil_div(m, ROWS) * C), (unsigned)batch);
    return launch_chained("skn::kernel", f, grid, dim3(THREADS), (size_t)smem, s, C, m, n, k,
                          alpha, A, X, beta, Y, C);
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
