// LU panel with partial pivoting, held in registers and spread over a thread
// block cluster.
//
// One cluster of C CTAs factors the columns [k0, k0 + kb) (kb <= W) of one
// matrix over the rows [k0, n).  Every thread keeps R rows x W columns from load
// to store, so a column step touches no memory but the pivot row: the rows are
// dealt to the CTAs in blocks of R * blockDim.x.  In registers, but for what does not
// fit in the 168 that 384 threads leave each: FP64 spills 44 bytes of stores and 356
// of loads (-Xptxas -v) with 32 columns, 40 and 108 with 16 of two rows, 416 and 624
// with 8 of four; FP32 with 32 columns takes 122 registers and none.
//
// What bounds it: the chain of kb dependent pivot steps.  A step is a warp
// and CTA reduction of the pivot candidates, one exchange between the CTAs,
// and the rank-1 update.  Each CTA's best row is pushed to every CTA of the
// cluster (distributed shared memory) together with its value before the
// exchange's one cluster barrier, so the winner's row is local to all CTAs
// when the barrier opens.  Rows never move: each carries the row position it
// would have after the interchanges so far (`pos`), an interchange swaps two
// positions, and the rows are stored at their final positions at the end.
//
// Two buffers alternate between steps: a push into buffer (j & 1) for step
// j + 2 comes after the barrier of step j + 1, which every thread reaches
// only after its reads of step j.  The last remote store precedes the last
// barrier, so no CTA of the cluster is written to after it has left.
//
// Measured (FP64 LU of one n x n matrix, all else equal) against the leaf it
// replaces, one CTA per matrix working in global memory: n = 284 1.44 -> 0.94
// ms, 1365 16.0 -> 7.5, 2884 63.7 -> 22.0, 7000 348 -> 106; 41 matrices of
// 1148 23.1 -> 16.9.  A pivot step takes 1.1 us in one CTA and 1.8 us in a
// cluster of 8 (1.4 and 2.1 before the reductions were redux.sync on the bit
// patterns instead of shuffles of the values).
#pragma once
#include "common.cuh"

namespace mnpb {
namespace lup {

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_rank(const void *p, uint32_t rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

// FP64 interleaved storage (column-major complex128).
struct F64 {
    typedef cd V;
    typedef double S;
    struct Mat {
        cd *A;
        int64_t lda, sA;
    };
    static __device__ __forceinline__ V zero() { return cmk(0.0, 0.0); }
    static __device__ __forceinline__ V load(const Mat &m, int64_t b, int64_t row, int64_t col) {
        return m.A[b * m.sA + col * m.lda + row];
    }
    static __device__ __forceinline__ void store(const Mat &m, int64_t b, int64_t row,
                                                 int64_t col, V v) {
        m.A[b * m.sA + col * m.lda + row] = v;
    }
    static __device__ __forceinline__ S mag(V v) { return cabs1(v); }
    // one division where the squares can neither overflow nor underflow
    static __device__ __forceinline__ V rcp(V v) {
        const double m = fmax(fabs(v.x), fabs(v.y));
        if (m > 1e-100 && m < 1e100) {
            const double i = 1.0 / (v.x * v.x + v.y * v.y);
            return cmk(v.x * i, -v.y * i);
        }
        return crcp(v);
    }
    static __device__ __forceinline__ V mul(V a, V b) { return cmul(a, b); }
    static __device__ __forceinline__ V fms(V a, V b, V c) { return cfms(a, b, c); }
    static __device__ __forceinline__ V rnd(V v) { return v; }   // storage precision of L and U
    static __device__ __forceinline__ void push(uint32_t addr, V v) {
        asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y)
                     : "memory");
    }
    static __device__ __forceinline__ void push_s(uint32_t addr, S v) {
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
    }
};

constexpr int MAXC = 8;          // CTAs per cluster (portable limit)
constexpr int MAXW = 12;         // warps per CTA
constexpr int NOROW = 0x7fffffff;

// Best (magnitude, position) of a warp: larger magnitude (>= 0), then smaller
// position.  The bit pattern of a non-negative number orders as an integer, so
// the reductions are redux.sync on 32-bit words.
__device__ __forceinline__ void warp_best(double &v, int &p) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    p = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? p : NOROW);
    v = __hiloint2double((int)mh, (int)ml);
}
__device__ __forceinline__ void warp_best(float &v, int &p) {
    const unsigned k = __float_as_uint(v), m = __reduce_max_sync(0xffffffffu, k);
    p = __reduce_min_sync(0xffffffffu, k == m ? p : NOROW);
    v = __uint_as_float(m);
}

template <typename T, int W, int R>
__global__ void __launch_bounds__(32 * MAXW, 1)
    panel_kernel(int n, int k0, int kb, typename T::Mat A, int32_t *ipiv, int64_t sP,
                 int32_t *info, int C) {
    typedef typename T::V V;
    typedef typename T::S S;
    constexpr int WIN = R == 1 ? 8 : 4;        // columns of an unrolled window
    __shared__ __align__(16) V rowbuf[2][MAXC][W];   // every CTA's best row
    __shared__ S cand_v[2][MAXC];
    __shared__ int cand_p[2][MAXC];
    __shared__ S red_v[2][MAXW];
    __shared__ int red_p[2][MAXW];
    grid_wait();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nw = blockDim.x >> 5;
    const uint32_t me = C > 1 ? cluster_rank() : 0;
    const int64_t b = blockIdx.x / C;
    const int m = n - k0;
    V a[R][W];
    int pos[R];                       // row position relative to k0; done rows: < jj
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = (int)me * R * blockDim.x + r * blockDim.x + tid;
        pos[r] = i < m ? i : NOROW;
#pragma unroll
        for (int j = 0; j < W; ++j)
            a[r][j] = (i < m && j < kb) ? T::load(A, b, k0 + i, k0 + j) : T::zero();
    }
    if (C > 1) cluster_sync();        // every CTA of the cluster has started
    // WIN steps are unrolled, with the current columns always in registers
    // 0 .. WIN - 1: after them the columns rotate, so that one copy of the code
    // serves all of them (unrolled over all W columns the code ran once per
    // launch, straight from the instruction fetch: FP64 LUs 2 % slower, FP32
    // LUs of one 2884 matrix 11.1 against 10.7 ms; the two-row instances are
    // quicker with windows of four, 54 x 2884 36.9 against 34.0 ms)
#pragma unroll 1
    for (int o = 0; o < W; o += WIN) {
#pragma unroll
        for (int w = 0; w < WIN; ++w) {
            const int jj = o + w;
            if (jj < kb) {
                const int buf = jj & 1;
                // best of this thread's active rows, then of the warp, then of the CTA
                S bv = (S)0;
                int bp = NOROW;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const S t = T::mag(a[r][w]);
                    const S v = t > (S)0 ? t : (S)0;       // NaN counts as zero
                    if (pos[r] != NOROW && pos[r] >= jj &&
                        (v > bv || (v == bv && pos[r] < bp))) {
                        bv = v;
                        bp = pos[r];
                    }
                }
                warp_best(bv, bp);
                if (lane == 0) { red_v[buf][wid] = bv; red_p[buf][wid] = bp; }
                __syncthreads();
                bv = lane < nw ? red_v[buf][lane] : (S)0;
                bp = lane < nw ? red_p[buf][lane] : NOROW;
                warp_best(bv, bp);
                // the warp that holds the CTA's best row publishes it
                bool mine = false;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (bp != NOROW && pos[r] == bp) {
                        mine = true;
#pragma unroll
                        for (int g = 0; g < W; g += WIN)
                            if (g < W - o) {
#pragma unroll
                                for (int j = g == 0 ? w : g; j < g + WIN; ++j)
                                    rowbuf[buf][me][j] = T::rnd(a[r][j]);
                            }
                    }
                if (C > 1) {
                    const bool ours = __any_sync(0xffffffffu, mine);
                    if (ours) {
                        __syncwarp();
                        if (lane >= w && lane < W - o) {
                            const V v = rowbuf[buf][me][lane];
#pragma unroll
                            for (int q = 0; q < MAXC; ++q)
                                if (q < C && q != (int)me)
                                    T::push(map_rank(&rowbuf[buf][me][lane], q), v);
                        }
                    }
                    // CTAs without active rows publish "none"
                    if (wid == 0 && lane < C) {
                        T::push_s(map_rank(&cand_v[buf][me], lane), bv);
                        asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(
                                         map_rank(&cand_p[buf][me], lane)),
                                     "r"(bp)
                                     : "memory");
                    }
                    cluster_sync();
                } else {
                    __syncthreads();
                }
                int win = 0;
                if (C > 1) {
                    bv = lane < C ? cand_v[buf][lane] : (S)0;
                    const int own = lane < C ? cand_p[buf][lane] : NOROW;
                    bp = own;
                    warp_best(bv, bp);
                    win = __ffs(__ballot_sync(0xffffffffu, own == bp)) - 1;
                }
                if (me == 0 && tid == 0) {
                    ipiv[b * sP + k0 + jj] = k0 + bp;
                    if (!(bv > (S)0) && info && info[b] == 0) info[b] = k0 + jj + 1;
                }
                const V *u = rowbuf[buf][win];
                const V pv = u[w];
                const bool nz = pv.x != (S)0 || pv.y != (S)0;
                const V inv = nz ? T::rcp(pv) : T::zero();
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    // the interchange of positions jj and bp
                    const int p = pos[r];
                    const bool done = p == bp;
                    if (done) pos[r] = jj;
                    else if (p == jj) pos[r] = bp;
                    // a finished row keeps its values (as stored), the others subtract
                    const bool upd = !done && pos[r] > jj && pos[r] != NOROW;
                    if (upd) {
                        V l = a[r][w];
                        if (nz) l = T::rnd(T::mul(l, inv));
                        a[r][w] = l;
#pragma unroll
                        for (int g = 0; g < W; g += WIN)
                            if (g < W - o) {
#pragma unroll
                                for (int j = g == 0 ? w + 1 : g; j < g + WIN; ++j)
                                    a[r][j] = T::fms(l, u[j], a[r][j]);
                            }
                    }
                    if (done) {
#pragma unroll
                        for (int g = 0; g < W; g += WIN)
                            if (g < W - o) {
#pragma unroll
                                for (int j = g == 0 ? w : g; j < g + WIN; ++j)
                                    a[r][j] = T::rnd(a[r][j]);
                            }
                    }
                }
            }
        }
        if (W > WIN) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                V t[WIN];
#pragma unroll
                for (int j = 0; j < WIN; ++j) t[j] = a[r][j];
#pragma unroll
                for (int j = 0; j + WIN < W; ++j) a[r][j] = a[r][j + WIN];
#pragma unroll
                for (int j = 0; j < WIN; ++j) a[r][W - WIN + j] = t[j];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (pos[r] != NOROW) {
#pragma unroll
            for (int j = 0; j < W; ++j)
                if (j < kb) T::store(A, b, k0 + pos[r], k0 + j, a[r][j]);
        }
}

// Launch shape for m rows of `batch` matrices: CTAs per cluster and threads
// per CTA; false if the rows do not fit in MAXC CTAs.
inline bool panel_shape(int m, int R, int &C, int &threads) {
    const int per = 32 * MAXW * R;
    C = ceil_div(m, per);
    if (C > MAXC) return false;
    threads = 32 * ceil_div(ceil_div(m, C * R), 32);
    return true;
}

template <typename T, int W, int R>
int launch_panel(cudaStream_t s, int n, int k0, int kb, typename T::Mat A, int32_t *ipiv,
                 int64_t sP, int32_t *info, int batch, int C, int threads) {
    return launch_chained("lup::panel_kernel", panel_kernel<T, W, R>, dim3((unsigned)(batch * C)),
                          dim3((unsigned)threads), 0, s, C, n, k0, kb, A, ipiv, sP, info, C);
}

}  // namespace lup
}  // namespace mnpb
