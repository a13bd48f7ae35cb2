// Triangular solve for a few right-hand sides, one thread block cluster per
// matrix (and per chunk of NC right-hand sides).
//
// What bounds it: the chain of n / 64 diagonal blocks, and below it the
// bandwidth the CTAs working on one matrix can draw.  Block rows of 64 are
// dealt to the C CTAs of the cluster round-robin and their right-hand sides
// stay in shared memory.  Step k: the owner of block k + 1 first subtracts
// T(k+1, k) x_k from its rows, solves the diagonal block and pushes x_{k+1}
// into every CTA's shared memory; all CTAs then arrive at the cluster barrier
// and use its latency for the rest of column k of the triangle, whose tiles
// are loaded one ahead into registers (they do not depend on x).
//
// x has three buffers: x_{k+2} is pushed after the barrier of step k + 1,
// which every CTA reaches only after its updates with x_{k-1} are done, while
// x_k may still be read.  The last push precedes the last barrier.
//
// The row interchanges of the LU (ipiv) are applied while the right-hand sides
// are read: composed in shared memory as a gather, the steps with one target
// chained so that each step looks only at those.
//
// Measured, FP64, both triangles with the interchanges, against the recursion
// of many-right-hand-side leaves this replaces: n = 2884, 1 / 4 columns 5.14 /
// 5.31 -> 0.62 / 0.87 ms; 1365, 12 columns 2.49 -> 0.39; 284, 1 column 452 ->
// 71 us, 41 matrices 4 columns 486 -> 86 us; 41 x 1148, 3 columns 2.48 -> 0.45.
//
// FP32 (512 threads, two block rows per update, the diagonal blocks through their halves'
// inverses, G1 and G2 in one launch) against the solves it replaces, per
// triangle: 2884, 4 columns 1.05 -> 0.16 ms for one matrix, 1.06 -> 0.41 ms for
// 27; 12 columns, 13 to 26 matrices of 284 to 2044 rows 0.78 -> 0.12 ms.
//
// An upper triangle is solved as a lower one with blocks and rows in reverse
// order; "logical" indices below count in the order of the solve.
#pragma once
#include "lu_panel.cuh"

namespace mnpb {
namespace trc {

constexpr int NB = 64, GROUP = 256, MAXC = 8;   // threads that update one tile together

__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// FP64: the diagonal blocks are solved by substitution.
struct F64 : lup::F64 {
    typedef lup::F64::Mat Mat;
    // staged diagonal block: the triangle in logical order, column by column
    static constexpr int DELEMS = NB * NB;
    static constexpr int P = 1, H = 1;   // block rows per update: P per thread group, H groups
    static constexpr int THREADS = GROUP * H;
    // 16 entries of one row, four columns apart
    static __device__ __forceinline__ void load16(const Mat &m, int64_t b, int row, int col,
                                                  V (&t)[16]) {
        const cd *p = m.A + b * m.sA + col * m.lda + row;
        const int64_t step = 4 * m.lda;
#pragma unroll
        for (int k = 0; k < 16; ++k) t[k] = p[k * step];
    }
    static __device__ __forceinline__ V fma(V a, V b, V c) { return cfma(a, b, c); }
    static __device__ __forceinline__ V shfl(V v, int l) {
        return cmk(__shfl_sync(0xffffffffu, v.x, l), __shfl_sync(0xffffffffu, v.y, l));
    }
    static __device__ __forceinline__ V shfl_xor(V v, int o) {
        return cmk(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
    }
    static __device__ __forceinline__ V sub(V a, V b) { return csub(a, b); }
    static __device__ __forceinline__ V add(V a, V b) { return cadd(a, b); }
    static __device__ __forceinline__ void stage(V *D, const Mat &A, const float *, int64_t b,
                                                 int n, int blk, bool lower, int tid) {
        V v[DELEMS / THREADS];
#pragma unroll
        for (int q = 0; q < DELEMS / THREADS; ++q) {
            const int e = tid + q * THREADS, p = e % NB, j = e / NB;   // physical row, column
            const int gr = blk * NB + p, gc = blk * NB + j;
            v[q] = (gr < n && gc < n) ? load(A, b, gr, gc) : cmk(p == j ? 1.0 : 0.0, 0.0);
        }
#pragma unroll
        for (int q = 0; q < DELEMS / THREADS; ++q) {
            const int e = tid + q * THREADS, p = e % NB, j = e / NB;
            D[lower ? e : (NB - 1 - j) * NB + NB - 1 - p] = v[q];
        }
    }
    // one warp, one right-hand side: r0, r1 = rows lane and lane + 32 in
    // logical order, overwritten by the solution
    static __device__ __forceinline__ void diag(const V *D, bool unit, int lane, V &r0, V &r1) {
        V i0 = cmk(1.0, 0.0), i1 = i0;
        if (!unit) {
            i0 = crcp(D[lane * NB + lane]);
            i1 = crcp(D[(lane + 32) * NB + lane + 32]);
        }
#pragma unroll 4
        for (int j = 0; j < 32; ++j) {
            const V x = shfl(unit ? r0 : cmul(r0, i0), j);
            if (lane > j) r0 = cfms(D[j * NB + lane], x, r0);
            r1 = cfms(D[j * NB + lane + 32], x, r1);
        }
#pragma unroll 4
        for (int j = 0; j < 32; ++j) {
            const V x = shfl(unit ? r1 : cmul(r1, i1), j);
            if (lane > j) r1 = cfms(D[(j + 32) * NB + lane + 32], x, r1);
        }
        if (!unit) {
            r0 = cmul(r0, i0);
            r1 = cmul(r1, i1);
        }
    }
};

// Systems of one launch: `groups` sets of `per` entries, the sets' triangles,
// inverses, right-hand sides and pivots these offsets (elements) apart.  G1
// and G2 of the BEM solve go through one launch this way.
struct Groups {
    int per, groups;
    int64_t A, D, X, P;
};

template <typename T, int NC>
struct Smem {
    typedef typename T::V V;
    static constexpr int XS = NC + 1;   // row stride of x: four column groups, four bank groups
    static int64_t bytes(int n, int C) {
        const int nb = ceil_div(n, NB), own = ceil_div(nb, C);
        return ((int64_t)T::DELEMS + 3 * NB * XS + (int64_t)own * NB * NC) * sizeof(V);
    }
    // the interchanges are composed where the diagonal block is staged later
    static bool composes(int n) {
        return 4 * (int64_t)n * sizeof(int) <=
               ((int64_t)T::DELEMS + 3 * NB * XS) * (int64_t)sizeof(V);
    }
};

// Gather equal to the interchanges (c, ipiv[c]), c = 0 .. n - 1 in order: row c
// of the result is row src[c].  w: 4 n ints of shared memory, src = w on return.
// V(c), the row whose value sits in row c before step c, is V of the last
// earlier step that targeted c, or c itself; row c ends with V of the last
// earlier step with the same target as step c, or with the target's own row.
// That takes ipiv[c] >= c, as an LU gives it; a caller's sequence with other
// targets, whose chains could close to a ring, is followed step by step instead.
__device__ __forceinline__ void compose(int *w, const int32_t *ipiv, int n) {
    int *p = w, *head = w + n, *next = w + 2 * n, *par = w + 3 * n;
    int down = 1;
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
        p[c] = ipiv[c];
        head[c] = -1;
        if (p[c] < c) down = 0;
    }
    if (!__syncthreads_and(down)) {
        for (int c = threadIdx.x; c < n; c += blockDim.x) head[c] = c;
        __syncthreads();
        if (threadIdx.x == 0)
            for (int c = 0; c < n; ++c) {
                const int t = p[c], r = head[c];
                head[c] = head[t];
                head[t] = r;
            }
        __syncthreads();
        for (int c = threadIdx.x; c < n; c += blockDim.x) p[c] = head[c];
        __syncthreads();
        return;
    }
    for (int c = threadIdx.x; c < n; c += blockDim.x)
        if (p[c] != c) next[c] = atomicExch(&head[p[c]], c);
    __syncthreads();
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
        int q = -1;
        for (int e = head[c]; e >= 0; e = next[e]) q = max(q, e);
        par[c] = q;
    }
    __syncthreads();
    for (int c0 = 0; c0 < n; c0 += blockDim.x) {
        const int c = c0 + threadIdx.x;
        int v = 0;
        if (c < n) {
            const int t = p[c];
            int q = -1;
            if (t != c)
                for (int e = head[t]; e >= 0; e = next[e])
                    if (e < c) q = max(q, e);
            v = t;
            if (t == c || q >= 0) {
                v = t == c ? c : q;
                while (par[v] >= 0) v = par[v];
            }
        }
        // p[c] is read by step c only, from here on
        if (c < n) p[c] = v;
    }
    __syncthreads();
}

template <typename T, int NC>
__global__ void __launch_bounds__(T::THREADS, 1)
    trsv_kernel(int n, int m, int lower_, int unit_, typename T::Mat A,
                const float *Dinv, typename T::Mat X, const int32_t *ipiv, int64_t sP, int C,
                int chunks, Groups gr_) {
    typedef typename T::V V;
    constexpr int XS = Smem<T, NC>::XS, THREADS = T::THREADS;
    grid_wait();
    extern __shared__ __align__(16) unsigned char trc_sm[];
    V *D = (V *)trc_sm;              // staged diagonal block
    V *xs = D + T::DELEMS;           // [3][NB][XS]
    V *rs = xs + 3 * NB * XS;        // [own blocks][NB][NC]
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    // thread group, tile row, column group
    const int hg = tid / GROUP, rl = (wid & 7) * 8 + (lane & 7), q = lane >> 3;
    const bool lower = lower_, unit = unit_;
    const int me = C > 1 ? (int)lup::cluster_rank() : 0;
    const int64_t unitid = blockIdx.x / C;
    const int64_t b = (unitid / chunks) % gr_.per;
    {
        const int64_t g = (unitid / chunks) / gr_.per;
        A.A += g * gr_.A;
        X.A += g * gr_.X;
        Dinv += g * gr_.D;
        if (ipiv) ipiv += g * gr_.P;
    }
    const int c0 = (int)(unitid % chunks) * NC;
    const int mc = min(NC, m - c0);
    const int nb = (n + NB - 1) / NB;
    auto phys = [&](int k) { return lower ? k : nb - 1 - k; };

    const int *src = nullptr;
    if (ipiv) {
        compose((int *)trc_sm, ipiv + b * sP, n);
        src = (const int *)trc_sm;
    }
    for (int k = me, o = 0; k < nb; k += C, ++o)
        for (int e = tid; e < NB * NC; e += THREADS) {
            const int p = e % NB, c = e / NB, gr = phys(k) * NB + p;
            rs[(o * NB + p) * NC + c] =
                (gr < n && c < mc) ? T::load(X, b, src ? src[gr] : gr, c0 + c) : T::zero();
        }
    if (ipiv) __syncthreads();
    if (me < nb) T::stage(D, A, Dinv, b, n, phys(me), lower, tid);
    __syncthreads();

    // solve the owned block o (logical block k), publish x_k
    auto solve = [&](int k, int o) {
        for (int c = wid; c < NC; c += THREADS / 32) {
            const int p0 = lower ? lane : NB - 1 - lane, p1 = lower ? lane + 32 : NB - 33 - lane;
            V r0 = rs[(o * NB + p0) * NC + c], r1 = rs[(o * NB + p1) * NC + c];
            T::diag(D, unit, lane, r0, r1);
            const int g0 = phys(k) * NB + p0, g1 = phys(k) * NB + p1;
            V *x0 = xs + ((k % 3) * NB + p0) * XS + c, *x1 = xs + ((k % 3) * NB + p1) * XS + c;
            if (C > 1) {
                for (int t = 0; t < C; ++t) {
                    T::push(lup::map_rank(x0, t), r0);
                    T::push(lup::map_rank(x1, t), r1);
                }
            } else {
                *x0 = r0;
                *x1 = r1;
            }
            if (c < mc) {
                if (g0 < n) T::store(X, b, g0, c0 + c, r0);
                if (g1 < n) T::store(X, b, g1, c0 + c, r1);
            }
        }
    };
    // tiles (i, k), (i + C, k), ...: 16 entries of each per thread (row rl,
    // columns 4 kk + q); a thread group takes P tiles, which share the reads of x
    constexpr int P = T::P, H = T::H;
    auto fetch = [&](int i, int k, V (&t)[P][16]) {
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const int it = i + (hg * P + p) * C;
            const int gr = it < nb ? phys(it) * NB + rl : n;
            // a tile inside the matrix: no bounds and addresses by steps, which
            // were as many instructions as the products (FP64 2884, 1 / 4 columns
            // 0.71 / 1.00 -> 0.62 / 0.87 ms; FP32 27 x 2884 5 to 9 % less)
            if (it < nb && max(phys(it), phys(k)) * NB + NB <= n) {
                T::load16(A, b, gr, phys(k) * NB + q, t[p]);
                continue;
            }
#pragma unroll
            for (int kk = 0; kk < 16; ++kk) {
                const int gc = phys(k) * NB + 4 * kk + q;
                t[p][kk] = (gr < n && gc < n) ? T::load(A, b, gr, gc) : T::zero();
            }
        }
    };
    auto update = [&](int i, int k, const V (&t)[P][16]) {
        const V *x = xs + (k % 3) * NB * XS;
        V acc[P][NC];
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
            for (int c = 0; c < NC; ++c) acc[p][c] = T::zero();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const V xv = x[(4 * kk + q) * XS + c];
#pragma unroll
                for (int p = 0; p < P; ++p) acc[p][c] = T::fma(t[p][kk], xv, acc[p][c]);
            }
#pragma unroll
        for (int p = 0; p < P; ++p) {
            if (i + (hg * P + p) * C >= nb) break;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                acc[p][c] = T::add(acc[p][c], T::shfl_xor(acc[p][c], 8));
                acc[p][c] = T::add(acc[p][c], T::shfl_xor(acc[p][c], 16));
            }
            V *r = rs + (((i - me) / C + hg * P + p) * NB + rl) * NC;
#pragma unroll
            for (int c = 0; c < NC; ++c)
                if ((c & 3) == q) r[c] = T::sub(r[c], acc[p][c]);
        }
    };

    V cur[P][16];
    // the tiles in the order of their use: column k, owned block rows i > k
    // ascending, P H at a time
    int ti = me, tk = 0;             // next tiles to fetch
    auto first_row = [&](int k) { return k + 1 + ((me - (k + 1)) % C + C) % C; };
    ti = first_row(0);
    auto valid = [&]() { return ti < nb; };
    auto advance = [&]() {
        ti += P * H * C;
        if (ti >= nb) {
            ++tk;
            ti = first_row(tk);
        }
    };
    if (C > 1) lup::cluster_sync();  // every CTA has started
    if (valid()) fetch(ti, tk, cur);
    if (me == 0) solve(0, 0);
    if (C > 1) cluster_arrive();
    int staged = me;                 // logical block whose diagonal D holds
    for (int k = 0; k < nb; ++k) {
        if (C > 1) cluster_wait();
        __syncthreads();             // x_k visible; D free if block k was ours
        if (staged == k && k + C < nb) {
            staged = k + C;
            T::stage(D, A, Dinv, b, n, phys(staged), lower, tid);
        }
        const bool next_mine = k + 1 < nb && (k + 1) % C == me;
        V nxt[P][16];
        if (next_mine) {
            // tile (k + 1, k) is among the first of this column
            const int i = ti;
            advance();
            if (valid()) fetch(ti, tk, nxt);
            update(i, k, cur);
#pragma unroll
            for (int e = 0; e < P * 16; ++e) cur[e / 16][e % 16] = nxt[e / 16][e % 16];
            __syncthreads();         // rows of block k + 1 and its staged diagonal complete
            solve(k + 1, (k + 1) / C);
        }
        if (C > 1 && k + 1 < nb) cluster_arrive();
        while (valid() && tk == k) {
            const int i = ti;
            advance();
            if (valid()) fetch(ti, tk, nxt);
            update(i, k, cur);
#pragma unroll
            for (int e = 0; e < P * 16; ++e) cur[e / 16][e % 16] = nxt[e / 16][e % 16];
        }
    }
}

// CTAs per cluster for `units` systems of n rows: as many as leave every
// system a cluster at once, more where the right-hand sides need the room;
// 0 if they do not fit.
template <typename T, int NC>
int cluster_size(int n, int64_t units) {
    const int nb = ceil_div(n, NB);
    int C = 1;
    while (C < MAXC && 2 * C <= nb && units * 2 * C <= device_sms()) C *= 2;
    while (C < MAXC && Smem<T, NC>::bytes(n, C) > 200 * 1024) C *= 2;
    return Smem<T, NC>::bytes(n, C) <= 200 * 1024 ? C : 0;
}

template <typename T, int NC>
int launch_trsv(cudaStream_t s, bool lower, bool unit, int n, int m, const Groups &gr,
                typename T::Mat A, const float *Dinv, typename T::Mat X, const int32_t *ipiv,
                int64_t sP, int C) {
    const int chunks = ceil_div(m, NC);
    const int smem = (int)Smem<T, NC>::bytes(n, C);
    MNPB_TRY(smem_opt_in(trsv_kernel<T, NC>, smem, "trc::trsv_kernel"));
    return launch_chained("trc::trsv_kernel", trsv_kernel<T, NC>,
                          dim3((unsigned)(gr.per * gr.groups * chunks * C)), dim3(T::THREADS),
                          (size_t)smem, s, C, n, m, lower ? 1 : 0, unit ? 1 : 0, A, Dinv, X, ipiv,
                          sP, C, chunks, gr);
}

}  // namespace trc
}  // namespace mnpb
