// Batched dense complex linear algebra in FP32 on planar storage (real plane,
// imaginary plane), column-major, for the mixed-precision solver.
//
// LU is recursive down to blocks of 128 columns (split the columns in halves;
// factor the left half; update the right half with a triangular solve and a
// GEMM; factor the rest), so nearly all flops land in large GEMMs that run on
// the tensor cores (tc::cgemm_tf32).  A block goes leaf by leaf: 32-column LU
// panel, fused interchange and solve of the block's other columns, GEMM.  Only
// the panels, those strips, the 128 x 128 diagonal-block inverses and the
// 32-row leaves of small triangular solves run on CUDA cores.
#include "common.cuh"
#include "dense_f32.cuh"
#include "interchange.cuh"
#include "lu_panel.cuh"
#include "skinny.cuh"
#include "trsv_cluster.cuh"

namespace mnpb {
namespace f32 {

using tc::CMatF;

namespace {

constexpr int PANEL_THREADS = 512;
constexpr int TS = 32;

struct cf {
    float x, y;
};
__device__ __forceinline__ cf fmk(float r, float i) { return cf{r, i}; }
__device__ __forceinline__ cf fmul(cf a, cf b) { return cf{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
__device__ __forceinline__ cf ffms(cf a, cf b, cf c) {   // c - a*b
    c.x = fmaf(-a.x, b.x, c.x);
    c.x = fmaf(a.y, b.y, c.x);
    c.y = fmaf(-a.x, b.y, c.y);
    c.y = fmaf(-a.y, b.x, c.y);
    return c;
}
__device__ __forceinline__ cf frcp(cf b) {
    if (fabsf(b.x) >= fabsf(b.y)) {
        float r = b.y / b.x, d = b.x + b.y * r;
        return cf{1.f / d, -r / d};
    } else {
        float r = b.x / b.y, d = b.y + b.x * r;
        return cf{r / d, -1.f / d};
    }
}
// nearest TF32 (10-bit mantissa), ties away from zero
__device__ __forceinline__ float tf32_rna(float v) {
    uint32_t t;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(t) : "f"(v));
    return __uint_as_float(t);
}
__device__ __forceinline__ cf rna(cf v) { return cf{tf32_rna(v.x), tf32_rna(v.y)}; }
__device__ __forceinline__ cf ld(const float *p, int64_t plane, int64_t o) {
    return cf{p[o], p[o + plane]};
}
__device__ __forceinline__ void st(float *p, int64_t plane, int64_t o, cf v) {
    p[o] = v.x;
    p[o + plane] = v.y;
}

// Planar FP32 storage for the cluster kernels (LU panels, triangular solves,
// products with a few vectors).
struct Planar {
    typedef cf V;
    typedef float S;
    typedef float Scale;
    struct Mat {
        float *A;
        int64_t lda, plane, sA;
    };
    static __device__ __forceinline__ V zero() { return fmk(0.f, 0.f); }
    static __device__ __forceinline__ V load(const Mat &m, int64_t b, int64_t row, int64_t col) {
        return ld(m.A + b * m.sA, m.plane, col * m.lda + row);
    }
    static __device__ __forceinline__ void store(const Mat &m, int64_t b, int64_t row,
                                                 int64_t col, V v) {
        st(m.A + b * m.sA, m.plane, col * m.lda + row, v);
    }
    static __device__ __forceinline__ S mag(V v) { return fabsf(v.x) + fabsf(v.y); }
    static __device__ __forceinline__ V rcp(V v) { return frcp(v); }
    static __device__ __forceinline__ V mul(V a, V b) { return fmul(a, b); }
    static __device__ __forceinline__ V fms(V a, V b, V c) { return ffms(a, b, c); }
    static __device__ __forceinline__ V fma(V a, V b, V c) {
        c.x = fmaf(a.x, b.x, c.x);
        c.x = fmaf(-a.y, b.y, c.x);
        c.y = fmaf(a.x, b.y, c.y);
        c.y = fmaf(a.y, b.x, c.y);
        return c;
    }
    static __device__ __forceinline__ V add(V a, V b) { return fmk(a.x + b.x, a.y + b.y); }
    static __device__ __forceinline__ V sub(V a, V b) { return fmk(a.x - b.x, a.y - b.y); }
    static __device__ __forceinline__ V rnd(V v) { return rna(v); }   // L and U are stored as TF32
    static __device__ __forceinline__ void push(uint32_t addr, V v) {
        asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y)
                     : "memory");
    }
    static __device__ __forceinline__ void push_s(uint32_t addr, S v) {
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
    }
    static __device__ __forceinline__ V shfl(V v, int l) {
        return fmk(__shfl_sync(0xffffffffu, v.x, l), __shfl_sync(0xffffffffu, v.y, l));
    }
    static __device__ __forceinline__ V shfl_xor(V v, int o) {
        return fmk(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
    }
};

// Triangular solves: the 64-row diagonal blocks are solved through the
// precomputed inverses of their two 32-row halves (dinv: diag_inv_kernel).
struct PlanarTri : Planar {
    typedef Planar::Mat Mat;
    // staged diagonal block: inverse of the first half, the block below it,
    // inverse of the second half, each column by column in solve order
    static constexpr int DELEMS = 3 * 32 * 32;
    // two thread groups with a block row each: against one group with two block
    // rows per thread, 12 columns (whose diagonal solves get a warp each) take
    // 0.240 instead of 0.277 ms, 1 and 4 columns 1 to 3 % less
    static constexpr int P = 1, H = 2, THREADS = trc::GROUP * H;
    // 16 entries of one row, four columns apart
    static __device__ __forceinline__ void load16(const Mat &m, int64_t b, int row, int col,
                                                  V (&t)[16]) {
        const float *re = m.A + b * m.sA + col * m.lda + row, *im = re + m.plane;
        const int64_t step = 4 * m.lda;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            t[k] = fmk(*re, *im);
            re += step;
            im += step;
        }
    }
    static __device__ __forceinline__ void stage(V *D, const Mat &A, const float *dinv, int64_t b,
                                                 int n, int blk, bool lower, int tid) {
        const int nb32 = (n + 31) / 32;
        const int h0 = lower ? 0 : 1, h1 = 1 - h0;       // physical halves in solve order
        V v[DELEMS / THREADS];
#pragma unroll
        for (int q = 0; q < DELEMS / THREADS; ++q) {
            const int e = tid + q * THREADS, w = e >> 10, i = e & 31, t = (e >> 5) & 31;
            v[q] = fmk(0.f, 0.f);
            if (w == 1) {
                const int gr = blk * 64 + 32 * h1 + i, gc = blk * 64 + 32 * h0 + t;
                if (gr < n && gc < n) v[q] = load(A, b, gr, gc);
            } else {
                const int sb = 2 * blk + (w == 0 ? h0 : h1);
                if (sb < nb32) {
                    const float *d = dinv + ((b * nb32 + sb) * 2) * 1024 + t * 32 + i;
                    v[q] = fmk(d[0], d[1024]);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < DELEMS / THREADS; ++q) {
            const int e = tid + q * THREADS, w = e >> 10, i = e & 31, t = (e >> 5) & 31;
            D[lower ? e : w * 1024 + (31 - t) * 32 + 31 - i] = v[q];
        }
    }
    static __device__ __forceinline__ void diag(const V *D, bool, int lane, V &r0, V &r1) {
        V y = fmk(0.f, 0.f);
#pragma unroll 8
        for (int t = 0; t < 32; ++t) y = fma(D[t * 32 + lane], shfl(r0, t), y);
        r0 = y;
#pragma unroll 8
        for (int t = 0; t < 32; ++t) r1 = ffms(D[1024 + t * 32 + lane], shfl(r0, t), r1);
        y = fmk(0.f, 0.f);
#pragma unroll 8
        for (int t = 0; t < 32; ++t) y = fma(D[2048 + t * 32 + lane], shfl(r1, t), y);
        r1 = y;
    }
};

// Products with a few vectors: two rows per thread in one 8-byte load per plane
// (leading dimension, plane and stride even and the base aligned to it), or
// R = 1 for any alignment.  Sixteen loads in flight per thread: with eight the
// 12-column products of 13 to 26 matrices of 284 to 2044 rows took 0.163 ms,
// now 0.118; four rows a thread with 16-byte loads read 27 x 2884 x 2884 at 3.4
// TB/s with 4 columns, two rows read it at 5.5.
template <int RR>
struct PlanarRows : Planar {
    typedef Planar::Mat Mat;
    static constexpr int R = RR, U = 8;
    struct Scale {
        float a;
        int rnd;        // store rounded to TF32
    };
    static __device__ __forceinline__ void rows(const Mat &m, int64_t b, int64_t row, int64_t col,
                                                V (&a)[R]) {
        const float *p = m.A + b * m.sA + col * m.lda + row;
        if constexpr (R == 2) {
            const float2 x = *reinterpret_cast<const float2 *>(p);
            const float2 y = *reinterpret_cast<const float2 *>(p + m.plane);
            a[0] = fmk(x.x, y.x);
            a[1] = fmk(x.y, y.y);
        } else {
            a[0] = fmk(p[0], p[m.plane]);
        }
    }
    static __device__ __forceinline__ void out(const Mat &m, int64_t b, int64_t row, int64_t col,
                                               Scale al, V v, Scale be) {
        float *y = m.A + b * m.sA + col * m.lda + row;
        V w = fmk(al.a * v.x, al.a * v.y);
        if (be.a != 0.f) w = fmk(w.x + be.a * y[0], w.y + be.a * y[m.plane]);
        if (al.rnd) w = rna(w);
        y[0] = w.x;
        y[m.plane] = w.y;
    }
};

// LU leaf: columns [k0, k0+kb) (kb <= 32) over rows [k0, n), one CTA per matrix.
__global__ void __launch_bounds__(PANEL_THREADS) panel_kernel(int n, int k0, int kb, float *A,
                                                              int64_t lda, int64_t plane,
                                                              int64_t sA, int32_t *ipiv,
                                                              int64_t sP, int32_t *info) {
    __shared__ float red_v[PANEL_THREADS / 32];
    __shared__ int red_i[PANEL_THREADS / 32];
    __shared__ cf prow[TS];
    __shared__ int s_piv;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t b = blockIdx.x;
    A += b * sA;
    ipiv += b * sP;
    for (int jj = 0; jj < kb; ++jj) {
        const int c = k0 + jj;
        const int64_t co = (int64_t)c * lda;
        float best = -1.f;
        int bi = n;
        for (int r = c + tid; r < n; r += PANEL_THREADS) {
            float v = fabsf(A[co + r]) + fabsf(A[co + r + plane]);
            if (v > best) { best = v; bi = r; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            float ov = __shfl_xor_sync(0xffffffffu, best, o);
            int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) { red_v[wid] = best; red_i[wid] = bi; }
        __syncthreads();
        if (wid == 0) {
            best = (lane < PANEL_THREADS / 32) ? red_v[lane] : -1.f;
            bi = (lane < PANEL_THREADS / 32) ? red_i[lane] : n;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                float ov = __shfl_xor_sync(0xffffffffu, best, o);
                int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
            }
            if (lane == 0) {
                int p = bi;
                if (!(best > 0.f)) {
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
                const int64_t o = (int64_t)(k0 + cc) * lda;
                cf t = ld(A, plane, o + c);
                st(A, plane, o + c, ld(A, plane, o + p));
                st(A, plane, o + p, t);
            }
        }
        __syncthreads();
        const int rest = kb - jj;
        for (int cc = tid; cc < rest; cc += PANEL_THREADS) {
            const int64_t o = (int64_t)(c + cc) * lda + c;
            const cf u = rna(ld(A, plane, o));
            prow[cc] = u;
            st(A, plane, o, u);
        }
        __syncthreads();
        const cf pv = prow[0];
        const bool nz = (pv.x != 0.f || pv.y != 0.f);
        const cf inv = nz ? frcp(pv) : fmk(0.f, 0.f);
        for (int r = c + 1 + tid; r < n; r += PANEL_THREADS) {
            cf l = ld(A, plane, co + r);
            if (nz) l = rna(fmul(l, inv));
            st(A, plane, co + r, l);
            for (int cc = 1; cc < rest; ++cc) {
                const int64_t o = (int64_t)(c + cc) * lda + r;
                st(A, plane, o, ffms(l, prow[cc], ld(A, plane, o)));
            }
        }
        __syncthreads();
    }
}

// LU leaf in shared memory: columns [k0, k0+kb) factored as kb/SW slabs of SW
// columns.  A slab (rows cs..n-1, SW columns, planar) is loaded into shared
// memory and factored there column by column (partial pivoting on |re|+|im|,
// as the global-memory leaf); row swaps are mirrored into the panel's other
// columns in global memory.  The 4-column slabs run two CTAs per SM (batches
// above the SM count), so that instantiation is held to 64 registers.  The panel's columns right of the slab then get
// one block update: U12 = L11^{-1} A12 on the slab's SW rows, A22 -= L21 U12
// below.  Compared with the global-memory leaf, each panel column is read and
// written once per slab instead of once per column.  Dynamic shared memory:
// SW * (n - k0) * 8 bytes.
constexpr int SLAB_THREADS = 512;
// D += A B for one m16n8k8 TF32 tile (A 16 x 8 row-major, B 8 x 8 column-major,
// FP32 accumulators in the mma.sync fragment layout)
__device__ __forceinline__ void mma_tf32(float (&d)[4], const unsigned (&a)[4],
                                         const unsigned (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
template <int SW>
__global__ void __launch_bounds__(SLAB_THREADS, SW == 4 ? 2 : 1) panel_slab_kernel(int n, int k0, int kb, float *A,
                                                                 int64_t lda, int64_t plane,
                                                                 int64_t sA, int32_t *ipiv,
                                                                 int64_t sP, int32_t *info) {
    extern __shared__ float slab_sm[];
    __shared__ float red_v[SLAB_THREADS / 32];
    __shared__ int red_i[SLAB_THREADS / 32];
    __shared__ cf u12[SW][TS];
    __shared__ int slab_piv[SW];   // local pivot row of each slab column
    __shared__ int sw_dst[2 * SW], sw_src[2 * SW], sw_n;   // the slab's composed interchanges
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t b = blockIdx.x;
    A += b * sA;
    ipiv += b * sP;
    const int mmax = n - k0;
    float *sre = slab_sm, *sim = slab_sm + (int64_t)SW * mmax;
    for (int cs = k0; cs < k0 + kb; cs += SW) {
        const int ms = n - cs;                         // slab rows cs .. n-1
        // every load of a thread's rows issued before its shared-memory stores
        // (SW columns x 2 rows x 2 planes in flight per thread).  Each step's
        // pivot search is carried along (cbest, cbi): over the first column
        // here, and over column jj + 1 in step jj's update, which touches the
        // same rows of this thread in the same order as a separate search
        float cbest = -1.f;
        int cbi = ms;
        {
            const float *src = A + (int64_t)cs * lda + cs;
            for (int i0 = tid; i0 < ms; i0 += 2 * SLAB_THREADS) {
                float vr[SW][2], vi[SW][2];
#pragma unroll
                for (int j = 0; j < SW; ++j)
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int i = i0 + u * SLAB_THREADS;
                        const int64_t o = (int64_t)j * lda + i;
                        vr[j][u] = i < ms ? __ldcg(src + o) : 0.f;
                        vi[j][u] = i < ms ? __ldcg(src + o + plane) : 0.f;
                    }
#pragma unroll
                for (int j = 0; j < SW; ++j)
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int i = i0 + u * SLAB_THREADS;
                        if (i < ms) {
                            sre[j * mmax + i] = vr[j][u];
                            sim[j * mmax + i] = vi[j][u];
                        }
                    }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int i = i0 + u * SLAB_THREADS;
                    if (i < ms) {
                        const float v = fabsf(vr[0][u]) + fabsf(vi[0][u]);
                        if (v > cbest) { cbest = v; cbi = i; }
                    }
                }
            }
        }
        __syncthreads();
        for (int jj = 0; jj < SW; ++jj) {
            const int c = cs + jj;
            float best = cbest;
            int bi = cbi;
            cbest = -1.f;
            cbi = ms;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
            }
            if (lane == 0) { red_v[wid] = best; red_i[wid] = bi; }
            // two barriers per step: (A) the partial maxima are visible and
            // every row update of the previous step is done; warp 0 then
            // picks the pivot and, one lane per slab column, swaps the pivot
            // row into place and stores its U entries as TF32; (B) the pivot
            // row is ready for the update.  The update's end needs no barrier
            // of its own: the next step's (A) follows it
            __syncthreads();
            if (wid == 0) {
                best = (lane < SLAB_THREADS / 32) ? red_v[lane] : -1.f;
                bi = (lane < SLAB_THREADS / 32) ? red_i[lane] : ms;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
                    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
                }
                // every lane holds the same (best, bi) after the butterfly
                const int ip = (best > 0.f) ? bi : jj;
                if (lane == 0) {
                    if (!(best > 0.f) && info && info[b] == 0) info[b] = c + 1;
                    slab_piv[jj] = ip;
                    ipiv[c] = cs + ip;
                }
                if (lane < SW) {
                    const int j = lane;
                    if (ip != jj) {
                        float t = sre[j * mmax + jj];
                        sre[j * mmax + jj] = sre[j * mmax + ip];
                        sre[j * mmax + ip] = t;
                        t = sim[j * mmax + jj];
                        sim[j * mmax + jj] = sim[j * mmax + ip];
                        sim[j * mmax + ip] = t;
                    }
                    if (j >= jj) {
                        sre[j * mmax + jj] = tf32_rna(sre[j * mmax + jj]);
                        sim[j * mmax + jj] = tf32_rna(sim[j * mmax + jj]);
                    }
                }
            }
            __syncthreads();
            const cf pv = fmk(sre[jj * mmax + jj], sim[jj * mmax + jj]);
            const bool nz = (pv.x != 0.f || pv.y != 0.f);
            const cf inv = nz ? frcp(pv) : fmk(0.f, 0.f);
            for (int i = jj + 1 + tid; i < ms; i += SLAB_THREADS) {
                cf l = fmk(sre[jj * mmax + i], sim[jj * mmax + i]);
                if (nz) l = rna(fmul(l, inv));
                sre[jj * mmax + i] = l.x;
                sim[jj * mmax + i] = l.y;
                for (int j = jj + 1; j < SW; ++j) {
                    const cf u = fmk(sre[j * mmax + jj], sim[j * mmax + jj]);
                    cf a = fmk(sre[j * mmax + i], sim[j * mmax + i]);
                    a = ffms(l, u, a);
                    sre[j * mmax + i] = a.x;
                    sim[j * mmax + i] = a.y;
                    if (j == jj + 1) {
                        const float v = fabsf(a.x) + fabsf(a.y);
                        if (v > cbest) { cbest = v; cbi = i; }
                    }
                }
            }
        }
        __syncthreads();
        {
            float *dst = A + (int64_t)cs * lda + cs;
            for (int i = tid; i < ms; i += SLAB_THREADS)
#pragma unroll
                for (int j = 0; j < SW; ++j) {
                    dst[(int64_t)j * lda + i] = sre[j * mmax + i];
                    dst[(int64_t)j * lda + i + plane] = sim[j * mmax + i];
                }
        }
        // the slab's SW row interchanges, applied to the panel's other columns:
        // warp 0 composes them (lane t holds touched row P and the original row
        // V whose value ends there) into at most 2 SW (destination, source)
        // pairs, then every other column is one gather and one scatter
        if (wid == 0) {
            int P = -1, V = -1, np = 0;
            for (int jj = 0; jj < SW; ++jj) {
                const int r2 = slab_piv[jj];
                unsigned m = __ballot_sync(0xffffffffu, P == jj);
                const int ia = m ? __ffs(m) - 1 : np;
                if (!m) {
                    if (lane == np) P = V = jj;
                    ++np;
                }
                m = __ballot_sync(0xffffffffu, P == r2);
                const int ib = m ? __ffs(m) - 1 : np;
                if (!m) {
                    if (lane == np) P = V = r2;
                    ++np;
                }
                const int va = __shfl_sync(0xffffffffu, V, ia);
                const int vb = __shfl_sync(0xffffffffu, V, ib);
                if (lane == ia) V = vb;
                if (lane == ib) V = va;
            }
            const bool keep = lane < np && V != P;
            const unsigned mk = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                const int at = __popc(mk & ((1u << lane) - 1u));
                sw_dst[at] = P;
                sw_src[at] = V;
            }
            if (lane == 0) sw_n = __popc(mk);
        }
        __syncthreads();
        {
            const int m = sw_n;
            for (int cc = tid; cc < kb; cc += SLAB_THREADS) {
                const int col = k0 + cc;
                if (col >= cs && col < cs + SW) continue;
                const int64_t o = (int64_t)col * lda + cs;
                cf vals[2 * SW];
                for (int t = 0; t < m; ++t) vals[t] = ld(A, plane, o + sw_src[t]);
                for (int t = 0; t < m; ++t) st(A, plane, o + sw_dst[t], vals[t]);
            }
        }
        __syncthreads();
        const int c1 = cs + SW, R = k0 + kb - c1;
        if (R > 0) {
            // U12 = L11^{-1} A12 (unit lower SW x SW from the slab's top rows)
            for (int q = tid; q < R; q += SLAB_THREADS) {
                const int64_t o = (int64_t)(c1 + q) * lda + cs;
                cf x[SW];
#pragma unroll
                for (int r = 0; r < SW; ++r) x[r] = ld(A, plane, o + r);
#pragma unroll
                for (int r = 1; r < SW; ++r)
#pragma unroll
                    for (int t = 0; t < r; ++t)
                        x[r] = ffms(fmk(sre[t * mmax + r], sim[t * mmax + r]), x[t], x[r]);
#pragma unroll
                for (int r = 0; r < SW; ++r) {
                    x[r] = rna(x[r]);
                    st(A, plane, o + r, x[r]);
                    u12[r][q] = x[r];
                }
            }
            __syncthreads();
            // A22 -= L21 U12 on rows cs+SW .. n-1.  8-column slabs: TF32
            // tensor-core tiles (mma.sync m16n8k8, FP32 accumulation); L21 and
            // U12 hold TF32 values, so every product is exact as in the FMA
            // loop.  One warp per 16-row x 8-column tile; real and imaginary
            // parts as  Cr += Lr (-Ur) + Li Ui,  Ci += Lr (-Ui) + Li (-Ur).
            // Measured on LUs of 2884 x 2884 matrices: -15 % for this phase
            // with 8-column slabs, +34 % with 4-column ones (K = 4 padded to
            // 8), which keep the FMA loop.
            if constexpr (SW == 8) {
                const int g = lane >> 2, t4 = lane & 3;
                const int nrt = (ms - SW + 15) / 16, nqt = (R + 7) / 8;
                for (int tile = wid; tile < nrt * nqt; tile += SLAB_THREADS / 32) {
                    const int tr = tile / nqt, q0 = 8 * (tile - tr * nqt);
                    const int r0 = SW + 16 * tr + g, r1 = r0 + 8;
                    unsigned ar[4], ai[4], bur[2], bui[2], buin[2];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int r = (e & 1) ? r1 : r0, k = t4 + 4 * (e >> 1);
                        const bool ok = r < ms && k < SW;
                        ar[e] = ok ? __float_as_uint(sre[k * mmax + r]) : 0u;
                        ai[e] = ok ? __float_as_uint(sim[k * mmax + r]) : 0u;
                    }
                    const int qb = q0 + g;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int k = t4 + 4 * e;
                        const bool ok = k < SW && qb < R;
                        const cf u = ok ? u12[k][qb] : fmk(0.f, 0.f);
                        bur[e] = __float_as_uint(-u.x);
                        bui[e] = __float_as_uint(u.y);
                        buin[e] = __float_as_uint(-u.y);
                    }
                    float cr[4], ci[4];
                    float *pc[4];
                    bool okc[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int r = (e & 2) ? r1 : r0, q = q0 + 2 * t4 + (e & 1);
                        okc[e] = r < ms && q < R;
                        pc[e] = A + (int64_t)(c1 + q) * lda + cs + r;
                        cr[e] = okc[e] ? pc[e][0] : 0.f;
                        ci[e] = okc[e] ? pc[e][plane] : 0.f;
                    }
                    mma_tf32(cr, ar, bur);
                    mma_tf32(cr, ai, bui);
                    mma_tf32(ci, ar, buin);
                    mma_tf32(ci, ai, bur);
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (okc[e]) {
                            pc[e][0] = cr[e];
                            pc[e][plane] = ci[e];
                        }
                }
            } else {
            // A22 -= L21 U12 on rows cs+SW .. n-1
            // all of a row's loads issued before its stores (one memory
            // round trip per row instead of one per column)
            for (int i = SW + tid; i < ms; i += SLAB_THREADS) {
                cf l[SW];
#pragma unroll
                for (int t = 0; t < SW; ++t) l[t] = fmk(sre[t * mmax + i], sim[t * mmax + i]);
                float *col = A + (int64_t)c1 * lda + cs + i;
                for (int q0 = 0; q0 < R; q0 += 8) {
                    cf a[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q0 + q < R)
                            a[q] = fmk(col[(int64_t)(q0 + q) * lda],
                                       col[(int64_t)(q0 + q) * lda + plane]);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        if (q0 + q < R) {
#pragma unroll
                            for (int t = 0; t < SW; ++t) a[q] = ffms(l[t], u12[t][q0 + q], a[q]);
                            col[(int64_t)(q0 + q) * lda] = a[q].x;
                            col[(int64_t)(q0 + q) * lda + plane] = a[q].y;
                        }
                    }
                }
            }
            }
        }
        __syncthreads();
    }
}

// The pivots of a leaf's columns [off, off + kb) (kb <= 32) on the other columns
// [j0, j1) of its block: the interchanges, composed into a gather, and for the
// columns right of the leaf U12 = L11^-1 A12 on its rows, stored as TF32.  A row is
// rounded when it is final and the rows after it are eliminated with what is stored,
// as the panels do: the rounding of U12 then enters A - L U once, not again through
// the rows below.  Rounding the finished FP32 rows instead leaves a larger residual
// of the stored factors (random matrices, relative: n = 256 1.41e-3 against 1.01e-3,
// 512 1.70e-3 against 1.37e-3, 1024 2.10e-3 against 1.86e-3).  One CTA per 32 columns, four
// lanes per column with eight rows each.  It replaces, inside a block of 128
// columns, an interchange launch and one or more 32-row solve leaves per level
// of the recursion (about 11 launches of 5 to 10 us per block become 4).
// Latency-bound (4 to 8 us a launch).  LU of n, batch, before -> after: 2884 x 1
// 10.8 -> 9.8 ms, 2884 x 27 20.7 -> 18.9 ms, 2884 x 162 82.3 -> 81.1 ms, 1148 x 54
// 5.35 -> 4.95 ms; 284 x 1 the same (0.65 ms).  Blocks of 128 columns: what is
// left to the recursion above has products deep enough for the tensor cores.
constexpr int SSV = 32, SST = SSV + 1;
__global__ void __launch_bounds__(128) swap_solve_kernel(int off, int kb, int j0, int j1, float *A,
                                                         int64_t lda, int64_t plane, int64_t sA,
                                                         const int32_t *ipiv, int64_t sP) {
    grid_wait();
    __shared__ cf X[32][SST], L[32][SST];
    __shared__ swp::Swaps sw;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t b = blockIdx.y;
    A += b * sA;
    // columns [j0, off), then [off + kb, j1)
    const int nl = (off - j0 + SSV - 1) / SSV;
    const bool solve = (int)blockIdx.x >= nl;
    const int v0 = solve ? off + kb + ((int)blockIdx.x - nl) * SSV : j0 + (int)blockIdx.x * SSV;
    const int nv = min(SSV, (solve ? j1 : off) - v0);
    if (solve)
        for (int e = tid; e < 1024; e += 128) {
            const int r = e & 31, c = e >> 5;
            L[c][r] = (r < kb && c < r) ? ld(A, plane, (int64_t)(off + c) * lda + off + r)
                                        : fmk(0.f, 0.f);
        }
    swp::compose(sw, ipiv + b * sP + off, off, kb);
    cf t[8], u[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int e = tid + 128 * q, c = e & 31, v = e >> 5;
        const int64_t o = (int64_t)(v0 + v) * lda + off;
        const bool on = c < kb && v < nv;
        t[q] = on ? ld(A, plane, o + sw.out[c]) : fmk(0.f, 0.f);
        u[q] = on && sw.tail[c] >= 0 ? ld(A, plane, o + sw.tail[c]) : fmk(0.f, 0.f);
    }
    __syncthreads();                 // every row read: A may be written
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int e = tid + 128 * q, c = e & 31, v = e >> 5;
        const int64_t o = (int64_t)(v0 + v) * lda + off;
        if (c < kb && v < nv) {
            if (sw.tail[c] >= 0) st(A, plane, o + sw.p[c], u[q]);
            if (!solve) st(A, plane, o + c, t[q]);
        }
        X[c][v] = t[q];
    }
    if (!solve) return;
    __syncthreads();
    const int v = wid * 8 + (lane >> 2), r = lane & 3;
    cf y[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = X[4 * i + r][v];
#pragma unroll
    for (int c = 0; c < 32; ++c) {
        if (r == (c & 3)) y[c >> 2] = rna(y[c >> 2]);
        const int src = (lane & ~3) | (c & 3);
        const cf x = fmk(__shfl_sync(0xffffffffu, y[c >> 2].x, src),
                         __shfl_sync(0xffffffffu, y[c >> 2].y, src));
        if (r > (c & 3)) y[c >> 2] = ffms(L[c][4 * (c >> 2) + r], x, y[c >> 2]);
#pragma unroll
        for (int i = (c >> 2) + 1; i < 8; ++i) y[i] = ffms(L[c][4 * i + r], x, y[i]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) X[4 * i + r][v] = y[i];
    __syncthreads();
    for (int e = tid; e < kb * nv; e += 128) {
        const int c = e % kb, w = e / kb;
        st(A, plane, (int64_t)(v0 + w) * lda + off + c, X[c][w]);
    }
}

// Row / column interchanges of a pivot range.  Pivoting on these matrices
// rarely moves a row, so each CTA first compacts the range's non-trivial
// interchanges (pivot p != c) into shared memory, in order, 1024 pivots at a
// time (warp 0, ballot + popc), and its threads then apply only those to
// their own column (laswp) or row (colswp).
constexpr int SWP_CHUNK = 1024;

__device__ int compact_swaps(const int32_t *pv, int lo, int hi, int2 *list) {
    // warp 0 fills list[0..count) with (c, pv[c]) for pv[c] != c, c in [lo, hi)
    __shared__ int s_count;
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int count = 0;
        for (int c0 = lo; c0 < hi; c0 += 32) {
            const int c = c0 + lane;
            const int p = c < hi ? pv[c] : c;
            const bool f = p != c;
            const unsigned m = __ballot_sync(0xffffffffu, f);
            if (f) list[count + __popc(m & ((1u << lane) - 1u))] = make_int2(c, p);
            count += __popc(m);
        }
        if (lane == 0) s_count = count;
    }
    __syncthreads();
    const int n = s_count;
    __syncthreads();
    return n;
}

// Column segments of one interchange launch: columns [brk[i], brk[i+1])
// take the interchanges [cs[i], end) (cs[i] == end: none).
constexpr int SWP_MAXSEG = 24;
struct SwpSegs {
    int n, end;
    int brk[SWP_MAXSEG + 1];
    int cs[SWP_MAXSEG];
};

// segs != nullptr: column j takes only the interchanges of its segment's
// range (the recursive LU's fused forward + deferred backward interchanges)
__global__ void laswp_kernel(float *A, int64_t lda, int64_t plane, int64_t sA, int j0, int j1,
                             const int32_t *ipiv, int64_t sP, int c0, int c1, int forward,
                             const SwpSegs segs, int use_segs) {
    grid_wait();
    __shared__ int2 list[SWP_CHUNK];
    const int64_t b = blockIdx.y;
    const int j = j0 + blockIdx.x * blockDim.x + threadIdx.x;
    float *col = A + b * sA + (int64_t)j * lda;
    const int32_t *pv = ipiv + b * sP;
    const int nch = (c1 - c0 + SWP_CHUNK - 1) / SWP_CHUNK;
    for (int q = 0; q < nch; ++q) {
        const int ch = forward ? q : nch - 1 - q;
        const int lo = c0 + ch * SWP_CHUNK, hi = min(c1, lo + SWP_CHUNK);
        const int cnt = compact_swaps(pv, lo, hi, list);
        if (j < j1) {
            int cmin = c0;
            if (use_segs) {
                cmin = segs.end;
                for (int q = 0; q < segs.n; ++q)
                    if (j >= segs.brk[q] && j < segs.brk[q + 1]) cmin = segs.cs[q];
            }
            for (int t = 0; t < cnt; ++t) {
                const int2 e = list[forward ? t : cnt - 1 - t];
                if (e.x < cmin) continue;
                const cf x = ld(col, plane, e.x);
                st(col, plane, e.x, ld(col, plane, e.y));
                st(col, plane, e.y, x);
            }
        }
        __syncthreads();
    }
}

__global__ void colswp_kernel(float *X, int64_t ldx, int64_t plane, int64_t sX, int m,
                              const int32_t *ipiv, int64_t sP, int n) {
    __shared__ int2 list[SWP_CHUNK];
    const int64_t b = blockIdx.y;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    float *x = X + b * sX + r;
    const int32_t *pv = ipiv + b * sP;
    const int nch = (n + SWP_CHUNK - 1) / SWP_CHUNK;
    for (int q = nch - 1; q >= 0; --q) {
        const int lo = q * SWP_CHUNK, hi = min(n, lo + SWP_CHUNK);
        const int cnt = compact_swaps(pv, lo, hi, list);
        if (r < m) {
            for (int t = cnt - 1; t >= 0; --t) {
                const int2 e = list[t];
                const cf v = ld(x, plane, (int64_t)e.x * ldx);
                st(x, plane, (int64_t)e.x * ldx, ld(x, plane, (int64_t)e.y * ldx));
                st(x, plane, (int64_t)e.y * ldx, v);
            }
        }
        __syncthreads();
    }
}

// Small triangular solves (kb <= 32), same modes as the FP64 version:
// 0 left lower unit, 1 left upper non-unit, 2 right upper non-unit,
// 3 right lower unit.
__global__ void __launch_bounds__(128) trsm_small_kernel(int mode, int kb, const float *T,
                                                         int64_t ldt, int64_t planeT, int64_t sT,
                                                         float *B, int64_t ldb, int64_t planeB,
                                                         int64_t sB, int nvec) {
    __shared__ cf Ts[TS][TS + 1];
    const int64_t b = blockIdx.y;
    T += b * sT;
    B += b * sB;
    for (int e = threadIdx.x; e < TS * TS; e += blockDim.x) {
        const int r = e % TS, c = e / TS;
        Ts[r][c] = (r < kb && c < kb) ? ld(T, planeT, (int64_t)c * ldt + r)
                                      : fmk(r == c ? 1.f : 0.f, 0.f);
    }
    __syncthreads();
    // non-unit modes: keep 1 / diagonal on the diagonal, so that no thread's
    // substitution chain contains a division
    if ((mode == 1 || mode == 2) && threadIdx.x < TS) Ts[threadIdx.x][threadIdx.x] = frcp(Ts[threadIdx.x][threadIdx.x]);
    __syncthreads();
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nvec) return;
    cf x[TS];
    const bool left = mode < 2;
#pragma unroll
    for (int e = 0; e < TS; ++e)
        x[e] = (e < kb) ? ld(B, planeB, left ? (int64_t)v * ldb + e : (int64_t)e * ldb + v)
                        : fmk(0.f, 0.f);
    if (mode == 0) {
#pragma unroll
        for (int r = 1; r < TS; ++r)
#pragma unroll
            for (int c = 0; c < r; ++c) x[r] = ffms(Ts[r][c], x[c], x[r]);
    } else if (mode == 1) {
#pragma unroll
        for (int r = TS - 1; r >= 0; --r) {
#pragma unroll
            for (int c = r + 1; c < TS; ++c) x[r] = ffms(Ts[r][c], x[c], x[r]);
            x[r] = fmul(x[r], Ts[r][r]);
        }
    } else if (mode == 2) {
#pragma unroll
        for (int c = 0; c < TS; ++c) {
#pragma unroll
            for (int r = 0; r < c; ++r) x[c] = ffms(x[r], Ts[r][c], x[c]);
            x[c] = fmul(x[c], Ts[c][c]);
        }
    } else {
#pragma unroll
        for (int c = TS - 1; c >= 0; --c)
#pragma unroll
            for (int r = c + 1; r < TS; ++r) x[c] = ffms(x[r], Ts[r][c], x[c]);
    }
#pragma unroll
    for (int e = 0; e < TS; ++e)
        if (e < kb) st(B, planeB, left ? (int64_t)v * ldb + e : (int64_t)e * ldb + v, rna(x[e]));
}

// Inverses of the 128 x 128 diagonal blocks of a unit-lower (lower = 1) or
// non-unit upper (lower = 0) triangle; the last block may be short (kb < 128)
// and is padded with the identity.  The triangle sits packed in shared memory,
// its columns contiguous (66 KB, so that up to three CTAs share an SM and one's
// loads and stores run beside another's arithmetic); a warp builds columns j of
// the inverse by column-oriented substitution (T x = e_j): rows 32r + lane live
// in the lane's registers x[r], the newly final entry x_k is broadcast by a
// shuffle and subtracted, times column k of T, from the rows it feeds.  Output:
// out[b][blk][2][128][128] (planar, column-major, leading dimension 128).
// Bound by issue where blocks are many, by a warp's 132 dependent steps where
// they are few: against one CTA of 512 threads per block with the square in
// shared memory, 23 to 46 blocks 36 -> 28 us, 1242 blocks 25 % less.
constexpr int TL = 128;
constexpr int TINV_THREADS = 512;
constexpr int TINV_CPW = 4;      // columns a warp inverts together


// entry (i, k) of the triangle in shared memory, packed column by column
__device__ __forceinline__ int tri_at(bool lower, int i, int k) {
    return lower ? k * TL - k * (k + 1) / 2 + i : k * (k + 1) / 2 + i;
}

__global__ void __launch_bounds__(TINV_THREADS, 2) tri_inv_kernel(int n, int lower_, const float *A,
                                                                  int64_t lda, int64_t plane,
                                                                  int64_t sA, float *out, int nb) {
    grid_wait();
    extern __shared__ __align__(16) unsigned char tinv_smem[];
    cf *Tc = reinterpret_cast<cf *>(tinv_smem);   // [TL (TL + 1) / 2]
    __shared__ cf dinv[TL];
    const bool lower = lower_;
    const int blk = blockIdx.x;
    const int64_t b = blockIdx.y;
    const int o = blk * TL, kb = min(TL, n - o);
    A += b * sA;
    for (int e0 = threadIdx.x; e0 < TL * TL; e0 += 8 * blockDim.x) {
        cf v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int e = e0 + u * blockDim.x, i = e % TL, k = e / TL;
            const bool in = lower ? i >= k : i <= k;      // the unit diagonal is not read
            v[u] = fmk(i == k ? 1.f : 0.f, 0.f);
            if (in && i < kb && k < kb) v[u] = ld(A, plane, (int64_t)(o + k) * lda + o + i);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int e = e0 + u * blockDim.x, i = e % TL, k = e / TL;
            if (lower ? i >= k : i <= k) Tc[tri_at(lower, i, k)] = v[u];
        }
    }
    __syncthreads();
    if (!lower && threadIdx.x < TL) {
        const cf d = Tc[tri_at(false, threadIdx.x, threadIdx.x)];
        dinv[threadIdx.x] = (d.x != 0.f || d.y != 0.f) ? frcp(d) : fmk(0.f, 0.f);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int w = blockIdx.z * (blockDim.x >> 5) + (threadIdx.x >> 5);   // of TINV_THREADS / 32
    float *ob = out + ((b * nb + blk) * 2) * TL * TL;
    // Each warp solves two groups of TINV_CPW consecutive columns, group g
    // paired with group (TL / TINV_CPW - 1 - g) so every warp carries the same
    // substitution length.  The columns of a group share every step's
    // triangle loads and run as independent chains; a column whose index is
    // past the step carries zeros there (x_k = 0 above / below its unit
    // entry), so running the group's common step range is exact.
    static_assert(TL / TINV_CPW == 2 * (TINV_THREADS / 32), "two column groups per warp");
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
        const int grp = half == 0 ? w : TL / TINV_CPW - 1 - w;
        const int j0 = grp * TINV_CPW;
        cf x[TINV_CPW][4];
#pragma unroll
        for (int c = 0; c < TINV_CPW; ++c)
#pragma unroll
            for (int r = 0; r < 4; ++r) x[c][r] = fmk(32 * r + lane == j0 + c ? 1.f : 0.f, 0.f);
        if (lower) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (32 * r + 31 < j0) continue;
                for (int kk = (32 * r < j0 ? j0 - 32 * r : 0); kk < 32; ++kk) {
                    const int k = 32 * r + kk;
                    cf t[4];
#pragma unroll
                    for (int r2 = 0; r2 < 4; ++r2)
                        t[r2] = r2 >= r ? Tc[tri_at(true, 32 * r2 + lane, k)] : fmk(0.f, 0.f);
#pragma unroll
                    for (int c = 0; c < TINV_CPW; ++c) {
                        const cf xk = fmk(__shfl_sync(0xffffffffu, x[c][r].x, kk),
                                          __shfl_sync(0xffffffffu, x[c][r].y, kk));
#pragma unroll
                        for (int r2 = r; r2 < 4; ++r2)
                            if (r2 > r || lane > kk) x[c][r2] = ffms(t[r2], xk, x[c][r2]);
                    }
                }
            }
        } else {
            const int jt = j0 + TINV_CPW - 1;      // largest column of the group
#pragma unroll
            for (int r = 3; r >= 0; --r) {
                if (32 * r > jt) continue;
                for (int kk = min(31, jt - 32 * r); kk >= 0; --kk) {
                    const int k = 32 * r + kk;
                    cf t[4];
#pragma unroll
                    for (int r2 = 0; r2 < 4; ++r2)
                        t[r2] = r2 <= r ? Tc[tri_at(false, 32 * r2 + lane, k)] : fmk(0.f, 0.f);
                    const cf dk = dinv[k];
#pragma unroll
                    for (int c = 0; c < TINV_CPW; ++c) {
                        const cf xk = fmul(fmk(__shfl_sync(0xffffffffu, x[c][r].x, kk),
                                               __shfl_sync(0xffffffffu, x[c][r].y, kk)),
                                           dk);
                        if (lane == kk) x[c][r] = xk;
#pragma unroll
                        for (int r2 = 0; r2 <= r; ++r2)
                            if (r2 < r || lane < kk) x[c][r2] = ffms(t[r2], xk, x[c][r2]);
                    }
                }
            }
        }
        // stored rounded to nearest TF32, the precision the leaf GEMM reads
#pragma unroll
        for (int c = 0; c < TINV_CPW; ++c)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                ob[(j0 + c) * TL + 32 * r + lane] = tf32_rna(x[c][r].x);
                ob[TL * TL + (j0 + c) * TL + 32 * r + lane] = tf32_rna(x[c][r].y);
            }
    }
}

// Round rows [0, rows) of every column of a planar block to nearest TF32 in
// place: the right-hand sides of a left leaf, read by the tensor cores as the
// B operand (which would otherwise drop the low mantissa bits, a bias towards
// zero) and overwritten by the leaf's result right after.
// One CTA rounds RT_COLS columns of `rows` (<= 128) entries, both planes.
constexpr int RT_COLS = 8;
__global__ void __launch_bounds__(128) round_tf32_kernel(float *B, int64_t ldb, int64_t plane,
                                                         int64_t sB, int rows, int cols) {
    grid_wait();
    const int i = threadIdx.x;
    if (i >= rows) return;
    const int c0 = blockIdx.x * RT_COLS, c1 = min(cols, c0 + RT_COLS);
    float *base = B + blockIdx.y * sB + i;
#pragma unroll
    for (int c = c0; c < c1; ++c) {
        float *p = base + (int64_t)c * ldb;
        p[0] = tf32_rna(p[0]);
        p[plane] = tf32_rna(p[plane]);
    }
}

// ---------------------------------------------------------------------------
// Few-RHS triangular solves: inverses of the 32 x 32 diagonal blocks.  Then the
// flag and mbarrier waits of mnpb_wait_probe, kinds 1 and 2: bounded waits for code
// that waits on device memory or a barrier.  The solves themselves wait on
// hardware cluster barriers only and record no error.
// ---------------------------------------------------------------------------
constexpr int TB = 32;

__device__ int g_trsv_error;

__device__ __forceinline__ uint64_t gtimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ int ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// Spins (acquire loads) until *p == want, for at most `limit` ns of wall
// time; false if it gave up.
__device__ __forceinline__ bool wait_flag(const int *p, int want, uint64_t limit) {
    const uint64_t t0 = gtimer();
    while (ld_acquire(p) != want)
        if (gtimer() - t0 > limit) return false;
    return true;
}

// Inverse of each 32 x 32 diagonal block of the unit-lower (lower = 1) or
// upper (lower = 0) factor; out[b][blk][2][32][32] (planar, column-major).
__global__ void __launch_bounds__(TB) diag_inv_kernel(int n, int lower, const float *A,
                                                      int64_t lda, int64_t plane, int64_t sA,
                                                      float *out, int nb) {
    __shared__ cf T[TB][TB + 1];
    const int blk = blockIdx.x;
    const int64_t b = blockIdx.y;
    const int r0 = blk * TB, kb = min(TB, n - r0);
    A += b * sA;
    for (int c = 0; c < TB; ++c) {
        const int r = threadIdx.x;
        cf v = fmk(r == c ? 1.f : 0.f, 0.f);
        if (r < kb && c < kb) {
            const bool in = lower ? (r > c) : (r <= c);
            if (in) v = ld(A, plane, (int64_t)(r0 + c) * lda + r0 + r);
            else v = (lower && r == c) ? fmk(1.f, 0.f) : fmk(0.f, 0.f);
        }
        T[r][c] = v;
    }
    __syncthreads();
    // column t of the inverse: solve T x = e_t
    const int t = threadIdx.x;
    cf x[TB];
#pragma unroll
    for (int e = 0; e < TB; ++e) x[e] = fmk(e == t ? 1.f : 0.f, 0.f);
    if (lower) {
#pragma unroll
        for (int r = 1; r < TB; ++r)
#pragma unroll
            for (int c = 0; c < r; ++c) x[r] = ffms(T[r][c], x[c], x[r]);
    } else {
#pragma unroll
        for (int r = TB - 1; r >= 0; --r) {
#pragma unroll
            for (int c = r + 1; c < TB; ++c) x[r] = ffms(T[r][c], x[c], x[r]);
            x[r] = fmul(x[r], frcp(T[r][r]));
        }
    }
    float *o = out + ((b * nb + blk) * 2) * TB * TB;
#pragma unroll
    for (int e = 0; e < TB; ++e) {
        o[t * TB + e] = x[e].x;
        o[TB * TB + t * TB + e] = x[e].y;
    }
}

__device__ __forceinline__ uint32_t s_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void sbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ bool sbar_wait(uint32_t bar, uint32_t parity, uint64_t limit) {
    const uint64_t t0 = gtimer();
    while (true) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (gtimer() - t0 > limit) return false;
    }
}
__global__ void set_identity_kernel(float *W, int64_t ldw, int64_t plane, int64_t sW, int n) {
    const int64_t b = blockIdx.z;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if (i >= n) return;
    float *w = W + b * sW + (int64_t)j * ldw + i;
    w[0] = (i == j) ? 1.f : 0.f;
    w[plane] = 0.f;
}

}  // namespace

// ---------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------
Ctx::Ctx(cudaStream_t s_, int batch_, float *work_, int64_t work_bytes_)
    : s(s_), batch(batch_), work(work_), work_bytes(work_bytes_) {}

int gemm(Ctx &c, int m, int n, int k, float alpha, CMatF A, CMatF B, float beta, CMatF C,
         bool round_out, bool a_tf32) {
    if (m <= 0 || n <= 0) return MNPB_OK;
    if (k <= 0) {
        if (beta == 1.f) return MNPB_OK;
        set_error("f32 gemm: k = 0 with beta != 1 is not supported");
        return MNPB_EINVAL;
    }
    if (n <= 16) {
        ProfScope ps(c.s, PC_SGEMM, 8.0 * (double)m * k * c.batch);   // bytes of A streamed
        prof_tag("M=%d N=%d K=%d B=%d", m, n, k, c.batch);
        // vector loads where A allows them and the row blocks (split eightfold
        // along k at most) still give every SM two CTAs
        const bool pairs = m % 2 == 0 && A.ld % 2 == 0 && A.plane % 2 == 0 && A.stride % 2 == 0 &&
                           ((uintptr_t)A.p & 7) == 0 &&
                           (int64_t)ceil_div(m, skn::ROWT * 2) * c.batch * skn::MAXC >=
                               2 * device_sms();
        const Planar::Mat a{A.p, A.ld, A.plane, A.stride}, x{B.p, B.ld, B.plane, B.stride},
            y{C.p, C.ld, C.plane, C.stride};
        const int rnd = round_out ? 1 : 0;
        if (pairs)
            return skn::run<PlanarRows<2>>(c.s, m, n, k, c.batch, {alpha, rnd}, a, x, {beta, 0}, y);
        return skn::run<PlanarRows<1>>(c.s, m, n, k, c.batch, {alpha, rnd}, a, x, {beta, 0}, y);
    }
    return tc::cgemm_tf32(c.s, m, n, k, c.batch, alpha, A, B, beta, C, c.work, c.work_bytes,
                          round_out, a_tf32);
}

static int trsm_small(Ctx &c, int mode, int kb, CMatF T, CMatF B, int nvec) {
    if (nvec <= 0 || kb <= 0) return MNPB_OK;
    dim3 grid(ceil_div(nvec, 128), c.batch);
    ProfScope ps(c.s, PC_TRSM, 4.0 * kb * kb * (double)nvec * c.batch);
    prof_tag("mode=%d kb=%d nvec=%d B=%d", mode, kb, nvec, c.batch);
    trsm_small_kernel<<<grid, 128, 0, c.s>>>(mode, kb, T.p, T.ld, T.plane, T.stride, B.p, B.ld,
                                             B.plane, B.stride, nvec);
    MNPB_LAUNCH_CHECK("trsm_small_kernel(f32)");
    return MNPB_OK;
}

static int dev_sms() { return device_sms(); }

static int split_point(int n) {
    int h = n / 2;
    h = (h / TS) * TS;
    return h < TS ? TS : h;
}

// Triangular solves with many right-hand sides, recursive: split the
// triangle, solve one half, update the other half's right-hand sides with a
// tensor-core GEMM, solve the other half.  Two leaf kinds:
//  * 32-row leaves on CUDA cores (trsm_small) with splits at multiples of 32;
//  * when there are at least TL right-hand sides and the workspace holds
//    the inverses of the triangle's 128 x 128 diagonal blocks, 128-row
//    leaves applied as one tensor-core GEMM with the block's inverse (splits
//    at multiples of 128).  The leaf GEMM overwrites its own right-hand
//    sides: for a left solve (inverse as A, the RHS rows as B, C = B) each
//    output tile is a single 128-row tile whose columns no other tile reads,
//    and its epilogue runs after all of its loads; for a right solve the RHS
//    block is A and is copied into the packed operand before the GEMM.
//  mode 0 left lower unit, 1 left upper non-unit, 2 right upper non-unit,
//  3 right lower unit.
struct InvSet {
    const float *p;   // tri_inv_kernel output of the whole triangle
    int nb;           // 128-blocks of that triangle
};

static CMatF inv_block(const InvSet &iv, int blk) {
    return CMatF{(float *)iv.p + (int64_t)blk * 2 * TL * TL, TL, (int64_t)TL * TL,
                 (int64_t)iv.nb * 2 * TL * TL};
}

static int split_tl(int n) {
    int h = n / 2;
    h = (h / TL) * TL;
    return h < TL ? TL : h;
}

// `fresh`: B still holds the caller's right-hand side (not TF32); otherwise
// every update that wrote it stored its output rounded to nearest TF32, so a
// leaf reads it as an exact tensor-core operand without a rounding pass.
static int trsm_rec(Ctx &c, int mode, int n, int m, CMatF T, CMatF B, const InvSet *iv,
                    int blk0, bool fresh = true) {
    if (!iv && n <= TS) return trsm_small(c, mode, n, T, B, m);
    if (iv && n <= TL) {
        const CMatF I = inv_block(*iv, blk0);
        if (mode >= 2) {
            // right leaf: A is the right-hand-side block; packed with rounding
            // while fresh, read in place once the updates have rounded it
            if (fresh) return gemm(c, m, n, n, 1.f, B, I, 0.f, B, true);
            return gemm(c, m, n, n, 1.f, B, I, 0.f, B, true, true);
        }
        if (fresh) {
            ProfScope ps(c.s, PC_PACK, 16.0 * (double)n * m * c.batch);   // bytes read + written
            prof_tag("round n=%d m=%d B=%d", n, m, c.batch);
            MNPB_TRY(launch_chained("round_tf32_kernel", round_tf32_kernel,
                                    dim3(ceil_div(m, RT_COLS), c.batch), dim3(TL), 0, c.s, 1, B.p,
                                    B.ld, B.plane, B.stride, n, m));
        }
        return gemm(c, n, m, n, 1.f, I, B, 0.f, B, true, true);
    }
    const int n1 = iv ? split_tl(n) : split_point(n);
    const int blk1 = blk0 + n1 / TL;
    // the A operand of every update is TF32 already: a factor block (stored
    // rounded by the LU) or right-hand-side rows a leaf has finished (stored
    // rounded), so the tensor cores read it in place.  With the block
    // inverses (iv) the updates store their output rounded to TF32 as well,
    // for the leaves that read it next.
    const bool rnd = iv != nullptr;
    switch (mode) {
    case 0:
        MNPB_TRY(trsm_rec(c, 0, n1, m, T, B, iv, blk0, fresh));
        MNPB_TRY(gemm(c, n - n1, m, n1, -1.f, T.sub(n1, 0), B, 1.f, B.sub(n1, 0), rnd, true));
        return trsm_rec(c, 0, n - n1, m, T.sub(n1, n1), B.sub(n1, 0), iv, blk1, fresh && !rnd);
    case 1:
        MNPB_TRY(trsm_rec(c, 1, n - n1, m, T.sub(n1, n1), B.sub(n1, 0), iv, blk1, fresh));
        MNPB_TRY(gemm(c, n1, m, n - n1, -1.f, T.sub(0, n1), B.sub(n1, 0), 1.f, B, rnd, true));
        return trsm_rec(c, 1, n1, m, T, B, iv, blk0, fresh && !rnd);
    case 2:
        MNPB_TRY(trsm_rec(c, 2, n1, m, T, B, iv, blk0, fresh));
        MNPB_TRY(gemm(c, m, n - n1, n1, -1.f, B, T.sub(0, n1), 1.f, B.sub(0, n1), rnd, true));
        return trsm_rec(c, 2, n - n1, m, T.sub(n1, n1), B.sub(0, n1), iv, blk1, fresh && !rnd);
    default:
        MNPB_TRY(trsm_rec(c, 3, n - n1, m, T.sub(n1, n1), B.sub(0, n1), iv, blk1, fresh));
        MNPB_TRY(gemm(c, m, n1, n - n1, -1.f, B.sub(0, n1), T.sub(n1, 0), 1.f, B, rnd, true));
        return trsm_rec(c, 3, n1, m, T, B, iv, blk0, fresh && !rnd);
    }
}

// Inverses of the TL x TL diagonal blocks of a triangle.  The columns of a block
// are spread over four or two CTAs while those fit the SMs at three each.
static int tri_inv(Ctx &c, int n, bool lower, CMatF T, float *inv, int nb) {
    constexpr int SMEM = TL * (TL + 1) / 2 * (int)sizeof(cf);
    MNPB_TRY(smem_opt_in(tri_inv_kernel, SMEM, "tri_inv_kernel"));
    const int64_t blocks = (int64_t)nb * c.batch, room = 3 * dev_sms();
    const int parts = 4 * blocks <= room ? 4 : 2 * blocks <= room ? 2 : 1;
    ProfScope ps(c.s, PC_TRSM, 8.0 * TL * TL * TL / 3.0 * nb * c.batch);
    prof_tag("tri_inv n=%d B=%d %s", n, c.batch, lower ? "L" : "U");
    return launch_chained("tri_inv_kernel", tri_inv_kernel, dim3(nb, c.batch, parts),
                          dim3(TINV_THREADS / parts), SMEM, c.s, 1, n, lower ? 1 : 0, T.p, T.ld,
                          T.plane, T.stride, inv, nb);
}

// Packed-operand bytes of the largest GEMM trsm_rec issues with 128-leaves.
static int64_t trsm_pack_bytes(int mode, int n, int m, int batch) {
    const int big = n - split_tl(n) > TL ? n - split_tl(n) : TL;
    return mode < 2 ? tc::cgemm_tf32_workspace(big, big, batch)
                    : tc::cgemm_tf32_workspace(m, big, batch);
}

static int trsm(Ctx &c, int mode, int n, int m, CMatF T, CMatF B) {
    if (n <= 0 || m <= 0) return MNPB_OK;
    const int nb = ceil_div(n, TL);
    const int64_t inv_bytes = ((int64_t)c.batch * nb * 2 * TL * TL * 4 + 255) / 256 * 256;
    const int64_t keep = (c.work_bytes - inv_bytes) / 256 * 256;
    if (n <= TS || m < TL || keep < trsm_pack_bytes(mode, n, m, c.batch))
        return trsm_rec(c, mode, n, m, T, B, nullptr, 0);
    float *inv = (float *)((char *)c.work + keep);
    MNPB_TRY(tri_inv(c, n, mode == 0 || mode == 3, T, inv, nb));
    Ctx c2(c.s, c.batch, c.work, keep);
    const InvSet iv{inv, nb};
    return trsm_rec(c2, mode, n, m, T, B, &iv, 0);
}

// ---- inverse of an LU factorisation: A^-1 = U^-1 L^-1 P^T ---------------------
// Copy of each matrix's n x n diagonal-block inverse (planar, ld TL) into X.
__global__ void copy_inv_block_kernel(int n, const float *__restrict__ inv, int64_t sinv,
                                      float *X, int64_t ldx, int64_t plane, int64_t sX) {
    const int64_t b = blockIdx.z;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (i >= n) return;
    const float *src = inv + b * sinv + (int64_t)j * TL + i;
    float *dst = X + b * sX + (int64_t)j * ldx + i;
    dst[0] = src[0];
    dst[plane] = src[(int64_t)TL * TL];
}

// X <- L^-1 for the unit lower factor in T, with X holding the identity on
// entry: the rows of an identity column above its diagonal stay zero, so
// X11 = L11^-1 (recursively), X21 = -L22^-1 (L21 X11) (one product and one
// general solve with n1 right-hand sides), X22 = L22^-1 (recursively), and a
// leaf is the stored inverse of its diagonal block -- a quarter fewer flops
// than solving against the full identity.
static int trsm_llu_eye_rec(Ctx &c, int n, CMatF T, CMatF X, const InvSet &iv, int blk0) {
    if (n <= TL) {
        const CMatF I = inv_block(iv, blk0);
        dim3 grid(ceil_div(n, 128), n, c.batch);
        copy_inv_block_kernel<<<grid, 128, 0, c.s>>>(n, I.p, I.stride, X.p, X.ld, X.plane,
                                                     X.stride);
        MNPB_LAUNCH_CHECK("copy_inv_block_kernel");
        return MNPB_OK;
    }
    const int n1 = split_tl(n);
    const int blk1 = blk0 + n1 / TL;
    MNPB_TRY(trsm_llu_eye_rec(c, n1, T, X, iv, blk0));
    MNPB_TRY(gemm(c, n - n1, n1, n1, -1.f, T.sub(n1, 0), X, 0.f, X.sub(n1, 0), true, true));
    MNPB_TRY(trsm_rec(c, 0, n - n1, n1, T.sub(n1, n1), X.sub(n1, 0), &iv, blk1, false));
    return trsm_llu_eye_rec(c, n - n1, T.sub(n1, n1), X.sub(n1, n1), iv, blk1);
}

int lu_inverse(Ctx &c, int n, CMatF LU, const int32_t *ipiv, int64_t sP, CMatF X) {
    MNPB_TRY(set_identity(c, n, X));
    const int nb = ceil_div(n, TL);
    const int64_t inv_bytes = ((int64_t)c.batch * nb * 2 * TL * TL * 4 + 255) / 256 * 256;
    const int64_t keep = (c.work_bytes - inv_bytes) / 256 * 256;
    if (n <= TL || keep < trsm_pack_bytes(0, n, n, c.batch)) {
        // no room for the block inverses: the plain getrs on the permuted identity
        MNPB_TRY(laswp(c, X, 0, n, ipiv, sP, 0, n, true));
        MNPB_TRY(trsm_llu(c, n, n, LU, X));
        return trsm_lun(c, n, n, LU, X);
    }
    float *inv = (float *)((char *)c.work + keep);
    MNPB_TRY(tri_inv(c, n, true, LU, inv, nb));
    Ctx c2(c.s, c.batch, c.work, keep);
    MNPB_TRY(trsm_llu_eye_rec(c2, n, LU, X, InvSet{inv, nb}, 0));
    MNPB_TRY(trsm_lun(c, n, n, LU, X));
    // X <- X P^T: the row interchanges of the factorisation, as column
    // interchanges in reverse order
    dim3 grid(ceil_div(n, 128), c.batch);
    ProfScope ps(c.s, PC_SWAP, 0.0);
    colswp_kernel<<<grid, 128, 0, c.s>>>(X.p, X.ld, X.plane, X.stride, n, ipiv, sP, n);
    MNPB_LAUNCH_CHECK("colswp_kernel(f32)");
    return MNPB_OK;
}

int trsm_llu(Ctx &c, int n, int m, CMatF L, CMatF B) { return trsm(c, 0, n, m, L, B); }
int trsm_lun(Ctx &c, int n, int m, CMatF U, CMatF B) { return trsm(c, 1, n, m, U, B); }
int trsm_run(Ctx &c, int n, int m, CMatF U, CMatF B) { return trsm(c, 2, n, m, U, B); }
int trsm_rlu(Ctx &c, int n, int m, CMatF L, CMatF B) { return trsm(c, 3, n, m, L, B); }

int laswp(Ctx &c, CMatF A, int j0, int j1, const int32_t *ipiv, int64_t sP, int c0, int c1,
          bool forward) {
    if (j1 <= j0 || c1 <= c0) return MNPB_OK;
    dim3 grid(ceil_div(j1 - j0, 128), c.batch);
    ProfScope ps(c.s, PC_SWAP, 0.0);
    SwpSegs none{};
    return launch_chained("laswp_kernel(f32)", laswp_kernel, grid, dim3(128), 0, c.s, 1, A.p, A.ld,
                          A.plane, A.stride, j0, j1, ipiv, sP, c0, c1, forward ? 1 : 0, none, 0);
}

// One launch of the segment table t (forward order): columns [t.brk[0],
// t.brk[t.n]), interchanges from the smallest segment start to t.end.
static int laswp_segs(Ctx &c, CMatF A, const int32_t *ipiv, int64_t sP, const SwpSegs &t) {
    if (t.n == 0) return MNPB_OK;
    int c0 = t.end;
    for (int q = 0; q < t.n; ++q) c0 = min(c0, t.cs[q]);
    const int j0 = t.brk[0], j1 = t.brk[t.n];
    if (j1 <= j0 || t.end <= c0) return MNPB_OK;
    dim3 grid(ceil_div(j1 - j0, 128), c.batch);
    ProfScope ps(c.s, PC_SWAP, 0.0);
    return launch_chained("laswp_kernel(f32, segments)", laswp_kernel, grid, dim3(128), 0, c.s, 1,
                          A.p, A.ld, A.plane, A.stride, j0, j1, ipiv, sP, c0, t.end, 1, t, 1);
}

// append segment [j0, j1) -> interchanges [cs, t.end) to table t
static int seg_push(SwpSegs &t, int j0, int j1, int cs) {
    if (j1 <= j0) return MNPB_OK;
    if (t.n >= SWP_MAXSEG) {
        set_error("getrf: interchange segment table full");
        return MNPB_EINVAL;
    }
    if (t.n == 0) t.brk[0] = j0;
    if (t.brk[t.n] != j0) {               // gap: nothing owed there
        t.cs[t.n] = t.end;
        t.brk[++t.n] = j0;
        if (t.n >= SWP_MAXSEG) {
            set_error("getrf: interchange segment table full");
            return MNPB_EINVAL;
        }
    }
    t.cs[t.n] = cs;
    t.brk[++t.n] = j1;
    return MNPB_OK;
}

// One LU leaf: columns [off, off + w) (w <= 32) over rows [off, n).
static int leaf(Ctx &c, int n, int off, int w, CMatF A, int32_t *ipiv, int64_t sP,
                int32_t *info) {
    ProfScope ps(c.s, PC_PANEL, 8.0 * w * w * (double)(n - off) * c.batch / 2);
    prof_tag("off=%d w=%d B=%d", off, w, c.batch);
    const Planar::Mat mat{A.p, A.ld, A.plane, A.stride};
    int C, threads;
    // registers of a cluster while that runs in one wave: one row per
    // thread if it does, two otherwise (LU of 2884 matrices: 1 16.4 ->
    // 10.7 ms, 8 19.5 -> 14.1, 27 24.7 -> 21.2).  More matrices keep one
    // CTA each and the slab in shared memory, whose pivot steps are longer
    // but leave no second wave (54: 33.2 against 34.0, 162: 83 against 91)
    if (lup::panel_shape(n - off, 1, C, threads) && (int64_t)C * c.batch <= dev_sms())
        return lup::launch_panel<Planar, TS, 1>(c.s, n, off, w, mat, ipiv, sP, info, c.batch,
                                                C, threads);
    if (lup::panel_shape(n - off, 2, C, threads) && (int64_t)C * c.batch <= dev_sms())
        return lup::launch_panel<Planar, TS, 2>(c.s, n, off, w, mat, ipiv, sP, info, c.batch,
                                                C, threads);
    MNPB_TRY(smem_opt_in(panel_slab_kernel<8>, 200 * 1024, "panel_slab_kernel<8>"));
    MNPB_TRY(smem_opt_in(panel_slab_kernel<4>, 200 * 1024, "panel_slab_kernel<4>"));
    // more matrices than SMs: 4-column slabs, half the shared memory, so
    // that two CTAs share an SM and the batch runs in one wave
    const int64_t slab8 = (int64_t)8 * (n - off) * 8, slab4 = slab8 / 2;
    if (c.batch > dev_sms() && w % 4 == 0 && w <= TS && slab4 <= 100 * 1024) {
        panel_slab_kernel<4><<<c.batch, SLAB_THREADS, (size_t)slab4, c.s>>>(
            n, off, w, A.p, A.ld, A.plane, A.stride, ipiv, sP, info);
        MNPB_LAUNCH_CHECK("panel_slab_kernel<4>(f32)");
        return MNPB_OK;
    }
    if (w % 8 == 0 && w <= TS && slab8 <= 200 * 1024) {
        panel_slab_kernel<8><<<c.batch, SLAB_THREADS, (size_t)slab8, c.s>>>(
            n, off, w, A.p, A.ld, A.plane, A.stride, ipiv, sP, info);
        MNPB_LAUNCH_CHECK("panel_slab_kernel(f32)");
        return MNPB_OK;
    }
    if (lup::panel_shape(n - off, 2, C, threads))
        return lup::launch_panel<Planar, TS, 2>(c.s, n, off, w, mat, ipiv, sP, info, c.batch,
                                                C, threads);
    panel_kernel<<<c.batch, PANEL_THREADS, 0, c.s>>>(n, off, w, A.p, A.ld, A.plane, A.stride,
                                                     ipiv, sP, info);
    MNPB_LAUNCH_CHECK("panel_kernel(f32)");
    return MNPB_OK;
}

// Blocks of up to LB columns are factored leaf by leaf (right-looking), wider
// ones by halves.
constexpr int LB = 128;
static int block_getrf(Ctx &c, int n, int off, int w, CMatF A, int32_t *ipiv, int64_t sP,
                       int32_t *info) {
    const int end = off + w;
    for (int c0 = off; c0 < end; c0 += TS) {
        const int kb = min(TS, end - c0), c1 = c0 + kb;
        MNPB_TRY(leaf(c, n, c0, kb, A, ipiv, sP, info));
        if (w == kb) break;
        {
            ProfScope ps(c.s, PC_SWAP, 0.0);
            const int strips = ceil_div(c0 - off, SSV) + ceil_div(end - c1, SSV);
            MNPB_TRY(launch_chained("swap_solve_kernel", swap_solve_kernel, dim3(strips, c.batch),
                                    dim3(128), 0, c.s, 1, c0, kb, off, end, A.p, A.ld, A.plane,
                                    A.stride, ipiv, sP));
        }
        // L21 and U12 are stored rounded to TF32: read in place
        MNPB_TRY(gemm(c, n - c1, end - c1, kb, -1.f, A.sub(c1, c0), A.sub(c0, c1), 1.f,
                      A.sub(c1, c1), false, true));
    }
    return MNPB_OK;
}

// Factor columns [off, off+w) over rows [off, n) of the full matrix A;
// pivots are absolute row indices.  The backward interchanges this node's
// columns still owe (its right half's pivots on its left half, and what its
// right half owes) are returned in `owed` (pivots up to off + w) instead of
// applied: the caller applies them in its next interchange launch, together
// with its own forward interchanges, before anything reads these columns.
static int rgetrf(Ctx &c, int n, int off, int w, CMatF A, int32_t *ipiv, int64_t sP,
                  int32_t *info, SwpSegs &owed) {
    owed.n = 0;
    owed.end = off + w;
    if (w <= LB) return block_getrf(c, n, off, w, A, ipiv, sP, info);
    const int w1 = split_tl(w);
    SwpSegs pl;
    MNPB_TRY(rgetrf(c, n, off, w1, A, ipiv, sP, info, pl));
    // one launch: what the left half owes (pivots up to off + w1) and the
    // left half's pivots on the right half's columns
    SwpSegs t = pl;
    MNPB_TRY(seg_push(t, off + w1, off + w, off));
    MNPB_TRY(laswp_segs(c, A, ipiv, sP, t));
    MNPB_TRY(trsm_llu(c, w1, w - w1, A.sub(off, off), A.sub(off, off + w1)));
    // L21 is stored rounded to TF32 by the panels: read in place
    MNPB_TRY(gemm(c, n - off - w1, w - w1, w1, -1.f, A.sub(off + w1, off),
                  A.sub(off, off + w1), 1.f, A.sub(off + w1, off + w1), false, true));
    SwpSegs pr;
    MNPB_TRY(rgetrf(c, n, off + w1, w - w1, A, ipiv, sP, info, pr));
    // owed: the right half's pivots on the left half's columns, and what the
    // right half owes (both up to off + w)
    MNPB_TRY(seg_push(owed, off, off + w1, off + w1));
    for (int q = 0; q < pr.n; ++q) MNPB_TRY(seg_push(owed, pr.brk[q], pr.brk[q + 1], pr.cs[q]));
    return MNPB_OK;
}

int getrf(Ctx &c, int n, CMatF A, int32_t *ipiv, int64_t sP, int32_t *info) {
    SwpSegs owed;
    MNPB_TRY(rgetrf(c, n, 0, n, A, ipiv, sP, info, owed));
    return laswp_segs(c, A, ipiv, sP, owed);
}

int getrs(Ctx &c, int n, int nrhs, CMatF LU, const int32_t *ipiv, int64_t sP, CMatF B) {
    MNPB_TRY(laswp(c, B, 0, nrhs, ipiv, sP, 0, n, true));
    MNPB_TRY(trsm_llu(c, n, nrhs, LU, B));
    return trsm_lun(c, n, nrhs, LU, B);
}

int right_solve(Ctx &c, int n, int m, CMatF LU, const int32_t *ipiv, int64_t sP, CMatF B) {
    MNPB_TRY(trsm_run(c, n, m, LU, B));
    MNPB_TRY(trsm_rlu(c, n, m, LU, B));
    dim3 grid(ceil_div(m, 128), c.batch);
    ProfScope ps(c.s, PC_SWAP, 0.0);
    colswp_kernel<<<grid, 128, 0, c.s>>>(B.p, B.ld, B.plane, B.stride, m, ipiv, sP, n);
    MNPB_LAUNCH_CHECK("colswp_kernel(f32)");
    return MNPB_OK;
}

// ---- few-RHS solves ---------------------------------------------------------
int64_t diag_inv_floats(int n, int batch) { return (int64_t)batch * ceil_div(n, TB) * 2 * TB * TB; }

int diag_inv(Ctx &c, int n, CMatF LU, float *invL, float *invU) {
    const int nb = ceil_div(n, TB);
    dim3 grid(nb, c.batch);
    ProfScope ps(c.s, PC_TRSM, 0.0);
    diag_inv_kernel<<<grid, TB, 0, c.s>>>(n, 1, LU.p, LU.ld, LU.plane, LU.stride, invL, nb);
    MNPB_LAUNCH_CHECK("diag_inv_kernel(L)");
    diag_inv_kernel<<<grid, TB, 0, c.s>>>(n, 0, LU.p, LU.ld, LU.plane, LU.stride, invU, nb);
    MNPB_LAUNCH_CHECK("diag_inv_kernel(U)");
    return MNPB_OK;
}

template <int NC>
static int getrs_few_nc(Ctx &c, int n, int m, const trc::Groups &gr, CMatF LU,
                        const int32_t *ipiv, int64_t sP, const float *invL, const float *invU,
                        CMatF B, int C) {
    const Planar::Mat A{LU.p, LU.ld, LU.plane, LU.stride}, X{B.p, B.ld, B.plane, B.stride};
    const bool ride = trc::Smem<PlanarTri, NC>::composes(n);
    if (!ride) {
        Ctx ce(c.s, gr.per, c.work, c.work_bytes);
        for (int g = 0; g < gr.groups; ++g) {
            CMatF Bg = B;
            Bg.p += g * gr.X;
            MNPB_TRY(laswp(ce, Bg, 0, m, ipiv + g * gr.P, sP, 0, n, true));
        }
    }
    ProfScope ps(c.s, PC_TRSV, 8.0 * (double)n * n * gr.per * gr.groups);   // both triangles
    prof_tag("n=%d m=%d B=%d C=%d", n, m, gr.per * gr.groups, C);
    MNPB_TRY((trc::launch_trsv<PlanarTri, NC>(c.s, true, true, n, m, gr, A, invL, X,
                                              ride ? ipiv : nullptr, sP, C)));
    return trc::launch_trsv<PlanarTri, NC>(c.s, false, false, n, m, gr, A, invU, X, nullptr, 0, C);
}

// 1: done (status in rc), 0: too many columns
static int getrs_few_groups(Ctx &c, int n, int m, const trc::Groups &gr, CMatF LU,
                            const int32_t *ipiv, int64_t sP, const float *invL,
                            const float *invU, CMatF B, int &rc) {
    if (m > 16) return 0;
    const int64_t units = (int64_t)gr.per * gr.groups;
    // the widest instance whose right-hand sides fit in shared memory; fewer
    // columns per cluster (and the triangle read once for each) beyond that
#define MNPB_FEW(NC)                                                                         \
    if (const int C = trc::cluster_size<PlanarTri, NC>(n, units * ceil_div(m, NC))) {        \
        rc = getrs_few_nc<NC>(c, n, m, gr, LU, ipiv, sP, invL, invU, B, C);                  \
        return 1;                                                                            \
    }
    if (m > 8) MNPB_FEW(12);
    if (m > 4) MNPB_FEW(8);
    if (m > 1) MNPB_FEW(4);
    MNPB_FEW(1);
#undef MNPB_FEW
    return 0;
}

int getrs_few(Ctx &c, int n, int m, CMatF LU, const int32_t *ipiv, int64_t sP,
              const float *invL, const float *invU, CMatF B) {
    const trc::Groups gr{c.batch, 1, 0, 0, 0, 0};
    int rc = MNPB_OK;
    if (getrs_few_groups(c, n, m, gr, LU, ipiv, sP, invL, invU, B, rc)) return rc;
    return getrs(c, n, m, LU, ipiv, sP, B);
}

int getrs_few_pair(Ctx &c, int n, int m, CMatF LU, const float *LU2, const int32_t *ipiv,
                   const int32_t *ipiv2, int64_t sP, const float *invL, const float *invU,
                   int64_t inv2, CMatF B, int64_t b2) {
    const trc::Groups gr{c.batch, 2, LU2 - LU.p, inv2, b2, ipiv2 - ipiv};
    int rc = MNPB_OK;
    if (getrs_few_groups(c, n, m, gr, LU, ipiv, sP, invL, invU, B, rc)) return rc;
    MNPB_TRY(getrs(c, n, m, LU, ipiv, sP, B));
    CMatF L2 = LU, B2 = B;
    L2.p = (float *)LU2;
    B2.p += b2;
    return getrs(c, n, m, L2, ipiv2, sP, B2);
}

// Failure-path probe of the two wait helpers above: kind 1 spins with
// wait_flag on a zeroed flag for the value 1 (which nothing writes), kind 2
// waits with sbar_wait on an mbarrier that expects one arrival and never gets
// it.  Each gives up after `limit_ns`, records code 9 in the error word and
// returns.
__global__ void trsv_wait_probe_kernel(int kind, const int *flag, uint64_t limit_ns) {
    __shared__ __align__(8) uint64_t bar;
    bool ok;
    if (kind == 1) {
        ok = wait_flag(flag, 1, limit_ns);
    } else {
        const uint32_t b = s_u32(&bar);
        sbar_init(b, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        ok = sbar_wait(b, 0, limit_ns);
    }
    if (!ok) atomicCAS(&g_trsv_error, 0, 9);
}

int trsv_wait_probe(cudaStream_t s, int kind, int *flag, uint64_t limit_ns) {
    if (cudaMemsetAsync(flag, 0, sizeof(int), s) != cudaSuccess) {
        set_error("trsv_wait_probe: cannot clear the flag");
        return MNPB_ECUDA;
    }
    trsv_wait_probe_kernel<<<1, 1, 0, s>>>(kind, flag, limit_ns);
    MNPB_LAUNCH_CHECK("trsv_wait_probe_kernel");
    return MNPB_OK;
}

int trsv_error_read_and_clear(cudaStream_t s, int *code) {
    int v = 0, z = 0;
    if (cudaMemcpyFromSymbolAsync(&v, g_trsv_error, sizeof(int), 0, cudaMemcpyDeviceToHost, s) !=
            cudaSuccess ||
        cudaMemcpyToSymbolAsync(g_trsv_error, &z, sizeof(int), 0, cudaMemcpyHostToDevice, s) !=
            cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
        set_error("trsv: cannot read the error word");
        return MNPB_ECUDA;
    }
    *code = v;
    return MNPB_OK;
}

int set_identity(Ctx &c, int n, CMatF W) {
    dim3 grid(ceil_div(n, 128), n, c.batch);
    set_identity_kernel<<<grid, 128, 0, c.s>>>(W.p, W.ld, W.plane, W.stride, n);
    MNPB_LAUNCH_CHECK("set_identity_kernel(f32)");
    return MNPB_OK;
}

}  // namespace f32
}  // namespace mnpb

using namespace mnpb;

extern "C" int64_t mnpb_f32_workspace(int64_t n, int64_t batch) {
    // packed-A buffer of the largest tensor-core GEMM the recursions issue
    return tc::cgemm_tf32_workspace((int)n, (int)n, (int)batch);
}

extern "C" int mnpb_getrf_c32p(void *stream, int64_t n, int64_t batch, float *A, int64_t ld,
                               int64_t plane, int64_t stride, int32_t *piv, int64_t pstride,
                               int32_t *info, void *work, int64_t work_bytes) {
    clear_error();
    MNPB_REQUIRE(n > 0 && batch > 0 && batch < 65536 && ld >= n, "getrf_c32p: bad sizes");
    MNPB_REQUIRE(A && piv && work, "getrf_c32p: null pointer");
    MNPB_REQUIRE(ld % 4 == 0 && plane % 4 == 0 && stride % 4 == 0 && ((uintptr_t)A & 15) == 0,
                 "getrf_c32p: ld, plane and stride must be multiples of 4 floats and A 16-byte "
                 "aligned");
    f32::Ctx c(as_stream(stream), (int)batch, (float *)work, work_bytes);
    return f32::getrf(c, (int)n, tc::CMatF{A, ld, plane, stride}, piv, pstride, info);
}

extern "C" int mnpb_getri_c32p(void *stream, int64_t n, int64_t batch, const float *LU,
                               int64_t ld, int64_t plane, int64_t stride, const int32_t *piv,
                               int64_t pstride, float *X, int64_t ldx, int64_t planeX,
                               int64_t xstride, void *work, int64_t work_bytes) {
    clear_error();
    MNPB_REQUIRE(n > 0 && batch > 0 && ld >= n && ldx >= n, "getri_c32p: bad sizes");
    MNPB_REQUIRE(ld % 4 == 0 && plane % 4 == 0 && stride % 4 == 0 && ldx % 4 == 0 &&
                     planeX % 4 == 0 && xstride % 4 == 0 && ((uintptr_t)LU & 15) == 0 &&
                     ((uintptr_t)X & 15) == 0,
                 "getri_c32p: leading dimensions, planes and strides must be multiples of 4 "
                 "floats and base pointers 16-byte aligned");
    MNPB_REQUIRE(LU && piv && X && work, "getri_c32p: null pointer");
    MNPB_REQUIRE(work_bytes >= mnpb_f32_workspace(n, batch), "getri_c32p: workspace too small");
    f32::Ctx c(as_stream(stream), (int)batch, (float *)work, work_bytes);
    return f32::lu_inverse(c, (int)n, tc::CMatF{(float *)LU, ld, plane, stride}, piv, pstride,
                           tc::CMatF{X, ldx, planeX, xstride});
}

extern "C" int mnpb_getrs_c32p(void *stream, int64_t n, int64_t batch, int64_t nrhs,
                               const float *LU, int64_t ld, int64_t plane, int64_t stride,
                               const int32_t *piv, int64_t pstride, float *B, int64_t ldb,
                               int64_t planeB, int64_t bstride, void *work, int64_t work_bytes) {
    clear_error();
    MNPB_REQUIRE(n > 0 && batch > 0 && nrhs > 0 && ld >= n && ldb >= n, "getrs_c32p: bad sizes");
    MNPB_REQUIRE(ld % 4 == 0 && plane % 4 == 0 && stride % 4 == 0 && ldb % 4 == 0 &&
                     planeB % 4 == 0 && bstride % 4 == 0 && ((uintptr_t)LU & 15) == 0 &&
                     ((uintptr_t)B & 15) == 0,
                 "getrs_c32p: leading dimensions, planes and strides must be multiples of 4 "
                 "floats and base pointers 16-byte aligned");
    MNPB_REQUIRE(LU && piv && B && work, "getrs_c32p: null pointer");
    f32::Ctx c(as_stream(stream), (int)batch, (float *)work, work_bytes);
    return f32::getrs(c, (int)n, (int)nrhs, tc::CMatF{(float *)LU, ld, plane, stride}, piv,
                      pstride, tc::CMatF{B, ldb, planeB, bstride});
}

// ---------------------------------------------------------------------------
// Failure-path probe of the bounded device waits (see the header).
// ---------------------------------------------------------------------------
#include "tc_gemm.cuh"

extern "C" int mnpb_wait_probe(void *stream, int32_t kind, int64_t limit_ns, int32_t *flag) {
    using namespace mnpb;
    clear_error();
    MNPB_REQUIRE(kind >= 0 && kind <= 2, "wait_probe: kind must be 0, 1 or 2");
    MNPB_REQUIRE(limit_ns > 0 && limit_ns <= 2000000000ll, "wait_probe: limit_ns in (0, 2e9]");
    MNPB_REQUIRE(kind != 1 || flag, "wait_probe: kind 1 needs a device int");
    cudaStream_t s = as_stream(stream);
    int code = 0;
    if (kind == 0) {
        MNPB_TRY(tc::wait_probe(s, (uint64_t)limit_ns));
        MNPB_TRY(tc::tc_error_read_and_clear(s, &code));
    } else {
        MNPB_TRY(f32::trsv_wait_probe(s, kind, (int *)flag, (uint64_t)limit_ns));
        MNPB_TRY(f32::trsv_error_read_and_clear(s, &code));
    }
    if (code) {
        set_error("wait_probe: the %s wait gave up after %lld ns (error word %d)",
                  kind == 0 ? "tensor-core mbarrier" : kind == 1 ? "triangular-solve flag"
                                                                 : "triangular-solve mbarrier",
                  (long long)limit_ns, code);
        return MNPB_ETIMEOUT;
    }
    return MNPB_OK;
}
