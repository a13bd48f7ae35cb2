// FP64 GMRES building blocks (the Krylov solver of the iterative retarded
// solver; the reference calls scipy.sparse.linalg.gmres with restart =
// min(n, maxit), mnpbem/bem/bem_iter.py:79-89).
//
//  * mnpb_gmres_arnoldi: one Arnoldi step with classical Gram-Schmidt run
//    twice (CGS2, as stable as modified Gram-Schmidt, but each pass is two
//    bandwidth-bound launches instead of j dependent dot products):
//    h = V^H w, w -= V h (twice), h_{j+1} = |w|, v_{j+1} = w / h_{j+1}.
//  * mnpb_gmres_givens: applies the previous Givens rotations to Hessenberg
//    column j, forms rotation j, updates g and reports |g_{j+1}| (the
//    residual norm of the least-squares problem), on the device.
//  * mnpb_gmres_update: back substitution R y = g, then x += V y.
//
// Vectors are complex128 of length L; the basis V is column-major with
// column stride ldv; H is column-major (ldh >= m + 1).  All arithmetic FP64.
#include "common.cuh"

namespace mnpb {
namespace gm {

constexpr int CH = 2048;   // elements per partial-sum chunk of the norms
constexpr int MAXCH = 32;  // chunks of a dot product at most
constexpr int PE = 64;     // elements per CTA of the projection (four lanes of q each)

// partial[q * nch + c] = sum over chunk c of conj(V[:, q]) w
__global__ void dots_kernel(int64_t L, int nq, const cd *__restrict__ V, int64_t ldv,
                            const cd *__restrict__ w, cd *__restrict__ partial, int nch,
                            int64_t chunk) {
    __shared__ cd sh[32];
    const int c = blockIdx.x, q = blockIdx.y;
    const int64_t e0 = (int64_t)c * chunk, e1 = min(L, e0 + chunk);
    const cd *v = V + (int64_t)q * ldv;
    cd a = cmk(0, 0);
    for (int64_t e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
        const cd x = v[e], y = w[e];
        a.x += x.x * y.x + x.y * y.y;
        a.y += x.x * y.y - x.y * y.x;
    }
    for (int o = 16; o > 0; o >>= 1) {
        a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
        a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
    }
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        cd t = cmk(0, 0);
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t = cadd(t, sh[k]);
        partial[(int64_t)q * nch + c] = t;
    }
}

// h[q] = sum_c partial[q][c] (fixed order; every CTA for itself, the first one
// keeps it), w -= V[:, 0:nq] h, and with `norms` the CTA's partial squared norm
// of the new w.  64 elements per CTA, four lanes of every fourth q each: the
// chain of products per element is a quarter as long and four times as many
// CTAs share the stream of V.  The separate launch for the sums and the one for
// the norm are gone: an Arnoldi step takes five launches instead of nine, 25 us
// instead of 45 on average over 130 vectors of 19,200 elements.
__global__ void __launch_bounds__(256) project_kernel(int64_t L, int nq, int nch,
                                                      const cd *__restrict__ V, int64_t ldv,
                                                      const cd *__restrict__ partial,
                                                      cd *__restrict__ hq, cd *__restrict__ w,
                                                      double *__restrict__ norms) {
    extern __shared__ cd sh_h[];
    __shared__ cd part[4][PE];
    __shared__ double sn[2];
    for (int q = threadIdx.x; q < nq; q += blockDim.x) {
        cd t = cmk(0, 0);
        for (int c = 0; c < nch; ++c) t = cadd(t, partial[(int64_t)q * nch + c]);
        sh_h[q] = t;
        if (blockIdx.x == 0) hq[q] = t;
    }
    __syncthreads();
    const int el = threadIdx.x & (PE - 1), ql = threadIdx.x / PE;
    const int64_t e = (int64_t)blockIdx.x * PE + el;
    cd acc = cmk(0, 0);
    if (e < L) {
#pragma unroll 4
        for (int q = ql; q < nq; q += 4) acc = cfma(V[(int64_t)q * ldv + e], sh_h[q], acc);
    }
    part[ql][el] = acc;
    __syncthreads();
    if (threadIdx.x < PE) {
        double a = 0.0;
        if (e < L) {
            cd t = cadd(cadd(part[0][el], part[1][el]), cadd(part[2][el], part[3][el]));
            t = csub(w[e], t);
            w[e] = t;
            a = t.x * t.x + t.y * t.y;
        }
        if (norms) {
            for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if ((threadIdx.x & 31) == 0) sn[threadIdx.x >> 5] = a;
        }
    }
    if (norms) {
        __syncthreads();
        if (threadIdx.x == 0) norms[blockIdx.x] = sn[0] + sn[1];
    }
}

// partial squared norms of w
__global__ void norm_kernel(int64_t L, const cd *__restrict__ w, double *__restrict__ partial) {
    __shared__ double sh[32];
    const int64_t e0 = (int64_t)blockIdx.x * CH, e1 = min(L, e0 + CH);
    double a = 0.0;
    for (int64_t e = e0 + threadIdx.x; e < e1; e += blockDim.x) a += w[e].x * w[e].x + w[e].y * w[e].y;
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += sh[k];
        partial[blockIdx.x] = t;
    }
}

// out[v] = sqrt(sum_c partial[v * nch + c])
__global__ void norm_finish_kernel(int nvec, int nch, const double *__restrict__ partial,
                                   double *out) {
    for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
        double t = 0.0;
        for (int c = 0; c < nch; ++c) t += partial[(int64_t)v * nch + c];
        out[v] = sqrt(t);
    }
}

// nrm = |w| from the partial squared norms (every CTA for itself, in one order),
// v_out = w / nrm (zero if nrm == 0: an exact breakdown); the first CTA writes
// Hcol[q] = h1[q] + h2[q] for q <= j, Hcol[j+1] = nrm_out = nrm.
__global__ void __launch_bounds__(256) finish_col_kernel(int64_t L, int j, int np,
                                                         const double *__restrict__ norms,
                                                         const cd *__restrict__ h1,
                                                         const cd *__restrict__ h2, cd *Hcol,
                                                         double *nrm_out,
                                                         const cd *__restrict__ w,
                                                         cd *__restrict__ v) {
    __shared__ double sh[8];
    double t = 0.0;
    for (int c = threadIdx.x; c < np; c += 256) t += norms[c];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
    __syncthreads();
    t = 0.0;
    for (int k = 0; k < 8; ++k) t += sh[k];
    const double s = sqrt(t);
    const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (e < L) v[e] = s > 0.0 ? cscale(w[e], 1.0 / s) : cmk(0, 0);
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            Hcol[j + 1] = cmk(s, 0.0);
            *nrm_out = s;
        }
        for (int q = threadIdx.x; q <= j; q += 256) Hcol[q] = cadd(h1[q], h2[q]);
    }
}

// Givens step j on column j of H (complex rotations, LAPACK zlartg-style
// with real cosine): apply rotations 0..j-1, form rotation j zeroing
// H[j+1, j], rotate g; out[0] = |g[j+1]|.
// The column and the rotations are staged in shared memory by the whole CTA;
// the chain of j dependent rotations then touches nothing slower (19 -> 5 us on
// average over 130 columns).
constexpr int GV_SEG = 1024;   // rotations staged at a time
__global__ void __launch_bounds__(128) givens_kernel(int j, cd *H, int64_t ldh, double *cs,
                                                     cd *sn, cd *g, double *out) {
    __shared__ cd ss[GV_SEG], hc[GV_SEG + 1];
    __shared__ double cc[GV_SEG];
    cd *h = H + (int64_t)j * ldh;
    for (int i0 = 0; i0 < j; i0 += GV_SEG) {
        const int ns = min(GV_SEG, j - i0);
        for (int i = threadIdx.x; i < ns; i += blockDim.x) {
            ss[i] = sn[i0 + i];
            cc[i] = cs[i0 + i];
        }
        for (int i = threadIdx.x; i <= ns; i += blockDim.x) hc[i] = h[i0 + i];
        __syncthreads();
        if (threadIdx.x == 0) {
            cd a = hc[0];
#pragma unroll 4
            for (int i = 0; i < ns; ++i) {
                // [c  s; -conj(s) c] [a; b]
                const cd b = hc[i + 1];
                hc[i] = cadd(cscale(a, cc[i]), cmul(ss[i], b));
                a = csub(cscale(b, cc[i]), cmul(cmk(ss[i].x, -ss[i].y), a));
            }
            hc[ns] = a;
        }
        __syncthreads();
        for (int i = threadIdx.x; i <= ns; i += blockDim.x) h[i0 + i] = hc[i];
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    const cd a = h[j], b = h[j + 1];
    const double na = hypot(a.x, a.y), nb = hypot(b.x, b.y);
    double c;
    cd s, r;
    if (nb == 0.0) {
        c = 1.0;
        s = cmk(0, 0);
        r = a;
    } else if (na == 0.0) {
        c = 0.0;
        s = cmk(b.x / nb, -b.y / nb);          // conj(b) / |b|
        r = cmk(nb, 0.0);
    } else {
        const double nrm = hypot(na, nb);
        c = na / nrm;
        const cd ph = cmk(a.x / na, a.y / na);   // a / |a|
        s = cmul(ph, cmk(b.x / nrm, -b.y / nrm));   // (a/|a|) conj(b) / nrm
        r = cscale(ph, nrm);
    }
    cs[j] = c;
    sn[j] = s;
    h[j] = r;
    h[j + 1] = cmk(0, 0);
    const cd gj = g[j];
    g[j] = cscale(gj, c);
    g[j + 1] = cmul(cmk(-s.x, s.y), gj);         // -conj(s) g_j
    out[0] = hypot(g[j + 1].x, g[j + 1].y);
}

// y = R^{-1} g (R = upper triangle of H, m x m), one CTA, column by column from
// the last; the next column is loaded while this one is subtracted (130 columns:
// 0.96 ms on one thread, 0.11 here).  Dynamic shared memory: g (m).
constexpr int BS_T = 256, BS_Q = 12;              // m < BS_T * BS_Q
__global__ void __launch_bounds__(BS_T) backsub_kernel(int m, const cd *H, int64_t ldh,
                                                       const cd *g, cd *y) {
    extern __shared__ cd bs_g[];
    __shared__ cd yi;
    for (int i = threadIdx.x; i < m; i += BS_T) bs_g[i] = g[i];
    const int nq = (m + BS_T - 1) / BS_T;
    cd col[BS_Q], nxt[BS_Q];
    auto load = [&](int i, cd (&t)[BS_Q]) {
#pragma unroll
        for (int q = 0; q < BS_Q; ++q)
            if (q < nq) {
                const int k = threadIdx.x + q * BS_T;
                t[q] = (i >= 0 && k <= i) ? H[(int64_t)i * ldh + k] : cmk(0, 0);
            }
    };
    load(m - 1, col);
    for (int i = m - 1; i >= 0; --i) {
        load(i - 1, nxt);
        __syncthreads();
        if (threadIdx.x == i % BS_T) {
            cd d = cmk(0, 0);
#pragma unroll
            for (int q = 0; q < BS_Q; ++q)
                if (q == i / BS_T) d = col[q];
            const cd v = (d.x == 0.0 && d.y == 0.0) ? cmk(0, 0) : cmul(bs_g[i], crcp(d));
            yi = v;
            y[i] = v;
        }
        __syncthreads();
        const cd v = yi;
#pragma unroll
        for (int q = 0; q < BS_Q; ++q)
            if (q < nq) {
                const int k = threadIdx.x + q * BS_T;
                if (k < i) bs_g[k] = csub(bs_g[k], cmul(col[q], v));
                col[q] = nxt[q];
            }
    }
}

// x += V[:, 0:m] y
__global__ void update_kernel(int64_t L, int m, const cd *__restrict__ V, int64_t ldv,
                              const cd *__restrict__ y, cd *__restrict__ x) {
    extern __shared__ cd sh_y[];
    for (int q = threadIdx.x; q < m; q += blockDim.x) sh_y[q] = y[q];
    __syncthreads();
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= L) return;
    cd acc = x[e];
    for (int q = 0; q < m; ++q) acc = cadd(acc, cmul(V[(int64_t)q * ldv + e], sh_y[q]));
    x[e] = acc;
}

}  // namespace gm
}  // namespace mnpb

using namespace mnpb;

static int64_t gm_chunks(int64_t L) { return (L + gm::CH - 1) / gm::CH; }
static int64_t gm_dot_chunks(int64_t L) {
    const int64_t c = gm_chunks(L);
    return c < gm::MAXCH ? c : gm::MAXCH;
}
static int64_t gm_projections(int64_t L) { return (L + gm::PE - 1) / gm::PE; }

// Scratch (bytes) for mnpb_gmres_arnoldi with basis index up to jmax.
extern "C" int64_t mnpb_gmres_workspace(int64_t L, int64_t jmax) {
    const int64_t nch = gm_dot_chunks(L);
    return (jmax + 1) * nch * 16 + 2 * (jmax + 1) * 16 + gm_projections(L) * 8 + 8 + 1024;
}

extern "C" int mnpb_gmres_arnoldi(void *stream, int64_t L, int64_t j, double *V, int64_t ldv,
                                  double *w, double *Hcol, double *nrm, void *work,
                                  int64_t work_bytes) {
    clear_error();
    MNPB_REQUIRE(L > 0 && j >= 0 && ldv >= L && j < 4096, "gmres_arnoldi: bad sizes");
    MNPB_REQUIRE(V && w && Hcol && nrm && work, "gmres_arnoldi: null pointer");
    MNPB_REQUIRE(work_bytes >= mnpb_gmres_workspace(L, j), "gmres_arnoldi: workspace too small");
    cudaStream_t s = as_stream(stream);
    const int nq = (int)j + 1;
    const int nch = (int)gm_dot_chunks(L);
    const int64_t chunk = (L + nch - 1) / nch;
    const int np = (int)gm_projections(L);
    char *wp = (char *)work;
    cd *partial = (cd *)wp;
    wp += (int64_t)nq * nch * 16;
    cd *h1 = (cd *)wp;
    cd *h2 = h1 + nq;
    double *norms = (double *)(h2 + nq);
    ProfScope ps(s, PC_GMRES, 4.0 * 16.0 * (double)L * nq);
    const size_t shq = (size_t)nq * 16;
    if (shq > 48 * 1024) {
        set_error("gmres_arnoldi: basis too large (%d vectors)", nq);
        return MNPB_EINVAL;
    }
    if (shq > 40 * 1024)   // beside the kernel's static 4 KB
        MNPB_TRY(smem_opt_in(gm::project_kernel, 48 * 1024, "project_kernel"));
    cd *hs[2] = {h1, h2};
    for (int pass = 0; pass < 2; ++pass) {
        gm::dots_kernel<<<dim3(nch, nq), 256, 0, s>>>(L, nq, (const cd *)V, ldv, (const cd *)w,
                                                     partial, nch, chunk);
        gm::project_kernel<<<np, 256, shq, s>>>(L, nq, nch, (const cd *)V, ldv, partial, hs[pass],
                                                (cd *)w, pass ? norms : nullptr);
    }
    gm::finish_col_kernel<<<(unsigned)((L + 255) / 256), 256, 0, s>>>(
        L, (int)j, np, norms, h1, h2, (cd *)Hcol, nrm, (const cd *)w,
        (cd *)V + (int64_t)(j + 1) * ldv);
    count_launch(4);
    MNPB_LAUNCH_CHECK("gmres arnoldi kernels");
    return MNPB_OK;
}

extern "C" int mnpb_gmres_givens(void *stream, int64_t j, double *H, int64_t ldh, double *cs,
                                 double *sn, double *g, double *out) {
    clear_error();
    MNPB_REQUIRE(j >= 0 && ldh >= j + 2, "gmres_givens: bad sizes");
    MNPB_REQUIRE(H && cs && sn && g && out, "gmres_givens: null pointer");
    cudaStream_t s = as_stream(stream);
    gm::givens_kernel<<<1, 128, 0, s>>>((int)j, (cd *)H, ldh, cs, (cd *)sn, (cd *)g, out);
    MNPB_LAUNCH_CHECK("givens_kernel");
    return MNPB_OK;
}

extern "C" int mnpb_gmres_update(void *stream, int64_t L, int64_t m, const double *H,
                                 int64_t ldh, const double *g, const double *V, int64_t ldv,
                                 double *y, double *x) {
    clear_error();
    MNPB_REQUIRE(L > 0 && m >= 0 && ldh >= m && ldv >= L && m < 3000, "gmres_update: bad sizes");
    if (m == 0) return MNPB_OK;
    MNPB_REQUIRE(H && g && V && y && x, "gmres_update: null pointer");
    cudaStream_t s = as_stream(stream);
    gm::backsub_kernel<<<1, gm::BS_T, (size_t)m * 16, s>>>((int)m, (const cd *)H, ldh,
                                                           (const cd *)g, (cd *)y);
    gm::update_kernel<<<(unsigned)((L + 255) / 256), 256, (size_t)m * 16, s>>>(
        L, (int)m, (const cd *)V, ldv, (const cd *)y, (cd *)x);
    count_launch(1);
    MNPB_LAUNCH_CHECK("gmres update kernels");
    return MNPB_OK;
}

// Euclidean norms of nvec vectors of L complex entries (stride ldx):
// out[v] = |x_v|, deterministic two-stage sums.  partial: nvec * ceil(L/2048)
// doubles of scratch.
extern "C" int mnpb_vec_norms(void *stream, int64_t L, int64_t nvec, const double *x,
                              int64_t ldx, double *partial, double *out) {
    clear_error();
    MNPB_REQUIRE(L > 0 && nvec > 0 && ldx >= L && x && partial && out, "vec_norms: bad arguments");
    cudaStream_t s = as_stream(stream);
    const int nch = (int)gm_chunks(L);
    for (int64_t v = 0; v < nvec; ++v)
        gm::norm_kernel<<<nch, 256, 0, s>>>(L, (const cd *)x + v * ldx, partial + v * nch);
    gm::norm_finish_kernel<<<1, 128, 0, s>>>((int)nvec, nch, partial, out);
    MNPB_LAUNCH_CHECK("vec_norms kernels");
    return MNPB_OK;
}
