// Complex GEMM on the 5th-generation tensor cores (tcgen05, sm_100a), TF32
// inputs with FP32 accumulation in tensor memory.
//
//   C = beta C + alpha A B      (planar complex FP32, column-major, batched)
//
// Cr = Ar Br - Ai Bi and Ci = Ar Bi + Ai Br are accumulated in two adjacent TMEM
// accumulators (128 lanes x BN columns each): Ar [Br | Bi] is one instruction of
// twice the width, -Ai Bi uses the negate-A bit of the instruction descriptor.
// B tiles (K x BN, K contiguous in a column-major matrix: K-major) are loaded by
// TMA straight from the caller's matrix.  A is read in place too (MN-major) where
// the caller guarantees TF32 values, else packed K-major first (a transpose) with
// round-to-nearest TF32 conversion.
//
// One CTA computes one 128 x BN output tile: warp 0 / lane 0 issues the TMA
// loads of a stage ring, warp 1 / lane 0 issues the MMAs, eight more warps read
// the accumulators and apply the epilogue to C (epi_store).  Every mbarrier wait
// is bounded: on timeout the kernel records an error, still frees its tensor
// memory and returns.
//
// Measured, one tile of K = 128: 18.2 us when four warps read C after the last
// MMA, 11.1 with eight that have C one chunk ahead, 7.3 with 32 columns; 27 x
// 2884 x 128 x 128 59 -> 50 us (bound by C's traffic, 4.8 TB/s), 1440 x 2884 x
// 1440 113 -> 84 us.  Large batched products are bound by the power limit and the
// shared-memory traffic of the operands: 27 x 1440 x 1440 x 1440 1191 -> 1168 us
// (552 TFLOP/s), most of it from the wide instruction's fewer reads of A.
#include "common.cuh"
#include "tc_gemm.cuh"

#include <cuda.h>
#include <mutex>

namespace mnpb {
namespace tc {

constexpr int BM = 128, BK = 32;   // BK: TF32 elements per 128-byte row
// warp 0 TMA producer, warp 1 MMA issuer, warps 2..9 epilogue
constexpr int EPI_THREADS = 256, GEMM_THREADS = 64 + EPI_THREADS;
constexpr int MAX_STAGES = 4;
constexpr int TILE_A_BYTES = BM * BK * 4;   // 16 KB
template <int BN> struct Tile {
    static constexpr int B_BYTES = BN * BK * 4;
    static constexpr int STAGE_BYTES = 2 * TILE_A_BYTES + 2 * B_BYTES;   // Ar, Ai, Br, Bi
    static constexpr int TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;          // re + im accumulators
    static constexpr int MAX_ST = ((227 * 1024 - 1280) / STAGE_BYTES) < MAX_STAGES
                                      ? ((227 * 1024 - 1280) / STAGE_BYTES)
                                      : MAX_STAGES;
    static int smem_bytes(int nst) { return nst * STAGE_BYTES + 1024 + 256; }
};
constexpr uint64_t WAIT_NS = 2000000000ull;    // a wait gives up after 2 s

__device__ int g_tc_error;                     // first timeout code seen (0 = none)

// ---------------------------------------------------------------------------
// PTX helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// Bounded parity wait (`limit` ns of wall time); returns false on timeout.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity,
                                          uint64_t limit = WAIT_NS) {
    const uint64_t t0 = global_ns();
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
        if (global_ns() - t0 > limit) return false;
    }
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar,
                                            int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
        "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
// K-major operand tile in shared memory, 128-byte swizzle, 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t smem_desc_k128(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);          // start address
    d |= (uint64_t)1 << 16;                          // leading byte offset (unused, 16 B)
    d |= (uint64_t)(1024 >> 4) << 32;                // stride byte offset: 8 rows x 128 B
    d |= (uint64_t)1 << 46;                          // descriptor version (sm_100)
    d |= (uint64_t)2 << 61;                          // swizzle: 128 B
    return d;
}
// MN-major operand tile (A read straight from a column-major matrix): four
// TMA boxes of 32 M x 32 K, 4096 B apart, each K row 128 B with its four 32-B
// chunks swizzled (TMA 128B_ATOM_32B mode, descriptor layout type 1 = 128-B
// swizzle on a 32-B base).  Leading byte offset: the 4096-B step between
// 32-element M groups; stride byte offset: the 512-B step between 4-row K
// groups.  One MMA (K = 8) reads 8 K rows = 1024 B from addr.
__device__ __forceinline__ uint64_t smem_desc_mn128_32b(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);          // start address
    d |= (uint64_t)(4096 >> 4) << 16;               // leading byte offset: M group step
    d |= (uint64_t)(512 >> 4) << 32;                // stride byte offset: 4-row K group step
    d |= (uint64_t)1 << 46;                          // descriptor version (sm_100)
    d |= (uint64_t)1 << 61;                          // layout: 128-B swizzle, 32-B atoms
    return d;
}
// Instruction descriptor: TF32 x TF32 -> F32, B K-major, A K-major (a_mn = false)
// or MN-major, M = 128, N = bn.
__host__ __device__ constexpr uint32_t idesc_tf32(bool neg_a, int bn, bool a_mn = false) {
    return (1u << 4)                    // D format F32
         | (2u << 7) | (2u << 10)       // A, B format TF32
         | ((neg_a ? 1u : 0u) << 13)    // negate A
         | ((a_mn ? 1u : 0u) << 15)     // A major-ness: 1 = MN-major
         | ((uint32_t)(bn >> 3) << 17)  // N / 8
         | ((uint32_t)(BM >> 4) << 24); // M / 16
}
__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
        : "memory");
}
__device__ __forceinline__ void fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
        "[%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

struct Epi {
    float *C;
    int64_t ldc, planeC, strideC;
    float alpha, beta;
    int M, N, ktiles;
    int round_out;   // 1: store C rounded to nearest TF32
};

__device__ __forceinline__ float rna_tf32(float v) {
    uint32_t t;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(t) : "f"(v));
    return __uint_as_float(t);
}

// Epilogue of one tile, eight warps: warp w reads TMEM lanes 32 (w % 4) .., its
// rows, and two warps of a lane quadrant take alternate chunks of CH columns.
// Bound by the latency of reading C, so a chunk's C is loaded a chunk ahead,
// the first one before the accumulators are waited for.
constexpr int CH = 16;   // columns per TMEM load (keeps the epilogue's registers low)

__device__ __forceinline__ void epi_fetch(const Epi &ep, const float *Cr, int row, int col,
                                          float (&cr)[CH], float (&ci)[CH]) {
    if (ep.beta == 0.f) return;
    const int ncol = row < ep.M ? min(CH, ep.N - col) : 0;
    const float *p = Cr + (int64_t)col * ep.ldc + row;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        cr[c] = c < ncol ? p[(int64_t)c * ep.ldc] : 0.f;
        ci[c] = c < ncol ? p[(int64_t)c * ep.ldc + ep.planeC] : 0.f;
    }
}

template <int BN>
__device__ __forceinline__ void epi_store(const Epi &ep, float *Cr, int row, int n0, int half,
                                          uint32_t d_re, uint32_t lane_base, float (&cr)[CH],
                                          float (&ci)[CH]) {
#pragma unroll 1
    for (int c0 = half * CH; c0 < BN; c0 += 2 * CH) {
        float vr[CH], vi[CH];
        tmem_ld16(d_re + lane_base + c0, vr);
        tmem_ld16(d_re + BN + lane_base + c0, vi);
        if (ep.beta != 0.f) {
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                vr[c] = fmaf(ep.beta, cr[c], ep.alpha * vr[c]);
                vi[c] = fmaf(ep.beta, ci[c], ep.alpha * vi[c]);
            }
            if (c0 + 2 * CH < BN) epi_fetch(ep, Cr, row, n0 + c0 + 2 * CH, cr, ci);
        } else {
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                vr[c] *= ep.alpha;
                vi[c] *= ep.alpha;
            }
        }
        if (ep.round_out) {
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                vr[c] = rna_tf32(vr[c]);
                vi[c] = rna_tf32(vi[c]);
            }
        }
        const int ncol = row < ep.M ? min(CH, ep.N - (n0 + c0)) : 0;
        float *p = Cr + (int64_t)(n0 + c0) * ep.ldc + row;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            if (c < ncol) {
                p[(int64_t)c * ep.ldc] = vr[c];
                p[(int64_t)c * ep.ldc + ep.planeC] = vi[c];
            }
        }
    }
}

template <int BN, bool AMN>
__global__ void __launch_bounds__(GEMM_THREADS, 2)
    cgemm_tf32_kernel(const __grid_constant__ CUtensorMap tmA,
                      const __grid_constant__ CUtensorMap tmAi,
                      const __grid_constant__ CUtensorMap tmBr,
                      const __grid_constant__ CUtensorMap tmBi, Epi ep, int STAGES) {
    using TL = Tile<BN>;
    grid_wait();
    constexpr int STAGE_BYTES = TL::STAGE_BYTES;
    constexpr int TILE_BYTES = TILE_A_BYTES;
    constexpr int TMEM_COLS = TL::TMEM_COLS;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // 1024-byte alignment for the swizzled tiles
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = (uint64_t *)(smem + STAGES * STAGE_BYTES);
    // bars[0..S): full, bars[S..2S): empty, bars[2S]: accumulator ready
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * MAX_STAGES + 1);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN, b = blockIdx.z;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&bars[s]), 1);
            mbar_init(smem_u32(&bars[STAGES + s]), 1);
        }
        mbar_init(smem_u32(&bars[2 * STAGES]), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t d_re = tmem, d_im = tmem + BN;
    const int KT = ep.ktiles;

    if (warp == 0 && lane == 0) {
        // TMA producer
        for (int kt = 0; kt < KT; ++kt) {
            const int s = kt % STAGES;
            if (kt >= STAGES) {
                if (!mbar_wait(smem_u32(&bars[STAGES + s]), ((kt / STAGES) - 1) & 1)) {
                    atomicCAS(&g_tc_error, 0, 1);
                    *abort_flag = 1;
                    break;
                }
            }
            if (*abort_flag) break;
            uint8_t *st = smem + s * STAGE_BYTES;
            const uint32_t full = smem_u32(&bars[s]);
            mbar_expect_tx(full, STAGE_BYTES);
            const int k0 = kt * BK;
            if (AMN) {
#pragma unroll
                for (int a = 0; a < BM / 32; ++a) {
                    tma_load_3d(smem_u32(st + a * 4096), &tmA, full, m0 + 32 * a, k0, b);
                    tma_load_3d(smem_u32(st + TILE_BYTES + a * 4096), &tmAi, full, m0 + 32 * a,
                                k0, b);
                }
            } else {
                tma_load_3d(smem_u32(st), &tmA, full, k0, m0, 2 * b);
                tma_load_3d(smem_u32(st + TILE_BYTES), &tmA, full, k0, m0, 2 * b + 1);
            }
            tma_load_3d(smem_u32(st + 2 * TILE_BYTES), &tmBr, full, k0, n0, b);
            tma_load_3d(smem_u32(st + 2 * TILE_BYTES + TL::B_BYTES), &tmBi, full, k0, n0, b);
        }
    } else if (warp == 1 && lane == 0) {
        // MMA issuer
        constexpr uint32_t ID = idesc_tf32(false, BN, AMN), IDN = idesc_tf32(true, BN, AMN);
        constexpr uint32_t ID2 = idesc_tf32(false, 2 * BN, AMN);
        for (int kt = 0; kt < KT; ++kt) {
            const int s = kt % STAGES;
            if (!mbar_wait(smem_u32(&bars[s]), (kt / STAGES) & 1)) {
                atomicCAS(&g_tc_error, 0, 2);
                *abort_flag = 1;
                break;
            }
            fence_after();
            const uint32_t st = smem_u32(smem + s * STAGE_BYTES);
#pragma unroll
            for (int j = 0; j < BK / 8; ++j) {      // 8 TF32 = 32 bytes per MMA
                const uint32_t off = 32 * j;
                const uint64_t ar = AMN ? smem_desc_mn128_32b(st + 1024 * j) : smem_desc_k128(st + off);
                const uint64_t ai = AMN ? smem_desc_mn128_32b(st + TILE_BYTES + 1024 * j)
                                        : smem_desc_k128(st + TILE_BYTES + off);
                const uint64_t br = smem_desc_k128(st + 2 * TILE_BYTES + off);
                const uint64_t bi = smem_desc_k128(st + 2 * TILE_BYTES + TL::B_BYTES + off);
                const uint32_t acc = (kt > 0 || j > 0) ? 1u : 0u;
                // Re(A) [Re(B) | Im(B)]: the tiles are adjacent, so are the sums
                mma_tf32(d_re, ar, br, ID2, acc);
                mma_tf32(d_re, ai, bi, IDN, 1u);
                mma_tf32(d_im, ai, br, ID, 1u);
            }
            mma_commit(smem_u32(&bars[STAGES + s]));   // frees this stage when done
        }
        // accumulator ready (or abort) -- commit tracks all MMAs issued above
        mma_commit(smem_u32(&bars[2 * STAGES]));
    }
    __syncwarp();

    if (warp >= 2) {
        const int q = warp & 3, half = (warp - 2) >> 2;
        const int row = m0 + q * 32 + lane;
        float *Cr = ep.C + (int64_t)b * ep.strideC;
        float cr[CH], ci[CH];
        epi_fetch(ep, Cr, row, n0 + half * CH, cr, ci);
        const bool acc_ok = mbar_wait(smem_u32(&bars[2 * STAGES]), 0);
        if (!acc_ok) atomicCAS(&g_tc_error, 0, 3);
        fence_after();
        if (acc_ok && *abort_flag == 0)
            epi_store<BN>(ep, Cr, row, n0, half, d_re, (uint32_t)(q * 32) << 16, cr, ci);
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(TMEM_COLS)
                     : "memory");
    }
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Persistent variant for large GEMMs: one CTA per SM walks the output tiles
// (t = blockIdx.x, blockIdx.x + gridDim.x, ...; M fastest, then N, then the
// batch).  Warp 0 issues the TMA loads of a stage ring that runs on across
// tiles, warp 1 allocates all 512 TMEM columns and issues the MMAs into two
// accumulator buffers (re + im, 2 x BN columns each), warps 2-9 drain a
// finished buffer into C (warp w owns TMEM lanes 32 (w % 4) .., two warps per
// lane quadrant on alternate column chunks, so twice the C traffic is in
// flight when the epilogue reads C) while the MMAs of the next tile fill the
// other one.  acc_full[b] (MMA -> epilogue, one commit) and acc_empty[b]
// (epilogue -> MMA, 256 arrivals) hand the buffers over.  Every wait is
// bounded as in cgemm_tf32_kernel.
template <int BN, bool AMN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    cgemm_tf32_persistent(const __grid_constant__ CUtensorMap tmA,
                          const __grid_constant__ CUtensorMap tmAi,
                          const __grid_constant__ CUtensorMap tmBr,
                          const __grid_constant__ CUtensorMap tmBi, Epi ep, int STAGES, int MT,
                          int NT, int ntiles) {
    using TL = Tile<BN>;
    grid_wait();
    constexpr int STAGE_BYTES = TL::STAGE_BYTES;
    constexpr int TILE_BYTES = TILE_A_BYTES;
    constexpr int ACC_COLS = 2 * BN;
    constexpr int TMEM_COLS = 2 * ACC_COLS;
    static_assert(TMEM_COLS <= 512, "two accumulator buffers must fit in TMEM");
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = (uint64_t *)(smem + STAGES * STAGE_BYTES);
    // bars: full [0, S), empty [S, 2S), acc_full 2S + {0,1}, acc_empty 2S + {2,3}
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * MAX_STAGES + 4);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int TPB = MT * NT;   // tiles per batch entry

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&bars[s]), 1);
            mbar_init(smem_u32(&bars[STAGES + s]), 1);
        }
        mbar_init(smem_u32(&bars[2 * STAGES + 0]), 1);
        mbar_init(smem_u32(&bars[2 * STAGES + 1]), 1);
        mbar_init(smem_u32(&bars[2 * STAGES + 2]), EPI_THREADS);
        mbar_init(smem_u32(&bars[2 * STAGES + 3]), EPI_THREADS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    const int KT = ep.ktiles;

    if (warp == 0) {
        if (lane == 0) {
            // TMA producer
            uint32_t g = 0;
            for (int t = blockIdx.x; t < ntiles && !*abort_flag; t += gridDim.x) {
                const int b = t / TPB, rem = t - b * TPB;
                const int nt = rem / MT, mt = rem - nt * MT;
                const int m0 = mt * BM, n0 = nt * BN;
                bool ok = true;
                for (int kt = 0; kt < KT; ++kt, ++g) {
                    const int s = g % STAGES;
                    if (g >= (uint32_t)STAGES &&
                        !mbar_wait(smem_u32(&bars[STAGES + s]), ((g / STAGES) - 1) & 1)) {
                        atomicCAS(&g_tc_error, 0, 1);
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    if (*abort_flag) {
                        ok = false;
                        break;
                    }
                    uint8_t *st = smem + s * STAGE_BYTES;
                    const uint32_t full = smem_u32(&bars[s]);
                    mbar_expect_tx(full, STAGE_BYTES);
                    const int k0 = kt * BK;
                    if (AMN) {
#pragma unroll
                        for (int a = 0; a < BM / 32; ++a) {
                            tma_load_3d(smem_u32(st + a * 4096), &tmA, full, m0 + 32 * a, k0, b);
                            tma_load_3d(smem_u32(st + TILE_BYTES + a * 4096), &tmAi, full,
                                        m0 + 32 * a, k0, b);
                        }
                    } else {
                        tma_load_3d(smem_u32(st), &tmA, full, k0, m0, 2 * b);
                        tma_load_3d(smem_u32(st + TILE_BYTES), &tmA, full, k0, m0, 2 * b + 1);
                    }
                    tma_load_3d(smem_u32(st + 2 * TILE_BYTES), &tmBr, full, k0, n0, b);
                    tma_load_3d(smem_u32(st + 2 * TILE_BYTES + TL::B_BYTES), &tmBi, full, k0, n0,
                                b);
                }
                if (!ok) break;
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // MMA issuer
            constexpr uint32_t ID = idesc_tf32(false, BN, AMN), IDN = idesc_tf32(true, BN, AMN);
            constexpr uint32_t ID2 = idesc_tf32(false, 2 * BN, AMN);
            uint32_t g = 0;
            int i = 0;
            for (int t = blockIdx.x; t < ntiles && !*abort_flag; t += gridDim.x, ++i) {
                const int buf = i & 1;
                if (i >= 2 && !mbar_wait(smem_u32(&bars[2 * STAGES + 2 + buf]), ((i >> 1) - 1) & 1)) {
                    atomicCAS(&g_tc_error, 0, 4);
                    *abort_flag = 1;
                    break;
                }
                fence_after();
                const uint32_t d_re = tmem + buf * ACC_COLS, d_im = d_re + BN;
                bool ok = true;
                for (int kt = 0; kt < KT; ++kt, ++g) {
                    const int s = g % STAGES;
                    if (!mbar_wait(smem_u32(&bars[s]), (g / STAGES) & 1)) {
                        atomicCAS(&g_tc_error, 0, 2);
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    fence_after();
                    const uint32_t st = smem_u32(smem + s * STAGE_BYTES);
#pragma unroll
                    for (int j = 0; j < BK / 8; ++j) {
                        const uint32_t off = 32 * j;
                        const uint64_t ar = AMN ? smem_desc_mn128_32b(st + 1024 * j)
                                                : smem_desc_k128(st + off);
                        const uint64_t ai = AMN ? smem_desc_mn128_32b(st + TILE_BYTES + 1024 * j)
                                                : smem_desc_k128(st + TILE_BYTES + off);
                        const uint64_t br = smem_desc_k128(st + 2 * TILE_BYTES + off);
                        const uint64_t bi = smem_desc_k128(st + 2 * TILE_BYTES + TL::B_BYTES + off);
                        const uint32_t acc = (kt > 0 || j > 0) ? 1u : 0u;
                        // Re(A) [Re(B) | Im(B)]: the tiles are adjacent, so are the sums
                        mma_tf32(d_re, ar, br, ID2, acc);
                        mma_tf32(d_re, ai, bi, IDN, 1u);
                        mma_tf32(d_im, ai, br, ID, 1u);
                    }
                    mma_commit(smem_u32(&bars[STAGES + s]));
                }
                mma_commit(smem_u32(&bars[2 * STAGES + buf]));
                if (!ok) break;
            }
        }
    } else {
        // epilogue warps 2..9: warp w reads TMEM lanes 32 (w % 4) .. +31 (its
        // rows), the two warps of a lane quadrant take alternate column chunks
        const int q = warp & 3;
        const int half = (warp - 2) >> 2;
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        int i = 0;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++i) {
            const int buf = i & 1;
            const int b = t / TPB, rem = t - b * TPB;
            const int nt = rem / MT, mt = rem - nt * MT;
            const int row = mt * BM + q * 32 + lane, n0 = nt * BN;
            float *Cr = ep.C + (int64_t)b * ep.strideC;
            float cr[CH], ci[CH];
            epi_fetch(ep, Cr, row, n0 + half * CH, cr, ci);
            const bool acc_ok = mbar_wait(smem_u32(&bars[2 * STAGES + buf]), (i >> 1) & 1);
            if (!acc_ok) {
                atomicCAS(&g_tc_error, 0, 3);
                *abort_flag = 1;
                break;
            }
            fence_after();
            if (*abort_flag) break;
            epi_store<BN>(ep, Cr, row, n0, half, tmem + buf * ACC_COLS, lane_base, cr, ci);
            fence_before();
            mbar_arrive(smem_u32(&bars[2 * STAGES + 2 + buf]));
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(TMEM_COLS)
                     : "memory");
    }
}

// Pack a column-major planar complex A (M x K) into K-major TF32 tiles:
// out[b][plane][Mp][Kp], zero outside M x K, round to nearest TF32.
__global__ void pack_a_tf32_kernel(const float *__restrict__ A, int64_t lda, int64_t planeA,
                                   int64_t strideA, int M, int K, int Mp, int Kp,
                                   float *__restrict__ out) {
    __shared__ float tile[32][33];
    const int b = blockIdx.z >> 1, pl = blockIdx.z & 1;
    const int mb = blockIdx.x * 32, kb = blockIdx.y * 32;
    const float *src = A + (int64_t)b * strideA + (int64_t)pl * planeA;
    // read: 32 k-columns x 32 m (m contiguous)
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int m = mb + threadIdx.x, k = kb + j;
        float v = (m < M && k < K) ? src[(int64_t)k * lda + m] : 0.f;
        uint32_t t;
        asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(t) : "f"(v));
        tile[j][threadIdx.x] = __uint_as_float(t);
    }
    __syncthreads();
    float *dst = out + ((int64_t)b * 2 + pl) * (int64_t)Mp * Kp;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int m = mb + i, k = kb + threadIdx.x;
        if (m < Mp && k < Kp) dst[(int64_t)m * Kp + k] = tile[threadIdx.x][i];
    }
}

// Same pack for 16-byte aligned operands (base, lda, plane and stride all
// multiples of 4 floats): 64 x 64 tiles, 16-byte loads and stores, four
// independent loads per thread in flight before any shared-memory traffic.
constexpr int PK = 64;
__global__ void __launch_bounds__(256) pack_a_tf32_vec_kernel(const float *__restrict__ A,
                                                              int64_t lda, int64_t planeA,
                                                              int64_t strideA, int M, int K,
                                                              int Mp, int Kp,
                                                              float *__restrict__ out) {
    __shared__ float tile[PK][PK + 1];   // tile[k][m]
    const int b = blockIdx.z >> 1, pl = blockIdx.z & 1;
    const int mb = blockIdx.x * PK, kb = blockIdx.y * PK;
    const float *src = A + (int64_t)b * strideA + (int64_t)pl * planeA;
    const int tid = threadIdx.x;
    float4 v[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int idx = tid + 256 * p, kc = idx >> 4, m = mb + 4 * (idx & 15), k = kb + kc;
        v[p] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k < K) {
            const float *s = src + (int64_t)k * lda + m;
            if (m + 3 < M) {
                v[p] = __ldg(reinterpret_cast<const float4 *>(s));
            } else {
                if (m < M) v[p].x = s[0];
                if (m + 1 < M) v[p].y = s[1];
                if (m + 2 < M) v[p].z = s[2];
            }
        }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int idx = tid + 256 * p, kc = idx >> 4, mm = 4 * (idx & 15);
        const float e[4] = {v[p].x, v[p].y, v[p].z, v[p].w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint32_t t;
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(t) : "f"(e[q]));
            tile[kc][mm + q] = __uint_as_float(t);
        }
    }
    __syncthreads();
    float *dst = out + ((int64_t)b * 2 + pl) * (int64_t)Mp * Kp;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int idx = tid + 256 * p, mr = idx >> 4, kq = 4 * (idx & 15);
        const int m = mb + mr, k = kb + kq;
        if (m < Mp && k < Kp)
            *reinterpret_cast<float4 *>(dst + (int64_t)m * Kp + k) =
                make_float4(tile[kq][mr], tile[kq + 1][mr], tile[kq + 2][mr], tile[kq + 3][mr]);
    }
}

// Failure-path probe: one thread initialises an mbarrier that expects one
// arrival, never arrives, and waits on it with mbar_wait -- the helper every
// wait of the tensor-core kernels uses -- for at most `limit_ns`.  The wait
// gives up, the error word gets code 9 as a kernel's would, and the kernel
// returns; nothing else is touched.
__global__ void wait_probe_kernel(uint64_t limit_ns) {
    __shared__ __align__(8) uint64_t bar;
    const uint32_t b = smem_u32(&bar);
    mbar_init(b, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (!mbar_wait(b, 0, limit_ns)) atomicCAS(&g_tc_error, 0, 9);
}

int wait_probe(cudaStream_t s, uint64_t limit_ns) {
    wait_probe_kernel<<<1, 1, 0, s>>>(limit_ns);
    MNPB_LAUNCH_CHECK("wait_probe_kernel");
    return MNPB_OK;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                             const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                             const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn get_encode() {
    static EncodeFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeFn)p;
    });
    return fn;
}

// 3-D FP32 map: inner dim d0 (contiguous), rows d1 (stride s1 elements),
// planes/batch d2 (stride s2 elements); box 32 x 128 x 1, 128-byte swizzle.
static int make_map(CUtensorMap *map, const float *base, uint64_t d0, uint64_t d1, uint64_t d2,
                    uint64_t s1, uint64_t s2, uint32_t box_rows,
                    CUtensorMapSwizzle swz = CU_TENSOR_MAP_SWIZZLE_128B) {
    EncodeFn enc = get_encode();
    if (!enc) {
        set_error("tc_gemm: cuTensorMapEncodeTiled unavailable");
        return MNPB_ECUDA;
    }
    if (((uintptr_t)base & 15) || ((s1 * 4) & 15) || ((s2 * 4) & 15)) {
        set_error("tc_gemm: operand not 16-byte aligned (base %p, strides %llu %llu)", base,
                  (unsigned long long)s1, (unsigned long long)s2);
        return MNPB_EINVAL;
    }
    cuuint64_t dims[3] = {d0, d1, d2};
    cuuint64_t strides[2] = {s1 * 4, s2 * 4};
    cuuint32_t box[3] = {BK, box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)base, dims, strides, box,
                     estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("tc_gemm: cuTensorMapEncodeTiled failed (%d)", (int)r);
        return MNPB_ECUDA;
    }
    return MNPB_OK;
}

int encode_map_f32(void *map, const float *base, const uint64_t dims[3],
                   const uint64_t stride_bytes[2], const uint32_t box[3], int swizzle) {
    EncodeFn enc = get_encode();
    if (!enc) {
        set_error("tma: cuTensorMapEncodeTiled unavailable");
        return MNPB_ECUDA;
    }
    if (((uintptr_t)base & 15) || (stride_bytes[0] & 15) || (stride_bytes[1] & 15)) {
        set_error("tma: operand not 16-byte aligned (base %p)", base);
        return MNPB_EINVAL;
    }
    cuuint64_t d[3] = {dims[0], dims[1], dims[2]};
    cuuint64_t st[2] = {stride_bytes[0], stride_bytes[1]};
    cuuint32_t bx[3] = {box[0], box[1], box[2]};
    cuuint32_t es[3] = {1, 1, 1};
    CUresult r = enc((CUtensorMap *)map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)base, d, st,
                     bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, (CUtensorMapSwizzle)swizzle,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("tma: cuTensorMapEncodeTiled failed (%d)", (int)r);
        return MNPB_ECUDA;
    }
    return MNPB_OK;
}

static int num_sms() { return device_sms(); }

// Launch configuration chosen by the autotuner (process-wide; the defaults
// are the hand-picked ones): the tile width used for N > 64 (64 or 128), the
// persistent kernel's threshold in tiles per SM (0: never persistent) and the
// stage count of the operand ring (0: as many as fit).  Every change bumps
// an epoch that cached launch sequences (CUDA graphs) are keyed on.
static std::atomic<int> g_cfg_bn{128}, g_cfg_persist{2}, g_cfg_stages{0};
// TF32-exact A operands are read in place (MN-major) when N >= this, else
// packed K-major first (exact for TF32 values).  Narrow products (N of one or
// two 128-column tiles) stream their tall A only once per tile column, where
// the MN-major boxes reach about half the HBM rate of the packed layout.
static std::atomic<int> g_cfg_mn_min_n{0};
static std::atomic<int64_t> g_cfg_epoch{0};

int64_t gemm_config_epoch() { return g_cfg_epoch.load(); }

int64_t cgemm_tf32_workspace(int M, int K, int batch) {
    const int64_t Mp = (M + BM - 1) / BM * BM, Kp = (K + BK - 1) / BK * BK;
    return (int64_t)batch * 2 * Mp * Kp * 4;
}

template <int BN, bool AMN>
static int launch_tf32(cudaStream_t s, const CUtensorMap &mA, const CUtensorMap &mAi,
                       const CMatF &B, int M, int N, int K, int Kp, int Mp, int batch, Epi ep) {
    using TL = Tile<BN>;
    MNPB_TRY(smem_opt_in(cgemm_tf32_kernel<BN, AMN>, TL::smem_bytes(TL::MAX_ST),
                         "cgemm_tf32_kernel"));
    CUtensorMap mBr, mBi;
    MNPB_TRY(make_map(&mBr, B.p, K, N, batch, B.ld, B.stride, BN));
    MNPB_TRY(make_map(&mBi, B.p + B.plane, K, N, batch, B.ld, B.stride, BN));
    // stages: as many as the K loop can use; the shared-memory request is at
    // least large enough that no more CTAs share an SM than fit their
    // accumulators in its 512 TMEM columns
    const int KT = Kp / BK;
    const int cst = g_cfg_stages.load(std::memory_order_relaxed);
    const int maxst = (cst >= 2 && cst < TL::MAX_ST) ? cst : TL::MAX_ST;
    const int nst = KT < maxst ? KT : maxst;
    const int max_ctas_tmem = 512 / TL::TMEM_COLS;
    int dyn = TL::smem_bytes(nst);
    const int floor_bytes = (228 * 1024) / (max_ctas_tmem + 1) + 1024;
    if (dyn < floor_bytes) dyn = floor_bytes;
    const int MT = Mp / BM, NT = (N + BN - 1) / BN;
    const int64_t ntiles = (int64_t)MT * NT * batch;
    // (narrower tiles already overlap epilogues across several CTAs per SM)
    const int persist = g_cfg_persist.load(std::memory_order_relaxed);
    if (BN == 128 && persist > 0 && ntiles >= (int64_t)persist * num_sms()) {
        // persistent: one CTA per SM, double-buffered accumulators
        MNPB_TRY(smem_opt_in(cgemm_tf32_persistent<BN, AMN>, TL::smem_bytes(TL::MAX_ST),
                             "cgemm_tf32_persistent"));
        const int pst = maxst;
        const int grid = (int)(ntiles < num_sms() ? ntiles : num_sms());
        return launch_chained("cgemm_tf32_persistent", cgemm_tf32_persistent<BN, AMN>, dim3(grid),
                              dim3(GEMM_THREADS), TL::smem_bytes(pst), s, 1, mA, mAi, mBr, mBi, ep,
                              pst, MT, NT, (int)ntiles);
    }
    dim3 grid(MT, NT, batch);
    return launch_chained("cgemm_tf32_kernel", cgemm_tf32_kernel<BN, AMN>, grid,
                          dim3(GEMM_THREADS), dyn, s, 1, mA, mAi, mBr, mBi, ep, nst);
}

template <bool AMN>
static int launch_any(cudaStream_t s, const CUtensorMap &mA, const CUtensorMap &mAi,
                      const CMatF &B, int M, int N, int K, int Kp, int Mp, int batch, Epi ep,
                      bool in_place) {
    // Narrow tiles while those are one wave: such a product is bound by one
    // tile's latency (loads of K, then its epilogue), not by the tensor cores.
    // M, N, K, matrices: 32 / 64 / 128 columns 2884, 128, 128, 1 (92 / 46 / 23
    // tiles) 7.4 / 8.8 / 11.6 us; 892, 892, 256, 1 (196 / 98 / 49) 20.0 / 12.2 /
    // 15.0; 768, 768, 768, 2 (288 / 144 / 72) 45.3 / 25.3 / 27.4; 1440, 1440,
    // 128, 1 (540 / 276 / 144) 26.3 / 16.6 / 11.8.  Not where C overwrites A:
    // one tile has to span the columns that its rows are read from.
    const int64_t rows = (int64_t)Mp / BM * batch;
    auto one_wave = [&](int bn) { return !in_place && rows * ceil_div(N, bn) <= num_sms(); };
    if (N <= 32 || one_wave(32))
        return launch_tf32<32, AMN>(s, mA, mAi, B, M, N, K, Kp, Mp, batch, ep);
    if (N <= 64 || one_wave(64) ||
        (!in_place && g_cfg_bn.load(std::memory_order_relaxed) == 64))
        return launch_tf32<64, AMN>(s, mA, mAi, B, M, N, K, Kp, Mp, batch, ep);
    return launch_tf32<128, AMN>(s, mA, mAi, B, M, N, K, Kp, Mp, batch, ep);
}

static bool aligned16(const CMatF &X) {
    return ((uintptr_t)X.p & 15) == 0 && X.ld % 4 == 0 && X.plane % 4 == 0 && X.stride % 4 == 0;
}

int cgemm_tf32(cudaStream_t s, int M, int N, int K, int batch, float alpha, CMatF A, CMatF B,
               float beta, CMatF C, float *work, int64_t work_bytes, bool round_out,
               bool a_tf32) {
    if (M <= 0 || N <= 0 || batch <= 0) return MNPB_OK;
    if (K <= 0) {
        set_error("tc_gemm: K must be positive");
        return MNPB_EINVAL;
    }
    const int Mp = (M + BM - 1) / BM * BM, Kp = (K + BK - 1) / BK * BK;
    Epi ep{C.p, C.ld, C.plane, C.stride, alpha, beta, M, N, Kp / BK, round_out ? 1 : 0};
    // narrow products of the 128-wide tile (96 < N < mn_min_n) pack A even when it
    // could be read in place; the 32/64-wide tiles and wide products read it in place
    const bool pack_narrow = N > 64 && N < g_cfg_mn_min_n.load(std::memory_order_relaxed) &&
                             work && work_bytes >= cgemm_tf32_workspace(M, K, batch);
    if (a_tf32 && aligned16(A) && !pack_narrow) {
        // A already holds TF32 values: the tensor cores read it in place (MN-major)
        CUtensorMap mAr, mAi;
        MNPB_TRY(make_map(&mAr, A.p, M, K, batch, A.ld, A.stride, 32,
                          CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B));
        MNPB_TRY(make_map(&mAi, A.p + A.plane, M, K, batch, A.ld, A.stride, 32,
                          CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B));
        ProfScope ps(s, PC_TCGEMM, 8.0 * M * N * (double)K * batch);
        prof_tag("M=%d N=%d K=%d B=%d mn", M, N, K, batch);
        return launch_any<true>(s, mAr, mAi, B, M, N, K, Kp, Mp, batch, ep, A.p == C.p);
    }
    if (work_bytes < cgemm_tf32_workspace(M, K, batch)) {
        set_error("tc_gemm: workspace too small");
        return MNPB_ENOMEM;
    }
    {
        ProfScope ps(s, PC_PACK, 8.0 * (double)M * K * batch);
        if (aligned16(A)) {
            dim3 g(Mp / PK, (Kp + PK - 1) / PK, batch * 2);
            pack_a_tf32_vec_kernel<<<g, 256, 0, s>>>(A.p, A.ld, A.plane, A.stride, M, K, Mp, Kp,
                                                     work);
            MNPB_LAUNCH_CHECK("pack_a_tf32_vec_kernel");
        } else {
            dim3 g(Mp / 32, Kp / 32, batch * 2), t(32, 8);
            pack_a_tf32_kernel<<<g, t, 0, s>>>(A.p, A.ld, A.plane, A.stride, M, K, Mp, Kp, work);
            MNPB_LAUNCH_CHECK("pack_a_tf32_kernel");
        }
    }
    CUtensorMap mA;
    MNPB_TRY(make_map(&mA, work, Kp, Mp, (uint64_t)batch * 2, Kp, (uint64_t)Mp * Kp, BM));
    ProfScope ps(s, PC_TCGEMM, 8.0 * M * N * (double)K * batch);
    prof_tag("M=%d N=%d K=%d B=%d", M, N, K, batch);
    return launch_any<false>(s, mA, mA, B, M, N, K, Kp, Mp, batch, ep, false);
}

int tc_error_read_and_clear(cudaStream_t s, int *code) {
    int v = 0, z = 0;
    if (cudaMemcpyFromSymbolAsync(&v, g_tc_error, sizeof(int), 0, cudaMemcpyDeviceToHost, s) !=
            cudaSuccess ||
        cudaMemcpyToSymbolAsync(g_tc_error, &z, sizeof(int), 0, cudaMemcpyHostToDevice, s) !=
            cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
        set_error("tc_gemm: cannot read the error word");
        return MNPB_ECUDA;
    }
    *code = v;
    return MNPB_OK;
}

}  // namespace tc
}  // namespace mnpb

using namespace mnpb;

extern "C" int64_t mnpb_cgemm_tf32_workspace(int64_t m, int64_t k, int64_t batch) {
    return tc::cgemm_tf32_workspace((int)m, (int)k, (int)batch);
}

extern "C" int mnpb_cgemm_tf32(void *stream, int64_t m, int64_t n, int64_t k, int64_t batch,
                               float alpha, const float *A, int64_t lda, int64_t planeA,
                               int64_t sA, const float *B, int64_t ldb, int64_t planeB,
                               int64_t sB, float beta, float *C, int64_t ldc, int64_t planeC,
                               int64_t sC, void *work, int64_t work_bytes) {
    clear_error();
    MNPB_REQUIRE(m >= 0 && n >= 0 && k > 0 && batch > 0 && batch < 65536,
                 "cgemm_tf32: bad sizes");
    MNPB_REQUIRE(A && B && C && work, "cgemm_tf32: null pointer");
    tc::CMatF a{(float *)A, lda, planeA, sA}, b{(float *)B, ldb, planeB, sB}, c{C, ldc, planeC, sC};
    return tc::cgemm_tf32(as_stream(stream), (int)m, (int)n, (int)k, (int)batch, alpha, a, b,
                          beta, c, (float *)work, work_bytes);
}

extern "C" int mnpb_cgemm_tf32_ex(void *stream, int64_t m, int64_t n, int64_t k, int64_t batch,
                                  float alpha, const float *A, int64_t lda, int64_t planeA,
                                  int64_t sA, const float *B, int64_t ldb, int64_t planeB,
                                  int64_t sB, float beta, float *C, int64_t ldc, int64_t planeC,
                                  int64_t sC, void *work, int64_t work_bytes, int32_t flags) {
    clear_error();
    MNPB_REQUIRE(m >= 0 && n >= 0 && k > 0 && batch > 0 && batch < 65536,
                 "cgemm_tf32_ex: bad sizes");
    MNPB_REQUIRE((flags & ~3) == 0, "cgemm_tf32_ex: unknown flag bits 0x%x", (unsigned)flags);
    const bool a_tf32 = (flags & MNPB_GEMM_A_TF32) != 0;
    MNPB_REQUIRE(A && B && C && (work || a_tf32), "cgemm_tf32_ex: null pointer");
    tc::CMatF a{(float *)A, lda, planeA, sA}, b{(float *)B, ldb, planeB, sB}, c{C, ldc, planeC, sC};
    if (a_tf32)
        MNPB_REQUIRE(((uintptr_t)A & 15) == 0 && lda % 4 == 0 && planeA % 4 == 0 && sA % 4 == 0,
                     "cgemm_tf32_ex: MNPB_GEMM_A_TF32 needs A, lda, planeA and sA aligned to "
                     "16 bytes");
    return tc::cgemm_tf32(as_stream(stream), (int)m, (int)n, (int)k, (int)batch, alpha, a, b,
                          beta, c, (float *)work, work_bytes, (flags & MNPB_GEMM_ROUND_C) != 0,
                          a_tf32);
}

extern "C" int mnpb_gemm_config_mn(int32_t mn_min_n) {
    clear_error();
    MNPB_REQUIRE(mn_min_n >= 0, "gemm_config_mn: mn_min_n must be >= 0");
    tc::g_cfg_mn_min_n.store(mn_min_n);
    tc::g_cfg_epoch.fetch_add(1);
    return MNPB_OK;
}

extern "C" int mnpb_gemm_config(int32_t bn_wide, int32_t persist_tiles_per_sm, int32_t stages) {
    clear_error();
    MNPB_REQUIRE(bn_wide == 64 || bn_wide == 128, "gemm_config: bn_wide must be 64 or 128");
    MNPB_REQUIRE(persist_tiles_per_sm >= 0 && persist_tiles_per_sm <= 64,
                 "gemm_config: persist_tiles_per_sm must be 0..64");
    MNPB_REQUIRE(stages == 0 || (stages >= 2 && stages <= 4), "gemm_config: stages 0 or 2..4");
    tc::g_cfg_bn.store(bn_wide);
    tc::g_cfg_persist.store(persist_tiles_per_sm);
    tc::g_cfg_stages.store(stages);
    tc::g_cfg_epoch.fetch_add(1);
    return MNPB_OK;
}

extern "C" int mnpb_tc_error(void *stream, int32_t *code) {
    clear_error();
    MNPB_REQUIRE(code, "tc_error: null pointer");
    int v = 0;
    MNPB_TRY(tc::tc_error_read_and_clear(as_stream(stream), &v));
    *code = v;
    return MNPB_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of mnpb_cgemm_tf32.
//
// Some callers cannot hand the library a device workspace: a host program in
// another language that binds the C ABI but owns no device allocator, a code
// whose memory pool has already claimed the whole GPU, or a loop that must not
// take the implicit device synchronisation that cudaMalloc/cudaFree imply.
// For them the only scratch this GEMM needs, the packed TF32 copy of A, is
// kept in a fixed array of this module's static device memory.  The array is
// reserved by the CUDA runtime when the module is loaded (64 MiB per device),
// whether or not this entry point is ever called.
//
// Nothing in the array has to start at zero: the pack kernel writes every
// element of the padded Mp x Kp tiles, padding included, before the GEMM
// reads them.  The error word the GEMM may set is the same one
// mnpb_cgemm_tf32 uses (read and cleared by mnpb_tc_error).
//
// There is ONE array per device: calls that may overlap in time on the same
// device (different streams, or different host threads) overwrite each
// other's packed operand and race.  Calls issued in order on one stream are
// safe.
// ---------------------------------------------------------------------------
namespace mnpb {
namespace tc {

constexpr int64_t kStaticPackBytes = int64_t(64) << 20;
static __device__ __align__(256) float g_static_pack[kStaticPackBytes / 4];

constexpr int kMaxDevices = 64;

// Device address of g_static_pack on the current device, looked up once per
// device under a lock.  (The kernels' shared-memory opt-in is made per device
// by the launch path itself, for every tile width and the persistent kernel.)
static int static_pack_scratch(float **out) {
    static std::mutex mu;
    static float *addr[kMaxDevices] = {};
    const int dev = current_device();
    if (dev < 0) {
        set_error("cgemm_tf32_noalloc: cudaGetDevice failed");
        return MNPB_ECUDA;
    }
    if (dev >= kMaxDevices) {
        set_error("cgemm_tf32_noalloc: device ordinal %d out of range", dev);
        return MNPB_EINVAL;
    }
    std::lock_guard<std::mutex> lk(mu);
    if (!addr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_static_pack);
        if (e != cudaSuccess || !p) {
            set_error("cgemm_tf32_noalloc: cudaGetSymbolAddress failed on device %d: %s", dev,
                      cudaGetErrorString(e));
            return MNPB_ECUDA;
        }
        addr[dev] = (float *)p;
    }
    *out = addr[dev];
    return MNPB_OK;
}

}  // namespace tc
}  // namespace mnpb

extern "C" int mnpb_cgemm_tf32_noalloc(void *stream, int64_t m, int64_t n, int64_t k,
                                       int64_t batch, float alpha, const float *A, int64_t lda,
                                       int64_t planeA, int64_t sA, const float *B, int64_t ldb,
                                       int64_t planeB, int64_t sB, float beta, float *C,
                                       int64_t ldc, int64_t planeC, int64_t sC) {
    clear_error();
    MNPB_REQUIRE(m >= 0 && n >= 0 && k > 0 && batch > 0 && batch < 65536,
                 "cgemm_tf32_noalloc: bad sizes");
    MNPB_REQUIRE(A && B && C, "cgemm_tf32_noalloc: null pointer");
    if (m > (int64_t(1) << 30) || k > (int64_t(1) << 30)) {
        set_error("cgemm_tf32_noalloc: m or k too large");
        return MNPB_EINVAL;
    }
    const int64_t need = tc::cgemm_tf32_workspace((int)m, (int)k, (int)batch);
    if (need > tc::kStaticPackBytes) {
        set_error("cgemm_tf32_noalloc: packed A needs %lld bytes (m=%lld k=%lld batch=%lld), "
                  "the static scratch holds %lld; use mnpb_cgemm_tf32 with a workspace",
                  (long long)need, (long long)m, (long long)k, (long long)batch,
                  (long long)tc::kStaticPackBytes);
        return MNPB_ENOMEM;
    }
    // the scratch array used is the current device's: the stream must be one of its streams
    MNPB_TRY(check_stream_device(as_stream(stream), "cgemm_tf32_noalloc"));
    float *scratch = nullptr;
    MNPB_TRY(tc::static_pack_scratch(&scratch));
    tc::CMatF a{(float *)A, lda, planeA, sA}, b{(float *)B, ldb, planeB, sB}, c{C, ldc, planeC, sC};
    return tc::cgemm_tf32(as_stream(stream), (int)m, (int)n, (int)k, (int)batch, alpha, a, b,
                          beta, c, scratch, tc::kStaticPackBytes);
}
