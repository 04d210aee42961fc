// Toeplitz row filter on the 5th-generation tensor cores (tcgen05), split BF16.
//
// Y[R][k] = du * sum_m X[R][m] h[k-m+nu-1] is a GEMM  D[M x N] = A[M x K] B[K x N]
// with M = rows*views sinogram rows, N = K = nu.  Each float32 operand is split into
// bf16 hi + lo parts and D = A_hi B_hi + A_hi B_lo + A_lo B_hi is accumulated in
// float32 in tensor memory (the dropped A_lo B_lo term is ~2^-16 relative).
// Replaces the row convolution of Mgfbp.ConvolveSgmAndKernel (run_mgfbp.py:1030-1046).
//
// Operand layout.  A and B^T are stored pre-tiled in global memory exactly as one
// pipeline stage needs them in shared memory (tcgen05 canonical K-major layout, no
// swizzle): a 128x32 (A) or 256x32 (B^T) bf16 tile is one contiguous block of 8x8
// "core matrices" (8 rows x 16 bytes each); core (row group i, k group j) sits at
// byte (i*4 + j)*128.  So the K-direction core stride (LBO) is 128 B and the
// row-direction stride (SBO) is 512 B, and each stage is filled by plain bulk copies
// (cp.async.bulk, the TMA engine) of contiguous tiles.
//
// Kernel structure: 128 threads, two CTAs per SM (98 KiB of shared memory and 256
// tensor-memory columns each), so that one CTA's epilogue overlaps the other's MMAs
// (with one CTA per SM the tensor pipe idled during every epilogue: 29 % busy).
// Thread 0 issues the bulk copies of a 2-stage ring (48 KiB per stage; 64-column tiles: 4
// smaller stages),
// thread 32 issues tcgen05.mma (M=128, N=256, K=16; 3 products per K step) and
// commits each stage back to the producer; after the last stage all four warps read
// the 128 x 256 (64) float32 accumulator from tensor memory (warp w owns lanes 32w..32w+31)
// and store du*D to the view-major output.  Every mbarrier wait is bounded (about 2 s
// of %globaltimer); a timeout sets an error flag, the kernel waits (bounded) for its
// own copies and MMAs, frees its tensor memory and returns; the host reports
// MCT_E_TIMEOUT on the next call that reads the flag.
#include <cmath>

#include "common.cuh"
#include "weight.cuh"

namespace mct {
namespace {

constexpr int TC_BM = 128, TC_BN = 256;  // operand tiles: rows of A, rows of B^T
constexpr unsigned long long TC_WAIT_NS = 2000000000ull;        // 2 s

// NS = number of bf16 parts each float32 operand is split into:
//   2: x = hi + lo, products hi*hi + hi*lo + lo*hi (~1e-5 relative; the mixed path);
//   3: x = hi + mid + lo, products of total order <= 2 (hi*hi, hi*mid, mid*hi, hi*lo,
//      lo*hi, mid*mid): the dropped terms are ~2^-24 relative; the result is within
//      ~1e-6 of float32 (the level of the tensor pipe's float32 accumulation).
// BK (K depth of one pipeline stage) keeps a stage small enough for two CTAs per SM.
template <int NS>
struct TcCfg;
template <>
struct TcCfg<2> {
    static constexpr int BK = 32, NPROD = 3;
};
template <>
struct TcCfg<3> {
    static constexpr int BK = 16, NPROD = 6;
};
template <int NS>
struct TcTiles {
    static constexpr int BK = TcCfg<NS>::BK;
    static constexpr int KG = BK / 8;                          // core matrices along K per row group
    static constexpr int SBO = KG * 128;                       // bytes between row groups
    static constexpr int A_TILE = TC_BM * BK * 2;
    static constexpr int B_TILE = TC_BN * BK * 2;
};
// One CTA's tile: 128 x BN of the output, BN = 256 or 64 (a quarter of a B^T tile, whose rows
// are contiguous).
template <int NS, int BN>
struct TcStage {
    using T = TcTiles<NS>;
    static constexpr int B_BYTES = BN * T::BK * 2;
    static constexpr int STAGE = NS * (T::A_TILE + B_BYTES);
    static constexpr int STAGES = BN == 256 ? 2 : 4;
    static constexpr int SMEM = STAGES * STAGE + 2048;         // + 1 KiB alignment slack + barriers
    static_assert(2 * SMEM <= 228 * 1024, "two CTAs per SM");
    static_assert(TC_BN % BN == 0 && BN % 32 == 0 && (BN & (BN - 1)) == 0, "N tile");
    static_assert(STAGES * STAGE >= 4 * 32 * 33 * 4, "the ring holds the epilogue's transposes");
};

struct TcDims {
    int64_t rows;    // M (sinogram rows)
    int nu;          // N = K
    int mb, kb, nb;  // tile counts along M, K, N
};

template <int NS>
inline TcDims tc_dims(int64_t rows, int nu) {
    TcDims d;
    d.rows = rows;
    d.nu = nu;
    d.mb = (int)((rows + TC_BM - 1) / TC_BM);
    d.kb = (nu + TcTiles<NS>::BK - 1) / TcTiles<NS>::BK;
    d.nb = (nu + TC_BN - 1) / TC_BN;
    return d;
}

// x as NS bf16 parts (bit patterns), largest first; each part is the bf16 rounding of
// what the previous parts leave
template <int NS>
__device__ __forceinline__ void split_parts(float x, uint32_t* out) {
    float r = x;
#pragma unroll
    for (int p = 0; p < NS; ++p) {
        const __nv_bfloat16 h = __float2bfloat16_rn(r);
        out[p] = (uint32_t)__bfloat16_as_ushort(h);
        r = r - __bfloat162float(h);
    }
}

// One 16-byte core-matrix row (8 bf16 along K) of every part of a tile.  Chunk i
// enumerates (tile, row group, k group kj, row r8) in storage order, so consecutive
// threads write consecutive 16-byte chunks.  ROWS = 128 (A) or 256 (B^T).
template <int NS, int ROWS>
__device__ __forceinline__ void tile_coords(int64_t i, int KB, int& r8, int& kj, int& gi, int& kb, int& tb) {
    constexpr int KG = TcTiles<NS>::KG;
    r8 = (int)(i & 7);
    kj = (int)((i >> 3) % KG);
    const int64_t rest = (i >> 3) / KG;
    gi = (int)(rest % (ROWS / 8));
    tb = (int)split_index(rest / (ROWS / 8), KB, kb);
}

template <int NS>
__device__ __forceinline__ void store_parts(uint4* const* dst, int64_t i, const uint32_t (*v)[NS]) {
#pragma unroll
    for (int p = 0; p < NS; ++p)
        dst[p][i] = make_uint4(v[0][p] | (v[1][p] << 16), v[2][p] | (v[3][p] << 16), v[4][p] | (v[5][p] << 16),
                               v[6][p] | (v[7][p] << 16));
}

struct Parts {
    uint4* p[3];
};

template <int NS>
__global__ void split_a_kernel(const float* __restrict__ x, int64_t rows, int nu, int KB, int64_t n_chunks, Parts a) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_chunks; i += (int64_t)gridDim.x * blockDim.x) {
        int r8, kj, mi, kb, mb;
        tile_coords<NS, TC_BM>(i, KB, r8, kj, mi, kb, mb);
        const int64_t R = (int64_t)mb * TC_BM + mi * 8 + r8;
        const int m0 = kb * TcTiles<NS>::BK + kj * 8;
        uint32_t v[8][NS];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int m = m0 + c;
            split_parts<NS>((R < rows && m < nu) ? x[R * nu + m] : 0.0f, v[c]);
        }
        store_parts<NS>(a.p, i, v);
    }
}

// split_a_kernel reading the raw sinogram and weighting each element on the way
// (weight_value, as the weighting kernels do), so the weighted float32 sinogram is never
// written: operand row R = r * views + j is detector row r of view j, as in the
// weighting kernels' output.
//
// Instructions bound it (a distance factor's square root and division per element, and for
// curved detectors and short scans a cosine and an arc tangent).  256 chunks share the BK
// columns of one K block and rows of at most a few detector rows, so the block takes each
// column's cosine and fan angle once, and the square roots once per column and detector row
// where its rows span at most two; each element goes through the same operations as before.
// 500 x 157 rows of 701 columns, curved short scan: 0.40 -> 0.29 ms.  The common case (PLAIN:
// flat detector, full scan, no polynomial) has its own instance, rows are read 16 bytes at a
// time where they are aligned and row indices are 32-bit: 1080 x 256 rows of 1024 columns 0.86
// -> 0.55 ms (its bytes: 0.41 ms), 180 x 64 rows of 256 columns 19.6 -> 12.0 us.
template <int NS, bool PLAIN>
__global__ void __launch_bounds__(256)
weight_split_a_kernel(WeightParams wp, const float* __restrict__ in, const float* __restrict__ bh,
                      const float* __restrict__ angles, int rows, int nu, int KB, int64_t n_chunks, Parts a, bool vec) {
    constexpr int BK = TcTiles<NS>::BK, KG = TcTiles<NS>::KG;
    constexpr int SPAN = 256 / KG;  // operand rows of 256 chunks
    static_assert(256 % KG == 0 && TC_BM % SPAN == 0, "256 chunks lie in one tile");
    __shared__ float cs_s[BK], ga_s[BK], den_s[2][BK];
    for (int64_t i0 = blockIdx.x * (int64_t)256; i0 < n_chunks; i0 += (int64_t)gridDim.x * 256) {
        const int64_t i = i0 + threadIdx.x;  // n_chunks is a multiple of 256
        int r8, kj, mi, kb, mb;
        tile_coords<NS, TC_BM>(i, KB, r8, kj, mi, kb, mb);
        // operand rows, fewer than 2^28 (checked on the host): this thread's, and the block's R0 to R1
        const int R = mb * TC_BM + mi * 8 + r8;
        const int R0 = R / SPAN * SPAN, R1 = min(R0 + SPAN, rows) - 1;
        const int first = R0 / wp.views;  // the block's first detector row
        const bool shared_den = R0 < rows && R1 - first * wp.views < 2LL * wp.views;
        __syncthreads();
        if (threadIdx.x < 3 * BK) {
            const int what = threadIdx.x / BK, c = threadIdx.x % BK;
            const float u = wp.u0 + (kb * BK + c) * wp.u_step;
            if (PLAIN && what == 0) {
            } else if (what == 0) {
                cs_s[c] = weight_cos(wp, u);
                ga_s[c] = wp.short_scan ? parker_gamma(wp, u) : 0.0f;
            } else {
                den_s[what - 1][c] = weight_den<PLAIN>(wp, u, wp.v0 + (first + what - 1) * wp.v_step);
            }
        }
        __syncthreads();
        const int c0 = kj * 8, m0 = kb * BK + c0;
        uint32_t v[8][NS];
        if (R < rows) {
            int r = first, j = R - first * wp.views;
            if (shared_den) {
                if (j >= wp.views) {
                    ++r;
                    j -= wp.views;
                }
            } else {
                r = R / wp.views;
                j = R - r * wp.views;
            }
            const float* src = in + r * wp.row_stride + j * wp.view_stride;
            const float vv = wp.v0 + r * wp.v_step;
            const float beta = !PLAIN && wp.short_scan ? fabsf(angles[wp.view_begin + j] - angles[0]) : 0.0f;
            float x8[8];
            if (vec && m0 + 8 <= nu) {
                const float4 lo = __ldg(reinterpret_cast<const float4*>(src + m0));
                const float4 hi = __ldg(reinterpret_cast<const float4*>(src + m0) + 1);
                x8[0] = lo.x; x8[1] = lo.y; x8[2] = lo.z; x8[3] = lo.w;
                x8[4] = hi.x; x8[5] = hi.y; x8[6] = hi.z; x8[7] = hi.w;
            } else {
#pragma unroll
                for (int c = 0; c < 8; ++c) x8[c] = m0 + c < nu ? __ldg(src + m0 + c) : 0.0f;
            }
            float den[8];
            if (shared_den) {
#pragma unroll
                for (int c = 0; c < 8; ++c) den[c] = den_s[r - first][c0 + c];
            } else {
#pragma unroll
                for (int c = 0; c < 8; ++c) den[c] = weight_den<PLAIN>(wp, wp.u0 + (m0 + c) * wp.u_step, vv);
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) {  // a column past nu is 0
                const float x = PLAIN ? weight_value<true>(wp, x8[c], bh, 0.0f, 0.0f, den[c], beta)
                                      : weight_value(wp, x8[c], bh, ga_s[c0 + c], cs_s[c0 + c], den[c], beta);
                split_parts<NS>(m0 + c < nu ? x : 0.0f, v[c]);
            }
        } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) split_parts<NS>(0.0f, v[c]);
        }
        store_parts<NS>(a.p, i, v);
    }
}

// B^T element (n, k) = T[k][n] = h[n - k + nu - 1] (output column n, input column k),
// tiled like A with 256-row tiles.
template <int NS>
__global__ void build_b_kernel(const float* __restrict__ taps, int nu, int KB, int64_t n_chunks, Parts b) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_chunks; i += (int64_t)gridDim.x * blockDim.x) {
        int r8, kj, ni, kb, nb;
        tile_coords<NS, TC_BN>(i, KB, r8, kj, ni, kb, nb);
        const int n = nb * TC_BN + ni * 8 + r8;
        const int k0 = kb * TcTiles<NS>::BK + kj * 8;
        uint32_t v[8][NS];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int k = k0 + c;
            split_parts<NS>((n < nu && k < nu) ? taps[n - k + nu - 1] : 0.0f, v[c]);
        }
        store_parts<NS>(b.p, i, v);
    }
}

// ---------------------------------------------------------------- PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.b32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait; returns false (and raises the error flag) after TC_WAIT_NS.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* err, int code) {
    const unsigned long long t0 = global_ns();
    while (!mbar_try_wait(bar, parity)) {
        if (global_ns() - t0 > TC_WAIT_NS) {
            atomicExch(err, code);
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    // start address >> 4 (bits 0-13), leading byte offset >> 4 (16-29), stride byte
    // offset >> 4 (32-45), fixed 0b001 (46-48), no swizzle (61-63 = 0)
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// kind::f16 instruction descriptor: D f32, A and B bf16, both K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
            d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

template <int NS, int BN>
__global__ void __launch_bounds__(128, 2)
tc_filter_kernel(TcDims d, int nv, int views, float du, Parts a, Parts b, float* __restrict__ F, int* __restrict__ err) {
    using T = TcTiles<NS>;
    using S = TcStage<NS, BN>;
    constexpr int TC_STAGES = S::STAGES;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // 1 KiB-aligned stage buffers: [A part 0..NS-1][B part 0..NS-1] per stage
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* ctrl = smem + TC_STAGES * S::STAGE;  // barriers and the TMEM address
    uint64_t* full = reinterpret_cast<uint64_t*>(ctrl);
    uint64_t* empty = full + TC_STAGES;
    uint64_t* done = empty + TC_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nbk = blockIdx.x;  // N tile of BN columns
    const int64_t mbk = blockIdx.y;  // M tile

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < TC_STAGES; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        mbar_init(smem_u32(done), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    bool ok = true;
    if (threadIdx.x == 0) {
        // producer: bulk copies of the A and B part tiles of every K block
        int issued = 0;
        for (int kb = 0; kb < d.kb && ok; ++kb) {
            const int s = kb % TC_STAGES;
            if (kb >= TC_STAGES) ok = mbar_wait(smem_u32(&empty[s]), ((kb / TC_STAGES) - 1) & 1, err, 1);
            if (!ok) break;
            unsigned char* st = smem + s * S::STAGE;
            const uint32_t bar = smem_u32(&full[s]);
            mbar_expect_tx(bar, S::STAGE);
            const int64_t at = mbk * d.kb + kb;
            // the BN rows of the B^T tile that holds them
            constexpr int PER = TC_BN / BN;
            const int64_t bt = (int64_t)(nbk / PER) * d.kb + kb;
            const int bsub = (nbk % PER) * (S::B_BYTES / 16);
#pragma unroll
            for (int p = 0; p < NS; ++p) {
                bulk_g2s(smem_u32(st + p * T::A_TILE), a.p[p] + at * (T::A_TILE / 16), T::A_TILE, bar);
                bulk_g2s(smem_u32(st + NS * T::A_TILE + p * S::B_BYTES), b.p[p] + bt * (T::B_TILE / 16) + bsub,
                         S::B_BYTES, bar);
            }
            issued = kb + 1;
        }
        // drain: the copies of the last issued block of every stage must have landed
        // before this CTA's shared memory is released (immediate on the normal path)
        for (int kb = (issued > TC_STAGES ? issued - TC_STAGES : 0); kb < issued; ++kb)
            mbar_wait(smem_u32(&full[kb % TC_STAGES]), (kb / TC_STAGES) & 1, err, 4);
    } else if (threadIdx.x == 32) {
        // MMA issuer: the products of total order <= 1 (NS = 2) or <= 2 (NS = 3)
        constexpr int NP = TcCfg<NS>::NPROD;
        constexpr int pa[6] = {0, 0, 1, 0, 2, 1};
        constexpr int pb[6] = {0, 1, 0, 2, 0, 1};
        const uint32_t idesc = idesc_bf16(TC_BM, BN);
        for (int kb = 0; kb < d.kb && ok; ++kb) {
            const int s = kb % TC_STAGES;
            ok = mbar_wait(smem_u32(&full[s]), (kb / TC_STAGES) & 1, err, 2);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t st = smem_u32(smem + s * S::STAGE);
#pragma unroll
            for (int ks = 0; ks < T::BK / 16; ++ks) {
                const uint32_t off = ks * 256;  // two core matrices along K
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    const uint64_t da = smem_desc(st + pa[q] * T::A_TILE + off, 128, T::SBO);
                    const uint64_t db = smem_desc(st + NS * T::A_TILE + pb[q] * S::B_BYTES + off, 128, T::SBO);
                    mma_bf16(tmem, da, db, idesc, (kb | ks | q) != 0);
                }
            }
            mma_commit(smem_u32(&empty[s]));  // stage free once these MMAs complete
        }
        mma_commit(smem_u32(done));  // accumulator complete (or all issued MMAs drained)
    }
    __syncwarp();
    // epilogue: every warp waits for the accumulator, then reads its 32 lanes
    ok = mbar_wait(smem_u32(done), 0, err, 3);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // tcgen05.ld is warp-collective: decide per warp
    const bool go = __all_sync(0xffffffffu, ok && *(volatile int*)err == 0);
    if (go) {
        const int64_t R = mbk * TC_BM + warp * 32 + lane;
        const bool row_ok = R < d.rows;
        int64_t at = -1;  // this lane's output row, -1 past the last
        if (row_ok) {
            const int r = (int)R / views, j = (int)R % views;  // fewer than 2^28 rows
            at = ((int64_t)j * nv + r) * d.nu;
        }
        const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
        const int cols = min(BN, d.nu - nbk * BN);  // this tile's, at least 1
        if ((d.nu & 3) == 0) {
            // rows are 16-byte aligned: each lane stores its row
            for (int c0 = 0; c0 < cols; c0 += 16) {
                float v[16];
                tmem_ld16(lanes + (uint32_t)c0, v);
                const int n0 = nbk * BN + c0;
                if (!row_ok) continue;
                if (n0 + 16 <= d.nu) {
                    float4* q = reinterpret_cast<float4*>(F + at + n0);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        q[i] = make_float4(v[4 * i] * du, v[4 * i + 1] * du, v[4 * i + 2] * du, v[4 * i + 3] * du);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (n0 + i < d.nu) F[at + n0 + i] = v[i] * du;
                }
            }
        } else {
            // others (stored by each lane, 4 bytes at 32 rows a time, these cost more than the
            // MMAs: 500 x 157 rows of 701 columns, with the weighting, 0.94 -> 0.66 ms): 32
            // columns at a time through this warp's part of the ring (its copies and
            // MMAs are done), so that a warp stores 32 consecutive floats of a row
            float* t = reinterpret_cast<float*>(smem) + warp * (32 * 33);
            for (int c0 = 0; c0 < cols; c0 += 32) {
                const int n = nbk * BN + c0 + lane;
#pragma unroll
                for (int h = 0; h < 32; h += 16) {
                    float v[16];
                    tmem_ld16(lanes + (uint32_t)(c0 + h), v);
#pragma unroll
                    for (int i = 0; i < 16; ++i) t[lane * 33 + h + i] = v[i] * du;
                }
                __syncwarp();
#pragma unroll 4
                for (int q = 0; q < 32; ++q) {
                    const int64_t row = __shfl_sync(0xffffffffu, at, q);
                    if (row >= 0 && n < d.nu) F[row + n] = t[q * 33 + lane];
                }
                __syncwarp();
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN));
    }
}

// Workspace layout: [A parts][B parts][flag]
template <int NS>
size_t tc_workspace(const mct_geom* g, Parts* a, Parts* b, int** flag, void* ws) {
    using T = TcTiles<NS>;
    const TcDims d = tc_dims<NS>((int64_t)g->nv * g->views, g->nu);
    const size_t as = (size_t)d.mb * d.kb * T::A_TILE, bs = (size_t)d.nb * d.kb * T::B_TILE;
    if (ws) {
        unsigned char* p = static_cast<unsigned char*>(ws);
        for (int i = 0; i < NS; ++i) {
            a->p[i] = reinterpret_cast<uint4*>(p + i * as);
            b->p[i] = reinterpret_cast<uint4*>(p + NS * as + i * bs);
        }
        *flag = reinterpret_cast<int*>(p + NS * (as + bs));
    }
    return NS * (as + bs) + 256;
}

template <int NS>
int tc_prepare(const mct_geom* g, const float* taps, void* ws, cudaStream_t s) {
    Parts a{}, b{};
    int* flag;
    tc_workspace<NS>(g, &a, &b, &flag, ws);
    const TcDims d = tc_dims<NS>((int64_t)g->nv * g->views, g->nu);
    cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), s);
    if (e != cudaSuccess) {
        set_error("mct_filter_tc_prepare: %s", cudaGetErrorString(e));
        return MCT_E_CUDA;
    }
    const int64_t chunks = (int64_t)d.nb * d.kb * (TcTiles<NS>::B_TILE / 16);
    const int grid = (int)std::min<int64_t>((chunks + 255) / 256, 152 * 32);
    build_b_kernel<NS><<<grid, 256, 0, s>>>(taps, g->nu, d.kb, chunks, b);
    return launched("build_b_kernel");
}

template <int NS, int BN>
int tc_launch(const mct_geom* g, const TcDims& d, const Parts& a, const Parts& b, float* filtered, int* flag,
              cudaStream_t s) {
    constexpr int smem = TcStage<NS, BN>::SMEM;
    // opt in to the large dynamic shared memory (per device, idempotent)
    cudaError_t e = cudaFuncSetAttribute(tc_filter_kernel<NS, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) {
        set_error("mct_filter_tc: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        return MCT_E_CUDA;
    }
    dim3 grid((d.nu + BN - 1) / BN, d.mb);
    tc_filter_kernel<NS, BN><<<grid, 128, smem, s>>>(d, g->nv, g->views, g->du, a, b, filtered, flag);
    return launched("tc_filter_kernel");
}

// weighted: the weighted sinogram [nv][views][nu]; or, with wp, the raw sinogram
// (strides in wp), weighted while it is split.
template <int NS>
int tc_run(const mct_geom* g, const float* weighted, void* ws, float* filtered, cudaStream_t s,
           const WeightParams* wp = nullptr, const float* bh = nullptr, const float* angles = nullptr) {
    Parts a{}, b{};
    int* flag;
    tc_workspace<NS>(g, &a, &b, &flag, ws);
    const TcDims d = tc_dims<NS>((int64_t)g->nv * g->views, g->nu);
    MCT_REQUIRE(d.mb < 65535 * 32, "mct_filter_tc: too many rows");
    const int64_t chunks = (int64_t)d.mb * d.kb * (TcTiles<NS>::A_TILE / 16);
    const int grid = (int)std::min<int64_t>((chunks + 255) / 256, 152 * 32);
    if (wp) {
        // rows that start on 16-byte boundaries are read 16 bytes at a time
        const bool vec = ((uintptr_t)weighted & 15) == 0 && wp->row_stride % 4 == 0 && wp->view_stride % 4 == 0;
        auto go = wp->curved || wp->short_scan || wp->n_bh > 0 ? weight_split_a_kernel<NS, false>
                                                               : weight_split_a_kernel<NS, true>;
        go<<<grid, 256, 0, s>>>(*wp, weighted, bh, angles, (int)d.rows, g->nu, d.kb, chunks, a,
                                                       vec);
        MCT_TRY(launched("weight_split_a_kernel"));
    } else {
        split_a_kernel<NS><<<grid, 256, 0, s>>>(weighted, d.rows, g->nu, d.kb, chunks, a);
        MCT_TRY(launched("split_a_kernel"));
    }
    // Few rows: N tiles of 64 columns, so that more SMs work (256^2 image, 720 x 512 sinogram:
    // 48 CTAs instead of 12, FBP 0.088 -> 0.078 ms; 92 CTAs of 256 columns 0.464 -> 0.453 ms
    // per FBP; from 96 on the wider tile, which reads A once instead of four times, is the
    // faster: 96 CTAs 1.193 against 1.202 ms, 135 CTAs 0.283 against 0.288).  Rings of 6 or 8
    // stages and 32 or 128 columns measured the same within 3 %: the chain of K steps binds.
    if ((int64_t)d.mb * d.nb >= 96) return tc_launch<NS, 256>(g, d, a, b, filtered, flag, s);
    return tc_launch<NS, 64>(g, d, a, b, filtered, flag, s);
}

}  // namespace
}  // namespace mct

using namespace mct;

extern "C" {

size_t mct_filter_tc_workspace_size(const mct_geom* g, int32_t dtype) {
    if (!g || g->nu < 2 || g->nv < 1 || g->views < 1 || (dtype != MCT_F32 && dtype != MCT_BF16)) return 0;
    Parts a, b;
    int* f;
    return dtype == MCT_F32 ? tc_workspace<3>(g, &a, &b, &f, nullptr) : tc_workspace<2>(g, &a, &b, &f, nullptr);
}

int mct_filter_tc_prepare(const mct_geom* g, const float* taps, int32_t dtype, void* workspace, void* stream) {
    MCT_TRY(check_geom(g, "mct_filter_tc_prepare"));
    MCT_REQUIRE(taps && workspace, "mct_filter_tc_prepare: NULL buffer");
    MCT_REQUIRE(dtype == MCT_F32 || dtype == MCT_BF16, "mct_filter_tc_prepare: dtype must be MCT_F32 or MCT_BF16");
    MCT_REQUIRE(((uintptr_t)workspace & 1023) == 0, "mct_filter_tc_prepare: workspace must be 1 KiB aligned");
    return dtype == MCT_F32 ? tc_prepare<3>(g, taps, workspace, as_stream(stream))
                            : tc_prepare<2>(g, taps, workspace, as_stream(stream));
}

int mct_filter_tc(const mct_geom* g, const float* weighted, int32_t dtype, void* workspace, float* filtered,
                  void* stream) {
    MCT_TRY(check_geom(g, "mct_filter_tc"));
    MCT_REQUIRE(weighted && workspace && filtered, "mct_filter_tc: NULL buffer");
    MCT_REQUIRE(dtype == MCT_F32 || dtype == MCT_BF16, "mct_filter_tc: dtype must be MCT_F32 or MCT_BF16");
    MCT_REQUIRE(((uintptr_t)workspace & 1023) == 0, "mct_filter_tc: workspace must be 1 KiB aligned");
    return dtype == MCT_F32 ? tc_run<3>(g, weighted, workspace, filtered, as_stream(stream))
                            : tc_run<2>(g, weighted, workspace, filtered, as_stream(stream));
}

int mct_weight_filter(const mct_geom* g, const mct_tables* t, const float* sgm, int64_t row_stride,
                      int64_t view_stride, const float* bh_coeffs, int32_t n_bh, int32_t dtype, void* workspace,
                      float* filtered, void* stream) {
    MCT_TRY(check_geom(g, "mct_weight_filter"));
    MCT_REQUIRE(sgm && workspace && filtered, "mct_weight_filter: NULL buffer");
    MCT_REQUIRE(n_bh >= 0 && (n_bh == 0 || bh_coeffs), "mct_weight_filter: bad BH coefficients");
    MCT_REQUIRE(dtype == MCT_F32 || dtype == MCT_BF16, "mct_weight_filter: dtype must be MCT_F32 or MCT_BF16");
    MCT_REQUIRE(((uintptr_t)workspace & 1023) == 0, "mct_weight_filter: workspace must be 1 KiB aligned");
    const bool short_scan = (g->flags & MCT_SHORT_SCAN) != 0;
    MCT_REQUIRE(!short_scan || (t && t->angles), "mct_weight_filter: short scan needs the angle table");
    MCT_REQUIRE(row_stride >= 0 && view_stride >= 0, "mct_weight_filter: negative stride");
    const WeightParams wp = weight_params(g, row_stride, view_stride, n_bh);
    const float* angles = t ? t->angles : nullptr;
    cudaStream_t s = as_stream(stream);
    return dtype == MCT_F32 ? tc_run<3>(g, sgm, workspace, filtered, s, &wp, bh_coeffs, angles)
                            : tc_run<2>(g, sgm, workspace, filtered, s, &wp, bh_coeffs, angles);
}

// 0 if no tensor-core filter launch on this workspace has timed out, else MCT_E_TIMEOUT
// (synchronises the stream).
int mct_filter_tc_status(const mct_geom* g, int32_t dtype, void* workspace, void* stream) {
    MCT_REQUIRE(g && workspace, "mct_filter_tc_status: NULL argument");
    MCT_REQUIRE(dtype == MCT_F32 || dtype == MCT_BF16, "mct_filter_tc_status: dtype must be MCT_F32 or MCT_BF16");
    Parts a, b;
    int* flag;
    if (dtype == MCT_F32) tc_workspace<3>(g, &a, &b, &flag, workspace);
    else tc_workspace<2>(g, &a, &b, &flag, workspace);
    int h = 0;
    cudaStream_t s = as_stream(stream);
    cudaError_t e = cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_error("mct_filter_tc_status: %s", cudaGetErrorString(e));
        return MCT_E_CUDA;
    }
    if (h != 0) {
        set_error("mct_filter_tc: a pipeline wait timed out (stage %d)", h);
        return MCT_E_TIMEOUT;
    }
    return MCT_OK;
}

}  // extern "C"
