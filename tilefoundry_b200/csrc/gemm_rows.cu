// Projection of many tokens on the tensor cores: Y[M, N] = X[M, K] . W[N, K]^T (+ residual, or SwiGLU), bf16 in, f32
// accumulate, bf16 out, for prompt chunks of more than 256 tokens (up to there gemm_tc.cu: the weight stream is the
// larger time and the split over K fills the chip).
//
// Compute-bound: 2 * M * N * K operations against N * K * 2 bytes of weights.  Tokens are the MMA's A rows (one per
// tensor-memory lane), weight rows its N; both operands through a TMA ring of 192 KB, K in stages of 128 elements (two
// 128-byte-swizzled tiles per request).  One persistent CTA per SM: warp 0 (one lane) requests tiles, warp 1 (one lane)
// issues tcgen05.mma, warps 2-5 read accumulators back and write results; two accumulators in tensor memory, so a tile's
// read-back runs under the next tile's products.  Tiles are dealt with the token tile running fastest: the tiles in flight
// share a few weight blocks and the whole X, which then come from L2.
//
// Two forms.  gemm_pair_kernel, 256 x 256 on two SMs: what the SMs can take from L2 is the bound (a lone CTA at 128 x 256
// needs 48 KB per K block where each CTA of a pair needs 32), 4093 tokens x 12288 x 2048: 137 us, 1.51 PFLOP/s (the lone
// form 172).  gemm_rows_kernel, 128 x 128 on one SM, where 256 x 256 tiles would leave SMs idle (512 tokens x 2048 x 2048:
// 12.2 us against 15.1).
//
// SwiGLU: the BN rows of a tile are BN/2 gate rows and the BN/2 up rows of the same outputs, so the thread that owns a
// token holds both halves in its own accumulator row.  Rounding points are those of gemm_tc.cu.
//
// Every mbarrier wait is bounded; a timeout sets *status, and the CTA still frees its tensor memory.
#include "common.cuh"
#include "kernels.h"
#include "launch.h"
#include "tc.cuh"

namespace tfb {
namespace {

constexpr int RW_BM = 128, RW_BK = 64, RW_KB = 2, RW_THREADS = 192;   // a stage holds RW_KB blocks of 64 elements
constexpr int RW_A_TILE = RW_BM * RW_BK * 2, RW_A_BYTES = RW_KB * RW_A_TILE;

constexpr int RW_BN = 128, RW_B_TILE = RW_BN * RW_BK * 2, RW_B_BYTES = RW_KB * RW_B_TILE, RW_STAGES = 3;

struct RwSmemTail {
    uint64_t full[RW_STAGES], empty[RW_STAGES], acc_full[2], acc_empty[2], drain;
    uint32_t tmem_base;
    volatile int aborted;
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(bar)) : "memory");
}
// One request for the RW_KB blocks of a stage: 64 elements x rows (x gate/up halves) x blocks.  A request costs the producer
// ~0.1 us however large it is: with one 64-element block per request the 128 x 64 form took 0.38 us a block, with two 0.26.
__device__ __forceinline__ void tma_load_x(void* dst, const CUtensorMap* map, uint64_t* bar, int row, int kb) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 :: "r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(0), "r"(row), "r"(kb) : "memory");
}
__device__ __forceinline__ void tma_load_w(void* dst, const CUtensorMap* map, uint64_t* bar, int row, int kb) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                 :: "r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(0), "r"(row), "r"(0), "r"(kb) : "memory");
}
// 32 bytes (one sector) per lane
__device__ __forceinline__ void st_global32(void* p, const uint32_t (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    return uint32_t(f32_to_bf16_bits(lo)) | (uint32_t(f32_to_bf16_bits(hi)) << 16);
}

// 16 finished sums of token row m, columns n .. n + 15 -> y
__device__ __forceinline__ void rw_store16(const TcParams& p, int m, int n, const uint32_t* v) {
    uint32_t out[8];
    if (p.residual) {                                     // bf16(acc), bf16(. * scale), then the add
        const uint4* rp = reinterpret_cast<const uint4*>(p.residual + size_t(m) * p.N + n);
        const uint4 r0 = rp[0], r1 = rp[1];
        const uint32_t r[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float a = round_bf16(__uint_as_float(v[2 * i])), b = round_bf16(__uint_as_float(v[2 * i + 1]));
            if (p.res_scale != 1.f) { a = round_bf16(a * p.res_scale); b = round_bf16(b * p.res_scale); }
            out[i] = pack_bf16(bf16_lo(r[i]) + a, bf16_hi(r[i]) + b);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = pack_bf16(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
    }
    st_global32(p.y + size_t(m) * p.N + n, out);
    if (p.y_lo) {
        uint32_t lo[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            lo[i] = pack_bf16(__uint_as_float(v[2 * i]) - bf16_lo(out[i]), __uint_as_float(v[2 * i + 1]) - bf16_hi(out[i]));
        st_global32(p.y_lo + size_t(m) * p.N + n, lo);
    }
}

// token row m of weight tile nt: this lane's accumulator row of BN columns -> y
template <int BN>
__device__ __forceinline__ void rw_epilogue(const TcParams& p, uint32_t taddr, int m, int nt) {
    if (p.swiglu) {
#pragma unroll 1
        for (int c = 0; c < BN / 2; c += 32) {
            uint32_t g[32], u[32];
            tmem_ld32_async(g, taddr + c);
            tmem_ld32_async(u, taddr + BN / 2 + c);
            tmem_wait_ld();
            tmem_pin(g);
            tmem_pin(u);
            const int n = nt * (BN / 2) + c;
            if (m < p.M && n < p.N) {
                uint32_t out[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float a = round_bf16(silu_f32(round_bf16(__uint_as_float(g[2 * i])))) * round_bf16(__uint_as_float(u[2 * i]));
                    const float b = round_bf16(silu_f32(round_bf16(__uint_as_float(g[2 * i + 1])))) * round_bf16(__uint_as_float(u[2 * i + 1]));
                    out[i] = pack_bf16(a, b);
                }
                uint16_t* y = p.y + size_t(m) * p.N + n;
                st_global32(y, *reinterpret_cast<uint32_t(*)[8]>(out));
                st_global32(y + 16, *reinterpret_cast<uint32_t(*)[8]>(out + 8));
            }
        }
        return;
    }
#pragma unroll 1
    for (int c = 0; c < BN; c += 32) {
        uint32_t v[32];
        tmem_ld32(v, taddr + c);
        const int n = nt * BN + c;
        if (m < p.M && n < p.N) {
            rw_store16(p, m, n, v);
            rw_store16(p, m, n + 16, v + 16);
        }
    }
}

__global__ void __launch_bounds__(RW_THREADS, 1) gemm_rows_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                  const __grid_constant__ CUtensorMap map_x, const TcParams p,
                                                                  int m_tiles, int n_tiles) {
    constexpr int ST = RW_STAGES, BB = RW_B_BYTES, BN = RW_BN;
    extern __shared__ unsigned char rw_smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(rw_smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* a_tiles = base;                                      // ST x RW_KB x 16 KB (tokens)
    unsigned char* b_tiles = base + ST * RW_A_BYTES;                    // ST x RW_KB x BN * 128 bytes (weights)
    RwSmemTail* t = reinterpret_cast<RwSmemTail*>(b_tiles + ST * BB);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total = m_tiles * n_tiles;

    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) { mbar_init(&t->full[s], 1); mbar_init(&t->empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&t->acc_full[b], 1); mbar_init(&t->acc_empty[b], 4); }
        mbar_init(&t->drain, 1);
        t->aborted = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(&t->tmem_base)), "r"(uint32_t(2 * BN)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = t->tmem_base;
    pdl_trigger();
    if (!(warp == 0 && lane == 0)) pdl_wait();

    // a bounded wait that also ends once any role of this CTA gave up
    auto wait = [&](uint64_t* bar, uint32_t parity, unsigned role) -> bool {
        if (t->aborted) return false;
        if (mbar_wait(bar, parity)) return true;
        t->aborted = 1;
        atomicExch(p.status, role);
        return false;
    };

    if (warp == 0) {
        if (lane == 0) {                                                // ---- TMA producer ----
            int s = 0;
            uint32_t ph = 0;
            auto load_w = [&](int tile, int k, int st) {                // (SwiGLU: BN/2 gate rows, then the up rows of the same outputs)
                tma_load_w(b_tiles + st * BB, &map_w, &t->full[st], tile / m_tiles * (p.swiglu ? BN / 2 : BN), k * RW_KB);
            };
            auto load_x = [&](int tile, int k, int st) {
                tma_load_x(a_tiles + st * RW_A_BYTES, &map_x, &t->full[st], tile % m_tiles * RW_BM, k * RW_KB);
            };
            // weights do not depend on the kernel before: the first tile's are requested ahead of the dependency wait
            const int pre = int(blockIdx.x) < total ? min(ST, p.ksteps) : 0;
            for (int k = 0; k < pre; ++k) {
                mbar_expect_tx(&t->full[k], RW_A_BYTES + BB);
                load_w(blockIdx.x, k, k);
            }
            pdl_wait();
            for (int k = 0; k < pre; ++k) load_x(blockIdx.x, k, k);
            int issued = pre;
            s = pre == ST ? 0 : pre;
            ph = pre == ST ? 1u : 0u;
            bool ok = true;
            for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
                for (int k = tile == int(blockIdx.x) ? pre : 0; k < p.ksteps; ++k) {
                    ok = wait(&t->empty[s], ph ^ 1u, 1u);
                    if (!ok) break;
                    mbar_expect_tx(&t->full[s], RW_A_BYTES + BB);
                    load_w(tile, k, s);
                    load_x(tile, k, s);
                    ++issued;
                    if (++s == ST) { s = 0; ph ^= 1u; }
                }
            }
            if (!ok) drain_copies(t->full, ST, issued);
        }
    } else if (warp == 1) {
        if (lane == 0) {                                                // ---- MMA issuer ----
            // D f32, A and B bf16, both K-major, N = BN, M = 128
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(BN >> 3) << 17) | (uint32_t(RW_BM >> 4) << 24);
            int s = 0, buf = 0;
            uint32_t ph = 0, aph = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
                ok = wait(&t->acc_empty[buf], aph ^ 1u, 4u);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + uint32_t(buf * BN);
                for (int k = 0; k < p.ksteps; ++k) {
                    ok = wait(&t->full[s], ph, 2u);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t da = umma_desc_sw128(a_tiles + s * RW_A_BYTES), db = umma_desc_sw128(b_tiles + s * BB);
#pragma unroll
                    for (int kk = 0; kk < RW_KB * RW_BK / 16; ++kk)
                        umma_bf16(d, da + (kk >> 2) * (RW_A_TILE >> 4) + 2 * (kk & 3), db + (kk >> 2) * (RW_B_TILE >> 4) + 2 * (kk & 3),
                                  idesc, (k > 0 || kk > 0) ? 1u : 0u);
                    umma_commit(&t->empty[s]);
                    if (++s == ST) { s = 0; ph ^= 1u; }
                }
                if (ok) umma_commit(&t->acc_full[buf]);
                if (++buf == 2) { buf = 0; aph ^= 1u; }
            }
            if (!ok) drain_products(&t->drain);
        }
    } else {                                                            // ---- epilogue: warps 2..5 ----
        const int quad = warp & 3;                                      // the tensor-memory lane quadrant this warp may read
        int buf = 0;
        uint32_t aph = 0;
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
            const bool ok = wait(&t->acc_full[buf], aph, 3u);
            if (!__all_sync(0xffffffffu, ok)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int m = (tile % m_tiles) * RW_BM + quad * 32 + lane, nt = tile / m_tiles;
            rw_epilogue<BN>(p, tmem + (uint32_t(quad * 32) << 16) + uint32_t(buf * BN), m, nt);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&t->acc_empty[buf]);
            if (++buf == 2) { buf = 0; aph ^= 1u; }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(uint32_t(2 * BN)) : "memory");
    }
}

// [rows][K] as (64 elements, rows of a half, halves, K blocks); boxes of 64 x box_rows x halves x RW_KB.  halves = 0: no such
// dimension.
bool make_block_map(CUtensorMap* map, const void* ptr, int rows, int k, int box_rows, int halves) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t kb = 64 * 2, pitch = cuuint64_t(k) * 2;
    const cuuint64_t dims4[4] = {64, cuuint64_t(rows), cuuint64_t(halves), cuuint64_t(k / 64)}, st4[3] = {pitch, pitch * rows, kb};
    const cuuint64_t dims3[3] = {64, cuuint64_t(rows), cuuint64_t(k / 64)}, st3[2] = {pitch, kb};
    const cuuint32_t box4[4] = {64, cuuint32_t(box_rows), cuuint32_t(halves), RW_KB}, box3[3] = {64, cuuint32_t(box_rows), RW_KB};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, halves ? 4 : 3, const_cast<void*>(ptr), halves ? dims4 : dims3, halves ? st4 : st3,
              halves ? box4 : box3, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_rows(const void* w, const void* x, TcParams p, cudaStream_t stream, bool pdl) {
    CUtensorMap map_w, map_x;
    if (!make_block_map(&map_w, w, p.N, p.K, p.swiglu ? RW_BN / 2 : RW_BN, p.swiglu ? 2 : 1) || !make_block_map(&map_x, x, p.M, p.K, RW_BM, 0))
        return cudaErrorInvalidValue;
    const size_t smem = 1024 + size_t(RW_STAGES) * (RW_A_BYTES + RW_B_BYTES) + sizeof(RwSmemTail);
    static PerDeviceOnce once;
    if (once.first()) {
        cudaError_t e = cudaFuncSetAttribute(gemm_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return e;
    }
    const int m_tiles = (p.M + RW_BM - 1) / RW_BM, per = p.swiglu ? RW_BN / 2 : RW_BN, n_tiles = (p.N + per - 1) / per;
    const int grid = min(sm_count(), m_tiles * n_tiles);
    return launch_kernel(gemm_rows_kernel, dim3(grid), dim3(RW_THREADS), smem, stream, pdl, map_w, map_x, p, m_tiles, n_tiles);
}

// ---- two SMs on one tile -----------------------------------------------------------------------------------------
// 256 tokens x 256 weight rows per pair of CTAs (cta_group::2): each CTA stages its own 128 tokens and HALF of the weight
// rows (rank 0 the first 128 of the tile -- the gate rows of a SwiGLU tile --, rank 1 the other 128), the MMA reads both
// halves, and each CTA's tensor memory receives its 128 tokens x all 256 columns.  Per CTA and K step 32 KB come from L2
// for the products a single CTA needs 48 KB for: the one-CTA form at 128 x 256 ran at 1.1 PFLOP/s, bound by that
// traffic.  Rank 0's barriers count both CTAs' copies; its one MMA thread issues for the pair.
constexpr int PR_BN = 256, PR_TILE = 128 * RW_BK * 2, PR_HALF = RW_KB * PR_TILE, PR_STAGES = 3;

struct PrSmemTail {
    uint64_t full[PR_STAGES], empty[PR_STAGES], acc_full[2], acc_empty[2], drain;
    uint32_t tmem_base;
    volatile int aborted;
};

__device__ __forceinline__ uint32_t map_to_rank(uint32_t local, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    return remote;
}
// a copy into this CTA's shared memory whose bytes are counted by a barrier of the pair (a cluster address)
__device__ __forceinline__ void tma_load_pair(void* dst, const CUtensorMap* map, uint32_t bar, int row, int kb) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 :: "r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(0), "r"(row), "r"(kb) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
                 :: "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {         // arrives at this barrier of both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 :: "r"(smem_u32(bar)), "h"(uint16_t(3)) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

__global__ void __launch_bounds__(RW_THREADS, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                  const __grid_constant__ CUtensorMap map_x, const TcParams p,
                                                                  int m_tiles, int n_tiles) {
    extern __shared__ unsigned char rw_smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(rw_smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* a_tiles = base;                                      // PR_STAGES x 32 KB (this CTA's tokens)
    unsigned char* b_tiles = base + PR_STAGES * RW_A_BYTES;             // PR_STAGES x 32 KB (this CTA's half of the weights)
    PrSmemTail* t = reinterpret_cast<PrSmemTail*>(b_tiles + PR_STAGES * PR_HALF);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int total = m_tiles * n_tiles, first = blockIdx.x >> 1, step = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < PR_STAGES; ++s) { mbar_init(&t->full[s], 1); mbar_init(&t->empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&t->acc_full[b], 1); mbar_init(&t->acc_empty[b], 8); }
        mbar_init(&t->drain, 1);
        t->aborted = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&t->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();                                                     // the peer's barriers exist before anything signals them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = t->tmem_base;
    pdl_trigger();
    if (!(warp == 0 && lane == 0)) pdl_wait();

    auto wait = [&](uint64_t* bar, uint32_t parity, unsigned role) -> bool {
        if (t->aborted) return false;
        if (mbar_wait(bar, parity)) return true;
        t->aborted = 1;
        atomicExch(p.status, role);
        return false;
    };

    if (warp == 0) {
        if (lane == 0) {                                                // ---- TMA producer: one in each CTA ----
            auto load_w = [&](int tile, int k, int s) {
                const int nt = tile / m_tiles;
                const int row = p.swiglu ? int(rank) * p.N + nt * 128 : nt * PR_BN + int(rank) * 128;
                tma_load_pair(b_tiles + s * PR_HALF, &map_w, map_to_rank(smem_u32(&t->full[s]), 0), row, k * RW_KB);
            };
            auto load_x = [&](int tile, int k, int s) {
                tma_load_pair(a_tiles + s * RW_A_BYTES, &map_x, map_to_rank(smem_u32(&t->full[s]), 0),
                              tile % m_tiles * 256 + int(rank) * 128, k * RW_KB);
            };
            auto expect = [&](int s) { if (rank == 0) mbar_expect_tx(&t->full[s], 2 * (RW_A_BYTES + PR_HALF)); };
            const int pre = first < total ? min(PR_STAGES, p.ksteps) : 0;
            for (int k = 0; k < pre; ++k) {                             // weights do not depend on the kernel before
                expect(k);
                load_w(first, k, k);
            }
            pdl_wait();
            for (int k = 0; k < pre; ++k) load_x(first, k, k);
            int issued = pre;
            int s = pre == PR_STAGES ? 0 : pre;
            uint32_t ph = pre == PR_STAGES ? 1u : 0u;
            bool ok = true;
            for (int tile = first; tile < total && ok; tile += step)
                for (int k = tile == first ? pre : 0; k < p.ksteps; ++k) {
                    ok = wait(&t->empty[s], ph ^ 1u, 1u);
                    if (!ok) break;
                    expect(s);
                    load_w(tile, k, s);
                    load_x(tile, k, s);
                    ++issued;
                    if (++s == PR_STAGES) { s = 0; ph ^= 1u; }
                }
            if (!ok && rank == 0) drain_copies(t->full, PR_STAGES, issued);      // (its barriers count the copies of both CTAs)
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {                                   // ---- MMA issuer of the pair ----
            // D f32, A and B bf16, both K-major, N = 256, M = 256
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(PR_BN >> 3) << 17) | (uint32_t(256 >> 4) << 24);
            int s = 0, buf = 0;
            uint32_t ph = 0, aph = 0;
            bool ok = true;
            for (int tile = first; tile < total && ok; tile += step) {
                ok = wait(&t->acc_empty[buf], aph ^ 1u, 4u);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + uint32_t(buf * PR_BN);
                for (int k = 0; k < p.ksteps; ++k) {
                    ok = wait(&t->full[s], ph, 2u);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t da = umma_desc_sw128(a_tiles + s * RW_A_BYTES), db = umma_desc_sw128(b_tiles + s * PR_HALF);
#pragma unroll
                    for (int kk = 0; kk < RW_KB * RW_BK / 16; ++kk)
                        umma_bf16_pair(d, da + (kk >> 2) * (RW_A_TILE >> 4) + 2 * (kk & 3), db + (kk >> 2) * (PR_TILE >> 4) + 2 * (kk & 3),
                                       idesc, (k > 0 || kk > 0) ? 1u : 0u);
                    umma_commit_pair(&t->empty[s]);
                    if (++s == PR_STAGES) { s = 0; ph ^= 1u; }
                }
                if (ok) umma_commit_pair(&t->acc_full[buf]);
                if (++buf == 2) { buf = 0; aph ^= 1u; }
            }
            if (!ok) {
                asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(&t->drain)) : "memory");
                mbar_wait(&t->drain, 0);
            }
        }
    } else {                                                            // ---- epilogue: warps 2..5 of both CTAs ----
        const int quad = warp & 3;
        int buf = 0;
        uint32_t aph = 0;
        for (int tile = first; tile < total; tile += step) {
            const bool ok = wait(&t->acc_full[buf], aph, 3u);
            if (!__all_sync(0xffffffffu, ok)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int m = (tile % m_tiles) * 256 + int(rank) * 128 + quad * 32 + lane, nt = tile / m_tiles;
            rw_epilogue<PR_BN>(p, tmem + (uint32_t(quad * 32) << 16) + uint32_t(buf * PR_BN), m, nt);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];"
                             :: "r"(map_to_rank(smem_u32(&t->acc_empty[buf]), 0)) : "memory");
            if (++buf == 2) { buf = 0; aph ^= 1u; }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();                                                     // nobody leaves while the pair's products or barriers need it
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u) : "memory");
    }
}

cudaError_t launch_pair(const void* w, const void* x, TcParams p, cudaStream_t stream, bool pdl) {
    CUtensorMap map_w, map_x;
    if (!make_block_map(&map_w, w, p.swiglu ? 2 * p.N : p.N, p.K, 128, 0) || !make_block_map(&map_x, x, p.M, p.K, RW_BM, 0))
        return cudaErrorInvalidValue;
    const size_t smem = 1024 + size_t(PR_STAGES) * (RW_A_BYTES + PR_HALF) + sizeof(PrSmemTail);
    static PerDeviceOnce once;
    if (once.first()) {
        cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return e;
    }
    const int m_tiles = (p.M + 255) / 256, per = p.swiglu ? PR_BN / 2 : PR_BN, n_tiles = (p.N + per - 1) / per;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * min(sm_count() / 2, m_tiles * n_tiles));
    cfg.blockDim = dim3(RW_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gemm_pair_kernel, map_w, map_x, p, m_tiles, n_tiles);
}

// Which kernel: the least of three fitted times (us; K blocks of 64; measured on distinct cold weights at 300 .. 4093 tokens,
// 2048 .. 6144 wide): a pair takes 0.33 a block and tile, the one-CTA form 0.27 for half the tile's columns and half its
// tokens, the split form of gemm_tc.cu 0.36 for a share of K; the constants are launch, ring fill and the last read-back.
enum Form { kPair, kRows, kSplit };
Form pick_form(const TcParams& p) {
    const int sms = sm_count(), kb = p.K / RW_BK, cols = p.swiglu ? 2 * p.N : p.N;
    auto up = [](int a, int b) { return (a + b - 1) / b; };
    const float pair = 5.5f + 0.33f * kb * up(up(p.M, 256) * up(cols, 256), sms / 2);
    const float rows = 4.2f + 0.27f * kb * up(up(p.M, 128) * up(cols, 128), sms);
    const int s = gemm_tc_splits_for(p.M, p.N, p.K, p.swiglu != 0);
    const float split = 9.f + (1.5f + 0.36f * kb / s) * up(up(cols, 128) * up(p.M, 256) * s, sms);
    return split < pair && split < rows ? kSplit : rows < pair ? kRows : kPair;
}

}  // namespace

cudaError_t gemm_rows_launch(const void* w, const void* x, TcParams p, cudaStream_t stream, bool pdl) {
    // up to 256 tokens the weight stream is the larger time; the wide forms take K in steps of 128 and 32 columns at a time
    // and store 32 bytes a lane
    const uintptr_t at = reinterpret_cast<uintptr_t>(p.y) | reinterpret_cast<uintptr_t>(p.y_lo) | (reinterpret_cast<uintptr_t>(p.residual) << 1);
    const Form f = p.M <= kTcMaxRows || p.K % (RW_KB * RW_BK) || p.N % (p.swiglu ? 64 : 32) || at % 32 ? kSplit : pick_form(p);
    if (f == kSplit) {
        p.splits = gemm_tc_splits_for(p.M, p.N, p.K, p.swiglu != 0);
        return gemm_tc_launch(w, x, p, stream, pdl);
    }
    p.ksteps = p.K / (RW_KB * RW_BK);
    return f == kPair ? launch_pair(w, x, p, stream, pdl) : launch_rows(w, x, p, stream, pdl);
}

}  // namespace tfb
