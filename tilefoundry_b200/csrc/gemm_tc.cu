// Small-batch projection on the 5th-generation tensor cores: Y[M, N] = X[M, K] . W[N, K]^T (+ residual) for
// few tokens (M <= 256; more where a split over K fills the chip best: gemm_rows.cu decides), bf16 in, f32 accumulate, bf16
// out.
//
// At batch 32 a projection is still HBM-bound (64 flop per weight byte against a ridge near 290), but the
// CUDA cores can no longer keep up with the weight stream (it would need ~200 TFLOP/s of FMA), so the
// products move to tcgen05.mma with the operands swapped: the WEIGHT tile is the MMA's 128-row A operand
// and the token block its B operand (BN = 32, 64, 128 or 256 tokens, the least that holds M: up to 256 tokens the weight
// stream is still the larger time, and the split over K is what fills the chip), both K-major in shared memory, the
// 128 x BN f32 accumulator in tensor memory.  The weight stream is what matters: a producer thread keeps a ring of TMA
// tiles of 128 rows x 64 columns (16 KB, 128-byte swizzle, and the BN tokens' 64 columns beside it) in flight per CTA,
// two CTAs per SM up to 128 tokens (one fills its ring while the other streams), completion counted by mbarriers.
//
// Roles in a CTA of 6 warps: warp 0 (one lane) issues TMA loads; warp 1 allocates tensor memory and (one lane)
// issues the MMAs, four per stage (K = 16 each), releasing a stage with tcgen05.commit; warps 2-5 read the
// accumulator back (tcgen05.ld, one TMEM lane quadrant each) and write it out.  K is split over the 1, 2, 3, 4 or 8
// CTAs of a thread-block cluster so that a 2048 x 2048 projection (16 row tiles) still reaches most SMs.  The
// splits' f32 partials never leave the chip: every CTA parks its 128 x BN tile in its own shared memory, and
// after a cluster barrier CTA c adds, in fixed split order (deterministic), token rows c, c + S, ... from all S CTAs through
// distributed shared memory and writes them out, a warp per row with 8 bytes per lane and two rows in flight (one row at a
// time in 2-byte stores: 193 tokens x 12288 x 2048 took 30.7 us, now 20.6; x 2048 x 6144 26.9, now 16.3).
//
// SwiGLU form (p.swiglu): a row tile holds 64 gate rows and the 64 up rows of the same outputs (one TMA box of both halves
// of a [gate; up] matrix), so one accumulator carries both halves; y = bf16(silu(bf16 g)) * bf16 u is written,
// rounding as the batch-1 epilogue.
//
// The weight tiles of the first ring pass do not depend on the kernel before: the producer requests them before
// griddepcontrol.wait and only the token tiles after it.
//
// Every mbarrier wait is bounded; a timeout sets *status, and the CTA still frees its tensor memory.
//
// HBM-bound: algorithmic bytes per launch = N*K*2 (weights) + M*K*2 per row tile from L2.
#include "common.cuh"
#include "kernels.h"
#include "launch.h"
#include "tc.cuh"

#include <algorithm>
#include <cuda.h>

namespace tfb {

constexpr int TC_BM = 128, TC_BK = 64, TC_THREADS = 192;
constexpr int TC_A_BYTES = TC_BM * TC_BK * 2;             // one 64-element K block of the weight tile

// Ring stages by token tile and CTAs per SM: what two resident CTAs (one at 256 tokens) fit into 227 KB.
template <int BN> struct TcShape {
    static constexpr int kStages = BN == 32 ? 5 : BN == 128 ? 3 : 4;
    static constexpr int kCtas = BN == 256 ? 1 : 2;
    static constexpr int kBBytes = BN * TC_BK * 2;
    static constexpr int kStageBytes = TC_A_BYTES + kBBytes;
};

template <int BN>
struct TcSmemTail {
    uint64_t full[TcShape<BN>::kStages], empty[TcShape<BN>::kStages], accum, drain;
    uint32_t tmem_base;
    int aborted;
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// 16 bytes of CTA `rank`'s shared memory at the address `local` has in this CTA's window
__device__ __forceinline__ float4 ld_dsmem_f4(uint32_t local, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

// One token row, tile rows 4q .. 4q+3 summed over the splits -> y.  SwiGLU: rows 4q .. of the gate half and the up rows
// of the same outputs.
__device__ __forceinline__ void tc_store4(const TcParams& p, uint16_t* out, int m, int n, const float (&o)[4]) {
    uint16_t* y = out + size_t(m) * p.N + n;
    if (p.vec4) {
        if (n < p.N)
            *reinterpret_cast<uint2*>(y) = make_uint2(uint32_t(f32_to_bf16_bits(o[0])) | (uint32_t(f32_to_bf16_bits(o[1])) << 16),
                                                      uint32_t(f32_to_bf16_bits(o[2])) | (uint32_t(f32_to_bf16_bits(o[3])) << 16));
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (n + i < p.N) y[i] = f32_to_bf16_bits(o[i]);
}
__device__ __forceinline__ void tc_residual4(const TcParams& p, int m, int n, float (&r)[4]) {
    const uint16_t* src = p.residual + size_t(m) * p.N + n;
    if (p.vec4) {
        const uint2 v = n < p.N ? *reinterpret_cast<const uint2*>(src) : make_uint2(0u, 0u);
        r[0] = bf16_lo(v.x); r[1] = bf16_hi(v.x); r[2] = bf16_lo(v.y); r[3] = bf16_hi(v.y);
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = n + i < p.N ? bf16_bits_to_f32(src[i]) : 0.f;
}

// Sum over the splits of 16 bytes at `local` in every CTA's shared memory, in split order.
__device__ __forceinline__ float4 tc_sum(const TcParams& p, uint32_t local) {
    if (p.splits == 1) {
        float4 v;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(local) : "memory");
        return v;
    }
    float4 part[8], acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int s = 0; s < 8; ++s)
        if (s < p.splits) part[s] = ld_dsmem_f4(local, uint32_t(s));
#pragma unroll
    for (int s = 0; s < 8; ++s)
        if (s < p.splits) { acc.x += part[s].x; acc.y += part[s].y; acc.z += part[s].z; acc.w += part[s].w; }
    return acc;
}

// The finished tile -> y: token rows are dealt to the CTAs of the cluster in turn, a warp takes a row at a time (lane q:
// tile rows 4q ..), two rows in flight.
__device__ __forceinline__ void tc_finish(const TcParams& p, uint32_t red, int mb, int rows, int tile, int split, int warp, int lane) {
    constexpr int NW = TC_THREADS / 32;
    if (p.swiglu) {                                          // lanes 0..15 one row, 16..31 the next
        const int q = lane & 15, n = tile * 64 + 4 * q;
        for (int i = warp * 2 + (lane >> 4); ; i += 2 * NW) {
            const int m = split + i * p.splits;
            if (m >= rows) break;
            const uint32_t at = red + uint32_t((m * TC_BM + 4 * q) * 4);
            const float4 g = tc_sum(p, at), u = tc_sum(p, at + 64 * 4);
            const float o[4] = {round_bf16(silu_f32(round_bf16(g.x))) * round_bf16(u.x), round_bf16(silu_f32(round_bf16(g.y))) * round_bf16(u.y),
                                round_bf16(silu_f32(round_bf16(g.z))) * round_bf16(u.z), round_bf16(silu_f32(round_bf16(g.w))) * round_bf16(u.w)};
            tc_store4(p, p.y, mb + m, n, o);
        }
        return;
    }
    const int n = tile * TC_BM + 4 * lane;
    for (int i = warp; split + i * p.splits < rows; i += 2 * NW) {
        const int m0 = split + i * p.splits, m1 = m0 + NW * p.splits;
        const bool two = m1 < rows;
        float r0[4] = {0.f, 0.f, 0.f, 0.f}, r1[4] = {0.f, 0.f, 0.f, 0.f};
        if (p.residual) {
            tc_residual4(p, mb + m0, n, r0);
            if (two) tc_residual4(p, mb + m1, n, r1);
        }
        const float4 s0 = tc_sum(p, red + uint32_t((m0 * TC_BM + 4 * lane) * 4));
        const float4 s1 = two ? tc_sum(p, red + uint32_t((m1 * TC_BM + 4 * lane) * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
        float o0[4] = {s0.x, s0.y, s0.z, s0.w}, o1[4] = {s1.x, s1.y, s1.z, s1.w};
        if (p.residual) {                                    // TFB_EPI_RESIDUAL's rounding: bf16(acc), bf16(. * scale), then the add
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                o0[e] = round_bf16(o0[e]);
                o1[e] = round_bf16(o1[e]);
                if (p.res_scale != 1.f) { o0[e] = round_bf16(o0[e] * p.res_scale); o1[e] = round_bf16(o1[e] * p.res_scale); }
                o0[e] += r0[e];
                o1[e] += r1[e];
            }
        }
        tc_store4(p, p.y, mb + m0, n, o0);
        if (two) tc_store4(p, p.y, mb + m1, n, o1);
        if (p.y_lo) {
#pragma unroll
            for (int e = 0; e < 4; ++e) { o0[e] -= round_bf16(o0[e]); o1[e] -= round_bf16(o1[e]); }
            tc_store4(p, p.y_lo, mb + m0, n, o0);
            if (two) tc_store4(p, p.y_lo, mb + m1, n, o1);
        }
    }
}

// A weight tile in one request, whatever its form: 128 rows, or 64 gate rows and the 64 up rows of the same outputs (each
// request costs ~0.1 us of the producer's time).
__device__ __forceinline__ void tma_load_w(void* dst, const CUtensorMap* map, uint64_t* bar, int kx, int row) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 :: "r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(kx), "r"(row), "r"(0) : "memory");
}
template <int BN>
__global__ void __launch_bounds__(TC_THREADS, TcShape<BN>::kCtas) gemm_tc_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                const __grid_constant__ CUtensorMap map_x, const TcParams p) {
    constexpr int ST = TcShape<BN>::kStages, STAGE = TcShape<BN>::kStageBytes;
    extern __shared__ unsigned char tc_smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~uintptr_t(1023));
    // stage: the weight tile of 16 KB, then the token tile of BN * 128 bytes (both 1024-byte aligned)
    TcSmemTail<BN>* t = reinterpret_cast<TcSmemTail<BN>*>(base + ST * STAGE);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x, m0 = blockIdx.z * BN, rows = min(p.M - m0, BN), split = p.splits > 1 ? int(cluster_ctarank()) : 0;
    // K steps, dealt to the splits as evenly as they go
    const int k_begin = int((long long)p.ksteps * split / p.splits), k_end = int((long long)p.ksteps * (split + 1) / p.splits);
    const int nsteps = k_end - k_begin;

    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) { mbar_init(&t->full[s], 1); mbar_init(&t->empty[s], 1); }
        mbar_init(&t->accum, 1); mbar_init(&t->drain, 1);
        t->aborted = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {                                                    // BN columns of tensor memory: the 128 x BN f32 tile
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&t->tmem_base)), "r"(uint32_t(BN)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = t->tmem_base;
    pdl_trigger();
    const bool producer = (warp == 0 && lane == 0);
    if (!producer) pdl_wait();

    if (warp == 0) {
        if (lane == 0) {                                                // ---- TMA producer ----
            const int row = p.swiglu ? tile * 64 : tile * TC_BM;
            auto stage = [&](int s) { return base + s * STAGE; };
            const int pre = min(nsteps, ST);
            for (int i = 0; i < pre; ++i) {                             // weights never depend on the kernel before
                mbar_expect_tx(&t->full[i], STAGE);
                tma_load_w(stage(i), &map_w, &t->full[i], (k_begin + i) * TC_BK, row);
            }
            pdl_wait();
            for (int i = 0; i < pre; ++i) tma_load_2d(stage(i) + TC_A_BYTES, &map_x, &t->full[i], (k_begin + i) * TC_BK, m0);
            for (int i = pre; i < nsteps; ++i) {
                const int s = i % ST;
                if (!mbar_wait(&t->empty[s], ((i / ST) & 1) ^ 1)) {
                    t->aborted = 1;
                    atomicExch(p.status, 1u);
                    drain_copies(t->full, ST, i);
                    break;
                }
                mbar_expect_tx(&t->full[s], STAGE);
                tma_load_w(stage(s), &map_w, &t->full[s], (k_begin + i) * TC_BK, row);
                tma_load_2d(stage(s) + TC_A_BYTES, &map_x, &t->full[s], (k_begin + i) * TC_BK, m0);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {                                                // ---- MMA issuer ----
            // instruction descriptor: D f32, A and B bf16, both K-major, N = BN, M = 128
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(BN >> 3) << 17) | (uint32_t(TC_BM >> 4) << 24);
            bool ok = true;
            for (int i = 0; i < nsteps && ok; ++i) {
                const int s = i % ST;
                ok = mbar_wait(&t->full[s], (i / ST) & 1);
                if (!ok) { t->aborted = 1; atomicExch(p.status, 2u); break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t da = umma_desc_sw128(base + s * STAGE), db = umma_desc_sw128(base + s * STAGE + TC_A_BYTES);
#pragma unroll
                for (int kk = 0; kk < TC_BK / 16; ++kk)                 // 16 bf16 = 32 bytes = 2 descriptor units per step
                    umma_bf16(tmem, da + 2 * kk, db + 2 * kk, idesc, (i > 0 || kk > 0) ? 1u : 0u);
                umma_commit(&t->empty[s]);                              // arrives when these MMAs have read the stage
            }
            if (ok) umma_commit(&t->accum);                             // arrives when the accumulator is complete
            else drain_products(&t->drain);
        }
    } else {                                                            // ---- warps 2..5 read the accumulator back ----
        const int quad = warp & 3;                                      // the TMEM lane quadrant this warp may read
        bool ok = nsteps > 0 ? mbar_wait(&t->accum, 0) : true;
        if (!ok) { t->aborted = 1; atomicExch(p.status, 3u); }
        // park this CTA's sums as red[m][r] in the ring: every load into it has landed and every MMA that read it has
        // completed once the accumulator barrier fires
        float* red = reinterpret_cast<float*>(base);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int c = 0; c < rows; c += 32) {
            uint32_t v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
            if (ok && nsteps > 0) tmem_ld32(v, tmem + (uint32_t(quad * 32) << 16) + uint32_t(c));
#pragma unroll
            for (int m = 0; m < 32; ++m) red[(c + m) * TC_BM + quad * 32 + lane] = __uint_as_float(v[m]);
        }
    }

    // ---- teardown, and the split-K reduction through distributed shared memory ----
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(uint32_t(BN)) : "memory");
    }
    if (p.splits > 1) cluster_sync_all();                               // every split's tile is parked
    tc_finish(p, smem_u32(base), m0, rows, tile, split, warp, lane);
    if (p.splits > 1) cluster_sync_all();                               // nobody leaves while its tile is still being read
}

// K splits = CTAs of one cluster, a power of two (or three, below): as many as keep the grid within `resident` CTAs, at most
// `most` (8 is the portable cluster size).
static int splits_for_tiles(int tiles, int k, int resident, int most) {
    int splits = 1;
    while (splits < most && tiles * splits * 2 <= resident && (k / TC_BK) % (splits * 2) == 0) splits *= 2;
    return splits;
}
// Up to 128 tokens two CTAs share an SM, worth it up to 4 splits (6400 gate/up pairs x 2560, 128 tokens: two splits 20.1 us,
// unsplit 23.8; 8192 x 2048: four 13.5, two 15.9; the MiniCPM3 prompt of 128 tokens 7.1 ms, one CTA per SM 7.6); 8 only within
// one CTA per SM (4096 x 2048, 128 tokens: eight 12.4 us, four 11.6; alone and with 32 tokens eight are 0.3 us faster, but the
// 32-sequence step of Qwen3 is 2.70 ms with them, 2.63 with four).  Up to 64 tokens a share of less than 20 blocks of K is not
// worth it where most SMs would have two CTAs (6144 gate/up pairs x 2048, 96 tiles, 32 tokens: two splits 14.7 us, unsplit
// 14.4; 16384 x 2048, 128 tiles, 64 tokens: 17.9, 17.6; but 10240 x 2048, 80 tiles: 14.0, 15.0; and 6400 x 2560: 16.1, 16.7).
static int splits_two_per_sm(int tiles, int k, bool few) {
    const int sms = sm_count(), s = splits_for_tiles(tiles, k, 2 * sms, 4);
    if (s == 2 && few && 8 * tiles > 5 * sms && k < 40 * TC_BK) return 1;
    return s == 4 ? std::max(s, splits_for_tiles(tiles, k, sms, 8)) : s;
}
int gemm_tc_splits(int n, int k) { return splits_two_per_sm((n + TC_BM - 1) / TC_BM, k, true); }
int gemm_tc_splits_swiglu(int n, int k) { return splits_two_per_sm((n + 63) / 64, k, true); }
// More than 192 of up to 256 tokens as two tiles of 128 beside one another, where the weight tiles are few: two CTAs share
// an SM again (256 tokens: 2304 x 2560 12.2 us, as one tile 13.4; 2048 x 2048 11.1, 12.2; 193: 11.4, 12.1 and 10.8, 11.0).
// With fewer tokens in the second tile the first is not worth its weights twice (129: 11.5, 10.7 and 10.8, 9.6).  More weight
// tiles fill the chip as they are (2560 x 2560, 20 tiles, 256 tokens: 15.4 us as halves, 13.4 as one).
static bool two_halves(int m, int tiles) { return m > 192 && m <= 256 && 8 * tiles <= sm_count(); }
int gemm_tc_splits_for(int m, int n, int k, bool swiglu) {
    const int tiles = swiglu ? (n + 63) / 64 : (n + TC_BM - 1) / TC_BM;
    if (two_halves(m, tiles)) return splits_for_tiles(2 * tiles, k, sm_count(), 4);
    if (m > 128) {
        // A CTA takes an SM to itself: at most 4 splits, and 4 or 3 only where that many clusters find room at the same time --
        // of 148 SMs 33 clusters of four and 45 of three do, one more and they run in two waves (K 2048, 256 tokens, four: 33
        // tiles 13.7 us, 34 24.6; three: 45 tiles 16.3, 46 28.3; 2048 x 2048 at 193 tokens took 19 us with clusters of 8).
        // Nine tenths of the SMs keep clear of both.  Three, where four is too many or does not divide K, against two (K steps
        // are dealt as evenly as they go): 40 tiles, K 2560, 256 tokens 16.2 us, 20.2.
        const int all = tiles * ((m + 255) / 256), room = sm_count() * 9 / 10, s = splits_for_tiles(all, k, sm_count(), 4);
        if (s == 4 && 4 * all <= room) return 4;
        return s >= 2 && 3 * all <= room ? 3 : std::min(s, 2);
    }
    return splits_two_per_sm(tiles, k, m <= 64);
}

// Weights [rows][K], boxes of 64 elements x box_rows of each half (halves = 2: gate rows, then up rows).
static bool make_w_map(CUtensorMap* map, const void* ptr, int n, int k, int box_rows, int halves) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {cuuint64_t(k), cuuint64_t(n), cuuint64_t(halves)};
    const cuuint64_t strides[2] = {cuuint64_t(k) * 2, cuuint64_t(n) * k * 2};
    const cuuint32_t box[3] = {TC_BK, cuuint32_t(box_rows), cuuint32_t(halves)};
    const cuuint32_t elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN>
static cudaError_t launch_bn(const void* w, const void* x, TcParams p, cudaStream_t stream, bool pdl) {
    CUtensorMap map_w, map_x;
    if (!make_w_map(&map_w, w, p.N, p.K, p.swiglu ? 64 : TC_BM, p.swiglu ? 2 : 1) || !make_map_bf16(&map_x, x, p.M, p.K, BN))
        return cudaErrorInvalidValue;
    p.ksteps = p.K / TC_BK;
    const int tiles = p.swiglu ? (p.N + 63) / 64 : (p.N + TC_BM - 1) / TC_BM;
    const size_t smem = 1024 + size_t(TcShape<BN>::kStages) * TcShape<BN>::kStageBytes + sizeof(TcSmemTail<BN>);
    static PerDeviceOnce once;
    if (once.first()) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return e;
    }
    const dim3 grid(tiles, p.splits, (p.M + BN - 1) / BN), block(TC_THREADS);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    if (p.splits > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = 1;
        attr[na].val.clusterDim.y = unsigned(p.splits);
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return cudaLaunchKernelEx(&cfg, gemm_tc_kernel<BN>, map_w, map_x, p);
}

// The least token tile that holds M (a wider one only adds token bytes per weight tile and shortens the ring); above 256
// tokens, tiles of 256.
cudaError_t gemm_tc_launch(const void* w, const void* x, TcParams p, cudaStream_t stream, bool pdl) {
    p.vec4 = (p.N & 3) == 0 && ((reinterpret_cast<uintptr_t>(p.y) | reinterpret_cast<uintptr_t>(p.y_lo) | reinterpret_cast<uintptr_t>(p.residual)) & 7) == 0;
    if (p.M <= 32) return launch_bn<32>(w, x, p, stream, pdl);
    if (p.M <= 64) return launch_bn<64>(w, x, p, stream, pdl);
    if (p.M <= 128 || two_halves(p.M, p.swiglu ? (p.N + 63) / 64 : (p.N + TC_BM - 1) / TC_BM)) return launch_bn<128>(w, x, p, stream, pdl);
    return launch_bn<256>(w, x, p, stream, pdl);
}

}  // namespace tfb
