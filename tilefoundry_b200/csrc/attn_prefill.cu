// Attention of a prompt chunk over the paged bf16 cache on the tensor cores: for grouped-query heads of width 128 q/k norm +
// RoPE + cache append (prefill_rows_kernel), then causal flash attention (prefill_attn_kernel); for latent attention
// (MiniCPM3) the same kernel over keys and values expanded from the latents.
//
// Compute-bound: every (query, cached position, query head) takes 128 multiply-adds for the score and 128 for the
// weighted V.  As one CTA per token over the batched decode kernel a 4093-token prompt spent most of its 448 ms here
// and in re-reading the cache once per token; here 128 query rows share every K/V tile.
//
// One CTA: KV head g, 128 query rows = 128/G tokens x its G query heads (they share the K/V tiles).  K/V in tiles of 128
// positions by TMA (two 64-position pages, two 64-element halves each; 128-byte swizzle).  Two CTAs are resident per SM
// (96 KB of shared memory and 256 tensor-memory columns each): one CTA's softmax runs under the other's products, so no
// tile is double-buffered.  Grid: query tiles from the last (longest) to the first.
//   warp 0     TMA requests: Q once, K and V of each tile as their stage becomes free
//   warp 1     tcgen05.mma: S = Q K^T (128 x 128, tensor memory); O += P V
//   warps 2-5  softmax, one thread per query row: running maximum and sum in registers, P back into tensor memory
// P keeps f32 accuracy: it goes in as two bf16 terms (hi = bf16(p), lo = bf16(p - hi)), each a product of its own with
// V, so the weighted sum is good to 2^-17 of its terms as the f32 sums of the decode kernels are (to within V's own
// rounding, which both share).  P overwrites S in place: columns 32c .. 32c+15 the hi terms of scores 32c .. 32c+31, the
// next 16 their lo terms.  O is only rescaled when a row's maximum has grown by more than 8 (in log2), exact either way.
//
// The product meets every row of a V tile, so a row that a query must not see is more than a weight of zero (0 x Inf and
// 0 x NaN are NaN).  Rows past the chunk (a page's stale rows) are zeroed in shared memory by the requesting
// warp while the softmax runs (by the softmax warps themselves it cost 1.5 us a layer); a warp one of whose
// results is not finite -- a later token of the tile may have done that, or an earlier one rightly -- takes its
// rows again by a plain walk over the positions each query sees (slow_rows), as the decode kernels take them.  (Looking through
// the V tile for such values instead cost 1.6 us a layer.)
//
// V as the second operand is [position][d] in shared memory, so N is its contiguous dimension: an MN-major descriptor
// (64-element blocks 16 KB apart, groups of eight positions 1 KB apart).
//
// Every mbarrier wait is bounded; a timeout sets *status, and the CTA still frees its tensor memory.
#include "common.cuh"
#include "kernels.h"
#include "launch.h"
#include "tc.cuh"

namespace tfb {
namespace {

constexpr int PA_D = 128, PA_KV = 128, PA_THREADS = 192;
constexpr int PA_HALF = 128 * 128;                       // bytes of 128 rows x 64 bf16
constexpr int PA_TILE = 2 * PA_HALF;
constexpr float kLog2e = 1.4426950408889634f;

struct PaTail {
    uint64_t q_full, k_full, v_full, v_clean, k_empty, v_empty, s_full, p_full, o_done, drain;
    uint32_t tmem_base;
    volatile int aborted;
};

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 :: "r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ uint64_t desc_mn_sw128(const void* tile) {
    uint64_t d = 0;
    d |= uint64_t((smem_u32(tile) & 0x3FFFF) >> 4);
    d |= uint64_t(PA_HALF >> 4) << 16;                   // between 64-element blocks of N
    d |= uint64_t(1024 >> 4) << 32;                      // between groups of eight K rows
    d |= uint64_t(1) << 46;
    d |= uint64_t(2) << 61;
    return d;
}
// K-major rows of 64 bytes with 64-byte swizzle, groups of eight rows 512 bytes apart
__device__ __forceinline__ uint64_t desc_k_sw64(const void* tile) {
    uint64_t d = 0;
    d |= uint64_t((smem_u32(tile) & 0x3FFFF) >> 4);
    d |= uint64_t(1) << 16;
    d |= uint64_t(512 >> 4) << 32;
    d |= uint64_t(1) << 46;
    d |= uint64_t(4) << 61;
    return d;
}
// A operand from tensor memory
__device__ __forceinline__ void umma_bf16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 :: "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
                 :: "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                    "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
                    "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
                    "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]),
                    "r"(taddr) : "memory");
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// c + 0 * a of bf16 pairs: NaN where a is not finite
__device__ __forceinline__ uint32_t times_zero(uint32_t a, uint32_t c) {
    uint32_t r;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(0u), "r"(c));
    return r;
}
__device__ __forceinline__ float ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// ---- q/k norm + RoPE + append -----------------------------------------------------------------------------------
// One CTA per token, one warp per 128-wide vector at a time: q heads are normalised, rotated, scaled and written back in
// place (bf16, the rounding points of the decode kernels), k goes to the cache likewise, v as it is.
__global__ void __launch_bounds__(256) prefill_rows_kernel(const PrefillAttnParams p) {
    const int m = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_trigger();
    pdl_wait();
    const int pos = p.pos_rows[m];
    if (pos < 0 || pos >= p.max_ctx) return;
    const int page = p.block_table[pos / p.page_size];
    const size_t row = size_t(page) * p.page_size + pos % p.page_size;
    uint16_t* qkv = p.qkv + size_t(m) * (p.hq + 2 * p.hkv) * PA_D;
    // lane l: elements 2l, 2l+1 and their rotate-half partners 64 + 2l, 65 + 2l
    auto at2 = [lane](const uint16_t* v, int half) { return *reinterpret_cast<const uint32_t*>(v + 64 * half + 2 * lane); };
    uint32_t c2[2], s2[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        c2[h] = at2(p.cos_table + size_t(pos) * PA_D, h);
        s2[h] = at2(p.sin_table + size_t(pos) * PA_D, h);
    }
    for (int vi = warp; vi < p.hq + 2 * p.hkv; vi += 8) {
        uint16_t* src = qkv + size_t(vi) * PA_D;
        const uint32_t w0 = at2(src, 0), w1 = at2(src, 1);
        if (vi >= p.hq + p.hkv) {                         // v
            uint16_t* dst = p.v_pool + (row * p.hkv + (vi - p.hq - p.hkv)) * PA_D + 2 * lane;
            *reinterpret_cast<uint32_t*>(dst) = w0;
            *reinterpret_cast<uint32_t*>(dst + 64) = w1;
            continue;
        }
        float x[4] = {bf16_lo(w0), bf16_hi(w0), bf16_lo(w1), bf16_hi(w1)};
        const float rstd = rsqrtf(warp_sum(fmaf(x[0], x[0], fmaf(x[1], x[1], fmaf(x[2], x[2], x[3] * x[3])))) / float(PA_D) + p.eps);
        const uint16_t* gm = vi < p.hq ? p.gamma_q : p.gamma_k;
        const uint32_t g0 = at2(gm, 0), g1 = at2(gm, 1);
        const float gain[4] = {bf16_lo(g0), bf16_hi(g0), bf16_lo(g1), bf16_hi(g1)};
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = round_bf16(round_bf16(x[i] * rstd) * gain[i]);
        const float c[4] = {bf16_lo(c2[0]), bf16_hi(c2[0]), bf16_lo(c2[1]), bf16_hi(c2[1])};
        const float s[4] = {bf16_lo(s2[0]), bf16_hi(s2[0]), bf16_lo(s2[1]), bf16_hi(s2[1])};
        float out[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float partner = i < 2 ? -x[i + 2] : x[i - 2];
            out[i] = round_bf16(__fadd_rn(__fmul_rn(x[i], c[i]), __fmul_rn(partner, s[i])));
            if (vi < p.hq) out[i] *= p.scale;
        }
        uint16_t* dst = vi < p.hq ? src : p.k_pool + (row * p.hkv + (vi - p.hq)) * PA_D;
        *reinterpret_cast<uint32_t*>(dst + 2 * lane) = pack2(out[0], out[1]);
        *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = pack2(out[2], out[3]);
    }
}

// ---- latent form: the rows of a chunk before its projections -------------------------------------------------------
// CTAs 0 .. m-1, one token each: the low-rank norm of the compressed query (-> qa), the norm of the compressed kv vector and
// the rotated shared key slice (-> the pool's row and, the former, lat[first + token]).  The CTAs behind them copy the
// latents of earlier positions from the pool to lat, a warp per row.
__global__ void __launch_bounds__(256) mla_chunk_rows_kernel(const MlaChunkParams p) {
    constexpr int KVL = 256, ROPE = 32, ROW = KVL + ROPE;
    __shared__ float red[32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_trigger();
    pdl_wait();
    auto pool_row = [&](int pos) { return p.pool + (size_t(p.block_table[pos / p.page_size]) * p.page_size + pos % p.page_size) * ROW; };
    if (int(blockIdx.x) >= p.m) {
        const int pos = (blockIdx.x - p.m) * 8 + warp;
        if (pos < p.first)
            *reinterpret_cast<uint4*>(p.lat + size_t(pos) * KVL + lane * 8) = *reinterpret_cast<const uint4*>(pool_row(pos) + lane * 8);
        return;
    }
    const int m = blockIdx.x, pos = p.pos_rows[m], QL = p.q_lora;
    if (pos < 0 || pos >= p.max_ctx) return;
    const uint16_t* row = p.qkv_a + size_t(m) * (QL + ROW);
    float v[4], ss = 0.f;                                 // q_lora <= 1024
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[i] = tid + 256 * i < QL ? bf16_bits_to_f32(row[tid + 256 * i]) : 0.f;
        ss = fmaf(v[i], v[i], ss);
    }
    const float c = bf16_bits_to_f32(row[QL + tid]);
    const float rq = rsqrtf(block_sum(ss, red) / float(QL) + p.lora_eps);
    const float rk = rsqrtf(block_sum(c * c, red) / float(KVL) + p.lora_eps);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (tid + 256 * i < QL)
            p.qa[size_t(m) * QL + tid + 256 * i] = f32_to_bf16_bits(round_bf16(v[i] * rq) * bf16_bits_to_f32(p.gamma_q_a[tid + 256 * i]));
    uint16_t* dst = pool_row(pos);
    const uint16_t lat = f32_to_bf16_bits(round_bf16(c * rk) * bf16_bits_to_f32(p.gamma_kv_a[tid]));
    dst[tid] = lat;
    p.lat[size_t(p.first + m) * KVL + tid] = lat;
    if (tid < ROPE) {
        const uint16_t* kr = row + QL + KVL;
        const float k0 = bf16_bits_to_f32(kr[tid]);
        const float kp = tid < ROPE / 2 ? -bf16_bits_to_f32(kr[tid + ROPE / 2]) : bf16_bits_to_f32(kr[tid - ROPE / 2]);
        dst[KVL + tid] = f32_to_bf16_bits(__fadd_rn(__fmul_rn(k0, bf16_bits_to_f32(p.cos_table[size_t(pos) * ROPE + tid])),
                                                    __fmul_rn(kp, bf16_bits_to_f32(p.sin_table[size_t(pos) * ROPE + tid]))));
    }
}

// The projected queries in place: scale on the 64 no-position values, rotation and scale on the 32 rotary ones.
__global__ void __launch_bounds__(256) mla_chunk_q_kernel(const MlaChunkParams p) {
    const int m = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_trigger();
    pdl_wait();
    const int pos = p.pos_rows[m];
    if (pos < 0 || pos >= p.max_ctx) return;
    const float c = bf16_bits_to_f32(p.cos_table[size_t(pos) * 32 + lane]), s = bf16_bits_to_f32(p.sin_table[size_t(pos) * 32 + lane]);
    for (int h = warp; h < p.heads; h += 8) {             // lane: two no-position values and one rotary one
        uint16_t* q = p.q + (size_t(m) * p.heads + h) * 96;
        uint32_t* nope = reinterpret_cast<uint32_t*>(q) + lane;
        const uint32_t w = *nope;
        *nope = pack2(bf16_lo(w) * p.scale, bf16_hi(w) * p.scale);
        const float x = bf16_bits_to_f32(q[64 + lane]);
        const float other = __shfl_xor_sync(0xffffffffu, x, 16), partner = lane < 16 ? -other : other;
        q[64 + lane] = f32_to_bf16_bits(round_bf16(__fadd_rn(__fmul_rn(x, c), __fmul_rn(partner, s))) * p.scale);
    }
}

// ---- the plain walk -------------------------------------------------------------------------------------------------
// 32 query rows from row0 of the tile, one after the other by a warp: f32 scores and sums over positions 0 .. the query's own,
// nothing else is read.  Only where a result was not finite; four positions in flight.
__device__ __forceinline__ float two_terms(uint16_t hi, uint16_t lo) {     // (of a value that is not finite, hi is the whole)
    const float h = bf16_bits_to_f32(hi);
    return (hi & 0x7f80u) == 0x7f80u ? h : h + bf16_bits_to_f32(lo);
}
template <int G, bool MLA>
__device__ __noinline__ void slow_rows(const PrefillAttnParams& p, int first, int m0, int g, int row0, int lane) {
    constexpr int OW = MLA ? 64 : PA_D, VPL = OW / 32, QPL = MLA ? 3 : 4;   // values a lane holds of an output, of a query
    for (int r = row0; r < row0 + 32; ++r) {
        const int tok = m0 + r / G, pos = first + tok, head = g * G + r % G;
        if (tok >= p.m || pos >= p.max_ctx) continue;
        float q[QPL], o[VPL], m = -INFINITY, l = 0.f;
#pragma unroll
        for (int i = 0; i < QPL; ++i)
            q[i] = bf16_bits_to_f32(MLA ? p.qkv[(size_t(tok) * p.hq + head) * 96 + lane + 32 * i]
                                        : p.qkv[(size_t(tok) * (p.hq + 2 * p.hkv) + head) * PA_D + lane + 32 * i]);
#pragma unroll
        for (int i = 0; i < VPL; ++i) o[i] = 0.f;
        for (int t0 = 0; t0 <= pos; t0 += 4) {
            float s[4], v[4][VPL];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int t = min(t0 + j, pos);
                const size_t row = size_t(p.block_table[t / p.page_size]) * p.page_size + t % p.page_size;
                s[j] = 0.f;
                if (MLA) {
                    const size_t at = (size_t(t) * p.hkv + g) * 128 + lane;
#pragma unroll
                    for (int i = 0; i < 2; ++i) s[j] = fmaf(q[i], two_terms(p.k_pool[at + 32 * i], p.v_pool[at + 32 * i]), s[j]);
                    s[j] = fmaf(q[QPL - 1], bf16_bits_to_f32(p.lat_pool[row * 288 + 256 + lane]), s[j]);
#pragma unroll
                    for (int i = 0; i < VPL; ++i) v[j][i] = two_terms(p.k_pool[at + 64 + 32 * i], p.v_pool[at + 64 + 32 * i]);
                } else {
                    const size_t at = (row * p.hkv + g) * PA_D + lane;
#pragma unroll
                    for (int i = 0; i < QPL; ++i) s[j] = fmaf(q[i], bf16_bits_to_f32(p.k_pool[at + 32 * i]), s[j]);
#pragma unroll
                    for (int i = 0; i < VPL; ++i) v[j][i] = bf16_bits_to_f32(p.v_pool[at + 32 * i]);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (t0 + j > pos) break;
                const float sc = warp_sum(s[j]), nm = fmaxf(m, sc);
                const float f = m == -INFINITY ? 0.f : __expf(m - nm), w = sc == -INFINITY ? 0.f : __expf(sc - nm);
                l = l * f + w;
#pragma unroll
                for (int i = 0; i < VPL; ++i) o[i] = fmaf(w, v[j][i], o[i] * f);
                m = nm;
            }
        }
#pragma unroll
        for (int i = 0; i < VPL; ++i) p.out[(size_t(tok) * p.hq + head) * OW + lane + 32 * i] = f32_to_bf16_bits(o[i] / l);
    }
}

// ---- flash attention ----------------------------------------------------------------------------------------------
// GQA form (G query heads per KV head): maps q, k, v.  Latent form (MLA, G = 1): a head's keys and values are expanded from
// the latents to hi + lo bf16 terms beforehand, so a tile is K_hi | K_lo (64 wide each) and the rotary part shared by all
// heads (32 wide, 64-byte swizzle, from the latent pool's pages), V_hi | V_lo; S = q_nope (K_hi + K_lo) + q_rope k_rope and
// O = P_hi V_hi + P_lo V_hi + P_hi V_lo, the f32 accuracy of the absorbed form.  Maps: q, q_rope, hi, lo, pool.
template <int G, bool MLA>
__global__ void __launch_bounds__(PA_THREADS, 2) prefill_attn_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                     const __grid_constant__ CUtensorMap map_k,
                                                                     const __grid_constant__ CUtensorMap map_v,
                                                                     const __grid_constant__ CUtensorMap map_qr,
                                                                     const __grid_constant__ CUtensorMap map_kr,
                                                                     const __grid_constant__ PrefillAttnParams p) {
    constexpr int TOK = 128 / G;                         // tokens of a query tile
    constexpr int OW = MLA ? 64 : PA_D;                  // width of a head's output
    constexpr int Q_BYTES = MLA ? PA_HALF + PA_HALF / 2 : PA_TILE, K_BYTES = MLA ? PA_TILE + PA_HALF / 2 : PA_TILE;
    extern __shared__ unsigned char pa_smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(pa_smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char *qs = base, *ks = base + Q_BYTES, *vs = ks + K_BYTES;   // (the latent form's split of the same 96 KB)
    PaTail* t = reinterpret_cast<PaTail*>(base + 3 * PA_TILE);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = (gridDim.y - 1 - blockIdx.y) * TOK, g = blockIdx.x;   // the longest tiles of every KV head first

    if (threadIdx.x == 0) {
        mbar_init(&t->q_full, 1); mbar_init(&t->k_full, 1); mbar_init(&t->v_full, 1); mbar_init(&t->v_clean, 1);
        mbar_init(&t->k_empty, 1); mbar_init(&t->v_empty, 1); mbar_init(&t->s_full, 1);
        mbar_init(&t->p_full, 4); mbar_init(&t->o_done, 1); mbar_init(&t->drain, 1);
        t->aborted = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {                                     // S / P: columns 0..127, O: 128..255
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&t->tmem_base)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = t->tmem_base;
    pdl_trigger();
    pdl_wait();

    const int first = p.pos_rows[0];                     // positions of a chunk are consecutive
    const int last = min(first + min(m0 + TOK, p.m) - 1, p.max_ctx - 1);
    const int n_tiles = first < 0 ? 0 : (last + 1 + PA_KV - 1) / PA_KV;
    // V rows of the last tile past the chunk, whatever the pages hold there (the latent form's tiles end with the chunk: zeros)
    const int stale = MLA || n_tiles == 0 ? 0 : max(n_tiles * PA_KV - min(first + p.m, p.max_ctx), 0);

    auto wait = [&](uint64_t* bar, uint32_t parity, unsigned role) -> bool {
        if (t->aborted) return false;
        if (mbar_wait(bar, parity)) return true;
        t->aborted = 1;
        atomicExch(p.status, role);
        return false;
    };

    if (warp == 0) {
        if (lane == 0 && n_tiles > 0) {
            mbar_expect_tx(&t->q_full, Q_BYTES);
            if (MLA) {
                tma_load_3d(qs, &map_q, &t->q_full, 0, g, m0);
                tma_load_3d(qs + PA_HALF, &map_qr, &t->q_full, 64, g, m0);
            } else {
                for (int h = 0; h < 2; ++h) tma_load_3d(qs + h * PA_HALF, &map_q, &t->q_full, 64 * h, g * G, m0);
            }
            auto page_row = [&](int tile, int q) {       // (a page past the context holds masked positions only: any page will do)
                const int pos = min(tile * PA_KV + q * 64, last);
                return p.block_table[pos / p.page_size] * p.page_size + (pos % p.page_size & ~63);
            };
            auto load = [&](unsigned char* dst, const CUtensorMap* map, uint64_t* bar, int tile) {
                mbar_expect_tx(bar, PA_TILE);
                for (int q = 0; q < 2; ++q)
                    for (int h = 0; h < 2; ++h)
                        tma_load_3d(dst + h * PA_HALF + q * (PA_HALF / 2), map, bar, 64 * h, g, page_row(tile, q));
            };
            auto load_mla = [&](unsigned char* dst, uint64_t* bar, int tile, bool keys) {
                mbar_expect_tx(bar, keys ? K_BYTES : PA_TILE);
                tma_load_3d(dst, &map_k, bar, keys ? 0 : 64, g, tile * PA_KV);
                tma_load_3d(dst + PA_HALF, &map_v, bar, keys ? 0 : 64, g, tile * PA_KV);
                if (keys)
                    for (int q = 0; q < 2; ++q) tma_load_3d(dst + PA_TILE + q * (PA_HALF / 4), &map_kr, bar, 256, 0, page_row(tile, q));
            };
            bool ok = true;
            int n_k = 0, n_v = 0;
            for (int i = 0; i < n_tiles && ok; ++i) {
                ok = wait(&t->k_empty, (i & 1) ^ 1, 1u);
                if (!ok) break;
                if (MLA) load_mla(ks, &t->k_full, i, true); else load(ks, &map_k, &t->k_full, i);
                n_k = i + 1;
                ok = wait(&t->v_empty, (i & 1) ^ 1, 1u);
                if (!ok) break;
                if (MLA) load_mla(vs, &t->v_full, i, false); else load(vs, &map_v, &t->v_full, i);
                n_v = i + 1;
            }
            if (!ok) {
                drain_copies(&t->q_full, 1, 1);
                drain_copies(&t->k_full, 1, n_k);
                drain_copies(&t->v_full, 1, n_v);
            }
        }
        __syncwarp();
        if (stale > 0) {                                 // zeros, under the softmax
            const bool ok = wait(&t->v_full, (n_tiles - 1) & 1, 1u);
            if (__all_sync(0xffffffffu, ok)) {
                for (int c = lane; c < stale * 16; c += 32)
                    reinterpret_cast<uint4*>(vs + (c & 8 ? PA_HALF : 0) + (PA_KV - 1 - (c >> 4)) * 128)[c & 7] = make_uint4(0u, 0u, 0u, 0u);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // before the products read them
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(&t->v_clean)) : "memory");
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && n_tiles > 0) {
            // D f32, A and B bf16, N = 128 (OW), M = 128; the second product's B is MN-major
            const uint32_t id_qk = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(PA_KV >> 3) << 17) | (uint32_t(128 >> 4) << 24);
            const uint32_t id_pv = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | (uint32_t(OW >> 3) << 17) | (uint32_t(128 >> 4) << 24);
            bool ok = wait(&t->q_full, 0, 2u);
            for (int i = 0; i < n_tiles && ok; ++i) {
                ok = wait(&t->k_full, i & 1, 2u);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                // (issued after the last tile's P V: the products run in order)
                if (MLA) {
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)        // K_hi, then K_lo
                        umma_bf16(tmem, umma_desc_sw128(qs) + 2 * (kk & 3), umma_desc_sw128(ks + (kk >> 2) * PA_HALF) + 2 * (kk & 3),
                                  id_qk, kk > 0 ? 1u : 0u);
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk)
                        umma_bf16(tmem, desc_k_sw64(qs + PA_HALF) + 2 * kk, desc_k_sw64(ks + PA_TILE) + 2 * kk, id_qk, 1u);
                } else {
#pragma unroll
                    for (int kk = 0; kk < PA_D / 16; ++kk)
                        umma_bf16(tmem, umma_desc_sw128(qs + (kk >> 2) * PA_HALF) + 2 * (kk & 3),
                                  umma_desc_sw128(ks + (kk >> 2) * PA_HALF) + 2 * (kk & 3), id_qk, kk > 0 ? 1u : 0u);
                }
                umma_commit(&t->k_empty);
                umma_commit(&t->s_full);
                ok = wait(&t->v_full, i & 1, 2u) && (stale == 0 || i + 1 < n_tiles || wait(&t->v_clean, 0, 2u)) && wait(&t->p_full, i & 1, 2u);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t dv = desc_mn_sw128(vs);
#pragma unroll
                for (int kk = 0; kk < PA_KV / 16; ++kk)
#pragma unroll
                    for (int term = 0; term < (MLA ? 3 : 2); ++term)      // P_hi V, P_lo V (and P_hi V_lo)
                        umma_bf16_ta(tmem + 128, tmem + 32 * (kk >> 1) + 8 * (kk & 1) + 16 * (term == 1 ? 1 : 0),
                                     dv + uint64_t(kk * (2048 >> 4)) + uint64_t(term == 2 ? PA_HALF >> 4 : 0), id_pv,
                                     (i > 0 || kk > 0 || term > 0) ? 1u : 0u);
                umma_commit(&t->v_empty);
                umma_commit(&t->o_done);
            }
            if (!ok) drain_products(&t->drain);
        }
    } else if (n_tiles > 0) {
        const int quad = warp & 3, r = quad * 32 + lane; // query row: token r / G of the tile, head r % G
        const uint32_t trow = tmem + (uint32_t(quad * 32) << 16);
        const int tok = m0 + r / G, my_pos = first + tok;
        // maximum in log2 units: below any score worth a weight, but a number (a row all of whose scores are -infinity or
        // lower than this gets no weight, and with it the plain walk)
        float m_run = -1e30f, l_run = 0.f;
        bool ok = true;
        for (int i = 0; i < n_tiles; ++i) {
            ok = wait(&t->s_full, i & 1, 3u);
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int valid = my_pos - i * PA_KV;        // scores 0 .. valid of this tile count
            const bool whole = __all_sync(0xffffffffu, valid >= PA_KV - 1);
            uint32_t v[PA_KV / 32][32];                  // the row's scores, in registers until they are probabilities
#pragma unroll
            for (int c = 0; c < PA_KV / 32; ++c) tmem_ld32_async(v[c], trow + 32 * c);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < PA_KV / 32; ++c) tmem_pin(v[c]);
            if (!whole) {
#pragma unroll
                for (int c = 0; c < PA_KV / 32; ++c)
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (32 * c + j > valid) v[c][j] = 0xff800000u;   // -infinity
            }
            float mq[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < PA_KV / 32; ++c)
#pragma unroll
                for (int j = 0; j < 32; j += 2)
                    mq[c] = fmaxf(mq[c], fmaxf(__uint_as_float(v[c][j]), __uint_as_float(v[c][j + 1])));
            float mx = fmaxf(fmaxf(mq[0], mq[1]), fmaxf(mq[2], mq[3]));
            mx *= kLog2e;
            // keep the reference maximum until a row outgrows it by 2^8 (always exact: it divides out)
            const bool grow = mx > m_run + 8.f;
            if (i > 0) {                                 // O holds the last tile's products before anything touches it
                ok = wait(&t->o_done, (i - 1) & 1, 3u);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            if (__any_sync(0xffffffffu, grow)) {
                const float m_new = grow ? mx : m_run;
                const float scale = grow ? ex2(m_run - m_new) : 1.f;
                if (i > 0) {
#pragma unroll 1
                    for (int c = 0; c < OW; c += 32) {
                        uint32_t v[32];
                        tmem_ld32(v, trow + 128 + c);
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * scale);
                        tmem_st32(trow + 128 + c, v);
                    }
                }
                l_run *= scale;
                m_run = m_new;
            }
#pragma unroll
            for (int c = 0; c < PA_KV / 32; ++c) {
                uint32_t o[32];
                float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
                for (int j = 0; j < 32; j += 2) {
                    const float a = ex2(fmaf(__uint_as_float(v[c][j]), kLog2e, -m_run));
                    const float b = ex2(fmaf(__uint_as_float(v[c][j + 1]), kLog2e, -m_run));
                    sum0 += a;
                    sum1 += b;
                    const uint32_t hi = pack2(a, b);
                    o[j / 2] = hi;
                    o[16 + j / 2] = pack2(a - bf16_lo(hi), b - bf16_hi(hi));
                }
                l_run += sum0 + sum1;
                tmem_st32(trow + 32 * c, o);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(&t->p_full)) : "memory");
        }
        if (ok) ok = wait(&t->o_done, (n_tiles - 1) & 1, 3u);
        if (__all_sync(0xffffffffu, ok)) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const float inv = 1.f / l_run;
            uint16_t* dst = p.out + (size_t(tok) * p.hq + g * G + r % G) * OW;
            const bool mine = tok < p.m && my_pos < p.max_ctx;
            uint32_t odd = 0;                            // two bf16 zeros as long as every result is finite
#pragma unroll 1
            for (int c = 0; c < OW; c += 32) {
                uint32_t v[32];
                tmem_ld32(v, trow + 128 + c);
                if (mine) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint4 w;
                        w.x = pack2(__uint_as_float(v[8 * q]) * inv, __uint_as_float(v[8 * q + 1]) * inv);
                        w.y = pack2(__uint_as_float(v[8 * q + 2]) * inv, __uint_as_float(v[8 * q + 3]) * inv);
                        w.z = pack2(__uint_as_float(v[8 * q + 4]) * inv, __uint_as_float(v[8 * q + 5]) * inv);
                        w.w = pack2(__uint_as_float(v[8 * q + 6]) * inv, __uint_as_float(v[8 * q + 7]) * inv);
                        *reinterpret_cast<uint4*>(dst + c + 8 * q) = w;
                        odd = times_zero(w.x, times_zero(w.y, times_zero(w.z, times_zero(w.w, odd))));
                    }
                }
            }
            if (__any_sync(0xffffffffu, (odd & 0x7fff7fffu) != 0u)) {
                __syncwarp();                            // (these results are written over)
                slow_rows<G, MLA>(p, first, m0, g, quad * 32, lane);
            }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(256u) : "memory");
    }
}

// [outer][mid][inner] bf16, boxes of box_outer x box_mid x box_inner elements (64: 128-byte swizzle, 32: 64-byte swizzle)
bool make_map3(CUtensorMap* map, const void* ptr, size_t inner, size_t mid, size_t outer, size_t outer_stride, int box_inner,
               int box_mid, int box_outer) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {inner, mid, outer};
    const cuuint64_t strides[2] = {inner * 2, outer_stride * 2};
    const cuuint32_t box[3] = {cuuint32_t(box_inner), cuuint32_t(box_mid), cuuint32_t(box_outer)};
    const cuuint32_t elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, box_inner == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int G, bool MLA>
cudaError_t launch_attn(const PrefillAttnParams& p, int kv_heads, const CUtensorMap (&map)[5], cudaStream_t stream, bool pdl) {
    const size_t smem = 1024 + 3 * PA_TILE + sizeof(PaTail);
    static PerDeviceOnce once;
    if (once.first()) {
        cudaError_t e = cudaFuncSetAttribute(prefill_attn_kernel<G, MLA>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return e;
    }
    const int tok = 128 / G;
    return launch_kernel(prefill_attn_kernel<G, MLA>, dim3(kv_heads, (p.m + tok - 1) / tok), dim3(PA_THREADS), smem, stream, pdl,
                         map[0], map[1], map[2], map[3], map[4], p);
}

const size_t kAnyRows = size_t(1) << 30;                 // (a pool: its pages are what the table names; only those boxes are touched)

}  // namespace

bool prefill_attn_supported(int hq, int hkv, int d, int page_size) {
    if (d != PA_D || hkv < 1 || hq % hkv || page_size % 64) return false;
    const int g = hq / hkv;
    return g == 1 || g == 2 || g == 4;
}

cudaError_t prefill_attn_launch(const PrefillAttnParams& p, cudaStream_t stream, bool pdl) {
    if (!prefill_attn_supported(p.hq, p.hkv, PA_D, p.page_size) || p.m < 1) return cudaErrorInvalidValue;
    cudaError_t e = launch_kernel(prefill_rows_kernel, dim3(p.m), dim3(256), 0, stream, pdl, p);
    if (e != cudaSuccess) return e;
    const int G = p.hq / p.hkv;
    CUtensorMap m[5];
    if (!make_map3(&m[0], p.qkv, PA_D, p.hq, p.m, size_t(p.hq + 2 * p.hkv) * PA_D, 64, G, 128 / G) ||
        !make_map3(&m[1], p.k_pool, PA_D, p.hkv, kAnyRows, size_t(p.hkv) * PA_D, 64, 1, 64) ||
        !make_map3(&m[2], p.v_pool, PA_D, p.hkv, kAnyRows, size_t(p.hkv) * PA_D, 64, 1, 64))
        return cudaErrorInvalidValue;
    m[3] = m[4] = m[0];
    switch (G) {
        case 1: return launch_attn<1, false>(p, p.hkv, m, stream, pdl);
        case 2: return launch_attn<2, false>(p, p.hkv, m, stream, pdl);
        default: return launch_attn<4, false>(p, p.hkv, m, stream, pdl);
    }
}

// ---- latent form -------------------------------------------------------------------------------------------------
bool mla_chunk_supported(int page_size) { return page_size % 64 == 0; }

cudaError_t mla_chunk_rows_launch(const MlaChunkParams& p, cudaStream_t stream, bool pdl) {
    return launch_kernel(mla_chunk_rows_kernel, dim3(p.m + (p.first + 7) / 8), dim3(256), 0, stream, pdl, p);
}

cudaError_t mla_chunk_attn_launch(const MlaChunkParams& c, cudaStream_t stream, bool pdl) {
    cudaError_t e = launch_kernel(mla_chunk_q_kernel, dim3(c.m), dim3(256), 0, stream, pdl, c);
    if (e != cudaSuccess) return e;
    PrefillAttnParams p = {};
    p.pos_rows = c.pos_rows; p.block_table = c.block_table; p.out = c.out; p.status = c.status;
    p.qkv = c.q; p.k_pool = const_cast<uint16_t*>(c.kv_hi); p.v_pool = const_cast<uint16_t*>(c.kv_lo); p.lat_pool = c.pool;
    p.m = c.m; p.hq = c.heads; p.hkv = c.heads; p.page_size = c.page_size; p.max_ctx = c.max_ctx;
    CUtensorMap m[5];
    const size_t ctx = size_t(c.first) + c.m, kvw = size_t(c.heads) * 128, qw = size_t(c.heads) * 96;
    if (!make_map3(&m[0], c.q, 96, c.heads, c.m, qw, 64, 1, 128) || !make_map3(&m[1], c.kv_hi, 128, c.heads, ctx, kvw, 64, 1, 128) ||
        !make_map3(&m[2], c.kv_lo, 128, c.heads, ctx, kvw, 64, 1, 128) || !make_map3(&m[3], c.q, 96, c.heads, c.m, qw, 32, 1, 128) ||
        !make_map3(&m[4], c.pool, 288, 1, kAnyRows, 288, 32, 1, 64))
        return cudaErrorInvalidValue;
    return launch_attn<1, true>(p, c.heads, m, stream, pdl);
}

}  // namespace tfb
