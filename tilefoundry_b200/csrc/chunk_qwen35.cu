// The row-wise, recurrent and attention kernels of a Qwen3.5 prompt chunk (the projections are gemm_rows.cu's, the expert
// block moe_grouped.cu's): M consecutive tokens go through a layer together, so every weight is read once per chunk
// instead of once per token (a 64-token prompt walked token by token took 170 ms; its weights are 60 GB, 9 ms).
//
// The recurrence stays a recurrence: gdn_chunk_kernel walks the tokens in order with the state in registers (128 CTAs, 32
// columns of one head each; per token two 128-long products, no barrier), so a chunk reads and writes the state once.
// Arithmetic and rounding points per token are those of the one-token kernels (gdn.cu, attn_gated.cu, gemv_f32.cu);
// projections hand over bf16, which is what those kernels' f32 outputs held.
#include "common.cuh"
#include "kernels.h"
#include "launch.h"

namespace tfb {
namespace {

__device__ __forceinline__ float softplus_f32(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float sigmoid_f32(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) { return uint32_t(f32_to_bf16_bits(lo)) | (uint32_t(f32_to_bf16_bits(hi)) << 16); }

// ---- s = x + y (y optional), sum_out = s, norm_out = bf16(s * rstd * gain) and, optionally, the same unrounded ------
// One CTA per row, width <= 8192, a multiple of 8.  Bound by its bytes (M * width * 4 .. 14).
__global__ void __launch_bounds__(256) add_norm_rows_kernel(const float* __restrict__ x, const uint16_t* __restrict__ y,
                                                            const float* __restrict__ gain, float* __restrict__ sum_out,
                                                            uint16_t* __restrict__ norm_out, float* __restrict__ norm_f32, int width,
                                                            float eps) {
    __shared__ float red[32];
    pdl_trigger();
    pdl_wait();
    const size_t row = size_t(blockIdx.x) * width;
    float f[4][8], ss = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int c = (threadIdx.x + i * 256) * 8;
        if (c < width) {
            const float4 a = *reinterpret_cast<const float4*>(x + row + c), b = *reinterpret_cast<const float4*>(x + row + c + 4);
            const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            uint4 u = make_uint4(0u, 0u, 0u, 0u);
            if (y) u = *reinterpret_cast<const uint4*>(y + row + c);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                f[i][2 * q] = v[2 * q] + bf16_lo(w[q]);
                f[i][2 * q + 1] = v[2 * q + 1] + bf16_hi(w[q]);
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) ss = fmaf(f[i][q], f[i][q], ss);
            if (sum_out) {
                *reinterpret_cast<float4*>(sum_out + row + c) = make_float4(f[i][0], f[i][1], f[i][2], f[i][3]);
                *reinterpret_cast<float4*>(sum_out + row + c + 4) = make_float4(f[i][4], f[i][5], f[i][6], f[i][7]);
            }
        }
    }
    const float rstd = rsqrtf(block_sum(ss, red) / float(width) + eps);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int c = (threadIdx.x + i * 256) * 8;
        if (c < width) {
            float o[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) o[q] = f[i][q] * rstd * gain[c + q];
            if (norm_out)
                *reinterpret_cast<uint4*>(norm_out + row + c) = make_uint4(pack2(o[0], o[1]), pack2(o[2], o[3]), pack2(o[4], o[5]), pack2(o[6], o[7]));
            if (norm_f32) {
                *reinterpret_cast<float4*>(norm_f32 + row + c) = make_float4(o[0], o[1], o[2], o[3]);
                *reinterpret_cast<float4*>(norm_f32 + row + c + 4) = make_float4(o[4], o[5], o[6], o[7]);
            }
        }
    }
}

// ---- Gated DeltaNet: convolution + SiLU, L2 norms, decay and write strength of every token -------------------------
// A warp takes one 128-wide head of one token (lane: four channels), q and k heads, then value heads: one trip for its loads.
// (A CTA per token whose warps walked eight heads each took 39 us for 64 tokens, now 11.)
__global__ void __launch_bounds__(256) gdn_chunk_prep_kernel(const GdnChunkParams p) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int key = p.hk * 128, val = p.hv * 128, conv = 2 * key + val;
    const int pos0 = p.pos_rows[0];
    const float* win = p.conv_state + size_t(pos0 & 1) * p.conv_state_stride;
    const uint16_t* row = p.proj + size_t(t) * p.proj_width;
    const int h = blockIdx.y * 8 + warp;
    if (h < 2 * p.hk + p.hv) {
        const int c0 = h * 128 + lane * 4;                // q heads, k heads, v heads follow one another in the channels
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int at = t - 3 + j;                     // tap j: the entry of token at, or the window before the chunk
            float e[4];
            if (at >= 0) {
                const uint2 w = *reinterpret_cast<const uint2*>(row + ptrdiff_t(at - t) * p.proj_width + c0);
                e[0] = bf16_lo(w.x); e[1] = bf16_hi(w.x); e[2] = bf16_lo(w.y); e[3] = bf16_hi(w.y);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) e[q] = win[size_t(c0 + q) * 3 + at + 3];
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[q] += e[q] * p.conv_w[size_t(c0 + q) * 4 + j];
        }
        float m[4], ss = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) { m[q] = silu_f32(acc[q]); ss += m[q] * m[q]; }
        if (h < 2 * p.hk) {
            const float r = rsqrtf(warp_sum(ss) + 1e-6f);
            const float s = h < p.hk ? p.q_scale : 1.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) { m[q] *= r; if (h < p.hk) m[q] *= s; }
            *reinterpret_cast<float4*>(p.qk + size_t(t) * 2 * key + c0) = make_float4(m[0], m[1], m[2], m[3]);
        } else {
            *reinterpret_cast<float4*>(p.v + size_t(t) * val + (c0 - 2 * key)) = make_float4(m[0], m[1], m[2], m[3]);
        }
    }
    if (blockIdx.y == 0 && int(threadIdx.x) < p.hv) {
        const int h = threadIdx.x;
        const float b = bf16_bits_to_f32(row[conv + val + h]), a = bf16_bits_to_f32(row[conv + val + p.hv + h]);
        p.gates[(size_t(t) * p.hv + h) * 2] = sigmoid_f32(b);
        p.gates[(size_t(t) * p.hv + h) * 2 + 1] = expf(-expf(p.a_log[h]) * softplus_f32(a + p.dt_bias[h]));
    }
}

// ---- Gated DeltaNet: the delta rule over the chunk's tokens ---------------------------------------------------------
// CTA (value head, 32 state columns), 128 threads: four neighbouring lanes share a column, each holding 32 of its 128 rows
// in registers (rows 16i + 4 part ..), so a token costs a lane 96 multiply-adds and two two-step shuffles and the warps
// never meet except to refill the shared-memory tile of 16 tokens' q, k, v.  Bound by that chain: ~0.15 us per token.
constexpr int kGdnTile = 16;

__global__ void __launch_bounds__(128) gdn_chunk_kernel(const GdnChunkParams p) {
    __shared__ __align__(16) float sq[kGdnTile][128], sk[kGdnTile][128];
    __shared__ float sv[kGdnTile][32], sg[kGdnTile][2];
    const int tid = threadIdx.x, hv = blockIdx.x, c0 = blockIdx.y * 32, part = tid & 3, col = tid >> 2;
    const int key = p.hk * 128, val = p.hv * 128, kh = hv / (p.hv / p.hk);
    float* state = p.state + size_t(hv) * 128 * 128 + c0 + col;
    float s[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) s[i][q] = state[size_t(16 * i + 4 * part + q) * 128];
    pdl_trigger();
    pdl_wait();
    const int pos0 = p.pos_rows[0];
    for (int t0 = 0; t0 < p.m; t0 += kGdnTile) {
        const int n = min(kGdnTile, p.m - t0);
        __syncthreads();
        for (int i = tid; i < n * 32; i += 128) {         // 16-byte pieces of q and k
            const int t = i >> 5, c = (i & 31) * 4;
            const float* src = p.qk + size_t(t0 + t) * 2 * key + kh * 128 + c;
            *reinterpret_cast<float4*>(&sq[t][c]) = *reinterpret_cast<const float4*>(src);
            *reinterpret_cast<float4*>(&sk[t][c]) = *reinterpret_cast<const float4*>(src + key);
        }
        for (int i = tid; i < n * 32; i += 128) sv[i >> 5][i & 31] = p.v[size_t(t0 + (i >> 5)) * val + hv * 128 + c0 + (i & 31)];
        for (int i = tid; i < n * 2; i += 128) sg[i >> 1][i & 1] = p.gates[(size_t(t0 + (i >> 1)) * p.hv + hv) * 2 + (i & 1)];
        __syncthreads();
        for (int t = 0; t < n; ++t) {
            const float beta = sg[t][0], decay = sg[t][1];
            float4 k[8];
            float r[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                k[i] = *reinterpret_cast<const float4*>(&sk[t][16 * i + 4 * part]);
                s[i][0] *= decay; s[i][1] *= decay; s[i][2] *= decay; s[i][3] *= decay;
                r[0] = fmaf(s[i][0], k[i].x, r[0]); r[1] = fmaf(s[i][1], k[i].y, r[1]);
                r[2] = fmaf(s[i][2], k[i].z, r[2]); r[3] = fmaf(s[i][3], k[i].w, r[3]);
            }
            float rec = (r[0] + r[1]) + (r[2] + r[3]);
            rec += __shfl_xor_sync(0xffffffffu, rec, 1);
            rec += __shfl_xor_sync(0xffffffffu, rec, 2);
            const float delta = (sv[t][col] - rec) * beta;
            float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 q = *reinterpret_cast<const float4*>(&sq[t][16 * i + 4 * part]);
                s[i][0] = fmaf(k[i].x, delta, s[i][0]); s[i][1] = fmaf(k[i].y, delta, s[i][1]);
                s[i][2] = fmaf(k[i].z, delta, s[i][2]); s[i][3] = fmaf(k[i].w, delta, s[i][3]);
                o[0] = fmaf(s[i][0], q.x, o[0]); o[1] = fmaf(s[i][1], q.y, o[1]);
                o[2] = fmaf(s[i][2], q.z, o[2]); o[3] = fmaf(s[i][3], q.w, o[3]);
            }
            float read = (o[0] + o[1]) + (o[2] + o[3]);
            read += __shfl_xor_sync(0xffffffffu, read, 1);
            read += __shfl_xor_sync(0xffffffffu, read, 2);
            if (part == 0) p.read[size_t(t0 + t) * val + hv * 128 + c0 + col] = read;
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) state[size_t(16 * i + 4 * part + q) * 128] = s[i][q];
    // Both windows, as the walk leaves them: the one the next token reads (the last three entries, in the buffer of its
    // position's parity) and the one before it (a session's state is both buffers).  Every reader of the old window was in the
    // kernel before this one; a thread has its channel's old entries in registers before it writes either buffer.
    const float* win = p.conv_state + size_t(pos0 & 1) * p.conv_state_stride;
    float* next = p.conv_state + size_t((pos0 + p.m) & 1) * p.conv_state_stride;
    float* last = p.conv_state + size_t((pos0 + p.m + 1) & 1) * p.conv_state_stride;
    const int conv = 2 * key + val, ctas = gridDim.x * gridDim.y;
    for (int c = (blockIdx.y * gridDim.x + blockIdx.x) * 128 + tid; c < conv; c += ctas * 128) {
        float e[4];                                       // entries m - 4 .. m - 1; a negative one is of the old window
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int at = p.m - 4 + j;                   // (m >= 2: not below -2)
            e[j] = at >= 0 ? bf16_bits_to_f32(p.proj[size_t(at) * p.proj_width + c]) : win[size_t(c) * 3 + at + 3];
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            next[size_t(c) * 3 + j] = e[j + 1];
            last[size_t(c) * 3 + j] = e[j];
        }
    }
}

// ---- Gated DeltaNet: per-head norm of the read-out times silu(z), rounded for the output projection -----------------
__global__ void __launch_bounds__(256) gdn_chunk_out_kernel(const GdnChunkParams p) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int val = p.hv * 128, conv = 2 * p.hk * 128 + val;
    const float4 g = *reinterpret_cast<const float4*>(p.gamma + lane * 4);
    for (int h = warp; h < p.hv; h += 8) {
        const int c = h * 128 + lane * 4;
        const float4 x = *reinterpret_cast<const float4*>(p.read + size_t(t) * val + c);
        const uint2 z = *reinterpret_cast<const uint2*>(p.proj + size_t(t) * p.proj_width + conv + c);
        const float ss = warp_sum(fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, x.w * x.w))));
        const float r = rsqrtf(ss / 128.f + p.eps);
        *reinterpret_cast<uint2*>(p.out + size_t(t) * val + c) =
            make_uint2(pack2(x.x * r * g.x * silu_f32(bf16_lo(z.x)), x.y * r * g.y * silu_f32(bf16_hi(z.x))),
                       pack2(x.z * r * g.z * silu_f32(bf16_lo(z.y)), x.w * r * g.w * silu_f32(bf16_hi(z.y))));
    }
}

// ---- gated attention: q/k norm + partial RoPE + append -------------------------------------------------------------
// One CTA per token, one warp per D-wide vector at a time; lane l holds elements l, l + 32, ... (the rotate-half partner is
// in the same lane: rotary_dim / 2 is a multiple of 32).
template <int D>
__global__ void __launch_bounds__(256) gated_chunk_rows_kernel(const GatedChunkParams p) {
    constexpr int EPL = D / 32;
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos = p.pos_rows[t];
    if (pos < 0 || pos >= p.max_ctx) return;
    const uint16_t* row = p.proj + size_t(t) * p.proj_width;
    const size_t cache = size_t(p.block_table[pos / p.page_size]) * p.page_size + pos % p.page_size;
    const int rd = p.rotary_dim, half = rd >> 1;
    for (int v = warp; v < p.hq + 2 * p.hkv; v += 8) {
        const bool is_q = v < p.hq, is_k = !is_q && v < p.hq + p.hkv;
        const uint16_t* src = is_q ? row + size_t(v) * 2 * D : row + size_t(p.hq) * 2 * D + size_t(v - p.hq) * D;
        float x[EPL];
#pragma unroll
        for (int i = 0; i < EPL; ++i) x[i] = bf16_bits_to_f32(src[lane + 32 * i]);
        if (is_q || is_k) {
            const float* gm = is_q ? p.gamma_q : p.gamma_k;
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < EPL; ++i) ss = fmaf(x[i], x[i], ss);
            const float rstd = rsqrtf(warp_sum(ss) / float(D) + p.eps);
#pragma unroll
            for (int i = 0; i < EPL; ++i) x[i] = x[i] * rstd * gm[lane + 32 * i];
            float y[EPL];
#pragma unroll
            for (int i = 0; i < EPL; ++i) {
                const int e = lane + 32 * i;
                y[i] = x[i];
                if (e < rd) {
                    const int pi = e < half ? i + half / 32 : i - half / 32;
                    float partner = 0.f;
#pragma unroll
                    for (int k = 0; k < EPL; ++k) if (k == pi) partner = x[k];
                    if (e < half) partner = -partner;
                    y[i] = __fadd_rn(__fmul_rn(x[i], p.cos_table[size_t(pos) * rd + e]), __fmul_rn(partner, p.sin_table[size_t(pos) * rd + e]));
                }
                if (is_q) y[i] *= p.scale;
            }
#pragma unroll
            for (int i = 0; i < EPL; ++i) x[i] = y[i];
        }
        float* dst = is_q ? p.q + (size_t(t) * p.hq + v) * D
                     : is_k ? p.k_pool + (cache * p.hkv + (v - p.hq)) * D : p.v_pool + (cache * p.hkv + (v - p.hq - p.hkv)) * D;
#pragma unroll
        for (int i = 0; i < EPL; ++i) dst[lane + 32 * i] = x[i];
    }
}

// ---- gated attention: causal flash attention in f32 -----------------------------------------------------------------
// CTA (KV head, 32 query rows = 32/G tokens x the G query heads of the KV head), K/V in tiles of 32 positions through shared
// memory; a warp owns four query rows.  Scores: lane = position, the row's q broadcast; weighted V: lane = D/32 dimensions.
// f32 throughout (the cache is f32), so CUDA cores: 2 * 32 * 32 * D multiply-adds per tile against 256 B * D of cache.
template <int D>
__global__ void __launch_bounds__(256) gated_chunk_attn_kernel(const GatedChunkParams p) {
    constexpr int EPL = D / 32, PITCH = D + 4;            // (row pitch: 16-byte reads of eight lanes hit 32 banks)
    extern __shared__ __align__(16) float gsm[];
    float* qs = gsm;                                      // [32][D]
    float* ks = qs + 32 * D;                              // [32][PITCH]
    float* vs = ks + 32 * PITCH;                          // [32][D]
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = p.hq / p.hkv, TOK = 32 / G, g = blockIdx.x, m0 = (gridDim.y - 1 - blockIdx.y) * TOK;
    const int first = p.pos_rows[0];
    const int last = min(first + min(m0 + TOK, p.m) - 1, p.max_ctx - 1);
    if (first < 0) return;
    for (int i = tid; i < 32 * (D / 4); i += 256) {
        const int r = i / (D / 4), c = (i % (D / 4)) * 4, t = m0 + r / G;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < p.m) v = *reinterpret_cast<const float4*>(p.q + (size_t(t) * p.hq + g * G + r % G) * D + c);
        *reinterpret_cast<float4*>(qs + r * D + c) = v;
    }
    float m_run[4], l_run[4], o[4][EPL];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        m_run[r] = -INFINITY;
        l_run[r] = 0.f;
#pragma unroll
        for (int i = 0; i < EPL; ++i) o[r][i] = 0.f;
    }
    for (int k0 = 0; k0 <= last; k0 += 32) {
        __syncthreads();
        for (int i = tid; i < 32 * (D / 4); i += 256) {
            const int r = i / (D / 4), c = (i % (D / 4)) * 4, pos = min(k0 + r, last);
            const size_t at = ((size_t(p.block_table[pos / p.page_size]) * p.page_size + pos % p.page_size) * p.hkv + g) * D + c;
            *reinterpret_cast<float4*>(ks + r * PITCH + c) = *reinterpret_cast<const float4*>(p.k_pool + at);
            *reinterpret_cast<float4*>(vs + r * D + c) = *reinterpret_cast<const float4*>(p.v_pool + at);
        }
        __syncthreads();
        float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int c = 0; c < D; c += 4) {
            const float4 k = *reinterpret_cast<const float4*>(ks + lane * PITCH + c);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float4 q = *reinterpret_cast<const float4*>(qs + (warp * 4 + r) * D + c);
                s[r] = fmaf(q.x, k.x, fmaf(q.y, k.y, fmaf(q.z, k.z, fmaf(q.w, k.w, s[r]))));
            }
        }
        float e[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int my_pos = first + m0 + (warp * 4 + r) / G;
            const float v = k0 + lane <= my_pos ? s[r] : -INFINITY;
            const float m = fmaxf(m_run[r], warp_max(v));
            const float f = m_run[r] == -INFINITY ? 0.f : expf(m_run[r] - m);
            e[r] = v == -INFINITY ? 0.f : expf(v - m);
            l_run[r] = l_run[r] * f + warp_sum(e[r]);
            m_run[r] = m;
#pragma unroll
            for (int i = 0; i < EPL; ++i) o[r][i] *= f;
        }
#pragma unroll 4
        for (int j = 0; j < 32; ++j) {
            float v[EPL];
#pragma unroll
            for (int i = 0; i < EPL; ++i) v[i] = vs[j * D + lane + 32 * i];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float w = __shfl_sync(0xffffffffu, e[r], j);
                if (k0 + j > first + m0 + (warp * 4 + r) / G) continue;      // (a later token's value is not multiplied: it may be NaN)
#pragma unroll
                for (int i = 0; i < EPL; ++i) o[r][i] = fmaf(w, v[i], o[r][i]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int row = warp * 4 + r, t = m0 + row / G, head = g * G + row % G;
        if (t >= p.m) continue;
        const uint16_t* gate = p.proj + size_t(t) * p.proj_width + size_t(head) * 2 * D + D;
#pragma unroll
        for (int i = 0; i < EPL; ++i)
            p.out[(size_t(t) * p.hq + head) * D + lane + 32 * i] =
                f32_to_bf16_bits((o[r][i] / l_run[r]) * sigmoid_f32(bf16_bits_to_f32(gate[lane + 32 * i])));
    }
}

template <int D>
cudaError_t gated_launch(const GatedChunkParams& p, cudaStream_t stream, bool pdl) {
    cudaError_t e = launch_kernel(gated_chunk_rows_kernel<D>, dim3(p.m), dim3(256), 0, stream, pdl, p);
    if (e != cudaSuccess) return e;
    const size_t smem = size_t(32) * (3 * D + 4) * sizeof(float);
    static PerDeviceOnce once;
    if (once.first()) {
        e = cudaFuncSetAttribute(gated_chunk_attn_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return e;
    }
    const int tok = 32 / (p.hq / p.hkv);
    return launch_kernel(gated_chunk_attn_kernel<D>, dim3(p.hkv, (p.m + tok - 1) / tok), dim3(256), smem, stream, pdl, p);
}

}  // namespace

cudaError_t add_norm_rows_launch(const float* x, const uint16_t* y, const float* gain, float* sum_out, uint16_t* norm_out,
                                 float* norm_f32, int rows, int width, float eps, cudaStream_t stream, bool pdl) {
    if (width % 8 || width > 8192) return cudaErrorInvalidValue;
    return launch_kernel(add_norm_rows_kernel, dim3(rows), dim3(256), 0, stream, pdl, x, y, gain, sum_out, norm_out, norm_f32, width, eps);
}

bool gdn_chunk_supported(int hk, int hv, int dk, int dv, int width) {
    // (an even hv: a token's row of the projection, with the two scalars per value head at its end, is read 8 bytes at a time)
    return dk == 128 && dv == 128 && width == 4 && hk > 0 && hv > 0 && hv % hk == 0 && hv % 2 == 0 && hv <= 256;
}
cudaError_t gdn_chunk_launch(const GdnChunkParams& p, cudaStream_t stream, bool pdl) {
    cudaError_t e = launch_kernel(gdn_chunk_prep_kernel, dim3(p.m, (2 * p.hk + p.hv + 7) / 8), dim3(256), 0, stream, pdl, p);
    if (e == cudaSuccess) e = launch_kernel(gdn_chunk_kernel, dim3(p.hv, 4), dim3(128), 0, stream, pdl, p);
    if (e == cudaSuccess) e = launch_kernel(gdn_chunk_out_kernel, dim3(p.m), dim3(256), 0, stream, pdl, p);
    return e;
}

bool gated_chunk_supported(int hq, int hkv, int d, int rotary_dim) {
    return (d == 128 || d == 256) && hkv > 0 && hq > 0 && hq % hkv == 0 && 32 % (hq / hkv) == 0 && rotary_dim > 0 &&
           rotary_dim % 64 == 0 && rotary_dim <= d;
}
cudaError_t gated_chunk_launch(const GatedChunkParams& p, int d, cudaStream_t stream, bool pdl) {
    return d == 256 ? gated_launch<256>(p, stream, pdl) : gated_launch<128>(p, stream, pdl);
}

}  // namespace tfb
