// Top-k expert selection by one warp, shared by the stand-alone router kernel and the kernels that select in
// their own prologue.
#pragma once
#include "common.cuh"

namespace tfb {

// mode 0 (granite, examples/granite_4_0_h_small-cuda/model.py:376-386): logits -> top-k -> softmax over the k.
// mode 1 (Qwen3.5, examples/qwen3_5_35b_a3b-tilelang/model.py:488-499): softmax over ALL experts in f32 ->
//        top-k -> renormalise by the sum of the k.
// Selection order is by value descending; equal values resolve to the lower index; a NaN comes after everything else.  On
// return lane j < top_k <= experts holds the j-th selection: top_k different experts, whatever the logits are (whoever
// gathers expert rows uses the index as an address), and their routing weights.
template <int MAXE>
__device__ __forceinline__ void route_select(const float* __restrict__ logits_f32, const uint16_t* __restrict__ logits_bf16,
                                             int experts, int top_k, int mode, int lane, float& weight, int& expert) {
    constexpr int PER = MAXE / 32;
    float v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int e = lane + 32 * i;
        v[i] = -INFINITY;
        if (e < experts) v[i] = logits_f32 ? __ldcg(logits_f32 + e) : bf16_bits_to_f32(logits_bf16[e]);
    }
    if (mode == 1) {                           // probabilities over all experts
        float m = -INFINITY;
#pragma unroll
        for (int i = 0; i < PER; ++i) m = fmaxf(m, v[i]);
        m = warp_max(m);
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < PER; ++i) { v[i] = (lane + 32 * i < experts) ? expf(v[i] - m) : -INFINITY; s += fmaxf(v[i], 0.f); }
        s = warp_sum(s);
#pragma unroll
        for (int i = 0; i < PER; ++i) if (lane + 32 * i < experts) v[i] = v[i] / s;
    }
    // A round is two warp reductions of integers (the value as an order-preserving key, then the lowest index that has it):
    // with shuffled (value, index) pairs the selection took 4.0 us for 10 of 72 and
    // 4.4 us for 8 of 256, now 2.9 and 3.2, launch included.  Keys: 0 taken or not there, 1 NaN (it counts as
    // -infinity where its turn comes), then the numbers from -infinity (0x007fffff) up.
    unsigned key[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const unsigned b = __float_as_uint(v[i] == 0.f ? 0.f : v[i]);
        key[i] = lane + 32 * i >= experts ? 0u : v[i] != v[i] ? 1u : (b & 0x80000000u) ? ~b : b | 0x80000000u;
    }
    float top_v = 0.f;                          // lane j keeps the j-th selection
    int top_i = 0;
    for (int j = 0; j < top_k; ++j) {
        unsigned most = 0u;
#pragma unroll
        for (int i = 0; i < PER; ++i) most = max(most, key[i]);
        most = __reduce_max_sync(0xffffffffu, most);
        unsigned first = 0x7fffffffu;
#pragma unroll
        for (int i = PER - 1; i >= 0; --i) if (key[i] == most && most != 0u) first = unsigned(lane + 32 * i);
        const int best_e = int(__reduce_min_sync(0xffffffffu, first));
        if (lane == j) {
            top_v = most <= 1u ? -INFINITY : __uint_as_float((most & 0x80000000u) ? most & 0x7fffffffu : ~most);
            top_i = best_e;
        }
#pragma unroll
        for (int i = 0; i < PER; ++i) if (lane + 32 * i == best_e) key[i] = 0u;
    }
    const bool mine = lane < top_k;
    if (mode == 0) {
        const float m = warp_max(mine ? top_v : -INFINITY);
        const float e = mine ? expf(top_v - m) : 0.f;
        weight = e / warp_sum(e);
    } else {
        weight = top_v / warp_sum(mine ? top_v : 0.f);
    }
    expert = top_i;
}

}  // namespace tfb
