// Router tail shared by the few-token and the many-token MoE kernels.
#pragma once

#include "common.cuh"

namespace b200 {

#ifdef __CUDACC__
// One warp: softmax over ne logits, K rounds of arg-max (value descending, index
// ascending, candidates must exceed -1e30), renormalised mixture weights -
// core/math_cpu.cpp:546-558 and core/moe_cpu.cpp:85-98,233-254 bit for bit except
// exp(), evaluated in double and rounded.  s_p / s_sel: ne floats of scratch.
__device__ __forceinline__ void route_finish_warp(const float* __restrict__ logits, const float* __restrict__ bias,
                                                  int ne, int K, float* s_p, float* s_sel, int* s_idx, float* s_w,
                                                  float* probs_out, int lane) {
    float mx = __ldcg(logits);   // L2 loads: another CTA of the same kernel may have written the logits
    for (int e = lane; e < ne; e += 32) mx = fmaxf(mx, __ldcg(logits + e));
    mx = warp_max(mx);
    for (int e = lane; e < ne; e += 32) s_p[e] = (float)exp((double)__fsub_rn(__ldcg(logits + e), mx));
    __syncwarp();
    float inv = 0.0f;
    if (lane == 0) {
        float sum = 0.0f;
        for (int e = 0; e < ne; ++e) sum = __fadd_rn(sum, s_p[e]);
        inv = (sum > 1e-12f) ? __fdiv_rn(1.0f, sum) : 0.0f;
    }
    inv = __shfl_sync(0xffffffffu, inv, 0);
    for (int e = lane; e < ne; e += 32) {
        const float pr = __fmul_rn(s_p[e], inv);
        s_p[e] = pr;
        s_sel[e] = bias ? __fadd_rn(pr, bias[e]) : pr;
        if (probs_out) probs_out[e] = pr;
    }
    __syncwarp();
    for (int k = 0; k < K; ++k) {
        float bv = -1e30f;
        int bi = -1;
        for (int e = lane; e < ne; e += 32) {
            bool taken = false;
            for (int j = 0; j < k; ++j) taken |= (s_idx[j] == e);
            const float v = s_sel[e];
            if (!taken && v > bv) { bv = v; bi = e; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (oi >= 0 && (bi < 0 || ov > bv || (ov == bv && oi < bi))) { bv = ov; bi = oi; }
        }
        if (lane == 0) s_idx[k] = bi < 0 ? 0 : bi;
        __syncwarp();
    }
    if (lane == 0) {
        float sum_w = 0.0f;
        for (int k = 0; k < K; ++k) { s_w[k] = s_p[s_idx[k]]; sum_w = __fadd_rn(sum_w, s_w[k]); }
        if (sum_w > 1e-8f) {
            const float inv_w = __fdiv_rn(1.0f, sum_w);
            for (int k = 0; k < K; ++k) s_w[k] = __fmul_rn(s_w[k], inv_w);
        } else {
            const float uni = __fdiv_rn(1.0f, (float)K);
            for (int k = 0; k < K; ++k) s_w[k] = uni;
        }
    }
    __syncwarp();
}

// The same result for K <= 16 with the candidates in registers (lane holds logits 32 i + lane, i < PER, and
// their biases; those past ne are repeats of the last and decide nothing): the exponentials side by side, the K
// rounds two warp reductions each (the largest value as an ordered word, then the lowest index that has it)
// instead of ten shuffles and a walk over the taken ones.  s: ne floats of shared scratch.  v becomes the
// probabilities; lane k < K gets choice k and its weight.
template <int PER>
__device__ __forceinline__ void route_pick(float (&v)[PER], const float (&bs)[PER], bool biased, int ne, int K, float* s, int lane,
                                           int& my_idx, float& my_w) {
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER; ++i) mx = fmaxf(mx, v[i]);
    mx = warp_max(mx);
#pragma unroll
    for (int i = 0; i < PER; ++i) v[i] = (float)exp((double)__fsub_rn(v[i], mx));
#pragma unroll
    for (int i = 0; i < PER; ++i)
        if (32 * i + lane < ne) s[32 * i + lane] = v[i];
    __syncwarp();
    // the sum in index order (every lane the same additions)
    float sum = 0.0f;
    int e0 = 0;
    for (; e0 + 16 <= ne; e0 += 16) {
        float p[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) p[i] = s[e0 + i];
#pragma unroll
        for (int i = 0; i < 16; ++i) sum = __fadd_rn(sum, p[i]);
    }
    for (; e0 < ne; ++e0) sum = __fadd_rn(sum, s[e0]);
    const float inv = sum > 1e-12f ? __fdiv_rn(1.0f, sum) : 0.0f;
    uint32_t key[PER];                                        // selection value as an ordered word; 0: not a candidate
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        v[i] = __fmul_rn(v[i], inv);
        float sel = biased ? __fadd_rn(v[i], bs[i]) : v[i];
        key[i] = 0;
        if (32 * i + lane < ne && sel > -1e30f) {
            if (sel == 0.0f) sel = 0.0f;                      // -0 ranks as +0
            const uint32_t u = __float_as_uint(sel);
            key[i] = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
        }
    }
    my_idx = 0;
    my_w = 0.0f;
    float sum_w = 0.0f;
    for (int k = 0; k < K; ++k) {
        uint32_t best = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) best = max(best, key[i]);
        best = __reduce_max_sync(0xffffffffu, best);
        int at = 0x7fffffff;
#pragma unroll
        for (int i = PER - 1; i >= 0; --i)
            if (key[i] == best) at = 32 * i + lane;
        at = __reduce_min_sync(0xffffffffu, at);
        const int e = best == 0 ? 0 : at;                     // no candidate left: index 0, as often as it takes
        float pw = 0.0f;
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (e == 32 * i + lane) {
                key[i] = 0;
                pw = v[i];
            }
        pw = __shfl_sync(0xffffffffu, pw, e & 31);
        if (lane == k) {
            my_idx = e;
            my_w = pw;
        }
        sum_w = __fadd_rn(sum_w, pw);
    }
    my_w = sum_w > 1e-8f ? __fmul_rn(my_w, __fdiv_rn(1.0f, sum_w)) : __fdiv_rn(1.0f, (float)K);
}
#endif

}  // namespace b200
