// What a decode matrix-vector product does with output element (row n, token m): store, residual add,
// or the Mamba in_proj's split into gate | convolution step | dt.  Shared by the streamed kernel for fp16 /
// fp32 weights and the digit kernel for packed ones.
#pragma once

#include "fused.cuh"

namespace b200 {

#ifdef __CUDACC__
template <int EPI>
struct GemvEpilogue {
    float pre = 0.0f, st[4] = {0, 0, 0, 0}, wc[5] = {0, 0, 0, 0, 0};
    __device__ __forceinline__ static bool is_conv(const SgArgs& a, int n) {
        return EPI == EPI_INPROJ && n >= a.p.d_inner && n < a.p.d_inner + a.p.conv_dim;
    }
    // operands that the product does not need, so that their latency hides behind it
    __device__ __forceinline__ void prefetch(const SgArgs& a, int n, int m) {
        if (EPI == EPI_RESIDUAL) {
            pre = a.resid[(int64_t)m * a.y_stride + n];
        } else if (is_conv(a, n) && a.p.k <= 5) {
            const int c = n - a.p.d_inner, win = a.p.k - 1;
            const float* sp = a.conv_state + ((int64_t)m * a.p.conv_dim + c) * win;
            const float* wp = a.conv_w + (int64_t)c * a.p.k;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < win) st[j] = sp[j];
#pragma unroll
            for (int j = 0; j < 5; ++j)
                if (j < a.p.k) wc[j] = wp[j];
            pre = a.conv_b ? a.conv_b[c] : 0.0f;
        }
    }
    __device__ __forceinline__ void finish(const SgArgs& a, int n, int m, float v, float* y, int y_stride) {
        if (EPI == EPI_STORE) {
            y[(int64_t)m * y_stride + n] = v * a.out_scale;
        } else if (EPI == EPI_RESIDUAL) {
            a.resid[(int64_t)m * a.y_stride + n] = pre + v * a.res_mult;
        } else {
            // Mamba in_proj row n: gate | conv channel (window of raw inputs, oldest
            // first; unfused ops in the reference's order) | dt
            const MambaDims& p = a.p;
            if (n < p.d_inner) {
                a.gate[(int64_t)m * p.d_inner + n] = v;
            } else if (is_conv(a, n)) {
                const int c = n - p.d_inner, win = p.k - 1;
                float* sp = a.conv_state + ((int64_t)m * p.conv_dim + c) * win;
                float t;
                if (p.k <= 5) {
                    t = pre;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j < win) {
                            t = __fadd_rn(t, __fmul_rn(wc[j], st[j]));
                            if (j > 0) sp[j - 1] = st[j];
                        }
                    float wl = wc[0];
#pragma unroll
                    for (int j = 1; j < 5; ++j)
                        if (j == win) wl = wc[j];
                    t = __fadd_rn(t, __fmul_rn(wl, v));
                } else {
                    const float* wp = a.conv_w + (int64_t)c * p.k;
                    t = a.conv_b ? a.conv_b[c] : 0.0f;
                    for (int j = 0; j < win; ++j) {
                        const float sv = sp[j];
                        t = __fadd_rn(t, __fmul_rn(wp[j], sv));
                        if (j > 0) sp[j - 1] = sv;
                    }
                    t = __fadd_rn(t, __fmul_rn(wp[win], v));
                }
                if (win > 0) sp[win - 1] = v;
                a.bc[(int64_t)m * p.conv_dim + c] = silu_acc(t);
            } else {
                a.dt_raw[(int64_t)m * p.n_heads + (n - p.d_inner - p.conv_dim)] = v;
            }
        }
    }
};
#endif

}  // namespace b200
