// The MoE layer for up to eight tokens and packed weights, three kernels on the digit engine
// (digit_tile.cuh); arithmetic of cpu::moe_forward_bias, core/moe_cpu.cpp:198-288.
//
//   1  a few CTAs: router logits (the reference's exact fp32 order) and, in the one that ends last, softmax,
//      top-K and mixture weights; all others: the shared expert's gate / up with SwiGLU
//   2  gate / up of the chosen experts with SwiGLU
//   3  all down projections as one contraction over [shared | expert k ...], the mixture weights folded into
//      the activations' scales; residual add or plain store
//
// A token moves 10.6 MB of weights through these (H-Tiny shape), 1.6 us at the copy rate: what counts is the
// chain of dependent steps.  So: a tile is 8 gate rows and the same 8 up rows, which end in one lane pair; the
// router's group sums are formed by all threads and only the ordered additions - one lane per (expert, token),
// 384 additions of four cycles - are serial; kernel 2 lets kernel 3 start only after its own wait, which
// proves the routing of kernel 1 complete, so kernel 3 fetches its experts' rows while kernel 2 runs.
// One token, H-Tiny shape, in the step's graph: 31 us before,
// 16 now.  The layer by itself at 3, 5 and 8 tokens: 28, 42 and 57 us before the router's CTAs read all tokens at once, the chunks
// were loaded four at a time and two CTAs shared an SM; 22, 27 and 36 now.
#include "digit_tile.cuh"
#include "route.cuh"

namespace b200 {

constexpr int DM_ROUTER = 4;                  // experts per router CTA

__host__ __device__ inline int dm_chain_stride(int d) { return ((d >> 2) + 31) / 32 * 32 + 4; }   // floats; 4 mod 32: no bank conflicts

// The tile loop shared by the three kernels: rounds of up to G tiles through `sets` sets of stages, each tile's
// chunks split over P warps.  issue(r, set): one thread starts round r's copies; dot(stage, part, acc): one warp's
// share; epilogue(first tile, tiles, red): all threads. prepare() stages the activations, barrier included.
// The epilogues' elements go to the threads from the last warp but one on: a round has few, and the first warps, which
// always have products, go on to the next round's.
template <int MT>
__device__ __forceinline__ int dm_element() {
    constexpr int T = dg_warps(MT) * 32;
    return threadIdx.x >= T - 64 ? threadIdx.x - (T - 64) : threadIdx.x + 64;
}
template <int KIND, int MT, typename Prepare, typename Issue, typename Dot, typename Epi>
__device__ __forceinline__ void dm_rounds(const MoeFusedArgs& a, int n_my, float* red, uint64_t* bar, Prepare prepare, Issue issue, Dot dot, Epi epilogue) {
    constexpr int W = dg_warps(MT);
    const int G = a.n_stages, P = a.parts, rounds = a.sets == 1 ? 1 : (n_my + G - 1) / G;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    bool ok = true;
    prepare();
    for (int r = 0; r < rounds; ++r) {
        const int n = min(G, n_my - r * G), set = a.sets == 1 ? 0 : r & 1;
        float* rr = red + (size_t)(r & 1) * G * P * dg_red_floats(MT);
        ok = ok && mbar_wait(&bar[set], (a.sets == 1 ? r : r >> 1) & 1, a.status);
        if (ok) {
            for (int u = warp; u < n * P; u += W) {
                const int tile = dg_div(u, a.parts_inv), part = u - tile * P;
                DgAcc<KIND, MT> acc;
                acc.clear();
                dot(set * G + tile, part, acc);
                dg_finish<KIND, MT>(acc, rr + u * dg_red_floats(MT), lane);
            }
        }
        if (!__syncthreads_and(ok)) break;
        if (warp == W - 1 && lane == 0 && r + 2 < rounds) issue(r + 2, set);
        epilogue(r * G, n, rr);
    }
    if (!ok && threadIdx.x == 0)              // no copy of this CTA may be left under way
        for (int set = 0; set < min(a.sets, rounds); ++set)
            for (int par = 0; par < 2 && !mbar_wait(&bar[set], par, a.status); ++par) {}
}

// Stages tokens [m0, m0 + n) of x [., K] (times norm_w when there is one) as slots 0 ..; per-chunk sums of
// squares to ssq.  The norm factor itself is applied by the epilogue.
template <int KIND, int MT>
__device__ __forceinline__ void dm_stage_norm(const MoeFusedArgs& a, const DgX<KIND, MT>& xd, int m0, int n, double* ssq) {
    constexpr int W = dg_warps(MT), B = dg_batch(MT);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, chunks = dg_chunks(a.d), all = chunks * n;
    for (int i0 = warp; i0 < all; i0 += B * W) {
        float v[B][8], nw[B][8];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int i = i0 + b * W, m = MT == 1 ? 0 : dg_div(i, a.chunks_inv), c = i - m * chunks;
            if (i >= all) break;
            dg_load8<true>(a.x + (int64_t)(m0 + m) * a.d, c * DG_CHUNK + 8 * lane, a.d, v[b]);
            if (a.norm_w) dg_norm8(a.norm_w, c * DG_CHUNK + 8 * lane, a.d, nw[b]);
        }
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int i = i0 + b * W, m = MT == 1 ? 0 : dg_div(i, a.chunks_inv), c = i - m * chunks;
            if (i >= all) break;
            double ss = 0.0;
            if (a.norm_w) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    ss += (double)v[b][j] * (double)v[b][j];
                    v[b][j] *= nw[b][j];
                }
            }
            dg_stage<KIND, MT>(xd, c, m, v[b], 1.0f, lane);
            if (a.norm_w) {
                ss = warp_sum_d(ss);
                if (lane == 0) ssq[c * MT + m] = ss;
            }
        }
    }
}
// After a barrier: the norm factors of n tokens by the last warp (visible after the next barrier).
template <int MT>
__device__ __forceinline__ void dm_inv(const MoeFusedArgs& a, int n, const double* ssq, float* inv) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == dg_warps(MT) - 1 && lane < n) {
        float f = 1.0f;
        if (a.norm_w) {
            double ss = 0.0;
            for (int c = 0; c < dg_chunks(a.d); ++c) ss += ssq[c * MT + lane];
            const double d = 1.0 / sqrt(ss / (double)a.d + (double)a.eps);
            f = isfinite(d) ? (float)d : 0.0f;
        }
        inv[lane] = f;
    }
}

// ---- the router's logits on their way to the CTA that routes ----------------------
// A logit is its own flag: the word is zero until it is there (the bits are stored inverted below the sign, and
// the one NaN that would give zero becomes another), so nothing has to be fenced and counted - a fence, an atomic
// and a second read took 3 us of this kernel's 12.  Kernel 2 puts the words back to zero.  The CTA that polls is
// the last of the router's, so those it waits for were scheduled before it; the poll is bounded.
constexpr int DM_MAX_EXPERTS = 256;
static __device__ uint32_t g_dm_logits[8 * DM_MAX_EXPERTS];
constexpr uint32_t DM_POLL_LIMIT = 1u << 20;

__device__ __forceinline__ void dm_post(int m, int e, float logit) {
    uint32_t u = __float_as_uint(logit);
    if (u == 0x7FFFFFFFu) u = 0x7FC00000u;
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(g_dm_logits + m * DM_MAX_EXPERTS + e), "r"(u ^ 0x7FFFFFFFu) : "memory");
}
template <int PER>
__device__ __forceinline__ void dm_biases(const MoeFusedArgs& a, float (&bs)[PER], int lane) {
#pragma unroll
    for (int i = 0; i < PER; ++i) bs[i] = a.router_bias ? a.router_bias[min(32 * i + lane, a.ne - 1)] : 0.0f;
}
// One warp per token: waits for the token's logits, routes it.  real = false: a run of the code without either.
template <int PER>
__device__ __noinline__ void dm_route(const MoeFusedArgs& a, float* scratch, const float (&bs)[PER], bool real, int warp, int lane) {
    if (warp >= a.M) return;
    float v[PER];
    bool ok = true;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        uint32_t u = 0x7FFFFFFFu;
        if (real) {
            const uint32_t* p = g_dm_logits + warp * DM_MAX_EXPERTS + min(32 * i + lane, a.ne - 1);
            uint32_t it = 0;
            do asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(u) : "l"(p) : "memory");
            while (u == 0 && ++it < DM_POLL_LIMIT);
            ok = ok && u != 0;
        }
        v[i] = __uint_as_float(u ^ 0x7FFFFFFFu);
    }
    if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicExch(a.status, 1);
        return;
    }
    int idx;
    float w;
    route_pick<PER>(v, bs, a.router_bias != nullptr, a.ne, a.K, scratch + warp * a.ne, lane, idx, w);
    if (!real) return;
    if (lane < a.K) {
        a.idx[(int64_t)warp * a.K + lane] = idx;
        a.w[(int64_t)warp * a.K + lane] = w;
    }
    if (a.probs_out)
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (32 * i + lane < a.ne) a.probs_out[(int64_t)warp * a.ne + 32 * i + lane] = v[i];
}

// ---- kernel 1 ------------------------------------------------------------------
// NORM: a norm may be in front (a.norm_w says).  One token without one has an instance of its own: its serial path is the whole
// kernel, and the code for a held row, which it never takes, cost it 0.3 us.
template <int KIND, int MT, bool NORM>
__global__ void __launch_bounds__(dg_warps(MT) * 32, 2) dm_router_shared_kernel(MoeFusedArgs a) {
    constexpr int W = dg_warps(MT);
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t bar[2];
    __shared__ double red_d[W * 8];
    __shared__ float inv[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_router = (a.ne + DM_ROUTER - 1) / DM_ROUTER;
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_fence_init();
    }
    if ((int)blockIdx.x < n_router) {
        const int e0 = blockIdx.x * DM_ROUTER, rows = min(DM_ROUTER, a.ne - e0), groups = a.d >> 2, stride = dm_chain_stride(a.d);
        float* w_s = reinterpret_cast<float*>(smem);                  // [rows][d]
        float* gs = w_s + DM_ROUTER * a.d;                            // [token * DM_ROUTER + expert][stride]
        if (threadIdx.x == 0) {
            mbar_expect_tx(&bar[0], (uint32_t)rows * a.d * 4);
            tma_load_1d(w_s, a.router_w + (int64_t)e0 * a.d, (uint32_t)rows * a.d * 4, &bar[0]);
        }
        pdl_launch_dependents();
        // the CTA that will route: its biases, and a rehearsal of the code
        float biases[2], biases8[8];
        if ((int)blockIdx.x == n_router - 1) {
            if (a.ne <= 64) {
                dm_biases(a, biases, lane);
                dm_route<2>(a, gs, biases, false, warp, lane);
            } else {
                dm_biases(a, biases8, lane);
                dm_route<8>(a, gs, biases8, false, warp, lane);
            }
        }
        // A thread's RG runs of four of every token stay in registers from the norm to the group sums where the row is
        // narrow enough (W * 32 * RG runs), all loads under way together: read token by token, and twice, five tokens of
        // 1536 took 16 500 cycles here (now the shared expert's CTAs, 12 000, are what the kernel takes).
        constexpr int RG = MT <= 2 ? 1 : 2;
        const int padded = (groups + 31) & ~31;                       // zeros up to whole runs of 32
        const bool norm = NORM && a.norm_w;
        const bool held = (MT > 2 || norm) && padded <= RG * W * 32;     // (one read is all there is without a norm)
        float4 nw[RG], xv[MT][RG];
        if (held)
#pragma unroll
            for (int q = 0; q < RG; ++q) {
                const int g = threadIdx.x + q * W * 32;
                nw[q] = norm && g < groups ? dg_norm4(a.norm_w + 4 * g) : make_float4(1.f, 1.f, 1.f, 1.f);
            }
        pdl_wait();
        auto load = [&](int m, int g) {
            return g < groups ? __ldcg(reinterpret_cast<const float4*>(a.x + (int64_t)m * a.d + 4 * g)) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        if (held)
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int q = 0; q < RG; ++q)
                    if (m < a.M) xv[m][q] = load(m, threadIdx.x + q * W * 32);
        if (norm) {
            auto square = [](float4 v) { return (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w; };
            if (held) {
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    if (m >= a.M) break;
                    double ss = 0.0;
#pragma unroll
                    for (int q = 0; q < RG; ++q) ss += square(xv[m][q]);
                    ss = warp_sum_d(ss);
                    if (lane == 0) red_d[m * W + warp] = ss;
                }
            } else {
                for (int m = 0; m < a.M; ++m) {
                    double ss = 0.0;
                    for (int g = threadIdx.x; g < groups; g += W * 32) ss += square(load(m, g));
                    ss = warp_sum_d(ss);
                    if (lane == 0) red_d[m * W + warp] = ss;
                }
            }
            __syncthreads();
            if (threadIdx.x < a.M) {
                double ss = 0.0;
#pragma unroll
                for (int w = 0; w < W; ++w) ss += red_d[threadIdx.x * W + w];
                const double d = 1.0 / sqrt(ss / (double)a.d + (double)a.eps);
                inv[threadIdx.x] = isfinite(d) ? (float)d : 0.0f;
            }
        }
        __syncthreads();
        const bool ok = mbar_wait(&bar[0], 0, a.status);
        // group sums ((a0 b0 + a1 b1) + a2 b2) + a3 b3 of every (token, expert)
        auto sums = [&](int m, int g, float4 x, float4 w) {
            if (norm) {
                const float f = inv[m];
                x = make_float4(x.x * f * w.x, x.y * f * w.y, x.z * f * w.z, x.w * f * w.w);
            }
#pragma unroll
            for (int e = 0; e < DM_ROUTER; ++e) {
                if (e < rows) {
                    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (g < groups) b = *reinterpret_cast<const float4*>(w_s + e * a.d + 4 * g);
                    float t = __fadd_rn(__fmul_rn(x.x, b.x), __fmul_rn(x.y, b.y));
                    t = __fadd_rn(t, __fmul_rn(x.z, b.z));
                    gs[(m * DM_ROUTER + e) * stride + g] = __fadd_rn(t, __fmul_rn(x.w, b.w));
                }
            }
        };
        if (held) {
#pragma unroll
            for (int q = 0; q < RG; ++q) {
                const int g = threadIdx.x + q * W * 32;
                if (g < padded)
#pragma unroll
                    for (int m = 0; m < MT; ++m)
                        if (m < a.M) sums(m, g, xv[m][q], nw[q]);
            }
        } else {
            for (int m = 0; m < a.M; ++m)
                for (int g = threadIdx.x; g < padded; g += W * 32)
                    sums(m, g, load(m, g), norm && g < groups ? dg_norm4(a.norm_w + 4 * g) : make_float4(1.f, 1.f, 1.f, 1.f));
        }
        __syncthreads();
        // the ordered additions: one lane per chain, the next 32 sums on their way while 32 are added
        if (warp == 0) {
            const int m = lane / DM_ROUTER, e = lane % DM_ROUTER;
            if (m < a.M && e < rows) {
                const float4* p = reinterpret_cast<const float4*>(gs + lane * stride);
                float s = 0.0f;
                float4 cur[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) cur[i] = p[i];
                for (int g = 32; g <= padded; g += 32) {
                    float4 nxt[8];
                    p += g < padded ? 8 : 0;
#pragma unroll
                    for (int i = 0; i < 8; ++i) nxt[i] = p[i];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, cur[i].x), cur[i].y), cur[i].z), cur[i].w);
                        cur[i] = nxt[i];
                    }
                }
                if (ok) dm_post(m, e0 + e, s);
            }
        }
        if ((int)blockIdx.x == n_router - 1) {
            if (a.ne <= 64) dm_route<2>(a, gs, biases, true, warp, lane);
            else dm_route<8>(a, gs, biases8, true, warp, lane);
        }
        return;
    }
    // shared expert: tiles of 8 gate and 8 up rows
    const int chunks = dg_chunks(a.d), nsub = a.d >> 5, G = a.n_stages;
    const uint32_t rb = (uint32_t)row_bytes_of(KIND, a.d);
    DgX<KIND, MT> xd;
    uint8_t* p = xd.carve(smem + (size_t)a.sets * G * a.stage_bytes, chunks);
    double* ssq = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15);
    float* red = reinterpret_cast<float*>(ssq + chunks * MT);
    const int first = blockIdx.x - n_router, step = gridDim.x - n_router;
    const int n_my = a.share + (first < a.share_rem ? 1 : 0);
    auto issue = [&](int r, int set) {
        const int n = min(G, n_my - r * G);
        mbar_expect_tx(&bar[set], n * 16 * rb);
        for (int i = 0; i < n; ++i) {
            const int64_t at = (int64_t)(first + (r * G + i) * step) * 8 * rb;
            uint8_t* dst = smem + (size_t)(set * G + i) * a.stage_bytes;
            tma_load_1d(dst, a.sh_g + at, 8 * rb, &bar[set]);
            tma_load_1d(dst + 8 * rb, a.sh_u + at, 8 * rb, &bar[set]);
        }
    };
    if (threadIdx.x == 0)
        for (int r = 0; r < a.sets && r * G < n_my; ++r) issue(r, r);
    pdl_launch_dependents();
    dm_rounds<KIND, MT>(a, n_my, red, bar,
        [&] {
            pdl_wait();
            dm_stage_norm<KIND, MT>(a, xd, 0, a.M, ssq);
            __syncthreads();
            dm_inv<MT>(a, a.M, ssq, inv);
        }, issue,
        [&](int stage, int part, DgAcc<KIND, MT>& acc) {
            const uint32_t at = smem_u32(smem) + stage * a.stage_bytes + (lane >> 2) * rb;
            for (int c = part; c < chunks; c += a.parts) {
                const uint32_t ac = at + c * dg_row_chunk<KIND>();
                dg_chunk<KIND, MT>(acc, ac, ac + 8 * rb, xd, c, min(8, nsub - 8 * c), lane);
            }
        },
        [&](int t0, int n, const float* rr) {
            for (int e = dm_element<MT>(); e < n * 8 * MT; e += W * 32) {
                const int m = e % MT, row = e / MT % 8, i = e / (8 * MT);
                if (m >= a.M) continue;
                const float* re = rr + i * a.parts * dg_red_floats(MT);
                const float gt = dg_value<KIND, MT>(re, a.parts, row, m) * inv[m], up = dg_value<KIND, MT>(re, a.parts, row + 8, m) * inv[m];
                a.sh_act[(int64_t)m * a.SH + (first + (t0 + i) * step) * 8 + row] = silu_acc(gt) * up;
            }
        });
}

// ---- kernel 2 ------------------------------------------------------------------
// grid (ctas, M): blockIdx.y is the token.
template <int KIND>
__global__ void __launch_bounds__(dg_warps(1) * 32, 2) dm_gateup_kernel(MoeFusedArgs a) {
    constexpr int W = dg_warps(1);
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t bar[2];
    __shared__ float inv[8];
    __shared__ int s_idx[16];
    const int lane = threadIdx.x & 31, m = blockIdx.y;
    const int chunks = dg_chunks(a.d), nsub = a.d >> 5, G = a.n_stages;
    const uint32_t rb = (uint32_t)row_bytes_of(KIND, a.d);
    DgX<KIND, 1> xd;
    uint8_t* p = xd.carve(smem + (size_t)a.sets * G * a.stage_bytes, chunks);
    double* ssq = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15);
    float* red = reinterpret_cast<float*>(ssq + chunks);
    const int per = a.E / 8, first = blockIdx.x, step = gridDim.x;      // tiles per expert
    const int n_my = a.share + (first < a.share_rem ? 1 : 0);
    auto issue = [&](int r, int set) {
        const int n = min(G, n_my - r * G);
        mbar_expect_tx(&bar[set], n * 16 * rb);
        for (int i = 0; i < n; ++i) {
            const int tile = first + (r * G + i) * step, k = __umulhi(tile, a.per_inv);
            const int64_t at = ((int64_t)s_idx[k] * a.E + (tile - k * per) * 8) * rb;
            uint8_t* dst = smem + (size_t)(set * G + i) * a.stage_bytes;
            tma_load_1d(dst, a.gates + at, 8 * rb, &bar[set]);
            tma_load_1d(dst + 8 * rb, a.ups + at, 8 * rb, &bar[set]);
        }
    };
    dm_rounds<KIND, 1>(a, n_my, red, bar,
        [&] {
            pdl_wait();
            pdl_launch_dependents();          // after the wait: kernel 3 may take kernel 1 for complete
            if ((int)threadIdx.x >= (W - 1) * 32) {
                // the last warp, which stages nothing here (or last): the chosen experts' rows
                if (lane < a.K) s_idx[lane] = __ldcg(a.idx + (int64_t)m * a.K + lane);
                __syncwarp();
                if (lane == 0) {
                    mbar_init(&bar[0], 1);
                    mbar_init(&bar[1], 1);
                    mbar_fence_init();
                    for (int r = 0; r < a.sets && r * G < n_my; ++r) issue(r, r);
                }
                __syncwarp();
                if (blockIdx.x == 0)
                    for (int e = lane; e < a.ne; e += 32) g_dm_logits[m * DM_MAX_EXPERTS + e] = 0;
            }
            dm_stage_norm<KIND, 1>(a, xd, m, 1, ssq);
            __syncthreads();
            dm_inv<1>(a, 1, ssq, inv);
        }, issue,
        [&](int stage, int part, DgAcc<KIND, 1>& acc) {
            const uint32_t at = smem_u32(smem) + stage * a.stage_bytes + (lane >> 2) * rb;
            for (int c = part; c < chunks; c += a.parts) {
                const uint32_t ac = at + c * dg_row_chunk<KIND>();
                dg_chunk<KIND, 1>(acc, ac, ac + 8 * rb, xd, c, min(8, nsub - 8 * c), lane);
            }
        },
        [&](int t0, int n, const float* rr) {
            for (int e = dm_element<1>(); e < n * 8; e += W * 32) {
                const int row = e % 8, i = e / 8, tile = first + (t0 + i) * step, k = __umulhi(tile, a.per_inv);
                const float* re = rr + i * a.parts * dg_red_floats(1);
                const float gt = dg_value<KIND, 1>(re, a.parts, row, 0) * inv[0], up = dg_value<KIND, 1>(re, a.parts, row + 8, 0) * inv[0];
                a.act[((int64_t)m * a.K + k) * a.E + (tile - k * per) * 8 + row] = silu_acc(gt) * up;
            }
        });
}

// ---- kernel 3 ------------------------------------------------------------------
// grid (ctas, M).  A tile is R = 16 output rows: of sh_down (SH wide), then of each chosen expert's down (E wide); fewer
// where 16 of all of these do not fit the shared memory (the products then leave operand rows unused).
template <int KIND>
__global__ void __launch_bounds__(dg_warps(1) * 32, 2) dm_down_kernel(MoeFusedArgs a) {
    constexpr int W = dg_warps(1);
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t bar[2];
    __shared__ int s_idx[16];
    __shared__ float s_w[16];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m = blockIdx.y;
    const int sc = dg_chunks(a.SH), ec = dg_chunks(a.E), chunks = sc + a.K * ec, G = a.n_stages, R = a.rows_per_tile;
    const uint32_t rb_s = a.SH > 0 ? (uint32_t)row_bytes_of(KIND, a.SH) : 0, rb_e = (uint32_t)row_bytes_of(KIND, a.E);
    DgX<KIND, 1> xd;
    uint8_t* p = xd.carve(smem + (size_t)a.sets * G * a.stage_bytes, chunks);
    float* red = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15);
    const int first = blockIdx.x, step = gridDim.x;
    const int n_my = a.share + (first < a.share_rem ? 1 : 0);
    auto issue = [&](int r, int set) {
        const int n = min(G, n_my - r * G);
        uint32_t rows_all = 0;
        for (int i = 0; i < n; ++i) rows_all += min(R, a.d - (first + (r * G + i) * step) * R);
        mbar_expect_tx(&bar[set], rows_all * (rb_s + a.K * rb_e));
        for (int i = 0; i < n; ++i) {
            const int r0 = (first + (r * G + i) * step) * R, rows = min(R, a.d - r0);
            uint8_t* dst = smem + (size_t)(set * G + i) * a.stage_bytes;
            if (a.SH > 0) tma_load_1d(dst, a.sh_d + (int64_t)r0 * rb_s, rows * rb_s, &bar[set]);
            for (int k = 0; k < a.K; ++k)
                tma_load_1d(dst + R * (rb_s + k * rb_e), a.downs + ((int64_t)s_idx[k] * a.d + r0) * rb_e, rows * rb_e, &bar[set]);
        }
    };
    if (threadIdx.x < 32) {
        // the routing is kernel 1's, complete before kernel 2 let this kernel start
        if (lane < a.K) {
            s_idx[lane] = __ldcg(a.idx + (int64_t)m * a.K + lane);
            s_w[lane] = __ldcg(a.w + (int64_t)m * a.K + lane);
        }
        __syncwarp();
        if (lane == 0) {
            mbar_init(&bar[0], 1);
            mbar_init(&bar[1], 1);
            mbar_fence_init();
            for (int r = 0; r < a.sets && r * G < n_my; ++r) issue(r, r);
        }
        __syncwarp();
    }
    pdl_launch_dependents();
    __syncthreads();
    float pre = 0.0f;
    dm_rounds<KIND, 1>(a, n_my, red, bar,
        [&] {
            pdl_wait();
            const int el = dm_element<1>(), row = el & 15, col = (first + el / 16 * step) * R + row;      // this thread's first element
            if (!a.out && el < 16 * min(G, n_my) && row < R && col < a.d) pre = a.resid[(int64_t)m * a.d + col];
            for (int i = warp; i < chunks; i += W) {
                float v[8], mul = 1.0f;
                if (i < sc) {
                    dg_load8<true>(a.sh_act + (int64_t)m * a.SH, i * DG_CHUNK + 8 * lane, a.SH, v);
                } else {
                    const int k = dg_div(i - sc, a.ec_inv);
                    dg_load8<true>(a.act + ((int64_t)m * a.K + k) * a.E, (i - sc - k * ec) * DG_CHUNK + 8 * lane, a.E, v);
                    mul = s_w[k];
                }
                dg_stage<KIND, 1>(xd, i, 0, v, mul, lane);
            }
            __syncthreads();
        }, issue,
        [&](int stage, int part, DgAcc<KIND, 1>& acc) {
            const uint32_t base = smem_u32(smem) + stage * a.stage_bytes, cb = dg_row_chunk<KIND>();
            const int ga = min(lane >> 2, R - 1), gb = min((lane >> 2) + 8, R - 1);
            for (int c = part; c < chunks; c += a.parts) {
                uint32_t at, rb;
                int cc = c, K = a.SH;
                if (c < sc) {
                    at = base;
                    rb = rb_s;
                } else {
                    const int k = dg_div(c - sc, a.ec_inv);
                    at = base + R * (rb_s + k * rb_e);
                    rb = rb_e;
                    cc = c - sc - k * ec;
                    K = a.E;
                }
                at += cc * cb;
                dg_chunk<KIND, 1>(acc, at + ga * rb, at + gb * rb, xd, c, min(8, (K >> 5) - 8 * cc), lane);
            }
        },
        [&](int t0, int n, const float* rr) {
            for (int e = dm_element<1>(); e < n * 16; e += W * 32) {
                const int row = e % 16, i = e / 16, col = (first + (t0 + i) * step) * R + row;
                if (row >= R || col >= a.d) continue;
                const float v = dg_value<KIND, 1>(rr + i * a.parts * dg_red_floats(1), a.parts, row, 0);
                const int64_t at = (int64_t)m * a.d + col;
                if (a.out) a.out[at] = v;
                else a.resid[at] = (t0 == 0 && e == dm_element<1>() ? pre : a.resid[at]) + v * a.res_mult;
            }
        });
}

// ---- host side -----------------------------------------------------------------
// Stages and contraction split for `share` tiles per CTA of tile_bytes each: the whole share in half an SM, or two
// sets of as much as fits there, or the same in a whole SM (unless two CTAs are to share it).  Returns the dynamic
// shared memory, 0 if nothing fits.
template <int KIND>
static size_t dm_plan(MoeFusedArgs& a, int tiles, int ctas, size_t tile_bytes, int chunks, int mt, size_t fixed, size_t floor_bytes, bool share = false) {
    const int most = ctas ? ceil_div(tiles, ctas) : 0;
    a.share = ctas ? tiles / ctas : 0;
    a.share_rem = ctas ? tiles % ctas : 0;
    a.stage_bytes = (int)((tile_bytes + 127) / 128 * 128);
    if (chunks > 255) return 0;
    for (const size_t budget : {(size_t)SMEM_BUDGET - 2048, (size_t)SMEM_BUDGET_FULL - 2048}) {
        if (share && budget > SMEM_BUDGET) break;
        for (int G = std::max(1, std::min(most, 8)); G >= 1; --G) {
            a.n_stages = G;
            a.sets = G >= most ? 1 : 2;
            a.parts = dg_parts(G, chunks, dg_warps(mt));
            a.parts_inv = dg_inv(a.parts);
            const size_t need = std::max(floor_bytes, (size_t)a.sets * G * a.stage_bytes + dg_x_bytes<KIND>(chunks, mt) + fixed + 64 +
                                                          (size_t)2 * G * a.parts * dg_red_floats(mt) * 4);
            if (need <= budget) return need;
        }
    }
    return 0;
}
template <typename Kern>
static int dm_launch(Kern kern, bool& configured, dim3 grid, int threads, size_t smem, const MoeFusedArgs& a) {
    if (!configured) {
        int rc = allow_smem(kern);
        if (rc) return rc;
        configured = true;
    }
    return launch_pdl(kern, grid, dim3(threads), smem, a);
}

template <int KIND, int MT, bool NORM = true>
static int dm_kernel1(MoeFusedArgs a, size_t smem, int grid) {
    static bool configured = false;
    return dm_launch(dm_router_shared_kernel<KIND, MT, NORM>, configured, dim3(grid), dg_warps(MT) * 32, smem, a);
}

// The three launches of a layer: arguments with their tiling, CTAs (per token in the second and third) and dynamic shared
// memory (0: does not fit).
struct DmPlan {
    MoeFusedArgs p1, p2, p3;
    int g1 = 0, g2 = 0, g3 = 0;
    size_t s1 = 0, s2 = 0, s3 = 0;
};
template <int KIND>
static DmPlan dm_plan_layer(const MoeFusedArgs& a) {
    DmPlan p;
    p.p1 = p.p2 = p.p3 = a;
    const size_t rb_d = row_bytes_of(KIND, a.d), rb_e = row_bytes_of(KIND, a.E), rb_s = a.SH > 0 ? row_bytes_of(KIND, a.SH) : 0;
    // One CTA of kernels 2 and 3 on an SM for one token, so that the next kernel's fits beside it and fetches early.  Two for more:
    // their time is a CTA's rounds of products (13 tiles each at five tokens), which twelve warps fill an SM with to 39 %
    // of its issue slots.  Us for gate / up at 2, 3, 5, 8 tokens (H-Tiny): 7.3, 11.5, 17.3, 24.2 with one, 5.7, 6.5, 9.7, 14.3 with two.
    // One again where two do not fit: the second would be a second wave, which stages its token again.  The layer in us with such a
    // second wave and without: 4096 x 768 in Q8_0 (gate / up), two tokens 134.6 / 128.7, in Q4_K (down) 77.2 / 72.6; 1536 x 1024 with
    // eight experts in Q4_K (down), five tokens 61.6 / 57.3; 1536 x 512 in Q8_0 (down), four tokens 33.4 / 31.8.  (2560 x 512 in
    // Q8_0, two tokens 27.5 / 29.8: 160 tiles per token for 74 CTAs are three to some, and two waves even that out.)
    // A layer by itself (not in a decode step) is shorter with one where the second CTA takes little: gate / up of less than seven
    // products of a chunk for a CTA, and down of three tiles and more in one set of half an SM, beside which the next
    // kernel's CTA fits.  Us from a graph, on other weights each, two and one: 768 x 512, two tokens in Q4_K 15.5 / 12.3, in Q8_0 15.6 /
    // 13.4 (gate / up); 4096 x 256, two tokens in Q4_K 24.1 / 20.6; 768 x 512, eight tokens 18.4 / 16.7; 2048 x 1024, three tokens
    // 21.8 / 19.8 (down).  On the other side: 768 x 512, three tokens 13.0 / 13.2 (gate / up); 2560 x 512, three tokens 27.1 / 30.1 (down).
    auto per_token = [&](int per_sm) { return std::max(1, per_sm * num_sms() / a.M); };
    const int most_per_sm = a.M > 1 ? 2 : 1;
    const bool alone = a.out != nullptr;
    const int n_router = ceil_div(a.ne, DM_ROUTER), sh_tiles = a.SH / 8;
    const int sh_ctas = std::min(sh_tiles, std::max(8, num_sms() - n_router));
    const size_t router_bytes = (size_t)DM_ROUTER * a.d * 4 + std::max<size_t>((size_t)DM_ROUTER * a.M * dm_chain_stride(a.d) * 4, (size_t)a.M * a.ne * 4);
    const int mt = dg_tokens(a.M);
    p.p1.chunks_inv = dg_inv(std::min(255, dg_chunks(a.d)));
    p.g1 = n_router + sh_ctas;
    p.s1 = dm_plan<KIND>(p.p1, sh_tiles, sh_ctas, sh_ctas ? 16 * rb_d : 0, sh_ctas ? dg_chunks(a.d) : 1, mt, (size_t)dg_chunks(a.d) * mt * 8, router_bytes);
    const int t2 = a.K * (a.E / 8);
    p.p2.per_inv = 0xFFFFFFFFu / (uint32_t)(a.E / 8) + 1u;      // exact quotients below 2^16 (E / 8 >= 4)
    auto gate_up = [&](int n, bool share) {
        p.g2 = std::min(t2, per_token(n));
        p.s2 = dm_plan<KIND>(p.p2, t2, p.g2, 16 * rb_d, dg_chunks(a.d), 1, (size_t)dg_chunks(a.d) * 8, 0, share);
    };
    if (most_per_sm == 2 && !(alone && t2 * dg_chunks(a.d) < 7 * per_token(1))) gate_up(2, true);
    if (!p.s2) gate_up(1, false);
    if (!p.s2 && most_per_sm == 2) gate_up(2, false);      // rows so wide that two tiles do not fit a whole SM, and one to each of two waves
    p.p3.ec_inv = dg_inv(std::min(255, dg_chunks(a.E)));
    // The down rows of the shared and all K experts: 16 to a tile, fewer where those do not fit (Q8_0, experts of 1024 and
    // eight of them: 4.5 KB of rows per output), while a copy still moves whole 16-byte words.
    auto down = [&](int R, int n, bool share) {
        const int t3 = ceil_div(a.d, R);
        p.g3 = std::min(t3, per_token(n));
        p.p3.rows_per_tile = R;
        p.s3 = dm_plan<KIND>(p.p3, t3, p.g3, R * (rb_s + a.K * rb_e), dg_chunks(a.SH) + a.K * dg_chunks(a.E), 1, 0, 0, share);
    };
    auto copies = [&](int R) { return (R * rb_e) % 16 == 0 && (R * rb_s) % 16 == 0; };
    if (most_per_sm == 2 && copies(TILE_ROWS)) {
        if (alone && ceil_div(a.d, TILE_ROWS) > 2 * per_token(1)) {
            down(TILE_ROWS, 1, true);
            if (p.p3.sets != 1) p.s3 = 0;
        }
        if (!p.s3) down(TILE_ROWS, 2, true);
    }
    for (int R = TILE_ROWS; R >= 1 && !p.s3 && copies(R); R >>= 1) down(R, 1, false);
    return p;
}
template <int KIND>
static int dm_kind(const MoeFusedArgs& a) {
    // all three are planned before the first is launched: a layer runs whole or not at all
    const DmPlan p = dm_plan_layer<KIND>(a);
    if (!p.s1 || !p.s2) return fail(B200_EUNSUPPORTED, "moe_fused: hidden size %d does not fit the shared-memory staging", a.d);
    if (!p.s3)
        return fail(B200_EUNSUPPORTED, "moe_fused: the down rows of %d experts of %d and a shared one of %d do not fit the shared-memory staging",
                    a.K, a.E, a.SH);
    int rc;
    switch (dg_tokens(a.M)) {
        case 1: rc = a.norm_w ? dm_kernel1<KIND, 1>(p.p1, p.s1, p.g1) : dm_kernel1<KIND, 1, false>(p.p1, p.s1, p.g1); break;
        case 2: rc = dm_kernel1<KIND, 2>(p.p1, p.s1, p.g1); break;
        case 4: rc = dm_kernel1<KIND, 4>(p.p1, p.s1, p.g1); break;
        default: rc = dm_kernel1<KIND, 8>(p.p1, p.s1, p.g1); break;
    }
    if (rc) return rc;
    static bool c2 = false, c3 = false;
    rc = dm_launch(dm_gateup_kernel<KIND>, c2, dim3(p.g2, a.M), dg_warps(1) * 32, p.s2, p.p2);
    return rc ? rc : dm_launch(dm_down_kernel<KIND>, c3, dim3(p.g3, a.M), dg_warps(1) * 32, p.s3, p.p3);
}

// moe_fused() for packed weights (kind 0 .. 3); sizes checked there.
int moe_digit(const MoeFusedArgs& a, int kind) {
    auto bad = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    if (bad(a.x) || bad(a.gates) || bad(a.ups) || bad(a.downs) || (a.SH > 0 && (bad(a.sh_g) || bad(a.sh_u) || bad(a.sh_d))))
        return fail(B200_EUNSUPPORTED, "moe_fused: tensors must be 16-byte aligned");
    switch (kind) {
        case 0: return dm_kind<0>(a);
        case 1: return dm_kind<1>(a);
        case 2: return dm_kind<2>(a);
        default: return dm_kind<3>(a);
    }
}

}  // namespace b200

// The three launches of a layer as they would be planned, for tests: CTAs and dynamic shared memory of a CTA of each.
extern "C" int b200_moe_digit_plan(int kind, int M, int d, int E, int ne, int K, int SH, int alone, int* ctas, int* smem) {
    using namespace b200;
    static float out;
    MoeFusedArgs a;
    if (alone) a.out = &out;
    a.M = M;
    a.d = d;
    a.E = E;
    a.ne = ne;
    a.K = K;
    a.SH = SH;
    const DmPlan p = kind == 0 ? dm_plan_layer<0>(a) : kind == 1 ? dm_plan_layer<1>(a) : kind == 2 ? dm_plan_layer<2>(a) : dm_plan_layer<3>(a);
    const int g[3] = {p.g1, p.g2 * M, p.g3 * M};
    const size_t s[3] = {p.s1, p.s2, p.s3};
    for (int i = 0; i < 3; ++i) {
        ctas[i] = g[i];
        smem[i] = (int)s[i];
    }
    return p.s1 && p.s2 && p.s3 ? B200_OK : B200_EUNSUPPORTED;
}
