// Mixture-of-experts layer: router (softmax + top-K), deterministic expert
// permutation, routed SwiGLU experts + shared expert, weighted combine.
//
// Reference arithmetic: cpu::moe_forward_bias, core/moe_cpu.cpp:198-288 (router
// dot order :76-83, softmax core/math_cpu.cpp:546-558, top-K :85-98); kernels
// replaced: cuda/moe.cu:170-333 (route), :623-651 (grouping), :731-958 (layer).
//
// Routing is reproduced bit for bit: the router logit of (token, expert) is the
// fp32 chain s += ((a0*b0 + a1*b1) + a2*b2) + a3*b3 over groups of four in k order
// with unfused multiplies and adds; the softmax sums in expert order; selection is
// strict '>' in ascending expert order (lowest index wins ties).  Expert outputs
// are combined per token in k order (no atomics), so results are run-to-run
// bit-stable.
#include "gemm.cuh"
#include "fused.cuh"
#include "linear.cuh"
#include "route.cuh"

namespace b200 {

// moe_grouped.cu
constexpr int MOE_UNITS_MAX_ROWS = 12;
int moe_forward_units(const float* x, const float* router_w, const float* router_bias, const void* gates,
                      const void* ups, const void* downs, const void* sh_g, const void* sh_u, const void* sh_d,
                      float* out, float* probs_cache, int32_t* idx_cache, float* w_cache, int64_t N, int d, int E,
                      int ne, int K, int SH, int kind);
int moe_forward_grouped(const float* x, const float* router_w, const float* router_bias, const void* gates,
                        const void* ups, const void* downs, const void* sh_g, const void* sh_u, const void* sh_d,
                        float* out, float* probs_cache, int32_t* idx_cache, float* w_cache, int64_t N, int d, int E,
                        int ne, int K, int SH, int kind);

constexpr int MOE_MAX_NE = 256;
constexpr int MOE_MAX_K = 16;

// ---------------------------------------------------------------------------
// Router: one block per token.
//   phase A  all threads: group sums g[i][e] = ((a0b0+a1b1)+a2b2)+a3b3 -> smem
//   phase B  thread e: the serial chain over the groups (and the scalar tail)
//   then     softmax in expert order, K rounds of warp arg-max, renormalise
// Shared memory: x[d] + g[chunk_groups][ne + 1] floats.
// ---------------------------------------------------------------------------
constexpr int ROUTE_THREADS = 256;

__global__ void __launch_bounds__(ROUTE_THREADS)
moe_route_kernel(const float* __restrict__ x, const float* __restrict__ router_w,
                 const float* __restrict__ router_bias, float* __restrict__ probs_out,
                 int32_t* __restrict__ idx_out, float* __restrict__ w_out, int d, int ne, int K,
                 int chunk_groups) {
    extern __shared__ float sm[];
    float* sx = sm;                          // [d]
    float* sg = sm + ((d + 3) & ~3);         // [chunk_groups][ne + 1] (padded: conflict-free both ways)
    __shared__ float s_logit[MOE_MAX_NE];    // logits -> exp -> probs
    __shared__ float s_sel[MOE_MAX_NE];
    __shared__ int s_idx[MOE_MAX_K];
    __shared__ float s_inv;
    const int64_t t = blockIdx.x;
    const float* xt = x + t * d;
    for (int i = threadIdx.x; i < d; i += blockDim.x) sx[i] = xt[i];
    const int groups = d >> 2;
    float chain = 0.0f;                      // thread e's running sum
    for (int g0 = 0; g0 < groups; g0 += chunk_groups) {
        const int ng = min(chunk_groups, groups - g0);
        __syncthreads();
        // phase A: item = (e, gi) with gi fastest so a thread's loads walk a weight row
        for (int item = threadIdx.x; item < ng * ne; item += blockDim.x) {
            const int e = item / ng, gi = item - e * ng;
            const int k = (g0 + gi) << 2;
            const float4 b = *reinterpret_cast<const float4*>(router_w + (int64_t)e * d + k);
            const float4 a = *reinterpret_cast<const float4*>(sx + k);
            float g = __fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y));
            g = __fadd_rn(g, __fmul_rn(a.z, b.z));
            g = __fadd_rn(g, __fmul_rn(a.w, b.w));
            sg[gi * (ne + 1) + e] = g;
        }
        __syncthreads();
        // phase B
        if (threadIdx.x < ne) {
            const int e = threadIdx.x;
#pragma unroll 8
            for (int gi = 0; gi < ng; ++gi) chain = __fadd_rn(chain, sg[gi * (ne + 1) + e]);
        }
    }
    if (threadIdx.x < ne) {
        const int e = threadIdx.x;
        for (int k = groups << 2; k < d; ++k)
            chain = __fadd_rn(chain, __fmul_rn(sx[k], router_w[(int64_t)e * d + k]));
        s_logit[e] = chain;
    }
    __syncthreads();
    // softmax: max (order-free), exp, then the sum in expert order by one thread
    if (threadIdx.x < 32) {
        float mx = s_logit[0];
        for (int e = threadIdx.x; e < ne; e += 32) mx = fmaxf(mx, s_logit[e]);
        mx = warp_max(mx);
        // exp in double, rounded to float: matches the CPU libm's correctly rounded expf
        for (int e = threadIdx.x; e < ne; e += 32)
            s_logit[e] = (float)exp((double)__fsub_rn(s_logit[e], mx));
        __syncwarp();
        if (threadIdx.x == 0) {
            float sum = 0.0f;
            for (int e = 0; e < ne; ++e) sum = __fadd_rn(sum, s_logit[e]);
            s_inv = (sum > 1e-12f) ? __fdiv_rn(1.0f, sum) : 0.0f;
        }
        __syncwarp();
        const float inv = s_inv;
        for (int e = threadIdx.x; e < ne; e += 32) {
            const float p = __fmul_rn(s_logit[e], inv);
            s_logit[e] = p;
            s_sel[e] = router_bias ? __fadd_rn(p, router_bias[e]) : p;
        }
        __syncwarp();
        // K rounds of arg-max: value descending, index ascending; candidates must
        // exceed -1e30 (the reference's initial best value); none left -> expert 0.
        for (int k = 0; k < K; ++k) {
            float bv = -1e30f;
            int bi = -1;
            for (int e = threadIdx.x; e < ne; e += 32) {
                bool taken = false;
                for (int j = 0; j < k; ++j) taken |= (s_idx[j] == e);
                const float v = s_sel[e];
                if (!taken && v > bv) { bv = v; bi = e; }   // ascending e: strict '>' keeps the lowest
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (oi >= 0 && (bi < 0 || ov > bv || (ov == bv && oi < bi))) { bv = ov; bi = oi; }
            }
            if (threadIdx.x == 0) s_idx[k] = bi < 0 ? 0 : bi;
            __syncwarp();
        }
        if (threadIdx.x == 0) {
            float tw[MOE_MAX_K];
            float sum_w = 0.0f;
            for (int k = 0; k < K; ++k) { tw[k] = s_logit[s_idx[k]]; sum_w = __fadd_rn(sum_w, tw[k]); }
            if (sum_w > 1e-8f) {
                const float inv_w = __fdiv_rn(1.0f, sum_w);
                for (int k = 0; k < K; ++k) tw[k] = __fmul_rn(tw[k], inv_w);
            } else {
                const float uni = __fdiv_rn(1.0f, (float)K);
                for (int k = 0; k < K; ++k) tw[k] = uni;
            }
            for (int k = 0; k < K; ++k) {
                idx_out[t * K + k] = s_idx[k];
                w_out[t * K + k] = tw[k];
            }
        }
        if (probs_out)
            for (int e = threadIdx.x; e < ne; e += 32) probs_out[t * ne + e] = s_logit[e];
    }
}

// ---------------------------------------------------------------------------
// Expert permutation: stable counting sort of slots s = t*K + k by expert, one block per expert and one launch.  A block
// reads all slots twice (from L2): counted below and at its expert, which gives the expert's offset and each warp's first
// position, then placed in order.  No block waits for another.  The three kernels before it (histograms, a scan, ranked
// placing) and the one for the inverse were bound by their launches: 24 576 slots of 64 experts 19.5 us and 4 for the
// inverse, 12.3 now; 3102 slots 17.4 + 4 -> 6.2, a decode batch of 384 8.2 -> 6.1.
// ---------------------------------------------------------------------------
constexpr int PERM_WARPS = 16;

__global__ void __launch_bounds__(PERM_WARPS * 32)
perm_kernel(const int32_t* __restrict__ idx, int NK, int32_t* __restrict__ grouped, int32_t* __restrict__ inv,
            int32_t* __restrict__ offsets) {
    __shared__ int s_below[PERM_WARPS], s_at[PERM_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, e = blockIdx.x;
    // a warp's run of slots: whole 128s
    const uint32_t run = (((uint32_t)NK + PERM_WARPS - 1) / PERM_WARPS + 127) & ~127u;
    const uint32_t s0 = min((uint32_t)NK, warp * run), s1 = min((uint32_t)NK, s0 + run);
    const bool wide = (reinterpret_cast<uintptr_t>(idx) & 15) == 0;
    auto load = [&](uint32_t s, int (&v)[4]) {                     // slots s .. s + 3; past the end: no expert
        if (wide && s + 4 <= s1) {
            const int4 q = *reinterpret_cast<const int4*>(idx + s);
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = s + j < s1 ? idx[s + j] : MOE_MAX_NE;
        }
    };
    pdl_launch_dependents();
    pdl_wait();
    int below = 0, at = 0;
#pragma unroll 2
    for (uint32_t s = s0 + 4 * lane; s < s1; s += 128) {
        int v[4];
        load(s, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            below += v[j] < e;
            at += v[j] == e;
        }
    }
    below = __reduce_add_sync(0xffffffffu, below);
    at = __reduce_add_sync(0xffffffffu, at);
    if (lane == 0) {
        s_below[warp] = below;
        s_at[warp] = at;
    }
    __syncthreads();
    int offset = 0, pos = 0;
#pragma unroll
    for (int w = 0; w < PERM_WARPS; ++w) {
        offset += s_below[w];
        pos += w < warp ? s_at[w] : 0;
    }
    if (threadIdx.x == 0) {
        offsets[e] = offset;
        if (e == (int)gridDim.x - 1) offsets[e + 1] = NK;
    }
    pos += offset;
    if (at == 0) return;                                      // whole warps
    for (uint32_t s = s0 + 4 * lane; s - 4 * lane < s1; s += 128) {
        int v[4];
        load(s, v);
        unsigned has[4];
        int before = 0, total = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            has[j] = __ballot_sync(0xffffffffu, v[j] == e);
            before += __popc(has[j] & ((1u << lane) - 1u));
            total += __popc(has[j]);
        }
        int p = pos + before;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (v[j] == e) {
                grouped[p] = (int32_t)(s + j);
                if (inv) inv[s + j] = p;
                ++p;
            }
        pos += total;
    }
}

// Many slots: every block above reads all of them twice, 0.27 us a thousand, whatever the device has to spare.
// Here each slot is read twice in all, by three kernels: per-block histograms, a scan over (expert, block), and a fill where each warp
// ranks its 32 slots with __match_any_sync and warps are ordered through shared-memory prefix sums.
// In us, the kernel above and these, 24 576 / 100 000 / 655 360 / 4 000 000 slots: 4 experts 7 / 28 / 170 / 1022 and 11 / 25 / 215 / 1215; 16
// experts 7 / 28 / 169 / 1015 and 12 / 25 / 135 / 1040; 64 experts 7 / 27 / 165 / 990 and 11 / 22 / 100 / 1124; 256 experts 12 / 44 / 266 / 1597
// and 15 / 25 / 193 / 1134.
constexpr int SORT_THREADS = 256;
constexpr int SORT_ITERS = 4;                              // slots per block = 256 * 4
constexpr int SORT_CHUNK = SORT_THREADS * SORT_ITERS;

__global__ void __launch_bounds__(SORT_THREADS)
sort_count_kernel(const int32_t* __restrict__ idx, int64_t NK, int ne, int32_t* __restrict__ block_counts) {
    __shared__ int cnt[MOE_MAX_NE];
    for (int e = threadIdx.x; e < ne; e += blockDim.x) cnt[e] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * SORT_CHUNK;
    for (int it = 0; it < SORT_ITERS; ++it) {
        const int64_t s = base + it * SORT_THREADS + threadIdx.x;
        const int e = s < NK ? idx[s] : -1;
        if ((unsigned)e < (unsigned)ne) atomicAdd(&cnt[e], 1);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < ne; e += blockDim.x) block_counts[(int64_t)blockIdx.x * ne + e] = cnt[e];
}

// One block; thread e walks the blocks of expert e.  block_counts becomes the
// first output position of (block, expert); offsets[ne+1] the expert boundaries.
__global__ void sort_scan_kernel(int32_t* __restrict__ block_counts, int nblocks, int ne,
                                 int32_t* __restrict__ offsets) {
    __shared__ int total[MOE_MAX_NE + 1];
    const int e = threadIdx.x;
    if (e < ne) {
        int run = 0;
        for (int b = 0; b < nblocks; ++b) {
            const int c = block_counts[(int64_t)b * ne + e];
            block_counts[(int64_t)b * ne + e] = run;
            run += c;
        }
        total[e] = run;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int i = 0; i < ne; ++i) { const int c = total[i]; total[i] = run; run += c; }
        total[ne] = run;
    }
    __syncthreads();
    if (e <= ne) offsets[e] = total[e];
    if (e < ne) {
        const int off = total[e];
        for (int b = 0; b < nblocks; ++b) block_counts[(int64_t)b * ne + e] += off;
    }
}

__global__ void __launch_bounds__(SORT_THREADS)
sort_fill_kernel(const int32_t* __restrict__ idx, int64_t NK, int ne, const int32_t* __restrict__ block_base,
                 int32_t* __restrict__ grouped) {
    constexpr int NW = SORT_THREADS / 32;
    __shared__ int cursor[MOE_MAX_NE];
    __shared__ int wcnt[NW][MOE_MAX_NE];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int e = threadIdx.x; e < ne; e += blockDim.x) cursor[e] = block_base[(int64_t)blockIdx.x * ne + e];
    const int64_t base = (int64_t)blockIdx.x * SORT_CHUNK;
    for (int it = 0; it < SORT_ITERS; ++it) {
        for (int i = threadIdx.x; i < NW * ne; i += blockDim.x) (&wcnt[0][0])[(i / ne) * MOE_MAX_NE + (i % ne)] = 0;
        __syncthreads();
        const int64_t s = base + it * SORT_THREADS + threadIdx.x;
        int e = s < NK ? idx[s] : -1;
        const bool live = (unsigned)e < (unsigned)ne;
        if (!live) e = -1 - lane;              // dead lanes match nobody
        const unsigned peers = __match_any_sync(0xffffffffu, e);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        if (live && rank == 0) wcnt[warp][e] = __popc(peers);
        __syncthreads();
        if (live) {
            int pos = cursor[e] + rank;
            for (int w = 0; w < warp; ++w) pos += wcnt[w][e];
            grouped[pos] = (int32_t)s;
        }
        __syncthreads();
        for (int ee = threadIdx.x; ee < ne; ee += blockDim.x) {
            int add = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) add += wcnt[w][ee];
            cursor[ee] += add;
        }
        __syncthreads();
    }
}

// inv[grouped[pos]] = pos
__global__ void sort_inverse_kernel(const int32_t* __restrict__ grouped, int32_t* __restrict__ inv, int64_t NK) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < NK) inv[grouped[p]] = (int32_t)p;
}

// grouped [NK]: slots sorted by expert, stable; inv (optional): where each slot went; offsets [ne + 1].
int moe_permutation(const int32_t* idx, int64_t NK, int ne, int32_t* grouped, int32_t* inv, int32_t* offsets) {
    B200_REQUIRE(idx && grouped && offsets, "moe_permutation: null pointer");
    B200_REQUIRE(ne > 0 && ne <= MOE_MAX_NE, "moe_permutation: ne out of range");
    B200_REQUIRE(NK >= 0 && NK < ((int64_t)1 << 31), "moe_permutation: slot count out of range");
    const bool two = ne > num_sms();                               // blocks of the one kernel on an SM
    const bool many = NK * (two ? 2 : 1) >= (inv ? 110000 : 90000) && (NK < 1 << 18 || (ne >= 16 && NK < 1 << 21) || two);
    if (!many) return launch_short(perm_kernel, dim3(ne), dim3(PERM_WARPS * 32), idx, (int)NK, grouped, inv, offsets);
    const int nblocks = (int)ceil_div64(NK, SORT_CHUNK);
    void* wsp;
    int rc = workspace(WS_PERM).ensure((size_t)nblocks * ne * sizeof(int32_t) + 256, &wsp);
    if (rc) return rc;
    int32_t* bc = static_cast<int32_t*>(wsp);
    sort_count_kernel<<<nblocks, SORT_THREADS, 0, stream()>>>(idx, NK, ne, bc);
    B200_LAUNCH_CHECK("sort_count_kernel");
    sort_scan_kernel<<<1, 320, 0, stream()>>>(bc, nblocks, ne, offsets);
    B200_LAUNCH_CHECK("sort_scan_kernel");
    sort_fill_kernel<<<nblocks, SORT_THREADS, 0, stream()>>>(idx, NK, ne, bc, grouped);
    B200_LAUNCH_CHECK("sort_fill_kernel");
    if (inv) {
        sort_inverse_kernel<<<(unsigned)ceil_div64(NK, 256), 256, 0, stream()>>>(grouped, inv, NK);
        B200_LAUNCH_CHECK("sort_inverse_kernel");
    }
    return B200_OK;
}

// ---------------------------------------------------------------------------
// Experts, token-major (small N): every (token, k) slot and every token's shared
// expert is an independent job.
//   kernel 1  act[job][i] = silu(gate_e[i].x_t) * up_e[i].x_t        (one warp per i)
//   kernel 2  out[t][j]   = shared_down[j].act_sh + sum_k w_k down_{e_k}[j].act_k
// ---------------------------------------------------------------------------
struct MoeArgs {
    const float* x;
    const uint8_t *gates, *ups, *downs, *sh_g, *sh_u, *sh_d;
    const int32_t* idx;     // [N,K]
    const float* w;         // [N,K]
    float* act;             // [N*K, E]
    float* sh_act;          // [N, SH]
    float *s_gate, *s_up;   // optional [N*K, E]
    float* out;             // [N, d]
    int N, d, E, ne, K, SH;
};

template <int KIND>
__global__ void __launch_bounds__(GEMV_THREADS) moe_gate_up_kernel(MoeArgs a) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * GEMV_WARPS + warp;
    const int job = blockIdx.y;
    const int routed = a.N * a.K;
    float g[1], u[1];
    if (job < routed) {
        if (i >= a.E) return;
        const int t = job / a.K, e = a.idx[job];
        const float* xt = a.x + (int64_t)t * a.d;
        gemv_row<KIND, 1>(xt, a.gates, (int64_t)e * a.E + i, 1, a.d, lane, g);
        gemv_row<KIND, 1>(xt, a.ups, (int64_t)e * a.E + i, 1, a.d, lane, u);
        if (lane == 0) {
            const int64_t o = (int64_t)job * a.E + i;
            a.act[o] = silu_acc(g[0]) * u[0];
            if (a.s_gate) a.s_gate[o] = g[0];
            if (a.s_up) a.s_up[o] = u[0];
        }
    } else {
        if (i >= a.SH) return;
        const int t = job - routed;
        const float* xt = a.x + (int64_t)t * a.d;
        gemv_row<KIND, 1>(xt, a.sh_g, i, 1, a.d, lane, g);
        gemv_row<KIND, 1>(xt, a.sh_u, i, 1, a.d, lane, u);
        if (lane == 0) a.sh_act[(int64_t)t * a.SH + i] = silu_acc(g[0]) * u[0];
    }
}

template <int KIND>
__global__ void __launch_bounds__(GEMV_THREADS) moe_down_combine_kernel(MoeArgs a) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = blockIdx.x * GEMV_WARPS + warp;
    const int t = blockIdx.y;
    if (j >= a.d) return;
    float r[1];
    float acc = 0.0f;
    if (a.sh_d) {
        gemv_row<KIND, 1>(a.sh_act + (int64_t)t * a.SH, a.sh_d, j, 1, a.SH, lane, r);
        acc = r[0];
    }
    for (int k = 0; k < a.K; ++k) {
        const int slot = t * a.K + k;
        const int e = a.idx[slot];
        gemv_row<KIND, 1>(a.act + (int64_t)slot * a.E, a.downs, (int64_t)e * a.d + j, 1, a.E, lane, r);
        acc = __fadd_rn(acc, __fmul_rn(a.w[slot], r[0]));
    }
    if (lane == 0) a.out[(int64_t)t * a.d + j] = acc;
}

template <int KIND>
static int launch_experts(const MoeArgs& a) {
    const bool shared = a.sh_g != nullptr;
    const int jobs = a.N * a.K + (shared ? a.N : 0);
    const int rows = std::max(a.E, shared ? a.SH : 0);
    moe_gate_up_kernel<KIND><<<dim3(ceil_div(rows, GEMV_WARPS), jobs), GEMV_THREADS, 0, stream()>>>(a);
    B200_LAUNCH_CHECK("moe_gate_up_kernel");
    moe_down_combine_kernel<KIND><<<dim3(ceil_div(a.d, GEMV_WARPS), a.N), GEMV_THREADS, 0, stream()>>>(a);
    B200_LAUNCH_CHECK("moe_down_combine_kernel");
    return B200_OK;
}

// ---------------------------------------------------------------------------
// Router.  The logit of (token, expert) keeps the reference's sequential fp32 chain over groups
// of four (products and sums rounded one by one: eight instructions per group, 23 us of a chip's fp32 rate for 4096 tokens
// of 1536 x 64 experts).  A thread carries TPT x EPT chains; token and expert rows come through a ring of asynchronous
// copies, RT_K columns at a time and a thousand columns deep where a block has few chains, because the chains advance
// faster than a cold load returns: the ring of three 64-column stages before it spent 1800 cycles per stage, a load's way.
// In us (before, now), router alone, launches included: 64 tokens of 1536 x 64
// 16.4 -> 14.3, 301 27.6 -> 20.5, 2048 44 -> 38; of 4096 x 72: 64 tokens 30 -> 25, 517 64 -> 50, 4096 210 -> 194; 4096 tokens of
// 768 x 16 34 -> 19.5.  (A layer's few tokens have the router of decode_moe.cu, unless it refuses their width.)  Larger thread tiles (4 x 4, 8 x 2) and packed additions were no faster: about two cycles a product or
// sum whatever their number.
// ---------------------------------------------------------------------------
constexpr int RT_K = 128, RT_LD = RT_K + 4, RT_THREADS = 256;

// One warp routes token t from its logits; s: ne floats of shared scratch.
template <int PER>
__device__ __forceinline__ void route_token(const float* __restrict__ logits, const float* __restrict__ router_bias, float* __restrict__ probs_out,
                                            int32_t* __restrict__ idx_out, float* __restrict__ w_out, int64_t t, int ne, int K, float* s, int lane) {
    float v[PER], bs[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int e = min(32 * i + lane, ne - 1);
        v[i] = __ldcg(logits + t * ne + e);
        bs[i] = router_bias ? router_bias[e] : 0.0f;
    }
    int idx;
    float w;
    route_pick<PER>(v, bs, router_bias != nullptr, ne, K, s, lane, idx, w);
    if (lane < K) {
        idx_out[t * K + lane] = idx;
        w_out[t * K + lane] = w;
    }
    if (probs_out)
#pragma unroll
        for (int i = 0; i < PER; ++i)
            if (32 * i + lane < ne) probs_out[t * ne + 32 * i + lane] = v[i];
}

// Two products, each rounded as __fmul_rn does, in one instruction (few warps: issue slots count).
__device__ __forceinline__ void mul_pair(float a, float b, float c, float d, float& ac, float& bd) {
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(ac), "=f"(bd)
        : "f"(a), "f"(b), "f"(c), "f"(d));
}

// Lanes: eight experts x four tokens; CW warps compute (one to a scheduler with the blocks that share an SM), all copy.
template <int TPT, int EPT, int CW, int STAGES>
struct RtShape {
    static constexpr int LE = 8, LT = 4, TOK = LT * TPT * CW, EXP = LE * EPT, ROWS = TOK + EXP, STAGE = ROWS * RT_LD, SMEM = STAGES * STAGE * 4;
};
template <int TPT, int EPT, int CW, int STAGES>
__global__ void __launch_bounds__(RT_THREADS)
route_logits_kernel(const float* __restrict__ x, const float* __restrict__ router_w, float* __restrict__ logits,
                    int64_t N, int d, int ne, const float* __restrict__ router_bias, float* __restrict__ probs_out,
                    int32_t* __restrict__ idx_out, float* __restrict__ w_out, int K, int* __restrict__ counters) {
    using S = RtShape<TPT, EPT, CW, STAGES>;
    extern __shared__ __align__(16) float rt_sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t t0 = (int64_t)blockIdx.x * S::TOK;
    const int e0 = blockIdx.y * S::EXP;
    // rows 0 .. TOK-1: tokens, then the experts; rows past the ends repeat the last one, columns past d are not read
    constexpr int PER = S::ROWS / (RT_THREADS / 32);
    static_assert(S::ROWS % (RT_THREADS / 32) == 0 && RT_K == 128, "a warp copies a row's 128 columns");
    const float* src[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int row = warp + u * (RT_THREADS / 32);
        src[u] = (row < S::TOK ? x + min(t0 + row, N - 1) * d : router_w + (int64_t)min(e0 + row - S::TOK, ne - 1) * d) + 4 * lane;
    }
    const uint32_t dst = smem_u32(rt_sm + warp * RT_LD + 4 * lane);
    const int chunks = (d + RT_K - 1) / RT_K;
    auto fetch = [&](int k) {
        if (k < chunks && k * RT_K + 4 * lane < d) {
            const uint32_t at = dst + (k % STAGES) * (S::STAGE * 4);
#pragma unroll
            for (int u = 0; u < PER; ++u)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at + u * (RT_THREADS / 32) * RT_LD * 4), "l"(src[u] + k * RT_K) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int te = lane % S::LE, tt = warp * S::LT * TPT + lane / S::LE;
    float acc[TPT][EPT] = {};
#pragma unroll
    for (int k = 0; k < STAGES - 1; ++k) fetch(k);
    pdl_launch_dependents();
    for (int k = 0; k < chunks; ++k) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                               // the stage is here, and the one before it is free
        fetch(k + STAGES - 1);
        if (warp >= CW) continue;
        const float* xs = rt_sm + (k % STAGES) * S::STAGE + tt * RT_LD;
        const float* ws = rt_sm + (k % STAGES) * S::STAGE + (S::TOK + te) * RT_LD;
        const int kc = min(RT_K, d - k * RT_K);        // a multiple of 4
        auto load = [&](int g, float4 (&a)[TPT], float4 (&b)[EPT]) {
#pragma unroll
            for (int j = 0; j < EPT; ++j) b[j] = *reinterpret_cast<const float4*>(ws + S::LE * j * RT_LD + g);
#pragma unroll
            for (int i = 0; i < TPT; ++i) a[i] = *reinterpret_cast<const float4*>(xs + S::LT * i * RT_LD + g);
        };
        auto group = [&](const float4 (&a)[TPT], const float4 (&b)[EPT]) {
#pragma unroll
            for (int i = 0; i < TPT; ++i)
#pragma unroll
                for (int j = 0; j < EPT; ++j) {
                    float px, py, pz, pw;
                    mul_pair(a[i].x, a[i].y, b[j].x, b[j].y, px, py);
                    mul_pair(a[i].z, a[i].w, b[j].z, b[j].w, pz, pw);
                    float s = __fadd_rn(px, py);
                    s = __fadd_rn(s, pz);
                    s = __fadd_rn(s, pw);
                    acc[i][j] = __fadd_rn(acc[i][j], s);
                }
        };
        float4 a[2][TPT], b[2][EPT];
        if (kc == RT_K) {
            // the next group's loads under this one's arithmetic
            load(0, a[0], b[0]);
            constexpr int UNROLL = TPT * EPT == 1 ? 8 : 4;
#pragma unroll UNROLL
            for (int g = 0; g < RT_K; g += 8) {
                load(g + 4, a[1], b[1]);
                group(a[0], b[0]);
                if (g + 8 < RT_K) load(g + 8, a[0], b[0]);
                group(a[1], b[1]);
            }
        } else {
            for (int g = 0; g < kc; g += 4) {
                load(g, a[0], b[0]);
                group(a[0], b[0]);
            }
        }
    }
    if (warp < CW) {
#pragma unroll
        for (int i = 0; i < TPT; ++i)
#pragma unroll
            for (int j = 0; j < EPT; ++j) {
                const int64_t t = t0 + tt + S::LT * i;
                const int e = e0 + te + S::LE * j;
                if (t < N && e < ne) logits[t * ne + e] = acc[i][j];
            }
    }
    // The block that completes a token tile's last expert tile turns the tile's logits into (idx, w), one warp per token:
    // nobody waits - each block counts itself in after publishing its logits, and whoever counts last finds all of them
    // (fence before the count and after it).
    __shared__ int s_last;
    if (!counters) return;                                   // the caller finishes with route_finish_kernel
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&counters[blockIdx.x], 1) == (int)gridDim.y - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int i = warp; i < S::TOK; i += RT_THREADS / 32) {
        const int64_t t = t0 + i;
        if (t >= N) break;
        float* s_p = rt_sm + (size_t)warp * MOE_MAX_NE;      // the tiles are dead
        if (ne <= 64) route_token<2>(logits, router_bias, probs_out, idx_out, w_out, t, ne, K, s_p, lane);
        else route_token<8>(logits, router_bias, probs_out, idx_out, w_out, t, ne, K, s_p, lane);
        __syncwarp();
    }
    if (threadIdx.x == 0) counters[blockIdx.x] = 0;           // ready for the next call
}
template <int TPT, int EPT, int CW, int STAGES>
static int launch_route_logits(const float* x, const float* router_w, float* logits, int64_t N, int d, int ne, const float* router_bias,
                               float* probs, int32_t* idx, float* w, int K, int* counters) {
    using S = RtShape<TPT, EPT, CW, STAGES>;
    static_assert(S::SMEM <= 227 * 1024 && S::SMEM >= RT_THREADS / 32 * MOE_MAX_NE * 4, "stages, and the finishing warps' scratch");
    auto kern = route_logits_kernel<TPT, EPT, CW, STAGES>;
    static bool configured = false;
    if (!configured) {
        B200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM));
        configured = true;
    }
    const dim3 grid((unsigned)ceil_div64(N, S::TOK), ceil_div(ne, S::EXP));
    kern<<<grid, RT_THREADS, S::SMEM, stream()>>>(x, router_w, logits, N, d, ne, router_bias, probs, idx, w, K, counters);
    B200_LAUNCH_CHECK("route_logits_kernel");
    return B200_OK;
}

// Tokens times experts enough to fill the device with blocks of 32 x 32: a thread carries eight tokens of one expert.  A warp reads its
// lanes' 32 expert rows (four wavefronts per group of columns) for eight token rows (one each, the same for all lanes), so that
// shared memory needs 12 cycles where the arithmetic needs 16.  In us, the form above and this one: 4096 and 16 384 tokens of 1536 x 64
// 58 / 54 and 195 / 164, 1024 and 4096 of 2048 x 256 77 / 70 and 252 / 212, 2048 of 8192 x 128 285 / 262; fewer tokens: 2048 of 1536 x 64 32 / 38,
// 700 of 2048 x 256 61 / 70, 1500 of 8192 x 128 222 / 263.  Not where a third of the experts' columns would be idle.
constexpr int RW_K = 64, RW_LD = RW_K + 4, RW_WARPS = 4, RW_THREADS = 32 * RW_WARPS, RW_STAGES = 3, RW_TOKENS = 8;
__global__ void __launch_bounds__(RW_THREADS)
route_logits_wide_kernel(const float* __restrict__ x, const float* __restrict__ router_w, float* __restrict__ logits,
                    int64_t N, int d, int ne) {
    constexpr int TOK = RW_WARPS * RW_TOKENS, ROWS = TOK + 32, STAGE = ROWS * RW_LD;
    extern __shared__ __align__(16) float rw_sm[];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t t0 = (int64_t)blockIdx.x * TOK;
    const int e0 = blockIdx.y * 32;
    // rows 0 .. TOK-1: tokens, then 32 experts; rows past the ends repeat the last one, columns past d are not read
    const int c4 = (threadIdx.x % (RW_K / 4)) * 4, r0 = threadIdx.x / (RW_K / 4);
    constexpr int STEP = RW_THREADS / (RW_K / 4), PER = ROWS / STEP;
    static_assert(ROWS % STEP == 0, "rows of a stage per copying thread");
    const int chunks = (d + RW_K - 1) / RW_K;
    auto fetch = [&](int k) {
        if (k < chunks) {
            float* st = rw_sm + (k % RW_STAGES) * STAGE;
            if (k * RW_K + c4 < d)
#pragma unroll
                for (int u = 0; u < PER; ++u) {
                    const int row = r0 + u * STEP;
                    const float* src = row < TOK ? x + min(t0 + row, N - 1) * d : router_w + (int64_t)min(e0 + row - TOK, ne - 1) * d;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(st + row * RW_LD + c4)), "l"(src + k * RW_K + c4) : "memory");
                }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[RW_TOKENS] = {};
#pragma unroll
    for (int k = 0; k < RW_STAGES - 1; ++k) fetch(k);
    for (int k = 0; k < chunks; ++k) {
        asm volatile("cp.async.wait_group %0;" ::"n"(RW_STAGES - 2) : "memory");
        __syncthreads();                               // the stage is here, and the one before it is free
        fetch(k + RW_STAGES - 1);
        const float* xs = rw_sm + (k % RW_STAGES) * STAGE + RW_TOKENS * ty * RW_LD;
        const float* ws = rw_sm + (k % RW_STAGES) * STAGE + (TOK + tx) * RW_LD;
        const int kc = min(RW_K, d - k * RW_K);        // a multiple of 4
        auto group = [&](int g) {
            const float4 b = *reinterpret_cast<const float4*>(ws + g);
#pragma unroll
            for (int i = 0; i < RW_TOKENS; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(xs + i * RW_LD + g);
                float s = __fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y));
                s = __fadd_rn(s, __fmul_rn(a.z, b.z));
                s = __fadd_rn(s, __fmul_rn(a.w, b.w));
                acc[i] = __fadd_rn(acc[i], s);
            }
        };
        // whole chunks with the loads of later groups under the additions of earlier ones (the chains are serial)
        if (kc == RW_K) {
#pragma unroll
            for (int g = 0; g < RW_K; g += 4) group(g);
        } else {
            for (int g = 0; g < kc; g += 4) group(g);
        }
    }
    const int e = e0 + tx;
#pragma unroll
    for (int i = 0; i < RW_TOKENS; ++i) {
        const int64_t t = t0 + RW_TOKENS * ty + i;
        if (t < N && e < ne) logits[t * ne + e] = acc[i];
    }
}
static int launch_route_logits_wide(const float* x, const float* router_w, float* logits, int64_t N, int d, int ne) {
    constexpr int SMEM = RW_STAGES * (RW_WARPS * RW_TOKENS + 32) * RW_LD * 4;
    static bool configured = false;
    if (!configured) {
        B200_CUDA(cudaFuncSetAttribute(route_logits_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured = true;
    }
    const dim3 grid((unsigned)ceil_div64(N, RW_WARPS * RW_TOKENS), ceil_div(ne, 32));
    route_logits_wide_kernel<<<grid, RW_THREADS, SMEM, stream()>>>(x, router_w, logits, N, d, ne);
    B200_LAUNCH_CHECK("route_logits_wide_kernel");
    return B200_OK;
}

// Arrival counters of the kernel above (one per token group), zeroed once; every call leaves them zero.
// Not created while the stream is being captured into a graph (an allocation and a memset on the
// default stream do not belong there): the caller then runs the separate finishing kernel.
constexpr int ROUTE_COUNTERS = 1024;
static int* route_counters() {
    static int* p = nullptr;
    if (!p) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream(), &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
            cudaGetLastError();
            return nullptr;
        }
        if (cudaMalloc(&p, ROUTE_COUNTERS * sizeof(int)) != cudaSuccess) { p = nullptr; cudaGetLastError(); return nullptr; }
        if (cudaMemset(p, 0, ROUTE_COUNTERS * sizeof(int)) != cudaSuccess) { cudaFree(p); p = nullptr; cudaGetLastError(); return nullptr; }
    }
    return p;
}

constexpr int RF_WARPS = 8;
template <int PER>
__global__ void __launch_bounds__(RF_WARPS * 32)
route_finish_kernel(const float* __restrict__ logits, const float* __restrict__ router_bias, float* __restrict__ probs_out,
                    int32_t* __restrict__ idx_out, float* __restrict__ w_out, int64_t N, int ne, int K) {
    __shared__ float s_p[RF_WARPS][32 * PER];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t t = (int64_t)blockIdx.x * RF_WARPS + warp;
    pdl_launch_dependents();
    pdl_wait();
    if (t < N) route_token<PER>(logits, router_bias, probs_out, idx_out, w_out, t, ne, K, s_p[warp], lane);
}

int moe_route(const float* x, const float* router_w, const float* router_bias, float* probs,
              int32_t* idx, float* w, int64_t N, int d, int ne, int K) {
    if (d % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        void* wsp;
        int rc = workspace(WS_ROUTE).ensure((size_t)N * ne * 4 + 256, &wsp);
        if (rc) return rc;
        float* logits = static_cast<float*>(wsp);
        // One chain per thread in blocks of 8 x 8 (most blocks, least latency) or four in blocks of 32 x 16 (a third of the
        // shared loads per product).  Times in units of some us, from 1536 columns and 64 experts: 128 / 256 / 517 / 1024 tokens
        // take 14 / 18 / 29 / 41 us with the first and 24 / 24 / 24 / 26 with the second, 2048 take 66 and 38.  (The fixed terms are those
        // of that width; wider rows come to the second form early: 517 tokens of 4096 x 72 are 85 blocks of it, 44 us.)
        auto rounds = [&](int tok, int exp) { return ceil_div64(ceil_div64(N, tok) * ceil_div(ne, exp), num_sms()); };
        int* counters = nullptr;
        const int64_t wide = ceil_div64(N, RW_WARPS * RW_TOKENS) * ceil_div(ne, 32);
        if (2 * wide > 3 * num_sms() && 6 * 32 * ceil_div(ne, 32) < 7 * 16 * ceil_div(ne, 16)) {
            rc = launch_route_logits_wide(x, router_w, logits, N, d, ne);
        } else if (5 * rounds(8, 8) + 4 <= 12 * rounds(32, 16) + 7) {
            if (N <= 8 * ROUTE_COUNTERS) counters = route_counters();
            rc = launch_route_logits<1, 1, 2, 8>(x, router_w, logits, N, d, ne, router_bias, probs, idx, w, K, counters);
        } else {
            rc = launch_route_logits<2, 2, 4, 4>(x, router_w, logits, N, d, ne, router_bias, probs, idx, w, K, nullptr);
        }
        if (rc || counters) return rc;
        const dim3 blocks((unsigned)ceil_div64(N, RF_WARPS)), threads(RF_WARPS * 32);
        if (ne <= 64) return launch_short(route_finish_kernel<2>, blocks, threads, logits, router_bias, probs, idx, w, N, ne, K);
        if (ne <= 128) return launch_short(route_finish_kernel<4>, blocks, threads, logits, router_bias, probs, idx, w, N, ne, K);
        return launch_short(route_finish_kernel<8>, blocks, threads, logits, router_bias, probs, idx, w, N, ne, K);
    }
    // shared memory: x + as many group rows as fit in ~96 KB
    const int groups = d >> 2;
    const size_t x_bytes = (size_t)((d + 3) & ~3) * 4;
    int chunk = (int)std::min<size_t>((size_t)std::max(groups, 1), (96 * 1024 - x_bytes) / ((size_t)(ne + 1) * 4));
    B200_REQUIRE(chunk >= 1, "moe: hidden size too large for the router kernel");
    const size_t smem = x_bytes + (size_t)chunk * (ne + 1) * 4;
    static size_t configured = 0;
    if (smem > 48 * 1024 && smem > configured) {
        B200_CUDA(cudaFuncSetAttribute(moe_route_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
        configured = 100 * 1024;
    }
    moe_route_kernel<<<(unsigned)N, ROUTE_THREADS, smem, stream()>>>(x, router_w, router_bias, probs, idx, w, d, ne,
                                                                     K, chunk);
    B200_LAUNCH_CHECK("moe_route_kernel");
    return B200_OK;
}

// kind: template tag.  Weight pointers are raw bytes in that kind.
int moe_forward(const float* x, const float* router_w, const float* router_bias, const void* gates,
                const void* ups, const void* downs, const void* sh_g, const void* sh_u, const void* sh_d,
                float* out, float* probs_cache, int32_t* idx_cache, float* w_cache, float* s_gate,
                float* s_up, float* s_act, int64_t N, int d, int E, int ne, int K, int SH, int kind) {
    if (N <= 0) return B200_OK;
    B200_REQUIRE(K >= 1 && K <= MOE_MAX_K, "moe_forward: K must be in [1,%d]", MOE_MAX_K);
    B200_REQUIRE(ne > 0 && ne <= MOE_MAX_NE && K <= ne, "moe_forward: ne out of range");
    B200_REQUIRE(d > 0 && E > 0, "moe_forward: bad dims");
    B200_REQUIRE(x && router_w && gates && ups && downs && out, "moe_forward: null pointer");
    B200_REQUIRE(d % 32 == 0 && E % 32 == 0, "moe_forward: d and E must be multiples of 32");
    B200_REQUIRE((reinterpret_cast<uintptr_t>(router_w) & 15) == 0 && d % 4 == 0, "moe_forward: router_w alignment");
    const bool shared = sh_g && sh_u && sh_d;
    if (shared) B200_REQUIRE(SH > 0 && SH % 32 == 0, "moe_forward: SH must be a positive multiple of 32");
    if (kind >= 0 && kind <= 3)
        B200_REQUIRE(d % q_block_elems(kind) == 0 && E % q_block_elems(kind) == 0 &&
                         (!shared || SH % q_block_elems(kind) == 0),
                     "moe_forward: d, E and SH must be multiples of the quantisation block");
    B200_REQUIRE(N * K < ((int64_t)1 << 31), "moe_forward: N too large");

    // Many tokens over fp16 / packed experts: expert-grouped tensor-core GEMMs.  The
    // optional fp32 scratch outputs only exist on the token-major path.
    auto aligned16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    // Up to eight tokens over packed experts: the decode step's three kernels (decode_moe.cu) with no norm in front and
    // the plain output (one token of the H-Tiny shape: 52 us of three dependent kernels here, 33 of them the router).
    if (N <= 8 && kind >= 0 && kind <= 3 && !s_gate && !s_up && !s_act) {
        size_t off = 0;
        auto take = [&](size_t bytes) { const size_t o = off; off += (bytes + 255) & ~(size_t)255; return o; };
        const size_t o_idx = take(N * K * 4), o_w = take(N * K * 4), o_act = take(N * K * E * 4), o_sh = take(N * (size_t)SH * 4);
        void* wsp;
        int rc = workspace(WS_MOE).ensure(off + 256, &wsp);
        if (rc) return rc;
        char* base = static_cast<char*>(wsp);
        MoeFusedArgs m;
        m.x = x; m.router_w = router_w; m.router_bias = router_bias;
        m.gates = static_cast<const uint8_t*>(gates); m.ups = static_cast<const uint8_t*>(ups); m.downs = static_cast<const uint8_t*>(downs);
        m.sh_g = static_cast<const uint8_t*>(sh_g); m.sh_u = static_cast<const uint8_t*>(sh_u); m.sh_d = static_cast<const uint8_t*>(sh_d);
        m.idx = idx_cache ? idx_cache : reinterpret_cast<int32_t*>(base + o_idx);
        m.w = w_cache ? w_cache : reinterpret_cast<float*>(base + o_w);
        m.probs_out = probs_cache;
        m.act = reinterpret_cast<float*>(base + o_act);
        m.sh_act = reinterpret_cast<float*>(base + o_sh);
        m.out = out;
        m.M = (int)N; m.d = d; m.E = E; m.ne = ne; m.K = K; m.SH = shared ? SH : 0;
        rc = moe_fused(m, kind);
        if (rc != B200_EUNSUPPORTED) return rc;
    }
    // A decode batch: at most MOE_UNITS_MAX_ROWS rows per expert on average.  The experts'
    // rows would leave the 128-row tensor-core tiles nearly empty; they run as weight streams
    // shared by their tokens instead (moe_exact.cu, moe_units.cu).
    // (Up to eight tokens come here where the three kernels above refuse them: 3, 5, 8 tokens of 768 x 4096 in Q8_0 took 397, 638
    // and 1000 us token by token.  Not in place, which every other form for few tokens takes: the units' shared expert writes out
    // beside the routed experts that read x.)
    const bool in_place = x < out + N * d && out < x + N * d;
    if ((N > 8 || (kind >= 0 && kind <= 3 && !in_place)) && N * K <= (int64_t)MOE_UNITS_MAX_ROWS * ne && kind != KIND_F32 && !s_gate && !s_up && !s_act && aligned16(x) &&
        aligned16(out) && aligned16(gates) && aligned16(ups) && aligned16(downs) && d % 8 == 0 &&
        (kind != 3 || (d % 256 == 0 && E % 256 == 0)) && ne <= 256 &&
        (!shared || (aligned16(sh_g) && aligned16(sh_u) && aligned16(sh_d) && (kind == KIND_F16 || SH % 256 == 0)))) {
        const int rc = moe_forward_units(x, router_w, router_bias, gates, ups, downs, sh_g, sh_u, sh_d, out, probs_cache,
                                         idx_cache, w_cache, N, d, E, ne, K, shared ? SH : 0, kind);
        if (rc != B200_EUNSUPPORTED) return rc;
    }
    if (N >= GEMM_MIN_ROWS && kind != KIND_F32 && !s_gate && !s_up && !s_act && aligned16(x) && aligned16(out) &&
        aligned16(gates) && aligned16(ups) && aligned16(downs) &&
        (!shared || (aligned16(sh_g) && aligned16(sh_u) && aligned16(sh_d))))
        return moe_forward_grouped(x, router_w, router_bias, gates, ups, downs, sh_g, sh_u, sh_d, out, probs_cache,
                                   idx_cache, w_cache, N, d, E, ne, K, shared ? SH : 0, kind);

    // workspace: idx | w | act | sh_act
    const size_t NK = (size_t)N * K;
    size_t off = 0;
    auto take = [&](size_t bytes) { const size_t o = off; off += (bytes + 255) & ~(size_t)255; return o; };
    const size_t o_idx = take(NK * 4), o_w = take(NK * 4);
    const size_t o_act = s_act ? 0 : take(NK * E * 4);
    const size_t o_sh = shared ? take((size_t)N * SH * 4) : 0;
    void* wsp;
    int rc = workspace(WS_MOE).ensure(off + 256, &wsp);
    if (rc) return rc;
    char* base = static_cast<char*>(wsp);
    int32_t* idx = idx_cache ? idx_cache : reinterpret_cast<int32_t*>(base + o_idx);
    float* w = w_cache ? w_cache : reinterpret_cast<float*>(base + o_w);

    rc = moe_route(x, router_w, router_bias, probs_cache, idx, w, N, d, ne, K);
    if (rc) return rc;

    MoeArgs a;
    a.x = x;
    a.gates = static_cast<const uint8_t*>(gates);
    a.ups = static_cast<const uint8_t*>(ups);
    a.downs = static_cast<const uint8_t*>(downs);
    a.sh_g = shared ? static_cast<const uint8_t*>(sh_g) : nullptr;
    a.sh_u = shared ? static_cast<const uint8_t*>(sh_u) : nullptr;
    a.sh_d = shared ? static_cast<const uint8_t*>(sh_d) : nullptr;
    a.idx = idx;
    a.w = w;
    a.act = s_act ? s_act : reinterpret_cast<float*>(base + o_act);
    a.sh_act = shared ? reinterpret_cast<float*>(base + o_sh) : nullptr;
    a.s_gate = s_gate;
    a.s_up = s_up;
    a.out = out;
    a.N = (int)N; a.d = d; a.E = E; a.ne = ne; a.K = K; a.SH = shared ? SH : 0;
    // grid.y carries the jobs: walk the tokens in chunks that keep it under 65535
    const int chunk_tokens = std::max(1, 65535 / (K + 1));
    for (int64_t t0 = 0; t0 < N; t0 += chunk_tokens) {
        MoeArgs c = a;
        c.N = (int)std::min<int64_t>(chunk_tokens, N - t0);
        c.x = a.x + t0 * d;
        c.idx = a.idx + t0 * K;
        c.w = a.w + t0 * K;
        c.act = a.act + t0 * K * E;
        if (a.sh_act) c.sh_act = a.sh_act + t0 * SH;
        if (a.s_gate) c.s_gate = a.s_gate + t0 * K * E;
        if (a.s_up) c.s_up = a.s_up + t0 * K * E;
        c.out = a.out + t0 * d;
        switch (kind) {
            case 0: rc = launch_experts<0>(c); break;
            case 1: rc = launch_experts<1>(c); break;
            case 2: rc = launch_experts<2>(c); break;
            case 3: rc = launch_experts<3>(c); break;
            case KIND_F16: rc = launch_experts<KIND_F16>(c); break;
            default: rc = launch_experts<KIND_F32>(c); break;
        }
        if (rc) return rc;
    }
    return B200_OK;
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_moe_forward(const float* x, const float* router_w, const float* gates, const float* ups,
                     const float* downs, const float* sh_g, const float* sh_u, const float* sh_d,
                     float* out, float* probs_cache, int32_t* idx_cache, float* w_cache,
                     float* s_gate, float* s_up, float* s_act,
                     int64_t N, int d, int E, int ne, int K, int SH) {
    return moe_forward(x, router_w, nullptr, gates, ups, downs, sh_g, sh_u, sh_d, out, probs_cache, idx_cache,
                       w_cache, s_gate, s_up, s_act, N, d, E, ne, K, SH, KIND_F32);
}
int b200_moe_forward_bias(const float* x, const float* router_w, const float* router_bias,
                          const float* gates, const float* ups, const float* downs,
                          const float* sh_g, const float* sh_u, const float* sh_d,
                          float* out, float* probs_cache, int32_t* idx_cache, float* w_cache,
                          float* s_gate, float* s_up, float* s_act,
                          int64_t N, int d, int E, int ne, int K, int SH) {
    return moe_forward(x, router_w, router_bias, gates, ups, downs, sh_g, sh_u, sh_d, out, probs_cache, idx_cache,
                       w_cache, s_gate, s_up, s_act, N, d, E, ne, K, SH, KIND_F32);
}
int b200_moe_forward_half(const float* x, const float* router_w, const uint16_t* gates,
                          const uint16_t* ups, const uint16_t* downs, const uint16_t* sh_g,
                          const uint16_t* sh_u, const uint16_t* sh_d, float* out,
                          float* probs_cache, int32_t* idx_cache, float* w_cache,
                          float* s_gate, float* s_up, float* s_act,
                          int64_t N, int d, int E, int ne, int K, int SH, int qkind) {
    B200_REQUIRE(qkind >= -1 && qkind <= 3, "moe_forward_half: unknown qkind %d", qkind);
    return moe_forward(x, router_w, nullptr, gates, ups, downs, sh_g, sh_u, sh_d, out, probs_cache, idx_cache,
                       w_cache, s_gate, s_up, s_act, N, d, E, ne, K, SH, tag_of_qkind(qkind));
}
int b200_moe_forward_bias_half(const float* x, const float* router_w, const float* router_bias,
                               const uint16_t* gates, const uint16_t* ups, const uint16_t* downs,
                               const uint16_t* sh_g, const uint16_t* sh_u, const uint16_t* sh_d,
                               float* out, float* probs_cache, int32_t* idx_cache, float* w_cache,
                               float* s_gate, float* s_up, float* s_act,
                               int64_t N, int d, int E, int ne, int K, int SH, int qkind) {
    B200_REQUIRE(qkind >= -1 && qkind <= 3, "moe_forward_bias_half: unknown qkind %d", qkind);
    return moe_forward(x, router_w, router_bias, gates, ups, downs, sh_g, sh_u, sh_d, out, probs_cache, idx_cache,
                       w_cache, s_gate, s_up, s_act, N, d, E, ne, K, SH, tag_of_qkind(qkind));
}
int b200_moe_permutation(const int32_t* idx, int64_t NK, int ne, int32_t* grouped, int32_t* offsets) {
    return moe_permutation(idx, NK, ne, grouped, nullptr, offsets);
}

}  // extern "C"
