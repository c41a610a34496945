// Single-token GQA attention over an fp16 ring or paged KV cache, head_dim 64 / 128, on
// mma.sync with every fp32 operand cut in three fp16 parts.
//
// Reference arithmetic: core/attn_cpu.cpp:151-254; kernels replaced: cuda/attention.cu:614-809.
//
// What bounds it: the K and V rows, read once (4 * len * KV * hd bytes).  The scalar form spent
// 8 FMAs, five shuffles and two exponentials per key and query head and reached 7 % of the copy
// rate; here a warp takes 16 keys at a time for the up to eight query heads of a KV head:
//   S[16, 16 keys]  = Q . K^T    rows 0-7 the heads' high parts, rows 8-15 their middle parts, so a
//                                thread's accumulators c0 + c2 are one head's; the low parts in a
//                                product of their own
//   O[16, hd]      += P . V      the same split of the probabilities; the parts are added at the end
// q is scaled by a power of two to at most 2^10 before the cut and p runs up to 2^10, so three parts
// hold all 24 bits of both; K and V are fp16 in memory.  The tensor cores cut a sum's last bits off where
// an addition rounds them, so the high parts' products are added up outside, 16 dims or keys at a time.
// Every warp keeps a ring of three 16-key stages of its own in shared memory, filled by cp.async and read
// by ldmatrix (rows padded by 16 bytes: no bank conflicts), so 17 KB per warp are always under way and no
// block-wide barrier is on the path.  (The same kernel with the rows in registers, loaded one tile ahead:
// 0.295 ms on the case below, 57 % of the warps' time in load latency.)
// 64 sequences of 256 .. 8192 tokens, 32 / 8 heads of 128: 2.50 ms before, 0.23 ms now
// (1.11 GB: 4.8 TB/s, 75 % of the measured copy rate).  With two parts and sums left to the tensor cores it took 0.21, at
// twice the error of fp32 arithmetic (3.6e-7 of the output's norm at scores of unit variance, where the scalar form
// has 1.9e-7 and this 2.2e-7; over the whole case above 4.7e-7, the scalar form's long sums, against 2.2e-7 here).
#include <algorithm>
#include <type_traits>

#include "attention_decode.cuh"
#include "fused_common.cuh"

namespace b200 {

constexpr int AD_WARPS = 4;
constexpr int AD_HEADS = 8;           // query heads of one KV head per block
constexpr int AD_TILE = 16;           // keys per warp step
constexpr int AD_STAGES = 3;
constexpr int AD_STEP = AD_WARPS * AD_TILE;
constexpr int AD_MAX_SPLITS = 128;
constexpr int AD_MAX_COUNTERS = 1 << 16;
constexpr float AD_P_UNIT = 1024.0f;  // probabilities carry a factor 2^10

// Blocks of a (sequence, KV head, head block) that have left their partial result; the last one
// merges and puts the word back to zero.
static __device__ unsigned int g_ad_count[AD_MAX_COUNTERS];

__device__ __forceinline__ void ad_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// c0, c1 of one product alone, for an addition that rounds; c2, c3 go on from c.
__device__ __forceinline__ void ad_mma_top(float (&d)[4], const float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                           uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%11,%12};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f), "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ uint32_t ad_pack(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void ad_ldsm(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ad_ldsm_t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// (a, b) as fp16 pairs: the rounded values, what rounding left of them, and of that
__device__ __forceinline__ void ad_split(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 r = __floats2half2_rn(a - f.x, b - f.y);
    const float2 g = __half22float2(r);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    mid = *reinterpret_cast<const uint32_t*>(&r);
    lo = ad_pack(a - f.x - g.x, b - f.y - g.y);
}

// An empty range gives zeros (the reference's sum > 0 guard); a sum that is not a number shows.
__device__ __forceinline__ float4 ad_over(const float4& o, float l) {
    return l == 0.0f ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(o.x / l, o.y / l, o.z / l, o.w / l);
}

// Row of logical position j: pinned prefix + rolling window (core/attn_cpu.cpp:151-156), or the page.
template <bool PAGED>
__device__ __forceinline__ int64_t ad_row(const DecodeMmaArgs& a, const int32_t* pages, int j) {
    if (PAGED) return (int64_t)pages[j / a.page] * a.page + j % a.page;
    return j < a.pinned ? j : (int64_t)a.pinned + (a.ring_start + (j - a.pinned)) % a.ring_cap;
}

template <int HD>
struct AdSmem {
    static constexpr int ROW = HD * 2 + 16;                   // bytes of a staged row
    static constexpr int STAGE = 2 * AD_TILE * ROW;           // K rows, then V rows
    static constexpr int WARP = AD_STAGES * STAGE;
    static constexpr int RING = AD_WARPS * WARP;              // re-used for the merges
    static constexpr int Q2 = HD / 16 * 32 * 16;              // high and middle parts of the queries
    static constexpr int Q = Q2 + HD / 16 * 32 * 8;           // and low ones
    static constexpr int BYTES = RING + Q + AD_WARPS * AD_HEADS * 2 * 4 + AD_HEADS * 4 + 16;
};

// grid (splits, KV * head blocks, batch)
// FOUR: at most four query heads to a KV head, so all three parts of each fit the sixteen rows: 0-3 high, 4-7 middle, 8-11
// low; lanes g and g + 4 hold the same head's score, probability and sum.
template <int HD, bool PAGED, bool FOUR>
__global__ void __launch_bounds__(AD_WARPS * 32, 2) attn_decode_mma_kernel(DecodeMmaArgs a) {
    using S = AdSmem<HD>;
    constexpr int NT = HD / 8;                                // output tiles of 8 dims
    constexpr int CH = HD / 8;                                // 16-byte pieces of a row
    extern __shared__ __align__(128) uint8_t ad_smem[];
    uint4(*s_q)[32] = reinterpret_cast<uint4(*)[32]>(ad_smem + S::RING);          // A fragments of Q, one per 16 dims
    uint2(*s_q3)[32] = reinterpret_cast<uint2(*)[32]>(ad_smem + S::RING + S::Q2); // and of its low parts, eight rows
    float(*s_ml)[AD_HEADS][2] = reinterpret_cast<float(*)[AD_HEADS][2]>(ad_smem + S::RING + S::Q);
    float* s_mul = reinterpret_cast<float*>(s_ml + AD_WARPS);                     // product -> score
    int* s_last = reinterpret_cast<int*>(s_mul + AD_HEADS);
    float(*s_o)[AD_HEADS][HD] = reinterpret_cast<float(*)[AD_HEADS][HD]>(ad_smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int gblocks = (a.group + AD_HEADS - 1) / AD_HEADS;
    const int kvh = blockIdx.y / gblocks, g0 = (blockIdx.y % gblocks) * AD_HEADS, b = blockIdx.z;
    const int G = min(AD_HEADS, a.group - g0);
    const int h0 = kvh * a.group + g0;
    pdl_launch_dependents();
    pdl_wait();
    const int len = PAGED ? __ldcg(a.seq_lens + b) : a.cur_len - a.j0;
    // this sequence's own cut: even pieces of whole steps, so a short sequence uses few blocks
    const int chunk = max(AD_STEP, ((len + a.splits - 1) / a.splits + AD_STEP - 1) / AD_STEP * AD_STEP);
    const int ns = max(1, (len + chunk - 1) / chunk);
    if (blockIdx.x >= ns) return;
    const int jbeg = blockIdx.x * chunk, jend = min(len, jbeg + chunk);
    const int32_t* pages = PAGED ? a.page_table + (int64_t)b * a.max_pages : nullptr;
    const int jofs = PAGED ? 0 : a.j0;
    const int64_t stride = (int64_t)a.KV * HD;
    const uint16_t* kc = a.kc + (int64_t)kvh * HD + lane % CH * 8;
    const uint16_t* vc = a.vc + (int64_t)kvh * HD + lane % CH * 8;
    const uint32_t ring = smem_u32(ad_smem) + warp * S::WARP;

    auto row_of = [&](int j) { return ad_row<PAGED>(a, pages, jofs + min(j, jend - 1)); };   // past the end: the last key again
    // one 16-key tile into stage s; lane l brings row (i * 32 + l) / CH, piece l % CH; r: the row of key l % 16
    auto issue = [&](int s, int64_t r) {
        const uint32_t dst = ring + s * S::STAGE + lane / CH * S::ROW + lane % CH * 16;
#pragma unroll
        for (int i = 0; i < AD_TILE * CH / 32; ++i) {
            const int64_t at = __shfl_sync(0xffffffffu, r, i * (32 / CH) + lane / CH) * stride;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * (32 / CH) * S::ROW), "l"(kc + at) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + AD_TILE * S::ROW + i * (32 / CH) * S::ROW), "l"(vc + at) : "memory");
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    int j = jbeg + warp * AD_TILE;
    int64_t row = 0;                                          // of the next tile to bring
#pragma unroll
    for (int s = 0; s < AD_STAGES - 1; ++s) {
        if (j + s * AD_STEP < jend) issue(s, row_of(j + s * AD_STEP + (lane & 15)));
        commit();
    }
    if (j + (AD_STAGES - 1) * AD_STEP < jend) row = row_of(j + (AD_STAGES - 1) * AD_STEP + (lane & 15));
    // Q of head g0 + w, w + 4: scaled by 2^-e to at most 2^10, cut, laid out as A fragments
    for (int w = warp; w < (FOUR ? AD_HEADS / 2 : AD_HEADS); w += AD_WARPS) {
        const float* q = a.q + ((int64_t)b * a.H + h0 + w) * HD;
        float v[HD / 32], mx = 0.0f;
#pragma unroll
        for (int i = 0; i < HD / 32; ++i) {
            v[i] = w < G ? __ldcg(q + 32 * i + lane) : 0.0f;
            mx = fmaxf(mx, fabsf(v[i]));
        }
        mx = warp_max(mx);
        int e = 0;
        if (mx > 0.0f && isfinite(mx)) frexpf(mx, &e);
        e = max(e, -100);                                     // a head of denormals stays as it is
        const float mul = ldexpf(1.0f, 10 - e);
        if (lane == 0) s_mul[w] = ldexpf(a.scale, e - 10);
#pragma unroll
        for (int i = 0; i < HD / 32; ++i) {
            // dim x of a step's 16 belongs to thread (x % 8) / 2, register pair x / 8, half x % 2
            const int x = lane & 15;
            const float f = v[i] * mul;
            const __half hi = __float2half_rn(f);
            const __half mid = __float2half_rn(f - __half2float(hi));
            const __half lo = __float2half_rn(f - __half2float(hi) - __half2float(mid));
            __half* dst = reinterpret_cast<__half*>(&s_q[2 * i + (lane >> 4)][4 * w + (x & 7) / 2]) + (x >> 3) * 4 + (x & 1);
            dst[0] = hi;                                      // a0 | a1 | a2 | a3, two halves each
            if (FOUR) {
                __half* dst4 = dst + 4 * 4 * 8;               // four rows on
                dst4[0] = mid;
                dst[2] = lo;
                dst4[2] = __ushort_as_half(0);
            } else {
                dst[2] = mid;
                *(reinterpret_cast<__half*>(&s_q3[2 * i + (lane >> 4)][4 * w + (x & 7) / 2]) + (x >> 3) * 2 + (x & 1)) = lo;
            }
        }
    }
    __syncthreads();
    const float mul = s_mul[FOUR ? g & 3 : g];
    float o[NT][4], m = -INFINITY, l = 0.0f;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[n][i] = 0.0f;
    // ldmatrix row addresses inside a stage: K (keys x dims) as it lies, V transposed
    const uint32_t k_at = ((lane & 7) + (lane >> 4) * 8) * S::ROW + ((lane >> 3) & 1) * 16;
    const uint32_t v_at = AD_TILE * S::ROW + (lane & 15) * S::ROW + (lane >> 4) * 16;

    for (int s = 0; j < jend; j += AD_STEP, s = s + 1 == AD_STAGES ? 0 : s + 1) {
        asm volatile("cp.async.wait_group %0;" ::"n"(AD_STAGES - 2) : "memory");
        __syncwarp();                                         // this tile is here, and the tile before it is read
        if (j + (AD_STAGES - 1) * AD_STEP < jend) {
            issue(s == 0 ? AD_STAGES - 1 : s - 1, row);
            if (j + AD_STAGES * AD_STEP < jend) row = row_of(j + AD_STAGES * AD_STEP + (lane & 15));
        }
        commit();
        const uint32_t st = ring + s * S::STAGE;
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f}, u0[4] = {0.f, 0.f, 0.f, 0.f}, u1[4] = {0.f, 0.f, 0.f, 0.f};
        float p0[2], p1[2];
#pragma unroll
        for (int c = 0; c < HD / 16; ++c) {
            const uint4 f = s_q[c][lane];
            uint32_t kr[4];
            float d0[4], d1[4];
            ad_ldsm(st + k_at + c * 32, kr);
            ad_mma_top(d0, s0, f.x, f.y, f.z, f.w, kr[0], kr[1]);
            ad_mma_top(d1, s1, f.x, f.y, f.z, f.w, kr[2], kr[3]);
            if (!FOUR) {
                const uint2 f3 = s_q3[c][lane];
                ad_mma(u0, f3.x, 0u, f3.y, 0u, kr[0], kr[1]);
                ad_mma(u1, f3.x, 0u, f3.y, 0u, kr[2], kr[3]);
            }
            s0[2] = d0[2]; s0[3] = d0[3]; s1[2] = d1[2]; s1[3] = d1[3];
            if (c & 1) {                                      // pairs first: fewer roundings in a row
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    s0[i] += p0[i] + d0[i];
                    s1[i] += p1[i] + d1[i];
                }
            } else {
#pragma unroll
                for (int i = 0; i < 2; ++i) { p0[i] = d0[i]; p1[i] = d1[i]; }
            }
        }
        float x[4] = {s0[0] + (s0[2] + u0[0]), s0[1] + (s0[3] + u0[1]), s1[0] + (s1[2] + u1[0]), s1[1] + (s1[3] + u1[1])};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (FOUR) x[i] += __shfl_xor_sync(0xffffffffu, x[i], 16);
            x[i] *= mul;
        }
        if (j + AD_TILE > jend) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (j + 2 * t + (i & 1) + 8 * (i >> 1) >= jend) x[i] = -INFINITY;
        }
        float mn = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
        mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
        mn = fmaxf(m, fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2)));
        if (__any_sync(0xffffffffu, mn != m)) {
            const float corr = expf(m - mn);                  // exp(-inf) = 0 on the first keys
            l *= corr;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) o[n][i] *= corr;
            m = mn;
        }
        uint32_t hi[2], mid[2], lo[2];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = expf(x[i] - m) * AD_P_UNIT;
        l += (x[0] + x[1]) + (x[2] + x[3]);
        ad_split(x[0], x[1], hi[0], mid[0], lo[0]);
        ad_split(x[2], x[3], hi[1], mid[1], lo[1]);
        if (FOUR) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                hi[i] = g < 4 ? hi[i] : mid[i];
                mid[i] = g < 4 ? lo[i] : 0u;
            }
        }
#pragma unroll
        for (int n = 0; n < NT; n += 2) {
            uint32_t vr[4];
            ad_ldsm_t(st + v_at + n * 16, vr);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float d[4];
                ad_mma_top(d, o[n + i], hi[0], mid[0], hi[1], mid[1], vr[2 * i], vr[2 * i + 1]);
                if (!FOUR) ad_mma(d, 0u, lo[0], 0u, lo[1], vr[2 * i], vr[2 * i + 1]);
                o[n + i][0] += d[0]; o[n + i][1] += d[1]; o[n + i][2] = d[2]; o[n + i][3] = d[3];
            }
        }
    }
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                          // the rings become s_o
    if (FOUR) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 2; ++i) o[n][2 + i] += __shfl_down_sync(0xffffffffu, o[n][i], 16);        // the middle part's row
    }
    if (g < G) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
            *reinterpret_cast<float2*>(&s_o[warp][g][8 * n + 2 * t]) = make_float2(o[n][0] + o[n][2], o[n][1] + o[n][3]);
        if (t == 0) { s_ml[warp][g][0] = m; s_ml[warp][g][1] = l; }
    }
    __syncthreads();
    constexpr int REC = HD + 4;
    for (int i = threadIdx.x; i < G * (HD / 4); i += AD_WARPS * 32) {
        const int hh = i / (HD / 4), c = i % (HD / 4) * 4;
        float mm = -INFINITY, ll = 0.0f;
#pragma unroll
        for (int w = 0; w < AD_WARPS; ++w) mm = fmaxf(mm, s_ml[w][hh][0]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < AD_WARPS; ++w) {
            const float mw = s_ml[w][hh][0];
            const float f = mw == -INFINITY ? 0.0f : expf(mw - mm);
            const float4 v = *reinterpret_cast<const float4*>(&s_o[w][hh][c]);
            ll += s_ml[w][hh][1] * f;
            acc.x += v.x * f; acc.y += v.y * f; acc.z += v.z * f; acc.w += v.w * f;
        }
        if (ns == 1) {
            *reinterpret_cast<float4*>(a.out + ((int64_t)b * a.H + h0 + hh) * HD + c) = ad_over(acc, ll);
        } else {
            float* dst = a.part + (((int64_t)b * a.H + h0 + hh) * a.splits + blockIdx.x) * REC;
            *reinterpret_cast<float4*>(dst + c) = acc;
            if (c == 0) { dst[HD] = mm; dst[HD + 1] = ll; }
        }
    }
    if (ns == 1) return;
    // the block that counts in last merges the pieces
    __threadfence();
    __syncthreads();
    unsigned int* count = g_ad_count + (int64_t)b * gridDim.y + blockIdx.y;
    if (threadIdx.x == 0) *s_last = atomicAdd(count, 1u) == (unsigned)ns - 1;
    __syncthreads();
    if (!*s_last) return;
    __threadfence();
    if (threadIdx.x == 0) *count = 0;
    float* s_w = &s_o[0][0][0];                               // [G][ns] weights, then the row sums
    for (int hh = warp; hh < G; hh += AD_WARPS) {
        const float* p = a.part + ((int64_t)b * a.H + h0 + hh) * a.splits * REC;
        float mv[AD_MAX_SPLITS / 32], lv[AD_MAX_SPLITS / 32], mm = -INFINITY, ll = 0.0f;
#pragma unroll
        for (int i = 0; i < AD_MAX_SPLITS / 32; ++i) {
            const int s = 32 * i + lane;
            mv[i] = s < ns ? __ldcg(p + (int64_t)s * REC + HD) : -INFINITY;
            lv[i] = s < ns ? __ldcg(p + (int64_t)s * REC + HD + 1) : 0.0f;
            mm = fmaxf(mm, mv[i]);
        }
        mm = warp_max(mm);
#pragma unroll
        for (int i = 0; i < AD_MAX_SPLITS / 32; ++i) {
            const float f = mv[i] == -INFINITY ? 0.0f : expf(mv[i] - mm);
            ll += lv[i] * f;
            if (32 * i + lane < ns) s_w[hh * AD_MAX_SPLITS + 32 * i + lane] = f;
        }
        ll = warp_sum(ll);
        if (lane == 0) s_ml[0][hh][0] = ll;
    }
    __syncthreads();
    constexpr int COLS = HD / 4, LANES = AD_WARPS * 32 / COLS;          // threads per head row, splits added side by side
    float4* s_acc = reinterpret_cast<float4*>(s_q);
    const int col = threadIdx.x % COLS, sl = threadIdx.x / COLS;
    for (int hh = 0; hh < G; ++hh) {
        const float* p = a.part + ((int64_t)b * a.H + h0 + hh) * a.splits * REC + 4 * col;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int s = sl; s < ns; s += LANES) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(p + (int64_t)s * REC));
            const float f = s_w[hh * AD_MAX_SPLITS + s];
            acc.x += v.x * f; acc.y += v.y * f; acc.z += v.z * f; acc.w += v.w * f;
        }
        s_acc[threadIdx.x] = acc;
        __syncthreads();
        if (sl == 0) {
            for (int k = 1; k < LANES; ++k) {
                const float4 v = s_acc[k * COLS + col];
                acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
            }
            *reinterpret_cast<float4*>(a.out + ((int64_t)b * a.H + h0 + hh) * HD + 4 * col) = ad_over(acc, s_ml[0][hh][0]);
        }
        __syncthreads();
    }
}

bool attention_decode_mma_takes(const DecodeMmaArgs& a) {
    auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    return (a.hd == 64 || a.hd == 128) && aligned(a.kc) && aligned(a.vc) && aligned(a.out) && aligned(a.q);
}

template <int HD, bool PAGED, bool FOUR>
static int launch_ad(dim3 grid, dim3 block, const DecodeMmaArgs& c) {
    auto kern = attn_decode_mma_kernel<HD, PAGED, FOUR>;
    static bool configured = false;
    if (!configured) {
        int rc = allow_smem(kern);
        if (rc) return rc;
        configured = true;
    }
    return launch_pdl(kern, grid, block, AdSmem<HD>::BYTES, c);
}

// fixed_part: the pieces' results go there (fixed_floats of room), else to the workspace.
int attention_decode_mma(DecodeMmaArgs a, int batch, int max_len, float* fixed_part, int64_t fixed_floats) {
    const int rows = a.KV * ceil_div(a.group, AD_HEADS);
    // About eight rounds of blocks over the SMs: enough pieces that a ragged batch ends evenly and a
    // lone sequence still covers the chip, none shorter than one step of the four warps.
    const int64_t want = ceil_div64((int64_t)8 * 2 * num_sms(), (int64_t)rows * batch);
    a.splits = (int)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(want, AD_MAX_SPLITS), ceil_div(std::max(max_len, 1), AD_STEP)));
    const int64_t rec = (int64_t)a.H * (a.hd + 4);
    if (fixed_part) {
        a.splits = (int)std::max<int64_t>(1, std::min<int64_t>(a.splits, fixed_floats / (batch * rec)));
        a.part = fixed_part;
    } else if (a.splits > 1) {
        void* wsp;
        int rc = workspace(WS_ATTN).ensure((size_t)batch * rec * a.splits * sizeof(float), &wsp);
        if (rc) return rc;
        a.part = static_cast<float*>(wsp);
    }
    // one launch, unless the batch has more (sequence, KV head) pairs than there are counters
    const int per = std::max(1, std::min(65535, AD_MAX_COUNTERS / rows));
    for (int b0 = 0; b0 < batch; b0 += per) {
        const int nb = std::min(per, batch - b0);
        DecodeMmaArgs c = a;
        c.q += (int64_t)b0 * a.H * a.hd;
        c.out += (int64_t)b0 * a.H * a.hd;
        if (a.page_table) c.page_table += (int64_t)b0 * a.max_pages;
        if (a.seq_lens) c.seq_lens += b0;
        if (a.splits > 1) c.part += (int64_t)b0 * rec * a.splits;
        const dim3 grid(a.splits, rows, nb), block(AD_WARPS * 32);
        const bool paged = a.page_table != nullptr;
        auto go = [&](auto hd, auto four) {
            return paged ? launch_ad<hd.value, true, four.value>(grid, block, c) : launch_ad<hd.value, false, four.value>(grid, block, c);
        };
        using Yes = std::true_type;
        using No = std::false_type;
        using H64 = std::integral_constant<int, 64>;
        using H128 = std::integral_constant<int, 128>;
        const int rc = a.hd == 64 ? (a.group <= 4 ? go(H64{}, Yes{}) : go(H64{}, No{})) : (a.group <= 4 ? go(H128{}, Yes{}) : go(H128{}, No{}));
        if (rc) return rc;
    }
    return B200_OK;
}

}  // namespace b200
