// The few-token dot engine for packed weights: integer tensor-core products of the weights' own
// integers with the activations cut into base-256 digits.
//
// What bounded the engine before it (mma_tile.cuh on fp16 pairs): instructions.  Turning nibbles into
// fp16, decoding the 6-bit scales to floats and spreading them with eight shuffles took 137 instructions
// per 1024 Q4_K weights, 215 in the kernels, on SMs that have about 1500 issue slots for the 1024 * 78
// weights HBM can deliver in a microsecond.  Here a nibble word needs one AND to become an operand:
//     x = 2^(e - 30) * sum_j 256^j D_j,   |x| < 2^e,  D_j signed bytes, j = 0 .. 3
// with e the exponent of the largest of the token's 256 activations (so no activation loses more than
// 2^-31 of that maximum; the fp16 pairs kept 22 bits of each; a NaN or an infinity among the 256 makes their
// scale, and so the token's outputs, NaN), and for every 32-weight sub-block one
// mma.m16n8k32 gives sum_k 16 (q_k - 8) D_jk exactly, the eight columns being the four digits of two tokens.
// The 6-bit scale of the sub-block multiplies the integer (exact: at most 63 * 32 * 128 * 128 * 8 = 2^28), so a
// super-block ends in one conversion and one multiply-add per digit.  What the centred integers leave of a
// sub-block, (8 d s - dmin m) times the sum of its activations, is small beside the products and added in fp32.
// (With q itself the products and the minimum terms are each two to three times their difference, and the last
// bits of both showed: 3e-7 .. 5e-7 of the output's norm against 64 bits, 1e-7 .. 2e-7 so.)
// About 40 instructions per 1024 weights for one or two tokens, 85 for eight.
#pragma once

#include "fused_common.cuh"

namespace b200 {

// Warps of a CTA: two CTAs of consecutive kernels share an SM, so twelve warps leave 80 registers, which one
// and two tokens fit; more tokens need the accumulators of eight warps at 128.
__host__ __device__ constexpr int dg_warps(int MT) { return MT <= 2 ? 12 : 8; }
// Token columns of the instance that takes M tokens.
inline int dg_tokens(int M) { return M <= 2 ? M : M <= 4 ? 4 : 8; }
constexpr int DG_CHUNK = 256;                 // activations that share a scale
// Chunks that a warp loads together before it stages them: the activations come from L2, and one after the other five tokens
// of 1536 were four such ways for each warp.  A batch's places past the last chunk load nothing: repeating the last chunk
// there had every CTA's idle loads meet in one line of L2 (768 -> 3224 at three tokens 11.3 us a call in a row, 5.8 without;
// 1536 -> 6448 9.6 and 5.7; a step of three sequences of a model 768 wide 335 and 265).
__host__ __device__ constexpr int dg_batch(int MT) { return MT == 1 ? 1 : MT == 2 ? 2 : 4; }
// a / b for 0 <= a < 4096, 1 <= b < 256, inv = dg_inv(b): no division on the kernels' serial path
__host__ __device__ constexpr uint32_t dg_inv(int b) { return ((1u << 20) + (uint32_t)b - 1) / (uint32_t)b; }
__host__ __device__ __forceinline__ int dg_div(int a, uint32_t inv) { return (int)(((uint32_t)a * inv) >> 20); }

template <int KIND>
struct DgKind {
    static constexpr bool offset = KIND == 3 || KIND == 1;       // the centred weights have an offset per 32
    // Q4_0 and Q4_1 pair element j with j + 16 of a block in one byte: their operand words are those of
    // elements 4t and 16 + 4t; the other kinds use 8t and 8t + 4.
    static constexpr bool split16 = KIND == 0 || KIND == 1;
};

__host__ __device__ inline int dg_chunks(int K) { return (K + DG_CHUNK - 1) / DG_CHUNK; }
// Staged activations of a chunk and token: four digit bytes each, the sub-block sums and the
// scale; for fp16 weights the three fp16 parts of each (all 24 bits), in columns of their own.
constexpr int DG_COL = DG_CHUNK * 2 + 64;     // bytes of an fp16 column: two neighbours fall into different halves of the banks
template <int KIND>
__host__ __device__ constexpr int dg_chunk_bytes() { return (KIND == KIND_F16 ? 3 * DG_COL : DG_CHUNK * 4 + 32) + 4; }
template <int KIND>
__host__ __device__ inline size_t dg_x_bytes(int chunks, int tokens) { return (size_t)chunks * tokens * dg_chunk_bytes<KIND>() + 16; }

int dg_parts(int tiles, int chunks, int warps);      // decode_gemv.cu

#ifdef __CUDACC__
// Packed weights: digits [sub-block][token][slot][32 bytes], slot = (digit + sub-block) & 3 (so that the stores
// of a warp spread over the banks); sub-block sums times the scale [chunk][token][8]; scales [chunk][token].
// fp16 weights: columns [chunk][part][token][DG_COL bytes]; scales.
template <int KIND, int MT>
struct DgX {
    uint32_t dig, sum, scale;                 // shared addresses
    __device__ __forceinline__ uint8_t* carve(uint8_t* p, int chunks) {
        dig = smem_u32(p);
        sum = dig + chunks * MT * (KIND == KIND_F16 ? 3 * DG_COL : DG_CHUNK * 4);
        scale = sum + (KIND == KIND_F16 ? 0 : chunks * MT * 32);
        return p + dg_x_bytes<KIND>(chunks, MT);
    }
};

__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ float lds_f32(uint32_t a) { return __uint_as_float(lds_u32(a)); }
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts_u32(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts_u2(uint32_t a, uint32_t x, uint32_t y) {
    asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void dg_mma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y), "r"(0));
}

// The scale of a chunk of packed weights is 2^(e - DG_UNIT) and dg_value puts 2^DG_UNIT back on the finished sum: the
// products and the offsets, and the digits, each up to 2^10 of its share of the output, do not overflow where the output
// does not; 2^-90 2^-24 leaves room for a weight's scale above.
constexpr int DG_UNIT = 24;

// Lane l's eight activations 256 * chunk + 8 l .. of token m (zeros past K), staged by one whole warp.
// mul: a factor of the token's contribution, folded into the scale (a mixture weight).
template <int KIND, int MT>
__device__ __forceinline__ void dg_stage(const DgX<KIND, MT>& xd, int chunk, int m, const float (&v)[8], float mul, int lane) {
    uint32_t bits = 0;                                                // of the largest magnitude: a NaN counts as one
#pragma unroll
    for (int i = 0; i < 8; ++i) bits = max(bits, __float_as_uint(v[i]) & 0x7FFFFFFFu);
    bits = __reduce_max_sync(0xffffffffu, bits);
    const int e = min(max((int)(bits >> 23) - 126, -90), 128);        // every finite |v| < 2^e
    // fp16 parts are kept at up to 2^10
    float unit = __uint_as_float((uint32_t)(127 + e - (KIND == KIND_F16 ? 10 : DG_UNIT)) << 23) * mul;
    if (bits >= 0x7F800000u) unit = __uint_as_float(0x7FFFFFFFu);
    if (lane == 0) sts_u32(xd.scale + (chunk * MT + m) * 4, __float_as_uint(unit));
    if (KIND == KIND_F16) {
        const float up = __uint_as_float((uint32_t)(127 + 10 - e) << 23);
        uint32_t p[3][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float2 r = make_float2(v[2 * i] * up, v[2 * i + 1] * up);
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const __half2 h = __floats2half2_rn(r.x, r.y);
                const float2 f = __half22float2(h);
                p[j][i] = *reinterpret_cast<const uint32_t*>(&h);
                r = make_float2(r.x - f.x, r.y - f.y);
            }
        }
        const uint32_t at = xd.dig + (chunk * 3 * MT + m) * DG_COL + 16 * lane;
#pragma unroll
        for (int j = 0; j < 3; ++j)
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(at + j * MT * DG_COL), "r"(p[j][0]), "r"(p[j][1]), "r"(p[j][2]), "r"(p[j][3])
                         : "memory");
        return;
    }
    const float to_int = __uint_as_float((uint32_t)(127 + 30 - e) << 23), down = to_int * 0x1p-30f;
    uint32_t w[2][4];
    float sum = 0.0f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t d[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            // the three low bytes become signed by carrying their top bit into the next digit
            d[i] = ((uint32_t)__float2int_rn(v[4 * h + i] * to_int) + 0x00808080u) ^ 0x00808080u;
            sum += v[4 * h + i] * down;
        }
        const uint32_t p0 = __byte_perm(d[0], d[1], 0x5140), p1 = __byte_perm(d[2], d[3], 0x5140);      // bytes 0, 1 of each
        const uint32_t p2 = __byte_perm(d[0], d[1], 0x7362), p3 = __byte_perm(d[2], d[3], 0x7362);      // bytes 2, 3
        w[h][0] = __byte_perm(p0, p1, 0x5410);
        w[h][1] = __byte_perm(p0, p1, 0x7632);
        w[h][2] = __byte_perm(p2, p3, 0x5410);
        w[h][3] = __byte_perm(p2, p3, 0x7632);
    }
    const int sub = 8 * chunk + (lane >> 2), l4 = lane & 3;
    const uint32_t at = xd.dig + (sub * MT + m) * 128;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t a = at + ((j + sub) & 3) * 32;
        if (DgKind<KIND>::split16) {
            const int p = l4 < 2 ? 4 * l4 : 4 * (l4 - 2) + 1;         // words 2 l4, 2 l4 + 1 go to pair positions
            sts_u32(a + 4 * p, w[0][j]);
            sts_u32(a + 4 * p + 8, w[1][j]);
        } else {
            sts_u2(a + 8 * l4, w[0][j], w[1][j]);
        }
    }
    if (DgKind<KIND>::offset) {
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if (l4 == 0) sts_u32(xd.sum + (chunk * MT + m) * 32 + (lane >> 2) * 4, __float_as_uint(sum * unit));
    }
}

// Bytes of a chunk of a row.
template <int KIND>
__host__ __device__ constexpr int dg_row_chunk() { return KIND == KIND_F16 ? DG_CHUNK * 2 : DG_CHUNK / q_block_elems(KIND) * q_block_bytes(KIND); }

// Loads for dg_stage; x 16-byte aligned.
// CG: from L2.
template <bool CG>
__device__ __forceinline__ void dg_load8(const float* x, int k, int K, float (&v)[8]) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (k < K) {                                                      // K % 32 == 0: a lane has all eight or none
        a = ld_f4<CG>(x + k);
        b = ld_f4<CG>(x + k + 4);
    }
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// The same of a norm's weights, which the caller may have put at any address.
__device__ __forceinline__ float4 dg_norm4(const float* w) {
    if ((reinterpret_cast<uintptr_t>(w) & 15) == 0) return *reinterpret_cast<const float4*>(w);
    return make_float4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void dg_norm8(const float* w, int k, int K, float (&v)[8]) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (k < K) {
        a = dg_norm4(w + k);
        b = dg_norm4(w + k + 4);
    }
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// One warp's accumulators for a 16-row tile.  Packed: f[q] the digit columns of tokens 2 q, 2 q + 1 (lane
// (g, t): rows g, g + 8; token 2 q + t / 2, digits 2 (t & 1), + 1), off the offsets of this lane's sub-blocks
// (rows g, g + 8; each token).  fp16: the operand's eight columns are Wd
// = 2, 4 or 8 tokens of 4, 2 or 1 parts; f[q] columns 2 t, 2 t + 1 (rows g, g + 8).
template <int KIND, int MT>
struct DgAcc {
    static constexpr int Wd = MT <= 2 ? 2 : MT;
    static constexpr int NT = KIND == KIND_F16 ? (3 * Wd + 7) / 8 : (MT <= 2 ? 1 : MT / 2);
    static constexpr int NO = DgKind<KIND>::offset ? MT : 1;
    float f[NT][4], off[2][NO];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int q = 0; q < NT; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) f[q][i] = 0.0f;
#pragma unroll
        for (int i = 0; i < NO; ++i) off[0][i] = off[1][i] = 0.0f;
    }
};

// Adds one chunk of 256 weights of 16 rows.  row_a / row_b: shared addresses of the chunk in this lane's
// rows g and g + 8; xc: the chunk's index among the staged activations; nb: its 32-weight blocks (8, fewer
// in a tail of kinds 0 .. 2).
template <int KIND, int MT>
__device__ __forceinline__ void dg_chunk(DgAcc<KIND, MT>& acc, uint32_t row_a, uint32_t row_b, const DgX<KIND, MT>& xd, int xc, int nb, int lane) {
    constexpr int NT = DgAcc<KIND, MT>::NT;
    const int g = lane >> 2, t = lane & 3, dgt = g & 3;
    if (KIND == KIND_F16) {
        constexpr int Wd = DgAcc<KIND, MT>::Wd;
        // a column past the third part repeats it (dg_finish leaves it out), one past the tokens repeats the last token
        uint32_t col[NT];
        float sum[NT][4];
#pragma unroll
        for (int q = 0; q < NT; ++q) {
            col[q] = xd.dig + ((xc * 3 + min((8 * q + g) / Wd, 2)) * MT + min(g % Wd, MT - 1)) * DG_COL + 16 * t;
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[q][i] = 0.0f;
        }
        // The tensor cores cut a sum's last bits off where an addition rounds them: 32 of K at a time.
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            if (s >= nb) break;
            const uint4 a = lds_u4(row_a + 64 * s + 16 * t), b = lds_u4(row_b + 64 * s + 16 * t);
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                float c[4] = {0.f, 0.f, 0.f, 0.f};
                const uint4 x = lds_u4(col[q] + 64 * s);
                mma_16816(c, a.x, b.x, a.y, b.y, x.x, x.y);
                mma_16816(c, a.z, b.z, a.w, b.w, x.z, x.w);
#pragma unroll
                for (int i = 0; i < 4; ++i) sum[q][i] += c[i];
            }
        }
        const uint32_t xs = xd.scale + xc * MT * 4;
        const float x0 = lds_f32(xs + min(2 * t % Wd, MT - 1) * 4), x1 = lds_f32(xs + min(2 * t % Wd + 1, MT - 1) * 4);
#pragma unroll
        for (int q = 0; q < NT; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc.f[q][i] += (i & 1 ? x1 : x0) * sum[q][i];
        return;
    }
    const uint32_t xb = xd.dig + xc * 8 * MT * 128 + 8 * t + (MT == 1 ? 0 : (g >> 2) * 128);
    uint32_t xo[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) xo[s] = xb + ((dgt + s) & 3) * 32;
    float xs[NT];
#pragma unroll
    for (int q = 0; q < NT; ++q) xs[q] = lds_f32(xd.scale + (xc * MT + (MT == 1 ? 0 : 2 * q + (t >> 1))) * 4);
    auto bfrag = [&](int s, int q) { return lds_u2(xo[s & 3] + (s * MT + 2 * q) * 128); };
    float oa[2] = {0.f, 0.f}, ob[2] = {0.f, 0.f};                      // offsets of sub-blocks 2 t, 2 t + 1 in the two rows
    float da, db;
    if (KIND == 3) {
        const uint4 ha = lds_u4(row_a), hb = lds_u4(row_b);
        const float2 fa = __half22float2(*reinterpret_cast<const __half2*>(&ha.x)), fb = __half22float2(*reinterpret_cast<const __half2*>(&hb.x));
        da = fa.x; db = fb.x;
        const uint32_t sca[2] = {ha.y & 0x3F3F3F3Fu, (ha.w & 0x0F0F0F0Fu) | ((ha.y >> 2) & 0x30303030u)};
        const uint32_t scb[2] = {hb.y & 0x3F3F3F3Fu, (hb.w & 0x0F0F0F0Fu) | ((hb.y >> 2) & 0x30303030u)};
        const uint32_t mna = t < 2 ? ha.z & 0x3F3F3F3Fu : ((ha.w >> 4) & 0x0F0F0F0Fu) | ((ha.z >> 2) & 0x30303030u);
        const uint32_t mnb = t < 2 ? hb.z & 0x3F3F3F3Fu : ((hb.w >> 4) & 0x0F0F0F0Fu) | ((hb.z >> 2) & 0x30303030u);
        // 8 d s - dmin m, both products exact
        auto offsets = [&](uint32_t sc, uint32_t mn, float2 f, float (&o)[2]) {
            const int sh = 16 * (t & 1);
            sc >>= sh;
            mn >>= sh;
            const float d8 = 8.0f * f.x;
            o[0] = __fsub_rn(d8 * (float)(sc & 0xFF), f.y * (float)(mn & 0xFF));
            o[1] = __fsub_rn(d8 * (float)((sc >> 8) & 0xFF), f.y * (float)((mn >> 8) & 0xFF));
        };
        offsets(t < 2 ? sca[0] : sca[1], mna, fa, oa);
        offsets(t < 2 ? scb[0] : scb[1], mnb, fb, ob);
        int v[NT][4];
#pragma unroll
        for (int q = 0; q < NT; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) v[q][i] = 0;
        auto high = [](uint32_t w) { return (w & 0xF0F0F0F0u) ^ 0x80808080u; };      // 16 (q - 8) as signed bytes
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint2 wa = lds_u2(row_a + 16 + 32 * j + 8 * t), wb = lds_u2(row_b + 16 + 32 * j + 8 * t);
            const int sa0 = (sca[j >> 1] >> (16 * (j & 1))) & 0xFF, sa1 = (sca[j >> 1] >> (16 * (j & 1) + 8)) & 0xFF;
            const int sb0 = (scb[j >> 1] >> (16 * (j & 1))) & 0xFF, sb1 = (scb[j >> 1] >> (16 * (j & 1) + 8)) & 0xFF;
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                int c[4];
                dg_mma(c, high(wa.x << 4), high(wb.x << 4), high(wa.y << 4), high(wb.y << 4), bfrag(2 * j, q));
                v[q][0] += sa0 * c[0]; v[q][1] += sa0 * c[1]; v[q][2] += sb0 * c[2]; v[q][3] += sb0 * c[3];
                dg_mma(c, high(wa.x), high(wb.x), high(wa.y), high(wb.y), bfrag(2 * j + 1, q));
                v[q][0] += sa1 * c[0]; v[q][1] += sa1 * c[1]; v[q][2] += sb1 * c[2]; v[q][3] += sb1 * c[3];
            }
        }
#pragma unroll
        for (int q = 0; q < NT; ++q) {
            const float ea = da * xs[q], eb = db * xs[q];
            acc.f[q][0] += ea * (float)v[q][0];
            acc.f[q][1] += ea * (float)v[q][1];
            acc.f[q][2] += eb * (float)v[q][2];
            acc.f[q][3] += eb * (float)v[q][3];
        }
    } else {
        constexpr int BB = q_block_bytes(KIND);
        if (KIND == 1) {
            // m + 8 d of blocks 2 t, 2 t + 1 (zero past the row's end: their sums are zero, but the bits may be anything)
            auto offset = [&](uint32_t row, int s) {
                const uint32_t dm = s < nb ? lds_u32(row + s * BB) : 0u;
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&dm));
                return fmaf(8.0f, f.x, f.y);
            };
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                oa[i] = offset(row_a, 2 * t + i);
                ob[i] = offset(row_b, 2 * t + i);
            }
        }
        // bytes [a, a + 4) at any even address
        auto word = [&](uint32_t a) { return __funnelshift_r(lds_u32(a & ~3u), lds_u32((a & ~3u) + 4), (a & 2) * 8); };
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            if (s >= nb) break;
            uint32_t a0, a1, a2, a3;
            const uint32_t ra = row_a + s * BB, rb = row_b + s * BB;
            if (KIND == 2) {
                auto two = [&](uint32_t a, uint32_t& x, uint32_t& y) {
                    const uint32_t base = a & ~3u, sh = (a & 2) * 8;
                    const uint32_t w0 = lds_u32(base), w1 = lds_u32(base + 4), w2 = lds_u32(base + 8);
                    x = __funnelshift_r(w0, w1, sh);
                    y = __funnelshift_r(w1, w2, sh);
                };
                two(ra + 2 + 8 * t, a0, a2);
                two(rb + 2 + 8 * t, a1, a3);
            } else {
                // 16 (q - 8) as signed bytes
                const uint32_t wa = (KIND == 0 ? word(ra + 2 + 4 * t) : lds_u32(ra + 4 + 4 * t)) ^ 0x88888888u;
                const uint32_t wb = (KIND == 0 ? word(rb + 2 + 4 * t) : lds_u32(rb + 4 + 4 * t)) ^ 0x88888888u;
                a0 = (wa << 4) & 0xF0F0F0F0u; a1 = (wb << 4) & 0xF0F0F0F0u;
                a2 = wa & 0xF0F0F0F0u; a3 = wb & 0xF0F0F0F0u;
            }
            da = half_bits_to_float((uint16_t)lds_u16(ra));
            db = half_bits_to_float((uint16_t)lds_u16(rb));
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                int c[4];
                dg_mma(c, a0, a1, a2, a3, bfrag(s, q));
                const float ea = da * xs[q], eb = db * xs[q];
                acc.f[q][0] += ea * (float)c[0]; acc.f[q][1] += ea * (float)c[1];
                acc.f[q][2] += eb * (float)c[2]; acc.f[q][3] += eb * (float)c[3];
            }
        }
    }
    if (DgKind<KIND>::offset) {
        const uint32_t at = xd.sum + xc * MT * 32 + 8 * t;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const uint2 u = lds_u2(at + m * 32);
            const float s0 = __uint_as_float(u.x), s1 = __uint_as_float(u.y);
            acc.off[0][m] = fmaf(oa[1], s1, fmaf(oa[0], s0, acc.off[0][m]));
            acc.off[1][m] = fmaf(ob[1], s1, fmaf(ob[0], s0, acc.off[1][m]));
        }
    }
}

// The warp's sums to red[16 rows][MT] (packed weights: in units of 2^DG_UNIT).
constexpr int dg_red_floats(int MT) { return 16 * MT; }
template <int KIND, int MT>
__device__ __forceinline__ void dg_finish(const DgAcc<KIND, MT>& acc, float* red, int lane) {
    const int g = lane >> 2, t = lane & 3;
    if constexpr (KIND == KIND_F16) {
        constexpr int Wd = DgAcc<KIND, MT>::Wd;
        float v[4];                           // tokens 2 t % Wd, + 1; rows g, g + 8
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if constexpr (Wd == 8) {
                v[i] = acc.f[0][i] + (acc.f[1][i] + acc.f[2][i]);
            } else if constexpr (Wd == 4) {   // f[0]: high parts in lanes 0, 1, middle ones in 2, 3; f[1]: low ones in 0, 1
                v[i] = acc.f[0][i] + (t < 2 ? acc.f[1][i] : 0.0f);
                v[i] += __shfl_xor_sync(0xffffffffu, v[i], 2);
            } else {                          // lane t: part t
                v[i] = t < 3 ? acc.f[0][i] : 0.0f;
                v[i] += __shfl_xor_sync(0xffffffffu, v[i], 2);
                v[i] += __shfl_xor_sync(0xffffffffu, v[i], 1);
            }
        }
        if (2 * t < Wd) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (2 * t + i < MT) {
                    red[g * MT + 2 * t + i] = v[i];
                    red[(g + 8) * MT + 2 * t + i] = v[2 + i];
                }
        }
        return;
    }
    const float scale = ((t & 1) ? 65536.0f : 1.0f) * (KIND == 2 ? 0x1p-30f : 0x1p-34f);
#pragma unroll
    for (int q = 0; q < DgAcc<KIND, MT>::NT; ++q) {
        float v[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            v[r] = (acc.f[q][2 * r] + 256.0f * acc.f[q][2 * r + 1]) * scale;
            if (DgKind<KIND>::offset) {
                // the four lanes of a row hold the offsets of two sub-blocks each for every token: lanes 0, 1 take the first
                // token of the pair from lanes 2, 3, which take the second
                const float o0 = acc.off[r][2 * q], o1 = acc.off[r][MT == 1 ? 0 : 2 * q + 1];
                v[r] += (t < 2 ? o0 : o1) + __shfl_xor_sync(0xffffffffu, t < 2 ? o1 : o0, 2);
            }
            v[r] += __shfl_xor_sync(0xffffffffu, v[r], 1);
        }
        const int tok = 2 * q + (t >> 1);
        if ((t & 1) == 0 && tok < MT) {
            red[g * MT + tok] = v[0];
            red[(g + 8) * MT + tok] = v[1];
        }
    }
}
// Element (row, token) from `parts` warps' results, each dg_red_floats apart.
template <int KIND, int MT>
__device__ __forceinline__ float dg_value(const float* red, int parts, int row, int tok) {
    const float* at = red + row * MT + tok;
    float v = 0.0f;
#pragma unroll 4
    for (int p = 0; p < parts; ++p, at += dg_red_floats(MT)) v += *at;
    return KIND == KIND_F16 ? v : v * (float)(1 << DG_UNIT);
}
#endif

}  // namespace b200
