// The routed Q4_K experts of a decode batch on tcgen05, exact to fp32: every expert's weights are expanded once
// for all the tokens that chose it.
//
// A Q4_K weight is d s (q - 8) + (8 d s - dmin m) with |s (q - 8)| <= 504, an integer that fp16 holds exactly; d and
// dmin are constant over 256 of K, s and m over 32.  So the tensor cores multiply the integers (expanded in registers,
// first operand in tensor memory, as in gemm_wt.cu), one accumulation per 256 of K, and the epilogue multiplies it by
// the row's d and adds the eight offsets times the sums of the activations.  (With s q and the minima alone the two terms
// cancel, and the tensor cores, which cut the last bits off a sum, show: 6e-7 .. 1.2e-6 of the output's norm against 64 bits,
// 2.6e-7 so.)  An activation is three fp16 columns,
// x = 2^e (a + 2^-11 b + 2^-22 c) with 2^e from the maximum of its 256 (33 bits below it), which the epilogue adds up:
// a tile of up to 24 slots of one expert is 72 columns.
// Everything moves in steps of 256 of K (per 64, as gemm_wt.cu does, the roles' waits took 4300 cycles per 256).
//   warp 0        activation columns by TMA
//   warp 2        packed rows by TMA
//   warp 1        MMA issue
//   warps 4..7, 24..27   epilogue: a lane holds one weight row, its sums of up to 12 slots in registers
//   warps 8..23   expansion: four groups of four warps, 64 of the 256 each, into one of two operands
// The SwiGLU form puts 64 gate rows and the same 64 up rows in one tile.  All waits are bounded (gemm_umma.cu).
//
// Bound by instructions issued (63 % of the slots: the expansion, the epilogue's sums) and the waits between the roles,
// 1930 cycles per 128 rows x 256 of K, 2.2 times what the bytes alone take.  Tried without effect: a third accumulator,
// packed rows by 16-byte asynchronous copies instead of TMA, deeper rings.
// 64 tokens, H-Tiny: gate / up 47 us and down 58 on the digit engine (moe_units.cu), 38 and 22 here; 48 tokens, H-Small:
// the layer 450 us before, 237 now.
#include <algorithm>

#include "gemm.cuh"
#include "linear.cuh"
#include "umma_ts.cuh"

namespace b200 {

int splitk_reduce(const float* part, float* c, int splits, int64_t stride, int M, int N, int64_t ldc);
int make_packed_map(CUtensorMap* out, const void* base, int64_t rows, int64_t row_bytes, int box_bytes, int box_rows);

constexpr int WX_CAP = 24;                    // slots of a tile
constexpr int WX_ROWS = 128;                  // weight rows of a tile
constexpr int WX_SBB = 144;                   // bytes of 256 weights
constexpr int WX_PACKED = WX_ROWS * WX_SBB;
constexpr int WX_BOX = 24;                    // rows of a TMA box of activation columns: eight slots
constexpr int WX_X_SUB = 3 * WX_CAP * 128;    // 64 of K
constexpr int WX_X_STAGE = 4 * WX_X_SUB;      // 256 of K
constexpr int WX_SX = 2, WX_SP = 5;
constexpr int WX_HDR = 4;                     // ring of eight offsets and d per weight row, from the expansion to the epilogue
constexpr int WX_AUX = 12;                    // floats per slot and 256 of K: 2^e, -, -, -, eight sub-block sums in units of 2^e
constexpr int WX_SET = 128;                   // tensor-memory columns between the two accumulators, between the two operands
constexpr int WX_OPERAND = 2 * WX_SET;
constexpr int WX_FIRST_EXPAND = 8, WX_EXPAND_WARPS = 16;
constexpr int WX_SECOND_EPI = WX_FIRST_EXPAND + WX_EXPAND_WARPS;
constexpr int WX_THREADS = (WX_SECOND_EPI + 4) * 32;
constexpr int WX_HALF = WX_CAP / 2;           // slots of an epilogue group
constexpr int WX_MAX_EXPERTS = 256, WX_TABLE = 64;
constexpr int WX_SWAP = 2 * WX_CAP * WX_ROWS * 4;     // SwiGLU: gate and up rows of a tile, double buffered
constexpr int WX_SMEM = 1024 + WX_SX * WX_X_STAGE + WX_SP * WX_PACKED + WX_SWAP + 8 * WX_HALF * WX_AUX * 4 + WX_HDR * WX_ROWS * 36 + 512 +
                        (WX_MAX_EXPERTS + 4) * 4 + WX_TABLE * 16;
static_assert(WX_SMEM <= 227 * 1024, "the stages do not fit the shared memory of an SM");

struct alignas(64) WxArgs {
    CUtensorMap map_x, map_w, map_w2;
    const int32_t* offsets;                   // device [ne + 1]: sorted slots of each expert; null: one of M rows
    const float* aux;                         // [NK, K / 256, WX_AUX]
    float* c;                                 // [NK, N]
    int ne, M, N, K, n_tiles;
    int k_splits, per_split;                  // ranges of K (in units of 256) whose partial sums are added afterwards
    int64_t split_stride;
    int* status;
};

// ---- activations to three fp16 columns: one warp per (slot, 256 of K) ------------
__global__ void __launch_bounds__(256)
wx_split_kernel(const float* __restrict__ x, const int32_t* __restrict__ grouped, int top_k, int NK, int K,
                __half* __restrict__ out, float* __restrict__ aux) {
    const int chunks = K >> 8, lane = threadIdx.x & 31;
    pdl_launch_dependents();                  // the products' kernel sets up and fetches its first weights meanwhile
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), slot = i / chunks, c = i - slot * chunks;
    if (slot >= NK) return;
    const float* row = x + (int64_t)(grouped ? grouped[slot] / top_k : slot) * K + 256 * c + 8 * lane;
    float v[8];
    const float4 lo4 = *reinterpret_cast<const float4*>(row), hi4 = *reinterpret_cast<const float4*>(row + 4);
    v[0] = lo4.x; v[1] = lo4.y; v[2] = lo4.z; v[3] = lo4.w;
    v[4] = hi4.x; v[5] = hi4.y; v[6] = hi4.z; v[7] = hi4.w;
    float mx = 0.0f, sum = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) mx = fmaxf(mx, fabsf(v[k]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const int e = min(max((__float_as_int(mx) >> 23) - 127, -126), 126);
    const float s = __int_as_float((e + 127) << 23), inv = __int_as_float((127 - e) << 23);
    __half p[3][8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float r = v[k] * inv;
        sum += r;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            p[j][k] = __float2half_rn(r);
            r = (r - __half2float(p[j][k])) * 2048.0f;
        }
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);          // of the lane's 32 values
#pragma unroll
    for (int j = 0; j < 3; ++j)
        *reinterpret_cast<uint4*>(out + ((int64_t)slot * 3 + j) * K + 256 * c + 8 * lane) = *reinterpret_cast<const uint4*>(p[j]);
    float* a = aux + ((int64_t)slot * chunks + c) * WX_AUX;
    if (lane == 0) *a = s;
    if ((lane & 3) == 0) a[4 + (lane >> 2)] = sum;
}

// ---- tiles ------------------------------------------------------------------------
struct WxTile {
    int slot0, slots, n0, brow;
    int sb0, sb1;                             // its range of K in units of 256
};
// first[e] = first token tile of expert e; first[ne] = all of them.  All threads.
__device__ __forceinline__ void wx_build(const WxArgs& a, int* first) {
    if (!a.offsets) {
        if (threadIdx.x == 0) {
            first[0] = 0;
            first[1] = (a.M + WX_CAP - 1) / WX_CAP;
        }
        __syncthreads();
        return;
    }
    if (threadIdx.x < 32) {
        int carry = 0;
        for (int e0 = 0; e0 < a.ne; e0 += 32) {
            const int e = e0 + threadIdx.x;
            const int n = e < a.ne ? (a.offsets[e + 1] - a.offsets[e] + WX_CAP - 1) / WX_CAP : 0;
            int incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)threadIdx.x >= o) incl += up;
            }
            if (e < a.ne) first[e] = carry + incl - n;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (threadIdx.x == 0) first[a.ne] = carry;
    }
    __syncthreads();
}
template <bool SPLIT>
__device__ __noinline__ WxTile wx_find(const WxArgs& a, const int* first, int t) {
    WxTile w;
    w.sb0 = 0;
    w.sb1 = a.K >> 8;
    if (SPLIT) {
        w.sb0 = t % a.k_splits * a.per_split;
        w.sb1 = min(w.sb1, w.sb0 + a.per_split);
        t /= a.k_splits;
    }
    const int tile = t / a.n_tiles;
    w.n0 = t - tile * a.n_tiles;
    int l = 0, h = a.ne;                      // the last expert whose first tile is <= tile owns it
    while (h - l > 1) {
        const int mid = (l + h) >> 1;
        if (first[mid] <= tile) l = mid; else h = mid;
    }
    const int lo = a.offsets ? a.offsets[l] : 0, rows = (a.offsets ? a.offsets[l + 1] : a.M) - lo, n = first[l + 1] - first[l], i = tile - first[l];
    const int size = ((rows + n - 1) / n + 7) & ~7;                // equal tiles of whole groups of eight
    w.slot0 = lo + i * size;
    w.slots = max(0, min(size, rows - i * size));
    w.brow = l * a.N;
    return w;
}
template <bool SPLIT>
__device__ __forceinline__ WxTile wx_tile_at(const WxArgs& a, const int* first, const int4* table, int i) {
    if (i >= WX_TABLE) return wx_find<SPLIT>(a, first, blockIdx.x + i * gridDim.x);
    const int4 e = table[i];
    if (!SPLIT) return WxTile{e.x, e.y, e.z, e.w, 0, a.K >> 8};
    const int sb0 = (e.z >> 20) * a.per_split;
    return WxTile{e.x, e.y, e.z & 0xFFFFF, e.w, sb0, min(a.K >> 8, sb0 + a.per_split)};
}

// 64 weights of a row (K step J of its 256) to the integers s (q - 8) as 32 fp16 pairs, exact.
// d: the row's factor; off: 8 d s - dmin m of the two 32.
template <int J>
__device__ __forceinline__ void wx_expand(uint32_t seg, uint32_t (&out)[32], float& d, float2& off) {
    auto vec = [&](int i) {
        uint4 v;
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(seg + 16 * i));
        return v;
    };
    const uint4 hdr = vec(0), q0 = vec(1 + 2 * J), q1 = vec(2 + 2 * J);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hdr.x));
    d = f.x;
    const uint32_t words[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        int s, m;
        q4k_scale_min_regs(2 * J + hh, hdr.y, hdr.z, hdr.w, s, m);
        (hh ? off.y : off.x) = __fsub_rn(8.0f * f.x * (float)s, f.y * (float)m);      // both products exact
        // high nibbles stay where they are, low ones move there: 1024 + 16 q, times s / 16, less 72 s
        const __half2 sc2 = __half2half2(__hmul(__int2half_rn(s), __float2half(0.0625f)));
        const __half2 nsc = __half2half2(__int2half_rn(-72 * s));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t x = (hh ? words[i] : words[i] << 4) & 0xF0F0F0F0u;
            out[16 * hh + 2 * i] = wt_bits(__hfma2(wt_magic(x, WT_SEL_01), sc2, nsc));
            out[16 * hh + 2 * i + 1] = wt_bits(__hfma2(wt_magic(x, WT_SEL_23), sc2, nsc));
        }
    }
}
// 12 consecutive columns of this warp's 32 lanes: four slots.
__device__ __forceinline__ void tmem_ld12(uint32_t at, float (&v)[12]) {
    uint32_t r[12];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%12];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8, %9, %10, %11}, [%13];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]),
          "=&r"(r[10]), "=&r"(r[11])
        : "r"(at), "r"(at + 8)
        : "memory");
#pragma unroll
    for (int i = 0; i < 12; ++i) v[i] = __uint_as_float(r[i]);
}

template <bool SWIGLU, bool SPLIT>
__global__ void __launch_bounds__(WX_THREADS, 1) wx_kernel(const __grid_constant__ WxArgs a) {
    constexpr int TILE_N = SWIGLU ? WX_ROWS / 2 : WX_ROWS;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sm_x = smem;
    uint8_t* sm_p = sm_x + WX_SX * WX_X_STAGE;
    float* swap = reinterpret_cast<float*>(sm_p + WX_SP * WX_PACKED);
    float* sm_aux = swap + WX_SWAP / 4;                                // [8 warps][WX_HALF][WX_AUX]
    float4* sm_off = reinterpret_cast<float4*>(sm_aux + 8 * WX_HALF * WX_AUX);    // [WX_HDR][2][WX_ROWS]
    float* sm_d = reinterpret_cast<float*>(sm_off + WX_HDR * 2 * WX_ROWS);        // [WX_HDR][WX_ROWS]
    uint64_t* x_full = reinterpret_cast<uint64_t*>(sm_d + WX_HDR * WX_ROWS);
    uint64_t* x_empty = x_full + WX_SX;
    uint64_t* p_full = x_empty + WX_SX;
    uint64_t* p_empty = p_full + WX_SP;
    uint64_t* a_full = p_empty + WX_SP;       // [2] the operand is expanded
    uint64_t* done = a_full + 2;              // [2] its products are in the accumulator
    uint64_t* acc_empty = done + 2;           // [2] and have been read
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    int4* table = reinterpret_cast<int4*>(x_full + 64);
    int* first = reinterpret_cast<int*>(table + WX_TABLE);
    const int warp = uniform_warp(), lane = threadIdx.x & 31, chunks = a.K >> 8;
    wx_build(a, first);
    const int total = first[a.ne] * a.n_tiles * (SPLIT ? a.k_splits : 1);
    const int mine = (int)blockIdx.x < total ? (total - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    if (threadIdx.x < WX_TABLE && (int)threadIdx.x < mine) {
        const WxTile w = wx_find<SPLIT>(a, first, blockIdx.x + threadIdx.x * gridDim.x);
        table[threadIdx.x] = make_int4(w.slot0, w.slots, SPLIT ? w.n0 | (w.sb0 / a.per_split) << 20 : w.n0, w.brow);
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < WX_SX; ++s) { mbar_init(&x_full[s], 1); mbar_init(&x_empty[s], 1); }
        for (int s = 0; s < WX_SP; ++s) { mbar_init(&p_full[s], 1); mbar_init(&p_empty[s], WX_EXPAND_WARPS); }
        for (int s = 0; s < 2; ++s) { mbar_init(&a_full[s], WX_EXPAND_WARPS); mbar_init(&done[s], 1); mbar_init(&acc_empty[s], 8); }
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        pdl_wait();                           // the activations come from the kernel before
        uint32_t it = 0, s = 0, ph = 0;
        bool ok = true;
        for (int i = 0; i < mine && ok; ++i) {
            const WxTile w = wx_tile_at<SPLIT>(a, first, table, i);
            const int boxes = (w.slots + 7) / 8;
            for (int sb = w.sb0; sb < w.sb1; ++sb, ++it) {
                if (it >= WX_SX) ok = mbar_wait_warp(&x_empty[s], ph ^ 1, a.status);
                if (!ok) break;
                if (elect_one()) {
                    mbar_expect_tx(&x_full[s], 4 * boxes * WX_BOX * 128);
                    for (int k = 0; k < 4; ++k)
                        for (int b = 0; b < boxes; ++b)
                            tma_load_2d(sm_x + s * WX_X_STAGE + k * WX_X_SUB + b * WX_BOX * 128, &a.map_x, sb * 256 + k * 64,
                                        3 * w.slot0 + b * WX_BOX, &x_full[s]);
                }
                if (++s == WX_SX) { s = 0; ph ^= 1; }
            }
        }
        if (!ok)
            for (uint32_t j = it > WX_SX ? it - WX_SX : 0; j < it; ++j)
                if (!mbar_wait_warp(&x_full[j % WX_SX], (j / WX_SX) & 1, a.status)) break;
    } else if (warp == 2) {
        uint32_t it = 0, p = 0, ph = 0;
        bool ok = true;
        for (int i = 0; i < mine && ok; ++i) {
            const WxTile w = wx_tile_at<SPLIT>(a, first, table, i);
            const int brow = w.brow + w.n0 * TILE_N;
            for (int sb = w.sb0; sb < w.sb1; ++sb, ++it) {
                if (it >= WX_SP) ok = mbar_wait_warp(&p_empty[p], ph ^ 1, a.status);
                if (!ok) break;
                if (elect_one()) {
                    uint8_t* dst = sm_p + p * WX_PACKED;
                    mbar_expect_tx(&p_full[p], WX_PACKED);
                    tma_load_2d(dst, &a.map_w, sb * (WX_SBB / 4), brow, &p_full[p]);
                    if (SWIGLU) tma_load_2d(dst + WX_PACKED / 2, &a.map_w2, sb * (WX_SBB / 4), brow, &p_full[p]);
                }
                if (++p == WX_SP) { p = 0; ph ^= 1; }
            }
        }
        if (!ok)
            for (uint32_t j = it > WX_SP ? it - WX_SP : 0; j < it; ++j)
                if (!mbar_wait_warp(&p_full[j % WX_SP], (j / WX_SP) & 1, a.status)) break;
    } else if (warp == 1) {
        uint32_t ci = 0, s = 0, ph = 0, ready = 0;
        bool ok = true;
        for (int i = 0; i < mine && ok; ++i) {
            const WxTile w = wx_tile_at<SPLIT>(a, first, table, i);
            const uint32_t idesc = umma_idesc_f16(WX_ROWS, ((w.slots + 7) / 8 * WX_BOX + 15) & ~15);
            for (int sb = w.sb0; sb < w.sb1; ++sb, ++ci) {
                const uint32_t as = ci & 1, d = tmem + as * WX_SET, op = tmem + WX_OPERAND + as * WX_SET;
                if (!__all_sync(0xffffffffu, ready != 0))
                    ok = (ci < 2 || mbar_wait_warp(&acc_empty[as], ((ci >> 1) - 1) & 1, a.status)) &&
                         mbar_wait_warp(&x_full[s], ph, a.status) && mbar_wait_warp(&a_full[as], (ci >> 1) & 1, a.status);
                if (!ok) break;
                tc_fence_after();
                const uint64_t desc = umma_smem_desc(smem_u32(sm_x + s * WX_X_STAGE));
                // the next step's barriers are looked at before this one's products are issued: a wait costs a few
                // hundred cycles even when there is nothing to wait for
                const uint32_t sn = s + 1 == WX_SX ? 0 : s + 1, phn = s + 1 == WX_SX ? ph ^ 1 : ph, nx = ci + 1;
                ready = (nx < 2 ? 1u : mbar_peek(&acc_empty[nx & 1], ((nx >> 1) - 1) & 1)) & mbar_peek(&x_full[sn], phn) &
                        mbar_peek(&a_full[nx & 1], (nx >> 1) & 1);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 16; ++k)          // 32 bytes of K per step: 2 in the descriptor's units
                        umma_f16_ts(d, op + k * 8, desc + (k >> 2) * (WX_X_SUB >> 4) + 2 * (k & 3), idesc, k > 0);
                    umma_commit(&x_empty[s]);
                    umma_commit(&done[as]);
                }
                if (++s == WX_SX) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp >= 4 && (warp < WX_FIRST_EXPAND || warp >= WX_SECOND_EPI)) {
        // Two groups of four warps take the fours of slots in turn.  An accumulation has to be read in the time that
        // the next one is expanded: with one group, which also decoded the headers, it took 2300 cycles, and a SwiGLU
        // tile's end, half the rows finishing all slots, 5500.
        const int e = warp >= WX_SECOND_EPI, q = warp & 3, tid = q * 32 + lane;
        float* aux = sm_aux + (4 * e + q) * WX_HALF * WX_AUX;
        auto slot_of = [&](int l) { return 4 * (2 * (l >> 2) + e) + (l & 3); };        // of the group's l-th sum
        uint32_t ci = 0, ti = 0, ready = 0;
        pdl_wait();
        // the next 256's scales and sums travel while this one's are used: a lane fetches one slot's
        float4 nx[3];
        auto source = [&](int i) {
            const WxTile w = wx_tile_at<SPLIT>(a, first, table, i);
            return reinterpret_cast<const float4*>(a.aux + (int64_t)(w.slot0 + min(slot_of(min(lane, WX_HALF - 1)), w.slots - 1)) * chunks * WX_AUX) + w.sb0 * 3;
        };
        const float4* src = mine > 0 ? source(0) : nullptr;
        if (mine > 0)
#pragma unroll
            for (int j = 0; j < 3; ++j) nx[j] = src[j];
        for (int i = 0; i < mine; ++i, ++ti) {
            const WxTile w = wx_tile_at<SPLIT>(a, first, table, i);
            bool ok = true;
            float acc[WX_HALF];
#pragma unroll
            for (int j = 0; j < WX_HALF; ++j) acc[j] = 0.0f;
            for (int sb = w.sb0; sb < w.sb1; ++sb, ++ci) {
                __syncwarp();
                if (lane < WX_HALF)
#pragma unroll
                    for (int j = 0; j < 3; ++j) *reinterpret_cast<float4*>(aux + lane * WX_AUX + 4 * j) = nx[j];
                src += 3;
                if (sb + 1 == w.sb1 && i + 1 < mine) src = source(i + 1);
                if (sb + 1 < w.sb1 || i + 1 < mine)
#pragma unroll
                    for (int j = 0; j < 3; ++j) nx[j] = src[j];
                const uint32_t as = ci & 1;
                if (!__all_sync(0xffffffffu, ready != 0)) ok = mbar_wait_warp(&done[as], (ci >> 1) & 1, a.status);
                if (!ok) break;
                ready = mbar_peek(&done[as ^ 1], ((ci + 1) >> 1) & 1);
                tc_fence_after();
                const float d = sm_d[(ci % WX_HDR) * WX_ROWS + tid];
                const float4 o0 = sm_off[(ci % WX_HDR) * 2 * WX_ROWS + tid], o1 = sm_off[((ci % WX_HDR) * 2 + 1) * WX_ROWS + tid];
                const uint32_t tq = tmem + as * WX_SET + ((uint32_t)(q * 32) << 16);
#pragma unroll
                for (int k = 0; k < WX_HALF / 4; ++k) {
                    if (slot_of(4 * k) < w.slots) {
                        float v[12];
                        tmem_ld12(tq + 12 * (2 * k + e), v);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float4* au = reinterpret_cast<const float4*>(aux + (4 * k + j) * WX_AUX);
                            const float4 s0 = au[1], s1 = au[2];
                            const float t = fmaf(fmaf(v[3 * j + 2], 0x1p-11f, v[3 * j + 1]), 0x1p-11f, v[3 * j]);
                            const float lo = fmaf(o0.w, s0.w, fmaf(o0.z, s0.z, fmaf(o0.y, s0.y, o0.x * s0.x)));
                            const float hi = fmaf(o1.w, s1.w, fmaf(o1.z, s1.z, fmaf(o1.y, s1.y, o1.x * s1.x)));
                            acc[4 * k + j] = fmaf(au[0].x, fmaf(d, t, lo + hi), acc[4 * k + j]);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[as]);
            }
            if (SWIGLU) {
                // gate and up rows to the exchange buffer; the group's four warps go on or stop together
                float* sw = swap + ((ti & 1) * 2 + e) * WX_HALF * WX_ROWS;
#pragma unroll
                for (int j = 0; j < WX_HALF; ++j)
                    if (slot_of(j) < w.slots) sw[j * WX_ROWS + tid] = acc[j];
                int all;
                asm volatile(
                    "{\n\t.reg .pred p, r;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.and.pred r, %2, 128, p;\n\t"
                    "selp.b32 %0, 1, 0, r;\n\t}"
                    : "=r"(all)
                    : "r"((int)ok), "r"(1 + e)
                    : "memory");
                if (!all) break;
                const int r = tid & 63, n = w.n0 * TILE_N + r;
#pragma unroll 1
                for (int l = tid >> 6; l < WX_HALF; l += 2) {
                    const int slot = slot_of(l);
                    if (slot < w.slots && n < a.N)
                        a.c[(int64_t)(w.slot0 + slot) * a.N + n] = silu_acc(sw[l * WX_ROWS + r]) * sw[l * WX_ROWS + 64 + r];
                }
            } else {
                if (!ok) break;
                const int n = w.n0 * TILE_N + tid;
                float* c = SPLIT ? a.c + w.sb0 / a.per_split * a.split_stride : a.c;
                if (n < a.N)
#pragma unroll
                    for (int j = 0; j < WX_HALF; ++j)
                        if (slot_of(j) < w.slots) c[(int64_t)(w.slot0 + slot_of(j)) * a.N + n] = acc[j];
            }
        }
    } else if (warp >= WX_FIRST_EXPAND) {
        const int slot = (warp - WX_FIRST_EXPAND) >> 2, q = warp & 3;
        const uint32_t dst = tmem + WX_OPERAND + slot * 32 + ((uint32_t)(q * 32) << 16);
        const uint32_t row_at = smem_u32(sm_p) + (q * 32 + lane) * WX_SBB;
        uint32_t p = 0, ph = 0, p_ready = 0;
        uint32_t stages = SPLIT ? 0 : (uint32_t)mine * chunks;
        for (int i = 0; SPLIT && i < mine; ++i) {
            const WxTile w = wx_tile_at<SPLIT>(a, first, table, i);
            stages += w.sb1 - w.sb0;
        }
        for (uint32_t ci = 0; ci < stages; ++ci) {
            if (!__all_sync(0xffffffffu, p_ready != 0) && !mbar_wait_warp(&p_full[p], ph, a.status)) break;
            const uint32_t free_ahead = ci > 1 ? mbar_peek(&done[ci & 1], ((ci >> 1) - 1) & 1) : 1u;
            const uint32_t seg = row_at + p * WX_PACKED;
            uint32_t out[32];
            float d;
            float2 off;
            if (slot == 0) wx_expand<0>(seg, out, d, off);
            else if (slot == 1) wx_expand<1>(seg, out, d, off);
            else if (slot == 2) wx_expand<2>(seg, out, d, off);
            else wx_expand<3>(seg, out, d, off);
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_empty[p]);
            if (++p == WX_SP) { p = 0; ph ^= 1; }
            p_ready = mbar_peek(&p_full[p], ph);
            // (ci - 2 done: the epilogue has read ci - 4, whose header is overwritten below)
            if (!__all_sync(0xffffffffu, free_ahead != 0) && !mbar_wait_warp(&done[ci & 1], ((ci >> 1) - 1) & 1, a.status)) break;
            if (slot == 0) sm_d[(ci % WX_HDR) * WX_ROWS + q * 32 + lane] = d;
            reinterpret_cast<float2*>(sm_off + ((ci % WX_HDR) * 2 + (slot >> 1)) * WX_ROWS + q * 32 + lane)[slot & 1] = off;
            tc_fence_after();
            tmem_st32(dst + (ci & 1) * WX_SET, out);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[ci & 1]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

template <bool SWIGLU, bool SPLIT>
static int launch_wx(const WxArgs& a, int64_t rows) {
    static bool configured = false;
    if (!configured) {
        B200_CUDA(cudaFuncSetAttribute(wx_kernel<SWIGLU, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, WX_SMEM));
        configured = true;
    }
    const int64_t most = (rows / WX_CAP + std::min<int64_t>(a.ne, rows)) * a.n_tiles * a.k_splits;      // an expert's last tile may be short
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::min<int64_t>(most, num_sms()));
    cfg.blockDim = dim3(WX_THREADS);
    cfg.dynamicSmemBytes = WX_SMEM;
    cfg.stream = stream();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    B200_CUDA(cudaLaunchKernelEx(&cfg, wx_kernel<SWIGLU, SPLIT>, a));
    ++g_kernel_launches;
    return B200_OK;
}

// See gemm.cuh.
size_t moe_exact_bytes(int64_t NK, int d, int E) {
    const size_t k = std::max(d, E);
    return ((size_t)NK * 3 * k * 2 + 255) / 256 * 256 + (size_t)NK * (k / 256) * WX_AUX * 4;
}
int moe_exact_forward(const float* x, const int32_t* grouped, const int32_t* offsets, const void* gates, const void* ups,
                      const void* downs, float* act, float* y, void* scratch, int64_t N, int d, int E, int ne, int K) {
    const int64_t NK = N * K;
    B200_REQUIRE(ne <= WX_MAX_EXPERTS && NK * 3 <= 0x7fffffff && d % 256 == 0 && E % 256 == 0, "moe_exact: shape");
    __half* cols = static_cast<__half*>(scratch);
    float* aux = reinterpret_cast<float*>(static_cast<char*>(scratch) + ((size_t)NK * 3 * std::max(d, E) * 2 + 255) / 256 * 256);
    WxArgs a;
    a.offsets = offsets; a.aux = aux; a.ne = ne; a.M = 0; a.k_splits = 1; a.split_stride = 0;
    a.status = stream_status_ptr();
    B200_REQUIRE(a.status, "moe_exact: status word allocation failed");
    for (int pass = 0; pass < 2; ++pass) {
        const bool down = pass == 1;
        const int Kd = down ? E : d, Nd = down ? d : E, tile = down ? WX_ROWS : WX_ROWS / 2;
        int rc = make_tile_map(&a.map_x, cols, 3 * NK, Kd, WX_BOX);
        if (!rc) rc = make_packed_map(&a.map_w, down ? downs : gates, (int64_t)ne * Nd, (int64_t)Kd / 256 * WX_SBB, WX_SBB, tile);
        if (!rc) rc = make_packed_map(&a.map_w2, down ? downs : ups, (int64_t)ne * Nd, (int64_t)Kd / 256 * WX_SBB, WX_SBB, tile);
        if (rc) return rc;
        wx_split_kernel<<<(unsigned)ceil_div64(NK * (Kd / 256), 8), 256, 0, stream()>>>(down ? act : x, down ? nullptr : grouped, K,
                                                                                       (int)NK, Kd, cols, aux);
        B200_LAUNCH_CHECK("wx_split_kernel");
        a.c = down ? y : act;
        a.N = Nd; a.K = Kd; a.n_tiles = ceil_div(Nd, tile); a.per_split = Kd / 256;
        rc = down ? launch_wx<false, false>(a, NK) : launch_wx<true, false>(a, NK);
        if (rc) return rc;
    }
    return B200_OK;
}

// One Q4_K matrix for a few tens of tokens, exact to fp32: y [M, N] = x [M, K] . w [N, K]^T; K a multiple of 256, N of 4.
// Few tiles: K is cut across CTAs and the partial sums are added in a fixed order.  With w_up: y = silu(x . w^T) * (x . w_up^T),
// K whole (a gate and its up must be complete).
int linear_exact(const float* x, const void* w, float* y, int M, int K, int N, const void* w_up) {
    WxArgs a;
    const int rows = w_up ? WX_ROWS / 2 : WX_ROWS;
    a.n_tiles = ceil_div(N, rows);
    const int chunks = K / 256, tiles = w_up ? num_sms() : ceil_div(M, WX_CAP) * a.n_tiles;
    a.per_split = ceil_div(chunks, std::max(1, std::min(chunks, num_sms() / tiles)));
    a.k_splits = ceil_div(chunks, a.per_split);
    a.split_stride = a.k_splits > 1 ? (int64_t)M * N : 0;
    void *ws, *part = nullptr;
    const size_t cols_bytes = ((size_t)M * 3 * K * 2 + 255) / 256 * 256;
    int rc = workspace(WS_LINEAR).ensure(cols_bytes + (size_t)M * chunks * WX_AUX * 4 + 256, &ws);
    if (!rc && a.k_splits > 1) rc = workspace(WS_SPLITK).ensure((size_t)a.k_splits * a.split_stride * 4 + 256, &part);
    if (rc) return rc;
    __half* cols = static_cast<__half*>(ws);
    float* aux = reinterpret_cast<float*>(static_cast<char*>(ws) + cols_bytes);
    if ((rc = make_tile_map(&a.map_x, cols, 3 * (int64_t)M, K, WX_BOX))) return rc;
    if ((rc = make_packed_map(&a.map_w, w, N, (int64_t)chunks * WX_SBB, WX_SBB, rows))) return rc;
    if ((rc = make_packed_map(&a.map_w2, w_up ? w_up : w, N, (int64_t)chunks * WX_SBB, WX_SBB, rows))) return rc;
    a.offsets = nullptr; a.aux = aux; a.ne = 1; a.M = M; a.N = N; a.K = K;
    a.c = part ? static_cast<float*>(part) : y;
    a.status = stream_status_ptr();
    B200_REQUIRE(a.status, "linear_exact: status word allocation failed");
    wx_split_kernel<<<(unsigned)ceil_div(M * chunks, 8), 256, 0, stream()>>>(x, nullptr, 1, M, K, cols, aux);
    B200_LAUNCH_CHECK("wx_split_kernel");
    if ((rc = w_up ? launch_wx<true, false>(a, M) : launch_wx<false, true>(a, M))) return rc;
    return part ? splitk_reduce(a.c, y, a.k_splits, a.split_stride, M, N, N) : B200_OK;
}

}  // namespace b200
