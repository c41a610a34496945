// The many-token GEMM for packed weights:  C[rows, N] = A[rows, K] . W[N, K]^T  on tcgen05 with the
// dequantised WEIGHTS as the MMA's first operand in TENSOR memory and the token rows as the second in shared
// memory: the accumulator of a tile is [128 weight rows (lanes) x up to 192 tokens (columns)].
//
// What bounded the form before it (weights expanded to fp16 tiles in shared memory, both operands read from
// there, 256 token rows per tile): shared-memory bandwidth - a 64-wide K step moved 131 KB (1020 cycles at
// 128 B per cycle) for 524 cycles of tensor work - and, with few tokens, one expanding warp pass per K step
// and MMA work for 128-row halves that were mostly empty.  Here a thread expands its own weight row in
// registers and writes it with one tcgen05.st; shared memory sees the token rows once in and once out and the
// packed bytes (29 + 29 KB per 393 tensor cycles), and the MMA's N is the tile's own token count rounded to 16.
//
// Tensor memory: two accumulator sets of 192 columns (the epilogue of a tile under the main loop of the next) and
// four operand slots of 32 columns (64 fp16 of K).  The SwiGLU form puts 64 gate rows and the same 64 up rows
// in one tile and exchanges them through shared memory in the epilogue.
//   warp 0        token rows by TMA: one load per stage of 64 of K (128 for at most 96 rows), from one of twelve 3-D maps
//   warp 2        packed rows by TMA (256 of K per stage)
//   warp 1        MMA issue, a stage per round
//   warps 4..7    epilogue: a lane holds one weight row, so a warp stores 32 consecutive outputs of a token
//   warps 8..23   expansion: four groups of four warps, group = operand slot = K step mod 4
// A stage of token rows has one pair of barriers for everything that its MMAs read and free: `full` counts the load and
// the expanding warps' arrivals, `empty` one commit; the operand slots need none of their own.
// Group lists (the MoE experts): rows of A cut into consecutive ranges by device offsets; a range is cut into
// equal token tiles.  All waits are bounded; see gemm_umma.cu for what happens when one runs out.
//
// What bounds it: with six warps at a scheduler an instruction of a role costs four to five cycles, so a role that does
// little per K step still takes hundreds of cycles for it.  Clock stamps showed the loads of token rows (two to four TMA
// instructions per K step with their addresses, a wait and two barriers) at some 600 cycles for 384 of tensor work, and the
// MMA warp's round (a wait, four MMAs, two commits) at 430.  Hence one load and one commit per stage, stages of 128 where
// the rows leave room, descriptors by their low word, and a look before the counted wait.  In us, before and after:
//   8188 x 6448 x 1536 Q4_K  164.9 -> 142.4 (16 of them round the activations; 1290 TFLOP/s without)
//   8188 x 1536 x 3072        107.6 -> 95.3      4096 x 6448 x 1536  93.2 -> 82.9
//   64 experts of 1536 x 512, gate | up and down: 384 rows each 156.7 -> 142.3, 192: 101 -> 91, 48: 76.8 -> 56.4, 16: 70.7 -> 52.1
//   72 experts of 4096 x 768, 72 rows each: 216 -> 157 (the weights' way from HBM: 60)
// With the expansion left out the last takes 130: few rows are bound by the hand-overs between the roles and by issue slots.
// Slower: two K steps per expanding warp and turn (the second one's expansion sits between two MMA rounds), stages of
// constant number in the MMA warp (no difference once the loads are quick).
#include <algorithm>

#include "gemm.cuh"
#include "linear.cuh"
#include "umma.cuh"
#include "umma_ts.cuh"

namespace b200 {

int make_packed_map(CUtensorMap* out, const void* base, int64_t rows, int64_t row_bytes, int box_bytes, int box_rows);
int splitk_reduce(const float* part, float* c, int splits, int64_t stride, int M, int N, int64_t ldc);

constexpr int WT_TOKENS = 192;                // most tokens of a tile
constexpr int WT_ROWS = 128;                  // weight rows of a tile
constexpr int WT_BOX = 16;                    // token rows are loaded in multiples of this, the MMA's granularity of N
constexpr int WT_X_STAGE = WT_TOKENS * 128;   // 64 fp16 of K per token row, or 128 of at most 96 rows
constexpr int WT_SLOT0 = 2 * WT_TOKENS;       // first tensor-memory column of the operand slots
constexpr int WT_SLOT = 32, WT_SLOTS = 4;
constexpr int WT_SWAP = 2 * 2 * 16 * 64 * 4;  // SwiGLU epilogue: [buffer][half][token][row] floats
constexpr int WT_FIRST_EXPAND = 8;
constexpr int WT_EXPAND_WARPS = 16;
constexpr int WT_THREADS = (WT_FIRST_EXPAND + WT_EXPAND_WARPS) * 32;
constexpr int WT_TABLE = 64;                  // a CTA's tiles worked out in advance; later ones on the way
constexpr int WT_LISTS = (3 * 256 + 2) * 4;
constexpr int WT_MAX_GROUPS = 256;            // group lists kept as a prefix table; longer ones are walked

struct alignas(64) WtArgs {
    CUtensorMap map_x[WT_TOKENS / WT_BOX];    // a stage of 16, 32 .. 192 token rows in one load
    CUtensorMap map_w, map_w2;
    const int32_t* offsets;                   // device [groups + 1], or null: one group of M rows
    const int32_t* group_map;                 // device [groups]: block of N weight rows a group uses (negative: skipped)
    int M, groups, N, K;
    int slots, n_tiles;                       // upper bound of the token tiles, weight tiles per token tile
    float* c;
    float* const* group_c;                    // see GemmArgs
    __half* c16;
    int64_t ldc;
    float scale;
    int* status;
    int k_splits, sb_split;                   // K ranges (in units of 256) whose partial products are added afterwards
    int64_t split_stride;
};

template <bool SWIGLU, int KIND>
struct WtShape {
    static constexpr int SBB = 8 * (KIND == 3 ? 18 : q_block_bytes(KIND));     // bytes of 256 weights
    static constexpr int PACKED = WT_ROWS * SBB;
    static constexpr int SX = SWIGLU ? 5 : 6;                                 // at least 4: see the expansion
    static constexpr int SP = KIND == 2 ? 2 : KIND == 1 && !SWIGLU ? 3 : 4;
    static constexpr int TILE_N = SWIGLU ? WT_ROWS / 2 : WT_ROWS;              // output columns of a tile
    static constexpr int SMEM = SX * WT_X_STAGE + SP * PACKED + (SWIGLU ? WT_SWAP : 0) + 1024 + 256 + WT_LISTS + WT_TABLE * 24;
    static_assert(SMEM <= 227 * 1024, "the stages do not fit the shared memory of an SM");
};

struct WtTile {
    int group, row0, rows, n0, brow, split;
};

__host__ __device__ __forceinline__ int wt_tiles(int rows) { return (rows + WT_TOKENS - 1) / WT_TOKENS; }
// Tile i of `rows` token rows cut into equal tiles of a multiple of 16.
__device__ __forceinline__ void wt_cut(int rows, int i, int& first, int& count) {
    const int n = max(1, wt_tiles(rows)), size = ((rows + n - 1) / n + 15) & ~15;
    first = i * size;
    count = max(0, min(size, rows - first));
}

// Group lists of at most WT_MAX_GROUPS: the offsets and each group's first token tile (first[groups] = all of them) in
// shared memory, so that the searches below touch global memory once, and with one latency.  All threads.
struct WtLists {
    int first[WT_MAX_GROUPS + 1], offset[WT_MAX_GROUPS + 1], block[WT_MAX_GROUPS];
};
__device__ __forceinline__ void wt_build(const WtArgs& a, WtLists& l) {
    if (!a.offsets || a.groups > WT_MAX_GROUPS) return;
    for (int g = threadIdx.x; g <= a.groups; g += blockDim.x) {
        l.offset[g] = a.offsets[g];
        if (g < a.groups) l.block[g] = a.group_map ? a.group_map[g] : g;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        int carry = 0;
        for (int g0 = 0; g0 < a.groups; g0 += 32) {
            const int g = g0 + threadIdx.x, n = g < a.groups && l.block[g] >= 0 ? wt_tiles(l.offset[g + 1] - l.offset[g]) : 0;
            int incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)threadIdx.x >= o) incl += up;
            }
            if (g < a.groups) l.first[g] = carry + incl - n;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (threadIdx.x == 0) l.first[a.groups] = carry;
    }
    __syncthreads();
}

__device__ __forceinline__ bool wt_find(const WtArgs& a, const WtLists& l, int t, WtTile& w) {
    w.split = 0;
    if (a.k_splits > 1) {
        w.split = t % a.k_splits;
        t /= a.k_splits;
    }
    const int slot = t / a.n_tiles;
    w.n0 = t - slot * a.n_tiles;              // weight tile; scaled by the caller's tile width
    w.group = 0;
    w.brow = 0;
    int lo = 0, hi = a.M, i = slot;
    if (a.offsets) {
        if (a.groups <= WT_MAX_GROUPS) {
            if (slot >= l.first[a.groups]) return false;
            int g = 0, h = a.groups;          // the last group whose first tile is <= slot owns it
            while (h - g > 1) {
                const int mid = (g + h) >> 1;
                if (l.first[mid] <= slot) g = mid; else h = mid;
            }
            w.group = g;
            i = slot - l.first[g];
            lo = l.offset[g];
            hi = l.offset[g + 1];
            w.brow = l.block[g] * a.N;
        } else {
            int g = 0;
            for (; g < a.groups; ++g) {
                const int n = (a.group_map && a.group_map[g] < 0) ? 0 : wt_tiles(a.offsets[g + 1] - a.offsets[g]);
                if (i < n) break;
                i -= n;
            }
            if (g == a.groups) return false;
            w.group = g;
            lo = a.offsets[g];
            hi = a.offsets[g + 1];
            w.brow = (a.group_map ? a.group_map[g] : g) * a.N;
        }
    }
    wt_cut(hi - lo, i, w.row0, w.rows);
    w.row0 += lo;
    return w.rows > 0;
}
__device__ __noinline__ bool wt_find_late(const WtArgs& a, const WtLists& l, int t, WtTile& w) { return wt_find(a, l, t, w); }

// A stage of token rows, and with it one round of the MMA warp, is 64 of K, or 128 where the tile's rows fill no more than
// half of it (a ring of mostly empty stages is shorter than the latency that it has to cover): log2 of the K steps of 64.
__host__ __device__ constexpr int wt_unit(int rows) { return rows > WT_TOKENS / 2 ? 0 : 1; }
__device__ __forceinline__ void mbar_arrive_n(uint64_t* bar, uint32_t n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}

// Tile number i of this CTA.  The search (divisions, bisection) takes over a thousand cycles, which every role would
// otherwise spend between two tiles of a few thousand: one thread per tile does it when the kernel starts.
__device__ __forceinline__ void wt_fill(const WtArgs& a, const WtLists& l, int* table, int total) {
    const int t = blockIdx.x + threadIdx.x * gridDim.x;
    if (threadIdx.x < WT_TABLE && t < total) {
        WtTile w{0, 0, 0, 0, 0, 0};
        if (!wt_find(a, l, t, w)) w.rows = 0;
        int* e = table + 6 * threadIdx.x;
        e[0] = w.group; e[1] = w.row0; e[2] = w.rows; e[3] = w.n0; e[4] = w.brow; e[5] = w.split;
    }
}
__device__ __forceinline__ bool wt_tile_at(const WtArgs& a, const WtLists& l, const int* table, int i, WtTile& w) {
    if (i >= WT_TABLE) {
        WtTile late;                          // its address is taken: w itself stays in registers
        const bool ok = wt_find_late(a, l, blockIdx.x + i * gridDim.x, late);
        w = late;
        return ok;
    }
    const int* e = table + 6 * i;
    w.group = e[0]; w.row0 = e[1]; w.rows = e[2]; w.n0 = e[3]; w.brow = e[4]; w.split = e[5];
    return w.rows > 0;
}

// ---- expansion: 64 weights of a row (K step J of its 256) to 32 fp16 pairs ----------------------
// fp16 arithmetic, two values per instruction: a byte b OR-ed into the mantissa of 0x6400 is 1024 + b.
//   Q4_0  (q - 8) * d,  Q8_0  q * d        exact products rounded once
//   Q4_1  q * d + m                         one rounding
//   Q4_K  (q * sc) * d - fp16(m * dmin)     q * sc exact; the minimum rounded first
// against the fp16-rounded value of the materialising dequantiser: equal for Q4_0 / Q8_0, within one ulp else.
template <int KIND, int J>
__device__ __forceinline__ void wt_expand(uint32_t seg, uint32_t (&out)[32]) {
    auto vec = [&](int i) {
        uint4 v;
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(seg + 16 * i));
        return v;
    };
    if (KIND == 3) {
        const uint4 hdr = vec(0), q0 = vec(1 + 2 * J), q1 = vec(2 + 2 * J);
        const __half2 d2 = wt_half2(hdr.x & 0xFFFFu);
        const float dmin = half_bits_to_float((uint16_t)(hdr.x >> 16));
        const uint32_t words[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            int s, m;
            q4k_scale_min_regs(2 * J + hh, hdr.y, hdr.z, hdr.w, s, m);
            // integers below 1024 become fp16 (and fp32) by their bits; conversions would take the slow pipe.
            // high nibbles stay where they are: 1024 + 16 q, times s / 16 (exact)
            const uint32_t sb = (uint32_t)s * 0x00010001u | 0x64006400u;
            const __half2 s2 = __hsub2(*reinterpret_cast<const __half2*>(&sb), wt_half2(0x6400u));
            const __half2 sc2 = hh ? __hmul2(s2, wt_half2(0x2C00u)) : s2;
            const __half2 nsc = __hmul2(s2, wt_half2(hh ? 0xD400u : 0xE400u));                          // -64 s, -1024 s: exact
            const float mf = __fsub_rn(__uint_as_float(0x4B000000u | (uint32_t)m), 8388608.0f);
            const __half2 nm = __half2half2(__float2half_rn(-__fmul_rn(dmin, mf)));
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t x = words[i] & (hh ? 0xF0F0F0F0u : 0x0F0F0F0Fu);
                out[16 * hh + 2 * i] = wt_bits(__hfma2(__hfma2(wt_magic(x, WT_SEL_01), sc2, nsc), d2, nm));
                out[16 * hh + 2 * i + 1] = wt_bits(__hfma2(__hfma2(wt_magic(x, WT_SEL_23), sc2, nsc), d2, nm));
            }
        }
    } else {
        // the 16-byte window that covers the two blocks, then words at compile-time places
        constexpr int WORDS = KIND == 2 ? 17 : KIND == 1 ? 10 : 9, W0 = WORDS * J, V0 = W0 / 4, OFF = W0 % 4, NV = (OFF + WORDS + 3) / 4;
        uint32_t w[4 * NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint4 v = vec(V0 + i);
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
        auto half_at = [&](int i) { return (w[OFF + (i >> 1)] >> (16 * (i & 1))) & 0xFFFFu; };
        constexpr int BH = q_block_bytes(KIND) / 2;                   // halfwords per block
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const __half2 d2 = wt_half2(half_at(b * BH));
            if (KIND == 2) {
                const __half2 bias = wt_half2(0x6480u);               // 1024 + 128
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int h = b * BH + 1 + i;
                    const uint32_t x = w[OFF + (h >> 1)] ^ 0x80808080u;          // int8 + 128
                    out[16 * b + i] = wt_bits(__hmul2(__hsub2(wt_magic(x, (h & 1) ? WT_SEL_23 : WT_SEL_01), bias), d2));
                }
            } else {
                const __half2 off = wt_half2(KIND == 0 ? 0x6408u : 0x6400u);     // 1032 / 1024
                const __half2 m2 = KIND == 1 ? wt_half2(half_at(b * BH + 1)) : wt_half2(0u);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int h = b * BH + (KIND == 0 ? 1 : 2) + i;
                    const uint32_t x = w[OFF + (h >> 1)], sel = (h & 1) ? WT_SEL_23 : WT_SEL_01;
                    const __half2 lo = __hsub2(wt_magic(x & 0x0F0F0F0Fu, sel), off), hi = __hsub2(wt_magic((x >> 4) & 0x0F0F0F0Fu, sel), off);
                    out[16 * b + i] = wt_bits(KIND == 0 ? __hmul2(lo, d2) : __hfma2(lo, d2, m2));
                    out[16 * b + 8 + i] = wt_bits(KIND == 0 ? __hmul2(hi, d2) : __hfma2(hi, d2, m2));
                }
            }
        }
    }
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// The fast exponential and reciprocal (a few fp32 ulp) are invisible after the rounding to fp16.
__device__ __forceinline__ float wt_silu(float v) { return __fdividef(v, 1.0f + __expf(-v)); }

template <bool SWIGLU, int KIND>
__global__ void __launch_bounds__(WT_THREADS, 1) umma_wt_kernel(const __grid_constant__ WtArgs a) {
    using S = WtShape<SWIGLU, KIND>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sm_x = smem;
    uint8_t* sm_p = sm_x + S::SX * WT_X_STAGE;
    float* swap = reinterpret_cast<float*>(sm_p + S::SP * S::PACKED);
    uint64_t* full = reinterpret_cast<uint64_t*>(sm_p + S::SP * S::PACKED + (SWIGLU ? WT_SWAP : 0));
    uint64_t* empty = full + S::SX;
    uint64_t* p_full = empty + S::SX;
    uint64_t* p_empty = p_full + S::SP;
    uint64_t* acc_full = p_empty + S::SP;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    WtLists& lists = *reinterpret_cast<WtLists*>(reinterpret_cast<int*>(full) + 64);
    int* table = reinterpret_cast<int*>(&lists + 1);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int total = a.slots * a.n_tiles * a.k_splits, sb_all = a.K / 256;
    // what does not depend on the kernels before
    if (threadIdx.x == 0) {
        tma_prefetch_map(&a.map_w);
        if (SWIGLU) tma_prefetch_map(&a.map_w2);
        for (int s = 0; s < S::SX; ++s) { mbar_init(&full[s], 1 + WT_EXPAND_WARPS); mbar_init(&empty[s], 1); }
        for (int s = 0; s < S::SP; ++s) { mbar_init(&p_full[s], 1); mbar_init(&p_empty[s], WT_EXPAND_WARPS); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 4); }
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    pdl_wait();                               // offsets, rows and everything that reads the output now: the kernels before
    wt_build(a, lists);
    wt_fill(a, lists, table, total);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    constexpr uint32_t tmem = 0;              // all 512 columns: the allocation starts at the first
    pdl_launch_dependents();
    const int mine = ((int)blockIdx.x < total ? total - (int)blockIdx.x + (int)gridDim.x - 1 : 0) / (int)gridDim.x;
    // every role walks the same tiles; sb0 .. sb1: a tile's range of K in units of 256
    auto range = [&](const WtTile& w, int& sb0, int& sb1) {
        sb0 = w.split * a.sb_split;
        sb1 = min(sb_all, sb0 + a.sb_split);
    };

    if (warp == 0) {
        const uint32_t x0 = smem_u32(sm_x), full0 = smem_u32(full);
        uint32_t it = 0, s = 0, ph = 0;
        bool ok = true;
        for (int i = 0; i < mine && ok; ++i) {
            WtTile w;
            if (!wt_tile_at(a, lists, table, i, w)) continue;
            int sb0, sb1;
            range(w, sb0, sb1);
            const int unit = wt_unit(w.rows), steps = 1 << unit, boxes = (w.rows + WT_BOX - 1) / WT_BOX;
            const uint32_t bytes = (boxes * WT_BOX * 128) << unit;
            const CUtensorMap* map = &a.map_x[boxes - 1];
            const int row0 = w.row0, k1 = 4 * sb1;
            for (int kb = 4 * sb0; kb < k1; kb += steps, ++it) {
                if (it >= S::SX && !__all_sync(0xffffffffu, mbar_try_wait(&empty[s], ph ^ 1))) {
                    ok = mbar_wait_warp(&empty[s], ph ^ 1, a.status);
                    if (!ok) break;
                }
                if (elect_one()) {
                    mbar_expect_tx(&full[s], bytes);
                    tma_load_3d(x0 + s * WT_X_STAGE, map, 0, row0, kb, full0 + s * 8);
                }
                if (++s == S::SX) { s = 0; ph ^= 1; }
            }
        }
        if (!ok)
            for (uint32_t j = it > S::SX ? it - S::SX : 0; j < it; ++j)
                if (!mbar_wait_warp(&full[j % S::SX], (j / S::SX) & 1, a.status)) break;
    } else if (warp == 2) {
        const uint32_t p0 = smem_u32(sm_p), full0 = smem_u32(p_full);
        uint32_t it = 0, p = 0, ph = 0;
        bool ok = true;
        for (int i = 0; i < mine && ok; ++i) {
            WtTile w;
            if (!wt_tile_at(a, lists, table, i, w)) continue;
            int sb0, sb1;
            range(w, sb0, sb1);
            const int brow = w.brow + w.n0 * S::TILE_N;
            for (int sb = sb0; sb < sb1; ++sb, ++it) {
                if (it >= S::SP && !__all_sync(0xffffffffu, mbar_try_wait(&p_empty[p], ph ^ 1))) {
                    ok = mbar_wait_warp(&p_empty[p], ph ^ 1, a.status);
                    if (!ok) break;
                }
                if (elect_one()) {
                    const uint32_t dst = p0 + p * S::PACKED, bar = full0 + p * 8;
                    mbar_expect_tx(&p_full[p], S::PACKED);
                    tma_load_2d(dst, &a.map_w, sb * (S::SBB / 4), brow, bar);
                    if (SWIGLU) tma_load_2d(dst + S::PACKED / 2, &a.map_w2, sb * (S::SBB / 4), brow, bar);
                }
                if (++p == S::SP) { p = 0; ph ^= 1; }
            }
        }
        if (!ok)
            for (uint32_t j = it > S::SP ? it - S::SP : 0; j < it; ++j)
                if (!mbar_wait_warp(&p_full[j % S::SP], (j / S::SP) & 1, a.status)) break;
    } else if (warp == 1) {
        const uint32_t desc0 = (uint32_t)umma_smem_desc(smem_u32(sm_x));
        uint32_t ti = 0, s = 0, ph = 0;
        bool ok = true;
        for (int i = 0; i < mine && ok; ++i) {
            WtTile w;
            if (!wt_tile_at(a, lists, table, i, w)) continue;
            int sb0, sb1;
            range(w, sb0, sb1);
            const uint32_t idesc = umma_idesc_f16(WT_ROWS, (w.rows + 15) & ~15), as = ti & 1;
            if (ti > 1) ok = mbar_wait_warp(&acc_empty[as], ((ti >> 1) - 1) & 1, a.status);
            if (!ok) break;
            tc_fence_after();
            const uint32_t d = tmem + as * WT_TOKENS;
            const int k0 = 4 * sb0, k1 = 4 * sb1;
            const uint32_t step = (w.rows + WT_BOX - 1) / WT_BOX * (WT_BOX * 128 / 16);   // 64 of K of the rows loaded
            auto rounds = [&](auto unit) {
                constexpr int STEPS = 1 << decltype(unit)::value;
                for (int kb = k0; kb < k1; kb += STEPS) {
                    if (!__all_sync(0xffffffffu, mbar_try_wait(&full[s], ph))) {
                        ok = mbar_wait_warp(&full[s], ph, a.status);
                        if (!ok) return;
                    }
                    tc_fence_after();
                    const uint32_t op = WT_SLOT0 + (kb & (WT_SLOTS - 1)) * WT_SLOT, desc = desc0 + s * (WT_X_STAGE / 16);
                    const uint32_t accumulate = kb > k0;
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < 4 * STEPS; ++k)   // 32 bytes of K per step: 2 in the descriptor's units
                            umma_f16_ts_lo(d, op + k * 8, desc + (k >> 2) * step + 2 * (k & 3), idesc, k > 0 ? 1u : accumulate);
                        umma_commit(&empty[s]);
                        if (kb + STEPS == k1) umma_commit(&acc_full[as]);
                    }
                    if (++s == S::SX) { s = 0; ph ^= 1; }
                }
            };
            if (wt_unit(w.rows) == 0) rounds(std::integral_constant<int, 0>{});
            else rounds(std::integral_constant<int, 1>{});
            ++ti;
        }
    } else if (warp >= 4 && warp < WT_FIRST_EXPAND) {
        const int q = warp & 3;
        uint32_t ti = 0;
        for (int i = 0; i < mine; ++i) {
            WtTile w;
            if (!wt_tile_at(a, lists, table, i, w)) continue;
            const uint32_t as = ti & 1;
            bool ok = mbar_wait(&acc_full[as], (ti >> 1) & 1, a.status);
            ok = __all_sync(0xffffffffu, ok && *reinterpret_cast<volatile int*>(a.status) == 0);
            if (SWIGLU) {
                // the four warps meet in the exchange: they go on or stop together
                int all;
                asm volatile(
                    "{\n\t.reg .pred p, r;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.and.pred r, 1, 128, p;\n\t"
                    "selp.b32 %0, 1, 0, r;\n\t}"
                    : "=r"(all)
                    : "r"((int)ok)
                    : "memory");
                ok = all != 0;
            }
            if (!ok) break;
            tc_fence_after();
            const uint32_t tq = tmem + as * WT_TOKENS + ((uint32_t)(q * 32) << 16);
            if (SWIGLU) {
                // lanes of warps 0, 1: gate rows; of 2, 3: up rows.  Of every 32 tokens warps 0, 1 finish the first
                // 16 and warps 2, 3 the rest: each side leaves the other's half in the exchange buffer.
                const int side = q >> 1, r = (q & 1) * 32 + lane, n = w.n0 * S::TILE_N + r;
                __half* dst = a.c16 + ((int64_t)w.row0 + 16 * side) * a.ldc + n;
                int buf = 0;
                for (int c0 = 0; c0 < w.rows; c0 += 32, dst += 32 * a.ldc, buf ^= 1) {
                    float mine[16], give[16];
                    tmem_ld16(tq + c0 + 16 * side, mine);
                    tmem_ld16(tq + c0 + 16 * (side ^ 1), give);
                    float* out = swap + (buf * 2 + side) * 16 * 64 + r;
                    const float* in = swap + (buf * 2 + (side ^ 1)) * 16 * 64 + r;
#pragma unroll
                    for (int i = 0; i < 16; ++i) out[i * 64] = give[i];
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    const int left = w.rows - c0 - 16 * side;
                    if (n < a.N) {
                        __half* o = dst;
#pragma unroll
                        for (int i = 0; i < 16; ++i, o += a.ldc) {
                            const float other = in[i * 64];
                            if (i < left) *o = __float2half_rn(side ? wt_silu(other) * mine[i] : wt_silu(mine[i]) * other);
                        }
                    }
                }
            } else {
                const int n = w.n0 * S::TILE_N + q * 32 + lane;
                const int64_t step = a.ldc;
                float* dst = (a.group_c ? a.group_c[w.group] : a.c + w.split * a.split_stride) + (int64_t)w.row0 * step + n;
                for (int c0 = 0; c0 < w.rows; c0 += 32) {
                    float v[32];
                    tmem_ld32(tq + c0, v);                    // columns past the tile's tokens are not stored
                    if (n < a.N) {
                        const int left = w.rows - c0;
                        if (left >= 32) {
#pragma unroll
                            for (int i = 0; i < 32; ++i, dst += step) *dst = v[i] * a.scale;
                        } else {
#pragma unroll
                            for (int i = 0; i < 32; ++i, dst += step)
                                if (i < left) *dst = v[i] * a.scale;
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[as]);
            ++ti;
        }
    } else if (warp >= WT_FIRST_EXPAND) {
        const int slot = (warp - WT_FIRST_EXPAND) >> 2, q = warp & 3;
        const uint32_t dst = tmem + WT_SLOT0 + slot * WT_SLOT + ((uint32_t)(q * 32) << 16);
        const uint32_t row_at = smem_u32(sm_p) + (q * 32 + lane) * S::SBB;
        uint32_t p = 0, ph = 0;
        uint32_t base = 0, bph = 0;                       // the token rows' first stage of these 256 of K
        uint32_t last = S::SX, lph = 0;                   // the stage whose MMAs read this slot last (SX: none)
        bool ok = true;
        for (int i = 0; i < mine && ok; ++i) {
            WtTile w;
            if (!wt_tile_at(a, lists, table, i, w)) continue;
            int sb0, sb1;
            range(w, sb0, sb1);
            const int unit = wt_unit(w.rows);
            for (int sb = sb0; sb < sb1; ++sb) {
                if (!__all_sync(0xffffffffu, mbar_try_wait(&p_full[p], ph))) {
                    ok = mbar_wait_warp(&p_full[p], ph, a.status);
                    if (!ok) break;
                }
                const uint32_t seg = row_at + p * S::PACKED;
                uint32_t out[32];
                if (slot == 0) wt_expand<KIND, 0>(seg, out);
                else if (slot == 1) wt_expand<KIND, 1>(seg, out);
                else if (slot == 2) wt_expand<KIND, 2>(seg, out);
                else wt_expand<KIND, 3>(seg, out);
                __syncwarp();                             // every lane has read its row: the stage goes back to TMA
                if (lane == 0) mbar_arrive(&p_empty[p]);
                if (++p == S::SP) { p = 0; ph ^= 1; }
                // The slot is free once the MMAs of four K steps ago are done.  With them every stage up to theirs has
                // been through, so that with SX >= 4 this step's stage is in the phase that the arrival is meant for;
                // and theirs cannot complete another phase before this step, so that the parity is not ambiguous.
                if (last < S::SX && !__all_sync(0xffffffffu, mbar_try_wait(&empty[last], lph))) {
                    ok = mbar_wait_warp(&empty[last], lph, a.status);
                    if (!ok) break;
                }
                tc_fence_after();
                tmem_st32(dst, out);
                tc_fence_before();
                const uint32_t at = base + (slot >> unit), over = at >= S::SX;
                last = at - (over ? S::SX : 0);
                lph = bph ^ over;
                __syncwarp();
                if (lane == 0) mbar_arrive_n(&full[last], 4 >> unit);     // 16 in all, whatever the unit
                base += WT_SLOTS >> unit;
                if (base >= S::SX) { base -= S::SX; bph ^= 1; }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// ---- host side ------------------------------------------------------------------
// The token rows' loads: 16 (i + 1) rows and the K steps of their stage.
struct WtBoxes {
    StageBox b[WT_TOKENS / WT_BOX];
    constexpr WtBoxes() : b() {
        for (int i = 0; i < WT_TOKENS / WT_BOX; ++i) b[i] = StageBox{(i + 1) * WT_BOX, 1 << wt_unit((i + 1) * WT_BOX)};
    }
};
static constexpr WtBoxes wt_boxes;

template <bool SWIGLU, int KIND>
static int launch_wt(WtArgs& a, bool allow_split, bool early) {
    using S = WtShape<SWIGLU, KIND>;
    auto kern = umma_wt_kernel<SWIGLU, KIND>;
    static bool configured = false;
    if (!configured) {
        B200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM));
        configured = true;
    }
    a.n_tiles = ceil_div(a.N, S::TILE_N);
    a.slots = wt_tiles(a.M) + (a.offsets ? a.groups : 0);
    const int tiles = a.slots * a.n_tiles, sb = a.K / 256;
    a.k_splits = 1;
    a.sb_split = sb;
    // Few tiles (a decode batch, the attention projections): K is cut across CTAs and the partial products are
    // added in a fixed order.  Not for group lists: the sum walks all M rows, a list may leave some untouched.
    if (!SWIGLU && !a.offsets && allow_split && sb >= 2 && tiles * 2 <= num_sms()) {
        const int per = ceil_div(sb, std::min(sb, num_sms() / tiles));
        a.k_splits = ceil_div(sb, per);
        a.sb_split = per;
    }
    float* c = a.c;
    if (a.k_splits > 1) {
        a.split_stride = (int64_t)a.M * a.ldc;
        void* wsp;
        int rc = workspace(WS_SPLITK).ensure((size_t)a.k_splits * a.split_stride * sizeof(float) + 256, &wsp);
        if (rc) return rc;
        a.c = static_cast<float*>(wsp);
    }
    // Set up (barriers, tensor memory, tensor maps: a microsecond) while the kernel before it ends: the projections, which have
    // the device to themselves (64 sequences 102.7 -> 100.1 ms).  Not the experts' products, routed and shared beside each other:
    // CTAs that wait hold SMs that the other stream's could use (five ragged prompts and steps 37.0 ms, 37.8 with them).
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::min(tiles * a.k_splits, num_sms()));
    cfg.blockDim = dim3(WT_THREADS);
    cfg.dynamicSmemBytes = S::SMEM;
    cfg.stream = stream();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    B200_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
    ++g_kernel_launches;
    return a.k_splits > 1 ? splitk_reduce(a.c, c, a.k_splits, a.split_stride, a.M, a.N, a.ldc) : B200_OK;
}

// See gemm.cuh.
int umma_gemm_q(int epi, int kind, const __half* A, int64_t a_rows, const void* B, const void* B2, int64_t b_rows,
                const int32_t* offsets, int groups, int M, int N, int K, float* c, __half* c16, int64_t ldc,
                float scale, const int32_t* group_map, float* const* group_c, bool allow_split_k, bool early) {
    if (M <= 0 || N <= 0) return B200_OK;
    B200_REQUIRE(kind >= 0 && kind <= 3, "umma_gemm_q: unknown kind %d", kind);
    B200_REQUIRE(!group_c || (offsets && epi == GEMM_EPI_STORE), "umma_gemm_q: per-group outputs need the grouped store form");
    B200_REQUIRE(A && B && K > 0 && K % 256 == 0, "umma_gemm_q: K must be a positive multiple of 256");
    B200_REQUIRE(groups >= 1 && (offsets || groups == 1), "umma_gemm_q: groups need a device offsets array");
    B200_REQUIRE((group_map || b_rows >= (int64_t)groups * N) && a_rows >= M, "umma_gemm_q: operand shapes do not cover the groups");
    WtArgs a;
    int rc = make_stage_maps(a.map_x, A, a_rows, K, wt_boxes.b, WT_TOKENS / WT_BOX);
    if (rc) return rc;
    const int64_t row_bytes = q_row_bytes(kind, K);
    const int sbb = 8 * (kind == 3 ? 18 : q_block_bytes(kind));
    const bool swiglu = epi == GEMM_EPI_SWIGLU;
    const int box_rows = swiglu ? WT_ROWS / 2 : WT_ROWS;
    rc = make_packed_map(&a.map_w, B, b_rows, row_bytes, sbb, box_rows);
    if (rc) return rc;
    a.map_w2 = a.map_w;
    if (swiglu) {
        B200_REQUIRE(B2 && c16 && ldc % 2 == 0, "umma_gemm_q: the SwiGLU form needs the second matrix and an fp16 output");
        rc = make_packed_map(&a.map_w2, B2, b_rows, row_bytes, sbb, box_rows);
        if (rc) return rc;
    } else {
        B200_REQUIRE(c || group_c, "umma_gemm_q: null output");
    }
    a.offsets = offsets; a.group_map = group_map; a.M = M; a.groups = groups; a.N = N; a.K = K;
    a.c = c; a.group_c = group_c; a.c16 = c16; a.ldc = ldc; a.scale = scale; a.split_stride = 0;
    a.status = stream_status_ptr();
    B200_REQUIRE(a.status, "umma_gemm_q: status word allocation failed");
    switch (kind) {
        case 0: return swiglu ? launch_wt<true, 0>(a, allow_split_k, early) : launch_wt<false, 0>(a, allow_split_k, early);
        case 1: return swiglu ? launch_wt<true, 1>(a, allow_split_k, early) : launch_wt<false, 1>(a, allow_split_k, early);
        case 2: return swiglu ? launch_wt<true, 2>(a, allow_split_k, early) : launch_wt<false, 2>(a, allow_split_k, early);
        default: return swiglu ? launch_wt<true, 3>(a, allow_split_k, early) : launch_wt<false, 3>(a, allow_split_k, early);
    }
}

}  // namespace b200
