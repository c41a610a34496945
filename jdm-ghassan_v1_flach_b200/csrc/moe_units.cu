// MoE layer for a decode batch (tens of tokens): the experts as weight streams shared by
// the tokens that chose them.
//
// With 64 tokens and top-6 of 64 experts nearly every expert is touched, by about six tokens
// each.  The tensor-core GEMM path would expand a 128-row weight tile per expert for six
// rows of activations; the token-major few-token path (decode_moe.cu) would stream an expert
// once per token.  Here the (token, k) slots are sorted by expert (the layer's own
// permutation), cut into *units* of up to eight slots of one expert, and a unit's rows are
// streamed once through the digit engine (digit_tile.cuh) with its tokens as columns: exact
// dequantised weights, activations to 2^-31 of their block's maximum, fp32 sums.
//
//   moe_units_build_kernel    offsets -> unit table (expert, first sorted slot, slots)
//   moe_units_kernel<gate/up> act[slot, :] = silu(gate_e x_t) * up_e x_t          [NK, E]
//   moe_units_kernel<down>    y[slot, :]   = down_e act[slot, :]                  [NK, d]
// The weighted combination over a token's K slots (k order) and the shared expert are the
// many-token path's (moe_grouped.cu).  Arithmetic followed: core/moe_cpu.cpp:198-288.
//
// Bound by the engine's instructions (about 85 per 1024 weights with eight tokens, 137 and more before it) and
// by how evenly the units spread: two CTAs per SM share the list of all (unit, tile) pairs in equal contiguous
// ranges, so a unit's tokens are staged by the few CTAs whose range it is in.
// 64 tokens, H-Tiny shape, Q4_K: 54 + 53 us before, 47 + 58 (beside the shared expert) now; Q4_K has a
// faster form since (moe_exact.cu: 38 + 22), the other kinds, whose scales change every 32 of K, have not.
#include "digit_tile.cuh"
#include "gemm.cuh"

namespace b200 {

constexpr int UNIT_SLOTS = 8;        // token columns of the dot engine

struct MoeUnitArgs {
    const float* x = nullptr;            // [T, d] layer input
    const int32_t* grouped = nullptr;    // [NK] slot numbers sorted by expert (slot / K = token)
    const int4* units = nullptr;         // (expert, first sorted position, slots <= 8, -)
    const int* n_units = nullptr;
    const uint8_t *gates = nullptr, *ups = nullptr, *downs = nullptr;
    float* act = nullptr;                // [NK, E], sorted order
    float* y = nullptr;                  // [NK, d], sorted order
    int d = 0, E = 0, K = 0;
    // filled per kernel: rows a tile takes of each of its parts (gate and up: two parts; down: one), tiles per set of
    // stages, warps per tile's contraction
    int part_rows = 8, stage_bytes = 0, G = 1, P = 1;
    uint32_t p_inv = 0, chunks_inv = 0;
    int* status = nullptr;
    bool dry = false;
};

// One block; ne <= 256 experts.
__global__ void moe_units_build_kernel(const int32_t* __restrict__ offsets, int ne, int4* __restrict__ units,
                                       int* __restrict__ n_units) {
    __shared__ int first[257];
    __shared__ int wsum[8];
    const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
    const int lo = e < ne ? offsets[e] : 0, hi = e < ne ? offsets[e + 1] : 0;
    const int chunks = (hi - lo + UNIT_SLOTS - 1) / UNIT_SLOTS;
    int incl = chunks;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int base = 0;
    for (int w = 0; w < warp; ++w) base += wsum[w];
    first[e] = base + incl - chunks;
    if (e == 255) *n_units = base + incl;
    for (int c = 0; c < chunks; ++c)
        units[first[e] + c] = make_int4(e, lo + c * UNIT_SLOTS, min(UNIT_SLOTS, hi - lo - c * UNIT_SLOTS), 0);
}

// Tiles [t0, t1) of one unit.  full / phase: the two stage sets' barriers and how often each was waited for.
template <int KIND, int MT, bool DOWN>
__device__ __forceinline__ bool unit_tiles(const MoeUnitArgs& a, const int4 unit, int t0, int t1, uint8_t* smem, uint64_t* full, int (&phase)[2]) {
    constexpr int W = dg_warps(UNIT_SLOTS), PARTS = DOWN ? 1 : 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int Kd = DOWN ? a.E : a.d, N = DOWN ? a.d : a.E, chunks = dg_chunks(Kd), nsub = Kd >> 5, G = a.G, P = a.P;
    const int e = unit.x, p0 = unit.y, M = unit.z, R = a.part_rows;
    const uint32_t rb = (uint32_t)row_bytes_of(KIND, Kd);
    DgX<KIND, MT> xd;
    xd.carve(smem + 2 * (size_t)G * a.stage_bytes, chunks);
    float* red = reinterpret_cast<float*>(smem + 2 * (size_t)G * a.stage_bytes + ((dg_x_bytes<KIND>(chunks, UNIT_SLOTS) + 15) & ~(size_t)15));
    const int rounds = (t1 - t0 + G - 1) / G;
    auto issue = [&](int r, int set) {
        const int n = min(G, t1 - t0 - r * G);
        uint32_t total = 0;
        for (int i = 0; i < n; ++i) total += PARTS * min(R, N - (t0 + r * G + i) * R) * rb;
        mbar_expect_tx(&full[set], total);
        for (int i = 0; i < n; ++i) {
            const int r0 = (t0 + r * G + i) * R;
            const uint32_t bytes = min(R, N - r0) * rb;
            const int64_t at = ((int64_t)e * N + r0) * rb;
            uint8_t* dst = smem + (size_t)(set * G + i) * a.stage_bytes;
            tma_load_1d(dst, (DOWN ? a.downs : a.gates) + at, bytes, &full[set]);
            if (!DOWN) tma_load_1d(dst + R * rb, a.ups + at, bytes, &full[set]);
        }
    };
    if (threadIdx.x == 0)
        for (int r = 0; r < min(rounds, 2); ++r) issue(r, r);
    for (int i = warp; i < chunks * M; i += W) {
        const int m = dg_div(i, a.chunks_inv), c = i - m * chunks;
        const float* row = DOWN ? a.act + (int64_t)(p0 + m) * a.E : a.x + (int64_t)(a.grouped[p0 + m] / a.K) * a.d;
        float v[8];
        dg_load8<true>(row, c * DG_CHUNK + 8 * lane, Kd, v);
        dg_stage<KIND, MT>(xd, c, m, v, 1.0f, lane);
    }
    __syncthreads();
    const int ga = min(lane >> 2, R - 1), gb = DOWN ? min((lane >> 2) + 8, R - 1) : R + ga;
    bool ok = true;
    for (int r = 0; r < rounds; ++r) {
        const int n = min(G, t1 - t0 - r * G), set = r & 1;
        float* rr = red + (size_t)set * G * P * dg_red_floats(MT);
        ok = ok && mbar_wait(&full[set], phase[set] & 1, a.status);
        ++phase[set];
        if (ok) {
            for (int u = warp; u < n * P; u += W) {
                const int tile = dg_div(u, a.p_inv), part = u - tile * P;
                const uint32_t base = smem_u32(smem) + (set * G + tile) * a.stage_bytes;
                DgAcc<KIND, MT> acc;
                acc.clear();
                for (int c = part; c < chunks; c += P) {
                    const uint32_t at = base + c * dg_row_chunk<KIND>();
                    dg_chunk<KIND, MT>(acc, at + ga * rb, at + gb * rb, xd, c, min(8, nsub - 8 * c), lane);
                }
                dg_finish<KIND, MT>(acc, rr + u * dg_red_floats(MT), lane);
            }
        }
        if (!__syncthreads_and(ok)) break;
        // The next copies and the outputs are the last warps' work: with one tile in six parts two warps have none of
        // the products, and the others go on to the next tile (by the first warps, a round of 1220 cycles of products
        // had 1900 more of this behind it).
        if (threadIdx.x == (W - 1) * 32 && r + 2 < rounds) issue(r + 2, set);
        // (row, token) with the row fastest: neighbouring threads store neighbouring outputs
        const int per = DOWN ? 16 : 8;
        for (int i = (threadIdx.x + 64) & (W * 32 - 1); i < n * per * MT; i += W * 32) {       // 0 at the last two warps' first thread
            const int row = i % per, m = i / per % MT, tile = i / (per * MT), at = (t0 + r * G + tile) * R + row;
            if (m >= M || row >= R || at >= N) continue;
            const float* re = rr + tile * P * dg_red_floats(MT);
            if (DOWN) {
                a.y[(int64_t)(p0 + m) * a.d + at] = dg_value<KIND, MT>(re, P, row, m);
            } else {
                const float g = dg_value<KIND, MT>(re, P, row, m), u = dg_value<KIND, MT>(re, P, row + 8, m);
                a.act[(int64_t)(p0 + m) * a.E + at] = silu_acc(g) * u;
            }
        }
    }
    return ok;
}

template <int KIND, bool DOWN>
__global__ void __launch_bounds__(dg_warps(UNIT_SLOTS) * 32, 2) moe_units_kernel(MoeUnitArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t full[2];
    if (threadIdx.x == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        mbar_fence_init();
    }
    pdl_launch_dependents();
    pdl_wait();                                   // the unit table comes from the kernels before
    __syncthreads();
    const int N = DOWN ? a.d : a.E, tpu = (N + a.part_rows - 1) / a.part_rows;
    const int64_t total = (int64_t)*a.n_units * tpu;
    int64_t t = total * blockIdx.x / gridDim.x;
    const int64_t end = total * (blockIdx.x + 1) / gridDim.x;
    int phase[2] = {0, 0};
    while (t < end) {
        const int u = (int)(t / tpu), t0 = (int)(t - (int64_t)u * tpu), t1 = (int)min((int64_t)tpu, end - (int64_t)u * tpu);
        const int4 unit = a.units[u];
        const bool ok = unit.z <= 2   ? unit_tiles<KIND, 2, DOWN>(a, unit, t0, t1, smem, full, phase)
                        : unit.z <= 4 ? unit_tiles<KIND, 4, DOWN>(a, unit, t0, t1, smem, full, phase)
                                      : unit_tiles<KIND, 8, DOWN>(a, unit, t0, t1, smem, full, phase);
        if (!ok) {
            // no copy of this CTA may be left under way
            if (threadIdx.x == 0)
                for (int s = 0; s < 2; ++s)
                    for (int par = 0; par < 2 && !mbar_wait(&full[s], par, a.status); ++par) {}
            return;
        }
        t += t1 - t0;
        __syncthreads();                          // the staged tokens and sums are free again
    }
}

// Rows of a tile, tiles of a set, warps of a contraction; dynamic shared memory, 0 if the width does not fit.
template <int KIND, bool DOWN>
static size_t plan_units(MoeUnitArgs& a) {
    const int Kd = DOWN ? a.E : a.d, N = DOWN ? a.d : a.E, chunks = dg_chunks(Kd);
    const size_t rb = row_bytes_of(KIND, Kd), x = (dg_x_bytes<KIND>(chunks, UNIT_SLOTS) + 15) & ~(size_t)15;
    if (chunks > 255) return 0;
    for (const size_t budget : {(size_t)SMEM_BUDGET - 1024, (size_t)SMEM_OPT_IN - 1024})        // two CTAs on an SM, or one
        for (int R = DOWN ? 16 : 8; R >= 1; R >>= 1)
            for (int G = 8; G >= 1; G >>= 1) {
                if ((R * rb) % 16 != 0 || ((N % R) * rb) % 16 != 0) continue;
                a.part_rows = R;
                a.G = G;
                a.P = dg_parts(G, chunks, dg_warps(UNIT_SLOTS));
                a.stage_bytes = (int)(((DOWN ? 1 : 2) * R * rb + 127) / 128 * 128);
                const size_t need = 2 * (size_t)G * a.stage_bytes + x + (size_t)2 * G * a.P * dg_red_floats(UNIT_SLOTS) * 4 + 128;
                if (need <= budget) return need;
            }
    return 0;
}
template <int KIND, bool DOWN>
static int launch_units(MoeUnitArgs a) {
    const int Kd = DOWN ? a.E : a.d;
    const size_t smem = plan_units<KIND, DOWN>(a);
    if (!smem) return fail(B200_EUNSUPPORTED, "moe_units: width %d does not fit the shared-memory staging", Kd);
    a.chunks_inv = dg_inv(dg_chunks(Kd));
    a.p_inv = dg_inv(a.P);
    auto kern = moe_units_kernel<KIND, DOWN>;
    static bool configured = false;
    if (!configured) {
        int rc = allow_smem(kern);
        if (rc) return rc;
        configured = true;
    }
    const int per_sm = smem <= (size_t)SMEM_BUDGET ? 2 : 1;
    return launch_pdl(kern, dim3(per_sm * num_sms()), dim3(dg_warps(UNIT_SLOTS) * 32), smem, a);
}
template <int KIND>
static bool units_take(int d, int E) {
    MoeUnitArgs a;
    a.d = d; a.E = E;
    return plan_units<KIND, false>(a) && plan_units<KIND, true>(a);
}
bool moe_units_takes(int d, int E, int kind) {
    switch (kind) {
        case 0: return units_take<0>(d, E);
        case 1: return units_take<1>(d, E);
        case 2: return units_take<2>(d, E);
        case 3: return units_take<3>(d, E);
        case KIND_F16: return units_take<KIND_F16>(d, E);
        default: return false;
    }
}
template <int KIND>
static int moe_units_kind(const MoeUnitArgs& a) {
    const int rc = launch_units<KIND, false>(a);
    return rc ? rc : launch_units<KIND, true>(a);
}

// The routed experts of N tokens whose slots have been sorted by expert: grouped / offsets as
// moe_dispatch_perm leaves them; act [N K, E] and y [N K, d] fp32 in sorted order; units:
// scratch for unit_table_bytes(N K, ne) bytes.  kind: a packed kind or KIND_F16.
size_t moe_units_table_bytes(int64_t NK, int ne) { return ((size_t)(ne + NK / UNIT_SLOTS + 1) * sizeof(int4) + 255) / 256 * 256 + 256; }
int moe_units_forward(const float* x, const int32_t* grouped, const int32_t* offsets, const void* gates, const void* ups,
                      const void* downs, float* act, float* y, void* units_scratch, int64_t N, int d, int E, int ne, int K,
                      int kind) {
    B200_REQUIRE(ne <= 256 && N * K <= 0x7fffffff, "moe_units: too many experts or slots");
    B200_REQUIRE(d % 32 == 0 && E % 32 == 0, "moe_units: d and E must be multiples of 32");
    if (kind == 3) B200_REQUIRE(d % 256 == 0 && E % 256 == 0, "moe_units: Q4_K needs multiples of 256");
    int* n_units = static_cast<int*>(units_scratch);
    int4* units = reinterpret_cast<int4*>(static_cast<char*>(units_scratch) + 256);
    moe_units_build_kernel<<<1, 256, 0, stream()>>>(offsets, ne, units, n_units);
    B200_LAUNCH_CHECK("moe_units_build_kernel");
    MoeUnitArgs a;
    a.x = x; a.grouped = grouped; a.units = units; a.n_units = n_units;
    a.gates = static_cast<const uint8_t*>(gates); a.ups = static_cast<const uint8_t*>(ups);
    a.downs = static_cast<const uint8_t*>(downs);
    a.act = act; a.y = y; a.d = d; a.E = E; a.K = K;
    a.status = stream_status_ptr();
    B200_REQUIRE(a.status, "moe_units: status word allocation failed");
    switch (kind) {
        case 0: return moe_units_kind<0>(a);
        case 1: return moe_units_kind<1>(a);
        case 2: return moe_units_kind<2>(a);
        case 3: return moe_units_kind<3>(a);
        case KIND_F16: return moe_units_kind<KIND_F16>(a);
        default: return fail(B200_EUNSUPPORTED, "moe_units: fp32 experts take the token-major path");
    }
}

}  // namespace b200
