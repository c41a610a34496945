// y[M,N] = f(x)[M,K] . W^T for up to eight tokens and packed weights, on the digit engine (digit_tile.cuh).
//
// A decode matrix is a few MB, so a CTA's whole share - two or three tiles of 16 rows - fits its shared memory
// and is on its way by TMA before the previous kernel has ended (griddepcontrol.wait).  After the wait only a
// short chain is left: the token's activations from L2, each warp cutting 256 of them into digits, one barrier,
// the tiles' products with the contraction split over the warps, one barrier, the epilogue.  The RMSNorm
// factor is a scalar of the token and is applied there, so its sum of squares is off that chain.
// Larger shares go round by round through two sets of stages.
// In_proj of the H-Tiny shape ([6448, 1536] Q4_K, one token) in the step's graph:
// 7.6 us before, 4.5 now, of which 1.5 are the hand-over between the two launches.
#include "digit_tile.cuh"
#include "gemv_epilogue.cuh"

namespace b200 {

constexpr int DG_MAX_SETS = 4;
constexpr size_t DG_SMEM_MAX = 224 * 1024;
constexpr size_t DG_SMEM_TWO = SMEM_BUDGET - 128;     // of two CTAs on an SM: the kernel's static variables come on top
constexpr size_t DG_SMEM_THIRD = 77 * 1024;           // from here on a third CTA does not fit

template <int KIND, int MT, int PRO, int EPI>
__global__ void __launch_bounds__(dg_warps(MT) * 32, 2) dg_gemv_kernel(SgArgs a) {
    constexpr int W = dg_warps(MT), ELEMS = 16 * MT;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t bar[DG_MAX_SETS];
    __shared__ float inv[8];
    const int G = a.n_stages, P = a.parts, chunks = dg_chunks(a.K), nsub = a.K >> 5;
    DgX<KIND, MT> xd;
    uint8_t* p = xd.carve(smem + (size_t)a.sets * G * a.stage_bytes, chunks);
    double* ssq = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15);
    float* red = reinterpret_cast<float*>(ssq + (PRO == PRO_RMS ? chunks : 0) * MT);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int first = blockIdx.x, step = gridDim.x;
    const int n_my = a.share + (first < a.share_rem ? 1 : 0);        // tiles of this CTA
    const int rounds = a.sets == 1 ? 1 : (n_my + G - 1) / G;

    // tile -> matrix of the launch, first row
    struct Seg { const uint8_t* w; float* y; int N, y_stride, r0; };
    auto seg_of = [&](int tile) {
        Seg s{a.w, a.y, a.N, a.y_stride, tile * a.rows_per_tile};
        if (EPI == EPI_STORE && tile >= a.t1) {
            const bool third = tile >= a.t2;
            s = Seg{third ? a.w3 : a.w2, third ? a.y3 : a.y2, third ? a.N3 : a.N2, third ? a.y3_stride : a.y2_stride,
                    (tile - (third ? a.t2 : a.t1)) * a.rows_per_tile};
        }
        return s;
    };
    auto issue = [&](int r, int set) {                                // one thread: the copies of round r
        const int n = min(G, n_my - r * G);
        uint32_t total = 0;
        for (int i = 0; i < n; ++i) {
            const Seg s = seg_of(first + (r * G + i) * step);
            total += (uint32_t)(min(a.rows_per_tile, s.N - s.r0) * (int)a.row_bytes);
        }
        mbar_expect_tx(&bar[set], total);
        for (int i = 0; i < n; ++i) {
            const Seg s = seg_of(first + (r * G + i) * step);
            tma_load_1d(smem + (size_t)(set * G + i) * a.stage_bytes, s.w + (int64_t)s.r0 * a.row_bytes,
                        (uint32_t)(min(a.rows_per_tile, s.N - s.r0) * (int)a.row_bytes), &bar[set]);
        }
    };
    if (threadIdx.x == 0) {
        for (int i = 0; i < a.sets; ++i) mbar_init(&bar[i], 1);
        mbar_fence_init();
        for (int r = 0; r < min(rounds, a.sets); ++r) issue(r, r);    // the weights do not depend on the previous kernel
    }
    pdl_launch_dependents();
    // element e of round r: token, output row; false when it does not exist
    auto element = [&](int r, int e, Seg& s, int& n_out, int& m) {
        m = e % MT;
        const int row = e / MT % 16;
        s = seg_of(first + (r * G + e / ELEMS) * step);
        n_out = s.r0 + row;
        return m < a.M && row < a.rows_per_tile && n_out < s.N;
    };
    // This thread's first element of round 0: what its epilogue reads is under way before the products.  The
    // convolution's window and taps are older than the previous kernel, the residual stream is not.
    GemvEpilogue<EPI> epi;
    Seg s0;
    int n0 = 0, m0 = 0;
    const bool own = (int)threadIdx.x < min(G, n_my) * ELEMS && element(0, threadIdx.x, s0, n0, m0);
    if (EPI == EPI_INPROJ && own) epi.prefetch(a, n0, m0);
    float nw[8];
    if (PRO == PRO_RMS) {
        const int c = MT == 1 ? warp : warp - dg_div(warp, a.chunks_inv) * chunks;
        dg_norm8(a.norm_w, c * DG_CHUNK + 8 * lane, a.K, nw);
    }
    pdl_wait();

    if (EPI == EPI_RESIDUAL && own) epi.prefetch(a, n0, m0);
    if (PRO != PRO_RMS && a.in_partials) {
        // the gated norm's factors from the state update's partial sums, by warps that stage least
        for (int m = W - 1 - warp; m < a.M; m += W) {
            const double* q = a.in_partials + (int64_t)m * a.n_partials;
            double t = 0.0;
            for (int i0 = 0; i0 < a.n_partials; i0 += 512) {
                double v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = i0 + 32 * i + lane < a.n_partials ? __ldcg(q + i0 + 32 * i + lane) : 0.0;
#pragma unroll
                for (int i = 0; i < 16; ++i) t += v[i];
            }
            t = warp_sum_d(t);
            if (lane == 0) inv[m] = 1.0f / sqrtf((float)(t / (double)a.in_dim) + a.eps);
        }
    }
    constexpr int B = dg_batch(MT);
    const int all = chunks * a.M;
    for (int i0 = warp; i0 < all; i0 += B * W) {
        float v[B][8], nv[B][8];
#pragma unroll
        for (int q = 0; q < B; ++q) {
            const int i = i0 + q * W, m = MT == 1 ? 0 : dg_div(i, a.chunks_inv), c = i - m * chunks;
            if (i >= all) break;
            dg_load8<true>(a.x + (int64_t)m * a.x_stride, c * DG_CHUNK + 8 * lane, a.K, v[q]);
            if (PRO == PRO_RMS && (q > 0 || i0 != warp)) dg_norm8(a.norm_w, c * DG_CHUNK + 8 * lane, a.K, nv[q]);
        }
#pragma unroll
        for (int q = 0; q < B; ++q) {
            const int i = i0 + q * W, m = MT == 1 ? 0 : dg_div(i, a.chunks_inv), c = i - m * chunks;
            if (i >= all) break;
            if (PRO == PRO_RMS) {
                double ss = 0.0;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    ss += (double)v[q][j] * (double)v[q][j];
                    v[q][j] *= q == 0 && i0 == warp ? nw[j] : nv[q][j];
                }
                dg_stage<KIND, MT>(xd, c, m, v[q], 1.0f, lane);
                ss = warp_sum_d(ss);
                if (lane == 0) ssq[c * MT + m] = ss;
            } else {
                dg_stage<KIND, MT>(xd, c, m, v[q], 1.0f, lane);
            }
        }
    }
    __syncthreads();
    if (PRO == PRO_RMS) {
        if (warp == W - 1 && lane < a.M) {
            double ss = 0.0;
            for (int c = 0; c < chunks; ++c) ss += ssq[c * MT + lane];
            const double d = 1.0 / sqrt(ss / (double)a.K + (double)a.eps);
            inv[lane] = isfinite(d) ? (float)d : 0.0f;
        }
    } else if (!a.in_partials) {
        if (threadIdx.x < 8) inv[threadIdx.x] = 1.0f;
    }

    const uint32_t ra = min(lane >> 2, a.rows_per_tile - 1) * (uint32_t)a.row_bytes, rb = min((lane >> 2) + 8, a.rows_per_tile - 1) * (uint32_t)a.row_bytes;
    for (int r = 0, set = 0, parity = 0; r < rounds; ++r) {
        const int n = min(G, n_my - r * G);
        float* rr = red + (size_t)(r & 1) * G * P * dg_red_floats(MT);
        if (r > 0 && EPI == EPI_RESIDUAL && (int)threadIdx.x < n * ELEMS && element(r, threadIdx.x, s0, n0, m0)) epi.prefetch(a, n0, m0);
        const bool ok = mbar_wait(&bar[set], parity, a.status);
        if (ok) {
            for (int u = warp; u < n * P; u += W) {
                const int tile = dg_div(u, a.parts_inv), part = u - tile * P;
                const uint32_t base = smem_u32(smem) + (set * G + tile) * a.stage_bytes;
                DgAcc<KIND, MT> acc;
                acc.clear();
                for (int c = part; c < chunks; c += P) {
                    const uint32_t at = base + c * dg_row_chunk<KIND>();
                    dg_chunk<KIND, MT>(acc, at + ra, at + rb, xd, c, min(8, nsub - 8 * c), lane);
                }
                dg_finish<KIND, MT>(acc, rr + u * dg_red_floats(MT), lane);
            }
        }
        if (!__syncthreads_and(ok)) {
            // a wait that ran out: no copy of this CTA may be left under way
            if (threadIdx.x == 0)
                for (int t = 0; t < min(a.sets, rounds); ++t)
                    for (int par = 0; par < 2 && !mbar_wait(&bar[t], par, a.status); ++par) {}
            break;
        }
        if (threadIdx.x == 0 && r + a.sets < rounds) issue(r + a.sets, set);
        for (int e = threadIdx.x; e < n * ELEMS; e += W * 32) {
            const float* re = rr + e / ELEMS * P * dg_red_floats(MT);
            const int row = e / MT % 16, m = e % MT;
            const bool fetched = e == (int)threadIdx.x && (r == 0 || EPI == EPI_RESIDUAL);
            if (!element(r, e, s0, n0, m0)) continue;
            if (!fetched) epi.prefetch(a, n0, m0);
            epi.finish(a, n0, m0, dg_value<KIND, MT>(re, P, row, m) * inv[m], s0.y, s0.y_stride);
        }
        if (++set == a.sets) {
            set = 0;
            parity ^= 1;
        }
    }
}

// Warps per tile's contraction: fewest passes of the warps over `tiles` tiles, ties to fewer parts.
int dg_parts(int tiles, int chunks, int warps) {
    int best = 1, cost = 1 << 30;
    for (int p = 1; p <= std::min(chunks, warps); ++p) {
        const int c = ceil_div(tiles * p, warps) * ceil_div(chunks, p);
        if (c < cost) { cost = c; best = p; }
    }
    return best;
}

// A launch's CTAs and their dynamic shared memory (0: K does not fit); fills the tiling of a.  plain: a product by itself,
// without the norm or the epilogues of a decode step.
struct DgPlan { int grid = 0; size_t smem = 0; };
template <int KIND>
static DgPlan dg_plan(SgArgs& a, int mt, bool norm, bool plain) {
    const int chunks = dg_chunks(a.K);
    DgPlan plan;
    if (chunks > 255) return plan;
    a.chunks_inv = dg_inv(chunks);
    const size_t fixed = dg_x_bytes<KIND>(chunks, mt) + 16 + (size_t)(norm ? chunks : 0) * mt * 8 + 128;
    // Rows per tile: 16, fewer only for rows so wide that a tile would not fit.  Stages: the CTA's whole
    // share when it fits half an SM (the next kernel's CTA fits beside it and streams early), else two sets of
    // as much as does; a whole SM for long shares (an fp16 lm_head: two sets of two tiles, whose products take
    // less time than their 98 KB - one tile at a time, the barriers between them held the stream at 4.3 TB/s).
    auto tile = [&](int R, int ctas) {
        a.rows_per_tile = R;
        a.t1 = ceil_div(a.N, R);
        a.t2 = a.t1 + ceil_div(a.N2, R);
        a.num_tiles = a.t2 + ceil_div(a.N3, R);
        a.stage_bytes = (int)((R * a.row_bytes + 127) / 128 * 128);
        plan.grid = std::min(a.num_tiles, ctas);
        a.share = a.num_tiles / plan.grid;
        a.share_rem = a.num_tiles % plan.grid;
        return ceil_div(a.num_tiles, plan.grid);
    };
    auto fits = [&](int G, int sets, size_t budget) {
        a.n_stages = G;
        a.sets = sets;
        a.parts = dg_parts(G, chunks, dg_warps(mt));
        a.parts_inv = dg_inv(a.parts);
        const size_t need = (size_t)sets * G * a.stage_bytes + fixed + (size_t)2 * G * a.parts * dg_red_floats(mt) * 4;
        if (need > budget) return false;
        plan.smem = need;
        return true;
    };
    auto half = [&](int most, size_t budget) {
        if (most > 8 || fits(most, 1, budget)) return;
        for (int G = std::min(most - 1, 4); G >= 1 && !plan.smem; --G) fits(G, 2, budget);
    };
    // From three tokens on the products outweigh the hand-over and two CTAs share an SM, where two of them fit: else the
    // grid is two waves, which both stage all activations, and no CTA of the next kernel is set up beside them.  A step of 3, 5 and 8
    // sequences with one CTA an SM and with two: H-Tiny in Q4_K 1611 / 1586, 2236 / 2160 and 2817 / 2740 us, in Q8_0 1878 / 1836, 2755 /
    // 2596 and 3405 / 3254, the small model in Q4_K 268 / 261, 310 / 306 and 351 / 346.  They do not fit (us a call in a row):
    // 2560 -> 10448, 5 tokens 11.7 / 14.6; 4096 -> 16768, 8 tokens 25.2 / 31.2, in Q8_0 64.7 / 69.3.
    // Products by themselves keep one CTA an SM where its share is one set in half an SM, beside which the next call fetches its
    // weights: from a graph, on other weights each, 1536 -> 6448 in Q4_K, 3, 5, 8 tokens 4.4 / 5.1, 5.9 / 7.1, 6.7 / 8.0; 768 -> 3224 in
    // Q8_0, 5 tokens 3.7 / 4.2.  A share that does not fit so: 2560 -> 10448 in Q4_K, 3 tokens 10.6 / 9.0; 512 -> 24000, 5 tokens 7.3 / 6.4.
    const bool whole = (TILE_ROWS * a.row_bytes) % 16 == 0;
    if (plain && whole) {
        const int most = tile(TILE_ROWS, num_sms());
        if (most <= 8) fits(most, 1, SMEM_BUDGET);
    }
    if (KIND != KIND_F16 && mt > 2 && whole && !plan.smem) half(tile(TILE_ROWS, 2 * num_sms()), DG_SMEM_TWO);
    for (int R = TILE_ROWS; R >= 1 && !plan.smem; R >>= 1) {
        if ((R * a.row_bytes) % 16 != 0) break;
        const int most = tile(R, num_sms());
        half(most, SMEM_BUDGET);
        for (int G = std::min(most, 4); G >= 2 && !plan.smem; --G) fits(G, most > G ? 2 : 1, DG_SMEM_MAX);
        // (one set holds a whole share or nothing: a share of several rounds takes two at least, at half the rows if it must)
        for (int sets = std::min(most, DG_MAX_SETS); sets >= std::min(most, 2) && !plan.smem; --sets) fits(1, sets, DG_SMEM_MAX);
    }
    return plan;
}

template <int KIND, int MT, int PRO, int EPI>
static int launch_dg(SgArgs a) {
    const DgPlan plan = dg_plan<KIND>(a, MT, PRO == PRO_RMS, PRO == PRO_NONE && EPI == EPI_STORE);
    if (!plan.smem) return fail(B200_EUNSUPPORTED, "stream_gemv: K = %d does not fit the shared-memory staging", a.K);
    auto kern = dg_gemv_kernel<KIND, MT, PRO, EPI>;
    // Where the instance's registers let a third CTA on an SM (56 of twelve warps), the CTAs of two kernels crowd on some SMs while others
    // have none: two tokens, 1536 -> 1536 in Q8_0 4.3 us with three, 3.7 with two; 3072 -> 1536 in Q4_0 7.4 and 5.9; a step of H-Tiny in
    // Q8_0, one sequence 1587 and 1541.  Shared memory that it does not use keeps it out.
    static size_t least = 0;
    static bool configured = false;
    if (!configured) {
        int rc = allow_smem(kern);
        if (rc) return rc;
        cudaFuncAttributes at;
        B200_CUDA(cudaFuncGetAttributes(&at, kern));
        if (3 * dg_warps(MT) * 32 * ((at.numRegs + 7) / 8 * 8) <= 65536) least = DG_SMEM_THIRD;
        configured = true;
    }
    return launch_pdl(kern, dim3(plan.grid), dim3(dg_warps(MT) * 32), std::max(plan.smem, least), a);
}

template <int KIND, int PRO, int EPI>
static int launch_dg_mt(const SgArgs& a) {
    switch (dg_tokens(a.M)) {
        case 1: return launch_dg<KIND, 1, PRO, EPI>(a);
        case 2: return launch_dg<KIND, 2, PRO, EPI>(a);
        case 4: return launch_dg<KIND, 4, PRO, EPI>(a);
        default: return launch_dg<KIND, 8, PRO, EPI>(a);
    }
}
template <int KIND>
static int launch_dg_kind(const SgArgs& a, int pro, int epi) {
    if (pro == PRO_RMS && epi == EPI_STORE) return launch_dg_mt<KIND, PRO_RMS, EPI_STORE>(a);
    if (pro == PRO_RMS && epi == EPI_INPROJ) return launch_dg_mt<KIND, PRO_RMS, EPI_INPROJ>(a);
    if (pro == PRO_NONE && epi == EPI_RESIDUAL) return launch_dg_mt<KIND, PRO_NONE, EPI_RESIDUAL>(a);
    if (pro == PRO_NONE && epi == EPI_STORE) return launch_dg_mt<KIND, PRO_NONE, EPI_STORE>(a);
    return fail(B200_EINVAL, "stream_gemv: unsupported prologue/epilogue pair");
}

// stream_gemv() for packed and fp16 weights; arguments checked there.
int digit_gemv(SgArgs a, int kind, int pro, int epi) {
    if ((reinterpret_cast<uintptr_t>(a.x) & 15) != 0 || (a.x_stride & 3) != 0)
        return fail(B200_EUNSUPPORTED, "stream_gemv: activations must be 16-byte aligned");
    switch (kind) {
        case 0: return launch_dg_kind<0>(a, pro, epi);
        case 1: return launch_dg_kind<1>(a, pro, epi);
        case 2: return launch_dg_kind<2>(a, pro, epi);
        case 3: return launch_dg_kind<3>(a, pro, epi);
        default: return launch_dg_kind<KIND_F16>(a, pro, epi);
    }
}

}  // namespace b200

// The launch of one matrix's product as it would be planned, for tests: CTAs and dynamic shared memory of a CTA.
extern "C" int b200_digit_gemv_plan(int kind, int M, int N, int K, int norm, int plain, int* ctas, int* smem) {
    using namespace b200;
    SgArgs a;
    a.M = M;
    a.N = N;
    a.K = K;
    a.row_bytes = row_bytes_of(kind, K);
    const int mt = dg_tokens(M);
    const DgPlan plan = kind == KIND_F16 ? dg_plan<KIND_F16>(a, mt, norm, plain) : dg_plan<0>(a, mt, norm, plain);
    *ctas = plan.grid;
    *smem = (int)plan.smem;
    return plan.smem ? B200_OK : B200_EUNSUPPORTED;
}
