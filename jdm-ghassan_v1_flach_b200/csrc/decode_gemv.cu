// y[M,N] = f(x)[M,K] . W^T for up to eight tokens and packed weights, on the digit engine (digit_tile.cuh).
//
// A decode matrix is a few MB, so a CTA's whole share - two or three tiles of 16 rows - fits its shared memory
// and is on its way by TMA before the previous kernel has ended (griddepcontrol.wait).  After the wait only a
// short chain is left: the token's activations from L2, each warp cutting 256 of them into digits, one barrier,
// the tiles' products with the contraction split over the warps, one barrier, the epilogue.  The RMSNorm
// factor is a scalar of the token and is applied there, so its sum of squares is off that chain.
// Larger shares go round by round through two sets of stages.
// In_proj of the H-Tiny shape ([6448, 1536] Q4_K, one token) in the step's graph: DGSTEP.
#include "digit_tile.cuh"
#include "gemv_epilogue.cuh"

namespace b200 {

template <int KIND, int MT, int PRO, int EPI>
__global__ void __launch_bounds__(DG_THREADS, 2) dg_gemv_kernel(SgArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int G = a.n_stages, P = a.parts, chunks = dg_chunks(a.K), nsub = a.K >> 5;
    DgX<MT> xd;
    uint8_t* p = xd.carve(smem + (size_t)a.sets * G * a.stage_bytes, chunks);
    double* ssq = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15);
    float* inv = reinterpret_cast<float*>(ssq + (PRO == PRO_RMS ? chunks : 1) * MT);
    float* red = inv + 8;
    uint64_t* bar = reinterpret_cast<uint64_t*>(red + 2 * G * P * dg_red_floats(MT));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int first = blockIdx.x, step = gridDim.x;
    const int n_my = first < a.num_tiles ? (a.num_tiles - first + step - 1) / step : 0;
    const int rounds = (n_my + G - 1) / G;

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
    auto issue = [&](int r) {                                         // one thread: the copies of round r
        const int n = min(G, n_my - r * G), set = a.sets == 1 ? 0 : r & 1;
        uint32_t total = 0;
        for (int i = 0; i < n; ++i) {
            const Seg s = seg_of(first + (r * G + i) * step);
            total += (uint32_t)(min(a.rows_per_tile, s.N - s.r0) * a.row_bytes);
        }
        mbar_expect_tx(&bar[set], total);
        for (int i = 0; i < n; ++i) {
            const Seg s = seg_of(first + (r * G + i) * step);
            tma_load_1d(smem + (size_t)(set * G + i) * a.stage_bytes, s.w + (int64_t)s.r0 * a.row_bytes,
                        (uint32_t)(min(a.rows_per_tile, s.N - s.r0) * a.row_bytes), &bar[set]);
        }
    };
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_fence_init();
        for (int r = 0; r < min(rounds, 2); ++r) issue(r);            // the weights do not depend on the previous kernel
    }
    pdl_launch_dependents();
    float nw[8];
    if (PRO == PRO_RMS) dg_load8(a.norm_w, (warp % chunks) * DG_CHUNK + 8 * lane, a.K, nw);
    pdl_wait();

    for (int i = warp; i < chunks * a.M; i += DG_WARPS) {
        const int m = i / chunks, c = i - m * chunks;
        float v[8];
        dg_load8(a.x + (int64_t)m * a.x_stride, c * DG_CHUNK + 8 * lane, a.K, v);
        if (PRO == PRO_RMS) {
            if (i != warp || c != warp % chunks) dg_load8(a.norm_w, c * DG_CHUNK + 8 * lane, a.K, nw);
            double ss = 0.0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                ss += (double)v[j] * (double)v[j];
                v[j] *= nw[j];
            }
            dg_stage<KIND, MT>(xd, c, m, v, 1.0f, lane);
            ss = warp_sum_d(ss);
            if (lane == 0) ssq[c * MT + m] = ss;
        } else {
            dg_stage<KIND, MT>(xd, c, m, v, 1.0f, lane);
        }
    }
    if (PRO != PRO_RMS && a.in_partials) {
        for (int m = DG_WARPS - 1 - warp; m < a.M; m += DG_WARPS) {
            double t = 0.0;
            for (int i = lane; i < a.n_partials; i += 32) t += a.in_partials[(int64_t)m * a.n_partials + i];
            t = warp_sum_d(t);
            if (lane == 0) inv[m] = 1.0f / sqrtf((float)(t / (double)a.in_dim) + a.eps);
        }
    }
    __syncthreads();
    if (PRO == PRO_RMS) {
        if (warp == DG_WARPS - 1 && lane < a.M) {
            double ss = 0.0;
            for (int c = 0; c < chunks; ++c) ss += ssq[c * MT + lane];
            const double d = 1.0 / sqrt(ss / (double)a.K + (double)a.eps);
            inv[lane] = isfinite(d) ? (float)d : 0.0f;
        }
    } else if (!a.in_partials) {
        if (threadIdx.x < 8) inv[threadIdx.x] = 1.0f;
    }

    bool ok = true;
    for (int r = 0; r < rounds; ++r) {
        const int n = min(G, n_my - r * G), set = a.sets == 1 ? 0 : r & 1;
        float* rr = red + (size_t)(r & 1) * G * P * dg_red_floats(MT);
        // element (tile, row, token) this thread finishes first: its operands before the products
        auto element = [&](int e, Seg& s, int& n_out, int& m) {
            m = e % MT;
            const int row = e / MT % 16;
            s = seg_of(first + (r * G + e / (16 * MT)) * step);
            n_out = s.r0 + row;
            return m < a.M && row < a.rows_per_tile && n_out < s.N;
        };
        GemvEpilogue<EPI> epi;
        Seg s0;
        int n0 = 0, m0 = 0;
        const bool own = (int)threadIdx.x < n * 16 * MT && element(threadIdx.x, s0, n0, m0);
        if (own) epi.prefetch(a, n0, m0);
        ok = ok && mbar_wait(&bar[set], (a.sets == 1 ? r : r >> 1) & 1, a.status);
        if (ok) {
            for (int u = warp; u < n * P; u += DG_WARPS) {
                const int tile = u / P, part = u - tile * P;
                const uint32_t base = smem_u32(smem) + (set * G + tile) * a.stage_bytes;
                const int ra = min(lane >> 2, a.rows_per_tile - 1), rb = min((lane >> 2) + 8, a.rows_per_tile - 1);
                DgAcc<MT> acc;
                acc.clear();
                for (int c = part; c < chunks; c += P) {
                    const uint32_t at = base + c * (DG_CHUNK / q_block_elems(KIND)) * q_block_bytes(KIND);
                    dg_chunk<KIND, MT>(acc, at + ra * (uint32_t)a.row_bytes, at + rb * (uint32_t)a.row_bytes, xd, c, min(8, nsub - 8 * c), lane);
                }
                dg_finish<KIND, MT>(acc, rr + u * dg_red_floats(MT), lane);
            }
        }
        if (!__syncthreads_and(ok)) break;
        if (threadIdx.x == 0 && r + 2 < rounds) issue(r + 2);
        for (int e = threadIdx.x; e < n * 16 * MT; e += DG_THREADS) {
            const float* re = rr + e / (16 * MT) * P * dg_red_floats(MT);
            const int row = e / MT % 16, m = e % MT;
            if (e == (int)threadIdx.x) {
                if (own) epi.finish(a, n0, m0, dg_value<KIND, MT>(re, P, row, m) * inv[m], s0.y, s0.y_stride);
            } else {
                GemvEpilogue<EPI> ep;
                Seg s;
                int nn, mm;
                if (!element(e, s, nn, mm)) continue;
                ep.prefetch(a, nn, mm);
                ep.finish(a, nn, mm, dg_value<KIND, MT>(re, P, row, m) * inv[m], s.y, s.y_stride);
            }
        }
    }
    // a wait that ran out: no copy of this CTA may be left under way
    if (!ok && threadIdx.x == 0)
        for (int set = 0; set < a.sets; ++set)
            for (int par = 0; par < 2 && !mbar_wait(&bar[set], par, a.status); ++par) {}
}

// Warps per tile's contraction: fewest passes of the eight warps over `tiles` tiles, ties to fewer parts.
static int dg_parts(int tiles, int chunks) {
    int best = 1, cost = 1 << 30;
    for (int p = 1; p <= std::min(chunks, DG_WARPS); ++p) {
        const int c = ceil_div(tiles * p, DG_WARPS) * ceil_div(chunks, p);
        if (c < cost) { cost = c; best = p; }
    }
    return best;
}

template <int KIND, int MT, int PRO, int EPI>
static int launch_dg(SgArgs a) {
    const int chunks = dg_chunks(a.K);
    const size_t fixed = dg_x_bytes(chunks, MT) + 16 + (size_t)(PRO == PRO_RMS ? chunks : 1) * MT * 8 + 32 + 16 + 128;
    int grid = 0;
    size_t smem = 0;
    // Rows per tile: 16, fewer only for rows so wide that a tile would not fit.  Stages: the CTA's whole
    // share when it fits half an SM (the next kernel's CTA fits beside it and streams early), else as much
    // as does, twice; a whole SM only when half of one holds less than that.
    for (int R = TILE_ROWS; R >= 1 && !smem; R >>= 1) {
        if ((R * a.row_bytes) % 16 != 0) break;
        a.rows_per_tile = R;
        a.t1 = ceil_div(a.N, R);
        a.t2 = a.t1 + ceil_div(a.N2, R);
        a.num_tiles = a.t2 + ceil_div(a.N3, R);
        a.stage_bytes = (int)((R * a.row_bytes + 127) / 128 * 128);
        grid = std::min(a.num_tiles, num_sms());
        const int share = ceil_div(a.num_tiles, grid);
        for (const size_t budget : {(size_t)SMEM_BUDGET, (size_t)SMEM_BUDGET_FULL}) {
            for (int G = std::min(share, 8); G >= 1 && !smem; --G) {
                a.n_stages = G;
                a.sets = G >= share ? 1 : 2;
                a.parts = dg_parts(G, chunks);
                const size_t need = (size_t)a.sets * G * a.stage_bytes + fixed + (size_t)2 * G * a.parts * dg_red_floats(MT) * 4;
                if (need <= budget) smem = need;
            }
            if (smem) break;
        }
    }
    if (!smem) return fail(B200_EUNSUPPORTED, "stream_gemv: K = %d does not fit the shared-memory staging", a.K);
    auto kern = dg_gemv_kernel<KIND, MT, PRO, EPI>;
    static bool configured = false;
    if (!configured) {
        int rc = allow_smem(kern);
        if (rc) return rc;
        configured = true;
    }
    return launch_pdl(kern, dim3(grid), dim3(DG_THREADS), smem, a);
}

template <int KIND, int PRO, int EPI>
static int launch_dg_mt(const SgArgs& a) {
    if (a.M == 1) return launch_dg<KIND, 1, PRO, EPI>(a);
    if (a.M == 2) return launch_dg<KIND, 2, PRO, EPI>(a);
    if (a.M <= 4) return launch_dg<KIND, 4, PRO, EPI>(a);
    return launch_dg<KIND, 8, PRO, EPI>(a);
}
template <int KIND>
static int launch_dg_kind(const SgArgs& a, int pro, int epi) {
    if (pro == PRO_RMS && epi == EPI_STORE) return launch_dg_mt<KIND, PRO_RMS, EPI_STORE>(a);
    if (pro == PRO_RMS && epi == EPI_INPROJ) return launch_dg_mt<KIND, PRO_RMS, EPI_INPROJ>(a);
    if (pro == PRO_NONE && epi == EPI_RESIDUAL) return launch_dg_mt<KIND, PRO_NONE, EPI_RESIDUAL>(a);
    if (pro == PRO_NONE && epi == EPI_STORE) return launch_dg_mt<KIND, PRO_NONE, EPI_STORE>(a);
    return fail(B200_EINVAL, "stream_gemv: unsupported prologue/epilogue pair");
}

// stream_gemv() for packed weights (kind 0 .. 3); arguments checked there.
int digit_gemv(SgArgs a, int kind, int pro, int epi) {
    if ((reinterpret_cast<uintptr_t>(a.x) & 15) != 0 || (a.x_stride & 3) != 0 || (reinterpret_cast<uintptr_t>(a.norm_w) & 15) != 0)
        return fail(B200_EUNSUPPORTED, "stream_gemv: activations must be 16-byte aligned");
    switch (kind) {
        case 0: return launch_dg_kind<0>(a, pro, epi);
        case 1: return launch_dg_kind<1>(a, pro, epi);
        case 2: return launch_dg_kind<2>(a, pro, epi);
        default: return launch_dg_kind<3>(a, pro, epi);
    }
}

}  // namespace b200
