// Fused decode-step kernels, part 1: the streamed single-matrix GEMV (RMSNorm
// prologue; store / residual / Mamba in_proj+conv epilogues) for fp32 weights - fp16 and
// packed ones run on the digit engine (decode_gemv.cu) - and the Mamba-2 state update that
// also emits the gated-norm statistics.
//
// These fuse across the reference's op boundaries (rmsnorm_forward -> linear ->
// add_inplace in Generator::decode_step_logits, inference/generator.cpp:253-436),
// so they are reached only through the decoder's fused mode; the per-op C ABI keeps
// the reference's granularity.  All kernels are launched with programmatic
// dependent launch: barrier set-up, weight streaming and parameter prefetch run
// before griddepcontrol.wait and overlap the predecessor's tail.
#include "fused_common.cuh"
#include "gemv_epilogue.cuh"

namespace b200 {

static int* g_status_dev = nullptr;
int* stream_status_ptr() {
    if (!g_status_dev) {
        if (cudaMalloc(&g_status_dev, 256) != cudaSuccess) return nullptr;
        cudaMemset(g_status_dev, 0, 256);
    }
    return g_status_dev;
}
int stream_status_check(const char* who) {
    if (!g_status_dev) return B200_OK;
    int h = 0;
    B200_CUDA(cudaMemcpy(&h, g_status_dev, 4, cudaMemcpyDeviceToHost));
    if (h != 0) {
        cudaMemset(g_status_dev, 0, 4);
        return fail(B200_ECUDA, "%s: a bounded wait inside a streaming kernel ran out (status %d)", who, h);
    }
    return B200_OK;
}

// ===========================================================================
// streamed GEMV: y[M,N] = f(x)[M,K] . W^T, M <= 8
// ===========================================================================
template <int KIND, int MT, int PRO, int EPI>
__global__ void __launch_bounds__(SG_THREADS, 2) stream_gemv_kernel(SgArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    Ring ring;
    ring.stages = smem;
    ring.stage_bytes = a.stage_bytes;
    ring.n_stages = a.n_stages;
    ring.status = a.status;
    XAct xa;
    uint8_t* p = xact_carve<KIND>(xa, smem + (size_t)a.n_stages * a.stage_bytes, a.K, MT, PRO == PRO_RMS);
    float* nw_s = reinterpret_cast<float*>(p);                      // [K] when PRO_RMS
    p += (PRO == PRO_RMS ? (size_t)a.K * 4 : 0);
    float* red = reinterpret_cast<float*>(p);
    p += (size_t)RED_FLOATS * 4;
    ring.full = reinterpret_cast<uint64_t*>(p);
    ring.empty = ring.full + SG_MAX_STAGES;
    double* red_d = reinterpret_cast<double*>(ring.empty + SG_MAX_STAGES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int first = blockIdx.x, step = gridDim.x;
    const int n_my = first < a.num_tiles ? (a.num_tiles - first + step - 1) / step : 0;
    ring.init();
    if (threadIdx.x == 0) pdl_launch_dependents();

    if (warp == SG_CONSUMERS) {
        // producer: the weights do not depend on the previous kernel - start at once
        if (lane == 0) {
            int issued = 0;
            for (int i = 0; i < n_my; ++i) {
                if (!ring.acquire(i)) break;
                int tile = first + i * step;
                const uint8_t* wseg = a.w;
                int nseg = a.N;
                if (EPI == EPI_STORE && tile >= a.t1) {       // second / third matrix of the launch
                    const bool third = tile >= a.t2;
                    wseg = third ? a.w3 : a.w2;
                    nseg = third ? a.N3 : a.N2;
                    tile -= third ? a.t2 : a.t1;
                }
                const int rows = min(a.rows_per_tile, nseg - tile * a.rows_per_tile);
                const uint32_t bytes = (uint32_t)(rows * a.row_bytes);
                ring.expect(i, bytes);
                ring.copy(i, 0, wseg + (int64_t)tile * a.rows_per_tile * a.row_bytes, bytes);
                issued = i + 1;
            }
            ring.drain(issued);
        }
        return;
    }

    // consumers: everything independent of the previous kernel first
    if (PRO == PRO_RMS)
        for (int k = threadIdx.x; k < a.K; k += SG_CTHREADS) nw_s[k] = a.norm_w[k];
    xact_zero_row<KIND>(xa);
    pdl_wait();
    // element (row, token) this thread finishes
    const int e_row = threadIdx.x >> 3, e_m = threadIdx.x & 7;
    float in_scale = 1.0f;
    for (int m = 0; m < a.M; ++m) {
        const float* xm = a.x + (int64_t)m * a.x_stride;
        if (a.in_partials) {
            // gated-norm statistic: inv = 1/sqrt(mean + eps) from the scan kernel's block
            // partial sums, reduced together with the activation staging
            double t = 0.0;
            for (int i = threadIdx.x; i < a.n_partials; i += SG_CTHREADS) t += a.in_partials[(int64_t)m * a.n_partials + i];
            t = stage_x<KIND, PRO == PRO_RMS, true>(xm, nw_s, xa, m, a.eps, red_d, t) / (double)a.in_dim;
            if (e_m == m) in_scale = 1.0f / sqrtf((float)t + a.eps);
        } else {
            stage_x<KIND, PRO == PRO_RMS, false>(xm, nw_s, xa, m, a.eps, red_d, 0.0);
        }
    }

    for (int i = 0; i < n_my; ++i) {
        int tile = first + i * step;
        int nseg = a.N;
        float* yseg = a.y;
        int ystride = a.y_stride;
        if (EPI == EPI_STORE && tile >= a.t1) {
            const bool third = tile >= a.t2;
            nseg = third ? a.N3 : a.N2;
            yseg = third ? a.y3 : a.y2;
            ystride = third ? a.y3_stride : a.y2_stride;
            tile -= third ? a.t2 : a.t1;
        }
        const int rows = min(a.rows_per_tile, nseg - tile * a.rows_per_tile);
        const int n = tile * a.rows_per_tile + e_row;
        const bool owner = e_row < rows && e_m < a.M;
        // epilogue operands are fetched before the dot products so their latency hides
        GemvEpilogue<EPI> epi;
        if (owner) epi.prefetch(a, n, e_m);
        if (!ring.wait_full(i)) break;
        float* red_pass = red + (size_t)(i & 1) * RED_BUF;
        tile_compute<KIND, MT>(ring.stage(i), a.row_bytes, rows, a.K, xa, 0, a.M, red_pass, warp, lane);
        ring.release(i);
        consumer_sync();
        if (owner) {
            epi.finish(a, n, e_m, red_value<KIND>(red_pass, e_row, e_m) * in_scale, yseg, ystride);
        }
    }
}

// ===========================================================================
// Mamba-2 state update (decode) + gated-norm statistics
// ===========================================================================
// grid (rows / FS_WARPS, batch); one warp per state row.  Writes u = y * silu(gate)
// * norm_w and one double partial sum of (y*silu(gate))^2 per block; the
// out-projection turns the partials into inv = 1/sqrt(mean + eps) and computes
// inv * (W u) - algebraically the reference's rmsnorm(y*silu(gate))*norm_w -> W.
constexpr int FS_WARPS = 8;
// NV: state elements per lane, one vector load (d_state = 32 NV); 0 for any other d_state.
template <int NV>
__global__ void __launch_bounds__(FS_WARPS * 32)
mamba_scan_norm_kernel(const float* __restrict__ bc, const float* __restrict__ dt_raw,
                       const float* __restrict__ gate, const float* __restrict__ dt_bias,
                       const float* __restrict__ a_log, const float* __restrict__ Dv,
                       const float* __restrict__ norm_w, float* __restrict__ ssm_state,
                       float* __restrict__ u_out, double* __restrict__ partials, MambaDims p) {
    constexpr int N = NV > 0 ? NV : 1;
    __shared__ double wsum[FS_WARPS];
    if (threadIdx.x == 0) pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rows = p.n_heads * p.d_head;
    const int row = blockIdx.x * FS_WARPS + warp;
    const int m = blockIdx.y;
    const bool live = row < rows;
    const int h = live ? row / p.d_head : 0;
    float* s = ssm_state + ((int64_t)m * rows + (live ? row : 0)) * p.d_state;
    auto load = [&](const float* q, float (&v)[N]) {
        if (NV == 4) {
            const float4 f = *reinterpret_cast<const float4*>(q + lane * 4);
            v[0] = f.x; v[N > 1 ? 1 : 0] = f.y; v[N > 2 ? 2 : 0] = f.z; v[N > 3 ? 3 : 0] = f.w;
        } else if (NV == 2) {
            const float2 f = *reinterpret_cast<const float2*>(q + lane * 2);
            v[0] = f.x; v[N > 1 ? 1 : 0] = f.y;
        }
    };
    // everything that does not depend on this token's projection: before the wait
    float sv[N];
    if (NV > 0) load(s, sv);
    const float dtb = dt_bias[h], A = -expf(a_log[h]), dsk = Dv[h];
    const float nw = live ? norm_w[row] : 0.0f;
    pdl_wait();
    double sq = 0.0;
    if (live) {
        const float* bcm = bc + (int64_t)m * p.conv_dim;
        const float* Bv = bcm + p.d_inner;
        const float* Cv = Bv + p.d_state;
        float bv[N], cv[N];
        if (NV > 0) {
            load(Bv, bv);
            load(Cv, cv);
        }
        const float xv = bcm[row];
        const float gt = gate[(int64_t)m * p.d_inner + row];
        const float uu = dt_raw[(int64_t)m * p.n_heads + h] + dtb;
        float acc = 0.0f;
        const float dt = (uu > 20.0f) ? uu : log1pf(expf(uu));
        const float dA = expf(__fmul_rn(A, dt));
        const float sg = silu_acc(gt);
        if (NV > 0) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                sv[i] = __fadd_rn(__fmul_rn(dA, sv[i]), __fmul_rn(__fmul_rn(dt, bv[i]), xv));
                acc += cv[i] * sv[i];
            }
            if (NV == 4) *reinterpret_cast<float4*>(s + lane * 4) = make_float4(sv[0], sv[N > 1 ? 1 : 0], sv[N > 2 ? 2 : 0], sv[N > 3 ? 3 : 0]);
            else *reinterpret_cast<float2*>(s + lane * 2) = make_float2(sv[0], sv[N > 1 ? 1 : 0]);
        } else {
            for (int j = lane; j < p.d_state; j += 32) {
                const float sn = __fadd_rn(__fmul_rn(dA, s[j]), __fmul_rn(__fmul_rn(dt, Bv[j]), xv));
                s[j] = sn;
                acc += Cv[j] * sn;
            }
        }
        acc = warp_sum(acc);
        if (lane == 0) {
            const float y = acc + dsk * xv;
            const float v = y * sg;
            u_out[(int64_t)m * p.d_inner + row] = v * nw;
            sq = (double)v * v;
        }
    }
    if (lane == 0) wsum[warp] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < FS_WARPS; ++w) t += wsum[w];
        partials[(int64_t)m * gridDim.x + blockIdx.x] = t;
    }
}

// ===========================================================================
// host side
// ===========================================================================
template <int KIND, int MT, int PRO, int EPI>
static int launch_sg_inst(const SgArgs& a, int grid, size_t smem) {
    auto kern = stream_gemv_kernel<KIND, MT, PRO, EPI>;
    static bool configured = false;
    if (!configured) {
        int rc = allow_smem(kern);
        if (rc) return rc;
        configured = true;
    }
    return launch_pdl(kern, dim3(grid), dim3(SG_THREADS), smem, a);
}

template <int KIND, int PRO, int EPI>
static int launch_sg_mt(SgArgs a, int grid) {
    const int mt = a.M == 1 ? 1 : a.M == 2 ? 2 : a.M <= 4 ? 4 : 8;
    const size_t other = xact_bytes<KIND>(a.K, mt, PRO == PRO_RMS) + (PRO == PRO_RMS ? (size_t)a.K * 4 : 0) +
                         (size_t)RED_FLOATS * 4 + BAR_BYTES;
    a.n_stages = pick_stages(a.stage_bytes, other);
    if (a.n_stages < 2) return fail(B200_EUNSUPPORTED, "stream_gemv: K = %d does not fit the shared-memory staging", a.K);
    const size_t smem = (size_t)a.n_stages * a.stage_bytes + other;
    if (mt == 1) return launch_sg_inst<KIND, 1, PRO, EPI>(a, grid, smem);
    if (mt == 2) return launch_sg_inst<KIND, 2, PRO, EPI>(a, grid, smem);
    if (mt == 4) return launch_sg_inst<KIND, 4, PRO, EPI>(a, grid, smem);
    return launch_sg_inst<KIND, 8, PRO, EPI>(a, grid, smem);
}

// Fills the tiling fields and launches.  kind: template tag.
int stream_gemv(SgArgs a, int kind, int pro, int epi) {
    B200_REQUIRE(a.M >= 1 && a.M <= 8, "stream_gemv: 1..8 tokens per launch");
    B200_REQUIRE(a.K % 32 == 0 && (kind != 3 || a.K % 256 == 0), "stream_gemv: K not a multiple of the block size");
    B200_REQUIRE(((reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.w2) | reinterpret_cast<uintptr_t>(a.w3)) & 15) == 0,
                 "stream_gemv: weights must be 16-byte aligned");
    if (a.N2 > 0 || a.N3 > 0)
        B200_REQUIRE(epi == EPI_STORE && a.N2 > 0 && a.w2 && a.y2 && (a.N3 == 0 || (a.w3 && a.y3)),
                     "stream_gemv: extra matrices need the store epilogue and their pointers");
    a.row_bytes = row_bytes_of(kind, a.K);
    a.status = stream_status_ptr();
    B200_REQUIRE(a.status, "stream_gemv: status word allocation failed");
    // Rows per tile; a bulk copy moves a multiple of 16 bytes, the last tile of each matrix too.
    const int R = pick_rows(kind, a.row_bytes, a.row_bytes, a.row_bytes, a.N);
    if (R < 1 || (R * a.row_bytes) % 16 != 0 || !tail_tile_ok(a.N, R, a.row_bytes) || !tail_tile_ok(a.N2, R, a.row_bytes) ||
        !tail_tile_ok(a.N3, R, a.row_bytes))
        return fail(B200_EUNSUPPORTED, "stream_gemv: rows of %lld bytes cannot be tiled to 16 bytes", (long long)a.row_bytes);
    if (kind != KIND_F32) return digit_gemv(a, kind, pro, epi);
    a.rows_per_tile = R;
    a.t1 = ceil_div(a.N, R);
    a.t2 = a.t1 + ceil_div(a.N2, R);
    a.num_tiles = a.t2 + ceil_div(a.N3, R);
    a.stage_bytes = (int)((R * a.row_bytes + 127) / 128 * 128);
    const int grid = std::min(a.num_tiles, num_sms());
#define SG_DISPATCH(KIND)                                                                                   \
    if (pro == PRO_RMS && epi == EPI_STORE) return launch_sg_mt<KIND, PRO_RMS, EPI_STORE>(a, grid);         \
    if (pro == PRO_RMS && epi == EPI_INPROJ) return launch_sg_mt<KIND, PRO_RMS, EPI_INPROJ>(a, grid);       \
    if (pro == PRO_NONE && epi == EPI_RESIDUAL) return launch_sg_mt<KIND, PRO_NONE, EPI_RESIDUAL>(a, grid); \
    if (pro == PRO_NONE && epi == EPI_STORE) return launch_sg_mt<KIND, PRO_NONE, EPI_STORE>(a, grid);       \
    return fail(B200_EINVAL, "stream_gemv: unsupported prologue/epilogue pair");
    SG_DISPATCH(KIND_F32)
#undef SG_DISPATCH
}

int mamba_scan_norm_blocks(const MambaDims& p) { return ceil_div(p.n_heads * p.d_head, FS_WARPS); }

int mamba_scan_norm(const float* bc, const float* dt_raw, const float* gate, const float* dt_bias,
                    const float* a_log, const float* D, const float* norm_w, float* ssm_state, float* u_out,
                    double* partials, int batch, const MambaDims& p) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(mamba_scan_norm_blocks(p), batch);
    cfg.blockDim = dim3(FS_WARPS * 32);
    cfg.stream = stream();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto kern = p.d_state == 128 ? mamba_scan_norm_kernel<4> : p.d_state == 64 ? mamba_scan_norm_kernel<2> : mamba_scan_norm_kernel<0>;
    B200_CUDA(cudaLaunchKernelEx(&cfg, kern, bc, dt_raw, gate, dt_bias, a_log, D, norm_w, ssm_state, u_out, partials, p));
    ++g_kernel_launches;
    return B200_OK;
}

}  // namespace b200

extern "C" int b200_stream_status(void) {
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return b200::cuda_status(e, "stream_status: synchronize");
    return b200::stream_status_check("stream_status");
}
