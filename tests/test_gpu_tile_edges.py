"""GPU parity at the edges of the kernels' tiles: the few-token products, the exact tensor-core form for a few tens
of tokens, the GEMM whose token tiles follow the row count, the router's tiles, the one-chunk scan and the recorded
step of a caller whose buffers move."""
import numpy as np
import pytest
import torch

from cases import mamba_params, moe_case
from model_util import TINY, CudaDecoder, make_model

pytestmark = pytest.mark.gpu


# K: one chunk of 256, a partly filled one, several parts of a contraction; N: below a tile of 16 rows, one over
@pytest.mark.parametrize("kind", [-1, 0, 1, 2, 3])
@pytest.mark.parametrize("M", [1, 3, 8, 9, 24, 25, 31])
@pytest.mark.parametrize("K,N", [(256, 4), (288, 20), (2560, 132)])
def test_few_token_products(oracle, kind, M, K, N):
    from gpu_util import SUM_ORDER, close, dev, empty, host, ops
    if kind == 3 and K % 256:
        pytest.skip("Q4_K rows are multiples of 256 weights")
    r = np.random.default_rng(100 * M + K + kind)
    x = r.standard_normal((M, K)).astype(np.float32)
    x[0, :32] *= 1e4                                    # one block far above the rest of its row
    x[M - 1, 256:] = 0.0
    w = (r.standard_normal(N * K) * 0.02).astype(np.float32)
    y = empty((M, N))
    if kind < 0:
        w = w.astype(np.float16).reshape(N, K)
        ops.linear_forward_fp16(dev(x), dev(w.view(np.uint16)), y, M, K, N)
        want = (x.astype(np.float64) @ w.astype(np.float64).T).astype(np.float32)
    else:
        w = oracle.quantize(w, kind)
        ops.linear_forward_q4(dev(x), dev(w), y, M, K, N, kind)
        want = oracle.linear_exact(x, w, kind, M, K, N)
    tol = dict(SUM_ORDER, atol=SUM_ORDER["atol"] * max(1.0, float(np.abs(want).max())))
    np.testing.assert_allclose(host(y), want, **tol)


# More tiles than SMs, on both sides of the line from which two CTAs no longer fit an SM's shared memory.
@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("M", [3, 4, 5, 8])
@pytest.mark.parametrize("K", [1536, 2560])
def test_few_token_products_of_one_and_two_ctas(oracle, kind, M, K):
    from gpu_util import SUM_ORDER, dev, empty, host, ops
    N = 4772                                            # of 16 rows: two tiles for each of 148 SMs and three over, the last with four rows
    r = np.random.default_rng(K + 10 * M + kind)
    x = r.standard_normal((M, K)).astype(np.float32)
    w = oracle.quantize((r.standard_normal(N * K) * 0.02).astype(np.float32), kind)
    y = empty((M, N))
    ops.linear_forward_q4(dev(x), dev(w), y, M, K, N, kind)
    np.testing.assert_allclose(host(y), oracle.linear_exact(x, w, kind, M, K, N), **SUM_ORDER)


# Rows so wide that one tile of sixteen fills the shared memory, and more tiles than a round of the CTAs takes.
@pytest.mark.parametrize("kind,K,M", [(-1, 4096, 1), (-1, 2304, 8), (-1, 5632, 2), (0, 4608, 8), (1, 4352, 8), (2, 4096, 8), (2, 6144, 1),
                                      (2, 4608, 3), (3, 4608, 8), (3, 10496, 1)])
def test_few_token_products_of_wide_rows(oracle, kind, K, M):
    from gpu_util import SUM_ORDER, dev, empty, host, ops
    N = 2388                                            # of 16 rows: one tile for each of 148 SMs and two over
    r = np.random.default_rng(K + M)
    x = r.standard_normal((M, K)).astype(np.float32)
    w = (r.standard_normal(N * K) * 0.02).astype(np.float32)
    y = empty((M, N))
    if kind < 0:
        w = w.astype(np.float16).reshape(N, K)
        ops.linear_forward_fp16(dev(x), dev(w.view(np.uint16)), y, M, K, N)
        want = (x.astype(np.float64) @ w.astype(np.float64).T).astype(np.float32)
    else:
        w = oracle.quantize(w, kind)
        ops.linear_forward_q4(dev(x), dev(w), y, M, K, N, kind)
        want = oracle.linear_exact(x, w, kind, M, K, N)
    np.testing.assert_allclose(host(y), want, **SUM_ORDER)


# rows around one, two and three token tiles of 192 and around the 16 and 96 rows of a copy
@pytest.mark.parametrize("kind", [1, 2, 3])
@pytest.mark.parametrize("M", [33, 96, 97, 192, 193, 385])
@pytest.mark.parametrize("K,N", [(256, 132), (768, 260)])
def test_gemm_token_tiles(oracle, kind, M, K, N):
    from gpu_util import dev, empty, fp16_close, host, ops
    r = np.random.default_rng(M + K + kind)
    x = r.standard_normal((M, K)).astype(np.float32)
    w = oracle.quantize((r.standard_normal(N * K) * 0.02).astype(np.float32), kind)
    y = empty((M, N))
    ops.linear_forward_q4(dev(x), dev(w), y, M, K, N, kind)
    w16 = oracle.dequantize(w, N * K, kind).reshape(N, K).view(np.float16).astype(np.float64)
    want = (x.astype(np.float16).astype(np.float64) @ w16.T).astype(np.float32)
    fp16_close(host(y), want, frac=1e-3)


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("d,E", [(256, 256), (768, 512)])
def test_expert_rows_of_mixed_sizes(oracle, kind, d, E):
    """One group list with every form of a token tile: empty groups, one row, the multiples of 16 that a load brings and
    their neighbours, tiles of one and of two K steps per stage in turn (96 | 97 rows), groups of several tiles.  Norm-wise
    bound: weights within one fp16 ulp of their value in both products (2 x 2^-10) and fp16 activations between them (2^-11)."""
    from gpu_util import dev, empty, host, ops
    sizes = [0, 1, 15, 16, 17, 0, 95, 96, 97, 32, 33, 191, 192, 193, 300, 2, 48, 0]
    ne, R = len(sizes), sum(sizes)
    r = np.random.default_rng(kind)
    rows = r.standard_normal((R, d)).astype(np.float16)
    w = [oracle.quantize((r.standard_normal(ne * E * d) * 0.05).astype(np.float32), kind) for _ in range(3)]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    y = empty((R, d))
    ops.moe_experts_rows(dev(rows.view(np.uint16)), dev(off), None, ne, R, dev(w[0]), dev(w[1]), dev(w[2]), ne, y, d, E, kind)
    got = host(y)
    g, u, dn = (torch.from_numpy(oracle.dequantize(x, ne * E * d, kind).view(np.float16).astype(np.float64)).cuda() for x in w)
    g, u, dn = g.view(ne, E, d), u.view(ne, E, d), dn.view(ne, d, E)
    x = torch.from_numpy(rows.astype(np.float64)).cuda()
    for e in range(ne):
        xe = x[off[e]:off[e + 1]]
        if len(xe):
            act = (torch.nn.functional.silu(xe @ g[e].T) * (xe @ u[e].T)).half().double()
            ref = (act @ dn[e].T).cpu().numpy()
            mine = got[off[e]:off[e + 1]]
            err = np.linalg.norm(mine - ref, axis=1) / np.linalg.norm(ref, axis=1)
            assert err.max() < 2.5e-3, (e, sizes[e], err.max())


# the bias gathers the tokens: experts with none, one, a full tile (8 / 24 slots) and one more
@pytest.mark.parametrize("kind", [2, 3])
@pytest.mark.parametrize("N", [9, 24, 25, 48])
@pytest.mark.parametrize("d,E", [(256, 512), (768, 256)])
def test_expert_tiles(oracle, kind, N, d, E):
    from gpu_util import SUM_ORDER, dev, empty, host, ops
    ne, K = 8, 2
    c = moe_case(oracle, N + d, N, d, E, ne, K, 0, kind, bias_sigma=2.0)
    out, idx, w = empty((N, d)), empty((N, K), torch.int32), empty((N, K))
    args = [dev(c[k]) for k in ("gates", "ups", "downs", "sh_g", "sh_u", "sh_d")]
    ops.moe_forward_bias_half(dev(c["x"]), dev(c["router_w"]), dev(c["router_bias"]), *args, out, None, idx, w, None, None,
                              None, N, d, E, ne, K, 0, kind)
    want, _, widx, _ = oracle.moe_forward(c["x"], c["router_w"], c["router_bias"], c["gates"], c["ups"], c["downs"], None, None,
                                          None, d, E, ne, K, 0, kind)
    assert np.array_equal(host(idx), widx)
    np.testing.assert_allclose(host(out), want, **SUM_ORDER)


# Experts whose down rows do not fit sixteen to a tile: (kind, hidden, experts, width, top, shared width, sequences)
WIDE_EXPERTS = [(2, 2048, 64, 1024, 8, 2048, 1), (2, 2048, 128, 768, 8, 0, 2), (0, 1024, 16, 1024, 8, 1024, 8), (1, 1024, 16, 1024, 8, 1024, 8),
                (2, 512, 16, 1536, 16, 0, 5)]


@pytest.mark.parametrize("kind,d,ne,E,K,SH,B", WIDE_EXPERTS)
def test_fused_step_takes_wide_experts(kind, d, ne, E, K, SH, B):
    import ctypes as C
    from gpu_util import pkg
    lib, h = pkg.lib(), C.c_void_p()
    types = np.array([0], np.int32)
    lib.b200_decoder_create(C.byref(h), B, 512, d, 1, types.ctypes.data, d // 64, d // 64, 64, -1, 2 * d // 64, 64, 64, 4, ne, K, E, SH, 32,
                            16, kind, 1e-5, 1.0, 1.0, 0.0, 1.0)
    try:
        lib.b200_decoder_configure(h, 1, 0)
    finally:
        lib.b200_decoder_destroy(h)


@pytest.mark.parametrize("kind,ne,E,K,SH,N", [(2, 8, 1024, 8, 2048, 1), (0, 8, 1024, 8, 1024, 8), (1, 8, 1024, 8, 1024, 8),
                                              (2, 16, 1536, 16, 0, 1), (2, 16, 1536, 16, 0, 5)])
def test_wide_experts(oracle, kind, ne, E, K, SH, N):
    from gpu_util import SUM_ORDER, dev, empty, host, ops
    d = 544                                             # tiles of two and eight rows over the CTAs in several rounds
    c = moe_case(oracle, N + E, N, d, E, ne, K, SH, kind)
    out, idx, w = empty((N, d)), empty((N, K), torch.int32), empty((N, K))
    args = [dev(c[k]) for k in ("gates", "ups", "downs", "sh_g", "sh_u", "sh_d")]
    ops.moe_forward_bias_half(dev(c["x"]), dev(c["router_w"]), dev(c["router_bias"]), *args, out, None, idx, w, None, None, None, N, d, E,
                              ne, K, SH, kind)
    oracle.set_weight_rounding(False)
    want, _, widx, _ = oracle.moe_forward(c["x"], c["router_w"], c["router_bias"], c["gates"], c["ups"], c["downs"], c["sh_g"], c["sh_u"],
                                          c["sh_d"], d, E, ne, K, SH, kind)
    oracle.set_weight_rounding(True)
    assert np.array_equal(host(idx), widx)
    np.testing.assert_allclose(host(out), want, **SUM_ORDER)


# Up to eight tokens of rows so wide that the decode step's kernels refuse them (eight tokens of 4096 beside two tiles): they
# run as units, in fp32 on the exact weights as the others.  Two and four tokens still fit.
@pytest.mark.parametrize("kind", [2, 3])
@pytest.mark.parametrize("N", [2, 3, 4, 5, 8])
def test_few_tokens_of_wide_rows(oracle, kind, N):
    from gpu_util import SUM_ORDER, dev, empty, host, ops
    d, E, ne, K, SH = 4096, 256, 8, 2, 1536
    c = moe_case(oracle, N + kind, N, d, E, ne, K, SH, kind)
    out, idx, w = empty((N, d)), empty((N, K), torch.int32), empty((N, K))
    args = [dev(c[k]) for k in ("gates", "ups", "downs", "sh_g", "sh_u", "sh_d")]
    ops.moe_forward_bias_half(dev(c["x"]), dev(c["router_w"]), dev(c["router_bias"]), *args, out, None, idx, w, None, None, None, N, d, E,
                              ne, K, SH, kind)
    oracle.set_weight_rounding(False)
    want, _, widx, _ = oracle.moe_forward(c["x"], c["router_w"], c["router_bias"], c["gates"], c["ups"], c["downs"], c["sh_g"], c["sh_u"],
                                          c["sh_d"], d, E, ne, K, SH, kind)
    oracle.set_weight_rounding(True)
    assert np.array_equal(host(idx), widx)
    np.testing.assert_allclose(host(out), want, **SUM_ORDER)


# Up to eight tokens may be written over x, whatever the row's width and with or without the last elements of x in front of out.
@pytest.mark.parametrize("kind", [2, 3])
@pytest.mark.parametrize("N,d", [(5, 4096), (8, 4096), (8, 512)])
@pytest.mark.parametrize("shift", [0, 1])
def test_few_tokens_in_place(oracle, kind, N, d, shift):
    from gpu_util import SUM_ORDER, dev, empty, host, ops
    E, ne, K, SH = 256, 8, 2, 1536
    c = moe_case(oracle, N + kind, N, d, E, ne, K, SH, kind)
    args = [dev(c[k]) for k in ("router_w", "router_bias", "gates", "ups", "downs", "sh_g", "sh_u", "sh_d")]
    got = []
    for over in (False, True):
        room = empty(((N + shift) * d,))
        x = room[: N * d]
        x.copy_(dev(c["x"]).view(-1))
        out = room[shift * d:] if over else empty((N * d,))
        ops.moe_forward_bias_half(x, *args, out, None, None, None, None, None, None, N, d, E, ne, K, SH, kind)
        got.append(host(out))
    np.testing.assert_allclose(got[1], got[0], **SUM_ORDER)


# the decode step's kernels, the digit engine's units and the exact tensor-core form
@pytest.mark.parametrize("kind", [0, 2, 3])
@pytest.mark.parametrize("N", [1, 3, 8, 9, 24])
def test_experts_of_a_token_that_is_not_finite(oracle, kind, N):
    from gpu_util import dev, empty, host, ops
    d, E, ne, K = 256, 256, 8, 2
    c = moe_case(oracle, N, N, d, E, ne, K, 0, kind)
    x = c["x"].copy()
    x[N - 1, 5] = np.nan
    out, idx, w = empty((N, d)), empty((N, K), torch.int32), empty((N, K))
    args = [dev(c[k]) for k in ("gates", "ups", "downs", "sh_g", "sh_u", "sh_d")]
    ops.moe_forward_bias_half(dev(x), dev(c["router_w"]), dev(c["router_bias"]), *args, out, None, idx, w, None, None, None, N, d, E,
                              ne, K, 0, kind)
    got = host(out)
    assert np.isnan(got[N - 1]).all() and np.isfinite(got[:N - 1]).all()


# one to eight tokens; the 8- and 32-token tiles of the router; widths off its 128 columns
@pytest.mark.parametrize("d,ne,K", [(260, 33, 3), (1536, 64, 6)])
@pytest.mark.parametrize("N", [1, 7, 257, 600, 2401])
def test_router_tiles(oracle, d, ne, K, N):
    from gpu_util import dev, empty, host, ops
    r = np.random.default_rng(d + N)
    x = r.standard_normal((N, d)).astype(np.float32)
    rw = (r.standard_normal((ne, d)) / np.sqrt(d)).astype(np.float32)
    bias = (r.standard_normal(ne) * 0.5 / ne).astype(np.float32)
    _, idx, w = oracle.moe_route(x, rw, bias, ne, K)
    di, dw = empty((N, K), torch.int32), empty((N, K))
    ops.moe_route(dev(x), dev(rw), dev(bias), empty((N, ne)), di, dw, N, d, ne, K)
    assert np.array_equal(host(di), idx)
    np.testing.assert_array_max_ulp(host(dw), w, maxulp=4)


# the tiles of the router and their ragged ends: one chain per thread up to some 500 tokens, 2 x 2 above, 8 x 1 for many experts, one
# column tile and several, a last one of four columns; bit-exact as above
@pytest.mark.parametrize("d,ne,K", [(128, 16, 2), (132, 72, 10), (1028, 256, 16)])
@pytest.mark.parametrize("N", [9, 300, 1111])
def test_router_thread_tiles(oracle, d, ne, K, N):
    test_router_tiles(oracle, d, ne, K, N)


# 8 x 1 tiles: the last token and expert tiles with one row, a last column tile of four
@pytest.mark.parametrize("d,ne,K,N", [(68, 64, 6, 3585), (256, 97, 4, 1793)])
def test_router_wide_tiles(oracle, d, ne, K, N):
    test_router_tiles(oracle, d, ne, K, N)


# slots around a warp's 128 and a block's 2048, on both sides of the line to the three kernels for many; at a list that is no multiple
# of 16 bytes; experts without any
@pytest.mark.parametrize("NK", [1, 127, 129, 2047, 2049, 40001, 109999, 110001])
@pytest.mark.parametrize("shift", [0, 1])
def test_permutation_and_its_inverse(NK, shift):
    from gpu_util import dev, empty, host, ops
    ne = 72
    r = np.random.default_rng(NK)
    idx = r.choice(ne, size=NK + shift, p=r.dirichlet(np.full(ne, 0.3))).astype(np.int32)
    rows16, inv, offsets = empty((NK, 32), torch.int16), empty(NK, torch.int32), empty(ne + 1, torch.int32)
    didx, x = dev(idx), empty((NK, 32))
    ops.moe_dispatch_pack(x, didx[shift:], NK, 32, ne, 1, rows16, inv, offsets)
    want = np.argsort(idx[shift:], kind="stable")
    assert np.array_equal(host(inv)[want], np.arange(NK))
    assert np.array_equal(host(offsets), np.concatenate([[0], np.cumsum(np.bincount(idx[shift:], minlength=ne))]))


# a sequence of one chunk carries its state in the output kernel; 129 steps: two chunks
@pytest.mark.parametrize("kind", [-2, 2])
@pytest.mark.parametrize("d_state", [64, 128])
@pytest.mark.parametrize("T", [65, 128, 129])
def test_scan_chunks(oracle, kind, d_state, T):
    from gpu_util import dev, empty, fp16_close, host, ops
    r = np.random.default_rng(T + d_state)
    B, d, heads, P, k = 2, 256, 3, 64, 4
    p = mamba_params(oracle, r, d, heads, P, d_state, k, kind, 0.2)
    x = r.standard_normal((B, T, d)).astype(np.float32)
    state = (r.standard_normal((B, heads, P, d_state)) * 0.1).astype(np.float32)
    names = ("w_in", "conv_w", "conv_b", "dt_bias", "a_log", "D", "norm_w", "w_out")
    rest = (B, T, d, p["d_inner"], p["conv_dim"], heads, P, d_state, k, 1e-5)
    want, want_state = oracle.mamba2_forward(x, *(p[n] for n in names), state, *rest, kind)
    ds, out = dev(state), empty((B, T, d))
    weights = [dev(p[n]) for n in names]
    if kind == -2:
        ops.mamba2_forward(dev(x), *weights, ds, out, *rest)
    else:
        ops.mamba2_forward_half(dev(x), *weights, ds, out, *rest, kind)
    fp16_close(host(out), want)
    fp16_close(host(ds), want_state)


# buffers that stay, that move at every step, and that move and come back
@pytest.mark.parametrize("fused,batch", [(1, 1), (0, 3), (0, 9)])
def test_recorded_step_with_moving_buffers(oracle, fused, batch):
    model = make_model(oracle, TINY, 4)
    r = np.random.default_rng(5)
    steps = r.integers(0, TINY["vocab"], (6, batch)).astype(np.int32)
    outs = []
    for moving in (False, True):
        dec = CudaDecoder(model, batch=batch, max_ctx=64)
        dec.configure(fused, 1)
        tok, nxt = torch.zeros(batch, dtype=torch.int32, device="cuda"), torch.zeros(batch, dtype=torch.int32, device="cuda")
        kept, got = [], []
        for i, t in enumerate(steps):
            if moving and i != 3:
                tok, nxt = torch.zeros_like(tok), torch.zeros_like(nxt)
                kept.append((tok, nxt))
            tok.copy_(torch.from_numpy(t))
            torch.cuda.synchronize()
            dec.lib.b200_decoder_step(dec.handle, tok, nxt)
            dec.lib.b200_synchronize()
            got.append((nxt.cpu().numpy().copy(), dec.logits()))
        outs.append(got)
        dec.close()
    for (na, la), (nb, lb) in zip(*outs):
        assert np.array_equal(na, nb)
        assert np.array_equal(la.view(np.uint32), lb.view(np.uint32))


# norm weights where a caller's own packing put them: any address of a float
@pytest.mark.parametrize("B", [1, 2, 5])
@pytest.mark.parametrize("qkind", [2, 3])
def test_fused_step_with_norm_weights_at_odd_addresses(oracle, B, qkind):
    from model_util import T
    m = make_model(oracle, dict(TINY, qkind=qkind), seed=4)
    toks = np.random.default_rng(B).integers(0, TINY["vocab"], (3, B)).astype(np.int32)
    got = []
    for odd in (False, True):
        dec = CudaDecoder(m, B, 16)
        if odd:
            for l, L in [(-1, m)] + list(enumerate(m["layers"])):
                for name in ("final_norm", "attn_norm", "ffn_norm"):
                    if name in L:
                        t = torch.empty(L[name].size + 1, device="cuda")[1:]
                        t.copy_(torch.from_numpy(L[name]))
                        dec.keep.append(t)
                        dec.lib.b200_decoder_set_tensor(dec.handle, l, T[name], t)
        dec.configure(1, 0)
        for t in toks:
            dec.step_host(t)
        got.append(dec.logits())
    assert np.array_equal(got[0], got[1])
