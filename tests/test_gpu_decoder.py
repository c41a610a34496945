"""GPU parity at model level: the CUDA decoder against the oracle walking the
reference's per-token op sequence, teacher-forced."""
import numpy as np
import pytest

from model_util import CONFIG_1, TINY, CudaDecoder, OracleDecoder, cached_model, make_model

pytestmark = pytest.mark.gpu


def _teacher_forced(oracle, cfg, steps, graph, fused, seed=0, model=None):
    """Feed the same seeded token stream to both sides (greedy continuation of the
    oracle after a random prompt), compare logits and arg-max every step."""
    model = model or make_model(oracle, cfg, seed)
    ora = OracleDecoder(oracle, model, max_ctx=steps + 1)
    dec = CudaDecoder(model, batch=1, max_ctx=steps + 1)
    dec.configure(fused, graph)
    r = np.random.default_rng(seed + 1)
    prompt = r.integers(0, cfg["vocab"], steps // 2)
    tok = int(prompt[0])
    agree, margins, worst = 0, [], 0.0
    for s in range(steps):
        want = ora.step(tok)
        got_next = int(dec.step_host([tok])[0])
        got = dec.logits()[0]
        err = np.abs(got - want)
        worst = max(worst, float(err.max()))
        # stated tolerance for logits vs the reference CPU path
        assert np.all(err <= 2e-2 + 1e-2 * np.abs(want)), f"step {s}: max abs err {err.max()}"
        top2 = np.sort(want)[-2:]
        margins.append(float(top2[1] - top2[0]))
        want_next = oracle.argmax(want)
        agree += int(got_next == want_next)
        assert got_next == int(np.argmax(got)) or got[got_next] == got.max()
        tok = int(prompt[s + 1]) if s + 1 < len(prompt) else want_next       # teacher forcing
    dec.close()
    return agree / steps, worst, margins


@pytest.mark.parametrize("graph", [0, 1])
def test_tiny_model_teacher_forced(oracle, graph):
    rate, worst, _ = _teacher_forced(oracle, TINY, steps=24, graph=graph, fused=0)
    assert rate >= 0.99, f"greedy agreement {rate:.3f}"
    assert worst < 2e-3            # fp32 paths: far inside the stated tolerance


@pytest.mark.parametrize("graph", [0, 1])
def test_tiny_model_fused_teacher_forced(oracle, graph):
    """Cross-op fused kernels (norm prologue, conv / residual epilogues, streamed weights)."""
    rate, worst, _ = _teacher_forced(oracle, TINY, steps=24, graph=graph, fused=1)
    assert rate >= 0.99, f"greedy agreement {rate:.3f}"
    assert worst < 2e-3


@pytest.mark.parametrize("graph", [0, 1])
def test_tiny_model_persistent_teacher_forced(oracle, graph):
    """Persistent step kernel (fused = 2): Mamba and MoE phases of the token in one
    cooperative launch per run of layers, grid barriers between the phases."""
    rate, worst, _ = _teacher_forced(oracle, TINY, steps=24, graph=graph, fused=2)
    assert rate >= 0.99, f"greedy agreement {rate:.3f}"
    assert worst < 2e-3


def test_config1_persistent_teacher_forced(oracle):
    cfg = dict(CONFIG_1, vocab=4096)
    rate, worst, margins = _teacher_forced(oracle, cfg, steps=32, graph=1, fused=2)
    assert rate >= 0.99, f"greedy agreement {rate:.3f} (min top-2 margin {min(margins):.2e})"
    assert worst < 2e-3


def test_persistent_equals_fused_bitwise_stable(oracle):
    """Two runs of the persistent step give identical bits (fixed summation orders, no
    atomics on data), and it stays within summation-order distance of the fused mode."""
    model = make_model(oracle, TINY, 9)
    toks = [3, 77, 5, 400, 12, 12, 9, 250]
    runs = []
    for fused in (2, 2, 1):
        dec = CudaDecoder(model, batch=1, max_ctx=16)
        dec.configure(fused, 0)
        out = []
        for t in toks:
            dec.step_host([t])
            out.append(dec.logits()[0].copy())
        runs.append(np.stack(out))
        dec.close()
    assert np.array_equal(runs[0].view(np.uint32), runs[1].view(np.uint32))
    np.testing.assert_allclose(runs[0], runs[2], rtol=1e-3, atol=1e-4)


def test_persistent_barrier_timeout_reports_and_recovers(oracle):
    """A grid barrier one CTA never reaches: the other CTAs' bounded waits run out, the
    kernel returns, the step reports B200_ECUDA - and after a reset the decoder works."""
    from gpu_util import B200Error
    model = make_model(oracle, TINY, 2)
    dec = CudaDecoder(model, batch=1, max_ctx=16)
    dec.configure(2, 0)
    dec.step_host([1])
    dec.lib.b200_decoder_test_barrier(dec.handle, 20000, 3)
    with pytest.raises(B200Error, match="bounded wait"):
        dec.step_host([2])
    dec.lib.b200_decoder_test_barrier(dec.handle, 0, -1)
    assert dec.lib.raw("b200_stream_status") == 0
    dec.reset()
    ora = OracleDecoder(oracle, model, max_ctx=16)
    for t in (1, 2, 3):
        want = ora.step(t)
        dec.step_host([t])
        np.testing.assert_allclose(dec.logits()[0], want, rtol=1e-3, atol=1e-4)
    dec.close()


def test_persistent_needs_batch_one(oracle):
    from gpu_util import B200Error
    model = make_model(oracle, TINY, 2)
    dec = CudaDecoder(model, batch=2, max_ctx=8)
    with pytest.raises(B200Error, match="batch 1"):
        dec.configure(2, 0)
    dec.close()


@pytest.mark.parametrize("fused", [0, 1, 2])
def test_graph_is_recaptured_after_workspaces_move(oracle, fused):
    """Steps replayed from a captured graph, then a longer prefill that makes the library's
    workspaces grow (their old addresses are freed), then steps again: the stale recording
    must not be replayed.  Compared with the same sequence run without graphs."""
    model = make_model(oracle, TINY, 6)
    r = np.random.default_rng(8)
    first, second = r.integers(0, TINY["vocab"], 40), r.integers(0, TINY["vocab"], 200)
    tail = r.integers(0, TINY["vocab"], 4)
    outs = []
    for graph in (0, 1):
        dec = CudaDecoder(model, batch=1, max_ctx=256)
        dec.configure(fused, graph)
        got = []
        dec.prefill(first[None])
        for t in tail:
            dec.step_host([t])
            got.append(dec.logits()[0].copy())
        dec.reset()
        dec.prefill(second[None])           # grows the prefill / GEMM / attention workspaces
        for t in tail:
            dec.step_host([t])
            got.append(dec.logits()[0].copy())
        outs.append(np.stack(got))
        dec.close()
    assert np.array_equal(outs[0].view(np.uint32), outs[1].view(np.uint32))


def test_config1_fused_teacher_forced(oracle):
    cfg = dict(CONFIG_1, vocab=4096)
    rate, worst, margins = _teacher_forced(oracle, cfg, steps=32, graph=1, fused=1)
    assert rate >= 0.99, f"greedy agreement {rate:.3f} (min top-2 margin {min(margins):.2e})"
    assert worst < 2e-3


def test_config1_teacher_forced(oracle):
    """Config-1 shape (hidden 768, 8 layers, Q8_0) with a reduced vocabulary so the scalar
    oracle finishes in seconds."""
    cfg = dict(CONFIG_1, vocab=4096)
    rate, worst, margins = _teacher_forced(oracle, cfg, steps=32, graph=1, fused=0)
    assert rate >= 0.99, f"greedy agreement {rate:.3f} (min top-2 margin {min(margins):.2e})"
    assert worst < 2e-3


H_TINY_CUT = dict(vocab=2048, hidden=1536, n_layers=4, layer_types=[0, 1, 0, 0],
                  n_heads=12, n_kv=4, head_dim=128, rope_type=-1, rope_theta=1e4,
                  mamba_heads=48, mamba_d_head=64, mamba_d_state=128, mamba_d_conv=4,
                  n_experts=64, top_k=6, expert_dim=512, shared_dim=1024, qkind=3,
                  rms_eps=1e-5, embedding_multiplier=12.0, residual_multiplier=0.22,
                  attn_scale=0.0078125, logits_scaling=6.0)


@pytest.mark.parametrize("fused", [1, 2])
def test_h_tiny_width_cut_teacher_forced(oracle, fused):
    """Four layers at the widths of the Granite-4.0-H-Tiny-shaped model (hidden 1536, Mamba
    48 x 64 / state 128, 12 q / 4 kv heads x 128 without RoPE, 64 experts top-6 ffn 512, shared
    1024, Q4_K; reduced vocabulary) against the oracle's walk, fused and persistent modes."""
    model = cached_model(oracle, H_TINY_CUT, 0, share_experts=True)
    rate, worst, margins = _teacher_forced(oracle, H_TINY_CUT, steps=10, graph=1, fused=fused, model=model)
    assert rate >= 0.99, f"greedy agreement {rate:.3f} (min top-2 margin {min(margins):.2e})"
    assert worst < 2e-3


def test_batch_rows_are_independent(oracle):
    """batch 3 with different tokens per row == three batch-1 oracle runs."""
    model = make_model(oracle, TINY, 3)
    dec = CudaDecoder(model, batch=3, max_ctx=16)
    oras = [OracleDecoder(oracle, model, max_ctx=16) for _ in range(3)]
    r = np.random.default_rng(4)
    for s in range(6):
        toks = r.integers(0, TINY["vocab"], 3)
        dec.step_host(toks)
        got = dec.logits()
        for b in range(3):
            want = oras[b].step(int(toks[b]))
            np.testing.assert_allclose(got[b], want, rtol=1e-3, atol=1e-4)
    dec.close()


def test_reset_and_replay_is_bit_stable(oracle):
    model = make_model(oracle, TINY, 5)
    dec = CudaDecoder(model, batch=2, max_ctx=16)
    dec.configure(0, 1)
    toks = np.array([[1, 2], [3, 4], [5, 6], [7, 8]])
    runs = []
    for _ in range(2):
        dec.reset()
        out = []
        for t in toks:
            dec.step_host(t)
            out.append(dec.logits().copy())
        runs.append(np.stack(out))
    assert np.array_equal(runs[0].view(np.uint32), runs[1].view(np.uint32))
    assert dec.launches() > 0 and dec.step_bytes() > 0
    dec.close()


def test_errors(oracle):
    from gpu_util import B200Error, pkg
    import ctypes as C
    lib = pkg.lib()
    h = C.c_void_p()
    types = np.zeros(2, np.int32)
    with pytest.raises(B200Error, match="unknown qkind"):
        lib.b200_decoder_create(C.byref(h), 1, 64, 64, 2, types.ctypes.data, 2, 1, 32, -1, 2, 32, 16, 4, 4, 2, 32, 32,
                                8, 4, 9, 1e-5, 1.0, 1.0, 0.0, 1.0)
    lib.b200_decoder_create(C.byref(h), 1, 64, 64, 2, types.ctypes.data, 2, 1, 32, -1, 2, 32, 16, 4, 4, 2, 32, 32,
                            8, 4, 2, 1e-5, 1.0, 1.0, 0.0, 1.0)
    tok = np.zeros(1, np.int32)
    with pytest.raises(B200Error, match="not set"):
        lib.b200_decoder_step_host(h, tok.ctypes.data, tok.ctypes.data)
    lib.b200_decoder_destroy(h)


def test_recorded_step_of_experts_too_wide_for_the_unit_kernels(oracle):
    """Nine sequences, rows too wide for the unit kernels' staging: the layer is refused there before anything is on the
    second stream, so the recording of the step has no branch left open and its outputs are the eager step's."""
    cfg = dict(TINY, hidden=7168, n_layers=1, layer_types=[0], qkind=2, n_experts=4, top_k=1, expert_dim=64, shared_dim=256,
               mamba_heads=4, mamba_d_state=64)
    m = make_model(oracle, cfg, seed=1)
    toks = np.random.default_rng(2).integers(0, cfg["vocab"], (3, 9)).astype(np.int32)
    got = []
    for graph in (0, 1):
        dec = CudaDecoder(m, 9, 8)
        dec.configure(0, graph)
        for t in toks:
            dec.step_host(t)
        got.append(dec.logits())
    assert np.array_equal(got[0], got[1]) and np.isfinite(got[0]).all()


@pytest.mark.parametrize("B", [5, 8])
def test_fused_step_with_a_wide_lm_head(oracle, B):
    """Hidden size 4096: eight sequences' staged rows leave no room for an lm_head row, so it goes in groups."""
    cfg = dict(TINY, hidden=4096, n_layers=1, layer_types=[0], n_experts=4, top_k=1, mamba_heads=4, mamba_d_state=64)
    m = make_model(oracle, cfg, seed=3)
    toks = np.random.default_rng(B).integers(0, cfg["vocab"], (2, B)).astype(np.int32)
    got = []
    for fused in (0, 1):
        dec = CudaDecoder(m, B, 8)
        dec.configure(fused, 0)
        for t in toks:
            dec.step_host(t)
        got.append(dec.logits())
    np.testing.assert_allclose(got[1], got[0], rtol=1e-4, atol=1e-4 * np.abs(got[0]).max())


@pytest.mark.parametrize("qkind", [2, 3])
def test_batches_of_any_size_agree_when_the_routing_is_held(oracle, qkind):
    """The same sequence decoded alone, among 2, 5, 8, 9, 20 and 31: the step's kernels differ (digit engine of one to eight
    columns, exact tensor-core form, units), the logits must not by more than fp32 rounding.  The router is switched off
    (equal probabilities, the choice by the bias alone), as a near-tie that comes out the other way hides everything else.
    Per layer five products, each off by up to 2^-22 of its norm, of independent signs: 2^-22 sqrt(5 * 4 layers) on the logits;
    four times that where the products are the exact tensor-core form's (cut sums: 6.3 of 2^-24 each, one direction within a
    product, so that layers' errors add up rather than cancel).  Q8_0 from 9 sequences on: the shared expert's fp16 GEMM (2^-11 per activation, averaged over the row: 5e-4)."""
    m = make_model(oracle, dict(TINY, qkind=qkind), seed=11)
    for i, L in enumerate(m["layers"]):
        L["router"] = np.zeros_like(L["router"])
        L["router_bias"] = np.random.default_rng(i).permutation(L["router_bias"].size).astype(np.float32)
    toks = np.random.default_rng(5).integers(0, TINY["vocab"], (6, 31)).astype(np.int32)
    want = None
    for B in (1, 2, 5, 8, 9, 20, 31):
        dec = CudaDecoder(m, B, 16)
        dec.configure(1 if B <= 8 else 0, 0)
        for t in toks:
            dec.step_host(t[:B])
        got = dec.logits()[0].astype(np.float64)
        if want is None:
            want = got
        bound = 2.0 ** -22 * 20 ** 0.5 * (1 if B <= 8 else 4) if B <= 8 or qkind == 3 else 5e-4
        assert np.linalg.norm(got - want) < bound * np.linalg.norm(want), (B, np.linalg.norm(got - want) / np.linalg.norm(want))
