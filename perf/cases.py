"""The workloads the speed of this framework is judged by: what its users have it do, through its public
entry points, with the sizes of its benchmark configurations and the ragged and odd ones between them.

kind "generate"   a conversation of a decoder: reset, the prompts (b200_decoder_prefill, or _ragged when they differ
                  in length), then `steps` decode steps, greedy or sampled, device tokens or the host loop
kind "prompt"     the prompts alone (scoring, embedding, filling the caches of a serving batch)
kind "moe"        one MoE layer (b200_moe_forward_bias_half): router, top-K experts, shared expert
kind "mamba"      one Mamba-2 layer over whole sequences (b200_mamba2_forward_half)
kind "attention"  decode attention of a ragged batch over the paged KV cache (b200_attention_decode_paged_fp16)

Weights are random-init N(0, 0.02) quantised on the device, as in the benchmark.  A decoder is fed given tokens instead of
its own picks: a step does the same work for any token, and two implementations stay comparable when they round differently.
"""
import ctypes as C
import importlib
import math
import random

import numpy as np
import torch

PKG = "jdm-ghassan_v1_flach_b200"

# The benchmark's small hybrid model and the Granite-4.0-H-Tiny-shaped one (BASELINE configurations 1 and 4).
SMALL = dict(vocab=32768, hidden=768, layer_types=[0, 0, 0, 1, 0, 0, 0, 1], n_heads=12, n_kv=4, head_dim=64, rope_type=1,
             mamba_heads=24, d_head=64, d_state=64, d_conv=4, n_experts=16, top_k=2, expert_dim=512, shared_dim=1024,
             embedding_multiplier=1.0, residual_multiplier=1.0, attn_scale=0.0, logits_scaling=1.0)
H_TINY = dict(vocab=100352, hidden=1536, layer_types=[1 if l in (9, 19, 29, 39) else 0 for l in range(40)], n_heads=12, n_kv=4,
              head_dim=128, rope_type=-1, mamba_heads=48, d_head=64, d_state=128, d_conv=4, n_experts=64, top_k=6,
              expert_dim=512, shared_dim=1024, embedding_multiplier=12.0, residual_multiplier=0.22, attn_scale=0.0078125,
              logits_scaling=6.0)
MODELS = {"small": SMALL, "htiny": H_TINY}

# The MoE and attention widths of the three benchmark models (the H-Small-shaped one at the op level only).
MOE = {"small": dict(d=768, E=512, ne=16, K=2, SH=1024), "htiny": dict(d=1536, E=512, ne=64, K=6, SH=1024),
       "hsmall": dict(d=4096, E=768, ne=72, K=10, SH=1536)}
MAMBA = {"small": dict(d=768, heads=24, d_head=64, d_state=64), "htiny": dict(d=1536, heads=48, d_head=64, d_state=128)}
ATTN = {"small": dict(H=12, KV=4, hd=64), "htiny": dict(H=12, KV=4, hd=128), "hsmall": dict(H=32, KV=8, hd=128)}

KIND = {"Q8_0": 2, "Q4_K": 3}                            # storage kinds of include/b200ops.h
BLOCK = {"Q8_0": (32, 34), "Q4_K": (256, 144)}           # weights, bytes
PAGE = 64
DECODE_FUSED_MAX = 8                                     # include/b200step.h: fused steps take up to 8 sequences


def listed():
    return [
        # an assistant on the small model, token by token through host buffers: launches and latency
        dict(name="chat_small", kind="generate", model="small", quant="Q8_0", batch=1, lo=128, hi=128, steps=32, sampled=False,
             host=True),
        # the headline: one user on the H-Tiny-shaped model
        dict(name="chat_htiny", kind="generate", model="htiny", quant="Q4_K", batch=1, lo=301, hi=301, steps=16, sampled=False,
             host=False),
        # a handful of users with sampling on
        dict(name="few_users_htiny", kind="generate", model="htiny", quant="Q4_K", batch=5, lo=17, hi=160, steps=12,
             sampled=True, host=False),
        # a serving batch
        dict(name="serve64_htiny", kind="generate", model="htiny", quant="Q4_K", batch=64, lo=9, hi=120, steps=12, sampled=False,
             host=False),
        # one long prompt, and a ragged group of them
        dict(name="prompt_4096_htiny", kind="prompt", model="htiny", quant="Q4_K", batch=1, lo=4096, hi=4096),
        dict(name="prompts_ragged_htiny", kind="prompt", model="htiny", quant="Q4_K", batch=12, lo=31, hi=1400),
        # the MoE layer by itself: a token, a ragged middle, a long prompt's worth
        dict(name="moe_1_htiny", kind="moe", shape="htiny", quant="Q4_K", tokens=1),
        dict(name="moe_517_hsmall", kind="moe", shape="hsmall", quant="Q4_K", tokens=517),
        dict(name="moe_4096_htiny", kind="moe", shape="htiny", quant="Q4_K", tokens=4096),
        # the Mamba-2 layer by itself over a batch of sequences that is no multiple of any tile
        dict(name="mamba_4x2047_htiny", kind="mamba", shape="htiny", quant="Q4_K", batch=4, steps=2047),
        # decode attention of a ragged serving batch with long contexts
        dict(name="attention_64_hsmall", kind="attention", shape="hsmall", batch=64, lo=256, hi=8192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    quant = rng.choice(["Q4_K", "Q4_K", "Q8_0"])
    kind = rng.choice(["generate", "generate", "generate", "prompt", "prompt", "moe", "moe", "mamba", "attention"])
    if kind == "generate":
        batch = _log(rng, 1, 64)
        hi = _log(rng, 8, 300 if batch <= 8 else 120)
        return dict(kind=kind, model=rng.choice(["small", "htiny", "htiny"]), quant=quant, batch=batch,
                    lo=hi if batch == 1 else rng.randint(1, hi), hi=hi, steps=rng.randint(6, 16 if batch <= 8 else 8),
                    sampled=rng.random() < 0.3, host=rng.random() < 0.3)
    if kind == "prompt":
        batch = _log(rng, 1, 16)
        hi = _log(rng, 64, 4096 if batch <= 2 else 1024)
        return dict(kind=kind, model=rng.choice(["small", "htiny", "htiny"]), quant=quant, batch=batch,
                    lo=hi if batch == 1 else rng.randint(1, hi), hi=hi)
    if kind == "moe":
        shape = rng.choice(["small", "htiny", "htiny", "hsmall"])
        return dict(kind=kind, shape=shape, quant=quant, tokens=_log(rng, 1, 2048 if shape == "hsmall" else 4096))
    if kind == "mamba":
        batch = _log(rng, 1, 8)
        return dict(kind=kind, shape=rng.choice(["small", "htiny"]), quant=quant, batch=batch,
                    steps=_log(rng, 16, 8192 // batch))
    hi = _log(rng, 64, 8192)
    return dict(kind=kind, shape=rng.choice(list(ATTN)), batch=_log(rng, 1, 64), lo=rng.randint(1, hi), hi=hi)


def _lengths(case):
    """Lengths of the case's sequences: spread evenly over [lo, hi] in a shuffled order, one of them hi."""
    lo, hi, n = case["lo"], case["hi"], case["batch"]
    got = [lo + (hi - lo) * (i + 1) // n for i in range(n)]
    random.Random(n).shuffle(got)
    return got


class _Sampling(C.Structure):
    """struct b200_sampling of include/b200step.h."""
    _fields_ = [(n, C.c_float) for n in ("temperature", "top_p", "min_p", "repetition_penalty", "frequency_penalty",
                                         "presence_penalty")] + \
               [(n, C.c_int32) for n in ("top_k", "repetition_window", "no_repeat_ngram", "greedy")] + [("seed", C.c_uint64)]


class _Random:
    def __init__(self, seed, lib):
        self.g, self.lib = torch.Generator(device="cuda").manual_seed(seed), lib

    def normal(self, *shape):
        return torch.randn(*shape, device="cuda", generator=self.g)

    def uniform(self, n):
        return torch.rand(n, device="cuda", generator=self.g)

    def packed(self, n, quant, std=0.02):
        w = self.normal(n).mul_(std)
        be, bb = BLOCK[quant]
        out = torch.empty(n // be * bb, dtype=torch.uint8, device="cuda")
        self.lib.b200_quantize(w, out, n, KIND[quant])
        return out

    def tokens(self, vocab, *shape):
        return torch.randint(0, vocab, shape, device="cuda", generator=self.g, dtype=torch.int32)

    def mamba(self, d, heads, d_head, d_state, k, quant):
        d_inner = heads * d_head
        conv_dim = d_inner + 2 * d_state
        return dict(w_in=self.packed((d_inner + conv_dim + heads) * d, quant), conv_w=self.normal(conv_dim * k) * 0.1,
                    conv_b=self.normal(conv_dim) * 0.1, dt_bias=torch.log(torch.expm1(self.uniform(heads) * (1e-1 - 1e-3) + 1e-3)),
                    a_log=self.uniform(heads) * math.log(16.0), D=self.normal(heads), norm_w=1 + 0.1 * self.normal(d_inner),
                    w_out=self.packed(d * d_inner, quant))

    def moe(self, d, E, ne, SH, quant):
        """Router logits of unit variance and a bias on the scale of a probability: skewed, ragged expert loads."""
        return dict(router=self.normal(ne * d) / math.sqrt(d), router_bias=self.normal(ne) * 0.5 / ne,
                    gate=self.packed(ne * E * d, quant), up=self.packed(ne * E * d, quant), down=self.packed(ne * d * E, quant),
                    sh_gate=self.packed(SH * d, quant), sh_up=self.packed(SH * d, quant), sh_down=self.packed(d * SH, quant))


T_IDS = dict(embed=0, final_norm=1, lm_head=2, inv_freq=3, attn_norm=10, ffn_norm=11, w_in=20, conv_w=21, conv_b=22, dt_bias=23,
             a_log=24, D=25, norm_w=26, w_out=27, wq=30, wk=31, wv=32, wo=33, router=40, router_bias=41, gate=42, up=43, down=44,
             sh_gate=45, sh_up=46, sh_down=47)


class _Decoder:
    """A model's weights on the device, bound to a b200_decoder."""

    def __init__(self, lib, r, m, quant, batch, max_ctx):
        self.lib, self.kept, self.handle, self.model, self.batch = lib, [], C.c_void_p(), m, batch
        types = np.array(m["layer_types"], np.int32)
        d, hd, ne = m["hidden"], m["head_dim"], m["n_experts"]
        lib.b200_decoder_create(C.byref(self.handle), batch, m["vocab"], d, len(types), types.ctypes.data, m["n_heads"], m["n_kv"],
                                hd, m["rope_type"], m["mamba_heads"], m["d_head"], m["d_state"], m["d_conv"], ne, m["top_k"],
                                m["expert_dim"], m["shared_dim"], max_ctx, PAGE, KIND[quant], 1e-5, m["embedding_multiplier"],
                                m["residual_multiplier"], m["attn_scale"], m["logits_scaling"])
        emb = (r.normal(m["vocab"] * d) * 0.02).half()
        self.put(-1, embed=emb, lm_head=emb, final_norm=1 + 0.1 * r.normal(d))
        if m["rope_type"] >= 0:
            self.put(-1, inv_freq=(1.0 / 1e4 ** (torch.arange(hd // 2, device="cuda") * 2.0 / hd)).float())
        for l, t in enumerate(m["layer_types"]):
            self.put(l, attn_norm=1 + 0.1 * r.normal(d), ffn_norm=1 + 0.1 * r.normal(d))
            if t == 0:
                self.put(l, **r.mamba(d, m["mamba_heads"], m["d_head"], m["d_state"], m["d_conv"], quant))
            else:
                q, kv = m["n_heads"] * hd, m["n_kv"] * hd
                self.put(l, wq=r.packed(q * d, quant), wk=r.packed(kv * d, quant), wv=r.packed(kv * d, quant),
                         wo=r.packed(d * q, quant))
            self.put(l, **r.moe(d, m["expert_dim"], ne, m["shared_dim"], quant))
        # the fused step where the library takes the model and the batch, the per-op step otherwise
        if batch > DECODE_FUSED_MAX or lib.raw("b200_decoder_configure", self.handle, 1, 1) != 0:
            lib.b200_decoder_configure(self.handle, 0, 1)

    def put(self, layer, **tensors):
        for name, t in tensors.items():
            self.kept.append(t)
            self.lib.b200_decoder_set_tensor(self.handle, layer, T_IDS[name], t)

    def __del__(self):
        if self.handle:
            torch.cuda.synchronize()
            self.lib.b200_decoder_destroy(self.handle)
            self.handle = None


def prepare(case, seed):
    lib = importlib.import_module(PKG).lib()
    r = _Random(seed, lib)
    s = dict(case=case, lib=lib)
    if case["kind"] in ("generate", "prompt"):
        m, n, lens = MODELS[case["model"]], case["batch"], _lengths(case)
        steps = case.get("steps", 0)
        s["dec"] = _Decoder(lib, r, m, case["quant"], n, case["hi"] + steps + 1)
        s["ragged"] = None if len(set(lens)) == 1 else np.array(lens, np.int32)
        s["T"] = lens[0]
        s["prompt"] = r.tokens(m["vocab"], sum(lens))
        s["tokens"] = r.tokens(m["vocab"], max(steps, 1), n)
        s["tokens_host"] = s["tokens"].cpu().numpy()
        s["next"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        s["next_host"] = np.zeros(n, np.int32)
        s["logits"] = torch.zeros(n, m["vocab"], device="cuda")
        if case.get("sampled"):
            lib.b200_decoder_set_sampling(s["dec"].handle, C.byref(_Sampling(0.8, 0.95, 0.0, 1.1, 0.0, 0.0, 40, 64, 0, 0, seed)))
    elif case["kind"] == "moe":
        m, T = MOE[case["shape"]], case["tokens"]
        s.update(r.moe(m["d"], m["E"], m["ne"], m["SH"], case["quant"]))
        s["x"] = r.normal(T, m["d"])
        s["out"] = torch.empty(T, m["d"], device="cuda")
        s["idx"] = torch.empty(T, m["K"], dtype=torch.int32, device="cuda")
        s["w"] = torch.empty(T, m["K"], device="cuda")
    elif case["kind"] == "mamba":
        m, B, T = MAMBA[case["shape"]], case["batch"], case["steps"]
        s.update(r.mamba(m["d"], m["heads"], m["d_head"], m["d_state"], 4, case["quant"]))
        s["x"] = r.normal(B, T, m["d"])
        s["out"] = torch.empty(B, T, m["d"], device="cuda")
        s["state"] = torch.empty(B, m["heads"], m["d_head"], m["d_state"], device="cuda")
    else:
        m, lens = ATTN[case["shape"]], _lengths(case)
        pages = [-(-n // PAGE) for n in lens]
        pool, most = sum(pages), max(pages)
        order = torch.randperm(pool, device="cuda", generator=r.g).int()     # pages as a serving pool hands them out
        table = torch.zeros(len(lens), most, dtype=torch.int32, device="cuda")
        at = 0
        for i, p in enumerate(pages):
            table[i, :p] = order[at:at + p]
            at += p
        s["table"], s["most"] = table, most
        s["lens"] = torch.tensor(lens, dtype=torch.int32, device="cuda")
        s["q"] = r.normal(len(lens), m["H"], m["hd"])
        s["k"], s["v"] = (r.normal(pool * PAGE, m["KV"] * m["hd"]).half() for _ in range(2))
        s["out"] = torch.empty_like(s["q"])
    return s


def run(s):
    case, lib = s["case"], s["lib"]
    if case["kind"] in ("generate", "prompt"):
        h = s["dec"].handle
        lib.b200_decoder_reset(h)
        if s["ragged"] is None:
            lib.b200_decoder_prefill(h, s["prompt"], s["T"], s["next"])
        else:
            lib.b200_decoder_prefill_ragged(h, s["prompt"], s["ragged"].ctypes.data, s["next"])
        for i in range(case.get("steps", 0)):
            if case["host"]:
                lib.b200_decoder_step_host(h, s["tokens_host"][i].ctypes.data, s["next_host"].ctypes.data)
            else:
                lib.b200_decoder_step(h, s["tokens"][i], s["next"])
        p = C.c_void_p()
        lib.b200_decoder_logits(h, C.byref(p))
        lib.b200_copy_f32(s["logits"], p.value, s["logits"].numel())
        return {"logits": s["logits"]}
    if case["kind"] == "moe":
        m = MOE[case["shape"]]
        lib.b200_moe_forward_bias_half(s["x"], s["router"], s["router_bias"], s["gate"], s["up"], s["down"], s["sh_gate"],
                                       s["sh_up"], s["sh_down"], s["out"], None, s["idx"], s["w"], None, None, None,
                                       case["tokens"], m["d"], m["E"], m["ne"], m["K"], m["SH"], KIND[case["quant"]])
        return {"out": s["out"], "idx": s["idx"], "w": s["w"]}
    if case["kind"] == "mamba":
        m = MAMBA[case["shape"]]
        d_inner = m["heads"] * m["d_head"]
        s["state"].zero_()                                                   # empty sequences
        lib.b200_mamba2_forward_half(s["x"], s["w_in"], s["conv_w"], s["conv_b"], s["dt_bias"], s["a_log"], s["D"], s["norm_w"],
                                     s["w_out"], s["state"], s["out"], case["batch"], case["steps"], m["d"], d_inner,
                                     d_inner + 2 * m["d_state"], m["heads"], m["d_head"], m["d_state"], 4, 1e-5,
                                     KIND[case["quant"]])
        return {"out": s["out"], "state": s["state"]}
    m = ATTN[case["shape"]]
    lib.b200_attention_decode_paged_fp16(s["q"], s["k"], s["v"], s["table"], s["lens"], s["out"], case["batch"], s["most"], PAGE,
                                         m["H"], m["KV"], m["hd"], 1.0 / math.sqrt(m["hd"]))
    return {"out": s["out"]}


def _moe_work(T, d, E, ne, K, SH, wb):
    """Weights of the experts that T tokens touch (expected), router, shared expert; (weight bytes, flops)."""
    touched = ne * (1 - (1 - K / ne) ** T)
    return (touched * 3 * E * d + 3 * SH * d) * wb + ne * d * 4, 2.0 * T * (K * 3 * E * d + 3 * SH * d + ne * d)


def _model_work(m, wb, rows, ctx, seqs, heads):
    """One pass of `rows` new tokens of `seqs` sequences whose queries meet `ctx` keys in all; `heads` rows of logits."""
    d, di = m["hidden"], m["mamba_heads"] * m["d_head"]
    conv = di + 2 * m["d_state"]
    proj, q, kv = di + conv + m["mamba_heads"], m["n_heads"] * m["head_dim"], m["n_kv"] * m["head_dim"]
    state = m["mamba_heads"] * m["d_head"] * m["d_state"] + conv * (m["d_conv"] - 1)
    b, f = m["vocab"] * d * 2.0 + heads * m["vocab"] * 4, 2.0 * heads * m["vocab"] * d
    for t in m["layer_types"]:
        mb, mf = _moe_work(rows, d, m["expert_dim"], m["n_experts"], m["top_k"], m["shared_dim"], wb)
        b, f = b + mb, f + mf
        if t == 0:
            b += (proj + di) * d * wb + 2.0 * seqs * state * 4
            f += 2.0 * rows * (proj + di) * d + 6.0 * rows * di * m["d_state"]
        else:
            b += (2 * q + 2 * kv) * d * wb + 2.0 * 2 * kv * (ctx if rows == seqs else rows)
            f += 2.0 * rows * (2 * q + 2 * kv) * d + 4.0 * ctx * q
    return b, f


def work(case):
    wb = BLOCK[case["quant"]][1] / BLOCK[case["quant"]][0] if "quant" in case else 2.0
    if case["kind"] in ("generate", "prompt"):
        m, lens, n = MODELS[case["model"]], _lengths(case), case["batch"]
        b, f = _model_work(m, wb, sum(lens), sum(x * (x + 1) // 2 for x in lens), n, n)
        for i in range(case.get("steps", 0)):
            sb, sf = _model_work(m, wb, n, sum(lens) + (i + 1) * n, n, n)
            b, f = b + sb, f + sf
        return {"bytes": b, "flops": f}
    if case["kind"] == "moe":
        m, T = MOE[case["shape"]], case["tokens"]
        b, f = _moe_work(T, m["d"], m["E"], m["ne"], m["K"], m["SH"], wb)
        return {"bytes": b + 8.0 * T * (m["d"] + m["K"]), "flops": f}
    if case["kind"] == "mamba":
        m, rows = MAMBA[case["shape"]], case["batch"] * case["steps"]
        di = m["heads"] * m["d_head"]
        both = (3 * di + 2 * m["d_state"] + m["heads"]) * m["d"]               # in_proj and out_proj
        return {"bytes": both * wb + 8.0 * rows * m["d"] + 4.0 * case["batch"] * di * m["d_state"],
                "flops": 2.0 * rows * both + 6.0 * rows * di * m["d_state"]}
    m, n = ATTN[case["shape"]], sum(_lengths(case))
    return {"bytes": 4.0 * n * m["KV"] * m["hd"] + 8.0 * case["batch"] * m["H"] * m["hd"], "flops": 4.0 * n * m["H"] * m["hd"]}


def tolerance(case):
    if case["kind"] in ("generate", "prompt"):
        # fp16 operands through up to 40 layers, and near-ties of the router among the experts that come out the other way
        return {"rel": 1e-2, "max": 0.1} if case["model"] == "htiny" else {"rel": 3e-3, "max": 3e-2}
    if case["kind"] == "moe":
        # up to 8 tokens in fp32 on the exact weights; from there on fp16 operands.  The routing is exact.
        return {"rel": 5e-5, "max": 1e-3} if case["tokens"] <= 8 else {"rel": 2e-3, "max": 2e-2}
    if case["kind"] == "mamba":
        return {"rel": 3e-3, "max": 5e-2}                                    # fp16 operands in the projections and the scan
    return {"rel": 1e-4, "max": 1e-3}                                        # fp32 on fp16 keys and values
