"""What a program that serves with this package has it do, as cases that can be timed and checked one by one.

The kinds, and what each stands for:

  llama      a request of the prompt-cache path: `CacheEngine.process` on a prompt whose modules are cached, then the model's
             forward of the uncached suffix over them (7B layer sizes, four of the 32 layers and the head).  A short suffix
             reads the cached rows in place; a long one copies them first and runs the long-suffix attention.
  attn       attention over the slot pool, the call every slot-pool model makes once per attention layer: prompts and
             continued prompts of several sequences, and decoding (one token of each sequence).  `variant` is the model
             whose options are set: "bias" (logarithmic distance bias and a sink: Mutolix), "window" (capped scores under a sliding window that
             keeps the first keys: Raritar), "chunk" (tabulated bias inside chunks: Zovolorn), "gated" (per-head sinks and gates:
             Safilorn, Zovolorn), "plain" (Zepilix).  bfloat16, or float32 as `bin/trace_run --dtype float32` runs it.
  mlstm      the matrix-memory recurrence of a prompt (Mutolix, Tevilix)
  delta      the gated delta rule of a prompt, with one decay per channel (Zovolorn) or per head (Zepilix)
  gla        gated linear attention of a prompt (Safilorn)
  moe        a mixture-of-experts feed-forward of a prompt: router, chosen experts, weighted sum (Raritar)
  model      a whole Mutolix model of the benchmark's small size: prompts of a few sequences as one step, then decoding

Sizes are those of bench.py's models (widths 1024 and 2048; 8 or 16 heads of 128; recurrent heads of 128 x 256 and 256 x 512),
of the prompt-cache configuration (7 segments, 2048 cached tokens, 16 new ones) and the ranges around them.
"""
import math
import re

import torch
import torch.nn.functional as F

DEV = torch.device("cuda", 0)
BF, F32, F64 = torch.bfloat16, torch.float32, torch.float64
EPS = 1e-5


def listed():
    return [
        # the headline request: 16 new tokens over 7 cached segments of 2048 tokens
        dict(name="llama_cached_prompt", kind="llama", segments="24,400,400,400,400,400,24", suffix=16, layers=4),
        # a user's long question behind a cached document
        dict(name="llama_long_suffix", kind="llama", segments="24,400,400,176,24", suffix=700, layers=4),
        # an attention layer of the width-2048 benchmark model over one prompt
        dict(name="attn_prompt_2k", kind="attn", variant="bias", lens="2048", pos0="0", heads=16, kv=4, dim=128, vdim=128, dtype="bf16"),
        # long prompts of two users in one step
        dict(name="attn_prompt_long", kind="attn", variant="plain", lens="6144,2311", pos0="0,0", heads=16, kv=4, dim=128, vdim=128, dtype="bf16"),
        # chat turns that continue stored sequences under a window
        dict(name="attn_window_turns", kind="attn", variant="window", lens="700,1301,64,333", pos0="3000,511,1777,4096", heads=16, kv=4, dim=128,
             vdim=128, dtype="bf16"),
        # one decoded token of 16 sequences
        dict(name="attn_decode_16", kind="attn", variant="gated", lens=",".join(["1"] * 16),
             pos0=",".join(str(4096 - (i * 613) % 2049) for i in range(16)), heads=16, kv=4, dim=128, vdim=128, dtype="bf16"),
        # the 32-bit mode over a prompt
        dict(name="attn_prompt_f32", kind="attn", variant="bias", lens="1024", pos0="0", heads=8, kv=2, dim=128, vdim=128, dtype="f32"),
        # recurrent layers of the width-2048 benchmark models over one prompt, and of two unequal ones
        dict(name="mlstm_prompt", kind="mlstm", lens="2048", heads=4, dim=256, vdim=512),
        dict(name="delta_prompt", kind="delta", lens="2048", heads=4, kv=2, dim=256, vdim=512, per_head=False),
        dict(name="gla_prompts", kind="gla", lens="1500,548", heads=4, dim=256, vdim=512),
        # an expert layer of the width-2048 benchmark model over one prompt
        dict(name="moe_prompt", kind="moe", tokens=2048, width=2048, ff=1024, experts=16, top=4, groups=4, keep=2),
        # four short requests end to end
        dict(name="model_requests", kind="model", prompts="384,130,57,256", new=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _parts(rng, total, n, least=1):
    """`total` cut into n uneven parts of at least `least`."""
    w = [rng.uniform(0.2, 1.0) for _ in range(n)]
    return [max(least, int(total * x / sum(w))) for x in w]


def draw(rng):
    kind = rng.choice(("llama", "attn", "attn", "attn", "decode", "f32", "mlstm", "delta", "gla", "moe", "model"))
    csv = lambda v: ",".join(str(x) for x in v)
    if kind == "llama":
        return dict(kind="llama", segments=csv(_parts(rng, _log(rng, 200, 3000), rng.randint(2, 8), 8)), suffix=_log(rng, 2, 700), layers=rng.randint(2, 4))
    if kind in ("attn", "decode", "f32"):
        heads, kv = rng.choice(((8, 2), (16, 4), (16, 16), (12, 3)))
        dim, vdim = rng.choice(((128, 128), (128, 128), (64, 64), (192, 128)))
        variant = rng.choice(("bias", "window", "chunk", "gated", "plain"))
        if kind == "decode":
            n = _log(rng, 1, 16)
            lens, pos0 = [1] * n, [_log(rng, 100, 6000) for _ in range(n)]
        elif kind == "f32":
            n, heads, kv = rng.randint(1, 2), 8, 2
            lens = _parts(rng, _log(rng, 64, 1024), n, 16)
            pos0 = [rng.choice((0, _log(rng, 10, 400))) for _ in range(n)]
        else:
            n = rng.randint(1, 4)
            lens = _parts(rng, _log(rng, 200, 7000), n, 16)
            pos0 = [rng.choice((0, 0, _log(rng, 10, 4000))) for _ in range(n)]
        return dict(kind="attn", variant=variant, lens=csv(lens), pos0=csv(pos0), heads=heads, kv=kv, dim=dim, vdim=vdim,
                    dtype="f32" if kind == "f32" else "bf16")
    if kind in ("mlstm", "delta", "gla"):
        heads = rng.choice((2, 4, 8))
        dim, vdim = rng.choice(((64, 128), (128, 256), (128, 128), (256, 512)))
        case = dict(kind=kind, lens=csv(_parts(rng, _log(rng, 150, 4096), rng.randint(1, 3), 70)), heads=heads, dim=dim, vdim=vdim)
        if kind == "delta":
            case.update(kv=rng.choice((1, heads // 2, heads)), per_head=rng.random() < 0.5)
        return case
    if kind == "moe":
        return dict(kind="moe", tokens=_log(rng, 40, 4096), width=rng.choice((1024, 2048)), ff=rng.choice((512, 1024)), experts=rng.choice((8, 16)),
                    top=rng.choice((2, 4)), groups=rng.choice((2, 4)), keep=2)
    return dict(kind="model", prompts=csv([_log(rng, 20, 700) for _ in range(rng.randint(1, 4))]), new=rng.randint(4, 24))


def _ints(text):
    return [int(x) for x in str(text).split(",")]


# ---- inputs: plain tensors from the seed alone --------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _attn_inputs(case, seed):
    g = _gen(seed)
    lens, pos0 = _ints(case["lens"]), _ints(case["pos0"])
    H, G, D, V, dt = case["heads"], case["kv"], case["dim"], case["vdim"], F32 if case["dtype"] == "f32" else BF
    T, B = sum(lens), len(lens)
    cap = (max(n + p for n, p in zip(lens, pos0)) + 127) // 128 * 128
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x = dict(lens=lens, pos0=pos0, cap=cap, q=(rnd(T, H * D) * 1.5).to(dt), k=rnd(B, G, cap, D).to(dt), v=rnd(B, G, cap, V).to(dt), scale=D ** -0.5, opt={})
    # rows that no token may read hold what an earlier sequence of the slot left there: ordinary numbers
    if case["variant"] == "bias":
        x["opt"] = dict(r1=rnd(H).abs() * 0.1 + 0.5, r2=rnd(H).abs() * 0.1 + 0.5, sink=True)
    elif case["variant"] == "window":
        x["opt"] = dict(softcap=30.0, window=1024, keep_first=8)
    elif case["variant"] == "chunk":
        d = torch.arange(1024, device=DEV).float()
        x["opt"] = dict(chunk=1024, bias_table=(rnd(H, 1) * 0.3 - 0.2 * torch.log1p(d / 8)).contiguous(), head_scale=rnd(H).abs() * 0.2 + 0.9, out_scale=0.5 ** 0.5)
    elif case["variant"] == "gated":
        x["opt"] = dict(sink=True, sink_logit=rnd(H) * 0.5, head_gate=rnd(T, H).to(dt))
    return x


def _recurrent_inputs(case, seed):
    g = _gen(seed)
    lens, H, D, V = _ints(case["lens"]), case["heads"], case["dim"], case["vdim"]
    T = sum(lens)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x = dict(lens=lens, H=H, D=D, V=V)
    if case["kind"] == "mlstm":
        x.update(proj=rnd(T, 2 * H * D + 2 * H * V).to(BF), offs=(0, H * D, 2 * H * D, 2 * H * D + H * V), ig=rnd(T, H),
                 fg=F.logsigmoid(rnd(T, H) + 3.0), w=(1 + 0.05 * rnd(H * V)).to(BF))
    elif case["kind"] == "gla":
        x.update(proj=rnd(T, 2 * H * D + 2 * H * V).to(BF), offs=(0, H * D, 2 * H * D, 2 * H * D + H * V), ld=F.logsigmoid(rnd(T, H * D) + 1.0) / 16,
                 w=(1 + 0.05 * rnd(V)).to(BF))
    else:
        kv = case["kv"]
        unit = lambda t: t / t.norm(dim=-1, keepdim=True)
        q, k = unit(rnd(T, kv, D)) * D ** -0.5, unit(rnd(T, kv, D))
        x.update(kv=kv, qk=torch.cat([q.reshape(T, -1), k.reshape(T, -1)], 1).contiguous(), v=rnd(T, H * V).to(BF), b=rnd(T, H).to(BF),
                 gate=rnd(T, H * V).to(BF), w=(1 + 0.05 * rnd(V)).to(BF), ld=None, head=None)
        rate = torch.exp(rnd(H) * 0.5 - 2.0)
        if case["per_head"]:
            x["head"] = (rnd(T, H).to(BF), rnd(H) * 0.5, rate)
        else:
            x["ld"] = (-rate[:, None] * F.softplus(rnd(T, H, D))).reshape(T, H * D).contiguous()
    return x


def _moe_inputs(case, seed):
    g = _gen(seed)
    T, W, ff, E = case["tokens"], case["width"], case["ff"], case["experts"]
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    return dict(h=rnd(T, W).to(BF), router=(rnd(E, W) * 3 * W ** -0.5).to(BF), correction=rnd(E) * 0.05, w_gu=(rnd(E, 2 * ff, W) * W ** -0.5).to(BF),
                w_down=(rnd(E, W, ff) * ff ** -0.5).to(BF))


LLAMA = dict(vocab_size=32000, hidden_size=4096, intermediate_size=11008, num_attention_heads=32, num_key_value_heads=32, max_position_embeddings=4096,
             rms_norm_eps=1e-5)


def _llama_weights(case, seed):
    g = _gen(seed)
    hid, inter, vocab = LLAMA["hidden_size"], LLAMA["intermediate_size"], LLAMA["vocab_size"]
    rnd = lambda *s, std=0.02, mean=0.0: (torch.randn(*s, generator=g, device=DEV, dtype=torch.half) * std + mean)
    sd = {"model.embed_tokens.weight": rnd(vocab, hid, std=1.0), "model.norm.weight": rnd(hid, std=0.05, mean=1.0), "lm_head.weight": rnd(vocab, hid)}
    for l in range(case["layers"]):
        p = f"model.layers.{l}."
        for n in ("q", "k", "v", "o"):
            sd[p + f"self_attn.{n}_proj.weight"] = rnd(hid, hid)
        for n in ("gate", "up"):
            sd[p + f"mlp.{n}_proj.weight"] = rnd(inter, hid)
        sd[p + "mlp.down_proj.weight"] = rnd(hid, inter)
        for n in ("input_layernorm", "post_attention_layernorm"):
            sd[p + n + ".weight"] = rnd(hid, std=0.05, mean=1.0)
    return sd


def _llama_text(case, seed):
    from promptcache_b200.synthetic import flat_schema
    return flat_schema("doc", _ints(case["segments"]), case["suffix"], LLAMA["vocab_size"], seed=int(seed))


MUTOLIX = dict(width=1024, heads=8, kv_heads=2, dim=128, vdim=128, m_heads=4, m_dim=128, m_vdim=256, ff=4096, vocab=8192)


def _mutolix_config():
    m = MUTOLIX
    mlp = {"kind": "dense", "ff": m["ff"]}
    attn = {"type": "attention", "mlp": mlp, "mixer": {"heads": m["heads"], "kv_heads": m["kv_heads"], "dim": m["dim"], "vdim": m["vdim"], "scale": m["dim"] ** -0.5,
                                                       "v_mix": True, "q_temp": {"coef": 0.3, "every": 256}}}
    rec = {"type": "mlstm", "mlp": mlp, "mixer": {"heads": m["m_heads"], "dim": m["m_dim"], "vdim": m["m_vdim"], "gate_cap": 12.0}}
    return {"architecture": "Mutolix", "vocab": m["vocab"], "width": m["width"], "embedding": {"scale": 1.0}, "norm": {"eps": EPS},
            "layers": [rec, attn, attn, rec]}


def _mutolix_weights(cfg, seed):
    g = _gen(seed)
    W, t = cfg["width"], {}
    rnd = lambda *s, std=1.0, mean=0.0: (torch.randn(*s, generator=g, device=DEV) * std + mean).to(BF)
    lin = lambda o, i: rnd(o, i, std=i ** -0.5)
    t["embed"], t["final.norm"], t["head"] = rnd(cfg["vocab"], W), rnd(W, std=0.05, mean=1.0), lin(cfg["vocab"], W)
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        for n in ("norm1", "norm1b", "norm2", "norm2b"):
            t[p + n] = rnd(W, std=0.05, mean=1.0)
        for n in ("ls1", "ls2"):
            t[p + n] = rnd(W, std=0.1, mean=0.5)
        for n in ("rg1", "rg2"):
            t[p + n], t[p + n + ".b"] = lin(W, W), rnd(W, std=0.3)
        H, D, V = m["heads"], m["dim"], m["vdim"]
        if layer["type"] == "mlstm":
            for n, r in (("q", H * D), ("k", H * D), ("v", H * V), ("g", H * V)):
                t[p + "mix." + n] = lin(r, W)
            t[p + "mix.norm"] = rnd(H * V, std=0.05, mean=1.0)
            t[p + "mix.i"], t[p + "mix.i.b"], t[p + "mix.f"], t[p + "mix.f.b"] = lin(H, W), rnd(H), lin(H, W), rnd(H, mean=3.0)
        else:
            G = m["kv_heads"]
            for n, r in (("q", H * D), ("k", G * D), ("v", G * V)):
                t[p + "mix." + n], t[p + "mix." + n + ".b"] = lin(r, W), rnd(r, std=0.1)
            t[p + "mix.q.norm"], t[p + "mix.k.norm"] = rnd(H * D, std=0.1, mean=1.0), rnd(G * D, std=0.1, mean=1.0)
            t[p + "mix.vmix"], t[p + "mix.r1"], t[p + "mix.r2"] = rnd(1, std=0.05, mean=0.4).reshape(()), rnd(H, std=0.05, mean=0.5).abs(), rnd(H, std=0.1, mean=0.5).abs()
        t[p + "mix.o"] = lin(W, H * V)
        ff = layer["mlp"]["ff"]
        t[p + "mlp.up"], t[p + "mlp.down"], t[p + "mlp.act"] = lin(ff, W), lin(W, ff), rnd(2, std=0.3)
    return t


def _mutolix_tokens(case, seed):
    g = torch.Generator().manual_seed(int(seed) + 1)
    return [torch.randint(0, MUTOLIX["vocab"], (n + case["new"],), generator=g).tolist() for n in _ints(case["prompts"])]


# ---- what a program has in hand before the call ------------------------------------------------------------------------------
def prepare(case, seed):
    from promptcache_b200 import _native_seq as nsq
    kind = case["kind"]
    if kind == "attn":
        x = _attn_inputs(case, seed)
        x["batch"] = nsq.Batch(range(len(x["lens"])), x["pos0"], x["lens"], DEV)
        x["out"] = torch.empty(sum(x["lens"]), case["heads"] * case["vdim"], dtype=x["q"].dtype, device=DEV)
    elif kind in ("mlstm", "gla", "delta"):
        x = _recurrent_inputs(case, seed)
        B, H, D, V, T = len(x["lens"]), x["H"], x["D"], x["V"], sum(x["lens"])
        x["batch"] = nsq.Batch(range(B), [0] * B, x["lens"], DEV)   # sequences that begin: their states start from zero in every pass
        x["s"], x["out"] = torch.zeros(B, H, D, V, device=DEV), torch.empty(T, H * V, dtype=BF, device=DEV)
        if kind == "mlstm":
            x["n"], x["m"] = torch.zeros(B, H, D, device=DEV), torch.zeros(B, H, device=DEV)
    elif kind == "moe":
        x = _moe_inputs(case, seed)
        x["x"] = torch.empty(case["tokens"], case["width"], device=DEV)
    elif kind == "llama":
        from promptcache_b200 import CacheEngine, Prompt
        from promptcache_b200.model import Llama2, LlamaConfigLite, LlamaForCausalLM
        from promptcache_b200.synthetic import IdTokenizer
        model = LlamaForCausalLM(LlamaConfigLite(**LLAMA, num_hidden_layers=case["layers"]), device=DEV)
        model.load_hf_state_dict(_llama_weights(case, seed))
        lm = Llama2("llama", model=model, tokenizer=IdTokenizer(LLAMA["vocab_size"]))
        text = _llama_text(case, seed)
        eng = CacheEngine((text.n_cached + text.q_len + 256 + 127) // 128 * 128, lm)
        eng.prompt_cache.retain_prefix = False   # requests come with modules of their own: no rows are left from the one before
        eng.add_schema(text.schema_xml)
        x = dict(lm=lm, eng=eng, prompt=Prompt(text.prompt_xml))
    else:
        from promptcache_b200.model.mutolix import MutolixConfig, MutolixForCausalLM
        cfg = _mutolix_config()
        x = dict(model=MutolixForCausalLM(MutolixConfig(cfg), _mutolix_weights(cfg, seed), device=DEV, dtype=BF), tokens=_mutolix_tokens(case, seed))
        x["lens"], x["new"] = _ints(case["prompts"]), case["new"]
    x["case"] = dict(case)
    return x


# ---- one pass -------------------------------------------------------------------------------------------------------------
@torch.inference_mode()
def run(x):
    from promptcache_b200 import _native_seq as nsq
    case = x["case"]
    kind = case["kind"]
    if kind == "attn":
        opt = dict(x["opt"])
        r1, r2, sink = opt.pop("r1", None), opt.pop("r2", None), opt.pop("sink", False)
        T = x["q"].shape[0]
        if T <= 16:   # as the models call it for a decoding step
            opt.update(workspace=nsq.attn_workspace(T, case["heads"], case["vdim"], DEV), max_keys=min(x["cap"], opt.get("chunk") or x["cap"]))
        nsq.attention(x["q"], x["k"], x["v"], x["out"], case["heads"], x["scale"], r1, r2, sink, x["batch"], **opt)
        return x["out"]
    if kind == "mlstm":
        nsq.mlstm_scan(x["proj"], x["offs"], x["ig"], x["fg"], x["w"], x["out"], x["s"], x["n"], x["m"], EPS, x["batch"])
        return {"out": x["out"], "s": x["s"], "n": x["n"], "m": x["m"]}
    if kind == "gla":
        nsq.gla_scan(x["proj"], x["offs"], x["ld"], x["w"], x["out"], x["s"], EPS, x["batch"])
        return {"out": x["out"], "s": x["s"]}
    if kind == "delta":
        nsq.delta_scan(x["qk"], x["v"], x["ld"], x["b"], x["kv"], x["s"], x["w"], x["gate"], x["out"], EPS, x["batch"], head_decay=x["head"],
                       gate_silu=x["head"] is not None)
        return {"out": x["out"], "s": x["s"]}
    if kind == "moe":
        idx, wgt, _ = nsq.moe_route(x["h"], x["router"], x["correction"], None, case["top"], case["groups"], case["keep"])
        y, rows = nsq.moe_experts(x["h"], idx, x["w_gu"], x["w_down"])
        nsq.moe_combine(x["x"], y, idx, wgt, x["h"], case["experts"], 0.8, y_row=rows, overwrite=True)
        return {"x": x["x"], "idx": idx, "wgt": wgt}
    if kind == "llama":
        ids, pos, _, cache = x["eng"].process(x["prompt"])
        both = torch.tensor([ids, pos], device=DEV, dtype=torch.long)
        out = x["lm"](input_ids=both[0:1], position_ids=both[1:2], past_key_values=cache.batched(), use_cache=True, max_position=max(pos))
        return out.logits
    m, seqs, got = x["model"], [x["model"].new_sequence() for _ in x["lens"]], []
    got.append(m.step([(s, t[:n]) for s, t, n in zip(seqs, x["tokens"], x["lens"])]))
    for i in range(x["new"]):
        got.append(m.step([(s, t[n + i:n + i + 1]) for s, t, n in zip(seqs, x["tokens"], x["lens"])]))
    for s in seqs:
        s.free()
    return torch.stack(got)


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------
def _visible(case, lens, pos0):
    """((query, key) pairs, key rows read by some query) of all entries."""
    win, keep, chunk = (1024, 8, 0) if case["variant"] == "window" else (0, 0, 1024 if case["variant"] == "chunk" else 0)
    pairs = rows = 0
    for n, p0 in zip(lens, pos0):
        for p in range(p0, p0 + n):
            pairs += min(p + 1, win) + max(0, min(keep, p + 1 - win)) if win else p % chunk + 1 if chunk else p + 1
        lo = max(0, p0 - win + 1) if win else p0 // chunk * chunk if chunk else 0
        rows += p0 + n - lo + min(keep, lo)
    return pairs, rows


def work(case):
    kind = case["kind"]
    if kind == "attn":
        lens, pos0 = _ints(case["lens"]), _ints(case["pos0"])
        pairs, rows = _visible(case, lens, pos0)
        size, H, D, V = 4 if case["dtype"] == "f32" else 2, case["heads"], case["dim"], case["vdim"]
        return {"bytes": size * (rows * case["kv"] + sum(lens) * H) * (D + V), "flops": 2 * (D + V) * H * pairs}
    if kind in ("mlstm", "gla", "delta"):
        T, B, H, D, V = sum(_ints(case["lens"])), len(_ints(case["lens"])), case["heads"], case["dim"], case["vdim"]
        state = 4 * B * H * D * V
        if kind == "mlstm":
            return {"bytes": 2 * T * H * (2 * D + 3 * V) + 8 * T * H + state, "flops": 4 * T * H * D * V}
        if kind == "gla":
            return {"bytes": 2 * T * H * (2 * D + 3 * V) + 4 * T * H * D + state, "flops": 4 * T * H * D * V}
        return {"bytes": 8 * T * case["kv"] * D + 6 * T * H * V + (2 if case["per_head"] else 4 * D) * T * H + state, "flops": 6 * T * H * D * V}
    if kind == "moe":
        T, W, ff, E = case["tokens"], case["width"], case["ff"], case["experts"]
        return {"bytes": 6 * E * W * ff + 6 * T * W, "flops": 6 * T * case["top"] * W * ff + 2 * T * E * W}
    if kind == "llama":
        hid, inter, vocab, N, q = 4096, 11008, 32000, sum(_ints(case["segments"])), case["suffix"]
        params = case["layers"] * (4 * hid * hid + 3 * hid * inter) + vocab * hid
        return {"bytes": 2 * params + 4 * case["layers"] * hid * N + 4 * q * vocab, "flops": 2 * params * q + 4 * case["layers"] * hid * (N * q + q * (q + 1) // 2)}
    m, lens = MUTOLIX, _ints(case["prompts"])
    W = m["width"]
    rec = W * 2 * (m["m_heads"] * m["m_dim"] + m["m_heads"] * m["m_vdim"]) + W * m["m_heads"] * m["m_vdim"]
    att = W * (m["heads"] * m["dim"] + m["kv_heads"] * (m["dim"] + m["vdim"])) + W * m["heads"] * m["vdim"]
    params = 2 * (rec + att) + 4 * (2 * W * m["ff"] + 2 * W * W) + m["vocab"] * W
    steps, toks = case["new"] + 1, sum(lens) + case["new"] * len(lens)
    state = 2 * 8 * len(lens) * m["m_heads"] * m["m_dim"] * m["m_vdim"] + 2 * 4 * m["kv_heads"] * 128 * sum(lens)
    return {"bytes": steps * (2 * params + state), "flops": 2 * (params - m["vocab"] * W) * toks + 2 * m["vocab"] * W * steps * len(lens)}


def tolerance(case):
    """About four times what the path was measured to show against `exact`: 1.7e-3 where only the result is rounded to 16 bits (and over four fp16
    layers), 3.5e-3 over the three 16-bit products of the experts, 5.5e-3 over a whole bfloat16 model, 5.5e-7 in the 32-bit mode."""
    kind = case["kind"]
    if kind == "attn":
        return {"rel": 2.2e-6, "max": 1e-4} if case["dtype"] == "f32" else {"rel": 7e-3, "max": 0.06}
    if kind in ("mlstm", "gla", "delta"):
        return {"rel": 7e-3, "max": 0.06}
    if kind == "moe":
        return {"rel": 1.4e-2, "max": 0.1, "differ": 2e-3}   # choices whose scores lie within a rounding of each other
    if kind == "llama":
        return {"rel": 7e-3, "max": 0.06}
    return {"rel": 2.2e-2, "max": 0.2}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------------
def _rms(t, w=None):
    y = t / torch.sqrt((t * t).mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _attn64(q, k, v, p0, scale, o, h):
    """One head of one entry: q [n, D], k, v [p0 + n, *]; o: the options, h: the head."""
    n, dev = q.shape[0], q.device
    i, j = torch.arange(p0, p0 + n, device=dev)[:, None], torch.arange(p0 + n, device=dev)[None, :]
    s = q @ k.T * scale
    if "head_scale" in o:
        s = s * o["head_scale"][h].double()
    if "softcap" in o:
        s = o["softcap"] * torch.tanh(s / o["softcap"])
    if "r1" in o:
        s = s - o["r1"][h].double() * torch.log1p(o["r2"][h].double() * (i - j).clamp(min=0).double())
    if "bias_table" in o:
        t = o["bias_table"][h].double()
        s = s + t[(i - j).clamp(0, t.numel() - 1)]
    hidden = j > i
    if "window" in o:
        hidden = hidden | ((i - j >= o["window"]) & (j >= o["keep_first"]))
    if "chunk" in o:
        hidden = hidden | (i // o["chunk"] != j // o["chunk"])
    s = s.masked_fill_(hidden, -math.inf)
    sink = None if not o.get("sink") else o["sink_logit"][h].double() if "sink_logit" in o else torch.zeros((), dtype=F64, device=dev)
    mx = s.max(-1, keepdim=True).values
    if sink is not None:
        mx = torch.maximum(mx, sink)
    e = torch.exp(s - mx)
    den = e.sum(-1, keepdim=True) + (torch.exp(sink - mx) if sink is not None else 0.0)
    return e @ v / den


def _attn_exact(case, seed):
    x = _attn_inputs(case, seed)
    H, G, D, V = case["heads"], case["kv"], case["dim"], case["vdim"]
    out, off = torch.empty(sum(x["lens"]), H, V, dtype=F64, device=DEV), 0
    for b, (n, p0) in enumerate(zip(x["lens"], x["pos0"])):
        for h in range(H):
            g = h // (H // G)
            out[off:off + n, h] = _attn64(x["q"][off:off + n, h * D:(h + 1) * D].double(), x["k"][b, g, :p0 + n].double(), x["v"][b, g, :p0 + n].double(), p0,
                                          x["scale"], x["opt"], h)
        off += n
    if "head_gate" in x["opt"]:
        out *= torch.sigmoid(x["opt"]["head_gate"].double())[:, :, None]
    return (out * x["opt"].get("out_scale", 1.0)).reshape(-1, H * V)


def _mlstm64(q, k, v, ig, fg):
    """q (scaled), k [B, T, H, D], v [B, T, H, V], gates [B, T, H]: results [B, T, H, V] and the last S, n, m."""
    B, T, H, D = q.shape
    S, n, m = q.new_zeros(B, H, D, v.shape[-1]), q.new_zeros(B, H, D), q.new_zeros(B, H)
    out = torch.empty_like(v)
    for t in range(T):
        mn = torch.maximum(fg[:, t] + m, ig[:, t])
        a, b = torch.exp(fg[:, t] + m - mn), torch.exp(ig[:, t] - mn)
        kb = b[..., None] * k[:, t]
        S.mul_(a[..., None, None]).addcmul_(kb[..., None], v[:, t][..., None, :])
        n, m = a[..., None] * n + kb, mn
        den = torch.maximum((n * q[:, t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        out[:, t] = (S.transpose(-1, -2) @ q[:, t][..., None])[..., 0] / den[..., None]
    return out, S, n, m


def _recurrent_exact(case, seed):
    x = _recurrent_inputs(case, seed)
    H, D, V, kind, off, outs, states = x["H"], x["D"], x["V"], case["kind"], 0, [], []
    for T in x["lens"]:
        sl = slice(off, off + T)
        off += T
        if kind != "delta":
            o1, o2, o3, o4 = x["offs"]
            pr = x["proj"][sl].double()
            q, k, v, gate = pr[:, o1:o2].view(T, H, D) * D ** -0.5, pr[:, o2:o3].view(T, H, D), pr[:, o3:o4].view(T, H, V), pr[:, o4:]
        if kind == "mlstm":
            o, S, n, m = _mlstm64(q[None], k[None], v[None], x["ig"][sl].double()[None], x["fg"][sl].double()[None])
            outs.append(_rms(o[0]).reshape(T, H * V) * x["w"].double() * torch.sigmoid(gate))
            states.append((S[0], n[0], m[0]))
            continue
        S = torch.zeros(H, D, V, dtype=F64, device=DEV)
        o = torch.empty(T, H, V, dtype=F64, device=DEV)
        if kind == "gla":
            dec = torch.exp(x["ld"][sl].double()).view(T, H, D, 1)
            for t in range(T):
                S.mul_(dec[t]).addcmul_(k[t][..., None], v[t][:, None, :])
                o[t] = (S.transpose(-1, -2) @ q[t][..., None])[..., 0]
            gated = gate * torch.sigmoid(gate)
        else:
            kv = x["kv"]
            rep = lambda z: z.double().view(T, kv, D).repeat_interleave(H // kv, 1)
            q, k, v = rep(x["qk"][sl, :kv * D]), rep(x["qk"][sl, kv * D:]), x["v"][sl].double().view(T, H, V)
            if x["head"] is not None:
                a, bias, rate = x["head"]
                dec = torch.exp(-rate.double() * F.softplus(a[sl].double() + bias.double())).view(T, H, 1, 1).expand(T, H, D, 1)
            else:
                dec = torch.exp(x["ld"][sl].double()).view(T, H, D, 1)
            beta = torch.sigmoid(x["b"][sl].double())
            for t in range(T):
                S.mul_(dec[t])
                u = beta[t][:, None] * (v[t] - (S.transpose(-1, -2) @ k[t][..., None])[..., 0])
                S.addcmul_(k[t][..., None], u[:, None, :])
                o[t] = (S.transpose(-1, -2) @ q[t][..., None])[..., 0]
            gate = x["gate"][sl].double()
            gated = gate * torch.sigmoid(gate) if x["head"] is not None else torch.sigmoid(gate)
        outs.append((_rms(o) * x["w"].double()).reshape(T, H * V) * gated)
        states.append((S,))
    got = {"out": torch.cat(outs), "s": torch.stack([s[0] for s in states])}
    if kind == "mlstm":
        got.update(n=torch.stack([s[1] for s in states]), m=torch.stack([s[2] for s in states]))
    return got


def _moe_exact(case, seed):
    x = _moe_inputs(case, seed)
    E, top, ng, keep, ff = case["experts"], case["top"], case["groups"], case["keep"], case["ff"]
    h = x["h"].double()
    s = torch.softmax(h @ x["router"].double().T, -1)
    c = s + x["correction"].double()
    best = c.view(-1, ng, E // ng).max(-1).values.topk(keep, -1).indices
    open_ = torch.zeros(h.shape[0], ng, dtype=torch.bool, device=DEV).scatter_(1, best, True).repeat_interleave(E // ng, 1)
    idx = c.masked_fill(~open_, -math.inf).topk(top, -1).indices
    wgt = s.gather(1, idx)
    out = torch.zeros_like(h)
    for e in range(E):
        t, k = (idx == e).nonzero(as_tuple=True)
        gu = h[t] @ x["w_gu"][e].double().T
        out.index_add_(0, t, wgt[t, k][:, None] * ((F.silu(gu[:, :ff]) * gu[:, ff:]) @ x["w_down"][e].double().T))
    return {"x": 0.8 * out, "idx": None, "wgt": wgt}


def _llama_exact(case, seed):
    sd, text = _llama_weights(case, seed), _llama_text(case, seed)
    words = lambda xml: [int(n) for n in re.findall(r"\bt(\d+)\b", xml)]
    ids = torch.tensor(words(text.schema_xml) + words(text.prompt_xml), device=DEV)
    H, D, T = 32, 128, ids.numel()
    pos = torch.arange(T, device=DEV, dtype=F64)
    ang = pos[:, None] * (10000.0 ** (-torch.arange(0, D, 2, device=DEV, dtype=F64) / D))[None]
    cos, sin = torch.cat([ang.cos()] * 2, -1)[:, None], torch.cat([ang.sin()] * 2, -1)[:, None]
    turn = lambda z: z * cos + torch.cat([-z[..., D // 2:], z[..., :D // 2]], -1) * sin
    x = sd["model.embed_tokens.weight"][ids].double()
    for l in range(case["layers"]):
        w = lambda n: sd[f"model.layers.{l}.{n}.weight"].double()
        h = _rms(x, w("input_layernorm"))
        q, k, v = (h @ w(f"self_attn.{n}_proj").T for n in ("q", "k", "v"))
        q, k, v = turn(q.view(T, H, D)), turn(k.view(T, H, D)), v.view(T, H, D)
        a = torch.stack([_attn64(q[:, i], k[:, i], v[:, i], 0, D ** -0.5, {}, i) for i in range(H)], 1)
        x = x + a.reshape(T, H * D) @ w("self_attn.o_proj").T
        h = _rms(x, w("post_attention_layernorm"))
        x = x + (F.silu(h @ w("mlp.gate_proj").T) * (h @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T
    x = _rms(x[-case["suffix"]:], sd["model.norm.weight"].double())
    return (x @ sd["lm_head.weight"].double().T)[None]


def _xielu64(z, a):
    cp, cn = F.softplus(a[0]), 0.5 + F.softplus(a[1])
    neg = z.clamp(max=0.0)
    return torch.where(z > 0, cp * z * z + z / 2, cn * (torch.exp(neg) - 1 - neg) + z / 2)


def _mutolix_exact(case, seed):
    cfg = _mutolix_config()
    W = {k: t.double() for k, t in _mutolix_weights(cfg, seed).items()}
    logits = []
    for n, toks in zip(_ints(case["prompts"]), _mutolix_tokens(case, seed)):
        T = len(toks)
        x, first, pos = W["embed"][torch.tensor(toks, device=DEV)], None, torch.arange(T, device=DEV)
        for i, layer in enumerate(cfg["layers"]):
            w, m = (lambda s: W[f"l{i}.{s}"]), layer["mixer"]
            H, D, V = m["heads"], m["dim"], m["vdim"]
            h = _rms(x, w("norm1"))
            if layer["type"] == "mlstm":
                q, k, v = (h @ w("mix.q").T * D ** -0.5).view(1, T, H, D), (h @ w("mix.k").T).view(1, T, H, D), (h @ w("mix.v").T).view(1, T, H, V)
                capped = lambda s: m["gate_cap"] * torch.tanh((h @ w("mix." + s).T + w("mix." + s + ".b")) / m["gate_cap"])
                o = _mlstm64(q, k, v, capped("i")[None], F.logsigmoid(capped("f"))[None])[0][0]
                y = _rms(o).reshape(T, H * V) * w("mix.norm") * torch.sigmoid(h @ w("mix.g").T)
            else:
                G, t = m["kv_heads"], m["q_temp"]
                q, k = _rms(h @ w("mix.q").T + w("mix.q.b"), w("mix.q.norm")), _rms(h @ w("mix.k").T + w("mix.k.b"), w("mix.k.norm"))
                q = q * (1 + t["coef"] * torch.log(((pos + 1) // t["every"]).double() + 1))[:, None]
                v = h @ w("mix.v").T + w("mix.v.b")
                if first is None:
                    first = v
                else:
                    v = (1 - w("mix.vmix")) * v + w("mix.vmix") * first
                q, k, v = q.view(T, H, D), k.view(T, G, D), v.view(T, G, V)
                o = dict(r1=w("mix.r1"), r2=w("mix.r2"), sink=True)
                y = torch.stack([_attn64(q[:, j], k[:, j // (H // G)], v[:, j // (H // G)], 0, m["scale"], o, j) for j in range(H)], 1).reshape(T, H * V)
            y = y @ w("mix.o").T * torch.sigmoid(h @ w("rg1").T + w("rg1.b"))
            x = x + _rms(y, w("norm1b")) * w("ls1")
            h = _rms(x, w("norm2"))
            y = _xielu64(h @ w("mlp.up").T, w("mlp.act")) @ w("mlp.down").T * torch.sigmoid(h @ w("rg2").T + w("rg2.b"))
            x = x + _rms(y, w("norm2b")) * w("ls2")
        logits.append(_rms(x[n - 1:n + case["new"]], W["final.norm"]) @ W["head"].T)
    return torch.stack(logits, 1)


@torch.inference_mode()
def exact(case, seed):
    kind = case["kind"]
    return {"attn": _attn_exact, "moe": _moe_exact, "llama": _llama_exact, "model": _mutolix_exact}.get(kind, _recurrent_exact)(case, seed)
