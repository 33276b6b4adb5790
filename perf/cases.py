"""What a user of this library has it do, as cases that can be timed and compared.

Four kinds of pass, all through the public entry points:

* ``prompt``    ``Engine.step`` of whole prompts on fresh sequences, logits after each prompt's last token;
* ``decode``    one ``Engine.decode`` step of a batch whose sequences grow by a token per pass (a batch that has reached
                the longest context is released and its prompts run again, as a server takes the next batch);
* ``extend``    ``Engine.step`` that continues sequences by several tokens each, after which the cache goes back to where
                it was, as a conversation does when a reply is asked for again;
* ``generate``  ``LLM.generate``: prompts in as host lists, sampled ids out.

Tokens and weights are made from the seed.  Models have the layer sizes that ``bench.py`` measures: Gemma 2 2B (26 layers),
and eight layers of Fuposun, Tumudra and Vonulorn at the two widths that it sets side by side; the smallest is the tiny
Gemma 2 of the tests, in float32.  The tokens that a decode step is fed are drawn beforehand, so that the logits of two
implementations belong to the same sequence.  In Fuposun an embedding carries one of sixteen directions that the routers
look at: which experts a token goes to is then decided by a margin, as in a trained model, and not by a rounding.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from quicknn_b200.config import find_architecture
from quicknn_b200.engine import LLM, Model
from quicknn_b200.sampling import GenerationOptions

DEVICE = "cuda:0"
EXPERT_DIRECTIONS = 16
GROWTH = 1200                      # decode steps that a batch has room for before its prompts are run again


# ---- the models ---------------------------------------------------------------------------------------------------------

def config_of(model: str) -> dict:
    """``config.json`` of a model of the cases."""
    if model == "gemma2-tiny":
        return dict(architectures=["Gemma2ForCausalLM"], model_type="gemma2", hidden_size=96, intermediate_size=200,
                    num_attention_heads=6, num_key_value_heads=1, head_dim=24, vocab_size=1000, num_hidden_layers=3,
                    max_position_embeddings=1024, rope_theta=1e6, rms_norm_eps=1e-5, sliding_window=5,
                    attn_logit_softcapping=None, final_logit_softcapping=15.0, query_pre_attn_scalar=32, eos_token_id=1)
    if model == "gemma2-2b":
        return dict(architectures=["Gemma2ForCausalLM"], model_type="gemma2", hidden_size=2304, intermediate_size=9216,
                    num_attention_heads=8, num_key_value_heads=4, head_dim=256, vocab_size=256000, num_hidden_layers=26,
                    max_position_embeddings=8192, rope_theta=10000.0, rms_norm_eps=1e-6, sliding_window=4096,
                    attn_logit_softcapping=50.0, final_logit_softcapping=30.0, query_pre_attn_scalar=256, eos_token_id=1)
    design, size = model.split("-")
    W, ff, heads, hd, kvh, layers, vocab, window, rank, qr, d = {
        "2b": (2304, 9216, 8, 256, 4, 8, 32768, 4096, 256, 768, 128),
        "1b": (1536, 6144, 8, 128, 4, 8, 32768, 2048, 128, 512, 64)}[size]
    H = W // (2 * d)
    dense = {"kind": "dense", "ff": ff}
    if design == "fuposun":
        latent = {"heads": H, "dim": d, "vdim": d, "q_rank": qr, "kv_rank": rank, "scale": d ** -0.5, "mask": {"size": window}}
        gla = {"heads": H, "dim": d, "vdim": 2 * d, "tau": 8.0, "decay_rank": 64}
        moe = {"kind": "moe", "router": {"experts": 16, "top": 2}, "expert": {"ff": ff // 4, "limit": 7.0},
               "shared": {"ff": ff // 4, "limit": 7.0}}
        pattern = [("latent_attention", latent, dense), ("latent_attention", latent, moe), ("gla", gla, dense),
                   ("latent_attention", latent, moe)]
        return dict(architecture="Fuposun", vocab=vocab, width=W, residual_mult=0.5, logit_softcap=50.0, norm={"eps": 1e-6},
                    layers=[{"type": t, "mixer": m, "mlp": f} for t, m, f in (pattern * layers)[:layers]])
    if design == "tumudra":
        att = {"heads": heads, "kv_heads": kvh, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "rot": {"base": 1e4, "dims": hd}}
        left = dict(att, mask={"size": window},
                    rot={"base": 1e4, "dims": hd // 2, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}})
        right = {"heads": H, "dim": d, "vdim": 2 * d, "gate_cap": 15.0}
        ret = {"heads": H, "dim": d, "vdim": 2 * d, "rot": {"base": 1e4, "dims": d}, "decay": [1.0 - 2.0 ** -(5 + h % 8) for h in range(H)]}
        mixers = [("parallel", {"left": left, "right": right}), ("attention", att), ("retention", ret)]
        out = []
        for i in range(layers):
            t, m = mixers[i % 4] if i % 4 < 3 else ("attention", dict(att, kv_from=i - 2))
            out.append({"type": t, "mixer": m, "mlp": dense})
        return dict(architecture="Tumudra", vocab=vocab, width=W, embedding={"scale": 1.0}, norm={"eps": 1e-6}, layers=out)
    if design == "vonulorn":
        rot = d // 2
        delta = ("delta", {"heads": H, "kv_heads": H, "dim": d, "vdim": 2 * d, "conv": 4})
        att = ("attention", {"heads": heads, "kv_heads": kvh, "dim": hd // 2, "vdim": hd, "scale": (hd // 2) ** -0.5, "softcap": 50.0,
                             "diff": 0.35, "q_temp": {"coef": 0.1, "every": 1024}})
        lat = ("latent_attention", {"heads": H, "dim": d, "rot_dim": rot, "vdim": d, "q_rank": qr, "kv_rank": rank - rot,
                                    "scale": (d + rot) ** -0.5, "rot": {"base": 1e4, "dims": rot}})
        return dict(architecture="Vonulorn", vocab=vocab, width=W, norm={"eps": 1e-6}, residual_mult=0.5,
                    layers=[{"type": t, "mixer": m, "mlp": dense} for t, m in ((delta, delta, att, lat) * layers)[:layers]])
    raise ValueError(f"no such model: {model}")


def vocab_of(cfg: dict) -> int:
    return cfg["vocab_size"] if "vocab_size" in cfg else cfg["vocab"]


def tensor_shapes(cfg: dict):
    """[(checkpoint name, shape, what it is: "matrix", "scale" (around 1) or "small" (around 0))]."""
    out = []
    add = lambda n, s, k="matrix": out.append((n, s, k))  # noqa: E731
    if "hidden_size" in cfg:
        W, I, hd = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
        nq, nkv = cfg["num_attention_heads"], cfg["num_key_value_heads"]
        add("model.embed_tokens.weight", (cfg["vocab_size"], W))
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            for n, s in (("q", (nq * hd, W)), ("k", (nkv * hd, W)), ("v", (nkv * hd, W)), ("o", (W, nq * hd))):
                add(f"{p}self_attn.{n}_proj.weight", s)
            for n, s in (("gate", (I, W)), ("up", (I, W)), ("down", (W, I))):
                add(f"{p}mlp.{n}_proj.weight", s)
            for n in ("input", "post_attention", "pre_feedforward", "post_feedforward"):
                add(f"{p}{n}_layernorm.weight", (W,), "small")
        add("model.norm.weight", (W,), "small")
        return out
    W, design = cfg["width"], cfg["architecture"]
    add("embed", (cfg["vocab"], W))
    add("head", (cfg["vocab"], W))
    add("final.norm", (W,), "scale")
    if design == "Fuposun":
        add("embed.norm", (W,), "scale")
    for i, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.", layer["mixer"], layer["mlp"]
        add(p + "norm1", (W,), "scale")
        add(p + "norm2", (W,), "scale")
        p += "mix."
        if layer["type"] == "latent_attention":
            H, D, V, R, Q, K = m["heads"], m["dim"], m["vdim"], m.get("rot_dim", 0), m["q_rank"], m["kv_rank"]
            for n, s in (("dq", (Q, W)), ("uq", (H * (D + R), Q)), ("dkv", (K + R, W)), ("uk", (H * D, K)), ("uv", (H * V, K)), ("o", (W, H * V))):
                add(p + n, s)
            add(p + "dq.norm", (Q,), "scale")
            add(p + "dkv.norm", (K,), "scale")
            if design == "Fuposun":
                add(p + "g", (H, W))
            else:
                add(p + "sink", (H,), "small")
        elif layer["type"] == "attention" and design == "Vonulorn":
            H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            for n, s in (("q", (2 * H * D, W)), ("k", (2 * G * D, W)), ("v", (G * V, W)), ("o", (W, H * V))):
                add(p + n, s)
            for n in ("lq1", "lk1", "lq2", "lk2"):
                add(p + n, (D,), "small")
        elif layer["type"] in ("gla", "delta", "retention"):
            memory_shapes(add, p, layer["type"], m, W)
        elif layer["type"] == "attention":
            softmax_shapes(add, p, m, W, biases=True)
        elif layer["type"] == "parallel":
            softmax_shapes(add, p + "left.", m["left"], W, biases=False)
            memory_shapes(add, p + "right.", "mlstm", m["right"], W)
            add(p + "left.out", (W,), "scale")
            add(p + "right.out", (W,), "scale")
        p = f"l{i}.mlp."
        names = ("up", "down") if design == "Tumudra" else ("gate", "up", "down")
        if f["kind"] == "dense":
            for n in names:
                add(p + n, (W, f["ff"]) if n == "down" else (f["ff"], W))
        else:
            add(p + "router", (f["router"]["experts"], W))
            for e in [f"e{j}" for j in range(f["router"]["experts"])] + ["shared"]:
                for n in names:
                    add(f"{p}{e}.{n}", (W, f["expert"]["ff"]) if n == "down" else (f["expert"]["ff"], W))
    return out


def softmax_shapes(add, p, m, W, biases):
    H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    own = "kv_from" not in m
    for n, s in (("q", (H * D, W)), ("k", (G * D, W)), ("v", (G * V, W)), ("o", (W, H * V))):
        if own or n in "qo":
            add(p + n, s)
            if biases:
                add(f"{p}{n}.b", (s[0],), "small")
            if n in "qk":
                add(f"{p}{n}.norm", (D,), "scale")


def memory_shapes(add, p, kind, m, W):
    H, D, V = m["heads"], m["dim"], m["vdim"]
    G = m.get("kv_heads", H)
    for n, s in (("q", (G * D, W)), ("k", (G * D, W)), ("v", (H * V, W)), ("g", (H * V, W)), ("o", (W, H * V))):
        add(p + n, s)
        if kind == "delta" and n in "qkv":
            add(f"{p}{n}.conv", (s[0], m["conv"]), "scale")
    if kind == "gla":
        add(p + "norm", (V,), "scale")
        add(p + "a1", (m["decay_rank"], W))
        add(p + "a2", (H * D, m["decay_rank"]))
        add(p + "a2.b", (H * D,), "small")
    if kind == "delta":
        add(p + "norm", (V,), "scale")
        for n in "ab":
            add(p + n, (H, W))
        add(p + "A_log", (H,), "small")
        add(p + "dt_bias", (H,), "small")
    if kind == "mlstm":
        add(p + "norm", (H * V,), "scale")
        for n in "if":
            add(p + n, (H, W))
            add(f"{p}{n}.b", (H,), "small")


def make_weights(case: dict, seed: int) -> dict:
    cfg = config_of(case["model"])
    dtype = getattr(torch, case["dtype"])
    g = torch.Generator(device=DEVICE)
    g.manual_seed(1000003 * seed + 17)
    out = {}
    for name, shape, kind in tensor_shapes(cfg):
        t = torch.empty(shape, dtype=dtype, device=DEVICE)
        std = (0.05 if case["model"] == "gemma2-tiny" else 0.02) if kind == "matrix" else 0.1
        out[name] = t.normal_(1.0 if kind == "scale" else 0.0, std, generator=g)
    if cfg.get("architecture") == "Fuposun":
        give_directions(cfg, out, g)
    return out


def give_directions(cfg, w, g):
    """Half of an embedding's energy lies along one of sixteen directions; a router scores each direction with a ladder of
    its own, so that the best two experts of a token stand clear of the others."""
    E, W = EXPERT_DIRECTIONS, cfg["width"]
    dirs = torch.linalg.qr(torch.randn((W, E), generator=g, device=DEVICE))[0].T                    # [E, W], orthonormal
    kind = torch.arange(cfg["vocab"], device=DEVICE) % E
    w["embed"] = (0.5 ** 0.5 * (w["embed"].float() + 0.02 * W ** 0.5 * dirs[kind])).to(w["embed"].dtype)
    ladder = torch.linspace(2.0, -2.0, E, device=DEVICE)
    ladder[:2] += torch.tensor([0.8, 0.4], device=DEVICE)
    for i, layer in enumerate(cfg["layers"]):
        if layer["mlp"]["kind"] == "moe":
            shift = torch.randperm(E, generator=g, device=DEVICE)
            score = ladder[(torch.arange(E, device=DEVICE)[:, None] + shift[None, :]) % E]           # [expert, direction]
            w[f"l{i}.mlp.router"] = ((score @ dirs) / (0.7 * W ** 0.5)).to(w["embed"].dtype)


# ---- the cases ----------------------------------------------------------------------------------------------------------

def listed():
    B2 = dict(model="gemma2-2b", dtype="bfloat16")
    return [
        # the smallest: four short requests of the tiny float32 model, where launches and the host are all there is
        dict(name="generate_tiny_f32", kind="generate", model="gemma2-tiny", dtype="float32", batch=4, shortest=1, longest=29, new=12, greedy=True),
        # a small server's round: eight short questions, answers of 32 tokens with the default sampling
        dict(name="generate_2b_b8", kind="generate", batch=8, shortest=100, longest=400, new=32, greedy=False, **B2),
        # one user who reads along
        dict(name="decode_2b_b1", kind="decode", batch=1, shortest=900, longest=900, **B2),
        # the benchmark's batch near the end of the longest context
        dict(name="decode_2b_b8_long", kind="decode", batch=8, shortest=6900, longest=6900, **B2),
        # a full server, prompts of all lengths
        dict(name="decode_2b_b64", kind="decode", batch=64, shortest=512, longest=2048, **B2),
        # the benchmark's prompt
        dict(name="prompt_2b_2048", kind="prompt", batch=1, shortest=2048, longest=2048, **B2),
        # chat messages of odd lengths that arrive together
        dict(name="prompt_2b_chat", kind="prompt", batch=6, shortest=9, longest=333, **B2),
        # next turns of conversations
        dict(name="extend_2b", kind="extend", batch=3, shortest=1100, longest=2900, new=203, **B2),
        # latent attention, linear attention and routed experts
        dict(name="prompt_fuposun", kind="prompt", model="fuposun-2b", dtype="bfloat16", batch=1, shortest=2048, longest=2048),
        dict(name="decode_fuposun_b8", kind="decode", model="fuposun-2b", dtype="bfloat16", batch=8, shortest=1500, longest=3000),
        # matrix memories beside attention: documents of unequal length
        dict(name="prompt_tumudra", kind="prompt", model="tumudra-1b", dtype="bfloat16", batch=3, shortest=301, longest=1777),
        # the delta rule, differential and latent attention
        dict(name="decode_vonulorn_b8", kind="decode", model="vonulorn-2b", dtype="bfloat16", batch=8, shortest=2000, longest=2900),
    ]


def between(rng, lo, hi):
    """A whole number, its logarithm uniform."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["generate", "decode", "decode", "prompt", "prompt", "extend"])
    if kind == "generate" and rng.random() < 0.5:
        longest = between(rng, 2, 60)
        return dict(kind=kind, model="gemma2-tiny", dtype="float32", batch=rng.randint(1, 8), shortest=between(rng, 1, longest),
                    longest=longest, new=rng.randint(2, 24), greedy=rng.random() < 0.5)
    if kind == "generate":
        longest = between(rng, 20, 800)
        return dict(kind=kind, model="gemma2-2b", dtype="bfloat16", batch=between(rng, 1, 12), shortest=between(rng, 10, longest),
                    longest=longest, new=rng.randint(4, 32), greedy=rng.random() < 0.5)
    if kind == "extend":
        longest = between(rng, 200, 3300)
        return dict(kind=kind, model="gemma2-2b", dtype="bfloat16", batch=rng.randint(1, 4), shortest=between(rng, 100, longest),
                    longest=longest, new=between(rng, 2, 400))
    model = rng.choice(["gemma2-2b", "gemma2-2b", "fuposun-2b", "fuposun-1b", "tumudra-2b", "tumudra-1b", "vonulorn-2b", "vonulorn-1b"])
    if kind == "decode":
        batch = between(rng, 1, 64 if model == "gemma2-2b" else 24)
        longest = between(rng, 40, min(6900, 80000 // batch))
        return dict(kind=kind, model=model, dtype="bfloat16", batch=batch, shortest=between(rng, max(1, longest // 4), longest), longest=longest)
    batch = between(rng, 1, 6)
    longest = between(rng, 8, 2048 if batch == 1 else 4096 // batch)
    return dict(kind=kind, model=model, dtype="bfloat16", batch=batch, shortest=between(rng, max(1, longest // 8), longest), longest=longest)


def lengths_of(case: dict):
    """Prompt lengths: the shortest, the longest and, in equal ratios, what lies between, in an order that is not sorted."""
    n, lo, hi = case["batch"], case["shortest"], case["longest"]
    lens = [hi] if n == 1 else [int(round(lo * (hi / lo) ** (i / (n - 1)))) for i in range(n)]
    return lens[::2] + lens[1::2][::-1]


def make_tokens(case: dict, seed: int):
    """(prompts, what follows them: a list of [steps or new tokens] per sequence), host lists; ids from 2 up."""
    g = torch.Generator()
    g.manual_seed(7919 * seed + 3)
    vocab = vocab_of(config_of(case["model"]))
    ids = lambda n: torch.randint(2, vocab, (n,), generator=g).tolist()  # noqa: E731
    prompts = [ids(n) for n in lengths_of(case)]
    after = {"decode": GROWTH, "extend": case.get("new", 0)}.get(case["kind"], 0)
    return prompts, [ids(after) for _ in prompts]


def prepare(case: dict, seed: int):
    cfg = config_of(case["model"])
    arch = find_architecture(cfg)
    typed = arch.config_cls.from_dict(cfg)
    model = Model.from_tensors(arch, typed, make_weights(case, seed), case["dtype"], DEVICE)
    prompts, after = make_tokens(case, seed)
    more = {"generate": case.get("new", 0) + 2, "decode": GROWTH + 1, "extend": case.get("new", 0)}.get(case["kind"], 0)
    context = case["longest"] + more
    llm = LLM(model=model, dtype=case["dtype"], device=DEVICE, max_context=context, max_batch=case["batch"])
    st = dict(case=case, llm=llm, engine=llm.engine, prompts=prompts)
    if case["kind"] == "generate":
        new, seed_ = case["new"], 42
        st["options"] = GenerationOptions.greedy(new, seed=seed_) if case["greedy"] else GenerationOptions(max_new_tokens=new, seed=seed_)
        llm.warm_up(st["options"], batch_sizes=[case["batch"]])
    if case["kind"] == "decode":
        st["next"] = torch.tensor(after, dtype=torch.int32).T.contiguous().to(DEVICE)              # [step, sequence]
        begin_batch(st)
    if case["kind"] == "extend":
        st["slots"] = run_prompts(st)
        st["entries"] = list(zip(st["slots"], after))
        st["held"] = [(s, len(p)) for s, p in zip(st["slots"], prompts)]
    return st


def run_prompts(st):
    """Sequences that hold the prompts, a few thousand tokens per step."""
    eng, prompts = st["engine"], st["prompts"]
    slots = [eng.new_sequence() for _ in prompts]
    some, held = [], 0
    for slot, p in zip(slots, prompts):
        some.append((slot, p))
        held += len(p)
        if held >= 8192:
            eng.step(some, "last")
            some, held = [], 0
    if some:
        eng.step(some, "last")
    return slots


def begin_batch(st):
    """The batch's prompts, and its first decode step (the one that captures the graph)."""
    st["slots"] = run_prompts(st)
    st["engine"].decode(st["slots"], st["next"][0])
    st["at"] = 1


def run(st):
    kind, eng = st["case"]["kind"], st["engine"]
    if kind == "generate":
        return [np.array(r.tokens) for r in st["llm"].generate(st["prompts"], st["options"], stop_ids=[])]
    if kind == "decode":
        if st["at"] >= GROWTH:
            for s in st["slots"]:
                eng.release(s)
            begin_batch(st)
        st["at"] += 1
        return eng.decode(st["slots"], st["next"][st["at"] - 1])
    if kind == "extend":
        logits = eng.step(st["entries"], "last")
        eng.cache.truncate(st["held"])
        return logits
    slots = [eng.new_sequence() for _ in st["prompts"]]
    logits = eng.step(list(zip(slots, st["prompts"])), "last")
    for s in slots:
        eng.release(s)
    return logits


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------

def layers_of(cfg: dict):
    """Per layer: (window or None, bytes of keys and values per cached token at two bytes a value, flop per query row and
    key, elements of state per sequence)."""
    out = []
    if "hidden_size" in cfg:
        nq, nkv, hd = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
        return [(cfg["sliding_window"] if i % 2 == 0 else None, 4 * nkv * hd, 4 * nq * hd, 0) for i in range(cfg["num_hidden_layers"])]
    for layer in cfg["layers"]:
        t, m = layer["type"], layer["mixer"]
        att, mem = (m["left"], m["right"]) if t == "parallel" else (m, m)
        window, kv, per_key, state = (att.get("mask") or {}).get("size"), 0, 0, 0
        if t == "latent_attention":
            R = m.get("rot_dim", 0)
            kv, per_key = 2 * (m["kv_rank"] + R), 2 * m["heads"] * (2 * m["kv_rank"] + R)
        elif t in ("attention", "parallel"):
            maps = 2 if "diff" in att else 1
            kv = 2 * att["kv_heads"] * (maps * att["dim"] + att["vdim"])
            per_key = 2 * maps * att["heads"] * (att["dim"] + att["vdim"])
        if t not in ("latent_attention", "attention"):
            state = mem["heads"] * mem["dim"] * mem["vdim"]
        out.append((window, kv, per_key, state))
    return out


def parameters(cfg: dict):
    """(elements of the layers' tensors, of the routed experts among them, of the output head)."""
    layers = experts = 0
    for name, shape, _ in tensor_shapes(cfg):
        if "embed" in name or name == "head":
            continue
        n = math.prod(shape)
        layers += n
        experts += n if ".mlp.e" in name else 0
    return layers, experts, vocab_of(cfg) * (cfg["hidden_size"] if "hidden_size" in cfg else cfg["width"])


def step_work(cfg, size, starts, news, rows):
    """Bytes and flop of one step: sequences of ``starts`` cached tokens, each continued by ``news``; ``rows`` of logits."""
    layers, experts, head = parameters(cfg)
    T = sum(news)
    moe = next((l["mlp"] for l in cfg.get("layers", []) if l["mlp"]["kind"] == "moe"), None)
    share = moe["router"]["top"] / moe["router"]["experts"] if moe else 0.0
    nbytes = size * (layers - experts + experts * (1 - (1 - share) ** T) + head) + 4 * rows * vocab_of(cfg)
    flops = 2 * T * (layers - experts + experts * share) + 2 * rows * head
    for window, kv, per_key, state in layers_of(cfg):
        for s, n in zip(starts, news):
            cap = window or 1 << 30
            nbytes += kv * size / 2 * (min(s, cap) + n) + (8 * state if s else 4 * state)
            full = max(0, s + n - max(s, cap))                       # rows that see a whole window; the others see all before
            part = n - full
            flops += per_key * (full * min(cap, s + n) + part * s + part * (part + 1) // 2) + 6 * state * n
    return nbytes, flops


def work(case: dict):
    cfg = config_of(case["model"])
    size = 4 if case["dtype"] == "float32" else 2
    lens, B = lengths_of(case), case["batch"]
    zero = [0] * B
    if case["kind"] == "prompt":
        b, f = step_work(cfg, size, zero, lens, B)
    elif case["kind"] == "extend":
        b, f = step_work(cfg, size, lens, [case["new"]] * B, B)
    elif case["kind"] == "decode":
        b, f = step_work(cfg, size, [n + 1 for n in lens], [1] * B, B)
    else:
        b, f = step_work(cfg, size, zero, lens, B)
        for k in range(case["new"] - 1):
            more = step_work(cfg, size, [n + k for n in lens], [1] * B, B)
            b, f = b + more[0], f + more[1]
    return {"bytes": b, "flops": f}


def tolerance(case: dict):
    if case["kind"] == "generate":
        return "exact"
    # bfloat16 rows between float32 sums: measured 0.005 (Fuposun), 0.010 (Gemma 2, Tumudra) and 0.017 (Vonulorn, whose differential
    # attention subtracts two maps) against 64 bits; another order of the sums may be as far off in another direction
    return {"rel": 0.03 if case["model"].startswith("vonulorn") else 0.02, "max": 0.2}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------------

def exact(case: dict, seed: int):
    if case["kind"] == "generate":
        return None                                       # whole numbers
    cfg = config_of(case["model"])
    prompts, after = make_tokens(case, seed)
    n = {"decode": 2, "extend": case.get("new", 0)}.get(case["kind"], 0)
    seqs = [p + a[:n] for p, a in zip(prompts, after)]
    if step_work(cfg, 8, [0] * len(seqs), [len(s) for s in seqs], len(seqs))[1] > 4.5e14:
        return None                                       # over about 20 seconds
    with torch.no_grad():
        w = make_weights(case, seed)
        return (exact_gemma2 if "hidden_size" in cfg else exact_design)(cfg, w, seqs)


F64 = torch.float64


def rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def turn(x, freq, interleaved=False):
    """x: [n, heads, d]; the first 2 len(freq) columns turn by position times frequency (angles formed in 32 bits)."""
    half = freq.numel()
    a = (torch.arange(x.shape[0], device=x.device, dtype=torch.float32)[:, None] * freq.float()[None, :].to(x.device)).to(F64)
    c, s = a.cos()[:, None, :], a.sin()[:, None, :]
    out = x.clone()
    one, two = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if interleaved else (slice(0, half), slice(half, 2 * half))
    u, v = x[..., one], x[..., two]
    out[..., one], out[..., two] = u * c - v * s, v * c + u * s
    return out


def frequencies(rot):
    f = float(rot["base"]) ** (-2.0 * torch.arange(rot["dims"] // 2, dtype=F64) / rot["dims"])
    sc = rot.get("scaling")
    if sc:                                                # long wavelengths are slowed down, those between blended
        wave = 2.0 * math.pi / f
        s = ((sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])).clamp(0.0, 1.0)
        f = (1.0 - s) * f / sc["factor"] + s * f
    return f


def softmax_heads(q, k, v, scale, window=None, cap=None, sink=None):
    """q: [n, H, d], k: [n, G, d], v: [n, G, dv] -> [n, H, dv]; head h reads key head h // (H / G)."""
    n, H = q.shape[:2]
    g = H // k.shape[1]
    out = torch.empty((n, H, v.shape[2]), dtype=F64, device=q.device)
    for r0 in range(0, n, 2048):
        r1 = min(n, r0 + 2048)
        dist = torch.arange(r0, r1, device=q.device)[:, None] - torch.arange(r1, device=q.device)[None, :]
        hide = (dist < 0) if not window else ((dist < 0) | (dist >= window))
        for h in range(H):
            s = (q[r0:r1, h] @ k[:r1, h // g].T) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill_(hide, float("-inf"))
            top = s.amax(-1, keepdim=True)
            if sink is not None:
                top = top.clamp(min=float(sink[h]))
            s = torch.exp_(s.sub_(top))
            den = s.sum(-1, keepdim=True)
            if sink is not None:
                den = den + torch.exp(sink[h] - top)
            out[r0:r1, h] = (s @ v[:r1, h // g]) / den
    return out


def exact_gemma2(cfg, w, seqs):
    eps, hd, nq, nkv = cfg["rms_norm_eps"], cfg["head_dim"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
    flat = torch.tensor([t for s in seqs for t in s], device=DEVICE)
    x = w["model.embed_tokens.weight"][flat].to(F64) * float(torch.tensor(cfg["hidden_size"] ** 0.5, dtype=torch.float32))
    freq = frequencies({"base": cfg["rope_theta"], "dims": hd})
    lens = [len(s) for s in seqs]
    norm = lambda y, n: rms(y, eps) * (1.0 + w[n].to(F64))  # noqa: E731
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        mat = lambda n: w[p + n + "_proj.weight"].to(F64).T  # noqa: E731
        h = norm(x, p + "input_layernorm.weight")
        qkv = [(h @ mat("self_attn." + n)).view(-1, heads, hd) for n, heads in (("q", nq), ("k", nkv), ("v", nkv))]
        outs = []
        for q, k, v in zip(*(t.split(lens) for t in qkv)):
            outs.append(softmax_heads(turn(q, freq), turn(k, freq), v, cfg["query_pre_attn_scalar"] ** -0.5,
                                      cfg["sliding_window"] if i % 2 == 0 else None, cfg["attn_logit_softcapping"]))
        x = x + norm(torch.cat(outs).flatten(1) @ mat("self_attn.o"), p + "post_attention_layernorm.weight")
        h = norm(x, p + "pre_feedforward_layernorm.weight")
        y = torch.nn.functional.gelu(h @ mat("mlp.gate"), approximate="tanh") * (h @ mat("mlp.up"))
        x = x + norm(y @ mat("mlp.down"), p + "post_feedforward_layernorm.weight")
    last = torch.tensor(lens, device=DEVICE).cumsum(0) - 1
    z = norm(x[last], "model.norm.weight") @ w["model.embed_tokens.weight"].to(F64).T
    return cfg["final_logit_softcapping"] * torch.tanh(z / cfg["final_logit_softcapping"])


def silu(z):
    return z * torch.sigmoid(z)


def exact_design(cfg, w, seqs):
    """Fuposun, Tumudra or Vonulorn.  Sequences are padded at their ends: no row sees a later one."""
    design, eps, n = cfg["architecture"], cfg["norm"]["eps"], max(len(s) for s in seqs)
    ids = torch.tensor([s + [0] * (n - len(s)) for s in seqs], device=DEVICE)
    x = w["embed"][ids].to(F64)                                                          # [B, n, W]
    if design == "Fuposun":
        x = rms(x, eps) * w["embed.norm"].to(F64)
    kept = {}
    for i, layer in enumerate(cfg["layers"]):
        get = lambda name, i=i: w[f"l{i}.{name}"].to(F64)  # noqa: E731
        if design == "Tumudra":
            ln = lambda y, name: torch.nn.functional.layer_norm(y, y.shape[-1:], get(name), eps=eps)  # noqa: E731
            x = x + ln(tumudra_mixer(x, get, layer, eps, i, kept), "norm1")
            x = x + ln(torch.relu(x @ get("mlp.up").T) ** 2 @ get("mlp.down").T, "norm2")
            continue
        h = rms(x, eps) * get("norm1")
        x = x + cfg["residual_mult"] * MIXERS[design, layer["type"]](h, get, layer["mixer"], eps)
        h = rms(x, eps) * get("norm2")
        if layer["mlp"]["kind"] == "moe":
            y = routed(h, get, layer["mlp"])
        else:
            a = silu(h @ get("mlp.gate").T) if design == "Fuposun" else torch.nn.functional.gelu(h @ get("mlp.gate").T, approximate="tanh")
            y = (a * (h @ get("mlp.up").T)) @ get("mlp.down").T
        x = x + cfg["residual_mult"] * y
    last = x[torch.arange(len(seqs), device=DEVICE), torch.tensor([len(s) - 1 for s in seqs], device=DEVICE)]
    if design == "Tumudra":
        return torch.nn.functional.layer_norm(last, last.shape[-1:], w["final.norm"].to(F64), eps=eps) @ w["head"].to(F64).T
    z = (rms(last, eps) * w["final.norm"].to(F64)) @ w["head"].to(F64).T
    cap = cfg.get("logit_softcap")
    return cap * torch.tanh(z / cap) if cap else z


def heads(x, n):
    return x.view(*x.shape[:-1], n, -1)


def each(f, *batched):
    """f of every sequence, stacked."""
    return torch.stack([f(*row) for row in zip(*batched)])


def latent(h, get, m, eps):
    H, K = m["heads"], m["kv_rank"]
    q = heads((rms(h @ get("mix.dq").T, eps) * get("mix.dq.norm")) @ get("mix.uq").T, H)
    kv = h @ get("mix.dkv").T
    c = rms(kv[..., :K], eps) * get("mix.dkv.norm")
    k, v = heads(c @ get("mix.uk").T, H), heads(c @ get("mix.uv").T, H)
    if "rot" in m:
        freq, D = frequencies(m["rot"]), m["dim"]
        kr = each(lambda t: turn(t[:, None], freq, True), kv[..., K:])
        q = torch.cat([q[..., :D], each(lambda t: turn(t, freq, True), q[..., D:])], -1)
        k = torch.cat([k, kr.expand(-1, -1, H, -1)], -1)
    sink = get("mix.sink") if "rot" in m else None
    o = each(lambda a, b, d: softmax_heads(a, b, d, m["scale"], (m.get("mask") or {}).get("size"), sink=sink), q, k, v)
    if "rot" not in m:
        o = o * torch.sigmoid(h @ get("mix.g").T)[..., None]
    return o.flatten(2) @ get("mix.o").T


def gated_linear(h, get, m, eps):
    H, D = m["heads"], m["dim"]
    q, k, v = (heads(h @ get("mix." + n).T, H) for n in "qkv")
    a = torch.sigmoid((h @ get("mix.a1").T) @ get("mix.a2").T + get("mix.a2.b")) ** (1.0 / m["tau"])
    a = heads(a, H)
    S = torch.zeros((*q.shape[:1], H, D, v.shape[-1]), dtype=F64, device=h.device)
    out = torch.empty_like(v)
    for t in range(h.shape[1]):
        S = a[:, t, :, :, None] * S + k[:, t, :, :, None] * v[:, t, :, None, :]
        out[:, t] = (q[:, t, :, None, :] @ S)[..., 0, :] * D ** -0.5
    out = (rms(out, eps) * get("mix.norm")).flatten(2)
    return (out * silu(h @ get("mix.g").T)) @ get("mix.o").T


def routed(h, get, f):
    lim = f["expert"]["limit"]

    def expert(rows, e):
        g = (rows @ get(f"mlp.{e}.gate").T).clamp(max=lim)
        u = (rows @ get(f"mlp.{e}.up").T).clamp(-lim, lim)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ get(f"mlp.{e}.down").T

    rows = h.flatten(0, 1)
    s = torch.sigmoid(rows @ get("mlp.router").T)
    best = s.topk(f["router"]["top"], dim=-1).indices
    out = expert(rows, "shared")
    for e in range(f["router"]["experts"]):
        who = (best == e).any(-1).nonzero()[:, 0]
        if who.numel():
            out[who] += expert(s[who, e:e + 1] * rows[who], f"e{e}")
    return out.view_as(h)


def delta(h, get, m, eps):
    H, G, D, taps = m["heads"], m["kv_heads"], m["dim"], m["conv"]

    def conv(x, c):
        x = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
        return silu(sum(x[:, j:j + h.shape[1]] * c[:, j] for j in range(taps)))

    q, k, v = (conv(h @ get("mix." + n).T, get(f"mix.{n}.conv")) for n in "qkv")
    unit = lambda z: z * torch.rsqrt((z * z).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q, k = (unit(heads(z, G)).repeat_interleave(H // G, dim=2) for z in (q, k))
    q, v = q * D ** -0.5, heads(v, H)
    beta = torch.sigmoid(h @ get("mix.b").T)
    g = torch.exp(-torch.exp(get("mix.A_log")) * torch.nn.functional.softplus(h @ get("mix.a").T + get("mix.dt_bias"), threshold=100.0))
    S = torch.zeros((h.shape[0], H, D, v.shape[-1]), dtype=F64, device=h.device)
    out = torch.empty_like(v)
    for t in range(h.shape[1]):
        S = g[:, t, :, None, None] * S
        u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None, :] @ S)[..., 0, :])
        S = S + k[:, t, :, :, None] * u[:, :, None, :]
        out[:, t] = (q[:, t, :, None, :] @ S)[..., 0, :]
    out = (rms(out, eps) * get("mix.norm")).flatten(2)
    return (out * silu(h @ get("mix.g").T)) @ get("mix.o").T


def differential(h, get, m, eps):
    H, G, D = m["heads"], m["kv_heads"], m["dim"]
    p = torch.arange(h.shape[1], dtype=F64, device=h.device)
    temp = 1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((p + 1.0) / m["q_temp"]["every"]) + 1.0)
    q = heads(h @ get("mix.q").T, H) * temp[:, None, None]
    k, v = heads(h @ get("mix.k").T, G), heads(h @ get("mix.v").T, G)
    lam = torch.exp((get("mix.lq1") * get("mix.lk1")).sum()) - torch.exp((get("mix.lq2") * get("mix.lk2")).sum()) + m["diff"]
    one, two = (each(lambda a, b, c: softmax_heads(a, b, c, m["scale"], cap=m["softcap"]), q[..., s], k[..., s], v)
                for s in (slice(0, D), slice(D, 2 * D)))
    return (rms(one - lam * two, eps) * (1.0 - m["diff"])).flatten(2) @ get("mix.o").T


MIXERS = {("Fuposun", "latent_attention"): latent, ("Fuposun", "gla"): gated_linear, ("Vonulorn", "latent_attention"): latent,
          ("Vonulorn", "delta"): delta, ("Vonulorn", "attention"): differential}


def tumudra_mixer(x, get, layer, eps, i, kept):
    m = layer["mixer"]
    if layer["type"] == "attention":
        return tumudra_attention(x, get, "mix.", m, eps, False, i, kept)
    if layer["type"] == "retention":
        return retention(x, get, m, eps)
    a = tumudra_attention(x, get, "mix.left.", m["left"], eps, True, i, {})
    b = matrix_memory(x, get, m["right"], eps)
    return 0.5 * (rms(a, eps) * get("mix.left.out") + rms(b, eps) * get("mix.right.out"))


def tumudra_attention(x, get, p, m, eps, interleaved, i, kept):
    freq = frequencies(m["rot"])
    bias = (lambda n: 0.0) if interleaved else (lambda n: get(f"{p}{n}.b"))
    turned = lambda n, c: each(lambda t: turn(t, freq, interleaved), rms(heads(x @ get(p + n).T + bias(n), c), eps) * get(f"{p}{n}.norm"))  # noqa: E731
    q = turned("q", m["heads"])
    if "kv_from" in m:
        k, v = kept[m["kv_from"]]
    else:
        k, v = kept[i] = turned("k", m["kv_heads"]), heads(x @ get(p + "v").T + bias("v"), m["kv_heads"])
    o = each(lambda a, b, c: softmax_heads(a, b, c, m["scale"], (m.get("mask") or {}).get("size")), q, k, v)
    return o.flatten(2) @ get(p + "o").T + bias("o")


def matrix_memory(x, get, m, eps):
    H, D, cap = m["heads"], m["dim"], m["gate_cap"]
    q, k, v = (heads(x @ get("mix.right." + n).T, H) for n in "qkv")
    q = q * D ** -0.5
    gi, gf = (cap * torch.tanh((x @ get(f"mix.right.{n}").T + get(f"mix.right.{n}.b")) / cap) for n in "if")
    gf = torch.nn.functional.logsigmoid(gf)
    S = torch.zeros((x.shape[0], H, D, v.shape[-1]), dtype=F64, device=x.device)
    nv, mx = torch.zeros_like(S[..., 0]), torch.zeros_like(gi[:, 0])
    out = torch.empty_like(v)
    for t in range(x.shape[1]):
        new = torch.maximum(gf[:, t] + mx, gi[:, t])
        keep, take = torch.exp(gf[:, t] + mx - new)[..., None], torch.exp(gi[:, t] - new)[..., None]
        S = keep[..., None] * S + (take * k[:, t])[..., None] * v[:, t, :, None, :]
        nv, mx = keep * nv + take * k[:, t], new
        den = torch.maximum((nv * q[:, t]).sum(-1).abs(), torch.exp(-mx)) + 1e-6
        out[:, t] = (q[:, t, :, None, :] @ S)[..., 0, :] / den[..., None]
    out = rms(out, eps).flatten(2) * get("mix.right.norm")
    return (out * torch.sigmoid(x @ get("mix.right.g").T)) @ get("mix.right.o").T


def retention(x, get, m, eps):
    H, D = m["heads"], m["dim"]
    freq = frequencies(m["rot"])
    q, k = (each(lambda t: turn(t, freq), heads(x @ get("mix." + n).T, H)) for n in "qk")
    v = heads(x @ get("mix.v").T, H)
    k = k * D ** -0.5
    decay = torch.tensor(m["decay"], dtype=F64, device=x.device)[:, None, None]
    S = torch.zeros((x.shape[0], H, D, v.shape[-1]), dtype=F64, device=x.device)
    out = torch.empty_like(v)
    for t in range(x.shape[1]):
        S = decay * S + k[:, t, :, :, None] * v[:, t, :, None, :]
        out[:, t] = (q[:, t, :, None, :] @ S)[..., 0, :]
    return (rms(out, eps).flatten(2) * silu(x @ get("mix.g").T)) @ get("mix.o").T
