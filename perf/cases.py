"""What this framework is used for, as cases that can be timed and compared: the vision tower and projector over the crops of a request, the
decoder over packed prompts, whole Leopard-LLaVA prefills, cached single-token decoding, the SFT step, and prompts and decode steps of the
layer-list language models in both precisions.  Sizes are those of `leopard_b200.config`, of the crop planner (1 to 50 crops of 676 patches,
169 rows each) and of the benchmark's three model widths; weights and inputs are random, of the distributions of a fresh initialisation.

A case is a dict of plain values; `prepare` builds what a program holds before the call, `run` makes one pass through the public entry
points, `exact` says in 64 bits what that pass returns."""
import math
import zlib

import numpy as np
import torch
import torch.nn.functional as F

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
CROP_ROWS = 169            # decoder rows of one 364 x 364 crop
IMAGE_ID = 128200          # the placeholder id of the LLaVA prompt
SFT_VOCAB = 32000


# ------------------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the vision half of a 4-image request: 28 crops through tower layers and the projector
        {"name": "tower-28", "kind": "tower", "crops": 28, "layers": 4},
        # two prompts packed into one decoder pass, the second of an odd length; last-row logits and the cache that decoding continues from
        {"name": "decoder-4796", "kind": "decoder", "model": "llama", "first": 3559, "second": 1237, "layers": 2},
        # the smallest request: one small image and a short question, at full depth (latency)
        {"name": "request-1", "kind": "request", "crops": 1, "text": 32},
        # the headline request: four 896 x 1152 images, 28 crops, 4796 decoder rows, at full depth
        {"name": "request-28", "kind": "request", "crops": 28, "text": 92},
        # decoding after that prompt: single-token steps over the cache
        {"name": "decode-4796", "kind": "decode", "context": 4796, "tokens": 16, "layers": 8},
        # one SFT iteration of a short instruction with images
        {"name": "sft-2048", "kind": "sft", "length": 2048, "crops": 7},
        # a long prompt through retention + experts and latent attention + dense
        lm("zudalorn", "retention:moe,latent:dense", 2048, batch=1, prompt=4096, steps=0, score=64, name="zudalorn-prompt"),
        # a long prompt through the two windowed attentions and the gated recurrence
        lm("ronelorn", "attention:dense,attention_2:dense,mingru:none", 2048, batch=1, prompt=4096, steps=0, score=64, name="ronelorn-prompt"),
        # eight running requests with short prompts
        lm("zudalorn", "retention:moe,latent:dense", 2048, batch=8, prompt=120, steps=32, score=1, name="zudalorn-serve-8"),
        # one user talking to the widest model
        lm("ronelorn", "attention:dense,attention_2:dense,mingru:none", 4096, batch=1, prompt=500, steps=32, score=1, name="ronelorn-serve-1"),
        # a full batch on the small model
        lm("zudalorn", "retention:moe,latent:dense", 1024, batch=64, prompt=24, steps=24, score=1, name="zudalorn-serve-64"),
        # scoring and decoding in the 32-bit precision
        lm("zudalorn", "retention:dense,latent:moe", 1024, batch=3, prompt=777, steps=8, score=32, dtype="float32", name="zudalorn-float32"),
    ]


def lm(model, layers, width, batch, prompt, steps, score, dtype="bfloat16", name=None):
    """A layer-list model at the benchmark's proportions: heads of 128, feed-forward four widths, window half a width."""
    big = width >= 2048
    c = {"kind": "lm", "model": model, "layers": layers, "width": width, "heads": width // 128, "ff": 4 * width, "kv_rank": min(512, width // 4),
         "window": width // 2, "experts": 32 if width >= 4096 else 16 if big else 8, "top": 4 if big else 2,
         "expert_ff": 2048 if width >= 4096 else 1024, "vocab": 32000, "dtype": dtype, "batch": batch, "prompt": prompt, "steps": steps,
         "score": score}
    return dict(c, name=name) if name else c


def spread(rng, lo, hi):
    """a whole number of [lo, hi], even over its logarithm"""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["tower", "decoder", "request", "decode", "sft", "lm", "lm", "lm", "lm", "lm"])
    if kind == "tower":
        return {"kind": kind, "crops": spread(rng, 1, 50), "layers": rng.randint(2, 5)}
    if kind == "decoder":
        first = spread(rng, 33, 8192)
        return {"kind": kind, "model": rng.choice(["llama", "mistral"]), "first": first, "second": rng.choice([0, spread(rng, 17, 2048)]),
                "layers": rng.randint(1, 3)}
    if kind == "request":
        return {"kind": kind, "crops": rng.randint(1, 24), "text": spread(rng, 24, 300)}
    if kind == "decode":
        return {"kind": kind, "context": spread(rng, 150, 12000), "tokens": rng.randint(8, 24), "layers": rng.randint(4, 10)}
    if kind == "sft":
        length = 8 * spread(rng, 48, 512)
        return {"kind": kind, "length": length, "crops": rng.randint(1, max(1, min(21, length // CROP_ROWS - 1)))}
    model = rng.choice(["zudalorn", "ronelorn"])
    layers = rng.choice(["retention:moe,latent:dense", "retention:dense,latent:moe", "latent:moe,retention:dense"] if model == "zudalorn" else
                        ["attention:dense,attention_2:dense,mingru:none", "attention_2:dense,mingru:none", "mingru:none,attention:dense"])
    dtype = rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32"])
    if rng.random() < 0.4:       # prompts
        width = rng.choice([512, 768, 1024, 1536, 2048])
        batch = rng.choice([1, 1, 2, 5])
        return lm(model, layers, width, batch, spread(rng, 64, 4096) if dtype == "bfloat16" else spread(rng, 64, 1500), 0, rng.choice([1, 16, 64]), dtype)
    width = rng.choice([512, 1024, 1536, 2048, 3072, 4096])
    batch = spread(rng, 1, 64 if width <= 2048 and dtype == "bfloat16" else 12)
    return lm(model, layers, width, batch, spread(rng, 5, max(16, 800 // batch)), rng.randint(8, 32), 1, dtype)


# ------------------------------------------------------------------------------------------------------------------------ random data
def generator(seed, name):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFF)


def normal(seed, name, shape, scale=1.0, dtype=BF16):
    return (torch.randn(shape, device="cuda", generator=generator(seed, name)) * scale).to(dtype)


def uniform(seed, name, shape, lo, hi, dtype=BF16):
    return (torch.rand(shape, device="cuda", generator=generator(seed, name)) * (hi - lo) + lo).to(dtype)


def token_ids(seed, name, n, vocab):
    return np.random.RandomState((int(seed) * 7919 + zlib.crc32(name.encode())) & 0x7FFFFFFF).randint(0, vocab, n)


# ------------------------------------------------------------------------------------------------------------------------ Leopard-LLaVA
VT, PJ, LM = "vision_tower.vision_model.", "multi_modal_projector.", "language_model.model."
VIT = dict(hidden=1152, ffn=4304, heads=16, patches=676, eps=1e-6)
DEC = dict(hidden=4096, ffn=14336, heads=32, kv_heads=8, dim=128, eps=1e-5)


def leopard_config(case):
    from leopard_b200.config import leopard_idefics2_decoder, leopard_llava, reduced
    from dataclasses import replace
    kind = case["kind"]
    cfg = leopard_llava()
    if kind == "tower":
        return reduced(cfg, case["layers"], 1, 1024)
    if kind == "decoder":
        if case["model"] == "mistral":
            cfg = replace(cfg, dec=leopard_idefics2_decoder())
        return reduced(cfg, 1, case["layers"])
    if kind == "decode":
        return reduced(cfg, 1, case["layers"])
    if kind == "sft":
        return reduced(cfg, 1, 1, SFT_VOCAB)
    return cfg


def leopard_shape(name, vocab):
    """(shape, fan-in or None for vectors around 0 / 1) of a checkpoint tensor"""
    D, FF, d, ff = VIT["hidden"], VIT["ffn"], DEC["hidden"], DEC["ffn"]
    kv = DEC["kv_heads"] * DEC["dim"]
    last = name.split(".")[-2] + "." + name.split(".")[-1]
    if name.startswith(VT):
        table = {"patch_embedding.weight": (D, 3, 14, 14), "patch_embedding.bias": (D,), "position_embedding.weight": (VIT["patches"], D),
                 "fc1.weight": (FF, D), "fc1.bias": (FF,), "fc2.weight": (D, FF), "fc2.bias": (D,)}
        if last in table:
            return table[last]
        return (D, D) if "_proj" in name and last.endswith("weight") else (D,)
    if name.startswith(PJ):
        return {"linear_1.weight": (d, 4 * D), "linear_1.bias": (d,), "linear_2.weight": (d, d), "linear_2.bias": (d,)}[last]
    return {"embed_tokens.weight": (vocab, d), "lm_head.weight": (vocab, d), "norm.weight": (d,), "input_layernorm.weight": (d,),
            "post_attention_layernorm.weight": (d,), "q_proj.weight": (d, d), "k_proj.weight": (kv, d), "v_proj.weight": (kv, d),
            "o_proj.weight": (d, d), "gate_proj.weight": (ff, d), "up_proj.weight": (ff, d), "down_proj.weight": (d, ff)}[last]


def leopard_getter(seed, vocab):
    def get(name):
        shape = leopard_shape(name, vocab)
        if len(shape) == 1:
            if name.endswith("bias"):
                return normal(seed, name, shape, 0.02)
            return (1.0 + normal(seed, name, shape, 0.02, F32)).to(BF16)
        if "position_embedding" in name:
            return normal(seed, name, shape, 0.02)
        if "embed_tokens" in name:
            return normal(seed, name, shape, 0.05)
        return normal(seed, name, shape, math.prod(shape[1:]) ** -0.5)
    return get


def pixels(seed, crops):
    return uniform(seed, "pixels", (crops, 3, 364, 364), -1.0, 1.0, F32)


def request_ids(case, seed):
    """text with one placeholder per crop in its middle"""
    text = token_ids(seed, "text", case["text"], 128000)
    half = case["text"] // 2
    return torch.from_numpy(np.concatenate([text[:half], np.full(case["crops"], IMAGE_ID), text[half:]])).long()


def sft_batch(case, seed):
    s, n = case["length"], case["crops"] * CROP_ROWS
    ids = torch.from_numpy(token_ids(seed, "sft", s, SFT_VOCAB)).long()
    labels = torch.from_numpy(token_ids(seed, "labels", s, SFT_VOCAB)).long()
    at = min(16, s - n)
    ids[at:at + n] = -200
    mask = torch.ones(s)
    mask[: at + n] = 0
    if float(mask[1:].sum()) == 0:
        mask[-1] = 1
    return ids[None], labels[None], mask[None]


# ------------------------------------------------------------------------------------------------------------------------ layer-list models
def parts(case):
    return [tuple(p.split(":")) for p in case["layers"].split(",")]


def lm_config(case):
    H, D = case["heads"], case["width"]
    rows = []
    for mixer, ff in parts(case):
        if mixer == "retention":
            m = {"heads": H, "dim": 128, "vdim": 128, "decay": [1 - 2.0 ** (-4 - 4 * i / max(H - 1, 1)) for i in range(H)], "rot": {"base": 1e6, "dims": 128}}
        elif mixer == "latent":
            m = {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": case["kv_rank"], "scale": 192 ** -0.5, "mask": {"size": case["window"]},
                 "rot": {"base": 5e4, "dims": 64, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
        elif mixer == "mingru":
            m = {"width": D}
        else:
            m = {"heads": H, "kv_heads": max(H // 4, 1), "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "rot": {"base": 1e6, "dims": 64}}
            if mixer == "attention":
                m.update(softcap=30.0, mask={"size": case["window"], "pool": 64})
                m["rot"]["scaling"] = {"factor": 4.0}
            else:
                m.update(mask={"size": case["window"], "keep_first": 4})
        mlp = None
        if ff == "dense":
            mlp = {"kind": "dense", "ff": case["ff"]}
        elif ff == "moe":
            mlp = {"kind": "moe", "expert": {"ff": case["expert_ff"]}, "shared": {"ff": D},
                   "router": {"experts": case["experts"], "top": case["top"], "groups": {"count": 4, "keep": 2}}}
        rows.append({"type": {"latent": "latent_attention"}.get(mixer, mixer), "mixer": m, "mlp": mlp})
    c = {"architecture": case["model"].capitalize(), "vocab": case["vocab"], "width": D, "norm": {"eps": 1e-6}, "layers": rows}
    if case["model"] == "ronelorn":
        c.update(residual_mult=0.5, embedding={"scale": 1.0})
    return c


def lm_shapes(c):
    D, out = c["width"], {}
    out["embed"] = out["head"] = (c["vocab"], D)
    sandwich = c["architecture"] == "Zudalorn"
    out["final.norm"] = () if sandwich else (D,)
    for i, layer in enumerate(c["layers"]):
        p, m, kind = f"l{i}.", layer["mixer"], layer["type"]
        for n in ("norm1", "norm1b", "norm2", "norm2b") if sandwich else ("norm1", "norm2"):
            out[p + n] = () if sandwich else (D,)
        if kind == "mingru":
            out.update({p + "mix." + n: (m["width"], D) for n in "zxg"})
            out[p + "mix.z.b"] = out[p + "mix.x.b"] = (m["width"],)
            out[p + "mix.o"] = (D, m["width"])
        else:
            H = m["heads"]
            G = m.get("kv_heads", H)
            if kind == "latent_attention":
                out[p + "mix.q"], out[p + "mix.dkv"] = (H * (m["dim"] + m["rot_dim"]), D), (m["kv_rank"] + m["rot_dim"], D)
                out[p + "mix.dkv.norm"] = (m["kv_rank"],)
                out[p + "mix.uk"], out[p + "mix.uv"] = (H * m["dim"], m["kv_rank"]), (H * m["vdim"], m["kv_rank"])
            else:
                out[p + "mix.q"], out[p + "mix.k"], out[p + "mix.v"] = (H * m["dim"], D), (G * m["dim"], D), (G * m["vdim"], D)
                if kind == "retention":
                    out[p + "mix.g"] = (H * m["vdim"], D)
                else:
                    full = kind == "attention_2"
                    out[p + "mix.q.norm"], out[p + "mix.k.norm"] = ((H * m["dim"],), (G * m["dim"],)) if full else ((m["dim"],), (m["dim"],))
            out[p + "mix.o"] = (D, H * m["vdim"])
        f = layer["mlp"]
        if f is None:
            continue
        if f["kind"] == "dense":
            out[p + "mlp.up"], out[p + "mlp.down"] = (f["ff"], D), (D, f["ff"])
            if sandwich:
                out[p + "mlp.act"] = (2,)
            continue
        E = f["router"]["experts"]
        for e in [f"e{k}" for k in range(E)] + ["shared"]:
            n = f["shared"]["ff"] if e == "shared" else f["expert"]["ff"]
            out[f"{p}mlp.{e}.gate"] = out[f"{p}mlp.{e}.up"] = (n, D)
            out[f"{p}mlp.{e}.down"] = (D, n)
        out[p + "mlp.router"], out[p + "mlp.correction"], out[p + "mlp.shared.sg"] = (E, D), (E,), (1, D)
    return out


def lm_getter(c, seed):
    shapes = lm_shapes(c)

    def get(name):
        shape = shapes[name]
        if name == "embed":
            return normal(seed, name, shape, 4.0)      # the stream outweighs one sublayer's output, as it does inside a deep stack
        if name.endswith("router"):
            return normal(seed, name, shape, 4.0 * shape[1] ** -0.5)      # spread scores: few close calls
        if len(shape) == 2:
            return normal(seed, name, shape, shape[1] ** -0.5)
        if len(shape) == 0:
            return uniform(seed, name, shape, 0.6, 1.4)
        if name.endswith("correction"):
            return uniform(seed, name, shape, -0.3, 0.3)
        if name.endswith("mlp.act"):
            return uniform(seed, name, shape, -1.0, 1.0)
        if name.endswith((".q.norm", ".k.norm", ".dkv.norm")):
            return uniform(seed, name, shape, 0.75, 1.25)
        return uniform(seed, name, shape, -0.1, 0.1)
    return get


def lm_lengths(case):
    """prompt lengths of a batch: the first is `prompt`, the others shorter"""
    n = case["prompt"]
    return [max(1, n - (37 * i) % (n // 2 + 1)) for i in range(case["batch"])]


def lm_tokens(case, seed):
    """per request: its prompt and the tokens that follow"""
    got = []
    for i, n in enumerate(lm_lengths(case)):
        t = token_ids(seed, f"request {i}", n + case["steps"], case["vocab"]).tolist()
        got.append((t[:n], t[n:]))
    return got


# ------------------------------------------------------------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    if case["kind"] == "lm":
        from leopard_b200 import ronelorn, zudalorn
        from leopard_b200.seqlm import SeqLMEngine, SeqLMWeights
        c = lm_config(case)
        module = {"zudalorn": zudalorn, "ronelorn": ronelorn}[case["model"]]
        cfg = module.config_from_dict(c)
        weights = SeqLMWeights(cfg, lm_getter(c, seed), module.tensor_name, "cuda")
        room = sum(lm_lengths(case)) + case["batch"] * (case["steps"] + 64)
        return {"case": case, "requests": lm_tokens(case, seed),
                "engine": SeqLMEngine(cfg, weights, dtype=case["dtype"], max_tokens=room, max_seqs=case["batch"])}
    from leopard_b200.engine import PrefillEngine
    from leopard_b200.native_weights import load_hf
    cfg = leopard_config(case)
    weights = load_hf(cfg, leopard_getter(seed, cfg.dec.vocab), "cuda")
    state = {"case": case, "engine": PrefillEngine(cfg, weights)}
    kind = case["kind"]
    if kind == "tower":
        state["pixels"] = pixels(seed, case["crops"])
    elif kind == "request":
        state["samples"] = [(request_ids(case, seed), pixels(seed, case["crops"]))]
    elif kind == "decoder":
        state["samples"] = [(torch.from_numpy(token_ids(seed, k, case[k], min(cfg.dec.vocab, 31000))).long(), None) for k in ("first", "second") if case[k]]
    elif kind == "decode":
        from leopard_b200.hf import NativeKVCache, myLlavaForConditionalGeneration
        S, d = case["context"], cfg.dec
        kv = torch.zeros((d.layers, 2, S + case["tokens"], d.kv_heads * d.head_dim), dtype=BF16, device="cuda")
        kv[:, :, :S] = normal(seed, "cache", (d.layers, 2, S, d.kv_heads * d.head_dim))
        state["model"] = myLlavaForConditionalGeneration.from_native(cfg, weights)
        state["kv"], state["past"] = kv, NativeKVCache(kv, S, d.kv_heads, d.head_dim)
        state["tokens"] = [torch.tensor([[int(t)]], device="cuda") for t in token_ids(seed, "next", case["tokens"], 128000)]
    elif kind == "sft":
        from leopard_b200.train import SFTTrainer
        state["trainer"] = SFTTrainer(state["engine"])
        state["batch"] = (*sft_batch(case, seed), pixels(seed, case["crops"]))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "tower":
        return state["engine"].image_features(state["pixels"])
    if kind in ("decoder", "request"):
        logits, kv, _ = state["engine"].prefill(state["samples"], "last", want_kv=True)
        return {"logits": logits, "kv": kv}
    if kind == "decode":
        past, logits = state["past"], []
        for t in state["tokens"]:
            out = state["model"](input_ids=t, past_key_values=past)
            past = out.past_key_values
            logits.append(out.logits)
        return {"logits": logits, "kv": state["kv"][:, :, case["context"]:]}
    if kind == "sft":
        tr = state["trainer"]
        loss, norm = tr.step(*state["batch"])
        return {"loss": loss, "norm": norm, "grads": {n: tr.grad(n) for n in tr.names}}
    from leopard_b200.seqlm import StepEntry
    eng, score = state["engine"], case["score"]
    out = {"prompts": eng.step([StepEntry(i, p, range(max(0, len(p) - score), len(p))) for i, (p, _) in enumerate(state["requests"])])}
    steps = [eng.step([StepEntry(i, [nxt[t]], [0]) for i, (_, nxt) in enumerate(state["requests"])]) for t in range(case["steps"])]
    for i in range(case["batch"]):
        eng.finish(i)
    if steps:
        out["steps"] = torch.cat(steps)
    return out


# ------------------------------------------------------------------------------------------------------------------------ work and tolerance
def lm_params(case, tokens):
    """(weights a step over `tokens` tokens reads, weights one token meets), head excluded"""
    D, H, read, meet = case["width"], case["heads"], 0, 0
    for mixer, ff in parts(case):
        if mixer == "retention":
            n = 5 * D * H * 128
        elif mixer == "latent":
            n = D * (H * 192 + case["kv_rank"] + 64) + 2 * H * 128 * case["kv_rank"] + D * H * 128
        elif mixer == "mingru":
            n = 4 * D * D
        else:
            n = 2 * D * H * 128 + 2 * D * max(H // 4, 1) * 128
        read, meet = read + n, meet + n
        if ff == "dense":
            read, meet = read + 2 * D * case["ff"], meet + 2 * D * case["ff"]
        elif ff == "moe":
            one, shared = 3 * D * case["expert_ff"], 3 * D * D
            read += shared + one * min(case["experts"], tokens * case["top"])
            meet += shared + one * case["top"]
    return read, meet


def lm_attention_flops(case, first, n):
    """mixers' own multiply-adds over positions first .. first + n - 1 of one request, as operations"""
    H, W, f = case["heads"], case["window"], 0
    seen = sum(min(p + 1, W) for p in range(first, first + n))
    for mixer, _ in parts(case):
        if mixer == "retention":
            f += n * H * 4 * 128 * 128
        elif mixer == "latent":
            f += seen * H * 2 * (192 + 128)
        elif mixer != "mingru":
            f += seen * H * 4 * 128
    return f


def work(case):
    kind = case["kind"]
    D, FF, d, ff = VIT["hidden"], VIT["ffn"], DEC["hidden"], DEC["ffn"]
    vit_layer = 4 * D * D + 2 * D * FF
    dec_layer = 2 * d * d + 2 * d * 1024 + 3 * d * ff
    proj = d * 4 * D + d * d

    def tower(n, layers):
        t = n * VIT["patches"]
        f = layers * (2 * t * vit_layer + 4 * t * VIT["patches"] * D) + 2 * t * 588 * D + 2 * n * CROP_ROWS * proj
        return f, 2 * (layers * vit_layer + 588 * D + proj) + n * 3 * 364 * 364 * 4

    def prefill(lengths, layers, vocab):
        rows = sum(lengths)
        f = layers * (2 * rows * dec_layer + sum(2 * s * s * d for s in lengths)) + 2 * len(lengths) * d * vocab
        return f, 2 * (layers * dec_layer + vocab * d) + 4 * layers * rows * 1024 + 4 * vocab * len(lengths) + 2 * rows * d
    if kind == "tower":
        f, b = tower(case["crops"], case["layers"])
        return {"flops": f, "bytes": b + case["crops"] * CROP_ROWS * d * 2}
    if kind == "decoder":
        f, b = prefill([s for s in (case["first"], case["second"]) if s], case["layers"], 128256 if case["model"] == "llama" else 32003)
        return {"flops": f, "bytes": b}
    if kind == "request":
        f, b = tower(case["crops"], 27)
        g, c = prefill([case["text"] + case["crops"] * CROP_ROWS], 32, 128256)
        return {"flops": f + g, "bytes": b + c}
    if kind == "decode":
        n = case["tokens"]
        weights = case["layers"] * dec_layer + 128256 * d
        return {"flops": 2 * n * weights, "bytes": n * (2 * weights + case["layers"] * 4 * 1024 * (case["context"] + n // 2) + 4 * 128256)}
    if kind == "sft":
        s = case["length"]
        f, b = tower(case["crops"], 1)
        linear = dec_layer + SFT_VOCAB * d
        params = linear + SFT_VOCAB * d + proj
        # forward, backward by inputs and by weights, attention once forward and two and a half times back; gradients written, weights, main
        # copies and two moments read and written
        return {"flops": f + 6 * s * linear + 3.5 * 2 * s * s * d + 4 * case["crops"] * CROP_ROWS * proj, "bytes": b + params * (4 + 2 * 2 + 2 * 12)}
    flops = bytes_ = 0
    lens = lm_lengths(case)
    head = case["width"] * case["vocab"]
    wanted = [min(case["score"], n) for n in lens]
    for step, (rows, out) in enumerate([(sum(lens), sum(wanted))] + [(case["batch"], case["batch"])] * case["steps"]):
        read, meet = lm_params(case, rows)
        flops += 2 * rows * meet + 2 * out * head
        for n in lens:
            flops += lm_attention_flops(case, 0, n) if step == 0 else lm_attention_flops(case, n + step - 1, 1)
        kept = 0
        for mixer, _ in parts(case):
            for n in lens:
                if mixer == "retention":
                    kept += 4 * case["heads"] * 128 * 128 * (1 if step == 0 else 2)
                elif mixer == "latent":
                    kept += 4 * (case["kv_rank"] + 64) * (n if step == 0 else min(n + step, case["window"]))
                elif mixer != "mingru":
                    kept += 4 * max(case["heads"] // 4, 1) * 256 * (n if step == 0 else min(n + step, case["window"]))
        bytes_ += 2 * (read + head) + kept + 4 * out * case["vocab"]
    return {"flops": flops, "bytes": bytes_}


def tolerance(case):
    """About four times what another order of the sums shows; 16-bit roundings that fall the other way travel through the layers, and an
    expert chosen by a near tie exchanges a whole row."""
    if case["kind"] == "lm":
        if case["dtype"] == "float32":
            return {"rel": 2e-5, "max": 1e-3}
        return {"rel": 0.03, "max": 0.99} if "moe" in case["layers"] else {"rel": 0.01, "max": 0.2}
    return {"tower": {"rel": 0.025, "max": 0.4}, "decoder": {"rel": 0.03, "max": 0.4}, "request": {"rel": 0.03, "max": 0.9},
            "decode": {"rel": 0.03, "max": 0.4}, "sft": {"rel": 0.025, "max": 0.9}}[case["kind"]]


# ------------------------------------------------------------------------------------------------------------------------ 64 bits
def unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def half_turn(x, cos, sin):
    """entries i and i + n of the last dimension turn together, cos and sin [rows, n], x [rows, heads, 2 n]"""
    a, b = x.chunk(2, -1)
    c, s = cos[:, None], sin[:, None]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def exact_tower(get, layers, x):
    D, H, eps = VIT["hidden"], VIT["heads"], VIT["eps"]
    g = lambda n: get(VT + n).double()  # noqa: E731
    x = F.conv2d(x.double(), g("embeddings.patch_embedding.weight"), g("embeddings.patch_embedding.bias"), stride=14).flatten(2).transpose(1, 2)
    x = x + g("embeddings.position_embedding.weight")
    n, t, _ = x.shape
    for i in range(layers):
        p = f"encoder.layers.{i}."
        h = F.layer_norm(x, (D,), g(p + "layer_norm1.weight"), g(p + "layer_norm1.bias"), eps)
        q, k, v = (F.linear(h, g(p + f"self_attn.{c}_proj.weight"), g(p + f"self_attn.{c}_proj.bias")).view(n, t, H, D // H).transpose(1, 2) for c in "qkv")
        a = torch.cat([torch.softmax(q[j] @ k[j].transpose(-1, -2) * (D // H) ** -0.5, -1).matmul(v[j])[None] for j in range(n)])
        x = x + F.linear(a.transpose(1, 2).reshape(n, t, D), g(p + "self_attn.out_proj.weight"), g(p + "self_attn.out_proj.bias"))
        h = F.layer_norm(x, (D,), g(p + "layer_norm2.weight"), g(p + "layer_norm2.bias"), eps)
        h = F.gelu(F.linear(h, g(p + "mlp.fc1.weight"), g(p + "mlp.fc1.bias")), approximate="tanh")
        x = x + F.linear(h, g(p + "mlp.fc2.weight"), g(p + "mlp.fc2.bias"))
    x = F.layer_norm(x, (D,), g("post_layernorm.weight"), g("post_layernorm.bias"), eps)
    return x.view(n, 13, 2, 13, 2, D).permute(0, 1, 3, 2, 4, 5).reshape(n, CROP_ROWS, 4 * D)


def exact_project(get, x):
    g = lambda n: get(PJ + n).double()  # noqa: E731
    return F.linear(F.gelu(F.linear(x, g("linear_1.weight"), g("linear_1.bias"))), g("linear_2.weight"), g("linear_2.bias"))


def leopard_angles(positions, llama):
    theta = 500000.0 if llama else 10000.0
    inv = 1.0 / theta ** (torch.arange(0, 128, 2, dtype=F64) / 128)
    if llama:
        wave = 2 * math.pi / inv
        s = (8192 / wave - 1.0) / (4.0 - 1.0)
        inv = torch.where(wave > 8192, inv / 8.0, torch.where(wave < 2048, inv, (1 - s) * inv / 8.0 + s * inv))
    a = positions.double()[:, None] * inv.cuda()
    return a.cos(), a.sin()


def exact_attention(q, k, v, first):
    """causal grouped-query attention of rows first .. of one sequence, q [n, H, 128], k and v [first + n, G, 128]"""
    n, H, _ = q.shape
    rep = H // k.shape[1]
    hidden = torch.arange(k.shape[0], device=q.device)[None] > torch.arange(first, first + n, device=q.device)[:, None]
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h // rep].T * 128 ** -0.5).masked_fill(hidden, -math.inf)
        out.append(torch.softmax(s, -1) @ v[:, h // rep])
    return torch.cat(out, -1)


def exact_decoder_layer(get, i, x, lengths, llama, cache=None):
    """x [rows, 4096], the sequences' rows one after another (or the rows that follow `cache` = (k, v)) -> (x, k, v)"""
    g = lambda n: get(f"{LM}layers.{i}.{n}.weight").double()  # noqa: E731
    eps, past = DEC["eps"], 0 if cache is None else cache[0].shape[0]
    h = unit(x, eps) * g("input_layernorm")
    rows = x.shape[0]
    cos, sin = leopard_angles(torch.cat([torch.arange(past, past + n, device=x.device) for n in lengths]), llama)
    q = half_turn((h @ g("self_attn.q_proj").T).view(rows, 32, 128), cos, sin)
    k = half_turn((h @ g("self_attn.k_proj").T).view(rows, 8, 128), cos, sin)
    v = (h @ g("self_attn.v_proj").T).view(rows, 8, 128)
    a, at = [], 0
    for n in lengths:
        s = slice(at, at + n)
        a.append(exact_attention(q[s], k[s] if cache is None else torch.cat([cache[0], k]), v[s] if cache is None else torch.cat([cache[1], v]), past))
        at += n
    x = x + torch.cat(a) @ g("self_attn.o_proj").T
    h = unit(x, eps) * g("post_attention_layernorm")
    return x + (F.silu(h @ g("mlp.gate_proj").T) * (h @ g("mlp.up_proj").T)) @ g("mlp.down_proj").T, k, v


def exact_head(get, x):
    return (unit(x, DEC["eps"]) * get(LM + "norm.weight").double()) @ get("language_model.lm_head.weight").double().T


def exact_prefill(get, x, lengths, layers, llama):
    kv = torch.empty((layers, 2, x.shape[0], 1024), dtype=F64, device=x.device)
    for i in range(layers):
        x, k, v = exact_decoder_layer(get, i, x, lengths, llama)
        kv[i, 0], kv[i, 1] = k.flatten(1), v.flatten(1)
    ends = torch.tensor(lengths).cumsum(0) - 1
    return {"logits": exact_head(get, x[ends.to(x.device)]), "kv": kv}


def exact_sft(case, seed):
    base = leopard_getter(seed, SFT_VOCAB)
    ids, labels, mask = (t[0].cuda() for t in sft_batch(case, seed))
    leaves = {}

    def get(name):
        if name not in leaves:
            leaves[name] = base(name).double().requires_grad_(not name.startswith(VT))
        return leaves[name]
    with torch.no_grad():
        seen = exact_tower(base, 1, pixels(seed, case["crops"]))
    with torch.enable_grad():
        feats = exact_project(get, seen.reshape(-1, seen.shape[-1]))
        table = get(LM + "embed_tokens.weight")
        x = table[ids.clamp(min=0)]
        x = torch.where((ids < 0)[:, None], torch.zeros_like(x).index_put(((ids < 0).nonzero()[:, 0],), feats), x)
        x, _, _ = exact_decoder_layer(get, 0, x, [case["length"]], True)
        logits = exact_head(get, x)[:-1]
        loss = (F.cross_entropy(logits, labels[1:], reduction="none") * mask[1:].double()).sum() / mask[1:].double().sum()
    loss.backward()
    g = {n: t.grad for n, t in leaves.items() if t.grad is not None}
    p = LM + "layers.0."
    gate, up = (g[p + f"mlp.{n}_proj.weight"].reshape(-1, 1, 32, DEC["hidden"]) for n in ("gate", "up"))
    grads = {"dec.lm_head": g["language_model.lm_head.weight"], "dec.final_g": g[LM + "norm.weight"], "dec.0.down_w": g[p + "mlp.down_proj.weight"],
             "dec.0.gateup_w": torch.cat([gate, up], 1).reshape(2 * DEC["ffn"], DEC["hidden"]), "dec.0.ln2_g": g[p + "post_attention_layernorm.weight"],
             "dec.0.o_w": g[p + "self_attn.o_proj.weight"], "dec.0.qkv_w": torch.cat([g[p + f"self_attn.{c}_proj.weight"] for c in "qkv"]),
             "dec.0.ln1_g": g[p + "input_layernorm.weight"], "embed": g[LM + "embed_tokens.weight"], "proj.w2": g[PJ + "linear_2.weight"],
             "proj.b2": g[PJ + "linear_2.bias"], "proj.w1": g[PJ + "linear_1.weight"], "proj.b1": g[PJ + "linear_1.bias"]}
    norm = math.sqrt(sum(float((t * t).sum()) for t in grads.values()))
    return {"loss": float(loss), "norm": norm, "grads": grads}


def lm_frequencies(rot):
    dims, base = rot["dims"], rot["base"]
    i = torch.arange(dims // 2, dtype=F64)
    f, mag, s = base ** (-2.0 * i / dims), 1.0, rot.get("scaling")
    if s and "original" in s:
        at = lambda turns: dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(at(s["fast"])), 0), min(math.ceil(at(s["slow"])), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f, mag = f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1.0
    elif s:
        f = f / s["factor"]
    return f.float().double().cuda(), mag      # a table of 32-bit frequencies is part of the model


def lm_turn(x, rot, pairing="half", sign=1.0):
    n = rot["dims"]
    f, mag = lm_frequencies(rot)
    a = sign * torch.arange(x.shape[0], device=x.device, dtype=F64)[:, None] * f
    cos, sin = a.cos() * mag, a.sin() * mag
    head, rest = x[..., :n], x[..., n:]
    if pairing == "half":
        return torch.cat([half_turn(head, cos, sin), rest], -1)
    u, v = head[..., 0::2], head[..., 1::2]
    c, s = cos[:, None], sin[:, None]
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), rest], -1)


def exact_retention(h, w, m, eps):
    T, H = h.shape[0], m["heads"]
    q, k, v = ((h @ w[c].T).view(T, H, 128) for c in ("q", "k", "v"))
    q, k = lm_turn(q, m["rot"]), lm_turn(k, m["rot"]) * 128 ** -0.5
    t = torch.arange(T, device=h.device)
    gap = (t[:, None] - t[None]).double()
    out = torch.empty_like(v)
    for a in range(H):
        weight = torch.where(gap >= 0, float(np.float32(m["decay"][a])) ** gap.clamp(min=0), 0.0)
        out[:, a] = (q[:, a] @ k[:, a].T * weight) @ v[:, a]
    return unit(out, eps).reshape(T, -1) * F.silu(h @ w["g"].T)


def exact_latent(h, w, m, eps):
    T, H, R = h.shape[0], m["heads"], m["kv_rank"]
    q = (h @ w["q"].T).view(T, H, 192)
    down = h @ w["dkv"].T
    c = unit(down[:, :R], eps) * w["dkv.norm"]
    shared = lm_turn(down[:, None, R:], m["rot"], "adjacent")[:, 0]
    turned = lm_turn(q[..., 128:], m["rot"], "adjacent")
    k, v = (c @ w["uk"].T).view(T, H, 128), (c @ w["uv"].T).view(T, H, 128)
    t = torch.arange(T, device=h.device)
    hidden = (t[None] > t[:, None]) | (t[:, None] - t[None] >= m["mask"]["size"])
    out = torch.empty((T, H, 128), dtype=F64, device=h.device)
    for a in range(H):
        s = (q[:, a, :128] @ k[:, a].T + turned[:, a] @ shared.T) * m["scale"]
        out[:, a] = torch.softmax(s.masked_fill(hidden, -math.inf), -1) @ v[:, a]
    return out.reshape(T, -1)


def exact_window(h, w, m, eps, pooled):
    T, H, G = h.shape[0], m["heads"], m["kv_heads"]
    q, k, v = h @ w["q"].T, h @ w["k"].T, (h @ w["v"].T).view(T, G, 128)
    if pooled:
        q, k = unit(q.view(T, H, 128), eps) * w["q.norm"], unit(k.view(T, G, 128), eps) * w["k.norm"]
    else:
        q, k = (unit(q, eps) * w["q.norm"]).view(T, H, 128), (unit(k, eps) * w["k.norm"]).view(T, G, 128)
    q, k = lm_turn(q, m["rot"]), lm_turn(k, m["rot"])
    whole = {"dims": 128, "base": m["rot"]["base"]}
    t = torch.arange(T, device=h.device)
    size = m["mask"]["size"]
    seen = (t[None] <= t[:, None]) & (t[:, None] - t[None] < size)
    keys, values = k, v
    if pooled:
        v = values = lm_turn(v, whole)
        n, P = T // 64, 64
        keys = torch.cat([k[: n * P].view(n, P, G, 128).mean(1), k])
        values = torch.cat([v[: n * P].view(n, P, G, 128).mean(1), v])
        b = torch.arange(n, device=h.device)
        seen = torch.cat([b[None] * P + P - 1 <= t[:, None] - size, seen], 1)
    else:
        seen = seen | ((t[None] < m["mask"]["keep_first"]) & (t[None] <= t[:, None]))
    out = torch.empty((T, H, 128), dtype=F64, device=h.device)
    for a in range(H):
        s = q[:, a] @ keys[:, a // (H // G)].T * m["scale"]
        if pooled:
            s = m["softcap"] * torch.tanh(s / m["softcap"])
        s = s.masked_fill(~seen, -math.inf)
        if not pooled:       # one more term of weight exp(0) in the denominator
            s = torch.cat([torch.zeros((T, 1), dtype=F64, device=h.device), s], 1)
        p = torch.softmax(s, -1)
        out[:, a] = (p if pooled else p[:, 1:]) @ values[:, a // (H // G)]
    return (lm_turn(out, whole, sign=-1.0) if pooled else out).reshape(T, -1)


def exact_mingru(h, w, m):
    z, u = torch.sigmoid(h @ w["z"].T + w["z.b"]), h @ w["x"].T + w["x.b"]
    add = z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
    state, rows = torch.zeros_like(add[0]), []
    for t in range(h.shape[0]):
        state = torch.addcmul(add[t], 1.0 - z[t], state)
        rows.append(state)
    return torch.stack(rows) * F.silu(h @ w["g"].T)


def exact_experts(h, get, p, f):
    g = lambda n: get(p + n).double()  # noqa: E731
    unit_of = lambda x, e: (F.silu(x @ g(e + ".gate").T) * (x @ g(e + ".up").T)) @ g(e + ".down").T  # noqa: E731
    r = f["router"]
    E, top, G = r["experts"], r["top"], r["groups"]["count"]
    s = torch.sigmoid(h @ g("router").T)
    pick = s + g("correction")
    best = pick.view(-1, G, E // G).topk(2, -1).values.sum(-1).topk(r["groups"]["keep"], -1).indices
    allowed = torch.zeros((h.shape[0], G), dtype=torch.bool, device=h.device).scatter(1, best, True).repeat_interleave(E // G, 1)
    chosen = pick.masked_fill(~allowed, -math.inf).topk(top, -1).indices
    weight = torch.zeros_like(s).scatter(1, chosen, s.gather(1, chosen))
    weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)
    out = torch.sigmoid(h @ g("shared.sg").T) * unit_of(h, "shared")
    for e in range(E):
        rows = weight[:, e].nonzero()[:, 0]
        if rows.numel():
            out[rows] += weight[rows, e, None] * unit_of(h[rows], f"e{e}")
    return out


def exact_lm(case, seed):
    c = lm_config(case)
    get = lm_getter(c, seed)
    eps, sandwich, mult = c["norm"]["eps"], case["model"] == "zudalorn", c.get("residual_mult", 1.0)
    requests = lm_tokens(case, seed)
    ids = [torch.tensor(p + nxt) for p, nxt in requests]
    lengths = [len(t) for t in ids]
    x = get("embed").double()[torch.cat(ids).cuda()]

    def norm(x, name):
        return unit(x, eps) * (get(name).double() if sandwich else 1.0 + get(name).double())
    for i, layer in enumerate(c["layers"]):
        p, m, kind = f"l{i}.", layer["mixer"], layer["type"]
        w = {n: get(p + "mix." + n).double() for n in [k[len(p) + 4:] for k in lm_shapes(c) if k.startswith(p + "mix.")]}
        h = norm(x, p + "norm1")
        y = []
        for part in h.split(lengths):
            y.append(exact_retention(part, w, m, eps) if kind == "retention" else exact_latent(part, w, m, eps) if kind == "latent_attention" else
                     exact_mingru(part, w, m) if kind == "mingru" else exact_window(part, w, m, eps, kind == "attention"))
        y = torch.cat(y) @ w["o"].T
        x = x + (norm(y, p + "norm1b") if sandwich else mult * y)
        f = layer["mlp"]
        if f is None:
            continue
        h = norm(x, p + "norm2")
        if f["kind"] == "moe":
            y = exact_experts(h, get, p + "mlp.", f)
        else:
            z = h @ get(p + "mlp.up").double().T
            if sandwich:
                a = get(p + "mlp.act").double()
                pos, neg = F.softplus(a[0]), 0.5 + F.softplus(a[1])
                z = torch.where(z > 0, pos * z * z + z / 2, neg * (torch.expm1(z.clamp(max=0.0)) - z) + z / 2)
            else:
                z = torch.relu(z) ** 2
            y = z @ get(p + "mlp.down").double().T
        x = x + (norm(y, p + "norm2b") if sandwich else mult * y)
    rows, steps, at = [], [[] for _ in range(case["steps"])], 0
    for (prompt, _), n in zip(requests, lengths):
        last = at + len(prompt)
        rows += range(max(at, last - case["score"]), last)
        for t in range(case["steps"]):
            steps[t].append(last + t)
        at += n
    head, x = get("head").double().T, norm(x, "final.norm")
    out = {"prompts": x[torch.tensor(rows).cuda()] @ head}
    if steps:
        out["steps"] = x[torch.tensor(sum(steps, [])).cuda()] @ head
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "sft":
        return exact_sft(case, seed)
    with torch.no_grad():
        if kind == "lm":
            return exact_lm(case, seed)
        mistral = case.get("model") == "mistral"
        vocab = 32003 if mistral else 1024 if kind == "tower" else 128256
        get = leopard_getter(seed, vocab)
        if kind == "tower":
            return exact_project(get, exact_tower(get, case["layers"], pixels(seed, case["crops"])))
        table = get(LM + "embed_tokens.weight")
        if kind == "decoder":
            lengths = [case[k] for k in ("first", "second") if case[k]]
            ids = np.concatenate([token_ids(seed, k, case[k], min(vocab, 31000)) for k in ("first", "second") if case[k]])
            return exact_prefill(get, table[torch.from_numpy(ids).cuda()].double(), lengths, case["layers"], not mistral)
        if kind == "request":
            ids = request_ids(case, seed).cuda()
            feats = exact_project(get, exact_tower(get, 27, pixels(seed, case["crops"])))
            at = case["text"] // 2
            x = torch.cat([table[ids[:at]].double(), feats.flatten(0, 1), table[ids[at + case["crops"]:]].double()])
            return exact_prefill(get, x, [x.shape[0]], 32, True)
        S, n = case["context"], case["tokens"]
        kv = normal(seed, "cache", (case["layers"], 2, S, 1024))
        x = table[torch.from_numpy(token_ids(seed, "next", n, 128000)).cuda()].double()
        new = torch.empty((case["layers"], 2, n, 1024), dtype=F64, device="cuda")
        for i in range(case["layers"]):
            x, k, v = exact_decoder_layer(get, i, x, [n], True, tuple(t.double().view(S, 8, 128) for t in kv[i]))
            new[i, 0], new[i, 1] = k.flatten(1), v.flatten(1)
        return {"logits": [r.view(1, 1, -1) for r in exact_head(get, x)], "kv": new}
