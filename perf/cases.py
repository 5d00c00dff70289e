"""The work this framework does for its users, as cases that can be timed and checked.

A case is a dict of plain values; `kind` says which path it takes:

  tower      SigLIP vision encoder on a batch of images (`SiglipVisionModel.forward`)
  prompt     images + prompts -> last-position logits and a filled KV cache (`PaliGemmaForConditionalGeneration.forward`)
  answer     whole requests: prompt, then greedily decoded tokens (`PaliGemmaForConditionalGeneration.generate`)
  burst      text-only requests on the ragged-step engine: a step with the prompts, then steps of one token per request
             (`SequenceEngine.step`)
  attention  one windowed softmax-attention sub-layer over the paged cache (`mixers.WindowedSoftmaxAttention`)
  latent     one latent-attention sub-layer (`mixers.LatentAttention`)
  delta      one gated delta-rule sub-layer (`mixers.ChannelDeltaRule`)
  experts    one routed feed-forward (`mixers.RoutedFeedForward`)

The sub-layers and the shortened models have the full layer sizes; only `answer` runs every layer of the 3B model.
"""
import math
import random
import zlib

import torch

from paligemma_multimodal_system_b200 import mixers, seq_ops
from paligemma_multimodal_system_b200.cache import SequenceStore
from paligemma_multimodal_system_b200.engine import SequenceEngine
from paligemma_multimodal_system_b200.modeling_mapedra import MapedraConfig, MapedraForCausalLM
from paligemma_multimodal_system_b200.modeling_paligemma import KVCache, PaliGemmaConfig, PaliGemmaForConditionalGeneration
from paligemma_multimodal_system_b200.modeling_siglip import SiglipVisionConfig, SiglipVisionModel
from paligemma_multimodal_system_b200.random_init import make_state_dict, paligemma_3b_config

DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
LOWRANK = 64  # inner width of the delta rule's two low-rank projections


def listed():
    return [
        # one image at the smallest resolution: the latency of the vision encoder (256 patches)
        dict(name="tower-224-one", kind="tower", image=224, batch=1, layers=4),
        # a batch of images at the middle resolution: throughput (8192 patches in sequences of 1024)
        dict(name="tower-448-batch", kind="tower", image=448, batch=8, layers=4),
        # the first answer of one interactive request
        dict(name="prompt-224-one", kind="prompt", image=224, batch=1, text=7, vision_layers=2, text_layers=2),
        # prompts of a large image, sequences of 4119 tokens
        dict(name="prompt-896-pair", kind="prompt", image=896, batch=2, text=23, vision_layers=2, text_layers=2),
        # one interactive request from the image to the last token, every layer
        dict(name="answer-one", kind="answer", batch=1, text=8, tokens=24),
        # a full decode batch, every layer: the headline workload with shorter answers
        dict(name="answer-batch", kind="answer", batch=64, text=4, tokens=32),
        # 48 chats on the engine, bf16: prompts of 193 .. 256 tokens, then 24 decode steps
        dict(name="burst-bf16", kind="burst", dtype="bfloat16", requests=48, prompt=256, spread=64, steps=24, width=2048, layers=4),
        # a few chats served in full precision
        dict(name="burst-fp32", kind="burst", dtype="float32", requests=5, prompt=150, spread=37, steps=12, width=2048, layers=4),
        # prompts of 897 .. 1024 tokens through one attention sub-layer: sliding window, first tokens kept
        dict(name="attention-prompts", kind="attention", dtype="bfloat16", portions=8, new=1024, spread=128, behind=0, singles=0, context=0,
             width=2048, dim=64, window=1024, keep=4),
        # a mixed step of a serving engine: two portions of long prompts beside 40 decoding requests
        dict(name="latent-mixed", kind="latent", dtype="bfloat16", portions=2, new=333, spread=1, behind=1400, singles=40, context=1100, width=2048),
        # prompts through one recurrent sub-layer
        dict(name="delta-prompts", kind="delta", dtype="bfloat16", portions=6, new=700, spread=150, width=2048),
        # the tokens of one mixed step through one routed feed-forward
        dict(name="experts-step", kind="experts", dtype="bfloat16", rows=300, width=2048, experts=14, ff=1024),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choice(["tower", "tower", "prompt", "prompt", "answer", "burst", "burst", "attention", "attention", "latent", "latent", "delta", "experts"])
    width = rng.choice([1024, 2048, 2048])
    dtype = rng.choice(["bfloat16"] * 4 + ["float32"])
    slow = dtype == "float32"
    if kind == "tower":
        image = rng.choice([224, 448, 896])
        return dict(kind=kind, image=image, batch=_spread(rng, 1, 8192 // (image // 14) ** 2), layers=rng.choice([2, 3, 4]))
    if kind == "prompt":
        image = rng.choice([224, 448, 896])
        return dict(kind=kind, image=image, batch=_spread(rng, 1, 8192 // (image // 14) ** 2), text=_spread(rng, 2, 120), vision_layers=2, text_layers=2)
    if kind == "answer":
        return dict(kind=kind, batch=_spread(rng, 1, 64), text=_spread(rng, 2, 40), tokens=_spread(rng, 12, 32))
    if kind == "burst":
        prompt = _spread(rng, 20, 180 if slow else 400)
        return dict(kind=kind, dtype=dtype, requests=_spread(rng, 1, 6 if slow else min(48, 12000 // prompt)), prompt=prompt, spread=rng.randint(1, prompt // 2),
                    steps=_spread(rng, 6, 24), width=width, layers=4)
    if kind == "attention":
        portions = rng.randint(0, 8)
        singles = rng.randint(0 if portions else 1, 64)
        new = _spread(rng, 2, 256 if slow else 8192 // max(1, portions))
        return dict(kind=kind, dtype=dtype, portions=portions, new=min(new, 2048), spread=rng.randint(1, max(1, min(new, 2048) // 2)), behind=rng.choice([0, 0, rng.randint(1, 1500)]),
                    singles=singles, context=_spread(rng, 1, 3000), width=width, dim=rng.choice([64, 64, 128]), window=rng.choice([0, 512, 1024]), keep=rng.choice([0, 4, 16]))
    if kind == "latent":
        portions = rng.randint(0, 4)
        singles = rng.randint(0 if portions else 1, 64)
        new = _spread(rng, 2, 128 if slow else 1024)
        return dict(kind=kind, dtype=dtype, portions=portions, new=new, spread=rng.randint(1, max(1, new // 2)), behind=rng.choice([0, rng.randint(1, 1500)]),
                    singles=singles, context=_spread(rng, 1, 3000), width=width)
    if kind == "delta":
        portions = rng.randint(1, 8)
        new = _spread(rng, 2, 256 if slow else min(1024, 8192 // portions))
        return dict(kind=kind, dtype=dtype, portions=portions, new=new, spread=rng.randint(1, max(1, new // 2)), width=width)
    return dict(kind=kind, dtype=dtype, rows=_spread(rng, 1, 200 if slow else 8192), width=width, experts=rng.choice([6, 14, 30]), ff=rng.choice([512, 1024]))


# ---------------------------------------------------------------------------------------------------------------------- inputs
class _Tensors:
    """name, shape -> a tensor on the GPU made from (seed, name) alone.  Matrices N(0, 1 / columns), vectors near one; bf16 models get
    values that bf16 can hold."""

    def __init__(self, seed, dtype):
        self.seed, self.dtype, self.got = int(seed), dtype, {}

    def normal(self, name, shape, std=1.0, mean=0.0):
        g = torch.Generator(device="cuda").manual_seed((self.seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)
        return (torch.randn(tuple(shape), generator=g, device="cuda") * std + mean).to(self.dtype)

    def __call__(self, name, shape):
        if name not in self.got:
            shape = tuple(LOWRANK if n is None else n for n in shape)
            if name.endswith(("A_log", "dt_bias")):
                t = self.normal(name, shape, 0.6, -1.8)
            elif name.endswith("correction"):
                t = self.normal(name, shape, 0.02)
            elif name.endswith("conv"):
                t = self.normal(name, shape, 0.5)
            elif len(shape) == 1:
                t = self.normal(name, shape, 0.1, 1.0)
            else:
                t = self.normal(name, shape, shape[-1] ** -0.5)
            self.got[name] = t
        return self.got[name]


def _lengths(n, longest, spread):
    return [max(1, longest - (i * 37) % spread) for i in range(n)]


def _entries(c):
    """[(new tokens, tokens already stored)] of a sub-layer case."""
    got = [(n, c.get("behind", 0)) for n in _lengths(c["portions"], c["new"], c["spread"])]
    return got + [(1, max(0, c["context"] - (i * 53) % max(1, c["context"] // 2))) for i in range(c.get("singles", 0))]


# ---------------------------------------------------------------------------------------------------------------------- the models
def _paligemma(c):
    cfg = paligemma_3b_config(c.get("image", 224))
    if c["kind"] == "prompt":
        cfg["vision_config"]["num_hidden_layers"], cfg["text_config"]["num_hidden_layers"] = c["vision_layers"], c["text_layers"]
    return cfg


def _paligemma_inputs(c, seed, cfg):
    n = (cfg["vision_config"]["image_size"] // 14) ** 2
    g = torch.Generator(device="cuda").manual_seed(seed * 7 + 1)
    ids = torch.randint(3, 250000, (c["batch"], n + c["text"]), generator=g, device="cuda")
    ids[:, :n], ids[:, n], ids[:, -1] = cfg["image_token_index"], 2, 108
    size = cfg["vision_config"]["image_size"]
    px = torch.rand(c["batch"], 3, size, size, generator=g, device="cuda") * 2 - 1
    return ids, px.to(torch.bfloat16).float(), torch.ones_like(ids)


def _mapedra_config(c):
    """Three layers of decayed linear attention to one of softmax attention, 64-wide heads, four key / value heads to sixteen query heads."""
    w, heads = c["width"], c["width"] // 64
    ls = []
    for i in range(c["layers"]):
        mlp = {"kind": "dense", "ff": 4 * w}
        if i % 4 == 3:
            rot = {"base": 1e6, "dims": 32, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
            ls.append({"type": "attention", "mlp": mlp,
                       "mixer": {"heads": heads, "kv_heads": heads // 4, "dim": 64, "vdim": 64, "scale": 0.125, "softcap": 50.0, "rot": rot}})
        else:
            ls.append({"type": "lightning", "mlp": mlp,
                       "mixer": {"heads": heads, "dim": 64, "vdim": 64, "decay": [1.0 - 2.0 ** (-5 - 3 * h / heads) for h in range(heads)]}})
    return {"architecture": "Mapedra", "vocab": 32000, "width": w, "embedding": {"scale": w ** 0.5}, "norm": {"eps": 1e-6, "groups": 4},
            "token_side": {"dim": 64}, "layers": ls}


def _mapedra_weights(cfg, t):
    w, ff = cfg["width"], 4 * cfg["width"]
    out = {"embed": t.normal("embed", (cfg["vocab"], w), 0.05), "side.embed": t("side.embed", (cfg["vocab"], 64 * len(cfg["layers"]))),
           "final.norm": t("final.norm", (w,)), "head": t("head", (cfg["vocab"], w))}
    for i, l in enumerate(cfg["layers"]):
        m, p = l["mixer"], f"l{i}."
        shapes = {"norm1": (w,), "norm2": (w,), "mlp.gate": (ff, w), "mlp.up": (ff, w), "mlp.down": (w, ff), "side.gate": (64, w), "side.proj": (w, 64),
                  "side.norm": (w,), "mix.q": (w, w), "mix.g": (w, w), "mix.o": (w, w)}
        kv = w if l["type"] == "lightning" else m["kv_heads"] * 64
        shapes.update({"mix.k": (kv, w), "mix.v": (kv, w)})
        shapes.update({"mix.norm": (w,)} if l["type"] == "lightning" else {"mix.q.norm": (64,), "mix.k.norm": (64,)})
        out.update({p + n: t(p + n, s) for n, s in shapes.items()})
    return out


def _burst_tokens(c, seed):
    r = random.Random(seed * 31 + 5)
    prompts = [[r.randrange(32000) for _ in range(n)] for n in _lengths(c["requests"], c["prompt"], c["spread"])]
    return prompts, [[r.randrange(32000) for _ in range(c["requests"])] for _ in range(c["steps"])]


def _mixer(c):
    w, heads = c["width"], c["width"] // c.get("dim", 64)
    if c["kind"] == "attention":
        return mixers.WindowedSoftmaxAttention(w, heads, heads // 4, c["dim"], c["dim"], c["dim"] ** -0.5, 1e-5, window=c["window"] or None, keep_first=c["keep"],
                                               rot_dims=c["dim"], rot_base=1e6)
    if c["kind"] == "latent":
        return mixers.LatentAttention(w, heads, 64, 32, 64, 3 * w // 8, w // 8, 96 ** -0.5, 32, 1e6, 1e-6)
    return mixers.ChannelDeltaRule(w, heads, heads, 64, 64, 4, 1e-6)


def prepare(case, seed):
    c, kind = case, case["kind"]
    torch.cuda.set_device(0)
    if kind == "tower":
        cfg = dict(paligemma_3b_config(c["image"])["vision_config"], num_hidden_layers=c["layers"])
        sd = make_state_dict(dict(paligemma_3b_config(c["image"]), vision_config=cfg, text_config=dict(_tiny_text())), "R1", seed, device="cuda", dtype=torch.bfloat16)
        model = SiglipVisionModel(SiglipVisionConfig(**cfg), device="cuda", dtype=torch.bfloat16).eval()
        model.load_state_dict({k[len("vision_tower."):]: v for k, v in sd.items() if k.startswith("vision_tower.")}, strict=True, assign=True)
        model.pack()
        g = torch.Generator(device="cuda").manual_seed(seed * 7 + 1)
        return dict(kind=kind, model=model, px=torch.rand(c["batch"], 3, c["image"], c["image"], generator=g, device="cuda") * 2 - 1)
    if kind in ("prompt", "answer"):
        cfg = _paligemma(c)
        model = PaliGemmaForConditionalGeneration(PaliGemmaConfig(**cfg), device="meta", dtype=torch.bfloat16).eval()
        model.load_state_dict(make_state_dict(cfg, "R1", seed, device="cuda", dtype=torch.bfloat16), strict=True, assign=True)
        model.tie_weights()
        model.pack()
        ids, px, mask = _paligemma_inputs(c, seed, cfg)
        return dict(kind=kind, model=model, ids=ids, px=px, mask=mask, tokens=c.get("tokens"))
    dtype = DTYPES[c["dtype"]]
    t = _Tensors(seed, dtype)
    if kind == "burst":
        cfg = _mapedra_config(c)
        model = MapedraForCausalLM(MapedraConfig(cfg), dtype).load_weights(_mapedra_weights(cfg, t))
        model.pack()
        prompts, later = _burst_tokens(c, seed)
        pages = sum((len(p) + c["steps"] + 63) // 64 for p in prompts)
        return dict(kind=kind, engine=SequenceEngine(model, max_tokens=64 * pages, num_slots=c["requests"]), prompts=prompts, later=later)
    prec = seq_ops.Precision(dtype)
    if kind == "experts":
        ff = mixers.RoutedFeedForward(c["width"], c["experts"], 2, 4, 2, 1, 2.5, c["ff"], 2 * c["ff"])
        ff.load(t, "")
        ff.pack(prec)
        return dict(kind=kind, ff=ff, prec=prec, h=t.normal("h", (c["rows"], c["width"])))
    mixer, entries = _mixer(c), _entries(c)
    mixer.load(t, "")
    mixer.pack(prec)
    specs = mixer.cache_specs() if hasattr(mixer, "cache_specs") else [mixer.cache_spec()]
    store = SequenceStore(specs, 64 * sum((n + b + 63) // 64 for n, b in entries), len(entries), dtype)
    for pages, what in ((store.k_pages[0], "k"), (store.v_pages[0], "v")):  # what earlier steps left
        if pages is not None:
            pages.copy_(t.normal("cached " + what, pages.shape))
    rows = []
    for i, (n, behind) in enumerate(entries):
        rec = store.admit(i)
        store.reserve(i, behind + n)
        rows.append(dict(tokens=[1] * n, ctx=behind, slot=rec.slot, pages=rec.pages))
    b = seq_ops.make_step_batch(rows)
    return dict(kind=kind, mixer=mixer, prec=prec, store=store, batch=b, h=t.normal("h", (b.T, c["width"])))


def _tiny_text():
    return dict(hidden_size=64, intermediate_size=64, num_hidden_layers=0, num_attention_heads=1, num_key_value_heads=1, head_dim=64, vocab_size=8)


def run(state):
    s, kind = state, state["kind"]
    if kind == "tower":
        return s["model"](s["px"])
    if kind == "prompt":
        kv = KVCache()
        out = s["model"](input_ids=s["ids"], pixel_values=s["px"], attention_mask=s["mask"], kv_cache=kv, last_only=True)
        return {"logits": out["logits"], "k": kv.k_pages, "v": kv.v_pages}
    if kind == "answer":
        tokens = s["model"].generate(s["ids"], s["px"], s["mask"], s["tokens"])
        return {"tokens": tokens, "logits": s["model"].language_model.decode_buffers(tokens.shape[0])["logits"]}  # of the last step
    if kind == "burst":
        eng, ids = s["engine"], list(range(len(s["prompts"])))
        first = eng.step([(i, p, [len(p) - 1]) for i, p in enumerate(s["prompts"])])
        last = len(s["later"]) - 1
        return {"first": first, "later": [eng.step([(i, [t], [0]) for i, t in zip(ids, toks)], ids if k == last else ()) for k, toks in enumerate(s["later"])]}
    if kind == "experts":
        return s["ff"](s["h"], None, s["prec"])
    store = s["store"]
    y = s["mixer"](s["h"], s["batch"], store, 0, s["prec"])
    if kind == "delta":
        return {"y": y, "state": store.state[0], "rows": store.state[1]}
    return {"y": y, "k": store.k_pages[0], "v": store.v_pages[0]}


# ---------------------------------------------------------------------------------------------------------------------- cost
def _tower_work(cfg, batch):
    D, F, L, n = cfg["hidden_size"], cfg["intermediate_size"], cfg["num_hidden_layers"], (cfg["image_size"] // cfg["patch_size"]) ** 2
    params = L * (4 * D * D + 2 * D * F) + 588 * D
    return params, 2 * batch * n * params + L * 4 * batch * n * n * D, batch * n * D


def _pairs(entries, window=0, keep=0):
    """Query / key pairs of a causal step, with a window that keeps the first tokens."""
    total = 0
    for n, b in entries:
        if not window:
            total += n * b + n * (n + 1) // 2
        else:
            total += sum(min(p + 1, window + keep) for p in range(b, b + n))
    return total


def _keys(entries, window=0, keep=0):
    return sum(min(b + n, n + window + keep if window else b + n) for n, b in entries)


def work(case):
    c, kind = case, case["kind"]
    if kind == "tower":
        cfg = dict(paligemma_3b_config(c["image"])["vision_config"], num_hidden_layers=c["layers"])
        params, flops, out = _tower_work(cfg, c["batch"])
        return {"bytes": 2 * params + 4 * out + 12 * c["batch"] * c["image"] ** 2, "flops": flops}
    if kind in ("prompt", "answer"):
        cfg = _paligemma(c)
        tc, B = cfg["text_config"], c["batch"]
        vparams, vflops, vout = _tower_work(cfg["vision_config"], B)
        S, D, L, V = vout // B // 1152 + c["text"], 2048, tc["num_hidden_layers"], tc["vocab_size"]
        lparams = L * (2048 * 2560 + 2048 * 2048 + 3 * 2048 * 16384)
        flops = vflops + 2 * vout * 2048 + 2 * B * S * lparams + L * 4 * B * S * S * D + 2 * B * V * D
        kv = L * B * S * 256 * 2 * 2
        size = 2 * (vparams + lparams + 1152 * 2048 + V * D) + kv + 4 * B * V + 12 * B * cfg["vision_config"]["image_size"] ** 2
        if kind == "answer":
            n = c["tokens"] - 1
            flops += n * 2 * B * (lparams + V * D) + sum(L * 4 * B * (S + i) * D for i in range(1, n + 1))
            size += n * (2 * (lparams + V * D) + kv)
        return {"bytes": size, "flops": flops}
    e = 2 if c["dtype"] == "bfloat16" else 4
    w = c["width"]
    if kind == "burst":
        lens = _lengths(c["requests"], c["prompt"], c["spread"])
        cfg = _mapedra_config(c)
        params, flops, state, kv = 0, 0, 0, 0
        n, T, steps = len(lens), sum(lens), c["steps"]
        for l in cfg["layers"]:
            G = l["mixer"].get("kv_heads", w // 64)
            params += (3 * w + 2 * G * 64) * w + 12 * w * w + 128 * w
            if l["type"] == "lightning":
                state += n * w * 64 * 4
                flops += (T + n * steps) * 4 * w * 64
            else:
                kv += 2 * G * 64 * e
                flops += 4 * w * sum(_pairs([(m + steps, 0)]) for m in lens)
        flops += 2 * params * (T + n * steps) + 2 * n * (1 + steps) * w * 32000
        size = (1 + steps) * ((params + 32000 * w) * e + n * 32000 * 4) + T * w * e + state * (1 + 2 * steps) + kv * (T + sum(T + n * i for i in range(1, steps + 1)))
        return {"bytes": size, "flops": flops}
    if kind == "experts":
        T, D, F, n = c["rows"], w, c["ff"], c["experts"]
        used = n * (1 - (1 - 4 / (n + 2)) ** T)  # experts that are expected to be chosen at all
        flops = 2 * T * D * (n + 2) + 4 * T * 4 * n / (n + 2) * D * F + 4 * T * D * 2 * F
        return {"bytes": e * (used * 2 * D * F + 4 * D * F + (n + 2) * D + T * D) + 4 * T * D, "flops": flops}
    entries = _entries(c) if kind != "delta" else [(n, 0) for n in _lengths(c["portions"], c["new"], c["spread"])]
    T = sum(n for n, _ in entries)
    if kind == "attention":
        G = w // c["dim"] // 4
        proj = w * (2 * w + 2 * G * c["dim"])
        flops = 2 * T * proj + 4 * w * _pairs(entries, c["window"], c["keep"])
        return {"bytes": e * (proj + T * w + 2 * G * c["dim"] * _keys(entries, c["window"], c["keep"])) + 4 * T * w, "flops": flops}
    if kind == "latent":
        H, Q, R = w // 64, 3 * w // 8, w // 8
        proj = w * (Q + R + 32 + H) + Q * H * 96 + 2 * R * w + w * w
        return {"bytes": e * (proj + T * w + (R + 32) * _keys(entries)) + 4 * T * w, "flops": 2 * T * proj + 2 * H * 160 * _pairs(entries)}
    H = w // 64
    proj = 4 * w * w + w * (H + 2 * LOWRANK) + 2 * w * LOWRANK
    return {"bytes": e * (proj + T * w) + 4 * T * w + len(entries) * w * 64 * 4, "flops": 2 * T * proj + T * H * 6 * 64 * 64}


# ---------------------------------------------------------------------------------------------------------------------- closeness
def tolerance(case):
    """About four times what two runs of one build (split sums land in another order) or a run and the 64-bit result differ by."""
    kind = case["kind"]
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 2e-4}
    if kind == "answer":
        return {"rel": 2e-2, "max": 0.12, "differ": 0.0}
    return {"tower": {"rel": 4e-3, "max": 0.04}, "prompt": {"rel": 1.4e-2, "max": 0.12}, "burst": {"rel": 1.4e-2, "max": 0.12},
            "experts": {"rel": 6e-3, "max": 0.06}}.get(kind, {"rel": 1.4e-2, "max": 0.12})


# ---------------------------------------------------------------------------------------------------------------------- 64 bits
def _d(t):
    return t.detach().to("cuda", torch.float64)


def _lin(x, w, b=None):
    y = x @ _d(w).T
    return y if b is None else y + _d(b)


def _ln(x, w, b, eps=1e-6):
    m = x.mean(-1, keepdim=True)
    return (x - m) / torch.sqrt(((x - m) ** 2).mean(-1, keepdim=True) + eps) * _d(w) + _d(b)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _silu(x):
    return x * torch.sigmoid(x)


def _exact_tower(sd, cfg, px):
    p, D, H, P = "vision_tower.model.", cfg["hidden_size"], cfg["num_attention_heads"], cfg["patch_size"]
    dh = D // H
    w = _d(sd[p + "embeddings.patch_embedding.weight"]).reshape(D, -1)
    out = []
    for img in _d(px):
        cut = img.unfold(1, P, P).unfold(2, P, P)  # [C, n, n, P, P]
        x = cut.permute(1, 2, 0, 3, 4).reshape(-1, 3 * P * P) @ w.T + _d(sd[p + "embeddings.patch_embedding.bias"])
        x = x + _d(sd[p + "embeddings.positional_embeddings.weight"])
        for i in range(cfg["num_hidden_layers"]):
            l = f"{p}encoder.layers.{i}."

            def lin(v, name):
                return _lin(v, sd[l + name + ".weight"], sd[l + name + ".bias"])

            h = _ln(x, sd[l + "layer_norm1.weight"], sd[l + "layer_norm1.bias"])
            q, k, v = (lin(h, f"self_attn.{n}_proj").view(-1, H, dh).transpose(0, 1) for n in ("query", "key", "value"))
            a = torch.softmax(q @ k.transpose(1, 2) * dh ** -0.5, -1) @ v
            x = x + lin(a.transpose(0, 1).reshape(-1, D), "self_attn.out_proj")
            h = _ln(x, sd[l + "layer_norm2.weight"], sd[l + "layer_norm2.bias"])
            x = x + lin(_gelu(lin(h, "mlp.fc1")), "mlp.fc2")
        out.append(_ln(x, sd[p + "post_layernorm.weight"], sd[p + "post_layernorm.bias"]))
    return torch.stack(out)


def _turn_halves(x, pos, base):
    """x [..., S, heads, dh], pos [S]: element i turns with element i + dh / 2."""
    dh = x.shape[-1]
    a = pos[:, None, None] * base ** (-torch.arange(0, dh, 2, device="cuda", dtype=torch.float64) / dh)
    u, v = x[..., : dh // 2], x[..., dh // 2:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def _exact_decoder(sd, cfg, x, first_pos, caches):
    """x [B, s, D] through every layer; caches: per layer the keys and values so far, which every new token sees along with all of x."""
    B, s, D = x.shape
    H, dh = cfg["num_attention_heads"], cfg["head_dim"]
    pos = torch.arange(first_pos, first_pos + s, device="cuda", dtype=torch.float64)
    for i in range(cfg["num_hidden_layers"]):
        l = f"language_model.model.layers.{i}."
        h = _rms(x, 1e-6) * (1 + _d(sd[l + "input_layernorm.weight"]))
        q = _turn_halves(_lin(h, sd[l + "self_attn.q_proj.weight"]).view(B, s, H, dh), pos, 10000.0)
        k = _turn_halves(_lin(h, sd[l + "self_attn.k_proj.weight"]).view(B, s, 1, dh), pos, 10000.0)[:, :, 0]
        v = _lin(h, sd[l + "self_attn.v_proj.weight"])
        if len(caches) > i:
            k, v = torch.cat([caches[i][0], k], 1), torch.cat([caches[i][1], v], 1)
            caches[i] = (k, v)
        else:
            caches.append((k, v))
        a = torch.cat([torch.stack([torch.softmax(q[b, :, j] @ k[b].T * dh ** -0.5, -1) @ v[b] for j in range(H)], 1)[None] for b in range(B)])
        x = x + _lin(a.reshape(B, s, D), sd[l + "self_attn.o_proj.weight"])
        h = _rms(x, 1e-6) * (1 + _d(sd[l + "post_attention_layernorm.weight"]))
        x = x + _lin(_gelu(_lin(h, sd[l + "mlp.gate_proj.weight"])) * _lin(h, sd[l + "mlp.up_proj.weight"]), sd[l + "mlp.down_proj.weight"])
    x = _rms(x[:, -1], 1e-6) * (1 + _d(sd["language_model.model.norm.weight"]))
    return _lin(x, sd["language_model.lm_head.weight"], sd["language_model.lm_head.bias"])


def _exact_paligemma(c, seed):
    cfg = _paligemma(c)
    sd = make_state_dict(cfg, "R1", seed, device="cuda", dtype=torch.bfloat16)
    ids, px, _ = _paligemma_inputs(c, seed, cfg)
    D, (B, S) = 2048, ids.shape
    emb = sd["language_model.model.embed_tokens.weight"]
    img = _lin(_exact_tower(sd, cfg["vision_config"], px), sd["multi_modal_projector.linear.weight"]) * D ** -0.5
    x = torch.cat([img, _d(emb[ids[:, img.shape[1]:]])], 1) * D ** 0.5
    caches = []
    logits = _exact_decoder(sd, cfg["text_config"], x, 1, caches)
    if c["kind"] == "prompt":
        return {"logits": logits[:, None], "k": None, "v": None}
    tokens = [logits.argmax(-1)]
    for t in range(1, c["tokens"]):
        logits = _exact_decoder(sd, cfg["text_config"], _d(emb[tokens[-1]])[:, None] * D ** 0.5, S + t, caches)
        tokens.append(logits.argmax(-1))
    return {"tokens": torch.stack(tokens, 1), "logits": logits}


def _group_rms(x, w, groups, eps):
    return _rms(x.unflatten(-1, (groups, -1)), eps).flatten(-2) * _d(w)


def _turn_pairs(x, pos, freq):
    """x [n, heads, dim], pos [n]: neighbouring elements of the first 2 * len(freq) turn by pos * freq."""
    a, r = pos[:, None, None] * freq, 2 * len(freq)
    u, v = x[..., 0:r:2], x[..., 1:r:2]
    return torch.cat([torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2), x[..., r:]], -1)


def _attend(q, k, v, first, scale, softcap=0.0, window=0, keep=0):
    """q [n, H, dim] at positions first .. first + n - 1, k, v [L, G, .] -> [n, H, vdim]."""
    n, H, L, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    i, j = torch.arange(first, first + n, device="cuda")[:, None], torch.arange(L, device="cuda")[None]
    seen = (j <= i) & ((i - j < window) | (j < keep)) if window else j <= i
    out = torch.empty(n, H, v.shape[-1], device="cuda", dtype=torch.float64)
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].T * scale
        s = softcap * torch.tanh(s / softcap) if softcap else s
        out[:, h] = torch.softmax(s.masked_fill(~seen, -math.inf), -1) @ v[:, h * G // H]
    return out


def _scaled_frequencies(rot):
    f = rot["base"] ** (-torch.arange(0, rot["dims"], 2, device="cuda", dtype=torch.float64) / rot["dims"])
    s = rot["scaling"]
    wave = 2 * math.pi / f
    blend = (s["original"] / wave - s["low"]) / (s["high"] - s["low"])
    mid = (1 - blend) * f / s["factor"] + blend * f
    return torch.where(wave < s["original"] / s["high"], f, torch.where(wave > s["original"] / s["low"], f / s["factor"], mid))


def _exact_burst(c, seed):
    cfg = _mapedra_config(c)
    w = _mapedra_weights(cfg, _Tensors(seed, DTYPES[c["dtype"]]))
    prompts, later = _burst_tokens(c, seed)
    n, D, eps, H = len(prompts), c["width"], 1e-6, c["width"] // 64
    seqs = [p + [s[i] for s in later] for i, p in enumerate(prompts)]
    at = [0]
    for s in seqs:
        at.append(at[-1] + len(s))
    tokens = torch.tensor([t for s in seqs for t in s], device="cuda")
    x = _d(w["embed"][tokens]) * D ** 0.5
    for i, l in enumerate(cfg["layers"]):
        p, m = f"l{i}.", l["mixer"]
        G = m.get("kv_heads", H)
        q, k, v = (_lin(x, w[p + "mix." + s]) for s in "qkv")
        gate = torch.sigmoid(_lin(x, w[p + "mix.g"]))
        if l["type"] == "attention":
            f = _scaled_frequencies(m["rot"])
            out = []
            for a, b in zip(at, at[1:]):
                pos = torch.arange(b - a, device="cuda", dtype=torch.float64)
                qs = _turn_pairs(_rms(q[a:b].view(-1, H, 64), eps) * _d(w[p + "mix.q.norm"]), pos, f)
                ks = _turn_pairs(_rms(k[a:b].view(-1, G, 64), eps) * _d(w[p + "mix.k.norm"]), pos, f)
                out.append(_attend(qs, ks, _rms(v[a:b].view(-1, G, 64), eps), 0, m["scale"], m["softcap"]))
            y = torch.cat(out).reshape(-1, D) * gate
        else:
            longest = max(map(len, seqs))
            pad = torch.zeros(n, longest, 3, D, device="cuda", dtype=torch.float64)
            for j, (a, b) in enumerate(zip(at, at[1:])):
                pad[j, : b - a] = _silu(torch.stack([q[a:b], k[a:b], v[a:b]], 1))
            pad = pad.view(n, longest, 3, H, 64)
            S = torch.zeros(n, H, 64, 64, device="cuda", dtype=torch.float64)
            decay = torch.tensor(m["decay"], dtype=torch.float32, device="cuda").double().view(1, H, 1, 1)
            out = torch.empty(n, longest, H, 64, device="cuda", dtype=torch.float64)
            for t in range(longest):
                S = decay * S + pad[:, t, 1].unsqueeze(-1) * pad[:, t, 2].unsqueeze(-2)
                out[:, t] = (pad[:, t, 0].unsqueeze(-2) @ S).squeeze(-2)
            o = torch.cat([out[j, : b - a] for j, (a, b) in enumerate(zip(at, at[1:]))]).reshape(-1, D)
            y = _rms(o, eps) * _d(w[p + "mix.norm"]) * gate
        x = x + _group_rms(_lin(y, w[p + "mix.o"]), w[p + "norm1"], 4, eps)
        y = _lin(_gelu(_lin(x, w[p + "mlp.gate"])) * _lin(x, w[p + "mlp.up"]), w[p + "mlp.down"])
        x = x + _group_rms(y, w[p + "norm2"], 4, eps)
        e = _d(w["side.embed"][tokens][:, 64 * i:64 * i + 64])
        x = x + _group_rms(_lin(_gelu(_lin(x, w[p + "side.gate"])) * e, w[p + "side.proj"]), w[p + "side.norm"], 1, eps)
    x = _group_rms(x, w["final.norm"], 4, eps)

    def logits(step):
        return _lin(x[torch.tensor([at[i] + len(prompts[i]) + step for i in range(n)], device="cuda")], w["head"])

    return {"first": logits(-1), "later": [logits(s) for s in range(c["steps"])]}


def _exact_mixer(c, seed):
    """The sub-layers over the paged cache.  The state is laid out as `prepare` does: entry after entry, each on pages of its own."""
    t = _Tensors(seed, DTYPES[c["dtype"]])
    w, H = c["width"], c["width"] // c.get("dim", 64)
    entries = _entries(c)
    T = sum(n for n, _ in entries)
    h = _d(t.normal("h", (T, w)))
    pages = sum((n + b + 63) // 64 for n, b in entries)
    out, row, page = torch.empty(T, w, device="cuda", dtype=torch.float64), 0, 0
    if c["kind"] == "attention":
        dim, G = c["dim"], H // 4
        freq = 1e6 ** (-torch.arange(0, dim, 2, device="cuda", dtype=torch.float64) / dim)
        kc, vc = (_d(t.normal("cached " + s, (pages, 64, G * dim))).view(-1, G, dim) for s in "kv")
        q, k, v = (_lin(h, t(s, (n * dim, w))).view(T, n, dim) for s, n in (("q", H), ("k", G), ("v", G)))
    else:
        Q, R, dim = 3 * w // 8, w // 8, 64
        freq = 1e6 ** (-torch.arange(0, 32, 2, device="cuda", dtype=torch.float64) / 32)
        kc = _d(t.normal("cached k", (pages, 64, R + 32))).view(-1, R + 32)
        q = _lin(_rms(_lin(h, t("dq", (Q, w))), 1e-6) * _d(t("dq.norm", (Q,))), t("uq", (H * 96, Q))).view(T, H, 96)
        new = _lin(h, t("dkv", (R + 32, w)))
        new = torch.cat([_rms(new[:, :R], 1e-6) * _d(t("dkv.norm", (R,))), new[:, R:]], -1)
        gate = torch.sigmoid(_lin(h, t("g", (H, w))))
        uk, uv = t("uk", (H * 64, R)), t("uv", (H * 64, R))
    for n, behind in entries:
        a, b, p0 = row, row + n, page * 64
        pos = torch.arange(behind, behind + n, device="cuda", dtype=torch.float64)
        if c["kind"] == "attention":
            ks = torch.cat([kc[p0:p0 + behind], _turn_pairs(k[a:b], pos, freq)])
            o = _attend(_turn_pairs(q[a:b], pos, freq), ks, torch.cat([vc[p0:p0 + behind], v[a:b]]), behind, dim ** -0.5, window=c["window"], keep=c["keep"])
        else:
            rows = torch.cat([kc[p0:p0 + behind], torch.cat([new[a:b, :R], _turn_pairs(new[a:b, None, R:], pos, freq)[:, 0]], -1)])
            lat, rot = rows[:, :R], rows[:, None, R:].expand(-1, H, -1)
            qs = torch.cat([q[a:b, :, :64], _turn_pairs(q[a:b, :, 64:], pos, freq)], -1)
            o = _attend(qs, torch.cat([_lin(lat, uk).view(-1, H, 64), rot], -1), _lin(lat, uv).view(-1, H, 64), behind, 96 ** -0.5) * gate[a:b, :, None]
        out[a:b] = o.reshape(n, w)
        row, page = b, page + (n + behind + 63) // 64
    return {"y": _lin(out, t("o", (w, w))), "k": None, "v": None}


def _exact_delta(c, seed):
    t = _Tensors(seed, DTYPES[c["dtype"]])
    w, H = c["width"], c["width"] // 64
    lens = _lengths(c["portions"], c["new"], c["spread"])
    h = _d(t.normal("h", (sum(lens), w)))
    n, longest = len(lens), max(lens)
    x = torch.zeros(n, longest, w, device="cuda", dtype=torch.float64)
    at = 0
    for i, m in enumerate(lens):
        x[i, :m], at = h[at:at + m], at + m

    def conv(name):
        u, k = _lin(x, t(name, (w, w))), _d(t(name + ".conv", (w, 4)))
        u = torch.cat([torch.zeros(n, 3, w, device="cuda", dtype=torch.float64), u], 1)
        return _silu(sum(k[:, j] * u[:, j:j + longest] for j in range(4))).view(n, longest, H, 64)

    def low(a, b):
        return _lin(_lin(x, t(a, (LOWRANK, w))), t(b, (w, LOWRANK)))

    q, k, v = conv("q"), conv("k"), conv("v")
    q, k = (u / torch.sqrt((u * u).sum(-1, keepdim=True) + 1e-6) for u in (q, k))
    beta = torch.sigmoid(_lin(x, t("b", (H, w))))
    decay = torch.exp(-torch.exp(_d(t("A_log", (H,))))[:, None] * torch.nn.functional.softplus(low("a1", "a2") + _d(t("dt_bias", (w,)))).view(n, longest, H, 64))
    S = torch.zeros(n, H, 64, 64, device="cuda", dtype=torch.float64)
    out = torch.empty(n, longest, H, 64, device="cuda", dtype=torch.float64)
    going = torch.tensor(lens, device="cuda")
    for s in range(longest):
        new = S * decay[:, s].unsqueeze(-1)
        u = beta[:, s].unsqueeze(-1) * (v[:, s] - (k[:, s].unsqueeze(-2) @ new).squeeze(-2))
        new = new + k[:, s].unsqueeze(-1) * u.unsqueeze(-2)
        S = torch.where((going > s).view(-1, 1, 1, 1), new, S)
        out[:, s] = (q[:, s].unsqueeze(-2) @ S).squeeze(-2) / 8
    y = (_rms(out, 1e-6) * _d(t("norm", (64,)))).flatten(-2) * torch.sigmoid(low("g1", "g2"))
    return {"y": _lin(torch.cat([y[i, :m] for i, m in enumerate(lens)]), t("o", (w, w))), "state": S, "rows": None}


def _exact_experts(c, seed):
    t = _Tensors(seed, DTYPES[c["dtype"]])
    T, D, F, n = c["rows"], c["width"], c["ff"], c["experts"]
    h = _d(t.normal("h", (T, D)))
    p = torch.softmax(_lin(h, t("router", (n + 2, D))), -1)
    choice = p + _d(t("correction", (n + 2,)))
    half = choice.view(T, 2, -1)
    best = half.max(-1).values.argmax(-1)  # one of two groups is kept
    choice = torch.full_like(half, -math.inf).scatter(1, best.view(T, 1, 1).expand(-1, 1, half.shape[-1]),
                                                       half.gather(1, best.view(T, 1, 1).expand(-1, 1, half.shape[-1]))).view(T, -1)
    ids = choice.topk(4, -1).indices
    wt = p.gather(1, ids)
    wt = wt / wt.sum(-1, keepdim=True) * 2.5
    out = torch.relu(_lin(h, t("shared.up", (2 * F, D)))) ** 2 @ _d(t("shared.down", (D, 2 * F))).T
    for e in range(n + 2):
        rows, k = (ids == e).nonzero(as_tuple=True)
        if rows.numel():
            y = h[rows] if e >= n else torch.relu(_lin(h[rows], t(f"e{e}.up", (F, D)))) ** 2 @ _d(t(f"e{e}.down", (D, F))).T
            out.index_add_(0, rows, y * wt[rows, k][:, None])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "tower":
        full = paligemma_3b_config(case["image"])
        cfg = dict(full["vision_config"], num_hidden_layers=case["layers"])
        sd = make_state_dict(dict(full, vision_config=cfg, text_config=_tiny_text()), "R1", seed, device="cuda", dtype=torch.bfloat16)
        g = torch.Generator(device="cuda").manual_seed(seed * 7 + 1)
        return _exact_tower(sd, cfg, torch.rand(case["batch"], 3, case["image"], case["image"], generator=g, device="cuda") * 2 - 1)
    if kind in ("prompt", "answer"):
        return _exact_paligemma(case, seed)
    return {"burst": _exact_burst, "delta": _exact_delta, "experts": _exact_experts}.get(kind, _exact_mixer)(case, seed)
