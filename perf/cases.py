"""The framework's work as a list of timed cases: training steps, prompts and decode steps through the public entry points.

Two models stand for the framework: ``TransformerLM`` (training and serving) and, for the layered decoders, ``Tedirax`` (retention, latent
attention, experts chosen by token; its choices do not depend on rounding, so that its logits can be compared).  Sizes are those of
``configures/*.yaml`` and of ``bench.py``; where a training configuration has many equal layers, fewer of them are taken.

A case is a dict of plain values.  ``prepare`` makes what a program holds before the call (weights, optimizer, engine, requests), ``run`` is
one pass, ``exact`` states the same pass in 64 bits without this package."""
from __future__ import annotations

import math
import random

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

LR, BETAS, EPS, DECAY, CLIP = 3e-4, (0.9, 0.95), 1e-8, 0.1, 1.0      # configures/fsdp_1p3b.yaml
PAIR_EPS = 1e-5                                                       # RMSNorm of the TransformerLM
THETA = 10000.0

SAMPLE = dict(width=512, layers=4, heads=16, ff=1344, vocab=10000)
SMALL = dict(width=768, layers=12, heads=12, ff=2048, vocab=50257)
LARGE = dict(width=2048, layers=24, heads=16, ff=5504, vocab=50257)
WIDE = dict(width=4096, layers=2, heads=32, ff=11008, vocab=32000)


def listed():
    return [
        # configures/sample.yaml as it stands: the small run a user starts with, heads of 32; launches and host time count
        dict(name="train_sample", kind="train", batch=64, seq=256, recompute=False, **SAMPLE),
        # one GPU's share of configures/ddp_124m.yaml, whole: heads of 64, a vocabulary that is not a multiple of anything
        dict(name="train_124m", kind="train", batch=16, seq=1024, recompute=False, **SMALL),
        # one GPU's share of configures/fsdp_1p3b.yaml with 6 of its 24 layers: the headline training workload, heads of 128
        dict(name="train_1p3b", kind="train", batch=8, seq=2048, recompute=False, **{**LARGE, "layers": 6}),
        # one GPU's share of configures/fsdp_7b.yaml with 2 of its 32 layers: long sequences, activation checkpointing
        dict(name="train_7b_recompute", kind="train", batch=2, seq=4096, recompute=True, **WIDE),
        # a batch whose row count is not a multiple of any tile, the last batch of an epoch or a fine-tuning run
        dict(name="train_ragged", kind="train", batch=3, seq=777, recompute=False, **{**SMALL, "layers": 4}),
        # configures/serve_1p3b.yaml: the prompt of a lone user (time to first token), and a full prompt step of the scheduler
        dict(name="prompt_one", kind="prompt", requests=1, shortest=200, longest=200, mix=0, **LARGE),
        dict(name="prompt_many", kind="prompt", requests=8, shortest=128, longest=2048, mix=1, **LARGE),
        # the same model's decode steps: a lone user, a moderately loaded server, a full one
        dict(name="decode_one", kind="decode", requests=1, shortest=900, longest=900, mix=0, **LARGE),
        dict(name="decode_some", kind="decode", requests=20, shortest=128, longest=2400, mix=2, **LARGE),
        dict(name="decode_many", kind="decode", requests=128, shortest=128, longest=2400, mix=3, **LARGE),
        # configures/serve_tedirax.yaml: a full prompt step, and a decode step of a loaded server
        dict(name="layered_prompt", kind="layered_prompt", requests=8, shortest=128, longest=2048, mix=1, **LAYERED),
        dict(name="layered_decode", kind="layered_decode", requests=64, shortest=64, longest=1200, mix=4, **LAYERED),
    ]


LAYERED = dict(width=2048, heads=16, q_rank=1024, kv_rank=512, window=1024, ff=2752, experts=8, top=2, vocab=50257, times=6)


def _spread(rng: random.Random, low: int, high: int) -> int:
    """A whole number whose logarithm is spread evenly."""
    return min(high, int(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))


def draw(rng: random.Random) -> dict:
    most = {c["kind"]: work(c)["flops"] + 200 * work(c)["bytes"] for c in sorted(listed(), key=lambda c: work(c)["flops"])}
    while True:
        kind = rng.choice(["train", "train", "prompt", "decode", "layered_prompt", "layered_decode"])
        if kind == "train":
            head = rng.choice([32, 64, 128])
            heads = _spread(rng, max(2, 256 // head), 2048 // head)
            seq = _spread(rng, 64, 4096)
            case = dict(kind=kind, batch=max(1, _spread(rng, 256, 16384) // seq), seq=seq, recompute=rng.random() < 0.25, width=heads * head,
                        layers=rng.randint(1, 6), heads=heads, ff=8 * rng.randint(heads * head // 4, heads * head // 3),
                        vocab=_spread(rng, 1000, 50257))
        elif kind in ("prompt", "layered_prompt"):
            requests = _spread(rng, 1, 8)
            longest = _spread(rng, 64, 2048)
            case = dict(kind=kind, requests=requests, shortest=_spread(rng, 16, longest), longest=longest, mix=rng.randrange(1 << 20),
                        **(LARGE if kind == "prompt" else LAYERED))
        else:
            longest = _spread(rng, 64, 2400 if kind == "decode" else 1200)
            case = dict(kind=kind, requests=_spread(rng, 1, 128 if kind == "decode" else 64), shortest=_spread(rng, 16, longest),
                        longest=longest, mix=rng.randrange(1 << 20), **(LARGE if kind == "decode" else LAYERED))
        need = work(case)
        if need["flops"] + 200 * need["bytes"] <= most[kind] and (kind != "train" or case["width"] * case["ff"] % 64 == 0):
            return case


# ------------------------------------------------------------------------------------------------------------------- inputs
def _lengths(case) -> list[int]:
    """Tokens of every request; a prompt step holds at most 8192 (the scheduler's budget)."""
    rng = random.Random(case["mix"])
    out = [rng.randint(case["shortest"], case["longest"]) for _ in range(case["requests"])]
    over = sum(out) / 8192 if case["kind"].endswith("prompt") else 0.0
    return [max(1, int(n / over)) for n in out] if over > 1 else out


def _tokens(shape, vocab: int, seed: int, device="cuda"):
    """Token ids as text has them: the frequency of an id falls with its rank (Zipf)."""
    g = torch.Generator("cpu").manual_seed(seed)
    u = torch.rand(shape, generator=g, dtype=torch.float64)
    return (torch.pow(float(vocab), u).long() - 1).clamp_(0, vocab - 1).to(device)


class Weights:
    """Tensors by name, made when they are asked for: random values that bf16 represents exactly."""

    def __init__(self, shapes: dict, seed: int):
        self.shapes, self.seed = shapes, seed
        self.order = {name: i for i, name in enumerate(shapes)}

    def __getitem__(self, name):
        shape = self.shapes[name]
        g = torch.Generator("cuda").manual_seed(self.seed * 1000003 + self.order[name])
        if name.endswith(".table"):
            return torch.rand((shape[0], LAYERED["experts"]), generator=g, device="cuda").argsort(1)[:, :shape[1]].to(torch.int32)
        t = torch.randn(shape, generator=g, device="cuda")
        if len(shape) == 1:
            return (1.0 + 0.1 * t).bfloat16().float()
        std = 1.0 if name in ("embed", "token_embeddings.weight") else math.sqrt(2.0 / sum(shape))
        return (std * t.clamp_(-3.0, 3.0)).bfloat16().float()


def _lm_shapes(case) -> dict:
    d, f = case["width"], case["ff"]
    out = {}
    for i in range(case["layers"]):
        pre = f"layers.{i}."
        out.update({pre + f"attn.{n}.weight": (d, d) for n in ("q_proj", "k_proj", "v_proj", "output_proj")})
        out.update({pre + "ffn.gate_proj.weight": (f, d), pre + "ffn.up_proj.weight": (f, d), pre + "ffn.down_proj.weight": (d, f),
                    pre + "attn_norm.weight": (d,), pre + "ffn_norm.weight": (d,)})
    return {**out, "token_embeddings.weight": (case["vocab"], d), "final_norm.weight": (d,), "lm_head.weight": (case["vocab"], d)}


def _lm(case, seed: int, positions: int):
    from llm_systems_from_scratch_b200.models.transformer import TransformerLM
    with torch.device("cuda"):
        model = TransformerLM(case["vocab"], positions, case["width"], case["layers"], case["heads"], case["ff"], THETA,
                              use_flash_attn=True, use_custom_triton=True)
    weights = Weights(_lm_shapes(case), seed)
    with torch.no_grad():
        for name, p in model.named_parameters():
            if name.endswith("w_gate_up.weight"):
                pre = name[:-len("w_gate_up.weight")]
                p[:case["ff"]].copy_(weights[pre + "gate_proj.weight"])
                p[case["ff"]:].copy_(weights[pre + "up_proj.weight"])
            else:
                p.copy_(weights[name.replace("w_down", "down_proj")])
    return model


def _layered_config(case) -> dict:
    mlp = {"kind": "moe", "expert": {"ff": case["ff"]}, "router": {"experts": case["experts"], "top": case["top"]}}
    mixer = {"heads": case["heads"], "dim": 128, "vdim": 128}
    ret = {"type": "retention", "mlp": mlp, "mixer": {**mixer, "decay": _decay(case["heads"]), "rot": {"base": THETA, "dims": 128}}}
    lat = {"type": "latent_attention", "mlp": mlp, "mixer": {**mixer, "q_rank": case["q_rank"], "kv_rank": case["kv_rank"],
                                                             "scale": 128 ** -0.5, "mask": {"size": case["window"]}}}
    return {"architecture": "Tedirax", "vocab": case["vocab"], "width": case["width"], "norm": {"eps": 1e-6},
            "loop": {"start": 0, "stop": 4, "times": case["times"]}, "layers": [ret, ret, ret, lat]}


def _decay(heads: int) -> list[float]:
    return [1.0 - 2.0 ** (-5.0 - 2.0 * i / max(1, heads - 1)) for i in range(heads)]


def _layered_shapes(case) -> dict:
    w, hd, f = case["width"], case["heads"] * 128, case["ff"]
    out = {"embed": (case["vocab"], w)}
    for i in range(4):
        pre = f"l{i}."
        if i < 3:
            mix = {"q": (hd, w), "k": (hd, w), "v": (hd, w), "g": (hd, w), "o": (w, hd)}
        else:
            q, c = case["q_rank"], case["kv_rank"]
            mix = {"dq": (q, w), "dq.norm": (q,), "uq": (hd, q), "dkv": (c, w), "dkv.norm": (c,), "uk": (hd, c), "uv": (hd, c),
                   "g": (hd, w), "o": (w, hd)}
        out[pre + "norm1"] = (w,)
        out.update({pre + "mix." + k: v for k, v in mix.items()})
        for e in range(case["experts"]):
            out.update({f"{pre}mlp.e{e}.gate": (f, w), f"{pre}mlp.e{e}.up": (f, w), f"{pre}mlp.e{e}.down": (w, f)})
        out[pre + "mlp.table"] = (case["vocab"], case["top"])
    return {**out, "final.norm": (w,), "head": (case["vocab"], w)}


def _prompts(case, seed: int) -> list[list[int]]:
    return [_tokens((n,), case["vocab"], seed * 4099 + i, "cpu").tolist() for i, n in enumerate(_lengths(case))]


def _cached(case, seed: int, layer: int):
    """Keys and values of all requests' earlier tokens at one layer, one request after the other (tokens, width), as projections of normed rows
    have them."""
    g = torch.Generator("cuda").manual_seed(seed * 7919 + layer)
    total = sum(_lengths(case))
    std = math.sqrt(2.0 / (2 * case["width"])) * math.sqrt(case["width"])
    make = lambda: torch.randn((total, case["width"]), generator=g, device="cuda", dtype=torch.bfloat16).mul_(std)
    return make(), make()


# ------------------------------------------------------------------------------------------------------------------ prepare
class TrainState:
    def __init__(self, case, seed):
        from llm_systems_from_scratch_b200.ops.functional import clip_gradient
        from llm_systems_from_scratch_b200.optim import FusedAdamW
        self.model = _lm(case, seed, case["seq"])
        self.model.activation_checkpointing = case["recompute"]
        arena = self.model.engine().provider.arena
        arena.bind_grads()
        self.opt = FusedAdamW(self.model.parameters(), lr=LR, betas=BETAS, eps=EPS, weight_decay=DECAY)
        self.clip = clip_gradient
        ids = _tokens((case["batch"], case["seq"] + 1), case["vocab"], seed)
        self.x, self.y = ids[:, :-1].contiguous(), ids[:, 1:].contiguous()
        units = [arena.group_range(u) for u in [f"layer{i}" for i in range(case["layers"])] + ["embed", "lmhead"]]
        self.grads = [arena.grad[a:b] for a, b in units]
        self.weights = [arena.master[a:b] for a, b in units]

    def run(self):
        """One step of ``train.py``: loss, gradients, clipping, update."""
        loss = self.model.loss(self.x, self.y)
        loss.backward()
        self.clip(self.model.parameters(), CLIP)
        self.opt.step()
        return {"loss": loss.detach(), "grads": self.grads, "weights": self.weights}


def _model(case, seed: int, positions: int):
    if not case["kind"].startswith("layered"):
        return _lm(case, seed, positions)
    from llm_systems_from_scratch_b200.models.tedirax import Tedirax
    return Tedirax(_layered_config(case), Weights(_layered_shapes(case), seed))


def _cache(engine):
    """What a pass leaves behind for the next: pages and states of every layer run; of the TransformerLM, whose cache may be most of the memory,
    the last layer's keys and values."""
    cache = engine.cache
    return cache.entries if hasattr(cache, "entries") else [cache.k[-1], cache.v[-1]]


class PromptState:
    """Requests that bring their prompts to the serving engine; the logits behind each prompt come back, and what the cache holds then."""

    def __init__(self, case, seed):
        from llm_systems_from_scratch_b200.serving import ServingEngine
        self.prompts = _prompts(case, seed)
        context = max(256, -(-max(map(len, self.prompts)) // 64) * 64)
        pages = sum(-(-len(p) // 16) for p in self.prompts)
        self.engine = ServingEngine(_model(case, seed, context), num_pages=pages + 8, max_batch=len(self.prompts), max_context=context)

    def run(self):
        reqs = [self.engine.open(i) for i in range(len(self.prompts))]
        logits = self.engine.extend([(r, p, [len(p) - 1]) for r, p in zip(reqs, self.prompts)])
        for r in reqs:
            self.engine.close(r)
        return {"logits": logits, "cache": _cache(self.engine)}


class DecodeState:
    """Requests in the middle of their output: one captured decode step, whose inputs arrive in pinned memory as they do in the engine's loop."""

    def __init__(self, case, seed):
        from llm_systems_from_scratch_b200 import ops
        from llm_systems_from_scratch_b200.serving import ServingEngine
        from llm_systems_from_scratch_b200.serving.batch import StepBatch
        lens, layered = _lengths(case), case["kind"].startswith("layered")
        size = 64 if layered else 16
        self.engine = eng = ServingEngine(_model(case, seed, 2560), num_pages=sum(n // size + 1 for n in lens), max_batch=len(lens),
                                          max_context=2560)
        reqs = [eng.open(i) for i in range(len(lens))]
        if layered:
            part, prompts = 16, _prompts(case, seed)
            for at in range(0, len(lens), part):
                eng.extend([(r, p, []) for r, p in zip(reqs[at:at + part], prompts[at:at + part])])
        for r, n in zip(reqs, lens):
            eng.sched.grow(r, n + 1)
        if not layered:
            at = np.concatenate([np.asarray(r.pages)[np.arange(n) // size] * size + np.arange(n) % size for r, n in zip(reqs, lens)])
            at = torch.from_numpy(at).cuda()
            for i in range(case["layers"]):
                k, v = _cached(case, seed, i)
                eng.cache.k[i].view(-1, case["width"])[at] = k
                eng.cache.v[i].view(-1, case["width"])[at] = v
        next_ids = _tokens((len(lens),), case["vocab"], seed + 1, "cpu").tolist()
        self.batch = b = StepBatch.build([(r, n, [t]) for r, n, t in zip(reqs, lens, next_ids)], eng.page_size, eng.max_pages_per_req,
                                         eng.device)
        b.splits = eng.backend.choose_splits(len(lens), eng.max_context)
        self.fed = [(t, t.cpu().pin_memory()) for t in (b.tokens, b.positions, b.slots, b.ctx)]

        def step():
            with torch.no_grad():
                logits = eng.backend.logits(eng.backend.forward(b))
                return logits[:, :case["vocab"]], ops.argmax_rows(logits, case["vocab"])
        # the run before the capture sees idle rows only: a state must not advance
        state = b.state_slots.clone()
        b.slots.fill_(-1)
        b.state_slots.fill_(-1)
        step()
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.logits, self.tokens = step()
        b.state_slots.copy_(state)

    def run(self):
        for there, here in self.fed:
            there.copy_(here, non_blocking=True)
        self.graph.replay()
        return {"logits": self.logits, "tokens": self.tokens, "cache": _cache(self.engine)}


def prepare(case, seed: int):
    kind = case["kind"]
    return TrainState(case, seed) if kind == "train" else PromptState(case, seed) if kind.endswith("prompt") else DecodeState(case, seed)


def run(state):
    return state.run()


# ------------------------------------------------------------------------------------------------------------------- figures
def work(case) -> dict:
    d, v = case["width"], case["vocab"]
    if case["kind"] == "train":
        block = 4 * d * d + 3 * d * case["ff"]
        rows = case["batch"] * case["seq"]
        params = case["layers"] * (block + 2 * d) + 2 * v * d + d
        # weights and both moments are read and written, gradients written; every product three times (forward, both gradients); half of
        # the scores are masked
        return {"bytes": 28.0 * params + 16.0 * rows,
                "flops": 6.0 * rows * (case["layers"] * block + v * d) + 6.0 * case["layers"] * rows * case["seq"] * d}
    lens = _lengths(case)
    rows, last, full = sum(lens), len(lens), sum(n * (n + 1) / 2 for n in lens)
    prompt = case["kind"].endswith("prompt")
    fed = rows if prompt else last
    if not case["kind"].startswith("layered"):
        block = case["layers"] * (4 * d * d + 3 * d * case["ff"])
        pairs = case["layers"] * d * (full if prompt else rows)
        kept = case["layers"] * 4.0 * d * rows                                # keys and values, written by a prompt and read by a step
        return {"bytes": 2.0 * (block + v * d + fed * d) + kept + 4.0 * last * v, "flops": 2.0 * fed * block + 2.0 * last * v * d + 4.0 * pairs}
    hd, runs = case["heads"] * 128, case["times"]
    q, c = case["q_rank"], case["kv_rank"]
    ret, lat = 5 * d * hd, q * d + c * d + 2 * hd * d + hd * q + 2 * hd * c
    expert = 3 * d * case["ff"]
    mix = runs * (3 * ret + lat + 4 * case["top"] * expert)
    seen = sum(min(n, case["window"]) for n in lens)
    near = sum(n * (n + 1) / 2 - max(0, n - case["window"]) * (max(0, n - case["window"]) + 1) / 2 for n in lens)
    chosen = min(case["experts"], fed * case["top"])
    # weights of a pass that repeats its layers are read once
    weights = 3 * ret + lat + 4 * chosen * expert + v * d + fed * d
    states = 3 * runs * last * case["heads"] * 128 * 128 * 4.0 * (1 if prompt else 2)
    latents = runs * 2.0 * c * (rows if prompt else seen)
    recur = 3 * runs * fed * 4.0 * hd * 128
    return {"bytes": 2.0 * weights + states + latents + 4.0 * last * v,
            "flops": 2.0 * fed * mix + 2.0 * last * v * d + recur + 4.0 * runs * hd * (near if prompt else seen)}


def tolerance(case) -> dict:
    """About four times the error that this precision (bf16 operands, fp32 sums) shows against ``exact``: gradients up to 0.0065, logits of
    prompts 0.011, of decode steps 0.018, of the layered decoder 0.022.  Greedy tokens may differ where two logits tie."""
    if case["kind"] == "train":
        return {"rel": 0.025}
    return {"rel": {"prompt": 0.045, "decode": 0.07}.get(case["kind"], 0.09), "differ": 0.2}


# --------------------------------------------------------------------------------------------------------------------- exact
def _norm(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _turn_pairs(x, positions):
    """Rotary embedding of (rows, heads, dim) over pairs (2 i, 2 i + 1)."""
    dim = x.shape[-1]
    angle = positions.double()[:, None] * THETA ** -(torch.arange(0, dim, 2, device=x.device).double() / dim)
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * c - b * s, a * s + b * c), -1).flatten(-2)


def _turn_halves(x, positions):
    """The same over pairs (i, i + dim / 2)."""
    half = x.shape[-1] // 2
    angle = positions.double()[:, None] * THETA ** -(torch.arange(half, device=x.device).double() / half)
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat((a * c - b * s, a * s + b * c), -1)


def _attend(q, k, v, scale, window=0):
    """Causal softmax attention (rows, heads, dim); the queries are the last rows of the keys."""
    n, m = q.shape[0], k.shape[0]
    far = torch.arange(m - n, m, device=q.device)[:, None] - torch.arange(m, device=q.device)[None]
    hidden = (far < 0) | (far >= window) if window else far < 0
    s = torch.einsum("ihd,jhd->hij", q, k) * scale
    return torch.einsum("hij,jhe->ihe", torch.softmax(s.masked_fill(hidden, -math.inf), -1), v)


def _lm_block(x, w, heads, positions, spans, attend):
    """One block of the TransformerLM; ``attend(q, k, v)`` takes rotated heads of one span."""
    h = _norm(x, w("attn_norm"), PAIR_EPS)
    q, k, v = (torch.unflatten(h @ w(f"attn.{n}_proj").T, -1, (heads, -1)) for n in "qkv")
    q, k = _turn_pairs(q, positions), _turn_pairs(k, positions)
    o = torch.cat([attend(i, q[a:b], k[a:b], v[a:b]) for i, (a, b) in enumerate(spans)]).flatten(1)
    x = x + o @ w("attn.output_proj").T
    h = _norm(x, w("ffn_norm"), PAIR_EPS)
    return x + (torch.nn.functional.silu(h @ w("ffn.gate_proj").T) * (h @ w("ffn.up_proj").T)) @ w("ffn.down_proj").T


def _exact_train(case, seed):
    heads, rows = case["heads"], case["batch"] * case["seq"]
    scale = (case["width"] // heads) ** -0.5
    source = Weights(_lm_shapes(case), seed)
    w = {n: source[n].double().requires_grad_() for n in source.shapes}
    ids = _tokens((case["batch"], case["seq"] + 1), case["vocab"], seed)
    x, y = ids[:, :-1].reshape(-1), ids[:, 1:].reshape(-1)
    spans = [(i * case["seq"], (i + 1) * case["seq"]) for i in range(case["batch"])]
    positions = torch.arange(case["seq"], device="cuda").repeat(case["batch"])
    some = lambda i, q, k, v: checkpoint(lambda *t: _attend(*t, scale), q, k, v, use_reentrant=False)
    hidden = w["token_embeddings.weight"][x]
    for i in range(case["layers"]):
        hidden = checkpoint(lambda t, i=i: _lm_block(t, lambda n: w[f"layers.{i}.{n}.weight"], heads, positions, spans, some), hidden,
                            use_reentrant=False)
    hidden = _norm(hidden, w["final_norm.weight"], PAIR_EPS)
    part = lambda h, t: torch.nn.functional.cross_entropy(h @ w["lm_head.weight"].T, t, reduction="sum") / rows
    loss = sum(checkpoint(part, hidden[a:a + 2048], y[a:a + 2048], use_reentrant=False) for a in range(0, rows, 2048))
    loss.backward()
    coef = (CLIP / (torch.sqrt(sum(t.grad.square().sum() for t in w.values())) + 1e-6)).clamp(max=1.0)
    rate = LR * math.sqrt(1 - BETAS[1]) / (1 - BETAS[0])
    grads, weights = [], []
    attn = ["attn.q_proj", "attn.k_proj", "attn.v_proj", "attn.output_proj"]
    units = [[f"layers.{i}.{n}.weight" for n in (*attn, "ffn.gate_proj", "ffn.up_proj", "ffn.down_proj", "attn_norm", "ffn_norm")]
             for i in range(case["layers"])]
    with torch.no_grad():
        for unit in [*units, ["token_embeddings.weight"], ["final_norm.weight", "lm_head.weight"]]:
            g, p = [], []
            for name in unit:
                one, t = w[name].grad * coef, w[name].detach()
                new = t - rate * (1 - BETAS[0]) * one / (math.sqrt(1 - BETAS[1]) * one.abs() + EPS)
                pad = (0, -t.numel() % 64)                                   # tensors start at multiples of 64 elements
                g.append(torch.nn.functional.pad(one.flatten(), pad))
                p.append(torch.nn.functional.pad((new - LR * DECAY * new).flatten(), pad))
            grads.append(torch.cat(g))
            weights.append(torch.cat(p))
    return {"loss": loss.detach(), "grads": grads, "weights": weights}


@torch.no_grad()
def _exact_lm(case, seed):
    prompt, lens, heads = case["kind"] == "prompt", _lengths(case), case["heads"]
    scale = (case["width"] // heads) ** -0.5
    w = Weights(_lm_shapes(case), seed)
    if prompt:
        ids = torch.tensor(sum(_prompts(case, seed), []), device="cuda")
        positions = torch.cat([torch.arange(n, device="cuda") for n in lens])
        ends = np.cumsum(lens).tolist()
    else:
        ids = _tokens((len(lens),), case["vocab"], seed + 1)
        positions, ends = torch.tensor(lens, device="cuda"), list(range(1, len(lens) + 1))
    spans = list(zip([0, *ends[:-1]], ends))
    starts = [0, *np.cumsum(lens).tolist()]
    x = w["token_embeddings.weight"][ids].double()
    for i in range(case["layers"]):
        kept = None if prompt else _cached(case, seed, i)

        def attend(r, q, k, v):
            if kept is not None:
                before = [t[starts[r]:starts[r + 1]].double().unflatten(-1, (heads, -1)) for t in kept]
                k, v = torch.cat((before[0], k)), torch.cat((before[1], v))
            return _attend(q, k, v, scale)
        x = _lm_block(x, lambda n: w[f"layers.{i}.{n}.weight"].double(), heads, positions, spans, attend)
    h = _norm(x[[e - 1 for e in ends]], w["final_norm.weight"].double(), PAIR_EPS)
    return h @ w["lm_head.weight"].double().T


@torch.no_grad()
def _exact_layered(case, seed):
    eps, heads = 1e-6, case["heads"]
    source = Weights(_layered_shapes(case), seed)
    kept = {n: (t if t.dtype == torch.int32 else t.bfloat16()) for n, t in ((n, source[n]) for n in source.shapes)}
    w = lambda n: kept[n].double()
    seqs = _prompts(case, seed)
    if case["kind"] == "layered_decode":
        seqs = [s + [t] for s, t in zip(seqs, _tokens((len(seqs),), case["vocab"], seed + 1, "cpu").tolist())]
    ids = torch.tensor(sum(seqs, []), device="cuda")
    ends = np.cumsum([len(s) for s in seqs]).tolist()
    spans = list(zip([0, *ends[:-1]], ends))
    positions = torch.cat([torch.arange(len(s), device="cuda") for s in seqs])
    split = lambda t: t.unflatten(-1, (heads, 128))
    decay = torch.tensor(_decay(heads), dtype=torch.float32, device="cuda").double()
    x = w("embed")[ids]
    for i in list(range(4)) * case["times"]:
        pre = f"l{i}."
        h = _norm(x, w(pre + "norm1"), eps)
        m = lambda n, t: t @ w(pre + "mix." + n).T
        if i < 3:
            q, k, v = _turn_halves(split(m("q", h)), positions), _turn_halves(split(m("k", h)), positions) * 128 ** -0.5, split(m("v", h))
            o = torch.empty_like(v)
            for a, b in spans:
                far = positions[a:b, None] - positions[None, a:b]
                fade = torch.where(far < 0, 0.0, decay[:, None, None] ** far.clamp(min=0))
                o[a:b] = torch.einsum("hij,jhe->ihe", torch.einsum("ihd,jhd->hij", q[a:b], k[a:b]) * fade, v[a:b])
            y = m("o", _norm(o, 1.0, eps).flatten(1) * torch.nn.functional.silu(m("g", h)))
        else:
            c = _norm(m("dkv", h), w(pre + "mix.dkv.norm"), eps)
            q = split(m("uq", _norm(m("dq", h), w(pre + "mix.dq.norm"), eps)))
            k, v = split(m("uk", c)), split(m("uv", c))
            o = torch.cat([_attend(q[a:b], k[a:b], v[a:b], 128 ** -0.5, case["window"]) for a, b in spans])
            y = m("o", o.flatten(1) * torch.sigmoid(m("g", h)))
        for e in range(case["experts"]):
            rows = (kept[pre + "mlp.table"][ids] == e).any(1).nonzero().flatten()
            if rows.numel():
                g, u, d = (w(f"{pre}mlp.e{e}.{n}") for n in ("gate", "up", "down"))
                y[rows] += (torch.nn.functional.silu(h[rows] @ g.T) * (h[rows] @ u.T)) @ d.T / case["top"]
        x = x + y
    return _norm(x[[e - 1 for e in ends]], w("final.norm"), eps) @ w("head").T


def exact(case, seed: int):
    """64-bit results, laid out as ``run`` returns them (the cache's pages have an order of their own, and no such value)."""
    if case["kind"] == "train":
        return _exact_train(case, seed)
    logits = _exact_layered(case, seed) if case["kind"].startswith("layered") else _exact_lm(case, seed)
    return {"logits": logits, "cache": None, **({} if case["kind"].endswith("prompt") else {"tokens": logits.argmax(-1)})}
