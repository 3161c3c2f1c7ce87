"""What this framework's speed is measured on: the units of work its users run, through its public entry points.

Every case is a dict of plain values.  ``prepare`` builds what a program holds before the call (weights, inputs, the
key / value cache), ``run`` is one pass, ``exact`` states the same pass in plain 64-bit PyTorch.  Eight kinds of work:

* ``decode`` / ``prefill`` - one step of cached generation with the Qwen2.5-VL model (what ``VLMGenerator`` calls per
  token and once per prompt), 7B widths; 8 of the 28 (32) layers of each tower, since the layers of a tower are alike
* ``text``    - training step of a Qwen2.5-VL-7B decoder layer on packed documents (forward, all gradients)
* ``vision``  - training step of a vision-tower block, window or full attention, on packed images
* ``loss``    - final norm, vocabulary projection and cross entropy with all gradients
* ``experts`` - training step of the routed experts of Qwen3-VL-30B-A3B (128 experts, 8 per token)
* ``delta``   - training step of the gated-delta-net mixer of Qwen3.5-9B on packed documents
* ``video``   - a Wan2.1 transformer block: training step at 1.3B width, sampling pass at 14B width
"""
import math

import torch
import torch.nn.functional as F

from mindspeed_mm_b200.models.moe import FusedExperts, MoETextConfig
from mindspeed_mm_b200.models.qwen2_5_vl import DecoderLayer, LMHead, Qwen25VLConfig, Qwen25VLModel, TextConfig, VisionBlock, VisionConfig
from mindspeed_mm_b200.models.qwen3_5 import GatedDeltaNet, Qwen35Config
from mindspeed_mm_b200.models.wan import WanBlock, WanConfig
from mindspeed_mm_b200.data.collate import PackedVLMCollator

DEV = "cuda"
BF16 = torch.bfloat16
LAYERS = 8                                                # per tower in decode / prefill
H, FFN, NQ, NKV, HD, VOCAB = 3584, 18944, 28, 4, 128, 152064
VH, VFFN, VFFN_PAD, VN, VD = 1280, 3420, 3456, 16, 80     # vision tower; its FFN is stored padded to a multiple of 64
EXPERTS, TOPK, EH, EF = 128, 8, 2048, 768
GH, GHK, GHV, GD = 4096, 16, 32, 128
WAN = {"1.3B": (1536, 8960, 12), "14B": (5120, 13824, 40)}
TEXT_LEN = 512
EPS = 1e-6


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # a chat reply, one token: the smallest call, a matrix-vector product with every weight
        dict(name="decode_short", kind="decode", context=311),
        # the same late in a long document: a long cache beside the weights
        dict(name="decode_long", kind="decode", context=9000),
        # a question about one photograph (odd window grid, ragged prompt length)
        dict(name="prefill_image", kind="prefill", image="34x46", text=622),
        # the finetuning pack of bench.py: four samples of 2048 tokens
        dict(name="text_pack", kind="text", docs="2048,2048,2048,2048"),
        # a small ragged pack, as the last batch of an epoch or a short-answer dataset gives
        dict(name="text_ragged", kind="text", docs="517,33,1,870"),
        # the eight 448 x 448 images of that pack: window layers (28 of 32) ...
        dict(name="vision_window", kind="vision", images="32x32,32x32,32x32,32x32,32x32,32x32,32x32,32x32", full=False),
        # ... and a full-attention layer on images of native, uneven resolution
        dict(name="vision_full", kind="vision", images="34x46,22x58,64x80", full=True),
        # output head of the pack
        dict(name="loss_pack", kind="loss", tokens=8192),
        # expert layer of a MoE model, skewed routing
        dict(name="experts_pack", kind="experts", tokens=4096),
        # linear-attention layer on ragged documents
        dict(name="delta_ragged", kind="delta", docs="2048,1500,548"),
        # video DiT finetuning on a short clip (17 frames of 480 x 832)
        dict(name="video_train", kind="video", model="1.3B", grid="5x30x52", train=True),
        # one block of a sampling step on the full clip (81 frames of 480 x 832): the largest
        dict(name="video_sample", kind="video", model="14B", grid="21x30x52", train=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _split(rng, total, most):
    """``total`` cut into 1 .. ``most`` parts at random places."""
    n = rng.randint(1, max(1, min(most, total)))
    cuts = sorted(rng.sample(range(1, total), n - 1)) if n > 1 else []
    return ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]))


def draw(rng):
    kind = rng.choice(["decode", "prefill", "text", "vision", "loss", "experts", "delta", "video"])
    if kind == "decode":
        return dict(kind=kind, context=_log_int(rng, 32, 16000))
    if kind == "prefill":
        return dict(kind=kind, image="%dx%d" % (2 * rng.randint(4, 40), 2 * rng.randint(4, 40)), text=_log_int(rng, 16, 2000))
    if kind == "text":
        return dict(kind=kind, docs=_split(rng, _log_int(rng, 256, 8192), 8))
    if kind == "vision":
        images = ",".join("%dx%d" % (2 * rng.randint(4, 24), 2 * rng.randint(4, 24)) for _ in range(rng.randint(1, 8)))
        return dict(kind=kind, images=images, full=rng.random() < 0.3)
    if kind == "loss":
        return dict(kind=kind, tokens=_log_int(rng, 256, 8192))
    if kind == "experts":
        return dict(kind=kind, tokens=_log_int(rng, 64, 8192))
    if kind == "delta":
        return dict(kind=kind, docs=_split(rng, _log_int(rng, 256, 8192), 6))
    train = rng.random() < 0.6
    grid = "%dx%dx%d" % (rng.randint(1, 5 if train else 21), rng.randint(8, 30), rng.randint(8, 52))
    return dict(kind=kind, model="1.3B" if train else "14B", grid=grid, train=train)


def _ints(text, sep=","):
    return [int(t) for t in text.split(sep)]


def _images(text):
    return [_ints(t, "x") for t in text.split(",")]


# ------------------------------------------------------------------------------------------------ weights and inputs
def _decoder_shapes():
    return {"input_layernorm.weight": (H,), "post_attention_layernorm.weight": (H,),
            "qkv_proj.weight": ((NQ + 2 * NKV) * HD, H), "qkv_proj.bias": ((NQ + 2 * NKV) * HD,),
            "o_proj.weight": (H, NQ * HD), "gate_up_proj.weight": (2 * FFN, H), "down_proj.weight": (H, FFN)}


def _vision_shapes():
    return {"norm1.weight": (VH,), "norm2.weight": (VH,), "attn_qkv.weight": (3 * VH, VH), "attn_qkv.bias": (3 * VH,),
            "attn_proj.weight": (VH, VH), "attn_proj.bias": (VH,), "mlp_gate_up.weight": (2 * VFFN_PAD, VH),
            "mlp_gate_up.bias": (2 * VFFN_PAD,), "mlp_down.weight": (VH, VFFN_PAD), "mlp_down.bias": (VH,)}


def _loss_shapes():
    return {"norm.weight": (H,), "weight": (VOCAB, H)}


def _expert_shapes():
    return {"gate_up_proj": (EXPERTS, EH, 2 * EF), "down_proj": (EXPERTS, EF, EH)}


def _delta_shapes():
    kd, vd = GHK * GD, GHV * GD
    return {"in_proj.weight": (2 * kd + 2 * vd + 2 * GHV, GH), "conv_weight": (2 * kd + vd, 4), "A_log": (GHV,), "dt_bias": (GHV,),
            "norm_weight": (GD,), "out_proj.weight": (GH, vd)}


def _video_shapes(model):
    h, f, _ = WAN[model]
    s = {"modulation": (1, 6, h), "norm3.weight": (h,), "norm3.bias": (h,), "ffn_0.weight": (f, h), "ffn_0.bias": (f,),
         "ffn_2.weight": (h, f), "ffn_2.bias": (h,)}
    for name, out in (("self_attn.qkv", 3 * h), ("self_attn.proj_out", h), ("cross_attn.proj_q", h), ("cross_attn.kv", 2 * h),
                      ("cross_attn.proj_out", h)):
        s[name + ".weight"], s[name + ".bias"] = (out, h), (out,)
    for name in ("self_attn.q_norm", "self_attn.k_norm", "cross_attn.q_norm", "cross_attn.k_norm"):
        s[name + ".weight"] = (h,)
    return s


def _model_shapes():
    s = {"embed_tokens.weight": (VOCAB, H), "visual.patch_embed.proj.weight": (VH, 1176), "visual.merger.ln_q.weight": (VH,),
         "visual.merger.fc1.weight": (4 * VH, 4 * VH), "visual.merger.fc1.bias": (4 * VH,), "visual.merger.fc2.weight": (H, 4 * VH),
         "visual.merger.fc2.bias": (H,), "lm_head.norm.weight": (H,), "lm_head.weight": (VOCAB, H)}
    for i in range(LAYERS):
        s.update({"layers.%d.%s" % (i, k): v for k, v in _decoder_shapes().items()})
        s.update({"visual.blocks.%d.%s" % (i, k): v for k, v in _vision_shapes().items()})
    return s


def _generator(seed, stream):
    return torch.Generator(device=DEV).manual_seed(1000003 * (int(seed) + 1) + stream)


def _randn(g, *shape, std=1.0):
    return torch.empty(shape, dtype=BF16, device=DEV).normal_(0.0, std, generator=g)


def _weights(shapes, seed):
    """Weights as they are some way into a training: matrices of the usual scale, norms near one, small biases."""
    g = _generator(seed, 1)
    out = {}
    for name, shape in shapes.items():
        last = name.rsplit(".", 1)[-1]
        if last == "A_log":
            w = torch.linspace(1.0, 8.0, shape[0], device=DEV).log().to(BF16)
        elif last == "conv_weight":
            w = _randn(g, *shape, std=0.2)
        elif last == "modulation":
            w = _randn(g, *shape, std=0.1)
        elif len(shape) >= 2:
            w = _randn(g, *shape, std=0.02)
        elif last in ("bias", "dt_bias"):
            w = _randn(g, *shape, std=0.1)
        else:
            w = (1.0 + _randn(g, *shape, std=0.1).float()).to(BF16)
        if "mlp_gate_up" in name:
            w[VFFN:VFFN_PAD] = 0
            w[VFFN_PAD + VFFN:] = 0
        elif name.endswith("mlp_down.weight"):
            w[:, VFFN:] = 0
        out[name] = w
    return out


def _load(make, weights, train):
    with torch.device("meta"):
        module = make()
    module.load_state_dict(weights, assign=True)
    return module.requires_grad_(train)


def _cu(lens):
    return torch.tensor([0] + list(lens), device=DEV).cumsum(0).to(torch.int32)


def _text_rope(docs, dtype=BF16):
    pos = torch.cat([torch.arange(n, device=DEV) for n in docs]).double()
    inv = 1e6 ** (-torch.arange(0, HD // 2, device=DEV).double() / (HD // 2))
    f = torch.outer(pos, inv)
    f = torch.cat([f, f], -1)
    return f.cos().to(dtype), f.sin().to(dtype)


def _patches(images):
    """Row, column, window and image number of every patch, patches in the tower's input order (2 x 2 merge blocks)."""
    rows, cols, wins, which = [], [], [], []
    n_win = 0
    for i, (h, w) in enumerate(images):
        r = torch.arange(h).view(h, 1).expand(h, w)
        c = torch.arange(w).view(1, w).expand(h, w)
        r, c = (t.reshape(h // 2, 2, w // 2, 2).permute(0, 2, 1, 3).reshape(-1) for t in (r, c))
        across = -(-w // 8)
        rows.append(r), cols.append(c), which.append(torch.full((h * w,), i))
        wins.append(n_win + (r // 8) * across + c // 8)
        n_win += -(-h // 8) * across
    return (torch.cat(t).to(DEV) for t in (rows, cols, wins, which))


def _vision_rope(rows, cols, dtype):
    inv = 10000.0 ** (-torch.arange(0, VD // 2, 2, device=DEV).double() / (VD // 2))
    f = torch.cat([torch.outer(rows.double(), inv), torch.outer(cols.double(), inv)], -1)
    f = torch.cat([f, f], -1)
    return f.cos().to(dtype), f.sin().to(dtype)


def _video_rope(grid, dtype=torch.float32):
    f, h, w = grid
    parts = []
    for n, dim, shape in ((f, 44, (f, 1, 1)), (h, 42, (1, h, 1)), (w, 42, (1, 1, w))):
        a = torch.outer(torch.arange(n, device=DEV).double(), 1e4 ** (-torch.arange(0, dim, 2, device=DEV).double() / dim))
        parts.append(a.view(*shape, -1).expand(f, h, w, -1))
    a = torch.cat(parts, -1).reshape(f * h * w, -1)
    return a.cos().to(dtype), a.sin().to(dtype)


def _prompt(case, seed):
    """Token ids and pixels of a prompt: one image, then text."""
    (h, w), = _images(case["image"])
    g = torch.Generator().manual_seed(int(seed) + 77)
    n = h * w // 4
    ids = torch.cat([torch.randint(0, 150000, (5,), generator=g), torch.tensor([151652]), torch.full((n,), 151655),
                     torch.tensor([151653]), torch.randint(0, 150000, (case["text"],), generator=g)])
    return ids, torch.randn(h * w, 1176, generator=g).to(BF16), (h, w)


def _cache(case, seed):
    g = _generator(seed, 2)
    return [dict(k=_randn(g, case["context"], NKV, HD), v=_randn(g, case["context"], NKV, HD)) for _ in range(LAYERS)]


def _token(seed):
    return torch.randint(0, 150000, (1,), generator=torch.Generator().manual_seed(int(seed) + 77)).to(DEV)


def _inputs(case, seed):
    """The tensors of a training or sampling case."""
    g, kind = _generator(seed, 3), case["kind"]
    if kind == "text":
        docs = _ints(case["docs"])
        t = dict(x=_randn(g, sum(docs), H), dy=_randn(g, sum(docs), H), docs=docs)
        t["cos"], t["sin"] = _text_rope(docs)
    elif kind == "vision":
        rows, cols, wins, which = _patches(_images(case["images"]))
        # a block sees its patches in window order, images one after the other
        order = torch.argsort(wins, stable=True)
        seg = (which if case["full"] else wins)[order]
        t = dict(x=_randn(g, len(seg), VH), dy=_randn(g, len(seg), VH), docs=torch.unique_consecutive(seg, return_counts=True)[1].tolist())
        t["cos"], t["sin"] = _vision_rope(rows[order], cols[order], BF16)
    elif kind == "loss":
        T = case["tokens"]
        labels = torch.randint(0, VOCAB, (T,), device=DEV, generator=g)
        labels[torch.rand(T, device=DEV, generator=g) < 0.3] = -100          # prompt and image positions
        labels[0] = 17                                                       # at least one target
        t = dict(x=_randn(g, T, H), labels=labels)
    elif kind == "experts":
        T = case["tokens"]
        logits = torch.randn(T, EXPERTS, device=DEV, generator=g) + 0.7 * torch.randn(EXPERTS, device=DEV, generator=g)
        p, ids = torch.softmax(logits, -1).topk(TOPK, -1)
        t = dict(x=_randn(g, T, EH), ids=ids, probs=(p / p.sum(-1, keepdim=True)).to(BF16), dy=_randn(g, T, EH))
    elif kind == "delta":
        docs = _ints(case["docs"])
        t = dict(x=_randn(g, sum(docs), GH), dy=_randn(g, sum(docs), GH), docs=docs)
    else:
        h, grid = WAN[case["model"]][0], _ints(case["grid"], "x")
        S = grid[0] * grid[1] * grid[2]
        t = dict(x=_randn(g, 1, S, h), dy=_randn(g, 1, S, h) if case["train"] else None, time=_randn(g, 1, 6, h, std=0.3), ctx=_randn(g, 1, TEXT_LEN, h))
        t["cos"], t["sin"] = _video_rope(grid)
    return t


def _shapes(case):
    kind = case["kind"]
    return {"text": _decoder_shapes, "vision": _vision_shapes, "loss": _loss_shapes, "experts": _expert_shapes,
            "delta": _delta_shapes}[kind]() if kind != "video" else _video_shapes(case["model"])


def _config():
    return Qwen25VLConfig(vision=VisionConfig(depth=LAYERS, fullatt_block_indexes=(LAYERS - 1,)), text=TextConfig(num_layers=LAYERS))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        cfg = _config()
        model = _load(lambda: Qwen25VLModel(cfg), _weights(_model_shapes(), seed), False)
        if kind == "decode":
            batch = dict(input_ids=_token(seed), position_ids=torch.full((3, 1), case["context"], dtype=torch.long, device=DEV))
            return dict(kind=kind, model=model, batch=batch, cache=_cache(case, seed))
        ids, pixels, (h, w) = _prompt(case, seed)
        sample = dict(input_ids=ids, labels=ids.clone(), pixel_values=pixels, image_grid_thw=torch.tensor([[1, h, w]]))
        batch = PackedVLMCollator.for_config(cfg)([sample])
        batch.pop("labels")
        move = lambda v: v.to(DEV) if isinstance(v, torch.Tensor) else v  # noqa: E731
        batch = {k: {n: move(x) for n, x in v.items()} if isinstance(v, dict) else move(v) for k, v in batch.items()}
        return dict(kind=kind, model=model, batch=batch, cache=[dict() for _ in range(LAYERS)])
    train = case.get("train", True)
    make = {"text": lambda: DecoderLayer(TextConfig()), "vision": lambda: VisionBlock(VisionConfig()), "loss": lambda: LMHead(TextConfig()),
            "experts": lambda: FusedExperts(MoETextConfig(hidden_size=EH, num_attention_heads=32, num_key_value_heads=4)),
            "delta": lambda: GatedDeltaNet(Qwen35Config.qwen3_5_9b().text),
            "video": lambda: WanBlock(WanConfig.wan2_1_14b() if case["model"] == "14B" else WanConfig.wan2_1_1_3b())}[kind]
    state = _inputs(case, seed)
    state.update(kind=kind, train=train, module=_load(make, _weights(_shapes(case), seed), train))
    if "docs" in state:
        state["cu"], state["longest"] = _cu(state["docs"]), max(state["docs"])
    for name in ("x", "probs", "time", "ctx"):
        if name in state:
            state[name].requires_grad_(train)
    return state


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    s, kind = state, state["kind"]
    if kind in ("decode", "prefill"):
        cache = [dict(c) for c in s["cache"]]
        with torch.no_grad():
            logits = s["model"](s["batch"], kv_cache=cache)
        return dict(logits=logits, k=[c["k"] for c in cache], v=[c["v"] for c in cache])
    m = s["module"]
    if kind in ("text", "vision"):
        out = m(s["x"], s["cos"], s["sin"], s["cu"], s["longest"])
    elif kind == "loss":
        total, count = m(s["x"], s["labels"])
        out = total / count
    elif kind == "experts":
        out = m(s["x"], s["ids"], s["probs"])
    elif kind == "delta":
        out = m(s["x"], s["cu"])
    elif s["train"]:
        out = m(s["x"], s["time"], s["ctx"], s["cos"], s["sin"])
    else:
        with torch.no_grad():
            return m(s["x"], s["time"], s["ctx"], s["cos"], s["sin"])
    names = [n for n in ("x", "probs", "time", "ctx") if n in s]
    params = dict(m.named_parameters())
    grads = torch.autograd.grad(out, [s[n] for n in names] + list(params.values()), s.get("dy"))
    return dict(out=out.detach(), **{"d_" + n: g for n, g in zip(names + list(params), grads)})


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _size(shapes):
    return sum(math.prod(s) for s in shapes.values())


def _matrices(shapes):
    return sum(math.prod(s) for n, s in shapes.items() if len(s) == 2 and "conv" not in n)


def work(case):
    """Multiply-adds of the products (2 flops each; a training step makes three of every forward product) and attention
    (causal pairs counted once; five products in its backward against two), inputs and outputs moved once in bf16."""
    kind = case["kind"]
    dec, vis = _decoder_shapes(), _vision_shapes()
    if kind == "decode":
        n = LAYERS * _size(dec) + VOCAB * H
        kv = LAYERS * 2 * NKV * HD * case["context"]
        return dict(bytes=2.0 * (n + 2 * kv), flops=2.0 * n + 4.0 * LAYERS * NQ * HD * case["context"])
    if kind == "prefill":
        (h, w), = _images(case["image"])
        P, T = h * w, h * w // 4 + case["text"] + 7
        wins = P * 64
        flops = 2.0 * LAYERS * (P * _matrices(vis) + T * _matrices(dec)) + 2.0 * (P * VH * 1176 + P // 4 * 4 * VH * (4 * VH + H) + VOCAB * H)
        flops += 4.0 * VH * ((LAYERS - 1) * wins + P * P) + 2.0 * LAYERS * NQ * HD * T * T
        n = LAYERS * (_size(dec) + _size(vis)) + VOCAB * H + VH * 1176 + 4 * VH * (4 * VH + H)
        return dict(bytes=2.0 * (n + P * 1176 + T * H + LAYERS * 2 * NKV * HD * T), flops=flops)
    shapes = _shapes(case)
    if kind in ("text", "vision"):
        T = sum(_ints(case["docs"])) if kind == "text" else sum(h * w for h, w in _images(case["images"]))
        if kind == "text":
            att = sum(n * (n + 1) / 2 for n in _ints(case["docs"])) * NQ * HD
        elif case["full"]:
            att = sum((h * w) ** 2 for h, w in _images(case["images"])) * VH
        else:
            att = T * 64 * VH
        width = H if kind == "text" else VH
        return dict(bytes=2.0 * (2 * _size(shapes) + 4 * T * width), flops=6.0 * T * _matrices(shapes) + 14.0 * att)
    if kind == "loss":
        T = case["tokens"]
        return dict(bytes=2.0 * (2 * VOCAB * H + 2 * T * H), flops=6.0 * T * VOCAB * H)
    if kind == "experts":
        T = case["tokens"]
        return dict(bytes=2.0 * (2 * _size(shapes) + 4 * T * EH), flops=18.0 * T * TOPK * EH * EF)
    if kind == "delta":
        T = sum(_ints(case["docs"]))
        # state walk: two products with the 128 x 128 state per token and head
        return dict(bytes=2.0 * (2 * _size(shapes) + 4 * T * GH), flops=6.0 * T * _matrices(shapes) + 12.0 * T * GHV * GD * GD)
    h, f, _ = WAN[case["model"]]
    g = _ints(case["grid"], "x")
    S = g[0] * g[1] * g[2]
    lin = S * (3 * h * h + 3 * h * h + 2 * h * f) + TEXT_LEN * 2 * h * h
    att = h * S * (S + TEXT_LEN)
    if case["train"]:
        return dict(bytes=2.0 * (2 * _size(shapes) + 4 * S * h + 2 * TEXT_LEN * h), flops=6.0 * lin + 14.0 * att)
    return dict(bytes=2.0 * (_size(shapes) + 2 * S * h + TEXT_LEN * h), flops=2.0 * lin + 4.0 * att)


def tolerance(case):
    """bf16 operands and results with fp32 sums; the model cases pass their error on from layer to layer."""
    return {"rel": {"decode": 0.08, "prefill": 0.08, "text": 0.04, "video": 0.04, "delta": 0.04}.get(case["kind"], 0.02)}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


def _ln(x):
    x = x - x.mean(-1, keepdim=True)
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS)


def _rotate(x, cos, sin):
    a, b = x.chunk(2, -1)
    return x * cos[:, None] + torch.cat([-b, a], -1) * sin[:, None]


def _rotate_pairs(x, cos, sin):
    a, b = x[..., 0::2], x[..., 1::2]
    c, s = cos[:, None], sin[:, None]
    return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)


def _attend(q, k, v, causal=False):
    """One segment: q [S, N, D], k / v [L, M, D]; the last query sees the last key.  A head and 4096 queries at a time."""
    S, N, D = q.shape
    L, M = k.shape[0], k.shape[1]
    heads = []
    for n in range(N):
        kk, vv, parts = k[:, n * M // N], v[:, n * M // N], []
        for a in range(0, S, 4096):
            s = q[a:a + 4096, n] @ kk.t() / math.sqrt(D)
            if causal:
                i = torch.arange(a, a + s.shape[0], device=q.device)[:, None] + L - S
                s = s.masked_fill(torch.arange(L, device=q.device)[None] > i, float("-inf"))
            parts.append(torch.softmax(s, -1) @ vv)
        heads.append(torch.cat(parts))
    return torch.stack(heads, 1)


def _attend_docs(q, k, v, docs, causal):
    if len(set(docs)) <= 3 and len(docs) > 3 and max(docs) <= 256:         # many short segments: batches of equal length
        out = torch.empty_like(q)
        starts, a = [], 0
        for n in docs:
            starts.append(a)
            a += n
        index = [torch.cat([torch.arange(s, s + n, device=q.device) for s, m in zip(starts, docs) if m == n]) for n in sorted(set(docs))]
        for n, i in zip(sorted(set(docs)), index):
            qq, kk, vv = (t[i].view(-1, n, t.shape[1], t.shape[2]).transpose(1, 2) for t in (q, k, v))
            o = torch.softmax(qq @ kk.transpose(-1, -2) / math.sqrt(q.shape[-1]), -1) @ vv
            out = out.index_copy(0, i, o.transpose(1, 2).reshape(-1, q.shape[1], q.shape[2]))
        return out
    return torch.cat([_attend(*t, causal) for t in zip(q.split(docs), k.split(docs), v.split(docs))])


def _decoder(w, x, cos, sin, docs, cache=None):
    T = x.shape[0]
    q, k, v = F.linear(_rms(x, w["input_layernorm.weight"]), w["qkv_proj.weight"], w["qkv_proj.bias"]).view(T, -1, HD).split([NQ, NKV, NKV], 1)
    q, k = _rotate(q, cos, sin), _rotate(k, cos, sin)
    if cache is not None:
        if "k" in cache:
            k, v = torch.cat([cache["k"].double(), k]), torch.cat([cache["v"].double(), v])
        cache["k"], cache["v"] = k, v
        o = _attend(q, k, v, True)
    else:
        o = _attend_docs(q, k, v, docs, True)
    x = x + o.reshape(T, -1) @ w["o_proj.weight"].t()
    g, u = (_rms(x, w["post_attention_layernorm.weight"]) @ w["gate_up_proj.weight"].t()).chunk(2, -1)
    return x + (F.silu(g) * u) @ w["down_proj.weight"].t()


def _vision(w, x, cos, sin, docs):
    T = x.shape[0]
    q, k, v = F.linear(_rms(x, w["norm1.weight"]), w["attn_qkv.weight"], w["attn_qkv.bias"]).view(T, 3, VN, VD).unbind(1)
    o = _attend_docs(_rotate(q, cos, sin), _rotate(k, cos, sin), v, docs, False)
    x = x + F.linear(o.reshape(T, -1), w["attn_proj.weight"], w["attn_proj.bias"])
    g, u = F.linear(_rms(x, w["norm2.weight"]), w["mlp_gate_up.weight"], w["mlp_gate_up.bias"]).chunk(2, -1)
    return x + F.linear(F.silu(g) * u, w["mlp_down.weight"], w["mlp_down.bias"])


def _delta(w, x, docs):
    T, kd, vd = x.shape[0], GHK * GD, GHV * GD
    qkv, z, b, a = (x @ w["in_proj.weight"].t()).split([2 * kd + vd, vd, GHV, GHV], -1)
    conv = [F.conv1d(F.pad(t.t()[None], (3, 0)), w["conv_weight"][:, None], groups=2 * kd + vd)[0].t() for t in qkv.split(docs)]
    q, k, v = F.silu(torch.cat(conv)).split([kd, kd, vd], -1)
    unit = lambda t: (t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + EPS)).repeat_interleave(GHV // GHK, 1)  # noqa: E731
    q, k, v = unit(q.reshape(T, GHK, GD)) / math.sqrt(GD), unit(k.reshape(T, GHK, GD)), v.reshape(T, GHV, GD)
    beta, gate = torch.sigmoid(b), -torch.exp(w["A_log"]) * F.softplus(a + w["dt_bias"])
    o = torch.cat([_delta_rule(*t) for t in zip(*(u.split(docs) for u in (q, k, v, gate, beta)))])
    return (_rms(o, w["norm_weight"]) * F.silu(z.reshape(T, GHV, GD))).reshape(T, vd) @ w["out_proj.weight"].t()


def _delta_rule(q, k, v, gate, beta, C=64):
    """``S_t = exp(g_t) S_(t-1) + k_t (beta_t (v_t - exp(g_t) S_(t-1)^T k_t))^T``, ``o_t = S_t^T q_t``, C tokens at a time."""
    T, N = q.shape[0], q.shape[1]
    pad = (-T) % C
    q, k, v, gate, beta = (F.pad(t.transpose(0, 1), (0, 0, 0, pad) if t.dim() == 3 else (0, pad)).unflatten(1, (-1, C)) for t in (q, k, v, gate, beta))
    G = gate.cumsum(-1)
    decay = torch.exp((G[..., :, None] - G[..., None, :]).tril()).tril()
    eye = torch.eye(C, dtype=q.dtype, device=q.device)
    A = (beta[..., None] * (k @ k.mT) * decay).tril(-1)
    u, wk = torch.linalg.solve_triangular(eye + A, torch.cat([beta[..., None] * v, (beta * G.exp())[..., None] * k], -1), upper=False,
                                          unitriangular=True).split(GD, -1)
    qs, ks, at = q * G.exp()[..., None], k * (G[..., -1:] - G).exp()[..., None], (q @ k.mT) * decay
    S, out = q.new_zeros(N, GD, GD), []
    for c in range(q.shape[1]):
        new = u[:, c] - wk[:, c] @ S
        out.append(qs[:, c] @ S + at[:, c] @ new)
        S = S * G[:, c, -1].exp()[:, None, None] + ks[:, c].mT @ new
    return torch.cat(out, 1)[:, :T].transpose(0, 1)


def _video(w, x, time, ctx, cos, sin, heads):
    lin = lambda n, t: F.linear(t, w[n + ".weight"], w[n + ".bias"])  # noqa: E731
    x, ctx, (_, S, h) = x[0], ctx[0], x.shape
    e = (w["modulation"] + time)[0]
    q, k, v = lin("self_attn.qkv", _ln(x) * (1 + e[1]) + e[0]).split(h, -1)
    q, k = _rms(q, w["self_attn.q_norm.weight"]), _rms(k, w["self_attn.k_norm.weight"])
    q, k = (_rotate_pairs(t.view(S, heads, -1), cos, sin) for t in (q, k))
    x = x + e[2] * lin("self_attn.proj_out", _attend(q, k, v.view(S, heads, -1)).reshape(S, h))
    del q, k, v
    q = _rms(lin("cross_attn.proj_q", _ln(x) * w["norm3.weight"] + w["norm3.bias"]), w["cross_attn.q_norm.weight"])
    k, v = lin("cross_attn.kv", ctx).split(h, -1)
    k = _rms(k, w["cross_attn.k_norm.weight"])
    x = x + lin("cross_attn.proj_out", _attend(*(t.reshape(-1, heads, h // heads) for t in (q, k, v))).reshape(S, h))
    y = lin("ffn_2", F.gelu(lin("ffn_0", _ln(x) * (1 + e[4]) + e[3]), approximate="tanh"))
    return (x + e[5] * y)[None]


def _model(case, seed):
    """Logits of the last token and the caches; a layer's weights are widened when it runs."""
    w = _weights(_model_shapes(), seed)
    part = lambda p: {k[len(p):]: v.double() for k, v in w.items() if k.startswith(p)}  # noqa: E731
    embed = w["embed_tokens.weight"]
    half = torch.arange(HD // 2, device=DEV)
    inv = 1e6 ** (-half.double() / (HD // 2))
    if case["kind"] == "decode":
        x, cache = embed[_token(seed)].double(), _cache(case, seed)
        pos = torch.full((3, 1), float(case["context"]), device=DEV, dtype=torch.double)
    else:
        ids, pixels, (h, wd) = _prompt(case, seed)
        x, cache = embed[ids.to(DEV)].double(), [dict() for _ in range(LAYERS)]
        rows, cols, wins, which = _patches([(h, wd)])
        order = torch.argsort(wins, stable=True)
        docs = torch.unique_consecutive(wins[order], return_counts=True)[1].tolist()
        cos, sin = _vision_rope(rows[order], cols[order], torch.double)
        p = (pixels.to(DEV).double() @ w["visual.patch_embed.proj.weight"].double().t())[order]
        for i in range(LAYERS):
            p = _vision(part("visual.blocks.%d." % i), p, cos, sin, [h * wd] if i == LAYERS - 1 else docs)
        m = part("visual.merger.")
        p = _rms(p[torch.argsort(order)], m["ln_q.weight"]).view(-1, 4 * VH)
        x[(ids == 151655).to(DEV)] = F.linear(F.gelu(F.linear(p, m["fc1.weight"], m["fc1.bias"])), m["fc2.weight"], m["fc2.bias"])
        # rotary positions: text counts up; the image's tokens keep its start in time and add their row and column
        n, mh, mw = h * wd // 4, h // 2, wd // 2
        img = torch.stack([torch.zeros(n), torch.arange(mh).repeat_interleave(mw).float(), torch.arange(mw).repeat(mh).float()]) + 6
        rest = torch.arange(case["text"] + 1).float() + 6 + max(mh, mw)
        pos = torch.cat([torch.arange(6).float().expand(3, -1), img, rest.expand(3, -1)], 1).to(DEV).double()
    axis = (half >= 16).long() + (half >= 40).long()
    f = pos[axis].t() * inv
    f = torch.cat([f, f], -1)
    for i in range(LAYERS):
        x = _decoder(part("layers.%d." % i), x, f.cos(), f.sin(), None, cache[i])
    x = _rms(x[-1:], w["lm_head.norm.weight"].double())
    logits = torch.cat([x @ t.double().t() for t in w["lm_head.weight"].split(16384)], -1)
    return dict(logits=logits, k=[c["k"] for c in cache], v=[c["v"] for c in cache])


def _loss(t, w):
    """Loss and gradients by the softmax formula, 1024 tokens at a time."""
    x, labels, weight = t["x"].double().requires_grad_(), t["labels"], w["weight"]
    norm = w["norm.weight"].requires_grad_()
    hid = _rms(x, norm)
    valid = labels != -100
    count = valid.sum()
    loss, dh, dw = 0.0, torch.zeros_like(hid), torch.zeros_like(weight)
    with torch.no_grad():
        for a in range(0, x.shape[0], 1024):
            hs, lab, ok = hid[a:a + 1024], labels[a:a + 1024].clamp(min=0), valid[a:a + 1024]
            z = torch.log_softmax(hs @ weight.t(), -1)
            loss = loss - (z.gather(1, lab[:, None])[:, 0] * ok).sum()
            z = z.exp_()
            z.scatter_add_(1, lab[:, None], -torch.ones_like(z[:, :1]))
            z *= ok[:, None] / count
            dh[a:a + 1024] = z @ weight
            dw += z.t() @ hs
    dx, dn = torch.autograd.grad(hid, [x, norm], dh)
    return {"out": loss / count, "d_x": dx, "d_norm.weight": dn, "d_weight": dw}


def _experts(x, ids, probs, w):
    out = torch.zeros_like(x)
    for e in range(EXPERTS):
        tok, slot = (ids == e).nonzero(as_tuple=True)
        if len(tok):
            g, u = (x[tok] @ w["gate_up_proj"][e]).chunk(2, -1)
            out = out.index_add(0, tok, probs[tok, slot, None] * ((F.silu(g) * u) @ w["down_proj"][e]))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        with torch.no_grad():
            return _model(case, seed)
    t = _inputs(case, seed)
    w = {k: v.double() for k, v in _weights(_shapes(case), seed).items()}
    if kind == "loss":
        return _loss(t, w)
    names = [n for n in ("x", "probs", "time", "ctx") if n in t]
    train = case.get("train", True)
    leaf = {n: t[n].double().requires_grad_(train) for n in names}
    w = {k: v.requires_grad_(train) for k, v in w.items()}
    with torch.set_grad_enabled(train):
        if kind in ("text", "vision"):
            fn = _decoder if kind == "text" else _vision
            out = fn(w, leaf["x"], t["cos"].double(), t["sin"].double(), t["docs"])
        elif kind == "experts":
            out = _experts(leaf["x"], t["ids"], leaf["probs"], w)
        elif kind == "delta":
            out = _delta(w, leaf["x"], t["docs"])
        else:
            out = _video(w, leaf["x"], leaf["time"], leaf["ctx"], t["cos"].double(), t["sin"].double(), WAN[case["model"]][2])
        if not train:
            return out
        grads = torch.autograd.grad(out, list(leaf.values()) + list(w.values()), t["dy"].double())
    return dict(out=out.detach(), **{"d_" + n: g for n, g in zip(names + list(w), grads)})
