"""The work that users have this engine do, as measurable cases: one engine step through the executor that the scheduler drives
(`HybridExecutor.prefill` / `decode`) for every model family, and one image through the vision tower.

A decode pass is one step of `streams` sequences at their context, `width` rows each (a drafted block behind the last committed
token where the model drafts).  A prefill pass is one portion of `rows` prompt tokens behind `past` tokens of the same prompt, of
several prompts packed together where `seqs` is above one.  Weights are random and belong to the process, as in a running engine;
a state owns its caches, its slots and the programs of its shapes; tokens, image and everything that follows from them are made
from the seed.  A step may be repeated on the same state: it writes the same cache rows again and carries the recurrent states on.

Models are the built-in descriptions.  The 27B-class hybrid decoder and its mixture-of-experts relative repeat their layers 64 and
48 times; here they have 16 and 8 of them, at full width, which leaves a layer's share of a step what it is within a few percent.
"""
from __future__ import annotations

import dataclasses
import functools
import math
import random
import zlib

import torch

from saber_engine_b200.models import config as C
from saber_engine_b200.models import stack_weights as SW
from saber_engine_b200.models import weights as HW
from saber_engine_b200.models.hybrid import HybridModel
from saber_engine_b200.models.stack import StackModel
from saber_engine_b200.ops.functional import QuantWeight
from saber_engine_b200.runtime.hybrid_executor import HybridExecutor
from saber_engine_b200.sched.executor import SeqRun
from saber_engine_b200.vision.tower import VisionConfig, VisionWeights
from saber_engine_b200.vision.tower_gpu import VisionTowerGPU

RUNGS = (128, 512, 2048)          # prefill row counts that programs exist for
HYBRID_LAYERS, MOE_LAYERS = 16, 8
F64 = torch.float64


# ------------------------------------------------------------------------------------ the cases
def listed() -> list:
    decode = lambda name, model, streams, width, ctx: dict(name=name, do="decode", model=model, streams=streams, width=width, ctx=ctx)   # noqa: E731
    prefill = lambda name, model, rows, past, seqs=1: dict(name=name, do="prefill", model=model, rows=rows, past=past, seqs=seqs)          # noqa: E731
    return [
        # one chat user: a drafted block verified per step, short context; latency per token
        decode("hybrid_decode_single", "qwen38-27b", 1, 8, 700),
        # the engine's headline: eight chats at 4k, each with its own length
        decode("hybrid_decode_eight", "qwen38-27b", 8, 8, 4096),
        # a short question: time to the first token
        prefill("hybrid_prefill_short", "qwen38-27b", 389, 0),
        # a long document: one full portion behind an earlier one
        prefill("hybrid_prefill_long", "qwen38-27b", 2048, 2048),
        # many small chats on the mixture of 512 experts, one row each (it serves up to 32 at once)
        decode("experts_decode_batch", "flashnext-moe", 32, 1, 500),
        # fp32-stream decoders: document portions, packed prompts of several users, chats
        prefill("renosun_prefill_long", "renosun-4k", 2048, 2048),
        decode("renosun_decode_eight", "renosun-4k", 8, 1, 4096),
        prefill("tepavik_prefill_packed", "tepavik-4k", 1500, 0, 5),
        prefill("sofunex_prefill_long", "sofunex-4k", 2048, 2048),
        decode("fitatar_decode_eight", "fitatar-4k", 8, 1, 4096),
        # a thumbnail with odd sides, and a photograph of one megapixel
        dict(name="vision_thumbnail", do="vision", height=14, width=22),
        dict(name="vision_photo", do="vision", height=64, width=64),
    ]


def draw(rng: random.Random) -> dict:
    span = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))      # noqa: E731
    what = rng.choice(("hybrid_decode", "hybrid_prefill", "experts_decode", "stack_prefill", "stack_prefill", "stack_decode", "vision"))
    stack = rng.choice(("renosun", "tepavik", "fitatar", "sofunex")) + rng.choice(("-2k", "-4k"))
    if what == "hybrid_decode":
        return dict(do="decode", model="qwen38-27b", streams=rng.randint(1, 8), width=rng.choice((1, 5, 8)), ctx=span(60, 4096))
    if what == "hybrid_prefill":
        return dict(do="prefill", model="qwen38-27b", rows=span(20, 2048), past=rng.choice((0, span(64, 2048))), seqs=1)
    if what == "experts_decode":
        return dict(do="decode", model="flashnext-moe", streams=span(1, 32), width=1, ctx=span(60, 600))
    if what == "stack_prefill":
        rows = span(40, 2048)
        seqs = rng.choice((1, 1, rng.randint(2, 6)))
        return dict(do="prefill", model=stack, rows=rows, past=0 if seqs > 1 else rng.choice((0, span(64, 2048))), seqs=seqs)
    if what == "stack_decode":
        return dict(do="decode", model=stack, streams=rng.randint(1, 8), width=1, ctx=span(60, 4096))
    return dict(do="vision", height=2 * rng.randint(4, 32), width=2 * rng.randint(4, 32))


def description(model: str):
    cfg = C.by_name(model)
    if isinstance(cfg, C.HybridConfig):
        n = MOE_LAYERS if cfg.moe is not None else HYBRID_LAYERS
        return dataclasses.replace(cfg, n_layers=n, w8_linears=tuple(x for x in cfg.w8_linears if int(x.split(".")[1]) < n))
    return cfg


def contexts(case: dict) -> list:
    """Tokens that every sequence has in its caches ahead of the step (chats have different lengths)."""
    if case["do"] == "prefill":
        return [case["past"]] * case["seqs"]
    return [max(case["ctx"] // 2, case["ctx"] - 61 * j) for j in range(case["streams"])]


def portions(case: dict) -> list:
    """Rows of every sequence of the step."""
    if case["do"] == "decode":
        return [case["width"]] * case["streams"]
    n, left, out = case["seqs"], case["rows"], []
    for j in range(n - 1):                             # later prompts are longer; a single token may stand among them
        out.append(max(1, case["rows"] * (j + 1) * 2 // (n * (n + 1)) - 13 * (j % 2)))
        left -= out[-1]
    return out + [left]


def committed(case: dict, cfg) -> int:
    """Rows of the step before that were committed (models that draft carry them into their states in this step)."""
    return min(4, case["width"]) if case["do"] == "decode" and isinstance(cfg, C.HybridConfig) else 0


def token_lists(case: dict, cfg, seed: int) -> list:
    """Per sequence: context, committed rows of the step before, rows of the step."""
    rng = random.Random(seed)
    return [[rng.randrange(cfg.vocab) for _ in range(c + committed(case, cfg) + n)] for c, n in zip(contexts(case), portions(case))]


# ------------------------------------------------------------------------------------ weights
def _normal(name: str, shape, std: float) -> torch.Tensor:
    g = torch.Generator(device="cuda").manual_seed(zlib.crc32(name.encode()))
    return torch.randn(*shape, generator=g, device="cuda") * std


def _uniform(name: str, shape, lo: float, hi: float) -> torch.Tensor:
    g = torch.Generator(device="cuda").manual_seed(zlib.crc32(name.encode()))
    return torch.rand(*shape, generator=g, device="cuda") * (hi - lo) + lo


SHARE = 0.05       # a linear that ends a sublayer: a trained model's layer adds a fraction of the stream's size to it, so that what one
                   # layer rounds does not grow through the next ones


def quantised(name: str, shape, bits: int) -> tuple:
    """(whole numbers, scale per row) of a linear: symmetric, the largest value of a row at the end of the range."""
    w = _normal(name, shape, 0.02 * (SHARE if name.endswith((".mixer.out", ".mlp.down")) else 1.0))
    top = 2 ** (bits - 1) - 1
    s = (w.abs().amax(1) / top).clamp_min(1e-12)
    return torch.round(w / s[:, None]).clamp_(-top, top).to(torch.int8), s


def hybrid_shapes(cfg, i: int) -> dict:
    """Linears of a layer: (outputs, inputs)."""
    H, sh = cfg.hidden, C.shard(cfg, 1, 0)
    n_in, k_out = (sh.qkv_n, sh.o_k) if cfg.is_attention_layer(i) else (sh.gdn_in_n, sh.gdn_out_k)
    return {"mixer.in": (n_in, H), "mixer.out": (H, k_out), "mlp.gate_up": (2 * cfg.ffn_inter, H), "mlp.down": (H, cfg.ffn_inter)}


def bits_of(cfg, name: str) -> int:
    return 8 if name in cfg.w8_linears else 4


def hybrid_vectors(cfg, i: int) -> dict:
    p, H = f"layers.{i}.", cfg.hidden
    vec = lambda n, size, std, base=0.0: _normal(p + n, (size,), std) + base      # noqa: E731
    v = dict(in_norm=vec("in_norm", H, 0.1), post_norm=vec("post_norm", H, 0.1))
    if cfg.is_attention_layer(i):
        return dict(v, q_norm=vec("q_norm", cfg.head_dim, 0.1), k_norm=vec("k_norm", cfg.head_dim, 0.1))
    hv = cfg.gdn_v_heads
    return dict(v, conv_w=_normal(p + "conv", (C.shard(cfg, 1, 0).gdn_conv_c, 4), 0.5), A_log=vec("A_log", hv, 0.5), dt_bias=vec("dt_bias", hv, 0.5),
                gdn_norm=vec("gdn_norm", cfg.gdn_head_dim, 0.1, 1.0))


def hybrid_weights(cfg):
    quant = lambda name, shape, bits: QuantWeight.from_int(*quantised(name, shape, bits), bits, "cuda")      # noqa: E731
    layers = []
    for i in range(cfg.n_layers):
        lin = {n: quant(f"layers.{i}.{n}", s, bits_of(cfg, f"layers.{i}.{n}")) for n, s in hybrid_shapes(cfg, i).items()}
        layers.append(HW.LayerWeights("attn" if cfg.is_attention_layer(i) else "gdn", mixer_in=lin["mixer.in"], mixer_out=lin["mixer.out"],
                                      gate_up=lin["mlp.gate_up"], down=lin["mlp.down"], **hybrid_vectors(cfg, i)))
    H, d = cfg.hidden, cfg.drafter
    out = HW.ModelWeights(_normal("embed", (cfg.vocab, H), 1.0).bfloat16(), layers, _normal("final_norm", (H,), 0.1), quant("lm_head", (cfg.vocab, H), 8))
    out.drafter = HW.DrafterWeights(quant("draft.aux", (d.hidden, d.n_taps * H), 4), _normal("draft.pos", (d.block, d.hidden), 0.02).bfloat16())
    for i in range(d.n_layers):
        out.drafter.layers.append(dict(norm=_normal(f"draft.{i}.norm", (d.hidden,), 0.1), gate_up=quant(f"draft.{i}.gate_up", (2 * d.inter, d.hidden), 4),
                                       down=quant(f"draft.{i}.down", (d.hidden, d.inter), 4)))
    out.drafter.final_norm, out.drafter.head = _normal("draft.final_norm", (d.hidden,), 0.1), quant("draft.head", (cfg.vocab, d.hidden), d.head_bits)
    return out


ROUTED = 64        # coordinates of the stream that routers read and no layer writes: which experts a token meets then depends on the
                   # token alone, so that two correct implementations choose alike however they round


def stack_tensor(cfg, name: str, shape) -> torch.Tensor:
    leaf = name.rsplit(".", 1)[-1]
    mixed = any(type(l.mlp).__name__ == "ExpertMix" for l in cfg.layers)
    if leaf in ("norm", "norm1", "norm2", "norm1b", "norm2b"):
        t = _normal(name, shape, 0.1) + (1.0 if ".mix." in name else 1.0 - cfg.norm_offset)
    elif leaf in ("D", "sink"):
        t = _normal(name, shape, 0.1) + 1.0
    elif leaf == "b":
        t = _normal(name, shape, 0.05)
    elif leaf == "correction":
        t = torch.zeros(*shape, device="cuda")
    elif leaf == "shift":
        t = _uniform(name, shape, 0.0, 1.0)
    elif leaf == "w0":
        t = _uniform(name, shape, -7.0, -1.0)
    elif leaf == "A_log":
        t = torch.log(_uniform(name, shape, 1.0, 16.0))
    elif leaf == "dt_bias":
        t = torch.log(torch.expm1(torch.exp(_uniform(name, shape, math.log(1e-3), math.log(1e-1)))))
    else:
        t = _normal(name, shape, 0.02 if name in ("embed", "loop.step") else shape[-1] ** -0.5)
    if mixed:
        if name.endswith(".router"):
            t[:, : shape[1] - ROUTED] = 0
            t *= (shape[1] / ROUTED) ** 0.5
        elif name == "loop.step":
            t[:, shape[1] - ROUTED:] = 0
        elif leaf in ("o", "down"):
            t[shape[0] - ROUTED:] = 0
        elif name.endswith((".o.b", ".down.b")):
            t[shape[0] - ROUTED:] = 0
    return t.bfloat16()


def stack_get(cfg):
    shapes = SW.tensor_shapes(cfg)
    return lambda name: stack_tensor(cfg, name, shapes[name])


@functools.lru_cache(maxsize=1)
def weights_of(model: str):
    """What a running engine holds: one model's weights."""
    if model == "vision":
        return VisionTowerGPU(VisionConfig.qwen38(), vision_weights(VisionConfig.qwen38()), "cuda")
    cfg = description(model)
    if not isinstance(cfg, C.HybridConfig):
        return SW.build(cfg, stack_get(cfg), torch.bfloat16, "cuda")
    if cfg.moe is None:
        return hybrid_weights(cfg)
    w = HW.random_init(cfg, 1, 0, "cuda", seed=7)
    w.embed.mul_(50)
    for lw in w.layers:
        for end in (lw.mixer_out, lw.moe["down"], lw.moe["shared_down"]):
            end.scale.mul_(SHARE)
    return w


def vision_weights(cfg: VisionConfig) -> VisionWeights:
    W, M4 = cfg.width, cfg.width * cfg.merge ** 2
    mat = lambda n, o, i, s=0.02: _normal(n, (o, i), s).bfloat16()                 # noqa: E731
    vec = lambda n, size, s=0.02, base=0.0: _normal(n, (size,), s) + base         # noqa: E731
    blocks = []
    for i in range(cfg.depth):
        t = dict(ln1_w=vec(f"{i}.ln1_w", W, 0.05, 1.0), ln1_b=vec(f"{i}.ln1_b", W), ln2_w=vec(f"{i}.ln2_w", W, 0.05, 1.0), ln2_b=vec(f"{i}.ln2_b", W))
        for n, o, k in (("qkv", 3 * W, W), ("proj", W, W), ("fc1", cfg.mlp, W), ("fc2", W, cfg.mlp)):
            t[n + "_w"], t[n + "_b"] = mat(f"{i}.{n}", o, k), vec(f"{i}.{n}_b", o)
        blocks.append(t)
    merger = dict(ln_w=vec("m.ln_w", W, 0.05, 1.0), ln_b=vec("m.ln_b", W), fc1_w=mat("m.fc1", M4, M4), fc1_b=vec("m.fc1_b", M4),
                  fc2_w=mat("m.fc2", cfg.out_hidden, M4), fc2_b=vec("m.fc2_b", cfg.out_hidden))
    return VisionWeights(mat("patch", W, cfg.patch_row), vec("patch_b", W), mat("pos", cfg.pos_grid ** 2, W, 0.1), blocks, merger)


# ------------------------------------------------------------------------------------ one pass
def prepare(case: dict, seed: int) -> dict:
    if case["do"] == "vision":
        tower, grids = weights_of("vision"), [(1, case["height"], case["width"])]
        g = torch.Generator().manual_seed(seed)
        rows = case["height"] * case["width"]
        px = torch.rand(rows, tower.cfg.patch_row, generator=g).mul_(2).sub_(1).pin_memory()       # what the image processor leaves: values in [-1, 1]
        tower.forward(torch.zeros_like(px), grids, graph=True)                                       # the server has met images of this shape
        return dict(case=case, tower=tower, px=px, grids=grids)
    cfg = description(case["model"])
    hybrid = isinstance(cfg, C.HybridConfig)
    tokens, ctx, n = token_lists(case, cfg, seed), contexts(case), portions(case)
    seqs, done = len(tokens), committed(case, cfg)
    longest = max(len(t) for t in tokens) + 8
    if hybrid:
        model = HybridModel(cfg, max_seqs=seqs, max_ctx=longest, max_width=8 if cfg.drafter is not None else 1, weights=weights_of(case["model"]),
                            use_drafter=cfg.drafter is not None)
    else:
        model = StackModel(cfg, max_seqs=seqs, max_ctx=longest, weights=weights_of(case["model"]))
    ex = HybridExecutor(model, decode_batches=tuple(range(1, seqs + 1)), decode_widths=(1, 5, 8), prefill_rungs=RUNGS,
                        prefill_pack=seqs if case["do"] == "prefill" else 1)
    per = model.max_blocks
    blocks = [list(range(1 + j * per, 1 + (j + 1) * per)) for j in range(seqs)]

    def run_of(j: int, first: int, count: int, shift: int = 0, last: bool = True) -> SeqRun:
        return SeqRun(j, tokens[j][first:first + count], first, j + 1, shift, blocks[j], uid=j, last_chunk=last, blocks_key=("sequence", j))

    for j in range(seqs):
        model.reset_slot(j + 1)
        for at in range(0, ctx[j], RUNGS[-1]):
            ex.prefill([run_of(j, at, min(RUNGS[-1], ctx[j] - at))])
    if case["do"] == "decode":
        if done:                                        # a step ahead of the measured one: its first rows are committed by the next
            ex.decode([run_of(j, ctx[j], case["width"]) for j in range(seqs)], case["width"])
        runs = [run_of(j, ctx[j] + done, n[j], done) for j in range(seqs)]
        bucket = model.build_bucket("decode", seqs, case["width"])
    else:
        runs = [run_of(j, ctx[j], n[j]) for j in range(seqs)]
        bucket = model.build_bucket("prefill", ex.prefill_pack, next(r for r in RUNGS if r >= sum(n)))
    rows = sum(n) if case["do"] == "decode" else seqs
    out = {"logits": bucket.logits[:rows, : cfg.vocab]}
    state = model.gdn_state if hybrid else model.state
    in_order = lambda d: [d[k] for k in sorted(d, key=lambda k: int(str(k).split(".")[0]))]      # noqa: E731
    out["state"], pages = [s[1:seqs + 1] for s in in_order(state)], in_order(model.kv)
    out["pages"] = [p.view(torch.float8_e4m3fn) for p in pages] if hybrid else pages
    return dict(case=case, ex=ex, runs=runs, out=out)


def run(state: dict):
    """One engine step, or one image.  Committed tokens and drafts are the largest of logits (ties fall either way): the logits, the recurrent
    states and the cache pages stand for them."""
    case = state["case"]
    if case["do"] == "vision":
        return state["tower"].forward(state["px"], state["grids"], graph=True)
    if case["do"] == "decode":
        state["ex"].decode(state["runs"], case["width"])
    else:
        state["ex"].prefill(state["runs"])
    return state["out"]


# ------------------------------------------------------------------------------------ what a pass cannot do without
def _size(shape) -> int:
    return math.prod(shape)


def work(case: dict) -> dict:
    if case["do"] == "vision":
        return vision_work(case)
    cfg, ctx, n = description(case["model"]), contexts(case), portions(case)
    rows, done = sum(n), committed(case, cfg)
    heads = rows if case["do"] == "decode" else len(n)
    first = [c + done for c in ctx]                                     # tokens ahead of the step's rows
    pairs = lambda span: sum(sum(min(f + i + 1, span) for i in range(k)) for f, k in zip(first, n))     # noqa: E731
    seen = lambda span: sum(min(f + k, span + k) for f, k in zip(first, n))                              # noqa: E731
    return (hybrid_work if isinstance(cfg, C.HybridConfig) else stack_work)(cfg, rows, len(n), heads, pairs, seen, done)


def _met(experts: int, top: int, rows: int) -> float:
    return experts * (1 - (1 - top / experts) ** rows)                  # experts that some row chooses, choices alike


def hybrid_work(cfg, rows, seqs, heads, pairs, seen, done) -> dict:
    H, D, m = cfg.hidden, cfg.head_dim, cfg.moe
    by, fl, far = heads * cfg.vocab * 2.0 + cfg.vocab * H, 2.0 * heads * cfg.vocab * H, 1 << 60
    for i in range(cfg.n_layers):
        for name, shape in hybrid_shapes(cfg, i).items():
            if m is None or not name.startswith("mlp"):
                by += _size(shape) * bits_of(cfg, f"layers.{i}.{name}") / 8
                fl += 2.0 * rows * _size(shape)
        if m is not None:
            one = 3 * H * m.expert_inter
            by += 0.5 * one * _met(m.n_experts, m.top_k, rows) + 1.5 * H * m.shared_inter + H * m.n_experts
            fl += 2.0 * rows * (m.top_k * one + 3 * H * m.shared_inter + H * m.n_experts)
        if cfg.is_attention_layer(i):
            by += (seen(far) + rows) * 2.0 * cfg.n_kv_heads * D
            fl += 4.0 * pairs(far) * cfg.n_q_heads * D
        else:
            by += 8.0 * seqs * cfg.gdn_v_heads * cfg.gdn_head_dim ** 2
            fl += 8.0 * (rows + seqs * done) * cfg.gdn_v_heads * cfg.gdn_head_dim ** 2
    d = cfg.drafter
    if d is not None:
        w = d.hidden * d.n_taps * H + d.n_layers * 3 * d.hidden * d.inter + cfg.vocab * d.hidden
        by, fl = by + 0.5 * w, fl + 2.0 * seqs * d.block * (w - d.hidden * d.n_taps * H) + 2.0 * seqs * d.hidden * d.n_taps * H
    return {"bytes": by, "flops": fl}


def stack_work(cfg, rows, seqs, heads, pairs, seen, done) -> dict:
    shapes, far = SW.tensor_shapes(cfg), 1 << 60
    runs = {}
    for r in cfg.runs:
        runs[r.layer] = runs.get(r.layer, 0) + 1
    by, fl = 2.0 * cfg.vocab * cfg.width + 4.0 * heads * cfg.vocab + 2.0 * rows * cfg.width, 2.0 * heads * cfg.vocab * cfg.width
    for name, shape in shapes.items():
        if not name.startswith("l") or len(shape) < 2 or name.endswith(".conv") or name == "loop.step":
            continue
        times = cfg.loop.times if name == "loop.in" else runs[int(name[1:name.index(".")])]
        share, part = 1.0, 1.0
        if ".mlp.e" in name:
            f = cfg.layers[int(name[1:name.index(".")])].mlp
            share, part = _met(f.experts, f.top, rows) / f.experts, f.top / f.experts
        absorbed = name.endswith((".uk", ".uv")) and rows >= 64           # expanded keys and values of every token seen
        by += 2.0 * _size(shape) * share
        fl += 2.0 * (seen(far) if absorbed else rows) * _size(shape) * part * times
    for r in cfg.runs:
        for _, m, _ in cfg.layers[r.layer].mixer.parts():
            kind = type(m).__name__
            if kind == "GroupedMixer":
                span = m.window or m.chunk or far
                by += 2.0 * seen(span) * m.kv_heads * (m.dim + m.vdim)
                fl += 2.0 * pairs(span) * m.heads * (m.dim + m.vdim)
            elif kind == "LatentMixer":
                by += 2.0 * seen(far) * (m.kv_rank + m.rot_dim)
                fl += 2.0 * pairs(far) * m.heads * (m.dim + m.rot_dim + m.vdim if rows >= 64 else 2 * m.kv_rank + m.rot_dim)
            else:
                v = getattr(m, "vdim", m.dim)
                by += 8.0 * seqs * m.heads * m.dim * v
                fl += (4.0 if kind == "OuterMixer" else 8.0) * rows * m.heads * m.dim * v
    return {"bytes": by, "flops": fl}


def vision_work(case: dict) -> dict:
    cfg, L = VisionConfig.qwen38(), case["height"] * case["width"]
    W, M4 = cfg.width, cfg.width * cfg.merge ** 2
    block, merge = 4 * W * W + 2 * W * cfg.mlp, M4 * M4 + M4 * cfg.out_hidden
    by = 2.0 * (cfg.depth * block + merge + W * cfg.patch_row) + L * (4.0 * cfg.patch_row + 0.5 * cfg.out_hidden)
    return {"bytes": by, "flops": 2.0 * L * (cfg.depth * block + W * cfg.patch_row + merge / 4) + 4.0 * cfg.depth * L * L * W}


def tolerance(case: dict) -> dict:
    """Measured against 64 bits: logits are 0.3 to 1.4 % off, recurrent states of deep layers up to 2.8 % (bf16 operands); the hybrid's, whose
    rows are 8 bits wide, 3 and 4 %.  Implementations that round in another place differ by as much from one another."""
    return {"rel": 0.03}


# ------------------------------------------------------------------------------------ the same in 64 bits
def exact(case: dict, seed: int):
    if case["do"] == "vision":
        return vision_exact(case, seed)
    cfg = description(case["model"])
    tokens = token_lists(case, cfg, seed)
    lens, n = [len(t) for t in tokens], portions(case)
    with torch.no_grad():
        if not isinstance(cfg, C.HybridConfig):
            hidden, states = stack_exact(cfg, stack_get(cfg), tokens)
            keep = 1
        elif cfg.moe is not None or sum(lens) > 10000:
            return None      # experts are chosen on rows quantised to 8 bits: a near tie falls either way; or it would take too long
        else:
            hidden, states = hybrid_exact(cfg, tokens, [l - k for l, k in zip(lens, n)] if case["do"] == "decode" else lens)
            keep = n[0] if case["do"] == "decode" else 1
        rows = torch.cat([hidden[j, lens[j] - keep:lens[j]] for j in range(len(tokens))])
        if isinstance(cfg, C.HybridConfig):
            q, s = quantised("lm_head", (cfg.vocab, cfg.hidden), 8)
            logits = torch.cat([rows @ (a.to(F64) * b.to(F64)[:, None]).T for a, b in zip(q.split(1 << 15), s.split(1 << 15))], -1)
            pages = cfg.n_attn_layers
        else:
            head = stack_tensor(cfg, "head", (cfg.vocab, cfg.width))
            logits = torch.cat([rows @ a.to(F64).T for a in head.split(1 << 15)], -1)
            if cfg.logit_cap:
                logits = cfg.logit_cap * torch.tanh(logits / cfg.logit_cap)
            pages = 0
        return {"logits": logits, "state": states, "pages": [None] * pages}


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.nn.functional.softplus(x)


def _padded(tokens: list) -> torch.Tensor:
    """[sequences, longest]: shorter ones end in padding, which nothing before it sees."""
    n = max(len(t) for t in tokens)
    return torch.tensor([t + [0] * (n - len(t)) for t in tokens], device="cuda")


def _conv(x, w):
    """x [B, T, channels], w [channels, taps]: the last tap meets the current token."""
    T, taps = x.shape[1], w.shape[1]
    y = x * w[:, taps - 1]
    for back in range(1, min(taps, T)):
        y[:, back:] += x[:, :T - back] * w[:, taps - 1 - back]
    return y


def _live(lens, T):
    return (torch.arange(T, device="cuda")[None] < torch.tensor(lens, device="cuda")[:, None]).to(F64)


def _recur(decay, keys, values, reads, removal=None, rate=None, lens=None, write=None):
    """S <- decay S [- removal (rate-weighted key' S)] + key value'; o = S' read.  All [B, T, H, ...]; decay [.., 1 or D].
    removal / rate: the delta rule's terms.  Tokens behind a sequence's length leave its state alone.  Returns (o, S [B, H, V, D])."""
    B, T, H, D = keys.shape
    live = _live(lens, T)[..., None, None]
    decay, keys = decay * live + (1 - live), keys * live
    S = torch.zeros(B, H, D, values.shape[-1], dtype=F64, device="cuda")
    out = torch.empty(B, T, H, values.shape[-1], dtype=F64, device="cuda")
    for t in range(T):
        k, v = keys[:, t], values[:, t]
        if write is not None:                          # gated delta rule: decay, correct, write
            S = S * decay[:, t, ..., None]
            u = write[:, t, :, None] * (v - torch.einsum("bhdv,bhd->bhv", S, k))
            S = S + k[..., None] * u[..., None, :]
        elif removal is not None:                      # rates per key channel: both terms read the old state
            held = torch.einsum("bhdv,bhd->bhv", S, removal[:, t] * live[:, t])
            S = S * decay[:, t, ..., None] - (rate[:, t] * removal[:, t])[..., None] * held[..., None, :] + k[..., None] * v[..., None, :]
        else:
            S = S * decay[:, t, ..., None] + k[..., None] * v[..., None, :]
        out[:, t] = torch.einsum("bhdv,bhd->bhv", S, reads[:, t])
    return out, S.transpose(-1, -2)


def _angles(rot, T):
    i = torch.arange(rot.dims // 2, dtype=F64, device="cuda")
    f, amp = rot.base ** (-2 * i / rot.dims), 1.0
    if rot.yarn is None:
        f = f / rot.factor
    else:
        original, fast, slow = rot.yarn
        pair = lambda turns: rot.dims * math.log(original / (2 * math.pi * turns)) / (2 * math.log(rot.base))      # noqa: E731
        lo, hi = max(math.floor(pair(fast)), 0), min(math.ceil(pair(slow)), rot.dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f, amp = f / rot.factor * ramp + f * (1 - ramp), 0.1 * math.log(rot.factor) + 1
    a = torch.arange(T, dtype=F64, device="cuda")[:, None, None] * f
    return amp * torch.cos(a), amp * torch.sin(a)


def _rotate(x, rot):
    """x [B, T, heads, size]"""
    n = rot.dims
    c, s = _angles(rot, x.shape[1])
    a, b = (slice(0, n, 2), slice(1, n, 2)) if rot.interleaved else (slice(0, n // 2), slice(n // 2, n))
    u, v, out = x[..., a], x[..., b], x.clone()
    out[..., a], out[..., b] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, lens, cap=0.0, chunk=0, window=0, sink=None):
    """q [B, T, H, D], k [B, T, G, D], v [B, T, G, V]"""
    out = torch.zeros(*q.shape[:3], v.shape[-1], dtype=F64, device="cuda")
    H, G = q.shape[2], k.shape[2]
    for b, T in enumerate(lens):
        i = torch.arange(T, device="cuda")
        hide = i[None] > i[:, None]
        if chunk:
            hide |= i[None] // chunk != i[:, None] // chunk
        if window:
            hide |= i[:, None] - i[None] >= window
        for h in range(H):
            g = h // (H // G)
            s = q[b, :T, h] @ k[b, :T, g].T * scale
            s = (cap * torch.tanh(s / cap) if cap else s).masked_fill_(hide, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(T, 1)], 1)
            out[b, :T, h] = torch.softmax(s, -1)[:, :T] @ v[b, :T, g]
    return out


def stack_exact(cfg, get, tokens):
    """(normed rows ahead of the head [B, T, width], states of the recurrent runs)"""
    eps, off, lens = cfg.eps, cfg.norm_offset, [len(t) for t in tokens]
    w = lambda name: get(name).to(F64)                                    # noqa: E731
    x = get("embed")[_padded(tokens)].to(F64) * cfg.embed_scale
    x0, states, pages = x, [], {}
    for r in cfg.runs:
        spec, p = cfg.layers[r.layer], f"l{r.layer}."
        if r.enter is not None:
            step = w("loop.step")[r.enter]
            x = torch.cat([x, x0], -1) @ w("loop.in").T + step if cfg.loop_linear else x + step
        h = _rms(x, eps) * (off + w(p + "norm1"))
        if cfg.token_shift:
            before = torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1)
            h = h + (before - h) * w(p + "shift")
        y = 0
        for pre, m, scale in spec.mixer.parts():
            o, s, pages[r.index] = MIXERS[type(m).__name__](h, m, lambda n: w(f"{p}mix.{pre}{n}"), eps, lens, pages.get(m.kv_from))
            if s is not None:
                states.append(s)
            y = y + scale * o
        if cfg.post_norms:
            x = x + cfg.residual_mult * _rms(y, eps) * w(p + "norm1b")
            if spec.mlp is not None:
                h = _rms(x, eps) * w(p + "norm2")
                x = x + cfg.residual_mult * _rms(feed_forward(h, spec.mlp, lambda n: w(f"{p}mlp.{n}")), eps) * w(p + "norm2b")
        elif cfg.parallel:
            if spec.mlp is not None:
                h = _rms(x, eps) * (off + w(p + "norm2")) if cfg.two_norms else h
                y = y + feed_forward(h, spec.mlp, lambda n: w(f"{p}mlp.{n}"))
            x = x + y
        else:
            x = x + y
            if spec.mlp is not None:
                x = x + feed_forward(_rms(x, eps) * (off + w(p + "norm2")), spec.mlp, lambda n: w(f"{p}mlp.{n}"))
    return _rms(x, eps) * (off + w("final.norm")), states


def delta(h, m, w, eps, lens, kv):
    B, T, _ = h.shape
    q, k, v = (_silu(_conv(h @ w(n).T, w(n + ".conv"))) for n in ("q", "k", "v"))
    unit = lambda z: (z / torch.sqrt((z * z).sum(-1, keepdim=True) + m.unit_eps)).repeat_interleave(m.heads // m.kv_heads, 2)      # noqa: E731
    q, k = unit(q.view(B, T, m.kv_heads, m.dim)) * m.dim ** -0.5, unit(k.view(B, T, m.kv_heads, m.dim))
    g = torch.exp(-torch.exp(w("A_log")) * _softplus(h @ w("a").T + w("dt_bias")))
    o, S = _recur(g[..., None], k, v.view(B, T, m.heads, m.vdim), q, lens=lens, write=torch.sigmoid(h @ w("b").T) * _live(lens, T)[..., None])
    o = _rms(o, eps) * w("norm") * _silu(h @ w("g").T).view(B, T, m.heads, m.vdim)
    return o.flatten(2) @ w("o").T, S, None


def channel_delta(h, m, w, eps, lens, kv):
    B, T, _ = h.shape
    split = lambda z: z.view(B, T, m.heads, m.dim)                        # noqa: E731
    r, k, v = (split(h @ w(n).T) for n in ("r", "k", "v"))
    decay = split(torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ w("w1").T) @ w("w2").T + w("w0"))))
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + m.unit_eps)
    o, S = _recur(decay, k, v, r, removal=u, rate=split(torch.sigmoid(h @ w("a").T + w("a.b"))), lens=lens)
    return (_rms(o, eps).flatten(2) * w("norm") * torch.sigmoid(h @ w("g").T)) @ w("o").T, S, None


def outer(h, m, w, eps, lens, kv):
    B, T, _ = h.shape
    inner, kd = m.heads * m.vdim, m.kv_heads * m.dim
    spread = lambda z: z.view(B, T, m.kv_heads, m.dim).repeat_interleave(m.heads // m.kv_heads, 2)      # noqa: E731
    if m.decay is not None:
        q, k, v = (_silu(h @ w(n).T) for n in ("q", "k", "v"))
        o, S = _recur(torch.tensor(m.decay, dtype=F64, device="cuda").expand(B, T, -1)[..., None], spread(k), v.view(B, T, m.heads, m.vdim), spread(q), lens=lens)
        return (_rms(o.flatten(2), eps) * w("norm") * torch.sigmoid(h @ w("g").T)) @ w("o").T, S, None
    z, xbc, dt = torch.split(h @ w("in").T, [inner, inner + 2 * kd, m.heads], -1)
    v, k, q = torch.split(_silu(_conv(xbc, w("conv")) + w("conv.b")), [inner, kd, kd], -1)
    v, dt = v.reshape(B, T, m.heads, m.vdim), _softplus(dt + w("dt_bias"))
    o, S = _recur(torch.exp(-torch.exp(w("A_log")) * dt)[..., None], spread(k.contiguous()), dt[..., None] * v, spread(q.contiguous()), lens=lens)
    o = (o + w("D")[:, None] * v).flatten(2) * _silu(z)
    return (_rms(o.view(B, T, m.norm_groups, -1), eps).flatten(2) * w("norm")) @ w("o").T, S, None


def grouped(h, m, w, eps, lens, kv):
    B, T, _ = h.shape
    split = lambda z: z.view(B, T, -1, m.dim)                             # noqa: E731
    proj = lambda n: h @ w(n).T + (w(n + ".b") if m.bias else 0)          # noqa: E731
    if m.taps:
        q, k, v = (_conv(proj(n), w(n + ".conv")) for n in ("q", "k", "v"))
        q, k, v = split(_rms(q, eps) * w("q.norm")), split(_rms(k, eps) * w("k.norm")), _rms(v.view(B, T, m.kv_heads, m.vdim), eps)
    else:
        q = split(proj("q"))
        q = _rms(q, eps) if m.qk_norm else q
    if m.rot is not None:
        q = _rotate(q, m.rot)
    if kv is None:
        if not m.taps:
            k, v = split(proj("k")), proj("v").view(B, T, m.kv_heads, m.vdim)
            k = _rms(k, eps) if m.qk_norm else k
        kv = (_rotate(k, m.rot) if m.rot is not None else k), v
    o = _attend(q, *kv, m.scale, lens, m.softcap, m.chunk, m.window, w("sink") if m.sink else None).flatten(2)
    o = o * torch.sigmoid(h @ w("g").T) if m.gate else o
    return o @ w("o").T + (w("o.b") if m.out_bias else 0), None, kv


def latent(h, m, w, eps, lens, kv):
    B, T, _ = h.shape
    q = (_rms(h @ w("dq").T, eps) * w("dq.norm")) @ w("uq").T if m.q_rank else h @ w("q").T
    q = q.view(B, T, m.heads, m.dim + m.rot_dim)
    q = torch.cat([q[..., : m.dim], _rotate(q[..., m.dim:], m.rot)], -1)
    if kv is None:
        d = h @ w("dkv").T
        kv = _rms(d[..., : m.kv_rank], eps) * w("dkv.norm"), _rotate(d[..., None, m.kv_rank:], m.rot)
    c, kr = kv
    k = torch.cat([(c @ w("uk").T).view(B, T, m.heads, m.dim), kr.expand(-1, -1, m.heads, -1)], -1)
    o = _attend(q, k, (c @ w("uv").T).view(B, T, m.heads, m.vdim), m.scale, lens)
    gate = torch.sigmoid(h @ w("g").T)
    return (o * (gate[..., None] if m.gate_heads else gate.view_as(o))).flatten(2) @ w("o").T, None, kv


MIXERS = {"DeltaMixer": delta, "ChannelDeltaMixer": channel_delta, "OuterMixer": outer, "GroupedMixer": grouped, "LatentMixer": latent}


def feed_forward(h, f, w):
    kind = type(f).__name__
    if kind == "ClampedGlu":
        g, u = (h @ w("gate").T).clamp(max=f.limit), (h @ w("up").T).clamp(-f.limit, f.limit)
        return (g * torch.sigmoid(f.alpha * g) * (u + 1)) @ w("down").T
    if kind == "SquaredRelu":
        return torch.relu(h @ w("up").T) ** 2 @ w("down").T
    if kind == "Gelu":
        return torch.nn.functional.gelu(h @ w("up").T + w("up.b")) @ w("down").T + w("down.b")
    if kind == "GatedUnit":
        g = h @ w("gate").T
        return ((torch.nn.functional.gelu(g, approximate="tanh") if f.act == "gelu_tanh" else _silu(g)) * (h @ w("up").T)) @ w("down").T
    flat = h.flatten(0, 1)
    s = flat @ w("router").T
    s = torch.sigmoid(s) if f.sigmoid else torch.softmax(s, -1)
    c = s + w("correction") if f.sigmoid else s
    by_group = c.view(len(c), f.groups, -1)
    strength = by_group.topk(2, -1).values.sum(-1) if f.sigmoid else by_group.amax(-1)
    kept = torch.zeros_like(strength).scatter_(1, strength.topk(f.keep, -1).indices, 1.0).bool()
    chosen = by_group.masked_fill(~kept[..., None], -math.inf).flatten(1).topk(f.top, -1).indices
    share = s.gather(1, chosen)
    share = share / share.sum(-1, keepdim=True) * f.scale if f.sigmoid else share
    one = (lambda z, n: (_silu(z @ w(n + "gate").T) * (z @ w(n + "up").T)) @ w(n + "down").T) if f.gated else \
        (lambda z, n: torch.relu(z @ w(n + "up").T) ** 2 @ w(n + "down").T)
    out = torch.zeros_like(flat)
    for e in range(f.experts):
        t, k = (chosen == e).nonzero(as_tuple=True)
        if len(t):
            out[t] += share[t, k, None] * one(flat[t], f"e{e}.")
    if f.shared:
        y = one(flat, "shared.")
        out += y if f.gated else y * torch.sigmoid(flat @ w("shared.sg").T)
    return out.view_as(h)


def hybrid_exact(cfg, tokens, until):
    """The dense hybrid without its 8-bit rows: (normed rows ahead of the head, recurrent states after `until` tokens of each sequence)."""
    eps, lens, D, d = cfg.eps, [len(t) for t in tokens], cfg.head_dim, cfg.gdn_head_dim

    def lin(x, i, n):
        q, s = quantised(f"layers.{i}.{n}", hybrid_shapes(cfg, i)[n], bits_of(cfg, f"layers.{i}.{n}"))
        return x @ (q.to(F64) * s.to(F64)[:, None]).T

    x, states = _normal("embed", (cfg.vocab, cfg.hidden), 1.0).bfloat16()[_padded(tokens)].to(F64), []
    B, T, _ = x.shape
    a = torch.arange(T, dtype=F64, device="cuda")[:, None, None] * cfg.rope_theta ** (-2 * torch.arange(cfg.rot_dim // 2, dtype=F64, device="cuda") / cfg.rot_dim)
    for i in range(cfg.n_layers):
        v = {k: t.to(F64) for k, t in hybrid_vectors(cfg, i).items()}
        y = lin(_rms(x, eps) * (cfg.norm_offset + v["in_norm"]), i, "mixer.in")
        if cfg.is_attention_layer(i):
            nq, nk = cfg.n_q_heads * D, cfg.n_kv_heads * D
            q, g, k, val = torch.split(y, [nq, nq, nk, nk], -1)

            def turned(z, w):
                z = _rms(z.view(B, T, -1, D), eps) * (cfg.norm_offset + w)
                h = cfg.rot_dim // 2
                lo, hi = z[..., :h], z[..., h:2 * h]
                return torch.cat([lo * torch.cos(a) - hi * torch.sin(a), hi * torch.cos(a) + lo * torch.sin(a), z[..., 2 * h:]], -1)
            o = _attend(turned(q, v["q_norm"]), turned(k, v["k_norm"]), val.view(B, T, -1, D), D ** -0.5, lens).flatten(2) * torch.sigmoid(g)
        else:
            nk, nv = cfg.gdn_k_heads * d, cfg.gdn_v_heads * d
            qkv, z, b, al = torch.split(y, [2 * nk + nv, nv, cfg.gdn_v_heads, cfg.gdn_v_heads], -1)
            q, k, val = torch.split(_silu(_conv(qkv, v["conv_w"])), [nk, nk, nv], -1)
            unit = lambda t: (t.reshape(B, T, -1, d) / torch.sqrt((t.reshape(B, T, -1, d) ** 2).sum(-1, keepdim=True) + 1e-6)) \
                .repeat_interleave(cfg.gdn_v_heads // cfg.gdn_k_heads, 2)      # noqa: E731
            dec = torch.exp(-torch.exp(v["A_log"]) * _softplus(al + v["dt_bias"]))[..., None]
            args = dec, unit(k), val.reshape(B, T, -1, d), unit(q) * d ** -0.5
            beta = torch.sigmoid(b)
            o, S = _recur(*args, lens=lens, write=beta * _live(lens, T)[..., None])
            if until != lens:
                n = max(until)
                S = _recur(*(t[:, :n] for t in args), lens=until, write=(beta * _live(until, T)[..., None])[:, :n])[1]
            states.append(S)
            o = (_rms(o, eps) * v["gdn_norm"]).flatten(2) * _silu(z)
        x = x + lin(o, i, "mixer.out")
        g, u = lin(_rms(x, eps) * (cfg.norm_offset + v["post_norm"]), i, "mlp.gate_up").chunk(2, -1)
        x = x + lin(_silu(g) * u, i, "mlp.down")
    return _rms(x, eps) * (cfg.norm_offset + _normal("final_norm", (cfg.hidden,), 0.1).to(F64)), states


def vision_exact(case, seed):
    cfg = VisionConfig.qwen38()
    wts = vision_weights(cfg)
    H, W, m, D = case["height"], case["width"], cfg.merge, cfg.head_dim
    px = torch.rand(H * W, cfg.patch_row, generator=torch.Generator().manual_seed(seed)).mul_(2).sub_(1).cuda().to(F64)
    d = lambda t: t.cuda().to(F64)                                        # noqa: E731
    order = lambda t: t.view(H // m, m, W // m, m, -1).transpose(1, 2).reshape(H * W, -1)      # noqa: E731  (rows of a 2 x 2 neighbourhood follow one another)
    ln = lambda x, a, b: (x - x.mean(-1, keepdim=True)) / torch.sqrt(x.var(-1, unbiased=False, keepdim=True) + cfg.eps) * d(a) + d(b)      # noqa: E731
    table = d(wts.pos_table).view(cfg.pos_grid, cfg.pos_grid, -1)
    at = [torch.linspace(0, cfg.pos_grid - 1, n, dtype=F64, device="cuda") for n in (H, W)]
    lo = [t.floor().long().clamp(max=cfg.pos_grid - 1) for t in at]
    hi = [(t + 1).clamp(max=cfg.pos_grid - 1) for t in lo]
    fy, fx = (at[0] - lo[0])[:, None, None], (at[1] - lo[1])[None, :, None]
    pick = lambda y, x: table[y][:, x]                                    # noqa: E731
    pos = (1 - fy) * ((1 - fx) * pick(lo[0], lo[1]) + fx * pick(lo[0], hi[1])) + fy * ((1 - fx) * pick(hi[0], lo[1]) + fx * pick(hi[0], hi[1]))
    x = px @ d(wts.patch_w).T + d(wts.patch_b) + order(pos)
    inv = cfg.rope_theta ** (-torch.arange(0, D // 2, 2, dtype=F64, device="cuda") / (D // 2))
    y, z = torch.meshgrid(*(torch.arange(n, dtype=F64, device="cuda") for n in (H, W)), indexing="ij")
    a = order(torch.cat([y[..., None] * inv, z[..., None] * inv], -1))[:, None]
    for b in wts.blocks:
        q, k, v = (ln(x, b["ln1_w"], b["ln1_b"]) @ d(b["qkv_w"]).T + d(b["qkv_b"])).view(-1, 3, cfg.heads, D).unbind(1)
        rot = lambda t: torch.cat([t[..., :D // 2] * a.cos() - t[..., D // 2:] * a.sin(), t[..., D // 2:] * a.cos() + t[..., :D // 2] * a.sin()], -1)      # noqa: E731
        q, k = rot(q), rot(k)
        o = torch.stack([torch.softmax(q[:, h] @ k[:, h].T * D ** -0.5, -1) @ v[:, h] for h in range(cfg.heads)], 1)
        x = x + o.flatten(1) @ d(b["proj_w"]).T + d(b["proj_b"])
        f = torch.nn.functional.gelu(ln(x, b["ln2_w"], b["ln2_b"]) @ d(b["fc1_w"]).T + d(b["fc1_b"]), approximate="tanh")
        x = x + f @ d(b["fc2_w"]).T + d(b["fc2_b"])
    g = wts.merger
    y = torch.nn.functional.gelu(ln(x, g["ln_w"], g["ln_b"]).reshape(H * W // m ** 2, -1) @ d(g["fc1_w"]).T + d(g["fc1_b"]))
    return y @ d(g["fc2_w"]).T + d(g["fc2_b"])
