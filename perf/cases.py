"""The work whose time matters to a user of this engine, as cases that can be drawn, run and checked.

Seven kinds of case, each through an entry point that a program calls:

``decode``       ``ModelRunner.step`` with one new token per request (replayed from the step's CUDA graph): what every
                 generated token costs, from one request, where latency and launches count, to a full batch; float32 too.
``moe``          one routed feed-forward (``sparse_moe``) on the tokens of a step, shared expert included.
``attention``    one attention mixer on portions of prompts (projections, rotation, pages, attention, output projection).
``attn_decode``  paged attention of single tokens, one per request, behind long contexts.
``latent``       one latent attention mixer (shared rotated key part, learned sink, window) on portions of prompts.
``gla``          one gated linear attention mixer, from single tokens to whole prompts.
``delta``        one gated delta rule mixer, the same.

Sizes are those of ``bench.py`` (Qwen1.5-MoE-A2.7B and Qwen2-57B-A14B layer sizes) and of ``locus_b200/tools/arch_bench.py``
(size m).  Weights, inputs and caches are random and follow from the seed alone.
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

import locus_b200.models  # noqa: F401  (registers the architectures)
import locus_b200.parts  # noqa: F401  (registers the parts)
from locus_b200 import kernels as K
from locus_b200.cache import CacheManager
from locus_b200.config import find_arch
from locus_b200.csrc import build as kernel_build
from locus_b200.engine.batch import GroupBatch, LayerCache, Runtime, StepBatch
from locus_b200.engine.step import ModelRunner, StepEntry
from locus_b200.models.model import Model
from locus_b200.parts.base import PartSpec, iter_parts, make_part
from locus_b200.weights.loader import load_weights

DEV = "cuda:0"
F64 = torch.float64
PAGE = 64          # tokens of a page, the engine's default
VOCAB = 151936
EPS = 1e-6
SIZES = {
    # bench.py's configurations, by layer
    "a27b": dict(hidden=2048, heads=16, kv=16, dim=128, theta=1e6, experts=60, top=4, ff=1408, shared=5632),
    "57b": dict(hidden=3584, heads=28, kv=4, dim=128, theta=1e6, experts=64, top=8, ff=2560, shared=20480),
}
# arch_bench.py's size m: heads of 128 on a latent of 512 with 64 rotated dimensions; recurrences of 16 heads, 128 x 128
WIDE = dict(hidden=2048, heads=16, dim=128, rot=64, vdim=128, q_rank=768, kv_rank=512, window=4096, base=10000.0)
DECODE_STEPS = 64  # steps that a decoding request takes before its context is taken back to where it began


def _dtype(case):
    return torch.float32 if case.get("dtype") == "fp32" else torch.bfloat16


def _el(case):
    return 4 if case.get("dtype") == "fp32" else 2


def listed():
    return [
        # one user alone: the shortest step there is, a chain of short kernels
        dict(name="decode_1", kind="decode", sizes="a27b", dtype="bf16", layers=4, batch=1, ctx=1024),
        # the benchmark's headline: eight requests at 4,096 tokens
        dict(name="decode_8", kind="decode", sizes="a27b", dtype="bf16", layers=4, batch=8, ctx=4000),
        # the float32 configuration, a handful of requests
        dict(name="decode_fp32_8", kind="decode", sizes="a27b", dtype="fp32", layers=2, batch=8, ctx=1000),
        # the feed-forward of a whole prompt portion, and of a portion of the float32 configuration (512 tokens)
        dict(name="moe_2048", kind="moe", sizes="a27b", dtype="bf16", tokens=2048),
        dict(name="moe_fp32_512", kind="moe", sizes="a27b", dtype="fp32", tokens=512),
        # a 2,048-token prompt; a portion of a long prompt with grouped queries; a float32 portion behind others
        dict(name="attention_2048", kind="attention", sizes="a27b", dtype="bf16", requests=1, new=2048, ctx=0),
        dict(name="attention_57b_long", kind="attention", sizes="57b", dtype="bf16", requests=1, new=2048, ctx=8192),
        dict(name="attention_fp32_512", kind="attention", sizes="a27b", dtype="fp32", requests=1, new=512, ctx=1500),
        # eight users of the large model, 8,192 tokens each: 28 query heads on 4 key/value heads
        dict(name="attn_decode_57b_8", kind="attn_decode", sizes="57b", dtype="bf16", batch=8, ctx=8191),
        # a prompt of an odd length through a latent mixer
        dict(name="latent_1000", kind="latent", dtype="bf16", requests=1, new=1000, ctx=0),
        # a prompt through each of the recurrences: one long, three ragged ones
        dict(name="gla_2048", kind="gla", dtype="bf16", requests=1, new=2048),
        dict(name="delta_3x700", kind="delta", dtype="bf16", requests=3, new=700),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "moe", "attention", "attn_decode", "latent", "gla", "delta"])
    fp32 = rng.random() < 0.3
    if kind == "decode":
        batch = _log(rng, 1, 32)
        ctx = min(_log(rng, 64, 8000), (12000 if fp32 else 36000) // batch)
        sizes = "57b" if not fp32 and rng.random() < 0.3 else "a27b"
        return dict(kind=kind, sizes=sizes, dtype="fp32" if fp32 else "bf16", layers=2 if fp32 or sizes == "57b" else 4,
                    batch=batch, ctx=ctx)
    if kind == "moe":
        sizes = "57b" if not fp32 and rng.random() < 0.3 else "a27b"
        return dict(kind=kind, sizes=sizes, dtype="fp32" if fp32 else "bf16",
                    tokens=_log(rng, 16, 512 if fp32 else 512 if sizes == "57b" else 2048))
    if kind == "attention":
        requests = rng.choice([1, 1, 2, 3])
        sizes = "57b" if not fp32 and rng.random() < 0.4 else "a27b"
        return dict(kind=kind, sizes=sizes, dtype="fp32" if fp32 else "bf16", requests=requests,
                    new=_log(rng, 32, (512 if fp32 else 2048) // requests),
                    ctx=0 if rng.random() < 0.4 else _log(rng, 64, 1500 if fp32 else 8000))
    if kind == "attn_decode":
        batch = _log(rng, 1, 64)
        sizes = rng.choice(["a27b", "57b"])
        return dict(kind=kind, sizes=sizes, dtype="fp32" if fp32 else "bf16", batch=batch,
                    ctx=min(_log(rng, 128, 16000), (60000 if fp32 else 120000) // batch))
    if kind == "latent":
        requests = rng.choice([1, 1, 2])
        return dict(kind=kind, dtype="bf16", requests=requests, new=_log(rng, 16, 1500 // requests),
                    ctx=0 if rng.random() < 0.5 else _log(rng, 64, 3000))
    if rng.random() < 0.25:   # single tokens
        return dict(kind=kind, dtype="bf16", requests=_log(rng, 1, 64), new=1)
    requests = rng.randint(1, 8)
    return dict(kind=kind, dtype="bf16", requests=requests, new=_log(rng, 2, 2048 // requests))


# ---------------------------------------------------------------------------
# random values: each tensor follows from the seed and its name


def _rand(seed, name, shape, std=1.0, mean=0.0, dtype=torch.float32):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 2654435761 + zlib.crc32(name.encode())) % (1 << 62))
    t = torch.randn(tuple(shape), generator=g, device=DEV, dtype=torch.float32)
    t.mul_(std)
    if mean:
        t.add_(mean)
    return t.to(dtype)


def _weight(seed, name, shape, init, dtype):
    """Weights and biases N(0, 0.02), norm weights 1 + N(0, 0.01), as the engine's random-weights mode has them; a short
    convolution's taps and the step bias of a decay as large as trained ones are (decays near 1)."""
    if name.endswith(".conv"):
        return _rand(seed, name, shape, 0.5, 0.0, dtype)
    if name.endswith(".dt_bias"):
        return _rand(seed, name, shape, 0.5, -3.0, dtype)
    return _rand(seed, name, shape, 0.01 if init == "norm" else 0.02, 1.0 if init == "norm" else 0.0, dtype)


class _Source:
    """Weights by checkpoint name for ``load_weights``."""

    def __init__(self, model, seed, dtype):
        self.seed, self.dtype, self.src = seed, dtype, {s.name: s for _, s in model.tensor_sources()}

    def names(self):
        return list(self.src)

    def info(self, name):
        return self.dtype, tuple(self.src[name].shape)

    def tensor(self, name):
        s = self.src[name]
        return _weight(self.seed, name, s.shape, s.init, self.dtype)


def _part(kind, spec, prefix, seed, dtype, rt):
    """A part with its weights, bound to the runtime."""
    part = make_part(kind, spec, prefix)
    for p in iter_parts(part):
        for name, shape in p.param_shapes().items():
            p.params[name] = torch.zeros(shape, dtype=dtype, device=DEV)
        for s in p.sources():
            dest = p.params[s.param]
            flat = dest.view(-1, dest.shape[-1]) if dest.dim() >= 2 else dest
            rows = flat[s.row0 : s.row0 + s.shape[0]]
            rows.copy_(_weight(seed, s.name, s.shape, s.init, dtype).reshape(rows.shape))
    kernel_build.ensure(sorted({m for p in iter_parts(part) for m in p.kernel_modules(dtype)}))
    for p in iter_parts(part):
        p.bind(rt)
    return part


# ---------------------------------------------------------------------------
# steps


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _segments(case):
    """(new tokens, cached tokens) of each request: the first as the case says, the others a little shorter and later."""
    n, ctx = case["new"], case.get("ctx", 0)
    return [(max(1, n - 13 * i), ctx + 101 * i if ctx else 0) for i in range(case["requests"])]


def _step(segs, seed, part):
    """The descriptors of a step over requests whose pages lie scattered in the pool; (batch, pages, table on the host)."""
    qn, ctx = [s[0] for s in segs], [s[1] for s in segs]
    T, n_seg = sum(qn), len(segs)
    need = [-(-(a + b) // PAGE) for a, b in segs]
    width, total = max(need), sum(need)
    order = np.random.RandomState(seed % (1 << 31)).permutation(total).astype(np.int32)
    table = np.full((n_seg, width), -1, dtype=np.int32)
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = order[at : at + n]
        at += n
    pos, slots = [], []
    for i in range(n_seg):
        for p in range(ctx[i], ctx[i] + qn[i]):
            pos.append(p)
            slots.append(int(table[i, p // PAGE]) * PAGE + p % PAGE)
    q0 = [sum(qn[:i]) for i in range(n_seg)]
    plans = {}
    for pl in part.step_plans() if hasattr(part, "step_plans") else []:
        host = np.zeros(pl.capacity(T, n_seg), dtype=np.int32)
        res = pl.build(np.array(q0, dtype=np.int32), np.array(qn, dtype=np.int32), np.array(ctx, dtype=np.int32), host)
        dev = torch.from_numpy(host).to(DEV)
        plans[pl.key] = {k: (dev[v[0] : v[0] + v[1]].view(*v[2]) if len(v) > 2 and v[2] else dev[v[0] : v[0] + v[1]])
                         if isinstance(v, tuple) else v for k, v in res.items()}
    batch = StepBatch(T=T, n_seg=n_seg, tokens=_i32([0] * T), positions=_i32(pos), seg_q0=_i32(q0), seg_qn=_i32(qn),
                      seg_ctx=_i32(ctx), state_slots=_i32(list(range(n_seg))), want_rows=_i32([]), n_want=0,
                      longest=max(a + b for a, b in segs), plans=plans, host_seg_q0=q0, host_seg_qn=qn, host_seg_ctx=ctx,
                      host_state_slots=list(range(n_seg)))
    batch.groups[0] = GroupBatch(block_table=torch.from_numpy(table).to(DEV), slots=_i32(slots), page_tokens=PAGE)
    return batch, total, table


def _attention_spec(z):
    return PartSpec("attention", {"hidden": z["hidden"], "n_heads": z["heads"], "n_kv_heads": z["kv"], "head_dim": z["dim"],
                                  "qkv_bias": True, "position": PartSpec("rotary", {"head_dim": z["dim"], "theta": z["theta"]})})


def _moe_spec(z):
    return PartSpec("sparse_moe", {"hidden": z["hidden"], "n_experts": z["experts"], "top_k": z["top"], "norm_topk": False,
                                   "expert_intermediate": z["ff"], "shared_intermediate": z["shared"]})


def _latent_spec():
    z = WIDE
    return PartSpec("latent_attention", {
        "hidden": z["hidden"], "n_heads": z["heads"], "nope_dim": z["dim"], "rot_dim": z["rot"], "v_dim": z["vdim"],
        "q_rank": z["q_rank"], "kv_rank": z["kv_rank"], "scale": (z["dim"] + z["rot"]) ** -0.5, "eps": EPS,
        "window": z["window"], "sink": True,
        "position": PartSpec("rotary", {"head_dim": z["rot"], "theta": z["base"], "rot_dim": z["rot"], "interleaved": True})})


GLA_RANK, GLA_TAU = 16, 16.0


def _gla_spec():
    z = WIDE
    return PartSpec("gla", {"hidden": z["hidden"], "n_heads": z["heads"], "dim": z["dim"], "v_dim": z["vdim"],
                            "decay_rank": GLA_RANK, "tau": GLA_TAU, "eps": 1e-5})


def _delta_spec():
    z = WIDE
    return PartSpec("gated_delta", {"hidden": z["hidden"], "n_heads": z["heads"], "n_qk_heads": z["heads"], "dim": z["dim"],
                                    "v_dim": z["vdim"], "taps": 4, "eps": EPS})


def _raw_config(case):
    z = SIZES[case["sizes"]]
    return {"architectures": ["Qwen2MoeForCausalLM"], "model_type": "qwen2_moe", "num_hidden_layers": case["layers"],
            "hidden_size": z["hidden"], "num_attention_heads": z["heads"], "num_key_value_heads": z["kv"], "head_dim": z["dim"],
            "vocab_size": VOCAB, "rope_theta": z["theta"], "rms_norm_eps": EPS, "max_position_embeddings": 32768,
            "decoder_sparse_step": 1, "num_experts": z["experts"], "num_experts_per_tok": z["top"], "norm_topk_prob": False,
            "moe_intermediate_size": z["ff"], "shared_expert_intermediate_size": z["shared"], "intermediate_size": z["shared"],
            "qkv_bias": True, "tie_word_embeddings": False, "use_sliding_window": False, "mlp_only_layers": [],
            "hidden_act": "silu", "eos_token_id": -1}


def _context(case, seed, layer):
    """Cached keys and values of a layer: [batch, tokens (whole pages), K and V, kv heads, dim], tokens beyond the context included."""
    z = SIZES[case["sizes"]]
    n = -(-case["ctx"] // PAGE) * PAGE
    return _rand(seed, f"context {layer}", (case["batch"], n, 2, z["kv"], z["dim"]), dtype=_dtype(case))


def _decode_tokens(case, seed):
    return np.random.RandomState((seed * 7 + 3) % (1 << 31)).randint(0, VOCAB, (DECODE_STEPS, case["batch"])).tolist()


def _prepare_decode(case, seed):
    """A runner with its weights and graph, and requests whose contexts are cached."""
    dt, B, ctx = _dtype(case), case["batch"], case["ctx"]
    entry = find_arch("Qwen2MoeForCausalLM")
    model = Model(entry.build_plan(entry.parse_config(_raw_config(case))), dt, DEV)
    load_weights(model, _Source(model, seed, dt))
    limit = ctx + DECODE_STEPS
    cache = CacheManager(model.cache_needs(), page_tokens=PAGE, n_pages=B * -(-limit // PAGE), n_state_slots=B,
                         max_seq_tokens=limit, dtype=dt, device=DEV)
    runner = ModelRunner(model, cache, max_tokens=max(64, B), max_segments=B, max_wanted=B, use_graphs=True)
    tokens = _decode_tokens(case, seed)
    pool = cache.groups[0].pool
    pool.zero_()
    st = dict(kind="decode", runner=runner, cache=cache, tokens=tokens, ctx=ctx, batch=B, at=0, seqs=[])
    # the graph of this batch size is captured once, by requests of their own
    seqs = [cache.open(f"first {b}") for b in range(B)]
    for s in seqs:
        cache.ensure_capacity(s, 1)
    runner.step([StepEntry(s, [tokens[0][b]], [0]) for b, s in enumerate(seqs)])
    for s in seqs:
        cache.release(s)
    _open_requests(st)
    for layer in range(case["layers"]):
        kv = _context(case, seed, layer)
        n = kv.shape[1] // PAGE
        for b, s in enumerate(st["seqs"]):
            pages = torch.tensor(s.tables[0][:n], device=DEV)
            pool[layer, pages] = kv[b].view(n, PAGE, 2, kv.shape[3], kv.shape[4]).permute(0, 2, 3, 1, 4)
    return st


def _open_requests(st):
    """The requests at the context where they begin (again); the cached values are whatever their pages hold."""
    cache = st["cache"]
    for s in st["seqs"]:
        cache.release(s)
    st["seqs"] = [cache.open(f"request {b}") for b in range(st["batch"])]
    for s in st["seqs"]:
        cache.adopt(s, st["ctx"])
    st["at"] = 0


def prepare(case, seed):
    kind, dt = case["kind"], _dtype(case)
    torch.cuda.set_device(0)
    if kind == "decode":
        return _prepare_decode(case, seed)
    if kind == "attn_decode":
        z, B = SIZES[case["sizes"]], case["batch"]
        batch, pages, table = _step([(1, case["ctx"])] * B, seed, None)
        pool = _rand(seed, "pool", (pages, 2, z["kv"], PAGE, z["dim"]), dtype=dt)
        q = _rand(seed, "q", (B, z["heads"] * z["dim"]), 1.5, dtype=dt)
        splits = (table.shape[1] * PAGE - 1) // K.DECODE_SPLIT + 1
        units = K.decode_units(B, z["heads"], z["dim"], dt, splits, torch.device(DEV), PAGE, z["kv"])
        call = dict(items=_i32(list(range(B))), n_items=B, seg_q0=batch.seg_q0, seg_qn=batch.seg_qn, seg_ctx=batch.seg_ctx,
                    block_table=batch.groups[0].block_table, n_heads=z["heads"], n_kv_heads=z["kv"], head_dim=z["dim"],
                    page_tokens=PAGE, window=0, scale=z["dim"] ** -0.5, max_splits=splits,
                    part_o=torch.empty(units * z["dim"], device=DEV), part_ml=torch.empty(2 * units, device=DEV),
                    counters=torch.zeros(B * z["heads"], dtype=torch.int32, device=DEV))
        return dict(kind=kind, q=q, pool=pool, out=torch.empty_like(q), call=call)
    if kind == "moe":
        z, T = SIZES[case["sizes"]], case["tokens"]
        rt = Runtime(torch.device(DEV), dt, T, 1, 1)
        part = _part("feed_forward", _moe_spec(z), "mlp", seed, dt, rt)
        return dict(kind=kind, part=part, rt=rt, h=_rand(seed, "h", (T, z["hidden"]), dtype=dt),
                    x=_rand(seed, "x", (T, z["hidden"]), 0.5))
    segs = _segments(case)
    T = sum(n for n, _ in segs)
    rt = Runtime(torch.device(DEV), dt, T, len(segs), 1)
    if kind == "attention":
        z = SIZES[case["sizes"]]
        part = _part("mixer", _attention_spec(z), "attn", seed, dt, rt)
        hidden, row = z["hidden"], (2, z["kv"], PAGE, z["dim"])
    elif kind == "latent":
        z = WIDE
        part = _part("mixer", _latent_spec(), "attn", seed, dt, rt)
        hidden, row = z["hidden"], (1, 1, PAGE, z["kv_rank"] + z["rot"])
    else:
        z = WIDE
        part = _part("mixer", _gla_spec() if kind == "gla" else _delta_spec(), "mix", seed, dt, rt)
        hidden, row = z["hidden"], None
    batch, pages, _ = _step(segs, seed, part)
    h = _rand(seed, "h", (T, hidden), dtype=dt)
    x = _rand(seed, "x", (T, hidden), 0.02 if row else 0.5)
    if row:
        cache = LayerCache(group=0, pool=_rand(seed, "pool", (pages,) + row, dtype=dt), page_tokens=PAGE, state=None)
    else:
        shape = (len(segs),) + tuple(part.cache_needs()[1].shape)
        cache = LayerCache(group=None, pool=None, page_tokens=PAGE, state=_rand(seed, "state", shape, 0.1))
    return dict(kind=kind, part=part, rt=rt, batch=batch, cache=cache, h=h, x=x)


def run(state):
    kind = state["kind"]
    if kind == "decode":
        cache = state["cache"]
        if state["at"] == DECODE_STEPS:
            _open_requests(state)
        row = state["tokens"][state["at"]]
        state["at"] += 1
        for s in state["seqs"]:
            cache.ensure_capacity(s, 1)
        return state["runner"].step([StepEntry(s, [t], [0]) for s, t in zip(state["seqs"], row)])
    if kind == "attn_decode":
        K.attn_decode(state["q"], state["pool"], state["out"], **state["call"])
        return state["out"]
    with K.stream_scope():
        if kind == "moe":
            state["part"].forward(state["h"], None, state["x"], state["rt"])
            return state["x"]
        state["part"].forward(state["h"], state["batch"], state["cache"], state["x"], state["rt"])
    kept = state["cache"].pool if state["cache"].pool is not None else state["cache"].state
    return {"out": state["x"], "cache": kept}


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _attention_work(z, segs, el):
    T = sum(n for n, _ in segs)
    seen = sum(n * c + n * (n + 1) / 2 for n, c in segs)
    weights = z["hidden"] * z["dim"] * (2 * z["heads"] + 2 * z["kv"])
    bts = el * weights + el * 2 * z["kv"] * z["dim"] * sum(n + c for n, c in segs)
    return bts, 2.0 * T * weights + 4.0 * seen * z["heads"] * z["dim"]


def _moe_work(z, T, el):
    used = z["experts"] * (1 - (1 - z["top"] / z["experts"]) ** T)
    one = 3 * z["hidden"] * z["ff"]
    shared = 3 * z["hidden"] * z["shared"]
    router = z["hidden"] * (z["experts"] + 1)
    return el * (used * one + shared + router), 2.0 * T * (z["top"] * one + shared + router)


def work(case):
    kind, el = case["kind"], _el(case)
    if kind == "moe":
        z, T = SIZES[case["sizes"]], case["tokens"]
        b, f = _moe_work(z, T, el)
        return {"bytes": b + T * z["hidden"] * (el + 8), "flops": f}
    if kind == "decode":
        z, B = SIZES[case["sizes"]], case["batch"]
        b1, f1 = _attention_work(z, [(1, case["ctx"])] * B, el)
        b2, f2 = _moe_work(z, B, el)
        head = VOCAB * z["hidden"]
        return {"bytes": case["layers"] * (b1 + b2) + head * el + B * VOCAB * 4, "flops": case["layers"] * (f1 + f2) + 2.0 * B * head}
    if kind == "attn_decode":
        z, B = SIZES[case["sizes"]], case["batch"]
        keys = B * (case["ctx"] + 1)
        return {"bytes": keys * 2 * z["kv"] * z["dim"] * el + 2 * B * z["heads"] * z["dim"] * el,
                "flops": 4.0 * keys * z["heads"] * z["dim"]}
    segs = _segments(case)
    T = sum(n for n, _ in segs)
    if kind == "attention":
        z = SIZES[case["sizes"]]
        b, f = _attention_work(z, segs, el)
        return {"bytes": b + T * z["hidden"] * (el + 8), "flops": f}
    z = WIDE
    H, d, dv = z["heads"], z["dim"], z["vdim"]
    if kind == "latent":
        kv = H * (d + dv) * z["kv_rank"]
        weights = z["hidden"] * (z["q_rank"] + z["kv_rank"] + z["rot"]) + z["q_rank"] * H * (d + z["rot"]) + z["hidden"] * H * dv
        seen = sum(sum(min(c + i + 1, z["window"]) for i in range(n)) for n, c in segs)
        keys = sum(n + c for n, c in segs)
        # the least of the forms: every key's heads expanded once, then keys of dim + rot and values of vdim
        return {"bytes": el * (weights + kv + keys * (z["kv_rank"] + z["rot"])) + T * z["hidden"] * (el + 8),
                "flops": 2.0 * T * weights + 2.0 * keys * kv + 2.0 * seen * H * (d + z["rot"] + dv)}
    weights = z["hidden"] * H * (2 * d + 3 * dv)
    state = 4 * len(segs) * H * d * dv
    per = 4.0 if kind == "gla" else 6.0   # the update and the read-out; the delta rule reads the state once more
    return {"bytes": el * weights + 2 * state + T * z["hidden"] * (el + 8), "flops": 2.0 * T * weights + per * T * H * d * dv}


def tolerance(case):
    """About four times the largest error against 64 bits that was measured over listed and drawn cases of the kind.
    Where a rotation takes part in float32 (``decode``, ``attention``), its angles' rounding is the largest part of it."""
    if case.get("dtype") == "fp32":
        return {"rel": {"moe": 5e-6, "attn_decode": 5e-6}.get(case["kind"], 4e-5)}
    return {"rel": {"decode": 3.5e-2, "moe": 4e-3, "attention": 1.5e-2, "attn_decode": 8e-3, "latent": 1.5e-2, "gla": 6e-3,
                    "delta": 6e-3}[case["kind"]]}


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch


def _rotate(x, pos, theta, interleaved=False):
    """x [T, heads, dim], rotated by position: pairs (i, i + dim / 2), or (2 i, 2 i + 1)."""
    dim = x.shape[-1]
    f = torch.pow(torch.tensor(theta, dtype=F64, device=DEV), -2.0 * torch.arange(dim // 2, device=DEV, dtype=F64) / dim)
    a = pos.to(F64)[:, None] * f[None, :]
    c, s = torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]
    if interleaved:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).reshape(x.shape)
    u, v = x[..., : dim // 2], x[..., dim // 2 :]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _attend(q, k, v, first, scale, window=0, sink=None):
    """q [n, H, d] at positions first .., k [m, G, d], v [m, G, dv] at 0 .. -> [n, H, dv]."""
    n, H, _ = q.shape
    m, G = k.shape[0], k.shape[1]
    pos, j = torch.arange(first, first + n, device=DEV)[:, None], torch.arange(m, device=DEV)[None, :]
    seen = j <= pos
    if window:
        seen &= pos - j < window
    out = torch.empty(n, H, v.shape[2], dtype=F64, device=DEV)
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h] @ k[:, g].T * scale).masked_fill(~seen, -math.inf)
        if sink is not None:
            p = torch.softmax(torch.cat([s, sink[h].expand(n, 1)], 1), 1)[:, :m]
        else:
            p = torch.softmax(s, 1)
        out[:, h] = p @ v[:, g]
    return out


def _exact_moe(z, h, W, prefix):
    logits = h @ W(f"{prefix}.gate.weight", (z["experts"], z["hidden"])).T
    p = torch.softmax(logits, -1)
    wts, ids = torch.topk(p, z["top"], -1)
    out = torch.zeros(h.shape[0], z["hidden"], dtype=F64, device=DEV)

    def mlp(rows, name, ff):
        g, u = (W(f"{name}.{r}_proj.weight", (ff, z["hidden"])) for r in ("gate", "up"))
        return _silu(rows @ g.T) * (rows @ u.T) @ W(f"{name}.down_proj.weight", (z["hidden"], ff)).T

    for e in range(z["experts"]):
        t, slot = torch.nonzero(ids == e, as_tuple=True)
        if len(t):
            out.index_add_(0, t, mlp(h[t], f"{prefix}.experts.{e}", z["ff"]) * wts[t, slot][:, None])
    gate = torch.sigmoid(h @ W(f"{prefix}.shared_expert_gate.weight", (1, z["hidden"])).T)
    return out + gate * mlp(h, f"{prefix}.shared_expert", z["shared"])


def _exact_qkv(z, h, W, prefix, pos):
    def proj(r, heads):
        n = heads * z["dim"]
        return (h @ W(f"{prefix}.{r}_proj.weight", (n, z["hidden"])).T + W(f"{prefix}.{r}_proj.bias", (n,), "bias")).view(-1, heads, z["dim"])

    return _rotate(proj("q", z["heads"]), pos, z["theta"]), _rotate(proj("k", z["kv"]), pos, z["theta"]), proj("v", z["kv"])


def _exact_decode(case, seed, W):
    z, B, ctx = SIZES[case["sizes"]], case["batch"], case["ctx"]
    tokens = torch.tensor(_decode_tokens(case, seed)[0], device=DEV)
    x = _weight(seed, "model.embed_tokens.weight", (VOCAB, z["hidden"]), "linear", _dtype(case))[tokens].double()
    pos = torch.full((B,), ctx, device=DEV)
    for layer in range(case["layers"]):
        p = f"model.layers.{layer}"
        h = _rms(x, W(f"{p}.input_layernorm.weight", (z["hidden"],), "norm"), EPS)
        q, k, v = _exact_qkv(z, h, W, f"{p}.self_attn", pos)
        kv = _context(case, seed, layer)[:, :ctx]
        o = torch.empty(B, z["heads"] * z["dim"], dtype=F64, device=DEV)
        for b in range(B):
            keys, vals = (torch.cat([kv[b, :, i].double(), new[b : b + 1]]) for i, new in ((0, k), (1, v)))
            o[b] = _attend(q[b : b + 1], keys, vals, ctx, z["dim"] ** -0.5).view(-1)
        x = x + o @ W(f"{p}.self_attn.o_proj.weight", (z["hidden"], z["heads"] * z["dim"])).T
        h = _rms(x, W(f"{p}.post_attention_layernorm.weight", (z["hidden"],), "norm"), EPS)
        x = x + _exact_moe(z, h, W, f"{p}.mlp")
    h = _rms(x, W("model.norm.weight", (z["hidden"],), "norm"), EPS)
    return h @ W("lm_head.weight", (VOCAB, z["hidden"])).T


def _paged_rows(pool, table, n):
    """[n, planes, heads, dim]: the rows of positions 0 .. n - 1 of one request."""
    pages = pool[torch.from_numpy(table[: -(-n // PAGE)]).long().to(DEV)]            # [pages, planes, heads, PAGE, dim]
    return pages.permute(0, 3, 1, 2, 4).reshape(-1, pool.shape[1], pool.shape[2], pool.shape[4])[:n]


def _exact_latent(z, h, W, pos):
    def norm(x, name, n):
        return _rms(x, W(f"attn.{name}", (n,), "norm"), EPS)

    cq = norm(h @ W("attn.dq", (z["q_rank"], z["hidden"])).T, "dq.norm", z["q_rank"])
    q = (cq @ W("attn.uq", (z["heads"] * (z["dim"] + z["rot"]), z["q_rank"])).T).view(-1, z["heads"], z["dim"] + z["rot"])
    down = h @ W("attn.dkv", (z["kv_rank"] + z["rot"], z["hidden"])).T
    c = norm(down[:, : z["kv_rank"]], "dkv.norm", z["kv_rank"])
    rot = _rotate(down[:, None, z["kv_rank"] :], pos, z["base"], True)[:, 0]
    q = torch.cat([q[..., : z["dim"]], _rotate(q[..., z["dim"] :], pos, z["base"], True)], -1)
    return q, torch.cat([c, rot], -1)


def _exact_recurrent(case, seed, W, h, state):
    """(mixer's output, state) of the recurrences; ``state`` [requests, floats] is advanced in place."""
    z = WIDE
    H, d, dv, hid = z["heads"], z["dim"], z["vdim"], z["hidden"]
    out = torch.empty(h.shape[0], hid, dtype=F64, device=DEV)
    t0 = 0
    for r, (n, _) in enumerate(_segments(case)):
        hr = h[t0 : t0 + n]
        S = state[r, : H * d * dv].view(H, d, dv).clone()
        gate = hr @ W("mix.g", (H * dv, hid)).T
        if case["kind"] == "gla":
            q, k = ((hr @ W(f"mix.{c}", (H * d, hid)).T).view(n, H, d) for c in "qk")
            v = (hr @ W("mix.v", (H * dv, hid)).T).view(n, H, dv)
            lg = hr @ W("mix.a1", (GLA_RANK, hid)).T @ W("mix.a2", (H * d, GLA_RANK)).T + W("mix.a2.b", (H * d,), "bias")
            a = torch.sigmoid(lg).pow(1.0 / GLA_TAU).view(n, H, d)
            q, eps = q * d ** -0.5, 1e-5
        else:
            names, widths = ("q", "k", "v"), (H * d, H * d, H * dv)
            u = torch.cat([hr @ W(f"mix.{c}", (w, hid)).T for c, w in zip(names, widths)], 1)
            conv = torch.cat([W(f"mix.{c}.conv", (w, 4), "bias") for c, w in zip(names, widths)], 0)
            past = state[r, H * d * dv :].view(-1, 3)          # the last three projected rows, oldest first
            full = torch.cat([past.T, u], 0)
            state[r, H * d * dv :] = full[-3:].T.reshape(-1)
            u = _silu(sum(full[j : j + n] * conv[:, j] for j in range(4)))
            q, k, v = (x.view(n, H, -1) for x in u.split(list(widths), 1))
            q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
            q, eps = q * d ** -0.5, EPS
            beta = torch.sigmoid(hr @ W("mix.b", (H, hid)).T)
            dt = torch.nn.functional.softplus(hr @ W("mix.a", (H, hid)).T + W("mix.dt_bias", (H,), "bias"))
            a = torch.exp(-torch.exp(W("mix.A_log", (H,), "bias")) * dt)[:, :, None].expand(n, H, d)
        o = torch.empty(n, H, dv, dtype=F64, device=DEV)
        for t in range(n):
            S = S * a[t][:, :, None]
            u = v[t] if case["kind"] == "gla" else beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            o[t] = torch.einsum("hde,hd->he", S, q[t])
        state[r, : H * d * dv] = S.reshape(-1)
        o = _rms(o, W("mix.norm", (dv,), "norm"), eps).view(n, -1) * _silu(gate)
        out[t0 : t0 + n] = o @ W("mix.o", (hid, H * dv)).T
        t0 += n
    return out, state


def exact(case, seed):
    kind, dt = case["kind"], _dtype(case)

    def W(name, shape, init="linear"):
        return _weight(seed, name, shape, init, dt).double()

    if kind == "decode":
        return _exact_decode(case, seed, W)
    if kind == "attn_decode":
        z, B, n = SIZES[case["sizes"]], case["batch"], case["ctx"] + 1
        _, pages, table = _step([(1, case["ctx"])] * B, seed, None)
        pool = _rand(seed, "pool", (pages, 2, z["kv"], PAGE, z["dim"]), dtype=dt)
        q = _rand(seed, "q", (B, z["heads"] * z["dim"]), 1.5, dtype=dt).double().view(B, 1, z["heads"], z["dim"])
        out = torch.empty(B, z["heads"] * z["dim"], dtype=F64, device=DEV)
        for b in range(B):
            kv = _paged_rows(pool, table[b], n).double()
            out[b] = _attend(q[b], kv[:, 0], kv[:, 1], n - 1, z["dim"] ** -0.5).view(-1)
        return out
    if kind == "moe":
        z, T = SIZES[case["sizes"]], case["tokens"]
        h = _rand(seed, "h", (T, z["hidden"]), dtype=dt).double()
        return _rand(seed, "x", (T, z["hidden"]), 0.5).double() + _exact_moe(z, h, W, "mlp")
    segs = _segments(case)
    T = sum(n for n, _ in segs)
    z = SIZES[case["sizes"]] if kind == "attention" else WIDE
    h = _rand(seed, "h", (T, z["hidden"]), dtype=dt).double()
    if kind in ("gla", "delta"):
        shape = (len(segs), z["heads"] * z["dim"] * z["vdim"] + (0 if kind == "gla" else 3 * z["heads"] * (2 * z["dim"] + z["vdim"])))
        out, state = _exact_recurrent(case, seed, W, h, _rand(seed, "state", shape, 0.1).double())
        return {"out": _rand(seed, "x", (T, z["hidden"]), 0.5).double() + out, "cache": state}
    _, pages, table = _step(segs, seed, None)
    row = (2, z["kv"], PAGE, z["dim"]) if kind == "attention" else (1, 1, PAGE, z["kv_rank"] + z["rot"])
    pool = _rand(seed, "pool", (pages,) + row, dtype=dt).double()
    out = _rand(seed, "x", (T, z["hidden"]), 0.02).double()
    t0 = 0
    for r, (n, ctx) in enumerate(segs):
        hr, pos = h[t0 : t0 + n], torch.arange(ctx, ctx + n, device=DEV)
        page = torch.from_numpy(table[r]).long().to(DEV)[pos // PAGE]
        if kind == "attention":
            q, k, v = _exact_qkv(z, hr, W, "attn", pos)
            pool[page, 0, :, pos % PAGE], pool[page, 1, :, pos % PAGE] = k, v
            kv = _paged_rows(pool, table[r], n + ctx)
            o = _attend(q, kv[:, 0], kv[:, 1], ctx, z["dim"] ** -0.5)
            wo = W("attn.o_proj.weight", (z["hidden"], z["heads"] * z["dim"]))
        else:
            q, rows = _exact_latent(z, hr, W, pos)
            pool[page, 0, 0, pos % PAGE] = rows
            kv = _paged_rows(pool, table[r], n + ctx)[:, 0, 0]
            uk = W("attn.uk", (z["heads"] * z["dim"], z["kv_rank"]))
            uv = W("attn.uv", (z["heads"] * z["vdim"], z["kv_rank"]))
            c, rot = kv[:, : z["kv_rank"]], kv[:, z["kv_rank"] :]
            keys = torch.cat([(c @ uk.T).view(-1, z["heads"], z["dim"]), rot[:, None].expand(-1, z["heads"], -1)], -1)
            o = _attend(q, keys, (c @ uv.T).view(-1, z["heads"], z["vdim"]), ctx, (z["dim"] + z["rot"]) ** -0.5, z["window"],
                        W("attn.sink", (z["heads"],), "bias"))
            wo = W("attn.o", (z["hidden"], z["heads"] * z["vdim"]))
        out[t0 : t0 + n] += o.reshape(n, -1) @ wo.T
        t0 += n
    return {"out": out, "cache": pool}
