"""The work that a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values.  ``prepare`` makes what a program holds before the call (weights, cache pages,
inputs, a batch's context) on the GPU from a seed; ``run`` is one pass through a public entry point; ``exact`` is the
same in float64, written here in plain torch.  Kinds:

step        ``ModelRunner.step`` of a whole dense decoder: prompt portions, decoded tokens or both; logits
attention   the grouped-query mixer over a paged cache (projections, rotation, cache write, attention, projection)
mlp         the SiLU-gated feed-forward
experts     the feed-forward of routed experts
latent      the mixer over latent rows
recurrence  the mixers that keep a matrix state: lightning attention and the state-space mixer
sample      from logits to tokens
"""
import math
import random

import torch

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
DTYPES = {"bfloat16": BF16, "float32": F32}
PAGE = 16
DECAY_FIRST, DECAY_SPAN = 5.0, 3.0


# ---------------------------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------------------------
# "lens": the tokens that every sequence of the batch brings; "starts": how many it already has in the cache.
def listed():
    return [
        # one step of a server under load: a long prompt, the rest of another, and six requests that decode
        dict(name="serving_step", kind="step", layers=4, hidden=2048, heads=16, kv_heads=4, dim=128, inter=4096,
             vocab=32768, lens="1791,250,1,1,1,1,1,1", starts="0,1024,2047,1500,803,2048,77,1290", dtype="bfloat16"),
        # eight requests that decode behind prompts of about 2,048 tokens (the benchmark's batch), four layers of that model
        dict(name="decode_step", kind="step", layers=4, hidden=2048, heads=32, kv_heads=8, dim=64, inter=8192,
             vocab=32768, lens="1,1,1,1,1,1,1,1", starts="2048,2100,2047,2200,2061,2303,2048,2111", dtype="bfloat16"),
        # three prompts of different lengths, one of them a later portion
        dict(name="attention_prompts", kind="attention", hidden=2048, heads=32, kv_heads=8, dim=64, window=0,
             lens="4096,1531,700", starts="0,0,2048", dtype="bfloat16"),
        # a full batch that decodes, contexts of up to 4,096 tokens
        dict(name="attention_decode", kind="attention", hidden=2048, heads=16, kv_heads=4, dim=128, window=0,
             lens=",".join(["1"] * 64), starts=",".join(str(1500 + (i * 1237) % 2596) for i in range(64)), dtype="bfloat16"),
        # the smallest call: the feed-forward of one decoded token
        dict(name="mlp_one_token", kind="mlp", rows=1, hidden=2048, inter=8192, dtype="bfloat16"),
        # the exact path: a portion of 96 tokens in float32
        dict(name="mlp_float32", kind="mlp", rows=96, hidden=1024, inter=2048, dtype="float32"),
        # routed experts behind a prompt of 2,048 tokens
        dict(name="experts_prompt", kind="experts", rows=2048, hidden=2048, inner=1024, experts=32, top=4, dtype="bfloat16"),
        # a prompt of 2,048 tokens through the latent mixer
        dict(name="latent_prompt", kind="latent", hidden=2048, heads=16, nope=128, rot=64, vdim=128, q_rank=768,
             kv_rank=512, window=0, sink=True, lens="2048", starts="0", dtype="bfloat16"),
        # eight requests that decode through it
        dict(name="latent_decode", kind="latent", hidden=2048, heads=16, nope=128, rot=64, vdim=128, q_rank=768,
             kv_rank=512, window=0, sink=True, lens="1,1,1,1,1,1,1,1", starts="4000,3777,4095,2048,3001,3900,4064,3500",
             dtype="bfloat16"),
        # a prompt of 2,048 tokens through a linear attention
        dict(name="lightning_prompt", kind="recurrence", mixer="lightning_attention", hidden=2048, heads=16, dim=128, vdim=128,
             groups=0, lens="2048", starts="0", dtype="bfloat16"),
        # two prompts through a state-space mixer
        dict(name="state_space_prompt", kind="recurrence", mixer="state_space", hidden=2048, heads=64, dim=128, vdim=64,
             groups=2, lens="1500,548", starts="0,0", dtype="bfloat16"),
        # the next token of eight requests with a temperature and a nucleus
        dict(name="sample_top_p", kind="sample", rows=8, vocab=128256, mode="top_p"),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm; every other one odd or ragged as it comes."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _batch(rng, most_tokens, most_context, decode):
    """(lens, starts): a batch of single tokens, or of prompt portions."""
    if decode:
        n = _log(rng, 1, 64)
        most = min(most_context, 262144 // n)
        return [1] * n, [_log(rng, 16, most) for _ in range(n)]
    n = rng.choice([1, 1, 2, 3, 5])
    lens = [_log(rng, 33, max(64, most_tokens // n)) for _ in range(n)]
    return lens, [0 if rng.random() < 0.6 else _log(rng, 16, most_context // 4) for _ in range(n)]


def _text(v):
    return ",".join(str(x) for x in v)


def draw(rng):
    kind = rng.choice(["step", "attention", "mlp", "experts", "latent", "recurrence", "sample"])
    if kind == "step":
        size = rng.choice([dict(hidden=1024, heads=16, kv_heads=4, dim=64, inter=2048),
                           dict(hidden=2048, heads=16, kv_heads=4, dim=128, inter=4096),
                           dict(hidden=2048, heads=32, kv_heads=8, dim=64, inter=8192)])
        lens, starts = _batch(rng, 1024, 2048, rng.random() < 0.5)
        return dict(kind=kind, layers=rng.choice([1, 2]), vocab=rng.choice([32768, 16384]), lens=_text(lens),
                    starts=_text(starts), dtype="bfloat16", **size)
    if kind == "attention":
        size = rng.choice([dict(heads=32, kv_heads=8, dim=64), dict(heads=16, kv_heads=4, dim=128),
                           dict(heads=24, kv_heads=8, dim=128), dict(heads=16, kv_heads=4, dim=64)])
        lens, starts = _batch(rng, 4096, 4096, rng.random() < 0.5)
        dtype = "float32" if sum(lens) <= 256 and len(lens) <= 8 and rng.random() < 0.3 else "bfloat16"
        return dict(kind=kind, hidden=rng.choice([1024, 2048]), window=rng.choice([0, 0, 512, 1024]), lens=_text(lens),
                    starts=_text(starts), dtype=dtype, **size)
    if kind == "mlp":
        hidden, inter = rng.choice([(2048, 8192), (1024, 2048), (2048, 4096), (3072, 8192)])
        f32 = rng.random() < 0.2
        return dict(kind=kind, rows=_log(rng, 1, 128 if f32 else 4096), hidden=hidden, inter=inter,
                    dtype="float32" if f32 else "bfloat16")
    if kind == "experts":
        size = rng.choice([dict(hidden=2048, inner=1024, experts=32, top=4), dict(hidden=1024, inner=1024, experts=16, top=2)])
        return dict(kind=kind, rows=_log(rng, 1, 2048), dtype="bfloat16", **size)
    if kind == "latent":
        size = rng.choice([dict(hidden=2048, heads=16, nope=128, rot=64, vdim=128, q_rank=768, kv_rank=512),
                           dict(hidden=1024, heads=8, nope=64, rot=32, vdim=64, q_rank=384, kv_rank=256)])
        lens, starts = _batch(rng, 1800, 4096, rng.random() < 0.5)
        return dict(kind=kind, window=rng.choice([0, 0, 512, 1024]), sink=rng.random() < 0.5, lens=_text(lens),
                    starts=_text(starts), dtype="bfloat16", **size)
    if kind == "recurrence":
        size = rng.choice([dict(mixer="lightning_attention", hidden=2048, heads=16, dim=128, vdim=128, groups=0),
                           dict(mixer="lightning_attention", hidden=1024, heads=8, dim=64, vdim=128, groups=0),
                           dict(mixer="state_space", hidden=2048, heads=64, dim=128, vdim=64, groups=2),
                           dict(mixer="state_space", hidden=1024, heads=32, dim=128, vdim=64, groups=1)])
        lens, _ = _batch(rng, 2048, 64, rng.random() < 0.35)
        return dict(kind=kind, lens=_text(lens), starts=_text([0] * len(lens)), dtype="bfloat16", **size)
    return dict(kind=kind, rows=_log(rng, 1, 64), vocab=rng.choice([128256, 32768]),
                mode=rng.choice(["greedy", "temperature", "top_p", "top_k", "all"]))


# ---------------------------------------------------------------------------------------------------------------
# inputs, from the seed alone: float64 code below and the framework read the same tensors
# ---------------------------------------------------------------------------------------------------------------
class _Draw:
    def __init__(self, case, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed) * 1000003 + 17)
        self.dtype = DTYPES[case.get("dtype", "bfloat16")]

    def normal(self, *shape, std=1.0, mean=0.0, dtype=None):
        t = torch.randn(*shape, generator=self.g, device="cuda", dtype=F32)
        return t.mul_(std).add_(mean).to(dtype or self.dtype)


def _ints(text):
    return [int(v) for v in text.split(",")]


def _mlp_weights(d, hidden, inter, std=0.02):
    return {"gate": d.normal(inter, hidden, std=std), "up": d.normal(inter, hidden, std=std),
            "down": d.normal(hidden, inter, std=std)}


def _attention_weights(d, c):
    nq, nkv, h = c["heads"] * c["dim"], c["kv_heads"] * c["dim"], c["hidden"]
    return {"q": d.normal(nq, h, std=0.03), "k": d.normal(nkv, h, std=0.03), "v": d.normal(nkv, h, std=0.02),
            "o": d.normal(h, nq, std=0.02)}


def _old_rows(d, c, heads, dim):
    """What the cache already holds: for each sequence [start, heads, dim]."""
    return [d.normal(s, heads, dim) for s in _ints(c["starts"])]


def _draw_inputs(c, seed):
    d = _Draw(c, seed)
    k = c["kind"]
    if k == "mlp":
        return dict(w=_mlp_weights(d, c["hidden"], c["inter"]), x=d.normal(c["rows"], c["hidden"]))
    if k == "experts":
        n, f, h = c["experts"], c["inner"], c["hidden"]
        return dict(router=d.normal(n, h, std=0.03), gate=d.normal(n, f, h, std=0.03), up=d.normal(n, f, h, std=0.03),
                    down=d.normal(n, h, f, std=0.03), x=d.normal(c["rows"], h))
    if k == "sample":
        return dict(logits=d.normal(c["rows"], c["vocab"], std=2.0, dtype=F32))
    T = sum(_ints(c["lens"]))
    if k == "attention":
        return dict(w=_attention_weights(d, c), x=d.normal(T, c["hidden"]), k=_old_rows(d, c, c["kv_heads"], c["dim"]),
                    v=_old_rows(d, c, c["kv_heads"], c["dim"]))
    if k == "latent":
        H, kv, qr, h = c["heads"], c["kv_rank"], c["q_rank"], c["hidden"]
        w = {"dq": d.normal(qr, h, std=0.02), "dq_norm": d.normal(qr, std=0.1, mean=1.0, dtype=F32),
             "uq": d.normal(H * (c["nope"] + c["rot"]), qr, std=0.04), "dkv": d.normal(kv + c["rot"], h, std=0.02),
             "dkv_norm": d.normal(kv, std=0.1, mean=1.0, dtype=F32), "uk": d.normal(H * c["nope"], kv, std=0.04),
             "uv": d.normal(H * c["vdim"], kv, std=0.04), "o": d.normal(h, H * c["vdim"], std=0.02)}
        if c["sink"]:
            w["sink"] = d.normal(H, dtype=F32)
        return dict(w=w, x=d.normal(T, h), k=_old_rows(d, c, 1, kv + c["rot"]))
    if k == "recurrence":
        H, dk, dv, h = c["heads"], c["dim"], c["vdim"], c["hidden"]
        if c["mixer"] == "lightning_attention":
            w = {"q": d.normal(H * dk, h, std=0.02), "k": d.normal(H * dk, h, std=0.02), "v": d.normal(H * dv, h, std=0.02),
                 "g": d.normal(H * dv, h, std=0.02), "o": d.normal(h, H * dv, std=0.02),
                 "norm": d.normal(H * dv, std=0.1, mean=1.0, dtype=F32)}
        else:
            inner = H * dv
            ch = inner + 2 * c["groups"] * dk
            w = {"in": d.normal(inner + ch + H, h, std=0.02), "conv": d.normal(ch, 4, std=0.4, dtype=F32),
                 "conv_bias": d.normal(ch, std=0.1, dtype=F32), "dt_bias": d.normal(H, std=1.0, dtype=F32),
                 "a_log": d.normal(H, std=1.0, dtype=F32), "d": d.normal(H, std=0.1, mean=1.0, dtype=F32),
                 "norm": d.normal(inner, std=0.1, mean=1.0, dtype=F32), "o": d.normal(h, inner, std=0.02)}
        return dict(w=w, x=d.normal(T, h))
    # step
    w = {"embed": d.normal(c["vocab"], c["hidden"], std=1.0), "head": d.normal(c["vocab"], c["hidden"], std=0.02),
         "norm": d.normal(c["hidden"], std=0.1, mean=1.0, dtype=F32), "layers": []}
    for _ in range(c["layers"]):
        w["layers"].append(dict(att=_attention_weights(d, c), mlp=_mlp_weights(d, c["hidden"], c["inter"]),
                                n1=d.normal(c["hidden"], std=0.1, mean=1.0, dtype=F32),
                                n2=d.normal(c["hidden"], std=0.1, mean=1.0, dtype=F32)))
    rng = random.Random(int(seed) * 7919 + 5)
    tokens = [[rng.randrange(c["vocab"]) for _ in range(n)] for n in _ints(c["lens"])]
    old = [(_old_rows(d, c, c["kv_heads"], c["dim"]), _old_rows(d, c, c["kv_heads"], c["dim"])) for _ in range(c["layers"])]
    return dict(w=w, tokens=tokens, old=old)


# ---------------------------------------------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------------------------------------------
class _State:
    pass


def _device():
    return torch.device("cuda:0")


def _batch_of(c, needs, dtype):
    """A cache manager whose requests hold their pages (handed out in turns, as a server does), and their entries."""
    from rllm_b200.cache import CacheManager
    from rllm_b200.engine.runner import StepEntry
    lens, starts = _ints(c["lens"]), _ints(c["starts"])
    pages = sum(-(-(a + b) // PAGE) for a, b in zip(lens, starts)) + 8
    paged = [n for n in needs if hasattr(n, "num_kv_heads")]
    cache = CacheManager(needs, PAGE, [pages] * len(paged), len(lens))
    for s in range(len(lens)):
        cache.admit(s)
    top = max(a + b for a, b in zip(lens, starts))
    for at in range(256, top + 256, 256):
        for s, (a, b) in enumerate(zip(lens, starts)):
            # the first query at position 0: windows give no page back here
            if at - 256 < a + b and not cache.ensure(s, 0, min(at, a + b)):
                raise RuntimeError("the pool is too small")
    entries = [StepEntry(s, [0] * a, b, []) for s, (a, b) in enumerate(zip(lens, starts))]
    return cache, entries, pages


def _fill_pages(cache, group, buffer, rows):
    """Rows [start, heads, dim] of every sequence into its pages [pages, heads, PAGE, dim]."""
    for s, r in enumerate(rows):
        n = r.shape[0]
        if not n:
            continue
        table = torch.tensor(cache.table(s, group), device="cuda", dtype=torch.long)
        at = torch.arange(n, device="cuda")
        buffer[table[at // PAGE], :, at % PAGE] = r


def _pages_like(pages, heads, dim, dtype):
    return torch.zeros(pages + 1, heads, PAGE, dim, device="cuda", dtype=dtype)


def _part(family, kind, names, weights, **params):
    from rllm_b200.parts import PartSpec, build_part
    part = build_part(family, PartSpec.of(kind, tensor_names={k: k for k in names}, **params))
    part.load(weights)
    return part


def _rotary(dim, interleaved):
    from rllm_b200.parts import PartSpec
    return PartSpec.of("rotary", head_dim=dim, rotary_dim=dim, theta=500000.0, scaling=None, interleaved=interleaved)


def _context(c, part, dtype):
    """(cache manager, context on the device, number of pages) of a mixer's batch."""
    from rllm_b200.engine.runner import BatchBuilder
    need = part.cache_need()
    needs = list(need) if isinstance(need, (tuple, list)) else [need]
    cache, entries, pages = _batch_of(c, needs, dtype)
    ctx, _, _ = BatchBuilder(cache, _device(), dtype).build_context(entries)
    return cache, ctx, pages


def _flat_order(c):
    """Sequences in a flat batch: single tokens first; the order of the rows that ``BatchBuilder`` lays out."""
    lens = _ints(c["lens"])
    return sorted(range(len(lens)), key=lambda i: (lens[i] != 1, i))


def prepare(case, seed):
    c, s = case, _State()
    i = _draw_inputs(c, seed)
    k = c["kind"]
    dtype = DTYPES[c.get("dtype", "bfloat16")]
    s.kind = k
    if k == "mlp":
        s.part = _part("feed_forward", "gated_mlp", ("gate", "up", "down"), i["w"], hidden_size=c["hidden"],
                       intermediate_size=c["inter"])
        s.x = i["x"]
    elif k == "experts":
        tensors = {"router": i["router"]}
        for e in range(c["experts"]):
            tensors.update({f"gate{e}": i["gate"][e], f"up{e}": i["up"][e], f"down{e}": i["down"][e]})
        from rllm_b200.parts import PartSpec, build_part
        s.part = build_part("feed_forward", PartSpec.of(
            "routed_experts", hidden_size=c["hidden"], inner_size=c["inner"], num_experts=c["experts"], top=c["top"],
            tensor_names={"router": "router", "gate": "gate{e}", "up": "up{e}", "down": "down{e}"}))
        s.part.load(tensors)
        s.x = i["x"]
    elif k == "sample":
        from rllm_b200.sampling import SamplingParams
        from rllm_b200.sampling.sampler import Sampler, SamplingRow
        options = {"greedy": dict(temperature=0.0), "temperature": dict(temperature=0.8),
                   "top_p": dict(temperature=0.8, top_p=0.9), "top_k": dict(temperature=0.8, top_k=50),
                   "all": dict(temperature=0.7, top_p=0.95, top_k=100, min_p=0.02)}[c["mode"]]
        s.sampler, s.logits = Sampler(_device()), i["logits"]
        s.rows = [SamplingRow(SamplingParams(**options), seed=int(seed) * 131 + r, gen_index=r) for r in range(c["rows"])]
    elif k == "attention":
        s.part = _part("mixer", "attention", ("q", "k", "v", "o"), i["w"], hidden_size=c["hidden"], num_heads=c["heads"],
                       num_kv_heads=c["kv_heads"], head_dim=c["dim"], window=c["window"] or None,
                       position=_rotary(c["dim"], False))
        s.cache, s.ctx, pages = _context(c, s.part, dtype)
        from rllm_b200.parts.base import KVCacheView
        s.view = KVCacheView(_pages_like(pages, c["kv_heads"], c["dim"], dtype),
                             _pages_like(pages, c["kv_heads"], c["dim"], dtype), 0, True)
        _fill_pages(s.cache, 0, s.view.k, i["k"])
        _fill_pages(s.cache, 0, s.view.v, i["v"])
        s.x = i["x"]
    elif k == "latent":
        names = ["dq", "dq_norm", "uq", "dkv", "dkv_norm", "uk", "uv", "o"] + (["sink"] if c["sink"] else [])
        s.part = _part("mixer", "latent_attention", names, i["w"], hidden_size=c["hidden"], num_heads=c["heads"],
                       nope_dim=c["nope"], rot_dim=c["rot"], v_dim=c["vdim"], q_rank=c["q_rank"], kv_rank=c["kv_rank"],
                       scale=(c["nope"] + c["rot"]) ** -0.5, eps=1e-6, window=c["window"] or None, sink=c["sink"],
                       position=_rotary(c["rot"], True))
        s.cache, s.ctx, pages = _context(c, s.part, dtype)
        from rllm_b200.parts.base import KVCacheView
        s.view = KVCacheView(_pages_like(pages, 1, c["kv_rank"] + c["rot"], dtype), None, 0, True)
        _fill_pages(s.cache, 0, s.view.k, i["k"])
        s.x = i["x"]
    elif k == "recurrence":
        if c["mixer"] == "lightning_attention":
            s.part = _part("mixer", "lightning_attention", ("q", "k", "v", "g", "o", "norm"), i["w"], hidden_size=c["hidden"],
                           num_heads=c["heads"], head_dim=c["dim"], v_dim=c["vdim"], decay=_decays(c), eps=1e-6)
        else:
            s.part = _part("mixer", "state_space", ("in", "conv", "conv_bias", "dt_bias", "a_log", "d", "norm", "o"), i["w"],
                           hidden_size=c["hidden"], num_heads=c["heads"], v_dim=c["vdim"], state=c["dim"],
                           groups=c["groups"], conv=4, norm_groups=c["groups"], eps=1e-6)
        s.cache, s.ctx, _ = _context(c, s.part, dtype)
        from rllm_b200.parts.base import StateCacheView
        need = s.part.cache_need()
        n = len(_ints(c["lens"]))
        views = [StateCacheView(torch.zeros((n + 1,) + tuple(x.shape), device="cuda", dtype=F32), g, True)
                 for g, x in enumerate(need if isinstance(need, (tuple, list)) else [need])]
        s.view = tuple(views) if isinstance(need, (tuple, list)) else views[0]
        s.x = i["x"]
    else:
        s.runner, s.entries, s.kv = _runner(c, i, dtype)
    return s


def _decays(c):
    return [1.0 - 2.0 ** (-DECAY_FIRST - DECAY_SPAN * h / max(1, c["heads"] - 1)) for h in range(c["heads"])]


def _runner(c, i, dtype):
    from rllm_b200.cache import CacheStorage
    from rllm_b200.config import resolve_architecture
    from rllm_b200.engine.runner import ModelRunner, StepEntry
    from rllm_b200.models.decoder import DecoderModel
    from rllm_b200.weights.loader import WeightSource
    cfg = {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": c["layers"],
           "hidden_size": c["hidden"], "num_attention_heads": c["heads"], "num_key_value_heads": c["kv_heads"],
           "head_dim": c["dim"], "intermediate_size": c["inter"], "vocab_size": c["vocab"], "rope_theta": 500000.0,
           "max_position_embeddings": 131072, "rms_norm_eps": 1e-5, "tie_word_embeddings": False, "hidden_act": "silu",
           "torch_dtype": c["dtype"], "bos_token_id": 0, "eos_token_id": 1}
    w = i["w"]
    tensors = {"model.embed_tokens.weight": w["embed"], "lm_head.weight": w["head"], "model.norm.weight": w["norm"]}
    for n, layer in enumerate(w["layers"]):
        p = f"model.layers.{n}."
        for key in "qkvo":
            tensors[f"{p}self_attn.{key}_proj.weight"] = layer["att"][key]
        for key in ("gate", "up", "down"):
            tensors[f"{p}mlp.{key}_proj.weight"] = layer["mlp"][key]
        tensors[p + "input_layernorm.weight"] = layer["n1"]
        tensors[p + "post_attention_layernorm.weight"] = layer["n2"]

    class Source(WeightSource):
        def names(self):
            return list(tensors)

        def info(self, name):
            return tensors[name].dtype, tuple(tensors[name].shape)

        def read(self, name):
            return tensors[name]

    arch = resolve_architecture(cfg)
    model = DecoderModel(arch.build_spec(arch.parse_config(cfg)))
    model.load(Source(), dtype, _device())
    cache, entries, pages = _batch_of(c, model.layout.groups, dtype)
    storage = CacheStorage(model.layout, PAGE, [pages], len(entries), dtype, _device())
    kv = []
    for n in range(c["layers"]):
        view = storage.view(n)
        _fill_pages(cache, 0, view.k, i["old"][n][0])
        _fill_pages(cache, 0, view.v, i["old"][n][1])
        kv += [view.k, view.v]
    entries = [StepEntry(e.req, i["tokens"][s], e.start, [len(i["tokens"][s]) - 1]) for s, e in enumerate(entries)]
    return ModelRunner(model, cache, storage), entries, kv


# ---------------------------------------------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------------------------------------------
@torch.no_grad()
def run(state):
    s = state
    if s.kind in ("mlp", "experts"):
        return {"y": s.part.forward(s.x)}
    if s.kind == "sample":
        return {"tokens": s.sampler.sample(s.logits, s.rows)}
    if s.kind == "attention":
        return {"y": s.part.forward(s.x, s.ctx, s.view), "k": s.view.k, "v": s.view.v}
    if s.kind == "latent":
        return {"y": s.part.forward(s.x, s.ctx, s.view), "k": s.view.k}
    if s.kind == "recurrence":
        y = s.part.forward(s.x, s.ctx, s.view)
        views = s.view if isinstance(s.view, tuple) else (s.view,)
        return {"y": y, "state": [v.state for v in views]}
    return {"logits": s.runner.step(s.entries), "kv": s.kv}


# ---------------------------------------------------------------------------------------------------------------
# the least that a pass has to move and to multiply
# ---------------------------------------------------------------------------------------------------------------
def _pairs(c):
    """(query, key) pairs that are visible, and the cached rows that are read."""
    pairs = rows = 0
    w = c.get("window", 0)
    for n, s in zip(_ints(c["lens"]), _ints(c["starts"])):
        for_each = [min(p + 1, w) if w else p + 1 for p in (s, s + n - 1)]
        if not w or s + n <= w:
            pairs += n * (2 * s + n + 1) // 2
        else:
            pairs += sum(min(p + 1, w) for p in range(s, s + n))
        rows += min(s, for_each[0])
    return pairs, rows


def work(case):
    c = case
    e = 4 if c.get("dtype") == "float32" else 2
    k = c["kind"]
    if k == "mlp":
        p = 3 * c["hidden"] * c["inter"]
        return {"bytes": e * (p + 2 * c["rows"] * c["hidden"]), "flops": 2 * p * c["rows"]}
    if k == "experts":
        p = 3 * c["hidden"] * c["inner"]
        hit = c["experts"] * (1 - (1 - c["top"] / c["experts"]) ** c["rows"])
        return {"bytes": e * (p * hit + c["experts"] * c["hidden"] + 2 * c["rows"] * c["hidden"]),
                "flops": 2 * c["rows"] * (p * c["top"] + c["experts"] * c["hidden"])}
    if k == "sample":
        return {"bytes": 4 * c["rows"] * (c["vocab"] + 1), "flops": 4 * c["rows"] * c["vocab"]}
    T = sum(_ints(c["lens"]))
    pairs, rows = _pairs(c)
    if k == "attention":
        nq, nkv = c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
        p = c["hidden"] * (2 * nq + 2 * nkv)
        return {"bytes": e * (p + 2 * T * c["hidden"] + 2 * (rows + T) * nkv), "flops": 2 * p * T + 4 * pairs * nq}
    if k == "latent":
        H, kv, row = c["heads"], c["kv_rank"], c["kv_rank"] + c["rot"]
        p = c["hidden"] * (c["q_rank"] + row + H * c["vdim"]) + c["q_rank"] * H * (c["nope"] + c["rot"]) + \
            H * kv * (c["nope"] + c["vdim"])
        return {"bytes": e * (p + 2 * T * c["hidden"] + (rows + T) * row), "flops": 2 * p * T + 2 * pairs * H * (row + kv)}
    if k == "recurrence":
        H, dk, dv = c["heads"], c["dim"], c["vdim"]
        n = len(_ints(c["lens"]))
        if c["mixer"] == "lightning_attention":
            p, keep = c["hidden"] * H * (2 * dk + 3 * dv), H * dk * dv
        else:
            ch = H * dv + 2 * c["groups"] * dk
            p, keep = c["hidden"] * (2 * H * dv + ch + H), H * dk * dv + 3 * ch
        return {"bytes": e * (p + 2 * T * c["hidden"]) + 8 * n * keep, "flops": 2 * p * T + 4 * T * H * dk * dv}
    nq, nkv = c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
    p = c["layers"] * (c["hidden"] * (2 * nq + 2 * nkv) + 3 * c["hidden"] * c["inter"])
    head, n = c["hidden"] * c["vocab"], len(_ints(c["lens"]))
    return {"bytes": e * (p + head + T * c["hidden"] + 2 * c["layers"] * (rows + T) * nkv) + 4 * n * c["vocab"],
            "flops": 2 * p * T + 2 * head * n + 4 * c["layers"] * pairs * nq}


def tolerance(case):
    c = case
    if c["kind"] == "sample":
        return "exact"
    if c.get("dtype") == "float32":
        return {"rel": 5e-6, "max": 2e-4}         # 1.3e-6 against float64
    if c["kind"] == "step":
        return {"rel": 1.8e-2, "max": 0.15}       # 4.3e-3
    if c["kind"] in ("attention", "latent"):
        return {"rel": 2.0e-2, "max": 0.15}       # 6.2e-3 with probabilities in bfloat16
    return {"rel": 1.2e-2, "max": 0.1}            # 2.3e-3 to 4.1e-3


# ---------------------------------------------------------------------------------------------------------------
# the same in float64
# ---------------------------------------------------------------------------------------------------------------
def _silu(x):
    return x * torch.sigmoid(x)


def _lin(x, w):
    return x @ w.to(F64).t()


def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.to(F64)


def _rotate(x, positions, theta, pairs):
    """x [T, heads, dim]; pairs: (2i, 2i + 1) turn together, else (i, i + dim / 2)."""
    dim = x.shape[-1]
    f = theta ** (-torch.arange(0, dim, 2, device=x.device, dtype=F64) / dim)
    a = positions.to(F64)[:, None] * f
    cos, sin = torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]
    if pairs:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * cos - v * sin, u * sin + v * cos], -1).flatten(-2)
    u, v = x[..., : dim // 2], x[..., dim // 2:]
    return torch.cat([u * cos - v * sin, u * sin + v * cos], -1)


def _spans(c):
    """(sequence, first flat row, tokens, tokens already there) in the order of the flat batch."""
    lens, starts, at = _ints(c["lens"]), _ints(c["starts"]), 0
    for s in _flat_order(c):
        yield s, at, lens[s], starts[s]
        at += lens[s]


def _softmax_rows(q, k, v, first, window, sink=None):
    """q [n, d] at positions first ..., k [m, d], v [m, e]; in slices of queries, to bound the memory."""
    out = torch.empty(q.shape[0], v.shape[1], device=q.device, dtype=F64)
    key = torch.arange(k.shape[0], device=q.device)
    for a in range(0, q.shape[0], 512):
        pos = first + torch.arange(a, min(a + 512, q.shape[0]), device=q.device)[:, None]
        s = q[a: a + 512] @ k.t()
        s = s.masked_fill((key > pos) | ((key <= pos - window) if window else (key < 0)), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.expand(s.shape[0], 1)], 1)
        p = torch.softmax(s, 1)[:, : k.shape[0]]
        out[a: a + 512] = p @ v
    return out


def _exact_attention(c, w, x, old_k, old_v, window):
    T, H, G, d = x.shape[0], c["heads"], c["kv_heads"], c["dim"]
    q, k, v = (_lin(x, w[n]).view(T, -1, d) for n in "qkv")
    out = torch.empty(T, H, d, device=x.device, dtype=F64)
    for s, at, n, start in _spans(c):
        pos = torch.arange(start, start + n, device=x.device)
        qs, ks = _rotate(q[at: at + n], pos, 500000.0, False), _rotate(k[at: at + n], pos, 500000.0, False)
        keys = torch.cat([old_k[s].to(F64), ks])
        vals = torch.cat([old_v[s].to(F64), v[at: at + n]])
        for h in range(H):
            g = h // (H // G)
            out[at: at + n, h] = _softmax_rows(qs[:, h] * d ** -0.5, keys[:, g], vals[:, g], start, window)
    return _lin(out.view(T, H * d), w["o"])


def _exact_mlp(w, x):
    return _lin(_silu(_lin(x, w["gate"])) * _lin(x, w["up"]), w["down"])


def _exact_experts(c, i):
    x = i["x"].to(F64)
    scores, ids = torch.softmax(_lin(x, i["router"]), 1).topk(c["top"], 1)
    y = torch.zeros_like(x)
    for e in range(c["experts"]):
        row, slot = torch.nonzero(ids == e, as_tuple=True)
        if row.numel():
            part = _exact_mlp({k: i[k][e] for k in ("gate", "up", "down")}, x[row])
            y.index_add_(0, row, part * scores[row, slot][:, None])
    return y


def _exact_latent(c, i):
    w, x = i["w"], i["x"].to(F64)
    T, H, kv, nope, rot = x.shape[0], c["heads"], c["kv_rank"], c["nope"], c["rot"]
    q = _lin(_rms(_lin(x, w["dq"]), w["dq_norm"], 1e-6), w["uq"]).view(T, H, nope + rot)
    a = _lin(x, w["dkv"])
    latent, shared = _rms(a[:, :kv], w["dkv_norm"], 1e-6), a[:, kv:]
    uk, uv = w["uk"].to(F64).view(H, nope, kv), w["uv"].to(F64).view(H, c["vdim"], kv)
    out = torch.empty(T, H, c["vdim"], device=x.device, dtype=F64)
    scale = (nope + rot) ** -0.5
    for s, at, n, start in _spans(c):
        pos = torch.arange(start, start + n, device=x.device)
        qr = _rotate(q[at: at + n, :, nope:], pos, 500000.0, True)
        kr = _rotate(shared[at: at + n, None], pos, 500000.0, True)[:, 0]
        rows = torch.cat([i["k"][s][:, 0].to(F64), torch.cat([latent[at: at + n], kr], 1)])
        for h in range(H):
            qh = torch.cat([q[at: at + n, h, :nope] @ uk[h], qr[:, h]], 1) * scale
            o = _softmax_rows(qh, rows, rows[:, :kv], start, c["window"], w["sink"][h].to(F64) if c["sink"] else None)
            out[at: at + n, h] = o @ uv[h].t()
    return _lin(out.view(T, H * c["vdim"]), w["o"])


def _exact_lightning(c, i):
    w, x = i["w"], i["x"].to(F64)
    T, H, dk, dv = x.shape[0], c["heads"], c["dim"], c["vdim"]
    q, k = (_silu(_lin(x, w[n])).view(T, H, dk) for n in "qk")
    v = _silu(_lin(x, w["v"])).view(T, H, dv)
    decay = torch.tensor(_decays(c), device=x.device, dtype=F64)[:, None, None]
    lens = _ints(c["lens"])
    state = torch.zeros(len(lens) + 1, H, dk, dv, device=x.device, dtype=F64)
    o = torch.empty(T, H, dv, device=x.device, dtype=F64)
    for s, at, n, _ in _spans(c):
        S = state[s]
        for t in range(at, at + n):
            S.mul_(decay).addcmul_(k[t][:, :, None], v[t][:, None, :])
            o[t] = torch.bmm(q[t][:, None, :], S)[:, 0]
    y = _rms(o.view(T, H * dv), w["norm"], 1e-6) * torch.sigmoid(_lin(x, w["g"]))
    return {"y": _lin(y, w["o"]), "state": [state]}


def _exact_state_space(c, i):
    w, x = i["w"], i["x"].to(F64)
    T, H, N, dv, G = x.shape[0], c["heads"], c["dim"], c["vdim"], c["groups"]
    inner, taps = H * dv, 4
    a = _lin(x, w["in"])
    z, u, dt = a[:, :inner], a[:, inner:-H], a[:, -H:]
    dt = torch.nn.functional.softplus(dt + w["dt_bias"].to(F64))
    decay = torch.exp(-torch.exp(w["a_log"].to(F64)) * dt)
    lens = _ints(c["lens"])
    state = torch.zeros(len(lens) + 1, H, N, dv, device=x.device, dtype=F64)
    tails = torch.zeros(len(lens) + 1, taps - 1, u.shape[1], device=x.device, dtype=F64)
    y = torch.empty(T, H, dv, device=x.device, dtype=F64)
    conv = w["conv"].to(F64)
    for s, at, n, _ in _spans(c):
        padded = torch.cat([torch.zeros(taps - 1, u.shape[1], device=x.device, dtype=F64), u[at: at + n]])
        mixed = _silu(sum(conv[:, j] * padded[j: j + n] for j in range(taps)) + w["conv_bias"].to(F64))
        tails[s] = padded[n:]
        xs = mixed[:, :inner].view(n, H, dv)
        B, C = (mixed[:, inner + j * G * N: inner + (j + 1) * G * N].view(n, G, N).repeat_interleave(H // G, 1) for j in (0, 1))
        B = B * dt[at: at + n, :, None]
        S = state[s]
        for t in range(n):
            S.mul_(decay[at + t][:, None, None]).addcmul_(B[t][:, :, None], xs[t][:, None, :])
            y[at + t] = torch.bmm(C[t][:, None, :], S)[:, 0]
        y[at: at + n] += w["d"].to(F64)[:, None] * xs
    y = (y.view(T, inner) * _silu(z)).view(T, G, inner // G)
    y = (y * torch.rsqrt(y.square().mean(-1, keepdim=True) + 1e-6)).view(T, inner) * w["norm"].to(F64)
    return {"y": _lin(y, w["o"]), "state": [state, tails]}


def _exact_step(c, i):
    w = i["w"]
    order = _flat_order(c)
    ids = torch.tensor([t for s in order for t in i["tokens"][s]], device="cuda")
    h = w["embed"][ids].to(F64)
    for n, layer in enumerate(w["layers"]):
        h = h + _exact_attention(c, layer["att"], _rms(h, layer["n1"], 1e-5), i["old"][n][0], i["old"][n][1], 0)
        h = h + _exact_mlp(layer["mlp"], _rms(h, layer["n2"], 1e-5))
    last = {s: at + n - 1 for s, at, n, _ in _spans(c)}
    rows = torch.tensor([last[s] for s in range(len(last))], device="cuda")
    return _lin(_rms(h[rows], w["norm"], 1e-5), w["head"])


@torch.no_grad()
def exact(case, seed):
    c = case
    if c["kind"] == "sample":
        return None
    i = _draw_inputs(c, seed)
    if c["kind"] == "mlp":
        return {"y": _exact_mlp(i["w"], i["x"].to(F64))}
    if c["kind"] == "experts":
        return {"y": _exact_experts(c, i)}
    if c["kind"] == "attention":
        return {"y": _exact_attention(c, i["w"], i["x"].to(F64), i["k"], i["v"], c["window"]), "k": None, "v": None}
    if c["kind"] == "latent":
        return {"y": _exact_latent(c, i), "k": None}
    if c["kind"] == "recurrence":
        return (_exact_lightning if c["mixer"] == "lightning_attention" else _exact_state_space)(c, i)
    return {"logits": _exact_step(c, i), "kv": None}
