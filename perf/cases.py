"""Work that programs have this engine do, as cases that can be timed and checked.

A case is a dict of plain values.  ``prepare`` makes what a program holds before the call (weights, engine or session,
requests whose prompts are in the cache), ``run`` is one pass through ``Engine.step`` or ``Session.generate``, ``exact`` the
same logits in 64 bits from the architectures' equations.  Four kinds of pass:

* ``prompt``: the prompts of ``requests`` requests (``tokens`` tokens the longest, down to an eighth where they are
  ``ragged``) in one step, logits of each one's last token; then the requests end.
* ``decode``: ``new`` steps of one token per request behind prompts that are in the cache already (each pass starts on the
  shared pages of the resident requests), logits of the last step.
* ``reply``: the prompts in one step, ``new`` steps of one token each, logits of the last one.  For models that keep a
  state per request, which can't be shared as pages can.
* ``generate``: ``Session.generate``: host ids in and out, prompts in portions of ``chunk`` tokens beside single tokens,
  sampling; the tokens.

Weights have the scales of a trained model: matrices N(0, 1 / inputs), what a sublayer adds to the stream small beside the
stream, gates and decays where trained models have them, routers that decide clearly (a token's embedding holds the
directions of the experts it goes to), and, where a head is tied to the embedding, a clear first choice of the next token.
"""
import hashlib
import math
from functools import lru_cache

import torch

import hfcpu_b200
from hfcpu_b200.config import config_from_dict
from hfcpu_b200.models import Model, build_model_specs
from hfcpu_b200.weights.loader import TensorSource

BLOCK = 16                  # tokens a cache page
DEVICE = "cuda:0"


# ---- model sizes (the benchmark's) -----------------------------------------------------------------------------------
QWEN2 = {
    "0.5b": dict(num_hidden_layers=24, hidden_size=896, num_attention_heads=14, num_key_value_heads=2, intermediate_size=4864,
                 vocab_size=151936, tie_word_embeddings=True),
    "7b": dict(num_hidden_layers=28, hidden_size=3584, num_attention_heads=28, num_key_value_heads=4, intermediate_size=18944,
               vocab_size=152064, tie_word_embeddings=False),
}
SIZES = {"w1024": dict(width=1024, heads=16, kv=4, dim=64, rot=32, gated=2736), "w2048": dict(width=2048, heads=16, kv=4, dim=128, rot=64, gated=5464),
         "w4096": dict(width=4096, heads=32, kv=8, dim=128, rot=128, gated=10920)}
VOCAB = 32768


def qwen2(size):
    return dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", max_position_embeddings=32768, rms_norm_eps=1e-6,
                rope_theta=1e6, use_sliding_window=False, hidden_act="silu", **QWEN2[size])


def _att(z, **more):
    return dict(heads=z["heads"], kv_heads=z["kv"], dim=z["dim"], vdim=z["dim"], scale=z["dim"] ** -0.5, **more)


def _latent(z, **more):
    return dict(heads=16 if more.pop("sixteen", True) else z["heads"], dim=z["dim"], rot_dim=32, vdim=z["dim"], q_rank=3 * z["width"] // 8,
                kv_rank=96, scale=(z["dim"] + 32) ** -0.5, **more)


def _top(z, name, **more):
    return dict(architecture=name, vocab=VOCAB, width=z["width"], norm=dict(eps=1e-6), max_positions=8192, **more)


def manapel(size):
    z = SIZES[size]
    n, top = (16, 2) if size == "w1024" else (32, 4)
    ff = z["width"] // 2
    rot = dict(dims=z["rot"], base=10000.0)
    moe = dict(kind="moe", router=dict(experts=n, top=top), expert=dict(ff=ff), shared=dict(ff=2 * ff))
    dense = dict(kind="dense", ff=(2 * (top * ff + 2 * ff) // 3 + 7) // 8 * 8)
    layers = [dict(type="attention", mixer=_att(z, rot=rot, **({"kv_from": i - 1} if i % 2 else {})), mlp=moe if i else dense)
              for i in range(4 if size == "w4096" else 8)]
    return dict(_top(z, "Manapel", logit_scale=1.0, layers=layers), norm=dict(eps=1e-5))


def peludra(size):
    z = SIZES[size]
    chunk = 1024 if size == "w1024" else 2048
    yarn = dict(factor=4.0, original=4096, fast=32.0, slow=1.0)
    lat = dict(type="latent_attention", mixer=_latent(z, mask=dict(size=chunk // 2), rot=dict(dims=32, base=10000.0, scaling=yarn)))
    att = dict(type="attention", mixer=_att(z, mask=dict(size=chunk), v_mix=True))
    return _top(z, "Peludra", embedding=dict(scale=z["width"] ** 0.5, bigram=dict(buckets=65521, mul_prev=1000003, mul_cur=31)),
                layers=[dict(att if i % 3 == 1 else lat, mlp=dict(kind="dense", ff=4 * z["width"])) for i in range(3 if size == "w4096" else 9)])


def mokisun(size):
    z = SIZES[size]
    small = size == "w1024"
    rheads, rdim, rank = z["width"] // 128, 64 if small else 128, z["width"] // 16
    att = _att(z, mask=dict(size=512 if small else 1024))
    kinds = (dict(type="gla", mixer=dict(heads=rheads, dim=rdim, vdim=128, tau=16.0, a_rank=rank)),
             dict(type="attention", mixer=dict(att, rot=dict(dims=z["rot"], base=10000.0))),
             dict(type="parallel", mixer=dict(left=att, left_scale=1.0, right_scale=1.0, right=dict(
                 heads=rheads, kv_heads=rheads // 2, dim=rdim, vdim=128, conv=4, a_rank=rank, g_rank=rank))))
    router = dict(experts=14, identity=2, top=2, scale=1.0, groups=dict(count=4, keep=2)) if small else \
        dict(experts=28, identity=4, top=4, scale=1.0, groups=dict(count=8, keep=4))
    mlp = dict(kind="moe", expert=dict(ff=z["width"] // 2), router=router)
    return _top(z, "Mokisun", streams=2, layers=[dict(kinds[i % 3], mlp=mlp) for i in range(3 if size == "w4096" else 6)])


def silupel(size):
    z = SIZES[size]
    att = _att(z, mask=dict(size=1024 if size == "w1024" else 2048), softcap=30.0, rot=dict(
        dims=z["rot"], base=500000.0, scaling=dict(factor=8.0, low=1.0, high=4.0, original=8192)))
    kinds = (dict(type="latent_attention", mixer=_latent(z, rot=dict(dims=32, base=10000.0))),
             dict(type="mingru", mixer=dict(width=z["width"])), dict(type="attention", mixer=att))
    mlp = dict(kind="dense", ff=z["gated"])
    return _top(z, "Silupel", layers=[dict(kinds[i % 3], mlp=mlp) for i in range(6)], loop=dict(start=3, stop=6, times=2))


def _decays(n):
    return [1.0 - 2.0 ** (-5.0 - 4.0 * i / n) for i in range(n)]


def tupalorn(size):
    z = SIZES[size]
    rdim = 64 if size == "w1024" else 128
    n = z["width"] // rdim
    att = _att(z, mask=dict(size=1024))
    kinds = (dict(type="mamba2", mixer=dict(heads=z["width"] // 32, vdim=64, state=128, groups=1, conv=4, norm_groups=1)),
             dict(type="retention", mixer=dict(heads=n, dim=rdim, vdim=rdim, decay=_decays(n), rot=dict(dims=rdim, base=10000.0))),
             dict(type="attention", mixer=att))
    layers = [dict(kinds[i % 3], mlp=dict(kind="dense", ff=z["gated"], limit=7.0)) for i in range(9)]
    layers[8] = dict(layers[8], mixer=dict(att, kv_from=5))
    return _top(z, "Tupalorn", logit_softcap=30.0, layers=layers)


def birizen(size):
    z = SIZES[size]
    ldim = 64 if size == "w1024" else 128
    n = z["width"] // ldim
    light = dict(type="lightning", mixer=dict(heads=n, dim=ldim, vdim=ldim, decay=_decays(n)))
    lat = dict(type="latent_attention", mixer=_latent(z, sixteen=False, rot=dict(
        dims=32, base=10000.0, scaling=dict(factor=4.0, original=4096, fast=32.0, slow=1.0))))
    ff = 3 * z["width"] // 8
    router = dict(experts=16, top=2, groups=dict(count=4, keep=2)) if size == "w1024" else dict(experts=32, top=4, groups=dict(count=8, keep=4))
    mlp = dict(kind="moe", expert=dict(ff=ff, limit=7.0), shared=dict(ff=2 * ff, limit=7.0), router=router)
    return _top(z, "Birizen", layers=[dict((light, lat)[i % 2], mlp=mlp) for i in range(4)], loop=dict(start=0, stop=2, times=3))


ARCHITECTURES = {f.__name__: f for f in (qwen2, manapel, peludra, mokisun, silupel, tupalorn, birizen)}


def _config(case):
    return ARCHITECTURES[case["model"]](case["size"])


# ---- the cases -------------------------------------------------------------------------------------------------------
def _case(name, model, size, kind, requests, tokens, new=0, ragged=False, dtype="bfloat16", chunk=0):
    c = dict(model=model, size=size, kind=kind, requests=requests, tokens=tokens, new=new, ragged=ragged, dtype=dtype, chunk=chunk)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user in a chat with a small model: launches and latency
        _case("small_chat", "qwen2", "0.5b", "decode", 1, 208, new=8),
        # the headline: eight requests decode behind 2,048-token prompts
        _case("decode_8", "qwen2", "7b", "decode", 8, 2048, new=8),
        # a loaded server: 64 requests of very different lengths decode
        _case("decode_64", "qwen2", "7b", "decode", 64, 2048, new=8, ragged=True),
        # the time to the first token of a long prompt
        _case("prompt_2048", "qwen2", "7b", "prompt", 1, 2048),
        # the whole engine: scheduler, prompts in portions beside decoding requests, sampling, host ids in and out
        _case("serving", "qwen2", "0.5b", "generate", 32, 1024, new=24, ragged=True, chunk=256),
        # the true 32-bit run of a prompt of odd length and a short answer (checking a checkpoint)
        _case("float32", "qwen2", "0.5b", "reply", 1, 333, new=4, dtype="float32"),
        # a prompt through routed experts
        _case("experts_prompt", "manapel", "w2048", "prompt", 1, 2048),
        # answers to short prompts under latent and chunked attention
        _case("latent_reply", "peludra", "w2048", "reply", 8, 301, new=16, ragged=True),
        # a few prompts of odd lengths through gated linear attention, delta rule and routed experts
        _case("linear_prompts", "mokisun", "w2048", "prompt", 4, 777, ragged=True),
        # one user's answer from a small looped model with minGRU layers
        _case("looped_chat", "silupel", "w1024", "reply", 1, 97, new=24),
        # a long prompt through state-space, retention and windowed attention layers
        _case("states_prompt", "tupalorn", "w2048", "prompt", 1, 4000),
        # a batch's answers from lightning and latent attention with gated experts
        _case("lightning_reply", "birizen", "w4096", "reply", 16, 250, new=16, ragged=True),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    model = rng.choice(["qwen2"] * 6 + ["manapel", "peludra", "mokisun", "silupel", "tupalorn", "birizen"])
    if model == "qwen2":
        size, kind = rng.choice(["0.5b", "7b"]), rng.choice(["prompt", "decode", "decode", "reply", "generate"])
    else:
        size, kind = rng.choice(sorted(SIZES)), rng.choice(["prompt", "reply", "decode" if model == "manapel" else "reply"])
    if kind == "generate":
        size = "0.5b" if model == "qwen2" else size
        return _case("", model, size, kind, _log_uniform(rng, 1, 32), _log_uniform(rng, 8, 1024), new=rng.randint(4, 24), ragged=rng.random() < 0.7,
                     chunk=rng.choice([128, 256, 512, 1024]))
    if rng.random() < 0.12 and size in ("0.5b", "w1024"):
        return _case("", model, size, "reply", rng.randint(1, 3), _log_uniform(rng, 5, 160), new=rng.randint(1, 4), ragged=rng.random() < 0.5, dtype="float32")
    if kind == "decode":
        return _case("", model, size, kind, _log_uniform(rng, 1, 64), BLOCK * _log_uniform(rng, 1, 96), new=rng.randint(2, 7), ragged=rng.random() < 0.6)
    requests = _log_uniform(rng, 1, 12)
    longest = 2048 // requests if size == "7b" else min(4000 // requests, 3000)
    return _case("", model, size, kind, requests, _log_uniform(rng, 4, max(longest, 8)), new=rng.randint(2, 16) if kind == "reply" else 0, ragged=rng.random() < 0.6)


# ---- weights, by name and seed ---------------------------------------------------------------------------------------
def _generator(seed, name):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:7], "little"))
    return g


def _normal(seed, name, shape, std=1.0, mean=0.0):
    return torch.empty(shape, dtype=torch.float32, device=DEVICE).normal_(mean, std, generator=_generator(seed, name))


def _uniform(seed, name, shape, lo, hi):
    return torch.empty(shape, dtype=torch.float32, device=DEVICE).uniform_(lo, hi, generator=_generator(seed, name))


def _router_rows(seed, name, shape):
    return _normal(seed, name, shape, shape[1] ** -0.5)


def _embedding(cfg, seed, name, shape):
    x = _normal(seed, name, shape)
    for i, layer in enumerate(cfg.get("layers", ())):
        mlp = layer.get("mlp") or {}
        if mlp.get("kind") != "moe":
            continue
        r = mlp["router"]
        n, top = r["experts"] + r.get("identity", 0), r["top"]
        count, keep = (r["groups"]["count"], r["groups"]["keep"]) if r.get("groups") else (n, n)
        g = _generator(seed, f"choices.{i}")
        group = torch.rand((shape[0], count), device=DEVICE, generator=g).argsort(-1)
        member = torch.rand((shape[0], count, n // count), device=DEVICE, generator=g).argsort(-1)
        rows = _router_rows(seed, f"l{i}.mlp.router", (n, shape[1]))
        used = min(keep, top)
        for j in range(top):
            gj = group[:, j % used]
            x += 8.0 * rows[gj * (n // count) + member[torch.arange(shape[0], device=DEVICE), gj, j // used]]
    return x


def _weight(cfg, seed, name, shape):
    """The tensor ``name`` in float32; what is stored is its rounding to the run's type."""
    last = name.rsplit(".", 1)[-1]
    layers = cfg.get("num_hidden_layers") or len(cfg["layers"])
    if name in ("embed", "model.embed_tokens.weight"):
        return _embedding(cfg, seed, name, shape) * (1.0 if cfg.get("architecture") != "Peludra" else shape[1] ** -0.5)
    if name == "bigram":
        return _normal(seed, name, shape, 0.3)
    if last == "router":
        return _router_rows(seed, name, shape) * (0.6 if cfg["architecture"] == "Birizen" else 1.0)
    if name == "loop.in":
        eye = torch.eye(shape[0], device=DEVICE)
        return _normal(seed, name, shape, 0.2 * shape[1] ** -0.5) + 0.6 * torch.cat([eye, eye], 1)
    if name == "loop.step":
        return _normal(seed, name, shape, 0.1)
    if last == "conv":
        return _normal(seed, name, shape, 0.5)
    if last == "mix" and len(shape) == 2:
        return _normal(seed, name, shape, 0.05, 0.5)
    if len(shape) == 2:
        into_stream = last in ("o", "down") or name.endswith(("o_proj.weight", "down_proj.weight"))
        return _normal(seed, name, shape, (layers ** -0.5 if into_stream else 1.0) * shape[1] ** -0.5)
    if last == "alpha":
        return _uniform(seed, name, shape, 0.4, 0.9)
    if last in ("ls1", "ls2", "norm1b", "norm2b"):
        return _normal(seed, name, shape, 0.02, 0.2)
    if last == "A_log":
        return _uniform(seed, name, shape, 1.0, 16.0).log()
    if last == "dt_bias":
        return _uniform(seed, name, shape, math.log(1e-3), math.log(1e-1)).exp().expm1().log()
    if last == "sink":
        return _normal(seed, name, shape)
    if last == "correction":
        return _normal(seed, name, shape, 0.01)
    if name.endswith("a2.b"):
        return _normal(seed, name, shape, 1.0, 2.0)
    if last in ("b", "bias"):
        return _normal(seed, name, shape, 0.1)
    if last in ("vmix", "shift", "in"):
        return _normal(seed, name, shape, 0.05, 0.5)
    if cfg.get("architecture") == "Peludra" and last in ("norm1", "norm2", "norm") and ".mix." not in name:
        return _normal(seed, name, shape, 0.1)            # these norms' weights are stored around zero
    tied = cfg.get("tie_word_embeddings") or cfg.get("architecture") in ("Tupalorn", "Birizen")
    scale = cfg.get("hidden_size", cfg.get("width")) ** -0.5 if tied and name in ("model.norm.weight", "final.norm") else 1.0
    return _normal(seed, name, shape, 0.1, 1.0) * scale


@lru_cache(maxsize=64)
def _specs(model, size):
    return {s.name: tuple(s.shape) for s in build_model_specs(config_from_dict(ARCHITECTURES[model](size)))}


def _store(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


class _Weights(TensorSource):
    """The weights as the model asks for them, one tensor at a time."""

    def __init__(self, case, seed):
        super().__init__(_store(case), torch.device(DEVICE))
        self.case, self.cfg, self.seed, self.shapes = case, _config(case), seed, _specs(case["model"], case["size"])

    def names(self):
        return self.shapes.keys()

    def __contains__(self, name):
        return name in self.shapes

    def meta(self, name):
        return _store(self.case), self.shapes[name]

    def _make(self, name):
        return _weight(self.cfg, self.seed, name, self.shapes[name]).to(_store(self.case))


# ---- a pass ----------------------------------------------------------------------------------------------------------
def _lengths(case):
    """Prompt lengths: all ``tokens``, or spread evenly from ``tokens`` down to an eighth of it.  Resident prompts fill
    whole pages, as shared ones do."""
    n, longest = case["requests"], case["tokens"]
    lens = [max(1, round(longest * (1 - 7 / 8 * i / max(n - 1, 1)))) if case["ragged"] else longest for i in range(n)]
    return [max(BLOCK, L // BLOCK * BLOCK) for L in lens] if case["kind"] == "decode" else lens


def _tokens(case, seed):
    """(prompts, the tokens fed behind each) as lists of ids."""
    cfg = _config(case)
    g = torch.Generator().manual_seed(seed + 7919)
    ids = lambda n: torch.randint(0, cfg.get("vocab_size", cfg.get("vocab")), (n,), generator=g).tolist()  # noqa: E731
    return [ids(n) for n in _lengths(case)], [ids(case["new"]) for _ in range(case["requests"])]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    s.prompts, s.fed = _tokens(case, seed)
    model = Model(config_from_dict(_config(case)), _store(case), torch.device(DEVICE)).bind(_Weights(case, seed))
    n, longest = case["requests"], max(len(p) for p in s.prompts) + case["new"] + 1
    pages = sum((len(p) + case["new"]) // BLOCK + 2 for p in s.prompts)
    if case["kind"] == "generate":
        s.session = hfcpu_b200.Session(model, kv_block=BLOCK, kv_pages=pages, max_seqs=n, ctx_max=longest, max_batched_tokens=max(case["chunk"], n),
                                       batch=case["chunk"])
        return s
    resident = case["kind"] == "decode"
    s.engine = hfcpu_b200.Engine(model, block_size=BLOCK, num_pages=pages * 2 if resident else pages, max_requests=2 * n if resident else n, ctx_max=longest)
    if resident:
        for i, p in enumerate(s.prompts):
            s.engine.add_request(("resident", i))
            s.engine.step([hfcpu_b200.StepEntry(("resident", i), p)])
    return s


def run(s):
    case, n = s.case, s.case["requests"]
    if case["kind"] == "generate":
        done = s.session.generate(s.prompts, temp=0.7, seed=5, max_tokens=case["new"], eos_ids=[], prefix_cache=False)
        return {"tokens": torch.tensor([c[0].tokens for c in done])}
    eng, entry = s.engine, hfcpu_b200.StepEntry
    for i in range(n):
        eng.add_request(i)
    if case["kind"] == "decode":
        for i in range(n):
            eng.fork_request(("resident", i), i, len(s.prompts[i]))
    else:
        logits = eng.step([entry(i, p, [len(p) - 1]) for i, p in enumerate(s.prompts)])
    for j in range(case["new"]):
        logits = eng.step([entry(i, [s.fed[i][j]], [0]) for i in range(n)])
    for i in range(n):
        eng.finish_request(i)
    c = _checked(case)
    return {"checked": logits[:c], "others": logits[c:]} if c < n else {"checked": logits}


def _checked(case):
    """How many of the requests ``exact`` computes: a few seconds' worth."""
    if case["kind"] == "generate":
        return 0
    each = 2.0 * _active(case) * max(_lengths(case)) + 1e12
    return max(1, min(case["requests"], int(8e13 / each)))


# ---- what a pass can't do without ------------------------------------------------------------------------------------
def _runs(cfg):
    """How often each layer runs."""
    n, loop = cfg.get("num_hidden_layers") or len(cfg["layers"]), cfg.get("loop")
    return [loop["times"] if loop and loop["start"] <= i < loop["stop"] else 1 for i in range(n)]


def _layer_of(name):
    name = name.replace("model.layers.", "l")
    head = name.split(".", 1)[0]
    return int(head[1:]) if head[0] == "l" and head[1:].isdigit() else None


def _router_of(cfg, layer):
    mlp = cfg["layers"][layer].get("mlp") or {} if "layers" in cfg else {}
    return mlp["router"] if mlp.get("kind") == "moe" else None


def _is_expert(name):
    part = name.split(".")
    return len(part) > 2 and part[1] == "mlp" and part[2][0] == "e" and part[2][1:].isdigit()


def _matrices(case):
    """(name, values, layer) of every matrix a step multiplies by, the head left out."""
    return [(n, math.prod(s), _layer_of(n)) for n, s in _specs(case["model"], case["size"]).items()
            if len(s) == 2 and n not in ("embed", "bigram", "head", "lm_head.weight", "model.embed_tokens.weight", "loop.step") and not n.endswith((".conv", "hc1.mix", "hc2.mix"))]


def _active(case):
    """Values of the matrices a token goes through (the head left out), each as often as it does."""
    cfg = _config(case)
    runs, total = _runs(cfg), 0.0
    for name, n, layer in _matrices(case):
        share = 1.0
        if _is_expert(name):
            r = _router_of(cfg, layer)
            share = r["top"] / (r["experts"] + r.get("identity", 0))
        total += n * share * (runs[layer] if layer is not None else cfg["loop"]["times"] if name == "loop.in" else 1)
    return total


def _read(case, tokens):
    """Values of the weights a step of ``tokens`` tokens reads, each once; of a layer's experts those that uniform choices hit."""
    cfg = _config(case)
    total = float(_vocab(cfg) * _width(cfg))
    for name, n, layer in _matrices(case):
        if _is_expert(name):
            r = _router_of(cfg, layer)
            n *= 1 - (1 - 1 / (r["experts"] + r.get("identity", 0))) ** (tokens * r["top"])
        total += n
    return total


def _vocab(cfg):
    return cfg.get("vocab_size", cfg.get("vocab"))


def _width(cfg):
    return cfg.get("hidden_size", cfg.get("width"))


def _attentions(cfg):
    """Per layer run with attention: (values per key and value a token leaves, operations per (query, key) pair, window or 0, chunk or 0)."""
    if "layers" not in cfg:
        d = cfg["hidden_size"] // cfg["num_attention_heads"]
        return [(2 * cfg["num_key_value_heads"] * d, 4 * cfg["num_attention_heads"] * d, 0, 0)] * cfg["num_hidden_layers"]
    out = []
    for layer, runs in zip(cfg["layers"], _runs(cfg)):
        m = layer["mixer"].get("left", layer["mixer"])
        size = (m.get("mask") or {}).get("size", 0)
        if layer["type"] == "latent_attention":
            row = m["kv_rank"] + m["rot_dim"]
            out += [(row, 2 * m["heads"] * (row + m["kv_rank"]), size, 0)] * runs
        elif "kv_heads" in m and layer["type"] in ("attention", "parallel"):
            chunked = cfg["architecture"] in ("Peludra", "Silupel")
            kept = m["kv_heads"] * (m["dim"] + (0 if layer["type"] == "parallel" else m["vdim"]))
            out += [(kept, 2 * m["heads"] * (m["dim"] + m["vdim"]), 0 if chunked else size, size if chunked else 0)] * runs
    return out


def _seen(pos, window, chunk):
    return min(pos + 1, window) if window else pos % chunk + 1 if chunk else pos + 1


def work(case):
    cfg, lens, new = _config(case), _lengths(case), case["new"]
    item = 4 if case["dtype"] == "float32" else 2
    V, E, n = _vocab(cfg), _width(cfg), case["requests"]
    active, attentions = _active(case), _attentions(cfg)
    prompt_steps = 0 if case["kind"] == "decode" else max(1, math.ceil(sum(lens) / max(case["chunk"], n))) if case["kind"] == "generate" else 1
    single_steps = max(0, new - 1) if case["kind"] == "generate" else new
    run_tokens = [(0 if case["kind"] == "decode" else L, L, L + single_steps) for L in lens]       # (tokens computed of the prompt, prompt, end)
    tokens = sum(p + single_steps for p, _, _ in run_tokens)
    rows = n * (single_steps + (1 if prompt_steps else 0))
    flops, nbytes = 2.0 * active * tokens + 2.0 * rows * V * E, 0.0
    if prompt_steps:
        nbytes += item * (prompt_steps * _read(case, sum(lens) / prompt_steps))
    nbytes += item * single_steps * _read(case, n) + 4.0 * rows * V + tokens * E * item
    for kept, ops, window, chunk in attentions:
        for p, L, end in run_tokens:
            first = L - p
            pairs = sum(_seen(t, window, chunk) for t in range(first, end))
            flops += float(ops) * pairs
            nbytes += item * kept * ((end - first) + sum(_seen(t, window, chunk) for t in range(L, end)))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "generate":
        return {"differ": 0.01}              # a draw within rounding of the border between two tokens
    # four times what the runs are off the 64-bit logits: up to 1.1e-6 in float32, 3.5e-3 in bfloat16
    if case["dtype"] == "float32":
        return {"rel": 5e-6, "max": 5e-5}
    return {"rel": 0.014, "max": 0.14}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------
def exact(case, seed):
    c = _checked(case)
    if not c:
        return None
    source, prompts, fed = _Weights(case, seed), *_tokens(case, seed)
    W = lambda name: source._make(name).double()  # noqa: E731
    rows = [_forward(source.cfg, W, prompts[i] + fed[i]) for i in range(c)]
    out = {"checked": torch.stack(rows)}
    return out if c == case["requests"] else dict(out, others=None)


def _rms(x, eps):
    return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt()


def _layer_norm(x, w, eps):
    d = x - x.mean(-1, keepdim=True)
    return _rms(d, eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _clamped(g, u, limit):
    g = g.clamp(max=limit)
    return g * torch.sigmoid(1.702 * g) * (u.clamp(-limit, limit) + 1.0)


def _rotate(x, rot, interleaved):
    """x [T, heads, d]: the first ``dims`` of each head turn by position * frequency, in neighbouring pairs or half apart."""
    if not rot or not rot["dims"]:
        return x
    n, base, size = rot["dims"], float(rot["base"]), 1.0
    i = torch.arange(n // 2, dtype=torch.float64, device=x.device)
    f = base ** (-2.0 * i / n)
    sc = rot.get("scaling")
    if sc and "fast" in sc:
        at = lambda turns: n * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), n - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f, size = f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    elif sc:
        wave = 2 * math.pi / f
        s = ((sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])).clamp(0, 1)
        f = (1 - s) * f / sc["factor"] + s * f
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * f
    c, s = size * a.cos(), size * a.sin()
    out = x.clone()
    first, second = (slice(0, n, 2), slice(1, n, 2)) if interleaved else (slice(0, n // 2), slice(n // 2, n))
    u, v = x[..., first], x[..., second]
    out[..., first], out[..., second] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, window=0, chunk=0, sink=None, slopes=None, cap=0.0, factors=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H * dv]."""
    T, H = q.shape[:2]
    pos = torch.arange(T, device=q.device)
    far = pos[:, None] - pos[None, :]
    see = far >= 0
    if window:
        see = see & (far < window)
    if chunk:
        see = see & (pos[:, None] // chunk == pos[None, :] // chunk)
    out = []
    for h in range(H):
        g = h // (H // k.shape[1])
        s = q[:, h] @ k[:, g].T * scale
        if factors is not None:
            s = s * factors[h]
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes[h] * far
        s = s.masked_fill(~see, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out.append(torch.softmax(s, -1)[:, :T] @ v[:, g])
    return torch.stack(out, 1).reshape(T, -1)


def _scan(decay, k, v, q, beta=None):
    """Per head S <- decay S + k v^T (with ``beta`` the delta rule's k beta (v - S^T k)^T), o = S^T q; decay [T, H, 1 or d]."""
    T, H, d = k.shape
    S, out = torch.zeros((H, d, v.shape[2]), dtype=k.dtype, device=k.device), torch.empty_like(v)
    for t in range(T):
        S = decay[t][..., None] * S
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hdv,hd->hv", S, q[t])
    return out


def _conv(x, w, b=None):
    taps = w.shape[1]
    pad = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    y = sum(pad[i:i + x.shape[0]] * w[:, i] for i in range(taps))
    return y if b is None else y + b


def _latent_attention(m, W, p, h, eps, interleaved, sink):
    T, H, d, R = h.shape[0], m["heads"], m["dim"], m["kv_rank"]
    cq = _rms(h @ W(p + ".dq").T, eps) * W(p + ".dq.norm")
    q = (cq @ W(p + ".uq").T).view(T, H, -1)
    down = h @ W(p + ".dkv").T
    c = _rms(down[:, :R], eps) * W(p + ".dkv.norm")
    k = (c @ W(p + ".uk").T).view(T, H, d)
    v = (c @ W(p + ".uv").T).view(T, H, -1)
    turned = _rotate(down[:, None, R:], m["rot"], interleaved).expand(T, H, -1)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], m["rot"], interleaved)], -1)
    return _attend(q, torch.cat([k, turned], -1), v, m["scale"], window=(m.get("mask") or {}).get("size", 0), sink=W(p + ".sink") if sink else None)


def _routed(mlp, W, p, h, ids, weights, expert):
    y = torch.zeros_like(h)
    for e in ids.unique().tolist():
        rows, at = (ids == e).nonzero(as_tuple=True)
        y[rows] += weights[rows, at][:, None] * (expert(f"{p}.e{e}", h[rows]) if e < mlp["router"]["experts"] else h[rows])
    return y


def _choose(choice, r, best):
    """The ``top`` largest choice scores within the groups kept; a group counts as much as its ``best`` best together."""
    if r.get("groups"):
        count, keep = r["groups"]["count"], r["groups"]["keep"]
        value = choice.view(choice.shape[0], count, -1).topk(best, -1).values.sum(-1)
        kept = torch.zeros_like(value, dtype=torch.bool).scatter_(1, value.topk(keep, -1).indices, True)
        choice = choice.masked_fill(~kept.repeat_interleave(choice.shape[1] // count, 1), -math.inf)
    return choice.topk(r["top"], -1).indices


def _forward(cfg, W, ids):
    """Logits of the last of ``ids``."""
    ids = torch.tensor(ids, device=DEVICE)
    return globals()["_" + cfg.get("architecture", "Qwen2").lower() + "_forward"](cfg, W, ids)


def _qwen2_forward(cfg, W, ids):
    H, G, eps, T = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["rms_norm_eps"], ids.shape[0]
    d = cfg["hidden_size"] // H
    rot = dict(dims=d, base=cfg["rope_theta"])
    x = W("model.embed_tokens.weight")[ids]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * W(p + "input_layernorm.weight")
        q, k, v = ((h @ W(f"{p}self_attn.{n}_proj.weight").T + W(f"{p}self_attn.{n}_proj.bias")).view(T, -1, d) for n in "qkv")
        x = x + _attend(_rotate(q, rot, False), _rotate(k, rot, False), v, d ** -0.5) @ W(p + "self_attn.o_proj.weight").T
        h = _rms(x, eps) * W(p + "post_attention_layernorm.weight")
        x = x + (_silu(h @ W(p + "mlp.gate_proj.weight").T) * (h @ W(p + "mlp.up_proj.weight").T)) @ W(p + "mlp.down_proj.weight").T
    head = W("model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight")
    return head @ (_rms(x[-1], eps) * W("model.norm.weight"))


def _heads(m, W, p, h, names="qkv", bias=False):
    return [(h @ W(f"{p}.{n}").T + (W(f"{p}.{n}.b") if bias else 0.0)).view(h.shape[0], -1, m["vdim"] if n == "v" else m["dim"]) for n in names]


def _dyt(x, W, name):
    return torch.tanh(W(name + ".alpha") * x) * W(name) + W(name + ".b")


def _manapel_forward(cfg, W, ids):
    eps, x, kept = cfg["norm"]["eps"], W("embed")[ids], {}
    square = lambda q, h: torch.relu(h @ W(q + ".up").T).square() @ W(q + ".down").T  # noqa: E731
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}", layer["mixer"], layer["mlp"]
        h = _dyt(x, W, p + ".norm1")
        q, = _heads(m, W, p + ".mix", h, "q", True)
        if m.get("kv_from") is None:
            k, v = _heads(m, W, p + ".mix", h, "kv", True)
            kept[i] = _rms(_rotate(k, m["rot"], False), eps), v
        k, v = kept[m.get("kv_from", i)]
        x = x + _dyt(_attend(_rms(_rotate(q, m["rot"], False), eps), k, v, m["scale"]) @ W(p + ".mix.o").T, W, p + ".norm1b")
        h, p = _dyt(x, W, p + ".norm2"), p + ".mlp"
        if mlp["kind"] == "dense":
            y = (torch.relu(h @ W(p + ".gate").T) * (h @ W(p + ".up").T)) @ W(p + ".down").T
        else:
            z, chosen = (h @ W(p + ".router").T + W(p + ".router.b")).topk(mlp["router"]["top"], -1)
            y = _routed(mlp, W, p, h, chosen, torch.softmax(z, -1), square) + square(p + ".shared", h)
        x = x + _dyt(y, W, f"l{i}.norm2b")
    return W("head") @ _dyt(x[-1], W, "final.norm") * cfg["logit_scale"]


def _peludra_forward(cfg, W, ids):
    eps, e = cfg["norm"]["eps"], cfg["embedding"]
    b = e["bigram"]
    pair = torch.cat([ids.new_tensor([b["buckets"]]), (ids[:-1] * b["mul_prev"] + ids[1:] * b["mul_cur"]) % b["buckets"]])
    x, first = W("embed")[ids] * e["scale"] + W("bigram")[pair], None
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix", layer["mixer"]
        h = _rms(x, eps) * (1 + W(f"l{i}.norm1"))
        if layer["type"] == "attention":
            q, k, own = _heads(m, W, p, h)
            mix = W(p + ".vmix")
            first, v = (own, own) if first is None else (first, (1 - mix) * own + mix * first)
            y = _attend(_rms(q, eps) * W(p + ".q.norm"), _rms(k, eps) * W(p + ".k.norm"), v, m["scale"], chunk=m["mask"]["size"])
        else:
            y = _latent_attention(m, W, p, h, eps, True, False)
        x = x + y @ W(p + ".o").T
        h = _rms(x, eps) * (1 + W(f"l{i}.norm2"))
        x = x + torch.relu(h @ W(f"l{i}.mlp.up").T).square() @ W(f"l{i}.mlp.down").T
    return W("head") @ (_rms(x[-1], eps) * (1 + W("final.norm")))


def _mokisun_forward(cfg, W, ids):
    eps, T = cfg["norm"]["eps"], ids.shape[0]

    def biased(m, p, h):
        q, k = _heads(m, W, p, h, "qk")
        slopes = 2.0 ** (-8.0 * torch.arange(1, m["heads"] + 1, dtype=torch.float64, device=h.device) / m["heads"])
        zero = torch.zeros(m["heads"], dtype=h.dtype, device=h.device)
        return _attend(q, k, k, m["scale"], window=m["mask"]["size"], sink=zero, slopes=slopes) @ W(p + ".o").T

    def delta(m, p, h):
        H, d = m["heads"], m["dim"]
        q, k, v = (_silu(_conv(h @ W(f"{p}.{n}").T, W(f"{p}.{n}.conv"))).view(T, -1, m["vdim"] if n == "v" else d) for n in "qkv")
        unit = lambda a: (a * (a.square().sum(-1, keepdim=True) + 1e-6).rsqrt()).repeat_interleave(H // m["kv_heads"], 1)  # noqa: E731
        dt = torch.nn.functional.softplus((h @ W(p + ".a1").T) @ W(p + ".a2").T + W(p + ".dt_bias")).view(T, H, d)
        o = _scan((-W(p + ".A_log").exp()[:, None] * dt).exp(), unit(k), v, unit(q) * d ** -0.5, torch.sigmoid(h @ W(p + ".b").T))
        gate = torch.sigmoid((h @ W(p + ".g1").T) @ W(p + ".g2").T)
        return ((_rms(o, eps) * W(p + ".norm")).reshape(T, -1) * gate) @ W(p + ".o").T

    def gla(m, p, h):
        q, k, v = _heads(m, W, p, h)
        z = (h @ W(p + ".a1").T) @ W(p + ".a2").T + W(p + ".a2.b")
        o = _scan((torch.nn.functional.logsigmoid(z) / m["tau"]).exp().view(T, -1, m["dim"]), k, v, q * m["dim"] ** -0.5)
        return ((_rms(o, eps) * W(p + ".norm")).reshape(T, -1) * _silu(h @ W(p + ".g").T)) @ W(p + ".o").T

    def mixer(layer, p, h):
        m = layer["mixer"]
        if layer["type"] == "gla":
            return gla(m, p, h)
        if layer["type"] == "parallel":
            return m["left_scale"] * biased(m["left"], p + ".left", h) + m["right_scale"] * delta(m["right"], p + ".right", h)
        q, k, v = _heads(m, W, p, h)
        return _attend(_rotate(q, m["rot"], True), _rotate(k, m["rot"], True), v, m["scale"], window=m["mask"]["size"], sink=W(p + ".sink")) @ W(p + ".o").T

    def experts(mlp, p, h):
        r = mlp["router"]
        s = torch.softmax(h @ W(p + ".router").T, -1)
        chosen = _choose(s + W(p + ".correction"), r, 1)
        gated = lambda q, a: (_silu(a @ W(q + ".gate").T) * (a @ W(q + ".up").T)) @ W(q + ".down").T  # noqa: E731
        return _routed(mlp, W, p, h, chosen, s.gather(1, chosen) * r["scale"], gated)

    X = W("embed")[ids][None].repeat(cfg["streams"], 1, 1)
    for i, layer in enumerate(cfg["layers"]):
        for j, f in ((1, lambda h: mixer(layer, f"l{i}.mix", h)), (2, lambda h: experts(layer["mlp"], f"l{i}.mlp", h))):
            hc = f"l{i}.hc{j}"
            y = W(f"l{i}.ls{j}") * f(_dyt(torch.einsum("s,ste->te", W(hc + ".in"), X), W, f"l{i}.norm{j}"))
            X = torch.einsum("st,sne->tne", W(hc + ".mix"), X) + W(hc + ".out")[:, None, None] * y
    return W("head") @ _dyt(X.sum(0)[-1], W, "final.norm")


def _run_order(cfg):
    n, loop = len(cfg["layers"]), cfg.get("loop")
    a, b, times = (loop["start"], loop["stop"], loop["times"]) if loop else (n, n, 0)
    return [(i, None) for i in range(a)] + [(i, t if i == a else None) for t in range(times) for i in range(a, b)] + [(i, None) for i in range(b, n)]


def _silupel_forward(cfg, W, ids):
    eps, x = cfg["norm"]["eps"], W("embed")[ids]
    for i, _ in _run_order(cfg):
        layer, p = cfg["layers"][i], f"l{i}.mix"
        m = layer["mixer"]
        h = _layer_norm(x, W(f"l{i}.norm1"), eps)
        h = h + (torch.cat([torch.zeros_like(h[:1]), h[:-1]]) - h) * W(f"l{i}.shift")
        if layer["type"] == "mingru":
            z, u = torch.sigmoid(h @ W(p + ".z").T + W(p + ".z.b")), h @ W(p + ".x").T + W(p + ".x.b")
            new = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
            S, states = torch.zeros_like(z[0]), torch.empty_like(z)
            for t in range(h.shape[0]):
                S = (1 - z[t]) * S + z[t] * new[t]
                states[t] = S
            x = x + (states * _silu(h @ W(p + ".g").T)) @ W(p + ".o").T
        elif layer["type"] == "attention":
            q, k, v = _heads(m, W, p, h, bias=True)
            y = _attend(_rotate(q, m["rot"], False), _rotate(k, m["rot"], False), v, m["scale"], chunk=m["mask"]["size"], cap=m["softcap"], factors=W(p + ".temp"))
            x = x + (y * torch.sigmoid(h @ W(p + ".g").T)) @ W(p + ".o").T + W(p + ".o.b")
        else:
            x = x + _latent_attention(m, W, p, h, eps, False, False) @ W(p + ".o").T
        h, p = _layer_norm(x, W(f"l{i}.norm2"), eps), f"l{i}.mlp"
        x = x + (torch.nn.functional.gelu(h @ W(p + ".gate").T, approximate="tanh") * (h @ W(p + ".up").T)) @ W(p + ".down").T
    return W("head") @ _layer_norm(x[-1], W("final.norm"), eps)


def _tupalorn_forward(cfg, W, ids):
    eps, x, kept, T = cfg["norm"]["eps"], W("embed")[ids], {}, ids.shape[0]
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}.mix"
        h = _layer_norm(x, W(f"l{i}.norm1"), eps)
        if layer["type"] == "mamba2":
            H, dv, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            z, xbc, dt = (h @ W(p + ".in").T).split([H * dv, H * dv + 2 * G * N, H], -1)
            u, b, c = _silu(_conv(xbc, W(p + ".conv"), W(p + ".conv.b"))).split([H * dv, G * N, G * N], -1)
            u, b, c = u.view(T, H, dv), *(a.reshape(T, G, N).repeat_interleave(H // G, 1) for a in (b, c))
            dt = torch.nn.functional.softplus(dt + W(p + ".dt_bias"))
            o = _scan((-W(p + ".A_log").exp() * dt).exp()[..., None], b, dt[..., None] * u, c) + W(p + ".D")[:, None] * u
            o = (o.reshape(T, -1) * _silu(z)).view(T, m["norm_groups"], -1)
            y = _rms(o, eps).reshape(T, -1) * W(p + ".norm")
        elif layer["type"] == "retention":
            q, k, v = _heads(m, W, p, h)
            decay = torch.tensor(m["decay"], dtype=h.dtype, device=h.device)[None, :, None].expand(T, -1, 1)
            o = _scan(decay, _rotate(k, m["rot"], False) * m["dim"] ** -0.5, v, _rotate(q, m["rot"], False))
            y = _rms(o, eps).reshape(T, -1) * _silu(h @ W(p + ".g").T)
        else:
            if m.get("kv_from") is None:
                kept[i] = (_rms(h @ W(p + ".k").T, eps) * W(p + ".k.norm")).view(T, -1, m["dim"]), (h @ W(p + ".v").T).view(T, -1, m["vdim"])
            q = (_rms(h @ W(p + ".q").T, eps) * W(p + ".q.norm")).view(T, -1, m["dim"])
            y = _attend(q, *kept[m.get("kv_from", i)], m["scale"], window=m["mask"]["size"])
            y = (y.view(T, m["heads"], -1) * torch.sigmoid(h @ W(p + ".g").T)[..., None]).reshape(T, -1)
        y, p = y @ W(p + ".o").T, f"l{i}.mlp"
        g, u = (h @ W(f"{p}.{n}").T + W(f"{p}.{n}.b") for n in ("gate", "up"))
        x = x + y + _clamped(g, u, layer["mlp"]["limit"]) @ W(p + ".down").T + W(p + ".down.b")
    logits = W("embed") @ _layer_norm(x[-1], W("final.norm"), eps)
    return cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"])


def _birizen_forward(cfg, W, ids):
    eps, T = cfg["norm"]["eps"], ids.shape[0]
    x = start = W("embed")[ids]
    for i, enters in _run_order(cfg):
        if enters is not None:
            x = torch.cat([x, start], -1) @ W("loop.in").T + W("loop.step")[enters]
        layer, p = cfg["layers"][i], f"l{i}.mix"
        m, mlp = layer["mixer"], layer["mlp"]
        h = _rms(x, eps) * W(f"l{i}.norm1")
        if layer["type"] == "lightning":
            q, k, v = (_silu(a) for a in _heads(m, W, p, h))
            decay = torch.tensor(m["decay"], dtype=h.dtype, device=h.device)[None, :, None].expand(T, -1, 1)
            y = _rms(_scan(decay, k, v, q).reshape(T, -1), eps) * W(p + ".norm")
        else:
            y = _latent_attention(m, W, p, h, eps, True, True)
        x = x + _rms((y * torch.sigmoid(h @ W(p + ".g").T)) @ W(p + ".o").T, eps) * W(f"l{i}.norm1b")
        h, p = _rms(x, eps) * W(f"l{i}.norm2"), f"l{i}.mlp"
        s = torch.sigmoid(h @ W(p + ".router").T)
        chosen = _choose(s + W(p + ".correction"), mlp["router"], 2)
        w = s.gather(1, chosen)
        expert = lambda q, a, limit=mlp["expert"]["limit"]: _clamped(a @ W(q + ".gate").T, a @ W(q + ".up").T, limit) @ W(q + ".down").T  # noqa: E731
        y = _routed(mlp, W, p, h, chosen, w / (w.sum(-1, keepdim=True) + 1e-20), expert) + expert(p + ".shared", h, mlp["shared"]["limit"])
        x = x + _rms(y, eps) * W(f"l{i}.norm2b")
    return W("embed") @ (_rms(x[-1], eps) * W("final.norm"))
