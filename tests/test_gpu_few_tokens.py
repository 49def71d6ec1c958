"""Products of up to eight tokens from the stream on, against float64, at the edges of what the kernel takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
D = "cuda:0"
# (features, inner): less than a group of eight rows a block, ragged groups, an inner size below and beside a chunk of 32, shares of
# 1, 2, 3, 4, 5, 6, 8, 10 and 12 groups for each of 148 SMs, the 0.5B and width-1,024 sizes
SIZES = [(8, 8), (40, 72), (152, 1000), (896, 896), (2400, 264), (5472, 1024), (896, 4864), (9728, 896), (14200, 136),
         (1992, 136), (4096, 264), (7000, 264), (9000, 264)]
TOKENS = [1, 2, 3, 5, 8]


def _kernels():
    from hfcpu_b200 import kernels
    kernels.backend()
    return kernels


def _made(M, N, K, seed):
    g = torch.Generator(device=D).manual_seed(seed)
    r = lambda *s: torch.randn(*s, device=D, generator=g)  # noqa: E731
    return r(M, K) * 3, (r(N, K) * K ** -0.5).bfloat16(), (1 + 0.1 * r(K)), r(N).bfloat16()


def _sums(x, norm, w):
    """(x normed @ w.T, a bound of what rounding may change) in float64: a normed operand is rounded to bfloat16 once (half a unit
    of 2^-7), the sums of K products in float32 in any order."""
    x, w, K = x.double(), w.double(), x.shape[1]
    rel = (K + 32) * 2.0 ** -24
    if norm is not None:
        x = x * (x.square().mean(-1, keepdim=True) + norm[1]).rsqrt() * norm[0].double()
        rel += 2.0 ** -8 + 2.0 ** -20
    return x @ w.T, rel * (x.abs() @ w.abs().T)


@pytest.mark.parametrize("N,K", SIZES)
@pytest.mark.parametrize("M", TOKENS)
def test_few_linear(M, N, K):
    kernels = _kernels()
    x, w, nw, b = _made(M, N, K, M * N + K)
    assert kernels.few_tokens(M, torch.bfloat16, (nw, 1e-6), w)
    for norm in (None, (nw, 1e-6), (nw.bfloat16(), 1e-5)):
        a = x if norm is not None else x.bfloat16()
        want, bound = _sums(a, norm, w)
        out = torch.randn(M, N, device=D)
        before = out.clone()
        kernels.few_linear(a, norm, w, b, out, True)
        want_out = before.double() + want + b.double()
        assert ((out.double() - want_out).abs() <= bound + 2.0 ** -22 * (before.abs() + want.abs() + b.abs().double())).all()
        kernels.few_linear(a, norm, w, None, out, False)
        assert ((out.double() - want).abs() <= bound + 1e-30).all()
        alone = torch.empty(1, N, device=D)
        kernels.few_linear(a[:1].contiguous(), norm, w, None, alone, False)
        assert torch.equal(alone[0], out[0]) or norm is not None and torch.allclose(alone[0], out[0], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("activation", ["silu", "relu", "gelu_tanh", "clamped"])
@pytest.mark.parametrize("M,N,K", [(1, 16, 40), (3, 1008, 72), (8, 9728, 896)])
def test_few_glu(M, N, K, activation):
    kernels = _kernels()
    x, w, nw, b = _made(M, N, K, N)
    clamp = (7.0, 1.702, 1.0) if activation == "clamped" else None
    z, bound = _sums(x, (nw, 1e-6), w)
    z = z + b.double()
    act = {"silu": torch.nn.functional.silu, "relu": torch.relu, "gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}

    def pair(g, u):
        if clamp is None:
            return act[activation](g) * u
        g = g.clamp(max=7.0)
        return g * torch.sigmoid(1.702 * g) * (u.clamp(-7.0, 7.0) + 1.0)
    g, u = z[:, 0::2], z[:, 1::2]
    want = pair(g, u)
    # a gate's slope is below 1.2 in size, and a pair is linear in what is multiplied with it
    slack = 1.2 * (bound[:, 0::2] + 1e-5) * (u.abs() + 1) + (g.abs() + 0.3) * (bound[:, 1::2] + 1e-5)
    wide = torch.full((M, N // 2 + 8), 7.0, device=D, dtype=torch.bfloat16)
    kernels.few_glu(x, (nw, 1e-6), w, b, wide[:, :N // 2], activation, clamp)
    assert ((wide[:, :N // 2].double() - want).abs() <= slack + 2.0 ** -8 * want.abs()).all()
    assert (wide[:, N // 2:] == 7).all()


@pytest.mark.parametrize("M,K,H,G,d", [(1, 896, 14, 2, 64), (8, 896, 14, 2, 64), (3, 200, 5, 1, 64), (2, 1024, 6, 2, 128), (5, 2048, 16, 4, 128)])
def test_few_rope_kv_agrees_with_the_separate_kernels(M, K, H, G, d):
    kernels = _kernels()
    x, w, nw, b = _made(M, (H + 2 * G) * d, K, d)
    g = torch.Generator(device=D).manual_seed(1)
    angle = torch.rand(64, d // 2, device=D, generator=g) * 6
    table = torch.stack([angle.cos(), angle.sin()], -1).contiguous()
    pos = torch.randperm(64, device=D)[:M].int()
    slots = torch.tensor([3, -1, 17, 8, 30, 1, 12, 5], device=D, dtype=torch.int32)[:M].contiguous()
    got, want = ([torch.zeros(M, H * d, device=D, dtype=torch.bfloat16)] + [torch.zeros(4, 8, G, d, device=D, dtype=torch.bfloat16) for _ in range(2)]
                 for _ in range(2))
    kernels.few_rope_kv(x, (nw, 1e-6), w, b, table, pos, slots, got[0], got[1], got[2], H, G, d)
    sums, bound = _sums(x, (nw, 1e-6), w)
    kernels.rope_kv_write((sums + b.double()).to(torch.bfloat16).contiguous(), table, d, pos, slots, want[0], want[1], want[2], H, G, d)
    # rounding of the row and of the rotated values (2^-8 of a pair's size), and what the sums may differ
    top = float((bound.max() + 2.0 ** -7 * (sums + b.double()).abs().max()) * 2)
    for a, c in zip(got, want):
        assert (a.double() - c.double()).abs().max() <= top
        assert float((a.double() - c.double()).norm() / c.double().norm()) < 5e-3
    # only the slots that tokens have are written, each in full
    written = torch.zeros(4 * 8, dtype=torch.bool, device=D)
    written[slots[slots >= 0].long()] = True
    for cache in got[1:]:
        rows = cache.view(4 * 8, G * d)
        assert (rows[~written] == 0).all() and (rows[written] != 0).any(-1).all()


def test_few_tokens_refuses_what_it_does_not_take():
    kernels = _kernels()
    nw = torch.ones(896, device=D)
    small = torch.zeros(896, 896, device=D, dtype=torch.bfloat16)
    assert kernels.few_tokens(8, torch.bfloat16, (nw, 1e-6), small) and not kernels.few_tokens(9, torch.bfloat16, (nw, 1e-6), small)
    assert not kernels.few_tokens(1, torch.float32, (nw, 1e-6), small)
    assert not kernels.few_tokens(1, torch.bfloat16, (nw, 1e-6), torch.zeros(151936, 896, device=D, dtype=torch.bfloat16))
    assert not kernels.few_tokens(1, torch.bfloat16, (torch.ones(897, device=D)[1:], 1e-6), small)


ACTS = {"silu": torch.nn.functional.silu, "relu": torch.relu, "relu2": lambda z: z.clamp_min(0) ** 2,
        "gelu_tanh": lambda z: torch.nn.functional.gelu(z, approximate="tanh")}


# half a million weights and more, so that the products of all designs go to the kernel; ragged and whole shares of groups
@pytest.mark.parametrize("N,K", [(1024, 1024), (2000, 264), (7008, 136)])
@pytest.mark.parametrize("M", [1, 3, 8])
def test_products_of_few_tokens_in_every_design_form(M, N, K):
    """linear, linear_act, linear_swiglu and linear_glu with operands that are normed already: every activation, with and without a
    bias, both types, into an array of its own and into columns of a wider one."""
    kernels = _kernels()
    b = kernels.backend()
    x, w, _, bias = _made(M, N, K, M + N + K)
    a = (x / 3).bfloat16()
    z, bound = _sums(a, None, w)
    assert b._few(a, w)

    def check(got, want, slack):
        unit = 2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -18      # the fast quotient and exponential: some 2^-20
        assert ((got.double() - want).abs() <= unit * want.abs() + slack).all()
    for dtype in (torch.bfloat16, torch.float32):
        out = torch.full((M, N), float("nan"), device=D, dtype=dtype)
        kernels.linear(a, w, bias, out, False)
        check(out, z + bias.double(), bound + 2.0 ** -22 * (z.abs() + bias.abs().double()))
        for act in ("relu", "relu2", "gelu_tanh"):
            out.fill_(float("nan"))
            kernels.linear_act(a, w, out, act)
            # (a slope is below 1.2, the square's twice the value)
            check(out, ACTS[act](z), (bound + 2.0 ** -20) * (2 * z.abs() + 1.2))
        for act in ("silu", "relu", "relu2", "gelu_tanh", "clamped"):
            clamp = (1.5, 1.7, 1.0) if act == "clamped" else None
            for with_bias in (False, True):
                y = z + bias.double() if with_bias else z
                g, u = y[:, 0::2], y[:, 1::2]
                want = g.clamp(max=1.5) * torch.sigmoid(1.7 * g.clamp(max=1.5)) * (u.clamp(-1.5, 1.5) + 1.0) if clamp else ACTS[act](g) * u
                slack = ((bound[:, 0::2] + 2.0 ** -20) * (u.abs() + 2.5) * (2 * g.abs() + 1.2)
                         + (g.square() + g.abs() + 0.3) * (bound[:, 1::2] + 2.0 ** -20))
                wide = torch.full((M, N // 2 + 24), 7.0, device=D, dtype=dtype)
                got = wide[:, 8:8 + N // 2]
                kernels.linear_glu(a, w, torch.empty(M, N, device=D, dtype=dtype), got, act, bias=bias if with_bias else None, clamp=clamp)
                check(got, want, slack)
                assert (wide[:, :8] == 7).all() and (wide[:, 8 + N // 2:] == 7).all()
                if act == "silu" and not with_bias:
                    own = torch.empty(M, N // 2, device=D, dtype=dtype)
                    kernels.linear_swiglu(a, w, torch.empty(M, N, device=D, dtype=dtype), own)
                    assert torch.equal(own, got)
    kernels.check_device_errors()


class _Counted:
    """A library whose calls of the kernel of few tokens are counted."""

    def __init__(self, lib):
        self._lib, self.few = lib, 0

    def __getattr__(self, name):
        fn = getattr(self._lib, name)
        if not name.startswith("hfb_few_") or name == "hfb_few_takes":
            return fn

        def call(*args):
            self.few += 1
            return fn(*args)
        return call


@pytest.mark.parametrize("requests", [1, 8])
@pytest.mark.parametrize("model", ["qwen2", "manapel", "peludra", "mokisun", "silupel", "tupalorn", "birizen"])
def test_designs_with_finished_sums_in_front_of_their_tails(model, requests):
    """Answers at the benchmark's smallest widths, whose products go to the kernel (the designs' own test models have smaller ones): one
    plane of finished sums in front of every tail (norms of all kinds, latent rows and queries, rotation with head norms, routers,
    recurrences), against float64 and against split products."""
    import importlib.util
    import os
    spec = importlib.util.spec_from_file_location("perf_cases", os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "perf", "cases.py"))
    cases = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(cases)
    b = _kernels().backend()
    case = dict(model=model, size="0.5b" if model == "qwen2" else "w1024", kind="reply", requests=requests, tokens=11 if requests == 1 else 5, new=4,
                ragged=False, dtype="bfloat16", chunk=0)
    want = cases.exact(case, 3)["checked"].double()
    lib, errors = b.lib, {}
    for few in (True, False):
        b.lib = _Counted(lib)
        if not few:
            b._few = lambda a, w: False
        try:
            got = cases.run(cases.prepare(case, 3))["checked"].double()
            assert (b.lib.few > 0) == (few or model == "qwen2")                # (its layers take the stream)
        finally:
            b.lib = lib
            vars(b).pop("_few", None)
        errors[few] = float((got[:want.shape[0]] - want).norm() / want.norm())
    # rounding to bfloat16 in every layer: what any correct run is off, and no more than the split products by half
    assert errors[True] < cases.tolerance(case)["rel"] and errors[True] < 1.5 * errors[False] + 1e-4, errors


def test_layers_made_again_from_a_recording_give_the_same_bits():
    """A step through recorded launches against the same step layer by layer, prompts and single tokens."""
    import hfcpu_b200
    from hfcpu_b200 import kernels
    from hfcpu_b200.config import config_from_dict
    from hfcpu_b200.models import random_model
    cfg = dict(architectures=["Qwen2ForCausalLM"], num_hidden_layers=6, hidden_size=512, num_attention_heads=8, num_key_value_heads=2,
               intermediate_size=1024, vocab_size=1000, max_position_embeddings=1024, rms_norm_eps=1e-6, rope_theta=1e6, tie_word_embeddings=False)
    for dtype in (torch.bfloat16, torch.float32):
        model = random_model(config_from_dict(cfg), seed=5, dtype=dtype, device=D, std=0.08)
        assert model._alike[:5] == [0] * 5 and model._alike[5] is None
        got, made_again = _with_and_without_recording(model, (300, 40, 3, 1, 1))
        assert torch.equal(got[0], got[1])
        # a layer is handed its normed input, except where it takes the stream (bfloat16, up to eight tokens): then all five are alike
        assert made_again == [3 if dtype == torch.float32 or n > 4 else 4 for n in (300, 40, 3, 1, 1)]


def _with_and_without_recording(model, portions):
    """(logits of both ways, layers made again in each step)."""
    import hfcpu_b200
    from hfcpu_b200 import kernels
    from hfcpu_b200.kernels.native import Recording
    got, count, inner = [], [], Recording.replay

    def counting(self, tensors):
        done = inner(self, tensors)
        count[-1] += done
        return done
    for record in (True, False):
        eng = hfcpu_b200.Engine(model, block_size=16, max_tokens=2048, max_requests=4)
        eng.use_graphs = False
        saved = kernels.recorder
        if record:
            Recording.replay = counting
        else:
            kernels.recorder = lambda: None
        try:
            eng.add_request("a")
            eng.add_request("b")
            outs = []
            for n in portions:
                if record:
                    count.append(0)
                outs.append(eng.step([hfcpu_b200.StepEntry(r, [(7 * i + n) % 1000 for i in range(n)], [n - 1]) for r in "ab"]).clone())
            got.append(torch.stack(outs))
        finally:
            kernels.recorder, Recording.replay = saved, inner
    return got, count


def test_layers_of_several_kinds_made_again_give_the_same_bits():
    """Windows on some layers (their caches are of another group), biases missing in some, kinds in stretches and in turn, a loop of
    the run order over layers that ran before."""
    import dataclasses
    from hfcpu_b200.config import config_from_dict
    from hfcpu_b200.config.base import ScheduleEntry
    from hfcpu_b200.models import Model
    from hfcpu_b200.weights import RandomSource
    cfg = config_from_dict(dict(architectures=["Qwen2ForCausalLM"], num_hidden_layers=12, hidden_size=512, num_attention_heads=8, num_key_value_heads=2,
                                intermediate_size=1024, vocab_size=1000, max_position_embeddings=1024, rms_norm_eps=1e-6, rope_theta=1e6,
                                tie_word_embeddings=False))
    #        window 32: w; no biases: n; feed-forward's activation relu: r
    kinds = ["", "", "", "w", "w", "w", "n", "r", "n", "r", "nw", "nw"]
    plan = cfg.plan()
    layers = [dataclasses.replace(l, mixer=dataclasses.replace(l.mixer, args=dict(l.mixer.args, window=32 if "w" in k else 0, qkv_bias="n" not in k)),
                                  ffn=dataclasses.replace(l.ffn, args=dict(l.ffn.args, activation="relu" if "r" in k else "silu")))
              for l, k in zip(plan.layers, kinds)]
    plan = dataclasses.replace(plan, layers=layers, schedule=[ScheduleEntry(i) for i in range(12)] + [ScheduleEntry(i) for i in (3, 4, 5, 11)])
    for dtype in (torch.bfloat16, torch.float32):
        model = Model(cfg, dtype, torch.device(D), plan=plan)
        model.bind(RandomSource(model.tensor_specs(), 5, dtype, model.device, std=0.08))
        a = model._alike
        assert a[0] == a[1] == a[2] and a[3] == a[4] == a[5] == a[12] == a[13] == a[14] and a[10] == a[11] and len({a[0], a[3], a[6], a[7], a[10]}) == 5
        got, made_again = _with_and_without_recording(model, (200, 40, 3, 1, 1))
        assert torch.equal(got[0], got[1])
        # entry 0 has no normed input handed to it: 1 and 3 are written down, 2, 4 and 5 made again, 10 -> 11, 12 -> 13 and 14; from the
        # stream on 0 -> 1 and 2 too
        assert made_again == [6 if dtype == torch.float32 or n > 4 else 7 for n in (200, 40, 3, 1, 1)]

