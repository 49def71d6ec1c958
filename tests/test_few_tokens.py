"""Steps of few tokens through parts that read the stream themselves: whose code runs.  On the CPU, with a stand-in that has the
products of few tokens."""
import pytest
import torch

from emu_backend import EmuBackend

CFG = dict(architectures=["Qwen2ForCausalLM"], num_hidden_layers=3, hidden_size=64, num_attention_heads=2, num_key_value_heads=1, head_dim=64,
           intermediate_size=96, vocab_size=200, max_position_embeddings=128, rms_norm_eps=1e-6, rope_theta=1e4, tie_word_embeddings=False)


class FewEmu(EmuBackend):
    """The stand-in with products of few tokens."""

    def __init__(self, takes=True):
        self.takes, self.few = takes, 0

    def few_takes(self, M, w, rope=False):
        return self.takes and M <= 8

    def _normed(self, a, norm):
        if norm is None:
            return a
        self.few += 1
        out = torch.empty(a.shape, dtype=torch.bfloat16)
        self.rmsnorm(a, norm[0], norm[1], out, None)
        return out

    def few_linear(self, a, norm, w, bias, out, accumulate):
        self.linear(self._normed(a, norm), w, bias, out, accumulate)

    def few_glu(self, a, norm, w, bias, out, act, clamp):
        assert act == 0 and bias is None
        self.linear_swiglu(self._normed(a, norm), w, torch.empty(a.shape[0], w.shape[0], dtype=out.dtype), out)

    def few_rope_kv(self, a, norm, w, bias, cos_sin, positions, slots, q_out, k_cache, v_cache, H, G, d):
        qkv = torch.empty(a.shape[0], w.shape[0], dtype=q_out.dtype)
        self.linear(self._normed(a, norm), w, bias, qkv, False)
        self.rope_kv_write(qkv, cos_sin, d, positions, slots, q_out, k_cache, v_cache, H, G, d)


@pytest.fixture
def install():
    from hfcpu_b200 import kernels
    old = kernels._backend
    yield kernels.set_backend
    kernels.set_backend(old)


def _model():
    from hfcpu_b200.config import config_from_dict
    from hfcpu_b200.models import random_model
    return random_model(config_from_dict(CFG), seed=5, dtype=torch.bfloat16, device="cpu", std=0.2)


def _steps(model):
    import hfcpu_b200
    eng = hfcpu_b200.Engine(model, block_size=16, max_tokens=256, max_requests=2)
    eng.add_request("a")
    return torch.cat([eng.step([hfcpu_b200.StepEntry("a", [(7 * i + n) % 200 for i in range(n)], [n - 1])]).clone() for n in (12, 8, 1)])


def _derived(part, **functions):
    """``part`` as an object of a class that derives from its own."""
    part.__class__ = type("Derived", (type(part),), functions)


def _attend(self, ctx, xn, cache, write_cache):
    return torch.ones_like(xn).repeat(1, 2)


CHANGES = {
    "a mixer's class": lambda m: _derived(m.layers[1].mixer, _attend=_attend),
    "a feed-forward's class": lambda m: _derived(m.layers[1].ffn, _hidden=lambda self, ctx, xn: torch.ones(xn.shape[0], 96).bfloat16()),
    "a first norm's class": lambda m: _derived(m.layers[0].norm1, forward=lambda self, x, out, rows=None: out.fill_(1)),
    "a mixer's function": lambda m: setattr(m.layers[1].mixer, "_attend", lambda *a: _attend(None, *a)),
    "a feed-forward's function": lambda m: setattr(m.layers[1].ffn, "operand", lambda ctx, xn, out: out.fill_(1)),
    "a first norm's function": lambda m: setattr(m.layers[0].norm1, "forward", lambda x, out, rows=None: out.fill_(1)),
}


def test_plain_layers_take_the_stream(install):
    few = FewEmu()
    install(few)
    got = _steps(_model())
    assert few.few == 2 * 3 * 2                       # two norms a layer in each of the steps of eight and one token
    install(FewEmu(takes=False))
    assert torch.equal(got, _steps(_model()))


@pytest.mark.parametrize("what", list(CHANGES))
def test_parts_that_compute_something_else_run_their_own_code(install, what):
    install(FewEmu(takes=False))
    model = _model()
    before = _steps(model)
    CHANGES[what](model)
    want = _steps(model)
    assert not torch.equal(want[1:], before[1:])
    install(FewEmu())
    assert torch.equal(_steps(model), want)


def test_a_class_whose_function_was_replaced(install, monkeypatch):
    from hfcpu_b200.parts.ffn import SwiGlu
    install(FewEmu())
    model, seen, inner = _model(), [], SwiGlu._hidden

    def probe(self, ctx, xn):
        seen.append(xn.shape[0])
        return inner(self, ctx, xn)
    monkeypatch.setattr(SwiGlu, "_hidden", probe)
    _steps(model)
    assert seen == [12] * 3 + [8] * 3 + [1] * 3


def test_a_backend_around_another_sees_the_calls_it_knows(install):
    class Around:
        def __init__(self, inner):
            self.inner, self.calls = inner, 0

        def __getattr__(self, name):
            return getattr(self.inner, name)

        def linear_rope_kv(self, *args):
            self.calls += 1
            return self.inner.linear_rope_kv(*args)
    b = Around(FewEmu())
    install(b)
    _steps(_model())
    assert b.calls == 3 * 3


def test_products_of_more_tokens_ask_the_library_nothing():
    """In steps of any size a product is looked at first; the question costs about 1 us of a prompt's host time."""
    from types import SimpleNamespace

    from hfcpu_b200.kernels.native import NativeBackend
    asked = []
    b = object.__new__(NativeBackend)
    b.gemm, b._few_sizes, b.lib = "tc", {}, SimpleNamespace(hfb_few_takes=lambda *a: asked.append(a) or 1)
    w = torch.zeros(1024, 512, dtype=torch.bfloat16)
    for M, few in ((1, True), (8, True), (9, False), (2000, False)):
        asked.clear()
        assert b._few(torch.zeros(M, 512, dtype=torch.bfloat16), w) == few
        assert len(asked) == few
    asked.clear()
    assert b._few(torch.zeros(1, 512, dtype=torch.bfloat16), w) and not asked                  # nor a second time about the same sizes
    for M in range(1, 9):
        for n in range(1000):
            b._few_has(M, n, 8, 0)
    assert len(b._few_sizes) <= 4096                                                           # kept for so many


def test_ranges_of_decode_attention():
    """At the edges of the rule, in tiles of 64 keys."""
    from hfcpu_b200.kernels import decode_split_hint
    edges = {1: 1, 6: 1, 7: 4, 8: 8, 15: 8, 16: 16, 31: 16, 32: 16, 63: 16, 64: 32, 127: 32, 128: 64, 4096: 64}
    for tiles, ranges in edges.items():
        assert decode_split_hint(tiles * 64 - 63) == decode_split_hint(tiles * 64) == ranges, tiles
    assert decode_split_hint(0) == 1


# the sources of the kernels that a step of the first architecture runs
@pytest.mark.parametrize("name", ["few_tokens", "fused_decode", "gemm_tc", "attention_decode", "attention_fast", "attention_tc", "attention_tc2"])
def test_every_kernel_of_a_step_is_on_the_timeline(name):
    """The timeline pairs a kernel's entry with the next wait that returns: one kernel without an entry gives its times to the others."""
    import os
    import re

    from hfcpu_b200.kernels import build, timeline
    with open(os.path.join(build.CSRC, name + ".cu")) as f:
        source = f.read()
    bodies = source.split("__global__")[1:]
    assert bodies
    for body in bodies:
        found = re.search(r"HFB_TRACE_ENTRY\((\d+)\)", body)
        assert found and int(found.group(1)) in timeline.KERNELS, body[:80]


def test_sizes_beyond_32_bits_of_arithmetic_are_refused():
    """An inner size just below 2^31 wrapped to a small one when its row in shared memory was counted: the product of it was taken,
    and would have been sums of nothing."""
    import ctypes

    from hfcpu_b200.kernels import build
    lib = ctypes.CDLL(build.build())
    assert lib.hfb_few_takes(1, 8, 8, 0) == 1
    for N, K in ((8, 2 ** 31 - 8), (8, 2 ** 31 - 32), (8, 2 ** 30), (2 ** 31 - 1, 8), (2 ** 31 - 8, 2 ** 31 - 8), (8, 1 << 17)):
        for rope in (0, 1):
            assert lib.hfb_few_takes(1, N, K, rope) == 0, (N, K)
    for bad in ((0, 8, 8), (9, 8, 8), (1, 7, 8), (1, 8, 4), (1, 8, 12), (-1, 8, 8), (1, -8, 8), (1, 8, -8)):
        assert lib.hfb_few_takes(*bad, 0) == 0, bad
