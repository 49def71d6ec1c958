"""Layers whose launches are made again from another layer's recording: whatever has been changed since the weights were bound runs
its own code.  On the CPU, with a stand-in that writes down its calls as the CUDA backend does, and the CUDA backend's recording
itself against a stand-in library."""
import ctypes

import pytest
import torch

from emu_backend import EmuBackend

CFG = dict(architectures=["Qwen2ForCausalLM"], num_hidden_layers=6, hidden_size=64, num_attention_heads=4, num_key_value_heads=2,
           intermediate_size=96, vocab_size=200, max_position_embeddings=128, rms_norm_eps=1e-6, rope_theta=1e4, tie_word_embeddings=False)


class RecordingEmu(EmuBackend):
    """The stand-in with a recorder: a recording makes the calls again with other tensors in the places of the recorded ones."""

    def __init__(self):
        self.log, self.replayed = None, 0

    def __getattribute__(self, name):
        fn = object.__getattribute__(self, name)
        if name.startswith("_") or name == "record" or not callable(fn):
            return fn

        def call(*args, **kw):
            if self.log is not None:
                self.log.append((fn, args, kw))
            saved, self.log = self.log, None               # (a call that makes others is one call)
            try:
                return fn(*args, **kw)
            finally:
                self.log = saved
        return call

    def record(self, run, tensors):
        self.log = []
        out = run()
        calls, self.log = self.log, None
        owner = self

        class Recording:
            def replay(self, others):
                assert len(others) == len(tensors)
                ptrs = {t.data_ptr(): o for t, o in zip(tensors, others) if t is not None}

                def swap(a):
                    return ptrs.get(a.data_ptr(), a) if isinstance(a, torch.Tensor) else a
                for fn, args, kw in calls:
                    fn(*[swap(a) for a in args], **{k: swap(a) for k, a in kw.items()})
                owner.replayed += 1
                return True
        return out, Recording()


@pytest.fixture
def emu():
    from hfcpu_b200 import kernels
    old, b = kernels._backend, RecordingEmu()
    kernels.set_backend(b)
    yield b
    kernels.set_backend(old)


def _model():
    from hfcpu_b200.config import config_from_dict
    from hfcpu_b200.models import random_model
    return random_model(config_from_dict(CFG), seed=5, dtype=torch.float32, device="cpu", std=0.2)


def _steps(model, record=True):
    """Logits of a portion of 12 tokens and two single tokens."""
    import hfcpu_b200
    from hfcpu_b200 import kernels
    eng, saved = hfcpu_b200.Engine(model, block_size=16, max_tokens=256, max_requests=2), kernels.recorder
    eng.add_request("a")
    if not record:
        kernels.recorder = lambda: None
    try:
        return torch.cat([eng.step([hfcpu_b200.StepEntry("a", [(7 * i + n) % 200 for i in range(n)], [n - 1])]).clone() for n in (12, 1, 1)])
    finally:
        kernels.recorder = saved


def test_alike_layers_are_made_again(emu):
    model = _model()
    assert model._alike == [0] * 5 + [None]
    want = _steps(model, record=False)
    assert emu.replayed == 0
    assert torch.equal(_steps(model), want)
    assert emu.replayed == 3 * 3                       # three steps; of five alike layers the first gets its input otherwise, the second is written down


def _other_ffn(model):
    from hfcpu_b200.parts import make_part
    part = make_part("ffn", type(model.plan.layers[0].ffn)("swiglu", dict(model.plan.layers[0].ffn.args, activation="relu")))
    part.w_gate_up, part.w_down = model.layers[2].ffn.w_gate_up, model.layers[2].ffn.w_down
    return part


def _new_layer(model):
    from hfcpu_b200.models import Layer
    l = model.layers[3]
    return Layer(l.block, l.norm1, l.mixer, l.norm2, _other_ffn(model))


CHANGES = {
    "a part's method": lambda m: setattr(m.layers[2].mixer, "_attend", lambda ctx, xn, cache, write: torch.ones_like(xn)),
    "the feed-forward's method": lambda m: setattr(m.layers[3].ffn, "_hidden", lambda ctx, xn: torch.ones(xn.shape[0], 96)),
    "a block's forward": lambda m: setattr(m.layers[2].block, "forward", lambda ctx, x, *a, **k: None),
    "a constant": lambda m: setattr(m.layers[2].mixer, "scale", 0.9),
    "a norm's eps": lambda m: setattr(m.layers[4].norm1, "eps", 0.5),
    "a weight": lambda m: setattr(m.layers[1].ffn, "w_down", m.layers[1].ffn.w_down * 2),
    "a weight of other strides": lambda m: setattr(m.layers[2].mixer, "w_o", m.layers[2].mixer.w_o.T),
    "a bias that was not there": lambda m: setattr(m.layers[2].mixer, "b_o", torch.ones(64)),
    "another part": lambda m: setattr(m.layers[2], "ffn", _other_ffn(m)),
    "another layer": lambda m: m.layers.__setitem__(3, _new_layer(m)),
    "a norm taken from another layer": lambda m: setattr(m.layers[3], "norm1", m.layers[5].norm1),
}


@pytest.mark.parametrize("what", list(CHANGES))
def test_what_is_changed_after_binding_counts(emu, what):
    model = _model()
    before = _steps(model, record=False)
    CHANGES[what](model)
    want = _steps(model, record=False)
    assert not torch.equal(want, before)
    assert torch.equal(_steps(model), want)


def test_a_probe_put_over_a_method_sees_every_layer(emu, monkeypatch):
    from hfcpu_b200 import kernels
    from hfcpu_b200.parts.attention import OutputProduct, PagedAttention
    from hfcpu_b200.parts.ffn import SwiGlu
    model = _model()
    for owner, name in ((SwiGlu, "_hidden"), (OutputProduct, "forward_then_norm"), (PagedAttention, "forward_then_norm"), (kernels, "linear_glu"),
                        (kernels, "paged_attention")):
        seen, inner = [], getattr(owner, name)

        def probe(*args, **kw):
            seen.append(1)
            return inner(*args, **kw)
        with monkeypatch.context() as m:
            m.setattr(owner, name, probe)
            _steps(model)
        assert len(seen) == 3 * 6, (owner, name)
    before = emu.replayed
    _steps(model)
    assert emu.replayed == before + 3 * 3              # and with everything back in its place layers are made again


def test_a_backend_around_another_sees_every_call(emu):
    from hfcpu_b200 import kernels

    class Around:
        def __init__(self, inner):
            self.inner, self.calls = inner, 0

        def __getattr__(self, name):
            return getattr(self.inner, name)

        def paged_attention(self, *args, **kw):
            self.calls += 1
            return self.inner.paged_attention(*args, **kw)

    class Derived(RecordingEmu):
        calls = 0

        def paged_attention(self, *args, **kw):
            Derived.calls += 1
            return super().paged_attention(*args, **kw)
    model = _model()
    for b in (Around(emu), Derived()):
        kernels.set_backend(b)
        _steps(model)
        assert b.calls == 3 * 6


def _model_of(make_mixer, block=None):
    """Six layers with mixers (and blocks) made here."""
    from hfcpu_b200.config import config_from_dict
    from hfcpu_b200.models import Model
    from hfcpu_b200.weights import RandomSource
    model = Model(config_from_dict(CFG), torch.float32, torch.device("cpu"))
    for i, l in enumerate(model.layers):
        l.mixer = make_mixer(i)
        if block is not None:
            l.block = block()
    return model.bind(RandomSource(model.tensor_specs(), 3, torch.float32, model.device, std=0.2))


def _plain_mixer():
    from hfcpu_b200 import kernels
    from hfcpu_b200.parts import Mixer
    from hfcpu_b200.weights import TensorSpec

    class Straight(Mixer):
        """x += W norm(x): no cache, no state."""
        graph_safe = True

        def __init__(self, i):
            self.name, self.w = f"straight.{i}", None

        def tensor_specs(self):
            return [TensorSpec(self.name, (64, 64))]

        def bind(self, tensors, run_dtype, device):
            self.w = tensors[self.name].contiguous()

        def replay_key(self):
            return ("straight",)

        def replay_tensors(self):
            return (self.w,)

        def forward(self, ctx, xn, residual, cache, state, write_cache):
            assert cache is None
            kernels.linear(xn, self.w, None, residual, accumulate=True)
    return Straight


def test_mixers_without_a_cache(emu):
    model = _model_of(_plain_mixer())
    assert model._alike[:5] == [0] * 5
    want = _steps(model, record=False)
    assert torch.equal(_steps(model), want) and emu.replayed == 3 * 3


def test_a_block_with_state_of_its_own_is_alike_with_none(emu):
    from hfcpu_b200.parts import StateSpec
    from hfcpu_b200.parts.block import PreNormResidual

    class Counting(PreNormResidual):
        """Adds how many tokens its layer has seen to the stream."""

        def replay_key(self):
            return ("counting",)

        def state_spec(self):
            return StateSpec((1,))

        def forward(self, ctx, x, *args, block_state=None, **kw):
            x.add_(block_state[ctx.seq_slots.long()])
            block_state[ctx.seq_slots.long()] += x.shape[0]
            return super().forward(ctx, x, *args, **kw)
    model = _model_of(_plain_mixer(), Counting)
    want = _steps(model, record=False)
    assert torch.equal(_steps(model), want)


def test_copies_of_a_model(emu):
    """A model can be copied and stored; a copy's layers are alike among themselves, and what is changed in it counts there only."""
    import copy
    import pickle
    model = _model()
    want = _steps(model, record=False)
    for again in (copy.deepcopy(model), pickle.loads(pickle.dumps(model)), copy.copy(model)):
        emu.replayed = 0
        assert torch.equal(_steps(again), want) and emu.replayed == 3 * 3
        if again.layers is not model.layers:
            again.layers[2].mixer.scale = 0.9
            other = _steps(again, record=False)
            assert not torch.equal(other, want) and torch.equal(_steps(again), other)
            assert torch.equal(_steps(model), want)


def test_only_parts_that_may_be_alike_count_their_changes(emu):
    """Counting costs every attribute of every part that is made; a class that sets attributes its own way is alike with none."""
    from hfcpu_b200.parts.latent_attention import LatentAttention
    from hfcpu_b200.parts.norm import DynamicTanh
    for cls in (LatentAttention, DynamicTanh):
        assert cls.__setattr__ is object.__setattr__ and not cls.counts_changes
    Plain = _plain_mixer()
    part = Plain(0)
    before = part.changes
    part.w = 1
    del part.w
    assert Plain.counts_changes and part.changes == before + 2

    class Own(Plain):
        def __setattr__(self, name, value):
            super().__setattr__(name, value)
    assert not Own.counts_changes
    model = _model_of(Own)
    assert model._alike == [None] * 6
    assert torch.equal(_steps(model), _steps(model, record=False)) and emu.replayed == 0


# ---- the CUDA backend's own recording ----------------------------------------------------------------------------------
class Library:
    """Functions of any name that note their arguments' values and succeed."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def fn(*args):
            self.calls.append((name, [a.value if isinstance(a, ctypes._SimpleCData) else a for a in args]))
            return 0
        fn.__name__ = name
        setattr(self, name, fn)
        return fn


def _native():
    from hfcpu_b200.kernels.native import NativeBackend
    b = object.__new__(NativeBackend)
    lib = Library()
    b.launches = 0
    b.lib = lib
    return b, lib


def _recorded(b, tensors):
    from hfcpu_b200.kernels.native import _p

    def run():
        b._check(b.lib.hfb_thing(ctypes.c_int(3), *[_p(t) for t in tensors]), "thing")
        return "out"
    return b.record(run, tensors)


def test_recording_makes_the_calls_with_other_pointers():
    b, lib = _native()
    one = [torch.zeros(512, dtype=torch.uint8), None, torch.zeros(4, 64)]
    two = [torch.zeros(512, dtype=torch.uint8), None, torch.zeros(4, 64)]
    out, rec = _recorded(b, one)
    # (pointers agree in their low bits with the recorded ones, or the layer runs its own code)
    ok = all((x.data_ptr() ^ y.data_ptr()) & 255 == 0 for x, y in zip(one, two) if x is not None)
    assert out == "out" and b.launches == 1
    assert rec.replay(two) == ok
    if ok:
        assert lib.calls[1] == ("hfb_thing", [3, two[0].data_ptr(), None, two[2].data_ptr()]) and b.launches == 2


def test_recording_refuses_tensors_of_another_form():
    b, lib = _native()
    store = torch.zeros(1 << 16)
    base = -store.data_ptr() % 256 // 4

    def at(offset, *shape, dtype=None):
        t = store[base + offset:base + offset + 4096][:torch.Size(shape).numel()].view(*shape)
        return t if dtype is None else t.view(dtype)
    one = [at(0, 8, 8), at(4096, 64)]
    _, rec = _recorded(b, one)
    assert rec.replay([at(8192, 8, 8), at(12288, 64)]) and len(lib.calls) == 2
    for other in ([at(8192, 8, 8).T, at(12288, 64)],                                    # strides
                  [at(8192, 4, 16), at(12288, 64)], [at(8192, 8, 8), at(12288, 32)],     # shapes
                  [at(8192, 8, 8, dtype=torch.int32), at(12288, 64)],                    # type
                  [at(8192 + 1, 8, 8), at(12288, 64)],                                   # alignment
                  [None, at(12288, 64)], [at(8192, 8, 8)], [at(8192, 8, 8), at(12288, 64), at(0, 8)]):
        assert not rec.replay(other)
    assert len(lib.calls) == 2 and b.launches == 2


def test_a_changed_backend_is_not_recorded(monkeypatch):
    from hfcpu_b200.kernels.native import NativeBackend
    t = [torch.zeros(8)]
    b, _ = _native()
    b.linear = lambda *a: None
    assert _recorded(b, t) == ("out", None)
    b, _ = _native()
    with monkeypatch.context() as m:
        m.setattr(NativeBackend, "rmsnorm", lambda *a: None)
        assert _recorded(b, t) == ("out", None)
    assert _recorded(b, t)[1] is not None


def test_calls_outside_a_recording_go_straight_to_the_library():
    """A launch looks the library up two or three times: it is a plain attribute, not asked for through a thread's own storage."""
    b, lib = _native()
    assert b.lib is lib and vars(b)["lib"] is lib
    _recorded(b, [torch.zeros(8)])
    assert vars(b)["lib"] is lib and "_check" not in vars(b)
    with pytest.raises(RuntimeError):
        b.record(lambda: (_ for _ in ()).throw(RuntimeError("a part's own")), [])
    assert vars(b)["lib"] is lib and "_check" not in vars(b)
    assert _recorded(b, [torch.zeros(8)])[1] is not None


def test_another_threads_calls_are_not_in_a_recording():
    import threading
    b, lib = _native()
    t, other = torch.zeros(8), []

    def elsewhere():
        b._check(b.lib.hfb_elsewhere(ctypes.c_int(1)), "elsewhere")
        other.append(b.record(lambda: b._check(b.lib.hfb_second(ctypes.c_int(2)), "second"), [t])[1])

    def run():
        b.lib.hfb_question(ctypes.c_int(0))
        rc = b.lib.hfb_first(ctypes.c_int(0))
        th = threading.Thread(target=elsewhere)
        th.start()
        th.join()
        b._check(rc, "first")
    _, rec = b.record(run, [t])
    assert other == [None] and [c[0] for c in lib.calls] == ["hfb_question", "hfb_first", "hfb_elsewhere", "hfb_second"]
    lib.calls.clear()
    assert rec.replay([t]) and [c[0] for c in lib.calls] == ["hfb_first"]
