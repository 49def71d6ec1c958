"""Products of up to eight tokens from the stream on, against float64, at the edges of what the kernel takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
D = "cuda:0"
# (features, inner): less than a group of eight rows a block, ragged groups, an inner size below and beside a chunk of 32, shares of
# one to twelve groups an SM, the 0.5B and width-1,024 sizes
SIZES = [(8, 8), (40, 72), (152, 1000), (896, 896), (2400, 264), (5472, 1024), (896, 4864), (9728, 896), (14200, 136)]
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
        assert torch.equal(a == 0, c == 0) or (a.double() - c.double()).abs().max() <= top
    assert float((got[0].double() - want[0].double()).norm() / want[0].double().norm()) < 5e-3


def test_few_tokens_refuses_what_it_does_not_take():
    kernels = _kernels()
    nw = torch.ones(896, device=D)
    small = torch.zeros(896, 896, device=D, dtype=torch.bfloat16)
    assert kernels.few_tokens(8, torch.bfloat16, (nw, 1e-6), small) and not kernels.few_tokens(9, torch.bfloat16, (nw, 1e-6), small)
    assert not kernels.few_tokens(1, torch.float32, (nw, 1e-6), small)
    assert not kernels.few_tokens(1, torch.bfloat16, (nw, 1e-6), torch.zeros(151936, 896, device=D, dtype=torch.bfloat16))
    assert not kernels.few_tokens(1, torch.bfloat16, (torch.ones(897, device=D)[1:], 1e-6), small)


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
        got = []
        for record in (True, False):
            eng = hfcpu_b200.Engine(model, block_size=16, max_tokens=2048, max_requests=4)
            eng.use_graphs = False
            saved = kernels.recorder
            if not record:
                kernels.recorder = lambda: None
            try:
                eng.add_request("a")
                eng.add_request("b")
                outs = []
                for n in (300, 40, 3, 1, 1):
                    outs.append(eng.step([hfcpu_b200.StepEntry(r, [(7 * i + n) % 1000 for i in range(n)], [n - 1]) for r in "ab"]).clone())
                got.append(torch.stack(outs))
            finally:
                kernels.recorder = saved
        assert torch.equal(got[0], got[1])
