"""Each CUDA kernel alone against its plain torch reference, at sizes other than the engine tests'.

Inputs are built so that faults show: a far key among hundreds with a score that stands out, a key
just outside and just inside a window, keys on both sides of a page's edge, scattered pages.
"""
import math
from types import SimpleNamespace

import pytest
import torch

from emu_backend import EmuBackend

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
TOL = {"float32": 2e-5, "bfloat16": 2e-2}


def native():
    from hfcpu_b200 import kernels
    return kernels


@pytest.fixture
def both_tc_forms():
    """Lets small cases reach the attention kernel with two query tiles per CTA, which otherwise waits for enough
    CTAs to fill the SMs three times."""
    b = native().backend()
    old = b.tc2_min_rounds
    b.tc2_min_rounds = 0
    yield b
    b.tc2_min_rounds = old


def rel(a, b):
    return float((a.double() - b.double()).abs().max() / b.double().abs().max().clamp_min(1e-30))


def rnd(*shape, dtype=torch.float32, scale=1.0, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(dtype)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_embed(dtype):
    V, E, T = 777, 200, 45
    table = rnd(V, E, dtype=DT[dtype])
    ids = torch.randint(0, V, (T,), device=DEV, dtype=torch.int32)
    out = torch.empty(T, E, device=DEV)
    native().embed(ids, table, out)
    assert torch.equal(out, table[ids.long()].float())


@pytest.mark.parametrize("E", [48, 200, 3584, 5000])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_rmsnorm(dtype, E):
    x = rnd(37, E, scale=3.0)
    w = rnd(E, dtype=DT[dtype]) + 1
    rows = torch.tensor([36, 0, 5, 5, 17], device=DEV, dtype=torch.int32)
    for r in (None, rows):
        M = 37 if r is None else 5
        out, ref = torch.empty(M, E, device=DEV, dtype=DT[dtype]), torch.empty(M, E, device=DEV, dtype=DT[dtype])
        native().rmsnorm(x, w, 1e-5, out, r)
        EmuBackend().rmsnorm(x, w, 1e-5, ref, r)
        assert rel(out.float(), ref.float()) < (1e-6 if dtype == "float32" else 1e-2)


@pytest.mark.parametrize("E", [64, 1000, 3584, 5000, 8192, 8200])
def test_rmsnorm_many_rows(E):
    """From 64 rows on the bfloat16 form keeps a row in registers (up to 8,192 values): against float64."""
    x = rnd(200, E, scale=3.0)
    w = rnd(E, dtype=torch.bfloat16) + 1
    rows = torch.arange(199, 99, -1, device=DEV, dtype=torch.int32)
    for r in (None, rows):
        src = x if r is None else x[r.long()]
        out = torch.empty(src.shape[0], E, device=DEV, dtype=torch.bfloat16)
        native().rmsnorm(x, w, 1e-6, out, r)
        want = src.double() / torch.sqrt((src.double() ** 2).mean(-1, keepdim=True) + 1e-6) * w.double()
        assert rel(out.double(), want) < 5e-3
        assert torch.equal(out, want.float().to(torch.bfloat16)) or float((out.float() - want.float()).abs().max()) <= float(want.abs().max()) * 2 ** -7


@pytest.mark.parametrize("shape", [(1, 50, 70), (5, 130, 64), (67, 1000, 192), (130, 96, 333), (300, 257, 1030)])
@pytest.mark.parametrize("wdtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_linear(dtype, wdtype, shape):
    M, N, K = shape
    a, w = rnd(M, K, dtype=DT[dtype]), rnd(N, K, dtype=DT[wdtype], scale=0.1)
    bias = rnd(N, dtype=DT[wdtype])
    ref = a.double() @ w.double().T
    out = torch.empty(M, N, device=DEV, dtype=DT[dtype])
    native().linear(a, w, bias, out, False)
    assert rel(out, ref + bias.double()) < (1e-5 if dtype == "float32" else 1e-2)
    res = rnd(M, N, seed=5)
    want = res.double() + ref
    native().linear(a, w, None, res, True)
    assert rel(res, want) < 1e-5
    logits = torch.empty(M, N, device=DEV)
    native().linear(a, w, None, logits, False)
    assert rel(logits, ref) < 1e-5


# the last row count of the streaming form and the first of the tiles; rows and features one beside a tile's edge; an inner size
# of one value, of a piece less one, and sizes that are cut among the CTAs of a cluster (few tiles, long rows), evenly or not
@pytest.mark.parametrize("shape", [(8, 129, 1), (9, 33, 15), (1, 7, 4), (3, 31, 130), (16, 65, 1024), (17, 63, 1028), (128, 128, 2048),
                                   (129, 127, 4100), (64, 64, 260), (333, 896, 1184), (2049, 520, 36)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_linear_plain_forms(dtype, shape):
    """Sums of K products, each rounded to float32: the error of a sum is at most K 2^-24 of the sum of magnitudes, and the
    rounding of a random sign pattern far less; 4 sqrt(K) 2^-24 of the root sum of squares bounds every value here."""
    M, N, K = shape
    b = native()
    a, w = rnd(M, K, dtype=DT[dtype]), rnd(N, K)
    ref = a.double() @ w.double().T
    size = (a.double() ** 2) @ (w.double() ** 2).T                  # sum of squared products
    out = torch.full((M, N), float("nan"), device=DEV)
    b.linear(a, w, None, out, False)
    assert float(((out.double() - ref).abs() / (size.sqrt() * 4 * (K ** 0.5 + 1) * 2 ** -24 + 1e-30)).max()) < 1
    again = torch.empty_like(out)
    b.linear(a, w, None, again, False)
    assert torch.equal(out, again)


# features and inner sizes that are cut into one, two, four and eight slices, into slices of unequal length, a size of no whole pieces;
# few features (blocks of 32 slices of rows) and many (of 128)
@pytest.mark.parametrize("N,K,slices", [(33, 31, 1), (38000, 200, 1), (130, 128, 2), (20000, 260, 2), (1152, 897, 8), (9728, 896, 4), (40, 1028, 8),
                                        (896, 1184, 8), (3584, 520, 8)])
@pytest.mark.parametrize("dtype,wdtype", [("float32", "float32"), ("float32", "bfloat16"), ("bfloat16", "float32")])
def test_plain_product_gives_a_row_the_same_bits_in_any_company(N, K, slices, dtype, wdtype):
    """One order of summation over k whatever the number of rows: the row counts take the streaming form, its templates, the
    three tiles, and slices shared by a cluster as well as taken by one CTA."""
    b = native()
    a, w, bias = rnd(1100, K, dtype=DT[dtype]), rnd(N, K, dtype=DT[wdtype]), rnd(N)
    counts = [1, 2, 4, 5, 8, 9, 16, 17, 64, 65, 129, 333] + ([1100] if N < 4000 else [])

    def product(x, weights):
        out = torch.full((x.shape[0], N), float("nan"), device=DEV)
        b.linear(x, weights, bias, out, False)
        return out

    whole = product(a[:counts[-1]].contiguous(), w)
    assert bool(whole.isfinite().all())
    for m in counts[:-1]:
        assert torch.equal(product(a[:m].contiguous(), w), whole[:m]), m
    # ... and where the weights don't start on whole pieces
    store = torch.empty(N * K + 1, dtype=w.dtype, device=DEV)
    store[1:] = w.flatten()
    for m in (1, 9):
        assert torch.equal(product(a[:m].contiguous(), store[1:].view(N, K)), whole[:m])


@pytest.mark.parametrize("geom", [(5, 1, 48, 48), (6, 3, 32, 16), (8, 8, 128, 128), (2, 2, 256, 64)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_rope_kv_write(dtype, geom):
    H, G, d, n_rot = geom
    T, pages, bs, P = 23, 9, 4, 100
    dt = DT[dtype]
    qkv = rnd(T, (H + 2 * G) * d, dtype=dt)
    ang = torch.rand(P, n_rot // 2, device=DEV, dtype=torch.float64) * 6
    cos_sin = torch.stack([ang.cos(), ang.sin()], -1).float().contiguous()
    positions = torch.randint(0, P, (T,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(pages * bs, device=DEV)[:T].int()
    slots[3] = -1
    outs = []
    for impl in (native(), EmuBackend()):
        q = torch.zeros(T, H * d, device=DEV, dtype=dt)
        kc = torch.zeros(pages, bs, G, d, device=DEV, dtype=dt)
        vc = torch.zeros_like(kc)
        impl.rope_kv_write(qkv, cos_sin, n_rot, positions, slots, q, kc, vc, H, G, d)
        outs.append((q, kc, vc))
    tol = 1e-6 if dtype == "float32" else 1e-2
    for a, b in zip(*outs):
        assert rel(a.float(), b.float()) < tol
    q2 = torch.zeros(T, H * d, device=DEV, dtype=dt)
    kc2 = torch.zeros(pages, bs, G, d, device=DEV, dtype=dt)
    native().rope_kv_write(qkv, cos_sin, n_rot, positions, None, q2, kc2, kc2.clone(), H, G, d)
    assert torch.equal(q2, outs[0][0]) and not kc2.any()


def _attention_case(dtype, H, G, d, bs, lens_q, lens_kv, window, spike=None, seed=0):
    """Builds a paged cache with scattered pages for requests of ``lens_kv`` keys, the last ``lens_q`` of
    them being this step's queries.  ``spike = (request, key position, query offset)`` scales one key and one
    query so that their score stands out."""
    dt = DT[dtype]
    S = len(lens_q)
    MB = max((n + bs - 1) // bs for n in lens_kv)
    pages = sum((n + bs - 1) // bs for n in lens_kv) + 5
    g = torch.Generator().manual_seed(seed)
    perm = torch.randperm(pages, generator=g).tolist()
    table = torch.full((S, MB), -1, dtype=torch.int32)
    kc = rnd(pages, bs, G, d, dtype=dt, seed=seed + 1)
    vc = rnd(pages, bs, G, d, dtype=dt, seed=seed + 2)
    token_seq, positions = [], []
    for s in range(S):
        lo = max(0, lens_kv[s] - lens_q[s] - window + 1) if window > 0 else 0
        for b in range((lens_kv[s] + bs - 1) // bs):
            if b >= lo // bs:                      # blocks a window has passed stay unmapped
                table[s, b] = perm.pop()
        token_seq += [s] * lens_q[s]
        positions += list(range(lens_kv[s] - lens_q[s], lens_kv[s]))
    T = len(token_seq)
    q = rnd(T, H * d, dtype=dt, seed=seed + 3)
    if spike is not None:
        s, key_pos, q_off = spike
        t = sum(lens_q[:s]) + q_off
        page = int(table[s, key_pos // bs])
        assert page >= 0
        direction = torch.ones(d, device=DEV)
        kc[page, key_pos % bs] = (direction * 2).to(dt)
        q.view(T, H, d)[t] = (direction * 2).to(dt)
    meta = SimpleNamespace(block_table=table.to(DEV), block_size=bs, max_blocks=MB)
    ctx = SimpleNamespace(token_seq=torch.tensor(token_seq, dtype=torch.int32, device=DEV),
                          positions=torch.tensor(positions, dtype=torch.int32, device=DEV))
    return q, kc, vc, meta, ctx


def _run_attention(impl, case, H, G, d, window):
    q, kc, vc, meta, ctx = case
    out = torch.empty_like(q)
    impl.paged_attention(q, kc, vc, meta, ctx, H, G, d, window, 1.0 / math.sqrt(d), out, tiles=getattr(ctx, "tiles", None))
    return out


@pytest.mark.parametrize("geom", [(4, 2, 16, 16), (6, 3, 32, 8), (7, 7, 48, 4), (28, 4, 128, 16), (8, 1, 256, 32),
                                  (5, 5, 80, 16)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_attention_mixed_batch(dtype, geom):
    H, G, d, bs = geom
    lens_q, lens_kv = [1, 40, 1, 7, 2], [300, 40, 1, 133, 64]
    for window in (0, 50):
        case = _attention_case(dtype, H, G, d, bs, lens_q, lens_kv, window)
        out, ref = _run_attention(native(), case, H, G, d, window), _run_attention(EmuBackend(), case, H, G, d, window)
        assert rel(out.float(), ref.float()) < TOL[dtype]
    from hfcpu_b200 import kernels
    kernels.check_device_errors()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_attention_far_key_and_page_edges(dtype):
    """One key among hundreds carries nearly all the weight; it sits at a page's first slot, last slot, the
    very first position and the query's own position in turn."""
    H, G, d, bs = 4, 2, 64, 16
    for key_pos in (0, 15, 16, 31, 303, 304, 599):
        case = _attention_case(dtype, H, G, d, bs, [1, 3], [200, 600], 0, spike=(1, key_pos, 2), seed=key_pos)
        out, ref = _run_attention(native(), case, H, G, d, 0), _run_attention(EmuBackend(), case, H, G, d, 0)
        assert rel(out.float(), ref.float()) < TOL[dtype], f"key {key_pos}"


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_attention_window_edge(dtype):
    """A key that would take all the weight lies just outside the window (must be ignored), then just inside."""
    H, G, d, bs, window = 4, 4, 32, 8, 40
    n = 100                                   # the single query sits at position 99 and sees keys 60..99
    for key_pos, inside in ((59, False), (60, True), (99, True)):
        # map the block of key 59 too, so that a kernel that reads one key too many finds the spike
        case = _attention_case(dtype, H, G, d, bs, [1], [n], 0, spike=(0, key_pos, 0), seed=7)
        out, ref = _run_attention(native(), case, H, G, d, window), _run_attention(EmuBackend(), case, H, G, d, window)
        assert rel(out.float(), ref.float()) < TOL[dtype], f"key {key_pos}"
        q, kc, vc, meta, ctx = case
        page = int(meta.block_table[0, key_pos // bs])
        spike_v = vc[page, key_pos % bs, 0].float()
        close = rel(out.view(1, H, d)[0, 0].float(), spike_v) < 0.05
        assert close == inside


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_swiglu(dtype):
    T, F = 33, 999
    gu = rnd(T, 2 * F, dtype=DT[dtype], scale=3)
    out, ref = torch.empty(T, F, device=DEV, dtype=DT[dtype]), torch.empty(T, F, device=DEV, dtype=DT[dtype])
    for inter in (False, True):
        native().swiglu(gu, out, inter)
        EmuBackend().swiglu(gu, ref, inter)
        assert rel(out.float(), ref.float()) < (1e-6 if dtype == "float32" else 1e-2)


@pytest.mark.parametrize("V", [151937, 152064, 4096, 4100, 37])
def test_argmax_lowest_index_wins(V):
    """Rows that allow 16-byte reads (a vocabulary that is a multiple of 4) and rows that do not; ties within a
    16-byte piece, across warps, across chunks; a row of equal values; the maximum in the last, short chunk."""
    logits = rnd(9, V)
    logits[2, V // 2] = logits[2, V - 7] = 50.0
    logits[3, 5] = logits[3, 4] = 60.0
    logits[4] = 1.0
    logits[5, V - 1] = 70.0
    logits[6, 33] = logits[6, 32] = logits[6, 31] = 55.0
    out = torch.empty(9, device=DEV, dtype=torch.int32)
    native().argmax(logits, out)
    assert out.tolist() == torch.argmax(logits, -1).tolist()
    assert out[2] == V // 2 and out[3] == 4 and out[4] == 0 and out[5] == V - 1 and out[6] == 31


def test_refuses_unsupported_head_dim():
    from hfcpu_b200.config.base import UnsupportedError
    with pytest.raises(UnsupportedError):
        native().check_head_dim(40)
    with pytest.raises(UnsupportedError):
        native().check_head_dim(512)


TC_SHAPES = [(1, 128, 64), (1, 3584, 3584), (8, 4608, 3584), (8, 3584, 18944), (16, 1000, 192), (17, 320, 72),
             (64, 3584, 2048), (100, 1000, 200), (128, 512, 512), (129, 256, 64), (130, 1000, 192), (300, 777 * 8, 136),
             (2048, 1024, 512), (1000, 4608, 3584), (5, 152064, 256),
             # from 256 rows on, pairs of CTAs share tiles of 256 rows (cta_group::2): edges of the pair's halves
             (256, 96, 64), (257, 136, 192), (384, 1000, 72), (511, 3000, 320), (1024, 208, 128), (640, 37888 // 8, 256),
             # a few hundred rows, few output tiles and a long inner dimension: split over K (one CTA, and pairs; ragged K)
             (192, 512, 4096), (300, 256, 4168), (384, 520, 1096), (512, 3584, 18944),
             # the o product at 2,048 tokens; ragged in every dimension with pairs
             (2048, 3584, 3584), (1100, 2000, 640), (768, 3000, 1096)]


@pytest.mark.parametrize("shape", TC_SHAPES)
def test_linear_tensor_core(shape):
    """bfloat16 x bfloat16 products on the tcgen05 kernel (both operand orders, split-K, ragged edges) against
    float64, and bit-for-bit stable from call to call."""
    from hfcpu_b200 import kernels
    assert kernels.backend().gemm == "tc"
    M, N, K = shape
    a, w = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.05)
    bias = rnd(N, dtype=torch.bfloat16)
    ref = a.double() @ w.double().T
    scale = float(ref.abs().max())
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    native().linear(a, w, bias, out, False)
    err = float((out.double() - (ref + bias.double())).abs().max()) / float((ref + bias.double()).abs().max())
    assert err < 1e-2, f"bf16 store: {err}"
    logits = torch.empty(M, N, device=DEV)
    native().linear(a, w, None, logits, False)
    assert float((logits.double() - ref).abs().max()) / scale < 2e-5, "float32 store"
    again = torch.empty(M, N, device=DEV)
    native().linear(a, w, None, again, False)
    assert torch.equal(logits, again), "two calls differ"
    res = rnd(M, N, seed=5)
    want = res.double() + ref + bias.double()
    native().linear(a, w, bias, res, True)
    assert float((res.double() - want).abs().max()) / float(want.abs().max()) < 2e-5, "accumulate"
    plain_out = torch.empty(M, N, device=DEV)
    b = kernels.backend()
    b.gemm = "plain"
    try:
        native().linear(a, w, None, plain_out, False)
    finally:
        b.gemm = "tc"
    assert float((logits - plain_out).abs().max()) / scale < 2e-5, "differs from the plain kernel"
    kernels.check_device_errors()


def _with_tiles(case, lens_q, lens_kv, H, G, wide=False):
    """Adds what the tiled kernel needs to a case's context: the tile lists and the step's extents."""
    q, kc, vc, meta, ctx = case
    warps = 1 if max(lens_q) == 1 else (8 if wide else 4)
    dev = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)

    def tiling(per):
        t_seq, t_t0, t_nt, t0 = [], [], [], 0
        for s, n in enumerate(lens_q):
            for a in range(0, n, per):
                t_seq.append(s); t_t0.append(t0 + a); t_nt.append(min(per, n - a))
            t0 += n
        return {"seq": dev(t_seq), "t0": dev(t_t0), "nt": dev(t_nt)}
    ctx.tiles = {f"{warps}.{k}": v for k, v in tiling((16 * warps) // (H // G)).items()}
    if wide:                                                      # the kernel with two 128-row tiles per CTA
        ctx.tiles.update({f"16.{k}": v for k, v in tiling(2 * (128 // (H // G))).items()})
    ws = {}

    def buf(name, shape, dtype):
        return ws.setdefault((name, shape, dtype), torch.empty(shape, dtype=dtype, device=DEV))
    ctx.max_q_len, ctx.max_kv_len, ctx.buf = max(lens_q), max(lens_kv), buf
    return case


FAST_GEOMS = [(28, 4, 128, 16), (14, 2, 64, 16), (6, 3, 64, 8), (4, 4, 128, 64), (16, 1, 64, 4), (8, 2, 128, 32)]


@pytest.mark.parametrize("geom", FAST_GEOMS)
@pytest.mark.parametrize("window", [0, 50, 300])
def test_attention_tiled_mixed_and_decode(geom, window):
    """The tiled tensor-core kernel in both forms: portions beside decode tokens (4 warps), and pure decode
    with the keys split over CTAs (1 warp), against the torch reference and against the plain kernel."""
    from hfcpu_b200 import kernels
    H, G, d, bs = geom
    b = kernels.backend()
    for lens_q, lens_kv, wide in (([1, 70, 1, 7, 2, 130], [300, 70, 1, 133, 64, 700], False),
                                  ([1, 70, 1, 7, 2, 130], [300, 70, 1, 133, 64, 700], True),
                                  ([1, 1, 1, 1, 1], [1, 64, 65, 1000, 2311], False)):
        case = _with_tiles(_attention_case("bfloat16", H, G, d, bs, lens_q, lens_kv, window), lens_q, lens_kv, H, G, wide)
        b.launches = 0
        out = _run_attention(native(), case, H, G, d, window)
        ref = _run_attention(EmuBackend(), case, H, G, d, window)
        assert rel(out.float(), ref.float()) < TOL["bfloat16"], (lens_q, window)
        b.attention = "plain"
        try:
            plain_out = _run_attention(native(), case, H, G, d, window)
        finally:
            b.attention = "fast"
        assert rel(out.float(), plain_out.float()) < TOL["bfloat16"]
        again = _run_attention(native(), case, H, G, d, window)
        assert torch.equal(out, again), "two calls differ"
    kernels.check_device_errors()


def test_attention_tiled_far_key_window_edge_and_page_edges(both_tc_forms):
    H, G, d, bs = 28, 4, 128, 16
    for lens_q, lens_kv, spike_req in (([1, 1], [200, 600], 1), ([5, 40], [200, 600], 1)):
        for key_pos in (0, 15, 16, 63, 64, 303, 304, 559, 560, 599):
            q_off = lens_q[spike_req] - 1
            if key_pos > lens_kv[spike_req] - lens_q[spike_req] + q_off:
                continue
            for window in (0, 40):
                for wide in (False, True, "single"):  # wide: 128-row tiles, the tcgen05 kernels for prompt portions
                    case = _attention_case("bfloat16", H, G, d, bs, lens_q, lens_kv, 0, spike=(spike_req, key_pos, q_off), seed=key_pos)
                    case = _with_tiles(case, lens_q, lens_kv, H, G, bool(wide))
                    native().backend().attention_tc2 = wide != "single"
                    try:
                        out = _run_attention(native(), case, H, G, d, window)
                    finally:
                        native().backend().attention_tc2 = True
                    ref = _run_attention(EmuBackend(), case, H, G, d, window)
                    assert rel(out.float(), ref.float()) < TOL["bfloat16"], (lens_q, key_pos, window, wide)


@pytest.mark.parametrize("shape", [(1, 352, 64), (8, 37888, 3584), (5, 640, 192), (64, 2048, 512), (130, 640, 192),
                                   (300, 2048, 256), (2048, 4096, 512), (7, 352, 70)])
def test_linear_swiglu_fused(shape):
    """The product with the SwiGLU epilogue (both operand orders; odd K falls back to two kernels) against torch."""
    M, N, K = shape
    a, w = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.1)
    gu = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    out = torch.empty(M, N // 2, device=DEV, dtype=torch.bfloat16)
    native().linear_swiglu(a, w, gu, out)
    y = a.double() @ w.double().T
    g, u = y[:, 0::2], y[:, 1::2]
    ref = (g / (1 + torch.exp(-g))) * u
    assert rel(out, ref) < 1.5e-2


@pytest.mark.parametrize("shape", [(1, 3584, 3584), (8, 3584, 18944), (8, 192, 320), (64, 3584, 512), (128, 1000, 64),
                                   (200, 512, 256), (5, 64, 44), (200, 512, 4096), (512, 200, 4104), (320, 1000, 1032)])
@pytest.mark.parametrize("with_norm", [True, False])
def test_linear_residual_norm_fused(shape, with_norm):
    M, N, K = shape
    a, w = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.1)
    bias, nw = rnd(N, dtype=torch.bfloat16), rnd(N, dtype=torch.bfloat16) + 1
    res = rnd(M, N, seed=3)
    res_ref = res.double() + a.double() @ w.double().T + bias.double()
    xn = torch.empty(M, N, device=DEV, dtype=torch.bfloat16) if with_norm else None
    native().linear_residual_norm(a, w, bias, res, nw if with_norm else None, 1e-6, xn)
    assert rel(res, res_ref) < 2e-5
    if with_norm:
        r = 1 / torch.sqrt((res_ref ** 2).mean(-1, keepdim=True) + 1e-6)
        assert rel(xn, res_ref * r * nw.double()) < 1e-2


@pytest.mark.parametrize("geom", [(28, 4, 128, 3584, 8), (6, 3, 32, 192, 5), (4, 2, 16, 64, 1), (8, 8, 64, 512, 130), (5, 1, 48, 100, 3),
                                  (28, 4, 128, 3584, 512), (4, 2, 64, 4096, 200),
                                  # 256 tokens and more: rotation and cache write in the epilogue of the pair kernel (tiles of
                                  # whole heads; a last tile half outside the row; ragged token counts; head size 64)
                                  (28, 4, 128, 3584, 2048), (6, 2, 128, 256, 257), (14, 2, 64, 896, 300), (5, 5, 64, 136, 640)])
def test_linear_rope_kv_fused(geom):
    from hfcpu_b200 import kernels
    H, G, d, K, T = geom
    N = (H + 2 * G) * d
    a, w, bias = rnd(T, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.1), rnd(N, dtype=torch.bfloat16)
    pages, bs, P = max(40, T // 4 + 8), 4, 64
    ang = torch.rand(P, d // 2, device=DEV, dtype=torch.float64) * 6
    cos_sin = torch.stack([ang.cos(), ang.sin()], -1).float().contiguous()
    positions = torch.randint(0, P, (T,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(pages * bs, device=DEV)[:T].int()
    slots[::7] = -1                                      # tokens that are not cached
    outs = []
    b = kernels.backend()
    for impl, in_epilogue in ((native(), True), (native(), False), (EmuBackend(), False)):
        qkv = torch.empty(T, N, device=DEV, dtype=torch.bfloat16)
        q = torch.zeros(T, H * d, device=DEV, dtype=torch.bfloat16)
        kc = torch.zeros(pages, bs, G, d, device=DEV, dtype=torch.bfloat16)
        vc = torch.zeros_like(kc)
        b.rope_in_epilogue = in_epilogue
        before = b.launches
        try:
            impl.linear_rope_kv(a, w, bias, qkv, cos_sin, d, positions, slots, q, kc, vc, H, G, d)
        finally:
            b.rope_in_epilogue = True
        if impl is native() and T >= 256 and d in (64, 128):
            assert b.launches - before == (1 if in_epilogue else 2)
        outs.append((q, kc, vc))
    for x, y, z in zip(*outs):
        assert torch.equal(x, y), "the product's epilogue and the separate kernel differ"
        assert rel(x.float(), z.float()) < 1.5e-2
    kernels.check_device_errors()


@pytest.mark.parametrize("geom", [(28, 4, 128, 16), (4, 4, 128, 8), (16, 1, 128, 128), (5, 5, 128, 32),
                                  (14, 2, 64, 16), (6, 3, 64, 8), (8, 8, 64, 64), (3, 1, 64, 128)])
def test_attention_tensor_core_prompt_portions(geom, both_tc_forms):
    """The tcgen05 attention kernels (head_dim 128 in both forms, two query tiles per CTA and one; head_dim 64 in the
    first): long portions over long histories, several requests, windows, against the torch reference and against
    the mma.sync kernel."""
    from hfcpu_b200 import kernels
    H, G, d, bs = geom
    b = kernels.backend()
    assert b.attention_tc and b.attention_tc2
    for lens_q, lens_kv in (([300, 1, 40], [300, 900, 417]), ([130, 64], [700, 64]), ([2, 1], [2, 1])):
        for window in (0, 100):
            case = _with_tiles(_attention_case("bfloat16", H, G, d, bs, lens_q, lens_kv, window, seed=len(lens_q)), lens_q, lens_kv, H, G, wide=True)
            out = _run_attention(native(), case, H, G, d, window)          # two query tiles per CTA
            ref = _run_attention(EmuBackend(), case, H, G, d, window)
            assert rel(out.float(), ref.float()) < TOL["bfloat16"], (lens_q, window)
            b.attention_tc2 = False
            try:
                single = _run_attention(native(), case, H, G, d, window)   # one query tile per CTA
            finally:
                b.attention_tc2 = True
            assert rel(single.float(), ref.float()) < TOL["bfloat16"], (lens_q, window)
            b.attention_tc = False
            try:
                other = _run_attention(native(), case, H, G, d, window)
            finally:
                b.attention_tc = True
            assert rel(out.float(), other.float()) < TOL["bfloat16"]
            again = _run_attention(native(), case, H, G, d, window)
            assert torch.equal(out, again)
    kernels.check_device_errors()


@pytest.mark.parametrize("geom", [(28, 4, 128, 16), (14, 2, 64, 16)])
@pytest.mark.parametrize("lens_q", [[1, 1], [1, 300]])
def test_attention_long_context_far_keys(lens_q, geom, both_tc_forms):
    """33,000 cached keys: a decode token (the keys split over many CTAs) and a 300-token portion (hundreds of
    tiles per query tile), with one key made to stand out near the start, in the middle and at the very end."""
    H, G, d, bs = geom
    lens_kv = [700, 33000]
    for key_pos in (3, 16384, 32999 - (lens_q[1] - 1)):
        q_off = 0 if key_pos > 30000 else lens_q[1] - 1
        case = _attention_case("bfloat16", H, G, d, bs, lens_q, lens_kv, 0, spike=(1, key_pos, q_off), seed=7)
        case = _with_tiles(case, lens_q, lens_kv, H, G, wide=True)
        out, ref = _run_attention(native(), case, H, G, d, 0), _run_attention(EmuBackend(), case, H, G, d, 0)
        assert rel(out.float(), ref.float()) < TOL["bfloat16"], (lens_q, key_pos)
        t = sum(lens_q[:1]) + q_off
        row = out.view(-1, H, d)[t].float()
        assert rel(row, ref.view(-1, H, d)[t].float()) < TOL["bfloat16"]
    from hfcpu_b200 import kernels
    kernels.check_device_errors()


@pytest.mark.parametrize("geom", [(28, 4, 128, 16), (14, 2, 64, 16), (40, 8, 128, 32), (6, 3, 64, 8)])
def test_attention_short_portions_over_long_context(geom):
    """Portions of 2 to 63 tokens behind thousands of cached keys (the end of a prompt, a prompt behind a shared
    prefix) beside single tokens: their keys are split over CTAs and merged; one key far back made to stand out."""
    from hfcpu_b200 import kernels
    H, G, d, bs = geom
    b = kernels.backend()
    for lens_q, lens_kv in (([9], [3000]), ([2, 33, 1], [9000, 1500, 700]), ([63], [8200])):
        for window, key_pos in ((0, 5), (0, lens_kv[0] - lens_q[0]), (300, lens_kv[0] - lens_q[0] - 250)):
            case = _attention_case("bfloat16", H, G, d, bs, lens_q, lens_kv, window, spike=(0, key_pos, lens_q[0] - 1), seed=key_pos)
            case = _with_tiles(case, lens_q, lens_kv, H, G)
            before = b.launches
            out = _run_attention(native(), case, H, G, d, window)
            assert b.launches - before == 2, "the keys were split (attention and merge)"
            ref = _run_attention(EmuBackend(), case, H, G, d, window)
            assert rel(out.float(), ref.float()) < TOL["bfloat16"], (lens_q, window, key_pos)
            assert torch.equal(out, _run_attention(native(), case, H, G, d, window)), "two calls differ"
    kernels.check_device_errors()


@pytest.mark.parametrize("geom", [(28, 4, 128, 16), (14, 2, 64, 16), (8, 2, 128, 32), (16, 1, 64, 8)])
def test_decode_attention_merges_its_own_splits(geom):
    """The decode kernel with the keys split over CTAs: merged by the CTA that stores a tile's last split, it gives
    what the separate merge kernel gives, in one launch, and leaves its counters at zero."""
    from hfcpu_b200 import kernels
    H, G, d, bs = geom
    b = kernels.backend()
    for lens_kv in ([1, 64, 65, 1000, 2311], [2048] * 8, [700]):
        lens_q = [1] * len(lens_kv)
        for window in (0, 300):
            case = _with_tiles(_attention_case("bfloat16", H, G, d, bs, lens_q, lens_kv, window), lens_q, lens_kv, H, G)
            ref = _run_attention(EmuBackend(), case, H, G, d, window)
            before = b.launches
            out = _run_attention(native(), case, H, G, d, window)
            assert b.launches - before == 1, "one kernel, no separate merge"
            again = _run_attention(native(), case, H, G, d, window)
            b.merge_in_kernel = False
            try:
                apart = _run_attention(native(), case, H, G, d, window)
            finally:
                b.merge_in_kernel = True
            assert torch.equal(out, again) and rel(out.float(), ref.float()) < 3e-2
            assert rel(out.float(), apart.float()) < 1e-2
            assert int(b._counters.abs().sum()) == 0
    kernels.check_device_errors()


# places per expert at the edges of the tensor-core form's tiles (a chunk of 16 or 32 columns, a box of 32 rows, a tile of 256
# places and one beside it), an expert without any; inner sizes of one piece, less and more; features beside a tile's edge
@pytest.mark.parametrize("shape", [((1, 15, 16, 17, 0, 31, 32, 33, 400), 3, 128, 64), ((255, 256, 257, 513, 3), 2, 130, 200),
                                   ((700, 0, 0, 12), 4, 24, 8), ((64, 511), 1, 520, 1032)])
@pytest.mark.parametrize("act", ["none", "relu2", "silu", "clamped"])
def test_grouped_product(shape, act):
    """Both directions of a layer's experts: gathered rows into places of the lists, places into pairs.  Exact products of
    bfloat16 values summed in float32: 4 sqrt(K) 2^-24 of the root sum of squares; times what an activation can add, and one
    rounding to bfloat16 (2^-9) where the output is of that type."""
    counts, top, N, Kd = shape
    b = native()
    E, P = len(counts), -(-sum(counts) // top) * top
    T = P // top
    ids = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)] + [torch.full((P - sum(counts),), E)])
    ids = ids[torch.randperm(P, generator=torch.Generator().manual_seed(P))].to(torch.int32).to(DEV).view(T, top)
    order = torch.empty(P, dtype=torch.int32, device=DEV)
    tiles = [torch.empty(b.moe_max_tiles(P, E), dtype=torch.int32, device=DEV) for _ in range(3)]
    n_tiles = torch.empty(1, dtype=torch.int32, device=DEV)
    b.moe_group(ids, E, order, *tiles, n_tiles)
    n = int(n_tiles)
    assert sorted(order[:sum(counts)].tolist()) == [i for i, e in enumerate(ids.flatten().tolist()) if e < E]
    got = [0] * E
    for e, c in zip(tiles[0][:n].tolist(), tiles[2][:n].tolist()):
        got[e] += c
    assert got == list(counts)
    a, w = rnd(T, Kd, dtype=torch.bfloat16), rnd(E, N, Kd, dtype=torch.bfloat16, scale=Kd ** -0.5)
    glu = act in ("silu", "clamped")
    clamp = (1.5, 1.7, 1.0) if act == "clamped" else None

    def expected(z):
        if act == "relu2":
            return z.clamp_min(0) ** 2
        if act == "silu":
            return torch.nn.functional.silu(z[:, 0::2]) * z[:, 1::2]
        if act == "clamped":
            g, u = z[:, 0::2].clamp(max=1.5), z[:, 1::2].clamp(-1.5, 1.5)
            return g * torch.sigmoid(1.7 * g) * (u + 1.0)
        return z

    bound = 4 * (Kd ** 0.5 + 1) * 2 ** -24
    for src_div, scatter, rows, dt in ((top, False, a, torch.bfloat16), (0, True, rnd(P, Kd, dtype=torch.bfloat16, seed=5), torch.float32)):
        space = {"rows": torch.empty(P, Kd, dtype=torch.bfloat16, device=DEV)} if src_div else {}
        out = torch.full((P, N // 2 if glu else N), 7.0, dtype=dt, device=DEV)
        b.moe_gemm(rows, w, out, act, order, src_div, scatter, *tiles, n_tiles, P, glu=glu, clamp=clamp, **space)
        places = torch.arange(sum(counts), device=DEV)
        pair = order[:sum(counts)].long()
        x = rows[pair // top if src_div else places].double()
        e = ids.flatten()[pair].long()
        want = torch.empty(sum(counts), out.shape[1], dtype=torch.float64, device=DEV)
        for i in range(E):
            if counts[i]:
                want[e == i] = expected(x[e == i] @ w[i].double().T)
        at = pair if scatter else places
        err = (out[at].double() - want).abs()
        # (the factors of a gated pair and the square each carry the sums' error times the other factor, at most about 4 here)
        slack = 16 * bound * float(x.square().sum(-1).mean().sqrt()) + (2 ** -8 if dt == torch.bfloat16 else 2 ** -22) * want.abs()
        assert bool((err <= slack + 1e-12).all()), float((err - slack).max())
        untouched = torch.ones(P, dtype=torch.bool, device=DEV)
        untouched[at] = False
        assert bool((out[untouched] == 7.0).all())                       # no row of a place that does not exist is written
        again = torch.empty_like(out)
        b.moe_gemm(rows, w, again, act, order, src_div, scatter, *tiles, n_tiles, P, glu=glu, clamp=clamp, **space)
        assert torch.equal(out[at], again[at])
    b.check_device_errors()


# tokens whose pairs are above the border of 512 in one step and below it in portions; inner sizes of one piece, several, and many
@pytest.mark.parametrize("T,top,E,N,K", [(200, 4, 9, 136, 1032), (300, 2, 5, 64, 72), (700, 1, 3, 24, 4096), (129, 4, 32, 256, 512), (1100, 1, 2, 40, 136)])
@pytest.mark.parametrize("act", ["none", "relu2", "silu"])
def test_grouped_products_of_every_form_agree_to_the_bit(T, top, E, N, K, act):
    """What a token's experts give does not depend on the number of pairs in its step, nor on whether the caller brings scratch for
    the gathered rows, nor on which entry it calls: tcgen05, mma.sync on tiles of few places and (the entry that is not told how many
    rows its operands have) of many add the same products in the same order.  Values over a wide range of sizes, so that an order
    of its own would show."""
    import ctypes
    b = native()
    lib, ptr = b.backend().lib, lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)
    wide = lambda *shape, seed: (rnd(*shape, seed=seed) * 2.0 ** (3 * rnd(*shape, seed=seed + 1))).bfloat16()
    a, w, hidden = wide(T, K, seed=1), wide(E, N, K, seed=3), wide(T * top, K, seed=5)
    ids = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(t))[:top] for t in range(T)]).to(torch.int32).to(DEV)
    glu = act == "silu"

    def lists(part, tile=0):
        P = part.numel()
        order = torch.empty(P, dtype=torch.int32, device=DEV)
        tiles = [torch.empty(b.moe_max_tiles(P, E, tile), dtype=torch.int32, device=DEV) for _ in range(3)]
        n = torch.empty(1, dtype=torch.int32, device=DEV)
        if tile:
            b.backend().moe_group(part, E, order, *tiles, n, tile)
        else:
            b.moe_group(part, E, order, *tiles, n)
        return order, tiles, n

    def by_pair(out, order):                    # rows in the order of the places -> of the (token, choice) pairs
        y = torch.empty_like(out)
        y[order.long()] = out
        return y

    def up(lo, hi, scratch):
        part, P = ids[lo:hi].contiguous(), (hi - lo) * top
        order, tiles, n = lists(part)
        out = torch.full((P, N // 2 if glu else N), float("nan"), device=DEV)
        rows = {"rows": torch.empty(P, K, dtype=torch.bfloat16, device=DEV)} if scratch else {}
        b.moe_gemm(a[lo:hi].contiguous(), w, out, act, order, top, False, *tiles, n, P, glu=glu, **rows)
        return by_pair(out, order)

    def down(lo, hi):
        part, P = ids[lo:hi].contiguous(), (hi - lo) * top
        order, tiles, n = lists(part)
        out = torch.full((P, N), float("nan"), device=DEV)
        b.moe_gemm(hidden[lo * top:hi * top][order.long()].contiguous(), w, out, "none", order, 0, True, *tiles, n, P)
        return out

    whole, whole_down = up(0, T, True), down(0, T)
    few = 512 // top
    cuts = [(lo, min(lo + few, T)) for lo in range(0, T, few)]
    assert T * top > 512 and bool(whole.isfinite().all())
    assert torch.equal(up(0, T, False), whole)
    assert torch.equal(torch.cat([up(lo, hi, False) for lo, hi in cuts]), whole)
    assert torch.equal(torch.cat([down(lo, hi) for lo, hi in cuts]), whole_down)
    # the entry that is not told the operands' rows: tiles of up to 128 places
    order, tiles, n = lists(ids, 128)
    out = torch.full_like(whole, float("nan"))
    code = b.ACTIVATIONS[act] | (b.ACT_GLU if glu else 0)
    call = lambda tile: lib.hfb_moe_gemm(ptr(a), 1, ptr(w), 1, ptr(out), 0, code, *[ctypes.c_float(0)] * 3, N, K, ptr(order), top, 0, *[ptr(t) for t in tiles], ptr(n),
                                         tiles[0].numel(), tile, b.backend()._stream())
    assert call(128) == 0
    assert torch.equal(by_pair(out, order), whole)
    assert call(129) == 1                       # more places than its tiles hold are refused
    b.check_device_errors()


# rows by columns on both sides of where steps of many tokens take four columns a thread (148 * 4,096 values), the
# last block ragged, and a width that four does not divide
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("M,E,S,top,splits", [(296, 2044, 2, 4, 1), (297, 2044, 2, 4, 1), (300, 2046, 2, 2, 1), (1190, 512, 3, 5, 3), (150, 4100, 8, 1, 2),
                                              (600, 1024, 1, 3, 0)])
def test_stream_tails_of_many_tokens_are_those_of_few(dtype, M, E, S, top, splits):
    """The Dynamic Tanh tail and the write-back of the streams' copies: every value is its own sums in one order, so a step
    gives the bits that the same tokens give in small portions (whose values the tests against float64 cover)."""
    b, dt = native(), DT[dtype]
    y = rnd(max(splits, 1), M, E)
    ey, wts, h = rnd(M * top, E, seed=1), torch.rand(M, top, device=DEV), rnd(M, E, dtype=dt, seed=2)
    ids = torch.randint(0, 6, (M, top), device=DEV, dtype=torch.int32)
    P = [(rnd(1, dtype=dt, seed=3 + i).abs() + 0.2, rnd(E, dtype=dt, seed=4 + i), rnd(E, dtype=dt, seed=5 + i)) for i in range(2)]
    res, x = rnd(M, E, seed=7), rnd(M, S * E, seed=8)
    scale, B, d_out, nxt = rnd(E, dtype=dt, seed=9), rnd(S, S, seed=10), rnd(S, seed=11), rnd(S, seed=12)

    def run(lo, hi):
        r, out = res[lo:hi].clone(), torch.empty(hi - lo, E, dtype=dt, device=DEV)
        mix = (ey[lo * top:hi * top].contiguous(), wts[lo:hi].contiguous())
        b.dyt_residual(y[0, lo:hi].contiguous() if splits else None, P[0], r, P[1], out, mix=mix)
        plain = res[lo:hi].clone()
        b.dyt_residual(y[0, lo:hi].contiguous(), P[0], plain)
        xx, out2 = x[lo:hi].clone(), torch.empty(hi - lo, E, dtype=dt, device=DEV)
        planes = y[:, lo:hi].contiguous()
        sources = [(planes, splits, 0.7), (planes[:1].contiguous(), 1, 1.3)] if splits else []
        b.hc_update(xx, S, sources, mix + (ids[lo:hi].contiguous(), 4, h[lo:hi].contiguous()), scale, B, d_out, nxt, P[1], out2)
        return r, out, plain, xx, out2

    whole = run(0, M)
    parts = [run(lo, min(lo + 64, M)) for lo in range(0, M, 64)]
    for i, got in enumerate(whole):
        assert torch.equal(got, torch.cat([p[i] for p in parts])), i


def cluster_of(M, N, K):
    return native().backend().lib.hfb_linear_tc_cluster(M, N, K)


# more than 128 tokens and few tiles of 128 x 128: eight, four and two CTAs a tile, slices of unequal length, an empty last slice (K of
# 17 and 9 pieces), ragged tokens and features, K that ends inside a piece; then sizes that the tile kernels take (too few pieces of
# K, or more tiles than run at once).  The largest number of tiles for a cluster size is the device's: one size is given a choice
@pytest.mark.parametrize("shape,ctas", [((129, 128, 1088), (8,)), ((256, 896, 4864), (8,)), ((255, 1152, 896), (4,)), ((130, 8, 576), (4,)),
                                        ((640, 896, 904), (2, 4)), ((1000, 1024, 520), (2,)), ((300, 136, 200), (0,)), ((2048, 1024, 136), (0,)),
                                        ((256, 9472, 256), (0,)), ((257, 9480, 72), (0,))])
def test_products_whose_inner_size_a_cluster_shares(shape, ctas):
    assert cluster_of(*shape) in ctas
    check_product_of_many_tokens(*shape)


# (the inner sizes are those with which the products are worth a cluster at all)
@pytest.mark.parametrize("ctas,K", [(8, 1032), (4, 520), (2, 520)])
def test_products_of_as_many_tiles_as_clusters_run_at_once(ctas, K):
    """The most tiles that a cluster size takes on this device, and the first product that it leaves to another form."""
    M, taken = 257, [n for n in range(1, 60) if cluster_of(257, 128 * n, K) == ctas]
    assert taken == list(range(taken[0], taken[-1] + 1)) and 3 * taken[-1] * ctas <= 148
    for N in (128 * taken[-1], 128 * taken[-1] - 120, 128 * taken[-1] + 8):
        check_product_of_many_tokens(M, N, K)


def check_product_of_many_tokens(M, N, K):
    """Exact products of bfloat16 values summed in float32: 4 sqrt(K) 2^-24 of the root sum of squares; one rounding (2^-9)
    where the output is bfloat16."""
    b = native()
    a, w, bias = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16), rnd(N, dtype=torch.bfloat16)
    ref = a.double() @ w.double().T
    bound = (K ** 0.5 + 1) * 4 * 2 ** -24 * ((a.double() ** 2) @ (w.double() ** 2).T).sqrt()
    out = torch.full((M, N), float("nan"), device=DEV)
    b.linear(a, w, bias, out, False)
    want = ref + bias.double()
    assert bool(((out.double() - want).abs() <= bound + 2 ** -23 * want.abs()).all())
    again = torch.empty_like(out)
    b.linear(a, w, bias, again, False)
    assert torch.equal(out, again)
    half = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    b.linear(a, w, bias, half, False)
    assert torch.equal(half, out.bfloat16())
    res = rnd(M, N, seed=3)
    added = res.clone()
    b.linear(a, w, None, added, True)
    assert bool(((added.double() - res.double() - ref).abs() <= bound + 2 ** -23 * (ref.abs() + res.double().abs())).all())
    gated = torch.empty(M, N // 2, dtype=torch.bfloat16, device=DEV)
    b.linear_swiglu(a, (w.double() * K ** -0.5).bfloat16(), torch.empty(M, N, dtype=torch.bfloat16, device=DEV), gated)
    z = a.double() @ (w.double() * K ** -0.5).bfloat16().double().T
    h = torch.nn.functional.silu(z[:, 0::2]) * z[:, 1::2]
    assert bool(((gated.double() - h).abs() <= 2 ** -8 * h.abs() + 1e-4).all())
    b.check_device_errors()


# a cluster, one CTA a tile (129 to 255 tokens with many tiles) and pairs of CTAs; ragged tokens, features beside a tile's edge, K that
# ends inside a piece
@pytest.mark.parametrize("M,F,K,ctas", [(256, 448, 1032, 8), (300, 388, 520, 4), (201, 4740, 136, 0), (601, 4740, 136, 0)])
@pytest.mark.parametrize("act", ["silu", "relu", "gelu_tanh", "relu2", "clamped"])
def test_activations_in_the_epilogues_of_many_tokens(M, F, K, ctas, act):
    """act(g) * u with and without a bias, into an array of its own and into columns of a wider one, in both types; act(z) alone.
    Values around one: a sum is off by at most 4 (sqrt(K) + 1) 2^-24 of the root sum of squares of its products, a gated pair's or a
    square's factors carry that times the other factor (below 16 here), functions and factors a few roundings of 2^-24, which the
    fast quotient and exponential make some 2^-20, and bfloat16 outputs one rounding."""
    b = native()
    assert cluster_of(M, 2 * F, K) == ctas
    a, w, bias = rnd(M, K, dtype=torch.bfloat16), rnd(2 * F, K, dtype=torch.bfloat16, scale=K ** -0.5), rnd(2 * F, dtype=torch.bfloat16)
    clamp = (1.5, 1.7, 1.0) if act == "clamped" else None
    fn = {"silu": torch.nn.functional.silu, "relu": torch.relu, "relu2": lambda z: z.clamp_min(0) ** 2,
          "gelu_tanh": lambda z: torch.nn.functional.gelu(z, approximate="tanh")}.get(act)
    z = a.double() @ w.double().T
    slack = 32 * (K ** 0.5 + 1) * 4 * 2 ** -24 * float((a.double() ** 2).mean().sqrt())

    def check(got, want):
        assert bool(((got.double() - want).abs() <= (2 ** -8 if got.dtype == torch.bfloat16 else 2 ** -18) * want.abs() + slack).all())

    for with_bias in (False, True):
        y = z + bias.double() if with_bias else z
        g, u = y[:, 0::2], y[:, 1::2]
        want = g.clamp(max=1.5) * torch.sigmoid(1.7 * g.clamp(max=1.5)) * (u.clamp(-1.5, 1.5) + 1.0) if clamp else fn(g) * u
        for dtype in (torch.bfloat16, torch.float32):
            for wide in (0, 24):
                store = torch.full((M, F + wide), 7.0, dtype=dtype, device=DEV)
                out = store[:, 8:8 + F] if wide else store
                b.linear_glu(a, w, torch.empty(M, 2 * F, dtype=dtype, device=DEV), out, act, bias=bias if with_bias else None, clamp=clamp)
                check(out, want)
                if wide:
                    assert bool((store[:, :8] == 7.0).all()) and bool((store[:, 8 + F:] == 7.0).all())
    if not clamp:
        for dtype in (torch.bfloat16, torch.float32):
            out = torch.full((M, 2 * F), float("nan"), dtype=dtype, device=DEV)
            b.linear_act(a, w, out, act)
            if act == "silu" and dtype == torch.bfloat16:        # (a pass of its own: the product is rounded before it)
                assert rel(out, fn(z).float()) < 2 ** -7
            else:
                check(out, fn(z))
    b.check_device_errors()


@pytest.mark.parametrize("M,H,G,d,K,ctas", [(129, 14, 2, 64, 896, 4), (256, 14, 2, 64, 896, 4), (300, 6, 2, 128, 1032, 4), (500, 3, 1, 64, 1096, 8),
                                            (500, 16, 2, 64, 520, 2), (1000, 8, 2, 128, 520, 0)])
def test_rotating_product_of_a_cluster(M, H, G, d, K, ctas):
    """q|k|v with rotation and the cache write in the epilogue against the separate kernels: their sums may be cut differently, so
    a value may round to the neighbouring bfloat16 before the rotation (2^-8 of the pair's size).  The last size is the pair
    kernel's."""
    b = native()
    back = b.backend()
    assert cluster_of(M, (H + 2 * G) * d, K) == ctas
    a, w, bias = rnd(M, K, dtype=torch.bfloat16), rnd((H + 2 * G) * d, K, dtype=torch.bfloat16, scale=K ** -0.5), rnd((H + 2 * G) * d, dtype=torch.bfloat16)
    angle = torch.rand(M + 7, d // 2, device=DEV) * 6.28
    cs = torch.stack([angle.cos(), angle.sin()], -1).contiguous()
    pos = torch.randperm(M, device=DEV).to(torch.int32)
    slots = (torch.randperm(M + 16, device=DEV)[:M] - 8).to(torch.int32)           # some tokens are not cached
    pages = (M + 31) // 16
    got = []
    for fused in (True, False):
        old, back.rope_in_epilogue = back.rope_in_epilogue, fused
        q = torch.zeros(M, H * d, dtype=torch.bfloat16, device=DEV)
        kc, vc = (torch.zeros(pages, 16, G, d, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        try:
            b.linear_rope_kv(a, w, bias, torch.empty(M, (H + 2 * G) * d, dtype=torch.bfloat16, device=DEV), cs, d, pos, slots, q, kc, vc, H, G, d)
        finally:
            back.rope_in_epilogue = old
        got.append((q, kc, vc))
    for x, y in zip(*got):
        pair = y.float().unflatten(-1, (-1, d)) if x.dim() == 2 else y.float()
        size = (pair ** 2 + pair.roll(d // 2, -1) ** 2).sqrt().view(y.shape)
        assert bool(((x.float() - y.float()).abs() <= 2 ** -7 * size + 1e-6).all())
        assert float((x != y).float().mean()) < 0.02
    b.check_device_errors()


# few places (an expert's fit one tile of 16 or don't), many (tiles of 256), experts without any, and ids that are no expert
@pytest.mark.parametrize("counts", [(1, 0, 0, 2), (16, 17, 0, 1, 15, 33), (0, 0, 1), (500, 12), (512, 1), (256, 257, 0, 255, 600, 1)])
def test_places_of_the_experts(counts):
    """Every expert's places lie one behind the other, in as few tiles as hold them, all of one size but the last."""
    b = native()
    E, extra = len(counts), 3
    P = sum(counts) + extra
    limit = b.moe_tile(P)
    ids = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)] + [torch.tensor([E, E + 7, -1])])
    ids = ids[torch.randperm(P, generator=torch.Generator().manual_seed(P))].to(torch.int32).to(DEV)
    order = torch.full((P,), -5, dtype=torch.int32, device=DEV)
    tiles = [torch.empty(b.moe_max_tiles(P, E), dtype=torch.int32, device=DEV) for _ in range(3)]
    n_tiles = torch.empty(1, dtype=torch.int32, device=DEV)
    b.moe_group(ids.view(P, 1), E, order, *tiles, n_tiles)
    got = list(zip(*(t[:int(n_tiles)].tolist() for t in tiles)))
    at, want = 0, []
    for e, c in enumerate(counts):
        k = -(-c // limit)
        each = -(-c // k) if k else 0
        want += [(e, at + p, min(each, c - p)) for p in range(0, c, max(each, 1))]
        assert sorted(order[at:at + c].tolist()) == (ids == e).nonzero().flatten().tolist()
        at += c
    assert got == want and order[at:].tolist() == [-5] * extra
    b.check_device_errors()
