"""Window attention of prompts with heads of 128 through the engine (lp_window_attn_prompt, csrc/lp_split32.cu): every visibility rule and option, portions
behind pages that the window has given back, several ragged requests, against float64 on the same prepared queries and cache rows, and beside
lp_window_attn_tiles, which has the rows that the rule leaves it.

Bound: sums of fp32 rows on short chains measure 1.1e-7 to 1.8e-7 of the result here, as those of lp_window_attn_tiles do (1.2e-7 to 2.2e-7); 2.5e-7."""
import math

import pytest
import torch

from leopard_b200 import _lib, seqlm
from leopard_b200.seqlm import LayerConfig, RotaryConfig, SeqLMConfig, SeqLMEngine, SeqLMWeights, StepEntry, WindowAttentionConfig, _Batch

F32, F64, D = torch.float32, torch.float64, 128
pytestmark = pytest.mark.gpu
BOUND = 2.5e-7


@pytest.fixture(autouse=True)
def every_size(request, monkeypatch):
    """the tensor-core kernel has rows of any number here, but where the rule is what is tested"""
    if "rule" not in request.node.name:
        for name in ("WINDOW_FULL_ROWS", "WINDOW_TILE_ROWS", "WINDOW_WORK", "WINDOW_WORK_F32"):
            monkeypatch.setattr(seqlm, name, 0)


def engine(heads, kv_heads, dtype="float32", max_tokens=2048, width=64, **options):
    m = WindowAttentionConfig(heads=heads, kv_heads=kv_heads, dim=D, vdim=D, scale=D ** -0.5, rot=RotaryConfig(dims=32, base=1e4), **options)
    cfg = SeqLMConfig(architecture="window", vocab=64, width=width, eps=1e-6, layers=(LayerConfig(mixer=m, ff=None),), norm="pre")
    shapes = {"embed": (64, width), "head": (64, width), "final.norm": (width,), "norm1": (width,), "mix.q": (heads * D, width), "mix.k": (kv_heads * D, width),
              "mix.v": (kv_heads * D, width), "mix.o": (width, heads * D), "mix.g": (heads * D, width)}
    w = SeqLMWeights(cfg, lambda name: torch.full(shapes[name], 0.125), lambda layer, key: key, "cuda")
    return SeqLMEngine(cfg, w, dtype=dtype, max_tokens=max_tokens, page_size=16, max_seqs=4, lib=_lib.stream32_lib()), m


def reference(eng, m, lw, batch, qkv):
    """float64 from the prepared queries (first columns of qkv), the cache and the block means"""
    H, G, out = m.heads, m.kv_heads, []
    pool, summary = eng.cache.pools[0], eng.cache.summary_pool(0) if m.pool else None
    for s, n, r0 in zip(batch.seqs, batch.lens, batch.seq_row0.tolist()):
        first, total = s.length, s.length + n
        pages = torch.tensor(s.pages, device="cuda").clamp_min(0)      # given back: no row sees them
        rows = pool[pages].flatten(0, 1)[:total].double()
        pos, j = torch.arange(first, total, device="cuda")[:, None], torch.arange(total, device="cuda")[None]
        lo = (pos - m.window + 1).clamp_min(0) if m.window else torch.zeros_like(pos)
        if m.chunk:
            lo = torch.maximum(lo, pos // m.chunk * m.chunk)
        seen = (j <= pos) & ((j >= lo) | (j < m.keep_first))
        if m.pool:
            means = summary[torch.tensor(s.summary_pages[0], device="cuda")].flatten(0, 1)[:total // m.pool].double()
            b = torch.arange(means.shape[0], device="cuda")[None]
            rows, seen = torch.cat([rows, means]), torch.cat([seen, (b + 1) * m.pool <= pos - m.window + 1], 1)
        rows = torch.where(seen.any(0)[:, None] & rows.isfinite(), rows, torch.zeros((), dtype=F64, device="cuda"))      # (a value that is not finite counts as none)
        heads = []
        for h in range(H):
            g = h // (H // G)
            score = qkv[r0:r0 + n, h * D:(h + 1) * D].double() @ rows[:, g * D:(g + 1) * D].T * m.scale
            if m.softcap:
                score = m.softcap * torch.tanh(score / m.softcap)
            score = torch.cat([score.masked_fill(~seen, -math.inf), torch.full((n, 1), 0.0 if m.sink else -math.inf, dtype=F64, device="cuda")], 1)
            v = 0 if m.values_are_keys else G * D
            o = torch.softmax(score, 1)[:, :-1] @ rows[:, v + g * D:v + (g + 1) * D]
            if m.value_rot:
                angle = (pos * lw["v_inv_freq"][None]).double()
                k = angle.shape[1]
                a, c = (slice(0, 2 * k, 2), slice(1, 2 * k, 2)) if m.value_rot.layout == "interleaved" else (slice(0, k), slice(k, 2 * k))
                x, y = o[:, a].clone(), o[:, c].clone()
                o[:, a], o[:, c] = x * angle.cos() + y * angle.sin(), y * angle.cos() - x * angle.sin()
            heads.append(o)
        out.append(torch.cat(heads, 1))
    out = torch.cat(out)
    return out * torch.sigmoid(qkv[:, qkv.shape[1] - H * D:].double()) if m.out_gate else out


def portion(eng, m, lens, seed, plant=None, expect=True):
    """one step of requests 0, 1, .. : its results by both kernels and in 64 bits"""
    lw, parts = eng.w.layers[0], m.heads + m.kv_heads * (1 if m.values_are_keys else 2) + (m.heads if m.out_gate else 0)
    batch = _Batch(eng, [StepEntry(i, [1] * n, []) for i, n in enumerate(lens)])
    raw = torch.randn((batch.R, parts * D), device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
    got, taken, inner = [], [], eng._window_prompt      # `taken`: whether lp_window_attn_prompt has had them
    if plant is not None:
        plant(batch)
    for take in (True, False):
        eng._window_prompt = lambda *a: taken.append(take and inner(*a)) or taken[-1]
        qkv, o = raw.clone(), torch.full((batch.R, m.heads * D), 9.0, device="cuda", dtype=eng.act)
        eng._window_heads(0, m, lw, raw, batch, o, qkv)
        got.append(o.double())
    eng._window_prompt = inner
    assert taken == [expect, False]
    want = reference(eng, m, lw, batch, qkv)
    for s, n in zip(batch.seqs, batch.lens):
        eng.cache.advance(s, n)
    return (*got, want)


def error(a, want):
    return float((a - want).norm() / want.norm())


HALF, INTER = RotaryConfig(dims=64, base=100.0), RotaryConfig(dims=24, base=100.0, layout="interleaved")
FORMS = {
    "kept, gate": (4, 1, dict(window=40, keep_first=3, out_gate=True)),
    "pooled, cap, turned": (6, 2, dict(window=48, pool=8, softcap=30.0, value_rot=HALF)),
    "own block, sink": (2, 2, dict(chunk=48, sink=True)),
    "window and own block": (2, 1, dict(window=30, chunk=64)),
    "values are keys": (3, 1, dict(window=100, values_are_keys=True, sink=True)),
    "all, turned in pairs": (2, 1, dict(value_rot=INTER)),
    "pooled and kept, cap": (2, 1, dict(window=33, pool=5, keep_first=7, softcap=4.0, out_gate=True)),
}
PORTIONS = [(33, 130), (300, 5), (1, 129), (70, 256), (2, 64)]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("form", sorted(FORMS))
def test_portions_of_two_requests(form, dtype):
    heads, kv_heads, options = FORMS[form]
    eng, m = engine(heads, kv_heads, dtype, **options)
    for i, lens in enumerate(PORTIONS):
        got, _, want = portion(eng, m, lens, i)
        assert error(got, want) < (BOUND if dtype == "float32" else 3e-3)      # a bf16 result is rounded to 2^-9
    if "window" in options:
        assert -1 in eng.cache.get(0).pages


def test_a_row_that_sees_one_key_has_its_value():
    """exactly: its weight is one, and the value's three terms add up to it"""
    eng, m = engine(64, 2, chunk=16)
    got, _, want = portion(eng, m, (200,), 0)
    assert torch.equal(got[::16], want[::16])


@pytest.mark.parametrize("bad", [math.inf, math.nan])
def test_a_value_that_is_not_finite_stays_with_the_rows_that_see_it(bad):
    eng, m = engine(2, 1, window=100)
    portion(eng, m, (300,), 0)

    def plant(batch):      # position 250, channel 5 of the values: rows 300 .. 349 see it
        eng.cache.pools[0][batch.seqs[0].pages[250 // 16], 250 % 16, D + 5] = bad
    got, _, want = portion(eng, m, (150,), 1, plant)
    odd = torch.zeros_like(want, dtype=torch.bool)
    odd[:50, 5::D] = True
    assert torch.equal(~got.isfinite(), odd) and (bool(got[odd].isnan().all()) if math.isnan(bad) else bool((got[odd] == bad).all()))
    # these rows were taken again one multiply-add after the other: a rounding of 2^-24 for each of the 128 of a score, of either sign
    assert error(got[~odd], want[~odd]) < 2.0 ** -24 * 128 ** 0.5


@pytest.mark.parametrize("heads,kv_heads,options,lens", [
    (16, 4, dict(window=1024, keep_first=4), [(4096,)]), (16, 4, dict(window=512, pool=64, softcap=30.0), [(2048,)]), (8, 8, dict(window=256), [(2000,)]),
    (16, 4, dict(window=1024), [(3000,), (640,)]), (16, 4, dict(window=256, pool=16, softcap=6.0), [(700, 300)]), (32, 8, dict(), [(500,)]), (64, 64, dict(), [(200,)])])
def test_errors_are_no_larger_than_those_of_the_tiles(heads, kv_heads, options, lens):
    """of fp32 results (measured 0.73 to 0.95 of them)"""
    eng, m = engine(heads, kv_heads, max_tokens=8192, **options)
    for i, portions in enumerate(lens):
        got, tiles, want = portion(eng, m, portions, i)
        assert error(got, want) < min(BOUND, error(tiles, want))


@pytest.mark.parametrize("dtype,width,heads,lens,taken", [
    ("float32", 1000, 16, (625,), True), ("float32", 1000, 16, (624,), False), ("bfloat16", 1744, 16, (896,), True), ("bfloat16", 1736, 16, (896,), False),
    ("float32", 4000, 64, (112, 112), True), ("float32", 4000, 64, (112, 111), False), ("float32", 4000, 63, (224,), True), ("float32", 4000, 63, (129,), False),
    ("float32", 4000, 64, (64, 64), False), ("float32", 4000, 64, ((200, 64), (184, 64)), True), ("float32", 4000, 64, ((200, 64), (183, 64)), False),
    ("float32", 4000, 64, ((200, 64), (400, 63)), False)])
def test_both_sides_of_the_rule(dtype, width, heads, lens, taken):
    """rows x heads x width of 10 million in fp32, 25 million in bf16; 112 rows a tile of 128, or 64 where the keys are four times the rows (here: (past, rows))"""
    eng, m = engine(heads, 1, dtype, width=width)
    for i, n in enumerate(lens):
        if isinstance(n, tuple):
            eng.cache.reserve(eng.cache.open(i), n[0])
            eng.cache.advance(eng.cache.get(i), n[0])
    batch = _Batch(eng, [StepEntry(i, [1] * (n[1] if isinstance(n, tuple) else n), []) for i, n in enumerate(lens)])
    calls, L = [], eng.L

    class Spy:
        def __getattr__(self, name):
            if name in ("lp_window_attn_prompt", "lp_window_attn_tiles"):
                calls.append(name)
            return getattr(L, name)
    qkv = torch.zeros((batch.R, (heads + 2 * m.kv_heads) * D), device="cuda")
    eng.L = Spy()
    eng._window_heads(0, m, eng.w.layers[0], qkv, batch, torch.empty((batch.R, heads * D), device="cuda", dtype=eng.act), qkv)
    assert calls[-1] == ("lp_window_attn_prompt" if taken else "lp_window_attn_tiles")


def test_rows_that_leave_no_room_for_planes(monkeypatch):
    """earlier tokens' planes beyond the limit, or an allocation that fails: lp_window_attn_tiles has the rows; this step's own planes have no limit"""
    monkeypatch.setattr(seqlm, "SCRATCH_BYTES", 6 * 299 * 2 * D)
    eng, m = engine(64, 1)
    for seed, (n, expect) in enumerate([(299, True), (130, True), (130, False)]):      # behind 0, 299 and 429 tokens
        got, tiles, want = portion(eng, m, (n,), seed, expect=expect)
        assert error(got, want) < 4e-7 and (expect or torch.equal(got, tiles))
    inner = eng._empty

    def full(shape, dtype):
        if dtype == torch.uint8:
            raise torch.OutOfMemoryError("no room")
        return inner(shape, dtype)
    monkeypatch.setattr(seqlm, "SCRATCH_BYTES", 1 << 30)
    eng._empty = full
    portion(eng, m, (130,), 9, expect=False)
