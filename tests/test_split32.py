"""The SOURCE of leopard_b200/csrc/lp_split32.cu executed on the CPU (tests/emu/tc_emu.h): fp32 operands as three planes of bf16 terms, the
product and the attention kernel on them, against float64.  Errors are those of fp32 sums: the terms add up to their number exactly, so a
product of K terms differs from float64 by at most K roundings of 2^-24 of the sum of magnitudes, in practice far less."""
import ctypes as C
import math
import subprocess
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parents[1]
F32, BF, F64 = torch.float32, torch.bfloat16, torch.float64


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    out = tmp_path_factory.mktemp("emu_split32")
    common = (ROOT / "leopard_b200/csrc/lp_common.cuh").read_text()
    a = common.rindex("// ----", 0, common.index("// UMMA descriptors"))
    (out / "emu_helpers.inc").write_text("namespace lp {\n" + common[a:common.rindex("}  // namespace lp")] + "\n}\n")
    lib = out / "libsplit32.so"
    r = subprocess.run(["g++", "-std=c++20", "-O2", "-pthread", "-shared", "-fPIC", "-I", str(out), "-I", str(ROOT / "tests/emu"),
                        str(ROOT / "tests/emu/split32_emu.cpp"), "-o", str(lib)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return C.CDLL(str(lib))


def P(t):
    return C.c_void_p(t.data_ptr() if t is not None else None)


def LL(n):
    return C.c_longlong(n)


def planes(emu, x):
    """[3][rows][cols] of fp32 [rows, cols]"""
    x = x.contiguous()
    p = torch.empty((3, *x.shape), dtype=BF)
    emu.emu_split_rows(P(x), LL(x.shape[1]), x.shape[0], x.shape[1], P(p), LL(x.shape[1]), LL(x.numel()))
    return p


def test_terms_add_up_exactly(emu):
    g = torch.Generator().manual_seed(1)
    x = torch.randn((37, 64), generator=g) * torch.exp(torch.randn((37, 64), generator=g) * 8)
    x[0, :6] = torch.tensor([float("inf"), -float("inf"), float("nan"), 0.0, -0.0, 3.4028e38])
    p = planes(emu, x).double()
    total = p[0] + p[1] + p[2]
    fin = torch.isfinite(x)
    assert torch.equal(total[fin], x.double()[fin])
    assert torch.equal(total[0, :2].float(), x[0, :2]) and bool(torch.isnan(total[0, 2]))


@pytest.mark.parametrize("M,N,K,bn,ctas,out", [(130, 136, 72, 128, 2, 1), (40, 264, 200, 256, 1, 1), (128, 128, 64, 128, 1, 0), (257, 128, 328, 128, 3, 2),
                                               (100, 392, 136, 256, 2, 2)])
def test_product_of_three_planes(emu, M, N, K, bn, ctas, out):
    g = torch.Generator().manual_seed(M + N)
    x, w, bias = torch.randn((M, K), generator=g), torch.randn((N, K), generator=g).to(BF), torch.randn(N, generator=g)
    p = planes(emu, x)
    c = torch.full({0: (M, N), 1: (M, N), 2: (3, M, N)}[out], float("nan"), dtype=F32 if out == 1 else BF)
    emu.emu_gemm_split(P(p), LL(K), LL(M * K), P(w), LL(K), P(c), LL(N), LL(M * N), out, M, N, K, P(bias), bn, ctas)
    want = x.double() @ w.double().T + bias.double()
    got = c.double().sum(0) if out == 2 else c.double()
    assert float((got - want).norm() / want.norm()) < (4e-3 if out == 0 else 5e-7)


@pytest.mark.parametrize("groups,tile_group,N,K,gated,out,ctas,split", [(3, [2, -1, 0], 272, 136, True, 0, 2, False), (2, [1, 1], 144, 72, False, 1, 3, False),
                                                                        (2, [0, 1, -1], 304, 200, True, 1, 1, False), (4, [3], 256, 64, False, 0, 1, False),
                                                                        (2, [1, -1, 0], 272, 136, True, 2, 2, True), (3, [2, 0], 144, 200, False, 1, 1, True)])
def test_grouped_product(emu, groups, tile_group, N, K, gated, out, ctas, split):
    """bf16 rows, or fp32 rows in planes; an infinite weight beside a row that is zero there gives what fp32 multiply-adds give"""
    g, rows, n_out = torch.Generator().manual_seed(N), 128 * len(tile_group), N // 2 if gated else N
    a, w = torch.randn((rows, K), generator=g), (torch.randn((groups, N, K), generator=g) / K ** 0.5).to(BF)
    if split:
        w[:, 3, 5] = float("inf")      # (a gate, or a row of its own)
        a[7, 5], a[8:, 5] = 1.0, -a[8:, 5].abs() - 0.1
        a[:7, 5] = a[:7, 5].abs() + 0.1
    else:
        a = a.to(BF)
    scale = torch.rand(rows, generator=g) + 0.1 if gated else None
    c = torch.full((3, rows, n_out) if out == 2 else (rows, n_out), float("nan"), dtype=F32 if out == 1 else BF)
    tg = torch.tensor(tile_group, dtype=torch.int32)
    p = planes(emu, a) if split else a
    emu.emu_gemm_grouped(P(p), LL(rows * K if split else 0), P(w), groups, P(tg), len(tile_group), int(gated), P(scale), P(c), LL(rows * n_out), out, N, K, ctas)
    for t, e in enumerate(tile_group):
        r = slice(128 * t, 128 * t + 128)
        got = c[:, r].double().sum(0) if out == 2 else c[r].double()
        if e < 0:
            assert bool(torch.isnan(got).all())
            continue
        y = a[r].double() @ w[e].double().T
        if gated:
            y = y * scale[r, None].double()
            y = torch.nn.functional.silu(y[:, :N // 2]) * y[:, N // 2:]
        fin = torch.isfinite(y)
        assert float((got[fin] - y[fin]).norm() / y[fin].norm()) < (4e-3 if out == 0 else 1e-6)
        if split and not gated:
            assert torch.equal(got[:, 3], y[:, 3])      # infinities of the rows' signs


def test_product_with_infinite_weight(emu):
    """as fp32 multiply-adds: an infinite weight gives infinities, zero times it NaN"""
    x, w = torch.randn((5, 64), generator=torch.Generator().manual_seed(3)), torch.ones((128, 64)).to(BF)
    x[1, 7] = 0.0
    w[9, 7] = float("inf")
    p, c = planes(emu, x), torch.zeros((5, 128))
    emu.emu_gemm_split(P(p), LL(64), LL(5 * 64), P(w), LL(64), P(c), LL(128), LL(0), 1, 5, 128, 64, P(None), 128, 1)
    for r in range(5):
        assert bool(torch.isnan(c[r, 9])) if r == 1 else float(c[r, 9]) == math.copysign(math.inf, float(x[r, 7]))
    assert bool(torch.isfinite(c[:, :9]).all()) and bool(torch.isfinite(c[:, 10:]).all())


def seen(pos, window, chunk=0, keep_first=0, pool=0):
    """(kept tokens, blocks, first token) that a query at `pos` sees"""
    lo = max(0, pos - window + 1) if window else 0
    if chunk:
        lo = max(lo, pos // chunk * chunk)
    return min(keep_first, lo), ((pos - window + 1) // pool if pool and window and pos - window + 1 > 0 else 0), lo


def run_keys(p0, n, *rule):
    """the key rows of a request that brings n tokens from position p0 on"""
    keep, blocks, _ = seen(p0 + n - 1, *rule)
    return [("token", t) for t in range(keep)] + [("block", t) for t in range(blocks)] + [("token", t) for t in range(seen(p0, *rule)[2], p0 + n)]


def reference(q, k, kr, v, lens, pos0, rule, scale, heads, softcap=0.0, sink=None, gate=None, out_gate=None, turn=None):
    """float64; keys and values lie request by request as run_keys says; sink: a score per head that joins the denominator"""
    R, H, kvh = q.shape[0], heads, v.shape[1] // 128
    dq = q.shape[1] // H
    out, r, base = torch.zeros((R, H * 128), dtype=F64), 0, 0
    for n, p0 in zip(lens, pos0):
        run = run_keys(p0, n, *rule)
        n_blocks, n_keep = sum(kind == "block" for kind, _ in run), seen(p0 + n - 1, *rule)[0]
        for i in range(n):
            keep, blocks, lo = seen(p0 + i, *rule)
            first = seen(p0, *rule)[2]
            at = list(range(keep)) + list(range(n_keep, n_keep + blocks)) + [n_keep + n_blocks + t - first for t in range(lo, p0 + i + 1)]
            at = torch.tensor(at) + base
            for h in range(H):
                c = slice(h // (H // kvh) * 128, h // (H // kvh) * 128 + 128)
                kk = k[at][:, c].double()
                if kr is not None:
                    kk = torch.cat([kk, kr[at].double()], 1)
                s = kk @ q[r, h * dq:(h + 1) * dq].double() * scale
                if softcap:
                    s = softcap * torch.tanh(s / softcap)
                top = max(float(s.max()), float(sink[h]) if sink is not None else -math.inf)
                e = torch.exp(s - top)
                den = e.sum() + (math.exp(float(sink[h]) - top) if sink is not None else 0.0)
                o = e @ v[at][:, c].double() / den
                if turn is not None:      # frequencies and layout
                    angle = (p0 + i) * turn[0].double()
                    m = len(angle)
                    u, w = (o[0:2 * m:2].clone(), o[1:2 * m:2].clone()) if turn[1] else (o[:m].clone(), o[m:2 * m].clone())
                    u, w = u * torch.cos(angle) + w * torch.sin(angle), w * torch.cos(angle) - u * torch.sin(angle)
                    if turn[1]:
                        o[0:2 * m:2], o[1:2 * m:2] = u, w
                    else:
                        o[:m], o[m:2 * m] = u, w
                if gate is not None:
                    o = o * torch.sigmoid(gate[r, h].double())
                out[r, h * 128:(h + 1) * 128] = o
            r += 1
        base += len(run)
    return out * torch.sigmoid(out_gate.double()) if out_gate is not None else out


@pytest.mark.parametrize("lens,pos0,window,rot,opts", [
    ([130], [0], 0, True, {}), ([40, 129], [300, 0], 100, True, {"sink": True}), ([257], [70], 150, False, {"gates": True}),
    ([3, 1, 20], [0, 500, 127], 0, True, {}), ([200], [0], 40, False, {"keep": 4, "ratio": 2}), ([150, 30], [100, 900], 64, False, {"pool": 8, "cap": 3.0}),
    ([140], [20], 30, False, {"keep": 5, "pool": 3, "sink_one": True, "turn": (64, False)}), ([20], [9], 16, False, {"turn": (24, True), "pool": 2}),
    ([160, 9], [50, 7], 90, False, {"chunk": 32})])
def test_attention_of_three_planes(emu, lens, pos0, window, rot, opts):
    H, R, dq, ratio = 2, sum(lens), 192 if rot else 128, opts.get("ratio", 1)
    g = torch.Generator().manual_seed(R)
    rule = (window, opts.get("chunk", 0), opts.get("keep", 0), opts.get("pool", 0))
    n_keys = sum(len(run_keys(p, n, *rule)) for n, p in zip(lens, pos0))
    q, k = 2 * torch.randn((R, H * dq), generator=g), torch.randn((n_keys, H // ratio * 128), generator=g)
    kr, v = torch.randn((n_keys, 64), generator=g) if rot else None, torch.randn((n_keys, H // ratio * 128), generator=g)
    sink = torch.randn(H, generator=g) if "sink" in opts else None
    gate, og = (torch.randn((R, H), generator=g), torch.randn((R, H * 128), generator=g)) if "gates" in opts else (None, None)
    row0 = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    p0 = torch.tensor(pos0, dtype=torch.int32)
    out = torch.full((R, H * 128), float("nan"))
    tiles = sum(-(-n // 128) for n in lens)
    half, inter = opts.get("turn", (0, False))
    freq, table = 10.0 ** -torch.linspace(0, 2, max(half, 1)), torch.empty((R, max(half, 1), 2))

    def run():
        p = [planes(emu, x) if x is not None else None for x in (q, k, kr, v)]
        emu.emu_attn32(*[P(x) for x in p], R, H, ratio, len(lens), *rule, P(row0), P(p0), tiles, n_keys, C.c_float(dq ** -0.5),
                       C.c_float(opts.get("cap", 0.0)), int("sink_one" in opts), P(sink), P(gate), P(og), P(freq), half, int(inter), P(table),
                       P(out), 1)
    run()
    want = reference(q, k, kr, v, lens, pos0, rule, dq ** -0.5, H, opts.get("cap", 0.0), torch.zeros(H) if "sink_one" in opts else sink, gate, og,
                     (freq, inter) if half else None)
    assert float((out.double() - want).norm() / want.norm()) < 1e-6
    if "sink" in opts or "pool" in opts:      # a value that is not finite reaches only the rows that see it
        v[n_keys - 1, 3] = float("inf")
        run()
        assert not bool(torch.isfinite(out[R - 1, 3])) and bool(torch.isfinite(out[: R - 1]).all())
        assert half or bool(torch.isfinite(out[R - 1, 4:128]).all())
        assert float((out[: R - 1].double() - want[: R - 1]).norm() / want.norm()) < 1e-6


def serial_stats(emu):
    """(fewest registers of a thread that took results again, MMAs issued before the first one did or -1, MMAs) since the last call"""
    regs, first, total = C.c_int(), C.c_long(), C.c_long()
    emu.emu_serial_stats(C.byref(regs), C.byref(first), C.byref(total))
    return regs.value, first.value, total.value


@pytest.mark.parametrize("rot", [False, True])
def test_rows_are_taken_again_by_warps_that_have_the_registers(emu, rot):
    """the warps that load and multiply give registers up when they start: what takes rows again was compiled for as many as a thread starts with (168)"""
    R, keys, dq = 40, 200, 192 if rot else 128
    g = torch.Generator().manual_seed(R)
    q, k, v = torch.randn((R, dq), generator=g), torch.randn((keys, 128), generator=g), torch.randn((keys, 128), generator=g)
    kr = torch.randn((keys, 64), generator=g) if rot else None
    row0, p0 = torch.tensor([0, R], dtype=torch.int32), torch.tensor([keys - R], dtype=torch.int32)
    out = torch.empty((R, 128))
    for bad in (False, True):
        if bad:
            v[keys - 3, 9] = math.inf
        p = [planes(emu, x) if x is not None else None for x in (q, k, kr, v)]
        serial_stats(emu)
        emu.emu_attn32(*[P(x) for x in p], R, 1, 1, 1, 0, 0, 0, 0, P(row0), P(p0), 1, keys, C.c_float(dq ** -0.5), C.c_float(0.0), 0, P(None), P(None), P(None),
                       P(None), 0, 0, P(None), P(out), 1)
        regs, first, total = serial_stats(emu)
        assert (first == total and regs >= 168) if bad else first == -1
    want = reference(q, k, kr, v, [R], [keys - R], (0,), dq ** -0.5, 1)
    assert torch.equal(out.isinf(), want.isinf()) and float((out[:-3].double() - want[:-3]).norm() / want[:-3].norm()) < 1e-6


def test_a_closed_gate_does_not_hide_a_nan(emu):
    """zero times NaN is NaN: rows of a head whose gate's sigmoid is zero"""
    R, H = 3, 2
    g = torch.Generator().manual_seed(2)
    q, k, kr, v = (torch.randn((R, n), generator=g) for n in (H * 192, H * 128, 64, H * 128))
    v[1, 4] = math.nan
    gate = torch.tensor([[0.0, -200.0], [-200.0, 0.0], [-200.0, -200.0]])
    row0, p0, out = torch.tensor([0, R], dtype=torch.int32), torch.zeros(1, dtype=torch.int32), torch.empty((R, H * 128))
    p = [planes(emu, x) for x in (q, k, kr, v)]
    emu.emu_attn32(*[P(x) for x in p], R, H, 1, 1, 0, 0, 0, 0, P(row0), P(p0), 1, R, C.c_float(192 ** -0.5), C.c_float(0.0), 0, P(None),
                   P(gate), P(None), P(None), 0, 0, P(None), P(out), 1)
    nan = torch.zeros((R, H * 128), dtype=torch.bool)
    nan[1:, 4] = True
    assert torch.equal(out.isnan(), nan) and bool((out[2, 5:] == 0).all())


@pytest.mark.parametrize("gated", [None, False, True])
def test_products_are_taken_again_after_the_tiles(emu, gated):
    """one CTA, more than 32 tiles: outputs that came out NaN are looked at again when all of its MMAs have been issued, so no warp waits meanwhile"""
    M, N, K = 1408, 384, 64      # 33 tiles of 128 x 128; of groups 22 of 256 columns, 33 of a gated unit
    g = torch.Generator().manual_seed(9)
    x, w = torch.randn((M, K), generator=g), torch.ones((2 * N if gated else N, K)).to(BF)
    w[5, 7] = math.inf
    x[:, 7] = x[:, 7].abs() + 0.1
    x[1300, 7] = 0.0
    p, c = planes(emu, x), torch.zeros((M, N))
    serial_stats(emu)
    if gated is None:
        emu.emu_gemm_split(P(p), LL(K), LL(M * K), P(w), LL(K), P(c), LL(N), LL(0), 1, M, N, K, P(None), 128, 1)
    else:
        groups = torch.zeros(M // 128, dtype=torch.int32)
        groups[3] = -1
        emu.emu_gemm_grouped(P(p), LL(M * K), P(w), 1, P(groups), M // 128, int(gated), P(None), P(c), LL(0), 1, w.shape[0], K, 1)
    regs, first, total = serial_stats(emu)
    assert first == total > 0 and regs >= 168
    y = x.double() @ w.double().T
    if gated:
        y = torch.nn.functional.silu(y[:, :N]) * y[:, N:]
    rows = torch.tensor([r for r in range(M) if gated is None or r // 128 != 3])
    assert torch.equal(c.isnan()[rows], y.isnan()[rows]) and torch.equal(c.isinf()[rows], y.isinf()[rows]) and bool(c.isnan().any())


def test_gather_of_cache_rows(emu):
    g = torch.Generator().manual_seed(4)
    width, page, lens, pos0, rule = 24, 4, [3, 5], [6, 0], (4, 0, 2, 2)
    cache, blocks = torch.randn((8 * page, width), generator=g), torch.randn((4 * page, width), generator=g)
    table, block_table = torch.tensor([[5, 1, 7], [2, 0, -1]], dtype=torch.int32), torch.tensor([[3, 1, -1], [0, 2, -1]], dtype=torch.int32)
    row0, p0 = torch.tensor([0, 3, 8], dtype=torch.int32), torch.tensor(pos0, dtype=torch.int32)
    rows = [(s, kind, t) for s, (n, a) in enumerate(zip(lens, pos0)) for kind, t in run_keys(a, n, *rule)]
    got = torch.zeros((3, len(rows), width), dtype=BF)
    emu.emu_gather_keys(2, rule[0], rule[2], rule[3], P(row0), P(p0), len(rows), P(cache), page, P(table), 3, P(blocks), P(block_table), width, P(got),
                        LL(len(rows) * width))
    want = torch.stack([(blocks if kind == "block" else cache)[int((block_table if kind == "block" else table)[s, t // page]) * page + t % page]
                        for s, kind, t in rows])
    assert torch.equal(got.double().sum(0), want.double())


@pytest.mark.parametrize("rows,K,dtype", [(1, 8, F32), (37, 72, F32), (130, 16, BF), (9, 264, BF)])
def test_gather_of_rows(emu, rows, K, dtype):
    """by an index, rows that stand apart, a negative index zeros"""
    g = torch.Generator().manual_seed(rows)
    src = torch.randn((11, K + 8), generator=g).to(dtype)
    index = torch.randint(-1, 11, (rows,), generator=g).int()
    got = torch.full((3 if dtype == F32 else 1, rows, K), float("nan"), dtype=BF)
    emu.emu_gather_rows(P(src), LL(K + 8), int(dtype == F32), P(index), rows, K, P(got), LL(rows * K))
    want = torch.where(index[:, None] < 0, torch.zeros((), dtype=F64), src[index.clamp_min(0).long()][:, :K].double())
    assert torch.equal(got.double().sum(0), want)


# ------------------------------------------------------------------------------------------------------------------- on a GPU, through the engine
def latent_engine(dtype, heads, rank, window, max_tokens=2048, **options):
    from leopard_b200 import _lib
    from leopard_b200.seqlm import LatentAttentionConfig, LayerConfig, RotaryConfig, SeqLMConfig, SeqLMEngine, SeqLMWeights
    D, O = 256, heads * 128
    m = LatentAttentionConfig(heads=heads, dim=128, rot_dim=64, vdim=128, kv_rank=rank, scale=192 ** -0.5, rot=RotaryConfig(dims=64, base=1e4),
                              window=window, **options)
    cfg = SeqLMConfig(architecture="latent", vocab=64, width=D, eps=1e-6, layers=(LayerConfig(mixer=m, ff=None),), norm="pre")
    shapes = {"embed": (64, D), "head": (64, D), "final.norm": (D,), "norm1": (D,), "mix.q": (heads * 192, D), "mix.dkv": (rank + 64, D),
              "mix.dkv.norm": (rank,), "mix.uk": (heads * 128, rank), "mix.uv": (O, rank), "mix.o": (D, O), "mix.sink": (heads,),
              "mix.g": (heads if options.get("head_gate") else O, D)}

    def get(name):
        shape = shapes[name]
        x = torch.randn(shape, generator=torch.Generator().manual_seed(sum(map(ord, name))))
        return x * (2 * shape[1] ** -0.5 if len(shape) == 2 else 0.1)
    w = SeqLMWeights(cfg, get, lambda layer, key: key, "cuda")
    return SeqLMEngine(cfg, w, dtype=dtype, max_tokens=max_tokens, page_size=16, max_seqs=4, lib=_lib.stream32_lib()), m


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,heads,rank,window,options,lens", [
    ("float32", 3, 136, None, {}, [(17, 130), (1, 300)]), ("float32", 2, 64, 100, {"sink": True}, [(129, 257), (40, 5)]),
    ("float32", 2, 72, 128, {"out_gate": True}, [(256, 1), (128, 33)]), ("bfloat16", 4, 128, 50, {"head_gate": True}, [(300, 64), (20, 500)])])
def test_expanded_latent_attention_in_the_engine(dtype, heads, rank, window, options, lens):
    """prompts, and portions that continue them, as the general path computes them (fp32: both within a few roundings of float64)"""
    from leopard_b200.seqlm import StepEntry, _Batch
    eng, m = latent_engine(dtype, heads, rank, window, **options)
    lw, kv = eng.w.layers[0], None
    calls = []
    inner = eng._latent_expanded
    eng._latent_expanded = lambda *a: calls.append(1) or inner(*a)
    for a, b in lens:
        batch = _Batch(eng, [StepEntry("a", [1] * a, []), StepEntry("b", [2] * b, [])])
        h = torch.randn((a + b, 256), device="cuda", generator=torch.Generator("cuda").manual_seed(a)).to(eng.act)
        n = len(calls)
        got = eng._latent(0, m, lw, h, batch).double()
        assert len(calls) == n + 1
        kv = lw.pop("w_kv")
        want = eng._latent(0, m, lw, h, batch).double()
        lw["w_kv"] = kv
        assert float((got - want).norm() / want.norm()) < (3e-6 if dtype == "float32" else 1e-2)
        for s, ln in zip(batch.seqs, batch.lens):
            eng.cache.advance(s, ln)


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [math.inf, math.nan])
def test_a_latent_that_is_not_finite_stays_with_the_rows_that_see_it(bad):
    from leopard_b200.seqlm import StepEntry, _Batch
    eng, m = latent_engine("float32", 3, 136, 100)
    lw = eng.w.layers[0]

    def rows(ln):
        return torch.randn((ln, 256), device="cuda", generator=torch.Generator("cuda").manual_seed(ln))
    first = _Batch(eng, [StepEntry("a", [1] * 300, [])])
    eng._latent(0, m, lw, rows(300), first)
    eng.cache.advance(first.seqs[0], 300)
    batch = _Batch(eng, [StepEntry("a", [1] * 150, [])])
    kv = lw.pop("w_kv")
    want = eng._latent(0, m, lw, rows(150), batch)
    lw["w_kv"] = kv
    eng.cache.pools[0][batch.seqs[0].pages[250 // 16], 250 % 16, 3] = bad      # position 250: rows 300 .. 349 see it
    got = eng._latent(0, m, lw, rows(150), batch)
    assert not bool(got[:50].isfinite().any())
    assert float((got[50:].double() - want[50:].double()).norm() / want[50:].double().norm()) < 3e-6      # the bound of the test above


@pytest.mark.parametrize("reqs,heads,rank,window,expands", [
    ([(0, 17)], 16, 512, None, True), ([(64000, 17)], 16, 512, None, True), ([(0, 4096)], 16, 512, 1024, True), ([(3000, 64)], 8, 256, 512, True),
    ([(8000, 1)] * 31 + [(0, 20)], 16, 512, None, False), ([(8000, 1)] * 31 + [(0, 20)], 8, 256, None, False),
    ([(2000, 1)] * 31 + [(0, 500)], 16, 512, None, False), ([(2000, 1)] * 31 + [(0, 2000)], 16, 512, None, True), ([(2000, 1)] * 7 + [(0, 20)], 16, 512, None, True),
    ([(4000, 4)] * 64, 16, 512, None, False), ([(4000, 48)] * 64, 16, 512, None, True), ([(0, 12)] * 128, 8, 256, None, False), ([(0, 24)] * 64, 8, 256, 512, True),
    ([(8000, 1)] * 31 + [(0, 20)], 4, 128, 256, True), ([(8000, 1)] * 31 + [(0, 20)], 16, 512, 100, False), ([(8000, 1)] * 31 + [(0, 20)], 32, 512, 2048, False),
    ([(8000, 1)] * 7 + [(0, 300)], 32, 512, 2048, True), ([(0, 24)] * 64, 16, 128, None, False)])
def test_which_steps_expand_their_latents(native_lib, reqs, heads, rank, window, expands):
    """by the work of either way, measured on both sides: running requests with a long past beside a short prompt do not, portions behind a long past do"""
    row0, pos0 = torch.tensor([0] + [n for _, n in reqs]).cumsum(0).int(), torch.tensor([p for p, _ in reqs], dtype=torch.int32)
    tiles, keys = C.c_int(), C.c_int()
    assert native_lib.lp_latent_route(row0.data_ptr(), pos0.data_ptr(), len(reqs), heads, rank, window or 0, C.byref(tiles), C.byref(keys)) == expands
    assert tiles.value == sum(-(-n // 128) for _, n in reqs) and keys.value == sum(p + n - seen(p, window or 0)[2] for p, n in reqs)


@pytest.mark.parametrize("rule", [(0,), (40, 0, 3), (48, 0, 0, 8), (0, 48), (33, 0, 7, 5), (30, 64)])
def test_key_rows_of_a_step(native_lib, rule):
    """window, own block, kept tokens, pooled blocks: what the host counts is what the kernels walk"""
    from leopard_b200._lib import WindowAttnDesc
    reqs = [(0, 1), (0, 200), (47, 1), (48, 100), (500, 3), (129, 300)]
    row0, pos0 = torch.tensor([0] + [n for _, n in reqs]).cumsum(0).int(), torch.tensor([p for p, _ in reqs], dtype=torch.int32)
    window, chunk, keep, pool = (*rule, 0, 0, 0)[:4]
    d, tiles, keys = WindowAttnDesc(window=window, chunk=chunk, keep_first=keep, pool=pool), C.c_int(), C.c_int()
    assert native_lib.lp_window_prompt_count(C.byref(d), row0.data_ptr(), pos0.data_ptr(), len(reqs), C.byref(tiles), C.byref(keys)) == 0
    assert tiles.value == sum(-(-n // 128) for _, n in reqs) and keys.value == sum(len(run_keys(p, n, *rule)) for p, n in reqs)


@pytest.mark.gpu
@pytest.mark.parametrize("why", ["work", "limit", "full"])
def test_latents_are_attended_as_they_are_where_expanding_does_not_pay_or_fit(why, monkeypatch):
    from leopard_b200 import seqlm
    eng, m = latent_engine("float32", 2, 64, None)
    batch = seqlm._Batch(eng, [seqlm.StepEntry("a", [1] * 40, [])])
    h = torch.randn((40, 256), device="cuda")
    want = eng._latent(0, m, eng.w.layers[0], h, batch).double()
    if why == "work":
        batch.counts[(2, 64, None)] = (0, 1, 40)
    elif why == "limit":
        monkeypatch.setattr(seqlm, "SCRATCH_BYTES", 0)
    else:
        inner = eng._empty

        def full(shape, dtype):
            if dtype == torch.uint8:
                raise torch.OutOfMemoryError("no room")
            return inner(shape, dtype)
        eng._empty = full
    monkeypatch.setattr(eng, "_latent_expanded", None)
    got = eng._latent(0, m, eng.w.layers[0], h, batch).double()
    assert float((got - want).norm() / want.norm()) < 3e-6      # the bound of the test above


@pytest.mark.gpu
def test_queries_off_16_byte_boundaries_are_attended_too():
    """columns of a wider product at an odd offset: the expanded keys' kernel reads 16 bytes at a time, the other one takes them as they are"""
    from leopard_b200.seqlm import StepEntry, _Batch
    eng, m = latent_engine("float32", 2, 64, None)
    batch = _Batch(eng, [StepEntry("a", [1] * 40, [])])
    qd = torch.randn((40, 2 * 192 + 128), device="cuda")
    shifted = torch.empty((40, qd.shape[1] + 4), device="cuda")[:, 1:1 + qd.shape[1]].copy_(qd)
    want = eng._latent(0, m, eng.w.layers[0], None, batch, proj=qd).double()
    got = eng._latent(0, m, eng.w.layers[0], None, batch, proj=shifted).double()
    assert float((got - want).norm() / want.norm()) < 3e-6      # the bound of the test above


@pytest.mark.gpu
def test_expanded_heads_in_groups():
    """more keys than all heads' expanded keys and values are held for at a time: the heads run in groups, the last one smaller; every 500th row against float64.
    Scores, their exponentials and 148 tiles of keys are each a few roundings of 2^-24, and the output's product sums 2,432 of them: 1e-6"""
    from leopard_b200.seqlm import StepEntry, _Batch
    H, rank, n = 19, 64, 19000
    eng, m = latent_engine("float32", H, rank, None, max_tokens=20480)
    lw, calls, inner = eng.w.layers[0], [], eng._latent_expanded
    eng._latent_expanded = lambda *a: calls.append(1) or inner(*a)
    assert n * 1536 * H > 512 << 20
    w_kv, w_o = lw["w_kv"].double(), lw["w_o"].double()
    for ln in (n, 40):      # a prompt, then a portion over all of it
        batch = _Batch(eng, [StepEntry("a", [1] * ln, [])])
        qd = torch.randn((ln, H * 192 + rank + 64), device="cuda", generator=torch.Generator("cuda").manual_seed(ln))
        got = eng._latent(0, m, lw, None, batch, proj=qd)      # queries are turned in place
        first = batch.seqs[0].length
        cache = eng.cache.pools[0][torch.tensor(batch.seqs[0].pages, device="cuda")].flatten(0, 1)[:first + ln].double()
        rows = torch.arange(ln - 1, -1, -500, device="cuda")
        unseen = torch.arange(first + ln, device="cuda")[None] > first + rows[:, None]
        heads = []
        for h in range(H):
            keys = torch.cat([cache[:, :rank] @ w_kv[h * 128:h * 128 + 128].T, cache[:, rank:]], 1)
            weights = torch.softmax((qd[rows, h * 192:h * 192 + 192].double() @ keys.T * 192 ** -0.5).masked_fill(unseen, -math.inf), 1)
            heads.append(weights @ (cache[:, :rank] @ w_kv[(H + h) * 128:(H + h) * 128 + 128].T))
        want = torch.cat(heads, 1) @ w_o.T
        assert float((got[rows].double() - want).norm() / want.norm()) < 1e-6
        eng.cache.advance(batch.seqs[0], ln)
    assert len(calls) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(65, 128, 1024), (4100, 264, 1032), (1100, 1000, 1400), (257, 4096, 3000)])
def test_products_of_fp32_rows_in_the_engine(M, N, K, monkeypatch):
    """the split product and its epilogues are no further from float64 than lp_linear's (few weights too)"""
    from leopard_b200 import _lib, seqlm
    monkeypatch.setattr(seqlm, "SPLIT_MIN_WEIGHTS", 0)
    eng, _ = latent_engine("float32", 2, 64, None)
    g = torch.Generator("cuda").manual_seed(M)
    a, w = torch.randn((M, K + 4), device="cuda", generator=g)[:, :K], torch.randn((N, K), device="cuda", generator=g).to(BF)
    bias, x = torch.randn(N, device="cuda", generator=g), torch.randn((M, N), device="cuda", generator=g)
    want = a.double() @ w.double().T + bias.double()
    for epi, ref in ((_lib.EPI_NONE, want), (_lib.EPI_RELU2, want.clamp_min(0) ** 2)):
        err = []
        for rows in (eng.split_rows, None):
            saved, eng.split_rows = eng.split_rows, rows
            assert eng._on_split(a, w) == (rows is not None)
            y = eng.linear(a, w, F32, epi, bias=bias).double()
            z = eng.linear(a, w, F32, epi, bias=bias, into=(x.clone(), 0.5)).double()
            eng.split_rows = saved
            err.append(float((y - ref).norm() / ref.norm()))
            assert float((z - (x.double() + 0.5 * ref)).norm() / z.norm()) < 1e-6
        assert err[0] < err[1]


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,split", [(65, 2048, 1024, True), (64, 2048, 1024, False), (65, 2040, 1024, False), (65, 2052, 1024, False), (5000, 4096, 1016, False),
                                         (65, 120, 20000, False), (65, 128, 16384, True), (2048, 1024, 1024, True), (2047, 1024, 1024, False)])
def test_which_fp32_products_are_split(M, N, K, split):
    """65 rows, 128 columns, K = 1024, and 2^21 weights or 2^31 multiplications: below that lp_linear's sums are the more precise ones, or its one launch the faster"""
    eng, _ = latent_engine("float32", 2, 64, None)
    assert eng._on_split(torch.empty((M, K), device="cuda"), torch.empty((N, K), device="cuda", dtype=BF)) == split


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("T,width,ff,on_host", [(257, 80, 72, False), (256, 80, 72, None), (400, 64, 136, False), (300, 72, 64, True)])
def test_expert_products_of_prompts_are_one_launch(T, width, ff, on_host, dtype):
    """the fewest tokens whose pairs are sorted, one fewer, an expert whose rows are several tiles, and a width that is no multiple of 16 (a product an expert)"""
    from oracle import seqlm as O
    from seqlm_common import TOL, make_engine, model, moe, rel_err, retention_layer
    form = moe(experts=4, top=2, groups=2, keep=2, ff=ff, shared=16)
    cfg = model([retention_layer(mlp=form)], width=width)
    w = O.random_weights(cfg, seed=1)
    eng = make_engine(cfg, w, ("cuda", None), dtype)
    h = torch.randn(T, width, generator=torch.Generator().manual_seed(T)).to(eng.act)
    calls = []

    class Spy:
        def __getattr__(self, name):
            f = getattr(lib, name)
            return (lambda *a: calls.append(name) or f(*a)) if name in ("lp_gemm_grouped", "lp_moe_align") else f
    lib, eng.L = eng.L, Spy()
    got = eng._moe(eng.cfg.layers[0].ff, eng.w.layers[0], h.cuda())
    want = O.feed_forward(h.double(), {k: v.to(BF).double() if v.ndim == 2 else v.double() for k, v in w.items()}, "l0.mlp.", form)
    assert rel_err(got, want) < TOL[dtype]
    assert calls.count("lp_gemm_grouped") == (2 if on_host is False else 0) and calls.count("lp_moe_align") == (on_host is not None)


@pytest.mark.gpu
@pytest.mark.parametrize("T,width,experts,top,ff", [(4096, 512, 8, 2, 512), (1000, 1024, 8, 2, 1024), (300, 256, 4, 2, 128)])
def test_fp32_experts_are_no_further_from_float64_than_sorted_tiles(T, width, experts, top, ff):
    """the grouped launches and lp_linear_grouped, which took these rows before them (measured 0.84 to 0.86 of its error)"""
    from oracle import seqlm as O
    from seqlm_common import make_engine, model, moe, rel_err, retention_layer
    form = moe(experts=experts, top=top, groups=2, keep=2, ff=ff, shared=16)
    cfg = model([retention_layer(mlp=form)], width=width)
    w = O.random_weights(cfg, seed=1)
    eng = make_engine(cfg, w, ("cuda", None), "float32")
    h = torch.randn(T, width, generator=torch.Generator().manual_seed(T))
    want = O.feed_forward(h.double(), {k: v.to(BF).double() if v.ndim == 2 else v.double() for k, v in w.items()}, "l0.mlp.", form)
    err = []
    for rows in (eng.split_rows, None):
        eng.split_rows = rows
        err.append(rel_err(eng._moe(eng.cfg.layers[0].ff, eng.w.layers[0], h.cuda()), want))
    assert err[0] < err[1], err


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_experts_of_an_engine_without_tensor_core_rows(dtype):
    """`tensor_core_rows` = None keeps bf16 rows off the tcgen05 products, `split_rows` = None fp32 rows, each only its own"""
    from oracle import seqlm as O
    from seqlm_common import make_engine, model, moe, retention_layer
    cfg = model([retention_layer(mlp=moe(experts=4, top=2, groups=2, keep=2, ff=72, shared=16))], width=80)
    eng = make_engine(cfg, O.random_weights(cfg, seed=1), ("cuda", None), dtype)
    calls, lib = [], eng.L

    class Spy:
        def __getattr__(self, name):
            f = getattr(lib, name)
            return (lambda *a: calls.append(name) or f(*a)) if name in ("lp_gemm_grouped", "lp_linear_grouped") else f
    eng.L = Spy()
    h, own = torch.randn((1000, 80), device="cuda").to(eng.act), "tensor_core_rows" if dtype == "bfloat16" else "split_rows"
    for name in ("tensor_core_rows", "split_rows"):
        saved = getattr(eng, name)
        setattr(eng, name, None)
        calls.clear()
        eng._moe(eng.cfg.layers[0].ff, eng.w.layers[0], h)
        setattr(eng, name, saved)
        assert calls == 2 * (["lp_linear_grouped"] if name == own else ["lp_gemm_grouped"])
