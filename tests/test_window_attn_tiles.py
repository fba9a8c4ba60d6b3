"""Attention of prompts with heads of 128 (lp_window_attn_tiles on the matrix instructions) against float64: ragged chunks and last tiles,
every number of query heads to a key / value head, windows with kept tokens or pooled blocks, blocks, caps, sinks, distance terms, values turned
back; and that it is as near to float64 as the one-row kernel (lp_window_attn) is.  On the kernel sources under the CPU emulator and, marked
gpu, on the native library.

Bound: three-term products keep 2^-24 of each factor, sums are short chains added in fp32; with scores of size 4 an error of 1e-6 in a score is
1e-6 of a weight, so 4e-6 of the result's root mean square; the one-row kernel's FMA chains measure about 3e-7."""
import ctypes as C
import math

import pytest
import torch

from leopard_b200 import _lib
from seqlm_common import backend, emu_lib, rel_err  # noqa: F401

F32, D, PAGE = torch.float32, 128, 16

FORMS = {
    "window": dict(window=20),
    "kept": dict(window=16, keep_first=3, sink=1),
    "pooled": dict(window=24, pool=8, softcap=6.0),
    "all": dict(),
    "blocks": dict(chunk=24),
    "bias": dict(window=40, dist="log"),
    "slope": dict(dist="linear"),
    "turned": dict(window=30, vrot=64),
}


def _run(backend, form, heads, kv_heads, pos0, lens, seed=0, plant=None, rule=False):
    """errors of (tiles, one-row kernel) against float64; with plant(queries, cached row (request, position), pooled) the tiles' outputs
    and float64's.  The matrix-instruction kernel takes launches that fill the chip: here the emulator has no SMs to fill, and on a GPU the heads
    are so many times as many, unless `rule` leaves the sizes and the emulator's four SMs as they are."""
    device, lib = backend
    if device == "cuda" and not rule:
        qh = next(q for q in (4, 2, 1) if heads // kv_heads % q == 0)
        times = -(-(36 if qh == 1 else 14) * torch.cuda.get_device_properties(0).multi_processor_count // (sum(lens) * (heads // qh)))
        heads, kv_heads = heads * times, kv_heads * times
    L = lib if lib is not None else _lib.stream32_lib()
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream) if device == "cuda" else None
    g = torch.Generator().manual_seed(seed)
    f, R = FORMS[form], sum(lens)
    total = [p + n for p, n in zip(pos0, lens)]
    pages = [-(-t // PAGE) for t in total]
    q = torch.randn(R, heads * D, generator=g)
    roww = kv_heads * 2 * D
    cache = torch.randn(sum(pages), PAGE, roww, generator=g)
    table = torch.full((len(lens), max(pages)), -1, dtype=torch.int32)
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = torch.randperm(n, generator=g).to(torch.int32) + at
        at += n
    rows = [torch.stack([cache[int(table[i, p // PAGE]), p % PAGE] for p in range(t)]) for i, t in enumerate(total)]
    pool = f.get("pool", 0)
    pooled = ptab = None
    if pool:
        n_blocks = max(max(t // pool for t in total), 1)
        pooled = torch.zeros(len(lens), -(-n_blocks // PAGE), PAGE, roww)
        for i, t in enumerate(total):
            for b in range(t // pool):
                pooled[i, b // PAGE, b % PAGE] = rows[i][b * pool:(b + 1) * pool].mean(0)
        ptab = torch.arange(pooled.shape[0] * pooled.shape[1], dtype=torch.int32).view(len(lens), -1)
    if plant is not None:
        plant(q, lambda i, p: cache[int(table[i, p // PAGE]), p % PAGE], pooled)
        rows = [torch.stack([cache[int(table[i, p // PAGE]), p % PAGE] for p in range(t)]) for i, t in enumerate(total)]
    amp = torch.rand(heads, generator=g) * 0.3 if "dist" in f else None
    rate = torch.rand(heads, generator=g) if f.get("dist") == "log" else None
    vfreq = 100.0 ** (-torch.arange(f["vrot"] // 2) * 2.0 / f["vrot"]) if "vrot" in f else None
    row_pos = torch.cat([torch.arange(p, p + n) for p, n in zip(pos0, lens)]).to(torch.int32)
    row_seq = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).to(torch.int32)
    chunks, r0 = [], 0
    for i, n in enumerate(lens):
        chunks += [(i, r0 + a, min(32, n - a)) for a in range(0, n, 32)]
        r0 += n
    cs, cr, cl = (torch.tensor(x, dtype=torch.int32) for x in zip(*chunks))
    t = {k: (v.to(device) if v is not None else None) for k, v in dict(q=q, cache=cache, table=table, pooled=pooled, ptab=ptab, amp=amp, rate=rate,
                                                                        vfreq=vfreq, row_pos=row_pos, row_seq=row_seq, cs=cs, cr=cr, cl=cl).items()}
    one = torch.ones(1, device=device)
    d = _lib.WindowAttnDesc(
        qkv=_lib.ptr(t["q"]), ld=heads * D, q_off=0, k_off=0, v_off=0, heads=heads, kv_heads=kv_heads, dim=D, vdim=D, norm_mode=_lib.QKNORM_NONE,
        g_off=-1, eps=1e-6, inv_freq=_lib.ptr(one), rot_dims=0, rot_layout=_lib.ROT_HALF, rot_mscale=1.0, v_inv_freq=_lib.ptr(t["vfreq"]),
        v_rot_dims=f.get("vrot", 0), v_rot_layout=_lib.ROT_HALF, cache=_lib.ptr(t["cache"]), page_size=PAGE, page_table=_lib.ptr(t["table"]),
        max_pages=table.shape[1], pooled=_lib.ptr(t["pooled"]), pooled_table=_lib.ptr(t["ptab"]), max_pooled_pages=ptab.shape[1] if pool else 0, pool=pool,
        window=f.get("window", 0), keep_first=f.get("keep_first", 0), scale=D ** -0.5, softcap=f.get("softcap", 0.0), sink=f.get("sink", 0),
        chunk=f.get("chunk", 0), kv_shared=1, dist_amp=_lib.ptr(t["amp"]), dist_rate=_lib.ptr(t["rate"]), out_scale=1.0)
    got, row_wise = torch.full((R, heads * D), 9.0, device=device), torch.empty(R, heads * D, device=device)
    if lib is not None and not rule:
        lib.emu_set_sm_count(0)
    rc = L.lp_window_attn_tiles(C.byref(d), R, _lib.ptr(t["row_seq"]), _lib.ptr(t["row_pos"]), len(chunks), _lib.ptr(t["cs"]), _lib.ptr(t["cr"]),
                                _lib.ptr(t["cl"]), _lib.ptr(got), heads * D, 1, st)
    if lib is not None:
        lib.emu_set_sm_count(4)
    assert rc == 0, L.lp_last_error()
    assert L.lp_window_attn(C.byref(d), R, _lib.ptr(t["row_seq"]), _lib.ptr(t["row_pos"]), _lib.ptr(row_wise), heads * D, 1, st) == 0
    want = torch.zeros(R, heads, D, dtype=torch.float64)
    for r in range(R):
        i, p = int(row_seq[r]), int(row_pos[r])
        w, ch = f.get("window", 0), f.get("chunk", 0)
        lo = max(p - w + 1, 0) if w else 0
        lo = max(lo, p // ch * ch) if ch else lo
        seen = [j for j in range(p + 1) if j >= lo or j < f.get("keep_first", 0)]
        blocks = [b for b in range(total[i]) if pool and w and b * pool + pool - 1 <= p - w]
        kv = torch.cat([pooled[i].reshape(-1, roww)[blocks] if blocks else torch.zeros(0, roww), rows[i][seen]]).double()
        dist = torch.tensor([0.0] * len(blocks) + [float(p - j) for j in seen], dtype=torch.float64)
        k, v = kv[:, :kv_heads * D].view(-1, kv_heads, D), kv[:, kv_heads * D:].view(-1, kv_heads, D)
        for h in range(heads):
            s = k[:, h // (heads // kv_heads)] @ q[r, h * D:(h + 1) * D].double() * D ** -0.5
            if f.get("softcap"):
                s = f["softcap"] * torch.tanh(s / f["softcap"])
            if amp is not None:
                s = s - float(amp[h]) * (torch.log1p(float(rate[h]) * dist) if rate is not None else dist)
            top = max([0.0] + s[s.isfinite()].tolist())
            e = torch.exp(s - top)
            want[r, h] = (e / (e.sum() + f.get("sink", 0) * math.exp(-top))) @ v[:, h // (heads // kv_heads)]
        if vfreq is not None:
            n = f["vrot"] // 2
            ang = (float(p) * vfreq.float()).double()
            x, y = want[r, :, :n].clone(), want[r, :, n:2 * n].clone()
            want[r, :, :n], want[r, :, n:2 * n] = x * ang.cos() + y * ang.sin(), y * ang.cos() - x * ang.sin()
    if plant is not None:
        return got.cpu(), want.view(R, -1)
    return rel_err(got, want.view(R, -1)), rel_err(row_wise, want.view(R, -1))


@pytest.mark.parametrize("form", sorted(FORMS))
def test_forms(backend, form):
    """two requests, one from its beginning, one after 37 earlier tokens; last chunks of 1 and 9 rows"""
    tiles, row_wise = _run(backend, form, 4, 1, [0, 37], [33, 41] if backend[0] == "cuda" else [33, 9])
    assert tiles < 4e-6 and tiles < 2 * row_wise + 2e-7, (tiles, row_wise)


@pytest.mark.parametrize("heads,kv_heads", [(1, 1), (2, 2), (2, 1), (6, 1), (8, 1), (3, 1)])
def test_head_groups(backend, heads, kv_heads):
    tiles, row_wise = _run(backend, "kept", heads, kv_heads, [5], [40])
    assert tiles < 4e-6 and tiles < 2 * row_wise + 2e-7, (tiles, row_wise)


INF, NAN, TOP = float("inf"), float("nan"), torch.finfo(F32).max
def _value(row):
    return row[len(row) // 2 + 5:len(row) // 2 + 6]


# what is planted: (form, where, number); values and keys of head 0's key / value head, channel 5
ODD = {
    "later value": ("all", lambda q, row, pooled, x: _value(row(0, 20)).fill_(x)),
    "value that leaves the window": ("window", lambda q, row, pooled, x: _value(row(0, 4)).fill_(x)),
    "later key": ("all", lambda q, row, pooled, x: row(0, 20)[5:6].fill_(x)),
    "later key under a cap": ("pooled", lambda q, row, pooled, x: row(0, 25)[5:6].fill_(x)),
    "kept value": ("kept", lambda q, row, pooled, x: _value(row(0, 1)).fill_(x)),
    "kept key": ("kept", lambda q, row, pooled, x: row(0, 1)[5:6].fill_(x)),
    "pooled value": ("pooled", lambda q, row, pooled, x: _value(pooled[0, 0, 0]).fill_(x)),
    "pooled key": ("pooled", lambda q, row, pooled, x: pooled[0, 0, 0, 5:6].fill_(x)),
    "key with a distance term": ("bias", lambda q, row, pooled, x: row(0, 20)[5:6].fill_(x)),
    "query": ("window", lambda q, row, pooled, x: q[7, 5:6].fill_(x)),
    "query under a cap": ("pooled", lambda q, row, pooled, x: q[7, 5:6].fill_(x)),
}


@pytest.mark.parametrize("what", sorted(ODD))
@pytest.mark.parametrize("x", [NAN, INF, -INF, TOP], ids=["nan", "inf", "-inf", "largest"])
def test_unusual_numbers_stay_with_the_rows_that_see_them(backend, what, x):
    """41 rows in chunks of 32 and 9: what a row does not see does not reach it, a key of score -inf has no weight, an infinite value keeps
    its sign; the largest fp32 number (of a value: a score of it leaves fp32) rounds to infinity in a bf16 term and is none.  Bound as above."""
    form, plant = ODD[what]
    if x == TOP and "value" not in what:
        pytest.skip("leaves fp32")
    tiles, want = _run(backend, form, 4, 1, [0], [41], plant=lambda q, row, pooled: plant(q, row, pooled, x))
    fine = want.isfinite()
    assert fine.any() and torch.equal(tiles.isfinite(), fine) and torch.equal(tiles.isnan(), want.isnan())
    assert torch.equal(tiles[tiles.isinf()].double(), want[want.isinf()])
    usual = fine & (want.abs() < 1e30)
    assert rel_err(tiles[usual], want[usual]) < 4e-6 and rel_err(tiles[fine] * 2.0 ** -64, want[fine] * 2.0 ** -64) < 4e-6


@pytest.mark.parametrize("heads,kv_heads,lens", [
    (4, 1, [32, 24]), (4, 1, [32, 23]), (16, 4, [12, 12, 12]), (16, 4, [12, 12, 11]), (2, 2, [72]), (2, 2, [64]), (2, 2, [20, 20]), (2, 2, [20, 19])])
def test_both_sides_of_the_rule(backend, heads, kv_heads, lens):
    """on the emulator's four SMs the first of each pair has the rows and the filled chunks for the matrix-instruction kernel, the second just
    not"""
    tiles, row_wise = _run(backend, "window", heads, kv_heads, [7] * len(lens), lens, rule=True)
    assert tiles < 4e-6 and tiles < 2 * row_wise + 2e-7, (tiles, row_wise)


@pytest.mark.parametrize("heads,kv_heads,rows", [(4, 1, 1), (8, 1, 1), (16, 2, 1), (2, 1, 3), (2, 1, 4), (6, 1, 1)])
def test_one_row_steps_with_and_without_shared_rows(backend, heads, kv_heads, rows):
    """the one-row kernel with a query head a CTA and with two or four: on the emulator's four SMs the first, fourth and last launches have a head
    a CTA, the others share"""
    _, row_wise = _run(backend, "kept", heads, kv_heads, [9] * rows, [1] * rows, rule=True)
    assert row_wise < 4e-6


@pytest.mark.parametrize("heads,kv_heads,pos", [(4, 1, 255), (4, 1, 256), (2, 2, 700), (4, 1, 1100)])
def test_one_row_over_many_keys(backend, heads, kv_heads, pos):
    """a head a CTA: pages for 256 keys, which eight warps take at once, and for more, which up to 32 warps walk"""
    _, row_wise = _run(backend, "all", heads, kv_heads, [pos], [1], rule=True)
    assert row_wise < 4e-6
