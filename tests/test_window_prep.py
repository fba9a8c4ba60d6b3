"""lp_window_attn_prep: rows of 128-wide heads take a kernel that holds them in registers, others (here: rows off 16-byte boundaries) the general one.  Both against
the definition in float64 over the forms that the first one takes; angles are fp32 products of position and frequency in both.  Bounds: a few fp32 roundings, 1e-6,
and up to position 3000 the rounding of the angle, 2^-24 * 3000 = 2e-4, which both share with the reference."""
import ctypes as C
import math

import pytest
import torch

from leopard_b200 import _lib
from seqlm_common import backend, emu_lib, rel_err  # noqa: F401

F32, F64, I32 = torch.float32, torch.float64, torch.int32
D = 128
FORMS = {
    "head norm, half turned": dict(H=6, G=2, norm=1, rot=64, value_rot=128),
    "row norm": dict(H=5, G=5, norm=2, rot=8),
    "no norm, pairs": dict(H=3, G=1, norm=0, rot=24, layout=1, value_rot=20, value_layout=1),
    "all turned, value norm, temperatures": dict(H=4, G=4, norm=1, rot=128, v_norm=1, temps=True),
    "values are keys": dict(H=2, G=2, norm=1, rot=32, v_is_k=1),
    "another layer's keys": dict(H=9, G=3, norm=1, rot=16, shared=True),
    "many heads": dict(H=40, G=20, norm=2, rot=64),
}


def turned(x, pos, freq, layout):
    n = freq.numel()
    angle = (pos.float()[:, None] * freq[None]).double()
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    y = x.clone()
    a, b = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if layout else (slice(0, n), slice(n, 2 * n))
    y[..., a], y[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return y


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("R", [1, 7])
def test_both_kernels(backend, form, R):
    f = FORMS[form]
    H, G, dev, lib = f["H"], f["G"], backend[0], backend[1]
    L = lib if lib is not None else _lib.stream32_lib()
    g = torch.Generator().manual_seed(R + H)
    kvh = 0 if f.get("shared") else G
    v_at = (H + G) * D
    width = v_at + G * D
    pos = torch.randint(0, 3000, (R,), generator=g)
    raw = torch.randn(R, width, generator=g) * 2
    gain_shape = {0: None, 1: (D, D), 2: (H * D, G * D)}[f["norm"]]
    gains = [torch.rand(n, generator=g) + 0.5 for n in gain_shape] if gain_shape else [None, None]
    freq = 100.0 ** (-torch.arange(f["rot"] // 2, dtype=F32) * 2 / f["rot"])
    vfreq = 50.0 ** (-torch.arange(f["value_rot"] // 2, dtype=F32) * 2 / f["value_rot"]) if f.get("value_rot") else None
    temp = torch.rand(H, generator=g) + 0.5 if f.get("temps") else None
    page, pages = 16, 200
    roww = G * D * (1 if f.get("v_is_k") else 2)
    # the definition
    x = raw.double()
    q, k, v = x[:, : H * D].view(R, H, D), x[:, H * D: v_at].view(R, G, D), x[:, v_at:].view(R, G, D)
    if f["norm"] == 1:
        q, k = (t / torch.sqrt((t * t).mean(-1, keepdim=True) + 1e-5) * w.double() for t, w in zip((q, k), gains))
    elif f["norm"] == 2:
        q, k = (t / torch.sqrt((t * t).mean((1, 2), keepdim=True) + 1e-5) * w.double().view(-1, D) for t, w in zip((q, k), gains))
    if temp is not None:
        q = q * temp.double()[:, None] * (0.1 * torch.log(((pos + 1) // 7).double() + 1) + 1)[:, None, None]
    q, k = turned(q, pos, freq, f.get("layout", 0)), turned(k, pos, freq, f.get("layout", 0))
    if f.get("v_norm"):
        v = v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)
    if vfreq is not None:
        v = turned(v, pos, vfreq, f.get("value_layout", 0))
    to = lambda t: None if t is None else t.to(dev)  # noqa: E731
    dev_of = [to(t) for t in (*gains, freq, vfreq, temp)]
    table, seqs, posd = torch.arange(R * pages, dtype=I32).flip(0).to(dev), torch.arange(R, dtype=I32).to(dev), pos.to(I32).to(dev)
    for shift in (0, 1):      # off 16-byte boundaries: the general kernel
        flat = torch.zeros(R * width + 4, dtype=F32)
        flat[shift: shift + R * width] = raw.flatten()
        flat = flat.to(dev)
        cache = torch.full((R * pages * page, roww), 7.0, device=dev)
        d = _lib.WindowAttnDesc(qkv=flat.data_ptr() + 4 * shift, ld=width, q_off=0, k_off=H * D, v_off=v_at, heads=H, kv_heads=G, dim=D, vdim=D, norm_mode=f["norm"],
                                q_gain=_lib.ptr(dev_of[0]), k_gain=_lib.ptr(dev_of[1]), eps=1e-5, inv_freq=_lib.ptr(dev_of[2]), rot_dims=f["rot"],
                                rot_layout=f.get("layout", 0), rot_mscale=1.0, v_inv_freq=_lib.ptr(dev_of[3]), v_rot_dims=f.get("value_rot", 0),
                                v_rot_layout=f.get("value_layout", 0), cache=_lib.ptr(cache), page_size=page, page_table=_lib.ptr(table), max_pages=pages, scale=1.0,
                                v_norm=f.get("v_norm", 0), kv_shared=int(bool(f.get("shared"))), v_is_k=f.get("v_is_k", 0), q_temp=_lib.ptr(dev_of[4]), out_scale=1.0,
                                pos_temp_coef=0.1, pos_temp_every=7 if temp is not None else 0)
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream) if dev != "cpu" else None
        assert L.lp_window_attn_prep(C.byref(d), R, _lib.ptr(seqs), _lib.ptr(posd), stream) == 0, L.lp_last_error()
        got = flat.cpu()[shift: shift + R * width].view(R, width)
        assert rel_err(got[:, : H * D], q.flatten(1)) < 2e-6
        assert torch.equal(got[:, H * D:], raw[:, H * D:])
        rows = cache.cpu()[[int(table[i * pages + int(pos[i]) // page]) * page + int(pos[i]) % page for i in range(R)]]
        if kvh:
            assert rel_err(rows[:, : G * D], k.flatten(1)) < 2e-6
            if not f.get("v_is_k"):
                assert rel_err(rows[:, G * D:], v.flatten(1)) < 2e-6
        assert float((cache == 7.0).float().mean()) >= 1 - (R * roww if kvh else 0) / cache.numel() - 1e-6 and math.isfinite(float(cache.sum()))


@pytest.mark.parametrize("layout,rot,value_rot", [(0, 64, 32), (0, 0, 8), (1, 24, 20)])
def test_dimensions_that_are_not_turned_stay_apart(backend, layout, rot, value_rot):
    """an infinity or a NaN in one of them is nobody's partner: all others are what they are in the general kernel (the same fp32 products; 1e-6 of the result)"""
    H, G, R, dev, lib = 4, 2, 2, backend[0], backend[1]
    L = lib if lib is not None else _lib.stream32_lib()
    width = (H + 2 * G) * D
    raw = torch.randn(R, width, generator=torch.Generator().manual_seed(rot))
    for at, odd in ((100, float("inf")), (D + 127, float("nan")), (H * D + 90, float("-inf")), ((H + G) * D + 120, float("nan")), ((H + G + 1) * D + 33, float("inf"))):
        raw[1, at] = odd
    freq, vfreq = (torch.rand(max(n // 2, 1)).to(dev) for n in (rot, value_rot))
    table, seqs, posd = torch.arange(R, dtype=I32).to(dev), torch.arange(R, dtype=I32).to(dev), torch.full((R,), 5, dtype=I32).to(dev)
    seen = []
    for shift in (0, 1):
        flat = torch.zeros(R * width + 4, dtype=F32)
        flat[shift: shift + R * width] = raw.flatten()
        flat, cache = flat.to(dev), torch.zeros(R * 8, 2 * G * D, device=dev)
        d = _lib.WindowAttnDesc(qkv=flat.data_ptr() + 4 * shift, ld=width, q_off=0, k_off=H * D, v_off=(H + G) * D, heads=H, kv_heads=G, dim=D, vdim=D,
                                eps=1e-5, inv_freq=_lib.ptr(freq), rot_dims=rot, rot_layout=layout, rot_mscale=1.0, v_inv_freq=_lib.ptr(vfreq),
                                v_rot_dims=value_rot, v_rot_layout=layout, cache=_lib.ptr(cache), page_size=8, page_table=_lib.ptr(table), max_pages=1, scale=1.0,
                                out_scale=1.0)
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream) if dev != "cpu" else None
        assert L.lp_window_attn_prep(C.byref(d), R, _lib.ptr(seqs), _lib.ptr(posd), stream) == 0, L.lp_last_error()
        seen.append(torch.cat([flat.cpu()[shift: shift + R * width], cache.cpu().flatten()]))
    new, old = seen
    fine = torch.isfinite(old)
    assert int((~fine).sum()) == 8      # the five, of which three are in the cache too
    assert torch.equal(new[~fine].nan_to_num(7.0), old[~fine].nan_to_num(7.0)) and torch.isfinite(new[fine]).all()
    assert rel_err(new[fine], old[fine].double()) < 1e-6
