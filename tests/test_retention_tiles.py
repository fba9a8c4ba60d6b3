"""lp_retention_prefill: heads of whole 128s take the matrix instruction for a chunk's products, others (here: a state off 16-byte boundaries) fp32 sums.  Both
against the recurrence in float64, outputs and the state left behind, over chunks of every kind of length.  Bound: sums of at most 32 + 256 products of three bf16
terms each (2^-26 a factor) and their fp32 additions, a few 2^-24 of what is added up, whose terms cancel to about a tenth: 2e-6 relative."""
import ctypes as C

import pytest
import torch

from leopard_b200 import _lib
from seqlm_common import backend, emu_lib, rel_err  # noqa: F401

F32, F64, I32 = torch.float32, torch.float64, torch.int32


def problem(H, dim, vdim, lens, rot=0, act=0, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    R, n = sum(sum(cs) for cs in lens), len(lens)
    return dict(H=H, dim=dim, vdim=vdim, lens=lens, rot=rot, act=act, R=R, raw=torch.randn(R, 2 * H * (dim + vdim), generator=g) * scale,
                decay=torch.linspace(0.9, 0.999, H), freq=100.0 ** (-torch.arange(rot // 2, dtype=F32) * 2 / max(rot, 1)),
                pos0=torch.tensor([(37 * i) % 200 for i in range(n)]), state=torch.randn(n, H * dim * vdim, generator=g))


def definition(p):
    """outputs and states in float64 (angles are fp32 products, as in the kernels)"""
    H, dim, vdim, rot = p["H"], p["dim"], p["vdim"], p["rot"]
    x = p["raw"].double()
    q, k = x[:, : H * dim].view(-1, H, dim).clone(), x[:, H * dim: 2 * H * dim].view(-1, H, dim).clone()
    v, gate = x[:, 2 * H * dim: 2 * H * dim + H * vdim].view(-1, H, vdim), x[:, 2 * H * dim + H * vdim:].view(-1, H, vdim)
    pos = torch.cat([int(p0) + torch.arange(sum(cs)) for p0, cs in zip(p["pos0"], p["lens"])])
    if p["act"]:
        q, k, v = (t * torch.sigmoid(t) for t in (q, k, v))
    elif rot:
        angle = (pos.float()[:, None] * p["freq"][None]).double()
        c, s = angle.cos()[:, None], angle.sin()[:, None]
        for t in (q, k):
            a, b = t[..., : rot // 2].clone(), t[..., rot // 2: rot].clone()
            t[..., : rot // 2], t[..., rot // 2: rot] = a * c - b * s, b * c + a * s
    k = k * dim ** -0.5
    out, states, r = torch.empty(p["R"], H, vdim, dtype=F64), [], 0
    for i, cs in enumerate(p["lens"]):
        S = p["state"][i].double().view(H, dim, vdim) * (1 if p["pos0"][i] else 0)
        for _ in range(sum(cs)):
            S = S * p["decay"].double()[:, None, None] + k[r][:, :, None] * v[r][:, None]
            out[r] = torch.einsum("hd,hdv->hv", q[r], S)
            r += 1
        states.append(S.flatten())
    if not p["act"]:
        out = out / torch.sqrt((out * out).mean(-1, keepdim=True) + 1e-5) * gate * torch.sigmoid(gate)
    return out.flatten(1), torch.stack(states)


def run(p, dev, L, shift):
    H, dim, vdim, n = p["H"], p["dim"], p["vdim"], len(p["lens"])
    hs, chunks = H * dim * vdim, [c for cs in p["lens"] for c in cs]
    to = lambda t, dt=I32: torch.as_tensor(t).to(dt).to(dev)  # noqa: E731
    at = lambda xs: [sum(xs[:i]) for i in range(len(xs) + 1)]  # noqa: E731
    raw, decay, freq = p["raw"].to(dev), p["decay"].to(dev), p["freq"].to(dev)
    flat = torch.zeros(n * hs + 4, dtype=F32)
    flat[shift: shift + n * hs] = p["state"].flatten()
    flat = flat.to(dev)
    out = torch.full((p["R"], H * vdim), 7.0, device=dev)
    tables = [to(at([sum(cs) for cs in p["lens"]])), to(p["pos0"]), to(range(n)), to(at([len(cs) for cs in p["lens"]])),
              to([i for i, cs in enumerate(p["lens"]) for _ in cs]), to(at(chunks)[:-1]), to(chunks)]
    d = _lib.RetentionDesc(qkvg=_lib.ptr(raw), ld=raw.stride(0), q_off=0, k_off=H * dim, v_off=2 * H * dim, g_off=2 * H * dim + H * vdim, heads=H, dim=dim, vdim=vdim,
                           decay=_lib.ptr(decay), inv_freq=_lib.ptr(freq) if p["rot"] else None, rot_dims=p["rot"], rot_layout=_lib.ROT_HALF, rot_mscale=1.0,
                           k_scale=dim ** -0.5, eps=1e-5, state=flat.data_ptr() + 4 * shift, slot_stride=hs, out=_lib.ptr(out), ldo=out.stride(0), out_fp32=1,
                           in_act=p["act"], finish=_lib.RET_FINISH_RAW if p["act"] else _lib.RET_FINISH_GATED_NORM)
    nbytes = int(L.lp_retention_workspace_bytes(len(chunks), H, dim, vdim))
    ws = torch.full((nbytes // 4,), 9.0, device=dev)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream) if dev != "cpu" else None
    rc = L.lp_retention_prefill(C.byref(d), n, len(chunks), *(_lib.ptr(t) for t in tables), _lib.ptr(ws), nbytes, stream)
    assert rc == 0, L.lp_last_error()
    return out.cpu(), flat.cpu()[shift: shift + n * hs].view(n, hs)


FORMS = {
    "whole and ragged chunks": dict(H=2, dim=128, vdim=128, lens=[[32, 32, 5], [1], [31]], rot=128),
    "short chunks between": dict(H=1, dim=128, vdim=128, lens=[[7, 32, 16], [17, 15]], rot=64),
    "activations, o itself": dict(H=1, dim=128, vdim=128, lens=[[32, 9]], act=1),
    "wide keys": dict(H=1, dim=256, vdim=128, lens=[[32, 18]], rot=32),
    "wide values": dict(H=1, dim=128, vdim=256, lens=[[32, 33 - 32], [24]]),
    "not whole 128s": dict(H=1, dim=128, vdim=64, lens=[[32, 18]], rot=32),
}


@pytest.mark.parametrize("form", FORMS)
def test_both_products(backend, form):
    p = problem(**FORMS[form])
    L = backend[1] if backend[1] is not None else _lib.stream32_lib()
    want, left = definition(p)
    for shift in (0, 1):      # off 16-byte boundaries: fp32 sums
        out, state = run(p, backend[0], L, shift)
        assert rel_err(out, want) < 2e-6 and rel_err(state, left) < 2e-6


@pytest.mark.parametrize("where", ["query", "key", "value", "large"])
def test_what_is_not_finite(backend, where):
    """an infinity, a NaN or a value that no bf16 holds comes out as the fp32 sums have it, and reaches no other request"""
    p = problem(1, 128, 128, [[32, 3], [20]], act=1)
    L = backend[1] if backend[1] is not None else _lib.stream32_lib()
    col = {"query": 5, "key": 128 + 9, "value": 256 + 3, "large": 256 + 3}[where]
    p["raw"][18, col] = 3.4e38 if where == "large" else float("inf")
    if where == "key":
        p["raw"][33, 256 + 77] = float("nan")
    a, b = run(p, backend[0], L, 0), run(p, backend[0], L, 1)
    for x, y in zip(a, b):
        assert torch.equal(x.isnan(), y.isnan()) and torch.equal(x.isposinf(), y.isposinf()) and torch.equal(x.isneginf(), y.isneginf())
        ok = x.isfinite()
        assert torch.allclose(x[ok], y[ok], rtol=2e-5, atol=2e-5)
    assert bool(a[0][35:].isfinite().all()) and bool(a[0][: 35].isfinite().all()) == (where == "large")
