"""Retention and latent attention where rows are whole 16-byte pieces (the kernels read four columns at a time) and where they are not, with few
(request, head) pairs for the chip and with many: prompts of several chunks, portions, then token by token, against the plain implementation in oracle/seqlm.py."""
import ctypes as C

import pytest

from leopard_b200 import _lib
from leopard_b200.seqlm import StepEntry
from oracle import seqlm as O
from seqlm_common import TOL, backend, emu_lib, latent_layer, make_engine, model, rel_err, retention_layer  # noqa: F401

import torch


def _prompts(n, vocab, lens):
    g = torch.Generator().manual_seed(n)
    return [torch.randint(0, vocab, (ln,), generator=g).tolist() for ln in lens]


@pytest.mark.parametrize("layer", [retention_layer(heads=2, dim=8, vdim=8, rot_dims=8), retention_layer(heads=2, dim=16, vdim=24, rot_dims=4),
                                   retention_layer(heads=1, dim=24, vdim=12, rot_dims=24, decay=(0.98,)), retention_layer(heads=1, dim=40, vdim=72, rot_dims=8, decay=(0.9,)),
                                   latent_layer(heads=2, dim=4, rot_dim=8, vdim=4, kv_rank=136, window=20), latent_layer(heads=1, dim=4, rot_dim=4, vdim=4, kv_rank=260, window=None),
                                   latent_layer(heads=2, dim=4, rot_dim=6, vdim=4, kv_rank=132, window=7), latent_layer(heads=2, dim=4, rot_dim=4, vdim=4, kv_rank=20, window=9)],
                         ids=["8x8", "16x24", "24x12", "40x72", "rank136", "rank260", "rank132-rot6", "rank20"])
@pytest.mark.parametrize("n", [1, 5])
def test_prompts_portions_and_steps(backend, layer, n):
    cfg = model([layer])
    w = O.random_weights(cfg, seed=1)
    eng = make_engine(cfg, w, backend, max_tokens=512, max_seqs=n)
    toks = _prompts(n, cfg["vocab"], [71 - 5 * i for i in range(n)])
    want = [O.forward(cfg, w, t) for t in toks]
    done = [0] * n
    for part in (33, len(toks[-1]) - 33 - 2):      # a whole chunk and one row more, then the rest
        got = eng.step([StepEntry(i, t[d:d + part], list(range(part))) for i, (t, d) in enumerate(zip(toks, done))])
        for i in range(n):
            assert rel_err(got[i * part:(i + 1) * part], want[i][done[i]:done[i] + part]) < TOL["float32"]
            done[i] += part
    for _ in range(2):
        got = eng.step([StepEntry(i, [t[d]], [0]) for i, (t, d) in enumerate(zip(toks, done))])
        for i in range(n):
            assert rel_err(got[i:i + 1], want[i][done[i]:done[i] + 1]) < TOL["float32"]
            done[i] += 1


@pytest.mark.gpu
@pytest.mark.parametrize("layer", [latent_layer(heads=8, dim=4, rot_dim=8, vdim=4, kv_rank=136, window=20), latent_layer(heads=8, dim=4, rot_dim=6, vdim=4, kv_rank=132, window=7),
                                   latent_layer(heads=8, dim=4, rot_dim=4, vdim=4, kv_rank=512, window=None), latent_layer(heads=8, dim=4, rot_dim=4, vdim=4, kv_rank=20, window=9)],
                         ids=["rank136", "rank132-rot6", "rank512", "rank20"])
@pytest.mark.parametrize("n", [37, 38])
def test_latent_steps_of_more_pairs_than_two_a_processor(layer, n):
    """8 heads of 37 requests are 296 (row, head) pairs, two an SM, of 38 more: 16 warps a pair, then four"""
    cfg = model([layer])
    w = O.random_weights(cfg, seed=1)
    eng = make_engine(cfg, w, ("cuda", None), max_tokens=1024, max_seqs=n)
    toks = _prompts(n, cfg["vocab"], [23 - i % 17 for i in range(n)])
    eng.step([StepEntry(i, t[:-2], [0]) for i, t in enumerate(toks)])
    for k in (2, 1):
        got = eng.step([StepEntry(i, [t[-k]], [0]) for i, t in enumerate(toks)])
        assert rel_err(got, torch.stack([O.forward(cfg, w, t)[-k] for t in toks])) < TOL["float32"]


@pytest.mark.parametrize("rot_dims,rot_dim,interleaved", [(8192, 8192, 0), (8194, 8200, 1), (12280, 12280, 0), (12290, 12300, 1)])
def test_rotation_of_many_dimensions(backend, rot_dims, rot_dim, interleaved):
    """as many pairs as shared memory holds sines and cosines for, one more, and sizes at which such a table would not fit a launch.  Sums of two products of
    fp32 numbers; an angle of up to 3 is rounded to 2^-24 of itself: 3e-7 of the result"""
    device, lib = backend
    L = lib if lib is not None else _lib.stream32_lib()
    g = torch.Generator().manual_seed(rot_dims)
    q, x = torch.randn((2, 3 * rot_dim), generator=g), torch.randn((2, 4 + rot_dim), generator=g)
    freq = torch.rand(rot_dims // 2, generator=g)
    ints = [torch.tensor(v, dtype=torch.int32, device=device) for v in ([0], [0, 0], [2, 3])]
    t = [v.clone().to(device) for v in (q, x, freq, torch.ones(4))]      # queries are turned in place
    cache = torch.zeros((4, 4 + rot_dim), device=device)
    d = _lib.LatentDesc(q=_lib.ptr(t[0]), ldq=3 * rot_dim, dkv=_lib.ptr(t[1]), lddkv=4 + rot_dim, heads=3, dim=0, rot_dim=rot_dim, kv_rank=4, c_gain=_lib.ptr(t[3]),
                        eps=1e-6, inv_freq=_lib.ptr(t[2]), rot_dims=rot_dims, rot_layout=_lib.ROT_INTERLEAVED if interleaved else _lib.ROT_HALF, rot_mscale=1.0,
                        cache=_lib.ptr(cache), page_size=4, page_table=_lib.ptr(ints[0]), max_pages=1, scale=1.0)
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream) if device == "cuda" else None
    assert L.lp_latent_prep(C.byref(d), 2, _lib.ptr(ints[1]), _lib.ptr(ints[2]), st) == 0, L.lp_last_error()

    def turned(v):      # [2, n, rot_dim]
        n = rot_dims // 2
        a, c = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if interleaved else (slice(0, n), slice(n, 2 * n))
        angle = (torch.tensor([2.0, 3.0])[:, None] * freq)[:, None].double()
        out = v.double().clone()
        out[..., a], out[..., c] = v[..., a] * angle.cos() - v[..., c] * angle.sin(), v[..., c] * angle.cos() + v[..., a] * angle.sin()
        return out
    assert rel_err(t[0].cpu().view(2, 3, rot_dim), turned(q.view(2, 3, rot_dim))) < 3e-7
    assert rel_err(cache[2:, 4:].cpu()[:, None], turned(x[:, None, 4:])) < 3e-7
