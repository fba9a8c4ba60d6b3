"""Which kernels a step of the layer-list language models takes as its number of rows changes, and what captured steps keep: against the
plain implementation (oracle/seqlm.py) or float64.  On the kernel sources under the CPU emulator and, marked gpu, on the native library."""
import math

import pytest
import torch

from leopard_b200 import _lib
from leopard_b200.seqlm import MOE_PAIRS_ALONE, MOE_PAIRS_MAX, STREAM_MAX_OUTPUTS, StepEntry
from oracle import seqlm as O
from seqlm_common import TOL, backend, dense, emu_lib, latent_layer, make_engine, model, moe, rel_err, retention_layer  # noqa: F401  (fixtures)


def _tokens(n, vocab, seed=0):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(0, vocab, (n,), generator=g).tolist()


def test_expert_tables_stay_where_captured_steps_found_them(backend):
    """a decode layout that was captured with few (token, choice) pairs, then portions of a prompt with more pairs than any step before
    them, then the captured layout again: the table of the pairs' rows has not moved, and the logits are the oracle's"""
    cfg = model([retention_layer(mlp=moe(top=2))])
    w = O.random_weights(cfg, seed=21)
    toks, other = _tokens(9, cfg["vocab"], seed=1), _tokens(130 + 250, cfg["vocab"], seed=2)
    want = O.forward(cfg, w, toks)
    eng = make_engine(cfg, w, backend, max_tokens=512)
    got = [eng.step([StepEntry("r", toks[:4], [3])])]
    for t in range(4, 7):      # eager, captured, replayed
        got.append(eng.step([StepEntry("r", [toks[t]], [0])]))
    at = eng._pair_rows.data_ptr()
    eng.step([StepEntry("p", other[:130])])
    eng.step([StepEntry("p", other[130:])])      # 500 pairs, just below the limit of this route
    assert eng._pair_rows.data_ptr() == at and eng._pair_rows.tolist() == list(range(eng._pair_rows.numel()))
    for t in range(7, 9):
        got.append(eng.step([StepEntry("r", [toks[t]], [0])]))
    assert rel_err(torch.cat(got, 0), want[3:]) < TOL["float32"]


class _Spy:
    """a library that notes the names of the entry points that are called"""
    def __init__(self, lib):
        self.lib, self.called = lib, []

    def __getattr__(self, name):
        f = getattr(self.lib, name)
        return lambda *a: (self.called.append(name), f(*a))[1]


@pytest.mark.gpu
@pytest.mark.parametrize("M", [8, 9, 33, 63, 64, 65])
@pytest.mark.parametrize("wide", [False, True])
def test_products_on_both_sides_of_the_crossover(M, wide):
    """bf16 rows just below and just above the outputs from which the GEMM is faster, below 64 rows (never there), at 64 (beyond that line) and above
    (always): which kernel runs, and the result against float64: plain, gated, with a bias, added to a stream through a gate, and in bf16"""
    eng = make_engine(model([retention_layer()]), O.random_weights(model([retention_layer()]), seed=2), ("cuda", None), "bfloat16")
    g = torch.Generator().manual_seed(M)
    K, N = 192, STREAM_MAX_OUTPUTS // M // 16 * 16 + (16 if wide else 0)      # both halves of a gated unit are whole 8s
    a = torch.randn(M, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g) / math.sqrt(K)).to(torch.bfloat16)
    bias, x, gate = torch.randn(N, generator=g), torch.randn(M, N, generator=g), torch.randn(M, N, generator=g)
    want = a.double() @ w.double().T
    ad, wd = a.cuda(), w.cuda()
    eng.L = _Spy(eng.L)
    for dtype, tol in ((torch.float32, 2e-6), (torch.bfloat16, 3e-3)):
        assert rel_err(eng.linear(ad, wd, dtype, bias=bias.cuda()), want + bias.double()) < tol
    p, q = want[:, : N // 2], want[:, N // 2:]
    assert rel_err(eng.linear(ad, wd, torch.float32, _lib.EPI_SILU_GATE), p * torch.sigmoid(p) * q) < 5e-6
    xd = x.cuda()
    eng.linear(ad, wd, torch.float32, into=(xd, 0.5, gate.cuda()))
    assert rel_err(xd, x.double() + 0.5 * want * torch.sigmoid(gate.double())) < 2e-6
    assert ("lp_gemm_bf16" in eng.L.called) == (M > 64 or (M == 64 and wide))
    assert ("lp_linear" in eng.L.called) != ("lp_gemm_bf16" in eng.L.called)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,bound", [(9, 20000, 1024, 2.5e-7), (33, 6000, 2048, 3.9e-7), (63, 4096, 4096, 6.1e-7)])
def test_few_rows_lose_no_more_than_chains_of_multiply_adds(M, N, K, bound):
    """below 64 rows, with many columns: no further from float64 than the fp32 multiply-adds over K that such products ran on (the bounds are
    what those measure on such data; the GEMM's one chain over K is 4 to 7 times as far)"""
    eng = make_engine(model([retention_layer()]), O.random_weights(model([retention_layer()]), seed=2), ("cuda", None), "bfloat16")
    g = torch.Generator().manual_seed(M)
    a, w = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda(), (torch.randn(N, K, generator=g) / math.sqrt(K)).to(torch.bfloat16).cuda()
    assert rel_err(eng.linear(a, w, torch.float32), a.double() @ w.double().T) < bound


@pytest.mark.gpu
@pytest.mark.parametrize("requests", [9, 33, 63, 64])
@pytest.mark.parametrize("wide", [False, True])
def test_captured_steps_on_both_sides_of_the_crossover(requests, wide):
    """steps of so many requests, eager, captured and replayed, with the vocabulary's product on either kernel, against the oracle"""
    vocab = STREAM_MAX_OUTPUTS // requests // 8 * 8 + (8 if wide else 0)
    cfg = model([retention_layer(mlp=dense(ff=64))], width=64, vocab=vocab)
    w = O.random_weights(cfg, seed=4)
    eng = make_engine(cfg, w, ("cuda", None), "bfloat16", max_tokens=512, max_seqs=requests)
    toks = {k: _tokens(5, vocab, seed=k) for k in range(requests)}
    want = {k: O.forward(cfg, w, toks[k]) for k in toks}
    got = []
    eng.step([StepEntry(k, toks[k][:1]) for k in toks])
    for t in range(1, 5):
        spy = eng.L = _Spy(eng.L if t == 1 else eng.L.lib)
        got.append(eng.step([StepEntry(k, [toks[k][t]], [0]) for k in toks]))
        assert ("lp_gemm_bf16" in spy.called) == (wide and requests == 64 and bool(spy.called))      # a replay calls nothing
    assert not spy.called
    got = torch.stack(got, 1)
    assert rel_err(got, torch.stack([want[k][1:] for k in toks])) < TOL["bfloat16"]


@pytest.mark.parametrize("ff,width,limit", [(moe(), 32, MOE_PAIRS_MAX), (moe(experts=4, top=1, groups=1, keep=1, ff=8, shared=0), 32, MOE_PAIRS_MAX),
                                            (moe(ff=6), 32, MOE_PAIRS_ALONE), (moe(), 36, MOE_PAIRS_ALONE)], ids=["moe", "moe-top1", "ff6", "width36"])
@pytest.mark.parametrize("over", [0, 1])
def test_experts_on_both_sides_of_the_pair_limit(backend, ff, width, limit, over):
    """the most pairs that run without sorting, and one token more: tiles of the sorted rows; fewer where rows are not whole 16-byte pieces"""
    top = ff["router"]["top"]
    T = limit // top + over
    cfg = model([retention_layer(mlp=ff)], width=width)
    w = O.random_weights(cfg, seed=1)
    eng = make_engine(cfg, w, backend)
    h = torch.randn(T, width, generator=torch.Generator().manual_seed(T))
    want = O.feed_forward(h.double(), {k: v.double() for k, v in w.items()}, "l0.mlp.", ff)
    eng.L = _Spy(eng.L)
    got = eng._moe(eng.cfg.layers[0].ff, eng.w.layers[0], h.to(backend[0]))
    assert rel_err(got, want) < 1e-5
    assert ("lp_moe_align" in eng.L.called) == bool(over) and ("lp_linear_group_pairs" in eng.L.called) != bool(over)
