"""The product of up to 64 rows as one stream of weights through a ring of TMA pieces (lp_linear, lp_linear_group_pairs with K a multiple of 64) against a
float64 product: pieces that end within K, tiles that end within N, more tiles than CTAs and more pieces than the ring has places, both operand types, batches,
segments, gated units, groups whose pairs fill several blocks; weights that may be read early and weights that may not.  The dispatch takes the ring where it is the
faster kernel, by tiles per SM and K; the sizes lie on both sides of its lines, on the emulator's four or sixteen SMs and on the GPU's.

Error bounds: as for the weight-streaming kernel, products are exact and K / 16 fp32 sums follow, less than 2e-6 of the result's size for K <= 2112."""
import ctypes as C
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from leopard_b200 import _lib
from seqlm_common import backend, emu_lib, rel_err  # noqa: F401
from test_linear_stream import _call, _data

F32, BF16 = torch.float32, torch.bfloat16


def _leave_nans(backend):
    """shared memory as a product of NaNs leaves it (the emulated kernels find NaNs in any case)"""
    if backend[0] == "cuda":
        a, w = torch.full((64, 1664), float("nan"), dtype=BF16, device="cuda"), torch.full((3200, 1664), float("nan"), dtype=BF16, device="cuda")
        _call(backend, a, w, torch.empty(64, 3200, device="cuda"), 64)
        _call(backend, a, w, torch.empty(8, 3200, device="cuda"), 8)


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("M,N,K", [(1, 1, 64), (1, 1, 576), (1, 200, 2112), (3, 40, 576), (5, 90, 832), (5, 130, 512), (8, 16, 1600), (8, 300, 64), (8, 300, 576), (9, 33, 640), (16, 130, 448), (17, 40, 320), (32, 130, 576), (33, 72, 256), (64, 130, 832), (12, 200, 2112), (20, 100, 1088), (33, 64, 576), (64, 160, 2112)])
@pytest.mark.parametrize("constant", [0, 1])
def test_rows_tiles_and_pieces(backend, dtype, M, N, K, constant):
    a, w, want, ad, wd = _data(M, N, K, dtype, backend[0])
    out = torch.empty(M, N, device=backend[0])
    _call(backend, ad, wd, out, M, constant=constant)
    assert rel_err(out, want) < 2e-6
    again = torch.empty(M, N, device=backend[0])
    _call(backend, ad, wd, again, M, constant=1 - constant)
    assert torch.equal(out, again)


@pytest.fixture
def sixteen_sms(backend):
    """products of a tile an SM take the ring at a shorter K than those of several rounds"""
    if backend[1] is not None:
        backend[1].emu_set_sm_count(16)
    yield
    if backend[1] is not None:
        backend[1].emu_set_sm_count(4)


@pytest.mark.usefixtures("sixteen_sms")
@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("M", [3, 12, 20, 50])
def test_gated_and_added(backend, dtype, M):
    N, K = 76, 704
    a, w, z, ad, wd = _data(M, N, K, dtype, backend[0])
    half = torch.empty(M, N // 2, device=backend[0])
    _call(backend, ad, wd, half, M, epi=_lib.EPI_SILU_GATE, constant=1)
    p, q = z[:, : N // 2], z[:, N // 2:]
    assert rel_err(half, p * torch.sigmoid(p) * q) < 5e-6      # the unit's slope is below 1.1, its factors carry one error each
    g = torch.Generator().manual_seed(1)
    bias, scale, gate, x = torch.randn(N, generator=g), torch.rand(M, generator=g), torch.randn(M, N, generator=g), torch.randn(M, N, generator=g)
    out = x.clone().to(backend[0])
    _call(backend, ad, wd, out, M, bias=bias.to(backend[0]), row_scale=scale.to(backend[0]), gate=gate.to(backend[0]), ldg=N, epi=_lib.EPI_RELU2,
          c_accum=1, c_scale=0.5, constant=1)
    v = torch.relu(z * scale.double()[:, None] + bias.double()) ** 2 * torch.sigmoid(gate.double())
    assert rel_err(out, x.double() + 0.5 * v) < 2e-6


@pytest.mark.usefixtures("sixteen_sms")
@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("M", [2, 11, 30, 41])
def test_batches_and_segments(backend, dtype, M):
    g = torch.Generator().manual_seed(M)
    heads, N, K = 5, 40, 576
    a, w = torch.randn(M, heads * (K + 8), generator=g).to(dtype), torch.randn(heads, N, K, generator=g).to(BF16)
    ad, wd = a.to(backend[0]), w.to(backend[0])
    out = torch.empty(M, heads * N, device=backend[0])
    _call(backend, ad, wd, out, M, batch=heads, a_batch=K + 8, c_batch=N, constant=1)
    want = torch.cat([a[:, h * (K + 8): h * (K + 8) + K].double() @ w[h].double().T for h in range(heads)], 1)
    assert rel_err(out, want) < 2e-6
    _call(backend, ad, wd, out, M, batch=heads, a_batch=0, c_batch=N, constant=1)      # one operand for all problems: not a tensor map's stride
    want = torch.cat([a[:, :K].double() @ w[h].double().T for h in range(heads)], 1)
    assert rel_err(out, want) < 2e-6
    segs, seg, N = 3, 64, 200
    a, w = torch.randn(segs, M, K, generator=g).to(dtype), torch.randn(N, K, generator=g).to(BF16)
    ad, wd = a.to(backend[0]), w.to(backend[0])
    out = torch.empty(M, N, device=backend[0])
    _call(backend, ad, wd, out, M, seg_cols=seg, n_segs=segs, a_seg=M * K, constant=1)
    which = [min(n // seg, segs - 1) for n in range(N)]
    want = torch.stack([a[i].double() @ w[n].double() for n, i in enumerate(which)], 1)
    assert rel_err(out, want) < 2e-6


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("n_pairs,groups,a_div", [(1, 4, 1), (10, 3, 2), (37, 9, 1), (64, 33, 4), (70, 200, 2)])
def test_pairs(backend, dtype, n_pairs, groups, a_div):
    g = torch.Generator().manual_seed(n_pairs)
    N, K = 44, 1088
    a, w = torch.randn((n_pairs + a_div - 1) // a_div, K, generator=g).to(dtype), torch.randn(groups, N, K, generator=g).to(BF16)
    of = torch.randint(0, groups, (n_pairs,), generator=g)
    of[: n_pairs // 2] = groups - 1      # more than a tile's rows in one group, groups without pairs
    ad, wd = a.to(backend[0]), w.to(backend[0])
    out = torch.full((n_pairs, N), 7.0, device=backend[0])
    _call(backend, ad, wd, out, 1, pairs=of.to(torch.int32).to(backend[0]), groups=groups, a_div=a_div)
    want = torch.stack([a[z // a_div].double() @ w[int(of[z])].double().T for z in range(n_pairs)])
    assert rel_err(out, want) < 2e-6


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("of", [[4], [4, 1, 4, 5], [0] * 7 + [2] * 3, [3] * 12])
@pytest.mark.parametrize("K", [192, 704, 1088])
def test_few_pairs_of_many_tiles(backend, dtype, of, K):
    """forty tiles an SM, of which most belong to groups without pairs: K of odd multiples of 64 ends within what a warp takes of a piece; more than 8 pairs in a group"""
    g = torch.Generator().manual_seed(K + len(of))
    N, groups = (432, 6) if backend[0] == "cpu" else (7904, 12)
    assert groups * (N // 16) >= 40 * (4 if backend[0] == "cpu" else 148)      # the dispatch's line
    a, w = torch.randn(len(of), K, generator=g).to(dtype), torch.randn(groups, N, K, generator=g).to(BF16)
    ad, wd = a.to(backend[0]), w.to(backend[0])
    _leave_nans(backend)
    out = torch.full((len(of), N), 7.0, device=backend[0])
    _call(backend, ad, wd, out, 1, pairs=torch.tensor(of, dtype=torch.int32).to(backend[0]), groups=groups)
    want = torch.stack([ad[z].double() @ wd[of[z]].double().T for z in range(len(of))])
    assert rel_err(out, want) < 2e-6


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("n_pairs,groups,N,K,a_div", [(12, 4, 4096, 1088, 1), (30, 8, 2064, 1088, 4), (32, 8, 432, 704, 1)])
def test_pairs_in_blocks(backend, dtype, n_pairs, groups, N, K, a_div):
    """enough weights for the ring, or tiles (on the emulator's four SMs): groups of more than 8 and more than 16 pairs, a block of 8 after the other, and groups without any"""
    g = torch.Generator().manual_seed(n_pairs)
    a, w = torch.randn((n_pairs + a_div - 1) // a_div, K, generator=g).to(dtype), torch.randn(groups, N, K, generator=g).to(BF16)
    of = torch.full((n_pairs,), groups - 1)
    of[1::7] = 1
    ad, wd = a.to(backend[0]), w.to(backend[0])
    _leave_nans(backend)
    out = torch.full((n_pairs, N), 7.0, device=backend[0])
    _call(backend, ad, wd, out, 1, pairs=of.to(torch.int32).to(backend[0]), groups=groups, a_div=a_div)
    want = torch.stack([a[z // a_div].double() @ w[int(of[z])].double().T for z in range(n_pairs)])
    assert rel_err(out, want) < 2e-6


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("M,N,K", [(1, 3600, 8256), (8, 3200, 3136), (8, 11200, 5184), (16, 2500, 8256), (13, 5000, 2112), (30, 2400, 5184), (64, 4800, 4160)])
def test_more_tiles_than_sms_and_more_pieces_than_stages(dtype, M, N, K):
    """the ring goes round several times within a tile and from tile to tile; fp32 rows with two tiles a piece (149 to 222 tiles, and more than 592).  K / 16 sums that are kept
    exactly, or for more than 16 rows rounded: below 3e-6 of the result for K <= 8256."""
    backend = "cuda", None
    a, w, want, ad, wd = _data(M, N, K, dtype, "cuda")
    out, again = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    _call(backend, ad, wd, out, M, constant=1)
    assert rel_err(out, want) < 3e-6
    _call(backend, ad, wd, again, M)
    assert torch.equal(out, again)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("n_pairs,groups,N,K", [(16, 8, 1216, 5824), (30, 8, 2104, 5824), (100, 50, 1944, 1344)])
def test_pairs_of_many_tiles(dtype, n_pairs, groups, N, K):
    backend = "cuda", None
    g = torch.Generator().manual_seed(n_pairs)
    a, w = torch.randn(n_pairs, K, generator=g).to(dtype), torch.randn(groups, N, K, generator=g).to(BF16)
    of = torch.randint(0, groups, (n_pairs,), generator=g)
    ad, wd = a.cuda(), w.cuda()
    _leave_nans(backend)
    out = torch.full((n_pairs, N), 7.0, device="cuda")
    _call(backend, ad, wd, out, 1, pairs=of.to(torch.int32).cuda(), groups=groups)
    want = torch.stack([a[z].double() @ w[int(of[z])].double().T for z in range(n_pairs)])
    assert rel_err(out, want) < 3e-6


def test_operands_that_lie_far_apart(emu_lib):
    """the operands of two problems, 32 TiB of addresses from one to the other: more than a tensor map's stride can be"""
    libc = C.CDLL(None, use_errno=True)
    libc.mmap.restype, libc.mmap.argtypes = C.c_void_p, [C.c_void_p, C.c_size_t, C.c_int, C.c_int, C.c_int, C.c_long]
    M, N, K, far = 2, 24, 576, 1 << 45
    a = torch.randn(2, M, K, generator=torch.Generator().manual_seed(1))
    base = 1 << 44
    for z in range(2):
        at = libc.mmap(base + z * far, 1 << 16, 3, 0x100022, -1, 0)      # private and anonymous, at this address or nowhere
        assert at == base + z * far
        C.memmove(at, a[z].data_ptr(), 4 * M * K)
    w = torch.randn(2, N, K, generator=torch.Generator().manual_seed(2)).to(BF16)
    out = torch.empty(M, 2 * N)
    d = _lib.LinearDesc(A=base, lda=K, a_batch=far // 4, a_fp32=1, W=_lib.ptr(w), ldw=K, w_batch=N * K, C=_lib.ptr(out), ldc=2 * N, c_batch=N, c_fp32=1, M=M, N=N, K=K, batch=2)
    assert emu_lib.lp_linear(C.byref(d), None) == 0, emu_lib.lp_last_error()
    assert rel_err(out, torch.cat([a[z].double() @ w[z].double().T for z in range(2)], 1)) < 2e-6


@pytest.mark.parametrize("warp,pairs", [(0, False), (0, True), (13, True), (1, False), (9, False)])
def test_lanes_that_lag_behind(emu_lib, warp, pairs):
    """the warps that fill the ring, take the products and add them up: lanes that only look on may run as late as they like (a block that gets stuck ends the process, so it is another one)"""
    r = subprocess.run([sys.executable, "-c", f"import test_linear_ring as t; t.product_with_lagging_lanes({emu_lib._name!r}, {warp}, {pairs})"],
                       cwd=Path(__file__).parent, env={**os.environ, "PYTHONPATH": str(Path(__file__).resolve().parents[1])}, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]


def product_with_lagging_lanes(path, warp, pairs):
    """one row, pieces for two rounds of the ring and more in every CTA"""
    lib = _lib.bind_stream32(C.CDLL(path))
    lib.emu_set_lagging(warp, 1)
    N, K = (2560, 192) if pairs else (256, 2048)
    a, w, want, ad, wd = _data(1, N, K, BF16, "cpu")
    out = torch.empty(1, N)
    _call(("cpu", lib), ad, wd[None] if pairs else wd, out, 1, **({"pairs": torch.zeros(1, dtype=torch.int32), "groups": 1} if pairs else {}))
    assert rel_err(out, want) < 2e-6


def test_numbers_that_are_not_finite(backend):
    """an fp32 row with an infinity: its products are those of the uncut number; rows and columns beside it keep theirs"""
    M, N, K = 5, 40, 640
    a, w, want, ad, wd = _data(M, N, K, F32, "cpu")
    a = a.clone()
    a[2, 600] = float("inf")
    a[4, 3] = float("nan")
    w[7, 600] = 0.0
    want = a.double() @ w.double().T
    out = torch.empty(M, N, device=backend[0])
    _call(backend, a.to(backend[0]), w.to(backend[0]), out, M, constant=1)
    out = out.cpu().double()
    fine = torch.isfinite(want)
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(out[torch.isinf(want)], want[torch.isinf(want)])
    assert rel_err(out[fine], want[fine]) < 2e-6


@pytest.mark.parametrize("M", [3, 12, 20])
def test_weights_that_are_not_finite(backend, M):
    """infinite weights times fp32 rows whose terms differ in sign: each such sum is taken again, and is infinite or a NaN as the uncut product's is"""
    N, K = 40, 640
    a, w, _, _, _ = _data(M, N, K, F32, "cpu")
    a, w = a.to(BF16).float(), w.clone()      # two terms that are zero
    w[:, 77] = float("inf")
    w[5, 600] = float("-inf")
    a[1, 77] = 0.0
    want = a.double() @ w.double().T
    out = torch.empty(M, N, device=backend[0])
    _call(backend, a.to(backend[0]), w.to(backend[0]), out, M, constant=1)
    out = out.cpu().double()
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(out[torch.isinf(want)], want[torch.isinf(want)])
