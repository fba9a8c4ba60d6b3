"""The weight-streaming product of up to 64 rows (lp_linear), of grouped pairs (lp_linear_group_pairs) and the tile
product of more rows (lp_linear, lp_linear_grouped) against a float64 product: the edges of their row groups, column tiles and K steps, both
operand types, every kind of epilogue; on the kernel sources under the CPU emulator and, marked gpu, on the native library.

Error bounds: products are exact (a bf16 weight times a bf16 value or one of three bf16 terms of an fp32 one), at most about K / 16 fp32 sums
follow: for K <= 400 below 32 * 2^-24 < 2e-6 of the result's size in the root mean square."""
import ctypes as C

import pytest
import torch

from leopard_b200 import _lib
from seqlm_common import backend, emu_lib, rel_err  # noqa: F401

F32, BF16 = torch.float32, torch.bfloat16


def _lib_of(backend):
    return backend[1] if backend[1] is not None else _lib.stream32_lib()


def _call(backend, a, w, out, M, batch=1, pairs=None, groups=None, a_div=1, constant=0, **kw):
    L = _lib_of(backend)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream) if a.is_cuda else None
    d = _lib.LinearDesc(A=_lib.ptr(a), lda=a.stride(-2), a_batch=kw.pop("a_batch", 0), a_fp32=int(a.dtype == F32), W=_lib.ptr(w), ldw=w.stride(-2),
                        w_batch=w.stride(0) if w.dim() == 3 else 0, C=_lib.ptr(out), ldc=out.stride(0), c_batch=kw.pop("c_batch", 0),
                        c_fp32=int(out.dtype == F32), M=M, N=w.shape[-2], K=w.shape[-1], batch=batch, **{k: _lib.ptr(v) if isinstance(v, torch.Tensor) else v for k, v in kw.items()})
    if constant:
        d.epi |= _lib.LINEAR_W_CONSTANT
    if pairs is None:
        rc = L.lp_linear(C.byref(d), stream)
    elif groups is None:
        rc = L.lp_linear_pairs(C.byref(d), _lib.ptr(pairs), a_div, pairs.numel(), stream)
    else:
        rc = L.lp_linear_group_pairs(C.byref(d), _lib.ptr(pairs), groups, a_div, pairs.numel(), stream)
    assert rc == 0, L.lp_last_error()


def _data(M, N, K, dtype, device, seed=0):
    g = torch.Generator().manual_seed(seed + 1000 * M + N + K)
    a = torch.randn(M, K, generator=g).to(dtype)
    w = (torch.randn(N, K, generator=g) * K ** -0.5).to(BF16)
    return a, w, a.double() @ w.double().T, a.to(device), w.to(device)


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("M,N,K", [(1, 1, 8), (8, 17, 40), (9, 33, 256), (16, 16, 264), (33, 48, 400), (64, 40, 72), (65, 130, 40), (129, 9, 72),
                                   (33, 24, 16), (49, 24, 16), (64, 24, 32), (64, 24, 40), (65, 130, 32), (65, 130, 136), (129, 9, 136), (100, 300, 264)])
def test_rows_columns_and_steps(backend, dtype, M, N, K):
    a, w, want, ad, wd = _data(M, N, K, dtype, backend[0])
    out = torch.empty(M, N, device=backend[0])
    _call(backend, ad, wd, out, M)
    assert rel_err(out, want) < 2e-6
    low = torch.empty(M, N, dtype=BF16, device=backend[0])
    _call(backend, ad, wd, low, M)
    assert torch.equal(low, out.to(BF16))


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("M,K", [(11, 64), (70, 64), (70, 200)])
def test_epilogues(backend, dtype, M, K):
    N = 36
    a, w, z, ad, wd = _data(M, N, K, dtype, backend[0])
    g = torch.Generator().manual_seed(1)
    bias, scale, gate, x = torch.randn(N, generator=g), torch.rand(M, generator=g), torch.randn(M, N, generator=g), torch.randn(M, N, generator=g)
    out = x.clone().to(backend[0])
    _call(backend, ad, wd, out, M, bias=bias.to(backend[0]), row_scale=scale.to(backend[0]), gate=gate.to(backend[0]), ldg=N, epi=_lib.EPI_RELU2,
          c_accum=1, c_scale=0.5)
    v = torch.relu(z * scale.double()[:, None] + bias.double()) ** 2 * torch.sigmoid(gate.double())
    assert rel_err(out, x.double() + 0.5 * v) < 2e-6
    half = torch.empty(M, N // 2, device=backend[0])
    _call(backend, ad, wd, half, M, epi=_lib.EPI_SILU_GATE)
    p, q = z[:, : N // 2], z[:, N // 2:]
    assert rel_err(half, p * torch.sigmoid(p) * q) < 5e-6      # the unit's slope is below 1.1, its factors carry one error each


def test_batches_and_segments(backend):
    g = torch.Generator().manual_seed(3)
    for M, K in ((10, 40), (66, 200), (66, 40)):
        heads, N = 3, 24
        a, w = torch.randn(M, heads * (K + 8), generator=g), torch.randn(heads, N, K, generator=g).to(BF16)
        ad, wd = a.to(backend[0]), w.to(backend[0])
        out = torch.empty(M, heads * N, device=backend[0])
        _call(backend, ad, wd, out, M, batch=heads, a_batch=K + 8, c_batch=N)
        want = torch.cat([a[:, (K + 8) * h:(K + 8) * h + K].double() @ w[h].double().T for h in range(heads)], 1)
        assert rel_err(out, want) < 2e-6
        gate, x = torch.randn(M, heads * N, generator=g), torch.randn(M, heads * N, generator=g)      # a gate per problem, added to what is there
        out, gd = x.clone().to(backend[0]), gate.to(backend[0])
        _call(backend, ad, wd, out, M, batch=heads, a_batch=K + 8, c_batch=N, gate=gd, ldg=heads * N, gate_batch=N, c_accum=1, c_scale=0.5)
        assert rel_err(out, x.double() + 0.5 * want * torch.sigmoid(gate.double())) < 2e-6
        out = torch.empty(M, heads * N, dtype=BF16, device=backend[0])
        _call(backend, ad, wd, out, M, batch=heads, a_batch=K + 8, c_batch=N, gate=gd, ldg=heads * N, gate_batch=N)
        assert rel_err(out, want * torch.sigmoid(gate.double())) < 3e-3
    K = 40
    ops, w = torch.randn(2, 5, K, generator=g).to(BF16), torch.randn(40, K, generator=g).to(BF16)
    out = torch.empty(5, 40, device=backend[0])
    od, wd = ops.to(backend[0]), w.to(backend[0])
    _call(backend, od, wd, out, 5, seg_cols=16, n_segs=2, a_seg=od.stride(0))
    assert rel_err(out, torch.cat([ops[0].double() @ w[:16].double().T, ops[1].double() @ w[16:].double().T], 1)) < 2e-6


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("n_pairs,groups", [(1, 2), (40, 3), (150, 2)])
def test_pairs_of_groups(backend, dtype, n_pairs, groups):
    """a group without pairs, one pair, and more pairs than one round over the weights takes; two pairs to a row of A"""
    g = torch.Generator().manual_seed(n_pairs)
    N, K = 20, 48
    a = torch.randn((n_pairs + 1) // 2, K, generator=g).to(dtype)
    w = (torch.randn(groups + 1, N, K, generator=g) * K ** -0.5).to(BF16)      # nobody chooses the last group
    of = torch.randint(0, groups, (n_pairs,), generator=g).to(torch.int32)
    out = torch.empty(n_pairs, N, device=backend[0])
    _call(backend, a.to(backend[0]), w.to(backend[0]), out, 1, groups=groups + 1, pairs=of.to(backend[0]), a_div=2)
    want = torch.stack([w[int(e)].double() @ a[z // 2].double() for z, e in enumerate(of)])
    assert rel_err(out, want) < 2e-6
    # without the number of groups a description's batch means nothing, whatever it holds
    out.fill_(9.0)
    _call(backend, a.to(backend[0]), w.to(backend[0]), out, 1, batch=groups - 1, pairs=of.to(backend[0]), a_div=2)
    assert rel_err(out, want) < 2e-6


@pytest.mark.parametrize("M,N,K", [(4, 96, 512), (8, 48, 2048)])
def test_few_rows_lose_no_more_than_a_lane_of_multiply_adds(backend, M, N, K):
    """bf16 rows up to eight against float64, beside what fp32 multiply-adds of a warp's lanes and a tree over the lanes lose on the same data"""
    a, w, want, ad, wd = _data(M, N, K, BF16, backend[0])
    out = torch.empty(M, N, device=backend[0])
    _call(backend, ad, wd, out, M)
    lanes = torch.zeros(M, N, 32)
    for k in range(0, K, 256):
        for i in range(8):      # lane l takes k + 8 l .. k + 8 l + 7
            x, y = a[:, k + i:k + 256:8].double(), w[:, k + i:k + 256:8].double()
            lanes = (lanes.double() + x[:, None] * y[None]).float()      # one rounding, as a fused multiply-add
    for half in (16, 8, 4, 2, 1):
        lanes = lanes[..., :half] + lanes[..., half:2 * half]
    assert rel_err(out, want) < 1.05 * rel_err(lanes[..., 0], want)


def test_unusual_numbers(backend):
    """an infinity or a NaN in a row of A stays in its row, as it does in an fp32 product; the largest number is no infinity"""
    M, N, K = 5, 16, 40
    a, w, _, _, wd = _data(M, N, K, F32, backend[0])
    a[1, 3], a[2, 7], a[3, 9] = float("inf"), float("nan"), torch.finfo(F32).max
    a[4, 0] = torch.tensor(0x7F800001, dtype=torch.int32).view(F32)      # a NaN whose upper half reads as infinity
    w[:, 9] = 0.25
    out = torch.empty(M, N, device=backend[0])
    _call(backend, a.to(backend[0]), w.to(backend[0]), out, M)
    out = out.cpu()
    want = a.double() @ w.double().T
    assert torch.isfinite(out[0]).all() and torch.isnan(out[2]).all() and torch.isnan(out[4]).all()
    assert torch.equal(out[1].isinf(), want[1].isinf()) and torch.equal(out[1].sign(), want[1].sign().float())
    assert rel_err(out[3], want[3]) < 2e-6


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("M,kind", [(5, "rows"), (40, "rows"), (70, "rows"), (5, "pairs"), (64, "groups")])
def test_infinite_weights(backend, dtype, M, kind):
    """an infinite weight makes its column's outputs infinite, with the sign of the product, in both halves of a gated unit too; NaN where it
    meets a zero, an infinity of the other sign or a NaN"""
    N, K, dev = 24, 136, backend[0]
    a, w, _, _, _ = _data(M, N, K, dtype, dev)
    a[0, 3], a[1, 5] = 0.0, float("nan")
    w[2, 3], w[5, 3], w[7, 11], w[7, 12], w[N // 2 + 3, 30] = float("inf"), -float("inf"), float("inf"), -float("inf"), float("inf")
    want = a.double() @ w.double().T
    ad, wd = a.to(dev), w.to(dev)
    out, half = torch.empty(M, N, device=dev), torch.empty(M, N // 2, device=dev)

    def call(o, **kw):
        if kind == "groups":
            L = _lib_of(backend)
            d = _lib.LinearDesc(A=_lib.ptr(ad), lda=K, a_fp32=int(dtype == F32), W=_lib.ptr(wd), ldw=K, w_batch=N * K, C=_lib.ptr(o), ldc=o.stride(0),
                                c_fp32=1, M=M, N=N, K=K, batch=1, **kw)
            rows, group = torch.arange(M, dtype=torch.int32, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
            stream = C.c_void_p(torch.cuda.current_stream().cuda_stream) if ad.is_cuda else None
            assert L.lp_linear_grouped(C.byref(d), _lib.ptr(group), 1, _lib.ptr(rows), stream) == 0
        elif kind == "pairs":
            _call(backend, ad, wd[None].expand(2, N, K).contiguous(), o, 1, groups=2, pairs=torch.arange(M, device=dev).to(torch.int32) % 2, **kw)
        else:
            _call(backend, ad, wd, o, M, **kw)

    call(out)
    assert torch.equal(out.cpu().isnan(), want.isnan()) and torch.equal(out.cpu()[want.isinf()].double(), want[want.isinf()])
    assert rel_err(out.cpu()[want.isfinite()], want[want.isfinite()]) < 2e-6
    call(half, epi=_lib.EPI_SILU_GATE)
    g = want[:, : N // 2].float()
    unit = g / (1 + torch.exp(-g)) * want[:, N // 2:].float()      # in fp32, where exp(-(-inf)) is an infinity too
    assert torch.equal(half.cpu().isnan(), unit.isnan()) and torch.equal(half.cpu()[unit.isinf()], unit[unit.isinf()])


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("K", [24, 40, 136])
def test_row_tiles_of_groups(backend, dtype, K):
    """tiles of 64 gathered rows, each on its group's weight; padding rows are zeros, a tile without a group is left alone"""
    g = torch.Generator().manual_seed(9)
    N, T = 136, 30
    a, w = torch.randn(T, K, generator=g).to(dtype), (torch.randn(3, N, K, generator=g) * K ** -0.5).to(BF16)
    groups, rows = torch.tensor([2, -1, 0], dtype=torch.int32), torch.randint(-1, T, (192,), generator=g).to(torch.int32)
    out = torch.full((192, N), 7.0)
    od = out.clone().to(backend[0])
    L = _lib_of(backend)
    ad, wd, gd, rd = a.to(backend[0]), w.to(backend[0]), groups.to(backend[0]), rows.to(backend[0])
    d = _lib.LinearDesc(A=_lib.ptr(ad), lda=K, a_fp32=int(dtype == F32), W=_lib.ptr(wd), ldw=K, w_batch=N * K, C=_lib.ptr(od), ldc=N, c_fp32=1,
                        M=192, N=N, K=K, batch=1)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream) if ad.is_cuda else None
    assert L.lp_linear_grouped(C.byref(d), _lib.ptr(gd), 3, _lib.ptr(rd), stream) == 0
    picked = torch.where((rows >= 0)[:, None], a.double()[rows.clamp(min=0).long()], 0.0)
    want = torch.cat([picked[:64] @ w[2].double().T, out[64:128].double(), picked[128:] @ w[0].double().T])
    assert rel_err(od, want) < 2e-6
