"""The one-pass row norms (alone, into the stream, and the pair of norms around a residual update) and the elementwise passes in both of their
forms (four columns a thread; one where a width or a stride forbids it), against float64, on the kernel sources under the CPU emulator and,
marked gpu, on the native library.  Bounds: a norm is a sum of squares, a root, a division and two products in fp32, below 1e-6 of the
result; a bf16 store adds half a unit in the last of 8 bits, 2^-9 = 2e-3."""
import ctypes as C

import pytest
import torch

from leopard_b200 import _lib
from seqlm_common import backend, emu_lib, rel_err  # noqa: F401

F32, BF16 = torch.float32, torch.bfloat16
EPS = 1e-5


def _norm(x, g):
    x = x.double()
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * (g.double() if isinstance(g, torch.Tensor) else g)


def _setup(backend):
    device, lib = backend
    L = lib if lib is not None else _lib.stream32_lib()
    return device, L, C.c_void_p(torch.cuda.current_stream().cuda_stream) if device == "cuda" else None


@pytest.mark.parametrize("M,D", [(1, 4), (3, 36), (2, 30), (2, 4096), (5, 4104), (1, 8192), (1, 8196), (700, 64)])
@pytest.mark.parametrize("vector", [False, True])
def test_norms(backend, M, D, vector):
    device, L, st = _setup(backend)
    if device == "cpu" and M * D > 20000:
        M = 1
    g = torch.Generator().manual_seed(D + M)
    x, y = torch.randn(M, D, generator=g) * 3, torch.randn(M, D, generator=g)
    g1, g2 = (torch.rand(D, generator=g) + 0.5, torch.rand(D, generator=g) + 0.5) if vector else (1.25, 0.75)
    gd = [(1.0, t.to(device)) if vector else (t, None) for t in (g1, g2)]
    yd = y.to(device)
    for dt, tol in ((F32, 1e-6), (BF16, 3e-3)):
        out, xd = torch.empty(M, D, dtype=dt, device=device), x.clone().to(device)
        assert L.lp_rmsnorm_f32(_lib.ptr(yd), D, M, D, gd[0][0], _lib.ptr(gd[0][1]), EPS, _lib.ptr(out), D, int(dt == F32), None, 0, st) == 0
        assert rel_err(out, _norm(y, g1)) < tol
        assert L.lp_rmsnorm_add_norm_f32(_lib.ptr(yd), D, M, D, gd[0][0], _lib.ptr(gd[0][1]), EPS, _lib.ptr(xd), D, gd[1][0], _lib.ptr(gd[1][1]),
                                         _lib.ptr(out), D, int(dt == F32), st) == 0
        assert rel_err(xd, x.double() + _norm(y, g1)) < 1e-6
        assert rel_err(out, _norm(x.double() + _norm(y, g1), g2)) < tol
    xd = x.clone().to(device)
    assert L.lp_rmsnorm_f32(_lib.ptr(yd), D, M, D, gd[0][0], _lib.ptr(gd[0][1]), EPS, None, 0, 0, _lib.ptr(xd), D, st) == 0
    assert rel_err(xd, x.double() + _norm(y, g1)) < 1e-6


@pytest.mark.parametrize("N,ld", [(4, 8), (1032, 2064), (7, 14), (12, 27)])
def test_activations_and_update(backend, N, ld):
    device, L, st = _setup(backend)
    g = torch.Generator().manual_seed(N)
    M = 3
    z = torch.randn(M, ld, generator=g)
    for src in (F32, BF16):
        for dst, tol in ((F32, 1e-6), (BF16, 3e-3)):
            zi = z.to(src)
            a, b = zi[:, :N].double(), zi[:, N:2 * N].double()
            for mode, want in ((_lib.EPI_XIELU, torch.where(a > 0, 0.7 * a * a + a / 2, 0.9 * (torch.expm1(a.clamp(max=0)) - a) + a / 2)),
                               (_lib.EPI_RELU2, torch.relu(a) ** 2), (_lib.EPI_SILU_GATE, a * torch.sigmoid(a) * b)):
                out = torch.empty(M, N, dtype=dst, device=device)
                zd = zi.to(device)
                assert L.lp_glu_scaled_f32(_lib.ptr(zd), ld, int(src == F32), _lib.ptr(out), N, int(dst == F32), M, N, mode, 0.7, 0.9, None, st) == 0
                assert rel_err(out, want) < tol
    x, y = torch.randn(M, ld, generator=g), torch.randn(M, N, generator=g)
    xd, yd = x.clone().to(device), y.to(device)
    assert L.lp_axpy_f32(_lib.ptr(xd), ld, _lib.ptr(yd), N, 0.5, M, N, st) == 0
    assert rel_err(xd[:, :N], x[:, :N].double() + 0.5 * y.double()) < 1e-6 and torch.equal(xd[:, N:].cpu(), x[:, N:])


@pytest.mark.parametrize("D", [4, 30, 512, 516, 1030, 2052])
def test_embedding_rows(backend, D):
    """the numbers of threads that widths take, four columns a thread and one; an id outside the table reads its first row"""
    device, L, st = _setup(backend)
    g = torch.Generator().manual_seed(D)
    table, ids = torch.randn(7, D, generator=g).to(BF16), torch.tensor([3, 0, 6, 9, -1], dtype=torch.int32)
    out = torch.empty(5, D, device=device)
    td, idd = table.to(device), ids.to(device)
    assert L.lp_embed_rows_f32(_lib.ptr(idd), 5, _lib.ptr(td), D, 7, 0.5, _lib.ptr(out), D, D, st) == 0
    assert torch.equal(out.cpu(), table[[3, 0, 6, 0, 0]].float() * 0.5)
