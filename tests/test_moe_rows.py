"""lp_moe_combine takes four columns a thread where rows are whole 16-byte pieces: the same sums bit for bit."""
import ctypes as C

import pytest
import torch

from leopard_b200 import _lib
from seqlm_common import backend, emu_lib, rel_err  # noqa: F401

FEW = 296      # tokens up to which a CTA has as many threads as it can use


def _of(backend):
    return backend[0], backend[1] if backend[1] is not None else _lib.stream32_lib(), \
        C.c_void_p(torch.cuda.current_stream().cuda_stream) if backend[0] != "cpu" else None


@pytest.mark.parametrize("T,D,top", [(3, 520, 2), (FEW + 1, 36, 5), (FEW + 1, 516, 2), (2, 4100, 1), (5, 33, 9)])
@pytest.mark.parametrize("extras", [True, False])
def test_columns_together_and_alone(backend, T, D, top, extras):
    dev, L, stream = _of(backend)
    g = torch.Generator().manual_seed(D)
    y, shared = torch.randn(T * top, D, generator=g).to(dev), torch.randn(T, D, generator=g).to(dev)
    rows = torch.randperm(T * top, generator=g).to(torch.int32).to(dev)
    w, gate = torch.rand(T, top, generator=g).to(dev), torch.rand(T, generator=g).to(dev)
    got = []
    for shift in (0, 1):      # off 16-byte boundaries: a column a thread
        flat = torch.full((T * D + 4,), 7.0, device=dev)
        rc = L.lp_moe_combine(_lib.ptr(y), D, _lib.ptr(rows), _lib.ptr(w) if extras else None, top, _lib.ptr(shared) if extras else None, D,
                              _lib.ptr(gate) if extras else None, flat.data_ptr() + 4 * shift, D, T, D, stream)
        assert rc == 0, L.lp_last_error()
        assert bool((flat[T * D + shift:] == 7.0).all()) and bool((flat[:shift] == 7.0).all())
        got.append(flat[shift: shift + T * D].view(T, D).cpu())
    assert torch.equal(*got)
    picked = y.double().cpu()[rows.long().cpu()].view(T, top, D)
    want = (picked * w.double().cpu()[..., None]).sum(1) + gate.double().cpu()[:, None] * shared.double().cpu() if extras else picked.sum(1)
    assert rel_err(got[0], want) < 1e-6
