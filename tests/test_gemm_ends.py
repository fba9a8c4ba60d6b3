"""lp_gemm_linear: the tcgen05 product that ends with the squared relu, xIELU or x <- x + m * product, against the product in fp32 (lp_gemm_bf16) followed by the
kernel of its own (lp_glu_f32, lp_axpy_f32): the same sums, the same operations, so the same bits up to the contraction of xIELU's two terms (one unit
of fp32 in each, seldom a bf16 rounding that falls the other way)."""
import ctypes as C

import pytest
import torch

from leopard_b200 import _lib

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("M,N,K", [(64, 128, 64), (65, 136, 72), (201, 4096, 512), (300, 1160, 1000), (201, 1024, 4096), (2500, 2304, 192), (4096, 2048, 256)])
def test_ends_are_the_kernels_that_followed(native_lib, M, N, K):
    L = _lib.stream32_lib()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, K, device="cuda", generator=g).to(BF16)
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).to(BF16)
    bias = torch.randn(N, device="cuda", generator=g)
    x = torch.randn(M, N, device="cuda", generator=g)
    for b in (None, bias):
        raw = torch.empty(M, N, device="cuda")
        _lib.check_on(L, L.lp_gemm_bf16(_lib.ptr(a), K, _lib.ptr(w), K, _lib.ptr(raw), N, M, N, K, _lib.ptr(b), None, 0, 0, _lib.ACT_NONE, 1, 0, stream), "gemm")
        want = a.double() @ w.double().T + (b.double() if b is not None else 0.0)
        assert float((raw.double() - want).norm() / want.norm()) < 1e-5      # one chain of tcgen05 over K <= 4096 cuts off below 1e-7 sqrt(K) of the result

        def call(out, **kw):
            d = _lib.LinearDesc(A=_lib.ptr(a), lda=K, W=_lib.ptr(w), ldw=K, C=_lib.ptr(out), ldc=N, M=M, N=N, K=K, batch=1, bias=_lib.ptr(b), **kw)
            _lib.check_on(L, L.lp_gemm_linear(C.byref(d), stream), "lp_gemm_linear")
            return out
        added = call(x.clone(), c_fp32=1, c_accum=1, c_scale=0.37)
        ref = x.clone()
        _lib.check_on(L, L.lp_axpy_f32(_lib.ptr(ref), N, _lib.ptr(raw), N, 0.37, M, N, stream), "axpy")
        assert torch.equal(added, ref)
        for epi, p, q in ((_lib.EPI_RELU2, 0.0, 0.0), (_lib.EPI_XIELU, 0.9, 1.1)):
            got, ref = call(torch.empty(M, N, device="cuda", dtype=BF16), epi=epi, epi_a=p, epi_b=q), torch.empty(M, N, device="cuda", dtype=BF16)
            _lib.check_on(L, L.lp_glu_scaled_f32(_lib.ptr(raw), N, 1, _lib.ptr(ref), N, 0, M, N, epi, p, q, None, stream), "glu")
            if epi == _lib.EPI_RELU2:
                assert torch.equal(got, ref)
            else:
                assert float((got != ref).float().mean()) < 1e-3 and float((got.float() - ref.float()).abs().max()) <= 2.0 ** -7 * float(ref.float().abs().max())


def test_what_it_does_not_end_is_refused(native_lib):
    L = _lib.stream32_lib()
    a, w, out = torch.zeros(64, 64, device="cuda", dtype=BF16), torch.zeros(128, 64, device="cuda", dtype=BF16), torch.zeros(64, 128, device="cuda")
    base = dict(A=_lib.ptr(a), lda=64, W=_lib.ptr(w), ldw=64, C=_lib.ptr(out), ldc=128, M=64, N=128, K=64, batch=1)
    for kw in (dict(c_fp32=1), dict(c_fp32=1, c_accum=1, epi=_lib.EPI_RELU2), dict(a_fp32=1, epi=_lib.EPI_RELU2), dict(epi=_lib.EPI_SILU_GATE), dict(epi=_lib.EPI_RELU2, batch=2)):
        assert L.lp_gemm_linear(C.byref(_lib.LinearDesc(**{**base, **kw})), None) == -1
