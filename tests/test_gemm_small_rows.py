"""GEMMs of fewer 256-row tiles than CTA pairs run as pairs of 128-wide tiles: the same bits as CTAs of 256-wide ones, row statistics (one pair per 128 columns,
added up in the same order), rotated heads and residuals included; on the kernel source under the CPU emulator and, marked gpu, through the dispatch of
lp_gemm_bf16_ex (lp_gemm_set_pair_mode(0) keeps the single CTAs)."""
import ctypes as C

import pytest
import torch

from test_gemm_kernel_emulated import BF, _Fx, _gemm_ex, _split_stats, emu  # noqa: F401


@pytest.mark.parametrize("M,N,K,res", [(201, 256, 136, True), (300, 384, 72, True), (90, 392, 200, False)])
def test_statistics_of_wide_tiles(emu, M, N, K, res):
    g = torch.Generator().manual_seed(M)
    a = torch.randn((M, K), generator=g).to(BF)
    w = (torch.randn((N, K), generator=g) * K ** -0.5).to(BF)
    b = torch.randn(N, generator=g)
    r = torch.randn((M, N), generator=g).to(BF) if res else None
    parts, outs, stats = 2 * (-(-N // 256)), [], []
    for bn, pair, tma in ((256, False, 0), (128, True, 0), (128, True, 1)):
        out, st = torch.full((M, N), float("nan"), dtype=BF), torch.full((M, parts, 2), float("nan"))
        emu.emu_gemm_set_stat_256(1)
        emu.emu_gemm_set_tma_residual(tma)
        try:
            _gemm_ex(emu, a, w, out, bias=b, res=r, bn=bn, pair=pair, ctas=4, fx=_Fx(stats_out=st.data_ptr()))
        finally:
            emu.emu_gemm_set_stat_256(0)
            emu.emu_gemm_set_tma_residual(0)
        outs.append(out)
        stats.append(st)
    assert all(torch.equal(o, outs[0]) for o in outs) and all(torch.equal(s, stats[0]) for s in stats)


def test_a_tile_is_a_head(emu):
    M, K, heads, rot = 150, 136, 4, 3
    g = torch.Generator().manual_seed(5)
    x = torch.randn((M, K), generator=g).to(BF)
    w = (torch.randn((heads * 128, K), generator=g) * K ** -0.5).to(BF)
    ang = torch.rand((M, 64), generator=g) * 6.28
    cos, sin, stats = ang.cos().contiguous(), ang.sin().contiguous(), _split_stats(x, 1)
    outs = []
    for bn, pair in ((256, False), (128, True)):
        outs.append(torch.full((M, heads * 128), float("nan"), dtype=BF))
        fx = _Fx(norm_mode=1, stats_in=stats.data_ptr(), stats_in_parts=1, norm_eps=1e-5, rope_cos=cos.data_ptr(), rope_sin=sin.data_ptr(), rope_heads=rot)
        _gemm_ex(emu, x, w, outs[-1], bn=bn, pair=pair, ctas=4, fx=fx)
    assert torch.equal(outs[0], outs[1])


def test_statistics_of_rotated_heads(emu):
    """row statistics of heads that are rotated, and of those that are not"""
    M, K, heads, rot = 140, 72, 5, 3
    g = torch.Generator().manual_seed(6)
    x = torch.randn((M, K), generator=g).to(BF)
    w = (torch.randn((heads * 128, K), generator=g) * K ** -0.5).to(BF)
    ang = torch.rand((M, 64), generator=g) * 6.28
    cos, sin, parts, seen = ang.cos().contiguous(), ang.sin().contiguous(), 6, []
    for bn, pair in ((256, False), (128, True), (128, False)):
        out, st = torch.full((M, heads * 128), float("nan"), dtype=BF), torch.full((M, parts, 2), float("nan"))
        emu.emu_gemm_set_stat_256(1)
        try:
            _gemm_ex(emu, x, w, out, bn=bn, pair=pair, ctas=4, fx=_Fx(stats_out=st.data_ptr(), rope_cos=cos.data_ptr(), rope_sin=sin.data_ptr(), rope_heads=rot))
        finally:
            emu.emu_gemm_set_stat_256(0)
        seen.append((out, st))
    assert all(torch.equal(o, seen[0][0]) and torch.equal(s, seen[0][1]) for o, s in seen)
    y = seen[0][0].float().view(M, heads, 128)
    assert torch.allclose(seen[0][1][:, :heads, 0], y.sum(2), atol=1e-3) and torch.allclose(seen[0][1][:, :heads, 1], (y * y).sum(2), rtol=1e-5)      # 128 fp32 additions


@pytest.mark.parametrize("M", [1, 32, 97, 129, 201, 224])
@pytest.mark.parametrize("pair", [False, True])
def test_gated_rows_of_a_ragged_block(emu, M, pair):
    """the rows that are there have the bits they have in a whole block, beside warps and lanes without a row"""
    g = torch.Generator().manual_seed(M)
    x, w = torch.randn((256, 72), generator=g).to(BF), (torch.randn((320, 72), generator=g) * 0.1).to(BF)
    x[M - 1, :] = 0      # a row of zeros that is there
    seen = []
    for rows in (256, M):
        seen.append(torch.full((256, 160), float("nan"), dtype=BF))
        _gemm_ex(emu, x[:rows], w, seen[-1][:rows], act=3, bn=256, pair=pair, ctas=4)
    assert torch.equal(seen[0][:M], seen[1][:M]) and bool(seen[1][M:].isnan().all()) and not bool(seen[0].isnan().any())


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 33, 128, 129, 201, 256, 300, 513, 676, 1000])
@pytest.mark.parametrize("N,K,what", [(4096, 512, "stats"), (1152, 1160, "stats"), (6144, 256, "rope"), (512, 4304, "plain"), (1152, 256, "modulo"), (1408, 256, "rope, stats")])
def test_dispatch_keeps_the_bits(native_lib, M, N, K, what):
    from leopard_b200 import _lib
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, K, device="cuda", generator=g).to(BF)
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).to(BF)
    r = torch.randn(M, N, device="cuda", generator=g).to(BF)
    ang = torch.rand(M, 64, device="cuda", generator=g) * 6.28
    cos, sin, parts = ang.cos().contiguous(), ang.sin().contiguous(), 2 * (-(-N // 256))
    seen = []
    for mode in (0, 1):
        out, st = torch.full((M, N), float("nan"), device="cuda", dtype=BF), torch.full((M, parts, 2), float("nan"), device="cuda")
        d = _lib.GemmDesc(A=a.data_ptr(), lda=K, W=w.data_ptr(), ldw=K, C=out.data_ptr(), ldc=N, M=M, N=N, K=K)
        if what in ("stats", "modulo"):
            d.residual, d.ldr, d.block_n, d.stats_out, d.stats_out_parts = r.data_ptr(), N, 256, st.data_ptr(), parts
            d.res_row_mod = 17 if what == "modulo" else 0
        if what == "rope, stats":
            d.stats_out, d.stats_out_parts = st.data_ptr(), parts
        if what[:4] == "rope":
            d.rope_cos, d.rope_sin, d.rope_heads = cos.data_ptr(), sin.data_ptr(), N // 128 - 8
        old = L.lp_gemm_set_pair_mode(mode)
        try:
            _lib.check(L.lp_gemm_bf16_ex(C.byref(d), C.c_void_p(torch.cuda.current_stream().cuda_stream)), "lp_gemm_bf16_ex")
        finally:
            L.lp_gemm_set_pair_mode(old)
        seen.append((out, st))
    assert torch.equal(seen[0][0], seen[1][0]) and not bool(torch.isnan(seen[1][0].float()).any())
    if "stats" in what or what == "modulo":
        assert torch.equal(seen[0][1], seen[1][1])
    if what == "plain":
        want = a.float() @ w.float().T
        assert float((seen[1][0].float() - want).abs().max() / want.abs().max()) < 8e-3
