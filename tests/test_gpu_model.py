"""-m gpu: model-level parity of the CUDA path (through the C ABI) against the CPU oracle on identical seeded
weights and inputs.

Tolerance ladder: the CUDA path keeps bf16 activations with fp32 accumulation /
statistics, the oracle is fp32 math on the same bf16-rounded weights.  We bound  max|cuda - oracle| / max|oracle|
per stage; the measured values are printed (run with -s).  A 1e-3 logit
max-abs figure is below bf16 resolution for 32 layers and is NOT claimed.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

from leopard_b200.config import leopard_llava, reduced  # noqa: E402
from leopard_b200.engine import PrefillEngine  # noqa: E402
from leopard_b200.native_weights import load_hf  # noqa: E402
from leopard_b200.weights import SyntheticCheckpoint, synth_inputs  # noqa: E402
from oracle import model as om  # noqa: E402  (checker only)


def rel_err(got, ref):
    got, ref = got.float().cpu(), ref.float().cpu()
    return float((got - ref).abs().max() / ref.abs().max())


@pytest.fixture(scope="module")
def small(native_lib):
    cfg = reduced(leopard_llava(), vit_layers=2, dec_layers=2, vocab=2048)
    ck = SyntheticCheckpoint(cfg, seed=1234)
    eng = PrefillEngine(cfg, load_hf(cfg, lambda n: ck[n], "cuda"))
    return cfg, ck, eng


def test_vit_tower_and_shuffle(small):
    cfg, ck, eng = small
    pix, _ = synth_inputs(cfg, n_crops=2, n_text=8)
    ref = om.vit_forward(ck, cfg, pix.to(torch.bfloat16).float())
    got = eng.vit(pix.cuda(), shuffle=False).view(2, 676, 1152)
    e = rel_err(got, ref)
    print(f"\n[parity] vit(2 layers) last_hidden_state rel err {e:.4f}")
    assert e < 2e-2
    got_s = eng.vit(pix.cuda(), shuffle=True).view(2, 169, 4608)
    assert rel_err(got_s, om.pixel_shuffle(ref)) < 2e-2
    # fused shuffle store == standalone shuffle of the unshuffled output, bit for bit
    from leopard_b200 import ops
    assert torch.equal(ops.pixel_shuffle(got.view(-1, 1152), 26), got_s.view(-1, 4608))


def test_projector(small):
    cfg, ck, eng = small
    g = torch.Generator().manual_seed(4)
    x = torch.randn(3, 676, 1152, generator=g).to(torch.bfloat16)
    ref = om.projector(ck, cfg, x.float())
    from leopard_b200 import ops
    got = eng.project(ops.pixel_shuffle(x.cuda().view(-1, 1152), 26)).view(3, 169, 4096)
    e = rel_err(got, ref)
    print(f"\n[parity] projector rel err {e:.4f}")
    assert e < 1.5e-2


@pytest.mark.parametrize("crops", [1, 3, 28])
def test_projector_single_kernel_equals_two_launches(small, crops):
    """lp_project as ONE chained kernel (both GEMMs in a persistent launch with dataflow counters, lp_gemm_chain.cu) against the
    two-launch sequence: same bits, repeated launches leave the counters clean, and it really is a single launch."""
    cfg, ck, eng = small
    from leopard_b200 import _lib
    L = _lib.lib()
    g = torch.Generator().manual_seed(crops)
    x = torch.randn(crops * 169, 4608, generator=g).to(torch.bfloat16).cuda()
    try:
        L.lp_model_set_chained_projector(0)
        n0 = L.lp_launch_count()
        two = eng.project(x).clone()
        n_two = L.lp_launch_count() - n0
        L.lp_model_set_chained_projector(1)
        n0 = L.lp_launch_count()
        one = eng.project(x).clone()
        n_one = L.lp_launch_count() - n0
        again = eng.project(x).clone()
    finally:
        L.lp_model_set_chained_projector(1)
    torch.cuda.synchronize()
    assert (n_two, n_one) == (2, 1)
    assert torch.equal(one, two) and torch.equal(again, two)


def test_decoder_all_logits_and_kv(small):
    cfg, ck, eng = small
    g = torch.Generator().manual_seed(6)
    S = 201
    emb = (torch.randn(S, 4096, generator=g) * 0.5).to(torch.bfloat16)
    kv_ref = []
    ref = om.decoder_forward(ck, cfg, emb.float(), torch.arange(S), kv_out=kv_ref)
    logits, kv = eng.decoder(emb.cuda().clone(), torch.arange(S), [0, S], "all", torch.float32, want_kv=True)
    e = rel_err(logits, ref)
    print(f"\n[parity] decoder(2 layers) logits rel err {e:.4f}  max-abs {float((logits.cpu() - ref).abs().max()):.4f}")
    assert e < 3e-2
    # KV cache = K after RoPE, V, per layer
    for l in range(cfg.dec.layers):
        assert rel_err(kv[l, 0].view(S, 8, 128), kv_ref[l][0]) < 2e-2
        assert rel_err(kv[l, 1].view(S, 8, 128), kv_ref[l][1]) < 2e-2
    last, _ = eng.decoder(emb.cuda().clone(), torch.arange(S), [0, S], "last")
    assert rel_err(last, ref[-1:]) < 3e-2


def test_end_to_end_prefill_and_packing(small):
    cfg, ck, eng = small
    pix, ids = synth_inputs(cfg, n_crops=2, n_text=12)
    ref = om.prefill_logits(ck, cfg, ids, pix.to(torch.bfloat16).float())[0]
    logits, _, cu = eng.prefill([(ids[0], pix.cuda())], "all")
    assert cu == [0, 12 + 2 * 169]
    e = rel_err(logits, ref)
    print(f"\n[parity] e2e reduced logits rel err {e:.4f}  max-abs {float((logits.cpu() - ref).abs().max()):.4f}")
    assert e < 3e-2
    assert torch.equal(logits.argmax(-1).cpu()[-1], ref.argmax(-1)[-1])
    # two independent requests packed into one call == each alone (different lengths -> varlen attention path)
    pix2, ids2 = synth_inputs(cfg, n_crops=1, n_text=20, seed=7)
    ref2 = om.prefill_logits(ck, cfg, ids2, pix2.to(torch.bfloat16).float())[0]
    both, _, cu2 = eng.prefill([(ids[0], pix.cuda()), (ids2[0], pix2.cuda())], "all")
    assert cu2 == [0, 350, 350 + 20 + 169]
    assert rel_err(both[:350], ref) < 3e-2 and rel_err(both[350:], ref2) < 3e-2
    # text-only request
    t_ids = ids2[0][ids2[0] != cfg.image_token_index]
    ref3 = om.decoder_forward(ck, cfg, ck.f32("language_model.model.embed_tokens.weight")[t_ids], torch.arange(t_ids.numel()))
    l3, _, _ = eng.prefill([(t_ids, None)], "all")
    assert rel_err(l3, ref3) < 3e-2


def test_image_token_count_mismatch_raises(small):
    cfg, ck, eng = small
    pix, ids = synth_inputs(cfg, n_crops=2, n_text=6)
    with pytest.raises(ValueError, match="number of image tokens"):
        eng.prefill([(ids[0], pix[:1].cuda())])


def test_determinism_and_causality(small):
    cfg, ck, eng = small
    pix, ids = synth_inputs(cfg, n_crops=1, n_text=40)
    a, _, _ = eng.prefill([(ids[0], pix.cuda())], "all")
    b, _, _ = eng.prefill([(ids[0], pix.cuda())], "all")
    assert torch.equal(a, b)  # same launch configuration -> bit-identical
    ids_c = ids.clone()
    ids_c[0, -1] = (ids_c[0, -1] + 1) % 1000
    c, _, _ = eng.prefill([(ids_c[0], pix.cuda())], "all")
    assert torch.equal(a[:-1], c[:-1]) and not torch.equal(a[-1], c[-1])  # causal: only the last row may change


@pytest.mark.timeout(1500)
def test_full_depth_cfg1_parity(seeded_full_engine):
    """BASELINE config 1 shape at FULL depth (27 ViT + 32 decoder layers): 1 crop, 8 question + 24 frame ids ->
    S = 201; logits of every position vs the fp32 oracle."""
    cfg, ck, eng = seeded_full_engine
    pix, ids = synth_inputs(cfg, n_crops=1, n_text=32)
    assert ids.shape[1] + 168 == 201
    stages = {}
    torch.set_num_threads(max(1, torch.get_num_threads()))
    ref = om.prefill_logits(ck, cfg, ids, pix.to(torch.bfloat16).float(), stages=stages)[0]
    feats = eng.image_features(pix.cuda())
    e_img = rel_err(feats, stages["image_features"])
    logits, _, _ = eng.prefill([(ids[0], pix.cuda())], "all")
    e = rel_err(logits, ref)
    mad = float((logits.cpu() - ref).abs().max())
    top = float((logits.argmax(-1).cpu() == ref.argmax(-1)).float().mean())
    print(f"\n[parity] FULL depth cfg1: image_features rel err {e_img:.4f}; logits rel err {e:.4f}, max-abs {mad:.4f}, "
          f"ref absmax {float(ref.abs().max()):.3f}, greedy-token agreement {top:.3f}")
    assert e_img < 4e-2
    assert e < 6e-2
    assert top > 0.9


def test_fused_norm_layer_loops_match_the_standalone_norm_kernels(small):
    """lp_model_set_fused_norm(1) (default: LayerNorm / RMSNorm folded into the GEMM epilogues, RoPE in the QKV epilogue) against
    the standalone-kernel sequencing on the same weights: both within the oracle tolerance and close to each other; the KV
    cache path (RoPE applied by the append kernel) agrees with the cache-less path."""
    from leopard_b200 import _lib
    cfg, ck, eng = small
    pix, ids = synth_inputs(cfg, n_crops=2, n_text=24)
    ref = om.prefill_logits(ck, cfg, ids, pix.to(torch.bfloat16).float())[0]
    L = _lib.lib()
    try:
        assert L.lp_model_set_fused_norm(1) in (0, 1)
        n0 = L.lp_launch_count()
        fused, _, _ = eng.prefill([(ids[0], pix.cuda())], "all")
        n_fused = L.lp_launch_count() - n0
        with_kv, kv, _ = eng.prefill([(ids[0], pix.cuda())], "all", want_kv=True)
        L.lp_model_set_fused_norm(0)
        n0 = L.lp_launch_count()
        plain, _, _ = eng.prefill([(ids[0], pix.cuda())], "all")
        n_plain = L.lp_launch_count() - n0
        plain_kv, kv0, _ = eng.prefill([(ids[0], pix.cuda())], "all", want_kv=True)
    finally:
        L.lp_model_set_fused_norm(1)
    assert n_fused < n_plain                      # 2 norm launches per tower layer, 2 norms + RoPE per decoder layer are gone
    assert rel_err(fused, ref) < 3e-2 and rel_err(plain, ref) < 3e-2
    assert rel_err(fused, plain.cpu()) < 2e-2 and rel_err(with_kv, fused.cpu()) < 2e-2
    assert rel_err(kv.float(), kv0.float().cpu()) < 2e-2 and rel_err(with_kv, plain_kv.cpu()) < 2e-2
