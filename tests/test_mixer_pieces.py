"""Retention and latent attention where rows are whole 16-byte pieces (the kernels read four columns at a time) and where they are not, with few
(request, head) pairs for the chip and with many: prompts of several chunks, portions, then token by token, against the plain implementation in oracle/seqlm.py."""
import pytest

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
