"""Which kernels a step of the layer-list language models takes as its number of rows changes, and what captured steps keep: against the
plain implementation (oracle/seqlm.py) or float64.  On the kernel sources under the CPU emulator and, marked gpu, on the native library."""
import pytest
import torch

from leopard_b200.seqlm import StepEntry
from oracle import seqlm as O
from seqlm_common import TOL, backend, emu_lib, make_engine, model, moe, rel_err, retention_layer  # noqa: F401  (fixtures)


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
