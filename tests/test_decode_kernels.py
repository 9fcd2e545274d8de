"""GPU (-m gpu): the decode chain where its splits can go wrong: contexts around the turns, tiles and splits of the attention kernel, query groups of every
width a launch narrows or keeps, matrices whose rows and column chunks do not fill the GEMV's units and slices, groups of 1, 2 and 4 sequences, and forks
of more segments than one launch copies.

Tolerance: cached keys and values carry two bf16 planes (2^-17 of each), everything else 24 bits; three layers, logits relative to the largest: 1e-4
(measured 1e-5)."""
import numpy as np
import pytest

from conftest import rel_err
import crane_b200
from crane_b200 import synth
from oracle.qwen3 import Qwen3Oracle

pytestmark = pytest.mark.gpu
TOL = 1e-4


def _model(cfg, **kw):
    w = dict(synth.synth_checkpoint(cfg))
    m = crane_b200.Qwen3Model(cfg, device=0, **kw)
    m.load_checkpoint(w.items())
    return m, w


@pytest.mark.parametrize("heads", [(4, 2), (8, 2), (6, 2), (10, 2), (32, 8), (2, 2)], ids=lambda h: f"{h[0]}x{h[1]}")
@pytest.mark.parametrize("past", [1, 2, 16, 17, 33, 129, 260])
def test_one_sequence(heads, past):
    # widths: 256 .. 1024 columns of the o projection (1 to 16 chunks of 256), 3 and 9 chunks of the MLP
    cfg = dict(synth.TINY_QWEN3, num_attention_heads=heads[0], num_key_value_heads=heads[1], intermediate_size=768 if past % 2 else 2304, num_hidden_layers=2)
    m, w = _model(cfg, max_seq_len=320)
    ids = synth.synth_token_ids(past + 4, cfg["vocab_size"], f"d{past}")
    orc = Qwen3Oracle(cfg, w)
    assert rel_err(m.forward_step(ids[:past], 0), orc.forward(ids[:past], 0).numpy()) < TOL
    for i in range(past, past + 4):
        assert rel_err(m.forward_step(ids[i:i + 1], i), orc.forward(ids[i:i + 1], i).numpy()) < TOL
    m.close()


@pytest.mark.parametrize("n", [2, 4])
def test_groups_of_sequences(n):
    """Groups that go through the GEMVs (two sequences, and what a batch leaves over) against one sequence at a time."""
    cfg = dict(synth.TINY_QWEN3, intermediate_size=1280)
    m, w = _model(cfg, max_seq_len=320, max_batch=n)
    lens = [3, 130, 17, 66][:n]
    slots = [0] + [m.seq_create() for _ in range(n - 1)]
    ids = [synth.synth_token_ids(k + 1, cfg["vocab_size"], f"g{k}") for k in lens]
    for s, k, t in zip(slots, lens, ids):
        m.seq_select(s)
        m.forward_step(t[:k], 0)
    _, got = m.decode_batch(slots, [int(t[-1]) for t in ids], 1, want_logits=True)
    for row, k, t in zip(got, lens, ids):
        orc = Qwen3Oracle(cfg, w)
        orc.forward(t[:k], 0)
        assert rel_err(row, orc.forward(t[k:], k).numpy()) < TOL
    m.close()


@pytest.mark.parametrize("layers", [16, 17, 33])
def test_fork_copies_every_segment(layers):
    """Four segments per layer: 64, 68 and 132 of them."""
    cfg = dict(synth.TINY_QWEN3, num_hidden_layers=layers)
    m, _ = _model(cfg, max_seq_len=256, max_batch=2)
    ids = synth.synth_token_ids(72, cfg["vocab_size"], "fork")
    m.forward_step(ids[:70], 0)
    s = m.seq_fork(0)
    want = [m.forward_step(ids[i:i + 1], i) for i in (70, 71)]
    m.seq_select(s)
    assert all(np.array_equal(a, m.forward_step(ids[i:i + 1], i)) for a, i in zip(want, (70, 71)))
    m.close()
