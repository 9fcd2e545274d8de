"""GPU (-m gpu): the decode chain where its splits can go wrong: contexts around the turns, tiles and splits of the attention kernel in both its forms, rings that
come round several times, query groups of every width a launch narrows or keeps, matrices whose rows and column chunks do not fill the GEMV's units and slices,
groups of 1, 2 and 4 sequences, and forks of more segments than one launch copies.

Tolerance: cached keys and values carry two bf16 planes (2^-17 of each), everything else 24 bits; three layers, logits relative to the largest: 1e-4
(measured 1e-5)."""
import numpy as np
import pytest

from conftest import rel_err
import crane_b200
from crane_b200 import synth
from oracle import ggml_quant as gq
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
    """Two sequences, which go through the GEMVs, and four, which share a pass over the tensor cores, each against the oracle."""
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


@pytest.mark.parametrize("n,kv_heads,dim,precision", [(20, 2, 128, "split"), (20, 2, 128, "bf16"), (20, 2, 256, "split"), (40, 4, 128, "split")],
                         ids=["128 split", "128 bf16", "256 split", "two splits"])
def test_rings_that_come_round(n, kv_heads, dim, precision):
    """More (sequence, KV head) pairs than the tile form takes: a warp's ring has six places of two tokens (one at D = 256), and comes round behind 96 (48) tokens of each
    of the four splits, or two of 160 pairs.  Contexts around once, twice and three times round, and around a turn, against each sequence alone in the tile form.
    In plain bf16 a new key or value whose sums came in another order may round to the neighbouring bf16, 2^-8 of it; the results average over such values: 2^-9."""
    tol = TOL if precision == "split" else 2.0 ** -9
    cfg = dict(synth.TINY_QWEN3, num_hidden_layers=2, head_dim=dim, num_key_value_heads=kv_heads, num_attention_heads=2 * kv_heads)
    m, _ = _model(cfg, max_seq_len=1216, max_batch=n, precision=precision)
    turn = (4 if n == 20 else 2) * (16 if dim == 128 else 8)          # tokens that all splits' warps take at once
    lens = [1, turn - 1, turn, turn + 1, 2 * turn + 1, 3 * turn] + [k * 6 * turn + d for k in (1, 2, 3) for d in (-1, 0, 1)]
    lens = [min(k, 1200) for k in lens] + [int(k) for k in np.random.default_rng(dim).integers(2, 1200, n - len(lens))]
    slots = [0] + [m.seq_create() for _ in range(n - 1)]
    ids = [synth.synth_token_ids(k + 2, cfg["vocab_size"], f"r{i}") for i, k in enumerate(lens)]
    want = []
    for s, k, t in zip(slots, lens, ids):
        m.seq_select(s)
        m.forward_step(t[:k], 0)
        want.append([m.forward_step(t[k + i:k + i + 1], k + i) for i in range(2)])
        m.set_kv_caches([], k)
    for i in range(2):
        _, got = m.decode_batch(slots, [int(t[k + i]) for k, t in zip(lens, ids)], 1, want_logits=True)
        for row, w, k in zip(got, want, lens):
            assert rel_err(row, w[i]) < tol, k
    m.close()


@pytest.mark.parametrize("cfg", [
    # 3, 5 and 6 column chunks in several slices; 9 and 18 rows a CTA, a head of 1003
    dict(hidden_size=768, intermediate_size=1280, num_attention_heads=6, num_hidden_layers=2, vocab_size=1003),
    # 4864 rows of 10240 columns: five slices would be the fastest, and take the shared memory that the folded-in norm needs for itself
    dict(hidden_size=10240, intermediate_size=256, num_attention_heads=34, num_hidden_layers=1, vocab_size=257)], ids=["odd", "wide"])
def test_four_sequences_through_the_gemv(cfg):
    """A quantised embedding sends groups of four, and with them every bf16 linear, past the tensor cores: the GEMV of four sequences, against the oracle."""
    cfg = dict(synth.TINY_QWEN3_UNTIED, **dict(cfg, num_key_value_heads=2))
    m = crane_b200.Qwen3Model(cfg, device=0, max_seq_len=160, max_batch=4)
    w = {}
    for name, shape, kind in synth.text_tensor_specs(cfg):
        rng = np.random.default_rng(len(w))
        t = rng.standard_normal((min(shape[0], 97),) + tuple(shape[1:]) if len(shape) > 1 else shape, dtype=np.float32)
        t = t * shape[1] ** -0.5 if kind == "linear" else t if kind == "embed" else 1 + 0.02 * t
        t = np.resize(t, shape).astype(np.float32)       # (97 rows again and again)
        if kind == "embed":
            raw = gq.quantize(t, "Q8_0")
            m.load_tensor_ggml(name, gq.GGML_TYPE_ID["Q8_0"], shape, raw)
            w[name] = gq.dequantize(raw, "Q8_0", shape[1])
        else:
            bits = synth.f32_to_bf16_bits(t)
            m.load_tensor(name, bits)
            w[name] = synth.bf16_bits_to_f32(bits)
    m.finalize()
    lens = [3, 130, 17, 66]
    slots = [0] + [m.seq_create() for _ in range(3)]
    ids = [synth.synth_token_ids(k + 1, cfg["vocab_size"], f"q{k}") for k in lens]
    for s, k, t in zip(slots, lens, ids):
        m.seq_select(s)
        m.forward_step(t[:k], 0)
    _, got = m.decode_batch(slots, [int(t[-1]) for t in ids], 1, want_logits=True)
    orc = Qwen3Oracle(cfg, w)
    for row, k, t in zip(got, lens, ids):
        orc.clear_kv_cache()
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
