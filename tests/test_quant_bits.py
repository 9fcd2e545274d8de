"""GPU (-m gpu): logits of quantised models, bit for bit.

A quantised linear rounds its input to 8-bit codes.  A value on the border of two goes the other way when one addition ahead of it is done in another order, and the
logits move by up to 1e-2 of their size where f32 sums alone would move them by 1e-6.  So the order of every sum ahead of the codes -- the rows' 1 / rms, the sums of
q, k and v wherever their launches end, decode attention over its tokens -- is part of what a quantised model answers, and these checksums hold it: they were
recorded with one launch per linear and attention token after token.  A change that moves one has to say why the new order is the better one."""
import zlib

import numpy as np
import pytest

import crane_b200
from crane_b200 import synth
from oracle import ggml_quant as gq

pytestmark = pytest.mark.gpu

RECIPES = {"q8_0": ("Q8_0", "Q8_0"), "q4_k_m": ("Q4_K", "Q6_K")}       # the second: v, down and the head
# 4096 columns: more than one tile of super-blocks per row, and a q, k, v of 4096 rows whose work no 148 CTAs share evenly
CFG = dict(synth.TINY_QWEN3_UNTIED, hidden_size=4096, intermediate_size=1024, num_attention_heads=16, num_key_value_heads=8, head_dim=128, num_hidden_layers=2, vocab_size=512)


@pytest.fixture(scope="module", params=sorted(RECIPES))
def model(request):
    m = crane_b200.Qwen3Model(CFG, max_seq_len=320, max_batch=24)
    for name, shape, kind in synth.text_tensor_specs(CFG):
        rng = np.random.default_rng(zlib.crc32(name.encode()))
        if "proj" in name or name == "lm_head.weight":
            qt = RECIPES[request.param][any(s in name for s in ("v_proj", "down", "lm_head"))]
            rows = gq.quantize(rng.standard_normal((64, shape[1]), dtype=np.float32) * np.float32(shape[1] ** -0.5), qt)
            m.load_tensor_ggml(name, gq.GGML_TYPE_ID[qt], shape, np.tile(rows, (shape[0] // 64, 1)))
        else:
            m.load_tensor(name, synth.f32_to_bf16_bits(rng.standard_normal(shape, dtype=np.float32) + (kind == "norm")))
    m.finalize()
    yield request.param, m
    m.close()


def _ids(n, seed):
    return np.random.default_rng(seed).integers(0, 512, n).astype(np.uint32)


def _prompt(m, rows):
    m.seq_select(0)
    m.clear_kv_cache()
    return [m.forward_step(_ids(rows, rows), 0)]


def _tokens(m, past):
    out = _prompt(m, past)
    return out + [m.forward_step(_ids(1, past + i), past + i) for i in range(4)]


def _batch(m, n, past):
    m.seq_select(0)
    m.clear_kv_cache()
    slots = [0] + [m.seq_create() for _ in range(n - 1)]
    for i, s in enumerate(slots):
        m.seq_select(s)
        m.forward_step(_ids(max(1, past * (i + 1) // n), i), 0)
    out = [m.decode_batch(slots, _ids(n, 100 + r), 1, want_logits=True)[1] for r in range(2)]
    for s in slots[1:]:
        m.seq_free(s)
    m.seq_select(0)
    return out


CASES = {
    "three rows": lambda m: _prompt(m, 3), "forty rows": lambda m: _prompt(m, 40),
    "token behind 4": lambda m: _tokens(m, 4), "token behind 300": lambda m: _tokens(m, 300),
    "pair": lambda m: _batch(m, 2, 12), "24 short": lambda m: _batch(m, 24, 12), "24 long": lambda m: _batch(m, 24, 300),
}
BITS = {
    "q8_0": {"three rows": 860423412, "forty rows": 2319047176, "token behind 4": 915047249, "token behind 300": 70435833, "pair": 2572308134, "24 short": 351940177, "24 long": 908247942},
    "q4_k_m": {"three rows": 2799229761, "forty rows": 133175824, "token behind 4": 3687851847, "token behind 300": 2366858767, "pair": 14193225, "24 short": 2683411286, "24 long": 151590533},
}


@pytest.mark.parametrize("case", list(CASES))
def test_logits_keep_their_bits(model, case):
    recipe, m = model
    crc = 0
    for x in CASES[case](m):
        assert np.isfinite(x).all()
        crc = zlib.crc32(np.ascontiguousarray(x), crc)
    assert crc == BITS[recipe][case]
