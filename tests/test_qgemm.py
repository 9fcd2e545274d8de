"""Quantised linears on the tensor cores (csrc/qgemm.cu) against the oracle's integer dots, at the edges of the kernel's tiles: 16 / 32 / 64 /
128 activation rows, 128 weight rows, one and more super-blocks, work shared by several blocks and not."""
import os
import subprocess
import sys

import numpy as np
import pytest

from oracle import ggml_quant as gq

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# The integer dots are exact on both sides; what differs is the order of the f32 additions over K / 256 (K-quants) or K / 32 (Q8_0) block terms
# of either sign: under sqrt(blocks) * 2^-24 of the row's largest term, 2e-6 of the largest output at K = 4096.  Bound: five times that.
BAR = 1e-5


def blocks(rng, n, k, qt):
    w = rng.standard_normal((n, k)).astype(np.float32) * k ** -0.5
    w[:, :3] *= 6.0                                    # a few blocks with large scales
    return gq.quantize(w, qt)


@pytest.mark.parametrize("qt", ["Q4_K", "Q6_K", "Q8_0"])
@pytest.mark.parametrize("m,n,k", [(5, 128, 256), (16, 130, 512), (17, 384, 768), (32, 700, 1024), (33, 127, 256), (64, 128, 4096), (65, 129, 512),
                                   (128, 512, 256), (129, 640, 2048), (300, 1024, 512), (7, 2000, 2560)])
def test_rows_against_integer_dots(qt, m, n, k):
    import crane_b200
    rng = np.random.default_rng(m * 1000 + n + k)
    raw = blocks(rng, n, k, qt)
    x = rng.standard_normal((m, k)).astype(np.float32)
    x[0] = 0.0                                          # an all-zero row: codes and scales zero
    x[1, 5] = 400.0                                     # one value takes a whole block's range
    want = gq.qmatmul(x, raw, qt)
    got = crane_b200.op_qlinear(x, raw, gq.GGML_TYPE_ID[qt], n)
    assert np.abs(got - want).max() <= BAR * np.abs(want).max()
    assert not got[0].any()
    again = crane_b200.op_qlinear(x, raw, gq.GGML_TYPE_ID[qt], n)
    assert np.array_equal(got, again)                   # contributor order, whoever came last


@pytest.mark.parametrize("qt", ["Q4_K", "Q6_K"])
@pytest.mark.parametrize("m", [5, 40, 130])
def test_sums_above_24_bits(qt, m):
    """Scales, weights and activations of one sign near the ends of their ranges: a super-block's sum passes 2^24 (Q4_K up to 3.1e7, Q6_K 1.3e8 in the units it is
    summed in), where the accumulator rounds instead of counting.  Sixteen to 32 partial sums of at most a unit in the last place (2^-23) each, the f32
    terms beside them: under 40 * 2^-23 of a result that has no cancellation."""
    import crane_b200
    rng = np.random.default_rng(m)
    n, k = 130, 512
    nb = k // 256
    half = np.frombuffer(np.float16(0.01).tobytes(), np.uint8)
    if qt == "Q4_K":
        sc = rng.integers(48, 64, (n, nb, 8)).astype(np.uint8)
        head = np.concatenate([sc[..., :4] | ((sc[..., 4:] >> 4) << 6), np.zeros((n, nb, 4), np.uint8), sc[..., 4:] & 15], -1)
        qs = (rng.integers(11, 16, (n, nb, 128)) | (rng.integers(11, 16, (n, nb, 128)) << 4)).astype(np.uint8)
        raw = np.concatenate([np.broadcast_to(half, (n, nb, 2)), np.zeros((n, nb, 2), np.uint8), head, qs], -1)
    else:
        raw = np.concatenate([rng.integers(0, 256, (n, nb, 128)).astype(np.uint8), np.full((n, nb, 64), 255, np.uint8), rng.integers(96, 128, (n, nb, 16)).astype(np.uint8),
                              np.broadcast_to(half, (n, nb, 2))], -1)
    raw = np.ascontiguousarray(raw.reshape(n, -1))
    x = rng.uniform(0.8, 1.0, (m, k)).astype(np.float32)
    want = gq.qmatmul(x, raw, qt)
    got = crane_b200.op_qlinear(x, raw, gq.GGML_TYPE_ID[qt], n)
    assert (np.abs(got - want) <= 40 * 2.0 ** -23 * np.abs(want)).all()


@pytest.mark.parametrize("recipe", [("Q8_0", "Q8_0"), ("Q4_K", "Q8_0"), ("Q4_K", "Q6_K")])
def test_prompts_at_the_line(recipe):
    """Prompts of 4 to 8 tokens, where GEMVs and tensor-core linears meet (7 rows for Q8_0, 5 for K-quants), with value projections of another type than the
    queries': each row count against the oracle; a code on the border of two moves a one-layer model's logits by up to 1e-2."""
    import crane_b200
    from crane_b200 import synth
    from oracle.qwen3 import Qwen3Oracle
    cfg = dict(synth.TINY_QWEN3_UNTIED, num_hidden_layers=1)
    m = crane_b200.Qwen3Model(cfg, max_seq_len=64)
    w, qd = {}, {}
    for name, t in synth.synth_checkpoint(cfg):
        if "proj" in name or name == "lm_head.weight":
            qt = recipe["v_proj" in name or "down" in name]
            raw = gq.quantize(t, qt)
            m.load_tensor_ggml(name, gq.GGML_TYPE_ID[qt], t.shape, raw)
            w[name], qd[name] = gq.dequantize(raw, qt, t.shape[1]), (raw, qt)
        else:
            m.load_tensor(name, t)
            w[name] = t
    m.finalize()
    orc = Qwen3Oracle(cfg, w, quantised=qd)
    err = []
    for rows in (4, 5, 6, 7, 8):
        for seed in range(3):
            ids = synth.synth_token_ids(rows, cfg["vocab_size"], f"ql{seed}")
            orc.clear_kv_cache()
            m.clear_kv_cache()
            want = orc.forward(ids, 0).numpy().ravel()
            err.append(np.abs(m.forward_step(ids, 0).ravel() - want).max() / np.abs(want).max())
    print(recipe, " ".join(f"{e:.1e}" for e in err))
    assert max(err) < 3e-2 and min(err) < 1e-4
    m.close()


@pytest.mark.parametrize("qt", ["Q4_K", "Q6_K"])
@pytest.mark.parametrize("m,n,k", [(200, 12288, 512), (257, 12160, 512)])
def test_wide_row_tiles(qt, m, n, k):
    """Several tiles of 64 rows for every block (the plan's at 148 SMs)."""
    assert rows_of(qt, m, n, k) == 64
    test_rows_against_integer_dots(qt, m, n, k)


def rows_of(qt, m, n, k):
    """Activation rows of the tiles that the plan takes."""
    import crane_b200
    return crane_b200.load_library().crane_b200_debug_qgemm_rows(gq.GGML_TYPE_ID[qt], m, n, k)


# one row of a second half, a half less one, whole halves and tiles, one row of a third half and tile; weight rows that 128 does not divide; one super-block and many, a block's
# own and shared
EDGES = [(5, 128, 256), (65, 130, 512), (64, 384, 768), (127, 700, 1024), (128, 256, 4096), (129, 130, 2560), (191, 640, 512), (193, 2080, 1024), (256, 128, 2048), (257, 1000, 256)]


def edges(qt, height):
    """At tiles of `height` rows, pinned: every edge against the integer dots, the residual and the gated epilogue beside the plain one."""
    import ctypes
    import crane_b200
    fn = crane_b200.load_library().crane_b200_debug_qlinear
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    for m, n, k in EDGES:
        m = max(m, 7)                                       # (fewer rows are GEMVs)
        assert rows_of(qt, m, n, k) == height
        test_rows_against_integer_dots(qt, m, n, k)
        rng = np.random.default_rng(m + n + k)
        raw, x = blocks(rng, n, k, qt), rng.standard_normal((m, k)).astype(np.float32)
        want = gq.qmatmul(x, raw, qt)
        for epi, y in ((1, rng.standard_normal((m, n)).astype(np.float32)), (2, np.full((m, n // 2), 9.0, np.float32))):
            if epi == 1:
                ref = y + want.astype(np.float64)
            else:
                g, u = want[:, 0::2].astype(np.float64), want[:, 1::2].astype(np.float64)
                ref = g / (1.0 + np.exp(-g)) * u
            # (the gated unit: 1.1 |u| of a gate's error and |g| of an up's, both below 4 deviations here; expf and the division add a few units of 2^-24)
            bar = BAR * (np.abs(ref).max() if epi == 1 else 2.1 * np.abs(want).max() ** 2)
            rc = fn(0, ptr(x), ctypes.c_size_t(m), ctypes.c_size_t(k), ptr(raw), ctypes.c_size_t(raw.nbytes), gq.GGML_TYPE_ID[qt], ctypes.c_size_t(n), epi, ptr(y))
            assert rc == 0 and np.abs(y - ref).max() <= bar, (m, n, k, epi)


@pytest.mark.parametrize("qt,height", [(q, h) for q in ("Q4_K", "Q6_K", "Q8_0") for h in (16, 32, 64, 128) if q != "Q8_0" or h < 128])
def test_edges_of_every_tile(qt, height):
    """In a process of its own: the pin is read once."""
    code = "import sys; sys.path[:0] = [%r, %r]; import test_qgemm as t; t.edges(%r, %d)" % (ROOT, os.path.join(ROOT, "tests"), qt, height)
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, CRANE_B200_QGEMM_ROWS=str(height)), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("qt", ["Q4_K", "Q6_K", "Q8_0"])
@pytest.mark.parametrize("k", [256, 1280, 2048, 4096])
def test_codes_of_a_row_are_its_own(qt, k):
    """A row behind a folded-in norm has the same 8-bit codes alone, in groups of two and four, and in a prompt.  Every value lies on the border of two codes, so a
    last bit of 1 / rms decides for many at once; one code the other way moves a result by (1 / 128) / (0.58 sqrt(k)) of its size, 2e-4 at k = 4096, while
    the order of the additions alone keeps within BAR."""
    import crane_b200
    rng = np.random.default_rng(k + len(qt))
    top, blk = (127.0, 32) if qt == "Q8_0" else (128.0, 256)
    x = (rng.integers(0, int(top) - 1, (12, k)) + 0.5).astype(np.float32) * rng.choice([-1.0, 1.0], (12, k)).astype(np.float32)
    x[:, ::blk] = top
    x *= rng.uniform(0.1, 1.0, (12, 1)).astype(np.float32)      # (so that squares round)
    raw = blocks(rng, 384, k, qt)
    run = lambda rows: crane_b200.op_qlinear(rows, raw, gq.GGML_TYPE_ID[qt], 384, norm_w=np.ones(k, np.float32))  # noqa: E731
    prompt = run(x)                                     # 12 rows: tensor cores
    for n in (1, 2, 4):
        got = np.concatenate([run(x[i:i + n]) for i in range(0, 12, n)])
        assert (np.abs(got - prompt).max(1) <= BAR * np.abs(prompt).max(1)).all(), n


@pytest.mark.parametrize("qt,m,n", [("Q4_K", 1100, 8192), ("Q6_K", 700, 8192), ("Q6_K", 641, 8192)])
def test_tiles_of_128_rows(qt, m, n):
    """Enough work that the plan takes tiles of 128 activation rows (a ragged last one among them): the same rows in calls of 64, which do not.  Only the division along K, the
    order of the f32 additions, differs; the first rows and the last against the oracle."""
    import crane_b200
    assert rows_of(qt, m, n, 4096) == 128 and rows_of(qt, 64, n, 4096) == 64
    rng = np.random.default_rng(m)
    few = blocks(rng, 512, 4096, qt)
    raw = np.tile(few, (n // 512, 1))
    x = rng.standard_normal((m, 4096)).astype(np.float32)
    got = crane_b200.op_qlinear(x, raw, gq.GGML_TYPE_ID[qt], n)
    for r in [*range(0, m - 64, 64), m - 64]:
        part = crane_b200.op_qlinear(x[r: r + 64], raw, gq.GGML_TYPE_ID[qt], n)
        assert np.abs(got[r: r + 64] - part).max() <= BAR * np.abs(part).max()
    some = [0, 1, 63, 64, 127, 128, m - 2, m - 1]
    want = np.tile(gq.qmatmul(x[some], few, qt), (1, n // 512))
    assert np.abs(got[some] - want).max() <= BAR * np.abs(want).max()
    assert np.array_equal(got, crane_b200.op_qlinear(x, raw, gq.GGML_TYPE_ID[qt], n))


@pytest.mark.parametrize("types", [("Q4_K", "Q4_K", "Q6_K"), ("Q6_K", "Q4_K", "Q4_K"), ("Q8_0", "Q8_0", "Q8_0"), ("Q4_K", "Q8_0", "Q6_K")])
@pytest.mark.parametrize("hidden", [512, 2560])
def test_q_k_v_side_by_side(types, hidden):
    """q, k and v that share a launch (or two, or none: 2560 x 2560 takes all CTAs) give the bits each gives by itself."""
    import ctypes
    import crane_b200
    from crane_b200 import synth
    cfg = dict(synth.TINY_QWEN3_UNTIED, hidden_size=hidden, intermediate_size=256, num_attention_heads=hidden // 128, num_key_value_heads=hidden // 256, head_dim=128, num_hidden_layers=1,
               vocab_size=300)
    rng = np.random.default_rng(hidden)
    m = crane_b200.Qwen3Model(cfg, max_seq_len=256)
    raws, norm, table = {}, None, None
    for name, shape, kind in synth.text_tensor_specs(cfg):
        short = name.split(".")[-2]
        qt = dict(zip(("q_proj", "k_proj", "v_proj"), types)).get(short, "Q8_0") if "proj" in name else None
        if qt:
            raw = blocks(rng, shape[0], shape[1], qt)
            raws[short] = (raw, qt, shape[0])
            m.load_tensor_ggml(name, gq.GGML_TYPE_ID[qt], shape, raw)
        else:
            bits = synth.f32_to_bf16_bits(rng.standard_normal(shape, dtype=np.float32))
            value = (bits.astype(np.uint32) << 16).view(np.float32)
            norm, table = (value if name.endswith("input_layernorm.weight") else norm), (value if "embed" in name else table)
            m.load_tensor(name, bits)
    m.finalize()
    width = sum(raws[n][2] for n in ("q_proj", "k_proj", "v_proj"))
    for rows in (7, 16, 17, 33, 64, 65, 130):
        ids = rng.integers(0, 300, rows).astype(np.uint32)
        m.clear_kv_cache()
        m.forward_step(ids, 0)
        got = np.empty((rows, width), np.float32)
        assert m.lib.crane_b200_debug_peek(m.h, 1, got.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(got.size)) == 0
        want = np.concatenate([crane_b200.op_qlinear(table[ids], raws[n][0], gq.GGML_TYPE_ID[raws[n][1]], raws[n][2], norm_w=norm, eps=cfg["rms_norm_eps"])
                               for n in ("q_proj", "k_proj", "v_proj")], 1)
        assert np.array_equal(got, want), rows
    m.close()
