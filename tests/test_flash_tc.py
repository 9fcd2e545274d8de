"""Prefill attention on tcgen05 (csrc/flash_tc.cu) through one-layer models, at the edges of its tiles: 128 query rows, 128 keys (64 at D = 256), a last page that was never
written to its end, cached prefixes; the oracle in f32."""
import numpy as np
import pytest

from crane_b200 import synth

pytestmark = pytest.mark.gpu


# split precision keeps 16 bits of every operand (2^-17 each): 3e-5 of the largest logit over a layer, four-fold; plain bf16 2^-9: 2e-2
@pytest.mark.parametrize("rows,past", [(2, 0), (63, 0), (64, 1), (65, 63), (127, 0), (128, 64), (129, 7), (300, 0), (37, 200), (513, 130), (70, 600), (16, 640)])
@pytest.mark.parametrize("precision", ["split", "bf16"])
def test_dense_prefill(rows, past, precision):
    import crane_b200
    from oracle.qwen3 import Qwen3Oracle
    cfg = dict(synth.TINY_QWEN3_UNTIED, num_hidden_layers=1)
    w = dict(synth.synth_checkpoint(cfg))
    m = crane_b200.Qwen3Model(cfg, max_seq_len=704, precision=precision)
    m.load_checkpoint(w.items())
    orc = Qwen3Oracle(cfg, w)
    ids = synth.synth_token_ids(past + rows, cfg["vocab_size"], f"ftc-{rows}-{past}")
    if past:
        orc.forward(ids[:past], 0)
        m.forward_step(ids[:past], 0)
    ref, got = orc.forward(ids[past:], past).numpy(), m.forward_step(ids[past:], past)
    assert np.abs(got - ref).max() <= (1.2e-4 if precision == "split" else 2e-2) * np.abs(ref).max()
    m.close()


@pytest.mark.parametrize("rows,past", [(70, 0), (129, 90), (260, 0)])
def test_hybrid_prefill(rows, past):
    """D = 256, output gate applied behind it."""
    import crane_b200
    from oracle.qwen3_5 import Qwen3_5Oracle
    cfg = synth.TINY_QWEN3_5
    w = dict(synth.synth_checkpoint(cfg))
    m = crane_b200.Qwen3_5Model(cfg, max_seq_len=512)
    m.load_checkpoint(w.items())
    orc = Qwen3_5Oracle(cfg, w)
    ids = synth.synth_token_ids(past + rows, cfg["vocab_size"], f"ftch-{rows}")
    if past:
        orc.forward(ids[:past], 0)
        m.forward_step(ids[:past], 0)
    ref, got = orc.forward(ids[past:], past).numpy(), m.forward_step(ids[past:], past)
    assert np.abs(got - ref).max() <= 1.2e-4 * np.abs(ref).max()
    m.close()


@pytest.mark.parametrize("grids", [[(1, 2, 2)], [(1, 8, 18)], [(1, 16, 16), (1, 4, 6), (2, 6, 10)]])
def test_vision(grids):
    """Strided keys, no mask, several images in one call."""
    import crane_b200
    from oracle.qwen3_vl import VisionOracle
    cfg = synth.TINY_QWEN3_VL
    w = dict(synth.synth_checkpoint(cfg))
    m = crane_b200.Qwen3VLModel(cfg, max_seq_len=64)
    m.load_checkpoint(w.items())
    n = sum(t * h * x for t, h, x in grids)
    pv = np.random.default_rng(n).uniform(-1, 1, (n, 1536)).astype(np.float32)
    ref, deep = VisionOracle(cfg["vision_config"], w).forward(pv, grids)
    got, ds = m.encode_images(pv, grids, want_deepstack=3)
    for g, r in [(got, ref)] + list(zip(ds, deep)):
        assert np.abs(g - r.numpy()).max() <= 1.2e-4 * np.abs(r.numpy()).max()
    m.close()


@pytest.mark.parametrize("grid", [(1, 2, 2), (1, 8, 18), (1, 20, 20), (1, 16, 24)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_image_beside_one_that_is_not_finite(grid, bad):
    """The keys behind an image's last one are the next image's: whatever it holds, the first image's features are the same bits."""
    import crane_b200
    cfg = synth.TINY_QWEN3_VL
    m = crane_b200.Qwen3VLModel(cfg, max_seq_len=64)
    m.load_checkpoint(synth.synth_checkpoint(cfg))
    grids = [grid, (1, 12, 14)]
    n = grid[1] * grid[2]
    pv = np.random.default_rng(n).uniform(-1, 1, (n + 168, 1536)).astype(np.float32)
    clean, clean_ds = m.encode_images(pv, grids, want_deepstack=3)
    pv[n:, ::7] = bad
    got, ds = m.encode_images(pv, grids, want_deepstack=3)
    assert not np.isfinite(got[n // 4:]).any()
    for g, c in [(got, clean)] + list(zip(ds, clean_ds)):
        assert np.array_equal(g[: n // 4], c[: n // 4])
    m.close()


# the lines between the two attention kernels (flash_few_keys): 160 keys at D = 128 in split precision, 8 in plain bf16
@pytest.mark.parametrize("rows,past", [(95, 0), (96, 0), (97, 0), (16, 80), (16, 81), (160, 0), (161, 0), (2, 158), (2, 159), (40, 57), (8, 0), (9, 0), (2, 6), (2, 7)])
@pytest.mark.parametrize("precision", ["split", "bf16"])
def test_few_keys(rows, past, precision):
    test_dense_prefill(rows, past, precision)


@pytest.mark.parametrize("rows,past", [(31, 0), (32, 0), (33, 0), (2, 30), (8, 0), (9, 0), (2, 6), (2, 7)])
def test_few_keys_hybrid(rows, past):
    """... 8 at D = 256"""
    test_hybrid_prefill(rows, past)


@pytest.mark.parametrize("grids", [[(1, 16, 20)], [(1, 18, 18)], [(1, 10, 16)] * 2, [(1, 2, 2), (1, 18, 20)], [(1, 18, 22)], [(1, 8, 8)] * 80])
def test_few_keys_vision(grids):
    """... 360 at D = 64 without a mask, as long as the 64-row tiles of all images fit the chip (eighty of them with two heads do not)"""
    test_vision(grids)


# a cluster of CTAs shares the keys of a query tile: one of them has none (the first query tile has one key tile), and clusters of eight
@pytest.mark.parametrize("family,rows,past", [("dense", 700, 0), ("dense", 70, 2100), ("hybrid", 90, 1100)])
def test_shared_keys(family, rows, past):
    import crane_b200
    from oracle.qwen3 import Qwen3Oracle
    from oracle.qwen3_5 import Qwen3_5Oracle
    cfg = dict(synth.TINY_QWEN3_UNTIED, num_hidden_layers=1) if family == "dense" else synth.TINY_QWEN3_5
    w = dict(synth.synth_checkpoint(cfg))
    m = (crane_b200.Qwen3Model if family == "dense" else crane_b200.Qwen3_5Model)(cfg, max_seq_len=past + rows + 64)
    m.load_checkpoint(w.items())
    orc = (Qwen3Oracle if family == "dense" else Qwen3_5Oracle)(cfg, w)
    ids = synth.synth_token_ids(past + rows, cfg["vocab_size"], f"ftsk-{rows}-{past}")
    if past:
        orc.forward(ids[:past], 0)
        m.forward_step(ids[:past], 0)
    ref, got = orc.forward(ids[past:], past).numpy(), m.forward_step(ids[past:], past)
    assert np.abs(got - ref).max() <= 1.2e-4 * np.abs(ref).max()
    m.close()


def modified(which):
    """Layer lists whose attention has 128-wide heads and, between them, every score modifier and mask; windows at the edges of the 128-key tiles."""
    import test_gavipel as g
    import test_puzonex as p
    import test_suvapel as s
    wide = dict(width=256, vocab=300)
    if which == "window, gate, sink":
        return g, g.config([g.layer(g.mixer(heads=4, kv_heads=2, dim=128, vdim=128, scale=0.08, window=128, rot_dims=64), None),
                            g.layer(g.mixer(heads=4, kv_heads=2, dim=128, vdim=128, scale=0.08, window=0, rot_dims=64), None)], loop=(0, 1, 1), **wide)
    if which == "cap, distance":
        return p, p.config([p.layer(p.attention(heads=4, kv_heads=2, dim=128, vdim=128, window=129, scale=0.09), None),
                            p.layer(p.attention(heads=4, kv_heads=4, dim=128, vdim=128, window=0, scale=0.09), None)], **wide)
    if which == "cap, table":
        return p, p.config([p.layer(p.parallel(heads=2, kv_heads=1, dim=128, window=150, scale=0.09, rheads=2, rdim=64, rvdim=64), None)], **wide)
    return s, s.config([s.layer(s.parallel(heads=4, kv_heads=2, dim=128, vdim=128, size=127, keep=130, scale=0.09, right=s.rule(heads=2, kv_heads=1, dim=64, vdim=64, conv=3)), None)], side=40, **wide)


@pytest.mark.parametrize("which", ["window, gate, sink", "cap, distance", "cap, table", "window, kept first keys"])
def test_modifiers_in_a_ragged_batch(which):
    """Unequal prompts side by side, then their next portions, in 128-row tiles: every row against the oracle in f64."""
    mod, cfg = modified(which)
    m, w = mod.make(cfg, 21, precision="split", max_tokens=2048)
    lens, more = (400, 129, 257), (70, 128, 3)
    slots = [0, m.seq_create(), m.seq_create()]
    ids = [mod.tokens(a + b, cfg["vocab"], 30 + i) for i, (a, b) in enumerate(zip(lens, more))]
    first = m.step_batch([(s, t[:a], mod.all_rows(a)) for s, t, a in zip(slots, ids, lens)])
    second = m.step_batch([(s, t[a:], mod.all_rows(b)) for s, t, a, b in zip(slots, ids, lens, more)])
    fa, fb = np.cumsum((0,) + lens), np.cumsum((0,) + more)
    for i in range(3):
        got = np.concatenate([first[fa[i]: fa[i + 1]], second[fb[i]: fb[i + 1]]])
        assert mod.rel(got, mod.oracle_logits(cfg, w, ids[i])) < mod.SPLIT_TOL
    m.close()
