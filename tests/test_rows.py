"""Linears of few rows (csrc/gemm_rows.cu) and decode batches that share one pass over the weights, at the edges of their tiles."""
import numpy as np
import pytest

from crane_b200 import synth

pytestmark = pytest.mark.gpu


def planes(x):
    hi = synth.bf16_round(x)
    return hi, synth.bf16_round(x - hi)


# f32 accumulation over K terms of either sign: under sqrt(K) * 2^-24 of the largest sum (4e-6 at K = 4096), eight-fold; a bf16 output adds half a unit, 2^-9
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("m,n,k", [(1, 32, 64), (15, 96, 192), (16, 160, 256), (17, 128, 2048), (77, 4096, 320), (113, 2080, 1024), (128, 384, 4096)])
def test_few_rows(m, n, k, split):
    import crane_b200 as cb
    rng = np.random.default_rng(m * 7 + n + k)
    hi, lo = planes(rng.standard_normal((m, k)).astype(np.float32))
    w = synth.bf16_round((rng.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32))
    bias, init = rng.standard_normal(n).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
    a, al, wb = synth.f32_to_bf16_bits(hi), synth.f32_to_bf16_bits(lo) if split else None, synth.f32_to_bf16_bits(w)
    ref = (hi.astype(np.float64) + (lo.astype(np.float64) if split else 0.0)) @ w.astype(np.float64).T
    f32 = 8 * np.sqrt(k) * 2.0 ** -24

    def close(got, want, rel):
        assert np.abs(got - want).max() <= rel * np.abs(want).max()
    close(cb.op_gemm(a, wb, cb.EPI_STORE_F32, bias=bias, a_lo_bits=al), ref + bias, f32)
    out = cb.op_gemm(a, wb, cb.EPI_RESID_F32, out_init=init, a_lo_bits=al)
    close(out, ref + init, f32)
    assert np.array_equal(out, cb.op_gemm(a, wb, cb.EPI_RESID_F32, out_init=init, a_lo_bits=al))       # the same bits whoever came last
    g, u = ref[:, 0::2], ref[:, 1::2]
    close(synth.bf16_bits_to_f32(cb.op_gemm(a, wb, cb.EPI_SILU_MUL_BF16, a_lo_bits=al)), g / (1 + np.exp(-g)) * u, 2.0 ** -8)
    close(synth.bf16_bits_to_f32(cb.op_gemm(a, wb, cb.EPI_STORE_BF16, bias=bias, a_lo_bits=al)), ref + bias, 2.0 ** -8)


@pytest.mark.parametrize("n", [2, 3, 5, 16, 33, 64])
@pytest.mark.parametrize("kv", ["", "int8"])
def test_decode_batch_against_single_steps(n, kv):
    """Rounds of a batch against the same tokens fed to every sequence by itself; the two differ by rounding alone (24-bit activations on either side,
    KV rows rounded alike), 1e-5 over three layers; int8 pages turn that into a code here and there."""
    import crane_b200
    cfg = synth.TINY_QWEN3_UNTIED
    m = crane_b200.Qwen3Model(cfg, max_seq_len=128, max_batch=64, **({"kv_cache": kv} if kv else {}))
    m.load_checkpoint(synth.synth_checkpoint(cfg))
    slots = [0] + [m.seq_create() for _ in range(n - 1)]
    ids = {s: synth.synth_token_ids(5 + (7 * s) % 60, cfg["vocab_size"], f"rows-{s}") for s in slots}
    forced = [synth.synth_token_ids(n, cfg["vocab_size"], f"rows-forced-{r}") for r in range(3)]
    want = []
    for j, s in enumerate(slots):
        m.seq_select(s)
        m.forward_step(ids[s], 0)
        want.append([m.forward_step([int(f[j])], len(ids[s]) + r) for r, f in enumerate(forced)])
        m.set_kv_caches([], len(ids[s]))
    for r, f in enumerate(forced):
        toks, got = m.decode_batch(slots, f, 1, want_logits=True)
        ref = np.stack([w[r] for w in want])
        assert np.abs(got - ref).max() <= (2e-2 if kv else 3e-5) * np.abs(ref).max()
        assert np.array_equal(toks[:, 0], got.argmax(1))
    # greedy rounds on the device: what one round chooses is what the next one reads
    for s in slots:
        m.seq_select(s)
        m.set_kv_caches([], len(ids[s]))
    three, _ = m.decode_batch(slots, forced[0], 3)
    for s in slots:
        m.seq_select(s)
        m.set_kv_caches([], len(ids[s]))
    one = np.asarray(forced[0])
    for r in range(3):
        one = m.decode_batch(slots, one, 1)[0][:, 0]
        assert np.array_equal(one, three[:, r])
    m.close()


@pytest.mark.parametrize("recipe", ["Q4_K", "Q8_0"])
def test_quantised_decode_batch(recipe):
    """A batch of nine in one pass against the same in passes of up to four: the same codes and integer dots, so a one-layer model differs by f32 rounding
    until a code sits on a border (one in 128 of its block's largest value: 1e-2 of an output of K = 256 terms)."""
    import crane_b200
    from oracle import ggml_quant as gq
    cfg = dict(synth.TINY_QWEN3_UNTIED, num_hidden_layers=1)
    m = crane_b200.Qwen3Model(cfg, max_seq_len=64, max_batch=16)
    for name, shape, kind in synth.tensor_specs(cfg):
        t = synth.make_tensor(name, shape, kind)
        if "proj" in name or name == "lm_head.weight":
            m.load_tensor_ggml(name, gq.GGML_TYPE_ID[recipe], t.shape, gq.quantize(t, recipe))
        else:
            m.load_tensor(name, t)
    m.finalize()
    slots = [0] + [m.seq_create() for _ in range(8)]
    for s in slots:
        m.seq_select(s)
        m.forward_step(synth.synth_token_ids(4 + s, cfg["vocab_size"], f"q{s}"), 0)
    tok = synth.synth_token_ids(9, cfg["vocab_size"], "qt")

    def back():
        for s in slots:
            m.seq_select(s)
            m.set_kv_caches([], 4 + s)
    back()
    _, nine = m.decode_batch(slots, tok, 1, want_logits=True)
    back()
    four = np.concatenate([m.decode_batch(slots[i: i + 4], tok[i: i + 4], 1, want_logits=True)[1] for i in (0, 4, 8)])
    err = np.abs(nine - four).max(1) / np.abs(four).max()
    assert err.max() < 3e-2 and np.median(err) < 1e-2
    m.close()


@pytest.mark.parametrize("recipe", ["", "Q8_0"])
def test_batch_after_a_long_prompt(recipe):
    """A captured batch step, a prompt whose linears have more tiles than any call before it (Q8_0: 64 rows x 128 columns, 33 x 128 of them), the same
    step replayed: the same bits."""
    import crane_b200
    from oracle import ggml_quant as gq
    cfg = dict(synth.TINY_QWEN3_UNTIED, num_hidden_layers=1, hidden_size=256, intermediate_size=8192)
    m = crane_b200.Qwen3Model(cfg, max_seq_len=2176, max_batch=8)
    for name, shape, kind in synth.tensor_specs(cfg):
        t = synth.make_tensor(name, shape, kind)
        if recipe and "proj" in name:
            m.load_tensor_ggml(name, gq.GGML_TYPE_ID[recipe], t.shape, gq.quantize(t, recipe))
        else:
            m.load_tensor(name, t)
    m.finalize()
    slots = [0] + [m.seq_create() for _ in range(5)]
    extra = m.seq_create()
    for s in slots:
        m.seq_select(s)
        m.forward_step(synth.synth_token_ids(9 + s, cfg["vocab_size"], f"lp{s}"), 0)
    tok = synth.synth_token_ids(6, cfg["vocab_size"], "lpt")

    def batch():
        for s in slots:
            m.seq_select(s)
            m.set_kv_caches([], 9 + s)
        return m.decode_batch(slots, tok, 2, want_logits=True)
    toks, want = batch()
    for rows in (700, 2112, 2170):
        m.seq_select(extra)
        m.set_kv_caches([], 0)
        m.forward_step(synth.synth_token_ids(rows, cfg["vocab_size"], f"lpp{rows}"), 0)
        again, got = batch()
        assert np.array_equal(again, toks) and np.array_equal(got, want)
    m.close()


@pytest.mark.parametrize("vocab", [997, 998, 999])
def test_decode_batch_of_any_vocabulary(vocab):
    """Vocabularies that are not a multiple of four rows, against single steps (bounds as in test_decode_batch_against_single_steps)."""
    import crane_b200
    cfg = dict(synth.TINY_QWEN3_UNTIED, vocab_size=vocab)
    m = crane_b200.Qwen3Model(cfg, max_seq_len=64, max_batch=33)
    m.load_checkpoint(synth.synth_checkpoint(cfg))
    slots = [0] + [m.seq_create() for _ in range(32)]
    tok = synth.synth_token_ids(33, vocab, "anyv")
    want = []
    for s in slots:
        m.seq_select(s)
        m.forward_step(synth.synth_token_ids(3 + s, vocab, f"anyv{s}"), 0)
        want.append(m.forward_step([int(tok[s])], 3 + s))
    want = np.stack(want)
    for n in (2, 3, 5, 33):
        for s in slots[:n]:
            m.seq_select(s)
            m.set_kv_caches([], 3 + s)
        toks, got = m.decode_batch(slots[:n], tok[:n], 1, want_logits=True)
        assert np.abs(got - want[:n]).max() <= 3e-5 * np.abs(want).max()
        assert np.array_equal(toks[:, 0], got.argmax(1))
    for s in slots:
        m.seq_select(s)
        m.set_kv_caches([], 3 + s)
    assert np.array_equal(m.decode_batch_sample(slots, tok, [dict(temperature=0.0)] * 33), toks[:, 0])
    m.close()


def test_batches_of_many_sizes():
    """Steps launched kernel by kernel, captured after a while, replayed, dropped for other sizes' captures and captured again: the same bits as without graphs."""
    import crane_b200
    cfg = dict(synth.TINY_QWEN3_UNTIED, num_hidden_layers=1)
    out = []
    for graphs in (True, False):
        m = crane_b200.Qwen3Model(cfg, max_seq_len=64, max_batch=24, graphs=graphs)
        m.load_checkpoint(synth.synth_checkpoint(cfg))
        slots = [0] + [m.seq_create() for _ in range(23)]
        for s in slots:
            m.seq_select(s)
            m.forward_step(synth.synth_token_ids(5 + s, cfg["vocab_size"], f"ms{s}"), 0)
        tok = synth.synth_token_ids(24, cfg["vocab_size"], "mst")
        got = []
        for n in list(range(2, 25)) * 2 + [3, 24, 3]:
            for s in slots[:n]:
                m.seq_select(s)
                m.set_kv_caches([], 5 + s)
            got += m.decode_batch(slots[:n], tok[:n], 20, want_logits=True)
            got.append(m.decode_batch(slots[:n], tok[:n], 1)[0])
        out.append(got)
        m.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("recipe", ["Q4_K", "Q6_K", "Q8_0"])
@pytest.mark.parametrize("n", [3, 4, 9])
def test_quantised_decode_batch_against_the_oracle(recipe, n):
    """Three and nine sequences in one pass (four through the GEMVs), each row against the oracle's integer dots.  The same codes give the same sums: rows whose activations avoid the border of
    two codes agree to f32 rounding, a code on a border moves an output by up to 1e-2 (one in 128 of its block's largest value)."""
    import crane_b200
    from oracle import ggml_quant as gq
    from oracle.qwen3 import Qwen3Oracle
    cfg = dict(synth.TINY_QWEN3_UNTIED, num_hidden_layers=1)
    m = crane_b200.Qwen3Model(cfg, max_seq_len=64, max_batch=16)
    w, qd = {}, {}
    for name, t in synth.synth_checkpoint(cfg):
        if "proj" in name or name == "lm_head.weight":
            raw = gq.quantize(t, recipe)
            m.load_tensor_ggml(name, gq.GGML_TYPE_ID[recipe], t.shape, raw)
            w[name], qd[name] = gq.dequantize(raw, recipe, t.shape[1]), (raw, recipe)
        else:
            m.load_tensor(name, t)
            w[name] = t
    m.finalize()
    slots = [0] + [m.seq_create() for _ in range(n - 1)]
    ids = synth.synth_token_ids(18, cfg["vocab_size"], "qo")
    orc = Qwen3Oracle(cfg, w, quantised=qd)
    want = []
    for s in slots:
        m.seq_select(s)
        m.forward_step(ids[s: s + 1], 0)
        orc.clear_kv_cache()
        orc.forward(ids[s: s + 1], 0)
        want.append(orc.forward(ids[9 + s: 10 + s], 1).numpy().ravel())
    want = np.stack(want)
    _, got = m.decode_batch(slots, ids[9: 9 + n], 1, want_logits=True)
    err = np.abs(got - want).max(1) / np.abs(want).max(1)
    print(recipe, " ".join(f"{e:.1e}" for e in err))
    assert 3 * (err < 2e-5).sum() >= n and err.max() < 3e-2
    m.close()


# both sides of the lines between few-row tiles and 128-row tiles (gemm_rows_pays): one CTA per tile (75 tiles and more) and clusters
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("m,n,k", [(48, 9600, 64), (49, 9600, 64), (64, 9600, 128), (65, 9600, 128), (80, 9600, 64), (81, 9600, 64), (64, 2048, 1024), (65, 2048, 1024), (96, 2048, 1024),
                                   (97, 2048, 1024), (128, 2048, 2048), (128, 1024, 1088), (5, 19008, 64)])
def test_few_rows_at_the_lines(m, n, k, split):
    test_few_rows(m, n, k, split)


# f32 sums over W terms in some order: sqrt(W) * 2^-24 of the sum, below 4e-6 at 8192, half of it in 1 / rms; the two planes leave out 2^-17 of a value; the rest a few units of 2^-24.
@pytest.mark.parametrize("width", [4, 64, 1020, 1024, 1028, 1152, 2048, 2052, 2560, 4092, 4096, 4100, 5120, 8192])
@pytest.mark.parametrize("kind", ["rms", "layer"])
def test_row_norms(width, kind):
    """Rows held in registers (up to 1024, 2048 and 4096 columns), full and not, and the longer ones read again for every pass."""
    import ctypes as C
    import crane_b200 as cb
    rng = np.random.default_rng(width)
    x = (rng.standard_normal((7, width)) * rng.uniform(0.01, 30.0, (7, 1)) + (0.7 if kind == "layer" else 0.0)).astype(np.float32)
    x[3] = 0.0
    w, b = rng.uniform(0.5, 1.5, width).astype(np.float32), rng.standard_normal(width).astype(np.float32)
    hi, lo = np.empty((7, width), np.uint16), np.empty((7, width), np.uint16)
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert cb.load_library().crane_b200_debug_row_norm(ptr(x), 7, width, ptr(w), ptr(b) if kind == "layer" else None, C.c_float(1e-6), ptr(hi), ptr(lo)) == 0
    x64 = x.astype(np.float64)
    if kind == "layer":
        d = x64 - x64.mean(1, keepdims=True)
        want = d / np.sqrt((d * d).mean(1, keepdims=True) + 1e-6) * w + b
    else:
        want = x64 / np.sqrt((x64 * x64).mean(1, keepdims=True) + 1e-6) * w
    got = synth.bf16_bits_to_f32(hi).astype(np.float64) + synth.bf16_bits_to_f32(lo)
    assert np.abs(got - want).max() <= 2.0 ** -16 * np.abs(want).max()
