"""A wait of a tensor-core kernel that runs out: the call that hands out the results reports it, sequences do not move on, and the next call works.
The wait is one of a small kernel of the library's own, for a barrier that nothing arrives at (about a millisecond)."""
import ctypes as C

import numpy as np
import pytest

from crane_b200 import synth

pytestmark = pytest.mark.gpu


def expire(m=None):
    import crane_b200
    fn = crane_b200.load_library().crane_b200_debug_expire_wait
    fn.restype, fn.argtypes = C.c_int, [C.c_void_p]
    assert fn(m.h if m is not None else None) == 0


def reported(m, call):
    """`call` works, fails once when a wait ran out before it, and works again with the same result."""
    import crane_b200
    want = call()
    expire(m)
    with pytest.raises(crane_b200.CraneB200Error, match="wait ran out"):
        call()
    for a, b in zip(want, call()):
        assert np.array_equal(np.asarray(a), np.asarray(b))


def test_dense_calls():
    import crane_b200
    cfg = synth.TINY_QWEN3_UNTIED
    m = crane_b200.Qwen3Model(cfg, max_seq_len=128, max_batch=8)
    m.load_checkpoint(synth.synth_checkpoint(cfg))
    ids = synth.synth_token_ids(20, cfg["vocab_size"], "we")
    slots = [0] + [m.seq_create() for _ in range(5)]

    def back(n=20):
        for s in slots:
            m.seq_select(s)
            m.set_kv_caches([], n)
        m.seq_select(0)

    def fresh(f):
        def g():
            m.seq_select(0)
            m.set_kv_caches([], 0)
            return f()
        return g
    for s in slots:
        m.seq_select(s)
        m.forward_step(ids, 0)
    reported(m, fresh(lambda: [m.forward_step(ids, 0)]))
    reported(m, fresh(lambda: [m.forward_step_argmax(ids, 0)]))
    reported(m, fresh(lambda: [m.forward_step_sample(ids, 0, temperature=0.0)]))
    reported(m, fresh(lambda: [m.generate_greedy(ids, 4)]))
    back()
    m.forward_step([1], 20)
    reported(m, lambda: [m.copy_logits()])
    reported(m, lambda: m.topk(5))
    reported(m, lambda: [m.sample(temperature=0.0)])
    reported(m, lambda: [x for kv in m.get_kv_caches() for x in kv])
    tok = synth.synth_token_ids(6, cfg["vocab_size"], "wet")

    def batch(f):
        def g():
            back()
            out = f()
            assert [m.seq_len(s) for s in slots] == [21] * 6
            return out
        return g
    reported(m, batch(lambda: m.decode_batch(slots, tok, 1, want_logits=True)))
    reported(m, batch(lambda: [m.decode_batch_sample(slots, tok, [dict(temperature=0.0)] * 6)]))
    for f in (lambda: m.decode_batch(slots, tok, 1), lambda: m.decode_batch_sample(slots, tok, [dict(temperature=0.0)] * 6)):
        back()
        expire(m)
        with pytest.raises(crane_b200.CraneB200Error, match="wait ran out"):
            f()
        assert [m.seq_len(s) for s in slots] == [20] * 6
    m.close()


def test_vision_calls():
    import crane_b200
    cfg = synth.TINY_QWEN3_VL
    m = crane_b200.Qwen3VLModel(cfg, max_seq_len=64)
    m.load_checkpoint(synth.synth_checkpoint(cfg))
    pv = np.random.default_rng(3).uniform(-1, 1, (64, 1536)).astype(np.float32)
    reported(m, lambda: [m.encode_images(pv, [(1, 8, 8)])[0]])
    m.close()


def test_layer_list_calls():
    import crane_b200
    cfg = synth.fosovik_config(width=256, vocab=512, blocks=1, heads=4, kv_heads=2, dim=64, ssm_heads=4, ssm_vdim=64, state=32, ff=512)
    m = crane_b200.FosovikModel(cfg, max_tokens=4096, max_batch=8)
    m.load_checkpoint(synth.synth_checkpoint(cfg))
    slots = [0] + [m.seq_create() for _ in range(5)]
    ids = synth.synth_token_ids(30, 512, "wel")
    m.step_batch([(s, ids, [29]) for s in slots])
    reported(m, lambda: [m.sample_rows([dict(temperature=0.0)] * 6)])
    tok = synth.synth_token_ids(6, 512, "welt")
    for f in (lambda: m.decode_batch(slots, tok, 2), lambda: m.decode_batch_sample(slots, tok, [dict(temperature=0.0)] * 6)):
        expire(m)
        with pytest.raises(crane_b200.CraneB200Error, match="wait ran out"):
            f()
        f()
    m.close()


def test_single_operations():
    import crane_b200
    from oracle import ggml_quant as gq
    rng = np.random.default_rng(5)
    a = synth.f32_to_bf16_bits(rng.standard_normal((40, 128)).astype(np.float32))
    w = synth.f32_to_bf16_bits(rng.standard_normal((64, 128)).astype(np.float32))
    raw = gq.quantize(rng.standard_normal((64, 256)).astype(np.float32), "Q8_0")
    x = rng.standard_normal((9, 256)).astype(np.float32)
    for f in (lambda: [crane_b200.op_gemm(a, w, crane_b200.EPI_STORE_F32)], lambda: [crane_b200.op_qlinear(x, raw, 8, 64)]):
        want = f()
        expire()
        with pytest.raises(crane_b200.CraneB200Error):
            f()
        assert np.array_equal(f()[0], want[0])


def test_speech_calls():
    import crane_b200
    cfg = synth.TINY_QWEN3_TTS
    m = crane_b200.Qwen3TTSModel(cfg, device=0, max_seq_len=256)
    m.load_checkpoint(synth.synth_checkpoint(cfg))
    reported(m, lambda: [m.text_project([1, 2, 3])])
    m.close()


def test_pair_gives_up_together():
    """One CTA of a pair gives up after a millisecond; the other, whose wait would run for 4 s, is released by it, and the error is reported once."""
    import time
    import crane_b200
    cfg = synth.TINY_QWEN3_UNTIED
    m = crane_b200.Qwen3Model(cfg, max_seq_len=64)
    m.load_checkpoint(synth.synth_checkpoint(cfg))
    ids = synth.synth_token_ids(20, cfg["vocab_size"], "wp")
    want = m.forward_step(ids, 0)
    fn = crane_b200.load_library().crane_b200_debug_expire_wait_pair
    fn.restype, fn.argtypes = C.c_int, [C.c_void_p]
    t = time.perf_counter()
    assert fn(m.h) == 0
    m.clear_kv_cache()
    with pytest.raises(crane_b200.CraneB200Error, match="wait ran out"):
        m.forward_step(ids, 0)
    assert time.perf_counter() - t < 2.0
    m.clear_kv_cache()
    assert np.array_equal(m.forward_step(ids, 0), want)
    m.close()
