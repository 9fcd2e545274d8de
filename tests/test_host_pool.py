"""Results in pinned memory (csrc/host_pool.h): arrays own their buffers, kept results stay as they are, the pool's bound turns into ordinary memory, and nothing is handed
out without a handle."""
import ctypes as C
import gc
import threading

import numpy as np
import pytest

import crane_b200
from crane_b200 import synth


def test_without_a_handle_there_is_none():
    lib = crane_b200.load_library()
    p = C.c_void_p()
    assert lib.crane_b200_host_alloc(0, C.byref(p)) == crane_b200.INVALID_ARG
    assert lib.crane_b200_host_alloc(4096, None) == crane_b200.INVALID_ARG
    assert lib.crane_b200_host_alloc(64 << 20, C.byref(p)) == crane_b200.OOM          # above a buffer's bound
    assert lib.crane_b200_host_free(None) == crane_b200.INVALID_ARG
    assert crane_b200._result((3, 5000)).shape == (3, 5000)


@pytest.mark.gpu
def test_results_are_their_callers():
    cfg = dict(synth.TINY_QWEN3, vocab_size=40000)
    m = crane_b200.Qwen3Model(cfg, max_seq_len=128, max_batch=4)
    m.load_checkpoint(synth.synth_checkpoint(cfg))
    ids = synth.synth_token_ids(20, cfg["vocab_size"], "pool")
    kept = [m.forward_step(ids[:10], 0)] + [m.forward_step(ids[i: i + 1], i) for i in range(10, 20)]
    was = [k.copy() for k in kept]
    m.clear_kv_cache()
    again = [m.forward_step(ids[:10], 0)] + [m.forward_step(ids[i: i + 1], i) for i in range(10, 20)]
    for k, w, a in zip(kept, was, again):
        assert np.array_equal(k, w) and np.array_equal(a, w) and k.flags.writeable and k.ctypes.data != a.ctypes.data
    view = again[3][100:200]
    expect = view.copy()
    del again, kept, k, a
    gc.collect()
    m.clear_kv_cache()
    for _ in range(3):
        m.forward_step(ids[:10], 0)
        m.clear_kv_cache()
    assert np.array_equal(view, expect)                        # a view keeps its buffer
    held = [crane_b200._result((1 << 20,), np.uint8) for _ in range(80)]      # the bound: 64 of these at most, then ordinary memory
    for i, h in enumerate(held):
        h[:] = i
    assert all((h == i).all() for i, h in enumerate(held)) and sum(h.base is not None for h in held) <= 64
    m.close()
    del m
    gc.collect()
    assert np.array_equal(view, expect)                        # ... past the last handle too
    assert crane_b200._result((5000,)).base is None or crane_b200._result((5000,)).flags.owndata is False


@pytest.mark.gpu
def test_threads_share_the_pool():
    cfg = synth.TINY_QWEN3
    m = crane_b200.Qwen3Model(cfg, max_seq_len=64)
    bad = []

    def work(seed):
        r = np.random.default_rng(seed)
        for _ in range(300):
            a = crane_b200._result((int(r.integers(1024, 9000)),))
            a[:] = seed
            if not (a == seed).all():
                bad.append(seed)
    ts = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    m.close()
    assert not bad
