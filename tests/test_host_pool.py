"""Results in pinned memory (csrc/host_pool.h): arrays own their buffers, kept results stay as they are, the pool's bound turns into ordinary memory, and nothing is handed
out without a handle."""
import ctypes as C
import gc
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

import crane_b200
from crane_b200 import synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


@pytest.mark.gpu
def test_pieces_of_one_range():
    """Every piece lies in one range of up to 64 MiB, as far as the handles need it, whatever was asked for before: rounds of 32 rows over 151 936 logits (19.4 MB) with the last one still held, beside a row at
    a time, never leave it; a program that keeps everything ends in ordinary memory; and what was given back in any order is whole again.  (In a process of its own: the
    range is a process's.)"""
    r = subprocess.run([sys.executable, "-c", "import sys; sys.path[:0] = [%r, %r]; import test_host_pool as t; t.pieces()" % (ROOT, os.path.join(ROOT, "tests"))],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def pieces():
    small = dict(synth.TINY_QWEN3)
    large = dict(synth.TINY_QWEN3, vocab_size=151936)
    m = crane_b200.Qwen3Model(small, max_seq_len=64)                    # 2 MiB are enough for it
    assert crane_b200._result((1 << 18,)).base is not None and crane_b200._result((3 << 18,)).base is None
    early = crane_b200._result((1024,))
    n = crane_b200.Qwen3Model(large, max_seq_len=64, max_batch=32)      # ... and the rest for this one
    m.close()
    span = [early.ctypes.data, early.ctypes.data + early.nbytes]

    def take(*shape):
        a = crane_b200._result(shape)
        a[...] = len(span)
        if a.base is not None:
            span.extend((a.ctypes.data, a.ctypes.data + a.nbytes))
        return a
    for _ in range(4):
        out = None                                          # (a first round; those behind it hold the one before)
        for _ in range(5):
            out = take(32, 151936)
            row = take(151936)
            assert out.base is not None and row.base is not None
        del out, row
    rng = np.random.default_rng(0)
    kept = [take(int(rng.integers(1024, 1 << 20))) for _ in range(100)]
    marks = [k.flat[0] for k in kept]
    assert any(k.base is None for k in kept) and all((k == v).all() for k, v in zip(kept, marks))
    while kept:
        kept.pop(int(rng.integers(len(kept))))
    del early
    assert take(62 << 18).base is not None and crane_b200._result((64 << 18,)).base is None       # (no piece lies across what was added)
    first, rest = take(2 << 18), take(62 << 18)
    assert first.base is not None and rest.base is not None and max(span) - min(span) == 64 << 20
    n.close()
    assert (rest == rest.flat[0]).all()
    m = crane_b200.Qwen3Model(small, max_seq_len=64)                    # the range lives on with its pieces; the next handle finds it used up
    assert crane_b200._result((1024,)).base is None
    del first
    assert crane_b200._result((1024,)).base is not None
    m.close()
    del rest
    m = crane_b200.Qwen3Model(large, max_seq_len=64, max_batch=32)      # made anew, in one
    assert crane_b200._result((64 << 18,)).base is not None
    m.close()


@pytest.mark.gpu
def test_a_thread_keeps_its_context():
    """Taking and giving back results opens no context in a thread that has none, the range's making and release included."""
    cu = C.CDLL("libcuda.so.1")
    seen = []

    def current():
        c = C.c_void_p()
        assert cu.cuCtxGetCurrent(C.byref(c)) == 0
        seen.append(c.value)

    def work():
        current()
        lib, p = crane_b200.load_library(), C.c_void_p()
        assert lib.crane_b200_host_alloc(1 << 20, C.byref(p)) == crane_b200.OK
        current()
        assert lib.crane_b200_host_free(p) == crane_b200.OK
        current()

    m = crane_b200.Qwen3Model(synth.TINY_QWEN3, max_seq_len=64)
    t = threading.Thread(target=work)
    t.start()
    t.join()
    last = crane_b200._result((5000,))
    m.close()
    box = [last]
    del last
    t = threading.Thread(target=lambda: (current(), box.clear(), gc.collect(), current()))
    t.start()
    t.join()
    assert seen == [None] * 5


@pytest.mark.gpu
def test_a_forked_process_keeps_what_it_had():
    """A child's results are its own, as in ordinary memory, while its parent's later calls reuse their pieces, and the parent's later results are right although it has written
    to pages that the child shares.  (The child calls nothing of CUDA's.)"""
    r = subprocess.run([sys.executable, "-c", "import sys; sys.path[:0] = [%r, %r]; import test_host_pool as t; t.forked()" % (ROOT, os.path.join(ROOT, "tests"))],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def forked():
    cfg = dict(synth.TINY_QWEN3, vocab_size=40000)
    m = crane_b200.Qwen3Model(cfg, max_seq_len=64)
    m.load_checkpoint(synth.synth_checkpoint(cfg))
    got = m.forward_step([1, 2, 3], 0)
    was, at = got.copy(), got.ctypes.data
    assert got.base is not None
    to_child, go = os.pipe()
    pid = os.fork()
    if pid == 0:
        os.read(to_child, 1)
        os._exit(0 if np.array_equal(got, was) else 1)
    got[:] = 0.0
    del got
    m.clear_kv_cache()
    again = m.forward_step([1, 2, 3], 0)
    assert again.ctypes.data == at and np.array_equal(again, was)
    m.clear_kv_cache()
    m.forward_step([4, 5], 0)
    os.write(go, b"x")
    assert os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]) == 0
    m.close()
