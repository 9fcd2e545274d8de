"""GPU (-m gpu): GEMM tiles of CTA pairs (256 x 256, gemm_tc2_kernel) at their edges: one row more than a CTA's 128, one more than a pair's 256, rows that leave the odd CTA
without any, column tiles of 32, 160 and 288 columns, one k-step, whole tiles and tiles shared along K.  The width is pinned in a process of its own (the plan takes pairs
for large shapes only); three shapes that the plan gives to pairs by itself beside it; every check asks the plan for the tiles that it means.  Against float64: f32 results to
1e-5, bf16 results with their low-order plane to 2^-15 (test_gemm_edges.py derives the bounds).  One accumulator that takes all of K is off by an amount that grows with K: at
4096 products of two planes f32 results by up to 1.0e-5, both planes by 0.9 of 2^-15, the same in tiles of 64, 256 and 512 columns."""
import os
import re
import subprocess
import sys

import numpy as np
import pytest

import crane_b200
from crane_b200 import synth

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def tiles(M, N, K, split, modes=(crane_b200.EPI_STORE_F32, crane_b200.EPI_RESID_F32, crane_b200.EPI_SILU_MUL_BF16, crane_b200.EPI_STORE_BF16)):
    """Columns of the tiles that the plan takes, 1000 more where they are shared along K: one answer for all modes."""
    got = {crane_b200.load_library().crane_b200_debug_gemm_tiles(m, M, N, K, int(split)) for m in modes}
    return got.pop() if len(got) == 1 else got


def check(M, N, K, split, want):
    assert tiles(M, N, K, split) == want
    rng = np.random.default_rng(M * 3 + N + K)
    a = rng.standard_normal((M, K), dtype=np.float32)
    bits = synth.f32_to_bf16_bits(a)
    lo = synth.f32_to_bf16_bits(a - synth.bf16_round(a)) if split else None
    val = synth.bf16_round(a).astype(np.float64) + (synth.bf16_round(a - synth.bf16_round(a)).astype(np.float64) if split else 0.0)
    wf = rng.standard_normal((N, K), dtype=np.float32) / np.sqrt(K)
    ref = val @ synth.bf16_round(wf).astype(np.float64).T
    w = synth.f32_to_bf16_bits(wf)
    bias, init = rng.standard_normal(N).astype(np.float32), rng.standard_normal((M, N)).astype(np.float32)
    err = lambda got, want: np.abs(got - want).max() / np.abs(want).max()  # noqa: E731
    for _ in range(2):
        one = crane_b200.op_gemm(bits, w, crane_b200.EPI_STORE_F32, a_lo_bits=lo, bias=bias)
        two = crane_b200.op_gemm(bits, w, crane_b200.EPI_STORE_F32, a_lo_bits=lo, bias=bias)
        assert np.array_equal(one, two) and err(one, ref + bias) < 1e-5
    assert err(crane_b200.op_gemm(bits, w, crane_b200.EPI_RESID_F32, a_lo_bits=lo, out_init=init), init + ref) < 1e-5
    g, u = ref[:, 0::2], ref[:, 1::2]
    hi, low = crane_b200.op_gemm_epi(bits, w, crane_b200.EPI_SILU_MUL_BF16, a_lo_bits=lo, lo=True)
    assert err(synth.bf16_bits_to_f32(hi).astype(np.float64) + synth.bf16_bits_to_f32(low), g / (1 + np.exp(-g)) * u) < 2.0 ** -15
    hi, low = crane_b200.op_gemm_epi(bits, w, crane_b200.EPI_STORE_BF16, a_lo_bits=lo, lo=True)
    assert err(synth.bf16_bits_to_f32(hi).astype(np.float64) + synth.bf16_bits_to_f32(low), ref) < 2.0 ** -15


EDGES = {"1": [(129, 256, 64), (256, 288, 192), (257, 416, 512), (300, 544, 1024), (385, 1056, 128), (640, 256, 4096)],
         "2": [(129, 288, 4864), (256, 288, 4864), (257, 416, 2432), (300, 544, 2048), (385, 1056, 1024), (640, 256, 4096)]}      # (148 k-steps and more: two for each of 74 pairs)


def run(code, **env):
    r = subprocess.run([sys.executable, "-c", "import sys; sys.path[:0] = [%r, %r]; import test_gemm_pairs as t\n%s" % (ROOT, os.path.join(ROOT, "tests"), code)], env=dict(os.environ, **env),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("schedule", ["1", "2"], ids=["whole", "shared"])
def test_edges(schedule):
    run("for e in t.EDGES[%r]:\n    for s in (False, True): t.check(*e, s, %d)" % (schedule, 512 if schedule == "1" else 1512), CRANE_B200_GEMM_BN="512", CRANE_B200_GEMM_SCHED=schedule)


TURNS = [(2400, 2336, 128), (2050, 4640, 64), (1100, 9472, 192)]        # several tiles a CTA; rows of tiles that 8 does not divide


@pytest.mark.parametrize("width", ["64", "256", "512"])
def test_whole_tiles_in_turns(width):
    run("for e in t.TURNS: t.check(*e, e[0] == 2050, %s)" % width, CRANE_B200_GEMM_BN=width, CRANE_B200_GEMM_SCHED="1")


@pytest.mark.parametrize("shape,split,want", [((2000, 6176, 2048), False, 512), ((770, 6176, 4096), False, 1512), ((2200, 4128, 2048), True, 1512)], ids=["whole", "shared", "split"])
def test_shapes_of_the_plan(shape, split, want):
    check(*shape, split, want)


def test_timeline():
    """The timeline of a launch (tools/gemm_probe.py) where the plan takes pairs: every stage has a time, and none is longer than the launch."""
    code = ("import sys; sys.path[:0] = [%r]; import numpy as np, crane_b200; r = np.random.default_rng(0).integers(0x3c00, 0x3c80, (2, 1024, 2048)).astype(np.uint16);"
            "crane_b200.op_gemm(r[0], r[1], crane_b200.EPI_STORE_F32)" % ROOT)
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, CRANE_B200_GEMM_BN="512", CRANE_B200_GEMM_SCHED="1", CRANE_B200_GEMM_PROF="1"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    line = next(x for x in r.stderr.splitlines() if x.startswith("gemm_prof"))
    assert "one launch: 32 CTAs" in line
    span = float(re.search(r"span ([0-9.]+) us", line).group(1))
    stages = [float(x) for x in re.findall(r"(?:setup|operands|issue|wait|epilogue) ([0-9.+-]+)", line)]
    assert len(stages) == 5 and 1.0 < span < 1e4 and all(0.0 < x <= 1e3 * span for x in stages), line
