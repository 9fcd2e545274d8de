"""Quantised linears on the tensor cores (csrc/qgemm.cu) against the oracle's integer dots, at the edges of the kernel's tiles: 16 / 32 / 64 /
128 activation columns, 128 weight rows, one and more super-blocks, work shared by several blocks and not."""
import numpy as np
import pytest

from oracle import ggml_quant as gq

pytestmark = pytest.mark.gpu

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
