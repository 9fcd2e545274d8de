"""GPU (-m gpu): the 128-row GEMM tiles where their epilogue can go wrong: row counts around the 32-row store patches, a last column tile of 32 or 96
columns, one k-step, tiles shared by several CTAs, for every epilogue; against float64 and bit for bit from call to call.

Tolerances (largest difference over the largest result): f32 results 1e-5 (K <= 4096 products in f32, another order of additions: below sqrt(K) 2^-24
of the largest, times a few), residuals the same, bf16 results 2^-8 (their rounding, 2^-9 of the value, and the f32 part)."""
import numpy as np
import pytest
import torch

from conftest import rel_err
import crane_b200
from crane_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [False, True], ids=["plain", "split"])
@pytest.mark.parametrize("shape", [(129, 32, 64), (130, 96, 128), (160, 288, 1024), (161, 544, 1024), (255, 1024, 64), (257, 256, 512), (300, 160, 4096)])
def test_epilogues_at_tile_edges(shape, split):
    M, N, K = shape
    rng = np.random.default_rng(M * 3 + N + K)
    a = rng.standard_normal((M, K), dtype=np.float32)
    hi = synth.bf16_round(a)
    bits = synth.f32_to_bf16_bits(a)
    lo_bits = synth.f32_to_bf16_bits(a - hi) if split else None
    val = hi.astype(np.float64) + (synth.bf16_round(a - hi).astype(np.float64) if split else 0.0)
    wf = rng.standard_normal((N, K), dtype=np.float32) / np.sqrt(K)
    w, w_bits = synth.bf16_round(wf).astype(np.float64), synth.f32_to_bf16_bits(wf)
    bias = rng.standard_normal(N).astype(np.float32)
    init = rng.standard_normal((M, N)).astype(np.float32)
    ref = val @ w.T

    def run(mode, **kw):
        one = crane_b200.op_gemm(bits, w_bits, mode, a_lo_bits=lo_bits, **kw)
        assert np.array_equal(one, crane_b200.op_gemm(bits, w_bits, mode, a_lo_bits=lo_bits, **kw))
        return one if one.dtype == np.float32 else synth.bf16_bits_to_f32(one)
    assert rel_err(run(crane_b200.EPI_STORE_F32, bias=bias), ref + bias) < 1e-5
    assert rel_err(run(crane_b200.EPI_RESID_F32, bias=bias, out_init=init), init + ref + bias) < 1e-5
    assert rel_err(run(crane_b200.EPI_STORE_BF16), ref) < 2.0 ** -8
    g, u = ref[:, 0::2], ref[:, 1::2]
    assert rel_err(run(crane_b200.EPI_SILU_MUL_BF16), g / (1 + np.exp(-g)) * u) < 2.0 ** -8
    x = torch.from_numpy(ref + bias)
    for mode, approx in ((crane_b200.EPI_GELU_ERF_BF16, "none"), (crane_b200.EPI_GELU_TANH_BF16, "tanh")):
        assert rel_err(run(mode, bias=bias), torch.nn.functional.gelu(x, approximate=approx).numpy()) < 2.0 ** -8
