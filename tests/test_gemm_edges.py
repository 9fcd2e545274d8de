"""GPU (-m gpu): the 128-row GEMM tiles where their epilogue can go wrong: row counts around the 32-row store patches, a last column tile of 32 or 96
columns, one k-step, tiles of every width, whole and shared by several CTAs, for every epilogue; against float64 and bit for bit from call to call.

Tolerances (largest difference over the largest result): f32 results 1e-5 (K <= 4096 products in f32, another order of additions: below sqrt(K) 2^-24
of the largest, times a few), residuals the same, bf16 results 2^-8 (their rounding, 2^-9 of the value, and the f32 part), bf16 results with their low-order
plane 2^-15 (what the two leave out, 2^-17 of the value, and the f32 part with the functions' own error)."""
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


@pytest.mark.parametrize("split", [False, True], ids=["plain", "split"])
@pytest.mark.parametrize("shape", [(160, 288, 1024), (161, 544, 1024), (255, 1024, 64), (300, 160, 4096), (129, 6176, 512), (129, 4128, 4096), (257, 8224, 1024), (600, 4128, 4096)],
                         ids=["64", "64a", "64b", "64 shared", "128", "128 shared", "256", "256 shared"])
def test_every_part_of_the_epilogue(shape, split, request):
    """Bias, column scale, gate and both planes of every mode, in tiles of the width and schedule that the plan takes at 148 SMs."""
    M, N, K = shape
    name = request.node.callspec.id.replace("split", "").replace("plain", "").strip("-")
    plan = crane_b200.load_library().crane_b200_debug_gemm_tiles
    assert {plan(mode, M, N, K, int(split)) for mode in range(7)} == {int(name.split()[0].rstrip("ab")) + (1000 if "shared" in name else 0)}
    rng = np.random.default_rng(M + N * 3 + K)
    a = rng.standard_normal((M, K), dtype=np.float32)
    hi = synth.bf16_round(a)
    bits = synth.f32_to_bf16_bits(a)
    lo_bits = synth.f32_to_bf16_bits(a - hi) if split else None
    val = hi.astype(np.float64) + (synth.bf16_round(a - hi).astype(np.float64) if split else 0.0)
    wf = rng.standard_normal((N, K), dtype=np.float32) / np.sqrt(K)
    w, w_bits = synth.bf16_round(wf).astype(np.float64), synth.f32_to_bf16_bits(wf)
    bias, scale, gate_bias = (rng.standard_normal(N).astype(np.float32) for _ in range(3))
    gate, init = (rng.standard_normal((M, N)).astype(np.float32) for _ in range(2))
    ref = val @ w.T
    full = (ref + bias) * scale / (1.0 + np.exp(-(gate.astype(np.float64) + gate_bias)))

    def run(mode, **kw):
        one = crane_b200.op_gemm_epi(bits, w_bits, mode, a_lo_bits=lo_bits, **kw)
        two = crane_b200.op_gemm_epi(bits, w_bits, mode, a_lo_bits=lo_bits, **kw)
        assert all(np.array_equal(x, y) for x, y in zip(one, two))
        return one
    parts = dict(bias=bias, col_scale=scale, gate=gate, gate_bias=gate_bias)
    assert rel_err(run(crane_b200.EPI_STORE_F32, **parts), full) < 1e-5
    assert rel_err(run(crane_b200.EPI_RESID_F32, out_init=init, **parts), init + full) < 1e-5
    x = torch.from_numpy(ref + bias)
    g, u = (ref + bias)[:, 0::2], (ref + bias)[:, 1::2]
    cg, cu = np.minimum(g, 1.5), np.clip(u, -1.5, 1.5)
    sig = lambda t: 1.0 / (1.0 + np.exp(-t))  # noqa: E731
    for mode, kw, want in (
            (crane_b200.EPI_STORE_BF16, {}, ref + bias),
            (crane_b200.EPI_RELU2_BF16, {}, np.maximum(ref + bias, 0.0) ** 2),
            (crane_b200.EPI_GELU_ERF_BF16, {}, torch.nn.functional.gelu(x).numpy()),
            (crane_b200.EPI_GELU_TANH_BF16, {}, torch.nn.functional.gelu(x, approximate="tanh").numpy()),
            (crane_b200.EPI_SILU_MUL_BF16, {}, g * sig(g) * u),
            (crane_b200.EPI_SILU_MUL_BF16, {"glu_limit": 1.5}, cg * sig(1.702 * cg) * (cu + 1.0))):
        h, l = run(mode, bias=bias, lo=True, **kw)
        assert rel_err(synth.bf16_bits_to_f32(h), want) < 2.0 ** -8, (mode, kw)
        assert rel_err(synth.bf16_bits_to_f32(h).astype(np.float64) + synth.bf16_bits_to_f32(l), want) < 2.0 ** -15, (mode, kw)
        alone = crane_b200.op_gemm_epi(bits, w_bits, mode, a_lo_bits=lo_bits, bias=bias, **kw)
        assert np.array_equal(alone, h)                                               # without the low-order plane
