"""Products above 128 rows on pairs of CTAs: gate and up projection with their activation in one launch, the same bits as the products by themselves,
at the edges of tiles and of the deal and for operands whose quotients a fast division does not cover."""

import pytest
import torch

from extensions_b200 import tiny_llm_ext_b200 as ext
from tiny_llm_b200.quantize import QuantizedWeights, quantized_linear

pytestmark = pytest.mark.gpu


def weight(K, N, dtype, seed, gain=0.2):
    g = torch.Generator(device="cuda").manual_seed(seed)
    scales = (torch.randn(K, N // 128, generator=g, device="cuda") * gain / N**0.5).to(dtype)
    words = torch.randint(-(2**31), 2**31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    return QuantizedWeights(scales=scales, biases=(scales.float() * -7.5).to(dtype), group_size=128, bits=4, weight=words, use_simdgroup_matmul=True, use_split_k_matmul=True)


@pytest.mark.parametrize("M", [129, 255, 256, 257, 511, 513, 769, 1100])
@pytest.mark.parametrize("N,K", [(128, 136), (256, 1096), (384, 2504), (1024, 9728), (2560, 1001)])
def test_pairs_at_the_edges_of_tiles_and_rounds(M, N, K):
    """1001 columns: rows that TMA cannot store; 9728: more tiles than the chip has pairs, the last ones single."""
    gate, up = weight(K, N, torch.bfloat16, 1), weight(K, N, torch.bfloat16, 2)
    x = torch.randn(M, N, generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").bfloat16() * 4
    part = lambda w: (w.scales, w.biases, w.weight)  # noqa: E731
    flags = (True, True)
    want, before = ext.swiglu(quantized_linear(x, gate), quantized_linear(x, up)), ext.launch_count()
    got = ext.quantized_gate_up(x, part(gate), part(up), flags, flags)
    assert ext.launch_count() - before == 1
    assert torch.equal(got, want)
    assert ext.waits_given_up() == 0


@pytest.mark.parametrize("M", [130, 600])
def test_gates_outside_the_fast_division(M):
    """Gates of -1e4 to 1e4 and beyond, zeros, infinities and NaN: every bit as the activation's own kernel gives it."""
    N, K = 256, 264
    gate, up = weight(K, N, torch.bfloat16, 1, gain=40.0), weight(K, N, torch.bfloat16, 2, gain=0.01)
    x = torch.randn(M, N, generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").bfloat16()
    x[: M // 2] *= torch.logspace(-30, 4, M // 2, device="cuda").bfloat16()[:, None]
    x[5], x[6, 3], x[7, 100], x[8, 9] = 0, float("inf"), float("-inf"), float("nan")
    part = lambda w: (w.scales, w.biases, w.weight)  # noqa: E731
    want = ext.swiglu(quantized_linear(x, gate), quantized_linear(x, up))
    got = ext.quantized_gate_up(x, part(gate), part(up), (True, True), (True, True))
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(), want.nan_to_num())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,K", [(9728, 2560), (6144, 2048), (3072, 1024)])
def test_a_row_has_the_same_bits_in_any_portion(N, K, dtype):
    """Above 128 rows a reduction is one sum, whatever the number of rows and whichever kernel: a prompt may be cut anywhere."""
    w = weight(K, N, dtype, N)
    x = torch.randn(2048, N, generator=torch.Generator(device="cuda").manual_seed(K), device="cuda").to(dtype)
    whole = quantized_linear(x, w)
    for M in (129, 200, 256, 257, 300, 512, 700, 1024, 1500):
        assert torch.equal(quantized_linear(x[:M], w), whole[:M])
