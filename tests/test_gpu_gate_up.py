"""The gated MLP's first half in one call - the up projection applies the activation in its epilogue - against two products and swiglu:
the same bits from every kernel that a number of rows takes, whole and ragged feature tiles, unaligned rows, both types."""

import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from extensions_b200 import tiny_llm_ext_b200 as ext
from tiny_llm_b200.quantize import QuantizedWeights, quantized_gate_up, quantized_linear, quantized_mlp

pytestmark = pytest.mark.gpu


def weight(K, N, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    scales = (torch.randn(K, N // 128, generator=g, device="cuda") * 0.2 / N**0.5).to(dtype)
    words = torch.randint(-(2**31), 2**31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    return scales, (scales.float() * -7.5).to(dtype), words


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("K,N", [(1000, 256), (1001, 384), (9728, 2560), (130, 1024)])
@pytest.mark.parametrize("M", [0, 1, 5, 8, 9, 24, 64, 100, 128, 129, 300, 515, 2048])
def test_equals_two_products_and_swiglu(M, K, N, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    a = torch.randn(M, N, generator=g, device="cuda").to(dtype) * 4
    gate, up = weight(K, N, dtype, 1), weight(K, N, dtype, 2)
    for flags in ((True, False), (True, True)) + (((False, False),) if M * K < 10**6 else ()):
        product = lambda w: ext.quantized_matmul(w[0], w[1], 128, 4, a, w[2], True, *flags)
        want = ext.swiglu(product(gate), product(up))
        assert torch.equal(ext.quantized_gate_up(a, gate, up, flags, flags), want)
    if M == 2048:  # the kernel of thread-block pairs, for every size
        ext.set_gemm_pairs(2)
        try:
            want = ext.swiglu(product(gate), product(up))
            assert torch.equal(ext.quantized_gate_up(a, gate, up, flags, flags), want)
        finally:
            ext.set_gemm_pairs(1)


def test_layer_form_mixed_flags_and_refusals():
    gate, up, odd = (weight(k, 256, torch.bfloat16, s) for k, s in ((264, 1), (264, 2), (272, 3)))
    wrap = lambda w, **flags: QuantizedWeights(scales=w[0], biases=w[1], group_size=128, bits=4, weight=w[2], **flags)
    x = torch.randn(3, 40, 256, device="cuda").bfloat16().transpose(0, 1)
    a, b = wrap(gate), wrap(up, use_simdgroup_matmul=True)
    assert torch.equal(quantized_gate_up(x, a, b), ext.swiglu(quantized_linear(x, a), quantized_linear(x, b)))
    with pytest.raises(RuntimeError, match="swiglu: gate and up must have the same shape"):
        quantized_gate_up(x, a, wrap(odd))
    with pytest.raises(RuntimeError, match="a must be the same dtype as scales"):
        quantized_gate_up(x.half(), a, b)


def test_the_gate_is_kept_for_the_stream_that_reads_it():
    """On a stream of its own the intermediate outlives the call: what the caller allocates meanwhile must not lie in its place."""
    N, K, M = 1024, 2048, 6
    weights = [weight(K, N, torch.bfloat16, seed) for seed in (1, 2)]
    x = torch.randn(M, N, device="cuda").bfloat16()
    want = ext.quantized_gate_up(x, *weights)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)  # about 10 ms: the products are queued, not run, when the call returns
    got = ext.quantized_gate_up(x, *weights, stream=side)
    taken = [torch.full((M, K), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    torch.cuda.current_stream().synchronize()
    side.synchronize()
    assert torch.equal(got, want) and all(bool(t.isnan().all()) for t in taken)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [1, 8, 9, 52, 128, 129, 700])
def test_the_whole_mlp_in_one_call_equals_its_products(M, dtype):
    wrap = lambda w, **flags: QuantizedWeights(scales=w[0], biases=w[1], group_size=128, bits=4, weight=w[2], **flags)
    gate, up, down = (wrap(weight(k, n, dtype, s), use_simdgroup_matmul=True, use_split_k_matmul=True) for k, n, s in ((1408, 768, 1), (1408, 768, 2), (520, 1408, 3)))
    x = torch.randn(2, M, 768, device="cuda").to(dtype) * 4
    for form in (x[:1], x, x.transpose(0, 1), x[:, :, :768][0], x[:, ::2]):  # one, three and two dimensions, rows that do not follow one another
        want = quantized_linear(quantized_gate_up(form, gate, up), down)
        got = quantized_mlp(form, gate, up, down)
        assert got.shape == want.shape and torch.equal(got, want)
    with pytest.raises(RuntimeError, match="0 elements"):
        quantized_mlp(x[:, :0], gate, up, down)
    with pytest.raises(RuntimeError, match="a must be the same dtype as scales"):
        quantized_mlp(x.float(), gate, up, down)
    with pytest.raises(RuntimeError, match="one column per input group"):
        quantized_mlp(x[..., :640].contiguous(), gate, up, down)


def test_the_wide_geometry_is_not_mixed_with_the_other():
    """TL_SKINNY_WIDE1=1 (A/B runs) at 65 to 128 rows: its splits go with its own launches, a product and a sum of planes each."""
    program = """
import sys, torch
sys.path[:0] = ["tests", "tiny-llm_b200"]
from test_gpu_gate_up import weight
from extensions_b200 import tiny_llm_ext_b200 as ext
gate, up = weight(2560, 2560, torch.bfloat16, 1), weight(2560, 2560, torch.bfloat16, 2)
x = torch.randn(100, 2560, device="cuda").bfloat16()
before = ext.launch_count()
got = ext.quantized_gate_up(x, gate, up)
launches = ext.launch_count() - before
one, two = (ext.quantized_matmul(w[0], w[1], 128, 4, x, w[2], True) for w in (gate, up))
assert torch.equal(got, ext.swiglu(one, two))
print(launches)
"""
    run = lambda **env: int(subprocess.run([sys.executable, "-c", program], cwd=Path(__file__).parent.parent, env={**os.environ, **env}, check=True, capture_output=True, text=True).stdout)  # noqa: E731
    assert run(TL_SKINNY_WIDE1="0") == 2 and run(TL_SKINNY_WIDE1="1") == 4
