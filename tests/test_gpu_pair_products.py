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


@pytest.mark.parametrize("M,N,K", [(129, 4096, 2560), (300, 9728, 264), (512, 9728, 1004), (300, 9728, 1001)])
def test_gated_products_whose_reductions_run_in_pieces(M, N, K):
    gate, up = weight(K, N, torch.bfloat16, 1), weight(K, N, torch.bfloat16, 2)
    x = torch.randn(M, N, generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").bfloat16()
    part = lambda w: (w.scales, w.biases, w.weight)  # noqa: E731
    want = ext.swiglu(quantized_linear(x, gate), quantized_linear(x, up))
    assert torch.equal(ext.quantized_gate_up(x, part(gate), part(up), (True, True), (True, True)), want)


def unpacked(w):
    """The weights as the kernels see them: code x scale + bias in fp32, rounded to the storage type."""
    words = w.weight
    codes = ((words.unsqueeze(-1) >> torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)) & 15).reshape(words.shape[0], -1, 128).float()
    return (codes * w.scales.float()[..., None] + w.biases.float()[..., None]).to(w.scales.dtype).reshape(words.shape[0], -1)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(129, 9728, 2560), (256, 4096, 1000), (257, 3072, 1028), (300, 9728, 264), (512, 6144, 2048), (700, 9728, 1004), (1024, 6144, 512), (300, 9728, 1001)])
def test_reductions_in_runs(M, N, K, dtype):
    """Planes of ragged sizes against 64 bits, no further off than the product in one run, the same bits every time.  1001 columns: not cut."""
    w = weight(K, N, dtype, M)
    x = torch.randn(M, N, generator=torch.Generator(device="cuda").manual_seed(K), device="cuda").to(dtype)
    want = x.double() @ unpacked(w).double().t()
    code = {torch.float16: 1, torch.bfloat16: 2}[dtype]
    assert (ext._lib.tl_quantized_matmul_workspace(M, N, K, code, 1, 1) > 0) == (K % 4 == 0)
    got = quantized_linear(x, w)
    assert torch.equal(quantized_linear(x, w), got)
    try:
        ext.set_gemm_pairs(0)
        whole = quantized_linear(x, w)
    finally:
        ext.set_gemm_pairs(1)
    error = lambda y: float((y.double() - want).norm() / want.norm())  # noqa: E731
    # the output's rounding is 2^-9 (2^-12) an entry at most, 0.4 of that in the mean; what the sums leave is a hundredth of it
    assert error(got) <= 1.01 * error(whole) and error(got) < (2.0**-9 if dtype == torch.bfloat16 else 2.0**-12)


def test_runs_on_two_streams_do_not_share_planes():
    w = weight(2560, 9728, torch.bfloat16, 1)
    xs = [torch.randn(m, 9728, device="cuda").bfloat16() for m in (140, 300)]
    want = [quantized_linear(x, w) for x in xs]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in xs], [[], []]
    for _ in range(20):
        for i, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                got[i].append(quantized_linear(xs[i], w))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i]) for i in range(2) for y in got[i])


def test_planes_belong_to_the_stream_that_works_in_them():
    """Memory that the current stream has freed and has yet to write is no place for another stream's planes."""
    w = weight(2560, 9728, torch.bfloat16, 1)
    x = torch.randn(300, 9728, device="cuda").bfloat16()
    want, side = quantized_linear(x, w), torch.cuda.Stream()
    part = (w.scales, w.biases, 128, 4, x, w.weight, True, True, True)
    ext.quantized_matmul(*part, stream=side)
    torch.cuda.synchronize()
    late = [torch.empty(n * 300 * 2560, device="cuda") for n in range(2, 13)]  # as large as the planes of 2 to 12 runs
    torch.cuda._sleep(2_000_000)
    for t in late:
        t.fill_(float("nan"))
    del t, late
    got = ext.quantized_matmul(*part, stream=side)
    torch.cuda.synchronize()
    assert torch.equal(got, want)


def test_without_memory_for_planes_the_reduction_stays_whole(monkeypatch):
    w = weight(2560, 9728, torch.bfloat16, 1)
    x = torch.randn(300, 9728, device="cuda").bfloat16()
    try:
        ext.set_gemm_pairs(0)
        want = quantized_linear(x, w)
    finally:
        ext.set_gemm_pairs(1)

    def empty(*args, **kwargs):
        raise torch.OutOfMemoryError

    monkeypatch.setattr(ext.torch, "empty", empty)
    got = quantized_linear(x, w)
    monkeypatch.undo()
    # whole reductions have the same bits on either kernel
    assert torch.equal(got, want)
