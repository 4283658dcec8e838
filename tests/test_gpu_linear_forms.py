"""The short way through ``quantized_linear`` and ``ext.quantized_matmul``: every form of a call gives what the checked call gives, and
what was refused is refused with the same words."""

import pytest
import torch

from extensions_b200 import tiny_llm_ext_b200 as ext
from tiny_llm_b200.quantize import QuantizedWeights, quantized_linear, quantized_matmul

pytestmark = pytest.mark.gpu


def weights(K=72, N=256, **flags):
    g = torch.Generator(device="cuda").manual_seed(5)
    scales = torch.randn(K, N // 128, generator=g, device="cuda").bfloat16() * 0.02
    words = torch.randint(-(2**31), 2**31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    return QuantizedWeights(scales=scales, biases=scales * -7.5, group_size=128, bits=4, weight=words, **flags)


@pytest.mark.parametrize("flags", [{}, {"use_simdgroup_matmul": True, "use_simdgroup_matvec": True}, {"use_simdgroup_matmul": True, "use_split_k_matmul": True}])
@pytest.mark.parametrize("form", ["row", "rows", "batch", "turned", "strided", "wide"])
def test_every_form_equals_the_plain_call(form, flags):
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(3, 5, 256, generator=g, device="cuda").bfloat16()
    x = {"row": x[0, 0], "rows": x[0], "batch": x, "turned": x.transpose(0, 1), "strided": torch.cat([x, x], -1)[..., ::2], "wide": x.expand(4, 3, 5, 256)}[form]
    w = weights(**flags)
    rows = x.reshape(-1, 256).contiguous()
    few = rows.shape[0] <= 8 and w.use_simdgroup_matvec
    want = ext.quantized_matmul(w.scales, w.biases, 128, 4, rows, w.weight, True, True if few else w.use_simdgroup_matmul, False if few else w.use_split_k_matmul)
    got = quantized_linear(x, w)
    assert got.shape == (*x.shape[:-1], 72) and torch.equal(got.reshape(-1, 72), want)
    bias = torch.randn(72, generator=g, device="cuda").bfloat16()
    assert torch.equal(quantized_linear(x, w, bias), got + bias)


@pytest.mark.parametrize("change,words", [
    (dict(a=lambda t: t.half()), "dtype"), (dict(a=lambda t: t[:, :128]), "column"), (dict(a=lambda t: t.cpu()), ""), (dict(b=lambda t: t.long()), "b must be uint32"),
    (dict(scales=lambda t: t.float()), "float16 or bfloat16"), (dict(biases=lambda t: t.half()), "dtype"), (dict(b=lambda t: t.t()), ""), (dict(a=lambda t: t[0]), ""),
    (dict(scales=lambda t: t[:1]), ""), (dict(a=lambda t: torch.cat([t, t], 1)[:, ::2]), "contiguous"), (dict(transpose_b=lambda t: False), "transposed"),
    (dict(bits=lambda t: 8), ""), (dict(group_size=lambda t: 64), ""),
])
def test_what_was_refused_is_refused(change, words):
    w = weights()
    call = dict(scales=w.scales, biases=w.biases, group_size=128, bits=4, a=torch.zeros(3, 256, dtype=torch.bfloat16, device="cuda"), b=w.weight, transpose_b=True)
    for name, f in change.items():
        call[name] = f(call[name])
    with pytest.raises(RuntimeError, match="quantized_matmul.*" + words):
        ext.quantized_matmul(**call)


def test_the_callers_stream_is_used():
    w, x = weights(), torch.randn(64, 256, device="cuda").bfloat16()
    want = quantized_linear(x, w)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        later = quantized_linear(x * 2, w)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(later, want * 2)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        held = quantized_linear(x, w)
    graph.replay()
    assert torch.equal(held, want)
