"""The prefill GEMM's cut into groups of one to four token tiles, with a last partial wave in smaller pieces: the same bits as the kernel
of thread-block pairs, which has a cut of its own, where waves end even, uneven and in the middle of a group, and at ragged sizes."""

import pytest
import torch

from extensions_b200 import tiny_llm_ext_b200 as ext

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [
    (2048, 2560, 9728), (2048, 9728, 2560), (2048, 4096, 2560), (512, 2560, 4096), (257, 256, 19000), (1153, 3200, 2600), (700, 3072, 1001),
    (384, 3328, 6300), (900, 1024, 18944), (2500, 128, 1282), (300, 2560, 130),
])
def test_equals_the_kernel_of_pairs(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    scales = (torch.randn(K, N // 128, generator=g, device="cuda") * 0.2 / N**0.5).bfloat16()
    words = torch.randint(-(2**31), 2**31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    a = torch.randn(M, N, generator=g, device="cuda").bfloat16()
    try:
        ext.set_gemm_pairs(2)
        want = ext.quantized_matmul(scales, scales * -7.5, 128, 4, a, words, True)
        ext.set_gemm_pairs(0)
        got = ext.quantized_matmul(scales, scales * -7.5, 128, 4, a, words, True)
    finally:
        ext.set_gemm_pairs(1)
    assert torch.equal(got, want)
