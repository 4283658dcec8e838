"""The norm behind a residual projection of 9 to 128 rows whose reduction is split: its sum of squares in the order of one block of 256 threads,
whichever block adds which part of the row."""

import numpy as np
import pytest
import torch

from extensions_b200 import tiny_llm_ext_b200 as ext

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def butterfly(v):
    """The sum over the last axis as lanes exchange it: every step adds the lane 16, 8, .. further."""
    while v.shape[-1] > 1:
        half = v.shape[-1] // 2
        v = v[..., :half] + v[..., half:]
    return v[..., 0]


def sum_of_squares(x):
    """Thread t of 256 adds the squares (exact in fp32) of columns t, t + 256, ..; then its warp's 32, then the eight warps'."""
    rows, cols = x.shape
    parts = np.zeros((rows, 256), np.float32)
    for j in range(0, cols, 256):
        here = x[:, j : j + 256].float().cpu().numpy()
        parts[:, : here.shape[1]] = parts[:, : here.shape[1]] + here * here
    return torch.from_numpy(butterfly(butterfly(parts.reshape(rows, 8, 32)))).cuda()


@pytest.mark.parametrize("M", [9, 24, 77, 128])
@pytest.mark.parametrize("N,K", [(4096, 2560), (9728, 2560), (3072, 1024), (2048, 4096), (2560, 264), (2560, 1000)])
def test_the_row_is_added_in_the_order_of_one_block(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    scales = (torch.randn(K, N // 128, generator=g, device="cuda") * 0.2 / N**0.5).to(BF16)
    words = torch.randint(-(2**31), 2**31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    x, res = (torch.randn(M, n, generator=g, device="cuda").to(BF16) for n in (N, K))
    w = (1 + 0.1 * torch.randn(K, generator=g, device="cuda")).to(BF16)
    assert ext._lib.tl_quantized_matmul_fused_workspace(M, N, K, N, 0, ext._DTYPE_CODE[BF16]) > 0  # planes: the norm is in their launch
    row, normed = ext.quantized_matmul_residual_norm(scales, (scales.float() * -7.5).to(BF16), words, x, res, w, 1e-6)
    share = torch.rsqrt(sum_of_squares(row) / torch.full((M,), float(K), device="cuda") + torch.tensor(1e-6, device="cuda"))  # by a number: times its reciprocal
    assert torch.equal(normed, (row.float() * share[:, None] * w.float()).to(BF16))
