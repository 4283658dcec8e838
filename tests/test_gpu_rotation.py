"""Rotations whose angles the heads of a row share, against float64: fewer pairs than are shared at a time, exactly as many, and more."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def turned(x, pos, dims, base, interleaved):
    """``x [T, H, >= dims]`` with its first ``dims`` entries rotated, in float64, and the size of the terms that were added."""
    half = dims // 2
    angle = pos.double()[:, None, None] * base ** (-2.0 * torch.arange(half, dtype=torch.float64) / dims)
    c, s = angle.cos(), angle.sin()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, half), slice(half, dims))
    x, size = x.double(), x.double().abs()
    out, terms = x.clone(), torch.zeros_like(x)
    out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    terms[..., a] = terms[..., b] = size[..., a] + size[..., b]
    return out, terms


def close(got, want, terms, dtype):
    # half a unit of the stored type, and three roundings of 32 bits (cos, sin, the sum) of the terms
    unit = {torch.float32: 2.0**-24, torch.bfloat16: 2.0**-8}[dtype]
    return bool(((got.double() - want).abs() <= unit * want.abs() + 3 * 2.0**-24 * terms).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("heads,dims", [(1, 2), (3, 64), (16, 128), (2, 130), (5, 260)])
def test_latent_prepare_turns_every_head_and_the_key(heads, dims, interleaved, dtype):
    from extensions_b200.tiny_llm_ext_b200 import blocks

    T, rank, plain, page = 9, 40, 8, 4
    rot = dims + 6  # entries past the rotated ones pass
    g = torch.Generator().manual_seed(dims + heads)
    x = torch.randn(T, heads * (plain + rot) + rank + rot, generator=g).to(dtype)
    pos = torch.tensor([0, 1, 2, 3, 4, 5, 6, 7, 8], dtype=torch.int32)
    table = torch.tensor([[2, 0, 1]], dtype=torch.int32)
    slab = torch.zeros(3, page, rank + rot, dtype=dtype, device="cuda")
    q = x.cuda()
    blocks.latent_prepare(q, torch.ones(rank, dtype=dtype, device="cuda"), 1e-5, heads=heads, dim=plain, rot_dim=rot, rank=rank, rot_dims=dims,
                          interleaved=interleaved, base=300.0, tok_pos=pos.cuda(), tok_seq=torch.zeros(T, dtype=torch.int32, device="cuda"),
                          block_table=table.cuda(), slab=slab)
    q, slab = q.cpu(), slab.cpu()
    before, after = (t[:, : heads * (plain + rot)].reshape(T, heads, plain + rot) for t in (x, q))
    assert torch.equal(after[..., :plain], before[..., :plain]) and torch.equal(after[..., plain + dims :], before[..., plain + dims :])
    want, terms = turned(before[..., plain : plain + dims], pos, dims, 300.0, interleaved)
    assert close(after[..., plain : plain + dims], want, terms, dtype)
    key = x[:, heads * (plain + rot) + rank :]
    stored = slab[table[0].long()].reshape(-1, rank + rot)[:T, rank:]
    want, terms = turned(key[:, None, :dims], pos, dims, 300.0, interleaved)
    assert close(stored[:, None, :dims], want, terms, dtype) and torch.equal(stored[:, dims:], key[:, dims:])
