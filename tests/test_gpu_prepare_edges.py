"""What stands between the projections and the attention, at its edges: heads for more warps than a CTA has, heads longer than a warp's registers, one head, a page that
is not there; and the rotation's table where it is longer than a CTA."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def normed(x, w, eps):
    x = x.double()
    return x / (x.pow(2).mean(-1, keepdim=True) + eps).sqrt() * w.double()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads,kv_heads,dk,dv,q_normed,k_normed", [
    (16, 4, 192, 128, True, True), (40, 8, 33, 7, True, True), (31, 1, 256, 64, True, False), (5, 5, 257, 32, True, True), (1, 1, 300, 40, True, True), (4, 4, 64, 64, False, True), (3, 35, 16, 16, True, False),
])
def test_norms_per_head(dtype, heads, kv_heads, dk, dv, q_normed, k_normed):
    from extensions_b200.tiny_llm_ext_b200 import blocks

    g = torch.Generator(device="cuda").manual_seed(heads * dk)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)  # noqa: E731
    T, page, eps = 9, 4, 1e-5
    q, k, v = draw(T, heads, dk + 3)[..., :dk], draw(T, kv_heads, dk), draw(T, kv_heads, dv + 1)[..., :dv]
    wq, wk = draw(dk) if q_normed else None, draw(dk) if k_normed else None
    table = torch.tensor([[2, -1, 0]], dtype=torch.int32, device="cuda")  # tokens 4 to 7 have no page
    pos = torch.arange(T, dtype=torch.int32, device="cuda")
    slab, before = torch.zeros((3, page, kv_heads * (dk + dv)), dtype=dtype, device="cuda"), q.clone()
    blocks.kv_prepare(q, k, v, q_norm=wq, k_norm=wk, eps=eps, tok_pos=pos, tok_seq=torch.zeros_like(pos), block_table=table, slab=slab)
    # a rounding of the result; fp32: of its sum of dk squares and two products
    tol = dict(rtol=2.0**-8, atol=1e-6) if dtype == torch.bfloat16 else dict(rtol=1e-5, atol=1e-6)
    if q_normed:
        torch.testing.assert_close(q.double(), normed(before, wq, eps), **tol)
    else:
        assert torch.equal(q, before)
    want = torch.zeros_like(slab, dtype=torch.float64)
    for t in (0, 1, 2, 3, 8):
        want[table[0, t // page], t % page] = torch.cat([(normed(k[t], wk, eps) if k_normed else k[t].double()).flatten(), v[t].double().flatten()])
    torch.testing.assert_close(slab.double(), want, **tol)


@pytest.mark.parametrize("dk,interleaved", [(256, False), (512, False), (264, True)])
def test_a_table_longer_than_the_row(dk, interleaved):
    """One head, queries alone, all of it rotated: the same bits as from rows that no 16-byte access fits."""
    from extensions_b200.tiny_llm_ext_b200 import blocks

    T = 5
    q = torch.randn(T, dk, generator=torch.Generator(device="cuda").manual_seed(dk), device="cuda").bfloat16()
    pos = torch.arange(3, 3 + T, dtype=torch.int32, device="cuda")
    odd = torch.zeros(T, dk + 1, dtype=torch.bfloat16, device="cuda")
    odd[:, :dk] = q
    for rows in (q, odd[:, :dk]):
        blocks.qk_whole_prepare(rows, None, None, heads=1, kv_heads=1, rot_dims=dk, interleaved=interleaved, tok_pos=pos, rope=blocks.rope_table(pos, dims=dk, base=1e4))
    assert torch.equal(q, odd[:, :dk])
