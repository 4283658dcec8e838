"""The latent layer's own route to keys and values up-projected per head: through a page slab, with a window (rows that no query sees are
left out), sinks and a query latent, against the absorbed form; and back to that form when the buffers cannot be had."""

import pytest
import torch

from tiny_llm_b200 import latent_attention
from tiny_llm_b200.latent_attention import LatentAttention
from tiny_llm_b200.latent_kv_cache import LatentPagedCache, LatentPagedPool
from tiny_llm_b200.ragged import RaggedEntry, RaggedPlan

pytestmark = pytest.mark.gpu
DEV, PAGE = "cuda", 64


def step(counts, starts, *, heads=8, dim=128, rot=64, vdim=128, rank=256, width=512, window=None, sink=False, q_rank=0, seed=0):
    gen = torch.Generator().manual_seed(seed)
    bf = lambda *s, std=1.0: (torch.randn(*s, generator=gen) * std).to(torch.bfloat16).to(DEV)  # noqa: E731
    weights = dict(w_q=bf(heads * (dim + rot), q_rank or width, std=2 * (q_rank or width) ** -0.5), w_dkv=bf(rank + rot, width, std=2 * width**-0.5), dkv_norm=1 + bf(rank, std=0.1),
                   w_uk=bf(heads * dim, rank, std=rank**-0.5), w_uv=bf(heads * vdim, rank, std=rank**-0.5), w_o=bf(width, heads * vdim, std=(heads * vdim) ** -0.5))
    if q_rank:
        weights.update(w_q_down=bf(q_rank, width, std=width**-0.5), q_down_norm=1 + bf(q_rank, std=0.1))
    layer = LatentAttention(heads=heads, dim=dim, rot_dim=rot, vdim=vdim, kv_rank=rank, scale=(dim + rot) ** -0.5, rot_dims=rot, rot_base=10000.0, interleaved=False,
                            window=window, sink=torch.randn(heads, generator=gen).to(DEV) if sink else None, **weights)
    pool = LatentPagedPool([layer.cache_width], page_size=PAGE, dtype=torch.bfloat16, device=DEV, max_pages=sum(-(-(n + s) // PAGE) for n, s in zip(counts, starts)) + 3)
    pool.slabs[0].fill_(float("nan"))  # what an earlier owner of a page may have left
    owners = [LatentPagedCache(pool) for _ in starts]
    for owner, n in zip(owners, starts):
        if n:
            owner.append_slots(n)
            rows = bf(n, layer.cache_width)
            for i, page in enumerate(owner.page_ids):
                part = rows[i * PAGE : (i + 1) * PAGE]
                pool.slabs[0][page, : part.shape[0]] = part
    plan = RaggedPlan([RaggedEntry([0] * n, [o], want=[]) for n, o in zip(counts, owners)], DEV, [layer.attention_kernel(pool.slabs[0])[1]])
    return layer, bf(sum(counts), width), plan, pool.slabs[0]


CASES = [
    # new tokens, cached before; how many rows are up-projected
    (dict(), [1200, 198], [0, 1025], 64 * (19 + 20)),
    (dict(window=256), [700, 1, 300], [1000, 500, 0], 64 * (27 - 11 + 8 - 3 + 5)),
    (dict(window=100, sink=True, rank=512), [600, 200], [64, 333], 64 * (11 + 9 - 3)),
    (dict(sink=True, q_rank=192), [900], [100], 64 * 16),
    (dict(window=512, q_rank=128, rank=512, dim=64, rot=32, vdim=64, heads=16), [1024], [3000], 64 * (63 - 38)),
    (dict(window=1024, heads=16, rank=512), [2048], [30000], 64 * (501 - 452)),
]


@pytest.mark.parametrize("sizes,counts,starts,rows", CASES)
def test_layer_takes_the_rows_that_are_seen(sizes, counts, starts, rows, monkeypatch):
    from extensions_b200.tiny_llm_ext_b200 import blocks

    layer, h, plan, slab = step(counts, starts, **sizes)
    taken, call = [], blocks.latent_attention_heads
    monkeypatch.setattr(blocks, "latent_attention_heads", lambda q, k, *a, **kw: taken.append(k.shape[0]) or call(q, k, *a, **kw))
    got = layer(h, plan, slab).double()
    assert taken == [rows]
    layer.tc = False
    want = layer(h, plan, slab).double()
    assert len(taken) == 1 and torch.isfinite(got).all()
    # either form rounds about five tensors on its way to bf16 (2^-9 each, root mean square below that)
    assert float((got - want).norm() / want.norm()) < 2.0**-6
    assert blocks.library().tlb_tc_gave_up() == 0


@pytest.mark.parametrize("where", ["linear", "bmm"])
def test_without_memory_for_the_buffers_the_layer_runs_the_absorbed_form(where, monkeypatch):
    layer, h, plan, slab = step([1200, 198], [0, 1025])
    layer.tc = False
    want = layer(h, plan, slab)
    layer.tc = True
    assert layer._per_head(plan, h.new_empty(h.shape[0], layer.heads, layer.dim + layer.rot_dim))
    real, rows = {"linear": latent_attention.linear, "bmm": torch.bmm}[where], 64 * (19 + 20)

    def short_of_memory(a, *rest, **kw):
        if a.shape[-2] == rows:
            raise torch.OutOfMemoryError("CUDA out of memory")
        return real(a, *rest, **kw)

    monkeypatch.setattr(latent_attention if where == "linear" else torch, where, short_of_memory)
    assert torch.equal(layer(h, plan, slab), want)
