"""The tcgen05 attention kernel of prompt portions against float64: every mask, weight and gate, head sizes that end inside a 64-column
block, runs that end inside a tile, groups that do not divide 128, pages in any order with stale (NaN) rows past the context, and a
bad table entry; and the latent layers' form with keys and values up-projected per head."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def reference(q, k, v, pos, *, scale, see, cap=0.0, sink=None, sigmoid_bias=None):
    """``q [n, H, dk]``, ``k [m, G, dk]``, ``v [m, G, dv]`` float64, ``see [n, m]``."""
    group = q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(group, dim=1), v.repeat_interleave(group, dim=1)
    s = torch.einsum("nhd,mhd->hnm", q, k) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    if sigmoid_bias is not None:
        p = torch.where(see, torch.sigmoid(s + sigmoid_bias[:, None, None]), 0.0)
    else:
        s = s.masked_fill(~see, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(-1, s.shape[1], 1)], dim=2)
        p = torch.softmax(s, dim=2)[:, :, : k.shape[0]]
    return torch.einsum("hnm,mhd->nhd", p, v)


def visible(pos, m, mask, size, keep):
    i, j = pos[:, None], torch.arange(m, device=pos.device)[None, :]
    see = j <= i
    if mask == 1:
        see = see & ((i - j < size) | (j < keep))
    if mask == 2:
        see = see & (i // size == j // size)
    return see


CASES = [
    # heads, kv_heads, dk, dv, page, counts, starts, mask, size, keep, cap, sink, gate, sigmoid
    (4, 4, 64, 64, 64, [40], [0], 0, 0, 0, 0.0, "", "", False),
    (8, 2, 128, 128, 64, [33, 1, 200], [0, 70, 129], 0, 0, 0, 0.0, "", "head", False),
    (16, 4, 128, 128, 128, [150, 64], [0, 900], 1, 100, 16, 0.0, "bias", "head", False),
    (16, 4, 192, 128, 64, [127, 3, 65], [1, 300, 0], 2, 96, 0, 30.0, "zero", "head", False),
    (8, 2, 96, 64, 64, [300], [17], 1, 64, 0, 30.0, "zero", "wide", False),
    (6, 2, 72, 40, 64, [129, 20], [0, 63], 0, 0, 0, 0.0, "", "", False),
    (10, 2, 256, 256, 64, [60], [500], 0, 0, 0, 0.0, "bias", "", False),
    (12, 4, 64, 192, 192, [100, 31], [0, 1000], 1, 200, 70, 0.0, "", "", False),
    (8, 2, 128, 128, 64, [90, 40], [0, 333], 2, 128, 0, 0.0, "bias", "", True),
    (128, 1, 64, 64, 64, [5], [100], 0, 0, 0, 0.0, "", "", False),
    (4, 2, 128, 128, 64, [40] * 40, list(range(0, 400, 10)), 0, 0, 0, 0.0, "", "head", False),
]


@pytest.mark.parametrize("case", CASES)
def test_paged(case):
    from extensions_b200.tiny_llm_ext_b200 import blocks

    H, G, dk, dv, page, counts, starts, mask, size, keep, cap, sink, gate, sigmoid = case
    gen = torch.Generator().manual_seed(len(counts) * 100 + dk)
    bf = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16).to(DEV)  # noqa: E731
    T = sum(counts)
    wide_q = bf(T, H * dk + 16)  # queries as columns of a wider product
    q = wide_q[:, : H * dk].unflatten(1, (H, dk))
    pages = [-(-(n + s) // page) for n, s in zip(counts, starts)]
    order = torch.randperm(sum(pages), generator=gen).int()
    slab = torch.full((sum(pages), page, G * (dk + dv)), float("nan"), dtype=torch.bfloat16, device=DEV)
    table = torch.full((len(counts), max(pages)), -1, dtype=torch.int32)
    info, at, first, keys = [], 0, 0, []
    for s, (n, start) in enumerate(zip(counts, starts)):
        table[s, : pages[s]] = order[at : at + pages[s]]
        rows = bf(n + start, G * (dk + dv))
        keys.append(rows)
        for i in range(pages[s]):
            part = rows[i * page : (i + 1) * page]
            slab[int(table[s, i]), : part.shape[0]] = part
        info.append((first, n, start, -1))
        at, first = at + pages[s], first + n
    # not 16-byte aligned, as inside a step's one block of integers
    info = torch.tensor([0] + [v for row in info for v in row], dtype=torch.int32, device=DEV)[1:].view(-1, 4)
    bias = torch.randn(H, generator=gen).to(DEV) if sink == "bias" or sigmoid else None
    logits = bf(T, H) if gate == "head" else bf(T, H * dv) if gate == "wide" else None
    run = blocks.flash_tc_run(torch.bfloat16, H, G, dk, dv, page)
    assert run == 128 // (H // G)
    runs = sum(-(-n // run) for n in counts)
    got = blocks.paged_attention_tc(q, slab, table.to(DEV), info, runs + 2, kv_heads=G, dv=dv, mask=mask, mask_size=size, keep_first=keep, scale=dk**-0.5, softcap=cap,
                                    sink=bool(sink) and not sigmoid, gate=logits, head_bias=bias, weights=int(sigmoid))
    first = 0
    for s, (n, start) in enumerate(zip(counts, starts)):
        pos = torch.arange(start, start + n, device=DEV)
        rows = keys[s].double()
        want = reference(q[first : first + n].double(), rows[:, : G * dk].view(-1, G, dk), rows[:, G * dk :].view(-1, G, dv), pos, scale=dk**-0.5,
                         see=visible(pos, n + start, mask, size, keep), cap=cap,
                         sink=None if not sink or sigmoid else bias.double() if sink == "bias" else torch.zeros(H, dtype=torch.float64, device=DEV),
                         sigmoid_bias=bias.double() if sigmoid else None)
        if logits is not None:
            w = torch.sigmoid(logits[first : first + n].double())
            want = want * (w[:, :, None] if gate == "head" else w.view(n, H, dv))
        part = got[first : first + n].double()
        assert torch.isfinite(part).all()
        # P and the output are rounded to bf16 once each (2^-9 an entry); tanh.approx under a cap: 2^-11 of up to 30, in the exponent
        assert float((part - want).norm() / want.norm()) < (2.0**-7 if not cap else 2.0**-5), s
        first += n
    assert blocks.library().tlb_tc_gave_up() == 0


def test_bad_table_entry_reads_as_zeros():
    from extensions_b200.tiny_llm_ext_b200 import blocks

    gen = torch.Generator().manual_seed(1)
    q, slab = torch.randn(20, 2, 64, generator=gen).to(torch.bfloat16).to(DEV), torch.randn(2, 64, 2 * 128, generator=gen).to(torch.bfloat16).to(DEV)
    info = torch.tensor([[0, 20, 100, -1]], dtype=torch.int32, device=DEV)
    run = lambda table: blocks.paged_attention_tc(q, slab, torch.tensor([table], dtype=torch.int32, device=DEV), info, 1, kv_heads=2, dv=64, mask=0, mask_size=0, scale=0.125)  # noqa: E731
    bad = run([7, 1])
    slab[0] = 0
    assert torch.equal(bad, run([0, 1])) and torch.equal(bad, run([-1, 1]))


@pytest.mark.parametrize("heads,dim,rot,dv,rank,counts,starts,window,sink", [
    (4, 64, 32, 64, 72, [130, 1, 40], [0, 200, 64], 0, False),
    (3, 128, 64, 128, 512, [200], [77], 0, True),
    (16, 128, 64, 128, 256, [64, 129], [300, 0], 100, False),
    (2, 64, 0, 48, 40, [31], [0], 0, False),
    (5, 192, 64, 200, 64, [70], [10], 64, True),
])
def test_latent_heads(heads, dim, rot, dv, rank, counts, starts, window, sink):
    from extensions_b200.tiny_llm_ext_b200 import blocks

    gen = torch.Generator().manual_seed(heads)
    bf = lambda *s, std=1.0: (torch.randn(*s, generator=gen) * std).to(torch.bfloat16).to(DEV)  # noqa: E731
    page, T = 32, sum(counts)
    q = bf(T, heads * (dim + rot)).unflatten(1, (heads, dim + rot))
    w_uk, w_uv = bf(heads * dim, rank, std=rank**-0.5), bf(heads, rank, dv, std=rank**-0.5)
    bias = torch.randn(heads, generator=gen).to(DEV) if sink else None
    pages = [-(-(n + s) // page) for n, s in zip(counts, starts)]
    slab = torch.full((sum(pages), page, rank + rot), float("nan"), dtype=torch.bfloat16, device=DEV)
    table = torch.full((len(counts), max(pages)), -1, dtype=torch.int32)
    info, at, first, caches = [], 0, 0, []
    for s, (n, start) in enumerate(zip(counts, starts)):
        table[s, : pages[s]] = torch.arange(at, at + pages[s]).flip(0)
        caches.append(bf(n + start, rank + rot))
        for i in range(pages[s]):
            part = caches[-1][i * page : (i + 1) * page]
            slab[int(table[s, i]), : part.shape[0]] = part
        info.append((first, n, start, -1))
        at, first = at + pages[s], first + n
    info = torch.tensor(info, dtype=torch.int32, device=DEV)
    rows, where = blocks.latent_rows(slab, table.to(DEV), info, [n + s for n, s in zip(counts, starts)])
    c = rows[:, :rank]
    scale = (dim + rot) ** -0.5
    got = blocks.latent_attention_heads(q, c @ w_uk.t(), torch.bmm(c.expand(heads, -1, -1), w_uv), rows[:, rank:], where, info, sum(-(-n // 128) for n in counts), dim=dim,
                                        window=window, scale=scale, sink=bias)
    first = 0
    for s, (n, start) in enumerate(zip(counts, starts)):
        cache = caches[s].double()
        k = torch.cat([(cache[:, :rank] @ w_uk.double().t()).view(-1, heads, dim), cache[:, None, rank:].expand(-1, heads, -1)], dim=2)
        v = torch.einsum("nr,hrd->nhd", cache[:, :rank], w_uv.double())
        pos = torch.arange(start, start + n, device=DEV)
        want = reference(q[first : first + n].double(), k, v, pos, scale=scale, see=visible(pos, n + start, 1 if window else 0, window, 0), sink=None if bias is None else bias.double())
        # keys, values, P and the output rounded to bf16 once each
        assert float((got[first : first + n].double() - want).norm() / want.norm()) < 2.0**-6, s
        first += n
    assert blocks.library().tlb_tc_gave_up() == 0


@pytest.mark.parametrize("dk,dv,mask,size", [(128, 128, 0, 0), (192, 128, 2, 512), (64, 64, 1, 700)])
def test_weights_are_as_exact_as_against_their_own_maximum(dk, dv, mask, size):
    """Peaked scores (standard deviation 2), where the maximum grows over many tiles: no further from float64 than weights that are rounded
    against the maximum of the keys up to their own tile."""
    from extensions_b200.tiny_llm_ext_b200 import blocks

    gen = torch.Generator().manual_seed(dk)
    n, H, G, page = 1000, 8, 2, 64
    q = (2 * torch.randn(n, H, dk, generator=gen)).to(torch.bfloat16).to(DEV)
    rows = torch.randn(n, G * (dk + dv), generator=gen).to(torch.bfloat16).to(DEV)
    slab = torch.zeros(-(-n // page), page, G * (dk + dv), dtype=torch.bfloat16, device=DEV)
    slab.view(-1, G * (dk + dv))[:n] = rows
    table = torch.arange(slab.shape[0], dtype=torch.int32, device=DEV)[None]
    info = torch.tensor([[0, n, 0, -1]], dtype=torch.int32, device=DEV)
    run = blocks.flash_tc_run(torch.bfloat16, H, G, dk, dv, page)
    got = blocks.paged_attention_tc(q, slab, table, info, -(-n // run), kv_heads=G, dv=dv, mask=mask, mask_size=size, scale=dk**-0.5).double()
    r = rows.double()
    k, v, see = r[:, : G * dk].view(-1, G, dk), r[:, G * dk :].view(-1, G, dv), visible(torch.arange(n, device=DEV), n, mask, size, 0)
    want = reference(q.double(), k, v, torch.arange(n, device=DEV), scale=dk**-0.5, see=see)
    s = torch.einsum("nhd,mhd->hnm", q.double(), k.repeat_interleave(H // G, 1)) * dk**-0.5 * 1.4426950408889634
    s = s.masked_fill(~see, -math.inf)
    top = torch.nn.functional.pad(s, (0, -n % 64), value=-math.inf).view(H, n, -1, 64).amax(3).cummax(2).values.repeat_interleave(64, 2)[:, :, :n]
    p = torch.exp2((s - top).masked_fill(~see, -math.inf)).bfloat16().double() * torch.exp2(top - top[:, :, -1:]).masked_fill(~see, 0.0)
    model = (torch.einsum("hnm,mhd->nhd", p, v.repeat_interleave(H // G, 1)) / p.sum(2).t()[:, :, None]).bfloat16().double()
    assert float((got - want).norm()) < 1.02 * float((model - want).norm())  # 2 % for the 32-bit scores and sums
