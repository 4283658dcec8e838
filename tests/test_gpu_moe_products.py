"""The experts' grouped products on the tensor cores against float64: chunk sizes around the tile's edges, feature counts that are
no multiple of a weight block, reductions that end inside one, experts with no token, one token and more than a chunk holds."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def choices(tokens, top, experts, skew, gen):
    """Expert ids per token without repeats; ``skew``: every token names expert 1 first."""
    idx = torch.rand(tokens, experts, generator=gen).argsort(dim=1)[:, :top]
    if skew:
        idx = torch.where(idx == 1, idx[:, :1], idx)
        idx[:, 0] = 1
    return idx.to(torch.int32)


def reference(h, idx, gate, wg, wu, wd, act, scale_input):
    """In float64, with the operands' bf16 rounding of the intermediate left out (that is the tolerance)."""
    h, wu, wd = h.double(), wu.double(), wd.double()
    out = torch.zeros(h.shape[0], wd.shape[1], dtype=torch.float64, device=h.device)
    for e in range(wu.shape[0]):
        t, slot = (idx == e).nonzero(as_tuple=True)
        if not t.numel():
            continue
        g = gate[t, slot].double()[:, None]
        x = h[t] * g if scale_input else h[t]
        u = x @ wu[e].t()
        inner = torch.nn.functional.silu(x @ wg[e].double().t()) * u if wg is not None else torch.relu(u).square() if act == 2 else torch.nn.functional.silu(u)
        out.index_add_(0, t, (inner @ wd[e].t()) * (1.0 if scale_input else g))
    return out


@pytest.mark.parametrize("tokens,top,experts,dim,ff,gated,scale_input,skew", [
    (1, 1, 4, 64, 128, True, False, False),
    (15, 2, 5, 72, 40, True, False, False),
    (16, 3, 8, 200, 136, True, False, True),
    (17, 2, 4, 128, 264, False, False, False),
    (33, 1, 64, 264, 256, True, False, False),
    (130, 4, 6, 192, 392, True, False, True),
    (129, 2, 3, 136, 128, False, True, True),
    (257, 2, 4, 320, 200, True, False, True),
    (700, 3, 9, 512, 384, True, False, True),
    (1100, 2, 7, 256, 640, False, True, True),
])
def test_products(tokens, top, experts, dim, ff, gated, scale_input, skew):
    from extensions_b200.tiny_llm_ext_b200 import blocks

    gen = torch.Generator().manual_seed(tokens * 31 + top)
    bf = lambda *s, std=1.0: (torch.randn(*s, generator=gen) * std).to(torch.bfloat16).to(DEV)  # noqa: E731
    h, wu, wd = bf(tokens, dim), bf(experts, ff, dim, std=dim**-0.5), bf(experts, dim, ff, std=ff**-0.5)
    wg = bf(experts, ff, dim, std=dim**-0.5) if gated else None
    idx = choices(tokens, top, experts, skew, gen).to(DEV)
    gate = torch.rand(tokens, top, generator=gen).to(DEV)
    act = blocks.ACT_SILU if gated else blocks.ACT_RELU_SQUARED
    got = blocks.moe_experts(h, idx, gate, wg, wu, wd, act, scale_input=scale_input)
    want = reference(h, idx, gate, wg, wu, wd, act, scale_input)
    # the intermediate (and the scaled input) is rounded to bf16 once: 2^-9 an entry, times 2 for the square, random over the sum
    rel = float((got.double() - want).norm() / want.norm())
    assert rel < 2.0**-7, rel
    worst = float((got.double() - want).abs().max() / want.abs().max())
    assert worst < 2.0**-6, worst
    assert blocks.library().tlb_tc_gave_up() == 0


def test_a_token_does_not_depend_on_its_batch():
    """Whatever chunk a token's rows fall into, its result has the same bits."""
    from extensions_b200.tiny_llm_ext_b200 import blocks

    gen = torch.Generator().manual_seed(5)
    bf = lambda *s, std=1.0: (torch.randn(*s, generator=gen) * std).to(torch.bfloat16).to(DEV)  # noqa: E731
    experts, dim, ff, tokens = 5, 264, 200, 400
    h, wg, wu, wd = bf(tokens, dim), bf(experts, ff, dim, std=0.06), bf(experts, ff, dim, std=0.06), bf(experts, dim, ff, std=0.07)
    idx = choices(tokens, 2, experts, False, gen).to(DEV)
    gate = torch.rand(tokens, 2, generator=gen).to(DEV)
    whole = blocks.moe_experts(h, idx, gate, wg, wu, wd, blocks.ACT_SILU)
    for n in (1, 16, 37, 150, 300):
        part = blocks.moe_experts(h[:n].contiguous(), idx[:n].contiguous(), gate[:n].contiguous(), wg, wu, wd, blocks.ACT_SILU)
        assert torch.equal(part, whole[:n]), n


@pytest.mark.parametrize("tokens,top,experts", [(1, 1, 1), (40, 2, 3), (5000, 4, 300), (16, 6, 4096)])
def test_lists(tokens, top, experts):
    """Every pair whose expert exists is listed once, under its expert, in the tiles and in the chunks."""
    from extensions_b200.tiny_llm_ext_b200 import blocks

    lib = blocks.library()
    idx = torch.randint(-1, experts + 2, (tokens, top), generator=torch.Generator().manual_seed(tokens), dtype=torch.int32).to(DEV)
    lists = torch.full((int(lib.tlb_moe_lists_ints(tokens, top, experts)),), -7, dtype=torch.int32, device=DEV)
    assert lib.tlb_moe_sort(idx.data_ptr(), tokens, top, experts, lists.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    flat, at = idx.flatten().tolist(), lists.tolist()
    rows_max = int(lib.tlb_moe_max_rows(tokens, top, experts))
    tiles, rows, chunks = at[:3]
    tile_expert, pair = at[-rows_max - rows_max // 32 : -rows_max], at[-rows_max:]
    assert rows == tiles * 32 <= rows_max
    seen = {}
    for r in range(rows):
        if pair[r] >= 0:
            assert flat[pair[r]] == tile_expert[r // 32]
            seen[pair[r]] = r
    assert sorted(seen) == [p for p, e in enumerate(flat) if 0 <= e < experts]
    covered = []
    for i in range(chunks):
        e, first, n, _ = at[4 + 4 * i : 8 + 4 * i]
        assert 0 < n <= 256 and first % 16 == 0
        assert all(flat[pair[r]] == e for r in range(first, first + n))
        covered += range(first, first + n)
    assert sorted(covered) == sorted(seen.values())


def test_calls_that_follow_one_another_closely():
    """A call's launches start while the one before is ending: of many sizes in a row, with nothing waited for, and replayed from a graph, the same bits as one by one."""
    from extensions_b200.tiny_llm_ext_b200 import blocks

    gen = torch.Generator().manual_seed(5)
    bf = lambda *s, std=1.0: (torch.randn(*s, generator=gen) * std).to(torch.bfloat16).to(DEV)  # noqa: E731
    experts, dim, ff, top = 8, 256, 200, 3
    wg, wu, wd = bf(experts, ff, dim, std=dim**-0.5), bf(experts, ff, dim, std=dim**-0.5), bf(experts, dim, ff, std=ff**-0.5)
    parts = [(bf(n, dim), choices(n, top, experts, n % 2 == 0, gen).to(DEV), torch.rand(n, top, generator=gen).to(DEV)) for n in (1, 16, 40, 300, 17, 700, 2)]
    run = lambda i: blocks.moe_experts(*parts[i], wg, wu, wd, blocks.ACT_SILU)  # noqa: E731
    want = []
    for i in range(len(parts)):
        torch.cuda.synchronize()
        want.append(run(i).clone())
    torch.cuda.synchronize()
    got = [[run(i) for i in range(len(parts))] for _ in range(10)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        replayed = [run(i) for i in range(len(parts))]
    for _ in range(10):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i]) for row in got + [replayed] for i, y in enumerate(row))
