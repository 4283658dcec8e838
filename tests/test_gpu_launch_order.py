"""Launches that follow one another closely, each on what the one before it wrote."""

import pytest
import torch

from extensions_b200 import tiny_llm_ext_b200 as ext

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("rows", [1, 24, 128])
def test_positions_written_by_the_launch_before(rows):
    """The step's bookkeeping, then at once the rotation and append that read it, many times over: every row turned by its own position and
    every key in its own place, as when each launch is waited for."""
    Hq, Hkv, D, page, pages, steps = 16, 8, 128, 16, 4, 60
    g = torch.Generator(device="cuda").manual_seed(rows)
    normal = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(BF16)  # noqa: E731
    qkv, qw, kw = normal(steps, rows, (Hq + 2 * Hkv) * D), normal(D), normal(D)
    table = torch.randperm(rows * pages, generator=g, device="cuda").to(torch.int32).view(rows, pages)
    ints = lambda n: torch.zeros(n, dtype=torch.int32, device="cuda")  # noqa: E731

    def run(waiting):
        slabs = [torch.zeros(rows * pages, Hkv, page, D, dtype=BF16, device="cuda") for _ in range(2)]
        tokens, following, offsets, lens, log, counter = ints(rows), ints(rows), ints(rows), ints(rows) + 1, ints(steps * rows).view(steps, rows), ints(1)
        out = []
        for i in range(steps):
            ext.decode_advance(tokens, following, offsets, lens, log, counter)
            if waiting:
                torch.cuda.synchronize()
            out.append(ext.decode_qk_norm_rope_append(qkv[i], qw, kw, offsets, table, lens, *slabs, Hq, Hkv, 1e6, 1e-6))
            if waiting:
                torch.cuda.synchronize()
        return torch.stack(out), *slabs

    assert all(torch.equal(a, b) for a, b in zip(run(False), run(True)))


def test_lists_made_by_the_launch_before():
    """Experts' second product straight behind the sort of its lists, many times over lists of other routings: as when each launch is waited for."""
    from extensions_b200.tiny_llm_ext_b200 import blocks

    lib, tokens, top, experts, dim, ff = blocks.library(), 300, 3, 16, 256, 136
    g = torch.Generator(device="cuda").manual_seed(1)
    normal = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(BF16)  # noqa: E731
    choices = [torch.rand(tokens, experts, generator=g, device="cuda").argsort(dim=1)[:, :top].to(torch.int32).contiguous() for _ in range(40)]
    # rows all alike: an expert's pairs come in no particular order
    inter, wd = normal(1, ff).repeat(int(lib.tlb_moe_max_rows(tokens, top, experts)), 1), normal(experts, dim, ff)
    lists = torch.zeros(int(lib.tlb_moe_lists_ints(tokens, top, experts)), dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream

    def run(waiting):
        out = [torch.zeros(tokens * top, dim, device="cuda") for _ in choices]
        for idx, y in zip(choices, out):
            assert lib.tlb_moe_sort(idx.data_ptr(), tokens, top, experts, lists.data_ptr(), stream) == 0
            if waiting:
                torch.cuda.synchronize()
            assert lib.tlb_moe_down(inter.data_ptr(), wd.data_ptr(), lists.data_ptr(), tokens, top, experts, dim, ff, y.data_ptr(), 2, stream) == 0
            if waiting:
                torch.cuda.synchronize()
        return torch.stack(out)

    assert torch.equal(run(False), run(True))


def test_experts_with_the_switch_off():
    """``set_pdl(False)`` reaches the experts' launches; the same bits either way."""
    from extensions_b200.tiny_llm_ext_b200 import blocks

    g = torch.Generator(device="cuda").manual_seed(2)
    normal = lambda *shape: (torch.randn(*shape, generator=g, device="cuda") * shape[-1] ** -0.5).to(BF16)  # noqa: E731
    h, wg, wu, wd = normal(90, 256) * 16, normal(8, 136, 256), normal(8, 136, 256), normal(8, 256, 136)
    idx = torch.rand(90, 8, generator=g, device="cuda").argsort(dim=1)[:, :2].to(torch.int32).contiguous()
    weight = torch.rand(90, 2, generator=g, device="cuda")
    want = blocks.moe_experts(h, idx, weight, wg, wu, wd, blocks.ACT_SILU)
    try:
        ext.set_pdl(False)
        assert torch.equal(blocks.moe_experts(h, idx, weight, wg, wu, wd, blocks.ACT_SILU), want)
    finally:
        ext.set_pdl(True)
