"""Gates whose quotients come from a branch-free division where that cannot change the rounded result: to the bit what the exact division gives, whatever
the layout, for gates of all magnitudes."""

import pytest
import torch

from extensions_b200 import tiny_llm_ext_b200 as ext
from extensions_b200.tiny_llm_ext_b200 import blocks

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def spread(*shape, seed, lo=-30, hi=3):
    """Normal numbers, every eighth row scaled to another magnitude."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(*shape, generator=g, device="cuda") * 3
    x[::8] *= torch.logspace(lo, hi, x[::8].shape[0], device="cuda")[:, None]
    return x.to(BF16)


def same(got, want):
    return torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0))


def exact(gate, up, act, limit, slope):
    """Rounded from the fp32 form, whose division is exact."""
    return blocks.gated_act(torch.cat([gate, up], dim=1).float().contiguous(), act, limit, slope).to(BF16)


ACTS = [(blocks.ACT_SILU, 0.0, 1.0), (blocks.ACT_CLAMPED_SWISH, 7.0, 1.702), (blocks.ACT_CLAMPED_SWISH, 1e4, 0.01)]


@pytest.mark.parametrize("act,limit,slope", ACTS)
@pytest.mark.parametrize("rows,width", [(1, 8), (37, 1408), (2048, 1024)])
def test_gated_activation(rows, width, act, limit, slope):
    gate, up = spread(rows, width, seed=rows), spread(rows, width, seed=rows + 1, lo=-10)
    gate[0, :8] = torch.tensor([0.0, -0.0, float("inf"), float("-inf"), float("nan"), -88.0, -1e4, 1e-40])
    gu = torch.cat([gate, up], dim=1).contiguous()
    aside = torch.empty(rows, width + 1, dtype=BF16, device="cuda")[:, 1:]  # rows that 16-byte accesses cannot take
    got = blocks.gated_act(gu, act, limit, slope)
    assert same(got, exact(gate, up, act, limit, slope))
    assert same(blocks.gated_act(gu, act, limit, slope, out=aside), got)


@pytest.mark.parametrize("act,limit,slope", ACTS)
@pytest.mark.parametrize("tokens", [16, 190, 1500])
def test_experts(tokens, act, limit, slope):
    """One expert whose two products have one term each, so that their sums are exact."""
    dim, ff, lib = 64, 1032, blocks.library()
    h, wg, wu = (torch.zeros(n, dim, dtype=BF16, device="cuda") for n in (tokens, ff, ff))
    h[:, 0], h[:, 1] = spread(tokens, 1, seed=1)[:, 0], spread(tokens, 1, seed=2, lo=-10)[:, 0]
    wg[:, 0], wu[:, 1] = spread(ff, 1, seed=3, lo=-2, hi=0)[:, 0], spread(ff, 1, seed=4, lo=-2, hi=0)[:, 0]
    idx = torch.zeros(tokens, 1, dtype=torch.int32, device="cuda")
    lists = torch.empty(int(lib.tlb_moe_lists_ints(tokens, 1, 1)), dtype=torch.int32, device="cuda")
    rows = int(lib.tlb_moe_max_rows(tokens, 1, 1))
    inter = torch.zeros(rows, ff, dtype=BF16, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.tlb_moe_sort(idx.data_ptr(), tokens, 1, 1, lists.data_ptr(), stream) == 0
    assert lib.tlb_moe_gate_up(h.data_ptr(), wg.data_ptr(), wu.data_ptr(), lists.data_ptr(), tokens, 1, 1, dim, ff, act, limit, slope, inter.data_ptr(), blocks._code(BF16), stream) == 0
    used = int(lists[1])
    pair, inter = lists[-rows:][:used], inter[:used]
    live = pair >= 0
    token = pair[live].long()
    p, q = h[:, :1].float() * wg[:, 0].float(), h[:, 1:2].float() * wu[:, 1].float()
    want = blocks.gated_act(torch.cat([p, q], dim=1).contiguous(), act, limit, slope).to(BF16)
    assert int(live.sum()) == tokens and same(inter[live], want[token])


@pytest.mark.parametrize("dv", [64, 128, 512])
def test_gate_behind_a_head_norm(dv):
    """Heads of ones have a norm of one: what is left is the gate."""
    tokens, heads = 700, 4
    gate = spread(tokens, heads * dv, seed=dv)
    o = torch.ones(tokens, heads, dv, device="cuda")
    got = blocks.head_norm_gate(o, None, 0.0, gate)
    assert same(got, exact(gate, torch.ones_like(gate), blocks.ACT_SILU, 0.0, 1.0))


@pytest.mark.parametrize("M,gain", [(130, 0.2), (600, 40.0), (1024, 0.2)])
def test_packed_products_of_fp16(M, gain):
    """Results from fp16's subnormal numbers to beyond its largest, on thread-block pairs: as two products and their activation."""
    N, K = 256, 1032
    g = torch.Generator(device="cuda").manual_seed(M)

    def weight(scale):
        scales = (torch.randn(K, N // 128, generator=g, device="cuda") * scale / N**0.5).half()
        words = torch.randint(-(2**31), 2**31 - 1, (K, N // 8), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
        return scales, (scales.float() * -7.5).half(), words

    gate, up = weight(gain), weight(0.2)
    x = torch.randn(M, N, generator=g, device="cuda").half()
    x[: M // 2] *= torch.logspace(-6, 3, M // 2, device="cuda").half()[:, None]
    x[5], x[6, 3], x[7, 9] = 0, float("inf"), float("nan")
    product = lambda w: ext.quantized_matmul(w[0], w[1], 128, 4, x, w[2], True, True, True)  # noqa: E731
    assert same(ext.quantized_gate_up(x, gate, up, (True, True), (True, True)), ext.swiglu(product(gate), product(up)))
