"""The router: a token's choice and weights have the same bits however many tokens a call brings (one a CTA, or eight a CTA from 400 tokens on), for both
types, rows with and without 16-byte pieces, two or four rows of weights a warp, groups, a side output and outputs that end inside a warp's share."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("dim,experts,top,scoring,groups,side", [
    (64, 8, 2, 0, (0, 0), False), (2048, 64, 6, 0, (0, 0), True), (1024, 16, 2, 1, (0, 0), False), (1024, 16, 2, 0, (0, 0), True),
    (203, 33, 3, 2, (0, 0), True), (264, 24, 4, 2, (4, 2), False), (5008, 40, 2, 0, (0, 0), False),
])
def test_a_token_does_not_depend_on_the_others(dtype, dim, experts, top, scoring, groups, side):
    from extensions_b200.tiny_llm_ext_b200 import blocks

    g = torch.Generator(device="cuda").manual_seed(dim + experts)
    draw = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).to(dtype)  # noqa: E731
    h, w, b = draw(405, dim), draw(experts, dim, std=2 * dim**-0.5), draw(experts, std=0.3)
    aux = draw(1, dim, std=dim**-0.5) if side else None
    bias = draw(experts, std=0.1) if scoring == 2 else None
    route = lambda x: blocks.moe_route(x, w, b, top, scoring, bias, 1.0, groups, aux)  # noqa: E731
    whole = route(h)
    for n in (1, 148, 399, 400, 403):
        for part, all_ in zip(route(h[:n].contiguous()), whole):
            assert torch.equal(part, all_[:n]), n
    logits = h.double() @ w.double().t() + b.double()
    if scoring == 0:  # against 64 bits: the chosen logits are the largest, to what fp32 sums of dim terms leave open
        best = torch.topk(logits, top, dim=1).values
        mine = torch.gather(logits, 1, whole[0].long())
        assert float((best - mine).abs().max()) < 1e-5 * dim**0.5
        torch.testing.assert_close(whole[1].double(), torch.softmax(mine, dim=1), rtol=0, atol=1e-5 * dim**0.5)
