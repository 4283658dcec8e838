"""The decay scan's split of the state's columns among threads (four, two or one a thread), its row-wise reads and writes (whole 16-byte rows
or not) and its segments, against the recurrence in float64; and the router and the experts' sum at sizes that end inside their
strides."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,dk,dv", [(2, 64, 128), (3, 32, 66), (1, 128, 33), (2, 16, 256), (4, 48, 4), (2, 100, 130)])
@pytest.mark.parametrize("counts", [[300], [1, 70, 129, 64], [65, 3]])
def test_decay_scan_against_float64(H, dk, dv, counts, dtype):
    from extensions_b200.tiny_llm_ext_b200 import blocks

    T, g = sum(counts), torch.Generator(device="cuda").manual_seed(dk + dv)
    q, k = (torch.randn(T, H, dk, generator=g, device="cuda").to(dtype) for _ in range(2))
    v = torch.randn(T, H, dv, generator=g, device="cuda").to(dtype)
    z = torch.randn(T, H * dk, generator=g, device="cuda") + 2
    state = torch.randn(len(counts) + 1, H, dk, dv, generator=g, device="cuda")
    start, first, info = state.clone(), 0, []
    for s, n in enumerate(counts):
        info.append((first, n, 5, s + 1))
        first += n
    out = blocks.decay_scan(q, k, v, z, None, q_scale=dk**-0.5, seq_info=torch.tensor(info, dtype=torch.int32, device="cuda"), state=state)
    decay = torch.sigmoid(z.double()).view(T, H, dk)
    for first, n, _, slot in info:
        S, size = start[slot].double(), start[slot].double().abs()
        for t in range(first, first + n):
            pair = k[t].double()[:, :, None] * v[t].double()[:, None, :]
            S, size = decay[t][:, :, None] * S + pair, decay[t][:, :, None] * size + pair.abs()
            want, terms = (torch.einsum("hk,hkv->hv", x, y) * dk**-0.5 for x, y in ((q[t].double(), S), (q[t].double().abs(), size)))
            # a term passes at most n decays of a few units in 2^-24 each, n updates and the sum over the dk rows
            assert bool(((out[t].double() - want).abs() <= 2.0**-24 * (8 * n + dk) * terms).all())
        assert bool(((state[slot].double() - S).abs() <= 2.0**-24 * 8 * n * size).all())
    assert torch.equal(state[0], start[0])


@pytest.mark.parametrize("kind", [0, 2])
@pytest.mark.parametrize("H,dk,dv", [(2, 32, 32), (1, 64, 160), (3, 64, 96), (2, 32, 128)])
@pytest.mark.parametrize("counts,start", [([65], 0), ([64, 80], 63), ([200, 1, 17], 0), ([129, 128], 64)])
def test_long_portions_on_the_tensor_cores_against_float64(H, dk, dv, counts, start, kind):
    """Rows inside a fused projection, columns that end inside a warp's or a CTA's, strong and weak decays, a bias, a sequence without a slot."""
    from extensions_b200.tiny_llm_ext_b200 import blocks

    T, g = sum(counts), torch.Generator(device="cuda").manual_seed(11 + dk + dv)
    fused = torch.randn(T, H * (2 * dk + dv) + 8, generator=g, device="cuda").bfloat16()
    q, k, v = (x.unflatten(1, (H, -1)) for x in fused[:, 8:].split([H * dk, H * dk, H * dv], dim=1))
    z = torch.randn(T, H * dk, generator=g, device="cuda") * 3 - (2 if kind == 2 else 0)  # some channels forget everything within a token
    bias = torch.randn(H * dk, generator=g, device="cuda").bfloat16()
    state = torch.randn(len(counts) + 1, H, dk, dv, generator=g, device="cuda")
    before, first, info = state.clone(), 0, []
    for s, n in enumerate(counts):
        info.append((first, n, start, s + 1 if s != 1 else -1))
        first += n
    info_t = torch.tensor(info, dtype=torch.int32, device="cuda")
    out = blocks.decay_scan(q, k, v, z, bias, q_scale=dk**-0.5, seq_info=info_t, state=state, max_tokens=max(counts), tau=2.0, decay_kind=kind)
    zz = (z + bias.float()).double().view(T, H, dk)
    decay = torch.exp(-torch.exp(zz)) if kind == 2 else torch.exp(torch.nn.functional.logsigmoid(zz) / 2.0)
    for first, n, p, slot in info:
        S = before[slot].double() if p and slot > 0 else torch.zeros(H, dk, dv, dtype=torch.float64, device="cuda")
        size = S.abs()
        for t in range(first, first + n):
            pair = k[t].double()[:, :, None] * v[t].double()[:, None, :]
            S, size = decay[t][:, :, None] * S + pair, decay[t][:, :, None] * size + pair.abs()
            want, terms = (torch.einsum("hk,hkv->hv", x, y) * dk**-0.5 for x, y in ((q[t].double(), S), (q[t].double().abs(), size)))
            # a term passes at most n decays, each off by a few units in 2^-24 and, as an exponential, by that times its exponent (at most 16 where it still counts)
            assert bool(((out[t].double() - want).abs() <= 2.0**-24 * (24 * n + dk) * terms).all())
        if slot > 0:
            assert bool(((state[slot].double() - S).abs() <= 2.0**-24 * 24 * n * size).all())
    assert torch.equal(state[0], before[0]) and (len(counts) < 2 or torch.equal(state[2], before[2]))


@pytest.mark.parametrize("counts,start", [([65] * 40, 64), ([128, 65, 2, 300], 191), ([1000], 100)])
def test_portions_that_go_on_from_a_slot_and_write_it(counts, start):
    """The first segment starts from the state that the last one (of a single token, too) replaces in the end."""
    test_long_portions_on_the_tensor_cores_against_float64(2, 64, 96, counts, start, 0)


def test_a_value_that_is_no_number_stays_behind_its_token():
    from extensions_b200.tiny_llm_ext_b200 import blocks

    T, H, dk, dv, bad = 130, 2, 64, 128, 72
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(T, H, d, generator=g, device="cuda").bfloat16() for d in (dk, dk, dv))
    z = torch.randn(T, H * dk, generator=g, device="cuda")
    info = torch.tensor([(0, T, 0, 0)], dtype=torch.int32, device="cuda")
    state = torch.zeros(1, H, dk, dv, device="cuda")
    run = lambda: blocks.decay_scan(q, k, v, z, None, q_scale=1.0, seq_info=info, state=state, max_tokens=T)  # noqa: E731
    want = run()
    v[bad, 0, 5], v[bad, 1, 40] = float("inf"), float("nan")
    got = run()
    clean = torch.ones_like(got, dtype=torch.bool)
    clean[bad:, 0, 5] = clean[bad:, 1, 40] = False
    assert not got[~clean].isfinite().any() and bool(got[clean].isfinite().all())
    assert torch.allclose(got[clean], want[clean], rtol=2.0**-18, atol=2.0**-18 * float(want.abs().max()))


@pytest.mark.parametrize("dk", [32, 64])
@pytest.mark.parametrize("what", ["key", "value", "query", "decay", "state", "nothing"])
def test_infinities_stay_what_they_are_token_by_token(dk, what):
    """Against the walk, which 32-bit operands take: infinities and NaN in the same places, the rest the same up to the order of the sums."""
    from extensions_b200.tiny_llm_ext_b200 import blocks

    T, H, dv, start = 150, 2, 96, 30  # segments of 34, 64 and 52 tokens
    g = torch.Generator(device="cuda").manual_seed(5 + dk)
    q, k, v = (torch.randn(T, H, d, generator=g, device="cuda").bfloat16() for d in (dk, dk, dv))
    z = torch.randn(T, H * dk, generator=g, device="cuda") + 3
    state = torch.randn(2, H, dk, dv, generator=g, device="cuda")
    for t, sign in ((0, 1), (20, -1), (33, 1), (60, 1), (T - 1, -1)):
        if what == "key":
            k[t, t % 2, t % dk] = sign * float("inf")
        if what == "value":
            v[t, t % 2, t % dv] = sign * float("inf")
        if what == "query":
            q[t, t % 2, t % dk] = sign * float("inf")
        if what == "decay":
            z[t, t % dk] = float("nan") if sign > 0 else float("inf")
    if what == "state":
        state[1, 0, 3, 5], state[1, 1, dk - 1, dv - 1], state[1, 1, 0, 40] = float("inf"), -float("inf"), float("nan")
    info = torch.tensor([(0, T, start, 1)], dtype=torch.int32, device="cuda")

    def run(*qkv):
        s = state.clone()
        return blocks.decay_scan(*qkv, z, None, q_scale=1.0, seq_info=info, state=s, max_tokens=T), s[1]

    for got, want in zip(run(q, k, v), run(q.float(), k.float(), v.float())):
        if what == "query":  # the walk adds two parts of a segment's outputs, which may be two infinities
            assert torch.equal(got.isfinite(), want.isfinite())
        else:
            assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
        fine = want.isfinite()
        assert bool(fine.any()) and bool(fine.all()) == (what == "nothing" or (what == "query" and want.dim() == 3 and want.shape[0] == H))
        # sums of up to 2 T dk terms of the size of the largest results, in another order
        assert float((got[fine].double() - want[fine].double()).abs().max()) <= 2.0**-24 * 32 * float(want[fine].abs().max())


@pytest.mark.parametrize("act", [0, 1, 2])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,H,dv", [(1, 1, 4), (5, 3, 128), (3, 2, 132), (4, 2, 256), (2, 2, 512), (2, 2, 516), (3, 2, 66)])
def test_head_norm_and_gate_against_float64(T, H, dv, dtype, act):
    """Widths of one, two and four pieces a lane, ragged ones, and those that are not taken whole."""
    from extensions_b200.tiny_llm_ext_b200 import blocks

    g = torch.Generator(device="cuda").manual_seed(T + dv)
    o = torch.randn(T, H, dv, generator=g, device="cuda")
    gate = torch.randn(T, H * dv + 4, generator=g, device="cuda").to(dtype)[:, 4:]
    for w in (None, torch.randn(dv, generator=g, device="cuda").to(dtype), torch.randn(H * dv, generator=g, device="cuda").to(dtype)):
        for first in (False, True):
            got = blocks.head_norm_gate(o, w, 1e-5, gate, act=act, gate_first=first)
            x, y = o.double(), gate.double().view(T, H, dv)
            y = y * torch.sigmoid(y) if act == 1 else torch.sigmoid(y) if act == 2 else y
            n = x * y if first else x
            want = n * torch.rsqrt(n.square().mean(-1, keepdim=True) + 1e-5) * (1 if first else y)
            want = want.reshape(T, -1) * (1 if w is None else w.double() if w.numel() == H * dv else w.double().repeat(H))
            unit = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-20
            assert bool(((got.double() - want).abs() <= unit * want.abs() + 1e-30).all())


@pytest.mark.parametrize("T,D,E,top", [(1, 64, 8, 2), (5, 1000, 16, 2), (37, 2048, 64, 6), (150, 520, 24, 3)])
def test_router_and_expert_sum_against_float64(T, D, E, top):
    from extensions_b200.tiny_llm_ext_b200 import blocks

    g = torch.Generator(device="cuda").manual_seed(T + D)
    h, w = torch.randn(T, D, generator=g, device="cuda").bfloat16(), (torch.randn(E, D, generator=g, device="cuda") * 2 / D**0.5).bfloat16()
    idx, gate = blocks.moe_route(h, w, None, top)
    logits = h.double() @ w.double().T
    noise = 2.0**-24 * D * (h.double().abs() @ w.double().abs().T)  # of a 32-bit sum over D
    chosen = logits.gather(1, idx.long())
    kth = logits.topk(top, dim=1).values[:, -1:]
    assert bool((chosen >= kth - 2 * noise.amax(1, keepdim=True)).all()) and all(len(set(row)) == top for row in idx.tolist())
    torch.testing.assert_close(gate.double(), torch.softmax(chosen, 1), rtol=float(4 * noise.max()) + 1e-6, atol=0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,dk,dv", [(3, 128, 70), (2, 100, 33), (1, 112, 64)])
@pytest.mark.parametrize("counts", [[1, 1, 1], [64], [40, 3], [200, 70]])
def test_one_decay_per_head_against_float64(H, dk, dv, counts, dtype):
    """The form with the fewest registers: key rows that fill a thread's and such that do not, walked whole and in segments."""
    from extensions_b200.tiny_llm_ext_b200 import blocks

    T, g = sum(counts), torch.Generator(device="cuda").manual_seed(dk + dv)
    q, k = (torch.randn(T, H, dk, generator=g, device="cuda").to(dtype) for _ in range(2))
    v = torch.randn(T, H, dv, generator=g, device="cuda").to(dtype)
    decay = 0.9 + 0.1 * torch.rand(H, generator=g, device="cuda")
    state = torch.randn(len(counts), H, dk, dv, generator=g, device="cuda")
    start, first, info = state.clone(), 0, []
    for s, n in enumerate(counts):
        info.append((first, n, 30, s))
        first += n
    out = blocks.decay_scan(q, k, v, None, None, q_scale=dk**-0.5, seq_info=torch.tensor(info, dtype=torch.int32, device="cuda"), state=state, max_tokens=max(counts),
                            head_decay=decay)
    a = decay.double()[:, None, None]
    for first, n, _, slot in info:
        S, size = start[slot].double(), start[slot].double().abs()
        for t in range(first, first + n):
            pair = k[t].double()[:, :, None] * v[t].double()[:, None, :]
            S, size = a * S + pair, a * size + pair.abs()
            want, terms = (torch.einsum("hk,hkv->hv", x, y) * dk**-0.5 for x, y in ((q[t].double(), S), (q[t].double().abs(), size)))
            # a term passes at most n decays and n updates of half a unit each and the sum over the dk rows
            assert bool(((out[t].double() - want).abs() <= 2.0**-24 * (8 * n + dk) * terms).all())
        assert bool(((state[slot].double() - S).abs() <= 2.0**-24 * 8 * n * size).all())
