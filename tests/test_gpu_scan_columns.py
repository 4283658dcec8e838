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
