"""The barrier protocol of the TMA-fed kernels, every interleaving of it.

``mbarrier.try_wait.parity`` passes when the barrier's current phase has another parity than the one asked for: when the phase waited
for is over, and just as well while the phase BEFORE it is still running.  So no wait may be reached while that one runs.  The roles of a
CTA are written down here as the waits, loads, products and arrivals they make, in the kernels' order; loads land in any order, the
tensor core takes its products in order, and a breadth-first walk over all states looks at every wait that passes."""

import re
from pathlib import Path

import pytest

KERNEL = Path(__file__).resolve().parent.parent / "tiny-llm_b200" / "csrc" / "blocks" / "blocks_flash_tc.cu"

# An operation of a role: ("wait", barrier, phase) / ("may", barrier, phase), a wait that is made or not / ("load", barrier) /
# ("mma", barriers that its commit arrives at) / ("arrive", barrier).


def early_waits(roles, counts=None):
    """The waits that can pass before their phase is over.  ``counts``: arrivals a phase takes, where more than one."""
    counts = counts or {}
    bars = sorted({op[1] for r in roles for op in r if op[0] != "mma"} | {b for r in roles for op in r if op[0] == "mma" for b in op[1]})
    at = {b: i for i, b in enumerate(bars)}
    start = (tuple(0 for _ in roles), tuple(0 for _ in bars), (), ())  # positions, arrivals per barrier, loads under way, products queued
    seen, todo, early, ends = {start}, [start], set(), 0
    while todo:
        pcs, arrived, loads, queue = todo.pop()
        nexts = []

        def hit(names):
            a = list(arrived)
            for n in names:
                a[at[n]] += 1
            return tuple(a)

        for i, load in enumerate(loads):
            nexts.append((pcs, hit([load]), loads[:i] + loads[i + 1 :], queue))
        if queue:
            nexts.append((pcs, hit(queue[0]), loads, queue[1:]))
        for r, ops in enumerate(roles):
            if pcs[r] == len(ops):
                continue
            op, on = ops[pcs[r]], pcs[:r] + (pcs[r] + 1,) + pcs[r + 1 :]
            if op[0] in ("wait", "may"):
                over = arrived[at[op[1]]] // counts.get(op[1], 1)
                if op[0] == "may":
                    nexts.append((on, arrived, loads, queue))
                if over % 2 != op[2] % 2:
                    if over <= op[2]:
                        early.add((op[1], op[2]))
                    nexts.append((on, arrived, loads, queue))
            elif op[0] == "load":
                nexts.append((on, arrived, tuple(sorted(loads + (op[1],))), queue))
            elif op[0] == "mma":
                nexts.append((on, arrived, loads, queue + (tuple(op[1]),)))
            else:
                nexts.append((on, hit([op[1]]), loads, queue))
        ends += all(p == len(o) for p, o in zip(pcs, roles)) and not loads and not queue
        assert nexts or all(p == len(o) for p, o in zip(pcs, roles)) or early, ("stuck", [o[p] for p, o in zip(pcs, roles) if p < len(o)])
        for n in nexts:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    assert ends or early
    return early


def prompt_attention(tiles, value_stages, guard):
    """``flash_tc_kernel``: two key stages and ``value_stages``; the softmax warps (one of them here) clear rows of the last value tile."""
    tma, mma, soft = [], [], []
    for t in range(tiles):
        if t >= 2:  # the producer's first pass through a ring asks for the parity of a phase that never ran
            tma.append(("wait", f"k_empty{t % 2}", t // 2 - 1))
        tma.append(("load", f"k_full{t % 2}"))
        if t >= value_stages:
            tma.append(("wait", f"v_empty{t % value_stages}", t // value_stages - 1))
        tma.append(("load", f"v_full{t % value_stages}"))

    def scores(t):
        return [("wait", f"k_full{t % 2}", t // 2), ("mma", (f"k_empty{t % 2}", f"s_full{t % 2}"))]

    mma += scores(0)
    for t in range(tiles):
        mma += scores(t + 1) if t + 1 < tiles else []
        mma += [("wait", f"p_full{t % 2}", t // 2), ("wait", f"v_full{t % value_stages}", t // value_stages), ("mma", (f"v_empty{t % value_stages}", f"pv_done{t % 2}"))]
        soft.append(("wait", f"s_full{t % 2}", t // 2))
        if t:
            soft.append(("may", f"pv_done{(t - 1) % 2}", (t - 1) // 2))  # a maximum grew
        if t == tiles - 1:
            if guard and t:
                soft.append(("wait", f"pv_done{(t - 1) % 2}", (t - 1) // 2))
            soft.append(("wait", f"v_full{t % value_stages}", t // value_stages))
        soft.append(("arrive", f"p_full{t % 2}"))
    soft.append(("wait", f"pv_done{(tiles - 1) % 2}", (tiles - 1) // 2))
    return [tma, mma, soft]


def expert_products(tiles, blocks, stages, gathers):
    """``moe_tc_kernel`` with one accumulator buffer in turn: weights, rows (gathered and reported one stage late, or by TMA), products, epilogue."""
    w, x, mma, epi = [], [], [], []
    steps, before = [(t, k) for t in range(tiles) for k in range(blocks)], None
    for i, (t, k) in enumerate(steps):
        s, again = i % stages, i // stages
        wait = [("wait", f"empty{s}", again - 1)] if again else []
        w += wait + [("load", f"full{s}")]
        x += wait
        if gathers:
            x += [("arrive", f"full{before}")] if before is not None else []
            before = s
        else:
            x += [("load", f"full{s}")]  # its bytes are part of the stage's count
        if k == 0 and t >= 2:
            mma.append(("wait", f"acc_empty{t % 2}", t // 2 - 1))
        mma += [("wait", f"full{s}", again), ("mma", (f"empty{s}",) + ((f"acc_full{t % 2}",) if k == blocks - 1 else ()))]
    if gathers:
        x.append(("arrive", f"full{before}"))
    for t in range(tiles):
        epi += [("wait", f"acc_full{t % 2}", t // 2), ("arrive", f"acc_empty{t % 2}")]
    return [w, x, mma, epi], {f"full{s}": 2 for s in range(stages)}


def decode_attention(stretches, stages, query_stages):
    """``paged_decode_tc_kernel``: the tiles of several (request, head) stretches one after another, queries in a ring of their own."""
    tma, mma, soft = [], [], []
    tile_of = [(n, i) for n, length in enumerate(stretches) for i in range(length)]

    def scores(j):
        n, i = tile_of[j]
        q = [("wait", f"q_full{n % query_stages}", n // query_stages)] if i == 0 else []
        last = (f"q_empty{n % query_stages}",) if i == stretches[n] - 1 else ()
        return q + [("wait", f"k_full{j % stages}", j // stages), ("mma", (f"k_empty{j % stages}",) + last + (f"s_full{j % 2}",))]

    for j, (n, i) in enumerate(tile_of):
        if i == 0:
            tma += [("wait", f"q_empty{n % query_stages}", n // query_stages - 1)] if n >= query_stages else []
            tma.append(("load", f"q_full{n % query_stages}"))
        for kind in "kv":
            tma += [("wait", f"{kind}_empty{j % stages}", j // stages - 1)] if j >= stages else []
            tma.append(("load", f"{kind}_full{j % stages}"))
        mma += scores(0) if j == 0 else []
        mma += scores(j + 1) if j + 1 < len(tile_of) else []
        mma += [("wait", f"p_full{j % 2}", j // 2), ("wait", f"v_full{j % stages}", j // stages), ("mma", (f"v_empty{j % stages}", f"pv_done{j % 2}"))]
        soft.append(("wait", f"s_full{j % 2}", j // 2))
        if i:
            soft.append(("may", f"pv_done{(j - 1) % 2}", (j - 1) // 2))
        soft.append(("arrive", f"p_full{j % 2}"))
        if i == stretches[n] - 1:
            soft.append(("wait", f"pv_done{j % 2}", j // 2))
    return [tma, mma, soft]


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("value_stages", [1, 2])
def test_prompt_attention(tiles, value_stages):
    source = KERNEL.read_text()
    clearing = source[source.index("values past the newest key: cleared") :]
    clearing = clearing[: clearing.index("g_fence_proxy_async")]
    guard = value_stages == 1 and re.search(r"if constexpr \(VST == 1\)\s*if \(t > 0\b[^;]*tc_wait\(pv_done \+ 8 \* \(\(t - 1\) & 1\), \(\(t - 1\) >> 1\) & 1, dead\)[^;]*;"
                                            r"[^;]*tc_wait\(v_full", clearing) is not None
    assert not early_waits(prompt_attention(tiles, value_stages, guard))


def test_a_single_value_stage_needs_the_product_before():
    assert early_waits(prompt_attention(4, 1, guard=False)) == {("v_full0", 3)}


@pytest.mark.parametrize("gathers", [True, False])
@pytest.mark.parametrize("tiles,blocks,stages", [(1, 1, 3), (4, 1, 3), (2, 5, 3), (3, 2, 3)])
def test_expert_products(tiles, blocks, stages, gathers):
    assert not early_waits(*expert_products(tiles, blocks, stages, gathers))


@pytest.mark.parametrize("stretches", [(1,), (5,), (1, 1, 1, 1, 1), (2, 1, 3)])
@pytest.mark.parametrize("stages,query_stages", [(3, 2), (2, 1)])
def test_decode_attention(stretches, stages, query_stages):
    assert not early_waits(decode_attention(stretches, stages, query_stages))
