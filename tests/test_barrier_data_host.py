"""The barrier protocols of the packed products, every interleaving of them: no wait passes before its phase is over, nothing is written over
before it is read, nothing is read before it is written, and nothing gets stuck.

Each role is the sequence of its operations in the kernels' order.  ``wait``: (barrier, phase); ``load``: an asynchronous copy, which lands later, in any
order; ``mma``: products, which the tensor core takes in the order of issue and which arrive at their commits' barriers; ``arrive``.  An operation
says what must have happened when it takes effect: ``after`` = conditions on the state that the protocol has to bring about by itself."""

from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tiny-llm_b200" / "csrc"


class Op:
    def __init__(self, kind, barriers=(), phase=0, after=(), name=None):
        self.kind, self.barriers, self.phase, self.after, self.name = kind, tuple(barriers), phase, tuple(after), name


def walk(roles, counts):
    """-> set of violations over all interleavings (empty: the protocol holds).  ``after``: ("landed", name) / ("executed", name) / ("done", name) of a load, a
    product and any other operation."""
    bars = sorted({b for r in roles for op in r for b in op.barriers})
    at = {b: i for i, b in enumerate(bars)}
    place = {op.name: (r, i) for r, ops in enumerate(roles) for i, op in enumerate(ops) if op.name is not None}
    start = ((0,) * len(roles), (0,) * len(bars), frozenset(), ())  # positions, arrivals, loads under way, products queued
    seen, todo, wrong = {start}, [start], set()
    while todo:
        pcs, arrived, loads, queue = todo.pop()
        over = [a // counts.get(b, 1) for b, a in zip(bars, arrived)]

        def happened(kind, name):
            r, i = place[name]
            return pcs[r] > i and not (kind == "landed" and (r, i) in loads) and not (kind == "executed" and (r, i) in queue)

        def check(op):
            wrong.update((op.name, c) for c in op.after if not happened(*c))

        def hit(names):
            a = list(arrived)
            for n in names:
                a[at[n]] += 1
            return tuple(a)

        nexts = [(pcs, hit(roles[r][i].barriers), loads - {(r, i)}, queue) for r, i in loads]
        if queue:
            op = roles[queue[0][0]][queue[0][1]]
            check(op)
            nexts.append((pcs, hit(op.barriers), loads, queue[1:]))
        for r, ops in enumerate(roles):
            if pcs[r] == len(ops):
                continue
            op, on = ops[pcs[r]], pcs[:r] + (pcs[r] + 1,) + pcs[r + 1 :]
            if op.kind == "wait":
                done = over[at[op.barriers[0]]]
                if done % 2 != op.phase % 2:
                    if done <= op.phase:
                        wrong.add((op.barriers[0], op.phase))
                    nexts.append((on, arrived, loads, queue))
            elif op.kind == "load":
                check(op)
                nexts.append((on, arrived, loads | {(r, pcs[r])}, queue))
            elif op.kind == "mma":
                nexts.append((on, arrived, loads, queue + ((r, pcs[r]),)))
            else:
                check(op)
                nexts.append((on, hit(op.barriers), loads, queue))
        if not nexts and any(p < len(o) for p, o in zip(pcs, roles)):
            wrong.add("stuck")
        if wrong:
            return wrong
        for n in nexts:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return wrong


def pairs(tiles, blocks, stages, early_empty=False, peer_releases=True, peer_forwards=True, unpackers=(0,)):
    """``w4a16_gemm2_kernel``: two CTAs, items of ``tiles[n]`` token tiles (2: both accumulators) of ``blocks`` reduction blocks each.  The first blocks, as many as there
    are stages, go to the first accumulator, then to the second, whose last results may still be being read out.  ``unpackers``: CTAs whose dequantisers are roles
    of their own (elsewhere they keep step with the copies)."""
    tma, unpack, forward, mma, epilogue = [[], []], [[], []], [], [], [[], []]
    last_read, uses, first_of = {}, [0, 0], {}

    def full(c, b):
        return f"full{c}.{b % stages}"

    def empties(b):
        return [f"empty{c}.{b % stages}" for c in (0, 1)]

    def inputs(b):
        return [("landed", f"copy{c}.{b}") for c in (0, 1)] + [("done", f"unpacked{c}.{b}") for c in unpackers]

    b = 0
    for n, mt in enumerate(tiles):
        first, head = b, min(stages, blocks)
        for kb in range(blocks):  # what is issued when block b is taken up
            last_read[b + kb] = f"product{mt - 1}.{b + kb}"

        def product(acc, block, commits):
            after = inputs(block)
            if block == first and (acc, uses[acc]) not in first_of:
                first_of[acc, uses[acc]] = True
                after += [("done", f"read{c}.{acc}.{uses[acc] - 1}") for c in (0, 1)] if uses[acc] else []
            mma.append(Op("mma", commits, after=after, name=f"product{acc}.{block}"))

        def take(acc):
            if uses[acc]:
                mma.append(Op("wait", [f"acc_empty{acc}"], uses[acc] - 1))

        take(0)
        for kb in range(head):
            mma.append(Op("wait", [full(0, b + kb)], (b + kb) // stages))
            product(0, b + kb, empties(b + kb) if mt == 1 or early_empty else [])
        if mt > 1:
            take(1)
            for kb in range(head):
                product(1, b + kb, [] if early_empty else empties(b + kb))
        for kb in range(head, blocks):
            mma.append(Op("wait", [full(0, b + kb)], (b + kb) // stages))
            product(0, b + kb, ["acc_full0.0", "acc_full1.0"] * (kb == blocks - 1) + (empties(b + kb) if mt == 1 else []))
            if mt > 1:
                product(1, b + kb, empties(b + kb))
        if head == blocks:
            mma.append(Op("mma", ["acc_full0.0", "acc_full1.0"]))
        if mt > 1:
            mma.append(Op("mma", ["acc_full0.1", "acc_full1.1"]))
        for acc in range(mt):
            for c in (0, 1):
                epilogue[c].append(Op("wait", [f"acc_full{c}.{acc}"], uses[acc]))
                release = [f"acc_empty{acc}"] if c == 0 or peer_releases else []
                epilogue[c].append(Op("arrive", release, after=[("executed", f"product{acc}.{first + kb}") for kb in range(blocks)], name=f"read{c}.{acc}.{uses[acc]}"))
            uses[acc] += 1
        b += blocks
    for block in range(b):
        free = [("executed", last_read[block - stages])] if block >= stages else []
        for c in (0, 1):
            for role in (tma[c], unpack[c]):
                if block >= stages:
                    role.append(Op("wait", [f"empty{c}.{block % stages}"], block // stages - 1))
            tma[c].append(Op("load", [full(c, block)], after=free, name=f"copy{c}.{block}"))
            unpack[c].append(Op("arrive", [full(c, block)], after=free, name=f"unpacked{c}.{block}"))
        if peer_forwards:
            forward += [Op("wait", [full(1, block)], block // stages), Op("arrive", [full(0, block)])]
    counts = {f"full{c}.{s}": 1 + (c in unpackers) + (c == 0 and peer_forwards) for c in (0, 1) for s in range(stages)}
    counts.update({f"acc_empty{a}": 1 + peer_releases for a in (0, 1)})
    return [tma[0], tma[1], mma, forward, epilogue[0], epilogue[1]] + [unpack[c] for c in unpackers], counts


@pytest.mark.parametrize("tiles,blocks,stages", [((2, 2), 1, 2), ((2, 2), 2, 2), ((2, 1), 3, 2), ((1, 2, 2), 2, 2), ((1, 1, 1), 3, 2), ((2, 2), 4, 2), ((2, 2), 2, 3)])
def test_pairs(tiles, blocks, stages):
    assert not walk(*pairs(tiles, blocks, stages))


@pytest.mark.parametrize("unpackers", [(), (1,)])
def test_pairs_whose_peer_unpacks_at_its_own_pace(unpackers):
    assert not walk(*pairs((2, 1, 2), 3, 2, unpackers=unpackers))


@pytest.mark.parametrize("wrong", [dict(early_empty=True), dict(peer_releases=False), dict(peer_forwards=False)])
def test_pairs_that_the_walk_rejects(wrong):
    """Stages given back before the second accumulator has had them, accumulators given back by one of the two CTAs, products that wait for one CTA's inputs."""
    assert walk(*pairs((2, 2), 3, 2, **wrong))


def skinny(blocks, stages, boxes, one_group=False):
    """``w4a16_skinny_kernel``: packed boxes of two blocks, two dequantiser groups that take blocks in turn, one full and one empty barrier a stage.  ``one_group``:
    a box given back by the first group alone."""
    tma, packed, groups, mma = [], [], [[], []], []
    for i in range(blocks):
        again, free = i // stages, [("executed", f"product{i - stages}")] if i >= stages else []
        empty = [Op("wait", [f"empty{i % stages}"], again - 1)] if again else []
        tma += empty + [Op("load", [f"full{i % stages}"], after=free, name=f"rows{i}")]
        box, slot = i // 2, i // 2 % boxes
        mine = groups[i % 2]
        mine += [Op("wait", [f"p_full{slot}"], box // boxes)] + empty
        mine.append(Op("arrive", [f"full{i % stages}"], after=free + [("landed", f"box{box}")], name=f"unpacked{i}"))
        mine.append(Op("arrive", [f"p_empty{slot}"] * (i % 2 == 0 or not one_group), name=f"given{i}"))
        mma += [Op("wait", [f"full{i % stages}"], again), Op("mma", [f"empty{i % stages}"], after=[("landed", f"rows{i}"), ("done", f"unpacked{i}")], name=f"product{i}")]
    for box in range((blocks + 1) // 2):
        read = [("done", f"unpacked{i}") for i in (2 * (box - boxes), 2 * (box - boxes) + 1)] if box >= boxes else []
        packed += [Op("wait", [f"p_empty{box % boxes}"], box // boxes - 1)] if box >= boxes else []
        packed.append(Op("load", [f"p_full{box % boxes}"], after=read, name=f"box{box}"))
    return [tma, packed, groups[0], groups[1], mma], {**{f"full{s}": 2 for s in range(stages)}, **{f"p_empty{s}": 1 if one_group else 2 for s in range(boxes)}}


@pytest.mark.parametrize("blocks", [1, 2, 4, 7, 8])
@pytest.mark.parametrize("stages", [2, 3])
@pytest.mark.parametrize("boxes", [2, 3])
def test_skinny(blocks, stages, boxes):
    assert not walk(*skinny(blocks, stages, boxes))


def test_skinny_that_the_walk_rejects():
    assert walk(*skinny(8, 3, 2, one_group=True))
