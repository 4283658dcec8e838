"""The decoding step in one launch against the operator sequence over the same buffers (``DecodeEngine._forward_unfused``)."""

import pytest
import torch

from extensions_b200 import tiny_llm_ext_b200 as ext
from tiny_llm_b200 import Qwen3ModelWeek3
from tiny_llm_b200.engine import DecodeEngine
from tiny_llm_b200.synthetic import synthetic_qwen3

# the smallest sizes it takes (gate|up rows in every CTA), and one with a 19th of a piece's units odd, two heads a group and an untied head
SMALL = dict(hidden_size=512, num_hidden_layers=3, num_attention_heads=8, num_key_value_heads=2, head_dim=128, intermediate_size=1536, vocab_size=528)
WIDE = dict(hidden_size=1536, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=128, intermediate_size=2560, vocab_size=1040)
# two heads a group and o wider than the model: o's staged activations lie over the keys and values of an attention that is not split
OVER = dict(hidden_size=1024, num_hidden_layers=3, num_attention_heads=16, num_key_value_heads=8, head_dim=128, intermediate_size=3072, vocab_size=1040)


def test_sizes_it_does_not_take():
    """0 bytes of workspace: the engine stays with the chain of launches."""
    def takes(batch=1, layers=36, heads=32, kv=8, hidden=2560, inter=9728, vocab=151936):
        return ext.DecodeStep.workspace_bytes(batch, layers, heads, kv, hidden, inter, vocab) > 0

    assert takes() and takes(batch=4) and takes(heads=16, hidden=1024, inter=3072, layers=28)
    assert not takes(batch=5) and not takes(layers=97) and not takes(heads=40) and not takes(hidden=2560 + 256) and not takes(inter=9728 + 256)
    assert not takes(vocab=151930) and not takes(hidden=256, inter=512, heads=4, kv=2, vocab=512)
    assert not takes(hidden=8192, batch=4)  # the rows of a norm in one batch


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [SMALL, WIDE], ids=["small", "wide"])
@pytest.mark.parametrize("page,contexts", [(16, [1]), (64, [64]), (64, [65]), (16, [129]), (128, [1500]), (128, [6000]), (16, [33, 0]), (8, [200, 7]), (64, [640, 1, 128]), (128, [1025, 63, 2200, 16])])
def test_one_launch_equals_the_operator_sequence(cuda_device, dims, page, contexts):
    dev, B = cuda_device, len(contexts)
    model = Qwen3ModelWeek3(synthetic_qwen3(dims, seed=B, device=dev, realistic=True), page_size=page)
    engine = DecodeEngine(model, B, max(contexts) + 3, dev)
    assert engine._one_launch
    need = [-(-c // page) for c in contexts]
    engine.reserve_pools(sum(need) + 2)
    g = torch.Generator(device=dev).manual_seed(7)
    for pool in model.page_pools:
        for pages in (pool._key_pages, pool._value_pages):
            pages.copy_(torch.randn(pages.shape, generator=g, device=dev))
    engine._ensure_graph()
    order = torch.randperm(sum(need) + 2, generator=g, device=dev)[: sum(need)].to(torch.int32)
    engine.tables.fill_(-1)
    at = 0
    for b, n in enumerate(need):
        engine.tables[:, b, :n] = order[at : at + n]
        at += n
    if need[0] > 2:
        engine.tables[:, 0, 1] = -1  # a page that is not there: its keys are not seen
    engine.tokens.copy_(torch.randint(0, dims["vocab_size"], (B,), generator=g, device=dev))
    engine.context_lens.copy_(torch.tensor(contexts, device=dev))
    engine.offsets.copy_((engine.context_lens - 1).clamp(min=0))
    before = [(p._key_pages.clone(), p._value_pages.clone()) for p in model.page_pools]

    def run(step):
        for pool, (k, v) in zip(model.page_pools, before):
            pool._key_pages.copy_(k), pool._value_pages.copy_(v)
        step()
        return engine.logits.clone(), engine.next_tokens.clone(), [(p._key_pages.clone(), p._value_pages.clone()) for p in model.page_pools]

    got, tokens, pages = run(engine._step.launch)
    again, _, _ = run(engine._step.launch)
    assert torch.equal(got, again), "the same bits every time"
    assert torch.equal(tokens.long(), got.float().argmax(-1)), "the first of the largest"
    want, _, want_pages = run(engine._forward_unfused)
    # both round to bf16 a dozen times a block; an operator's own error is 2^-9 and they add up in quadrature
    blocks = dims["num_hidden_layers"]
    apart = ((got.double() - want.double()).norm(dim=-1) / want.double().norm(dim=-1)).max()
    assert apart < 2**-8 * (12 * blocks) ** 0.5, float(apart)
    for layer, ((k, v), (wk, wv), (k0, v0)) in enumerate(zip(pages, want_pages, before)):
        for a, w, old in ((k, wk, k0), (v, wv, v0)):
            touched = (w != old).any(-1)
            assert torch.equal(a[~touched], old[~touched]), "only the newest token's rows are written"
            if touched.any():
                assert (a[touched].double() - w[touched].double()).norm() < 2**-8 * (12 * (layer + 1)) ** 0.5 * w[touched].double().norm()
    assert ext.waits_given_up() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("layers", [1, 2])
def test_the_first_launch_on_a_fresh_workspace(cuda_device, layers):
    """Zeroed memory must not pass for packets: a new object's first step is the step that it repeats later, and no packet carries memory's tag."""
    dims, dev, contexts = dict(SMALL, num_hidden_layers=layers), cuda_device, [150, 200]
    model = Qwen3ModelWeek3(synthetic_qwen3(dims, seed=3, device=dev, realistic=True), page_size=64)
    engine = DecodeEngine(model, 2, 256, dev)
    engine.reserve_pools(8)
    g = torch.Generator(device=dev).manual_seed(5)
    slabs = [t for p in model.page_pools for t in (p._key_pages, p._value_pages)]
    for pages in slabs:
        pages.copy_(torch.randn(pages.shape, generator=g, device=dev))
    before = [t.clone() for t in slabs]
    engine.tables[:, :, :4] = torch.randperm(8, generator=g, device=dev).view(2, 4).to(torch.int32)
    engine.tokens.copy_(torch.tensor([7, 300], device=dev))
    engine.context_lens.copy_(torch.tensor(contexts, device=dev))
    engine.offsets.copy_(engine.context_lens - 1)

    def run(step):
        for pages, old in zip(slabs, before):
            pages.copy_(old)
        step.launch()
        return engine.logits.clone(), engine.next_tokens.clone(), [t.clone() for t in slabs]

    steps = [engine._one_launch_step() for _ in range(6)]
    first = [run(step) for step in steps]
    packets = steps[-1].workspace[256:].view(torch.int32).view(-1, 2)
    assert not bool(((packets[:, 0] != 0) & (packets[:, 1] == 0)).any()), "a packet with the tag of memory that was never written"
    logits, tokens, pages = run(steps[0])
    for got in first:
        assert torch.equal(got[0], logits) and torch.equal(got[1], tokens) and all(torch.equal(a, b) for a, b in zip(got[2], pages))


@pytest.mark.gpu
@pytest.mark.parametrize("page,contexts", [(16, [60]), (16, [60, 0]), (64, [64, 3]), (16, [40, 1, 64, 0]), (8, [7, 64, 200, 33])])
def test_short_contexts_where_o_is_wider_than_the_model(cuda_device, page, contexts):
    """Requests of one split beside idle and longer ones: their values are read before o's activations are staged over them.  (What the order prevents shows
    by timing alone.)"""
    for _ in range(4):
        test_one_launch_equals_the_operator_sequence(cuda_device, OVER, page, contexts)


@pytest.mark.gpu
def test_a_request_that_grows_long_goes_on_with_the_chain(cuda_device, monkeypatch):
    """Past so many keys a share the chain of launches is faster; the engine changes over between two steps, driven by the host or on the device."""
    ckpt, dev, prompt = synthetic_qwen3(SMALL, seed=2, device=cuda_device, realistic=True), cuda_device, list(range(3, 60))
    shares = torch.cuda.get_device_properties(dev).multi_processor_count // 2

    def generate(on_device, limit):
        model = Qwen3ModelWeek3(ckpt, page_size=16)
        engine = DecodeEngine(model, 1, 256, dev)
        engine.reserve_pools()
        if limit is None:
            assert not engine._one_launch
        else:
            assert engine._one_launch_keys == 700 * min(shares, 32)
            engine._one_launch_keys = limit
        cache = model.create_kv_cache()
        token = int(model(torch.tensor([prompt], dtype=torch.int32, device=dev), 0, cache, logits_to_keep=1)[0, -1].argmax())
        logits = []
        if on_device:
            tokens = engine.decode_on_device([token], [len(prompt)], cache, 24).reshape(-1).tolist()
        else:
            tokens = []
            for i in range(24):
                out, nxt = engine.step([token], [len(prompt) + i], cache)
                logits.append(out.clone())
                token = int(nxt[0])
                tokens.append(token)
        if limit is not None:
            assert (engine._long is not None) == (len(prompt) + 24 > limit) and engine.captures == 1
        for c in cache:
            c.release()
        return tokens, logits

    whole, long, over = (generate(False, limit) for limit in (10**6, 10, 70))
    monkeypatch.setenv("TL_DECODE_STEP", "0")
    chain = generate(False, None)
    monkeypatch.delenv("TL_DECODE_STEP")
    assert all(torch.equal(a, b) for a, b in zip(long[1], chain[1])) and long[0] == chain[0]
    at = 70 - len(prompt)  # steps of up to 70 tokens
    assert all(torch.equal(a, b) for a, b in zip(over[1][:at], whole[1][:at]))
    assert generate(True, 70)[0] == over[0]


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["huge pages", "unaligned norms", "two rotations"])
def test_what_the_chain_takes_is_still_taken(cuda_device, monkeypatch, form):
    """Forms that the one launch does not take as they are: a product of the page sizes past 32 bits, norm weights inside another buffer, blocks that differ."""
    ckpt, dev = synthetic_qwen3(SMALL, seed=4, device=cuda_device, realistic=True), cuda_device

    def logits():
        model = Qwen3ModelWeek3(ckpt, page_size=65536 if form == "huge pages" else 16)
        if form == "unaligned norms":
            for b in model.layers_inner:
                for n in (b.self_attn.q_norm, b.self_attn.k_norm):
                    n.weight = torch.cat([n.weight[:1], n.weight.to(torch.bfloat16)])[1:]
        if form == "two rotations":
            model.layers_inner[1].self_attn.rope.base = 5000
        engine = DecodeEngine(model, 1, 100, dev)
        engine.reserve_pools(8 if engine.page_size == 16 else 1)
        cache = model.create_kv_cache()
        model.use_decode_graph = False
        model(torch.tensor([[5, 6, 7, 8, 9]], dtype=torch.int32, device=dev), 0, cache, logits_to_keep=1)
        return engine._one_launch, [engine.step([11], [5 + i], cache)[0].clone() for i in range(3)]

    if form == "two rotations":
        monkeypatch.setenv("TL_ATTENTION_FUSED", "0")  # rotates block by block
    one, got = logits()
    assert one == (form == "unaligned norms")
    monkeypatch.setenv("TL_DECODE_STEP", "0")
    chain, want = logits()
    assert not chain
    for a, b in zip(got, want):
        assert (a.double() - b.double()).norm() < 2**-8 * (12 * 3) ** 0.5 * b.double().norm()


@pytest.mark.gpu
@pytest.mark.parametrize("on_device", [False, True])
@pytest.mark.parametrize("what", ["o", "down", "head", "nothing"])
def test_weights_written_in_place_are_seen(cuda_device, what, on_device):
    """o, down and the head as in the chain, which reads them where they lie: by the engine's next step, and by an engine that is made afterwards."""
    dev = cuda_device

    def second_step(afterwards, write):
        model = Qwen3ModelWeek3(synthetic_qwen3(SMALL, seed=6, device=dev, realistic=True), page_size=16)
        engine = DecodeEngine(model, 1, 100, dev)
        engine.reserve_pools()
        cache = model.create_kv_cache()
        model.use_decode_graph = False
        model(torch.tensor([[5, 6, 7]], dtype=torch.int32, device=dev), 0, cache, logits_to_keep=1)
        _, token = engine.step([8], [3], cache)
        block = model.layers_inner[1]
        w = {"o": block.self_attn.wo, "down": block.mlp.w_down, "head": model.w_lm_head if model.w_lm_head is not None else model.embedding.weight}.get(what)
        if w is not None and write:
            w.scales.mul_(0.5)
        if afterwards:
            token = token.clone()
            engine = DecodeEngine(model, 1, 100, dev)
        if on_device:
            engine.decode_on_device([9], [4], cache, 1)
            return engine.logits.clone(), engine.captures
        return engine.step(token, [4], cache)[0].clone(), engine.captures  # (the static buffer of the step before)

    got, captures = second_step(False, True)
    want, _ = second_step(True, True)
    old, _ = second_step(False, False)
    assert torch.equal(got, want) and torch.equal(got, old) == (what == "nothing") and captures == (1 if what == "nothing" else 2)


@pytest.mark.gpu
def test_two_engines_on_two_streams_at_once(cuda_device):
    """Steps that fill the GPU by themselves follow one another, whatever stream they come from; other kernels run between them."""
    dev = cuda_device
    model = Qwen3ModelWeek3(synthetic_qwen3(OVER, seed=8, device=dev, realistic=True), page_size=64)
    engines = [DecodeEngine(model, b, 256, dev) for b in (1, 3)]
    engines[0].reserve_pools(16)
    want = []
    for i, engine in enumerate(engines):
        engine._ensure_graph()
        engine.tables[:, :, :4] = torch.arange(4 * i, 4 * i + 4 * engine.B, device=dev, dtype=torch.int32).view(engine.B, 4)
        engine.tokens.fill_(3 + i)
        engine.context_lens.fill_(200)
        engine.offsets.fill_(199)
        engine._graph.replay()
        want.append(engine.logits.clone())
    count = ext.waits_given_up()
    streams = [torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    a = torch.randn(4096, 4096, device=dev).bfloat16()
    torch.cuda.synchronize()
    for _ in range(100):
        for engine, stream in zip(engines, streams):
            with torch.cuda.stream(stream):
                engine._graph.replay()
        with torch.cuda.stream(streams[2]):
            a @ a
    torch.cuda.synchronize()
    assert all(torch.equal(e.logits, w) for e, w in zip(engines, want)) and ext.waits_given_up() == count
