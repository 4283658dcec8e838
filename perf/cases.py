"""The work this framework is used for, as cases that can be timed and compared.

Two groups.  The Qwen3 W4A16 path: whole decoding steps (``Qwen3ModelWeek3``), the packed feed-forward (``Qwen3MLP``) from
one row to a prompt portion, and paged attention for prompts and for decoding.  The unquantised designs: a latent-attention
layer, a grouped-query attention layer over the paged cache, a mixture-of-experts feed-forward and a decayed linear-attention
layer, each over a ragged batch as a continuous-batching step brings it.  Sizes are those of the framework's configurations
(``synthetic.CONFIGS``) and of its benchmark workloads; weights and inputs are random.

A case is a dict of plain values; ``kind`` says which of the seven it is.  ``lengths`` / ``before`` are the new tokens of every
request of a step and the tokens its cache already holds.
"""

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "tiny-llm_b200"))

from tiny_llm_b200 import Qwen3ModelWeek3, paged_attention  # noqa: E402
from tiny_llm_b200.kv_cache import BatchingKvCache  # noqa: E402
from tiny_llm_b200.latent_attention import LatentAttention  # noqa: E402
from tiny_llm_b200.latent_kv_cache import LatentPagedCache, LatentPagedPool  # noqa: E402
from tiny_llm_b200.linear_attention import DecayedLinearAttention  # noqa: E402
from tiny_llm_b200.mlp import GatedMLP, MixtureOfExperts, TopKRouter  # noqa: E402
from tiny_llm_b200.paged_attention import FusedProjection, PagedGroupedAttention  # noqa: E402
from tiny_llm_b200.quantize import QuantizedWeights  # noqa: E402
from tiny_llm_b200.qwen3_week3 import Qwen3MLP  # noqa: E402
from tiny_llm_b200.ragged import RaggedEntry, RaggedPlan  # noqa: E402
from tiny_llm_b200.state_cache import HybridPagedCache, StateSlotPool  # noqa: E402
from tiny_llm_b200.synthetic import CONFIGS, synthetic_qwen3  # noqa: E402

DEV = "cuda"
BF16, F64 = torch.bfloat16, torch.float64
EPS = 1e-5
STEPS = 16   # decoded tokens per request in one pass over a whole model
# Of a model's layers, the first eight: through all 28 or 36 of them bf16 rounding alone moves the logits by 5 % (random
# weights), and two correct results could no longer be told from a wrong one; through eight it is 2 %.
DEPTH = 8
PAGE = 64    # page size of the unquantised designs' caches
QPAGE = 128  # page size of the Qwen3 models' caches

LATENT = {
    1024: dict(width=1024, heads=8, dim=64, rot_dim=32, vdim=64, rank=256, window=512),
    2048: dict(width=2048, heads=16, dim=128, rot_dim=64, vdim=128, rank=512, window=1024),
}
GROUPED = {
    # a window plus kept first positions, whole-projection norms, a stretched rotation, a learned sink, a gate per head
    "window": {1024: dict(width=1024, heads=8, kv_heads=2, dim=128, vdim=128, size=512, keep_first=4, rot=64),
               2048: dict(width=2048, heads=16, kv_heads=4, dim=128, vdim=128, size=1024, keep_first=16, rot=64)},
    # blocks of positions, norms per head, a soft cap, a fixed sink, a gate per head
    "chunk": {1024: dict(width=1024, heads=8, kv_heads=2, dim=96, vdim=64, size=512, softcap=30.0),
              2048: dict(width=2048, heads=16, kv_heads=4, dim=192, vdim=128, size=1024, softcap=30.0)},
    # everything before, rotated
    "causal": {1024: dict(width=1024, heads=8, kv_heads=2, dim=96, vdim=64, size=0, rot=64),
               2048: dict(width=2048, heads=16, kv_heads=4, dim=192, vdim=128, size=0, rot=128)},
}
YARN = dict(factor=4.0, original=4096, fast=32.0, slow=1.0)
EXPERTS = {
    1024: dict(width=1024, experts=16, top=2, ff=512, shared=1024),
    2048: dict(width=2048, experts=64, top=6, ff=1408, shared=2816),
}
DECAY = {
    1024: dict(width=1024, heads=8, dim=64, vdim=128, tau=16.0, low=64),
    2048: dict(width=2048, heads=16, dim=64, vdim=128, tau=16.0, low=128),
}


def listed():
    return [
        # one user's answer being written: every step depends on the last, one row through every weight
        {"name": "decode_1", "kind": "decode", "model": "qwen3-4b", "lengths": "1011"},
        # a serving step: two dozen answers of different lengths at once
        {"name": "decode_24", "kind": "decode", "model": "qwen3-4b", "lengths": ",".join(str(70 + 113 * i % 1901) for i in range(24))},
        # the smallest call a program makes by itself: one row through a packed feed-forward
        {"name": "mlp_1", "kind": "mlp", "model": "qwen3-4b", "rows": 1},
        # a serving batch through it
        {"name": "mlp_52", "kind": "mlp", "model": "qwen3-4b", "rows": 52},
        # a prompt portion through it
        {"name": "mlp_2048", "kind": "mlp", "model": "qwen3-4b", "rows": 2048},
        # a long prompt's second portion attends everything before it
        {"name": "attend_prompt", "kind": "attend", "heads": 32, "kv_heads": 8, "new": 2048, "lengths": "3500"},
        # decoding over caches of different lengths, a few of them long
        {"name": "attend_decode", "kind": "attend", "heads": 32, "kv_heads": 8, "new": 1, "lengths": ",".join(str(200 + 331 * i % 7001) for i in range(32))},
        # prompt portions of three requests through a latent-attention layer
        {"name": "latent_prompt", "kind": "latent", "width": 2048, "windowed": False, "lengths": "1200,650,198", "before": "0,300,1025"},
        # the same mix through a grouped-query layer with a window
        {"name": "grouped_prompt", "kind": "grouped", "design": "window", "width": 2048, "lengths": "1200,650,198", "before": "0,300,1025"},
        # a prompt portion through a layer of experts, and a decoding batch
        {"name": "experts_2048", "kind": "experts", "width": 2048, "tokens": 2048},
        {"name": "experts_16", "kind": "experts", "width": 2048, "tokens": 16},
        # prompt portions through a recurrent layer
        {"name": "decay_prompt", "kind": "decay", "width": 2048, "lengths": "1500,548", "before": "0,0"},
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))

    def split(total, most):
        """``total`` tokens over up to ``most`` requests, unevenly."""
        n = rng.randint(1, max(1, min(most, total)))
        cuts = sorted(rng.sample(range(1, total), n - 1)) if n > 1 else []
        return [b - a for a, b in zip([0] + cuts, cuts + [total])]

    def text(values):
        return ",".join(str(v) for v in values)

    kind = rng.choice(["decode", "mlp", "mlp", "attend", "attend", "latent", "latent", "grouped", "grouped", "experts", "experts", "decay"])
    if kind == "decode":
        return {"kind": kind, "model": rng.choice(sorted(n for n in CONFIGS if n.startswith("qwen3"))), "lengths": text(log(16, 2000) for _ in range(log(1, 24)))}
    if kind == "mlp":
        return {"kind": kind, "model": rng.choice(sorted(n for n in CONFIGS if n.startswith("qwen3"))), "rows": log(1, 2048)}
    if kind == "attend":
        heads = rng.choice([16, 32])
        if rng.random() < 0.5:
            return {"kind": kind, "heads": heads, "kv_heads": 8, "new": 1, "lengths": text(log(16, 7200) for _ in range(log(1, 32)))}
        new = log(9, 2048)
        return {"kind": kind, "heads": heads, "kv_heads": 8, "new": new, "lengths": text([new + (log(1, 1400) if rng.random() < 0.7 else 0)])}
    width = rng.choice([1024, 2048])
    if kind == "experts":
        return {"kind": kind, "width": width, "tokens": log(1, 2048)}
    if rng.random() < 0.35:  # a decoding step
        lengths = [1] * log(1, 32)
        before = [log(16, 2048) for _ in lengths]
    else:  # prompt portions, single tokens of other requests among them
        lengths = split(log(8, 2048), 6)
        before = [log(16, 1024) if n == 1 or rng.random() < 0.5 else 0 for n in lengths]
    case = {"kind": kind, "width": width, "lengths": text(lengths), "before": text(before)}
    if kind == "latent":
        case["windowed"] = rng.random() < 0.4
    if kind == "grouped":
        case["design"] = rng.choice(sorted(GROUPED))
    return case


# ---- inputs, from the seed alone -----------------------------------------------------------------
class Draw:
    """Random tensors on the GPU, in the order they are asked for."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=BF16):
        return (torch.randn(shape, generator=self.gen, device=DEV) * std + mean).to(dtype)

    def matrix(self, rows, cols, gain=1.0):
        return self.normal(rows, cols, std=gain / cols**0.5)

    def fill_packed(self, layer):
        """Random codes and scales; the weights they stand for have variance 1 / inputs (codes are uniform: 22.25 sigma^2)."""
        w = layer.weight.view(torch.int32)
        w.copy_(torch.randint(-(2**31), 2**31, w.shape, generator=self.gen, device=DEV, dtype=torch.int64))
        sigma = 1.0 / (4.717 * (w.shape[1] * 8) ** 0.5)
        scales = torch.randn(layer.scales.shape, generator=self.gen, device=DEV) * sigma
        layer.scales.copy_(scales)
        layer.biases.copy_(-7.5 * layer.scales.float() + torch.randn(scales.shape, generator=self.gen, device=DEV) * sigma)
        return layer


def ints(text):
    return [int(v) for v in text.split(",")]


def qwen(case, seed):
    """The checkpoint object, the requests' keys and values per layer and the tokens to decode."""
    d = Draw(seed)
    ckpt = synthetic_qwen3(case["model"], device=DEV, empty=True, num_hidden_layers=DEPTH)
    m = ckpt.model
    d.fill_packed(m.embed_tokens)
    for layer in m.layers:
        a, f = layer.self_attn, layer.mlp
        for packed in (a.q_proj, a.k_proj, a.v_proj, a.o_proj, f.gate_proj, f.up_proj, f.down_proj):
            d.fill_packed(packed)
    for norm in [m.norm] + [n for l in m.layers for n in (l.input_layernorm, l.post_attention_layernorm, l.self_attn.q_norm, l.self_attn.k_norm)]:
        norm.weight.copy_(d.normal(norm.weight.numel(), std=0.1, mean=1.0))
    lengths, args = ints(case["lengths"]), ckpt.args
    longest = max(lengths) + len(lengths)
    cached = [(d.normal(1, args.num_key_value_heads, longest, args.head_dim), d.normal(1, args.num_key_value_heads, longest, args.head_dim)) for _ in m.layers]
    tokens = torch.randint(0, args.vocab_size, (STEPS, len(lengths), 1), generator=d.gen, device=DEV, dtype=torch.int32)
    return ckpt, cached, tokens


def mlp_inputs(case, seed):
    d, dims = Draw(seed), CONFIGS[case["model"]]
    one = synthetic_qwen3(dict(dims, num_hidden_layers=1, vocab_size=128), device=DEV, empty=True).model.layers[0].mlp
    packed = [QuantizedWeights.from_mlx_layer(d.fill_packed(p), use_simdgroup_matmul=True, use_split_k_matmul=True) for p in (one.gate_proj, one.up_proj, one.down_proj)]
    return packed, d.normal(1, case["rows"], dims["hidden_size"])


def attend_inputs(case, seed):
    """Queries, pages in shuffled order, block table and context lengths."""
    d, lengths = Draw(seed), ints(case["lengths"])
    pages = [-(-n // QPAGE) for n in lengths]
    order = np.random.RandomState(seed % 2**31).permutation(sum(pages)).astype(np.int32)
    table = np.full((len(lengths), max(pages)), -1, dtype=np.int32)
    at = 0
    for b, n in enumerate(pages):
        table[b, :n], at = order[at : at + n], at + n
    q = d.normal(len(lengths), case["heads"], case["new"], 128)
    k, v = (d.normal(sum(pages), case["kv_heads"], QPAGE, 128) for _ in range(2))
    return q, k, v, table, np.asarray(lengths, dtype=np.int32)


def latent_inputs(case, seed):
    d, z = Draw(seed), LATENT[case["width"]]
    H, dn, dr, dv, R, D = z["heads"], z["dim"], z["rot_dim"], z["vdim"], z["rank"], z["width"]
    w = dict(w_q=d.matrix(H * (dn + dr), D, 2.0), w_dkv=d.matrix(R + dr, D, 2.0), dkv_norm=d.normal(R, std=0.1, mean=1.0), w_uk=d.matrix(H * dn, R),
             w_uv=d.matrix(H * dv, R), w_o=d.matrix(D, H * dv))
    return w, d.normal(sum(ints(case["lengths"])), D), [d.normal(n, R + dr) for n in ints(case["before"])]


def grouped_inputs(case, seed):
    d, z = Draw(seed), GROUPED[case["design"]][case["width"]]
    H, G, dk, dv, D = z["heads"], z["kv_heads"], z["dim"], z["vdim"], z["width"]
    w = dict(q=d.matrix(H * dk, D, 2.0), k=d.matrix(G * dk, D, 2.0), v=d.matrix(G * dv, D), g=d.matrix(H, D, 2.0), o=d.matrix(D, H * dv))
    if case["design"] == "window":
        w.update(q_norm=d.normal(H * dk, std=0.1, mean=1.0), k_norm=d.normal(G * dk, std=0.1, mean=1.0), sink=d.normal(H))
    elif case["design"] == "chunk":
        w.update(q_norm=d.normal(dk, std=0.2, mean=1.0), k_norm=d.normal(dk, std=0.2, mean=1.0))
    return w, d.normal(sum(ints(case["lengths"])), D), [d.normal(n, G * (dk + dv)) for n in ints(case["before"])]


def experts_inputs(case, seed):
    d, z = Draw(seed), EXPERTS[case["width"]]
    E, D, ff, sh = z["experts"], z["width"], z["ff"], z["shared"]
    w = dict(router=d.matrix(E, D, 2.0), bias=d.normal(E, std=0.3), gate=d.normal(E, ff, D, std=D**-0.5), up=d.normal(E, ff, D, std=D**-0.5),
             down=d.normal(E, D, ff, std=ff**-0.5), s_gate=d.matrix(sh, D), s_up=d.matrix(sh, D), s_down=d.matrix(D, sh))
    return w, d.normal(case["tokens"], D)


def decay_inputs(case, seed):
    d, z = Draw(seed), DECAY[case["width"]]
    H, dk, dv, D, low = z["heads"], z["dim"], z["vdim"], z["width"], z["low"]
    w = dict(q=d.matrix(H * dk, D, 2.0), k=d.matrix(H * dk, D, 2.0), v=d.matrix(H * dv, D), g=d.matrix(H * dv, D), a1=d.matrix(low, D), a2=d.matrix(H * dk, low, 2.0),
             bias=d.normal(H * dk, std=1.0, mean=2.0), norm=d.normal(dv, std=0.2, mean=1.0), o=d.matrix(D, H * dv))
    n = len(ints(case["lengths"]))
    return w, d.normal(sum(ints(case["lengths"])), D), d.normal(n, H, dk, dv, std=3.0, dtype=torch.float32)


# ---- what a program has in hand before the call ------------------------------------------------------
def prepare_decode(case, seed):
    ckpt, cached, tokens = qwen(case, seed)
    model = Qwen3ModelWeek3(ckpt, page_size=QPAGE)
    lengths = ints(case["lengths"])
    B = len(lengths)
    limit = -(-(max(lengths) + STEPS) // QPAGE) * QPAGE
    model.decode_graph_max_seq_len = limit
    model.decode_engine(B, limit)  # also sizes the page pools
    requests = [model.create_kv_cache() for _ in range(B)]
    for b, request in enumerate(requests):
        for one, (k, v) in zip(request, cached):
            one.update_and_fetch_paged(k[:, :, b : b + lengths[b]].contiguous(), v[:, :, b : b + lengths[b]].contiguous())
    if B == 1:
        caches = requests[0]
    else:
        caches = []
        for layer in range(model.num_hidden_layers):
            table = BatchingKvCache(max_active_requests=B, max_seq_len=limit)
            for b in range(B):
                table.add_request(requests[b][layer], b)
            caches.append(table)
    state = {"kind": "decode", "model": model, "requests": requests, "caches": caches, "tokens": tokens, "lengths": lengths}
    run_decode(state, steps=1)  # a server has decoded before: its step is captured
    return state


def run_decode(s, steps=STEPS):
    logits = []
    for t in range(steps):
        logits.append(s["model"](s["tokens"][t], [n + t for n in s["lengths"]], s["caches"], logits_to_keep=1))
    for request in s["requests"]:  # the answers are taken back, so that the next pass writes them again
        for one in request:
            one.rewind(steps)
    return logits


def prepare_mlp(case, seed):
    (gate, up, down), x = mlp_inputs(case, seed)
    dims = CONFIGS[case["model"]]
    return {"kind": "mlp", "layer": Qwen3MLP(dims["hidden_size"], dims["intermediate_size"], gate, up, down), "x": x}


def run_mlp(s):
    return s["layer"](s["x"])


def prepare_attend(case, seed):
    q, k, v, table, lengths = attend_inputs(case, seed)
    return {"kind": "attend", "q": q, "k": k, "v": v, "table": torch.from_numpy(table).to(DEV), "lens": torch.from_numpy(lengths).to(DEV), "table_host": table, "lens_host": lengths}


def run_attend(s):
    return paged_attention(s["q"], s["k"], s["v"], s["table"], s["lens"], QPAGE, mask="causal", block_table_host=s["table_host"], context_lens_host=s["lens_host"])


def plan_for(case, owners, tile_sizes, before, slabs):
    """The step's plan, with the rows the caches already hold written to their pages."""
    lengths = ints(case["lengths"])
    for owner, rows in zip(owners, before):
        n = rows if isinstance(rows, int) else rows.shape[0]
        if n:
            owner.append_slots(n)
            if slabs is not None:
                for i, page in enumerate(owner.page_ids):
                    part = rows[i * PAGE : (i + 1) * PAGE]
                    slabs[0][page, : part.shape[0]] = part
    return RaggedPlan([RaggedEntry([0] * n, [o], want=[]) for n, o in zip(lengths, owners)], DEV, tile_sizes)


def page_pool(case, width):
    pages = sum(-(-(n + b) // PAGE) for n, b in zip(ints(case["lengths"]), ints(case["before"])))
    return LatentPagedPool([width], page_size=PAGE, dtype=BF16, device=DEV, max_pages=pages)


def prepare_latent(case, seed):
    w, h, before = latent_inputs(case, seed)
    z = LATENT[case["width"]]
    layer = LatentAttention(heads=z["heads"], dim=z["dim"], rot_dim=z["rot_dim"], vdim=z["vdim"], kv_rank=z["rank"], scale=(z["dim"] + z["rot_dim"]) ** -0.5,
                            rot_dims=z["rot_dim"], rot_base=10000.0, interleaved=False, window=z["window"] if case["windowed"] else None, eps=EPS, **w)
    pool = page_pool(case, layer.cache_width)
    owners = [LatentPagedCache(pool) for _ in before]
    plan = plan_for(case, owners, [layer.attention_kernel(pool.slabs[0])[1]], before, pool.slabs)
    return {"kind": "latent", "layer": layer, "h": h, "plan": plan, "slab": pool.slabs[0]}


def run_latent(s):
    return s["layer"](s["h"], s["plan"], s["slab"])


def prepare_grouped(case, seed):
    w, h, before = grouped_inputs(case, seed)
    z, design = GROUPED[case["design"]][case["width"]], case["design"]
    more = {}
    if design == "window":
        more = dict(mask="window", keep_first=z["keep_first"], sink=True, head_bias=w["sink"], q_norm=w["q_norm"], k_norm=w["k_norm"], qk_norm="whole",
                    rot={"dims": z["rot"], "base": 100000.0, "yarn": YARN})
    elif design == "chunk":
        more = dict(mask="chunk", softcap=z["softcap"], sink=True, q_norm=w["q_norm"], k_norm=w["k_norm"])
    else:
        more = dict(mask="causal", rot={"dims": z["rot"], "base": 10000.0, "factor": 8.0, "interleaved": True})
    layer = PagedGroupedAttention(heads=z["heads"], kv_heads=z["kv_heads"], dim=z["dim"], vdim=z["vdim"], scale=z["dim"] ** -0.5, mask_size=z["size"], w_o=w["o"], eps=EPS,
                                  page_size=PAGE, **more)
    pool = page_pool(case, layer.cache_width)
    owners = [LatentPagedCache(pool) for _ in before]
    plan = plan_for(case, owners, layer.tile_sizes, before, pool.slabs)
    proj = FusedProjection([(n, w[n], None) for n in ("q", "k", "v", "g")], BF16, DEV)
    return {"kind": "grouped", "layer": layer, "proj": proj, "h": h, "plan": plan, "slab": pool.slabs[0], "gated": design != "causal"}


def run_grouped(s):
    y = s["proj"](s["h"])
    return s["layer"](y["q"], y["k"], y["v"], y["g"] if s["gated"] else None, s["plan"], s["slab"])


def prepare_experts(case, seed):
    w, h = experts_inputs(case, seed)
    shared = GatedMLP(w["s_gate"], w["s_up"], w["s_down"], "silu")
    router = TopKRouter(w["router"], w["bias"], EXPERTS[case["width"]]["top"])
    return {"kind": "experts", "layer": MixtureOfExperts(router, w["gate"], w["up"], w["down"], "silu", shared), "h": h}


def run_experts(s):
    return s["layer"](s["h"])


def prepare_decay(case, seed):
    w, h, initial = decay_inputs(case, seed)
    z = DECAY[case["width"]]
    layer = DecayedLinearAttention(heads=z["heads"], dim=z["dim"], vdim=z["vdim"], tau=z["tau"], w_a2=w["a2"], a2_bias=w["bias"], norm_weight=w["norm"], w_o=w["o"], eps=EPS)
    floats = z["heads"] * z["dim"] * z["vdim"]
    before = ints(case["before"])
    states = StateSlotPool(floats, device=DEV, max_slots=len(before))
    pool = page_pool(case, 8)
    owners = [HybridPagedCache(pool, states) for _ in before]
    plan = plan_for(case, owners, [64], before, None)
    view = states.layer_view(0, layer.state_shape)
    slots = [o.state_slot for o in owners]
    first = torch.zeros_like(initial)
    first[slots] = initial
    proj = FusedProjection([(n, w[n], None) for n in ("q", "k", "v", "g", "a1")], BF16, DEV)
    return {"kind": "decay", "layer": layer, "proj": proj, "h": h, "plan": plan, "state": view, "first": first, "slots": torch.tensor(slots, device=DEV)}


def run_decay(s):
    s["state"].copy_(s["first"])  # the requests' states as they were before this step
    y = s["proj"](s["h"])
    out = s["layer"](y["q"], y["k"], y["v"], y["g"], y["a1"], s["plan"], s["state"])
    return {"out": out, "state": s["state"][s["slots"]]}


KINDS = ("decode", "mlp", "attend", "latent", "grouped", "experts", "decay")
PREPARE = {k: globals()["prepare_" + k] for k in KINDS}
RUN = {k: globals()["run_" + k] for k in KINDS}


def prepare(case, seed):
    return PREPARE[case["kind"]](case, seed)


def run(state):
    return RUN[state["kind"]](state)


# ---- what a pass cannot do without -----------------------------------------------------------------
def seen_keys(case):
    """Per request (how many keys its new tokens see, summed; how many cached rows they see together)."""
    out = []
    for n, b in zip(ints(case["lengths"]), ints(case["before"])):
        pos = np.arange(b, b + n)
        first = np.zeros(n, dtype=np.int64)
        kept = 0
        if case["kind"] == "latent" and case["windowed"]:
            first = np.maximum(0, pos - LATENT[case["width"]]["window"] + 1)
        elif case["kind"] == "grouped" and case["design"] != "causal":
            z = GROUPED[case["design"]][case["width"]]
            if case["design"] == "window":
                first = np.maximum(0, pos - z["size"] + 1)
                kept = z["keep_first"]
            else:
                first = pos // z["size"] * z["size"]
        seen = pos - first + 1 + np.minimum(first, kept)
        out.append((int(seen.sum()), int(b + n - first[0] + min(first[0], kept))))
    return out


def work(case):
    kind = case["kind"]
    if kind == "decode":
        z, lengths = CONFIGS[case["model"]], ints(case["lengths"])
        q, kv, D, ff, V = z["num_attention_heads"] * 128, z["num_key_value_heads"] * 128, z["hidden_size"], z["intermediate_size"], z["vocab_size"]
        weights = DEPTH * (D * (2 * q + 2 * kv) + 3 * D * ff) + V * D
        cached = DEPTH * 2 * kv * sum(n + STEPS / 2 for n in lengths)
        flops = 2.0 * weights * len(lengths) + 4.0 * DEPTH * q * sum(n + STEPS / 2 for n in lengths)
        return {"bytes": STEPS * (weights * 0.53125 + cached * 2 + len(lengths) * V * 2), "flops": STEPS * flops}
    if kind == "mlp":
        z, M = CONFIGS[case["model"]], case["rows"]
        weights = 3 * z["hidden_size"] * z["intermediate_size"]
        return {"bytes": weights * 0.53125 + 4 * M * z["hidden_size"], "flops": 2.0 * M * weights}
    if kind == "attend":
        lengths, H, G, n = ints(case["lengths"]), case["heads"], case["kv_heads"], case["new"]
        pairs = sum(n * c - n * (n - 1) // 2 for c in lengths)
        return {"bytes": sum(lengths) * G * 128 * 4 + len(lengths) * H * n * 128 * 4, "flops": 4.0 * 128 * H * pairs}
    if kind == "experts":
        z, T = EXPERTS[case["width"]], case["tokens"]
        D, E = z["width"], z["experts"]
        touched = E * (1.0 - (1.0 - z["top"] / E) ** T)
        return {"bytes": 2.0 * D * (E + 3 * z["shared"] + 3 * z["ff"] * touched) + T * D * 6, "flops": 2.0 * T * D * (3 * z["top"] * z["ff"] + 3 * z["shared"] + E)}
    T, D = sum(ints(case["lengths"])), case["width"]
    if kind == "decay":
        z = DECAY[D]
        H, dk, dv, low = z["heads"], z["dim"], z["vdim"], z["low"]
        weights = D * (2 * H * dk + 3 * H * dv + low) + low * H * dk
        states = len(ints(case["lengths"])) * H * dk * dv * 8
        return {"bytes": weights * 2.0 + T * D * 6 + states, "flops": 2.0 * T * weights + 5.0 * T * H * dk * dv}
    pairs, rows = (sum(v) for v in zip(*seen_keys(case)))
    if kind == "latent":
        z = LATENT[D]
        H, dn, dr, dv, R = z["heads"], z["dim"], z["rot_dim"], z["vdim"], z["rank"]
        weights = D * (H * (dn + dr) + R + dr) + R * H * (dn + dv) + D * H * dv
        return {"bytes": 2.0 * weights + 2.0 * rows * (R + dr) + T * D * 6, "flops": 2.0 * T * weights + 2.0 * H * pairs * (2 * R + dr)}
    z = GROUPED[case["design"]][D]
    H, G, dk, dv = z["heads"], z["kv_heads"], z["dim"], z["vdim"]
    weights = D * (H * dk + G * (dk + dv) + H + H * dv)
    return {"bytes": 2.0 * weights + 2.0 * rows * G * (dk + dv) + T * D * 6, "flops": 2.0 * T * weights + 2.0 * H * pairs * (dk + dv)}


# About four times the distance from 64 bits (mlp 0.0044, attend 0.0023, latent 0.0070, grouped 0.0044, experts 0.0032, decay
# 0.0038).  Decoding: the captured step and the operator sequence, both correct, are 0.023 apart, each 0.023 from 64 bits.
TOLERANCE = {"decode": 3e-2, "mlp": 1.6e-2, "attend": 8e-3, "latent": 2.4e-2, "grouped": 1.6e-2, "experts": 1.2e-2, "decay": 1.4e-2}


def tolerance(case):
    return {"rel": TOLERANCE[case["kind"]]}


# ---- the same in 64 bits, in plain torch ------------------------------------------------------------
def wide(t):
    return t.to(F64)


def unpack(layer):
    """The weights a packed layer stands for, ``[out, in]``."""
    words = layer.weight.view(torch.int32)
    codes = (words.unsqueeze(-1) >> torch.arange(0, 32, 4, device=DEV, dtype=torch.int32)) & 15
    rows = words.shape[0]
    codes = codes.reshape(rows, -1, 128).to(F64)
    return (codes * wide(layer.scales).unsqueeze(-1) + wide(layer.biases).unsqueeze(-1)).reshape(rows, -1)


def rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def frequencies(dims, base, factor=1.0, yarn=None):
    """One frequency per rotated pair and the factor on cos and sin."""
    f = [base ** (-2.0 * i / dims) / factor for i in range(dims // 2)]
    gain = 1.0
    if yarn:
        at = lambda turns: dims * math.log(yarn["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(at(yarn["fast"])), 0), min(math.ceil(at(yarn["slow"])), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        f = [v / yarn["factor"] * r + v * (1.0 - r) for v, r in zip(f, ramp)]
        gain = 0.1 * math.log(yarn["factor"]) + 1.0
    return torch.tensor(f, dtype=F64, device=DEV), gain


def rotate(x, pos, dims, base, factor=1.0, interleaved=False, yarn=None):
    """``x [T, heads, d]``: the first ``dims`` entries of every head, by its token's position."""
    f, gain = frequencies(dims, base, factor, yarn)
    angle = pos.to(F64)[:, None, None] * f
    c, s = torch.cos(angle) * gain, torch.sin(angle) * gain
    out = x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, dims // 2), slice(dims // 2, dims))
    u, v = x[..., a], x[..., b]
    out[..., a], out[..., b] = u * c - v * s, v * c + u * s
    return out


def softmax_attention(q, k, v, scale, see, cap=None, sink=None):
    """``q [n, H, dk]``, ``k [m, G, dk]``, ``v [m, G, dv]``, ``see [n, m]``; ``sink [H]``: one more exp(sink) in the denominator."""
    n, H, _ = q.shape
    group = H // k.shape[1]
    out = torch.empty((n, H, v.shape[2]), dtype=F64, device=DEV)
    for h in range(H):
        s = (q[:, h] @ k[:, h // group].t()) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~see, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], dim=1)
        p = torch.softmax(s, dim=1)
        out[:, h] = p[:, : k.shape[0]] @ v[:, h // group]
    return out


def exact_decode(case, seed):
    ckpt, cached, tokens = qwen(case, seed)
    lengths, a, m = ints(case["lengths"]), ckpt.args, ckpt.model
    H, G, d, eps = a.num_attention_heads, a.num_key_value_heads, a.head_dim, a.rms_norm_eps
    B = len(lengths)
    table = unpack(m.embed_tokens)
    x = table[tokens[:, :, 0].t().reshape(-1).long()]  # request by request, its steps in order
    pos = torch.cat([torch.arange(n, n + STEPS, device=DEV) for n in lengths])
    f = torch.arange(STEPS, device=DEV)
    for layer, (ck, cv) in zip(m.layers, cached):
        at, mlp = layer.self_attn, layer.mlp
        h = rms(x, eps) * wide(layer.input_layernorm.weight)
        q, k, v = (h @ unpack(p).t() for p in (at.q_proj, at.k_proj, at.v_proj))
        q = rotate(rms(q.view(-1, H, d), eps) * wide(at.q_norm.weight), pos, d, float(a.rope_theta))
        k = rotate(rms(k.view(-1, G, d), eps) * wide(at.k_norm.weight), pos, d, float(a.rope_theta))
        v = v.view(-1, G, d)
        o = torch.empty_like(q)
        for b, n in enumerate(lengths):
            rows = slice(b * STEPS, (b + 1) * STEPS)
            keys = torch.cat([wide(ck[0, :, b : b + n]), k[rows].transpose(0, 1)], dim=1)  # [G, n + STEPS, d]
            vals = torch.cat([wide(cv[0, :, b : b + n]), v[rows].transpose(0, 1)], dim=1)
            see = torch.arange(n + STEPS, device=DEV)[None, :] <= n + f[:, None]
            s = torch.einsum("tghd,gjd->gthj", q[rows].view(STEPS, G, H // G, d), keys) * d**-0.5
            p = torch.softmax(s.masked_fill(~see[None, :, None, :], -math.inf), dim=-1)
            o[rows] = torch.einsum("gthj,gjd->tghd", p, vals).reshape(STEPS, H, d)
        x = x + o.reshape(-1, H * d) @ unpack(at.o_proj).t()
        h = rms(x, eps) * wide(layer.post_attention_layernorm.weight)
        g, u = h @ unpack(mlp.gate_proj).t(), h @ unpack(mlp.up_proj).t()
        x = x + (g * torch.sigmoid(g) * u) @ unpack(mlp.down_proj).t()
    logits = (rms(x, eps) * wide(m.norm.weight)) @ table.t()
    return [logits.view(B, STEPS, -1)[:, t : t + 1] for t in range(STEPS)]


def exact_mlp(case, seed):
    (gate, up, down), x = mlp_inputs(case, seed)
    x = wide(x)
    g, u = x @ unpack(gate).t(), x @ unpack(up).t()
    return (g * torch.sigmoid(g) * u) @ unpack(down).t()


def exact_attend(case, seed):
    q, k, v, table, lengths = attend_inputs(case, seed)
    out = torch.empty(q.shape, dtype=F64, device=DEV)
    for b, n in enumerate(lengths.tolist()):
        ids = torch.from_numpy(table[b, : -(-n // QPAGE)]).to(DEV).long()
        keys, vals = (wide(t[ids].transpose(0, 1).reshape(t.shape[1], -1, 128)[:, :n]).transpose(0, 1) for t in (k, v))
        see = torch.arange(n, device=DEV)[None, :] <= torch.arange(n - case["new"], n, device=DEV)[:, None]
        out[b] = softmax_attention(wide(q[b]).transpose(0, 1), keys, vals, 128**-0.5, see).transpose(0, 1)
    return out


def positions(case):
    return [torch.arange(b, b + n, device=DEV) for n, b in zip(ints(case["lengths"]), ints(case["before"]))]


def exact_latent(case, seed):
    w, h, before = latent_inputs(case, seed)
    w, h, z = {k: wide(t) for k, t in w.items()}, wide(h), LATENT[case["width"]]
    H, dn, dr, dv, R = z["heads"], z["dim"], z["rot_dim"], z["vdim"], z["rank"]
    pos = positions(case)
    q = (h @ w["w_q"].t()).view(-1, H, dn + dr)
    down = h @ w["w_dkv"].t()
    every = torch.cat(pos)
    q_rot = rotate(q[..., dn:], every, dr, 10000.0)
    rows = torch.cat([rms(down[:, :R], EPS) * w["dkv_norm"], rotate(down[:, None, R:], every, dr, 10000.0)[:, 0]], dim=1)
    q_lat = torch.einsum("thd,hdr->thr", q[..., :dn], w["w_uk"].view(H, dn, R))
    o = torch.empty((h.shape[0], H, R), dtype=F64, device=DEV)
    at = 0
    for p, old in zip(pos, before):
        n = p.numel()
        keys = torch.cat([wide(old), rows[at : at + n]])
        j = torch.arange(keys.shape[0], device=DEV)[None, :]
        see = j <= p[:, None]
        if case["windowed"]:
            see = see & (p[:, None] - j < z["window"])
        o[at : at + n] = softmax_attention(torch.cat([q_lat[at : at + n], q_rot[at : at + n]], dim=2), keys[:, None], keys[:, None, :R], (dn + dr) ** -0.5, see)
        at += n
    return torch.einsum("thr,hvr->thv", o, w["w_uv"].view(H, dv, R)).reshape(-1, H * dv) @ w["w_o"].t()


def exact_grouped(case, seed):
    w, h, before = grouped_inputs(case, seed)
    w, h, z, design = {k: wide(t) for k, t in w.items()}, wide(h), GROUPED[case["design"]][case["width"]], case["design"]
    H, G, dk, dv = z["heads"], z["kv_heads"], z["dim"], z["vdim"]
    pos = positions(case)
    every = torch.cat(pos)
    q, k, v = h @ w["q"].t(), h @ w["k"].t(), (h @ w["v"].t()).view(-1, G, dv)
    if design == "window":
        q, k = (rms(q, EPS) * w["q_norm"]).view(-1, H, dk), (rms(k, EPS) * w["k_norm"]).view(-1, G, dk)
        q, k = (rotate(t, every, z["rot"], 100000.0, yarn=YARN) for t in (q, k))
    elif design == "chunk":
        q, k = rms(q.view(-1, H, dk), EPS) * w["q_norm"], rms(k.view(-1, G, dk), EPS) * w["k_norm"]
    else:
        q, k = (rotate(t.view(-1, n, dk), every, z["rot"], 10000.0, factor=8.0, interleaved=True) for t, n in ((q, H), (k, G)))
    o = torch.empty((h.shape[0], H, dv), dtype=F64, device=DEV)
    at = 0
    for p, old in zip(pos, before):
        n, b = p.numel(), old.shape[0]
        keys = torch.cat([wide(old[:, : G * dk]).view(b, G, dk), k[at : at + n]])
        vals = torch.cat([wide(old[:, G * dk :]).view(b, G, dv), v[at : at + n]])
        j = torch.arange(b + n, device=DEV)[None, :]
        i = p[:, None]
        see = j <= i
        if design == "window":
            see = see & ((i - j < z["size"]) | (j < z["keep_first"]))
        elif design == "chunk":
            see = see & (i // z["size"] == j // z["size"])
        sink = w["sink"] if design == "window" else torch.zeros(H, dtype=F64, device=DEV) if design == "chunk" else None
        o[at : at + n] = softmax_attention(q[at : at + n], keys, vals, dk**-0.5, see, cap=z.get("softcap"), sink=sink)
        at += n
    if design != "causal":
        o = o * torch.sigmoid(h @ w["g"].t())[:, :, None]
    return o.reshape(-1, H * dv) @ w["o"].t()


def exact_experts(case, seed):
    w, h = experts_inputs(case, seed)
    h = wide(h)

    def ff(x, gate, up, down):
        g = x @ wide(gate).t()
        return (g * torch.sigmoid(g) * (x @ wide(up).t())) @ wide(down).t()

    logits = h @ wide(w["router"]).t() + wide(w["bias"])
    val, idx = torch.topk(logits, EXPERTS[case["width"]]["top"], dim=-1)
    share = torch.softmax(val, dim=-1)
    out = ff(h, w["s_gate"], w["s_up"], w["s_down"])
    for e in range(w["gate"].shape[0]):
        t, slot = (idx == e).nonzero(as_tuple=True)
        if t.numel():
            out[t] += share[t, slot][:, None] * ff(h[t], w["gate"][e], w["up"][e], w["down"][e])
    return out


def exact_decay(case, seed):
    w, h, initial = decay_inputs(case, seed)
    w, h, z = {k: wide(t) for k, t in w.items()}, wide(h), DECAY[case["width"]]
    H, dk, dv = z["heads"], z["dim"], z["vdim"]
    q, k, v = (h @ w["q"].t()).view(-1, H, dk) * dk**-0.5, (h @ w["k"].t()).view(-1, H, dk), (h @ w["v"].t()).view(-1, H, dv)
    alpha = torch.exp(torch.nn.functional.logsigmoid((h @ w["a1"].t()) @ w["a2"].t() + w["bias"]) / z["tau"]).view(-1, H, dk)
    o = torch.empty((h.shape[0], H, dv), dtype=F64, device=DEV)
    states = []
    at = 0
    for s, (n, b) in enumerate(zip(ints(case["lengths"]), ints(case["before"]))):
        S = wide(initial[s]) if b else torch.zeros((H, dk, dv), dtype=F64, device=DEV)
        for t in range(at, at + n):
            S = alpha[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
            o[t] = (q[t][:, None, :] @ S)[:, 0]
        states.append(S)
        at += n
    g = h @ w["g"].t()
    out = ((rms(o, EPS) * w["norm"]).reshape(-1, H * dv) * g * torch.sigmoid(g)) @ w["o"].t()
    return {"out": out, "state": torch.stack(states)}


EXACT = {k: globals()["exact_" + k] for k in KINDS}


def exact(case, seed):
    return EXACT[case["kind"]](case, seed)
