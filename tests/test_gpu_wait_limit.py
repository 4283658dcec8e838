"""A wait that nothing ends: the CTA is marked, further waits return, what it stores is NaN, and the host can read the count."""

import ctypes
import subprocess
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "tiny-llm_b200" / "csrc"

SOURCE = """
#include <cuda_runtime.h>
#include "tc_wait.cuh"
// CTA 0 waits on a barrier at which nothing arrives, CTA 1 on one that is over.  out: per CTA (answer, answer of a second wait, factor).
__global__ void wait_kernel(float *out) {
    __shared__ __align__(8) unsigned long long bars[2];
    __shared__ int mark;
    volatile int *dead = &mark;
    const uint32_t first = tl::g_smem_u32(&bars[0]), second = tl::g_smem_u32(&bars[1]);
    if (threadIdx.x == 0) {
        *dead = 0;
        tl::g_mbar_init(first, 1), tl::g_mbar_init(second, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0 && blockIdx.x == 1) tl::g_mbar_arrive(first), tl::g_mbar_arrive(second);
    __syncthreads();
    if (threadIdx.x < 32) {
        const bool ok = tl::tc_wait(first, 0, dead, 1000);
        const bool more = tl::tc_wait(second, 0, dead);  // of a marked CTA: at once, whatever the limit
        if (threadIdx.x == 31) out[3 * blockIdx.x] = ok, out[3 * blockIdx.x + 1] = more, out[3 * blockIdx.x + 2] = tl::tc_verdict(ok, dead);
    }
    __syncthreads();
    tl::tc_settle(dead);
}
extern "C" long long run(float *out) {
    wait_kernel<<<2, 64>>>(out);
    return cudaDeviceSynchronize() == cudaSuccess ? tl::read_gave_up() : -2;
}
"""


@pytest.mark.gpu
def test_expired_wait_is_counted_and_poisons(tmp_path):
    source, lib = tmp_path / "wait.cu", tmp_path / "wait.so"
    source.write_text(SOURCE)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", str(CSRC),
                    "-o", str(lib), str(source)], check=True)
    run = ctypes.CDLL(str(lib)).run
    run.restype, run.argtypes = ctypes.c_longlong, [ctypes.c_void_p]
    out = torch.full((6,), -1.0, device="cuda")
    torch.cuda.synchronize()
    assert run(out.data_ptr()) == 1
    got = out.tolist()
    assert got[:2] == [0.0, 0.0] and got[2] != got[2] and got[3:] == [1.0, 1.0, 1.0]


def test_batcher_hands_over_no_answer_after_a_wait_gave_up(cpu_ext, monkeypatch):
    import tiny_llm_b200.batch as batch

    given_up = [3]  # of an earlier batcher
    monkeypatch.setattr(batch, "_waits_given_up", lambda: given_up[0])

    class Model:
        num_hidden_layers = 0

        def create_kv_cache(self):
            return []

        def __call__(self, tokens, offsets, caches, logits_to_keep=1):
            return torch.nn.functional.one_hot(torch.full((tokens.shape[0], 1), 2), 5).float()

    def serve():
        return batch.ContinuousBatcher(Model(), None, [[1, 2], [3]], max_seq_len=8, batch_size=1, verbose=False, max_new_tokens=[2, 2])

    assert [i for i, _ in serve().run()] == [0, 1]
    late = serve()
    given_up[0] = 4
    with pytest.raises(RuntimeError, match="gave up waiting"):
        late.run()
    assert late.results == []


@pytest.mark.gpu
@pytest.mark.parametrize("contexts", [[131072], [40, 131072, 0]])
def test_a_decoding_step_whose_waits_run_out_shows_it(cuda_device, contexts):
    """A limit of 64 polls, some 50 us, where others attend 7000 keys a CTA (about 360 us): no logit, token, key or value that looks right; the next step is
    as before."""
    from extensions_b200 import tiny_llm_ext_b200 as ext
    from tiny_llm_b200 import Qwen3ModelWeek3
    from tiny_llm_b200.engine import DecodeEngine
    from tiny_llm_b200.synthetic import synthetic_qwen3

    dims = dict(hidden_size=512, num_hidden_layers=3, num_attention_heads=8, num_key_value_heads=2, head_dim=128, intermediate_size=1536, vocab_size=528)
    dev, B = cuda_device, len(contexts)
    model = Qwen3ModelWeek3(synthetic_qwen3(dims, seed=1, device=dev, realistic=True), page_size=128)
    pages = [-(-c // 128) for c in contexts]
    engine = DecodeEngine(model, B, max(contexts), dev)
    engine.reserve_pools(sum(pages))
    slabs = [t for p in model.page_pools for t in (p._key_pages, p._value_pages)]
    for slab in slabs:
        slab.normal_()
    before = [t.clone() for t in slabs]
    engine.tables.fill_(-1)
    for b, n in enumerate(pages):
        engine.tables[:, b, :n] = torch.arange(sum(pages[:b]), sum(pages[: b + 1]), device=dev, dtype=torch.int32)
    engine.tokens.fill_(9)
    engine.context_lens.copy_(torch.tensor(contexts, device=dev))
    engine.offsets.copy_((engine.context_lens - 1).clamp(min=0))
    step = engine._one_launch_step()
    limit = step.workspace[4:8].view(torch.int32)

    def run(polls):
        for slab, old in zip(slabs, before):
            slab.copy_(old)
        limit.fill_(polls)
        step.launch()
        return engine.logits.clone(), engine.next_tokens.tolist(), [t.clone() for t in slabs]

    logits, tokens, right = run(0)
    count = ext.waits_given_up()
    assert bool(logits.isfinite().all()) and min(tokens) >= 0
    late, none, _ = run(1)
    assert bool(late.isnan().all()) and none == [-1] * B and ext.waits_given_up() > count
    for k, old, good in zip(slabs, before, right):  # a row of the newest token is the right one or no number
        changed = (k != old).any(-1)
        assert bool((~k[changed].isfinite() | (k[changed] == good[changed])).all())
    count = ext.waits_given_up()
    again, same, kept = run(0)
    assert torch.equal(again, logits) and same == tokens and all(torch.equal(a, b) for a, b in zip(kept, right)) and ext.waits_given_up() == count
