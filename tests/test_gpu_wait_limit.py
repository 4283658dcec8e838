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
