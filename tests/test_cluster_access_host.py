"""Kernels that reach into the shared memory of another CTA of their cluster: a CTA that has not started has none, and being scheduled together is no
promise of having started, so a cluster barrier comes before the first access, and one after the last before a CTA may leave."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tiny-llm_b200" / "csrc"
ACCESS = re.compile(r"mapa\.|st\.shared::cluster|ld\.shared::cluster|map_shared_rank|\bp_mbar_arrive_leader\(|\bp_tc_commit2\(|\bp_tc_mma2\(")
BARRIER = re.compile(r"barrier\.cluster\.wait|\bp_cluster_sync\(\)|cluster\.sync\(\)")


def kernels(source):
    """Name and body of every kernel, comments taken out."""
    source = re.sub(r"//[^\n]*|__(launch_bounds|cluster_dims|maxnreg)__\s*\((?:[^()]|\([^()]*\))*\)", "", source)
    for head in re.finditer(r"__global__[^;{(]*?(\w+)\s*\([^;{]*\)\s*\{", source):
        depth, end = 1, head.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(source[end], 0)
            end += 1
        yield head.group(1), source[head.end() : end]


CASES = [(path.name, name, body) for path in sorted(CSRC.rglob("*.cu")) for name, body in kernels(path.read_text()) if ACCESS.search(body)]


def test_the_kernels_are_found():
    assert {name for _, name, _ in CASES} >= {"w4a16_gemm2_kernel", "w4a16_skinny_reduce_norm_kernel", "paged_attention_flash_kernel"}


@pytest.mark.parametrize("path,name,body", CASES, ids=[name for _, name, _ in CASES])
def test_a_cluster_barrier_on_either_side(path, name, body):
    accesses, barriers = ([m.start() for m in pattern.finditer(body)] for pattern in (ACCESS, BARRIER))
    assert barriers and barriers[0] < accesses[0], f"{path}: {name} reaches into another CTA before that is known to run"
    assert barriers[-1] > accesses[-1], f"{path}: {name} may leave while another CTA reaches into it"
