"""Operands that the launch before may have written are read behind the wait for it (programmatic dependent launch: a kernel may become resident while
its predecessor still runs)."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tiny-llm_b200" / "csrc"
WAIT = re.compile(r"griddep_wait\(\)")


def body_of(path, kernel):
    source = re.sub(r"//[^\n]*", "", (CSRC / path).read_text())
    head = re.search(r"\b" + kernel + r"\s*\([^;{]*\)\s*\{", source)
    depth, end = 1, head.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(source[end], 0)
        end += 1
    return source[head.end() : end]


@pytest.mark.parametrize(
    "path,kernel,operands",
    [
        ("elementwise.cu", "decode_qk_norm_rope_append_d128_kernel", "qkv part offsets bt cl kp vp"),
        ("elementwise.cu", "decode_qk_norm_rope_append_kernel", "qkv offsets bt cl"),
        ("w4a16_skinny.cu", "w4a16_skinny_reduce_norm_kernel", "part res norm_w"),
        ("w4a16_skinny.cu", "w4a16_skinny_reduce4_kernel", "part res"),
    ],
)
def test_nothing_of_the_predecessor_is_read_ahead(path, kernel, operands):
    body = body_of(path, kernel)
    ahead = body[: WAIT.search(body).start()]
    read = [name for name in operands.split() if re.search(r"\b" + name + r"\s*\[|\b(ld_cg|__ldg|ldg_stream)\(\s*" + name + r"\b|\*\s*" + name + r"\b", ahead)]
    assert not read, f"{kernel} reads {read} before griddep_wait()"


def test_the_experts_sum_reads_through_l2():
    """Its operands are the launch before's, or the other stream's joined right ahead of it: loads that the compiler may move ahead of the wait (plain ones,
    of pointers that it takes for read-only) are not used."""
    body = body_of("blocks/blocks_moe.cu", "moe_combine_kernel")
    behind = body[WAIT.search(body).end() :]
    plain = [name for name in ("pair_out", "gate", "shared", "shared_gate", "idx", "h") if re.search(r"\b" + name + r"\s*\[|moe_load<\w+>\(\s*" + name + r"\b", behind)]
    assert not plain and "griddep_wait" not in behind


def test_lists_are_read_ahead_only_where_the_caller_says_what_is_before():
    """The experts' second product reads the lists before its wait behind a first product of theirs, and nowhere else."""
    kernel = body_of("blocks/blocks_moe_tc.cu", "moe_tc_kernel")
    first_read = re.search(r"a\.(counters|chunks|sorted_pair)\b", kernel).start()
    assert re.search(r"if \(!a\.second\) \{\s*tl::griddep_wait\(\);", kernel[:first_read])
    assert re.search(r"a\.second = p\.second;", body_of("blocks/blocks_moe_tc.cu", "moe_tc_product"))
    assert "stream, false)" in body_of("blocks/blocks_moe.cu", "tlb_moe_down")
    for entry in ("tlb_moe_gate_up", "tlb_moe_up"):
        assert "true" not in body_of("blocks/blocks_moe.cu", entry)


@pytest.mark.parametrize("loaded_before", [True, False])
def test_one_switch_for_both_libraries(monkeypatch, loaded_before):
    """``set_pdl`` reaches the blocks library whether it was loaded before the call or after it."""
    from extensions_b200 import tiny_llm_ext_b200 as ext
    from extensions_b200.tiny_llm_ext_b200 import blocks

    asked, real = [], ext.ctypes.CDLL

    class Library:
        def __init__(self, path):
            self.real = real(path)

        def __getattr__(self, name):
            return asked.append if name == "tlb_set_pdl" else getattr(self.real, name)

    monkeypatch.setattr(blocks, "_lib", None)
    monkeypatch.setattr(blocks, "_pdl", None)
    monkeypatch.setattr(blocks.ctypes, "CDLL", Library)
    monkeypatch.setattr(blocks, "_SIGNATURES", {k: v for k, v in blocks._SIGNATURES.items() if k != "tlb_set_pdl"})
    try:
        if loaded_before:
            blocks.load_library()
        ext.set_pdl(False)
        if not loaded_before:
            blocks.load_library()
        assert asked == [0]
    finally:
        ext.set_pdl(True)
