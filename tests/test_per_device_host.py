"""Kernel attributes are set once per device, and a failure is not remembered."""

import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "tiny-llm_b200" / "csrc"

PROGRAM = """
#include "per_device.h"
#include <cstdio>
int main() {
    static tl::PerDevice ready;
    int calls = 0;
    bool works = false;
    auto set = [&] { return ++calls, works; };
    if (ready(0, set) || ready(0, set) || calls != 2) return 1;            // failed twice, tried twice
    works = true;
    if (!ready(0, set) || !ready(0, set) || calls != 3) return 2;          // set once
    if (!ready(1, set) || !ready(1, set) || calls != 4) return 3;          // another device's own
    if (!ready(63, set) || !ready(63, set) || calls != 5) return 4;
    if (!ready(64, set) || !ready(64, set) || calls != 7) return 5;        // past the mask: every time
    return 0;
}
"""


def test_set_once_per_device(tmp_path):
    source, program = tmp_path / "p.cpp", tmp_path / "p"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-o", str(program), str(source)], check=True)
    assert subprocess.run([str(program)]).returncode == 0


def test_the_paged_attention_kernels_use_it():
    source = (CSRC / "attention_prefill_tc.cu").read_text()
    assert source.count("cudaFuncSetAttribute") == 2 and source.count("static PerDevice") == 1  # in the one helper that all launches go through
    assert "static bool configured" not in source and "static const bool configured" not in source


def test_the_kernels_of_packed_products_of_few_rows_use_it():
    for name in ("w4a16_matvec.cu", "w4a16_skinny.cu", "decode_step.cu"):
        source = (CSRC / name).read_text()
        assert "cudaFuncSetAttribute" in source and "static PerDevice" in source and "static bool configured" not in source
