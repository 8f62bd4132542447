"""The projections' register limits, as the compiler reports them: the largest CTAs of fp16 rows of a multiple of 4 columns in grids
of more CTAs than SMs (six slices, 768 threads) fit an SM twice, and nothing spills."""
import os
import re
import subprocess

import pytest

from mx230_b200 import build


def test_registers_and_spills(tmp_path):
    nvcc = build.find_nvcc()
    if nvcc is None:
        pytest.skip("no nvcc")
    out = subprocess.run([nvcc, *build.ARCH_FLAGS, "-O3", "-std=c++17", "-I", os.path.join(build.ROOT, "include"), "-Xptxas", "-v",
                          "-c", os.path.join(build.CSRC, "proj.cu"), "-o", str(tmp_path / "proj.o")],
                         capture_output=True, text=True, check=True)
    found = {}
    for m in re.finditer(r"Compiling entry function '\S*gemv_heads_kernelI(\S+?)Li(\d)E\S*'(.*?)Used (\d+) registers",
                         out.stdout + out.stderr, re.S):
        found[(m.group(1), int(m.group(2)))] = int(m.group(4))
        assert "0 bytes spill stores, 0 bytes spill loads" in m.group(3), m.group(0)
    assert set(found) == {("f", 4), ("6__half", 4), ("6__half", 8), ("a", 4)}
    per_thread = {k: -(-r // 8) * 8 for k, r in found.items()}   # allocated in eights
    assert 2 * 768 * per_thread[("6__half", 4)] <= 65536
    assert 2 * 640 * per_thread[("f", 4)] <= 65536 and 2 * 320 * per_thread[("6__half", 8)] <= 65536
