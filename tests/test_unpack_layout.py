"""Unpacking's shared memory: what a decoder sets aside holds the full layout
for every number of groups and segments, and the lean one with the bytes that
are left over."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "svt-jpeg-xs_gb300", "csrc")

MAIN = r"""
#include <stdio.h>
#include "jxs_kernels.cuh"
int main() {
    long bad = 0;
    for (uint32_t g = 0; g < 66000; g += g < 9000 ? 1 : 13)
        for (uint32_t s = 1; s <= JXS_MAXSEG; s += s < 8 ? 1 : 7) {
            bad += uk_layout(0, g, s, false).end > uk_reserved(g, s, 0);
            bad += uk_layout(0, g, s, false).top_end > uk_reserved(g, s, 1);
            bad += uk_layout(0, g, s, true).end > uk_reserved(g, s, 0) + UK_LEAN_MORE;
        }
    printf("%ld layouts do not fit\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir("/usr/local/cuda/include"), reason="no host compiler or CUDA headers")
def test_layouts_fit(tmp_path):
    src, exe = tmp_path / "t.cpp", str(tmp_path / "t")
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", "/usr/local/cuda/include", "-o", exe, str(src)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
