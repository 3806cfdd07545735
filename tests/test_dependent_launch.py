"""Kernels that may be launched before the kernel ahead of them in the stream
has finished (jxs_launch, dep_wait) make no promise to the compiler about
memory which that kernel may still write: `__restrict__` would let loads move
above the wait, or through the non-coherent path, and is for the handle's
configuration alone."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "svt-jpeg-xs_gb300", "csrc")


def code(path):
    with open(path) as f:
        text = f.read()
    return re.sub(r"/\*.*?\*/|//[^\n]*", "", text, flags=re.S)


SOURCES = [p for p in sorted(glob.glob(os.path.join(CSRC, "*.cu"))) if "dep_wait()" in code(p)]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_restrict_only_on_the_configuration(path):
    text = code(path)
    for m in re.finditer(r"__restrict__|__ldg\b", text):
        assert m.group() == "__restrict__" and re.search(r"const\s+jxs_cfg_t\s*\*\s*$", text[:m.start()]), text[m.start() - 60:m.end() + 20]


def test_sources_found():
    assert {os.path.basename(p) for p in SOURCES} >= {"jxs_gpu.cu", "jxs_enc_kernels.cu", "jxs_dec_kernels.cu", "jxs_fwd_dwt.cu",
                                                      "jxs_inv_dwt.cu"}
