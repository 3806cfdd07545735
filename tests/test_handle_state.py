"""What a handle's frames share on the host, compiled with the host compiler."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "svt-jpeg-xs_gb300", "csrc")


def run(tmp_path, body, *flags):
    src, exe = tmp_path / "t.cpp", str(tmp_path / "t")
    src.write_text('#include <stdio.h>\n#include <thread>\n#include <vector>\n#include "jxs_handle.h"\n'
                   "#define CHECK(x) do { if (!(x)) { printf(\"line %d: %s\\n\", __LINE__, #x); return 1; } } while (0)\n"
                   "int main() {\n" + body + "\nreturn 0; }\n")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", "-I", CSRC, *flags, "-o", exe, str(src)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


needs_compiler = pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")


@needs_compiler
def test_results_in_place_exactly_for_a_frame_alone(tmp_path):
    """From the handle's first frame on and however many came before."""
    run(tmp_path, """
    HandleLoad l;
    for (int i = 0; i < 1000; i++) {
        CHECK(l.submit() == 1);
        for (int k = 0; k < i % 3; k++) CHECK(l.submit() == 0);
        for (int k = 0; k < i % 3; k++) l.done();
        CHECK(l.submit() == 0);
        l.done();
        l.done();
    }
    CHECK(sizeof(l) == sizeof(int));  /* no count that could overflow */
    """)
