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


@needs_compiler
def test_frames_located_first(tmp_path):
    """None, then for a while after each frame that was not at the split,
    twice as long each time up to a limit; then the split is tried again."""
    run(tmp_path, """
    DecHints h;
    for (int i = 0; i < 100; i++) CHECK(!h.locate());
    int want = DecHints::kFirst;
    for (int round = 0; round < 20; round++) {
        h.elsewhere();
        h.elsewhere();  /* found by another frame in flight at the same time: no more for that */
        for (int i = 0; i < want; i++) CHECK(h.locate());
        CHECK(!h.locate());
        if (want < DecHints::kMost) want *= 2;
    }
    CHECK(want == DecHints::kMost);
    """)


@needs_compiler
def test_no_data_race(tmp_path):
    """Frames submitted and completed by several threads at a time."""
    probe = tmp_path / "p.cpp"
    probe.write_text("int main() { return 0; }")
    exe = str(tmp_path / "p")
    if subprocess.run(["g++", "-fsanitize=thread", "-o", exe, str(probe)], capture_output=True).returncode or subprocess.run([exe]).returncode:
        pytest.skip("no thread sanitizer here")
    run(tmp_path, """
    DecHints h;
    HandleLoad l;
    std::atomic<long> located{0}, alone{0};
    std::vector<std::thread> t;
    for (int k = 0; k < 4; k++)
        t.emplace_back([&, k] {
            for (int i = 0; i < 20000; i++) {
                alone += l.submit();
                located += h.locate();
                if (i % 1000 == k) h.elsewhere();
                if (i == 500) h.vpred.store(1);
                located += h.vpred.load() < 0;
                l.done();
            }
        });
    for (auto& x : t) x.join();
    CHECK(l.submit() == 1 && located > 0 && alone > 0);
    """, "-fsanitize=thread")
