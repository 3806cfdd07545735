"""Rate control's search over known answers with all 32 values of a word
(quantizations 0 to 31, the most there are): every threshold, the words of all
ones and all zeros, and patterns without a threshold, against the reference's
binary search."""
import shutil
import subprocess

import pytest

import test_rate_control_forms as forms

FULL_WORDS = r"""
int main() {
    const int n = 31;
    const uint32_t all = 0xffffffffu;
    auto low = [](int k) { return k >= 32 ? 0xffffffffu : (1u << k) - 1u; };
    long bad = 0, seen = 0;
    for (int a = 0; a <= 32; a++)
        for (int b = a; b <= 32; b++) {
            bad += check(low(a), all & ~low(b), n); /* too small, out of range, too big */
            bad += check(low(a), low(b) & ~low(a), n); /* too small, too big, out of range */
            seen += 2;
        }
    uint32_t x = 12345u;
    for (int i = 0; i < 200000; i++) {
        uint32_t w[2];
        for (int k = 0; k < 2; k++) {
            w[k] = 0;
            for (int h = 0; h < 2; h++) {
                x = x * 1664525u + 1013904223u;
                w[k] = (w[k] << 16) | (x >> 16);
            }
        }
        bad += check(w[0], w[1] & ~w[0], n);
        bad += check(w[0] & w[1], all & ~(w[0] & w[1]), n);
        seen += 2;
    }
    printf("%ld of %ld\n", bad, seen);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_search_over_32_values(tmp_path):
    text = open(forms.SOURCE).read()
    src = tmp_path / "words.cpp"
    src.write_text("#include <stdint.h>\n#include <stdio.h>\n#define DEV static inline\n"
                   "static int __popc(uint32_t x) { return __builtin_popcount(x); }\n"
                   + forms.between(text, "struct BSearch {", "/* A slice's even split")
                   + forms.between(text, "DEV int mask_search(", "/* The precinct searches of")
                   + forms.MAIN[:forms.MAIN.index("int main()")] + FULL_WORDS)
    exe = str(tmp_path / "words")
    subprocess.run(["g++", "-O2", "-fsanitize=undefined", "-fno-sanitize-recover=undefined", "-o", exe, str(src)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
