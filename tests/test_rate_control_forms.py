"""Rate control's closed forms against the step-by-step ones, over all inputs:
the search over known answers (every pattern of answers for up to 10 values,
thresholds for up to 32) against the reference's binary search, and the number
of gtli values at which a coefficient stays non-zero against trying each."""
import os
import shutil
import subprocess

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "svt-jpeg-xs_gb300", "csrc", "jxs_enc_kernels.cu")

MAIN = r"""
static int steps(uint32_t small, uint32_t big, int n, int below, int step) {
    BSearch bs;
    bs_init(bs, 0, n, below, step);
    int res, next = BS_BEGIN, v = 0;
    while ((res = bs_next(bs, next, &v)) == BS_CONTINUE)
        next = (small >> v) & 1u ? BS_TOO_SMALL : (big >> v) & 1u ? BS_TOO_BIG : BS_OUT_OF_RANGE;
    return res == BS_FOUND ? v : -1;
}
static long check(uint32_t small, uint32_t big, int n) {
    long bad = 0;
    for (int below = 0; below < 2; below++)
        for (int step = 0; step <= 6; step += 6) {
            const int s = (below ? 6 >= n : 6 > n) ? 0 : step;
            bad += mask_search(small, big, n, below, s) != steps(small, big, n, below, s);
        }
    return bad;
}
int main() {
    long bad = 0;
    for (int n = 0; n <= 9; n++) {
        long all = 1;
        for (int i = 0; i <= n; i++) all *= 3;
        for (long x = 0; x < all; x++) {
            uint32_t small = 0, big = 0;
            long y = x;
            for (int i = 0; i <= n; i++, y /= 3) {
                small |= (uint32_t)(y % 3 == 1) << i;
                big |= (uint32_t)(y % 3 == 2) << i;
            }
            bad += check(small, big, n);
        }
    }
    for (int n = 10; n <= 30; n++)
        for (int a = 0; a <= n + 1; a++)
            for (int b = a; b <= n + 1; b++) {
                const uint32_t in = (1u << (n + 1)) - 1u, small = ((1u << a) - 1u) & in;
                bad += check(small, in & ~((1u << b) - 1u) & ~small, n);
            }
    for (uint32_t m = 0; m < 32768; m++)
        for (uint32_t g = m ? 32 - __builtin_clz(m) : 0; g <= 15; g++) {
            uint32_t n = 0, bits = 0;
            while (n < g && m * ((2u << (g - n)) - 1u) >= (1u << g)) n++;
            while (bits < 15 && m >> bits) bits++;
            bad += nz_levels(m, g, 1) != n;
            bad += nz_levels(m, g, 0) != bits;
        }
    printf("%ld\n", bad);
    return bad != 0;
}
"""


def between(text, first, last):
    i = text.index(first)
    return text[i:text.index(last, i)]


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_forms_equal_the_steps(tmp_path):
    text = open(SOURCE).read()
    parts = ["#include <stdint.h>\n#include <stdio.h>\n#define DEV static inline\n"
             "static int __popc(uint32_t x) { return __builtin_popcount(x); }\n"
             "static int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }\n",
             between(text, "struct BSearch {", "/* A slice's even split"),
             between(text, "DEV int mask_search(", "/* The precinct searches of"),
             between(text, "DEV uint32_t nz_levels(", "/* Byte cost of every"), MAIN]
    src = tmp_path / "forms.cpp"
    src.write_text("".join(parts))
    exe = str(tmp_path / "forms")
    subprocess.run(["g++", "-O2", "-o", exe, str(src)], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout.strip() == "0"
