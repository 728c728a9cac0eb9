"""over_h (csu_b200/csrc/cuda/kernels.cuh) itself, compiled for the host from its source text: equal to the division by
the step, bit for bit, on random doubles of every exponent, on quotients beside a midpoint of two doubles, zeros of both
signs, both edges of its range, subnormals, the largest doubles, infinities and NaN."""
import os
import random
import re
import struct
import subprocess

import pytest

import test_block_step

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
int main()
{
    unsigned long long b, n = 0, bad = 0;
    while (scanf("%llx", &b) == 1) {
        double a, q, w;
        memcpy(&a, &b, 8);
        q = over_h(a);
        volatile double h = BLOCK_H;
        w = a / h;
        n++;
        if (memcmp(&q, &w, 8) != 0 && !(isnan(q) && isnan(w))) {
            if (bad++ < 10) printf("%a: %a instead of %a\n", a, q, w);
        }
    }
    printf("n=%llu bad=%llu\n", n, bad);
    return bad ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    src = open(os.path.join(ROOT, "csu_b200", "csrc", "cuda", "kernels.cuh")).read()
    parts = [re.search(r"^constexpr double BLOCK_H = [^;]*;$", src, re.M).group(0)]
    for name in ("over_h_any", "over_h"):
        parts.append(re.search(r"^[^\n]*\bdouble %s\(double a\)\n\{\n.*?^\}$" % name, src, re.M | re.S).group(0))
    d = tmp_path_factory.mktemp("over_h")
    cpp = "#include <math.h>\n#include <stdio.h>\n#include <string.h>\n" + "".join(
        "#define %s\n" % w for w in ("__host__", "__device__", "__noinline__", "__forceinline__"))
    (d / "over_h.cpp").write_text(cpp + "\n\n".join(parts) + MAIN)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(d / "over_h"), str(d / "over_h.cpp")],
                   check=True)

    def run(bits):
        r = subprocess.run([str(d / "over_h")], input="\n".join("%x" % b for b in bits), capture_output=True, text=True)
        assert r.returncode == 0 and "n=%d bad=0" % len(bits) in r.stdout, r.stdout
    return run


def _bits(a):
    return struct.unpack("<Q", struct.pack("<d", a))[0]


def test_random_doubles_of_every_exponent(check):
    rng = random.Random(11)
    check([rng.getrandbits(1) << 63 | e << 52 | rng.getrandbits(52) for e in range(0x7ff) for _ in range(60)])


def test_special_values_and_range_edges(check):
    edges = [_bits(v) for v in (0.0, 2.0 ** -900, 2.0 ** 900, 5e-324, 2.2250738585072014e-308,
                                1.7976931348623157e308, float("inf"), 1e-6, 1.0)]
    near = [b + k for b in edges for k in (-1, 0, 1) if 0 <= b + k <= 0x7ff8000000000000]
    check(near + [0x7ff8000000000000] + [b | 1 << 63 for b in near])


def test_quotients_beside_midpoints(check):
    """The dividends that test_block_step finds near a midpoint, through the function, at both signs and four scales."""
    found = []
    keep = test_block_step._right
    test_block_step._right = lambda a, zh, zl: found.append(a) or True
    try:
        test_block_step.test_every_quotient_near_a_midpoint()
    finally:
        test_block_step._right = keep
    assert len(found) > 20
    check([_bits(s * a * 2.0 ** e) for a in found for s in (1, -1) for e in (-300, -60, 0, 800)])
