"""csrc/fp64_exact.cuh compiled as host C++: every form gives the bits of the
plain double operation it stands for, over random and edge operands."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "stochastic-parker_gb300" / "csrc"

PROGRAM = r"""
#include "fp64_exact.cuh"
#include <cstdio>
#include <random>
using namespace gpat;
static bool same(double a, double b) { return hi_word(a) == hi_word(b) && lo_word(a) == lo_word(b); }
int main() {
    std::mt19937_64 r(12345);
    long bad = 0, used = 0;
    for (long i = 0; i < 4000000; ++i) {
        const uint64_t a = r(), b = r();
        uint32_t fu = (uint32_t)a;
        if (i % 7 == 0) fu &= 0xffff0000u;
        if (i % 11 == 0) fu = (fu & 0xff800000u) | ((fu & 3) ? 0x7fffffu : 1u);
        if (i % 19 == 0) fu &= 0x80000000u;
        if (i % 23 == 0) fu &= 0x807fffffu;          // subnormals
        const float v = bits_float(fu);
        const bool sub = v != 0.0f && std::fabs(v) < 1.17549435e-38f;
        if (odd_float(v) != (sub || !(std::fabs(v) <= 3.4028235e38f))) ++bad;
        double w = from_words(0x3f000000u + ((uint32_t)(b >> 32) & 0x00ffffffu), (uint32_t)b);
        if (i % 5 == 0) w = from_words(hi_word(w), 0u);
        if (i % 17 == 0) w = from_words(hi_word(w) | 0xfffffu, 0xffffffffu);
        const Weight t = weight(w);
        if (!odd_float(v) && t.ok) {
            ++used;
            if (!same(scaled(v, t), 0.0 + (double)v * w)) ++bad;
            if (!same(widen(v), 0.0 + (double)v)) ++bad;
        }
        const double d = from_words(0x3ff00000u + ((uint32_t)(a >> 32) & 0xfffffu) +
                                        (((uint32_t)(a >> 60) - 8u) << 20), (uint32_t)(a >> 7));
        double x = from_words(0x3ff00000u + ((uint32_t)(b >> 32) & 0xfffffu) +
                                  (((uint32_t)(b >> 58) - 32u) << 20), (uint32_t)b);
        if (i % 3 == 0) x = from_words(hi_word(x), 0u);
        if (i % 29 == 0) x = 0.0;
        if (i % 31 == 0) x = from_words(0x00100000u + (uint32_t)(a & 0xff), (uint32_t)b);
        for (double q : {d, 3.0, 1.0 / 2048, 0.125 / 48, 0.1, 1e300, 4.9e-324, 0.0})
            if (!same(div_by(x, q, reciprocal(q)), x / q) && !(x == 0.0 && q == 0.0)) ++bad;
        const uint32_t A = (uint32_t)a, B = (uint32_t)b;
        const double u = ((double)(A >> 5) * 67108864.0 + (double)(B >> 6)) / 9007199254740992.0;
        if (2.0 * u - 1.0 != symmetric_uniform(A, B)) ++bad;
        const double y = (b & 1) ? -x : x;
        int fl;
        double next;
        if (floor_next(y, fl, next)) {
            if (fl != (int)std::floor(y) || next != std::floor(y) + 1.0) ++bad;
        } else if (std::fabs(y) < 1073741824.0) {
            ++bad;
        }
        bool ok = true;
        const float f = rough(y, ok);
        if (ok && !(f <= std::fabs(y) && f >= std::fabs(y) * (1.0 - 1e-6))) ++bad;
        const double near = from_words(hi_word(d), (uint32_t)r());
        for (double p : {x, y, d, near, 0.0, -0.0, std::nan(""), (double)INFINITY})
            for (double q : {d, y, 0.0, -1.0, std::nan(""), -(double)INFINITY}) {
                if (less(p, q) != (p < q)) ++bad;
                if (surely_inside(p, q, d) && !(q < p && p < d) && q == q) ++bad;
                if (is_zero(p) != (p == 0.0) || finite_bits(p) != (bool)std::isfinite(p)) ++bad;
            }
    }
    std::printf("%ld %ld\n", used, bad);
    return bad != 0 || used < 1000000;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_exact_forms_match_plain_operations(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC),
                    str(tmp_path / "t.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
