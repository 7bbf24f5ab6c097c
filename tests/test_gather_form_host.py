"""csrc/gather_form.h compiled as host C++: which form of gather a launch of the
split-precision mover takes, at the points where both were measured (the faster
one is expected where they differ by more than 5 %), and that no load leaves the
rule without an answer."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "stochastic-parker_gb300" / "csrc"

# ndim, two frames, grid (nodes a side), particles a cell, step, groups expected; the
# launch makes 128 pushes
POINTS = [
    (2, 0, 64, 8.0, 0.03, 0), (2, 0, 64, 2.0, 0.3, 0), (2, 0, 256, 2.0, 0.01, 0),
    (2, 0, 256, 0.5, 0.3, 0), (2, 0, 256, 0.1, 0.5, 0), (2, 0, 64, 2.0, 0.5, 0), (2, 0, 512, 2.0, 0.5, 1),
    (2, 0, 64, 2.0, 3.0, 1), (2, 1, 64, 0.4, 3.0, 0), (2, 1, 1024, 0.006, 2.9, 1),
    (2, 0, 512, 2.0, 0.1, 0), (2, 0, 1024, 2.0, 0.03, 0), (2, 0, 1024, 0.5, 0.3, 1),
    (2, 0, 1024, 2.0, 0.5, 1), (2, 0, 1024, 0.5, 0.5, 1), (2, 0, 2048, 0.1, 0.003, 1),
    (2, 0, 2048, 0.5, 0.5, 1),
    (2, 1, 64, 8.0, 0.03, 0), (2, 1, 256, 8.0, 0.003, 0), (2, 1, 256, 8.0, 0.3, 1),
    (2, 1, 64, 2.0, 0.5, 0), (2, 0, 2048, 0.002, 0.5, 0), (2, 1, 2048, 0.002, 0.003, 0),
    (2, 1, 64, 8.0, 0.5, 1), (2, 1, 1024, 0.5, 0.003, 1), (2, 1, 2048, 0.5, 0.5, 1),
    (3, 0, 32, 8.0, 0.003, 0), (3, 0, 64, 2.0, 0.03, 0), (3, 0, 64, 0.5, 0.1, 0),
    (3, 0, 128, 0.5, 0.03, 0), (3, 0, 32, 8.0, 0.1, 1), (3, 0, 64, 2.0, 0.5, 1),
    (3, 0, 128, 0.5, 0.3, 1), (3, 0, 128, 0.1, 0.003, 1),
    (3, 1, 32, 32.0, 0.003, 0), (3, 1, 64, 2.0, 0.03, 0), (3, 1, 64, 8.0, 0.03, 1),
    (3, 1, 32, 2.0, 0.1, 1), (3, 1, 64, 0.5, 0.3, 1), (3, 1, 64, 0.1, 0.003, 1),
    (3, 1, 128, 0.5, 0.3, 1),
]

PROGRAM = r"""
#include <cstdio>
#include <limits>
#include "gather_form.h"
using namespace gpat;
int main() {
    int ndim, two;
    double side, ppc, step;
    while (std::scanf("%d %d %lf %lf %lf", &ndim, &two, &side, &ppc, &step) == 5) {
        const double cells = std::pow(side + 4, ndim);
        const int64_t n = (int64_t)(ppc * std::pow(side, ndim));
        std::printf("%d\n", (int)gathers_in_groups({ndim, two != 0, n, cells, n / cells, step, 152, 128.0}));
    }
    const double nan = std::numeric_limits<double>::quiet_NaN(), d = 1.0 / 128;
    // sqrt(2) / d; no diffusion: no step; the smallest side, twice at p0
    std::printf("%.3f %.3f %.3f\n", gather_step(2, 1.0, false, 1.0, d, d, 1.0),
                gather_step(3, 0.0, true, 1.0, d, d, d),
                gather_step(3, d * d / 8, true, 0.01, d, 2 * d, d / 2));
    std::printf("%d\n", (int)gathers_in_groups({3, false, 1, 8.0, 0.125, nan, 152, nan}));
    // launches of few pushes, right after a binning: by single lanes, unless each
    // particle has a group of its own
    std::printf("%d %d %d\n", (int)gathers_in_groups({2, true, 2000000, 4e6, 0.5, 0.5, 152, 16.0}),
                (int)gathers_in_groups({3, true, 1000000, 2e6, 0.5, 0.5, 152, 10.0}),
                (int)gathers_in_groups({3, true, 30000, 2e6, 0.015, 0.5, 152, 10.0}));
    std::printf("%d %d %d %d\n", long_steps(0.1), long_steps(0.3), long_steps(0.2), long_steps(0.0));
    return 0;
}
"""


def test_forms_at_the_measured_points(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    src = tmp_path / "form.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "form"
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    text = "\n".join(" ".join(str(v) for v in p[:5]) for p in POINTS)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True,
                         check=True).stdout.split("\n")
    got = [int(v) for v in out[:len(POINTS)]]
    assert got == [p[5] for p in POINTS], [p for p, g in zip(POINTS, got) if g != p[5]]
    # 0.2 = 2 sqrt(2 (d^2 / 8) 0.01) / (d / 2)
    assert out[len(POINTS)] == "181.019 0.000 0.200"
    assert out[len(POINTS) + 1] in ("0", "1")
    assert out[len(POINTS) + 2] == "0 0 1"
    assert out[len(POINTS) + 3] == "0 1 1 0"
