"""The autotuner's choice of a level tile (csrc/ga_tune.h), compiled for the
host with given times: the current tile stays unless another is clearly
faster, whatever the order of the candidates."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "model_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "ga_tune.h"
// argv: keep, its time, smallest tile, largest that fits, then the times of 1, 2, 4, ...
int main(int argc, char **argv)
{
    const int keep = std::atoi(argv[1]), lo = std::atoi(argv[3]), fit = std::atoi(argv[4]);
    float best = (float)std::atof(argv[2]);
    const int kt = ga::faster_tile(keep, lo, 64, best, [&](int k) { return k <= fit; }, [&](int k) {
        int n = 0;
        while ((1 << n) < k) n++;
        return (float)std::atof(argv[5 + n]);
    });
    std::printf("%d %.3f\n", kt, best);
}
"""


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("tune")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I" + CSRC, str(src), "-o", str(exe)], check=True)

    def run(keep, t_keep, lo, fit, times):
        out = subprocess.run([str(exe), str(keep), str(t_keep), str(lo), str(fit)] + [str(t) for t in times], check=True,
                             capture_output=True, text=True).stdout.split()
        return int(out[0]), float(out[1])
    return run


@pytest.mark.parametrize("keep,t_keep,lo,fit,times,want", [
    (8, 1.00, 1, 64, [1.50, 1.20, 1.10, 9.0, 1.05, 1.2, 1.4], 8),   # the best tile is the current one
    (8, 1.00, 1, 64, [0.998, 1.01, 0.997, 9.0, 1.00, 1.0, 1.0], 8),  # nothing clearly faster
    (8, 1.00, 1, 64, [0.97, 0.90, 1.10, 9.0, 1.05, 1.2, 1.4], 2),   # two faster ones: the fastest
    (4, 1.00, 1, 8, [1.20, 1.10, 9.0, 0.90, 0.1, 0.1, 0.1], 8),     # tiles that do not fit are not timed
    (1, 1.00, 1, 1, [9.0], 1),
    (8, 1.00, 2, 64, [0.10, 0.90, 1.10, 9.0, 1.05, 1.2, 1.4], 2),  # 1 is below the smallest
    (0, 1.00, 1, 64, [1.10, 1.05, 0.997, 1.2, 1.3, 1.4, 1.5], 0),   # nothing beats the fused kernel
    (0, 1.00, 1, 64, [1.10, 0.80, 0.70, 0.698, 1.3, 1.4, 1.5], 4),
])
def test_choice(choose, keep, t_keep, lo, fit, times, want):
    kt, best = choose(keep, t_keep, lo, fit, times)
    assert kt == want
    t = t_keep if kt == keep else times[kt.bit_length() - 1]
    assert best == pytest.approx(t)
