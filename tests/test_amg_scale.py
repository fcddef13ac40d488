"""Choice of the AMG correction scale (csrc/amg_scale.h), compiled for the host: a trial that breaks down is the
worst one, not a good one; a good start ends the trials; where nothing is better the start stays."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "babelsim_b200", "csrc")
PROGRAM = r"""
#include "amg_scale.h"
#include <cstdio>
#include <cstdlib>
int main(int, char** argv) {
    int trials = 0;
    const double chosen = bsg::chooseCorrection(1.8, [&](double scale, double) {
        ++trials;
        const double r = std::atof(argv[scale == 1.8 ? 1 : scale == 1.2 ? 2 : 3]);
        return r < 0.0 ? bsg::kTrialFailed : r;
    });
    std::printf("%g %d\n", chosen, trials);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("amg_scale")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, str(d / "t.cpp"), "-o", str(d / "t")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("reductions,chosen,trials", [
    ((1e-6, 0.5, 0.5), "1.8", "1"),     # good enough: nothing else is tried
    ((3e-5, 1e-9, 1e-9), "1.8", "1"),
    ((1e-2, 1e-4, 1e-3), "1.2", "3"),
    ((1e-2, 1e-3, 1e-4), "1.5", "3"),
    ((1e-2, 1e-2, 2e-2), "1.8", "3"),   # no better
    ((-1, 1e-3, 1e-2), "1.2", "3"),     # the start breaks down
    ((-1, -1, 0.9), "1.5", "3"),
    ((-1, -1, -1), "1.8", "3"),
    ((1e-2, -1, -1), "1.8", "3"),
])
def test_choice(program, reductions, chosen, trials):
    out = subprocess.run([program] + [str(r) for r in reductions], check=True, capture_output=True, text=True).stdout
    assert out.split() == [chosen, trials]
