"""What neighbours hold of a row's residual between CG iterations (sweptResidual and sweptUpdate of
csrc/pcg_tree.cuh), compiled for the host: with FP64 Krylov vectors and an FP32 V-cycle the updated sweep is
omega / diagonal * (r - alpha q) rounded to FP32 once, however far the residual falls in one iteration.

Bound: the product and the difference each round in FP64, which is 2^-53 of the old values, so 1e-9 times the
new one where it is 1e7 times smaller; the FP32 rounding adds 2^-24.  1.01 * 2^-24 relative."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "babelsim_b200", "csrc")
CUDA = "/usr/local/cuda/include"
PROGRAM = r"""
#include "pcg_tree.cuh"
#include <cmath>
#include <cstdio>
#include <random>
int main() {
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> u(0.5, 2.0);
    double worst[2] = {0.0, 0.0};
    for (int k = 0; k < 100000; ++k) {
        const float rd = static_cast<float>(u(rng));
        const double r = u(rng), q = u(rng), left = std::pow(10.0, -7.0 * (k % 1000) / 1000.0), alpha = r * (1.0 - left) / q;
        const long double exact = static_cast<long double>(rd) * (static_cast<long double>(r) - static_cast<long double>(alpha) * q);
        const float mixed = bsg::sweptUpdate<float>(bsg::sweptResidual(rd, r), alpha, static_cast<double>(rd) * q);
        worst[0] = std::fmax(worst[0], std::fabs(static_cast<double>((mixed - exact) / exact)));
        const double rd64 = u(rng), w = bsg::sweptUpdate<double>(bsg::sweptResidual(rd64, r), alpha, rd64 * q);
        const long double e64 = static_cast<long double>(rd64) * (static_cast<long double>(r) - static_cast<long double>(alpha) * q);
        worst[1] = std::fmax(worst[1], std::fabs(static_cast<double>((w - e64) / (rd64 * r))));
    }
    std::printf("%.17g %.17g\n", worst[0], worst[1]);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="needs g++ and the CUDA headers")
def test_updated_sweep_is_rounded_once(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + CUDA, str(src), "-o", exe], check=True)
    mixed, double = (float(v) for v in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert mixed <= 1.01 * 2.0 ** -24
    assert double <= 4 * 2.0 ** -53  # of the old value: the product, the difference and alpha q
