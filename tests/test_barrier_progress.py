"""The record of how far each CTA of a persistent launch got (takeProgress of csrc/bsg_internal.h), compiled for the
host: launches that follow one another before the host reads a report keep apart, inside the record."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "babelsim_b200", "csrc")
CUDA = "/usr/local/cuda/include"
PROGRAM = r"""
#include "bsg_internal.h"
#include <cstdio>
int main() {
    int next = 0, bad = 0;
    std::vector<std::pair<int, int>> kept;
    for (int k = 0; k < 500; ++k) {
        const int ctas = k % 7 == 0 ? 148 : 1 + (37 * k) % 444;
        const int at = bsg::takeProgress(next, ctas);
        if (at < 0 || at + ctas > bsg::kMaxPersistentCtas) ++bad;
        for (std::size_t j = kept.size() > 8 ? kept.size() - 8 : 0; j < kept.size(); ++j)
            if (at < kept[j].second && kept[j].first < at + ctas) ++bad;
        kept.push_back({at, at + ctas});
    }
    const int whole = bsg::takeProgress(next, bsg::kMaxPersistentCtas);
    std::printf("%d %d\n", bad, whole);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="needs g++ and the CUDA headers")
def test_launches_keep_apart(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "t")
    link = ["-L/usr/local/cuda/lib64", "-lcudart"]
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + CUDA, str(src), "-o", exe] + link, check=True)
    env = dict(os.environ, LD_LIBRARY_PATH="/usr/local/cuda/lib64:" + os.environ.get("LD_LIBRARY_PATH", ""))
    assert subprocess.run([exe], check=True, capture_output=True, text=True, env=env).stdout.split() == ["0", "0"]
