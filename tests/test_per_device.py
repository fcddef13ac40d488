"""Launch set-up per device (csrc/per_device.h), compiled for the host: threads that arrive together on several
devices run it once per device and all see its result, and a failed attempt is tried again."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "babelsim_b200", "csrc")
PROGRAM = r"""
#include "per_device.h"
#include <atomic>
#include <chrono>
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>
int main() {
    bsg::PerDevice set;
    std::atomic<int> ran[3] = {}, wrong{0}, ready{0};
    std::vector<std::thread> pool;
    for (int t = 0; t < 12; ++t)
        pool.emplace_back([&, t] {
            const int device = t % 3;
            ++ready;
            while (ready < 12) {}
            const int v = set.get(device, [&] {
                ++ran[device];
                std::this_thread::sleep_for(std::chrono::milliseconds(5));
                return 16 + device;
            });
            if (v != 16 + device) ++wrong;
        });
    for (auto& t : pool) t.join();
    bsg::PerDevice fails;
    int attempts = 0;
    try { fails.get(0, [&]() -> int { ++attempts; throw std::runtime_error("no"); }); } catch (const std::runtime_error&) {}
    const int second = fails.get(0, [&] { ++attempts; return 8; });
    std::printf("%d %d %d %d %d %d\n", ran[0].load(), ran[1].load(), ran[2].load(), wrong.load(), attempts, second);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_runs_once_per_device(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + CSRC, str(src), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["1", "1", "1", "0", "2", "8"]


def test_every_launch_attribute_is_kept_per_device():
    """A function attribute or cluster size kept in a plain static is the first device's alone."""
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        for word in ("cudaFuncSetAttribute(", "cudaOccupancyMaxActiveClusters("):
            at = text.find(word)
            while at >= 0:
                assert ".get(currentDevice()" in text[max(0, at - 1200):at], (name, text[at:at + 80])
                at = text.find(word, at + 1)
