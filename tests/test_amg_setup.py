"""The host part of the AMG set-up (csrc/amg_setup.cpp), compiled for the host: its loops over several threads
give what one thread gives, to the bit, and the maps are what they say (Galerkin sums, members by position,
padded entries), against a plain restatement in the program.  Sizes around the grain at which threads start."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "babelsim_b200", "csrc")
PROGRAM = r"""
#include "amg_setup.h"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <random>
using namespace bsg;
static unsigned long long hash_ = 1469598103934665603ull;
static void mix(const void* p, std::size_t n) {
    const unsigned char* c = static_cast<const unsigned char*>(p);
    for (std::size_t i = 0; i < n; ++i) hash_ = (hash_ ^ c[i]) * 1099511628211ull;
}
template <class T> static void mix(const std::vector<T>& v) { mix(v.data(), v.size() * sizeof(T)); }
int main(int, char** argv) {
    const int n = std::atoi(argv[1]);
    std::mt19937 rng(n);
    std::uniform_real_distribution<double> u(0.1, 1.0);
    std::vector<std::vector<std::pair<int, double>>> rows(n);
    for (int i = 0; i < n; ++i)
        for (int d : {1, 17, 211})
            if (i + d < n && u(rng) < 0.8) {
                const double c = -u(rng);
                rows[i].push_back({i + d, c});
                rows[i + d].push_back({i, c});
                if (u(rng) < 0.15) { rows[i].push_back({i + d, c / 2}); rows[i + d].push_back({i, c / 2}); }
            }
    HostCsr a;
    a.n = n;
    a.ptr.push_back(0);
    for (int i = 0; i < n; ++i) {
        double s = 0.01;
        for (auto& e : rows[i]) { a.col.push_back(e.first); a.val.push_back(e.second); s -= e.second; }
        a.ptr.push_back(static_cast<int>(a.col.size()));
        a.diag.push_back(s);
    }
    int n1 = 0, n2 = 0, bad = 0;
    const std::vector<int> p = pairwise(a, n1);
    const HostCsr half = coarsen(a, p, n1, nullptr);
    const std::vector<int> q = pairwise(half, n2);
    std::vector<int> agg(n), target, aptr, arows;
    for (int i = 0; i < n; ++i) agg[i] = q[p[i]];
    const HostCsr c = coarsen(a, agg, n2, &target);
    aggregateLists(agg, n2, aptr, arows);
    const GalerkinMaps g = galerkinMaps(a, target, aptr, arows, static_cast<int>(c.col.size()));
    for (int I = 0; I < n2; ++I) {
        double d = 0.0;
        for (int m = aptr[I]; m < aptr[I + 1]; ++m) d += a.diag[arows[m]];
        for (int k = g.cintra_ptr[I]; k < g.cintra_ptr[I + 1]; ++k) d += a.val[g.cintra_src[k]];
        if (std::fabs(d - c.diag[I]) > 1e-12 * std::fabs(d) + 1e-13) ++bad;
        for (int e = c.ptr[I]; e < c.ptr[I + 1]; ++e) {
            double v = 0.0;
            for (int k = g.cslot_ptr[e]; k < g.cslot_ptr[e + 1]; ++k) v += a.val[g.cslot_src[k]];
            if (v != c.val[e]) ++bad;
        }
    }
    const Members members = membersOf(agg, n2);
    std::vector<int> order(n2);
    std::iota(order.begin(), order.end(), 0);
    std::shuffle(order.begin(), order.end(), rng);
    const std::vector<int> coarse = order;
    const TreeMaps t = treeMaps(n, members, order);
    std::vector<int> seen(n, 0);
    double padded = 0.0;
    for (std::size_t s = 0; s < t.row.size(); s += 32) {
        int w = 0;
        for (std::size_t k = s; k < std::min(t.row.size(), s + 32); ++k) {
            const int i = t.row[k];
            if (i < 0) continue;
            ++seen[i];
            w = std::max(w, a.ptr[i + 1] - a.ptr[i]);
            if (agg[i] != coarse[k / 4] || t.at[i] != static_cast<int>(k) || t.pos[t.rank[k]] != static_cast<int>(k)) ++bad;
        }
        padded += 32.0 * w;
    }
    for (int s : seen) bad += s != 1;
    if (padded != paddedEntries(t, a.ptr)) ++bad;
    Members fine(n);
    for (int i = 0; i < n; ++i) fine[i] = {4 * i, 4 * i + 1, -1, -1};
    std::vector<int> by(4 * t.row.size(), -7);
    membersByPosition(t, fine, by.data());
    for (std::size_t k = 0; k < t.row.size(); ++k)
        for (int j = 0; j < 4; ++j) bad += by[4 * k + j] != (t.row[k] < 0 ? -7 : fine[t.row[k]][j]);
    mix(c.ptr); mix(c.col); mix(c.val); mix(c.diag); mix(target); mix(g.cslot_ptr); mix(g.cslot_src);
    mix(g.cintra_ptr); mix(g.cintra_src); mix(by);
    std::printf("%d %d %llx\n", hostThreads(), bad, hash_);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("amg_setup")
    (d / "t.cpp").write_text("#include <algorithm>\n" + PROGRAM)
    exes = []
    for threads in (1, 8):  # the number of threads is the machine's: let the program see one, or eight
        exe = str(d / f"t{threads}")
        stub = d / f"threads{threads}.h"
        stub.write_text("#pragma once\n#include <thread>\n#define hardware_concurrency() hardware_concurrency() * 0 + "
                        f"{threads}\n")
        subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I" + CSRC, "-include", str(stub), str(d / "t.cpp"),
                        os.path.join(CSRC, "amg_setup.cpp"), "-o", exe], check=True)
        exes.append(exe)
    return exes


@pytest.mark.parametrize("n", [1, 2, 37, 1000, 16384, 16385, 40001, 140000])
def test_threads_and_maps(program, n):
    one, eight = (subprocess.run([exe, str(n)], check=True, capture_output=True, text=True).stdout.split()
                  for exe in program)
    assert (one[0], eight[0]) == ("1", "8")
    assert one[1] == eight[1] == "0"
    assert one[2] == eight[2]
