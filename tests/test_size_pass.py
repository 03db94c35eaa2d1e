"""The host bookkeeping of a size-measuring pass (szx_gb300/csrc/size_pass.h):
every field's bounds are asked for once each, whatever other fields ask for,
and the cost of a pass grows with its fields, not with their square: 200,000
fields take a fraction of a second (comparing every pair of them: minutes)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <chrono>
#include <cmath>
#include <cstdio>
#include "size_pass.h"
using namespace szxg;
static int bad = 0;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); bad = 1; } } while (0)
int main() {
    float x = 0;
    {
        SizePass p(3);
        KnownRatios known(3);
        for (int f = 0; f < 3; f++) p.ask(f, &x, 500 + 513 * f, f == 1 ? NAN : 0.5f);   // steps 1, 2, 3
        CHECK(p.items.size() == 3 && p.steps == 6 && p.items[1].step0 == 1 && p.items[2].step0 == 3);
        p.begin_turn();
        p.ask_more(1, &x, 1013, NAN);      // its own first bound again
        p.ask_more(1, &x, 1013, 0.5f);     // another field's
        p.ask_more(1, &x, 1013, 0.25f);
        p.ask_more(1, &x, 1013, 0.5f);     // this turn's again
        CHECK(p.items.size() == 5 && p.owner[3] == 1 && p.owner[4] == 1 && p.items[4].step0 == 8 && p.steps == 10);
        p.begin_turn();
        p.ask_more(2, &x, 1526, 0.25f);    // asked for in another field's turn
        CHECK(p.items.size() == 6 && p.owner[5] == 2 && p.items[5].n == 1526);
        for (size_t k = 0; k < p.items.size(); k++) known.add(p.owner[k], p.items[k].eb, 1.0 + k);
        CHECK(*known.find(0, 0.5f) == 1.0 && *known.find(1, NAN) == 2.0 && *known.find(1, 0.25f) == 5.0);
        CHECK(*known.find(2, 0.25f) == 6.0 && !known.find(0, 0.25f) && !known.find(0, NAN));
        p.clear();
        CHECK(p.items.empty() && p.owner.empty() && p.steps == 0);
    }
    const int nf = 200000;
    const auto t0 = std::chrono::steady_clock::now();
    SizePass p(nf);
    KnownRatios known(nf);
    for (int f = 0; f < nf; f++) p.ask(f, &x, 1000, 1.0f + f);
    for (int f = 0; f < nf; f++) {
        p.begin_turn();
        for (int k = 1; k < 7; k++) p.ask_more(f, &x, 1000, 1.0f + f + 0.125f * k);
    }
    for (size_t k = 0; k < p.items.size(); k++) known.add(p.owner[k], p.items[k].eb, 1.0 + k);
    double sum = 0;
    for (int f = 0; f < nf; f++) sum += *known.find(f, 1.0f + f);
    const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    CHECK(p.items.size() == 7u * nf && p.steps == 14ull * nf && sum > 0);
    std::printf("%.3f s\n", s);
    CHECK(s < 5.0);
    return bad;
}
"""


def test_bookkeeping_of_a_size_pass(tmp_path):
    cxx = shutil.which("g++")
    inc = "/usr/local/cuda/include"
    if not cxx or not os.path.isdir(inc):
        pytest.skip("g++ and the CUDA headers are required")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run([cxx, "-O2", "-std=c++17", "-Wall", "-I", inc, "-I", os.path.join(ROOT, "szx_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
