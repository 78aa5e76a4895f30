"""CPU test of the automatic sweep configuration's schedule in a scene that
collapses after its first trial: the next trials come soon enough to follow.
Costs in the shape of the measured 2,097,152-particle dam break: the mixed sweeps
lead until substep 50, then the direct ones by more and more."""
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

HARNESS = r"""
#include <cmath>
#include <cstdio>
#include <vector>
#include "auto_policy.h"
using namespace pbf;
static double cost(uint32_t pass, double t) {  // ms per substep
    const double mixed = t < 20 ? 5.0 : 5.0 + 0.62 * (t - 20) * (t - 20);
    if (pass == PBF_PASS_MIXED) return mixed;
    if (pass == PBF_PASS_DIRECT) return t < 20 ? 9.0 : 9.0 + 18.0 * (t - 20);
    return 3.0 * mixed;
}
// Total time of the first 100 substeps; *trials and the substep from which the
// direct sweeps ran.
static double run(int* trials, int* direct_from) {
    AutoPolicy p;
    p.reset(0);
    uint32_t solver = PBF_PASS_MIXED, vort = solver;
    double total = 0;
    *trials = 0;
    *direct_from = -1;
    while (p.count < 100) {
        if (p.trial_due()) {
            const std::vector<uint32_t> c = p.candidates(solver, vort, false, true);
            std::vector<double> s, v;
            for (size_t k = 0; k < c.size(); ++k) {
                s.push_back(cost(c[k], (double)p.count));
                v.push_back(0.3 * s.back());
                total += s.back() + v.back();
                if (k + 1 < c.size()) ++p.count;
            }
            p.finish(c, s.data(), v.data(), true, solver, vort);
            ++p.count;
            ++*trials;
            if (solver == PBF_PASS_DIRECT && *direct_from < 0) *direct_from = (int)p.count;
        } else {
            total += cost(solver, (double)p.count) + 0.3 * cost(vort, (double)p.count);
            ++p.count;
        }
    }
    return total;
}
int main() {
    int trials = 0, from = -1;
    const double t = run(&trials, &from);
    double best = 0;
    for (int k = 0; k < 100; ++k)
        best += 1.3 * std::fmin(cost(PBF_PASS_MIXED, k), cost(PBF_PASS_DIRECT, k));
    std::printf("%.3f of the best, %d trials, direct from %d\n", t / best, trials, from);
    AutoPolicy q;  // a calm scene: half a period, then doubling up to the cap
    q.reset(0);
    uint32_t a = PBF_PASS_MIXED, b = a;
    std::vector<uint32_t> want = {16, 32, 64, 128, 256, 256}, got;
    for (size_t k = 0; k < want.size(); ++k) {
        const std::vector<uint32_t> c = q.candidates(a, b, false, true);
        std::vector<double> s;
        for (uint32_t x : c) s.push_back(x == PBF_PASS_MIXED ? 1.0 : 1.5);
        q.finish(c, s.data(), s.data(), true, a, b);
        got.push_back(q.period);
    }
    return !(t < 1.15 * best && from > 0 && from < 75 && trials <= 5 && got == want);
}
"""


def test_collapse_is_followed(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "collapse.cpp", tmp_path / "collapse"
    src.write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "pbf_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
