"""The 3D autotuner's table (pfast_gb300/csrc/tune_policy.h: TuneTable), compiled with g++: a time is used
for the cluster sizes it was measured with only, and one measured alone comes first for an evaluation
that runs alone."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

CHECK = r"""
#include <cstdio>
#include "tune_policy.h"
using namespace pfast;
static int n = 0;
static void eq(int got, int want) { ++n; std::printf("%s %d: %d %d\n", got == want ? "ok" : "FAIL", n, got, want); }
static void fill(TuneTable& t, const TuneTable::Phase& p, bool alone, const int cl[2], const double (&ms)[6]) {
    for (int c = 0; c < 6; ++c) t.record(p, alone, c, cl, ms[c]);
}
int main() {
    const TuneTable::Phase p = {0, 2, 64, 128, 128, 9}, q = {0, 2, 64, 128, 128, 10};
    const int one[2] = {1, 1}, many[2] = {16, 16}, mixed[2] = {16, 8};
    TuneTable t;
    eq(t.pick(p, true, 0x3f, many, 152), -1);
    fill(t, p, true, many, {60, 65, 20, 25, 30, 35});
    eq(t.pick(p, true, 0x3f, many, 152), 2);
    eq(t.pick(p, false, 0x3f, many, 152), 2);     // beside others, with the same clusters
    eq(t.pick(p, false, 0x3f, one, 152), -1);     // beside others, one block per source: not measured
    eq(t.pick(p, true, 0x3f, mixed, 152), -1);
    eq(t.pick(p, false, 0x03, one, 152), 0);      // per diagonal does not depend on the clusters
    eq(t.pick(p, false, 0x0c, one, 152), -1);
    eq(t.pick(q, true, 0x3f, many, 152), -1);
    fill(t, p, false, one, {90, 80, 200, 210, 220, 230});
    eq(t.pick(p, false, 0x3f, one, 152), 1);
    eq(t.pick(p, true, 0x3f, one, 152), 1);       // measured beside others only
    eq(t.pick(p, true, 0x3f, many, 152), 2);
    t.record(p, true, 2, many, 180);              // means: 100
    eq(t.pick(p, true, 0x3f, many, 152), 3);
    t.record(p, true, 3, many, 0.0);              // no time
    eq(t.pick(p, true, 0x3f, many, 152), 3);
}
"""


def test_times_belong_to_their_cluster_sizes(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "check.cpp", str(tmp_path / "check")
    src.write_text(CHECK)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "pfast_gb300", "csrc"), str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout
    assert "FAIL" not in out and out.count("ok ") == 13, out
