"""Dynamic shared-memory limits are raised per device and kernel (a second GPU in the
process needs its own), never lowered, and not remembered when the call failed."""
import glob
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "arec3d_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "arec_limits.h"
int main() {
    arecgb::RaisedLimits L;
    int k0 = 0, k1 = 0, calls = 0;
    size_t last = 0;
    auto ok = [&](size_t n) { calls++; last = n; return 0; };
    auto bad = [&](size_t) { calls++; return 7; };
#define CHECK(c) if (!(c)) { std::printf("line %d\n", __LINE__); return 1; }
    CHECK(L.raise(0, &k0, 100, ok) == 0 && calls == 1 && last == 100);
    CHECK(L.raise(0, &k0, 80, ok) == 0 && calls == 1);          // never lowered
    CHECK(L.raise(1, &k0, 100, ok) == 0 && calls == 2);         // the other device
    CHECK(L.raise(0, &k1, 100, ok) == 0 && calls == 3);         // the other kernel
    CHECK(L.raise(0, &k0, 200, bad) == 7 && calls == 4);
    CHECK(L.raise(0, &k0, 200, ok) == 0 && calls == 5);         // a failure is tried again
    CHECK(L.raise(1, &k0, 200, ok) == 0 && calls == 6 && last == 200);
    std::vector<std::thread> t;
    for (int i = 0; i < 8; i++)
        t.emplace_back([&, i] { for (size_t n = 1; n < 2000; n++) L.raise(2, &k0, (n * 7 + i) % 1999, ok); });
    for (auto &x : t) x.join();
    CHECK(last == 1998);                                        // raised in order
    std::puts("ok");
}
"""


def test_limits_per_device_and_kernel(tmp_path):
    src, exe = tmp_path / "limits.cpp", tmp_path / "limits"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout.strip() == "ok"


def test_every_kernel_raises_its_limit_there():
    hits = {}
    for f in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(f) as fh:
            n = len(re.findall(r"cudaFuncSetAttribute\(", fh.read()))
        if n:
            hits[os.path.basename(f)] = n
    assert hits == {"arec_project.cu": 1}, hits
