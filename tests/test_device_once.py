"""Kernel set-up per device (device_once.h): a second device of the process gets
its own, a device gets one, several threads are safe.  Host code, compiled and
run here."""

import os
import re
import shutil
import subprocess

import pytest
from conftest import ROOT

CSRC = os.path.join(ROOT, "surfacelets.jl_b200", "csrc")

PROGRAM = r"""
#include <thread>
#include <vector>
#include "device_once.h"
int main() {
    static sfl::DeviceOnce once;
    int runs[66] = {};
    for (int pass = 0; pass < 3; ++pass)
        for (int d : {0, 1, 7, 63}) once.run(d, [&] { ++runs[d]; });
    for (int d : {0, 1, 7, 63})
        if (runs[d] != 1) return 1;
    for (int pass = 0; pass < 3; ++pass) once.run(64, [&] { ++runs[64]; });   // no slot: set up every time
    if (runs[64] != 3) return 2;
    try {
        once.run(2, [] { throw 1; });
        return 3;
    } catch (int) {
    }
    once.run(2, [&] { ++runs[2]; });   // a set-up that failed is run again
    if (runs[2] != 1) return 4;
    static sfl::DeviceOnce shared;
    std::atomic<int> ready{0}, early{0};
    std::vector<std::thread> ts;
    for (int t = 0; t < 8; ++t)
        ts.emplace_back([&] {
            shared.run(3, [&] { ready = 1; });
            if (!ready) ++early;
        });
    for (auto& t : ts) t.join();
    return early == 0 ? 0 : 5;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_set_up_once_a_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_kernel_attributes_are_set_per_device():
    """No launcher keeps its set-up in a flag of the process."""
    for name in os.listdir(CSRC):
        text = open(os.path.join(CSRC, name), encoding="utf-8").read()
        assert not re.search(r"static (bool|size_t) configured", text), name
