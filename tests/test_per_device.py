"""Host values kept per device ordinal (csrc/per_device.h): one device's answer
is not another's, failures are tried again, threads may ask at once.  The step
launcher keeps its kernels' attributes, their resident blocks and the SM count
this way; no other static of it holds an answer of a device."""
from __future__ import annotations

import re
import subprocess

from conftest import ROOT

CSRC = ROOT / "lbm_bench_gpu_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"

int main()
{
    static lbm::PerDevice<int> p;
    int calls = 0, v = -1;
    auto find = [&](int value) { return [&calls, value](int &out) { calls++; out = value; return true; }; };
    // two devices, two answers, each found once
    if (!p.get(0, v, find(152)) || v != 152) return 1;
    if (!p.get(1, v, find(148)) || v != 148) return 2;
    if (!p.get(0, v, find(-5)) || v != 152 || !p.get(1, v, find(-5)) || v != 148 || calls != 2) return 3;
    // a failure is not kept
    if (p.get(2, v, [](int &) { return false; })) return 4;
    if (!p.get(2, v, find(7)) || v != 7) return 5;
    // ordinals outside the table are found every time
    if (!p.get(lbm::kMaxDevices, v, find(1)) || v != 1 || !p.get(lbm::kMaxDevices, v, find(2)) || v != 2) return 6;
    if (!p.get(-1, v, find(3)) || v != 3) return 7;
    std::vector<std::thread> ts;
    std::atomic<int> wrong{0};
    for (int t = 0; t < 8; t++)
        ts.emplace_back([&wrong] {
            for (int d = 3; d < lbm::kMaxDevices; d++) {
                int x = 0;
                if (!p.get(d, x, [d](int &out) { out = 10 * d; return true; }) || x != 10 * d) wrong++;
            }
        });
    for (auto &t : ts) t.join();
    return wrong ? 8 : 0;
}
"""


def test_answers_belong_to_a_device(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0


def test_step_launcher_keeps_no_process_wide_answer():
    text = (CSRC / "zsc_step.cu").read_text()
    host = text[text.index("cudaError_t configure("):]
    kept = re.findall(r"^\s*static (?!_)([^;{=]*)", host, re.M)
    allowed = ("PerDevice<int>", "const EncodeTiled fn", "thread_local")   # per device; a host entry point; keyed below
    assert all(k.startswith(allowed) for k in kept), kept
    assert "last[3] == device" in host
