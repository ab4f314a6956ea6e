"""Tables that every device of the process needs its own copy of are set up once per device."""
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "lighttransportsimulation_gb300", "csrc")

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "once_per_device.hpp"
int main() {
    lts::OncePerDevice once;
    std::atomic<int> runs[3] = {{0}, {0}, {0}}, seen_unset{0};
    std::atomic<bool> set[3] = {{false}, {false}, {false}};
    std::vector<std::thread> ts;
    for (int t = 0; t < 12; ++t)
        ts.emplace_back([&, t] {
            const int d = t % 3;
            const std::string e = once.run(d, [&]() -> std::string {
                ++runs[d];
                std::this_thread::sleep_for(std::chrono::milliseconds(5));
                set[d] = true;
                return "";
            });
            if (!e.empty() || !set[d]) ++seen_unset;
        });
    for (auto& t : ts) t.join();
    int fails = 0;
    const std::string a = once.run(7, [&]() -> std::string { ++fails; return "no"; });  // a failure is tried again
    const std::string b = once.run(7, [&]() -> std::string { ++fails; return ""; });
    const std::string c = once.run(7, [&]() -> std::string { ++fails; return ""; });
    std::printf("%d %d %d %d %d %d %d %d\n", (int)runs[0], (int)runs[1], (int)runs[2], (int)seen_unset, fails, a == "no",
                b.empty(), c.empty());
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.split()
    assert [int(x) for x in out] == [1, 1, 1, 0, 2, 1, 1, 1]


def test_no_flag_for_the_whole_process_guards_device_tables():
    for f in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, f)).read()
        assert not re.search(r"static bool \w+ = false;(?s:.){0,400}cudaMemcpyToSymbol", text), f
