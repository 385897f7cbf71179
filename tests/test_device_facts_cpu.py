"""What launches remember about a device between calls (the clusters that fit, the number of SMs) is shared by threads
and belongs to one device: no function keeps such a number in a plain static, and the class that keeps them
is free of races (run under the thread sanitizer) and of mix-ups between devices."""

import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bobcat_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "device_facts.h"
int main() {
    static bc::k::DeviceFacts<3> facts;
    std::atomic<int> wrong{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&] {
            for (int round = 0; round < 1000; ++round)
                for (int device : {0, 1, 63, 64, 1000})
                    for (int i = 0; i < 3; ++i) {
                        int got = 0;
                        if (!facts.get(device, i, [&](int* n) { *n = 1 + device * 3 + i; return true; }, &got) || got != 1 + device * 3 + i) ++wrong;
                    }
        });
    for (std::thread& t : threads) t.join();
    int got = 0;
    static bc::k::DeviceFacts<1> failing;
    if (failing.get(0, 0, [](int*) { return false; }, &got)) ++wrong;
    if (!failing.get(0, 0, [](int* n) { *n = 7; return true; }, &got) || got != 7) ++wrong;
    std::printf("%d wrong\n", wrong.load());
    return wrong.load() != 0;
}
"""


def test_no_function_keeps_a_plain_number():
    found = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cpp", ".h", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                found += ["%s: %s" % (name, line.strip()) for line in f if re.match(r"\s+static (?:unsigned |u?int\w* |size_t |bool |float |double )+\w+(?:\[[^]]*\])* *=", line)]
    assert not found, found


def test_device_facts_under_the_thread_sanitizer(tmp_path):
    source, binary = tmp_path / "facts.cpp", tmp_path / "facts"
    source.write_text(PROGRAM)
    built = subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=thread", "-I", CSRC, "-o", str(binary), str(source), "-lpthread"], capture_output=True, text=True)
    if built.returncode != 0 and "tsan" in built.stderr:
        pytest.skip("g++ has no thread sanitizer here")
    assert built.returncode == 0, built.stderr
    # The sanitizer wants a plain address-space layout.
    ran = subprocess.run((["setarch", "-R"] if shutil.which("setarch") else []) + [str(binary)], capture_output=True, text=True)
    assert ran.returncode == 0 and "0 wrong" in ran.stdout, ran.stdout + ran.stderr
