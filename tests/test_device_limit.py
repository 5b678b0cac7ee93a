"""A kernel's raised limit of shared memory is kept per device: the class that keeps account of it, against a driver of the test's own."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pulsar_b200", "csrc")

PROGRAM = r"""
#include "device_limit.h"
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

// The test's driver: one limit per device, raising refused beyond 1000 bytes, the current device a thread's own.
static std::atomic<size_t> limit_of[80];
static std::atomic<int> calls;
static thread_local int current = 0;
static int device(int* d) { if (current < 0) return 100; *d = current; return 0; }
static int raise_to(size_t n) { ++calls; if (n > 1000) return 1; limit_of[current] = n; return 0; }
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::exit(1); } } while (0)

int main() {
    static pb::DeviceLimit a, b;
    // a device at a time: the second one is raised too, each only once
    for (int round = 0; round < 3; ++round)
        for (current = 0; current < 2; ++current) {
            CHECK(a.allow(300, device, raise_to) == 0);
            CHECK(limit_of[current] == 300);
        }
    CHECK(calls == 2);
    // another kernel has limits of its own; a larger request raises, a smaller one does not lower
    current = 1;
    CHECK(b.allow(10, device, raise_to) == 0 && calls == 3);
    CHECK(a.allow(500, device, raise_to) == 0 && calls == 4 && limit_of[1] == 500);
    CHECK(a.allow(200, device, raise_to) == 0 && calls == 4 && limit_of[1] == 500 && limit_of[0] == 300);
    // a refusal is returned and not remembered as done, and so is the failure to name the device
    CHECK(a.allow(2000, device, raise_to) == 1);
    CHECK(a.allow(2000, device, raise_to) == 1 && calls == 6);
    CHECK(a.allow(400, device, raise_to) == 0 && calls == 6);
    current = -1;
    CHECK(a.allow(400, device, raise_to) == 100);
    // devices beyond those that are kept account of are raised on every call
    current = 70;
    CHECK(a.allow(400, device, raise_to) == 0 && a.allow(400, device, raise_to) == 0 && limit_of[70] == 400 && calls == 8);
    // many threads, growing and shrinking requests: what a call was granted holds when it returns
    static pb::DeviceLimit c;
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([t] {
            current = 2 + t % 2;
            unsigned x = 12345u + t;
            for (int i = 0; i < 20000; ++i) {
                x = x * 1664525u + 1013904223u;
                const size_t n = 1 + (x >> 8) % (i / 20 % 1000 + 1);
                if (c.allow(n, device, raise_to) != 0 || limit_of[current] < n) { std::printf("lowered\n"); std::exit(2); }
            }
        });
    for (auto& t : threads) t.join();
    return 0;
}
"""


def test_limits_are_kept_per_device(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++")) or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "limits.cpp"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O2", "-pthread", "-I", CSRC, str(src), "-o", str(tmp_path / "limits")], check=True)
    done = subprocess.run([str(tmp_path / "limits")], stdout=subprocess.PIPE, text=True, timeout=120)
    assert done.returncode == 0, done.stdout


COUNTS = r"""
#include "device_limit.h"
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
static thread_local int current = 0;
static std::atomic<int> asked;
static int ask(int* n) { ++asked; *n = 10 * (current + 1); return 0; }
static int fail(int* n) { ++asked; *n = 5; return 2; }
static int none(int* n) { ++asked; *n = 0; return 0; }
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::exit(1); } } while (0)

int main() {
    static pb::DeviceCount a, b;
    // a failure and an answer of none are not remembered; each device has its own number, asked for once
    CHECK(a.get(0, fail) == 0 && a.get(0, none) == 0 && asked == 2);
    for (int round = 0; round < 3; ++round)
        for (current = 0; current < 3; ++current) CHECK(a.get(current, ask) == 10 * (current + 1));
    CHECK(asked == 5);
    CHECK(a.get(1, fail) == 20 && b.get(1, fail) == 0);
    current = 70;                                       // beyond the devices that are kept account of
    CHECK(a.get(70, ask) == 710 && a.get(70, ask) == 710 && asked == 8);
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([t] { current = 10 + t % 4; for (int i = 0; i < 10000; ++i) CHECK(b.get(current, ask) == 10 * (current + 1)); });
    for (auto& t : threads) t.join();
    return 0;
}
"""


def test_counts_are_kept_per_device(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++")) or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "counts.cpp"
    src.write_text(COUNTS)
    subprocess.run([cxx, "-std=c++17", "-O2", "-pthread", "-I", CSRC, str(src), "-o", str(tmp_path / "counts")], check=True)
    done = subprocess.run([str(tmp_path / "counts")], stdout=subprocess.PIPE, text=True, timeout=120)
    assert done.returncode == 0, done.stdout


def test_nothing_is_asked_of_a_device_once_for_the_whole_process():
    """How many clusters a device holds belongs to the device: no launcher keeps the answer in a static of its own."""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                text = f.read()
            for at in re.finditer(r"cudaOccupancyMaxActiveClusters\(", text):
                before = text[max(0, at.start() - 600):at.start()]
                before = before[before.rfind("\n}") + 1:]
                assert "static std::atomic" not in before and "DeviceCount" in before, name


def test_no_launch_remembers_a_raised_limit_for_the_whole_process():
    """Every launch with more shared memory than any kernel may have raises the limit through ``SmemLimit``, or on every call."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        for at in re.finditer(r"cudaFuncSetAttribute\(", text):
            before = text[max(0, at.start() - 400):at.start()]
            before = before[before.rfind("\n}") + 1:]
            assert "static " not in before or name == "common.cuh", f"{name}: {before[-200:]}"
