"""Once-per-device set-up of the launchers (csrc/once.h), compiled for the host: a thread that comes while another one is
still setting up must not go on before that has succeeded, and a set-up that failed is repeated."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "llm-sys-project_b200", "csrc", "once.h")

SOURCE = r"""
#include "%s"
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

static int fail(const char* what) { std::printf("%%s\n", what); return 1; }

int main() {
    // eight threads on two devices: nobody returns 0 before the set-up of that device is through, and it runs once
    B200PerDeviceOnce once;
    std::atomic<int> ready[2] = {{0}, {0}}, calls[2] = {{0}, {0}}, early{0}, errors{0};
    std::vector<std::thread> threads;
    for (int i = 0; i < 8; i++)
        threads.emplace_back([&, i] {
            const int dev = i & 1;
            const int st = once.run(dev, [&]() -> int {
                calls[dev]++;
                std::this_thread::sleep_for(std::chrono::milliseconds(50));
                ready[dev] = 1;
                return 0;
            });
            if (st) errors++;
            if (!ready[dev]) early++;
        });
    for (auto& t : threads) t.join();
    if (early) return fail("a thread went on before the set-up was through");
    if (errors || calls[0] != 1 || calls[1] != 1) return fail("the set-up did not run once per device");

    // an error is reported, not remembered as done
    B200PerDeviceOnce retry;
    int tries = 0;
    auto flaky = [&]() -> int { return ++tries == 1 ? 7 : 0; };
    if (retry.run(3, flaky) != 7) return fail("the error of a set-up was lost");
    if (retry.run(3, flaky) != 0 || tries != 2) return fail("a set-up that failed was not repeated");
    if (retry.run(3, flaky) != 0 || tries != 2) return fail("a set-up that succeeded was repeated");
    // a device beyond the table is set up on every call
    if (retry.run(64, flaky) != 0 || retry.run(64, flaky) != 0 || tries != 4) return fail("device beyond the table");
    return 0;
}
"""


def test_once_per_device_with_threads_and_errors(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(SOURCE % HEADER)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-Wall", "-Werror", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
