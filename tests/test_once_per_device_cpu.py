"""Kernel attributes are set before any thread launches: gk::once_per_device returns
to no caller before its setting has been made, on each of two devices (a stub of
cudaGetDevice), and makes it once for calls that follow one another."""
import os
import subprocess

from gaukuk_b200 import _build

SOURCE = r"""
#include "gk_internal.h"
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
thread_local int device = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
static std::atomic<unsigned long long> mask{0};
static std::atomic<int> set[2], calls[2], early{0};
static void user(int dev) {
    device = dev;
    gk::once_per_device(mask, [&] {
        std::this_thread::sleep_for(std::chrono::milliseconds(100));
        set[dev] = 1;
        ++calls[dev];
    });
    if (!set[dev]) ++early;
}
int main() {
    std::vector<std::thread> t;
    for (int i = 0; i < 16; ++i) t.emplace_back(user, i & 1);
    for (auto& x : t) x.join();
    const int after = calls[0] + calls[1];
    user(0);
    user(1);
    std::printf("%d %d\n", early.load(), calls[0] + calls[1] - after);
}
"""


def test_no_thread_is_ahead_of_the_setting(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(SOURCE)
    cuda = os.path.dirname(os.path.dirname(_build.NVCC))
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + _build.CSRC, "-I" + _build.INCLUDE,
                    "-I" + os.path.join(cuda, "include"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60, check=True)
    assert r.stdout.split() == ["0", "0"]
