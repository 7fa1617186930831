"""What a kernel needs once per device (the limit of its dynamic shared
memory): compiled on the host against fake devices, each with a limit of its
own that a launch must find raised."""
import os
import subprocess

from conftest import ROOT

SRC = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "st_once.h"

constexpr int kNdev = 70;                  // more devices than marks
constexpr int kMax = 227;                  // what a device allows at most
std::atomic<int> limit[kNdev], calls[kNdev];
st::OncePerDevice once;                    // one kernel
int fails = 0;
void check(bool ok, const char *what) { if (!ok) { fails++; std::printf("%s\n", what); } }

int launch(int dev, int need) {
    const int e = once(dev, [&] { calls[dev]++; limit[dev] = kMax; return 0; });
    return e ? e : need <= limit[dev].load() ? 0 : 1;
}

int main() {
    for (auto &l : limit) l = 48;
    // an error is returned and the next call tries again
    check(once(0, [] { return 2; }) == 2, "error not returned");
    check(launch(0, 100) == 0, "not raised after an error");
    check(launch(0, 200) == 0 && calls[0] == 1, "raised twice");
    // a second device has a limit of its own
    check(launch(1, 100) == 0 && calls[1] == 1, "second device not raised");
    check(launch(kNdev - 1, 100) == 0, "device beyond the marks");
    // threads with large and small launches never lower the limit
    std::atomic<int> bad{0};
    std::vector<std::thread> t;
    for (int k = 0; k < 8; k++)
        t.emplace_back([&, k] {
            for (int r = 0; r < 1000; r++)
                for (int d = 2; d < kNdev; d++) bad += launch(d, k % 2 ? kMax : 60) != 0;
        });
    for (auto &x : t) x.join();
    check(bad == 0, "launch above the limit");
    return fails;
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-Wall",
                           "-I" + os.path.join(ROOT, "shock_turbulence_b200", "csrc"), str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
