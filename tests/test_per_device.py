"""Set-up done once per device (csrc/per_device.h) against a fake device query:
every device gets its own, a failure is tried again, threads run it once."""
import subprocess

from ray_tracing_gb300 import build as _build

SOURCE = """
#include "per_device.h"
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
static thread_local int current = 0;
extern "C" cudaError_t cudaGetDevice(int* d) {
    *d = current;
    return current >= 0 ? cudaSuccess : cudaErrorNoDevice;
}
#define EXPECT(x) if (!(x)) { std::printf("failed: %s\\n", #x); return 1; }
int main() {
    rtgb::OncePerDevice once;
    int made[3] = {0, 0, 0};
    auto make = [&](int d) { ++made[d]; return cudaSuccess; };
    for (int d : {0, 1, 0, 1, 2, 0}) {
        current = d;
        EXPECT(once.run(make) == cudaSuccess);
    }
    EXPECT(made[0] == 1 && made[1] == 1 && made[2] == 1);
    rtgb::OncePerDevice failing;
    int tries = 0;
    auto fail_once = [&](int) { return ++tries == 1 ? cudaErrorMemoryAllocation : cudaSuccess; };
    EXPECT(failing.run(fail_once) == cudaErrorMemoryAllocation);
    EXPECT(failing.run(fail_once) == cudaSuccess && failing.run(fail_once) == cudaSuccess && tries == 2);
    current = rtgb::kMaxDevices;
    EXPECT(once.run(make) == cudaErrorInvalidDevice);
    current = -1;
    EXPECT(once.run(make) == cudaErrorNoDevice);
    rtgb::OncePerDevice shared;
    std::atomic<int> runs{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t) {
        threads.emplace_back([&, t] { current = t & 1; shared.run([&](int) { ++runs; return cudaSuccess; }); });
    }
    for (auto& t : threads) t.join();
    EXPECT(runs == 2);
    return 0;
}
"""


def test_once_per_device(tmp_path):
    (tmp_path / "once.cpp").write_text(SOURCE)
    subprocess.run(["g++", *_build.CXX_FLAGS, "-I", str(_build.CSRC), "-I", str(_build._cuda_home() / "include"),
                    str(tmp_path / "once.cpp"), "-o", str(tmp_path / "once"), "-lpthread"], check=True)
    res = subprocess.run([str(tmp_path / "once")], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
