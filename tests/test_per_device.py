"""PerDevice (csrc/vsc_device.h): launch preparation once per device, compiled on
the host against a stand-in for the runtime's cudaGetDevice; and every kernel's
dynamic shared memory opt-in goes through per-device state."""
import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "video-stream-consistency_gb300" / "csrc"
CUDA = Path("/usr/local/cuda/include")

PROGRAM = r"""
#include "vsc_device.h"
#include <cassert>
#include <thread>
#include <vector>
static thread_local int device = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
int main()
{
    static vsc::PerDevice<int> p;
    int made[3] = {}, got = 0;
    auto make = [&](int* v) { ++made[device]; *v = 100 + device; return cudaSuccess; };
    auto fail = [&](int*) { return cudaErrorInvalidValue; };
    assert(p.get(fail, &got) == cudaErrorInvalidValue);  // not kept
    for (int round = 0; round < 2; ++round)
        for (device = 0; device < 3; ++device)
            assert(p.get(make, &got) == cudaSuccess && got == 100 + device && made[device] == 1);
    device = vsc::kMaxDevices;
    assert(p.get(make, &got) == cudaErrorInvalidDevice);
    static vsc::PerDevice<int> q;
    int count = 0;
    std::vector<std::thread> t;
    for (int i = 0; i < 8; ++i)
        t.emplace_back([&] { int v = 0; q.get([&](int* x) { ++count; *x = 7; return cudaSuccess; }, &v); assert(v == 7); });
    for (auto& x : t) x.join();
    assert(count == 1);
}
"""


def test_per_device_state(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(CSRC), "-I", str(CUDA), str(src), "-o", str(exe)],
                   check=True)
    subprocess.run([str(exe)], check=True)


def test_opt_ins_are_not_once_per_process():
    """A once_flag would opt in on the first device alone."""
    for f in sorted(CSRC.glob("*.cu")):
        for body in re.findall(r"call_once\(\w+, \[[^\]]*\] \{(.*?)\n    \}\);", f.read_text(), re.S):
            assert "cudaFuncSetAttribute" not in body, f.name
