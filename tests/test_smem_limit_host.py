"""Dynamic shared memory past 48 KB is an attribute of a kernel on one device. csrc/smem_limit.h sets it
once on every device a process launches from; the test compiles it against a stand-in of the runtime's two
calls, and checks that no launch sets the attribute in another way."""

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "av-denoise_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <map>
#include <utility>
#include "smem_limit.h"

static int current = 0, fail_next = 0;
static std::map<std::pair<const void*, int>, int> calls;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int) {
    if (fail_next) { fail_next = 0; return cudaErrorInvalidValue; }
    ++calls[{f, current}];
    return cudaSuccess;
}
void first(int) {}
void second(int) {}

int main() {
    auto times = [](void (*f)(int), int dev) { return calls[{reinterpret_cast<const void*>(f), dev}]; };
    for (int round = 0; round < 3; ++round)
        for (int dev : {0, 1, 7, 64}) {
            current = dev;
            if (avd::allow_smem<first>(60000) != cudaSuccess) return 1;
        }
    if (times(first, 0) != 1 || times(first, 1) != 1 || times(first, 7) != 1 || times(first, 64) != 3) return 2;
    current = 0;  // another kernel of the same signature has its own
    fail_next = 1;
    if (avd::allow_smem<second>(60000) != cudaErrorInvalidValue || times(second, 0) != 0) return 3;
    if (avd::allow_smem<second>(60000) != cudaSuccess || times(second, 0) != 1) return 4;
    return 0;
}
"""


def test_every_device_gets_the_attribute_once(tmp_path):
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", "-I/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_launch_sets_the_attribute_itself():
    users = [p.name for p in sorted(CSRC.iterdir()) if "MaxDynamicSharedMemorySize" in p.read_text()]
    assert users == ["smem_limit.h"]
