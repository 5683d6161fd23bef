"""Which memory a kernel copies in place of the driver (csrc/runtime/device_range.h), against a CUDA runtime of this
file's own with two devices: one allocation of 4,096 bytes at 0x10000 on device 0. No GPU is used."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include "runtime/device_range.h"
#include <cstdio>
#include <cstdlib>
static int current_device = 0;
static int range_of(unsigned long long* base, size_t* size, unsigned long long p) {
    if (p < 0x10000 || p >= 0x11000) return 1;
    *base = 0x10000;
    *size = 0x1000;
    return 0;
}
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = current_device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    const auto at = reinterpret_cast<uintptr_t>(p);
    a->type = at >= 0x10000 && at < 0x11000 ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    a->device = 0;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned int, unsigned long long,
                                             cudaDriverEntryPointQueryResult*) {
    *f = reinterpret_cast<void*>(&range_of);
    return cudaSuccess;
}
}
int main(int argc, char** argv) {
    current_device = std::atoi(argv[1]);
    const auto at = std::strtoull(argv[3], nullptr, 0);
    std::printf("%d\n", flamegpu::detail::device_range(reinterpret_cast<void*>(at), std::strtoull(argv[4], nullptr, 0),
                                                       std::atoi(argv[2])));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from flamegpu2_gb300.build import CUDA_HOME
    d = tmp_path_factory.mktemp("device_range")
    (d / "fake.cpp").write_text(FAKE)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "flamegpu2_gb300", "csrc"),
                    "-I", os.path.join(CUDA_HOME, "include"), str(d / "fake.cpp"), "-o", str(d / "fake")], check=True)
    return str(d / "fake")


@pytest.mark.parametrize("current,simulation,at,size,want", [
    (0, 0, 0x10000, 4096, True), (0, 0, 0x10010, 4080, True), (0, 0, 0x10010, 4081, False), (0, 0, 0x10008, 16, False),
    (0, 0, 0x20000, 16, False), (0, 0, 0, 16, False),
    (1, 0, 0x10000, 4096, False),  # the simulation's memory, but the thread is on another device
    (1, 1, 0x10000, 4096, False), (0, 1, 0x10000, 4096, False)])
def test_device_range(program, current, simulation, at, size, want):
    out = subprocess.run([program, str(current), str(simulation), str(at), str(size)], capture_output=True, text=True, check=True)
    assert out.stdout.strip() == str(int(want))
