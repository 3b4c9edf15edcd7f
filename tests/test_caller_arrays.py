"""Which of a caller's arrays the scene update's kernel reads by itself and which it has copied: the
rule of host_util.h over every kind of memory the runtime reports, compiled for the host alone (a
machine of this project's tests has one GPU, so that memory of another one exists only here)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include <cstdio>
#include "host_util.h"
using namespace helio;
static int check(cudaMemoryType type, int owner, bool mapped_here, uintptr_t at, bool direct, bool mapped) {
    cudaPointerAttributes a{};
    a.type = type;
    a.device = owner;
    const void* p = reinterpret_cast<const void*>(at);
    a.devicePointer = mapped_here ? const_cast<void*>(p) : nullptr;
    const bool d = reads_directly(a, 0, p, 16), m = reads_mapped(a, 0, p, 16);
    if (d == direct && m == mapped) return 0;
    std::printf("type %d owner %d mapped %d at %zx: %d %d\n", (int)type, owner, (int)mapped_here, (size_t)at, d, m);
    return 1;
}
int main() {
    int bad = 0;
    bad += check(cudaMemoryTypeDevice, 0, true, 0x1000, true, true);
    bad += check(cudaMemoryTypeDevice, 0, true, 0x1004, false, false);       // not for 16-byte loads
    bad += check(cudaMemoryTypeDevice, 1, true, 0x1000, false, false);       // another device's
    bad += check(cudaMemoryTypeDevice, 0, true, 0, false, false);
    bad += check(cudaMemoryTypeManaged, 0, true, 0x1000, false, true);
    bad += check(cudaMemoryTypeManaged, 0, true, 0x1008, false, false);
    bad += check(cudaMemoryTypeHost, 0, true, 0x1000, false, true);          // page-locked and mapped
    bad += check(cudaMemoryTypeHost, 0, false, 0x1000, false, false);        // page-locked, not mapped at its address
    bad += check(cudaMemoryTypeUnregistered, 0, false, 0x1000, false, false);  // no memory of CUDA's
    return bad;
}
"""


def test_only_this_devices_memory_is_read_directly(tmp_path):
    from helio_b200 import build

    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(SOURCE)
    inc = [f"-I{ROOT / 'helio_b200' / 'csrc'}", f"-I{build.CUDA_HOME / 'include'}", f"-L{build.CUDA_HOME / 'lib64'}"]
    subprocess.run(["g++", "-std=c++17", str(src), "-o", str(exe), *inc, "-lcudart_static", "-lrt", "-lpthread", "-ldl"],
                   check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
