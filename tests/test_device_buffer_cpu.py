"""The device buffer that the engines keep between calls (csrc/nbg_common.cuh): after a failed allocation it is empty, so that
the next call allocates again instead of launching on a null pointer, and the error is not found again by a later check.

The program asks for more than any device has; without a device every allocation fails, which is the same case."""
import os
import subprocess

from neuronbridge_gb300 import build

PROGRAM = r"""
#include <cstdio>
#include "nbg_common.cuh"
int main() {
    const size_t most = (size_t)1 << 58; // bytes that no device has
    DevBuf<char> a;
    if (a.alloc(most) == cudaSuccess || a.n != 0 || a.p != nullptr) return 1;
    if (a.alloc(0) != cudaSuccess || a.n != 0) return 2;
    DevBuf<int> b; // a kept buffer that cannot grow
    if (b.alloc(4) == cudaSuccess && (b.n != 4 || b.p == nullptr)) return 3;
    if (b.alloc(most / sizeof(int)) == cudaSuccess || b.n != 0 || b.p != nullptr) return 4;
    int devices = 0;
    if (cudaGetDeviceCount(&devices) == cudaSuccess && cudaGetLastError() != cudaSuccess) return 5;
    std::puts("ok");
    return 0;
}
"""


def test_a_failed_allocation_leaves_the_buffer_empty(tmp_path):
    src, exe = tmp_path / "buffer.cu", tmp_path / "buffer"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", build.INCLUDE, "-I", build.CSRC, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, env={**os.environ})
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)
