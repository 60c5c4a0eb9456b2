"""Kernels whose shared memory depends on the shape, launched from two threads with different shapes: the limit that one
thread's launch needs is not taken back by the other's.  A host program, whose threads really launch at the same time."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <thread>
#include "nbg_adjoint.h"
template <class Call> static int two_threads(Call call) { // refused launches
    int fails[2] = {0, 0};
    auto work = [&](int k) {
        cudaStream_t st;
        if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) { fails[k] = 1; return; }
        for (int i = 0; i < 20000; ++i) {
            fails[k] += call(k, st) != NBG_OK;
            if (i % 500 == 499) cudaStreamSynchronize(st);
        }
        cudaStreamSynchronize(st);
    };
    std::thread other(work, 1);
    work(0);
    other.join();
    return fails[0] + fails[1];
}
int main() {
    float *zero, *out[2];
    int *lists[2];
    if (cudaMalloc(&zero, 4 << 20) != cudaSuccess || cudaMemset(zero, 0, 4 << 20) != cudaSuccess) return 1;
    for (int k = 0; k < 2; ++k) {
        if (cudaMalloc(&out[k], 1 << 20) != cudaSuccess || cudaMemset(out[k], 0, 1 << 20) != cudaSuccess) return 1;
        if (cudaMalloc(&lists[k], 1 << 20) != cudaSuccess || cudaMemset(lists[k], 0, 1 << 20) != cudaSuccess) return 1;
    }
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    const int products = two_threads([&](int k, cudaStream_t st) { // 32 x K by K x 32
        return nbg_product_nt(zero, zero, out[k], 32, 32, k ? 4096 : 2000, st);
    });
    nbg_lif_grad_params p = {};
    p.slope = 10.0f;
    const int forwards = two_threads([&](int k, cudaStream_t st) { // one step of one row of 64 neurons
        const int c = k ? 4000 : 1000, n = 64;
        float *const v = out[k], *const s = v + n;
        return nbg_lif_forward_segment_gather(zero, zero, c, zero, lists[k], lists[k] + n, v, lists[k] + 2 * n, nullptr, s,
                                              nullptr, nullptr, nullptr, nullptr, zero, zero, zero, &p, 1, 1, n, st);
    });
    std::printf("%d %d %d\n", products, forwards, (int)cudaDeviceSynchronize());
    return 0;
}
"""


def test_two_threads_of_two_shapes(tmp_path):
    from neuronbridge_gb300 import build

    build.build()
    src, exe = tmp_path / "threads.cu", tmp_path / "threads"
    src.write_text(PROGRAM)
    libdir = os.path.dirname(build.LIB)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", build.INCLUDE, str(src), "-L", libdir, "-lnbg", "-lpthread",
                    "-Xlinker", f"-rpath={libdir}", "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.split() == ["0", "0", "0"], (r.returncode, r.stdout, r.stderr)
