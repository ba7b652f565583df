"""Shared memory that a kernel is given once per device must not depend on the call that comes first: two host threads may both come
first, and the smaller size would then stand under the larger.  The launcher of the delta rule's chunks, compiled for the host with a
stand-in for the CUDA call, in which another thread's call happens (no GPU: nothing is launched)."""
import subprocess

from tensorline_b200.csrc.build import ARCH_FLAGS, CSRC, _nvcc

HARNESS = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <map>
static std::map<const void*, int> given;
static void (*other_thread)() = nullptr;
template <typename F> static cudaError_t set_attribute(F f, cudaFuncAttribute, int bytes) {
    given[(const void*)f] = bytes;
    if (other_thread) { void (*run)() = other_thread; other_thread = nullptr; run(); }
    return cudaSuccess;
}
static cudaError_t get_device(int* dev) { *dev = 0; return cudaSuccess; }
#define cudaFuncSetAttribute set_attribute
#define cudaGetDevice get_device
#include "delta_chunk.cu"
alignas(16) static unsigned char memory[64];
static void call(int dv) {
    float* f = (float*)memory;
    int* i = (int*)memory;
    tl_delta_chunks(f, 2 * 128 + dv, 0, 128, 256, f, 2, f, f, f, 0, i, i, i, 1, i, 1, memory, i, f, 1, 1, 128, dv, 0);
}
int main() {
    other_thread = [] { call(64); };                     // comes between the first thread's call and its note of it
    call(1024);
    call(1024);
    const int needs = (2 * 32 * (128 + 4) + 32 * 1024) * 4;
    const int got = given[(const void*)dc_prepare_kernel<128>];
    std::printf("%d of %d\n", got, needs);
    return got >= needs ? 0 : 1;
}
"""


def test_two_threads_first_calls_leave_the_larger_size(tmp_path):
    (tmp_path / "harness.cu").write_text(HARNESS)
    cmd = [_nvcc(), *ARCH_FLAGS, "-O0", "-Xcicc", "-O0", "-Xptxas", "-O0", "-std=c++17", "-I", str(CSRC), "-o", str(tmp_path / "harness"), str(tmp_path / "harness.cu")]
    built = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert built.returncode == 0, built.stderr
    run = subprocess.run([str(tmp_path / "harness")], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
