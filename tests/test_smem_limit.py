"""Shared-memory limits of kernels (host code, on stand-ins for the two CUDA calls): each device is asked once, and again where a launch needs more."""
import os
import subprocess

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "distributed-llama-multiusers_b200", "csrc", "cuda")


def test_each_device_is_asked_once_and_for_more(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text("""
#pragma once
#include <cstddef>
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize };
inline int fake_device = 0, fake_calls = 0, fake_bytes = 0;
inline cudaError_t cudaGetDevice(int* d) { *d = fake_device; return cudaSuccess; }
template <typename K> cudaError_t cudaFuncSetAttribute(K, cudaFuncAttribute, int bytes) { fake_calls++; fake_bytes = bytes; return bytes > 1000 ? cudaErrorInvalidValue : cudaSuccess; }
inline const char* cudaGetErrorString(cudaError_t) { return "invalid"; }
""")
    (tmp_path / "t.cpp").write_text("""
#include <cstdio>
#include <initializer_list>
#include "smem_limit.cuh"
void dl_set_error(const char*, ...) {}
static void kernel(int) {}
static int ask(int device, size_t bytes) {
    static SmemLimit given;
    fake_device = device;
    const int before = fake_calls, rc = dl_smem_limit("t", kernel, bytes, given);
    return rc < 0 ? rc : fake_calls - before;
}
int main() {
    for (auto c : {ask(0, 100), ask(0, 100), ask(1, 100), ask(1, 50), ask(0, 200), ask(0, 100), ask(0, 2000), ask(0, 200), ask(99, 10), ask(99, 10)}) printf("%d ", c);
}
""")
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", CUDA, str(tmp_path / "t.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split() == ["1", "0", "1", "0", "1", "0", "-1", "0", "1", "1"]


def test_no_limit_is_raised_once_per_process():
    for f in sorted(os.listdir(CUDA)):
        lines = open(os.path.join(CUDA, f)).read().split("\n")
        for i, line in enumerate(lines):
            if "cudaFuncSetAttribute(" in line:
                assert not any(w in " ".join(lines[max(0, i - 4):i]) for w in ("static bool", "static size_t")), (f, i + 1)
