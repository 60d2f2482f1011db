"""What the launchers remember of a device, on the CPU: compiled from the library's header against a fake runtime."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r'''
#include "pk100_internal.h"
#include <cstdio>
#include <thread>
#include <vector>

static thread_local int device = 0;
static std::atomic<int> grants[128], asked[128];
static std::atomic<int> failing{-1};
static const void* granted_to = nullptr;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    if (device == failing.load()) return cudaErrorInvalidValue;
    if (a != cudaFuncAttributeMaxDynamicSharedMemorySize || v != 1000) return cudaErrorInvalidValue;
    granted_to = f;
    grants[device]++;
    return cudaSuccess;
}
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int d) { asked[d]++; *v = d == 2 ? 0 : 100 + d; return cudaSuccess; }
extern "C" cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
void kernel_a(int) {}
void kernel_b(int) {}
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    for (int d : {0, 1, 0, 1}) {
        device = d;
        CHECK(pk100_grant_smem<kernel_a>(1000) == cudaSuccess && pk100_sm_count() == 100 + d);
    }
    CHECK(grants[0] == 1 && grants[1] == 1 && asked[0] == 1 && asked[1] == 1);     // once on each device
    CHECK(pk100_grant_smem<kernel_b>(1000) == cudaSuccess && grants[1] == 2);       // each kernel by itself
    CHECK(granted_to == reinterpret_cast<const void*>(&kernel_b));
    device = 3;
    failing = 3;
    CHECK(pk100_grant_smem<kernel_a>(1000) == cudaErrorInvalidValue);               // a refusal is not remembered
    failing = -1;
    CHECK(pk100_grant_smem<kernel_a>(1000) == cudaSuccess && grants[3] == 1);
    device = 100;                                                                   // behind the table
    CHECK(pk100_grant_smem<kernel_a>(1000) == cudaSuccess && pk100_grant_smem<kernel_a>(1000) == cudaSuccess && grants[100] == 2);
    CHECK(pk100_sm_count() == 200 && pk100_sm_count() == 200);
    device = 2;
    CHECK(pk100_sm_count() == 148);
    std::vector<std::thread> threads;
    std::atomic<int> wrong{0};
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            device = 8 + t % 4;
            for (int i = 0; i < 1000; ++i)
                if (pk100_grant_smem<kernel_a>(1000) != cudaSuccess || pk100_sm_count() != 100 + device) wrong++;
        });
    for (auto& t : threads) t.join();
    CHECK(wrong == 0);
    for (int d = 8; d < 12; ++d) CHECK(grants[d] >= 1 && grants[d] <= 2);
    return 0;
}
'''


def test_attributes_and_sm_counts_are_kept_per_device(tmp_path):
    """Dynamic shared memory is granted to a kernel on every device that it runs on, and the SMs counted are those of the
    current device."""
    include = Path("/usr/local/cuda/include")
    if not (include / "cuda_runtime.h").exists():
        pytest.skip("CUDA headers not found")
    src = tmp_path / "per_device.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "per_device"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{include}", f"-I{ROOT / 'l4-parakeet-rs_b200' / 'csrc'}",
                    str(src), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert res.returncode == 0, res.stdout
