"""A kernel's dynamic shared memory is allowed on each device that needs it.

The attribute belongs to the function on one device. A process that runs on a
second one has to raise it there too, and must not lower what a larger launch
was granted. The host code is compiled against a stand-in for the two calls.
"""

import os
import shutil
import subprocess

import pytest

from tangle_b200.build import HERE

RUNTIME = """
#pragma once
typedef int cudaError_t;
enum { cudaSuccess = 0, cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
struct cudaFuncAttributes { int maxDynamicSharedSizeBytes; };
cudaError_t cudaGetDevice(int *device);
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *attributes, const void *kernel);
cudaError_t cudaFuncSetAttribute(const void *kernel, int attribute, int value);
"""

PROGRAM = """
#include <cstdio>
#include "dynamic_smem.h"
static int device = 0, allowed[2][2] = {{49152, 49152}, {49152, 49152}};
static const char a = 0, b = 0;
static bool verbose = false;
cudaError_t cudaGetDevice(int *current) { *current = device; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *attributes, const void *kernel) {
    if (verbose) std::printf("? ");
    attributes->maxDynamicSharedSizeBytes = allowed[device][kernel == &a];
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *kernel, int, int value) {
    allowed[device][kernel == &a] = value;
    std::printf("%d%c%d ", device, kernel == &a ? 'a' : 'b', value);
    return cudaSuccess;
}
int main() {
    tgl::allow_dynamic_smem(&a, 100000);
    tgl::allow_dynamic_smem(&a, 100000);
    tgl::allow_dynamic_smem(&a, 50000);
    tgl::allow_dynamic_smem(&b, 60000);
    tgl::allow_dynamic_smem(&b, 49152);
    device = 1;  // a second device
    tgl::allow_dynamic_smem(&a, 70000);
    tgl::allow_dynamic_smem(&a, 80000);
    device = 0;
    tgl::allow_dynamic_smem(&a, 90000);
    allowed[0][1] = 49152;  // the device was reset
    tgl::allow_dynamic_smem(&a, 90000);
    std::printf("| ");
    verbose = true;  // kept grants ask once for each size and device
    static tgl::DynamicSmem kept;
    kept.allow(&b, 70000);
    kept.allow(&b, 70000);
    kept.allow(&b, 60000);
    device = 1;
    kept.allow(&b, 70000);
    device = 200;
    kept.allow(&b, 1000);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_every_device_is_allowed_its_largest(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(PROGRAM)
    program = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", os.path.join(HERE, "csrc"), "-o", program,
                    str(tmp_path / "main.cpp")], check=True)
    out = subprocess.run([program], check=True, capture_output=True, text=True).stdout
    once, kept = out.split("|")
    assert once.split() == ["0a100000", "0b60000", "1a70000", "1a80000", "0a90000"]
    assert kept.split() == ["?", "0b70000", "?", "1b70000"]
