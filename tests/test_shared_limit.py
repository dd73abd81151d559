"""The process-wide limit of a kernel's dynamic shared memory (csrc/shared_limit.h), compiled against
stand-ins for the runtime's calls: whatever two contexts created at the same time do between each
other's calls, every context's kernels can be launched afterwards."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ether_gb300", "csrc")

RUNTIME = """
#pragma once
#include <cstddef>
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum cudaDeviceAttr { cudaDevAttrMaxSharedMemoryPerBlockOptin = 97 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
struct cudaFuncAttributes { size_t sharedSizeBytes; int maxDynamicSharedSizeBytes; };
cudaError_t cudaGetDevice(int *dev);
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int dev);
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *f);
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v);
"""

# another context's whole call runs before the step-th call of this one
PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "shared_limit.h"
static const int kOptin = 232448, kStatic = 1000;
static int limit = 49152, step = 0, calls = 0;
static bool inside = false;
static void between() {
    if (inside || ++calls != step) return;
    inside = true;
    if (ether::allow_shared(&limit) != cudaSuccess) exit(3);
    inside = false;
}
cudaError_t cudaGetDevice(int *dev) { between(); *dev = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { between(); *v = kOptin; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
    between();
    a->sharedSizeBytes = kStatic;
    a->maxDynamicSharedSizeBytes = limit;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int v) {
    between();
    if (v < 0 || v + kStatic > kOptin) return cudaErrorInvalidValue;  // as the runtime answers
    limit = v;
    return cudaSuccess;
}
int main(int, char **argv) {
    step = atoi(argv[1]);
    if (ether::allow_shared(&limit) != cudaSuccess) return 2;
    printf("%d", limit);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("limit")
    (d / "cuda_runtime.h").write_text(RUNTIME)
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(d), "-I", CSRC, str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    return str(d / "main")


@pytest.mark.parametrize("step", range(6))
def test_limit_holds_whatever_comes_between(program, step):
    r = subprocess.run([program, str(step)], capture_output=True, text=True)
    assert r.returncode == 0
    assert int(r.stdout) == 232448 - 1000


def test_nothing_else_sets_a_limit_that_varies():
    """Every other call of cudaFuncSetAttribute in the sources sets a constant of its kernel."""
    for f in sorted(os.listdir(CSRC)):
        for line in open(os.path.join(CSRC, f)):
            if "cudaFuncAttributeMaxDynamicSharedMemorySize" in line and f != "shared_limit.h":
                assert any(c in line for c in ("SM_BYTES + 1024", "XSM_BYTES")), (f, line)
