"""Launches of the training chain, on the CPU: csrc/chain_launch.h compiled with g++ against a launch call of the test's own
that records what it is given and can refuse."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = "/usr/local/cuda/include"

PROGRAM = r"""
#include <stdio.h>
#include "chain_launch.h"
static int calls = 0, fail_at = 0, cleared = 0;
static void first(int, float) {}
static void second(const char *) {}
extern "C" {
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *kernel, void **args) {
    ++calls;
    if (kernel == reinterpret_cast<const void *>(&first))
        printf("call first %u %u %zu %u %d %g\n", c->gridDim.x, c->blockDim.x, c->dynamicSmemBytes, c->numAttrs,
               *static_cast<int *>(args[0]), double(*static_cast<float *>(args[1])));
    else printf("call second %u %u %zu %u %s\n", c->gridDim.x, c->blockDim.x, c->dynamicSmemBytes, c->numAttrs,
                *static_cast<const char **>(args[0]));
    return calls == fail_at ? cudaErrorInvalidConfiguration : cudaSuccess;
}
cudaError_t cudaGetLastError() { ++cleared; return cudaSuccess; }
}
int main() {
    for (fail_at = 0; fail_at <= 3; ++fail_at) {
        calls = cleared = 0;
        fpt::ChainLaunch chain(nullptr);
        chain.launch(first, dim3(3), 64, 128, false, 7, 2.5);
        chain.launch(second, dim3(4), 32, 0, true, "text");
        chain.launch(first, dim3(5), 96, 0, true, 8, 0.5f);
        printf("end %d %d %d %d\n", fail_at, int(chain.status), calls, cleared);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime_api.h")):
        pytest.skip("g++ or the CUDA headers are not available")
    tmp = tmp_path_factory.mktemp("chain")
    (tmp / "main.cpp").write_text(PROGRAM)
    exe = str(tmp / "chain")
    subprocess.run([gxx, "-std=c++17", "-I", os.path.join(ROOT, "fractalpathtracer_gb300", "csrc"), "-I", CUDA_INCLUDE,
                    str(tmp / "main.cpp"), "-o", exe], check=True, capture_output=True, text=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()


def test_launches_pass_their_arguments(lines):
    assert lines[:3] == ["call first 3 64 128 0 7 2.5", "call second 4 32 0 1 text", "call first 5 96 0 1 8 0.5"]


def test_refused_launch_is_kept_and_ends_the_chain(lines):
    ends = [[int(v) for v in line.split()[1:]] for line in lines if line.startswith("end")]
    assert ends == [[0, 0, 3, 0], [1, 9, 1, 1], [2, 9, 2, 1], [3, 9, 3, 1]]   # 9: invalid configuration


GAPS = r"""
#include <stdio.h>
#include "chain_launch.h"
static int refuse = 0;
static void kernel(int) {}
extern "C" {
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **) { printf("%u ", c->numAttrs); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int v, size_t n, cudaStream_t) {
    printf("zero%d:%zu ", v, n);
    return refuse == 1 ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *, const void *, size_t n, cudaMemcpyKind k, cudaStream_t) {
    printf("read%d:%zu ", int(k), n);
    return refuse == 2 ? cudaErrorInvalidValue : cudaSuccess;
}
}
int main() {
    for (refuse = 0; refuse < 3; ++refuse) {
        float loss = 0.0f;
        fpt::ChainLaunch chain(nullptr);
        for (int step = 0; step < 4; ++step) {   // a training of four steps: the loss of the first and the last is read
            const bool probe = step == 0 || step == 3;
            if (probe) chain.zero(&loss, 4);
            chain.launch(kernel, dim3(1), 32, 0, true, 1);
            chain.launch(kernel, dim3(1), 32, 0, false, 1);
            chain.launch(kernel, dim3(1), 32, 0, true, 1);
            if (probe) chain.read(&loss, &loss, 4);
        }
        printf("status%d\n", int(chain.status));
    }
    return 0;
}
"""


def test_no_overlap_behind_copies_and_memsets(tmp_path):
    """A kernel of the chain may start early behind another kernel of it only, and a refused memset or copy ends the chain."""
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime_api.h")):
        pytest.skip("g++ or the CUDA headers are not available")
    (tmp_path / "main.cpp").write_text(GAPS)
    exe = str(tmp_path / "gaps")
    subprocess.run([gxx, "-std=c++17", "-I", os.path.join(ROOT, "fractalpathtracer_gb300", "csrc"), "-I", CUDA_INCLUDE,
                    str(tmp_path / "main.cpp"), "-o", exe], check=True, capture_output=True, text=True)
    lines = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()
    assert lines[0] == "zero0:4 0 0 1 read2:4 0 0 1 1 0 1 zero0:4 0 0 1 read2:4 status0"
    assert lines[1] == "zero0:4 status1"
    assert lines[2] == "zero0:4 0 0 1 read2:4 status1"
