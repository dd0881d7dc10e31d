"""Streams and events of the batch's parallel branches, on the CPU: csrc/batch_branches.h compiled with g++ against runtime
calls of the test's own, one of which fails."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = "/usr/local/cuda/include"

PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include "batch_branches.h"
static int calls = 0, fail_at = 0, made = 0;
static cudaError_t step() { return ++calls == fail_at ? cudaErrorMemoryAllocation : cudaSuccess; }
template <class T> static cudaError_t make(T *out) {
    const cudaError_t e = step();
    if (e == cudaSuccess) *out = reinterpret_cast<T>(size_t(++made) * 16u);
    return e;
}
template <class T> static cudaError_t use(T handle) { return handle ? step() : cudaErrorInvalidResourceHandle; }
extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned int) { return make(e); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned int) { return make(s); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return s ? use(e) : cudaErrorInvalidResourceHandle; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned int) { return s ? use(e) : cudaErrorInvalidResourceHandle; }
}
constexpr int N = 5;
int main() {
    cudaStream_t own = reinterpret_cast<cudaStream_t>(size_t(8));
    for (int at = 1; at <= 2 * N - 1; ++at) {   // the fork event, N - 1 join events, N - 1 streams
        fpt::BranchSet<N> set;
        calls = made = 0;
        fail_at = at;
        const cudaError_t first = set.create();
        const cudaError_t second = set.create();
        bool whole = set.fork != nullptr;
        for (int k = 1; k < N; ++k) whole = whole && set.join[k] && set.stream[k];
        const cudaError_t third = set.create();
        printf("create %d %d %d %d %d %d\n", at, first != cudaSuccess, second == cudaSuccess, whole, third == cudaSuccess, made);
    }
    fpt::BranchSet<N> set;
    fail_at = 0;
    set.create();
    for (int at = 0; at <= 3 * (N - 1) + 1; ++at) {   // record the fork; per branch wait, record, wait
        calls = 0;
        fail_at = at;
        cudaError_t e = set.begin(own);
        for (int k = 0; k < N && e == cudaSuccess; ++k) {
            e = set.enter(k);
            if (e == cudaSuccess) e = set.branch(k, own) ? set.leave(k, own) : cudaErrorInvalidResourceHandle;
        }
        printf("pass %d %d %d\n", at, e != cudaSuccess, calls);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime_api.h")):
        pytest.skip("g++ or the CUDA headers are not available")
    tmp = tmp_path_factory.mktemp("branches")
    (tmp / "main.cpp").write_text(PROGRAM)
    exe = str(tmp / "branches")
    subprocess.run([gxx, "-std=c++17", "-I", os.path.join(ROOT, "fractalpathtracer_gb300", "csrc"), "-I", CUDA_INCLUDE,
                    str(tmp / "main.cpp"), "-o", exe], check=True, capture_output=True, text=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return [line.split() for line in out.splitlines()]


def test_creation_goes_on_after_a_failure(lines):
    """Whichever creation fails, the call reports it, the next one makes what is missing and nothing is made twice."""
    rows = [[int(v) for v in r[1:]] for r in lines if r[0] == "create"]
    assert len(rows) == 9
    for at, failed, second, whole, third, made in rows:
        assert (failed, second, whole, third, made) == (1, 1, 1, 1, 9), at


def test_fork_and_join_failures_are_reported(lines):
    rows = [[int(v) for v in r[1:]] for r in lines if r[0] == "pass"]
    assert rows[0] == [0, 0, 13]
    for at, failed, calls in rows[1:]:
        assert failed == 1 and calls == at, at      # nothing is called after the failure
