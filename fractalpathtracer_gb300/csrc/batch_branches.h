// batch_branches.h -- side streams of the batch's pass graph and the events
// that fork and join them.
#pragma once

#include <cuda_runtime_api.h>

namespace fpt {

template <int N> struct BranchSet {
    cudaStream_t stream[N] = {};   // of branches 1 .. N-1; branch 0 is the stream that forks
    cudaEvent_t fork = nullptr, join[N] = {};

    // Creates what is not there yet: after a failure the next call goes on with the missing ones.
    cudaError_t create() {
        cudaError_t e = cudaSuccess;
        if (!fork) e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
        for (int k = 1; k < N && e == cudaSuccess; ++k) {
            if (!join[k]) e = cudaEventCreateWithFlags(&join[k], cudaEventDisableTiming);
            if (e == cudaSuccess && !stream[k]) e = cudaStreamCreateWithFlags(&stream[k], cudaStreamNonBlocking);
        }
        return e;
    }
    // Branch k forks from `st` (which recorded `fork`), and joins it again.
    cudaStream_t branch(int k, cudaStream_t st) const { return k == 0 ? st : stream[k]; }
    cudaError_t begin(cudaStream_t st) { return cudaEventRecord(fork, st); }
    cudaError_t enter(int k) { return k == 0 ? cudaSuccess : cudaStreamWaitEvent(stream[k], fork, 0); }
    cudaError_t leave(int k, cudaStream_t st) {
        if (k == 0) return cudaSuccess;
        const cudaError_t e = cudaEventRecord(join[k], stream[k]);
        return e == cudaSuccess ? cudaStreamWaitEvent(st, join[k], 0) : e;
    }
};

}  // namespace fpt
