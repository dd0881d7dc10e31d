// chain_launch.h -- kernels of one stream that are launched one after the
// other and may overlap (programmatic dependent launch), with the copies and
// memsets between them.
#pragma once

#include <cuda_runtime_api.h>
#include <stddef.h>
#include <tuple>
#include <utility>

namespace fpt {

struct ChainLaunch {
    cudaStream_t stream;
    cudaError_t status = cudaSuccess;   // of the first refused operation; none is tried after it
    bool after_kernel = false;          // the stream's last operation is a kernel of this chain

    explicit ChainLaunch(cudaStream_t st) : stream(st) {}

    // `waits`: the kernel waits for the one before it (wait_previous) and may start while that one ends.  It does so
    // behind a kernel of the chain only: behind a copy or a memset it is launched as any other.
    template <class... P, class... A>
    void launch(void (*kernel)(P...), dim3 grid, int threads, size_t smem, bool waits, A... args) {
        if (status != cudaSuccess) return;
        std::tuple<P...> values(args...);
        start(reinterpret_cast<const void *>(kernel), grid, threads, smem, waits && after_kernel, values, std::index_sequence_for<P...>());
        after_kernel = true;
    }
    void zero(void *dst, size_t bytes) { other(status == cudaSuccess ? cudaMemsetAsync(dst, 0, bytes, stream) : status); }
    void read(void *dst, const void *src, size_t bytes) {
        other(status == cudaSuccess ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream) : status);
    }

private:
    void other(cudaError_t e) {
        after_kernel = false;
        status = e;
        clear();
    }
    template <class T, size_t... K>
    void start(const void *kernel, dim3 grid, int threads, size_t smem, bool early, T &values, std::index_sequence<K...>) {
        void *params[] = {static_cast<void *>(&std::get<K>(values))...};
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = grid;
        cfg.blockDim = dim3(unsigned(threads));
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = &attr;
        cfg.numAttrs = early ? 1u : 0u;
        status = cudaLaunchKernelExC(&cfg, kernel, params);
        clear();
    }
    void clear() {
        if (status != cudaSuccess) (void)cudaGetLastError();   // reported here, not by the next call that looks
    }
};

}  // namespace fpt
