// chain_launch.h -- kernels of one stream that are launched one after the
// other and may overlap (programmatic dependent launch).
#pragma once

#include <cuda_runtime_api.h>
#include <stddef.h>
#include <tuple>
#include <utility>

namespace fpt {

struct ChainLaunch {
    cudaStream_t stream;
    cudaError_t status = cudaSuccess;   // of the first refused launch; none is tried after it

    explicit ChainLaunch(cudaStream_t st) : stream(st) {}

    // `early`: the kernel may start while the one before it ends.
    template <class... P, class... A>
    void launch(void (*kernel)(P...), dim3 grid, int threads, size_t smem, bool early, A... args) {
        if (status != cudaSuccess) return;
        std::tuple<P...> values(args...);
        start(reinterpret_cast<const void *>(kernel), grid, threads, smem, early, values, std::index_sequence_for<P...>());
    }

private:
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
        if (status != cudaSuccess) (void)cudaGetLastError();   // reported here, not by the next call that looks
    }
};

}  // namespace fpt
