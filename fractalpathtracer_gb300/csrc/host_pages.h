// host_pages.h -- memory of result arrays on the host (plain C++, no CUDA).
#pragma once

#include <stddef.h>
#include <initializer_list>

namespace fpt {

// Gives the pages of result arrays that the caller has only reserved so far
// their memory, while the GPU works on the results.
struct HostRange {
    void *data;
    size_t bytes;
};
void populate_pages(std::initializer_list<HostRange> ranges);

}  // namespace fpt
