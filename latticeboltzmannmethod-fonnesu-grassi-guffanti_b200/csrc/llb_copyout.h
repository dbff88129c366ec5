// Results from device memory into the caller's (pageable) host arrays.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace llb {

struct HostCopy {
    void* dst;        // host
    const void* src;  // device
    size_t bytes;
};

// Copies n pieces in the order of `stream` and returns when they are in host
// memory and the stream is idle.
cudaError_t copy_to_host(cudaStream_t stream, const HostCopy* c, int n);

// The staging memory lives while lattices do: freed with the last one.
void staging_add_user();
void staging_drop_user();

}  // namespace llb
