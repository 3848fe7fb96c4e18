// Partition sort: the plain (keys-only, whole-key) device sort. Host-side
// interface; the kernels and their reasons are in partition_sort.cu.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "launch.cuh"

namespace mgs {

// Scratch bytes of one partition sort of n keys, its ping-pong buffer included.
size_t partition_sort_temp_bytes(int dtype, size_t n);

// Sorts d_keys[0..n) ascending in place, with the bytes a stable sort in the
// engine's key order gives. n below 2^32. Asynchronous; device-side failures
// are OR-ed into *d_status when it is not null.
cudaError_t partition_sort(int dtype, void* d_keys, size_t n, void* d_temp, size_t temp_bytes, cudaStream_t stream,
                           uint32_t* d_status, LaunchRecorder* rec);

}  // namespace mgs
