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

// Polls of the grid barrier of the sort's last kernel on the current device, for
// sorts launched afterwards (0: the default). When they run out the kernel ends,
// the keys are left unspecified and *d_status gets kStatusQueueTimeout.
cudaError_t set_barrier_spins(uint32_t spins);

// The large segments of a segmented sort of integer keys: segment ids[i], i <
// *d_count <= max_segments, is [d_offsets[ids[i]], d_offsets[ids[i] + 1]) of
// d_keys (all device arrays), of more than two blocks' worth of keys; each is
// sorted on its own. A segment that starts before an earlier one's end is left
// as it is and reported (kStatusBadInput). (Not IEEE keys: the order of zeros of both signs is kept
// for a whole array only.) Temp bytes 0 for IEEE types.
size_t partition_segments_temp_bytes(int dtype, size_t n, size_t max_segments);
cudaError_t partition_segments(int dtype, void* d_keys, size_t n, const unsigned long long* d_offsets,
                               const uint32_t* d_ids, const uint32_t* d_count, size_t max_segments, void* d_temp,
                               size_t temp_bytes, cudaStream_t stream, uint32_t* d_status, LaunchRecorder* rec);

// K-way merge tiles of integer keys, sorted in shared memory: tile j in [tile0,
// tile0 + tiles) of the output is out[j*T, (j+1)*T) (T = kway_unit_tile_keys,
// the last tile shorter; 0 for IEEE types), from the slices splits[j*k + r] ..
// splits[(j+1)*k + r) of the k device runs (d_runs: a device array of k run
// pointers; splits: a (tiles + 1) x k device matrix at spacing T).
constexpr int kMaxUnitTileRuns = 1024;
size_t kway_unit_tile_keys(int dtype);
cudaError_t kway_unit_tiles(int dtype, const void* d_runs, int k, const uint64_t* d_splits, void* out, uint64_t total,
                            uint64_t tile0, uint64_t tiles, cudaStream_t stream, LaunchRecorder* rec);

}  // namespace mgs
