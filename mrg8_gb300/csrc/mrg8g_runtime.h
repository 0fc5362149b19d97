// mrg8g_runtime.h -- host runtime helpers shared by the C ABI translation
// units (errors, per-device setup, launch planning, state bookkeeping).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <vector>

#include "mrg8g_internal.h"

namespace mrg8g {

struct DeviceInfo;

// Record an error for mrg8g_last_error() and return `code`.
int fail(int code, const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);

// Make the current device ready (tables uploaded, limits queried).
int ensure_device(int* dev_out, const DeviceInfo** info);
int device_sms();
// An error if a kernel of an earlier launch on the current device gave up one
// of its bounded waits; the word such a kernel sets (device address).
int check_waits();
uint32_t* device_fault();

// Resident blocks of the recurrence batch kernel on each SM, of 128 or 256 threads.
int device_batch_blocks(int threads);

int kind_elem_bytes(int kind);
bool kind_valid(int kind);
int default_layout_V(int kind);
// A batch's tile rows are of 32 kBatchLayoutV outputs.
constexpr int kBatchLayoutV = 2;
// Streams of a batch launch on each SM, the fewest of any kind (mixed batches:
// three producers of four).
constexpr uint64_t kBatchStreamsPerSM = 12;

// Order of the kinds in a mixed batch: with the tiles of a kind together the
// writers mostly run the code of one kind at a time (10,000 uneven instances of
// three kinds: 2,660 -> 2,443 microseconds).
inline int kind_order(int kind) { return kind_elem_bytes(kind) == 8 ? 0 : kind == 0 ? 2 : 1; }

// Host -> device copy from pageable memory that has reached the device when
// it returns.  A plain cudaMemcpy from pageable memory may return once the
// data is staged, before the copy lands, and nothing orders that copy (on the
// legacy default stream) before work on a non-blocking stream, such as the
// serving slots or a caller's stream.
inline cudaError_t copy_to_device(void* dst, const void* src, size_t bytes) {
    cudaError_t e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
    return e != cudaSuccess ? e : cudaStreamSynchronize(0);
}

int validate_state(const uint32_t st[8]);
void advance_state(uint32_t st[8], uint64_t n);
// Enqueue a batch on the kernel that recurrence_blocks names.  kind: of all its instances, or
// -1; longest: outputs of its longest tile; threads, blocks_per_sm: as
// mrg8g_batch_config.
cudaError_t launch_batch(const BatchArgs& a, int kind, uint64_t longest, int threads, int blocks_per_sm,
                         cudaStream_t st);
int launch_plain_call(const uint32_t st[8], void* d_out, uint64_t n, int kind, cudaStream_t s, int V);

}  // namespace mrg8g

// Tiles of a batch: make_tiles, sort_largest_first, count_tiles, tile_prefix.
#include "mrg8g_tiles.h"
