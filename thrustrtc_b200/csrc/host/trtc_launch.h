// trtc_launch.h -- entry points of the nvcc-built (built-in type / operator) kernels.
#pragma once
#include <string>
#include <cstddef>
#include <cuda_runtime.h>

namespace trtc_host {

// compaction selector codes (same values as trtc::CompactMode)
enum : int { COMPACT_NOT_EQUAL = 2, COMPACT_UNIQUE = 5 };

// CTAs per SM of the reduce kernel: 4 x 256 threads with 16 loads each cover the memory latency, and
// the last CTA folds half as many partials as with 8 (B200, per launch, float sums of 2^28 / 67 M /
// 16.8 M / 4 M: 2 CTAs 191 / 56 / 21.8 / 12.1 us, 3: 166 / 50 / 20.7 / 11.9, 4: 160 / 48 / 20.7 / 11.8,
// 8: 167 / 51 / 23.4 / 14.4.  Per call with L2 flushed before each, 2^28 / 2^27 / 2^26 / 16.8 M floats:
// 4: 195 / 121 / 76 / 36 us, 8: 197 / 117 / 74 / 39)
enum : int { REDUCE_CTAS = 4 };

// compactions of fewer elements keep the two-phase kernel, whose one tile per CTA is done before the
// pipeline has handed a tile through its roles (B200, us per Copy_If / Remove_Copy call, two-phase
// against pipeline: 5,000 int32 20.3 / 16.9 against 22.2 / 20.9, 1 M 21.0 / 18.0 against 22.7 / 21.3,
// 4 M 25.8 / 24.7, 10 M 33 / 35 against 30.8 / 32.7)
enum : unsigned long long { COMPACT_PIPE_N = 1ull << 22 };

// radix sort of built-in key types; vals may be null; vsize = payload bytes per element
bool sort_raw(int key_tc, void* keys, void* vals, size_t vsize, size_t n, bool desc, cudaStream_t s);
bool sort_raw_narrow(int key_tc, void* keys, void* vals, size_t vsize, size_t n, bool desc, cudaStream_t s);
bool sort_raw_32(int key_tc, void* keys, void* vals, size_t vsize, size_t n, bool desc, cudaStream_t s);
bool sort_raw_64(int key_tc, void* keys, void* vals, size_t vsize, size_t n, bool desc, cudaStream_t s);
// index of the minimum in the reference's Min_Element tree order (synchronous)
bool min_element_raw(int tc, const void* keys, size_t n, cudaStream_t s, unsigned long long* idx);

// mode 0 inclusive, 1 exclusive with *init; in/out same type
bool scan_raw(int tc, int op, int mode, const void* in, void* out, size_t n, const void* init, cudaStream_t s);
// init may be null; result written to host memory (synchronous)
bool reduce_raw(int tc, int op, const void* in, size_t n, const void* init, void* result_host, cudaStream_t s);
// kernel-only variant: result left in device memory at *result_dev (asynchronous)
bool reduce_raw_async(int tc, int op, const void* in, size_t n, const void* init, void** result_dev, cudaStream_t s);
// segmented scan, EqualTo keys / Plus values; mode 0 inclusive, 1 exclusive with *init (or 0)
bool scan_by_key_raw(int key_tc, int val_tc, int mode, const void* keys, const void* vals, void* out, size_t n,
                     const void* init, cudaStream_t s);
// compaction with built-in selectors: CM_NOT_EQUAL (value) or CM_UNIQUE; count is synchronous
bool compact_raw(int tc, int mode, const void* in, void* out, size_t n, const void* value, cudaStream_t s,
                 unsigned long long* count);

// batched segmented sort + exclusive scan (launch_segmented.cu); 4-byte values
size_t segmented_workspace_bytes(int tc, size_t n, size_t nseg);
int segmented_tuned_items(int tc);
bool segmented_sort_scan_raw(int tc, void* keys, void* vals, void* scan, const unsigned long long* off, size_t nseg,
                             size_t n, void* ws, size_t ws_bytes, bool desc, cudaStream_t s);
bool segmented_autotune(int tc, const unsigned long long* off, size_t nseg, size_t n, cudaStream_t s, int* chosen);
std::string segmented_tuning_json();
bool segmented_tuning_load(const char* json);

}  // namespace trtc_host
