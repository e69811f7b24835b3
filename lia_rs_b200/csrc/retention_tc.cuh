// Retention's prompt portions on the tensor cores (retention_tc.cu), as retention.cu launches them.
#pragma once
#include "common.cuh"

constexpr int RETENTION_TC_CHUNK = 128;         // tokens of a chunk

// d and dv 64 or 128, rows and ld readable 16 bytes at a time; `chunks`: at least as many as the portions are cut into.  `sums` [chunks, heads, d, dv].
int retention_tc_sums(const float* rows, long long ld, const float* decay, const int* segments, int n_segments, int chunks, float* sums,
                      int heads, int d, int dv, int* error_flag, cudaStream_t stream);
// `sums`: the states that the chunks start from; out [n, heads dv] bfloat16, 8-byte aligned.
int retention_tc_output(const float* rows, long long ld, const float* decay, const int* segments, int n_segments, int chunks,
                        const float* sums, void* out, int heads, int d, int dv, float eps, int* error_flag, cudaStream_t stream);
