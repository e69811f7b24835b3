// What the chunked kernels of the linear recurrences share (retention with one fixed decay a head, gated linear
// attention with a decay per token and key channel): the chunk's length, how a CTA finds its chunk among a step's
// portions, and how a chunk's rows come into shared memory.
#pragma once
#include "common.cuh"

namespace {
constexpr int CHUNK = 32;

__device__ __forceinline__ float4 scaled(float4 v, float w) { return make_float4(v.x * w, v.y * w, v.z * w, v.w * w); }

// [CHUNK][width] of a chunk's rows into shared memory (row stride `stride`, zero behind `len` rows), each row times
// weight^(len - 1 - t) when weight_log2 is given; four elements at a time (`vec`: width and ld multiples of four, the
// base 16-byte aligned), several loads in flight.
__device__ __forceinline__ void load_chunk(float* __restrict__ dst, int stride, const float* __restrict__ src, long long ld,
                                           int len, int width, bool vec, bool weighted, float weight_log2) {
    if (vec) {
        const int w4 = width / 4;
#pragma unroll 4
        for (int e = threadIdx.x; e < CHUNK * w4; e += blockDim.x) {
            const int t = e / w4, i4 = e - t * w4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (t < len) v = *reinterpret_cast<const float4*>(src + (size_t)t * ld + 4 * i4);
            if (weighted) v = scaled(v, exp2f((float)(len - 1 - t) * weight_log2));
            *reinterpret_cast<float4*>(dst + t * stride + 4 * i4) = v;
        }
        return;
    }
    const int padded = (width + 3) & ~3;
    for (int e = threadIdx.x; e < CHUNK * padded; e += blockDim.x) {
        const int t = e / padded, i = e - t * padded;
        float value = 0.f;
        if (t < len && i < width) value = src[(size_t)t * ld + i] * (weighted ? exp2f((float)(len - 1 - t) * weight_log2) : 1.0f);
        dst[t * stride + i] = value;
    }
}

// 16 bytes into shared memory (zeros where there is nothing to bring), asynchronously; a thread's copies since the last commit are
// a group, and bring_wait<N> leaves at most the N youngest groups in flight.
__device__ __forceinline__ void bring16(float* dst, const float* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void bring_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void bring_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// acc[i][j] += sum_k a[2 i rows][k] b[k][j] over `count` k (a multiple of four): a thread's part of a product of two tiles in shared
// memory, I rows two apart and CJ groups of four columns 64 apart.
template <int I, int CJ>
__device__ __forceinline__ void multiply_tiles(float (&acc)[I][CJ * 4], const float* a_row, int a_stride, const float* b_row, int b_stride,
                                               int count) {
#pragma unroll 2
    for (int k = 0; k < count; k += 4) {
        float4 a[I];
#pragma unroll
        for (int i = 0; i < I; ++i) a[i] = *reinterpret_cast<const float4*>(a_row + 2 * i * a_stride + k);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            float b[CJ * 4];
#pragma unroll
            for (int c = 0; c < CJ; ++c) {
                const float4 x = *reinterpret_cast<const float4*>(b_row + (k + kk) * b_stride + c * 64);
                b[4 * c] = x.x, b[4 * c + 1] = x.y, b[4 * c + 2] = x.z, b[4 * c + 3] = x.w;
            }
#pragma unroll
            for (int i = 0; i < I; ++i) {
                const float w = kk == 0 ? a[i].x : kk == 1 ? a[i].y : kk == 2 ? a[i].z : a[i].w;
#pragma unroll
                for (int j = 0; j < CJ * 4; ++j) acc[i][j] = fmaf(w, b[j], acc[i][j]);
            }
        }
    }
}

// which portion and which of its chunks (of LENGTH tokens) the CTA `index` serves: false when there is none
template <int LENGTH = CHUNK>
__device__ __forceinline__ bool find_chunk(const int* __restrict__ segments, int n_segments, int index, int* first_row,
                                           int* length, int* segment, int* chunk) {
    for (int s = 0; s < n_segments; ++s) {
        const int count = segments[3 * s + 2];
        const int chunks = (count + LENGTH - 1) / LENGTH;
        if (index < chunks) {
            *first_row = segments[3 * s] + index * LENGTH;
            *length = min(LENGTH, count - index * LENGTH);
            *segment = s;
            *chunk = index;
            return true;
        }
        index -= chunks;
    }
    return false;
}
}  // namespace
