// Causal attention of prompt portions over the paged 32-bit cache, in tiles: what attention_generic.cu computes, a warp a token
// and head, for the rows of a portion together.
//
// A CTA owns 64 rows = (64 / g) consecutive tokens x the g query heads of one kv head (rows beyond them are idle) and walks
// the keys they can see 32 at a time; keys and values come by 16-byte asynchronous copies a chunk ahead, once for all 64 rows.
// Eight lanes share four rows: each scores four of a chunk's keys against them (keys 8 apart and rows 16 apart, so that the
// 16-byte loads of a warp meet no bank twice), the row's maximum and sum meet by shuffles, the probabilities go through shared
// memory inside the warp, and each lane owns an eighth of the head's columns of its four rows.
//
// Every number is formed as attention_generic.cu forms it, in the same order: a score is one chain of multiply-adds over
// ascending elements, a chunk's maximum moves the reference point, the chunk's exponentials are summed pairwise 16, 8, 4, 2 and 1
// keys apart, and an output element is one chain over ascending keys.  So a row's result is the same bits as there, however its
// request's tokens are cut into portions and single tokens (all keys visible: a window would cut a row's chunks elsewhere).
// What bounds it is the loads from shared memory beside the multiply-adds (a half of a score's, a third of an output's).
#include <type_traits>

#include "common.cuh"

namespace {
constexpr int ROWS = 64, KEYS = 32, THREADS = 128;

__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <int D>
__global__ void __launch_bounds__(THREADS)
attention_prefill_f32_kernel(const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
                             const int* __restrict__ segments, int n_segments, const int* __restrict__ slots,
                             const int* __restrict__ block_table, int table_stride, float* __restrict__ out, int nq, int nkv,
                             int page_size, int page_shift, int tokens_per_tile, float scale, int num_pages,
                             int* __restrict__ error_flag) {
    constexpr int LD = D + 4, LP = KEYS + 4, GROUPS = D / 32;
    extern __shared__ __align__(16) float prefill_shared[];
    float* qs = prefill_shared;                       // [ROWS][LD]
    float* kv = qs + ROWS * LD;                       // [2][K, V][KEYS][LD]
    float* ps = kv + 4 * KEYS * LD;                   // [ROWS][LP]
    pdl_launch_dependents();
    pdl_wait();
    const int group = nq / nkv, kvh = blockIdx.x % nkv;
    // (later tiles first: they have the most keys)
    int tile = (gridDim.x - 1 - blockIdx.x) / nkv, seg = 0, offset = 0, start = 0, count = 0;
    for (; seg < n_segments; ++seg) {
        offset = segments[3 * seg];
        start = segments[3 * seg + 1];
        count = segments[3 * seg + 2];
        const int tiles = (count + tokens_per_tile - 1) / tokens_per_tile;
        if (tile < tiles) break;
        tile -= tiles;
    }
    if (seg >= n_segments) return;
    const int slot = slots[offset];
    if (slot < 0) return;
    const int tok0 = tile * tokens_per_tile, tok_count = min(tokens_per_tile, count - tok0);
    const int pos_first = start + tok0, key_end = pos_first + tok_count;
    const int* table = block_table + (size_t)slot * table_stride;
    const int tid = threadIdx.x, lane = tid & 31, tx = lane & 7, ty = (tid >> 5) * 4 + (lane >> 3);
    const int rows_used = tok_count * group;

    for (int e = tid; e < ROWS * (D / 4); e += THREADS) {
        const int r = e / (D / 4), c = (e % (D / 4)) * 4, tok = r / group;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows_used) v = *reinterpret_cast<const float4*>(q + ((size_t)(offset + tok0 + tok) * nq + kvh * group + (r - tok * group)) * D + c);
        *reinterpret_cast<float4*>(qs + r * LD + c) = v;
    }
    auto fetch = [&](int base, int buffer) {
        float* ks = kv + buffer * 2 * KEYS * LD;
        // four threads bring a key's and a value's row; a key without a page (the flag is up) counts for nothing and reads zeros
        const int r = tid >> 2, j = base + r;
        const int row = j < key_end ? cache_row_of(table, j, page_size, page_shift, num_pages, error_flag) : -1;
        const float* k = k_pages + ((size_t)max(row, 0) * nkv + kvh) * D;
        const float* v = v_pages + ((size_t)max(row, 0) * nkv + kvh) * D;
#pragma unroll
        for (int c = (tid & 3) * 4; c < D; c += 16) {
            if (row >= 0) {
                copy16(ks + r * LD + c, k + c);
                copy16(ks + (KEYS + r) * LD + c, v + c);
            } else {
                *reinterpret_cast<float4*>(ks + r * LD + c) = make_float4(0.f, 0.f, 0.f, 0.f);
                *reinterpret_cast<float4*>(ks + (KEYS + r) * LD + c) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        return row;
    };
    int pos[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        const int r = ty + 16 * x;
        pos[x] = r < rows_used ? pos_first + r / group : -1;           // an idle row sees nothing
    }
    float acc[4][D / 8], running_max[4], running_sum[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        running_max[x] = -INFINITY;
        running_sum[x] = 0.f;
#pragma unroll
        for (int c = 0; c < D / 8; ++c) acc[x][c] = 0.f;
    }
    __shared__ unsigned present[2][THREADS / 32];      // which of a chunk's keys have a page: a bit a key, eight keys a warp
    auto note = [&](int row, int buffer) {
        const unsigned lanes = __ballot_sync(0xffffffffu, row >= 0);
        if (lane == 0) {
            unsigned keys = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) keys |= ((lanes >> (4 * i)) & 1u) << i;
            present[buffer][tid >> 5] = keys;
        }
    };
    note(fetch(0, 0), 0);
    int chunk = 0;
    for (int base = 0; base < key_end; base += KEYS, ++chunk) {
        const int buffer = chunk & 1;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                               // this chunk is there (at first: the queries too), the one before is used up
        if (base + KEYS < key_end) note(fetch(base + KEYS, buffer ^ 1), buffer ^ 1);
        const float* ks = kv + buffer * 2 * KEYS * LD;
        const float* vs = ks + KEYS * LD;
        float s[4][4];
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[x][j] = 0.f;
#pragma unroll 4
        for (int i = 0; i < D; i += 4) {
            float4 a[4], b[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) a[x] = *reinterpret_cast<const float4*>(qs + (ty + 16 * x) * LD + i);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(ks + (tx + 8 * j) * LD + i);
#define LIA_SCORE(E)                                                                                     \
    _Pragma("unroll") for (int x = 0; x < 4; ++x) _Pragma("unroll") for (int j = 0; j < 4; ++j) s[x][j] = \
        fmaf(a[x].E, b[j].E, s[x][j]);
            LIA_SCORE(x) LIA_SCORE(y) LIA_SCORE(z) LIA_SCORE(w)
#undef LIA_SCORE
        }
        const bool masked = base + KEYS - 1 > pos_first;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            bool seen[4];
            float top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                seen[j] = base + tx + 8 * j <= pos[x] && ((present[buffer][j] >> tx) & 1u);
                s[x][j] = seen[j] ? s[x][j] * scale : -INFINITY;
                top = fmaxf(top, s[x][j]);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float new_max = fmaxf(running_max[x], top);
            const bool none = new_max == -INFINITY;     // the row has seen no key yet: nothing to add
            const float correction = none ? 1.f : expf(running_max[x] - new_max);
            float p[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) p[j] = seen[j] ? expf(s[x][j] - new_max) : 0.f;
            float sum = (p[0] + p[2]) + (p[1] + p[3]);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            running_sum[x] = running_sum[x] * correction + sum;
            running_max[x] = new_max;
#pragma unroll
            for (int c = 0; c < D / 8; ++c) acc[x][c] *= correction;
#pragma unroll
            for (int j = 0; j < 4; ++j) ps[(ty + 16 * x) * LP + tx + 8 * j] = p[j];
        }
        __syncwarp();
        // (a row's own later keys carry no weight, but their values may be anything: they are left out, not multiplied by zero)
        auto outputs = [&](auto with_mask) {
#pragma unroll 2
            for (int j = 0; j < KEYS; j += 4) {
                float4 w[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) w[x] = *reinterpret_cast<const float4*>(ps + (ty + 16 * x) * LP + j);
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    float4 b[GROUPS];
#pragma unroll
                    for (int c = 0; c < GROUPS; ++c) b[c] = *reinterpret_cast<const float4*>(vs + (j + jj) * LD + 32 * c + 4 * tx);
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        if (decltype(with_mask)::value && base + j + jj > pos[x]) continue;
                        const float p = jj == 0 ? w[x].x : jj == 1 ? w[x].y : jj == 2 ? w[x].z : w[x].w;
#pragma unroll
                        for (int c = 0; c < GROUPS; ++c) {
                            acc[x][4 * c] = fmaf(p, b[c].x, acc[x][4 * c]);
                            acc[x][4 * c + 1] = fmaf(p, b[c].y, acc[x][4 * c + 1]);
                            acc[x][4 * c + 2] = fmaf(p, b[c].z, acc[x][4 * c + 2]);
                            acc[x][4 * c + 3] = fmaf(p, b[c].w, acc[x][4 * c + 3]);
                        }
                    }
                }
            }
        };
        if (masked) outputs(std::true_type{});
        else outputs(std::false_type{});
        __syncwarp();
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        const int r = ty + 16 * x, tok = r / group;
        if (r >= rows_used) continue;
        float* dst = out + ((size_t)(offset + tok0 + tok) * nq + kvh * group + (r - tok * group)) * D;
        const float inv = 1.0f / running_sum[x];
#pragma unroll
        for (int c = 0; c < GROUPS; ++c)
            *reinterpret_cast<float4*>(dst + 32 * c + 4 * tx) = make_float4(acc[x][4 * c] * inv, acc[x][4 * c + 1] * inv,
                                                                            acc[x][4 * c + 2] * inv, acc[x][4 * c + 3] * inv);
    }
}

template <int D>
int launch_f32(const float* q, const float* k_pages, const float* v_pages, const int* segments, int n_segments, int n_tiles,
               const int* slots, const int* block_table, int table_stride, float* out, int nq, int nkv, int page_size,
               int tokens_per_tile, float scale, int num_pages, int* error_flag, cudaStream_t stream) {
    constexpr size_t smem = ((size_t)(ROWS + 4 * KEYS) * (D + 4) + ROWS * (KEYS + 4)) * sizeof(float);
    static std::atomic<bool> configured{false};
    if (!configured.load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(attention_prefill_f32_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            return LIA_ERR_LAUNCH;
        }
        configured.store(true, std::memory_order_release);
    }
    int page_shift = -1;
    for (int b = 0; b < 31; ++b)
        if (page_size == (1 << b)) page_shift = b;
    return lia_launch(attention_prefill_f32_kernel<D>, dim3((unsigned)n_tiles * nkv), dim3(THREADS), smem, stream, q, k_pages, v_pages,
                      segments, n_segments, slots, block_table, table_stride, out, nq, nkv, page_size, page_shift, tokens_per_tile,
                      scale, num_pages, error_flag);
}
}  // namespace

// Tokens of a portion that one CTA takes for `group` query heads per kv head of size d (0: the kernel does not take them).
LIA_EXPORT int lia_attention_prefill_f32_tokens_per_tile(int group, int d) {
    if (d != 32 && d != 64 && d != 96 && d != 128) return 0;
    return group >= 1 && group <= ROWS ? ROWS / group : 0;
}

// q, out [tokens, nq, d]; k_pages, v_pages [num_pages, page_size, nkv, d], all 32-bit; segments [n_segments][3]: first token's
// batch index, its position, count; n_tiles = sum over portions of ceil(count / tokens_per_tile).  All keys are visible.
LIA_EXPORT int lia_attention_prefill_f32(const void* q, const void* k_pages, const void* v_pages, const int* segments, int n_segments,
                                         int n_tiles, const int* slots, const int* block_table, int table_stride, void* out, int nq,
                                         int nkv, int d, int page_size, float scale, int num_pages, int* error_flag,
                                         cudaStream_t stream) {
    if (n_segments <= 0 || n_tiles <= 0) return LIA_OK;
    if (nq <= 0 || nkv <= 0 || nq % nkv || page_size <= 0 || (long long)n_tiles * nkv > 2147483647LL) return LIA_ERR_SIZE;
    const int per_tile = lia_attention_prefill_f32_tokens_per_tile(nq / nkv, d);
    if (per_tile == 0) return LIA_ERR_SIZE;
    if (((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)out) & 15u) return LIA_ERR_ALIGN;
#define LIA_F32_CASE(D)                                                                                                          \
    case D: return launch_f32<D>((const float*)q, (const float*)k_pages, (const float*)v_pages, segments, n_segments, n_tiles, slots, \
                                 block_table, table_stride, (float*)out, nq, nkv, page_size, per_tile, scale, num_pages, error_flag, stream)
    switch (d) {
        LIA_F32_CASE(32);
        LIA_F32_CASE(64);
        LIA_F32_CASE(96);
        LIA_F32_CASE(128);
    }
#undef LIA_F32_CASE
    return LIA_ERR_SIZE;
}
