// Matrix product on the 32-bit pipes, for every size and element type:
//     acc[m, n] = sum_k A[m, k] * W[n, k]        (W is [out, in] row-major, as in the checkpoint)
// It is the product of the true 32-bit path (plain FMA, no tensor-core mode that would round the
// operands) and the fallback of the bfloat16 path for shapes the tcgen05 kernel refuses.
// The sum over k runs in ascending order for each output element, whatever M and N are, so a
// row's result does not depend on which other rows are in the batch.
//
// Epilogues:
//   STORE   out[m, n]  = alpha * acc
//   ACCUM   out[m, n] += alpha * acc                       (32-bit out: the residual stream)
//   SWIGLU  out[m, n]  = up * gate / (1 + exp(-gate)),  gate = acc over W rows [0, N),
//                                                        up   = acc over W rows [N, 2N)
#include <type_traits>

#include "common.cuh"

#define GEMM_STORE 0
#define GEMM_ACCUM 1
#define GEMM_SWIGLU 2

namespace {
constexpr int BM = 64, BN = 64, BK = 16;

template <typename TA, typename TW, typename TO, int MODE>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, int ldw,
                 TO* __restrict__ out, int ldo, int M, int N, int K, float alpha, long long a_batch,
                 long long w_batch, long long out_batch, int act) {
    constexpr int NW = (MODE == GEMM_SWIGLU) ? 2 : 1;
    A += (size_t)blockIdx.z * a_batch;                      // one product per blockIdx.z (a single one: all zero)
    W += (size_t)blockIdx.z * w_batch;
    out += (size_t)blockIdx.z * out_batch;
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[NW][BK][BN + 4];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[NW][4][4];
#pragma unroll
    for (int w = 0; w < NW; ++w)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[w][i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int e = tid; e < BM * BK; e += 256) {
            const int r = e / BK, k = e % BK;
            const int gm = m0 + r, gk = k0 + k;
            As[k][r] = (gm < M && gk < K) ? to_float(A[(size_t)gm * lda + gk]) : 0.f;
        }
#pragma unroll
        for (int w = 0; w < NW; ++w)
#pragma unroll
            for (int e = tid; e < BN * BK; e += 256) {
                const int r = e / BK, k = e % BK;
                const int gn = n0 + r, gk = k0 + k;
                Ws[w][k][r] = (gn < N && gk < K) ? to_float(W[((size_t)w * N + gn) * ldw + gk]) : 0.f;
            }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                float b[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = Ws[w][k][tx * 4 + j];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[w][i][j] = fmaf(a[i], b[j], acc[w][i][j]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= N) continue;
            TO* dst = out + (size_t)gm * ldo + gn;
            if (MODE == GEMM_STORE) {
                *dst = from_float<TO>(alpha * acc[0][i][j]);
            } else if (MODE == GEMM_ACCUM) {
                *dst = from_float<TO>(to_float(*dst) + alpha * acc[0][i][j]);
            } else {
                const float gate = acc[0][i][j], up = acc[NW - 1][i][j];
                *dst = from_float<TO>(up * (act == 4 ? fmaxf(gate, 0.f) : gate / (1.0f + expf(-gate))));       // act 4: a ReLU gate
            }
        }
    }
}

// ---- the same product of 32-bit operands in larger tiles ----
// BM x BN outputs a CTA (two of them side by side for the gated form), TM x TN a thread, K in steps of 16 or 32 through a ring of
// four shared-memory stages that 16-byte asynchronous copies fill three steps ahead: a step of a small tile is far shorter than a
// trip to L2.  Rows lie in shared memory as they do in memory, a step's elements and a pad of 4 (eight neighbouring rows' pieces fall into
// different banks); a thread's rows and columns lie BM / TM and BN / TN apart, so that a warp's 16-byte loads meet no bank twice
// and its stores are neighbours.  Each output is still one chain of multiply-adds over ascending k from zero: the results are
// those of the kernel above, bit for bit.  What bounds it is the issue of the multiply-adds.
template <int BM_, int BN_, int TM_, int TN_, int MODE>
struct Tile {
    static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, NW = MODE == GEMM_SWIGLU ? 2 : 1;
    static constexpr int THREADS = (BM / TM) * (BN / TN);
    static constexpr int ROWS = BM + NW * BN;                                   // rows of a stage: of A, then of W
    static constexpr int BK = ROWS <= 80 ? 32 : 16, LD = BK + 4, PIECES = BK / 4;
    static constexpr int LOADS = ROWS * PIECES / THREADS;                       // 16-byte copies a thread and step
    static constexpr int STAGES = 4;
    static constexpr size_t SMEM = (size_t)STAGES * ROWS * LD * sizeof(float);
    static_assert(ROWS * PIECES % THREADS == 0 && THREADS % PIECES == 0, "whole copies a thread");
    static_assert((BN / TN) % 8 == 0 && (BM / TM) % 4 == 0, "warps of eight by four threads");
};

template <int BM, int BN, int TM, int TN, int MODE>
__global__ void __launch_bounds__(Tile<BM, BN, TM, TN, MODE>::THREADS)
gemm_simt_tiled_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ out, int ldo,
                       int M, int N, int K, float alpha, long long a_batch, long long w_batch, long long out_batch, int act) {
    using T = Tile<BM, BN, TM, TN, MODE>;
    constexpr int NW = T::NW, THREADS = T::THREADS, BK = T::BK, LD = T::LD, ROWS = T::ROWS, STAGES = T::STAGES;
    constexpr int GX = BN / TN, GY = BM / TM;
    extern __shared__ __align__(16) float tile_shared[];                        // [STAGES][ROWS][LD]
    // a warp is eight threads across and four down: a warp's loads name the fewest different pieces of shared memory
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (warp % (GX / 8)) * 8 + (lane & 7), ty = (warp / (GX / 8)) * 4 + (lane >> 3);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    pdl_launch_dependents();
    pdl_wait();
    A += (size_t)blockIdx.z * a_batch;
    W += (size_t)blockIdx.z * w_batch;
    out += (size_t)blockIdx.z * out_batch;
    // this thread's copies: which row of the stage, and where that row begins in memory (beyond the product's rows: zeros)
    const float* source[T::LOADS];
    uint32_t target[T::LOADS], there[T::LOADS];
    const int piece = (tid % T::PIECES) * 4;
#pragma unroll
    for (int i = 0; i < T::LOADS; ++i) {
        const int r = (tid + i * THREADS) / T::PIECES;
        const float* row;
        bool valid;
        if (r < BM) {
            valid = m0 + r < M;
            row = A + (size_t)(valid ? m0 + r : 0) * lda;
        } else {
            const int half = (r - BM) / BN, n = n0 + (r - BM) - half * BN;
            valid = n < N;
            row = W + (valid ? (size_t)half * N + n : 0) * ldw;
        }
        source[i] = row + piece;
        there[i] = valid ? 16u : 0u;
        target[i] = (uint32_t)__cvta_generic_to_shared(tile_shared + r * LD + piece);
    }
    const int steps = (K + BK - 1) / BK;
    auto fetch = [&](int step) {
        const int k = step * BK;
        if (step < steps) {
            const uint32_t at = (uint32_t)(step % STAGES) * (ROWS * LD * 4u);
            const bool inside = k + piece < K;                                  // (K is a multiple of four)
#pragma unroll
            for (int i = 0; i < T::LOADS; ++i)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(target[i] + at),
                             "l"(source[i] + (inside ? k : 0)), "r"(inside ? there[i] : 0u) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[NW][TM][TN];
#pragma unroll
    for (int w = 0; w < NW; ++w)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[w][i][j] = 0.f;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                                        // the step is there, and the one before is used up
        fetch(s + STAGES - 1);
        const float* stage = tile_shared + (s % STAGES) * (ROWS * LD);
        const float* as = stage + ty * LD;
        const float* ws = stage + (BM + tx) * LD;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * GY * LD + k);
#pragma unroll
            for (int w = 0; w < NW; ++w)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float4 b = *reinterpret_cast<const float4*>(ws + (w * BN + j * GX) * LD + k);
                    // (element after element over all rows: a sum's next addition comes TM instructions behind its last one)
#pragma unroll
                    for (int i = 0; i < TM; ++i) acc[w][i][j] = fmaf(a[i].x, b.x, acc[w][i][j]);
#pragma unroll
                    for (int i = 0; i < TM; ++i) acc[w][i][j] = fmaf(a[i].y, b.y, acc[w][i][j]);
#pragma unroll
                    for (int i = 0; i < TM; ++i) acc[w][i][j] = fmaf(a[i].z, b.z, acc[w][i][j]);
#pragma unroll
                    for (int i = 0; i < TM; ++i) acc[w][i][j] = fmaf(a[i].w, b.w, acc[w][i][j]);
                }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty + i * GY;
        if (gm >= M) continue;
        float* row = out + (size_t)gm * ldo;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx + j * GX;
            if (gn >= N) continue;
            const float x = acc[0][i][j];
            if (MODE == GEMM_STORE) row[gn] = alpha * x;
            else if (MODE == GEMM_ACCUM) row[gn] = row[gn] + alpha * x;
            else row[gn] = acc[NW - 1][i][j] * (act == 4 ? fmaxf(x, 0.f) : x / (1.0f + expf(-x)));
        }
    }
}

template <int BM, int BN, int TM, int TN, int MODE>
int launch_tile(const float* A, int lda, const float* W, int ldw, float* out, int ldo, int M, int N, int K, float alpha,
                cudaStream_t stream, int batch, long long a_batch, long long w_batch, long long out_batch, int act) {
    using T = Tile<BM, BN, TM, TN, MODE>;
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
    if (grid.y > 65535 || batch < 1 || batch > 65535) return LIA_ERR_SIZE;
    if (T::SMEM > 48 * 1024) {
        static std::atomic<bool> configured{false};
        if (!configured.load(std::memory_order_acquire)) {
            if (cudaFuncSetAttribute(gemm_simt_tiled_kernel<BM, BN, TM, TN, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)T::SMEM) != cudaSuccess) {
                cudaGetLastError();
                return LIA_ERR_LAUNCH;
            }
            configured.store(true, std::memory_order_release);
        }
    }
    return lia_launch(gemm_simt_tiled_kernel<BM, BN, TM, TN, MODE>, grid, dim3(T::THREADS), T::SMEM, stream, A, lda, W, ldw, out, ldo, M,
                      N, K, alpha, a_batch, w_batch, out_batch, act);
}

int sm_count_of_device() {
    static std::atomic<int> known{0};
    int count = known.load(std::memory_order_relaxed);
    if (count == 0) {
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess ||
            cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || count <= 0) {
            cudaGetLastError();
            return 148;
        }
        known.store(count, std::memory_order_relaxed);
    }
    return count;
}

// Which tile.  Measured on a B200 (us; K 1,024).  A CTA's chain over K is the product's time while there are few of them: 8 x 1,280
// outputs take 12.5 in tiles of 8 x 16, 18.6 in 16 x 32 and 24.7 in 16 x 64; 100 x 1,024: 17.4, 20.6 and 24.7.  Larger tiles load
// less from shared memory per multiply-add: 450 x 1,280: 65.8 in 8 x 16, 41.1 in 16 x 32, 53 in 32 x 32; 600 x 1,024: 69.8, 59.5 and 53.4
// (the kernel above: 107); 600 x 32,000: 1,129 in 16 x 32, 1,058 in 32 x 32, 983 in 32 x 64 (40 TFLOP/s, 54% of the pipes).  So by how many
// tiles of a shape an SM would get; at most 16 rows keep 16 x 32 however many columns (8 x 32,000: 46.9 against 69.5 in 32 x 64).  The
// gated form, 4,096 pairs: 264 at 600 rows in 64 x 32 pairs (32 x 32: 273; the kernel above: 511), 41.1 at 48 rows in 16 x 32 pairs (47.3);
// 100 rows 84 in 32 x 32 pairs, 91 in 16 x 32, 98 in 64 x 32 (two CTAs on some SMs, none on others; the kernel above: 85), 8,192 pairs 121,
// 162 and the kernel above 134.
template <int MODE>
int launch_tiled(const float* A, int lda, const float* W, int ldw, float* out, int ldo, int M, int N, int K, float alpha,
                 cudaStream_t stream, int batch, long long a_batch, long long w_batch, long long out_batch, int act) {
#define LIA_TILE(BM, BN, TM, TN)                                                                                       \
    return launch_tile<BM, BN, TM, TN, MODE>(A, lda, W, ldw, out, ldo, M, N, K, alpha, stream, batch, a_batch, w_batch, out_batch, act)
    if constexpr (MODE == GEMM_SWIGLU) {
        if (M <= 64) LIA_TILE(16, 32, 2, 4);
        if (M <= 128) LIA_TILE(32, 32, 4, 4);
        LIA_TILE(64, 32, 4, 4);
    } else {
        const long long sms = sm_count_of_device();
        auto tiles = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn) * batch; };
        if (tiles(8, 16) <= 10 * sms) LIA_TILE(8, 16, 2, 2);
        if (tiles(16, 32) <= 8 * sms || M <= 16) LIA_TILE(16, 32, 4, 4);
        if (tiles(32, 64) <= 4 * sms) LIA_TILE(32, 32, 4, 4);
        LIA_TILE(32, 64, 4, 4);
    }
#undef LIA_TILE
}

template <typename TA, typename TW, typename TO>
int launch_modes(int mode, const void* A, int lda, const void* W, int ldw, void* out, int ldo, int M,
                 int N, int K, float alpha, cudaStream_t stream, int batch = 1, long long a_batch = 0,
                 long long w_batch = 0, long long out_batch = 0, int act = 0) {
    // 32-bit operands whose rows can be read 16 bytes at a time (and no more of them than the smallest tiles' grid holds)
    if constexpr (std::is_same<TA, float>::value) {
        if (K % 4 == 0 && M <= 65535 * 8 && lda % 4 == 0 && ldw % 4 == 0 && a_batch % 4 == 0 && w_batch % 4 == 0 &&
            (((uintptr_t)A | (uintptr_t)W) & 15u) == 0) {
#define LIA_TILED(MODE)                                                                                                       \
    return launch_tiled<MODE>((const float*)A, lda, (const float*)W, ldw, (float*)out, ldo, M, N, K, alpha, stream, batch, a_batch, w_batch, \
                              out_batch, act)
            if (mode == GEMM_STORE) LIA_TILED(GEMM_STORE);
            if (mode == GEMM_ACCUM) LIA_TILED(GEMM_ACCUM);
            if (mode == GEMM_SWIGLU) LIA_TILED(GEMM_SWIGLU);
            return LIA_ERR_SIZE;
#undef LIA_TILED
        }
    }
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
    if (grid.y > 65535 || batch < 1 || batch > 65535) return LIA_ERR_SIZE;
#define LIA_GEMM(MODE)                                                                          \
    gemm_simt_kernel<TA, TW, TO, MODE><<<grid, 256, 0, stream>>>((const TA*)A, lda, (const TW*)W, \
                                                                 ldw, (TO*)out, ldo, M, N, K, alpha, \
                                                                 a_batch, w_batch, out_batch, act)
    if (mode == GEMM_STORE) LIA_GEMM(GEMM_STORE);
    else if (mode == GEMM_ACCUM) LIA_GEMM(GEMM_ACCUM);
    else if (mode == GEMM_SWIGLU) LIA_GEMM(GEMM_SWIGLU);
    else return LIA_ERR_SIZE;
#undef LIA_GEMM
    return lia_check_launch();
}
}  // namespace

// A [M, K] (a_dtype), W [N, K] or, for SWIGLU, [2N, K] (w_dtype), out [M, N] (out_dtype).
// ACCUM needs a 32-bit out.  Supported element types: (f32, f32 -> f32) and
// (bf16, bf16 -> f32 | bf16).
LIA_EXPORT int lia_gemm_simt(int mode, const void* A, int a_dtype, int lda, const void* W, int w_dtype,
                             int ldw, void* out, int out_dtype, int ldo, int M, int N, int K,
                             float alpha, cudaStream_t stream) {
    const int act = mode >> 8;           // SWIGLU: 4 above the mode's byte makes the gate a ReLU
    mode &= 0xff;
    if (act != 0 && !(mode == GEMM_SWIGLU && act == 4)) return LIA_ERR_SIZE;
    if (M <= 0 || N <= 0) return LIA_OK;
    if (K <= 0 || lda < K || ldw < K || ldo < N) return LIA_ERR_SIZE;
    if (mode == GEMM_ACCUM && out_dtype != LIA_F32) return LIA_ERR_DTYPE;
    if (a_dtype == LIA_F32 && w_dtype == LIA_F32 && out_dtype == LIA_F32)
        return launch_modes<float, float, float>(mode, A, lda, W, ldw, out, ldo, M, N, K, alpha, stream, 1, 0, 0, 0, act);
    if (a_dtype == LIA_BF16 && w_dtype == LIA_BF16 && out_dtype == LIA_F32)
        return launch_modes<__nv_bfloat16, __nv_bfloat16, float>(mode, A, lda, W, ldw, out, ldo, M, N, K,
                                                                 alpha, stream, 1, 0, 0, 0, act);
    if (a_dtype == LIA_BF16 && w_dtype == LIA_BF16 && out_dtype == LIA_BF16)
        return launch_modes<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(mode, A, lda, W, ldw, out, ldo, M,
                                                                         N, K, alpha, stream, 1, 0, 0, 0, act);
    return LIA_ERR_DTYPE;
}

// `batch` products of one shape in one launch: product b reads A + b a_batch, W + b w_batch and writes out + b out_batch
// (strides in elements).  The products of the heads of an attention whose keys and values are expanded from a shared
// latent are of this kind: every head has a matrix of its own and rows of its own.
LIA_EXPORT int lia_gemm_simt_batched(int mode, const void* A, int a_dtype, int lda, long long a_batch, const void* W,
                                     int w_dtype, int ldw, long long w_batch, void* out, int out_dtype, int ldo,
                                     long long out_batch, int batch, int M, int N, int K, float alpha,
                                     cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return LIA_OK;
    if (K <= 0 || lda < K || ldw < K || ldo < N || mode == GEMM_SWIGLU) return LIA_ERR_SIZE;
    if (mode == GEMM_ACCUM && out_dtype != LIA_F32) return LIA_ERR_DTYPE;
    if (a_dtype == LIA_F32 && w_dtype == LIA_F32 && out_dtype == LIA_F32)
        return launch_modes<float, float, float>(mode, A, lda, W, ldw, out, ldo, M, N, K, alpha, stream, batch, a_batch,
                                                 w_batch, out_batch);
    if (a_dtype == LIA_BF16 && w_dtype == LIA_BF16 && out_dtype == LIA_F32)
        return launch_modes<__nv_bfloat16, __nv_bfloat16, float>(mode, A, lda, W, ldw, out, ldo, M, N, K, alpha, stream,
                                                                 batch, a_batch, w_batch, out_batch);
    if (a_dtype == LIA_BF16 && w_dtype == LIA_BF16 && out_dtype == LIA_BF16)
        return launch_modes<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(mode, A, lda, W, ldw, out, ldo, M, N, K, alpha,
                                                                         stream, batch, a_batch, w_batch, out_batch);
    return LIA_ERR_DTYPE;
}
