// Matrix product for many tokens on PAIRS of SMs (tcgen05 with cta_group::2):
//     acc[t, f] = sum_k X[t, k] * W[f, k]       X [M, K] bf16 activations, W [N, K] bf16 weights
//
// Two CTAs of a cluster share a tile of 256 tokens by up to 256 weight rows.  The tokens are the MMA's M dimension, 128 of
// them each CTA's own; the weight rows are its N dimension, half of them brought by each CTA.  One tcgen05.mma of the first
// CTA multiplies the whole tile, reading the operands from both CTAs' shared memory and leaving each CTA's 128 tokens in that
// CTA's TMEM.  A K block of 64 costs a CTA 16 KB of X and up to 16 KB of W for 4.2 MFLOP: two thirds of what one CTA alone
// brings for a 128 x 256 tile, and the MMAs read two thirds of the bytes from shared memory, whose 128 bytes a cycle
// bound the one-CTA kernel's main loop (csrc/gemm_tc.cu).
//
// The gated product (SWIGLU, REGLU) takes its tile's rows of W half from the gate and half from the up matrix (the first CTA brings
// the gate's rows, the second the up's): gate and up of a feature then lie in the same TMEM lane, n / 2 columns apart, and
// the accumulator still has two buffers.
//
// The kernel is persistent: one pair per two SMs walks the tiles round-robin.  Roles:
//   warp 0      one lane issues the TMA loads into a ring of 128-byte-swizzled stages (both CTAs; what they bring is
//               counted on the FIRST CTA's barriers: .cta_group::2, the barrier's address with the CTA bit cleared);
//   warp 1      allocates TMEM; in the first CTA one lane issues the MMAs into one of two accumulator buffers.  "Stage free" and
//               "accumulator complete" reach both CTAs by tcgen05.commit with a multicast mask;
//   warps 2..9  the epilogue: a warp reads 32 tokens (TMEM lanes) by 32 features at a time, turns them into the output's
//               type in a swizzled piece of shared memory of its own and sends it off by TMA (a store, or a reduce-add for ACCUM):
//               no warp waits for another.  "Accumulator drained" is counted in the first CTA from the warps of both.
// Tiles are narrower than 256 rows of W (a multiple of 32; of 64 for the gated product) where that leaves the pairs less idle in
// the last round: see plan_width.
//
// Programmatic dependent launch: the first ring of W boxes is asked for before the kernel ahead has finished; X waits.
// Every wait on an mbarrier is bounded; a role that gives up raises the error flag and leaves its loop, and all threads of both
// CTAs still meet at the cluster barrier before TMEM is freed.
#include <algorithm>

#include "gemm_pair.cuh"
#include "tcgen05.cuh"

using namespace tc5;

namespace {
constexpr int THREADS = 320;
constexpr int EPILOGUE_WARPS = 8;                // per CTA: two for each quarter of the TMEM lanes
constexpr int MAX_STAGES = 8;
constexpr int SMEM_BYTES = 226 * 1024;           // dynamic shared memory asked for (a CTA may have 227 KB; the rest is static)
constexpr int PAIR_M = 256, HALF_M = 128;        // tokens per tile, and per CTA
constexpr int CHUNK_F = 32;                      // features of an epilogue piece
constexpr int RASTER = 8;                        // token tiles that neighbouring pairs share the rows of W of
constexpr uint32_t PEER_BIT_MASK = 0xFEFFFFFFu;  // clears the bit of a shared::cluster address that tells the pair's CTAs apart

struct Shape {
    int M, N;
    int n_tile;               // rows of W per tile (gated: gate and up rows together)
    int width;                // output features per tile: n_tile, or half of it for the gated product
    int stages, kblocks, f_tiles, t_tiles;
    int tmem_cols;
    float alpha;
    float act_p, act_n;       // xIELU's two constants
    int* error_flag;
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// TMA load of one box whose completion is counted on the FIRST CTA's barrier, whichever CTA issues it.
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar & PEER_BIT_MASK), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive, when the MMAs issued so far are done, on the barrier at this offset in BOTH CTAs of the pair.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
    const uint16_t mask = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"(mask) : "memory");
}
// Arrive on the barrier at this offset in the FIRST CTA's shared memory.
__device__ __forceinline__ void arrive_on_first(uint32_t bar) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(bar), "r"(0));
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}

// The index-th tile: RASTER token tiles walk the rows of W together, so that what runs at the same time shares both operands in L2.
struct Unit {
    int t0, f0;               // first token, first output feature
};
__device__ __forceinline__ Unit unit_at(const Shape& s, int index) {
    const int band = index / (RASTER * s.f_tiles), t_first = band * RASTER;
    const int across = min(RASTER, s.t_tiles - t_first), rest = index - band * RASTER * s.f_tiles;
    Unit u;
    u.t0 = (t_first + rest % across) * PAIR_M;
    u.f0 = (rest / across) * s.width;
    return u;
}

template <int MODE>
__device__ __forceinline__ float finish(float acc, float up, const Shape& s) {
    if (MODE == GEMM_SWIGLU) return up * __fdividef(acc, 1.0f + __expf(-acc));
    if (MODE == GEMM_REGLU) return up * fmaxf(acc, 0.f);
    if (MODE == GEMM_STORE_RELU2) {
        const float r = fmaxf(s.alpha * acc, 0.f);
        return r * r;
    }
    if (MODE == GEMM_STORE_XIELU) return lia_xielu_fast(s.alpha * acc, s.act_p, s.act_n);
    return s.alpha * acc;
}

// A lane's 32 features of its token into the warp's piece of shared memory, 16 bytes at a time, swizzled as the output's tensor map
// says (rows of 128 bytes: the 16-byte chunk's number xor the row's low three bits; of 64: xor bits 1 and 2): eight lanes' stores meet 32 banks.
__device__ __forceinline__ void put_row(uint8_t* piece, int lane, const float (&v)[32], float*) {
    uint8_t* row = piece + lane * 128;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        *reinterpret_cast<float4*>(row + ((j ^ (lane & 7)) * 16)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
}
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void put_row(uint8_t* piece, int lane, const float (&v)[32], __nv_bfloat16*) {
    uint8_t* row = piece + lane * 64;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        *reinterpret_cast<uint4*>(row + ((j ^ ((lane >> 1) & 3)) * 16)) =
            make_uint4(pack_pair(v[8 * j], v[8 * j + 1]), pack_pair(v[8 * j + 2], v[8 * j + 3]), pack_pair(v[8 * j + 4], v[8 * j + 5]),
                       pack_pair(v[8 * j + 6], v[8 * j + 7]));
}

template <int MODE, typename TO>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                 const __grid_constant__ CUtensorMap map_o, Shape s) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_slot;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const bool leader = elect_one();
    const uint32_t rank = cluster_rank();
    const int half_n = s.n_tile / 2;                                   // rows of W that a CTA brings
    constexpr uint32_t A_BYTES = HALF_M * BLOCK_K * 2;
    const uint32_t stage_bytes = A_BYTES + (uint32_t)half_n * BLOCK_K * 2;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t staging_base = smem_base + (uint32_t)s.stages * stage_bytes;      // a piece of [32 tokens][32 features] a warp
    const int units = s.f_tiles * s.t_tiles;
    const int first_unit = blockIdx.x >> 1, stride = gridDim.x >> 1;

    if (warp == 0 && lane == 0) {
        for (int i = 0; i < s.stages; ++i) {
            mbar_init(smem_u32(&full_bar[i]), 1);          // the first CTA's producer; the bytes of both CTAs
            mbar_init(smem_u32(&empty_bar[i]), 1);         // one multicast commit
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&acc_full[i]), 1);          // one multicast commit
            mbar_init(smem_u32(&acc_empty[i]), 2 * EPILOGUE_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_o) : "memory");
    }
    if (warp == 1) {
        // both CTAs of the pair allocate, with the same destination offset
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                     "r"((uint32_t)s.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                    // the partner's barriers exist before anything of ours reaches them
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    pdl_launch_dependents();

    if (warp == 0 && leader) {
        // ---- TMA producer (both CTAs): this CTA's 128 tokens, its half of the tile's rows of W ----
        // gated: the first CTA brings gate rows, the second up rows of the same features
        const int w_first = GEMM_GATED(MODE) ? (rank == 0 ? 0 : s.N) : (int)rank * half_n;
        bool ok = true;
        int ahead = 0;
        {   // the first ring of W boxes goes out before the kernel ahead has finished: weights depend on nothing
            int it = 0;
            for (int index = first_unit; index < units && it < s.stages; index += stride) {
                const Unit u = unit_at(s, index);
                for (int kb = 0; kb < s.kblocks && it < s.stages; ++kb, ++it) {
                    const uint32_t full = smem_u32(&full_bar[it]);
                    if (rank == 0) mbar_expect_tx(full, 2 * stage_bytes);
                    tma_load_pair(smem_base + (uint32_t)it * stage_bytes + A_BYTES, &map_w, kb * BLOCK_K, w_first + u.f0, full);
                }
            }
            ahead = it;
        }
        pdl_wait();
        int it = 0, st = 0;
        uint32_t phase = 0;
        for (int index = first_unit; index < units && ok; index += stride) {
            const Unit u = unit_at(s, index);
            const int t_mine = u.t0 + (int)rank * HALF_M, w_mine = w_first + u.f0;
            for (int kb = 0; kb < s.kblocks; ++kb, ++it) {
                const uint32_t full = smem_u32(&full_bar[st]);
                const uint32_t dst = smem_base + (uint32_t)st * stage_bytes;
                if (it >= ahead) {
                    if (!mbar_wait(smem_u32(&empty_bar[st]), phase ^ 1u)) { ok = false; break; }
                    if (rank == 0) mbar_expect_tx(full, 2 * stage_bytes);
                    tma_load_pair(dst + A_BYTES, &map_w, kb * BLOCK_K, w_mine, full);
                }
                tma_load_pair(dst, &map_x, kb * BLOCK_K, t_mine, full);
                if (++st == s.stages) { st = 0; phase ^= 1u; }
            }
        }
        if (!ok) {
            if (s.error_flag) atomicExch(s.error_flag, 3);
            // copies of this CTA may still be in flight (they complete on the first CTA's barriers, which the second
            // CTA cannot poll): give them a bounded time to land before the CTA goes on to leave
            for (int i = 0; i < 64; ++i) __nanosleep(1000);
        }
    } else if (warp == 1 && leader && rank == 0) {
        // ---- MMA issuer (first CTA only): 256 tokens x n_tile rows per instruction ----
        const uint32_t idesc = instr_desc(PAIR_M, s.n_tile);
        bool ok = true;
        int n_unit = 0, st = 0;
        uint32_t phase = 0;
        const uint64_t desc_a0 = smem_desc(smem_base), desc_b0 = smem_desc(smem_base + A_BYTES), stage_step = stage_bytes >> 4;
        uint64_t stage_offset = 0;
        for (int index = first_unit; index < units && ok; index += stride, ++n_unit) {
            const int buf = n_unit & 1;
            if (!mbar_wait(smem_u32(&acc_empty[buf]), (((uint32_t)n_unit >> 1) & 1u) ^ 1u)) { ok = false; break; }
            tc_fence_after();
            const uint32_t acc = tmem_base + (uint32_t)(buf * s.n_tile);
            for (int kb = 0; kb < s.kblocks; ++kb) {
                if (!mbar_wait(smem_u32(&full_bar[st]), phase)) { ok = false; break; }
                tc_fence_after();
                const uint64_t da = desc_a0 + stage_offset, db = desc_b0 + stage_offset;
                const uint32_t first = kb > 0 ? 1u : 0u;
#pragma unroll
                for (int k = 0; k < BLOCK_K / 16; ++k) mma_pair(acc, da + 2 * k, db + 2 * k, idesc, k > 0 ? 1u : first);
                commit_pair(smem_u32(&empty_bar[st]));        // the stage is free in both CTAs when these MMAs have read it
                if (++st == s.stages) { st = 0; stage_offset = 0; phase ^= 1u; }
                else stage_offset += stage_step;
            }
            if (ok) commit_pair(smem_u32(&acc_full[buf]));    // the accumulator is complete, in both CTAs
        }
        if (!ok && s.error_flag) atomicExch(s.error_flag, 3);
    } else if (warp >= 2) {
        // ---- epilogue (both CTAs): warp w reads TMEM lanes 32 (w % 4) .. +31 = 32 of this CTA's tokens, every other piece of features ----
        const int group = warp & 3, set = (warp - 2) >> 2;
        constexpr int PIECE_BYTES = 32 * CHUNK_F * (int)sizeof(TO);
        const uint32_t piece_addr = staging_base + (uint32_t)((warp - 2) * PIECE_BYTES);
        uint8_t* piece = smem_raw + (piece_addr - smem_u32(smem_raw));
        pdl_wait();
        bool ok = true;
        int n_unit = 0;
        for (int index = first_unit; index < units && ok; index += stride, ++n_unit) {
            const Unit u = unit_at(s, index);
            const int t = u.t0 + (int)rank * HALF_M + group * 32;
            const int buf = n_unit & 1;
            if (!mbar_wait(smem_u32(&acc_full[buf]), ((uint32_t)n_unit >> 1) & 1u)) { ok = false; break; }
            tc_fence_after();
            const uint32_t lane_addr = tmem_base + ((uint32_t)(group * 32) << 16) + (uint32_t)(buf * s.n_tile);
            if (t < s.M) {
                for (int c0 = set * CHUNK_F; c0 < s.width; c0 += 2 * CHUNK_F) {
                    if (u.f0 + c0 >= s.N) break;
                    float acc[32], up[32];
                    tmem_load32_nowait(lane_addr + (uint32_t)c0, acc);
                    if (GEMM_GATED(MODE)) tmem_load32_nowait(lane_addr + (uint32_t)(s.width + c0), up);
                    tmem_load_wait();
#pragma unroll
                    for (int c = 0; c < 32; ++c) acc[c] = finish<MODE>(acc[c], GEMM_GATED(MODE) ? up[c] : 0.f, s);
                    if (lane == 0) tma_wait_read<0>();            // the store that read this piece last is done with it
                    __syncwarp();
                    put_row(piece, lane, acc, (TO*)nullptr);
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (MODE == GEMM_ACCUM) tma_reduce_add_2d(&map_o, piece_addr, u.f0 + c0, t);
                        else tma_store_2d(&map_o, piece_addr, u.f0 + c0, t);
                        tma_commit_group();
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_on_first(smem_u32(&acc_empty[buf]));
        }
        if (!ok && lane == 0 && s.error_flag) atomicExch(s.error_flag, 3);
        if (lane == 0) tma_wait_all();                 // shared memory must outlive the stores that read it
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                    // neither CTA frees TMEM (or leaves) while the other may still use the pair's
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)s.tmem_cols) : "memory");
    }
}

int pow2_columns(int x) {
    int p = 32;
    while (p < x) p *= 2;
    return p;
}

// The output [M, N] (row stride ldo elements) for the epilogue's pieces: boxes of [32 tokens, 32 features], swizzled over the box's rows.
int make_piece_map(CUtensorMap* map, void* base, int out_dtype, int M, int N, int ldo) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return LIA_ERR_DRIVER;
    const int esize = out_dtype == LIA_F32 ? 4 : 2;
    cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)M};
    cuuint64_t strides[1] = {(cuuint64_t)ldo * esize};
    cuuint32_t box[2] = {CHUNK_F, 32};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = fn(map, out_dtype == LIA_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base,
                    dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    out_dtype == LIA_F32 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                    CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? LIA_OK : LIA_ERR_DRIVER;
}

template <int MODE, typename TO>
int launch(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& mo, const Shape& s, int pairs, cudaStream_t stream) {
    static std::atomic<bool> configured{false};
    if (!configured.load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(gemm_pair_kernel<MODE, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) {
            cudaGetLastError();
            return LIA_ERR_LAUNCH;
        }
        configured.store(true, std::memory_order_release);
    }
    return lia_launch(gemm_pair_kernel<MODE, TO>, dim3(2 * pairs), dim3(THREADS), (size_t)SMEM_BYTES, stream, mw, mx, mo, s);
}

// Rows of W per tile, and the time this is expected to take (us).  Measured on a B200 (2,023 products of 160 to 4,096 tokens by 160 to 8,192
// features, K 128 to 8,192, in tiles of 32 to 256 rows; within 7%): a product begins and ends in 3.8 us, a round of tiles costs 0.54 and per
// K block its MMAs' time, or 0.15 (what an MMA on two SMs takes at least, and the threads that issue it), and the stores 0.16 a megabyte.
// A tile of 256 rows takes 0.30 a K block, 1,680 TFLOP/s over the device, so wide tiles are the rule, and narrower ones what fills the
// last round: 2,048 x 6,144 pairs x 2,048 in 512 tiles of 96 pairs (6.9 rounds) 66.1, in 384 of 128 (5.2) 68.9; 1,111 x 2,048 x 6,144 24.2 in
// tiles of 160 rows (one round), 36.5 in tiles of 256.
double plan_width(bool gated, int M, int N, int K, int out_bytes, int sm_count, int* n_tile) {
    const int kblocks = (K + BLOCK_K - 1) / BLOCK_K, t_tiles = (M + PAIR_M - 1) / PAIR_M, pairs = std::max(1, sm_count / 2);
    const int step = gated ? 64 : 32;
    double best = -1;
    for (int n = 256; n >= step; n -= step) {
        const int width = gated ? n / 2 : n;
        const long long tiles = (long long)t_tiles * ((N + width - 1) / width);
        const long long rounds = (tiles + pairs - 1) / pairs;
        const double cost = 3.8 + rounds * (kblocks * std::max(0.152, 0.026 + 0.00108 * n) + 0.54) + 0.16e-6 * out_bytes * M * N;
        if (best < 0 || cost < best) { best = cost; *n_tile = n; }
    }
    return best;
}
}  // namespace

double gemm_pair_estimate(int mode, int M, int N, int K, int out_bytes, int sm_count) {
    int n_tile;
    return plan_width(GEMM_GATED(mode), M, N, K, out_bytes, sm_count, &n_tile);
}

int gemm_pair_launch(int mode, const void* X, int ldx, const void* W, int ldw, void* out, int out_dtype, int ldo, int M, int N,
                     int K, float alpha, int sm_count, int n_tile, float act_p, float act_n, int* error_flag, cudaStream_t stream) {
    const bool gated = GEMM_GATED(mode);
    if (n_tile == 0) plan_width(gated, M, N, K, out_dtype == LIA_F32 ? 4 : 2, sm_count, &n_tile);
    if (n_tile < 32 || n_tile > 256 || n_tile % (gated ? 64 : 32) || sm_count < 2) return LIA_ERR_SIZE;
    Shape s;
    s.M = M; s.N = N; s.n_tile = n_tile; s.width = gated ? n_tile / 2 : n_tile;
    s.kblocks = (K + BLOCK_K - 1) / BLOCK_K;
    s.f_tiles = (N + s.width - 1) / s.width;
    s.t_tiles = (M + PAIR_M - 1) / PAIR_M;
    s.tmem_cols = pow2_columns(2 * n_tile);
    s.alpha = alpha; s.act_p = act_p; s.act_n = act_n; s.error_flag = error_flag;
    const int esize = out_dtype == LIA_F32 ? 4 : 2;
    const int staging = EPILOGUE_WARPS * 32 * CHUNK_F * esize;
    const int stage_bytes = HALF_M * BLOCK_K * 2 + (n_tile / 2) * BLOCK_K * 2;
    s.stages = std::min(MAX_STAGES, (SMEM_BYTES - 1024 - staging) / stage_bytes);

    CUtensorMap mw, mx, mo;
    int rc;
    if ((rc = make_map(&mw, W, gated ? 2 * N : N, K, ldw, n_tile / 2)) != LIA_OK) return rc;
    if ((rc = make_map(&mx, X, M, K, ldx, HALF_M)) != LIA_OK) return rc;
    if ((rc = make_piece_map(&mo, out, out_dtype, M, N, ldo)) != LIA_OK) return rc;
    const int pairs = (int)std::min((long long)(sm_count / 2), (long long)s.f_tiles * s.t_tiles);
#define LIA_PAIR(MODE)                                                                             \
    case MODE:                                                                                     \
        return out_dtype == LIA_F32 ? launch<MODE, float>(mw, mx, mo, s, pairs, stream)            \
                                    : launch<MODE, __nv_bfloat16>(mw, mx, mo, s, pairs, stream)
    switch (mode) {
        LIA_PAIR(GEMM_STORE);
        LIA_PAIR(GEMM_SWIGLU);
        LIA_PAIR(GEMM_REGLU);
        LIA_PAIR(GEMM_STORE_RELU2);
        LIA_PAIR(GEMM_STORE_XIELU);
        case GEMM_ACCUM: return launch<GEMM_ACCUM, float>(mw, mx, mo, s, pairs, stream);
    }
#undef LIA_PAIR
    return LIA_ERR_SIZE;
}

// The product on pairs of SMs with tiles of `n_tile` rows of W (0: as many as it would choose), for tests and measurements; lia_gemm_tc
// chooses it by itself.
LIA_EXPORT int lia_gemm_pair(int mode, const void* X, int ldx, const void* W, int ldw, void* out, int out_dtype, int ldo, int M,
                             int N, int K, float alpha, int sm_count, int n_tile, int* error_flag, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return LIA_OK;
    if (K <= 0 || K % 8 || ldx < K || ldw < K || ldo < N || (mode != GEMM_STORE && mode != GEMM_ACCUM && mode != GEMM_SWIGLU))
        return LIA_ERR_SIZE;
    if ((out_dtype != LIA_F32 && out_dtype != LIA_BF16) || (mode == GEMM_ACCUM && out_dtype != LIA_F32)) return LIA_ERR_DTYPE;
    if (((uintptr_t)out & 15u) || ((long long)ldo * (out_dtype == LIA_F32 ? 4 : 2)) % 16) return LIA_ERR_ALIGN;
    return gemm_pair_launch(mode, X, ldx, W, ldw, out, out_dtype, ldo, M, N, K, alpha, sm_count, n_tile, 0.f, 0.f, error_flag, stream);
}
