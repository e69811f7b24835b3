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
// Grouped products (a mixture of experts): the first product's token tiles are those of a list on the device, each with a group whose
// matrix it is multiplied with (see lia_gemm_pair_grouped); a second, plain product (a shared expert's) may share the launch.
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
// Clears the bit of a shared::cluster address that tells the pair's CTAs apart, as public sources for two-CTA loads have it (CUTLASS's copy_sm100_tma.hpp).
constexpr uint32_t PEER_BIT_MASK = 0xFEFFFFFFu;

// One product of a launch.
struct Part {
    int M, N, kblocks, f_tiles, t_tiles;
};
struct Shape {
    Part part[2];             // the second only in launches of two products
    int n_tile;               // rows of W per tile (gated: gate and up rows together)
    int width;                // output features per tile: n_tile, or half of it for the gated product
    int stages, tmem_cols;
    const int* group_tiles;   // grouped: per token tile of the first product (group, first row, rows)
    const int* group_count;   // grouped: the number of token tiles
    int group_rows;           // grouped: rows of W per group
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
    int w0;                   // first row of W: f0, plus the group's first row
    int t_end;                // tokens from here on are not the tile's
    int second;               // the second product's
};
// GROUPED: the first product's tiles are the list's (`first_units` of them by width), the second product's follow.
template <bool GROUPED>
__device__ __forceinline__ Unit unit_at(const Shape& s, int index, int first_units, int listed) {
    Unit u;
    u.second = GROUPED && index >= first_units ? 1 : 0;
    if (u.second) index -= first_units;
    const Part& p = s.part[GROUPED ? u.second : 0];
    const int t_tiles = GROUPED && !u.second ? listed : p.t_tiles;
    const int band = index / (RASTER * p.f_tiles), t_first = band * RASTER;
    const int across = min(RASTER, t_tiles - t_first), rest = index - band * RASTER * p.f_tiles;
    const int tile = t_first + rest % across;
    u.f0 = u.w0 = (rest / across) * s.width;
    if (GROUPED && !u.second) {
        u.w0 += s.group_tiles[3 * tile] * s.group_rows;
        u.t0 = s.group_tiles[3 * tile + 1];
        u.t_end = u.t0 + s.group_tiles[3 * tile + 2];
    } else {
        u.t0 = tile * PAIR_M;
        u.t_end = p.M;
    }
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

// The tensor maps of a launch's products: W, X and the output of the first, then of the second.
template <bool GROUPED>
struct Maps {
    CUtensorMap w[GROUPED ? 2 : 1], x[GROUPED ? 2 : 1], o[GROUPED ? 2 : 1];
};

template <int MODE, typename TO, bool GROUPED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const __grid_constant__ Maps<GROUPED> maps, const __grid_constant__ Shape s) {
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
    int first_units = s.part[0].f_tiles * s.part[0].t_tiles, listed = s.part[0].t_tiles;
    int units = first_units + (GROUPED ? s.part[1].f_tiles * s.part[1].t_tiles : 0);
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
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.w[0]) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.x[0]) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.o[0]) : "memory");
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
    if (GROUPED) {
        pdl_wait();           // the list of tiles is the work of a kernel ahead
        listed = min(*s.group_count, s.part[0].t_tiles);
        first_units = listed * s.part[0].f_tiles;
        units = first_units + s.part[1].f_tiles * s.part[1].t_tiles;
    }

    if (warp == 0 && leader) {
        // ---- TMA producer (both CTAs): this CTA's 128 tokens, its half of the tile's rows of W ----
        // gated: the first CTA brings gate rows, the second up rows of the same features
        const auto w_first = [&](const Part& p) { return GEMM_GATED(MODE) ? (rank == 0 ? 0 : p.N) : (int)rank * half_n; };
        bool ok = true;
        int ahead = 0;
        if (!GROUPED) {   // the first ring of W boxes goes out before the kernel ahead has finished: weights depend on nothing
            int it = 0;
            for (int index = first_unit; index < units && it < s.stages; index += stride) {
                const Unit u = unit_at<GROUPED>(s, index, first_units, listed);
                for (int kb = 0; kb < s.part[0].kblocks && it < s.stages; ++kb, ++it) {
                    const uint32_t full = smem_u32(&full_bar[it]);
                    if (rank == 0) mbar_expect_tx(full, 2 * stage_bytes);
                    tma_load_pair(smem_base + (uint32_t)it * stage_bytes + A_BYTES, &maps.w[0], kb * BLOCK_K, w_first(s.part[0]) + u.w0, full);
                }
            }
            ahead = it;
        }
        pdl_wait();
        int it = 0, st = 0;
        uint32_t phase = 0;
        for (int index = first_unit; index < units && ok; index += stride) {
            const Unit u = unit_at<GROUPED>(s, index, first_units, listed);
            const int which = GROUPED ? u.second : 0;
            const Part& p = s.part[which];
            const CUtensorMap *map_w = &maps.w[which], *map_x = &maps.x[which];
            const int t_mine = u.t0 + (int)rank * HALF_M, w_mine = w_first(p) + u.w0;
            for (int kb = 0; kb < p.kblocks; ++kb, ++it) {
                const uint32_t full = smem_u32(&full_bar[st]);
                const uint32_t dst = smem_base + (uint32_t)st * stage_bytes;
                if (it >= ahead) {
                    if (!mbar_wait(smem_u32(&empty_bar[st]), phase ^ 1u)) { ok = false; break; }
                    if (rank == 0) mbar_expect_tx(full, 2 * stage_bytes);
                    tma_load_pair(dst + A_BYTES, map_w, kb * BLOCK_K, w_mine, full);
                }
                tma_load_pair(dst, map_x, kb * BLOCK_K, t_mine, full);
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
            const int kblocks = s.part[GROUPED && index >= first_units ? 1 : 0].kblocks;
            for (int kb = 0; kb < kblocks; ++kb) {
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
            const Unit u = unit_at<GROUPED>(s, index, first_units, listed);
            const int N = s.part[GROUPED ? u.second : 0].N;
            const CUtensorMap* map_o = &maps.o[GROUPED ? u.second : 0];
            const int t = u.t0 + (int)rank * HALF_M + group * 32;
            const int buf = n_unit & 1;
            if (!mbar_wait(smem_u32(&acc_full[buf]), ((uint32_t)n_unit >> 1) & 1u)) { ok = false; break; }
            tc_fence_after();
            const uint32_t lane_addr = tmem_base + ((uint32_t)(group * 32) << 16) + (uint32_t)(buf * s.n_tile);
            if (t < u.t_end) {
                for (int c0 = set * CHUNK_F; c0 < s.width; c0 += 2 * CHUNK_F) {
                    if (u.f0 + c0 >= N) break;
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
                        if (MODE == GEMM_ACCUM) tma_reduce_add_2d(map_o, piece_addr, u.f0 + c0, t);
                        else tma_store_2d(map_o, piece_addr, u.f0 + c0, t);
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

template <int MODE, typename TO, bool GROUPED>
int launch(const Maps<GROUPED>& maps, const Shape& s, int pairs, cudaStream_t stream) {
    static std::atomic<bool> configured{false};
    if (!configured.load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(gemm_pair_kernel<MODE, TO, GROUPED>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) {
            cudaGetLastError();
            return LIA_ERR_LAUNCH;
        }
        configured.store(true, std::memory_order_release);
    }
    return lia_launch(gemm_pair_kernel<MODE, TO, GROUPED>, dim3(2 * pairs), dim3(THREADS), (size_t)SMEM_BYTES, stream, maps, s);
}

// The parts of a launch that follow from the tile's width.
void set_width(Shape* s, bool gated, int n_tile, int out_bytes) {
    s->n_tile = n_tile;
    s->width = gated ? n_tile / 2 : n_tile;
    s->tmem_cols = pow2_columns(2 * n_tile);
    const int staging = EPILOGUE_WARPS * 32 * CHUNK_F * out_bytes, stage_bytes = HALF_M * BLOCK_K * 2 + (n_tile / 2) * BLOCK_K * 2;
    s->stages = std::min(MAX_STAGES, (SMEM_BYTES - 1024 - staging) / stage_bytes);
}
Part part_of(int M, int N, int K, int width) {
    return {M, N, (K + BLOCK_K - 1) / BLOCK_K, (N + width - 1) / width, (M + PAIR_M - 1) / PAIR_M};
}

// What a tile of n rows of W and so many K blocks takes in a round of tiles (us; see plan_width).
double tile_cost(int kblocks, int n) { return kblocks * std::max(0.152, 0.026 + 0.00108 * n) + 0.54; }

// Rows of W per tile, and the time this is expected to take (us).  Measured on a B200 (2,023 products of 160 to 4,096 tokens by 160 to 8,192
// features, K 128 to 8,192, in tiles of 32 to 256 rows; within 7%, and within a tenth for 1,206 of 1,520 others, one behind the other): a product begins and ends in 3.8 us, a round of tiles costs 0.54 and per
// K block its MMAs' time, or 0.15 (what an MMA on two SMs takes at least, and the threads that issue it), and the stores 0.16 a megabyte.
// A tile of 256 rows takes 0.30 a K block (8.4 MFLOP on two SMs: 2,070 TFLOP/s over the device while it lasts, at a short product's clocks; with its ends, and
// at the clocks that the power cap leaves a long one, 4,096 x 10,240 x 4,096 takes 215, 1,600 TFLOP/s), so wide tiles are the rule, and narrower ones what fills the
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
        const double cost = 3.8 + rounds * tile_cost(kblocks, n) + 0.16e-6 * out_bytes * M * N;
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
    Shape s = {};
    set_width(&s, gated, n_tile, out_dtype == LIA_F32 ? 4 : 2);
    s.part[0] = part_of(M, N, K, s.width);
    s.alpha = alpha; s.act_p = act_p; s.act_n = act_n; s.error_flag = error_flag;
    Maps<false> maps;
    int rc;
    if ((rc = make_map(&maps.w[0], W, gated ? 2 * N : N, K, ldw, n_tile / 2)) != LIA_OK) return rc;
    if ((rc = make_map(&maps.x[0], X, M, K, ldx, HALF_M)) != LIA_OK) return rc;
    if ((rc = make_piece_map(&maps.o[0], out, out_dtype, M, N, ldo)) != LIA_OK) return rc;
    const int pairs = (int)std::min((long long)(sm_count / 2), (long long)s.part[0].f_tiles * s.part[0].t_tiles);
#define LIA_PAIR(MODE)                                                                             \
    case MODE:                                                                                     \
        return out_dtype == LIA_F32 ? launch<MODE, float, false>(maps, s, pairs, stream)           \
                                    : launch<MODE, __nv_bfloat16, false>(maps, s, pairs, stream)
    switch (mode) {
        LIA_PAIR(GEMM_STORE);
        LIA_PAIR(GEMM_SWIGLU);
        LIA_PAIR(GEMM_REGLU);
        LIA_PAIR(GEMM_STORE_RELU2);
        LIA_PAIR(GEMM_STORE_XIELU);
        case GEMM_ACCUM: return launch<GEMM_ACCUM, float, false>(maps, s, pairs, stream);
    }
#undef LIA_PAIR
    return LIA_ERR_SIZE;
}

// A grouped product and, in the same launch, a plain one.  The first: X [rows_cap, K] bf16 = the tokens' rows sorted by group, every group's
// rows beginning at a multiple of 32 (a warp's stores, beyond which a tile writes nothing); W [groups, n_total, K] (n_total = N, or 2N for SWIGLU: gate rows then up rows); out [rows_cap, N].  `tiles`
// [3 * max_tiles] on the device lists (group, first row, rows) per token tile, `n_tiles` [1] how many there are; `expected` (a number of
// tiles) decides the tiles' width only.  Rows of out that belong to no tile's rows may be written.  The second (M2 0: none): out2 [M2, N2] = X2 [M2, K2] W2^T
// in the same form.  mode: GEMM_SWIGLU (bf16 or f32 out), GEMM_STORE, or GEMM_STORE with 3 above its byte (relu(sum)^2).
// What bounds it is W: eight experts of 2,048 pairs x 2,048 are 134 MB, 20 us of memory.  A launch for either product of a
// mixture, routed and shared expert in tiles of one CTA each, took 2 x 32 and 2 x 22 us at 512 tokens (eight experts of 2,048, two chosen); so the whole
// part went from 102 to 77.
LIA_EXPORT int lia_gemm_pair_grouped(int mode, const void* X, int ldx, int rows_cap, const void* W, int ldw, int groups, void* out,
                                     int out_dtype, int ldo, int N, int K, const int* tiles, const int* n_tiles, int max_tiles, int expected,
                                     const void* X2, int ldx2, int M2, const void* W2, int ldw2, void* out2, int ldo2, int N2, int K2,
                                     int sm_count, int* error_flag, cudaStream_t stream) {
    const int act = mode >> 8;
    mode &= 0xff;
    if ((mode != GEMM_STORE && mode != GEMM_SWIGLU) || (act != 0 && !(mode == GEMM_STORE && act == 3))) return LIA_ERR_SIZE;
    if (rows_cap <= 0 || N <= 0 || max_tiles <= 0) return LIA_ERR_SIZE;
    if (K <= 0 || K % 8 || ldx < K || ldw < K || ldo < N || sm_count < 2 || groups <= 0 || !tiles || !n_tiles || M2 < 0)
        return LIA_ERR_SIZE;
    if (M2 > 0 && (N2 <= 0 || K2 <= 0 || K2 % 8 || ldx2 < K2 || ldw2 < K2 || ldo2 < N2)) return LIA_ERR_SIZE;
    if (out_dtype != LIA_F32 && out_dtype != LIA_BF16) return LIA_ERR_DTYPE;
    const bool gated = mode == GEMM_SWIGLU;
    const int out_bytes = out_dtype == LIA_F32 ? 4 : 2, n_total = gated ? 2 * N : N;
    if (((uintptr_t)out & 15u) || ((long long)ldo * out_bytes) % 16 || (M2 > 0 && (((uintptr_t)out2 & 15u) || ((long long)ldo2 * out_bytes) % 16)))
        return LIA_ERR_ALIGN;
    if ((long long)groups * n_total > 0x7fffffffLL) return LIA_ERR_SIZE;
    // the width that leaves the pairs least idle, with as many tiles in the list as are expected
    const int pairs = sm_count / 2, kblocks = (std::max(K, M2 > 0 ? K2 : 0) + BLOCK_K - 1) / BLOCK_K, step = gated ? 64 : 32;
    double best = -1;
    int n_tile = 256;
    for (int n = 256; n >= step; n -= step) {
        const int width = gated ? n / 2 : n;
        const long long units = (long long)std::max(1, std::min(expected, max_tiles)) * ((N + width - 1) / width) +
                                (M2 > 0 ? (long long)((M2 + PAIR_M - 1) / PAIR_M) * ((N2 + width - 1) / width) : 0);
        const double cost = (units + pairs - 1) / pairs * tile_cost(kblocks, n);
        if (best < 0 || cost < best) { best = cost; n_tile = n; }
    }
    Shape s = {};
    set_width(&s, gated, n_tile, out_bytes);
    s.part[0] = part_of(rows_cap, N, K, s.width);
    s.part[0].t_tiles = max_tiles;
    if (M2 > 0) s.part[1] = part_of(M2, N2, K2, s.width);
    s.alpha = 1.0f; s.error_flag = error_flag;
    s.group_tiles = tiles; s.group_count = n_tiles; s.group_rows = n_total;
    Maps<true> maps;
    int rc;
    if ((rc = make_map(&maps.w[0], W, groups * n_total, K, ldw, n_tile / 2)) != LIA_OK) return rc;
    if ((rc = make_map(&maps.x[0], X, rows_cap, K, ldx, HALF_M)) != LIA_OK) return rc;
    if ((rc = make_piece_map(&maps.o[0], out, out_dtype, rows_cap, N, ldo)) != LIA_OK) return rc;
    if (M2 > 0) {
        if ((rc = make_map(&maps.w[1], W2, gated ? 2 * N2 : N2, K2, ldw2, n_tile / 2)) != LIA_OK) return rc;
        if ((rc = make_map(&maps.x[1], X2, M2, K2, ldx2, HALF_M)) != LIA_OK) return rc;
        if ((rc = make_piece_map(&maps.o[1], out2, out_dtype, M2, N2, ldo2)) != LIA_OK) return rc;
    } else {
        maps.w[1] = maps.w[0]; maps.x[1] = maps.x[0]; maps.o[1] = maps.o[0];
    }
    const long long units = (long long)s.part[0].f_tiles * max_tiles + (long long)s.part[1].f_tiles * s.part[1].t_tiles;
    const int grid = (int)std::min((long long)pairs, units);
    const bool f32 = out_dtype == LIA_F32;
    if (gated) return f32 ? launch<GEMM_SWIGLU, float, true>(maps, s, grid, stream) : launch<GEMM_SWIGLU, __nv_bfloat16, true>(maps, s, grid, stream);
    if (act == 3)
        return f32 ? launch<GEMM_STORE_RELU2, float, true>(maps, s, grid, stream) : launch<GEMM_STORE_RELU2, __nv_bfloat16, true>(maps, s, grid, stream);
    return f32 ? launch<GEMM_STORE, float, true>(maps, s, grid, stream) : launch<GEMM_STORE, __nv_bfloat16, true>(maps, s, grid, stream);
}

// The product on pairs of SMs with tiles of `n_tile` rows of W (0: as many as it would choose), for tests and measurements; lia_gemm_tc
// chooses it by itself.  The epilogue's variant rides above the mode's byte, as there.
LIA_EXPORT int lia_gemm_pair(int mode, const void* X, int ldx, const void* W, int ldw, void* out, int out_dtype, int ldo, int M,
                             int N, int K, float alpha, int sm_count, int n_tile, float act_p, float act_n, int* error_flag, cudaStream_t stream) {
    const int act = mode >> 8;
    mode &= 0xff;
    if (act != 0 && !(mode == GEMM_SWIGLU && act == 4) && !(mode == GEMM_STORE && (act == 3 || act == 5))) return LIA_ERR_SIZE;
    if (M <= 0 || N <= 0) return LIA_OK;
    if (K <= 0 || K % 8 || ldx < K || ldw < K || ldo < N || (mode != GEMM_STORE && mode != GEMM_ACCUM && mode != GEMM_SWIGLU))
        return LIA_ERR_SIZE;
    if ((out_dtype != LIA_F32 && out_dtype != LIA_BF16) || (mode == GEMM_ACCUM && out_dtype != LIA_F32)) return LIA_ERR_DTYPE;
    if (((uintptr_t)out & 15u) || ((long long)ldo * (out_dtype == LIA_F32 ? 4 : 2)) % 16) return LIA_ERR_ALIGN;
    const int form = act == 5 ? GEMM_STORE_XIELU : act == 3 ? GEMM_STORE_RELU2 : act == 4 ? GEMM_REGLU : mode;
    return gemm_pair_launch(form, X, ldx, W, ldw, out, out_dtype, ldo, M, N, K, alpha, sm_count, n_tile, act_p, act_n, error_flag, stream);
}
