// Retention's prompt portions on tcgen05, for heads of 64 or 128 elements and bfloat16 outputs (csrc/retention.cu has the formulas, the other
// sizes and the 32-bit path): chunks of 128 tokens side by side, a CTA a chunk and head.
//
//   sums     U_c [d, dv] = sum_j (decay^(len-1-j) k_j) v_j^T
//   carry    csrc/retention.cu's
//   output   A = Q K^T and O1 = Q S_in in one pass over d, P = A times decay^(t-j) for j <= t, O2 = P V; o = decay^(t+1) O1 + O2, the
//            head's norm, the gate.
//
// The operands are 32-bit numbers and stay so: each is two tf32 numbers, the nearest one and what is left (see split), and a product is hi hi
// + hi lo + lo hi, accumulated in 32 bits in TMEM.  What is left out, lo lo and the last bit of lo, is some 2^-24 of a term, as much as a 32-bit
// multiply-add rounds away.  Against 64 bits, beside the 32-bit pipes: state after 100, 700, 2,048 tokens of 16 heads of 128 x 128 1.1e-7, 1.6e-7, 1.66e-7
// (1.2e-7, 1.6e-7, 1.64e-7), of 64 x 64 1.2e-7, 1.6e-7, 1.66e-7 (1.2e-7, 1.6e-7, 1.64e-7); outputs 0.00166 either way, their last rounding.
//
// What bounds these kernels is the way of the operands: 32-bit rows from L2 into registers, split, into shared memory as the tensor cores
// want them (rows of 32 tf32 numbers, 128 bytes, swizzled; tokens as the contracted dimension mean a transposed tile, which squares of four by four
// go to).  The multiply-adds of a chunk are 9,000 cycles of the tensor cores for outputs, 3,000 for
// sums, of some 34,000 and 20,000 that a CTA lives: a chain of trips and phases, one CTA an SM (200 KB of shared memory, all of TMEM).
// 2,048 tokens of 16 heads, us: 128 x 128 sums 23, carry 8, outputs 44 (32-bit pipes, chunks of 64: 33, 13, 95), 64 x 64 13, 4, 20.  The three launches in a
// row: 128 x 128, 33 tokens 43 -> 23, 700 64 -> 34, 2,048 140 -> 78; 64 x 64 22 -> 15, 38 -> 19, 61 -> 36.
//
// Every wait on an mbarrier is bounded: a role that gives up raises the error flag and leaves its loop; TMEM is freed behind the CTA's last
// barrier, which everyone reaches.
#include "linear_recurrence.cuh"
#include "retention_tc.cuh"
#include "tcgen05.cuh"

using namespace tc5;

namespace {
constexpr int TOKENS = RETENTION_TC_CHUNK;       // a chunk: the MMA's M (outputs), its K (sums)
// Warps that bring operands and empty TMEM (one more issues): sixteen for values of 64 elements, eight for 128, whose squares in flight need the
// registers (2,048 tokens of 16 heads, us for sums and outputs: 64 x 64 with eight 12.1 and 21.4, with sixteen 12.2 and 19.7; 128 x 128 22 and 42, 28 and 44).
template <int DV>
struct Crew {
    static constexpr int WORKERS = DV == 64 ? 512 : 256, THREADS = WORKERS + 32;
    static constexpr int PARTS = WORKERS / 128;      // warps that share the TMEM lanes of 32 rows
};
constexpr int BLOCK = 32;                        // tf32 numbers in a row of 128 bytes
constexpr int ROW = 128;
constexpr uint32_t TILE_BYTES = 128 * ROW;       // 128 rows

// x = hi + lo exactly: hi the nearest number with ten bits behind the leading one, lo at most eleven, of which the tensor cores read ten
// (integer operations: the conversion instruction has a quarter of their rate, and took as long as the products).
__device__ __forceinline__ void split(float x, float& hi, float& lo) {
    hi = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
    lo = x - hi;
}
// Instruction descriptor: 32-bit accumulator, tf32 A and B, both K-major.
__device__ __forceinline__ uint32_t instr_desc_tf32(int m, int n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// A from tensor memory: rows = lanes, a tf32 number a column.
__device__ __forceinline__ void mma_tf32_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_store32(uint32_t addr, const float* v) {
    const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// N (16 or 32) columns of this warp's 32 TMEM lanes, without waiting.
template <int N>
__device__ __forceinline__ void tmem_load_columns(uint32_t addr, float (&v)[N]) {
    if constexpr (N == 32) tmem_load32_nowait(addr, v);
    else tmem_load16_nowait(addr, v);
}
template <int WORKERS>
__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory"); }

// Four numbers of a row of a tile (its 16-byte piece `piece`), split.
__device__ __forceinline__ void put_piece(uint8_t* hi_tile, uint8_t* lo_tile, int row, int piece, float4 v) {
    float4 h, l;
    split(v.x, h.x, l.x);
    split(v.y, h.y, l.y);
    split(v.z, h.z, l.z);
    split(v.w, h.w, l.w);
    const uint32_t at = (uint32_t)(row * ROW + ((piece ^ (row & 7)) << 4));
    *reinterpret_cast<float4*>(hi_tile + at) = h;
    *reinterpret_cast<float4*>(lo_tile + at) = l;
}
// A square of four tokens by four columns, for a tile with the tokens along its rows.  A warp's lanes read whole lines of four tokens; in
// what they store, every lane turns its columns so that eight neighbours fall into eight different 16-byte places of the swizzle (rows
// 4 quad + i alone differ in one of their low three bits for the same i).
struct Square {
    float4 token[4];
};
__device__ __forceinline__ Square load_square(const float* __restrict__ src, long long ld, int j, int len, int quad) {
    Square q;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const bool there = j + r < len;
        q.token[r] = __ldg(reinterpret_cast<const float4*>(src + (size_t)(there ? j + r : 0) * ld + quad * 4));
        if (!there) q.token[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return q;
}
__device__ __forceinline__ void put_square(uint8_t* hi_tile, uint8_t* lo_tile, int quad, int group, const Square& q) {
    const float* x = reinterpret_cast<const float*>(q.token);                 // [token][column]
    const int turn = (quad >> 1) & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int c = (i + turn) & 3, row = 4 * quad + c;
        float h[4], l[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            // (x[4 r + c], c known only to the lane)
            const float even = c & 2 ? x[4 * r + 2] : x[4 * r], odd = c & 2 ? x[4 * r + 3] : x[4 * r + 1];
            split(c & 1 ? odd : even, h[r], l[r]);
        }
        const uint32_t at = (uint32_t)(row * ROW + ((group ^ (row & 7)) << 4));
        *reinterpret_cast<float4*>(hi_tile + at) = make_float4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<float4*>(lo_tile + at) = make_float4(l[0], l[1], l[2], l[3]);
    }
}
// The three products of K steps FROM .. TO - 1 of the four of a block of 32: acc (+)= (ah + al) (bh + bl) without al bl.  The small ones come first: the unit cuts
// every sum off (it does not round), by so much of what the accumulator holds.
template <int FROM = 0, int TO = BLOCK / 8>
__device__ __forceinline__ void multiply_block(uint32_t acc, uint64_t ah, uint64_t al, uint64_t bh, uint64_t bl, uint32_t idesc, bool first) {
#pragma unroll
    for (int k = FROM; k < TO; ++k) {
        mma_tf32(acc, ah + 2 * k, bl + 2 * k, idesc, first && k == FROM ? 0u : 1u);
        mma_tf32(acc, al + 2 * k, bh + 2 * k, idesc, 1u);
    }
#pragma unroll
    for (int k = FROM; k < TO; ++k) mma_tf32(acc, ah + 2 * k, bh + 2 * k, idesc, 1u);
}

// Bytes of a stage, of which there are two. Sums: K^T hi, lo (128 rows, of which D are filled), V^T hi, lo.  Outputs: Q hi, lo, K hi, lo, S^T hi, lo.
template <int DV>
struct Bytes {
    static constexpr uint32_t SUMS_STAGE = 2 * TILE_BYTES + 2 * DV * ROW, OUTPUT_STAGE = 4 * TILE_BYTES + 2 * DV * ROW;
    static constexpr size_t SUMS = 1024 + 2 * SUMS_STAGE, OUTPUT = 1024 + 2 * OUTPUT_STAGE;
};

struct Rows {
    const float* rows; long long ld;
    const float* decay; const int* segments; int n_segments; int heads;
    int* error_flag;
};

// ---- U [chunk, head, D, DV] ----
template <int D, int DV>
__global__ void __launch_bounds__(Crew<DV>::THREADS, 1)
retention_tc_sums_kernel(Rows p, float* __restrict__ sums) {
    constexpr int WORKERS = Crew<DV>::WORKERS, PARTS = Crew<DV>::PARTS;
    constexpr int STAGES = 2, BLOCKS = TOKENS / BLOCK;
    // Sixteen tokens have an accumulator of their own, and those are added in 32 bits, rounded: the unit cuts a sum off at every step (state's
    // error after 2,048 tokens, 16 heads of 64 x 64: 8.4e-7 with a chunk in one accumulator, 1.9e-7 with 32 tokens, 1.7e-7 so, 1.6e-7 on the
    // 32-bit pipes).  TMEM holds as many as ACCUMULATORS: values of 128 elements empty them half way.
    constexpr int ACCUMULATORS = 512 / DV, PER_BLOCK = 2, BLOCKS_HELD = ACCUMULATORS / PER_BLOCK;
    constexpr uint32_t COLUMNS = ACCUMULATORS * DV;
    static_assert(BLOCKS_HELD == BLOCKS || BLOCKS_HELD == STAGES, "emptied when the stages are used again");
    constexpr uint32_t V_BYTES = DV * ROW, STAGE = Bytes<DV>::SUMS_STAGE;
    static_assert(D * (DV + 4) * 4 <= 2 * STAGE, "the sums leave through the stages");
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], done_bar;
    __shared__ uint32_t tmem_slot;
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const bool leader = elect_one();
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - smem_u32(smem_raw));
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(smem_u32(&full_bar[i]), WORKERS);
            mbar_init(smem_u32(&empty_bar[i]), 1);
        }
        mbar_init(smem_u32(&done_bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == WORKERS / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(COLUMNS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();
    pdl_wait();
    int first = 0, len = 0, segment, chunk;
    const bool here = find_chunk<TOKENS>(p.segments, p.n_segments, blockIdx.x, &first, &len, &segment, &chunk);
    const int h = blockIdx.y, blocks = here ? (len + BLOCK - 1) / BLOCK : 0;
    if (warp < WORKERS / 32 && here) {
        const float* k = p.rows + (size_t)first * p.ld + (size_t)(p.heads + h) * D;
        const float* v = p.rows + (size_t)first * p.ld + (size_t)2 * p.heads * D + (size_t)h * DV;
        const float log_a = log2f(p.decay[h]);
        // a block's squares: eight groups of four tokens by the values' and the keys' quads of columns, AHEAD blocks ahead (eight warps keep
        // 64 numbers of U a thread beside them)
        constexpr int VQ = DV / 4, KQ = D / 4, UNITS = 8 * (VQ + KQ), PER = (UNITS + WORKERS - 1) / WORKERS;
        constexpr int AHEAD = PARTS == 2 ? 1 : 2;
        Square squares[AHEAD][PER];
        auto place = [&](int i, bool& key, int& group, int& quad) {
            const int u = threadIdx.x + i * WORKERS, w = u - 8 * VQ;
            key = w >= 0;
            group = key ? w / KQ : u / VQ;
            quad = key ? w % KQ : u % VQ;
            return UNITS % WORKERS == 0 || u < UNITS;
        };
        auto load = [&](int b) {
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                bool key; int group, quad;
                if (place(i, key, group, quad) && b < blocks) squares[b % AHEAD][i] = load_square(key ? k : v, p.ld, b * BLOCK + group * 4, len, quad);
            }
        };
        load(0);
        if (AHEAD == 2) load(1);
        // this thread's part of U: a row (a TMEM lane) of d, COLS columns
        constexpr int COLS = DV / PARTS, COLUMNS_AT_ONCE = COLS < 32 ? COLS : 32;
        const int quarter = warp & 3, c0 = (warp >> 2) * COLS;
        float u[COLS] = {};
        auto drain = [&](int accumulators) {
            tc_fence_after();
            if (quarter * 32 < D) {
                for (int a = 0; a < accumulators; ++a)
#pragma unroll
                    for (int c = 0; c < COLS; c += COLUMNS_AT_ONCE) {
                        float y[COLUMNS_AT_ONCE];
                        tmem_load_columns(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(a * DV + c0 + c), y);
                        tmem_load_wait();
#pragma unroll
                        for (int i = 0; i < COLUMNS_AT_ONCE; ++i) u[c + i] += y[i];
                    }
            }
            tc_fence_before();
        };
        bool ok = true;
#pragma unroll
        for (int b = 0; b < BLOCKS; ++b) {
            if (b >= blocks) break;
            if (b >= STAGES) ok = mbar_wait(smem_u32(&empty_bar[b % STAGES]), ((uint32_t)(b / STAGES) & 1u) ^ 1u);
            if (b == BLOCKS_HELD) {
                // (the second half's first products wait for every worker's arrival below)
                if (ok) ok = mbar_wait(smem_u32(&empty_bar[1]), 0u);
                ok = __all_sync(0xffffffffu, ok);
                if (ok) drain(ACCUMULATORS);
            }
            if (!ok) break;
            uint8_t* stage = smem + (b % STAGES) * STAGE;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                bool key; int group, quad;
                if (!place(i, key, group, quad)) continue;
                Square& q = squares[b % AHEAD][i];
                if (key) {
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        q.token[r] = scaled(q.token[r], exp2f((float)max(len - 1 - (b * BLOCK + group * 4 + r), 0) * log_a));
                }
                uint8_t* tile = stage + (key ? 0 : 2 * TILE_BYTES);
                put_square(tile, tile + (key ? TILE_BYTES : V_BYTES), quad, group, q);
            }
            fence_async_smem();
            mbar_arrive(smem_u32(&full_bar[b % STAGES]));
            if (b + AHEAD < BLOCKS) load(b + AHEAD);
        }
        if (ok) ok = mbar_wait(smem_u32(&done_bar), 0u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && lane == 0 && p.error_flag) atomicExch(p.error_flag, 3);
        if (ok) drain(PER_BLOCK * (blocks > BLOCKS_HELD ? blocks - BLOCKS_HELD : blocks));
        // rows of U through shared memory (the stages are free), so that they leave as whole lines
        constexpr int LD = DV + 4;
        float* tile = reinterpret_cast<float*>(smem);
        if (quarter * 32 < D) {
            float* dst = tile + (quarter * 32 + lane) * LD + c0;
#pragma unroll
            for (int i = 0; i < COLS; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(u[i], u[i + 1], u[i + 2], u[i + 3]);
        }
        workers_sync<WORKERS>();
        float* U = sums + ((size_t)blockIdx.x * p.heads + h) * D * DV;
#pragma unroll
        for (int e = threadIdx.x; e < D * (DV / 4); e += WORKERS) {
            const int r = e / (DV / 4), c = (e % (DV / 4)) * 4;
            *reinterpret_cast<float4*>(U + (size_t)r * DV + c) = *reinterpret_cast<const float4*>(tile + r * LD + c);
        }
    } else if (warp == WORKERS / 32 && leader && here) {
        const uint32_t idesc = instr_desc_tf32(128, DV);
        bool ok = true;
        for (int b = 0; b < blocks; ++b) {
            if (!mbar_wait(smem_u32(&full_bar[b % STAGES]), (uint32_t)(b / STAGES) & 1u)) { ok = false; break; }
            tc_fence_after();
            const uint32_t at = base + (uint32_t)(b % STAGES) * STAGE;
            const uint64_t kh = smem_desc(at), kl = smem_desc(at + TILE_BYTES), vh = smem_desc(at + 2 * TILE_BYTES), vl = smem_desc(at + 2 * TILE_BYTES + V_BYTES);
            const uint32_t acc = tmem + (uint32_t)(PER_BLOCK * (b % BLOCKS_HELD) * DV);
            multiply_block<0, BLOCK / 16>(acc, kh, kl, vh, vl, idesc, true);
            multiply_block<BLOCK / 16, BLOCK / 8>(acc + DV, kh, kl, vh, vl, idesc, true);
            tc_commit(smem_u32(&empty_bar[b % STAGES]));
        }
        if (ok) tc_commit(smem_u32(&done_bar));
        else if (p.error_flag) atomicExch(p.error_flag, 3);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == WORKERS / 32) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLUMNS) : "memory");
    }
}

// ---- outputs ----
template <int D, int DV>
__global__ void __launch_bounds__(Crew<DV>::THREADS, 1)
retention_tc_output_kernel(Rows p, const float* __restrict__ sums, __nv_bfloat16* __restrict__ out, float eps) {
    constexpr int WORKERS = Crew<DV>::WORKERS, PARTS = Crew<DV>::PARTS;
    constexpr int STAGES = 2, BLOCKS = D / BLOCK;
    constexpr uint32_t S_BYTES = DV * ROW, STAGE = Bytes<DV>::OUTPUT_STAGE;
    constexpr uint32_t V_BLOCK = 2 * S_BYTES;                                          // V^T hi, lo of 32 tokens, later in the stages' place
    static_assert(TOKENS / BLOCK * V_BLOCK <= 2 * STAGE && TOKENS * (DV + 4) * 4 <= 2 * STAGE, "the values, and the outputs, lie where the stages were");
    constexpr uint32_t COL_A = 0, COL_LO = 128, COL_O1 = 256, COL_O2 = 384;            // A (then P's hi), P's lo, O1, O2
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], scores_bar, weights_bar, done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ float powers[TOKENS + 1], squares[PARTS][TOKENS], inverse[TOKENS];
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const bool leader = elect_one();
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - smem_u32(smem_raw));
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(smem_u32(&full_bar[i]), WORKERS);
            mbar_init(smem_u32(&empty_bar[i]), 1);
        }
        mbar_init(smem_u32(&scores_bar), 1);
        mbar_init(smem_u32(&weights_bar), WORKERS);
        mbar_init(smem_u32(&done_bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == WORKERS / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();
    pdl_wait();
    int first = 0, len = 0, segment, chunk;
    const bool here = find_chunk<TOKENS>(p.segments, p.n_segments, blockIdx.x, &first, &len, &segment, &chunk);
    const int h = blockIdx.y, key_blocks = here ? (len + BLOCK - 1) / BLOCK : 0;
    if (warp < WORKERS / 32 && here) {
        const int tid = threadIdx.x;
        const float log_a = log2f(p.decay[h]);
        if (tid <= TOKENS) powers[tid] = exp2f((float)tid * log_a);
        const float* q = p.rows + (size_t)first * p.ld + (size_t)h * D;
        const float* k = q + (size_t)p.heads * D;
        const float* v = p.rows + (size_t)first * p.ld + (size_t)2 * p.heads * D + (size_t)h * DV;
        const float* S = sums + ((size_t)blockIdx.x * p.heads + h) * D * DV;
        constexpr int PER = TOKENS * 8 / WORKERS;                                      // 16-byte pieces of Q and of K a thread and block
        constexpr int VQ = DV / 4, SETS = WORKERS / (8 * VQ);                          // a block of the state is eight groups of rows by VQ quads of columns: a set's squares
        const int set = tid / (8 * VQ), s_group = tid % (8 * VQ) / VQ, s_quad = tid % VQ;      // set n takes blocks n, n + SETS, ..
        float4 qs[2][PER], ks[2][PER];                                                 // two blocks ahead
        Square state[SETS == 1 ? 2 : 1];                                               // (one set of threads: it has two blocks in flight)
        auto load = [&](int b) {
            float4 (&qv)[PER] = qs[b & 1], (&kv)[PER] = ks[b & 1];
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int e = tid + i * WORKERS, t = e >> 3, c = b * BLOCK + (e & 7) * 4;
                const bool there = t < len;
                const size_t at = (size_t)(there ? t : 0) * p.ld + c;
                qv[i] = __ldg(reinterpret_cast<const float4*>(q + at));
                kv[i] = __ldg(reinterpret_cast<const float4*>(k + at));
                if (!there) qv[i] = kv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            if (b % SETS == set) state[SETS == 1 ? b & 1 : 0] = load_square(S, DV, b * BLOCK + s_group * 4, D, s_quad);
        };
        bool ok = true;
        load(0);
        load(1);
#pragma unroll
        for (int b = 0; b < BLOCKS; ++b) {
            if (ok && b >= STAGES) ok = mbar_wait(smem_u32(&empty_bar[b % STAGES]), ((uint32_t)(b / STAGES) & 1u) ^ 1u);
            uint8_t* stage = smem + (b % STAGES) * STAGE;
            if (ok) {
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int e = tid + i * WORKERS;
                    put_piece(stage, stage + TILE_BYTES, e >> 3, e & 7, qs[b & 1][i]);
                    put_piece(stage + 2 * TILE_BYTES, stage + 3 * TILE_BYTES, e >> 3, e & 7, ks[b & 1][i]);
                }
                if (b % SETS == set) put_square(stage + 4 * TILE_BYTES, stage + 4 * TILE_BYTES + S_BYTES, s_quad, s_group, state[SETS == 1 ? b & 1 : 0]);
                fence_async_smem();
                mbar_arrive(smem_u32(&full_bar[b % STAGES]));
            }
            if (b + 2 < BLOCKS) load(b + 2);
        }
        // the values, asked for while the products run, go where the stages were
        constexpr int PER_V = TOKENS / 4 * VQ / WORKERS;                               // squares a thread
        Square values[PER_V];
#pragma unroll
        for (int i = 0; i < PER_V; ++i) {
            const int u = tid + i * WORKERS;
            values[i] = load_square(v, p.ld, u / VQ * 4, len, u % VQ);
        }
        if (ok) ok = mbar_wait(smem_u32(&scores_bar), 0u);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        if (ok) {
#pragma unroll
            for (int i = 0; i < PER_V; ++i) {
                const int u = tid + i * WORKERS, group = u / VQ;
                uint8_t* tile = smem + group / 8 * V_BLOCK;
                put_square(tile, tile + S_BYTES, u % VQ, group % 8, values[i]);
            }
        }
        workers_sync<WORKERS>();                                      // (the powers are there)
        // P = A decay^(t-j), split, in A's place and beside it: a thread a token and a part of the keys
        const int quarter = warp & 3, part = warp >> 2, t = quarter * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
        if (ok) {
#pragma unroll
            for (int c0 = part * (TOKENS / PARTS); c0 < (part + 1) * (TOKENS / PARTS); c0 += 32) {
                float x[32], lo[32];
                tmem_load32_nowait(lanes + COL_A + (uint32_t)c0, x);
                tmem_load_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const int back = t - (c0 + i);
                    const float w = back >= 0 ? x[i] * powers[back >= 0 ? back : 0] : 0.f;
                    split(w, x[i], lo[i]);
                }
                tmem_store32(lanes + COL_A + (uint32_t)c0, x);
                tmem_store32(lanes + COL_LO + (uint32_t)c0, lo);
            }
            tmem_store_wait();
            tc_fence_before();
            fence_async_smem();
            mbar_arrive(smem_u32(&weights_bar));
        }
        // the gates, asked for while the last products run
        constexpr int LANES = DV / 4, AT_ONCE = WORKERS / LANES, TURNS = TOKENS / AT_ONCE;      // threads a token, tokens at a time
        const int col = (tid % LANES) * 4;
        const float* g = p.rows + (size_t)first * p.ld + (size_t)2 * p.heads * D + (size_t)(p.heads + h) * DV + col;
        float4 gates[TURNS];
#pragma unroll
        for (int i = 0; i < TURNS; ++i) {
            const int r = tid / LANES + i * AT_ONCE;
            gates[i] = __ldg(reinterpret_cast<const float4*>(g + (size_t)(r < len ? r : 0) * p.ld));
        }
        if (ok) ok = mbar_wait(smem_u32(&done_bar), 0u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && lane == 0 && p.error_flag) atomicExch(p.error_flag, 3);
        tc_fence_after();
        // o = decay^(t+1) O1 + O2 and its sum of squares; through shared memory, so that gates and outputs are whole lines
        constexpr int LD = DV + 4;
        float* tile = reinterpret_cast<float*>(smem);
        const float power = powers[t + 1];
        float sum = 0.f;
        constexpr int COLS = DV / PARTS, STEP = COLS < 32 ? COLS : 32;
#pragma unroll
        for (int c0 = part * COLS; c0 < (part + 1) * COLS; c0 += STEP) {
            float a[STEP], b[STEP];
            tmem_load_columns(lanes + COL_O1 + (uint32_t)c0, a);
            tmem_load_columns(lanes + COL_O2 + (uint32_t)c0, b);
            tmem_load_wait();
            float* dst = tile + t * LD + c0;
#pragma unroll
            for (int i = 0; i < STEP; ++i) {
                a[i] = fmaf(power, a[i], b[i]);
                sum = fmaf(a[i], a[i], sum);
            }
#pragma unroll
            for (int i = 0; i < STEP; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(a[i], a[i + 1], a[i + 2], a[i + 3]);
        }
        squares[part][t] = sum;
        workers_sync<WORKERS>();
        if (part == 0) {
            float all = 0.f;
#pragma unroll
            for (int n = 0; n < PARTS; ++n) all += squares[n][t];
            inverse[t] = 1.0f / sqrtf(all / (float)DV + eps);
        }
        workers_sync<WORKERS>();
        __nv_bfloat16* dst = out + (size_t)first * p.heads * DV + (size_t)h * DV + col;
#pragma unroll
        for (int i = 0; i < TURNS; ++i) {
            const int r = tid / LANES + i * AT_ONCE;
            if (r >= len) break;
            const float4 z = gates[i];
            const float4 o = *reinterpret_cast<const float4*>(tile + r * LD + col);
            const float inv = inverse[r];
            const float zs[4] = {z.x, z.y, z.z, z.w}, os[4] = {o.x, o.y, o.z, o.w};
            struct alignas(8) Four { __nv_bfloat16 v[4]; } f;
#pragma unroll
            for (int e = 0; e < 4; ++e) f.v[e] = __float2bfloat16_rn(os[e] * inv * (zs[e] / (1.0f + expf(-zs[e]))));
            *reinterpret_cast<Four*>(dst + (size_t)r * p.heads * DV) = f;
        }
    } else if (warp == WORKERS / 32 && leader && here) {
        const uint32_t idesc_a = instr_desc_tf32(128, TOKENS), idesc_o = instr_desc_tf32(128, DV);
        bool ok = true;
        for (int b = 0; b < BLOCKS; ++b) {
            if (!mbar_wait(smem_u32(&full_bar[b % STAGES]), (uint32_t)(b / STAGES) & 1u)) { ok = false; break; }
            tc_fence_after();
            const uint32_t at = base + (uint32_t)(b % STAGES) * STAGE;
            const uint64_t qh = smem_desc(at), ql = smem_desc(at + TILE_BYTES);
            multiply_block(tmem + COL_A, qh, ql, smem_desc(at + 2 * TILE_BYTES), smem_desc(at + 3 * TILE_BYTES), idesc_a, b == 0);
            multiply_block(tmem + COL_O1, qh, ql, smem_desc(at + 4 * TILE_BYTES), smem_desc(at + 4 * TILE_BYTES + S_BYTES), idesc_o, b == 0);
            tc_commit(smem_u32(&empty_bar[b % STAGES]));
        }
        if (ok) {
            tc_commit(smem_u32(&scores_bar));
            ok = mbar_wait(smem_u32(&weights_bar), 0u);
        }
        if (ok) {
            tc_fence_after();
            for (int b = 0; b < key_blocks; ++b) {
                const uint64_t vh = smem_desc(base + b * V_BLOCK), vl = smem_desc(base + b * V_BLOCK + S_BYTES);
#pragma unroll
                for (int k = 0; k < BLOCK / 8; ++k) {
                    const uint32_t hi = tmem + COL_A + (uint32_t)(b * BLOCK + k * 8), lo = tmem + COL_LO + (uint32_t)(b * BLOCK + k * 8);
                    mma_tf32_ts(tmem + COL_O2, hi, vh + 2 * k, idesc_o, b > 0 || k > 0 ? 1u : 0u);
                    mma_tf32_ts(tmem + COL_O2, hi, vl + 2 * k, idesc_o, 1u);
                    mma_tf32_ts(tmem + COL_O2, lo, vh + 2 * k, idesc_o, 1u);
                }
            }
            tc_commit(smem_u32(&done_bar));
        } else if (p.error_flag) {
            atomicExch(p.error_flag, 3);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == WORKERS / 32) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

template <typename Kernel>
int raise(Kernel kernel, size_t bytes, std::atomic<bool>& done) {
    if (done.load(std::memory_order_acquire)) return LIA_OK;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) {
        cudaGetLastError();
        return LIA_ERR_LAUNCH;
    }
    done.store(true, std::memory_order_release);
    return LIA_OK;
}

template <int D, int DV>
int launch_sums(const Rows& p, int chunks, float* sums, cudaStream_t stream) {
    static std::atomic<bool> raised{false};
    const int rc = raise(retention_tc_sums_kernel<D, DV>, Bytes<DV>::SUMS, raised);
    return rc != LIA_OK ? rc : lia_launch(retention_tc_sums_kernel<D, DV>, dim3(chunks, p.heads), dim3(Crew<DV>::THREADS), Bytes<DV>::SUMS, stream, p, sums);
}
template <int D, int DV>
int launch_output(const Rows& p, int chunks, const float* sums, __nv_bfloat16* out, float eps, cudaStream_t stream) {
    static std::atomic<bool> raised{false};
    const int rc = raise(retention_tc_output_kernel<D, DV>, Bytes<DV>::OUTPUT, raised);
    return rc != LIA_OK ? rc : lia_launch(retention_tc_output_kernel<D, DV>, dim3(chunks, p.heads), dim3(Crew<DV>::THREADS), Bytes<DV>::OUTPUT, stream, p, sums, out, eps);
}
}  // namespace

int retention_tc_sums(const float* rows, long long ld, const float* decay, const int* segments, int n_segments, int chunks, float* sums,
                      int heads, int d, int dv, int* error_flag, cudaStream_t stream) {
    const Rows p = {rows, ld, decay, segments, n_segments, heads, error_flag};
    if (d == 64) return dv == 64 ? launch_sums<64, 64>(p, chunks, sums, stream) : launch_sums<64, 128>(p, chunks, sums, stream);
    return dv == 64 ? launch_sums<128, 64>(p, chunks, sums, stream) : launch_sums<128, 128>(p, chunks, sums, stream);
}
int retention_tc_output(const float* rows, long long ld, const float* decay, const int* segments, int n_segments, int chunks,
                        const float* sums, void* out, int heads, int d, int dv, float eps, int* error_flag, cudaStream_t stream) {
    const Rows p = {rows, ld, decay, segments, n_segments, heads, error_flag};
    __nv_bfloat16* o = (__nv_bfloat16*)out;
    if (d == 64) return dv == 64 ? launch_output<64, 64>(p, chunks, sums, o, eps, stream) : launch_output<64, 128>(p, chunks, sums, o, eps, stream);
    return dv == 64 ? launch_output<128, 64>(p, chunks, sums, o, eps, stream) : launch_output<128, 128>(p, chunks, sums, o, eps, stream);
}
