// A recurrent mixer with input-dependent decay (selective scan), as three kernels over a step's rows.  A step brings
// runs of consecutive tokens (prompt portions) and single tokens of several requests; what a request carries from step
// to step lives in its slot of two state tensors, both 32-bit: the last taps - 1 inputs of the short convolution and
// the recurrence's state [channels, states].
//
//  * `causal_conv`: y_t[c] = act(bias[c] + sum_j taps[c, j] x_(t - n + 1 + j)[c]) (act: SiLU or none), inputs before the
//    run taken from the slot's state, zeros before the sequence's start.  It reads the state and does not change it,
//    except in a step of single tokens only, where it can leave the new state itself.
//  * `conv_state_update`: the slot's state becomes the last taps - 1 inputs up to the end of the run.  A kernel of its
//    own, after the convolution: a run's first tokens read what its last tokens overwrite.
//  * `selective_scan`: dt = softplus(dt_raw + dt_bias);  S[c, n] <- exp(dt[c] A[c, n]) S[c, n] + dt[c] x[c] B[n];
//    y[c] = (sum_n S[c, n] C[n] + D[c] x[c]) * silu(z[c]), token by token along each run, the state read from and left
//    in the slot.  Decay, step size, exponentials and the state are 32-bit.  A channel is owned by 1 to 32 lanes, each
//    keeping up to 8 states in registers (up to 256 states).
//
// A row whose slot is negative belongs to nobody and is skipped.
#include <type_traits>

#include "common.cuh"

namespace {
constexpr int MAX_TAPS = 8;
// rows x channels of a step from which eight rows share a thread's window: below, eight times fewer threads are too few (us, a row a
// thread / eight, four taps: 100 x 2,048 4.4/5.6, 64 x 4,096 6.0/5.6, 100 x 4,096 6.2/5.7, 1,024 x 256 5.7/5.6, 300 x 2,048 8.9/6.1; two
// taps: 64 x 4,096 4.3/4.9, 100 x 4,096 4.7/4.9, 1,024 x 256 4.2/4.9, 2,048 x 256 5.5/5.0, 300 x 2,048 7.1/5.0)
constexpr long long CONV_TILED_FROM = 3 << 17;

// how many of the rows just before row t continue the same run (at most `most`)
__device__ __forceinline__ int run_before(const int* __restrict__ positions, const int* __restrict__ slots, int t,
                                          int slot, int pos, int most) {
    int m = 0;
    while (m < most && t - m - 1 >= 0 && slots[t - m - 1] == slot && positions[t - m - 1] == pos - m - 1) ++m;
    return m;
}

// input of channel c at distance k (>= 1) before row t, whose run has m rows before t
__device__ __forceinline__ float input_before(const float* __restrict__ x, long long ld, const float* state,
                                              int channels, int taps, int t, int pos, int m, int k, int c) {
    if (pos - k < 0) return 0.f;
    if (k <= m) return x[(size_t)(t - k) * ld + c];
    return state[(size_t)(taps - 1 - (k - m)) * channels + c];     // the state's last row is the input just before the run
}

template <typename TO>
__global__ void causal_conv_kernel(const float* __restrict__ x, long long ld, const float* __restrict__ taps_weight,
                                   const float* __restrict__ bias, const float* state,
                                   long long state_stride, const int* __restrict__ positions, const int* __restrict__ slots,
                                   float* __restrict__ out, TO* __restrict__ out_copy, int n_tokens, int channels,
                                   int taps, int act, float* state_out) {           // (state_out, if given, IS state)
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    if (t >= n_tokens) return;
    const int slot = slots[t];
    if (slot < 0) return;
    const int pos = positions[t];
    const int m = run_before(positions, slots, t, slot, pos, taps - 1);
    const float* own = state + (size_t)slot * state_stride;
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < channels; c += gridDim.y * blockDim.x) {
        float y = bias ? bias[c] : 0.f;
        for (int j = 0; j < taps - 1; ++j)
            y = fmaf(taps_weight[(size_t)c * taps + j], input_before(x, ld, own, channels, taps, t, pos, m, taps - 1 - j, c), y);
        y = fmaf(taps_weight[(size_t)c * taps + taps - 1], x[(size_t)t * ld + c], y);
        if (act == 1) y = y / (1.0f + expf(-y));
        out[(size_t)t * channels + c] = y;
        if (out_copy) out_copy[(size_t)t * channels + c] = from_float<TO>(y);
        if (state_out) {
            // A step of single tokens: nobody else reads this slot's state, so the thread that read a channel's inputs
            // moves them up by one and appends its own, and no second kernel runs.
            float* mine = state_out + (size_t)slot * state_stride;
            float kept[MAX_TAPS];
#pragma unroll
            for (int i = 0; i < MAX_TAPS - 1; ++i)
                if (i < taps - 1) kept[i] = i + 1 < taps - 1 ? mine[(size_t)(i + 1) * channels + c] : x[(size_t)t * ld + c];
#pragma unroll
            for (int i = 0; i < MAX_TAPS - 1; ++i)
                if (i < taps - 1) mine[(size_t)i * channels + c] = kept[i];
        }
    }
}

// The same convolution for many tokens: a thread owns four channels of CONV_ROWS neighbouring rows, asks for all of them at once
// and shifts the window of earlier inputs along; only the tile's first row, and a row that begins a run, look further back (into
// the rows before the tile, or the slot's state).  The sums are those of the kernel above, term by term.  Bound by memory: 2,048
// rows of 4,096 channels read 33 MB and write 50 (32-bit and bfloat16).
constexpr int CONV_ROWS = 8, CONV_THREADS = 128;

template <typename TO, int TAPS>
__global__ void __launch_bounds__(CONV_THREADS)
causal_conv_tile_kernel(const float* __restrict__ x, long long ld, const float* __restrict__ taps_weight,
                        const float* __restrict__ bias, const float* __restrict__ state, long long state_stride,
                        const int* __restrict__ positions, const int* __restrict__ slots, float* __restrict__ out,
                        TO* __restrict__ out_copy, int n_tokens, int channels, int act) {
    const int c = (blockIdx.x * CONV_THREADS + threadIdx.x) * 4;
    float w[4][TAPS], b[4];
    if (c < channels) {                                            // (weights wait for no one)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            b[i] = bias ? bias[c + i] : 0.f;
#pragma unroll
            for (int j = 0; j < TAPS; ++j) w[i][j] = taps_weight[(size_t)(c + i) * TAPS + j];
        }
    }
    pdl_launch_dependents();
    pdl_wait();
    if (c >= channels) return;
    const int t0 = blockIdx.y * CONV_ROWS, rows = min(CONV_ROWS, n_tokens - t0);
    float4 v[CONV_ROWS];
    int slot[CONV_ROWS], pos[CONV_ROWS];
#pragma unroll
    for (int r = 0; r < CONV_ROWS; ++r) {
        const int t = min(t0 + r, n_tokens - 1);
        v[r] = __ldg(reinterpret_cast<const float4*>(x + (size_t)t * ld + c));
        slot[r] = slots[t];
        pos[r] = positions[t];
    }
    float before[TAPS][4];                                         // [k]: the input k rows back (k >= 1)
#pragma unroll
    for (int r = 0; r < CONV_ROWS; ++r) {
        if (r >= rows) break;
        const int t = t0 + r;
        const float now[4] = {v[r].x, v[r].y, v[r].z, v[r].w};
        if (slot[r] >= 0) {
            const bool goes_on = r > 0 && slot[r > 0 ? r - 1 : 0] == slot[r] && pos[r > 0 ? r - 1 : 0] == pos[r] - 1;
            if (!goes_on && TAPS > 1) {
                const int m = run_before(positions, slots, t, slot[r], pos[r], TAPS - 1);
                const float* own = state + (size_t)slot[r] * state_stride;
#pragma unroll
                for (int k = 1; k < TAPS; ++k)
#pragma unroll
                    for (int i = 0; i < 4; ++i) before[k][i] = input_before(x, ld, own, channels, TAPS, t, pos[r], m, k, c + i);
            }
            float y[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                y[i] = b[i];
#pragma unroll
                for (int j = 0; j < TAPS - 1; ++j) y[i] = fmaf(w[i][j], before[TAPS - 1 - j][i], y[i]);
                y[i] = fmaf(w[i][TAPS - 1], now[i], y[i]);
                if (act == 1) y[i] = y[i] / (1.0f + expf(-y[i]));
            }
            *reinterpret_cast<float4*>(out + (size_t)t * channels + c) = make_float4(y[0], y[1], y[2], y[3]);
            if (out_copy) {
                struct alignas(4 * sizeof(TO)) Four { TO v[4]; } f;
#pragma unroll
                for (int i = 0; i < 4; ++i) f.v[i] = from_float<TO>(y[i]);
                *reinterpret_cast<Four*>(out_copy + (size_t)t * channels + c) = f;
            }
        }
#pragma unroll
        for (int k = TAPS - 1; k > 1; --k)
#pragma unroll
            for (int i = 0; i < 4; ++i) before[k][i] = before[k - 1][i];
        if (TAPS > 1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) before[1][i] = now[i];
        }
    }
}

__global__ void conv_state_update_kernel(const float* __restrict__ x, long long ld, float* __restrict__ state,
                                         long long state_stride, const int* __restrict__ positions, const int* __restrict__ slots, int n_tokens,
                                         int channels, int taps) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    if (t >= n_tokens) return;
    const int slot = slots[t];
    if (slot < 0) return;
    const int pos = positions[t];
    if (t + 1 < n_tokens && slots[t + 1] == slot && positions[t + 1] == pos + 1) return;      // not the run's last row
    const int m = run_before(positions, slots, t, slot, pos, taps - 1);
    float* own = state + (size_t)slot * state_stride;
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < channels; c += gridDim.y * blockDim.x) {
        float kept[MAX_TAPS];
#pragma unroll
        for (int i = 0; i < MAX_TAPS - 1; ++i) {
            if (i < taps - 1) {
                const int k = taps - 2 - i;                     // row i of the new state lies k inputs before this row's
                kept[i] = k == 0 ? x[(size_t)t * ld + c] : input_before(x, ld, own, channels, taps, t, pos, m, k, c);
            }
        }
#pragma unroll
        for (int i = 0; i < MAX_TAPS - 1; ++i)
            if (i < taps - 1) own[(size_t)i * channels + c] = kept[i];
    }
}

constexpr int SCAN_THREADS = 64;
constexpr int STATES_PER_LANE = 8;

__device__ __forceinline__ float softplus(float v) { return v > 20.f ? v : log1pf(expf(v)); }

constexpr int CHUNK = 64;             // tokens of a long run that one CTA walks when the run is cut

struct ScanArgs {
    const float* x; const float* dt_raw; const float* dt_bias; const float* A; const float* bc; long long ld_bc;
    int b_offset, c_offset;
    const float* D; const float* z; long long ld_z;
    float* state; long long state_stride;
    const int* segments; int n_segments; const int* single_rows; int n_single; const int* slots;
    void* out; int channels, states;
    float* chunk_state;               // [chunks][channels][states]: a chunk's end state from zero, later its start state
    float* chunk_dt;                  // [chunks][channels]: the sum of a chunk's step sizes
};

// Walks rows first .. first + count - 1 of one run for this thread's channel and states.  Tokens in groups of AHEAD:
// everything a group reads is asked for before its first token is computed, so that only the recurrence itself (an
// exponential and a multiply-add per state) lies between one token and the next.  Returns the sum of the step sizes.
template <typename TO, int LPC, bool OUTPUT>
__device__ __forceinline__ float walk(const ScanArgs& p, int first, int count, int cc, int sub, bool live,
                                      float (&S)[STATES_PER_LANE], const float (&a)[STATES_PER_LANE]) {
    const int channels = p.channels, states = p.states;
    const float bias = p.dt_bias[cc], skip = p.D[cc];
    TO* out = reinterpret_cast<TO*>(p.out);
    float dt_sum = 0.f;
    constexpr int AHEAD = 4;
    for (int r0 = 0; r0 < count; r0 += AHEAD) {
        float xv[AHEAD], dtv[AHEAD], gv[AHEAD], bv[AHEAD][STATES_PER_LANE], cv[AHEAD][STATES_PER_LANE];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const bool there = r0 + u < count;
            const size_t t = (size_t)first + (there ? r0 + u : r0);
            xv[u] = p.x[t * channels + cc];
            dtv[u] = p.dt_raw[t * channels + cc];
            if (OUTPUT) gv[u] = p.z[t * p.ld_z + cc];
            const float* b = p.bc + t * p.ld_bc + p.b_offset;
            const float* cvec = p.bc + t * p.ld_bc + p.c_offset;
#pragma unroll
            for (int i = 0; i < STATES_PER_LANE; ++i) {
                const int n = sub + i * LPC;
                bv[u][i] = n < states ? b[n] : 0.f;
                if (OUTPUT) cv[u][i] = n < states ? cvec[n] : 0.f;
            }
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            if (r0 + u >= count) break;
            const size_t t = (size_t)first + r0 + u;
            const float dt = softplus(dtv[u] + bias);
            const float dx = dt * xv[u];
            dt_sum += dt;
            float y = 0.f;
#pragma unroll
            for (int i = 0; i < STATES_PER_LANE; ++i) {
                if (sub + i * LPC < states) {
                    S[i] = fmaf(expf(dt * a[i]), S[i], dx * bv[u][i]);
                    if (OUTPUT) y = fmaf(S[i], cv[u][i], y);
                }
            }
            if (OUTPUT) {
#pragma unroll
                for (int o = LPC / 2; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
                if (live && sub == 0) out[t * channels + cc] = from_float<TO>((y + skip * xv[u]) * (gv[u] / (1.0f + expf(-gv[u]))));
            }
        }
    }
    return dt_sum;
}

// The chunk of the cut runs that CTA `id` serves: (first row, rows, first row of its run), or rows 0 if there is none.
__device__ __forceinline__ void chunk_of(const ScanArgs& p, int id, int& first, int& count, int& run_first) {
    count = 0;
    for (int s = 0; s < p.n_segments; ++s) {
        const int seg_first = p.segments[3 * s], seg_count = p.segments[3 * s + 2];
        const int chunks = (seg_count + CHUNK - 1) / CHUNK;
        if (id < chunks) {
            first = seg_first + id * CHUNK;
            count = min(CHUNK, seg_count - id * CHUNK);
            run_first = seg_first;
            return;
        }
        id -= chunks;
    }
}

// MODE 0: whole runs (grid x: the portions, then the single tokens), state read from and left in the slot.
// MODE 1: chunks of the portions from a zero state; leaves each chunk's end state and the sum of its step sizes.
// MODE 2: chunks of the portions from the start states that `scan_carry_kernel` left; writes the outputs.
template <typename TO, int LPC, int MODE>
__global__ void __launch_bounds__(SCAN_THREADS)
selective_scan_kernel(ScanArgs p) {
    pdl_launch_dependents();
    pdl_wait();
    int first = 0, count = 0, run_first = 0;
    if (MODE == 0) {
        if ((int)blockIdx.x < p.n_segments) {
            first = p.segments[3 * blockIdx.x];
            count = p.segments[3 * blockIdx.x + 2];
        } else {
            first = p.single_rows[blockIdx.x - p.n_segments];
            count = 1;
        }
        run_first = first;
    } else {
        chunk_of(p, blockIdx.x, first, count, run_first);
    }
    if (first < 0 || count <= 0) return;
    const int slot = p.slots[run_first];
    if (slot < 0) return;
    const int sub = threadIdx.x % LPC;
    const int c = blockIdx.y * (SCAN_THREADS / LPC) + threadIdx.x / LPC;
    const bool live = c < p.channels;
    const int cc = live ? c : 0;
    float S[STATES_PER_LANE], a[STATES_PER_LANE];
    float* own = MODE == 0 ? p.state + (size_t)slot * p.state_stride + (size_t)cc * p.states
                           : p.chunk_state + ((size_t)blockIdx.x * p.channels + cc) * p.states;
#pragma unroll
    for (int i = 0; i < STATES_PER_LANE; ++i) {
        const int n = sub + i * LPC;
        S[i] = (MODE != 1 && live && n < p.states) ? own[n] : 0.f;
        a[i] = (live && n < p.states) ? p.A[(size_t)cc * p.states + n] : 0.f;
    }
    const float dt_sum = walk<TO, LPC, MODE != 1>(p, first, count, cc, sub, live, S, a);
    if (live && MODE != 2) {
#pragma unroll
        for (int i = 0; i < STATES_PER_LANE; ++i) {
            const int n = sub + i * LPC;
            if (n < p.states) own[n] = S[i];
        }
        if (MODE == 1 && sub == 0) p.chunk_dt[(size_t)blockIdx.x * p.channels + cc] = dt_sum;
    }
}

// Between the two chunked passes: along each portion, the state at the start of every chunk (in place of the chunk's
// end state from zero), S <- exp(A sum(dt)) S + end, beginning with the slot's state; the last one is the slot's new state.
template <int LPC>
__global__ void __launch_bounds__(SCAN_THREADS)
scan_carry_kernel(ScanArgs p) {
    pdl_launch_dependents();
    pdl_wait();
    int base = 0;
    for (int s = 0; s < (int)blockIdx.x; ++s) base += (p.segments[3 * s + 2] + CHUNK - 1) / CHUNK;
    const int run_first = p.segments[3 * blockIdx.x];
    const int chunks = (p.segments[3 * blockIdx.x + 2] + CHUNK - 1) / CHUNK;
    const int slot = p.slots[run_first];
    if (slot < 0) return;
    const int sub = threadIdx.x % LPC;
    const int c = blockIdx.y * (SCAN_THREADS / LPC) + threadIdx.x / LPC;
    if (c >= p.channels) return;
    float* own = p.state + (size_t)slot * p.state_stride + (size_t)c * p.states;
    float S[STATES_PER_LANE], a[STATES_PER_LANE];
#pragma unroll
    for (int i = 0; i < STATES_PER_LANE; ++i) {
        const int n = sub + i * LPC;
        S[i] = n < p.states ? own[n] : 0.f;
        a[i] = n < p.states ? p.A[(size_t)c * p.states + n] : 0.f;
    }
    for (int k = 0; k < chunks; ++k) {
        float* at = p.chunk_state + ((size_t)(base + k) * p.channels + c) * p.states;
        const float dt_sum = p.chunk_dt[(size_t)(base + k) * p.channels + c];
#pragma unroll
        for (int i = 0; i < STATES_PER_LANE; ++i) {
            const int n = sub + i * LPC;
            if (n < p.states) {
                const float end = at[n];
                at[n] = S[i];
                S[i] = fmaf(expf(a[i] * dt_sum), S[i], end);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < STATES_PER_LANE; ++i) {
        const int n = sub + i * LPC;
        if (n < p.states) own[n] = S[i];
    }
}
// Whole portions of up to 64 states a channel, walked once: sixteen lanes own a channel, SPL neighbouring states each, and a CTA
// eight channels of one portion.  The rows of 32 tokens (x, step size, gate of the eight channels, B and C of all states) lie in
// shared memory and the next 32 are on their way.  Every lane forms the step sizes of every sixteenth token, side by side, and
// hands them round through shared memory; behind a group of sixteen tokens' recurrence (per state: an exponential, two
// multiply-adds) the sixteen sums over the lanes' states meet so that every lane is left with one token's, whose skip, gate and
// store are its own: what is not the recurrence is done once per token and channel.
// A token costs its exponentials: 2,048 tokens x 4,096 channels x 16 states are 134 M, 40 us of issue over the device with the
// multiply-adds around them.  Cutting the portions into chunks (below, for other sizes) does each of them twice, and one that
// reads B and C from memory per thread spends more on the loads: 539 us for the same tokens.
// With `conv_state` the CTA also leaves its channels' last taps - 1 inputs there (the convolution has long read them).
constexpr int RUN_CHANNELS = 8, RUN_LANES = 16, RUN_TOKENS = 32, RUN_THREADS = RUN_CHANNELS * RUN_LANES;

struct ConvTail {
    float* state; long long state_stride;           // null: nothing to leave
    const float* x; long long ld; int taps;
};

template <typename TO, int SPL>
__global__ void __launch_bounds__(RUN_THREADS)
scan_run_kernel(ScanArgs p, ConvTail tail) {
    constexpr int GROUP = RUN_LANES, GROUPS = RUN_TOKENS / GROUP;         // a token of a group a lane
    struct __align__(16) Stage {
        float x[RUN_TOKENS][RUN_CHANNELS], dt[RUN_TOKENS][RUN_CHANNELS], z[RUN_TOKENS][RUN_CHANNELS];
        float bc[RUN_TOKENS][RUN_LANES][2 * SPL];            // a lane's B and then its C
    };
    __shared__ Stage stages[2];
    __shared__ __align__(16) float steps[RUN_CHANNELS][RUN_TOKENS][2];       // step size, step size times input
    __shared__ __align__(16) TO results[RUN_TOKENS][RUN_CHANNELS];
    pdl_launch_dependents();
    pdl_wait();
    const int first = p.segments[3 * blockIdx.y], start = p.segments[3 * blockIdx.y + 1], count = p.segments[3 * blockIdx.y + 2];
    if (first < 0 || count <= 0) return;
    const int slot = p.slots[first];
    if (slot < 0) return;
    const int tid = threadIdx.x, lane = tid % RUN_LANES, ch = tid / RUN_LANES, c0 = blockIdx.x * RUN_CHANNELS, c = c0 + ch;
    const int states = p.states;
    // (channels and states are multiples of four: a piece of four lies inside or outside)
    auto fetch = [&](int t0, int buffer) {
        Stage& s = stages[buffer];
        auto bring = [&](float* dst, const float* src, bool there) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                         "r"(there ? 16 : 0) : "memory");
        };
        if (tid < 2 * RUN_TOKENS) {
            const int r = tid >> 1, piece = (tid & 1) * 4;
            const bool there = t0 + r < count && c0 + piece < p.channels;
            const size_t t = (size_t)first + (there ? t0 + r : 0);
            const int column = there ? c0 + piece : 0;
            bring(&s.x[r][piece], p.x + t * p.channels + column, there);
            bring(&s.dt[r][piece], p.dt_raw + t * p.channels + column, there);
            bring(&s.z[r][piece], p.z + t * p.ld_z + column, there);
        }
        // a lane's B (and its C) of a token: SPL elements, in pieces of at most 16 bytes
        constexpr int PIECE = SPL < 4 ? SPL : 4, PER = SPL / PIECE;
#pragma unroll
        for (int e = tid; e < RUN_TOKENS * RUN_LANES * 2 * PER; e += RUN_THREADS) {
            const int part = e % PER, l = (e / PER) % RUN_LANES, which = (e / (PER * RUN_LANES)) & 1, r = e / (PER * RUN_LANES * 2);
            const int column = l * SPL + part * PIECE;
            const bool there = t0 + r < count && column < states;
            const float* src = p.bc + ((size_t)first + (there ? t0 + r : 0)) * p.ld_bc + (which ? p.c_offset : p.b_offset) + (there ? column : 0);
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::
                         "r"((uint32_t)__cvta_generic_to_shared(&s.bc[r][l][which * SPL + part * PIECE])), "l"(src), "n"(PIECE * 4),
                         "r"(there ? PIECE * 4 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0, 0);
    const bool live = c < p.channels;
    const int cc = live ? c : 0;
    const float bias = p.dt_bias[cc], skip = p.D[cc];
    float* own = p.state + (size_t)slot * p.state_stride + (size_t)cc * states + lane * SPL;
    float S[SPL], a[SPL];
#pragma unroll
    for (int i = 0; i < SPL; ++i) {
        const bool there = live && lane * SPL + i < states;
        S[i] = there ? own[i] : 0.f;
        a[i] = there ? p.A[(size_t)cc * states + lane * SPL + i] : 0.f;
    }
    if (tail.state && live && lane == 0) {
        // row i of the new state lies taps - 2 - i inputs before the run's last; rows before the run come from the old state, zeros
        // before the sequence's start
        float kept[MAX_TAPS];
        float* mine = tail.state + (size_t)slot * tail.state_stride + c;
#pragma unroll
        for (int i = 0; i < MAX_TAPS - 1; ++i) {
            if (i < tail.taps - 1) {
                const int r = count - 1 - (tail.taps - 2 - i);
                kept[i] = start + r < 0 ? 0.f : r >= 0 ? tail.x[((size_t)first + r) * tail.ld + c] : mine[(size_t)(i + count) * p.channels];
            }
        }
#pragma unroll
        for (int i = 0; i < MAX_TAPS - 1; ++i)
            if (i < tail.taps - 1) mine[(size_t)i * p.channels] = kept[i];
    }
    int buffer = 0;
    for (int t0 = 0; t0 < count; t0 += RUN_TOKENS, buffer ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                     // these tokens are there, the ones before and their results are done with
        if (t0 + RUN_TOKENS < count) fetch(t0 + RUN_TOKENS, buffer ^ 1);
        const Stage& s = stages[buffer];
        const bool full = t0 + RUN_TOKENS <= count;
        // step sizes: a token of every group a lane, side by side (a chain of some hundred cycles each)
        float xv[GROUPS];
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            xv[g] = s.x[g * GROUP + lane][ch];
            const float dt = softplus(s.dt[g * GROUP + lane][ch] + bias);
            *reinterpret_cast<float2*>(steps[ch][g * GROUP + lane]) = make_float2(dt, dt * xv[g]);
        }
        __syncwarp();
        float sum[GROUPS];
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            float y[GROUP];
            auto recur = [&](auto whole) {
#pragma unroll
                for (int u = 0; u < GROUP; u += 2) {
                    const float4 step = *reinterpret_cast<const float4*>(steps[ch][g * GROUP + u]);
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        const float dtu = v ? step.z : step.x, dxu = v ? step.w : step.y;
                        float bc[2 * SPL];
                        if constexpr (SPL >= 2) {
#pragma unroll
                            for (int i = 0; i < 2 * SPL; i += 4) {
                                const float4 four = *reinterpret_cast<const float4*>(&s.bc[g * GROUP + u + v][lane][i]);
                                bc[i] = four.x, bc[i + 1] = four.y, bc[i + 2] = four.z, bc[i + 3] = four.w;
                            }
                        } else {
                            const float2 pair = *reinterpret_cast<const float2*>(s.bc[g * GROUP + u + v][lane]);
                            bc[0] = pair.x, bc[1] = pair.y;
                        }
                        y[u + v] = 0.f;
                        if (!decltype(whole)::value && t0 + g * GROUP + u + v >= count) continue;
#pragma unroll
                        for (int i = 0; i < SPL; ++i) {
                            S[i] = fmaf(expf(dtu * a[i]), S[i], dxu * bc[i]);
                            y[u + v] = fmaf(S[i], bc[SPL + i], y[u + v]);
                        }
                    }
                }
            };
            if (full) recur(std::true_type{});
            else recur(std::false_type{});
            // as many sums as lanes: at every turn a lane keeps half of its tokens and hands the other half on
#pragma unroll
            for (int half = GROUP / 2; half > 0; half >>= 1) {
#pragma unroll
                for (int u = 0; u < half; ++u) {
                    const float mine = lane & half ? y[u + half] : y[u], other = lane & half ? y[u] : y[u + half];
                    y[u] = mine + __shfl_xor_sync(0xffffffffu, other, half);
                }
            }
            sum[g] = y[0];
        }
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            const float zv = s.z[g * GROUP + lane][ch];
            results[g * GROUP + lane][ch] = from_float<TO>((sum[g] + skip * xv[g]) * (zv / (1.0f + expf(-zv))));
        }
        __syncthreads();
        // a token's eight results lie side by side
        constexpr int PER = 16 / (int)sizeof(TO), PIECES = RUN_CHANNELS / PER;
        TO* out = reinterpret_cast<TO*>(p.out);
        if (tid < RUN_TOKENS * PIECES) {
            const int r = tid / PIECES, piece = (tid % PIECES) * PER;
            if (t0 + r < count) {
                TO* dst = out + ((size_t)first + t0 + r) * p.channels + c0 + piece;
                if (c0 + RUN_CHANNELS <= p.channels && p.channels % PER == 0) {
                    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(&results[r][piece]);
                } else {
                    for (int i = 0; i < PER; ++i)
                        if (c0 + piece + i < p.channels) dst[i] = results[r][piece + i];
                }
            }
        }
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < SPL; ++i)
            if (lane * SPL + i < states) own[i] = S[i];
    }
}
}  // namespace

// x [n, ld] 32-bit (the first `channels` columns), taps_weight [channels, taps], bias [channels] or null,
// state (slot s at state + s state_stride: [taps - 1, channels]), all 32-bit.  out [n, channels] 32-bit; out_copy (optional) the same in `copy_dtype`.
LIA_EXPORT int lia_causal_conv(const float* x, long long ld, const float* taps_weight, const float* bias,
                               const float* state, long long state_stride, const int* positions, const int* slots,
                               float* out, void* out_copy,
                               int copy_dtype, int n_tokens, int channels, int taps, int act, int update_single,
                               cudaStream_t stream) {
    if (n_tokens <= 0) return LIA_OK;
    if (channels <= 0 || taps < 1 || taps > MAX_TAPS || ld < channels || (taps > 1 && !state) || act < 0 || act > 1)
        return LIA_ERR_SIZE;
    const size_t copy_size = copy_dtype == LIA_BF16 ? 2 : 4;
    if (!update_single && (long long)n_tokens * channels >= CONV_TILED_FROM && taps >= 2 && taps <= 4 && channels % 4 == 0 && ld % 4 == 0 &&
        (((uintptr_t)x | (uintptr_t)out) & 15u) == 0 && ((uintptr_t)out_copy & (4 * copy_size - 1)) == 0 &&
        (n_tokens + CONV_ROWS - 1) / CONV_ROWS <= 65535) {
        const dim3 tiles((channels / 4 + CONV_THREADS - 1) / CONV_THREADS, (n_tokens + CONV_ROWS - 1) / CONV_ROWS);
#define LIA_CONV(TO, TAPS)                                                                                              \
    return lia_launch(causal_conv_tile_kernel<TO, TAPS>, tiles, dim3(CONV_THREADS), 0, stream, x, ld, taps_weight, bias, state, \
                      state_stride, positions, slots, out, (TO*)out_copy, n_tokens, channels, act)
        if (!out_copy || copy_dtype == LIA_F32) {
            if (taps == 2) LIA_CONV(float, 2);
            if (taps == 3) LIA_CONV(float, 3);
            LIA_CONV(float, 4);
        }
        if (copy_dtype == LIA_BF16) {
            if (taps == 2) LIA_CONV(__nv_bfloat16, 2);
            if (taps == 3) LIA_CONV(__nv_bfloat16, 3);
            LIA_CONV(__nv_bfloat16, 4);
        }
#undef LIA_CONV
        return LIA_ERR_DTYPE;
    }
    const int threads = 128;
    // few tokens: a token's channels over several CTAs, so that the step's rows fill the device
    const dim3 grid(n_tokens, n_tokens >= 512 ? 1 : min(16, (channels + threads - 1) / threads));
    // `update_single`: every run of the step is a single token; the kernel then leaves the new state itself
    float* state_out = (update_single && taps > 1) ? const_cast<float*>(state) : nullptr;
    if (!out_copy || copy_dtype == LIA_F32)
        return lia_launch(causal_conv_kernel<float>, grid, dim3(threads), 0, stream, x, ld, taps_weight, bias,
                          state, state_stride, positions, slots, out, (float*)out_copy, n_tokens, channels, taps, act,
                          state_out);
    if (copy_dtype == LIA_BF16)
        return lia_launch(causal_conv_kernel<__nv_bfloat16>, grid, dim3(threads), 0, stream, x, ld, taps_weight,
                          bias, state, state_stride, positions, slots, out, (__nv_bfloat16*)out_copy, n_tokens, channels,
                          taps, act, state_out);
    return LIA_ERR_DTYPE;
}

LIA_EXPORT int lia_conv_state_update(const float* x, long long ld, float* state, long long state_stride,
                                     const int* positions, const int* slots, int n_tokens, int channels, int taps, cudaStream_t stream) {
    if (n_tokens <= 0 || taps <= 1) return LIA_OK;
    if (channels <= 0 || taps > MAX_TAPS || ld < channels || !state) return LIA_ERR_SIZE;
    const int threads = 128;
    const dim3 grid(n_tokens, n_tokens >= 512 ? 1 : min(16, (channels + threads - 1) / threads));
    return lia_launch(conv_state_update_kernel, grid, dim3(threads), 0, stream, x, ld, state, state_stride,
                      positions, slots, n_tokens, channels, taps);
}

// x, dt_raw [n, channels]; dt_bias, D [channels]; A [channels, states] (negative: the decay's rate); bc [n, ld_bc] with B
// at column b_offset and C at c_offset (`states` each); z [n, ld_z]; state (slot s at state + s state_stride:
// [channels, states]): all 32-bit.  segments [n_segments, 3] (first row, first position, count) and single_rows
// [n_single] name the step's runs.  out [n, channels] of `out_dtype`.
// `chunk_scratch` (32-bit, `chunk_floats` words; may be null): with it, and portions in the step, the portions are cut
// into chunks of 64 tokens that run side by side (a pass from zero states, a carry along each portion, a pass from the
// true start states); it must hold lia_selective_scan_chunk_floats(n_tokens, n_segments, channels, states) words.
// Without it every run is walked by one CTA per block of channels.
LIA_EXPORT long long lia_selective_scan_chunk_floats(int n_tokens, int n_segments, int channels, int states) {
    const long long chunks = (long long)n_tokens / CHUNK + n_segments;
    return chunks * channels * (states + 1);
}

namespace {
template <typename TO, int LPC>
int launch_scan(ScanArgs p, int n_tokens, bool chunked, cudaStream_t stream) {
    const int per_block = SCAN_THREADS / LPC;
    const unsigned blocks_y = (p.channels + per_block - 1) / per_block;
    if (blocks_y > 65535) return LIA_ERR_SIZE;
    if (!chunked) {
        const dim3 grid(p.n_segments + p.n_single, blocks_y);
        return lia_launch(selective_scan_kernel<TO, LPC, 0>, grid, dim3(SCAN_THREADS), 0, stream, p);
    }
    int rc = LIA_OK;
    if (p.n_single > 0) {                                   // the single tokens: whole runs, as ever
        ScanArgs q = p;
        q.n_segments = 0;
        rc = lia_launch(selective_scan_kernel<TO, LPC, 0>, dim3(p.n_single, blocks_y), dim3(SCAN_THREADS), 0, stream, q);
        if (rc != LIA_OK) return rc;
    }
    const dim3 chunks(n_tokens / CHUNK + p.n_segments, blocks_y);        // as many as the portions can have at most
    rc = lia_launch(selective_scan_kernel<TO, LPC, 1>, chunks, dim3(SCAN_THREADS), 0, stream, p);
    if (rc != LIA_OK) return rc;
    rc = lia_launch(scan_carry_kernel<LPC>, dim3(p.n_segments, blocks_y), dim3(SCAN_THREADS), 0, stream, p);
    if (rc != LIA_OK) return rc;
    return lia_launch(selective_scan_kernel<TO, LPC, 2>, chunks, dim3(SCAN_THREADS), 0, stream, p);
}
}  // namespace

namespace {
template <typename TO>
int launch_runs(const ScanArgs& p, const ConvTail& tail, cudaStream_t stream) {
    const dim3 grid((p.channels + RUN_CHANNELS - 1) / RUN_CHANNELS, p.n_segments);
    // (launched the ordinary way: CTAs that begin under the product ahead, whose own CTAs fill most SMs' shared memory, would all
    // gather on the few SMs that it leaves free and stay there; 2,048 tokens of a whole layer took 603 us so, 343 in turn)
    if (p.states <= 16) return lia_launch_in_turn(scan_run_kernel<TO, 1>, grid, dim3(RUN_THREADS), 0, stream, p, tail);
    if (p.states <= 32) return lia_launch_in_turn(scan_run_kernel<TO, 2>, grid, dim3(RUN_THREADS), 0, stream, p, tail);
    return lia_launch_in_turn(scan_run_kernel<TO, 4>, grid, dim3(RUN_THREADS), 0, stream, p, tail);
}
}  // namespace

namespace {
bool run_sizes(const void* x, const void* dt_raw, const void* bc, long long ld_bc, int b_offset, int c_offset, const void* z, long long ld_z,
               const void* out, int channels, int states) {
    return channels > 0 && states > 0 && states <= 64 && ((channels | states | b_offset | c_offset) & 3) == 0 && ((ld_bc | ld_z) & 3) == 0 &&
           (((uintptr_t)x | (uintptr_t)dt_raw | (uintptr_t)bc | (uintptr_t)z | (uintptr_t)out) & 15u) == 0;
}

// Which way the portions go where all are open (`tokens` of them in `portions` portions; us on a B200, the run kernel beside the other).
// Short ones, under eight tokens on average: the kernel for every size, which takes the step's single tokens in the same launch, where
// there are any or where the run kernel's CTAs are more than one round (3 tokens and 32 single ones, 16 states: 7.1 beside 4.4 at 256
// channels, 17.7 beside 13.9 at 4,096; 4 x 3 tokens of 4,096 channels 11.6 beside 5.6; 8 tokens and 32 single ones 7.3 beside 7.4).
// Long ones of few channels: the run kernel's time is a chain, that of one token times the tokens, while the device is nearly idle, and
// chunks side by side are faster.  Both times are estimated: a run's as its chain or the device's rate, whichever is longer; the chunks' as
// their launches and their chains of 64 tokens, and a rate.  2,048 tokens of 256 channels and 4 / 16 / 32 / 64 states: 89 beside 77, 89
// beside 107, 119 beside 126, 193 beside 132; 4,096 tokens of them 175 beside 101, 145, 153, 235; of 1,024 channels 175 beside 132 with 4
// states and 175 beside 241 with 16; 2,048 tokens of 4,096 channels and 16 states 164 beside 406.  Over 756 sizes (128 to 4,096
// channels, 4 to 64 states, 256 to 8,192 tokens in one to four portions) the choice costs more than 4% in seven, 18% at most.
enum ScanRoute { SCAN_WHOLE, SCAN_RUNS, SCAN_CHUNKS };
ScanRoute scan_route(int channels, int states, int tokens, int portions, int n_single) {
    if (portions <= 0) return SCAN_WHOLE;
    if (tokens < 8 * portions && (n_single > 0 || (long long)channels * portions > 8192)) return SCAN_WHOLE;
    const int wide = states <= 16 ? 0 : states <= 32 ? 1 : 2;                     // states a lane: 1, 2 or 4
    constexpr float CHAIN[3] = {0.0432f, 0.0578f, 0.0943f}, RATE[3] = {1.96e-5f, 2.75e-5f, 4.7e-5f};
    const float n = (float)tokens, width = (float)channels;
    const float runs = fmaxf(n / (float)portions * CHAIN[wide], n * width * RATE[wide]);
    const float chunks = (states <= 4 ? 50.f : 75.f) + n * (0.005f + width * (9e-6f + 2e-6f * (float)states));
    return runs > chunks ? SCAN_CHUNKS : SCAN_RUNS;
}
}  // namespace

// 1 if the kernel that walks whole portions serves these (at most 64 states, every row's pieces of four elements aligned, and faster
// than the others for a step of `n_tokens` rows, `n_single` of them single tokens, in `n_segments` portions).
LIA_EXPORT int lia_selective_scan_walks_runs(const void* x, const void* dt_raw, const void* bc, long long ld_bc, int b_offset,
                                             int c_offset, const void* z, long long ld_z, const void* out, int channels, int states,
                                             int n_tokens, int n_segments, int n_single) {
    return run_sizes(x, dt_raw, bc, ld_bc, b_offset, c_offset, z, ld_z, out, channels, states) &&
                   scan_route(channels, states, n_tokens - n_single, n_segments, n_single) == SCAN_RUNS
               ? 1 : 0;
}

// `conv_state` (or null; slot s at conv_state + s conv_stride: [taps - 1, channels]): the portions leave their last taps - 1 inputs
// there, read from conv_x [n, conv_ld]; only where lia_selective_scan_walks_runs says yes and the step has no single tokens.  Without
// chunk_scratch no portion is cut into chunks.
LIA_EXPORT int lia_selective_scan(const float* x, const float* dt_raw, const float* dt_bias, const float* A,
                                  const float* bc, long long ld_bc, int b_offset, int c_offset, const float* D,
                                  const float* z, long long ld_z, float* state, long long state_stride,
                                  const int* segments, int n_segments,
                                  const int* single_rows, int n_single, const int* slots, void* out, int out_dtype,
                                  int channels, int states, int n_tokens, float* chunk_scratch, long long chunk_floats,
                                  float* conv_state, long long conv_stride, const float* conv_x, long long conv_ld, int taps,
                                  cudaStream_t stream) {
    const int runs = n_segments + n_single;
    if (runs <= 0) return LIA_OK;
    if ((conv_state && (!conv_x || taps < 2 || taps > MAX_TAPS || n_single > 0)) || n_segments > 65535) return LIA_ERR_SIZE;
    if (channels <= 0 || states <= 0 || states > 32 * STATES_PER_LANE || n_segments < 0 || n_single < 0 ||
        ld_bc < b_offset + states || ld_bc < c_offset + states || ld_z < channels || n_tokens < n_single + 2 * n_segments)
        return LIA_ERR_SIZE;
    bool chunked = chunk_scratch && n_segments > 0;
    if (chunked && chunk_floats < lia_selective_scan_chunk_floats(n_tokens, n_segments, channels, states)) return LIA_ERR_SIZE;
    ScanArgs p;
    p.x = x; p.dt_raw = dt_raw; p.dt_bias = dt_bias; p.A = A; p.bc = bc; p.ld_bc = ld_bc; p.b_offset = b_offset;
    p.c_offset = c_offset; p.D = D; p.z = z; p.ld_z = ld_z; p.state = state; p.state_stride = state_stride;
    p.segments = segments; p.n_segments = n_segments; p.single_rows = single_rows; p.n_single = n_single; p.slots = slots;
    p.out = out; p.channels = channels; p.states = states;
    p.chunk_state = chunk_scratch;
    p.chunk_dt = chunk_scratch ? chunk_scratch + ((long long)n_tokens / CHUNK + n_segments) * channels * states : nullptr;
    const bool open = n_segments > 0 && run_sizes(x, dt_raw, bc, ld_bc, b_offset, c_offset, z, ld_z, out, channels, states);
    const ScanRoute route = scan_route(channels, states, n_tokens - n_single, n_segments, n_single);
    if (open && route == SCAN_WHOLE) chunked = false;
    if (open && (conv_state || route == SCAN_RUNS || (route == SCAN_CHUNKS && !chunked))) {
        const int rc = out_dtype == LIA_F32 ? launch_runs<float>(p, {conv_state, conv_stride, conv_x, conv_ld, taps}, stream)
                     : out_dtype == LIA_BF16 ? launch_runs<__nv_bfloat16>(p, {conv_state, conv_stride, conv_x, conv_ld, taps}, stream)
                                             : LIA_ERR_DTYPE;
        if (rc != LIA_OK || n_single <= 0) return rc;
        p.n_segments = 0;
        chunked = false;
    } else if (conv_state) {
        return LIA_ERR_SIZE;
    }
    int lpc = 1;
    while (lpc * STATES_PER_LANE < states) lpc *= 2;
#define LIA_SCAN_LANES(TO)                                                     \
    switch (lpc) {                                                             \
        case 1: return launch_scan<TO, 1>(p, n_tokens, chunked, stream);       \
        case 2: return launch_scan<TO, 2>(p, n_tokens, chunked, stream);       \
        case 4: return launch_scan<TO, 4>(p, n_tokens, chunked, stream);       \
        case 8: return launch_scan<TO, 8>(p, n_tokens, chunked, stream);       \
        case 16: return launch_scan<TO, 16>(p, n_tokens, chunked, stream);     \
        default: return launch_scan<TO, 32>(p, n_tokens, chunked, stream);     \
    }
    if (out_dtype == LIA_F32) LIA_SCAN_LANES(float)
    if (out_dtype == LIA_BF16) LIA_SCAN_LANES(__nv_bfloat16)
#undef LIA_SCAN_LANES
    return LIA_ERR_DTYPE;
}
