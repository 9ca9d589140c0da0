// The selective scan of the first Mamba mixer: a state vector per channel, with its state in the request's slot.
//
// Per channel c and state entry n, with dt_t[c] = softplus(step_t[c]) (the step projection's result with its bias) and
// A[c][n] = -exp(A_log[c][n]) formed once when the weights are loaded:
//
//     S[c][n] <- exp(dt_t[c] A[c][n]) S[c][n] + dt_t[c] x_t[c] B_t[n]
//     y_t[c]  =  sum_n S[c][n] C_t[n] + D[c] x_t[c],        out_t[c] = y_t[c] * silu(z_t[c])
//
// SL lanes share a channel and hold NR state entries each; a block owns SCAN_CHANNELS channels of one request and
// walks the request's new tokens in order; a token's B and C are staged once for all of the block's channels, and the
// next tile's inputs are loaded into registers while the current one is worked on.  The
// step size, the decay, the state and the sums are float32 whatever the activation dtype.  State row of a slot:
// [inner][state] (state fastest) at the row's start.
//
// A long portion is cut into chunks that run side by side (the recurrence is diagonal): a first pass runs every chunk
// from a zero state and leaves its end state L_c and the sum of its steps in a workspace; `selective_combine` walks a
// request's chunks in order, S <- exp(A sum_c dt) S + L_c, leaves in the workspace the state each chunk starts from
// and writes the slot; a second pass runs every chunk from there and writes the outputs.
#include "common.cuh"

namespace lily {

constexpr int SL = 8;                   // lanes that share a channel
constexpr int SCAN_TOKENS = 16;         // tokens staged at a time
constexpr int SCAN_THREADS = 128;
constexpr int SCAN_CHANNELS = SCAN_THREADS / SL;

struct SelectiveArgs {
    const void* x;            // [tokens, inner]: the convolved and activated inputs
    const void* low;          // [tokens, low_stride]: B at b_col, C at c_col (n_state columns each)
    int low_stride, b_col, c_col;
    const float* step;        // [tokens, inner]: W_dt . + bias, before softplus
    const void* z;            // [tokens, z_stride]: the gate's columns start at z_col
    int z_stride, z_col;
    const float* A;           // [inner, n_state]
    const float* D;           // [inner]
    float* state;             // [slots, state_stride]
    size_t state_stride;
    void* out;                // [tokens, inner]
    const int* cu_seqlens;
    const int* slots;
    int inner, n_state;
    // the work of block x: request work_req[x] (null: request x), its tokens [work_start[x], + work_len[x]) (null: all)
    const int* work_req;
    const int* work_start;
    const int* work_len;
    int mode;                 // 0: from and to the slot; 1: chunk x from zero, end state and sum of steps to the workspace,
                              // no outputs; 2: chunk x from the workspace's state, outputs, no state written
    float* ws_state;          // [chunks][inner][n_state]
    float* ws_steps;          // [chunks][inner]
};

// grid (requests, ceil(inner / SCAN_CHANNELS)), block SCAN_THREADS; n_state <= SL * NR
// AHEAD: a tile's inputs are loaded one tile ahead (portions of prompts); without it they are loaded when their turn
// comes, which keeps fewer registers alive (steps in which every request brings one token).
template <typename T, int NR, bool AHEAD>
__global__ void __launch_bounds__(SCAN_THREADS) selective_scan_kernel(const SelectiveArgs a) {
    constexpr int SP = SL * NR;
    __shared__ float Bs[SCAN_TOKENS][SP], Cs[SCAN_TOKENS][SP];
    __shared__ float dts[SCAN_TOKENS][SCAN_CHANNELS], xs[SCAN_TOKENS][SCAN_CHANNELS], zs[SCAN_TOKENS][SCAN_CHANNELS],
        ys[SCAN_TOKENS][SCAN_CHANNELS];
    pdl_enter_small();
    const int req = a.work_req ? a.work_req[blockIdx.x] : blockIdx.x, ch0 = blockIdx.y * SCAN_CHANNELS;
    const int l = threadIdx.x % SL, cg = threadIdx.x / SL;
    const int ch = ch0 + cg, inner = a.inner, ns = a.n_state;
    const bool ch_ok = ch < inner;
    const int first = a.work_start ? a.work_start[blockIdx.x] : 0;
    const int tok0 = a.cu_seqlens[req] + first, len = a.work_len ? a.work_len[blockIdx.x] : a.cu_seqlens[req + 1] - tok0;
    if (len <= 0) return;
    const int mode = a.mode;
    float* st = mode == 0 ? a.state + (size_t)a.slots[req] * a.state_stride + (size_t)(ch_ok ? ch : 0) * ns
                          : a.ws_state + ((size_t)blockIdx.x * inner + (ch_ok ? ch : 0)) * ns;
    float S[NR], A[NR], steps = 0.f;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int n = l + SL * r;
        const bool ok = ch_ok && n < ns;
        S[r] = ok && mode != 1 ? st[n] : 0.f;
        A[r] = ok ? a.A[(size_t)ch * ns + n] * 1.4426950408889634f : 0.f;      // in units of log2: the decay is one exp2 an entry
    }
    const float skip = ch_ok ? a.D[ch] : 0.f;
    const T* x = (const T*)a.x;
    const T* low = (const T*)a.low;
    const T* z = (const T*)a.z;
    T* out = (T*)a.out;

    // A tile's inputs are asked for into registers one tile ahead, so that they travel while the tile before is worked on.
    constexpr int PER = SCAN_TOKENS * SP / SCAN_THREADS;                    // B (and C) entries a thread stages: NR
    constexpr int CPER = SCAN_TOKENS * SCAN_CHANNELS / SCAN_THREADS;        // step, x and z entries a thread stages: 2
    float rB[PER], rC[PER], rs[CPER], rx[CPER], rz[CPER];
    auto fetch = [&](int t0) {
        const int n = min(SCAN_TOKENS, len - t0);
#pragma unroll
        for (int it = 0; it < PER; ++it) {
            const int e = it * SCAN_THREADS + threadIdx.x, t = e / SP, i = e % SP;
            const bool ok = t < n && i < ns;
            const T* row = low + (size_t)(tok0 + t0 + (ok ? t : 0)) * a.low_stride + (ok ? i : 0);
            rB[it] = ok ? to_float(row[a.b_col]) : 0.f;
            rC[it] = ok ? to_float(row[a.c_col]) : 0.f;
        }
#pragma unroll
        for (int it = 0; it < CPER; ++it) {
            const int e = it * SCAN_THREADS + threadIdx.x, t = e / SCAN_CHANNELS, c = e % SCAN_CHANNELS;
            const bool ok = t < n && ch0 + c < inner;
            const size_t tok = tok0 + t0 + (ok ? t : 0);
            rs[it] = ok ? a.step[tok * inner + ch0 + c] : 0.f;
            rx[it] = ok ? to_float(x[tok * inner + ch0 + c]) : 0.f;
            rz[it] = ok ? to_float(z[tok * a.z_stride + a.z_col + ch0 + c]) : 0.f;
        }
    };
    if (AHEAD) fetch(0);

    for (int t0 = 0; t0 < len; t0 += SCAN_TOKENS) {
        const int n = min(SCAN_TOKENS, len - t0);
        if (!AHEAD) fetch(t0);
        __syncthreads();
#pragma unroll
        for (int it = 0; it < PER; ++it) {
            const int e = it * SCAN_THREADS + threadIdx.x;
            Bs[e / SP][e % SP] = rB[it];
            Cs[e / SP][e % SP] = rC[it];
        }
#pragma unroll
        for (int it = 0; it < CPER; ++it) {
            const int e = it * SCAN_THREADS + threadIdx.x, t = e / SCAN_CHANNELS, c = e % SCAN_CHANNELS;
            dts[t][c] = rs[it] > 20.f ? rs[it] : log1pf(expf(rs[it]));
            xs[t][c] = rx[it];
            zs[t][c] = rz[it];
        }
        __syncthreads();
        if (AHEAD && t0 + SCAN_TOKENS < len) fetch(t0 + SCAN_TOKENS);
#pragma unroll 4
        for (int t = 0; t < n; ++t) {                 // the exponentials and the lane sums of neighbouring tokens overlap
            const float dt = dts[t][cg], xv = xs[t][cg], dx = dt * xv;
            steps += dt;
            float acc = 0.f;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                S[r] = fmaf(exp2f(dt * A[r]), S[r], dx * Bs[t][l + SL * r]);
                acc = fmaf(S[r], Cs[t][l + SL * r], acc);
            }
#pragma unroll
            for (int o = SL / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);      // every thread of the block is in this turn
            if (l == 0) {
                const float zv = zs[t][cg];
                ys[t][cg] = fmaf(skip, xv, acc) * (zv / (1.f + expf(-zv)));
            }
        }
        __syncthreads();
        if (mode != 1)
            for (int e = threadIdx.x; e < n * SCAN_CHANNELS; e += SCAN_THREADS) {
                const int t = e / SCAN_CHANNELS, c = e % SCAN_CHANNELS;
                if (ch0 + c < inner) out[(size_t)(tok0 + t0 + t) * inner + ch0 + c] = from_float<T>(ys[t][c]);
            }
    }
    if (ch_ok && mode != 2) {
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const int n = l + SL * r;
            if (n < ns) st[n] = S[r];
        }
        if (mode == 1 && l == 0) a.ws_steps[(size_t)blockIdx.x * inner + ch] = steps;
    }
}

// Chunks with up to 16 state entries a channel: a thread has a channel, all its entries in registers, so nothing is summed over lanes and
// a token costs a channel one softplus and one SiLU where eight lanes took eight.  A token's B and C come from shared memory 16 bytes a
// read for all of the block's channels, the next tile's on their way in registers; step, x and z are the thread's own, asked for ROW_STEP tokens ahead.
// Bound by the exponentials and the instructions around them.  (The decay's exponent is at most zero; where it is below float32's
// range the decay is zero.)  A portion in one piece stays with the kernel above, whose token is the shorter chain (0.27 us against 0.42
// where a scheduler has one warp).  Both passes and the combination, 1,999 tokens, 4,096 channels of 16: 381 -> 174 us; 2,048 tokens, 1,024
// channels of 8: 118 -> 58.  grid (work items, ceil(inner / 128)), block 128; OUT: outputs are wanted.
constexpr int ROW_CHANNELS = 128, ROW_STEP = 4;
static_assert(SCAN_TOKENS % ROW_STEP == 0, "a tile is whole steps");
__device__ __forceinline__ float ex2(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
template <typename T, int NS, bool OUT>
__global__ void __launch_bounds__(ROW_CHANNELS) selective_rows_kernel(const SelectiveArgs a) {
    __shared__ __align__(16) float Bs[2][SCAN_TOKENS][NS], Cs[2][SCAN_TOKENS][NS];
    pdl_enter_small();
    const int req = a.work_req[blockIdx.x], tid = threadIdx.x, ch = blockIdx.y * ROW_CHANNELS + tid;
    const int inner = a.inner, ns = a.n_state;
    const bool ok = ch < inner;
    const int tok0 = a.cu_seqlens[req] + a.work_start[blockIdx.x], len = a.work_len[blockIdx.x];
    if (len <= 0) return;
    const int col = ok ? ch : 0;
    float* st = a.ws_state + ((size_t)blockIdx.x * inner + col) * ns;
    float S[NS], A[NS], steps = 0.f;
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        S[n] = n < ns && OUT ? st[n] : 0.f;
        A[n] = n < ns ? a.A[(size_t)col * ns + n] * 1.4426950408889634f : 0.f;
    }
    const float skip = a.D[col];
    const T* x = (const T*)a.x + (size_t)tok0 * inner + col;
    const T* low = (const T*)a.low + (size_t)tok0 * a.low_stride;
    const T* z = (const T*)a.z + (size_t)tok0 * a.z_stride + a.z_col + col;
    const float* step = a.step + (size_t)tok0 * inner + col;
    T* out = (T*)a.out + (size_t)tok0 * inner + col;

    constexpr int PER = (SCAN_TOKENS * NS + ROW_CHANNELS - 1) / ROW_CHANNELS;      // B (and C) entries a thread stages
    float rB[PER], rC[PER];
    auto fetch = [&](int t0) {
#pragma unroll
        for (int it = 0; it < PER; ++it) {
            const int e = it * ROW_CHANNELS + tid, t = e / NS, n = e % NS;
            const bool in = e < SCAN_TOKENS * NS && t0 + t < len && n < ns;
            const T* row = low + (size_t)(in ? t0 + t : 0) * a.low_stride + (in ? n : 0);
            rB[it] = in ? to_float(row[a.b_col]) : 0.f;
            if (OUT) rC[it] = in ? to_float(row[a.c_col]) : 0.f;
        }
    };
    float rs[ROW_STEP], rx[ROW_STEP], rz[ROW_STEP];
    int left = len;                                            // tokens from the next one to be asked for on
    auto ask = [&]() {
#pragma unroll
        for (int k = 0; k < ROW_STEP; ++k) {
            const bool in = k < left;
            rs[k] = in ? step[(size_t)k * inner] : -INFINITY;  // a token that is not there: a step of zero
            rx[k] = in ? to_float(x[(size_t)k * inner]) : 0.f;
            if (OUT) rz[k] = in ? to_float(z[(size_t)k * a.z_stride]) : 0.f;
        }
        left -= ROW_STEP;
        step += ROW_STEP * (size_t)inner;
        x += ROW_STEP * (size_t)inner;
        if (OUT) z += ROW_STEP * (size_t)a.z_stride;
    };
    fetch(0);
    ask();
    for (int t0 = 0, buf = 0; t0 < len; t0 += SCAN_TOKENS, buf ^= 1) {
#pragma unroll
        for (int it = 0; it < PER; ++it) {
            const int e = it * ROW_CHANNELS + tid;
            if (e < SCAN_TOKENS * NS) {
                Bs[buf][e / NS][e % NS] = rB[it];
                if (OUT) Cs[buf][e / NS][e % NS] = rC[it];
            }
        }
        __syncthreads();                                       // (the other buffer's readers passed the one before)
        if (t0 + SCAN_TOKENS < len) fetch(t0 + SCAN_TOKENS);
        const int n_tok = min(SCAN_TOKENS, len - t0);
#pragma unroll 1
        for (int k0 = 0; k0 < n_tok; k0 += ROW_STEP) {
            float dt[ROW_STEP], xv[ROW_STEP], zv[ROW_STEP], y[ROW_STEP];
#pragma unroll
            for (int k = 0; k < ROW_STEP; ++k) {
                dt[k] = rs[k] > 20.f ? rs[k] : log1pf(expf(rs[k]));
                xv[k] = rx[k];
                if (OUT) zv[k] = rz[k];
            }
            if (left > 0) ask();
            const float4 *bp = reinterpret_cast<const float4*>(&Bs[buf][k0][0]), *cp = reinterpret_cast<const float4*>(&Cs[buf][k0][0]);
#pragma unroll
            for (int k = 0; k < ROW_STEP; ++k) {
                if (!OUT && k0 + k >= n_tok) break;            // a step of zero and an infinite rate make a NaN: the state that is kept meets neither
                const float dx = dt[k] * xv[k];
                steps += dt[k];
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int n = 0; n < NS; n += 4) {
                    const float4 b = bp[(k * NS + n) / 4], c = OUT ? cp[(k * NS + n) / 4] : make_float4(0.f, 0.f, 0.f, 0.f);
                    const float bs[4] = {b.x, b.y, b.z, b.w}, cs[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        S[n + e] = fmaf(ex2(dt[k] * A[n + e]), S[n + e], dx * bs[e]);
                        if (OUT) acc[e] = fmaf(S[n + e], cs[e], acc[e]);
                    }
                }
                y[k] = fmaf(skip, xv[k], (acc[0] + acc[1]) + (acc[2] + acc[3]));
            }
            if (OUT && ok) {
#pragma unroll
                for (int k = 0; k < ROW_STEP; ++k)
                    if (k0 + k < n_tok) out[(size_t)k * inner] = from_float<T>(y[k] * (zv[k] / (1.f + expf(-zv[k]))));
                out += ROW_STEP * (size_t)inner;
            }
        }
    }
    if (ok && !OUT) {
#pragma unroll
        for (int n = 0; n < NS; ++n)
            if (n < ns) st[n] = S[n];
        a.ws_steps[(size_t)blockIdx.x * inner + ch] = steps;
    }
}

template <typename T>
static void launch_rows(const SelectiveArgs& a, int items, cudaStream_t stream) {
    const dim3 grid(items, (a.inner + ROW_CHANNELS - 1) / ROW_CHANNELS), block(ROW_CHANNELS);
#define GO(NS)                                                                                                      \
    do {                                                                                                            \
        if (a.mode == 1) launch_pdl(selective_rows_kernel<T, NS, false>, grid, block, 0, stream, a);                \
        else launch_pdl(selective_rows_kernel<T, NS, true>, grid, block, 0, stream, a);                             \
    } while (0)
    if (a.n_state <= 4) GO(4);
    else if (a.n_state <= 8) GO(8);
    else GO(16);
#undef GO
}

// grid (long requests, ceil(inner * n_state / 256)): a thread an entry of a request's state, its chunks in order.
__global__ void selective_combine_kernel(float* __restrict__ state, size_t state_stride, const int* __restrict__ slots,
                                         const int* __restrict__ long_req, const int* __restrict__ long_first,
                                         const int* __restrict__ long_count, const float* __restrict__ A,
                                         float* __restrict__ ws_state, const float* __restrict__ ws_steps, int inner, int ns) {
    pdl_enter_small();
    const int e = blockIdx.y * blockDim.x + threadIdx.x;
    if (e >= inner * ns) return;
    const int ch = e / ns;
    float* slot = state + (size_t)slots[long_req[blockIdx.x]] * state_stride + e;
    const float rate = A[e];
    float S = *slot;
    const int c0 = long_first[blockIdx.x], c1 = c0 + long_count[blockIdx.x];
    for (int c = c0; c < c1; ++c) {
        float* at = ws_state + (size_t)c * inner * ns + e;
        const float own = *at;
        *at = S;                                                     // what chunk c starts from
        S = fmaf(expf(rate * ws_steps[(size_t)c * inner + ch]), S, own);
    }
    *slot = S;
}

}  // namespace lily

using namespace lily;

LILY_API int lily_selective_scan_max_state() { return SL * 32; }

LILY_API int lily_selective_scan(const void* x, const void* low, int low_stride, int b_col, int c_col, const float* step,
                                 const void* z, int z_stride, int z_col, const float* A, const float* D, float* state,
                                 size_t state_stride, void* out, const int* cu_seqlens, const int* slots, int requests, int tokens,
                                 int inner, int n_state, int dtype, const int* work_req, const int* work_start,
                                 const int* work_len, int mode, float* ws_state, float* ws_steps, cudaStream_t stream) {
    // `requests`: the blocks along x (requests, or the entries of the work lists)
    if (requests == 0) return 0;
    LILY_REQUIRE(mode >= 0 && mode <= 2 && (mode == 0 || (work_req && work_start && work_len && ws_state && ws_steps)),
                 "selective_scan: chunks come with their lists and a workspace");
    LILY_REQUIRE(inner > 0 && n_state > 0 && n_state <= SL * 32, "selective_scan: %d channels of %d state entries (up to %d)", inner, n_state, SL * 32);
    LILY_REQUIRE((size_t)inner * n_state <= state_stride, "selective_scan: the state row is shorter than %d x %d", inner, n_state);
    LILY_REQUIRE((inner + SCAN_CHANNELS - 1) / SCAN_CHANNELS <= 65535, "selective_scan: %d channels", inner);
    SelectiveArgs a{};
    a.x = x; a.low = low; a.low_stride = low_stride; a.b_col = b_col; a.c_col = c_col; a.step = step;
    a.z = z; a.z_stride = z_stride; a.z_col = z_col; a.A = A; a.D = D; a.state = state; a.state_stride = state_stride;
    a.out = out; a.cu_seqlens = cu_seqlens; a.slots = slots; a.inner = inner; a.n_state = n_state;
    a.work_req = work_req; a.work_start = work_start; a.work_len = work_len; a.mode = mode; a.ws_state = ws_state; a.ws_steps = ws_steps;
    dim3 grid(requests, (inner + SCAN_CHANNELS - 1) / SCAN_CHANNELS), block(SCAN_THREADS);
    const int per = (n_state + SL - 1) / SL;
    const bool ahead = mode != 0 || tokens > requests;  // some request brings more than one token
    if (mode != 0 && n_state <= 16) {
        if (dtype == kBF16) launch_rows<__nv_bfloat16>(a, requests, stream);
        else launch_rows<float>(a, requests, stream);
        LILY_CHECK_LAUNCH("selective_scan");
        return 0;
    }
#define GO(NR)                                                                                                            \
    do {                                                                                                                  \
        if (dtype == kBF16) {                                                                                             \
            if (ahead) launch_pdl(selective_scan_kernel<__nv_bfloat16, NR, true>, grid, block, 0, stream, a);             \
            else launch_pdl(selective_scan_kernel<__nv_bfloat16, NR, false>, grid, block, 0, stream, a);                  \
        } else {                                                                                                          \
            if (ahead) launch_pdl(selective_scan_kernel<float, NR, true>, grid, block, 0, stream, a);                     \
            else launch_pdl(selective_scan_kernel<float, NR, false>, grid, block, 0, stream, a);                          \
        }                                                                                                                 \
    } while (0)
    if (per <= 1) GO(1);
    else if (per <= 2) GO(2);
    else if (per <= 4) GO(4);
    else if (per <= 8) GO(8);
    else if (per <= 16) GO(16);
    else GO(32);
#undef GO
    LILY_CHECK_LAUNCH("selective_scan");
    return 0;
}

LILY_API int lily_selective_combine(float* state, size_t state_stride, const int* slots, const int* long_req, const int* long_first,
                                    const int* long_count, int num_long, const float* A, float* ws_state, const float* ws_steps,
                                    int inner, int n_state, cudaStream_t stream) {
    if (num_long == 0) return 0;
    const int entries = inner * n_state;
    launch_pdl(selective_combine_kernel, dim3(num_long, (entries + 255) / 256), dim3(256), 0, stream, state, state_stride, slots,
               long_req, long_first, long_count, A, ws_state, ws_steps, inner, n_state);
    LILY_CHECK_LAUNCH("selective_combine");
    return 0;
}
