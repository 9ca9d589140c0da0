// The state-space scan (see ssm.cu) over chunks of a prompt in bfloat16: a chunk's sums as matrix products on the tensor cores
// (mma.sync m16n8k16, float32 accumulation).
//
// With a_t = A dt_t and L_t the sum of the a up to and with token t of the chunk, for a chunk that starts from S_0:
//
//     own state   S = sum_t w_t x_t B_t^T,  w_t = dt_t e^(L - L_t);      S_end = e^L S_0 + S        (L of the last token)
//     output      y_t = e^(L_t) S_0 C_t + sum_(s <= t) e^(L_t - L_s) dt_s (C_t . B_s) x_s + D x_t
//
//   ssd_chunk_write   the own state and e^L: a block a (head, chunk, 64 value columns), warp w its 16 value columns w
//   ssd_combine       (ssm.cu) leaves each chunk's starting state in the workspace and the last state in the slot
//   ssd_chunk_read    the outputs: a block 64 tokens of a chunk and 64 value columns of a head, warp w its 16 tokens w
//
// B, C and x are the convolution's own bfloat16 numbers.  What meets the tensor cores as float32 (a weighted value, a decayed
// score, an entry of the starting state) is cut into the sum of three bfloat16 numbers, all 24 bits of it, and multiplied three
// times; the L are summed in float64 and kept as two float32, so that the difference of two large ones loses nothing.
// (The chunked form of the scan is Dao and Gu's, "Transformers are SSMs", 2024.)  A number that is not finite reaches what it would token
// by token: its own column and head, from its token on.
// Bound by the tensor cores and the reads of shared memory that feed them.  The scan one token after another took a chunk's
// 128 steps twice, each step a round of shared memory, FMAs and shuffles: 2,048 tokens, 64 heads of 64 x 128: 139 (own states) and
// 270 us (outputs), now 33 and 94; against 64 bits the outputs are 1.0e-7 off in the 2-norm, where they were 2 to 4e-7.
#include "common.cuh"
#include "mma.cuh"

namespace lily {
namespace ssdc {

using namespace mma16;

constexpr int THREADS = 128;
constexpr int CHUNK = 128;                 // tokens of a chunk, at most
constexpr int TOK = 64;                    // tokens of a block of the read kernel, keys of a turn of it
constexpr int PV = 64;                     // value columns of a block
constexpr int NMAX = 128;                  // n_state, at most (a multiple of 16)
constexpr int PAD = 8;                     // an odd number of 16-byte pieces a row: ldmatrix without bank conflicts

struct Args {
    const __nv_bfloat16* xbc;              // [tokens, channels]: x [heads, pd] | B [groups, n] | C [groups, n]
    int channels;
    const __nv_bfloat16* proj;
    int proj_stride, dt_col;
    const float* dt_bias;
    const float* a_log;
    const float* d_skip;
    const int* cu_seqlens;
    const int* item_req;
    const int* item_start;
    const int* item_len;
    float* chunk_state;                    // [items, heads, pd, n]: own states, or (read) starting states
    float* chunk_decay;                    // [items, heads]
    float* y;                              // [tokens, heads * pd]
    int heads, pd, n, groups;
};

__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }

// Which of a pair of bfloat16 numbers are infinities or NaN, as a mask over the pair's bits.
__device__ __forceinline__ uint32_t not_finite(uint32_t pair) {
    return ((pair & 0x7f80u) == 0x7f80u ? 0xffffu : 0u) | ((pair & 0x7f800000u) == 0x7f800000u ? 0xffff0000u : 0u);
}

__device__ __forceinline__ float half_of(uint32_t pair, int upper) { return __uint_as_float(upper ? pair & 0xffff0000u : pair << 16); }

// A token's step size and L (as two numbers) for the chunk's tokens, a thread each; the chunk's L for everyone.  All threads call it.
// e^-110 is zero in float32, so a decay beyond e^-200 counts as that: the sums stay finite and keep the bits of the slow decays behind it.
struct Gates {
    float dt[CHUNK], hi[CHUNK], lo[CHUNK];
    double warp_sum[THREADS / 32];
};
__device__ __forceinline__ double chunk_gates(const Args& a, Gates& s, size_t tok0, int len, int head) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float A = -expf(a.a_log[head]);
    const float dt = tid < len ? softplus_f(__bfloat162float(a.proj[(tok0 + tid) * a.proj_stride + a.dt_col + head]) + a.dt_bias[head]) : 0.f;
    const float step = tid < len ? A * dt : 0.f;
    double L = (double)(step < -200.f ? -200.f : step);          // (a NaN stays one)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double left = __shfl_up_sync(0xffffffffu, L, o);
        if (lane >= o) L += left;
    }
    if (lane == 31) s.warp_sum[warp] = L;
    __syncthreads();
    double total = 0.0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) {
        if (w < warp) L += s.warp_sum[w];
        total += s.warp_sum[w];
    }
    s.dt[tid] = dt;
    s.hi[tid] = (float)L;
    s.lo[tid] = (float)(L - (double)(float)L);
    __syncthreads();
    return total;
}

// Rows [0, rows) of `cols` bfloat16 from `src` (rows `ld` apart) into `total` rows `stride` apart in shared memory; zeros outside
// the rows and from column `have` on.  cols and have are multiples of 8.
__device__ __forceinline__ void stage_rows(__nv_bfloat16* dst, int stride, const __nv_bfloat16* src, size_t ld, int rows, int total, int cols, int have) {
    const int per = cols / 8;
    for (int e = threadIdx.x; e < total * per; e += THREADS) {
        const int r = e / per, c = (e % per) * 8;
        const bool in = r < rows && c < have;
        cp_async16(smem_u32(dst + r * stride + c), src + (in ? (size_t)r * ld + c : 0), in);
    }
}

struct WriteTile {
    __nv_bfloat16 b[CHUNK][NMAX + PAD], v[3][CHUNK][PV + PAD];
    Gates gates;
};

// grid (heads, chunks, ceil(pd / PV))
__global__ void __launch_bounds__(THREADS) write_kernel(const Args a) {
    extern __shared__ __align__(16) unsigned char smem[];
    WriteTile& s = *reinterpret_cast<WriteTile*>(smem);
    pdl_wait();
    pdl_launch_dependents();
    const int head = blockIdx.x, item = blockIdx.y, v0 = blockIdx.z * PV;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
    const int len = a.item_len[item];
    const size_t tok0 = (size_t)a.cu_seqlens[a.item_req[item]] + a.item_start[item];
    const int inner = a.heads * a.pd, grp = head / (a.heads / a.groups), have = min(PV, a.pd - v0);
    stage_rows(&s.b[0][0], NMAX + PAD, a.xbc + tok0 * a.channels + inner + (size_t)grp * a.n, a.channels, len, CHUNK, NMAX, a.n);
    cp_async_commit();
    const __nv_bfloat16* xsrc = a.xbc + tok0 * a.channels + (size_t)head * a.pd + v0;
    constexpr int VPER = CHUNK * (PV / 8) / THREADS;             // 16-byte pieces of values a thread weighs
    uint4 raw[VPER];
#pragma unroll
    for (int k = 0; k < VPER; ++k) {
        const int e = k * THREADS + tid, t = e / (PV / 8), col = (e % (PV / 8)) * 8;
        raw[k] = t < len && col < have ? *reinterpret_cast<const uint4*>(xsrc + (size_t)t * a.channels + col) : make_uint4(0, 0, 0, 0);
    }
    const double total = chunk_gates(a, s.gates, tok0, len, head);
    if (tid == 0 && blockIdx.z == 0) a.chunk_decay[(size_t)item * a.heads + head] = (float)exp(total);
    // w_t in the place of dt_t
    if (tid < len) s.gates.dt[tid] *= expf((float)(total - (double)s.gates.hi[tid]) - s.gates.lo[tid]);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < VPER; ++k) {
        const int e = k * THREADS + tid, t = e / (PV / 8), col = (e % (PV / 8)) * 8;
        const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw[k]);
        const float w = s.gates.dt[t];
        uint32_t part[3][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float2 f = __bfloat1622float2(p[q]);
            split3(f.x * w, f.y * w, part[0][q], part[1][q], part[2][q]);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(&s.v[q][t][col]) = make_uint4(part[q][0], part[q][1], part[q][2], part[q][3]);
    }
    cp_async_wait<0>();
    __syncthreads();
    float acc[NMAX / 8][4];
#pragma unroll
    for (int j = 0; j < NMAX / 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    const int steps = (len + 15) / 16;
    for (int k16 = 0; k16 < steps; ++k16) {
        uint32_t v[3][4];
        const int ar = k16 * 16 + (lane & 7) + ((lane >> 4) << 3), ac = warp * 16 + (((lane >> 3) & 1) << 3);
#pragma unroll
        for (int q = 0; q < 3; ++q) ldmatrix_x4_trans(smem_u32(&s.v[q][ar][ac]), v[q][0], v[q][1], v[q][2], v[q][3]);
        // the parts of a sum are a run of products apart, so that no product waits for the one before it
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            if (half * 64 >= a.n) break;
            uint32_t b[4][4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                ldmatrix_x4_trans(smem_u32(&s.b[k16 * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)][half * 64 + u * 16 + ((lane >> 4) << 3)]),
                                  b[u][0], b[u][1], b[u][2], b[u][3]);
            float sum[8][4] = {};
#pragma unroll
            for (int q = 2; q >= 0; --q)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    mma_bf16(sum[2 * u], v[q], b[u][0], b[u][1]);
                    mma_bf16(sum[2 * u + 1], v[q], b[u][2], b[u][3]);
                }
            add<8>(&acc[half * 8], sum);
        }
    }
    float* dst = a.chunk_state + ((size_t)item * a.heads + head) * a.pd * a.n;
    const int r_lo = v0 + warp * 16 + g, r_hi = r_lo + 8;
#pragma unroll
    for (int j = 0; j < NMAX / 8; ++j) {
        const int col = j * 8 + 2 * c;
        if (col >= a.n) continue;
        if (r_lo < a.pd) *reinterpret_cast<float2*>(dst + (size_t)r_lo * a.n + col) = make_float2(acc[j][0], acc[j][1]);
        if (r_hi < a.pd) *reinterpret_cast<float2*>(dst + (size_t)r_hi * a.n + col) = make_float2(acc[j][2], acc[j][3]);
    }
}

// Shared memory: C [TOK][n + PAD]; then the starting state's three parts [PV][n + PAD], or (behind a barrier) B [TOK][n + PAD] and x
// [TOK][PV + PAD] of a turn.
__host__ __device__ constexpr int read_smem() { return (4 * TOK * (NMAX + PAD)) * 2; }
static_assert(PV == TOK && TOK * (NMAX + PAD) + TOK * (PV + PAD) <= 3 * PV * (NMAX + PAD), "a turn's keys and values fit the state's room");

// grid (heads, 2 tiles of every chunk, ceil(pd / PV))
__global__ void __launch_bounds__(THREADS, 3) read_kernel(const Args a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Gates gates;
    pdl_wait();
    pdl_launch_dependents();
    const int head = blockIdx.x, item = blockIdx.y >> 1, start = (1 - (blockIdx.y & 1)) * TOK, v0 = blockIdx.z * PV;   // the longer tile first
    const int len = a.item_len[item];
    if (start >= len) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
    const size_t tok0 = (size_t)a.cu_seqlens[a.item_req[item]] + a.item_start[item];
    const int inner = a.heads * a.pd, grp = head / (a.heads / a.groups), have = min(PV, a.pd - v0), n16 = a.n / 16;
    constexpr int LD = NMAX + PAD, XLD = PV + PAD;
    __nv_bfloat16* c_s = reinterpret_cast<__nv_bfloat16*>(smem);
    __nv_bfloat16* rest = c_s + TOK * LD;
    const __nv_bfloat16* bsrc = a.xbc + tok0 * a.channels + inner + (size_t)grp * a.n;
    const __nv_bfloat16* xsrc = a.xbc + tok0 * a.channels + (size_t)head * a.pd + v0;
    stage_rows(c_s, LD, bsrc + (size_t)start * a.channels + (size_t)a.groups * a.n, a.channels, len - start, TOK, a.n, a.n);
    cp_async_commit();
    {
        const float* st = a.chunk_state + (((size_t)item * a.heads + head) * a.pd + v0) * a.n;
        const int per = a.n / 4;
#pragma unroll 4
        for (int e = tid; e < PV * per; e += THREADS) {
            const int r = e / per, col = e % per * 4;
            const float4 v = r < have ? *reinterpret_cast<const float4*>(st + (size_t)r * a.n + col) : make_float4(0.f, 0.f, 0.f, 0.f);
            uint2 part[3];
            split3(v.x, v.y, part[0].x, part[1].x, part[2].x);
            split3(v.z, v.w, part[0].y, part[1].y, part[2].y);
#pragma unroll
            for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(rest + (q * PV + r) * LD + col) = part[q];
        }
    }
    chunk_gates(a, gates, tok0, len, head);
    cp_async_wait<0>();
    __syncthreads();

    // ---- what the starting state answers
    float o[PV / 8][4];
#pragma unroll
    for (int j = 0; j < PV / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    const __nv_bfloat16* crow = c_s + (warp * 16 + (lane & 15)) * LD + ((lane >> 4) << 3);
    const int br = (lane & 7) + ((lane >> 4) << 3), bc = ((lane >> 3) & 1) << 3;
    for (int kk = 0; kk < n16; ++kk) {
        uint32_t q[4];
        ldmatrix_x4(smem_u32(crow + kk * 16), q[0], q[1], q[2], q[3]);
        float sum[PV / 8][4] = {};
#pragma unroll
        for (int part = 2; part >= 0; --part)
#pragma unroll
            for (int u = 0; u < PV / 16; ++u) {
                uint32_t b[4];
                ldmatrix_x4(smem_u32(rest + (part * PV + u * 16 + br) * LD + kk * 16 + bc), b[0], b[1], b[2], b[3]);
                mma_bf16(sum[2 * u], q, b[0], b[1]);
                mma_bf16(sum[2 * u + 1], q, b[2], b[3]);
            }
        add<PV / 8>(o, sum);
    }
    const int t_lo = start + warp * 16 + g, t_hi = t_lo + 8;     // this lane's two tokens of the chunk
    const float hi0 = gates.hi[t_lo], lo0 = gates.lo[t_lo], hi1 = gates.hi[t_hi], lo1 = gates.lo[t_hi];
    {
        const float e0 = expf(hi0 + lo0), e1 = expf(hi1 + lo1);
#pragma unroll
        for (int j = 0; j < PV / 8; ++j) {
            o[j][0] *= e0; o[j][1] *= e0;
            o[j][2] *= e1; o[j][3] *= e1;
        }
    }

    // ---- what the chunk's own tokens add, 64 of them a turn
    __nv_bfloat16 *b_s = rest, *x_s = rest + TOK * LD;
    for (int s0 = 0; s0 <= start; s0 += TOK) {
        __syncthreads();                                         // the room's last readers are done
        stage_rows(b_s, LD, bsrc + (size_t)s0 * a.channels, a.channels, len - s0, TOK, a.n, a.n);
        stage_rows(x_s, XLD, xsrc + (size_t)s0 * a.channels, a.channels, len - s0, TOK, PV, have);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        const int upto = s0 == start ? warp + 1 : TOK / 16;      // runs of 16 keys that this warp's tokens see
        for (int k16 = 0; k16 < upto; ++k16) {
            float sc[2][4] = {};
            for (int kk = 0; kk < n16; ++kk) {
                uint32_t q[4], b[4];
                ldmatrix_x4(smem_u32(crow + kk * 16), q[0], q[1], q[2], q[3]);
                ldmatrix_x4(smem_u32(b_s + (k16 * 16 + br) * LD + kk * 16 + bc), b[0], b[1], b[2], b[3]);
                float sum[2][4] = {};
                mma_bf16(sum[0], q, b[0], b[1]);
                mma_bf16(sum[1], q, b[2], b[3]);
                add<2>(sc, sum);
            }
            uint32_t w[3][4];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int s = s0 + k16 * 16 + j * 8 + 2 * c;
                const float h0 = gates.hi[s], l0 = gates.lo[s], d0 = gates.dt[s], h1 = gates.hi[s + 1], l1 = gates.lo[s + 1], d1 = gates.dt[s + 1];
                const float p00 = s <= t_lo ? sc[j][0] * (expf((hi0 - h0) + (lo0 - l0)) * d0) : 0.f;
                const float p01 = s + 1 <= t_lo ? sc[j][1] * (expf((hi0 - h1) + (lo0 - l1)) * d1) : 0.f;
                const float p10 = s <= t_hi ? sc[j][2] * (expf((hi1 - h0) + (lo1 - l0)) * d0) : 0.f;
                const float p11 = s + 1 <= t_hi ? sc[j][3] * (expf((hi1 - h1) + (lo1 - l1)) * d1) : 0.f;
                split3(p00, p01, w[0][2 * j], w[1][2 * j], w[2][2 * j]);
                split3(p10, p11, w[0][2 * j + 1], w[1][2 * j + 1], w[2][2 * j + 1]);
            }
            uint32_t xb[PV / 16][4];
#pragma unroll
            for (int u = 0; u < PV / 16; ++u)
                ldmatrix_x4_trans(smem_u32(x_s + (k16 * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)) * XLD + u * 16 + ((lane >> 4) << 3)),
                                  xb[u][0], xb[u][1], xb[u][2], xb[u][3]);
            // A weight of zero takes finite values away, but not infinities and NaN: in the run that a warp's tokens see only part of, those
            // are left out of the product and meet the tokens that see them one by one.
            bool odd = false;
            if (s0 == start && k16 == warp) {
                uint32_t any = 0;                                // an exponent of all ones leaves a half of zeros, which borrows
#pragma unroll
                for (int u = 0; u < PV / 16; ++u)
#pragma unroll
                    for (int q = 0; q < 4; ++q) any |= ((xb[u][q] & 0x7f807f80u) ^ 0x7f807f80u) - 0x00010001u;
                odd = __any_sync(0xffffffffu, (any & 0x80008000u) != 0);
                if (odd)
#pragma unroll
                    for (int u = 0; u < PV / 16; ++u)
#pragma unroll
                        for (int q = 0; q < 4; ++q) xb[u][q] &= ~not_finite(xb[u][q]);
            }
            float sum[PV / 8][4] = {};
#pragma unroll
            for (int part = 2; part >= 0; --part)
#pragma unroll
                for (int u = 0; u < PV / 16; ++u) {
                    mma_bf16(sum[2 * u], w[part], xb[u][0], xb[u][1]);
                    mma_bf16(sum[2 * u + 1], w[part], xb[u][2], xb[u][3]);
                }
            add<PV / 8>(o, sum);
            if (odd) {
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll 1
                    for (int k = 0; k < 8; ++k) {
                        const int row = warp * 16 + half * 8 + k, from = (lane & 28) | (k >> 1);
                        float p_lo = 0.f, p_hi = 0.f;            // the key's weights of this lane's two tokens
#pragma unroll
                        for (int part = 0; part < 3; ++part) {
                            p_lo += half_of(__shfl_sync(0xffffffffu, w[part][2 * half], from), k & 1);
                            p_hi += half_of(__shfl_sync(0xffffffffu, w[part][2 * half + 1], from), k & 1);
                        }
#pragma unroll
                        for (int j = 0; j < PV / 8; ++j) {
                            const uint32_t pair = *reinterpret_cast<const uint32_t*>(x_s + row * XLD + j * 8 + 2 * c), m = not_finite(pair);
#pragma unroll
                            for (int q = 0; q < 2; ++q)
                                if (m >> (16 * q) & 1) {
                                    if (start + row <= t_lo) o[j][q] = fmaf(p_lo, half_of(pair, q), o[j][q]);
                                    if (start + row <= t_hi) o[j][2 + q] = fmaf(p_hi, half_of(pair, q), o[j][2 + q]);
                                }
                        }
                    }
            }
        }
    }
    // the last turn's values are the tile's own tokens
    const float D = a.d_skip[head];
#pragma unroll
    for (int j = 0; j < PV / 8; ++j) {
        const int col = j * 8 + 2 * c;
        if (col >= have) continue;
        float* dst = a.y + (tok0 + t_lo) * inner + (size_t)head * a.pd + v0 + col;
        if (t_lo < len) {
            const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(x_s + (t_lo - start) * XLD + col));
            *reinterpret_cast<float2*>(dst) = make_float2(fmaf(D, x.x, o[j][0]), fmaf(D, x.y, o[j][1]));
        }
        if (t_hi < len) {
            const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(x_s + (t_hi - start) * XLD + col));
            *reinterpret_cast<float2*>(dst + (size_t)8 * inner) = make_float2(fmaf(D, x.x, o[j][2]), fmaf(D, x.y, o[j][3]));
        }
    }
}

}  // namespace ssdc
}  // namespace lily

using namespace lily;

// Whether the chunk kernels take the shape: states and head sizes of whole tiles, rows on 16 bytes.
LILY_API int lily_ssd_chunk_takes(const void* xbc, int channels, int heads, int pd, int n_state, int chunk) {
    return n_state >= 16 && n_state <= ssdc::NMAX && n_state % 16 == 0 && pd >= 16 && pd % 16 == 0 && chunk <= ssdc::CHUNK &&
           (uintptr_t)xbc % 16 == 0 && channels % 8 == 0 && heads <= 65535;
}

// outputs 0: the chunks' own states and decays; 1: the outputs from the starting states that ssd_combine left.
LILY_API int lily_ssd_chunk(const void* xbc, int channels, const void* proj, int proj_stride, int dt_col, const float* dt_bias, const float* a_log,
                            const float* d_skip, float* y, const int* cu_seqlens, int chunks, int heads, int pd, int n_state, int groups,
                            const int* item_req, const int* item_start, const int* item_len, float* chunk_state, float* chunk_decay, int chunk,
                            int outputs, cudaStream_t stream) {
    if (chunks == 0) return 0;
    LILY_REQUIRE(heads > 0 && groups > 0 && heads % groups == 0, "ssd_chunk: %d heads over %d groups", heads, groups);
    LILY_REQUIRE(lily_ssd_chunk_takes(xbc, channels, heads, pd, n_state, chunk) && 2 * chunks <= 65535 && (uintptr_t)chunk_state % 16 == 0,
                 "ssd_chunk: %d chunks of %d, heads of %d x %d", chunks, chunk, pd, n_state);
    const ssdc::Args a{(const __nv_bfloat16*)xbc, channels, (const __nv_bfloat16*)proj, proj_stride, dt_col, dt_bias, a_log, d_skip, cu_seqlens,
                       item_req, item_start, item_len, chunk_state, chunk_decay, y, heads, pd, n_state, groups};
    const int smem = outputs ? ssdc::read_smem() : (int)sizeof(ssdc::WriteTile), wide = (pd + ssdc::PV - 1) / ssdc::PV;
    auto kern = outputs ? ssdc::read_kernel : ssdc::write_kernel;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    LILY_REQUIRE(e == cudaSuccess, "ssd_chunk: cannot get %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
    launch_pdl(kern, dim3(heads, outputs ? 2 * chunks : chunks, wide), dim3(ssdc::THREADS), smem, stream, a);
    LILY_CHECK_LAUNCH("ssd_chunk");
    return 0;
}
