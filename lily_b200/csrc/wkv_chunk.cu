// The recurrence with a decay a channel (see wkv.cu) over chunks of a prompt in bfloat16, on the tensor cores (mma.sync m16n8k16, float32
// accumulation).
//
// A chunk is up to four segments of 16 tokens.  With w_t the token's decays (a number a key channel), p_t the product of the segment's
// decays before token t, q_s that of those behind token s, and W the product over a segment, for a chunk that starts from S_0:
//
//     own state   S = sum_s (k_s * q_s * the later segments' W) v_s^T,   S_end = diag(all W) S_0 + S
//     output      o_t = (r_t * p_t * the earlier segments' W)^T S_0 + sum_s A_ts v_s,   and A_ts is, for s
//                   in an earlier segment        sum_i (r_t p_t * the W between them)_i (k_s q_s)_i
//                   in t's segment, before t     sum_i r_ti k_si (product of the decays between them)_i
//                   t itself                     sum_i r_ti u_i k_ti
//
// Every factor is a product of decays, at most one: nothing is divided by a decay, however fast it is.
//
//   wkv_chunk_write   the own state and the product of the decays: a block a (head, chunk), a warp a segment, then 16 key channels
//   wkv_combine       (wkv.cu) leaves each chunk's starting state in the workspace and the last state in the slot
//   wkv_chunk_read    the outputs: a block a (head, chunk), a warp the 16 tokens of a segment; the weights within the segment are
//                     formed on CUDA cores, lanes over channels, 32 sums over the lanes in 31 exchanges
//
// v is the convolution-free projection's own bfloat16; what meets the tensor cores as float32 (decayed keys and queries, weights, S_0) is cut into
// the sum of three bfloat16 numbers, all 24 bits of it, and of two such numbers the products down to 2^-27 are taken.  Runs of 16
// products are added to a total by rounded additions.  What is not finite stays behind its token, as token by token.
// Bound by the instructions around the products (cutting, the weights within a segment).  The token-by-token scan took a chunk's tokens twice,
// each a round of shared memory and FMAs: 1,999 tokens, 32 heads of 64 x 64, own states, combination and outputs 249 -> 73 us, 2,048 tokens,
// 64 heads 450 -> 134, 32 heads of 32 147 -> 59.  Against 64 bits outputs and states of 33 to 1,000 tokens are 0.92 to 0.98 of as far off as they
// were token by token (1.3e-7 to 2.7e-7).
#include "common.cuh"
#include "mma.cuh"

namespace lily {
namespace wkvc {

using namespace mma16;

constexpr int THREADS = 128;
constexpr int CHUNK = 64, SEG = 16, SEGS = CHUNK / SEG;
constexpr int D = 64;                      // head size, at most (a multiple of 16)
constexpr int LD = D + 8;                  // an odd number of 16-byte pieces a row: ldmatrix without bank conflicts

struct Args {
    const __nv_bfloat16 *r, *k, *v;        // [tokens, heads * d], rows `ld` apart
    int ld;
    const float* lw;                       // [tokens, heads * d]: the decays' logarithms
    const float* u;                        // [heads, d]
    float* y;                              // [tokens, heads * d]
    const int* cu_seqlens;
    const int* item_req;
    const int* item_start;
    const int* item_len;
    float* ws_state;                       // [items, heads, d, d]: own states, or (read) starting states
    float* ws_decay;                       // [items, heads, d]
    int heads, d;
};

// The three parts of a pair of columns into their planes.
__device__ __forceinline__ void put(__nv_bfloat16 (*planes)[CHUNK][LD], int row, int col, float x, float y) {
    uint32_t p[3];
    split3(x, y, p[0], p[1], p[2]);
#pragma unroll
    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint32_t*>(&planes[q][row][col]) = p[q];
}

__device__ __forceinline__ void stage_values(__nv_bfloat16 (*dst)[LD], const __nv_bfloat16* src, int ld, int rows, int d) {
#pragma unroll
    for (int k = 0; k < CHUNK * D / 8 / THREADS; ++k) {
        const int e = k * THREADS + threadIdx.x, r = e / (D / 8), c = e % (D / 8) * 8;
        const bool in = r < rows && c < d;
        cp_async16(smem_u32(&dst[r][c]), src + (in ? (size_t)r * ld + c : 0), in);
    }
}

struct WriteTile {
    __nv_bfloat16 k[3][CHUNK][LD], v[CHUNK][LD];
    float w[SEGS][D];                      // the segments' products of decays
};

// grid (heads, chunks)
__global__ void __launch_bounds__(THREADS) write_kernel(const Args a) {
    extern __shared__ __align__(16) unsigned char smem[];
    WriteTile& s = *reinterpret_cast<WriteTile*>(smem);
    pdl_wait();
    pdl_launch_dependents();
    const int head = blockIdx.x, item = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int len = a.item_len[item], d = a.d;
    const size_t tok0 = (size_t)a.cu_seqlens[a.item_req[item]] + a.item_start[item], hd = (size_t)a.heads * d;
    stage_values(s.v, a.v + tok0 * a.ld + (size_t)head * d, a.ld, len, d);
    cp_async_commit();
    // a lane has channels 2 lane, 2 lane + 1 of its warp's segment
    const int ch = 2 * lane;
    uint32_t kr[SEG];
    float2 w[SEG];
#pragma unroll
    for (int t = 0; t < SEG; ++t) {
        const int at = warp * SEG + t;
        const bool in = at < len && ch < d;
        kr[t] = in ? *reinterpret_cast<const uint32_t*>(a.k + (tok0 + at) * a.ld + (size_t)head * d + ch) : 0u;
        w[t] = in ? *reinterpret_cast<const float2*>(a.lw + (tok0 + at) * hd + (size_t)head * d + ch) : make_float2(0.f, 0.f);
    }
    float kx[SEG], ky[SEG], qx = 1.f, qy = 1.f;
#pragma unroll
    for (int t = SEG - 1; t >= 0; --t) {
        kx[t] = lower(kr[t]) * qx;
        ky[t] = upper(kr[t]) * qy;
        qx *= expf(w[t].x);
        qy *= expf(w[t].y);
    }
    *reinterpret_cast<float2*>(&s.w[warp][ch]) = make_float2(qx, qy);
    __syncthreads();
    float bx = 1.f, by = 1.f;                                  // the later segments
#pragma unroll
    for (int j = 1; j < SEGS; ++j)
        if (j > warp) {
            bx *= s.w[j][ch];
            by *= s.w[j][ch + 1];
        }
    if (warp == 0 && ch < d)
        *reinterpret_cast<float2*>(a.ws_decay + ((size_t)item * a.heads + head) * d + ch) = make_float2(qx * bx, qy * by);
#pragma unroll
    for (int t = 0; t < SEG; ++t) put(s.k, warp * SEG + t, ch, kx[t] * bx, ky[t] * by);
    cp_async_wait<0>();
    __syncthreads();
    if (warp * 16 >= d) return;
    float acc[D / 8][4] = {};
    const int steps = (len + 15) / 16;
    for (int k16 = 0; k16 < steps; ++k16) {
        uint32_t q[3][4], b[4][4];
#pragma unroll
        for (int p = 0; p < 3; ++p)
            ldmatrix_x4_trans(smem_u32(&s.k[p][k16 * 16 + (lane & 7) + ((lane >> 4) << 3)][warp * 16 + (((lane >> 3) & 1) << 3)]), q[p][0], q[p][1], q[p][2], q[p][3]);
#pragma unroll
        for (int n = 0; n < 4; ++n)
            ldmatrix_x4_trans(smem_u32(&s.v[k16 * 16 + (lane & 7) + (((lane >> 3) & 1) << 3)][n * 16 + ((lane >> 4) << 3)]), b[n][0], b[n][1], b[n][2], b[n][3]);
        float sum[D / 8][4] = {};
#pragma unroll
        for (int p = 2; p >= 0; --p)
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                mma_bf16(sum[2 * n], q[p], b[n][0], b[n][1]);
                mma_bf16(sum[2 * n + 1], q[p], b[n][2], b[n][3]);
            }
        add<D / 8>(acc, sum);
    }
    float* dst = a.ws_state + (((size_t)item * a.heads + head) * d + warp * 16 + g) * d;
#pragma unroll
    for (int n = 0; n < D / 8; ++n) {
        const int col = n * 8 + 2 * c;
        if (col >= d) continue;
        *reinterpret_cast<float2*>(dst + col) = make_float2(acc[n][0], acc[n][1]);
        *reinterpret_cast<float2*>(dst + (size_t)8 * d + col) = make_float2(acc[n][2], acc[n][3]);
    }
}

struct ReadTile {
    __nv_bfloat16 k[3][CHUNK][LD];         // k_s q_s in three parts, then S_0 in three parts
    __nv_bfloat16 v[CHUNK][LD];
    float s0[D][D];
    float r[CHUNK][D + 2];                 // r_t p_t
    float w[SEGS][D];
    float a[SEGS][SEG][SEG + 1];           // the weights within a segment
};
static_assert(3 * (sizeof(ReadTile) + 1024) <= 228 * 1024, "three blocks a SM");

// grid (heads, chunks)
__global__ void __launch_bounds__(THREADS, 3) read_kernel(const Args a) {
    extern __shared__ __align__(16) unsigned char smem[];
    ReadTile& s = *reinterpret_cast<ReadTile*>(smem);
    pdl_wait();
    pdl_launch_dependents();
    const int head = blockIdx.x, item = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int len = a.item_len[item], d = a.d;
    const size_t tok0 = (size_t)a.cu_seqlens[a.item_req[item]] + a.item_start[item], hd = (size_t)a.heads * d;
    stage_values(s.v, a.v + tok0 * a.ld + (size_t)head * d, a.ld, len, d);
    {
        const float* st = a.ws_state + ((size_t)item * a.heads + head) * d * d;
#pragma unroll
        for (int k = 0; k < D * D / 4 / THREADS; ++k) {
            const int e = k * THREADS + threadIdx.x, i = e / (D / 4), j = e % (D / 4) * 4;
            const bool in = i < d && j < d;
            cp_async16(smem_u32(&s.s0[i][j]), st + (in ? (size_t)i * d + j : 0), in);
        }
    }
    cp_async_commit();
    {
        const int ch = 2 * lane;
        uint32_t kr[SEG], rr[SEG];
        float2 w[SEG];
#pragma unroll
        for (int t = 0; t < SEG; ++t) {
            const int at = warp * SEG + t;
            const bool in = at < len && ch < d;
            const size_t src = (tok0 + at) * a.ld + (size_t)head * d + ch;
            kr[t] = in ? *reinterpret_cast<const uint32_t*>(a.k + src) : 0u;
            rr[t] = in ? *reinterpret_cast<const uint32_t*>(a.r + src) : 0u;
            w[t] = in ? *reinterpret_cast<const float2*>(a.lw + (tok0 + at) * hd + (size_t)head * d + ch) : make_float2(0.f, 0.f);
        }
        const float2 u = ch < d ? *reinterpret_cast<const float2*>(a.u + (size_t)head * d + ch) : make_float2(0.f, 0.f);
#pragma unroll
        for (int t = 0; t < SEG; ++t) w[t] = make_float2(expf(w[t].x), expf(w[t].y));
        float px = 1.f, py = 1.f;
#pragma unroll
        for (int t = 0; t < SEG; ++t) {
            *reinterpret_cast<float2*>(&s.r[warp * SEG + t][ch]) = make_float2(lower(rr[t]) * px, upper(rr[t]) * py);
            px *= w[t].x;
            py *= w[t].y;
        }
        *reinterpret_cast<float2*>(&s.w[warp][ch]) = make_float2(px, py);
        px = py = 1.f;
#pragma unroll
        for (int t = SEG - 1; t >= 0; --t) {
            put(s.k, warp * SEG + t, ch, lower(kr[t]) * px, upper(kr[t]) * py);
            px *= w[t].x;
            py *= w[t].y;
        }
        // The weights within the segment.  Columns m and 16 - m of its lower triangle have 16 entries: one is (row p, column m) for p >= m
        // and (row 16 - m + p, column 16 - m) for p < m.  Two such pairs of columns are summed over the lanes at a time.
        auto column = [&](int m, float* val, int from, int count, int row0) {      // entries row0 .. row0 + count - 1 of column m into val[from ...]
            float gx = lower(kr[m]), gy = upper(kr[m]);
#pragma unroll
            for (int p = 0; p < SEG; ++p) {
                if (p >= count) break;
                const int t = row0 + p;
                if (t == m) val[from + p] = fmaf(lower(rr[t]) * u.x, gx, upper(rr[t]) * u.y * gy);
                else {
                    val[from + p] = fmaf(lower(rr[t]), gx, upper(rr[t]) * gy);
                    gx *= w[t].x;
                    gy *= w[t].y;
                }
            }
        };
#pragma unroll
        for (int m = 0; m <= SEG / 2; m += 2) {
            float val[32];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int col = m + h;
                if (col > SEG / 2) {
#pragma unroll
                    for (int p = 0; p < SEG; ++p) val[h * 16 + p] = 0.f;
                    continue;
                }
                column(col, val, h * 16 + col, SEG - col, col);
                if (col > 0 && col < SEG / 2) column(SEG - col, val, h * 16, col, SEG - col);
                if (col == SEG / 2)
#pragma unroll
                    for (int p = 0; p < SEG / 2; ++p) val[h * 16 + p] = val[h * 16 + SEG / 2 + p];
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                const bool up = lane & off;
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (i < off) {
                        const float give = up ? val[i] : val[i + off], keep = up ? val[i + off] : val[i];
                        val[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
                    }
            }
            const int col = m + (lane >> 4), p = lane & 15;
            if (col <= SEG / 2) {
                if (p >= col) s.a[warp][p][col] = val[0];
                else s.a[warp][SEG - col + p][SEG - col] = val[0];
            }
        }
    }
    cp_async_wait<0>();
    __syncthreads();

    float o[D / 8][4] = {};
    const int br = (lane & 7) + ((lane >> 4) << 3), bc = ((lane >> 3) & 1) << 3;        // rows of n, columns of k
    const int tr = (lane & 7) + (((lane >> 3) & 1) << 3), tc = (lane >> 4) << 3;        // rows of k, columns of n
    const bool live = warp * SEG < len;
    auto values = [&](int seg, uint32_t (&b)[4][4]) {
#pragma unroll
        for (int n = 0; n < 4; ++n) ldmatrix_x4_trans(smem_u32(&s.v[seg * SEG + tr][n * 16 + tc]), b[n][0], b[n][1], b[n][2], b[n][3]);
    };
    // o += (16 weights a row, in three parts) . a segment's values
    auto product = [&](const uint32_t (&p)[3][4], const uint32_t (&b)[4][4]) {
        float sum[D / 8][4] = {};
#pragma unroll
        for (int q = 2; q >= 0; --q)
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                mma_bf16(sum[2 * n], p[q], b[n][0], b[n][1]);
                mma_bf16(sum[2 * n + 1], p[q], b[n][2], b[n][3]);
            }
        add<D / 8>(o, sum);
    };
    float R[4][8];                         // r_t p_t (times the W between), a lane's fragments
    if (live) {
        {   // ---- the segment's own tokens
            uint32_t p[3][4], b[4][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int t = g + (q & 1) * 8, col = 2 * c + (q >> 1) * 8;
                const float x = col <= t ? s.a[warp][t][col] : 0.f, y = col + 1 <= t ? s.a[warp][t][col + 1] : 0.f;
                split3(x, y, p[0][q], p[1][q], p[2][q]);
            }
            values(warp, b);
            // A weight of zero takes finite values away, but not infinities and NaN: those are left out of the product and meet the tokens
            // that see them one by one.
            bool odd = false;
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int q = 0; q < 4; ++q) odd |= (b[n][q] & 0x7f80u) == 0x7f80u || (b[n][q] & 0x7f800000u) == 0x7f800000u;
            odd = __any_sync(0xffffffffu, odd);
            if (!odd) product(p, b);
            else {
#pragma unroll 1
                for (int k = 0; k < SEG; ++k) {
                    const float w_lo = k <= g ? s.a[warp][g][k] : 0.f, w_hi = k <= g + 8 ? s.a[warp][g + 8][k] : 0.f;
#pragma unroll
                    for (int n = 0; n < D / 8; ++n) {
                        const uint32_t pair = *reinterpret_cast<const uint32_t*>(&s.v[warp * SEG + k][n * 8 + 2 * c]);
                        if (k <= g) {
                            o[n][0] = fmaf(w_lo, lower(pair), o[n][0]);
                            o[n][1] = fmaf(w_lo, upper(pair), o[n][1]);
                        }
                        if (k <= g + 8) {
                            o[n][2] = fmaf(w_hi, lower(pair), o[n][2]);
                            o[n][3] = fmaf(w_hi, upper(pair), o[n][3]);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 x = *reinterpret_cast<const float2*>(&s.r[warp * SEG + g + (q & 1) * 8][kk * 16 + 2 * c + (q >> 1) * 8]);
                R[kk][2 * q] = x.x;
                R[kk][2 * q + 1] = x.y;
            }
        // ---- the segments before, nearest first
        for (int j = warp - 1; j >= 0; --j) {
            float sc[2][4] = {};
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                uint32_t p[3][4], b[3][4];
#pragma unroll
                for (int q = 0; q < 4; ++q) split3(R[kk][2 * q], R[kk][2 * q + 1], p[0][q], p[1][q], p[2][q]);
#pragma unroll
                for (int q = 0; q < 3; ++q) ldmatrix_x4(smem_u32(&s.k[q][j * SEG + br][kk * 16 + bc]), b[q][0], b[q][1], b[q][2], b[q][3]);
                float low[2][4] = {}, high[2][4] = {};
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    mma_bf16(low[n], p[2], b[0][2 * n], b[0][2 * n + 1]);
                    mma_bf16(high[n], p[1], b[0][2 * n], b[0][2 * n + 1]);
                    mma_bf16(low[n], p[0], b[2][2 * n], b[2][2 * n + 1]);
                    mma_bf16(high[n], p[0], b[1][2 * n], b[1][2 * n + 1]);
                    mma_bf16(low[n], p[1], b[1][2 * n], b[1][2 * n + 1]);
                    mma_bf16(high[n], p[0], b[0][2 * n], b[0][2 * n + 1]);
                }
                add<2>(high, low);
                add<2>(sc, high);
                // the next segment is one further away
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 f = *reinterpret_cast<const float2*>(&s.w[j][kk * 16 + 2 * c + h * 8]);
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        R[kk][4 * h + 2 * q] *= f.x;
                        R[kk][4 * h + 2 * q + 1] *= f.y;
                    }
                }
            }
            uint32_t p[3][4], b[4][4];
            split3(sc[0][0], sc[0][1], p[0][0], p[1][0], p[2][0]);
            split3(sc[0][2], sc[0][3], p[0][1], p[1][1], p[2][1]);
            split3(sc[1][0], sc[1][1], p[0][2], p[1][2], p[2][2]);
            split3(sc[1][2], sc[1][3], p[0][3], p[1][3], p[2][3]);
            values(j, b);
            product(p, b);
        }
    }
    // ---- what the starting state answers
    __syncthreads();                                           // the keys have been read
#pragma unroll
    for (int k = 0; k < D * D / 2 / THREADS; ++k) {
        const int e = k * THREADS + threadIdx.x, i = e / (D / 2), j = e % (D / 2) * 2;
        const float2 x = *reinterpret_cast<const float2*>(&s.s0[i][j]);
        put(s.k, i, j, x.x, x.y);
    }
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        if (kk * 16 >= d) break;
        uint32_t p[3][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) split3(R[kk][2 * q], R[kk][2 * q + 1], p[0][q], p[1][q], p[2][q]);
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            uint32_t b[3][4];
#pragma unroll
            for (int q = 0; q < 3; ++q) ldmatrix_x4_trans(smem_u32(&s.k[q][kk * 16 + tr][n * 16 + tc]), b[q][0], b[q][1], b[q][2], b[q][3]);
            float low[2][4] = {}, high[2][4] = {};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                mma_bf16(low[h], p[2], b[0][2 * h], b[0][2 * h + 1]);
                mma_bf16(high[h], p[1], b[0][2 * h], b[0][2 * h + 1]);
                mma_bf16(low[h], p[0], b[2][2 * h], b[2][2 * h + 1]);
                mma_bf16(high[h], p[0], b[1][2 * h], b[1][2 * h + 1]);
                mma_bf16(low[h], p[1], b[1][2 * h], b[1][2 * h + 1]);
                mma_bf16(high[h], p[0], b[0][2 * h], b[0][2 * h + 1]);
            }
            add<2>(high, low);
            add<2>(&o[2 * n], high);
        }
    }
    float* dst = a.y + (tok0 + warp * SEG) * hd + (size_t)head * d;
#pragma unroll
    for (int n = 0; n < D / 8; ++n) {
        const int col = n * 8 + 2 * c;
        if (col >= d) continue;
        if (warp * SEG + g < len) *reinterpret_cast<float2*>(dst + (size_t)g * hd + col) = make_float2(o[n][0], o[n][1]);
        if (warp * SEG + g + 8 < len) *reinterpret_cast<float2*>(dst + (size_t)(g + 8) * hd + col) = make_float2(o[n][2], o[n][3]);
    }
}

}  // namespace wkvc
}  // namespace lily

using namespace lily;

// Whether the chunk kernels take the shape (bfloat16 activations): heads of up to 64 in whole tiles, rows on 16 bytes.
LILY_API int lily_wkv_chunk_takes(const void* r, const void* k, const void* v, int in_stride, const float* lw, const float* u, int heads, int d, int chunk) {
    return (((uintptr_t)lw | (uintptr_t)u) & 7) == 0 && d >= 16 && d <= wkvc::D && d % 16 == 0 && chunk <= wkvc::CHUNK && in_stride % 8 == 0 &&
           (((uintptr_t)r | (uintptr_t)k | (uintptr_t)v) & 15) == 0 && heads <= 0x7fffffff / wkvc::D;
}

// outputs 0: the chunks' own states and decays; 1: the outputs from the starting states that wkv_combine left.
LILY_API int lily_wkv_chunk(const void* r, const void* k, const void* v, int in_stride, const float* lw, const float* u, float* y,
                            const int* cu_seqlens, int items, int heads, int d, const int* item_req, const int* item_start, const int* item_len,
                            float* ws_state, float* ws_decay, int chunk, int outputs, cudaStream_t stream) {
    if (items == 0) return 0;
    LILY_REQUIRE(heads > 0 && items <= 65535 && lily_wkv_chunk_takes(r, k, v, in_stride, lw, u, heads, d, chunk), "wkv_chunk: %d chunks of %d, %d heads of %d",
                 items, chunk, heads, d);
    LILY_REQUIRE((((uintptr_t)ws_state) & 15) == 0 && (((uintptr_t)y | (uintptr_t)ws_decay) & 7) == 0,
                 "wkv_chunk: operands do not start on 16 bytes");
    const wkvc::Args a{(const __nv_bfloat16*)r, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, in_stride, lw, u, y, cu_seqlens, item_req, item_start,
                       item_len, ws_state, ws_decay, heads, d};
    const int smem = outputs ? (int)sizeof(wkvc::ReadTile) : (int)sizeof(wkvc::WriteTile);
    auto kern = outputs ? wkvc::read_kernel : wkvc::write_kernel;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    LILY_REQUIRE(e == cudaSuccess, "wkv_chunk: cannot get %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
    launch_pdl(kern, dim3(heads, items), dim3(wkvc::THREADS), smem, stream, a);
    LILY_CHECK_LAUNCH("wkv_chunk");
    return 0;
}
