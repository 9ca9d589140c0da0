// The gated delta rule (see delta_rule.cu) over chunks of a prompt in bfloat16, on the tensor cores (mma.sync m16n8k16, float32
// accumulation).
//
// With L_t the sum of the log decays up to and with token t of a chunk that starts from S_0, g_t = e^(L_t), and k, q the unit vectors:
//
//     (1 + A) U = R,   A_ts = b_t e^(L_t - L_s) (k_t . k_s) for s < t,   r_t = b_t (v_t - g_t S_0^T k_t)
//     o_t = g_t S_0^T q_t + sum_(s <= t) e^(L_t - L_s) (q_t . k_s) u_s,   S_end = e^L S_0 + sum_s e^(L - L_s) k_s u_s^T
//
// (the chunked form of Yang, Wang, Zhang, Shen and Kim, "Parallelizing Linear Transformers with the Delta Rule over Sequence Length",
// 2024, with decays).
//
//   delta_prepare  what does not depend on the state, for all chunks side by side: a block a (chunk, query/key head) forms the products
//                  of the chunk's keys and queries once for the value heads that share them, then per value head T = (1 + A)^-1 by
//                  forward substitution, a thread a column, and M (the weights of the u_s in o_t), in float32
//   delta_chunks   the chunks of a request one after another: a block 16 value columns of a head, two teams of eight warps with eight
//                  columns each, the state in the registers of the product that updates it; warps 0 to 3 of a team have the keys' rows
//                  (R, U = T R), 4 to 7 the queries' (o); the next chunk's keys, queries, T and M arrive asynchronously
//
// q, k and v are the convolution's own bfloat16 numbers, the unit vectors' divisors stay factors of the rows.  What meets the tensor cores as
// float32 (S, R, U, T, M) is cut into the sum of three bfloat16 numbers, all 24 bits of it; of two such numbers the products down to
// 2^-27 are taken.  Runs of 16 products are added to a total by rounded additions.  The L are summed in float64 and kept as two
// float32.  What is not finite stays behind its token, as token by token.
// Bound by the chain of a chunk (products with the state, R, U, the state again: three barriers) and by the reads of shared memory that
// feed its products, 3,200 of its 6,900 cycles: 3.6 us for 64 tokens where 64 tokens one after another take 27.  1,999 tokens, 16 heads of 128 x 128:
// 843 -> 141 us, of them the preparation 20.  (One team of 16 columns and 256 threads, two blocks a SM: 202; T and M cut into parts by
// their readers: 226.)  Against 64 bits the outputs are 1.2e-7 to 3.8e-7 off in the 2-norm, where they were 1.2e-7 to 2.5e-6.
#include "common.cuh"
#include "mma.cuh"

namespace lily {
namespace deltac {

using namespace mma16;

constexpr int CHUNK = 64;                  // tokens of a chunk
constexpr int BLOCKS = CHUNK / 16;         // rows of 16 x 16 tiles; T and M are their lower triangles, tile by tile
constexpr int TILES = BLOCKS * (BLOCKS + 1) / 2;
constexpr int DMAX = 128;                  // head size of queries and keys, at most (a multiple of 16)
constexpr int THREADS = 256;               // of delta_prepare
constexpr int COLS = 8;                    // value columns of eight warps
constexpr int TEAMS = 2;                   // such groups of warps in a block of delta_chunks
constexpr int SIDE = 4;                    // value heads a block of delta_prepare works on at a time
constexpr int PAD = 8;                     // an odd number of 16-byte pieces a row: ldmatrix without bank conflicts

// The workspace of a (chunk, value head), in words: T, M (their tiles' three parts in the order of a lane's fragment: [tile][part][lane][4]), then
// the tokens' factors (b, b g / |k|, g q_scale / |q|, e^(L - L_t) / |k|) and e^L.
constexpr int TILE_WORDS = 3 * 32 * 4, FACTORS = 2 * TILES * TILE_WORDS, END = FACTORS + CHUNK * 4, FLOATS = END + 4;

struct Args {
    const __nv_bfloat16* qkv;              // [tokens, qkv_stride]
    int qkv_stride, q_col, k_col, v_col;
    const __nv_bfloat16* proj;
    int proj_stride, b_col, a_col;
    const float* a_log;
    const float* dt_bias;
    float* state;                          // [slots, state_stride]: [heads][dv][d]
    size_t state_stride;
    float* y;                              // [tokens, heads * dv]
    const int* cu_seqlens;
    const int* slots;
    const int* item_req;                   // [items]: request of each chunk
    const int* item_start;                 // [items]: its first token
    const int* first_item;                 // [requests]: a request's first chunk
    float* work;                           // [items, heads, FLOATS]
    int heads, kv_heads, d, dv;
    float unit_eps, q_scale;
};

__device__ __forceinline__ void stage_rows(__nv_bfloat16* dst, const __nv_bfloat16* src, size_t ld, int rows, int d) {
    const int per = d / 8;
    for (int e = threadIdx.x; e < CHUNK * per; e += THREADS) {
        const int r = e / per, c = (e % per) * 8;
        cp_async16(smem_u32(dst + r * (DMAX + PAD) + c), src + (r < rows ? (size_t)r * ld + c : 0), r < rows);
    }
}

// e^x of a sum of decays, to float32
__device__ __forceinline__ float exp_of(double x) {
    const float hi = (float)x, e = expf(hi);
    return fmaf(e, (float)(x - (double)hi), e);
}

// f x for a product x of two rows that may have overflowed: then one of the rows' divisors in f is zero, and so is the product of the unit vectors
__device__ __forceinline__ float times(float f, float x) { return f == 0.f ? 0.f : f * x; }

__device__ __forceinline__ int tile_of(int i, int j) { return i * (i + 1) / 2 + j; }      // the lower triangle's tiles, row by row

struct Prepare {
    __nv_bfloat16 k[CHUNK][DMAX + PAD], q[CHUNK][DMAX + PAD];
    float kk[CHUNK][CHUNK + 1], qk[CHUNK][CHUNK + 1];         // the raw products
    float a[SIDE][CHUNK][CHUNK + 4];                          // below the diagonal A, from it on the transposed M
    float x[SIDE][CHUNK][CHUNK];                              // T as it is solved: [row][column]
    float fk[CHUNK], fq[CHUNK], b[SIDE][CHUNK], hi[SIDE][CHUNK], lo[SIDE][CHUNK];
    double warp_sum[THREADS / 32];
};

// grid (items, kv_heads)
__global__ void __launch_bounds__(THREADS) prepare_kernel(const Args a) {
    extern __shared__ __align__(16) unsigned char smem[];
    Prepare& s = *reinterpret_cast<Prepare*>(smem);
    pdl_wait();
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
    const int item = blockIdx.x, kvh = blockIdx.y, req = a.item_req[item], start = a.item_start[item];
    const size_t tok0 = (size_t)a.cu_seqlens[req] + start;
    const int len = min(CHUNK, a.cu_seqlens[req + 1] - a.cu_seqlens[req] - start), group = a.heads / a.kv_heads;
    stage_rows(&s.k[0][0], a.qkv + tok0 * a.qkv_stride + a.k_col + (size_t)kvh * a.d, a.qkv_stride, len, a.d);
    stage_rows(&s.q[0][0], a.qkv + tok0 * a.qkv_stride + a.q_col + (size_t)kvh * a.d, a.qkv_stride, len, a.d);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    {                                                          // the divisors: four threads a token
        const int t = tid >> 2;
        float sk = 0.f, sq = 0.f;
        for (int i = tid & 3; i < a.d; i += 4) {
            const float x = __bfloat162float(s.k[t][i]), z = __bfloat162float(s.q[t][i]);
            sk = fmaf(x, x, sk + (x - x));                     // an infinity makes the divisor a NaN, squares that overflow a zero
            sq = fmaf(z, z, sq + (z - z));
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            sk += __shfl_xor_sync(0xffffffffu, sk, o);
            sq += __shfl_xor_sync(0xffffffffu, sq, o);
        }
        if ((tid & 3) == 0) {
            s.fk[t] = 1.f / sqrtf(sk + a.unit_eps);
            s.fq[t] = a.q_scale / sqrtf(sq + a.unit_eps);
        }
    }
    {                                                          // warps 0 to 3: rows of k . k, 4 to 7: of q . k
        const int row = (warp & 3) * 16;
        const __nv_bfloat16(*rows)[DMAX + PAD] = warp < 4 ? s.k : s.q;
        float(*out)[CHUNK + 1] = warp < 4 ? s.kk : s.qk;
        for (int j = 0; j <= (warp & 3); ++j) {
            float sc[2][4] = {};
            for (int kk = 0; kk < a.d / 16; ++kk) {
                uint32_t q[4], b[4];
                ldmatrix_x4(smem_u32(&rows[row + (lane & 15)][kk * 16 + ((lane >> 4) << 3)]), q[0], q[1], q[2], q[3]);
                ldmatrix_x4(smem_u32(&s.k[j * 16 + (lane & 7) + ((lane >> 4) << 3)][kk * 16 + (((lane >> 3) & 1) << 3)]), b[0], b[1], b[2], b[3]);
                float sum[2][4] = {};
                mma_bf16(sum[0], q, b[0], b[1]);
                mma_bf16(sum[1], q, b[2], b[3]);
                add<2>(sc, sum);
            }
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) out[row + g + (e >> 1) * 8][j * 16 + n * 8 + 2 * c + (e & 1)] = sc[n][e];
        }
    }
    const int side = tid / CHUNK, t = tid % CHUNK;            // a thread a (value head, token or column)
    for (int h0 = 0; h0 < group; h0 += SIDE) {
        const int head = kvh * group + h0 + side;
        const bool on = h0 + side < group;
        float b = 0.f;
        double L = 0.0;
        if (on && t < len) {
            const __nv_bfloat16* row = a.proj + (tok0 + t) * a.proj_stride + head;
            const float alpha = __bfloat162float(row[a.a_col]) + a.dt_bias[head];
            const float step = -expf(a.a_log[head]) * (alpha > 20.f ? alpha : log1pf(expf(alpha)));
            b = 1.f / (1.f + expf(-__bfloat162float(row[a.b_col])));
            L = (double)(step < -200.f ? -200.f : step);       // e^-200 is zero in float32 (a NaN stays one)
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double left = __shfl_up_sync(0xffffffffu, L, o);
            if (lane >= o) L += left;
        }
        if (lane == 31) s.warp_sum[warp] = L;
        __syncthreads();                                       // (also behind the last round's readers and the products)
        if (warp & 1) L += s.warp_sum[warp - 1];
        const double total = s.warp_sum[warp | 1] + s.warp_sum[warp & ~1];
        const float hi = (float)L, lo = (float)(L - (double)hi);
        s.b[side][t] = b;
        s.hi[side][t] = hi;
        s.lo[side][t] = lo;
        __syncthreads();
        float* work = a.work + ((size_t)item * a.heads + head) * FLOATS;
        if (on) {
            const float decay = exp_of(L), rest = exp_of(total - L);
            *reinterpret_cast<float4*>(work + FACTORS + t * 4) =
                t < len ? make_float4(b, b * decay * s.fk[t], decay * s.fq[t], rest * s.fk[t]) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (t == 0) work[END] = exp_of(total);
            // A and M: column t, a row a turn
            const float own = s.fk[t];
            for (int r = t; r < CHUNK; ++r) {
                const float w = expf((s.hi[side][r] - hi) + (s.lo[side][r] - lo)) * own;
                if (r > t) s.a[side][r][t] = times(s.b[side][r] * s.fk[r] * w, s.kk[r][t]);
                s.a[side][t][r] = times(s.fq[r] * w, s.qk[r][t]);
            }
        }
        __syncthreads();
        if (on) {
            // T, column t: eight rows at a time, what the rows above give first
            for (int r0 = 0; r0 < CHUNK; r0 += 8) {
                float acc[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) acc[r] = r0 + r == t ? 1.f : 0.f;
                for (int k = t & ~31; k < r0; k += 4) {       // the column begins with zeros
                    const float x0 = s.x[side][k][t], x1 = s.x[side][k + 1][t], x2 = s.x[side][k + 2][t], x3 = s.x[side][k + 3][t];
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        const float4 w = *reinterpret_cast<const float4*>(&s.a[side][r0 + r][k]);
                        acc[r] = fmaf(-w.w, x3, fmaf(-w.z, x2, fmaf(-w.y, x1, fmaf(-w.x, x0, acc[r]))));
                    }
                }
#pragma unroll
                for (int r = 0; r < 8; ++r) {
#pragma unroll
                    for (int k = 0; k < r; ++k) acc[r] = fmaf(-s.a[side][r0 + r][r0 + k], acc[k], acc[r]);
                    acc[r] = r0 + r >= t ? acc[r] : 0.f;
                    s.x[side][r0 + r][t] = acc[r];
                }
            }
        }
        __syncthreads();
        // T and M in three parts: a thread a lane of a tile
        const int heads_on = min(SIDE, group - h0);
        for (int e = tid; e < heads_on * 2 * TILES * 32; e += THREADS) {
            const int at = e & 31, tile = (e >> 5) % TILES, which = (e >> 5) / TILES, hs = which >> 1;
            const int ti = tile >= 6 ? 3 : (tile >= 3 ? 2 : (tile >= 1 ? 1 : 0)), tj = tile - tile_of(ti, 0);
            uint32_t p[3][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = ti * 16 + (at >> 2) + (q & 1) * 8, col = tj * 16 + (at & 3) * 2 + (q >> 1) * 8;
                float v[2];
#pragma unroll
                for (int o = 0; o < 2; ++o) v[o] = col + o > r ? 0.f : ((which & 1) ? s.a[hs][col + o][r] : s.x[hs][r][col + o]);
                split3(v[0], v[1], p[0][q], p[1][q], p[2][q]);
            }
            uint32_t* dst = reinterpret_cast<uint32_t*>(a.work + ((size_t)item * a.heads + kvh * group + h0 + hs) * FLOATS) +
                            ((which & 1) * TILES + tile) * TILE_WORDS + at * 4;
#pragma unroll
            for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(dst + q * 128) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
        }
    }
}

struct Stage {
    __nv_bfloat16 k[CHUNK][DMAX + PAD], q[CHUNK][DMAX + PAD];
    uint32_t tm[2][TILES * TILE_WORDS];                        // T, M
};
struct Team {                                                  // rows of eight columns: 16 bytes, ldmatrix without bank conflicts
    __nv_bfloat16 st[3][DMAX][COLS];                           // the state's three parts
    __nv_bfloat16 r[3][CHUNK][COLS], u[3][CHUNK][COLS], w[3][CHUNK][COLS];      // R, U, e^(L - L_s) U / |k_s|
    int odd[BLOCKS];                                           // whether U's rows of a tile hold an infinity or a NaN
};
struct Tile {
    Stage stage[2];
    Team team[TEAMS];
};

__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u; }

// o += row i of the lower triangle's tiles times the rows of `rows`; `odd`: the rows of the tile on the diagonal hold an infinity or
// a NaN, and are taken entry by entry so that a zero above the diagonal meets none.
__device__ __forceinline__ void triangle(float (&o)[4], const uint32_t* tiles, const __nv_bfloat16 (*rows)[CHUNK][COLS], int i, bool odd, int lane) {
    const uint32_t* mine = tiles + tile_of(i, 0) * TILE_WORDS + lane * 4;
#pragma unroll
    for (int j = 0; j < BLOCKS; ++j) {
        if (j > i || (j == i && odd)) continue;
        uint32_t p[3][4], b[3][2], none[2];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const uint4 f = *reinterpret_cast<const uint4*>(mine + j * TILE_WORDS + q * 128);
            p[q][0] = f.x, p[q][1] = f.y, p[q][2] = f.z, p[q][3] = f.w;
        }
        // lanes 0 to 15 name the rows of one part, 16 to 31 those of another
        ldmatrix_x4_trans(smem_u32(&rows[lane >> 4][j * 16 + (lane & 15)][0]), b[0][0], b[0][1], b[1][0], b[1][1]);
        ldmatrix_x4_trans(smem_u32(&rows[2][j * 16 + (lane & 15)][0]), b[2][0], b[2][1], none[0], none[1]);
        // of the products of parts those down to 2^-27, the small ones in sums of their own
        float low[4] = {}, mid[4] = {}, high[4] = {};
        mma_bf16(low, p[2], b[0][0], b[0][1]);
        mma_bf16(mid, p[1], b[0][0], b[0][1]);
        mma_bf16(high, p[0], b[0][0], b[0][1]);
        mma_bf16(low, p[0], b[2][0], b[2][1]);
        mma_bf16(mid, p[0], b[1][0], b[1][1]);
        mma_bf16(low, p[1], b[1][0], b[1][1]);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] += high[e] + (mid[e] + low[e]);
    }
    if (odd) {
        const int g = lane >> 2, c = lane & 3;
        const uint32_t* tile = tiles + tile_of(i, i) * TILE_WORDS;
#pragma unroll 1
        for (int k = 0; k < 16; ++k) {
            const int at = i * 16 + k;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = g + (e >> 1) * 8, col = 2 * c + (e & 1);
                float w = 0.f, x = 0.f;
#pragma unroll
                for (int q = 2; q >= 0; --q) {
                    const uint32_t pair = tile[q * 128 + (g * 4 + ((k & 7) >> 1)) * 4 + (k >> 3) * 2 + (e >> 1)];
                    w += k & 1 ? upper(pair) : lower(pair);
                    x += __bfloat162float(rows[q][at][col]);
                }
                if (k <= r) o[e] = fmaf(w, x, o[e]);
            }
        }
    }
}

// rows g and g + 8 of a tile (columns 2c and 2c + 1), times their factors, in three parts
__device__ __forceinline__ void put_rows(__nv_bfloat16* dst, int part, const float (&x)[4], float f_lo, float f_hi, int g, int c) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float f = e ? f_hi : f_lo;
        uint32_t p[3];
        split3(x[2 * e] * f, x[2 * e + 1] * f, p[0], p[1], p[2]);
#pragma unroll
        for (int q = 0; q < 3; ++q) *reinterpret_cast<uint32_t*>(dst + q * part + (g + 8 * e) * COLS + 2 * c) = p[q];
    }
}
__device__ __forceinline__ bool any_odd(const float (&x)[4]) {
    return __any_sync(0xffffffffu, not_finite(x[0]) || not_finite(x[1]) || not_finite(x[2]) || not_finite(x[3]));
}

// grid (requests, heads, dv / 16); KS: runs of 16 of the head size, the last ones zeros.  Eight warps a team: 0 to 3 the keys' rows, 4 to 7
// the queries'; a warp's 16 rows of the chunk, and in the state its 16 rows of d.
template <int KS>
__global__ void __launch_bounds__(TEAMS * 256, 1) chunks_kernel(const Args a) {
    extern __shared__ __align__(16) unsigned char smem[];
    Tile& s = *reinterpret_cast<Tile*>(smem);
    pdl_wait();
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, team = tid >> 8, warp = (tid >> 5) & 7, g = lane >> 2, c = lane & 3;
    const int req = blockIdx.x, head = blockIdx.y, v0 = blockIdx.z * (TEAMS * COLS) + team * COLS, kvh = head / (a.heads / a.kv_heads);
    const int tok0 = a.cu_seqlens[req], len = a.cu_seqlens[req + 1] - tok0;
    if (len <= 0) return;
    Team& t = s.team[team];
    const int d = a.d, out_ld = a.heads * a.dv;
    const size_t ld = a.qkv_stride;
    const __nv_bfloat16* base = a.qkv + (size_t)tok0 * ld;
    const __nv_bfloat16 *ksrc = base + a.k_col + (size_t)kvh * d, *qsrc = base + a.q_col + (size_t)kvh * d;
    const __nv_bfloat16* vsrc = base + a.v_col + (size_t)head * a.dv + v0;
    const float* work = a.work + ((size_t)a.first_item[req] * a.heads + head) * FLOATS;
    const size_t work_step = (size_t)a.heads * FLOATS;
    const int i = warp & 3, row = i * 16;
    const bool keys = warp < 4;

    // eight threads a row of keys and queries, then T and M
    auto stage = [&](Stage& dst, int t0, const float* w) {
        const int r = tid >> 3, at = t0 + r;
#pragma unroll
        for (int k = 0; k < (KS + 3) / 4; ++k) {
            const int col = (tid & 7) * 8 + k * 64;
            const bool in = at < len && col < d;
            cp_async16(smem_u32(&dst.k[r][col]), ksrc + (in ? (size_t)at * ld + col : 0), in);
            cp_async16(smem_u32(&dst.q[r][col]), qsrc + (in ? (size_t)at * ld + col : 0), in);
        }
        constexpr int PIECES = FACTORS / 4;
#pragma unroll
        for (int k = 0; k < (PIECES + TEAMS * 256 - 1) / (TEAMS * 256); ++k) {
            const int e = k * TEAMS * 256 + tid;
            if (e < PIECES) cp_async16(smem_u32(&dst.tm[0][0] + e * 4), w + e * 4, true);
        }
    };
    float4 fac[2];                                             // the rows' factors
    uint32_t v[2] = {};
    float end = 0.f;
    auto fetch = [&](const float* w, int t0) {
        const float4* factors = reinterpret_cast<const float4*>(w + FACTORS);
        fac[0] = factors[row + g];
        fac[1] = factors[row + g + 8];
        end = w[END];
        if (keys) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int at = t0 + row + g + e * 8;
                v[e] = at < len ? *reinterpret_cast<const uint32_t*>(vsrc + (size_t)at * ld + 2 * c) : 0u;
            }
        }
    };
    stage(s.stage[0], 0, work);
    cp_async_commit();
    fetch(work, 0);

    // the state: rows d of this warp's 16, value columns 2c and 2c + 1
    const bool holds = warp * 16 < d;
    float* st = a.state + (size_t)a.slots[req] * a.state_stride + ((size_t)head * a.dv + v0 + 2 * c) * d + warp * 16 + g;
    float S[4] = {};
    if (holds) S[0] = st[0], S[1] = st[d], S[2] = st[8], S[3] = st[d + 8];
    if (warp < KS) put_rows(&t.st[0][warp * 16][0], DMAX * COLS, S, 1.f, 1.f, g, c);        // zeros beyond d
    cp_async_wait<0>();
    __syncthreads();

    for (int t0 = 0, buf = 0; t0 < len; t0 += CHUNK, buf ^= 1) {
        const Stage& now = s.stage[buf];
        const bool more = t0 + CHUNK < len;
        if (more) stage(s.stage[buf ^ 1], t0 + CHUNK, work + work_step);
        cp_async_commit();
        // ---- this warp's rows times the state
        float acc[4] = {};
        const __nv_bfloat16* rows = (keys ? &now.k[0][0] : &now.q[0][0]) + (row + (lane & 15)) * (DMAX + PAD) + ((lane >> 4) << 3);
#pragma unroll
        for (int kk = 0; kk < KS; kk += 2) {                   // two runs at a time: one ldmatrix for a part of both
            uint32_t q[2][4], b[3][4];
            ldmatrix_x4(smem_u32(rows + kk * 16), q[0][0], q[0][1], q[0][2], q[0][3]);
            ldmatrix_x4(smem_u32(rows + kk * 16 + 16), q[1][0], q[1][1], q[1][2], q[1][3]);
#pragma unroll
            for (int part = 0; part < 3; ++part) ldmatrix_x4_trans(smem_u32(&t.st[part][kk * 16 + lane][0]), b[part][0], b[part][1], b[part][2], b[part][3]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float sum[4] = {};
#pragma unroll
                for (int part = 2; part >= 0; --part) mma_bf16(sum, q[h], b[part][2 * h], b[part][2 * h + 1]);
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[e] += sum[e];
            }
        }
        if (keys) {
            // ---- R, then U = T R, as it is and weighed for the state
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float value = e & 1 ? upper(v[e >> 1]) : lower(v[e >> 1]);
                acc[e] = fac[e >> 1].x * value - fac[e >> 1].y * acc[e];
            }
            put_rows(&t.r[0][row][0], CHUNK * COLS, acc, 1.f, 1.f, g, c);
            const bool odd = any_odd(acc);
            asm volatile("bar.sync %0, 128;\n" ::"r"(1 + team) : "memory");
            float U[4] = {};
            triangle(U, now.tm[0], t.r, i, odd, lane);
            put_rows(&t.u[0][row][0], CHUNK * COLS, U, 1.f, 1.f, g, c);
            put_rows(&t.w[0][row][0], CHUNK * COLS, U, fac[0].w, fac[1].w, g, c);
            const bool odd_u = any_odd(U);
            if (lane == 0) t.odd[i] = odd_u;
        }
        asm volatile("bar.sync %0, 256;\n" ::"r"(3 + team) : "memory");
        if (holds) {
            // ---- the state behind the chunk
#pragma unroll
            for (int e = 0; e < 4; ++e) S[e] *= end;
#pragma unroll
            for (int k32 = 0; k32 < BLOCKS / 2; ++k32) {
                uint32_t q[2][4], b[3][4];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    ldmatrix_x4_trans(smem_u32(&now.k[k32 * 32 + h * 16 + (lane & 7) + ((lane >> 4) << 3)][warp * 16 + (((lane >> 3) & 1) << 3)]), q[h][0], q[h][1], q[h][2], q[h][3]);
#pragma unroll
                for (int part = 0; part < 3; ++part) ldmatrix_x4_trans(smem_u32(&t.w[part][k32 * 32 + lane][0]), b[part][0], b[part][1], b[part][2], b[part][3]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float sum[4] = {};
#pragma unroll
                    for (int part = 2; part >= 0; --part) mma_bf16(sum, q[h], b[part][2 * h], b[part][2 * h + 1]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) S[e] += sum[e];
                }
            }
            put_rows(&t.st[0][warp * 16][0], DMAX * COLS, S, 1.f, 1.f, g, c);
        }
        if (!keys) {
            // ---- outputs
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[e] *= fac[e >> 1].z;
            triangle(acc, now.tm[1], t.u, i, t.odd[i] != 0, lane);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int at = t0 + row + g + 8 * e;
                if (at < len)
                    *reinterpret_cast<float2*>(a.y + (size_t)(tok0 + at) * out_ld + (size_t)head * a.dv + v0 + 2 * c) = make_float2(acc[2 * e], acc[2 * e + 1]);
            }
        }
        work += work_step;
        if (more) fetch(work, t0 + CHUNK);
        cp_async_wait<0>();
        __syncthreads();
    }
    if (holds) st[0] = S[0], st[d] = S[1], st[8] = S[2], st[d + 8] = S[3];
}

}  // namespace deltac
}  // namespace lily

using namespace lily;

// Whether the chunk kernels take the shape (bfloat16 activations): heads of whole tiles, rows on 16 bytes.
LILY_API int lily_delta_chunks_take(const void* qkv, int qkv_stride, int q_col, int k_col, int v_col, int heads, int kv_heads, int d, int dv) {
    return d >= 16 && d <= deltac::DMAX && d % 16 == 0 && dv >= 16 && dv % 16 == 0 && dv / 16 <= 65535 && heads <= 65535 &&
           (uintptr_t)qkv % 16 == 0 && (qkv_stride | q_col | k_col | v_col) % 8 == 0 && heads % kv_heads == 0;
}
LILY_API int lily_delta_chunk_tokens() { return deltac::CHUNK; }
LILY_API int lily_delta_chunk_floats() { return deltac::FLOATS; }

LILY_API int lily_delta_chunks(const void* qkv, int qkv_stride, int q_col, int k_col, int v_col, const void* proj, int proj_stride,
                               int b_col, int a_col, const float* a_log, const float* dt_bias, float* state, size_t state_stride,
                               float* y, const int* cu_seqlens, const int* slots, int requests, const int* item_req, const int* item_start,
                               const int* first_item, int items, float* work, int heads, int kv_heads, int d, int dv, float unit_eps,
                               float q_scale, cudaStream_t stream) {
    if (requests == 0 || items == 0) return 0;
    LILY_REQUIRE(heads > 0 && kv_heads > 0 && lily_delta_chunks_take(qkv, qkv_stride, q_col, k_col, v_col, heads, kv_heads, d, dv),
                 "delta_chunks: %d heads over %d of %d x %d", heads, kv_heads, d, dv);
    LILY_REQUIRE((size_t)heads * d * dv <= state_stride && ((uintptr_t)work & 15) == 0 &&
                     ((uintptr_t)y & 7) == 0, "delta_chunks: state, workspace or outputs of %d matrices of %d x %d", heads, d, dv);
    const deltac::Args a{(const __nv_bfloat16*)qkv, qkv_stride, q_col, k_col, v_col, (const __nv_bfloat16*)proj, proj_stride, b_col, a_col,
                         a_log, dt_bias, state, state_stride, y, cu_seqlens, slots, item_req, item_start, first_item, work, heads, kv_heads,
                         d, dv, unit_eps, q_scale};
    auto chunks = d <= 64 ? deltac::chunks_kernel<4> : deltac::chunks_kernel<8>;
    cudaError_t e = cudaFuncSetAttribute(deltac::prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(deltac::Prepare));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(chunks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(deltac::Tile));
    LILY_REQUIRE(e == cudaSuccess, "delta_chunks: cannot get the shared memory: %s", cudaGetErrorString(e));
    launch_pdl(deltac::prepare_kernel, dim3(items, kv_heads), dim3(deltac::THREADS), sizeof(deltac::Prepare), stream, a);
    launch_pdl(chunks, dim3(requests, heads, dv / (deltac::TEAMS * deltac::COLS)), dim3(deltac::TEAMS * 256), sizeof(deltac::Tile), stream, a);
    LILY_CHECK_LAUNCH("delta_chunks");
    return 0;
}
