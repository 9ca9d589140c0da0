// Decode attention in float32 (one query token a request) for head sizes that are multiples of four up to 256 and up to eight
// query heads a kv head: the other shapes of the 32-bit path stay with attention_simt.cu, whose cache layout, key ranges,
// scratch and options these are.
//
// A decode row is a chain of trips to memory and little arithmetic, so the keys are cut over warps: warp w of a block takes
// four neighbouring keys of every 4 * WARPS, for all query heads of the kv head.  A lane holds four neighbouring columns (and the four
// 128 columns further) of the queries and of the outputs, so a key or value row is one coalesced read straight into registers, the
// next four keys' while these are worked on; the scores of 4 keys x G heads are summed over the lanes by halving what a lane
// holds at each exchange (31 exchanges for 32 sums, where a sum alone takes five).  Each warp keeps its own (max, sum,
// output), merged in the order of the warps at the end.  Nothing passes through shared memory but the weights and that merge.
// Against the tiles of attention_simt.cu, us: 3 rows of 250 keys, 16 heads of 128 over 4: 39 -> 10.7 (6.8 in four ranges); 8 rows of
// 1,000: 56 -> 14; 64 rows of 1,000 over 8 kv heads: 348 -> 134; 64 of 4,000, 32 heads over 4: 1,270 -> 506 (4.3 TB/s); heads of 16
// over 8: 160 -> 99; 20 heads of 40, no sharing: 846 -> 675.  It was not behind at any of 24 shapes from heads of 16 to 256.
#include "attention_args.cuh"
#include "common.cuh"

namespace lily {
namespace f32d {

constexpr int KB = 4;                      // keys a warp works on at a time
constexpr int MAX_G = 8;

// Query heads a block takes (G, at least the heads of a kv head) x pieces of 128 columns (C): as many warps as the registers allow.
__host__ __device__ constexpr int warps_of(int g, int c) { return c == 1 && g <= 4 ? 16 : 8; }

template <int G, int C>
__global__ void __launch_bounds__(warps_of(G, C) * 32)
attention_decode_f32_kernel(const AttnArgs a) {
    constexpr int WARPS = warps_of(G, C), N = KB * G, STEP = WARPS * KB;
    constexpr bool AHEAD = WARPS == 16;                          // registers for the next keys
    extern __shared__ __align__(16) float merge[];             // [WARPS][G][dv] outputs, then [WARPS][G][2] (max, sum)
    __shared__ __align__(16) float p_s[WARPS][G][KB];
    __shared__ float alpha_s[WARPS][G];
    pdl_enter_small();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int d = a.d, dv = a.dv, group = a.nq / a.nkv;
    const int req = blockIdx.x, kvh = blockIdx.y;
    const int seq = a.seq_lens[req];
    const int klo = (a.window > 0 && seq > a.window) ? seq - a.window : 0;
    const int nkeep = min(a.keep_first, klo);
    const int total = nkeep + seq - klo;
    int per = (total + a.splits - 1) / a.splits;
    per = (per + 31) / 32 * 32;
    const int ubeg = blockIdx.z * per, uend = min(total, ubeg + per);
    const float* kv = (const float*)a.kv;
    const int* table = a.block_table + (size_t)req * a.bt_stride;
    const size_t khead = (size_t)a.page_size * d, vhead = (size_t)a.page_size * dv, page_stride = (size_t)a.nkv * (khead + vhead);
    const size_t kbase = (size_t)kvh * khead, vbase = (size_t)a.nkv * khead + (size_t)((kvh + a.v_shift) % a.nkv) * vhead;

    float4 k[KB][C], v[KB][C], kn[AHEAD ? KB : 1][C], vn[AHEAD ? KB : 1][C];
    auto fetch = [&](int u0, float4 (*kd)[C], float4 (*vd)[C]) {
#pragma unroll
        for (int j = 0; j < KB; ++j) {
            const int u = u0 + j, kpos = u < nkeep ? u : klo + (u - nkeep);
            const bool in = u < uend;
            const float* page = kv + (in ? (size_t)table[kpos / a.page_size] * page_stride : 0);
            const size_t row = in ? kpos % a.page_size : 0;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int col = c * 128 + lane * 4;
                kd[j][c] = in && col < d ? *reinterpret_cast<const float4*>(page + kbase + row * d + col) : make_float4(0.f, 0.f, 0.f, 0.f);
                vd[j][c] = in && col < dv ? *reinterpret_cast<const float4*>(page + vbase + row * dv + col) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    };
    int u0 = ubeg + warp * KB;
    if (u0 < uend) fetch(u0, k, v);
    float4 q[G][C], o[G][C];
#pragma unroll
    for (int h = 0; h < G; ++h)
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int col = c * 128 + lane * 4;
            q[h][c] = h < group && col < d ? *reinterpret_cast<const float4*>((const float*)a.q + ((size_t)req * a.nq + kvh * group + h) * d + col)
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
            o[h][c] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    // after the exchanges lane l holds the sum of head l / (32 / G), key (l / (32 / N)) % KB
    constexpr int PER_HEAD = 32 / G;
    const int head = lane / PER_HEAD;
    const bool sunk = a.sink && blockIdx.z == 0 && warp == 0 && head < group;
    float m = sunk ? (a.sinks ? a.sinks[kvh * group + head] : 0.f) : -INFINITY, l = sunk ? 1.f : 0.f;
    const float cap = a.softcap, cap_in = cap > 0.f ? a.scale / cap : 0.f;
    for (; u0 < uend; u0 += STEP) {
        if (AHEAD && u0 + STEP < uend) fetch(u0 + STEP, kn, vn);
        float s[N];
#pragma unroll
        for (int h = 0; h < G; ++h)
#pragma unroll
            for (int j = 0; j < KB; ++j) {
                float t = 0.f;
#pragma unroll
                for (int c = 0; c < C; ++c)
                    t = fmaf(q[h][c].w, k[j][c].w, fmaf(q[h][c].z, k[j][c].z, fmaf(q[h][c].y, k[j][c].y, fmaf(q[h][c].x, k[j][c].x, t))));
                s[h * KB + j] = t;
            }
#pragma unroll
        for (int off = 16, n = N; off > 0; off >>= 1) {
            if (n > 1) {
                n >>= 1;
                const bool upper = lane & off;
#pragma unroll
                for (int i = 0; i < N / 2; ++i)
                    if (i < n) {
                        const float give = upper ? s[i] : s[i + n], keep = upper ? s[i + n] : s[i];
                        s[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
                    }
            } else s[0] += __shfl_xor_sync(0xffffffffu, s[0], off);
        }
        constexpr int REST = 32 / N;                          // lanes that hold the same sum
        const int key = lane / REST % KB;
        const float sv = u0 + key < uend ? (cap > 0.f ? cap * tanhf(s[0] * cap_in) : s[0] * a.scale) : -INFINITY;
        float mx = sv;
#pragma unroll
        for (int off = REST; off < PER_HEAD; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const float m_new = fmaxf(m, mx);
        float p = sv == sv ? 0.f : sv, alpha = 1.f;              // a NaN is no maximum: as a weight it reaches the row
        if (m_new > -INFINITY) {
            alpha = expf(m - m_new);
            p = expf(sv - m_new);
        }
        m = m_new;
        float sum = p;
#pragma unroll
        for (int off = REST; off < PER_HEAD; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        l = l * alpha + sum;
        __syncwarp();                                          // the weights before these have been read
        if (lane % REST == 0) p_s[warp][head][key] = p;
        if (lane % PER_HEAD == 0) alpha_s[warp][head] = alpha;
        __syncwarp();
#pragma unroll
        for (int h = 0; h < G; ++h) {
            const float4 w = *reinterpret_cast<const float4*>(p_s[warp][h]);
            const float f = alpha_s[warp][h], pw[KB] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int c = 0; c < C; ++c) {
                o[h][c].x *= f, o[h][c].y *= f, o[h][c].z *= f, o[h][c].w *= f;
#pragma unroll
                for (int j = 0; j < KB; ++j) {
                    o[h][c].x = fmaf(pw[j], v[j][c].x, o[h][c].x);
                    o[h][c].y = fmaf(pw[j], v[j][c].y, o[h][c].y);
                    o[h][c].z = fmaf(pw[j], v[j][c].z, o[h][c].z);
                    o[h][c].w = fmaf(pw[j], v[j][c].w, o[h][c].w);
                }
            }
        }
        if constexpr (AHEAD) {
#pragma unroll
            for (int j = 0; j < KB; ++j)
#pragma unroll
                for (int c = 0; c < C; ++c) k[j][c] = kn[j][c], v[j][c] = vn[j][c];
        } else if (u0 + STEP < uend) fetch(u0 + STEP, k, v);
    }

    float* ml = merge + WARPS * G * dv;
#pragma unroll
    for (int h = 0; h < G; ++h)
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int col = c * 128 + lane * 4;
            if (col < dv) *reinterpret_cast<float4*>(merge + (warp * G + h) * dv + col) = o[h][c];
        }
    if (lane % PER_HEAD == 0) {
        ml[(warp * G + head) * 2] = m;
        ml[(warp * G + head) * 2 + 1] = l;
    }
    __syncthreads();
    for (int i = threadIdx.x * 4; i < group * dv; i += WARPS * 32 * 4) {
        const int h = i / dv, col = i % dv;
        float mx = -INFINITY;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) mx = fmaxf(mx, ml[(w * G + h) * 2]);
        float den = 0.f;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float mw = ml[(w * G + h) * 2], lw = ml[(w * G + h) * 2 + 1];
            if (mw == -INFINITY && lw == 0.f) continue;          // no keys
            const float f = expf(mw - mx);
            const float4 t = *reinterpret_cast<const float4*>(merge + (w * G + h) * dv + col);
            sum.x = fmaf(t.x, f, sum.x), sum.y = fmaf(t.y, f, sum.y), sum.z = fmaf(t.z, f, sum.z), sum.w = fmaf(t.w, f, sum.w);
            den = fmaf(lw, f, den);
        }
        const size_t row = (size_t)req * a.nq + kvh * group + h;
        if (a.splits > 1) {
            const size_t at = row * a.splits + blockIdx.z;
            *reinterpret_cast<float4*>(a.part_o + at * dv + col) = sum;
            if (col == 0) {
                a.part_ml[at * 2] = mx;
                a.part_ml[at * 2 + 1] = den;
            }
        } else {
            const float inv = den == 0.f ? 0.f : 1.f / den;
            *reinterpret_cast<float4*>((float*)a.out + row * dv + col) = make_float4(sum.x * inv, sum.y * inv, sum.z * inv, sum.w * inv);
        }
    }
}

template <int G, int C>
static int launch(const AttnArgs& a, int requests, cudaStream_t stream) {
    constexpr int WARPS = warps_of(G, C);
    const size_t smem = sizeof(float) * WARPS * G * ((size_t)a.dv + 2);
    auto kern = attention_decode_f32_kernel<G, C>;
    static bool configured = false;                            // set once for the widest head, never while a graph is captured
    if (!configured) {
        const size_t most = sizeof(float) * WARPS * G * (128 * C + 2);
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        LILY_REQUIRE(e == cudaSuccess, "attention_decode: cannot get %zu bytes of shared memory: %s", most, cudaGetErrorString(e));
        configured = true;
    }
    launch_pdl(kern, dim3(requests, a.nkv, a.splits), dim3(WARPS * 32), smem, stream, a);
    return 0;
}

}  // namespace f32d

bool attention_decode_f32_takes(const AttnArgs& a) {
    return ((a.d | a.dv) & 3) == 0 && a.d <= 256 && a.dv <= 256 && a.nq / a.nkv <= f32d::MAX_G && !a.v_all && !a.v_in_k &&
           (((uintptr_t)a.q | (uintptr_t)a.kv | (uintptr_t)a.out | (uintptr_t)a.part_o) & 15) == 0;
}

int attention_decode_f32(const AttnArgs& a, int requests, cudaStream_t stream) {
    const int g = a.nq / a.nkv;
    const bool wide = a.d > 128 || a.dv > 128;
#define GO(G) return wide ? f32d::launch<G, 2>(a, requests, stream) : f32d::launch<G, 1>(a, requests, stream)
    if (g == 1) GO(1);
    if (g == 2) GO(2);
    if (g <= 4) GO(4);
    GO(8);
#undef GO
}

}  // namespace lily
