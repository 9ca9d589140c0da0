// The chosen experts' feed-forwards for a few tokens (a decode step), bfloat16: two kernels from the routing to the layer's sum.
//
// With a few tokens the layer is bound by reading the weights of the experts that were chosen once, so both kernels are
// that stream (tiles of [rows][64 k] in flight by cp.async in a ring of each warp's own, read by ldmatrix for mma.sync
// m16n8k16: weight rows on the 16-row side, tokens on the 8-column side), and the grouping of pairs by expert that a
// grouped product needs is left out: every block reads the few choices itself, and all tokens are the columns of every expert's
// product, of which only those that chose it are kept.
//
//   up     grid (ceil(rows of an expert / 32), experts that can have been chosen): a block takes 32 weight rows of one
//          chosen expert (16 gate rows and the 16 up rows that meet them, or 32 up rows of an ungated expert), its four warps a
//          quarter of k each, and writes the activation in bfloat16, a row per (token, choice) pair.
//   down   grid (width / 16): a block takes 16 rows of W_down of every chosen expert in turn, its eight warps an eighth of
//          k each, as one pipeline over all of them; the pairs' weights multiply the sums in registers, so the pairs'
//          outputs are never written and nothing is left to combine.  The ring starts on the first experts while the up
//          kernel still runs (the choices are older than that kernel).
//
// The kernels take up to 16 tokens and 128 pairs, as far as the columns' fragments go (lily_moe_few_pays says where they are the faster
// way); against the grouping, the library's two grouped products and the sum, us with router and choice (weights read at the copy rate):
// 16 experts of 2,048 x 2,048, gated, top 4: 62 -> 31 (16) with 1 token, 84 -> 42 (25) with 2, 120 -> 76 (57) with 8, 125 -> 96
// (62) with 16; 64 of 4,096 x 1,536, top 8: 116 -> 70 (47), 172 -> 115 (89), 364 -> 276 (237), 498 -> 459 (328).  The columns
// ride in the ring beside the weights: read by the lanes in pieces of 4 bytes, 8 tokens took 113 us and 16 took 162.
//
// Everything between the bfloat16 inputs, the activation and the result is float32.  A pair's sums run in an order of their own
// whatever else is in the step, and a token's experts are added in the order of their numbers.
#include "common.cuh"
#include "expert_act.cuh"
#include "mma.cuh"
#include "operand.cuh"

namespace lily {
namespace few {

using mma16::cp_async_commit;
using mma16::cp_async_wait;
using mma16::ldmatrix_x4;
using mma16::mma_bf16;
using mma16::smem_u32;

constexpr int MAX_EXPERTS = 256, MAX_PAIRS = 128;
constexpr int KT = 64, PITCH = KT * 2, PIECES = KT / 8;

__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}

// The experts that were chosen, in order: their number is returned, list[i] the i-th, rank[e] its place (valid where chosen).
// All threads of the block call it.
__device__ __forceinline__ int used_experts(const int* __restrict__ chosen, int pairs, int experts, short* list, short* rank, int* count) {
    for (int e = threadIdx.x; e < experts; e += blockDim.x) rank[e] = -1;
    __syncthreads();
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        const int e = chosen[p];
        if (e >= 0 && e < experts) rank[e] = 0;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        int n = 0;
        for (int e0 = 0; e0 < experts; e0 += 32) {
            const int e = e0 + (int)threadIdx.x;
            const bool used = e < experts && rank[e] == 0;
            const unsigned all = __ballot_sync(0xffffffffu, used);
            if (used) {
                const int at = n + __popc(all & ((1u << threadIdx.x) - 1));
                list[at] = (short)e;
                rank[e] = (short)at;
            }
            n += __popc(all);
        }
        if (threadIdx.x == 0) *count = n;
    }
    __syncthreads();
    return *count;
}

// A stage of a warp's ring: MT tiles of 16 weight rows x 64 k, then the NT * 8 columns' rows x 64 k; 16-byte pieces swizzled.
__host__ __device__ constexpr int stage_bytes(int rows, int nt) { return (rows + nt * 8) * PITCH; }

// One stage's product: MT tiles of 16 weight rows, NT tiles of 8 columns.
template <int MT, int NT>
__device__ __forceinline__ void multiply(uint32_t stage, float (&acc)[MT][NT][4]) {
    const int lane = threadIdx.x & 31;
    uint32_t x[NT][8];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int q = 0; q < 2; ++q) {                    // a read brings the columns' numbers of two steps of 16 k
            const int r = (lane & 7), ch = q * 4 + (lane >> 3);
            ldmatrix_x4(stage + (MT * 16 + nt * 8 + r) * PITCH + (((ch ^ r) & 7) << 4), x[nt][4 * q], x[nt][4 * q + 1], x[nt][4 * q + 2],
                        x[nt][4 * q + 3]);
        }
#pragma unroll
    for (int kk = 0; kk < KT / 16; ++kk)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            uint32_t a[4];
            const int r = mt * 16 + (lane & 15), ch = kk * 2 + (lane >> 4);
            ldmatrix_x4(stage + r * PITCH + (((ch ^ r) & 7) << 4), a[0], a[1], a[2], a[3]);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_bf16(acc[mt][nt], a, x[nt][2 * kk], x[nt][2 * kk + 1]);
        }
}

// The columns' part of a stage: row(column) is where a column's 64 numbers lie (null: zeros).
template <int NT, typename Row>
__device__ __forceinline__ void copy_columns(uint32_t at, Row row) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < NT * 2; ++i) {
        const int r = i * 4 + lane / PIECES, piece = lane % PIECES;
        const __nv_bfloat16* src = row(r);
        mma16::cp_async16(at + r * PITCH + (((piece ^ r) & 7) << 4), src ? src + piece * 8 : nullptr, src != nullptr);
    }
}

constexpr int UP_WARPS = 4, UP_ROWS = 32;
__host__ __device__ constexpr int up_stages(int nt) { return nt == 1 ? 5 : 4; }        // two blocks a SM
__host__ __device__ constexpr int up_smem(int nt) { return UP_WARPS * up_stages(nt) * stage_bytes(UP_ROWS, nt); }

template <int NT, bool GATED>
__global__ void __launch_bounds__(UP_WARPS * 32)
moe_up_few_kernel(const __nv_bfloat16* __restrict__ h, int ldh, int tokens, int K, const __nv_bfloat16* __restrict__ W, int ff,
                  const int* __restrict__ chosen, int top, int experts, const float* __restrict__ in_weight, int act, float limit,
                  float alpha, __nv_bfloat16* __restrict__ out) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ short list[MAX_PAIRS], rank[MAX_EXPERTS];
    __shared__ int count, pair_of[NT * 8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
    pdl_wait();
    pdl_launch_dependents();
    const int pairs = tokens * top;
    if (tid < NT * 8) pair_of[tid] = -1;
    const int used = used_experts(chosen, pairs, experts, list, rank, &count);
    if ((int)blockIdx.y >= used) return;
    const int e = list[blockIdx.y];
    for (int p = tid; p < pairs; p += UP_WARPS * 32)
        if (chosen[p] == e) pair_of[p / top] = p;

    constexpr int PER = GATED ? 16 : 32;               // activations a block gives
    const int n0 = blockIdx.x * PER;
    const __nv_bfloat16* We = W + (size_t)e * (GATED ? 2 : 1) * ff * K;
    const int kblocks = K / KT, per = (kblocks + UP_WARPS - 1) / UP_WARPS, kb0 = warp * per, nkb = max(0, min(per, kblocks - kb0));
    constexpr int STAGES = up_stages(NT), STAGE = stage_bytes(UP_ROWS, NT);
    const uint32_t ring = smem_u32(smem + warp * STAGES * STAGE);
    constexpr int COPIES = UP_ROWS * PIECES / 32;
    const __nv_bfloat16* src[COPIES];
    uint32_t dst[COPIES];
#pragma unroll
    for (int i = 0; i < COPIES; ++i) {
        const int r = (32 * i + lane) / PIECES, piece = (32 * i + lane) % PIECES;
        const int row = GATED ? (r < 16 ? min(n0 + r, ff - 1) : ff + min(n0 + r - 16, ff - 1)) : min(n0 + r, ff - 1);
        src[i] = We + (size_t)row * K + (size_t)kb0 * KT + piece * 8;
        dst[i] = (uint32_t)(r * PITCH + (((piece ^ r) & 7) << 4));
    }
    auto issue = [&](int kb) {
        const uint32_t base = ring + (kb % STAGES) * STAGE;
#pragma unroll
        for (int i = 0; i < COPIES; ++i) copy16(base + dst[i], src[i] + (size_t)kb * KT);
        copy_columns<NT>(base + UP_ROWS * PITCH, [&](int t) { return t < tokens ? h + (size_t)t * ldh + (size_t)(kb0 + kb) * KT : nullptr; });
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < nkb) issue(s);
        cp_async_commit();
    }
    float acc[2][NT][4] = {};
    for (int kb = 0; kb < nkb; ++kb) {
        cp_async_wait<STAGES - 2>();
        __syncwarp();
        if (kb + STAGES - 1 < nkb) issue(kb + STAGES - 1);
        cp_async_commit();
        multiply<2, NT>(ring + (kb % STAGES) * STAGE, acc);
    }
    // the quarters of k meet in shared memory: [warp][32 rows][NT * 8]
    __syncthreads();
    float* part = reinterpret_cast<float*>(smem);
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                part[(warp * UP_ROWS + mt * 16 + g + (j >> 1) * 8) * (NT * 8) + nt * 8 + 2 * c + (j & 1)] = acc[mt][nt][j];
    __syncthreads();
    for (int i = tid; i < PER * tokens; i += UP_WARPS * 32) {
        const int r = i % PER, t = i / PER, p = pair_of[t];
        if (p < 0 || n0 + r >= ff) continue;
        auto sum = [&](int row) {
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < UP_WARPS; ++w) v += part[(w * UP_ROWS + row) * (NT * 8) + t];
            return v;
        };
        const float w = in_weight ? in_weight[p] : 1.f;
        const float v = GATED ? expert_gate(act, w * sum(r), w * sum(r + 16), limit, alpha) : squared_relu(w * sum(r));
        out[(size_t)p * ff + n0 + r] = __float2bfloat16_rn(v);
    }
}

constexpr int DN_WARPS = 8, DN_STAGES = 6, DN_ROWS = 16;
__host__ __device__ constexpr int dn_smem(int nt) { return DN_WARPS * DN_STAGES * stage_bytes(DN_ROWS, nt); }

template <int NT>
__global__ void __launch_bounds__(DN_WARPS * 32)
moe_down_few_kernel(const __nv_bfloat16* __restrict__ a, int ff, const __nv_bfloat16* __restrict__ W, int width,
                    const int* __restrict__ chosen, const float* __restrict__ weights, int tokens, int top, int experts,
                    const __nv_bfloat16* __restrict__ h, int ldh, const Operand shared_out, const float* __restrict__ gate, float* __restrict__ out) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ short list[MAX_PAIRS], rank[MAX_EXPERTS], pair_of[MAX_PAIRS * NT * 8];       // [chosen experts][column]: the pair, or -1
    __shared__ int count;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
    const int pairs = tokens * top, n0 = blockIdx.x * DN_ROWS;
    // the choices were made ahead of the up kernel, which waited for them before it let this one start
    const int used = used_experts(chosen, pairs, experts, list, rank, &count);
    for (int i = tid; i < used * NT * 8; i += DN_WARPS * 32) pair_of[i] = -1;
    __syncthreads();
    for (int p = tid; p < pairs; p += DN_WARPS * 32) {
        const int e = chosen[p];
        if (e >= 0 && e < experts) pair_of[rank[e] * (NT * 8) + p / top] = (short)p;
    }
    __syncthreads();

    const int kblocks = ff / KT, per = (kblocks + DN_WARPS - 1) / DN_WARPS, kb0 = warp * per, nkb = max(0, min(per, kblocks - kb0));
    const int steps = used * nkb;
    constexpr int STAGE = stage_bytes(DN_ROWS, NT);
    const uint32_t ring = smem_u32(smem + warp * DN_STAGES * STAGE);
    constexpr int COPIES = DN_ROWS * PIECES / 32;
    size_t src[COPIES];
    uint32_t dst[COPIES];
#pragma unroll
    for (int i = 0; i < COPIES; ++i) {
        const int r = (32 * i + lane) / PIECES, piece = (32 * i + lane) % PIECES;
        src[i] = (size_t)(n0 + r) * ff + (size_t)kb0 * KT + piece * 8;
        dst[i] = (uint32_t)(r * PITCH + (((piece ^ r) & 7) << 4));
    }
    int w_x = 0, w_kb = 0, a_x = 0, a_kb = 0;          // the place in the list and the tile whose weights and columns are fetched next
    auto issue_w = [&](int step) {
        const uint32_t base = ring + (step % DN_STAGES) * STAGE;
        const __nv_bfloat16* We = W + (size_t)list[w_x] * width * ff + (size_t)w_kb * KT;
#pragma unroll
        for (int i = 0; i < COPIES; ++i) copy16(base + dst[i], We + src[i]);
        if (++w_kb == nkb) w_kb = 0, ++w_x;
    };
    auto issue_a = [&](int step) {
        copy_columns<NT>(ring + (step % DN_STAGES) * STAGE + DN_ROWS * PITCH, [&](int col) {
            const int p = pair_of[a_x * (NT * 8) + col];
            return p >= 0 ? a + (size_t)p * ff + (size_t)(kb0 + a_kb) * KT : nullptr;
        });
        if (++a_kb == nkb) a_kb = 0, ++a_x;
    };
#pragma unroll
    for (int s = 0; s < DN_STAGES - 1; ++s)
        if (s < steps) issue_w(s);
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int s = 0; s < DN_STAGES - 1; ++s) {
        if (s < steps) issue_a(s);
        cp_async_commit();
    }

    float total[1][NT][4] = {};
    int step = 0;
    for (int x = 0; x < used && nkb > 0; ++x) {
        float acc[1][NT][4] = {};
        for (int kb = 0; kb < nkb; ++kb, ++step) {
            cp_async_wait<DN_STAGES - 2>();
            __syncwarp();
            if (step + DN_STAGES - 1 < steps) {
                issue_w(step + DN_STAGES - 1);
                issue_a(step + DN_STAGES - 1);
            }
            cp_async_commit();
            multiply<1, NT>(ring + (step % DN_STAGES) * STAGE, acc);
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int p = pair_of[x * (NT * 8) + nt * 8 + 2 * c + q];
                if (p < 0) continue;
                const float w = weights ? weights[p] : 1.f;
                total[0][nt][q] = fmaf(w, acc[0][nt][q], total[0][nt][q]);
                total[0][nt][2 + q] = fmaf(w, acc[0][nt][2 + q], total[0][nt][2 + q]);
            }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    float* part = reinterpret_cast<float*>(smem);      // [warp][NT * 8][16 rows]
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int j = 0; j < 4; ++j) part[(warp * NT * 8 + nt * 8 + 2 * c + (j & 1)) * DN_ROWS + g + (j >> 1) * 8] = total[0][nt][j];
    __syncthreads();
    for (int i = tid; i < tokens * DN_ROWS; i += DN_WARPS * 32) {
        const int t = i / DN_ROWS, n = n0 + i % DN_ROWS;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < DN_WARPS; ++w) v += part[w * NT * 8 * DN_ROWS + i];
        for (int k = 0; k < top; ++k)                  // choices that have no weights of their own stand for the input
            if (chosen[t * top + k] >= experts) v = fmaf(weights ? weights[t * top + k] : 1.f, __bfloat162float(h[(size_t)t * ldh + n]), v);
        const size_t at = (size_t)t * width + n;
        if (gate) v = fmaf(gate[t], shared_out(at), v);
        out[at] = v;
    }
}

}  // namespace few
}  // namespace lily

using namespace lily;

// Whether the two kernels take the step: whole tiles of 64 numbers along both sums, up to 16 tokens.
LILY_API int lily_moe_few_takes(int tokens, int top, int experts, int width, int ff) {
    return tokens >= 1 && tokens <= 16 && tokens * top <= few::MAX_PAIRS && experts >= 1 && experts <= few::MAX_EXPERTS &&
           width > 0 && ff > 0 && width % few::KT == 0 && ff % few::KT == 0;
}

// Whether they are the faster way.  A block of the down kernel takes every chosen expert's 16 rows, 1.25 us for 1,000 numbers of them up to 8
// tokens and 1.85 beyond (an expert counts 512 at least, a tile of k a warp), where the grouped products take 1 us a 1,000 for a width of
// 1,000 and 33 us of launches and grouping: a wide layer is always ahead, a narrow one while it meets few experts or short ones.
// Grouped / here, 64 experts, top 8: width 512, ff 2,048: 1.60 with 1 token, 1.13 with 2, 0.89 with 4, 0.60 with 16; width 1,024: 1.45,
// 1.28, 1.15, 0.86; width 1,024, ff 512: 2.00, 1.68, 1.37, 1.02; from width 2,048 on 1.05 to 3.
LILY_API int lily_moe_few_pays(int tokens, int top, int experts, int width, int ff) {
    const long long chosen = min(experts, tokens * top), a_number = tokens <= 8 ? 1250 : 1850;
    return width >= a_number || chosen * max(ff, 512) * (a_number - width) <= 33000000;
}

// act [tokens * top, ff] from h [tokens, ldh]: W [experts, 2 ff, width] (an expert's gate rows, then its up rows) with
// activation 0 or 1, [experts, ff, width] with activation 2 (ungated, the squared relu); in_weight as in lily_moe_gemm.
LILY_API int lily_moe_up_few(const void* h, int ldh, int tokens, int width, const void* W, int ff, const int* chosen, int top, int experts,
                             const float* in_weight, int act, float limit, float alpha, void* out, cudaStream_t stream) {
    LILY_REQUIRE(lily_moe_few_takes(tokens, top, experts, width, ff), "moe_up_few: %d tokens x %d of %d experts, width %d, ff %d", tokens, top, experts, width, ff);
    LILY_REQUIRE(ldh >= width && ldh % 8 == 0 && (((uintptr_t)h | (uintptr_t)W) & 15) == 0, "moe_up_few: operands are not aligned");
    const bool gated = act != 2;
    dim3 grid((ff + (gated ? 16 : 32) - 1) / (gated ? 16 : 32), min(experts, tokens * top));
#define GO(NT, G)                                                                                                                \
    do {                                                                                                                         \
        auto kern = few::moe_up_few_kernel<NT, G>;                                                                               \
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, few::up_smem(NT));                   \
        LILY_REQUIRE(e == cudaSuccess, "moe_up_few: %s", cudaGetErrorString(e));                                                 \
        launch_pdl(kern, grid, dim3(few::UP_WARPS * 32), few::up_smem(NT), stream, (const __nv_bfloat16*)h, ldh, tokens, width,      \
                   (const __nv_bfloat16*)W, ff, chosen, top, experts, in_weight, act, limit, alpha, (__nv_bfloat16*)out);        \
    } while (0)
    if (tokens <= 8) { if (gated) GO(1, true); else GO(1, false); }
    else { if (gated) GO(2, true); else GO(2, false); }
#undef GO
    LILY_CHECK_LAUNCH("moe_up_few");
    return 0;
}

// out [tokens, width] float32 = the pairs' sums times their weights (null: 1) + the identity choices' inputs + gate * shared.
LILY_API int lily_moe_down_few(const void* a, int ff, const void* W, int width, const int* chosen, const float* weights, int tokens, int top,
                               int experts, const void* h, int ldh, const void* shared, int shared_dtype, int shared_splits, size_t shared_stride,
                               const float* gate, float* out, cudaStream_t stream) {
    LILY_REQUIRE(lily_moe_few_takes(tokens, top, experts, width, ff), "moe_down_few: %d tokens x %d of %d experts, width %d, ff %d", tokens, top, experts, width, ff);
    LILY_REQUIRE((((uintptr_t)a | (uintptr_t)W) & 15) == 0 && ldh >= width, "moe_down_few: operands are not aligned");
    LILY_REQUIRE(!gate || (shared && shared_splits >= 1 && (shared_splits == 1 || shared_dtype == kF32)), "moe_down_few: the shared expert's output");
    const Operand sh{shared, shared_dtype == kBF16, shared_splits, shared_stride};
#define GO(NT)                                                                                                                   \
    do {                                                                                                                         \
        auto kern = few::moe_down_few_kernel<NT>;                                                                                \
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, few::dn_smem(NT));                   \
        LILY_REQUIRE(e == cudaSuccess, "moe_down_few: %s", cudaGetErrorString(e));                                               \
        launch_pdl(kern, dim3(width / few::DN_ROWS), dim3(few::DN_WARPS * 32), few::dn_smem(NT), stream, (const __nv_bfloat16*)a, ff, \
                   (const __nv_bfloat16*)W, width, chosen, weights, tokens, top, experts, (const __nv_bfloat16*)h, ldh, sh, gate, out); \
    } while (0)
    if (tokens <= 8) GO(1); else GO(2);
#undef GO
    LILY_CHECK_LAUNCH("moe_down_few");
    return 0;
}
