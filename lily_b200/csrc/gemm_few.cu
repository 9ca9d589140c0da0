// Matrix product for up to 16 tokens whose result is wanted whole: out[m][n] = sum_k x[m][k] w[n][k] (+ bias[n]), bfloat16 in,
// float32 sums, bfloat16 or float32 out.  (gemm_skinny.cu leaves float32 partial sums to a consumer that adds them up; this
// kernel serves the ones that want finished rows: projections with a convolution, a recurrence or a table behind them.)
//
// Bound by reading w once.  A block of eight warps takes tiles of 16 weight rows, each warp an eighth of k: tiles of [16 rows][64 k]
// by cp.async in a ring of the warp's own, the tokens' [8 or 16][64 k] beside them, ldmatrix and mma.sync m16n8k16 (weight rows on
// the 16-row side, tokens on the 8-column side); the eighths meet in shared memory.  Two blocks a SM walk the tiles as one pipeline
// each, up to 96 KB in flight a SM, and the first stages of w, which depends on no one, are asked for before the kernel ahead has
// finished (three of the four tiles of k that a warp has at K 2,048).
// A token's sums run in the same order whatever else is in the step.  With the gate/up product's activation (GATED) the tile's two
// halves are the gate and the up rows of 8 outputs.
//
// What the product adds to a chain of norms and products, the library's and this one, us (in brackets w over the copy's rate, which is no
// floor: w's first tiles come under the kernel ahead, and a copy writes as much as it reads; alone 24,576 x 4,096 takes 35): N x K 64 x 2,048
// 5.1 -> 2.0; 2,048 x
// 2,048 7.9 -> 3.2 (1.3) with 5 tokens, 6.4 -> 3.8 with 16; 2,048 x 4,096 12 -> 4.5 (2.6); 10,304 x 2,048 9.8 -> 7.9 (6.5) with 8, 11.3 ->
// 9.1 with 16; 24,576 x 4,096 35.3 -> 31.5 (31.2), 35.8 -> 34.2 with 16; 32,000 x 4,096 46 -> 39 (41), 47 -> 41.  Gate/up with SiLU, against
// stretches of (128 outputs, 64 k) dealt out evenly and finished through scratch by the block that comes last: 8,192 x 2,048 14.6 ->
// 11.5 (10.4), 12,288 x 4,096 36.9 -> 30.7 (31.2), 25,600 x 5,120 85 -> 75 (81), 28,672 x 8,192 155 -> 139 (146).
#include "common.cuh"
#include "mma.cuh"

namespace lily {
namespace fewrows {

using mma16::cp_async_commit;
using mma16::cp_async_wait;
using mma16::ldmatrix_x4;
using mma16::mma_bf16;
using mma16::smem_u32;

constexpr int KT = 64, PITCH = KT * 2, WARPS = 8, ROWS = 16;
__host__ __device__ constexpr int stages(int nt) { return nt == 1 ? 4 : 3; }
__host__ __device__ constexpr int stage_bytes(int nt) { return (ROWS + nt * 8) * PITCH; }
__host__ __device__ constexpr int part_floats(int nt) { return WARPS * nt * 8 * ROWS; }
__host__ __device__ constexpr int smem_bytes(int nt) { return WARPS * stages(nt) * stage_bytes(nt) + part_floats(nt) * (int)sizeof(float); }
static_assert(smem_bytes(1) <= 113 * 1024 && smem_bytes(2) <= 113 * 1024, "two blocks a SM");

// The gate/up product with its activation (GATED): w holds runs of `run` gate rows and the `run` up rows of the same outputs, a tile is
// the 8 gate rows and the 8 up rows of 8 outputs, and the sums meet in the activation instead of in `out`'s row.
struct Gate {
    int run, act;                  // act 0: SiLU, 1: GELU in its tanh form, 2: clamped
    float limit, alpha;
};

template <int NT, bool GATED>
__global__ void __launch_bounds__(WARPS * 32)
gemm_few_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, const void* __restrict__ bias, int bias_f32,
                void* __restrict__ out, int out_f32, int M, int N, int K, const Gate gate) {
    constexpr int STAGES = stages(NT), STAGE = stage_bytes(NT);
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
    const uint32_t ring = smem_u32(smem + warp * STAGES * STAGE);
    float* part = reinterpret_cast<float*>(smem + WARPS * STAGES * STAGE);      // [warp][NT * 8][16 rows]
    const int kblocks = K / KT, per = (kblocks + WARPS - 1) / WARPS, kb0 = warp * per, nkb = max(0, min(per, kblocks - kb0));
    const int tiles = (N + ROWS - 1) / ROWS, mine = (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1, steps = mine * nkb;

    // a copy of the warp covers four rows of 128 bytes; rows beyond N repeat the last one
    const int r4 = lane >> 3, piece = lane & 7;
    auto row_of = [&](int tile, int r) {
        if (!GATED) return min(tile * ROWS + r, N - 1);
        const int o = tile * 8 + (r & 7);                    // N / 2 outputs, a multiple of 8, as a run is
        return o / gate.run * 2 * gate.run + o % gate.run + (r < 8 ? 0 : gate.run);
    };
    int w_tile = blockIdx.x, w_kb = 0, x_kb = 0;
    auto issue_w = [&](int step) {
        const uint32_t base = ring + (step % STAGES) * STAGE;
        const __nv_bfloat16* src = w + (size_t)(kb0 + w_kb) * KT + piece * 8;
#pragma unroll
        for (int i = 0; i < ROWS / 4; ++i) {
            const int r = i * 4 + r4;
            asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;\n" ::"r"(base + r * PITCH + (((piece ^ r) & 7) << 4)),
                         "l"(src + (size_t)row_of(w_tile, r) * K) : "memory");
        }
        if (++w_kb == nkb) w_kb = 0, w_tile += gridDim.x;
    };
    auto issue_x = [&](int step) {
        const uint32_t base = ring + (step % STAGES) * STAGE + ROWS * PITCH;
#pragma unroll
        for (int i = 0; i < NT * 2; ++i) {
            const int r = i * 4 + r4;
            mma16::cp_async16(base + r * PITCH + (((piece ^ r) & 7) << 4), x + (size_t)min(r, M - 1) * K + (size_t)(kb0 + x_kb) * KT + piece * 8, r < M);
        }
        if (++x_kb == nkb) x_kb = 0;
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s)
        if (s < steps) issue_w(s);
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) issue_x(s);
        cp_async_commit();
    }

    int step = 0;
    for (int it = 0; it < mine; ++it) {
        float acc[NT][4] = {};
        for (int kb = 0; kb < nkb; ++kb, ++step) {
            cp_async_wait<STAGES - 2>();
            __syncwarp();
            if (step + STAGES - 1 < steps) {
                issue_w(step + STAGES - 1);
                issue_x(step + STAGES - 1);
            }
            cp_async_commit();
            const uint32_t stage = ring + (step % STAGES) * STAGE;
            uint32_t xf[NT][8];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int q = 0; q < 2; ++q) {                // a read brings the tokens' numbers of two steps of 16 k
                    const int r = lane & 7, ch = q * 4 + (lane >> 3);
                    ldmatrix_x4(stage + (ROWS + nt * 8 + r) * PITCH + (((ch ^ r) & 7) << 4), xf[nt][4 * q], xf[nt][4 * q + 1], xf[nt][4 * q + 2],
                                xf[nt][4 * q + 3]);
                }
#pragma unroll
            for (int kk = 0; kk < KT / 16; ++kk) {
                uint32_t a[4];
                const int r = lane & 15, ch = kk * 2 + (lane >> 4);
                ldmatrix_x4(stage + r * PITCH + (((ch ^ r) & 7) << 4), a[0], a[1], a[2], a[3]);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) mma_bf16(acc[nt], a, xf[nt][2 * kk], xf[nt][2 * kk + 1]);
            }
        }
        if (it > 0) __syncthreads();                         // the tile before has been added up
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 4; ++j) part[(warp * NT * 8 + nt * 8 + 2 * c + (j & 1)) * ROWS + g + (j >> 1) * 8] = acc[nt][j];
        __syncthreads();
        const int tile = blockIdx.x + it * gridDim.x;
        auto sum = [&](int m, int r) {
            float v = 0.f;
#pragma unroll
            for (int q = 0; q < WARPS; ++q) v += part[q * NT * 8 * ROWS + m * ROWS + r];
            return v;
        };
        if (GATED) {
            for (int i = tid; i < M * 8; i += WARPS * 32) {
                const int m = i / 8, o = tile * 8 + i % 8;
                float g_ = sum(m, i % 8), u = sum(m, i % 8 + 8);
                if (gate.act == 2) {                         // the clamped form: g' sigmoid(alpha g') (u' + 1)
                    g_ = fminf(g_, gate.limit);
                    u = fminf(fmaxf(u, -gate.limit), gate.limit) + 1.f;
                }
                // act(g) = g * sigmoid(t): t = g for SiLU; t = 2 sqrt(2/pi) (g + 0.044715 g^3) for the tanh form of GELU; alpha g for the clamped form
                const float t = gate.act == 0 ? g_ : (gate.act == 2 ? gate.alpha * g_ : 1.5957691216057308f * (g_ + 0.044715f * g_ * g_ * g_));
                ((__nv_bfloat16*)out)[(size_t)m * (N / 2) + o] = __float2bfloat16_rn(g_ / (1.f + __expf(-t)) * u);
            }
            continue;
        }
        for (int i = tid; i < M * ROWS; i += WARPS * 32) {
            const int m = i / ROWS, n = tile * ROWS + i % ROWS;
            if (n >= N) continue;
            float v = sum(m, i % ROWS);
            if (bias) v += bias_f32 ? ((const float*)bias)[n] : __bfloat162float(((const __nv_bfloat16*)bias)[n]);
            if (out_f32) ((float*)out)[(size_t)m * N + n] = v;
            else ((__nv_bfloat16*)out)[(size_t)m * N + n] = __float2bfloat16_rn(v);
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

template <int NT, bool GATED>
static int launch(int grid, const void* x, const void* w, const void* bias, int bias_f32, void* out, int out_f32, int M, int N, int K,
                  const Gate& gate, cudaStream_t stream) {
    auto kern = gemm_few_kernel<NT, GATED>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(NT));
    LILY_REQUIRE(e == cudaSuccess, "gemm_few: %s", cudaGetErrorString(e));
    launch_pdl(kern, dim3(grid), dim3(WARPS * 32), smem_bytes(NT), stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, bias, bias_f32,
               out, out_f32, M, N, K, gate);
    LILY_CHECK_LAUNCH("gemm_few");
    return 0;
}

}  // namespace fewrows
}  // namespace lily

using namespace lily;

// Whether the kernel takes the product.
LILY_API int lily_gemm_few_takes(int M, int N, int K) {
    return M >= 1 && M <= 16 && N >= 1 && K >= fewrows::KT && K % fewrows::KT == 0;
}

// Whether it is the faster way to the product than the library's.  A block has a tile's whole k to itself, so it falls behind where a
// very long k meets too few tiles for the SMs, where a second turn of tiles leaves most blocks idle, and, beyond 8 tokens, whose
// stages are three, where it is not ahead of the memory any more.  Library / here, timed over N from 16 to 128,256 and K from 512 to
// 28,672:
//   up to 8 tokens   1.05 to 3.5 but for K 28,672 with N up to 256 (0.85 to 0.94) and N 5,120 (320 tiles for 296 blocks) from K
//                    9,728 on (0.89 to 0.97)
//   9 to 16, tiles for one turn   1.0 to 2.7 up to K 18,944; beyond that 0.56 to 0.99 up to N 2,560, 0.97 to 1.2 from 3,072 on
//   9 to 16, more tiles           0.99 to 1.7 up to K 4,096 (0.76 at K 512, 0.95 at 1,024 with N 128,256; 1.09 at 1,024 with 50,000);
//                                 beyond it 0.76 to 0.99 in up to four turns, but 1.02 to 1.06 up to K 12,288 where two or three turns
//                                 are full (N 8,192 and 12,288), and 0.97 to 1.15 in five turns and more
LILY_API int lily_gemm_few_pays(int M, int N, int K) {
    const int tiles = (N + fewrows::ROWS - 1) / fewrows::ROWS, slots = 2 * sm_count(), turns = (tiles + slots - 1) / slots;
    if (M <= 8) return turns == 1 ? K <= 25600 || tiles >= 32 : K <= 8192 || 10ll * tiles >= 6ll * turns * slots;
    if (turns == 1) return K <= 18944 || tiles >= 192;
    if (turns <= 4) return K <= 4096 || (turns <= 3 && K <= 12288 && 10ll * tiles >= 8ll * turns * slots);
    return K >= (turns <= 16 ? 1024 : 2048);
}

LILY_API int lily_gemm_few(const void* x, const void* w, const void* bias, int bias_f32, void* out, int out_f32, int M, int N, int K,
                           cudaStream_t stream) {
    LILY_REQUIRE(lily_gemm_few_takes(M, N, K), "gemm_few: M=%d N=%d K=%d", M, N, K);
    LILY_REQUIRE((((uintptr_t)x | (uintptr_t)w) & 15) == 0, "gemm_few: operands do not start on 16 bytes");
    const int tiles = (N + fewrows::ROWS - 1) / fewrows::ROWS, grid = min(tiles, 2 * sm_count());
    if (M <= 8) return fewrows::launch<1, false>(grid, x, w, bias, bias_f32, out, out_f32, M, N, K, fewrows::Gate{}, stream);
    return fewrows::launch<2, false>(grid, x, w, bias, bias_f32, out, out_f32, M, N, K, fewrows::Gate{}, stream);
}

// out [M, I] bfloat16 = act(x . gate^T) * (x . up^T), up to 8 tokens; w [2 I, K] holds runs of `run` gate rows and the `run` up
// rows of the same outputs (run == I: all gate rows, then all up rows).  Against the product followed by the activation, us: 12,288 x 4,096
// 32.1 -> 31.0 with 1 token, 32.2 -> 31.3 with 8; 25,600 x 5,120 75.1 -> 73.8, 76.7 -> 75.6; 28,672 x 8,192 135.7 -> 136.6, 141.5 -> 139.5.
LILY_API int lily_swiglu_few_takes(int M, int I, int K, int run) {
    return M <= 8 && lily_gemm_few_takes(M, I, K) && I >= 8 && run >= 8 && run % 8 == 0 && I % run == 0;
}

LILY_API int lily_swiglu_few(const void* x, const void* w, void* out, int M, int I, int K, int run, int act, float limit, float alpha,
                             cudaStream_t stream) {
    LILY_REQUIRE(lily_swiglu_few_takes(M, I, K, run), "swiglu_few: M=%d I=%d K=%d run=%d", M, I, K, run);
    LILY_REQUIRE(act >= 0 && act <= 2 && (act != 2 || limit > 0.f), "swiglu_few: activation %d (0: SiLU, 1: GELU, tanh form, 2: clamped with a positive limit)", act);
    LILY_REQUIRE((((uintptr_t)x | (uintptr_t)w) & 15) == 0, "swiglu_few: operands do not start on 16 bytes");
    const int grid = min(I / 8, 2 * sm_count());
    const fewrows::Gate gate{run, act, limit, alpha};
    return fewrows::launch<1, true>(grid, x, w, nullptr, 0, out, 0, M, 2 * I, K, gate, stream);
}
