// True float32 matrix product for the 32-bit path: C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]).
//
// FFMA only (no tensor cores, no TF32).  Each output element is summed over k in a fixed order
// whatever M and N are (runs of 256 products, each run summed left to right, the runs' sums added
// left to right), so a row's result does not depend on what else is in the batch; summing in runs
// keeps the rounding error of a sum over 12,288 products near that of one over a few hundred.
// Both kernels below keep that order and give the same bits.
// Takes the place of F.linear in float32 (lily/layers/quantization/base.py:69-72).
//
//  * few rows (a decode step): bound by reading W once.  The unit of work is one run of one row of W (1 KB): a thread sums
//    two of them, so no order is cut and a 2,048 x 2,048 product still has 8,192 threads.  A block walks tiles of 16 rows
//    of W as one pipeline of cp.async stages (two blocks a SM, up to 96 KB in flight on each), and starts it before the
//    kernel ahead has finished: W depends on no one.  3 rows, 16,384 x 2,048 (134 MB): 217 us as a padded tile, 46 here
//    (21 at the copy rate); 2,048 x 8,192: 615 -> 33 (10).
//  * many rows (a prompt): bound by FFMA and the shared-memory reads that feed it.  A block of 128 threads has a tile of
//    64 x 128, a thread 8 x 8 outputs as packed pairs (fma.rn.f32x2: two IEEE fmas an instruction, the same bits), a
//    warp 32 x 64 so that an operand's read is one row of banks, the next tile of A and W in registers while this one is
//    multiplied.  451 rows, 16,384 x 2,048: 1,450 -> 695 us (409 at the FFMA rate); plain fmaf 853, 32 rows a block 821,
//    128 rows 760.
#include "common.cuh"

namespace lily {

constexpr int RUN = 256;               // products per run

// ------------------------------------------------------------------------------ few rows

constexpr int RN = 16;                 // rows of W (output columns) of a tile; a thread has two of them
constexpr int RUNS = 8;                // runs a pass covers
constexpr int ROWS_THREADS = RN / 2 * RUNS;
constexpr int PIECE = 32;              // floats of a run a stage holds
constexpr int PIECES = RUN / PIECE;
constexpr int PLD = PIECE + 4;         // floats between units in shared memory: 16-byte reads of 8 units meet 32 banks

// Two blocks a SM whatever MB is: of W 2 x 3 (2 x 2 beyond four rows) stages of 16 KB are in flight on each.
__host__ __device__ constexpr int rows_stages(int mb) { return mb <= 4 ? 4 : 3; }
__host__ __device__ constexpr int rows_stage_floats(int mb) { return (RN + mb) * RUNS * PLD; }

__device__ __forceinline__ void cp_async16(float* dst, const float* src, int bytes) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <int MB>
__global__ void __launch_bounds__(ROWS_THREADS)
gemm_fp32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
                      int M, int N, int K, int lda, int ldc, size_t a_head, size_t w_head, size_t c_head) {
    constexpr int STAGES = rows_stages(MB), STAGE = rows_stage_floats(MB), OUTS = (MB * RN + ROWS_THREADS - 1) / ROWS_THREADS;
    extern __shared__ __align__(16) float rows_smem[];
    float* sums = rows_smem + STAGES * STAGE;                  // [RUNS][MB][RN]: the runs of the pass that ended last
    A += blockIdx.z * a_head;
    W += blockIdx.z * w_head;
    C += blockIdx.z * c_head;
    const int m0 = blockIdx.y * MB, rows = min(MB, M - m0), tid = threadIdx.x;
    const int passes = (K + RUN * RUNS - 1) / (RUN * RUNS), per_tile = passes * PIECES;
    const int tiles = (N + RN - 1) / RN;
    const int steps = ((tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * per_tile;    // the block's tiles, one behind the other

    // a stage of W is RN x RUNS units of PIECE floats: 8 neighbouring threads fetch one unit's 128 bytes
    auto fetch_w = [&](int step) {
        float* dst = rows_smem + (step % STAGES) * STAGE;
        const int n0 = (blockIdx.x + step / per_tile * gridDim.x) * RN, at_k = step % per_tile;
        const int k0 = at_k / PIECES * RUNS * RUN + at_k % PIECES * PIECE + tid % 8 * 4;
#pragma unroll
        for (int i = 0; i < RN * RUNS / 8; ++i) {
            const int unit = i * 8 + tid / 8;
            const int n = n0 + unit % RN, k = k0 + unit / RN * RUN;
            const bool in = n < N && k < K;
            cp_async16(dst + unit * PLD + tid % 8 * 4, in ? W + (size_t)n * K + k : W, in ? 16 : 0);
        }
    };
    auto fetch_x = [&](int step) {
        float* dst = rows_smem + (step % STAGES) * STAGE + RN * RUNS * PLD;
        const int at_k = step % per_tile, k0 = at_k / PIECES * RUNS * RUN + at_k % PIECES * PIECE + tid % 8 * 4;
#pragma unroll
        for (int i = 0; i < MB; ++i) {
            const int unit = i * 8 + tid / 8;                  // RUNS units a row: row i, run tid / 8
            const int k = k0 + tid / 8 * RUN;
            const bool in = i < rows && k < K;
            cp_async16(dst + unit * PLD + tid % 8 * 4, in ? A + (size_t)(m0 + i) * lda + k : A, in ? 16 : 0);
        }
    };

    // W first, then the wait for whoever writes A
    for (int s = 0; s < STAGES - 1 && s < steps; ++s) fetch_w(s);
    pdl_launch_dependents();
    pdl_wait();
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) fetch_x(s);
        cp_commit();
    }

    float acc[MB][2], total[OUTS];
#pragma unroll
    for (int m = 0; m < MB; ++m) acc[m][0] = acc[m][1] = 0.f;
#pragma unroll
    for (int o = 0; o < OUTS; ++o) total[o] = 0.f;
    // after the barrier behind a pass's last step: its runs onto the totals, in order, and the tile's results out
    auto add_pass = [&](int step) {
        const int n0 = (blockIdx.x + step / per_tile * gridDim.x) * RN;
        const bool last = step % per_tile == per_tile - 1;
#pragma unroll
        for (int o = 0; o < OUTS; ++o) {
            const int at = o * ROWS_THREADS + tid;
            if (at >= MB * RN) continue;
            for (int r = 0; r < RUNS; ++r) total[o] += sums[r * MB * RN + at];
            if (last) {
                const int m = at / RN, n = n0 + at % RN;
                if (m < rows && n < N) C[(size_t)(m0 + m) * ldc + n] = total[o] + (bias ? bias[n] : 0.f);
                total[o] = 0.f;
            }
        }
    };
    for (int step = 0; step < steps; ++step) {
        cp_wait<STAGES - 2>();
        __syncthreads();
        if (step + STAGES - 1 < steps) {
            fetch_w(step + STAGES - 1);
            fetch_x(step + STAGES - 1);
        }
        cp_commit();
        if (step != 0 && step % PIECES == 0) add_pass(step - 1);
        const float* stage = rows_smem + (step % STAGES) * STAGE;
        const float* w = stage + (tid / 8 * RN + tid % 8) * PLD;
        const float* x = stage + (RN * RUNS + tid / 8) * PLD;
#pragma unroll
        for (int k = 0; k < PIECE; k += 4) {
            const float4 b0 = *reinterpret_cast<const float4*>(w + k), b1 = *reinterpret_cast<const float4*>(w + 8 * PLD + k);
#pragma unroll
            for (int m = 0; m < MB; ++m) {
                const float4 a = *reinterpret_cast<const float4*>(x + m * RUNS * PLD + k);
                acc[m][0] = fmaf(a.w, b0.w, fmaf(a.z, b0.z, fmaf(a.y, b0.y, fmaf(a.x, b0.x, acc[m][0]))));
                acc[m][1] = fmaf(a.w, b1.w, fmaf(a.z, b1.z, fmaf(a.y, b1.y, fmaf(a.x, b1.x, acc[m][1]))));
            }
        }
        if (step % PIECES == PIECES - 1) {
#pragma unroll
            for (int m = 0; m < MB; ++m) {
                sums[(tid / 8 * MB + m) * RN + tid % 8] = acc[m][0];
                sums[(tid / 8 * MB + m) * RN + tid % 8 + 8] = acc[m][1];
                acc[m][0] = acc[m][1] = 0.f;
            }
        }
    }
    __syncthreads();
    add_pass(steps - 1);
}

template <int MB>
static int launch_rows(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldc, int heads,
                       size_t a_head, size_t w_head, size_t c_head, cudaStream_t stream) {
    constexpr int smem = (int)sizeof(float) * (rows_stages(MB) * rows_stage_floats(MB) + RUNS * MB * RN);
    static_assert(smem <= 113 * 1024, "two blocks a SM");
    auto kern = gemm_fp32_rows_kernel<MB>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    LILY_REQUIRE(e == cudaSuccess, "gemm_fp32: cannot get %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
    // as many blocks as are resident at once, each with the same number of tiles (give or take one)
    const int tiles = (N + RN - 1) / RN, chunks = (M + MB - 1) / MB;
    const int room = max(1, 2 * sm_count() / (chunks * heads)), turns = (tiles + room - 1) / room;
    launch_pdl(kern, dim3((tiles + turns - 1) / turns, chunks, heads), dim3(ROWS_THREADS), smem, stream, A, W, bias, C, M, N, K, lda, ldc,
               a_head, w_head, c_head);
    return 0;
}

// ------------------------------------------------------------------------------ many rows

constexpr int BM = 64, BN = 128, BK = 16, TILE_THREADS = 128;
constexpr int ALD = BM + 4, WLD = BN + 4;

__device__ __forceinline__ uint64_t pack2(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// four neighbours of a row, zeros beyond the matrix; VEC: the row starts on 16 bytes and K is a multiple of four
template <bool VEC>
__device__ __forceinline__ float4 row4(const float* __restrict__ src, bool in, int k, int K) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (VEC) {
        if (in && k < K) v = *reinterpret_cast<const float4*>(src + k);
    } else if (in) {
        if (k < K) v.x = src[k];
        if (k + 1 < K) v.y = src[k + 1];
        if (k + 2 < K) v.z = src[k + 2];
        if (k + 3 < K) v.w = src[k + 3];
    }
    return v;
}

template <bool VEC>
__global__ void __launch_bounds__(TILE_THREADS, 2)
gemm_fp32_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                 float* __restrict__ C, int M, int N, int K, int lda, int ldc, size_t a_head, size_t w_head, size_t c_head) {
    // blockIdx.z: one of several products of the same sizes (a product per head), their operands these strides apart
    A += blockIdx.z * a_head;
    W += blockIdx.z * w_head;
    C += blockIdx.z * c_head;
    __shared__ __align__(16) float As[2][BK][ALD];
    __shared__ __align__(16) float Ws[2][BK][WLD];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    constexpr int QUADS = BK / 4, STEP = TILE_THREADS / QUADS;
    const int lr = tid / QUADS, lc = tid % QUADS * 4;          // loader: rows lr, lr + STEP, ..., k offset lc
    constexpr int AL = BM / STEP, WL = BN / STEP;
    float4 an[AL], wn[WL];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < AL; ++i) {
            const int m = m0 + lr + STEP * i;
            an[i] = row4<VEC>(A + (size_t)m * lda, m < M, k0 + lc, K);
        }
#pragma unroll
        for (int i = 0; i < WL; ++i) {
            const int n = n0 + lr + STEP * i;
            wn[i] = row4<VEC>(W + (size_t)n * K, n < N, k0 + lc, K);
        }
    };
    auto store = [&](int b) {
#pragma unroll
        for (int i = 0; i < AL; ++i) {
            As[b][lc][lr + STEP * i] = an[i].x;
            As[b][lc + 1][lr + STEP * i] = an[i].y;
            As[b][lc + 2][lr + STEP * i] = an[i].z;
            As[b][lc + 3][lr + STEP * i] = an[i].w;
        }
#pragma unroll
        for (int i = 0; i < WL; ++i) {
            Ws[b][lc][lr + STEP * i] = wn[i].x;
            Ws[b][lc + 1][lr + STEP * i] = wn[i].y;
            Ws[b][lc + 2][lr + STEP * i] = wn[i].z;
            Ws[b][lc + 3][lr + STEP * i] = wn[i].w;
        }
    };
    // a warp has 32 x 64 outputs: a thread the rows ar .. + 3 and ar + 16 .. + 3, the columns wc .. + 3 and wc + 32 .. + 3
    const int ar = warp / 2 * 32 + lane / 8 * 4, wc = warp % 2 * 64 + lane % 8 * 4;
    uint64_t acc[8][4];
    float total[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) total[i][j] = 0.f;
    }
    auto close_run = [&]() {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float x, y;
                unpack2(acc[i][j], x, y);
                total[i][2 * j] += x;
                total[i][2 * j + 1] += y;
                acc[i][j] = 0;
            }
    };
    const int tiles = (K + BK - 1) / BK;
    fetch(0);
    store(0);
    __syncthreads();
    for (int t = 0; t < tiles; ++t) {
        const int b = t & 1;
        if (t + 1 < tiles) fetch((t + 1) * BK);
        if (t != 0 && t % (RUN / BK) == 0) close_run();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            const float4 a0 = *reinterpret_cast<const float4*>(&As[b][k][ar]), a1 = *reinterpret_cast<const float4*>(&As[b][k][ar + 16]);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&Ws[b][k][wc]), b1 = *reinterpret_cast<const ulonglong2*>(&Ws[b][k][wc + 32]);
            const uint64_t bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint64_t aa = pack2(av[i], av[i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma2(aa, bv[j], acc[i][j]);
            }
        }
        if (t + 1 < tiles) store(b ^ 1);
        __syncthreads();
    }
    close_run();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ar + (i & 3) + (i >> 2) * 16;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int n = n0 + wc + (j & 3) + (j >> 2) * 32;
            if (n < N) C[(size_t)m * ldc + n] = total[i][j] + (bias ? bias[n] : 0.f);
        }
    }
}

// Whether a product goes to the kernel for few rows.  In units of 0.175 ns: that one takes, for every 2,048 numbers of k or part of them, 10
// for every output column of 8 rows (W comes from L2 again for each 8, and a product's row is read from shared memory; 5.5 for a single
// row), 25,000 for one row to 49,000 for 8 at least; the tile takes 13,000 and 290 for every k in one wave of blocks and 0.8 of that for each
// further one, however many of its 64 rows are there.  Tile / rows, us: N 2,048, K 2,048: 121 / 40 with 64 rows, 122 / 119 with 200, 122 /
// 187 with 300; N 8,192, K 2,048: 126 / 21 with 8, 127 / 139 with 64; N 512, K 512: 32 / 26 with 200, 32 / 42 with 300; 16 heads of N
// 512, K 128: 9.4 / 17 with 8; N 64, K 32: 3.2 / 4.5 with 1.
static bool few_rows(long long M, long long N, long long K, long long heads) {
    const long long chunks = (M + 7) / 8, blocks = (M + BM - 1) / BM * ((N + BN - 1) / BN) * heads, m = min(M, 8ll);
    const long long waves = (blocks + sm_count() - 1) / sm_count(), passes = (K + RUN * RUNS - 1) / (RUN * RUNS);
    const long long rows = passes * max(22000 + 3400 * m, (96 + 13 * m) * chunks * N * heads / 20);
    return chunks <= 65535 && rows < (13000 + 290 * K) * max(10ll, 8 * waves) / 10;
}

static int gemm_fp32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldc, int heads,
                     size_t a_head, size_t w_head, size_t c_head, cudaStream_t stream) {
    const bool vec = (((uintptr_t)A | (uintptr_t)W) & 15) == 0 && ((K | lda) & 3) == 0 && ((a_head | w_head) & 3) == 0;
    if (vec && few_rows(M, N, K, heads)) {
#define LILY_ROWS(MB) return launch_rows<MB>(A, W, bias, C, M, N, K, lda, ldc, heads, a_head, w_head, c_head, stream)
        if (M == 1) LILY_ROWS(1);
        if (M == 2) LILY_ROWS(2);
        if (M == 3) LILY_ROWS(3);
        if (M == 4) LILY_ROWS(4);
        if (M <= 6) LILY_ROWS(6);
        LILY_ROWS(8);
#undef LILY_ROWS
    }
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, heads);
    LILY_REQUIRE(grid.y <= 65535, "gemm_fp32: M=%d is too large for one launch", M);
    auto kern = vec ? gemm_fp32_kernel<true> : gemm_fp32_kernel<false>;
    kern<<<grid, TILE_THREADS, 0, stream>>>(A, W, bias, C, M, N, K, lda, ldc, a_head, w_head, c_head);
    return 0;
}

}  // namespace lily

using namespace lily;

LILY_API int lily_gemm_fp32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K,
                            int lda, int ldc, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    LILY_REQUIRE(K > 0 && lda >= K && ldc >= N, "gemm_fp32: bad sizes M=%d N=%d K=%d lda=%d ldc=%d", M, N, K, lda, ldc);
    if (int rc = gemm_fp32(A, W, bias, C, M, N, K, lda, ldc, 1, 0, 0, 0, stream)) return rc;
    LILY_CHECK_LAUNCH("gemm_fp32");
    return 0;
}

// `heads` products of the same sizes in one launch: head h reads A + h * a_head (rows lda apart) and W + h * w_head
// ([N, K]) and writes C + h * c_head (rows ldc apart).
LILY_API int lily_gemm_fp32_heads(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldc, int heads,
                                  size_t a_head, size_t w_head, size_t c_head, cudaStream_t stream) {
    if (M == 0 || N == 0 || heads == 0) return 0;
    LILY_REQUIRE(K > 0 && lda >= K && ldc >= N && heads <= 65535, "gemm_fp32_heads: bad sizes M=%d N=%d K=%d lda=%d ldc=%d heads=%d", M, N, K, lda, ldc, heads);
    if (int rc = gemm_fp32(A, W, nullptr, C, M, N, K, lda, ldc, heads, a_head, w_head, c_head, stream)) return rc;
    LILY_CHECK_LAUNCH("gemm_fp32_heads");
    return 0;
}
