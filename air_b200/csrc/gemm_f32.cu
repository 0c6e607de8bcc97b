// True 32-bit matrix product on the CUDA cores: C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]), for matrices W that gemm_f32_tc.cu does not
// take (short k, few columns, rows that are not whole aligned 16-byte pieces).  No reduced-precision mode.  The sum of an element of C is the same whatever kernel takes it: k is cut
// into PARTS ranges of equal length (a multiple of 16), each accumulated in ascending order by one thread with fused
// multiply-adds, and the ranges' sums are added in ascending order.  So a row of C does not depend on which other rows are
// in the batch: the 32-bit path gives the same bits for a token whether it is computed alone, in a portion of a prompt or
// in a mixed batch.  (One chain over all of k left a product of few rows waiting for its own additions, and one of few
// tiles could not use more blocks.  Four shorter chains also err half as much.)
//
//   gemm_f32_few_kernel    up to FEW_ROWS rows: a stream of weights
//   gemm_f32_tile_kernel   more rows: tiles of C in registers, a block for all ranges or a cluster with a block for each
//   gemm_f32_kernel        rows that are not whole aligned 16-byte pieces, at any number of rows
//
// Measured, us, from memory, against tiles of 64 x 64 with scalar reads at every size (also at sizes that gemm_f32_tc.cu takes now): 4 rows by 4,608 x 3,584 281 -> 23, by
// 37,888 x 3,584 631 -> 135 (4.0 TB/s), by 3,584 x 18,944 1,485 -> 74; 300 rows by 2,048 x 2,048 223 -> 83, by 16,384 x 2,048 886
// -> 533 (38 TFLOP/s), by 2,048 x 8,192 870 -> 295; 2,048 rows by 16,384 x 2,048 5,368 -> 3,297 (42 TFLOP/s; the multiply-add
// pipe alone gives 72).
#include "common.cuh"

#include <cooperative_groups.h>

namespace air {

constexpr int PARTS = 4;
__host__ __device__ __forceinline__ int part_of(int K) { return ((K + PARTS - 1) / PARTS + 15) / 16 * 16; }

__device__ __forceinline__ void gf_copy16(float* smem_dst, const float* src, bool valid) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem_dst);
    const int bytes = valid ? 16 : 0;             // 0: the 16 bytes are zero-filled, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gf_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void gf_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ---------------------------------------------------------------------------------------------- many rows
// Tiles are staged as they lie in memory, [row][k]: a thread reads four k of a row at once and multiplies them in turn, so
// nothing is transposed.  Rows of TILE_K + 4 floats put the eight rows that a quarter of a warp reads into different banks.
// A thread's rows and columns lie (BM / TM) and (BN / TN) apart.  (Staged transposed, and with 8 x 8 or 8 x 16 sums per
// thread, the same product stayed within 5 %.)
// CL 1: a block takes all of k in one go and keeps the sum of the ranges that are done in shared memory (a number of its own per
// thread).  CL PARTS: the blocks of a cluster take a range each and add the sums up through one another's shared memory, a
// quarter of the tile each.
constexpr int TILE_K = 16, TILE_LD = TILE_K + 4, TILE_STAGES = 4;

template <int BM, int BN, int TM, int TN, int CL>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), 4)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     float* __restrict__ C, int M, int N, int K) {
    constexpr int THREADS = (BM / TM) * (BN / TN), DY = BM / TM, DX = BN / TN, ROWS = BM + BN,
                  COPIES = ROWS * (TILE_K / 4) / THREADS;
    static_assert(ROWS * (TILE_K / 4) % THREADS == 0 && DX % 8 == 0 && DY % 4 == 0, "whole copies, whole warps");
    extern __shared__ __align__(16) float smem[];
    pdl_enter(TR_GEMM_F32);
    // (a warp is 8 columns by 4 rows of threads: what it reads at once is at most 8 pieces of 16 bytes, the least that a
    // read takes)
    const int tid = threadIdx.x, tx = tid / 32 % (DX / 8) * 8 + tid % 8, ty = tid / 32 / (DX / 8) * 4 + tid % 32 / 8;
    const int rank = CL > 1 ? blockIdx.x % CL : 0;
    const int m0 = (blockIdx.x / CL) * BM, n0 = blockIdx.y * BN;        // (blocks beside one another share their weights)
    const int Kp = part_of(K), k_lo = CL > 1 ? rank * Kp : 0, k_hi = CL > 1 ? min(K, k_lo + Kp) : K;
    float* const done = smem + TILE_STAGES * ROWS * TILE_LD + threadIdx.x;      // CL 1: [TM * TN][THREADS]
    // this thread's pieces of a stage: the same rows at every step, TILE_K further on
    const int k_mine = (tid % (TILE_K / 4)) * 4;
    const float* src[COPIES];
#pragma unroll
    for (int c = 0; c < COPIES; ++c) {
        const int row = tid / (TILE_K / 4) + c * (THREADS / (TILE_K / 4)), r = row < BM ? m0 + row : n0 + row - BM;
        src[c] = r < (row < BM ? M : N) ? (row < BM ? A : W) + (size_t)r * K + k_lo + k_mine : nullptr;
    }
    float* const dst = smem + (tid / (TILE_K / 4)) * TILE_LD + k_mine;
    auto bring = [&](int step) {
        float* to = dst + (step % TILE_STAGES) * ROWS * TILE_LD;
        const bool in_k = k_lo + step * TILE_K + k_mine < k_hi;
#pragma unroll
        for (int c = 0; c < COPIES; ++c) {
            const bool in = in_k && src[c];
            gf_copy16(to + c * (THREADS / (TILE_K / 4)) * TILE_LD, in ? src[c] + step * TILE_K : A, in);
        }
    };
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    const int steps = max(0, (k_hi - k_lo + TILE_K - 1) / TILE_K);
#pragma unroll
    for (int s = 0; s < TILE_STAGES - 1; ++s) {
        if (s < steps) bring(s);
        gf_commit();
    }
    for (int step = 0; step < steps; ++step) {
        gf_wait<TILE_STAGES - 2>();
        __syncthreads();
        if (step + TILE_STAGES - 1 < steps) bring(step + TILE_STAGES - 1);
        gf_commit();
        if (CL == 1 && step > 0 && step % (Kp / TILE_K) == 0) {       // a range is done
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    float* sum = done + (i * TN + j) * THREADS;
                    *sum = step > Kp / TILE_K ? *sum + acc[i][j] : acc[i][j];
                    acc[i][j] = 0.f;
                }
        }
        const float* as = smem + (step % TILE_STAGES) * ROWS * TILE_LD + ty * TILE_LD;
        const float* ws = smem + (step % TILE_STAGES) * ROWS * TILE_LD + (BM + tx) * TILE_LD;
#pragma unroll
        for (int k = 0; k < TILE_K; k += 4) {          // (beyond the range both operands hold zeros)
            float a[TM][4], w[2][4];
#pragma unroll
            for (int i = 0; i < TM; ++i) load4(as + i * DY * TILE_LD + k, a[i]);
            load4(ws + k, w[0]);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                if (j + 1 < TN) load4(ws + (j + 1) * DX * TILE_LD + k, w[(j + 1) & 1]);
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i][e], w[j & 1][e], acc[i][j]);
            }
        }
    }
    gf_wait<0>();
    if constexpr (CL == 1) {
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + j * DX;
            if (n >= N) continue;
            const float b = bias ? bias[n] : 0.f;
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const int m = m0 + ty + i * DY;
                if (m >= M) continue;
                const float sum = K > Kp ? done[(i * TN + j) * THREADS] + acc[i][j] : acc[i][j];
                C[(size_t)m * N + n] = bias ? sum + b : sum;
            }
        }
    } else {
        __syncthreads();                               // (the stages' memory takes the tile's sums)
#pragma unroll
        for (int j = 0; j < TN; ++j)
#pragma unroll
            for (int i = 0; i < TM; ++i) smem[(ty + i * DY) * BN + tx + j * DX] = acc[i][j];
        cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
        cluster.sync();
        const float* from[CL];
#pragma unroll
        for (int r = 0; r < CL; ++r) from[r] = cluster.map_shared_rank(smem, r);
        for (int i = tid * 4; i < BM / CL * BN; i += THREADS * 4) {
            const int at = rank * (BM / CL) * BN + i, m = m0 + at / BN, n = n0 + at % BN;
            float v[CL][4];
#pragma unroll
            for (int r = 0; r < CL; ++r) load4(from[r] + at, v[r]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (m >= M || n + e >= N) continue;
                float sum = v[0][e];
#pragma unroll
                for (int r = 1; r < CL; ++r) sum += v[r][e];
                C[(size_t)m * N + n + e] = bias ? sum + bias[n + e] : sum;
            }
        }
        cluster.sync();                                // (nobody leaves while its memory is read)
    }
}

// ---------------------------------------------------------------------------------------------- few rows
// A block takes `cols` rows of W and all rows of A, FEW_K numbers of every range of k at a time.  A warp's lanes are 8
// columns in each of the PARTS ranges; a lane has RN columns, 8 apart, and RM rows, so that RN + RM numbers are read from
// shared memory for RN * RM multiply-adds.  The last COPIERS threads only copy.  What is left is the stream of the weights.
constexpr int FEW_ROWS = 16, FEW_COLS = 32, FEW_K = 64, FEW_LD = PARTS * FEW_K + 4, COPIERS = 128, FEW_STAGES = 4;

template <int RM>
__global__ void __launch_bounds__(384)
gemm_f32_few_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                    float* __restrict__ C, int M, int N, int K, int cols, int w_ready) {
    constexpr int RN = 2;
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, workers = blockDim.x - COPIERS;
    const int n0 = blockIdx.x * cols, rows = cols + M;
    const int Kp = part_of(K), steps = (Kp + FEW_K - 1) / FEW_K;
    // this thread's pieces: one place of a row's k at a time, every other row
    constexpr int PIECES = PARTS * FEW_K / 4, ROW_STEP = COPIERS / PIECES;
    const bool copies = tid >= workers;
    const int place = copies ? tid - workers : 0, c = place % PIECES, row0 = place / PIECES;
    const int in_part = (c % (FEW_K / 4)) * 4, k_mine = (c / (FEW_K / 4)) * Kp + in_part;
    auto bring = [&](int step, bool of_w, bool of_a) {
        float* to = smem + ((step % FEW_STAGES) * rows + row0) * FEW_LD + 4 * c;
        const int at = step * FEW_K;
        const bool in_k = in_part + at < Kp && k_mine + at < K;
        if (of_w) {
            const float* src = W + (size_t)(n0 + row0) * K + k_mine + at;
#pragma unroll 4
            for (int row = row0; row < cols; row += ROW_STEP, src += (size_t)ROW_STEP * K) {
                const bool in = in_k && n0 + row < N;
                gf_copy16(to + (row - row0) * FEW_LD, in ? src : W, in);
            }
        }
        if (of_a) {
            const float* src = A + (size_t)row0 * K + k_mine + at;
            for (int row = row0; row < M; row += ROW_STEP, src += (size_t)ROW_STEP * K)
                gf_copy16(to + (row - row0 + cols) * FEW_LD, in_k ? src : A, in_k);
        }
    };
    // (w_ready, a model's weights: their first stages are asked for before the predecessor has ended)
    if (copies && w_ready)
        for (int s = 0; s < min(FEW_STAGES - 1, steps); ++s) bring(s, true, false);
    pdl_enter(TR_GEMM_F32);
    if (copies)
        for (int s = 0; s < FEW_STAGES - 1; ++s) {
            if (s < steps) bring(s, !w_ready, true);
            gf_commit();
        }
    const int warp = tid >> 5, lane = tid & 31, part = lane >> 3;
    const int groups = (cols + 8 * RN - 1) / (8 * RN);
    const int c0 = (warp % groups) * 8 * RN + (lane & 7), m0 = (warp / groups) * RM;
    const bool works = !copies && m0 < M;
    float acc[RN][RM];
    int w_at[RN], a_at[RM];                      // (beyond the last column or row: the last one again, not stored)
#pragma unroll
    for (int j = 0; j < RN; ++j) {
        w_at[j] = min(c0 + 8 * j, cols - 1) * FEW_LD + part * FEW_K;
#pragma unroll
        for (int i = 0; i < RM; ++i) acc[j][i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < RM; ++i) a_at[i] = (cols + min(m0 + i, M - 1)) * FEW_LD + part * FEW_K;
    for (int step = 0; step < steps; ++step) {
        if (copies) gf_wait<FEW_STAGES - 2>();
        __syncthreads();
        if (copies) {
            if (step + FEW_STAGES - 1 < steps) bring(step + FEW_STAGES - 1, true, true);
            gf_commit();
        }
        if (!works) continue;
        const float* base = smem + (step % FEW_STAGES) * rows * FEW_LD;
        float w[2][RN][4], a[2][RM][4];
        auto fetch = [&](int b, int k) {
#pragma unroll
            for (int j = 0; j < RN; ++j) load4(base + w_at[j] + k, w[b][j]);
#pragma unroll
            for (int i = 0; i < RM; ++i) load4(base + a_at[i] + k, a[b][i]);
        };
        auto multiply = [&](int b) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int j = 0; j < RN; ++j)
#pragma unroll
                    for (int i = 0; i < RM; ++i) acc[j][i] = fmaf(a[b][i][e], w[b][j][e], acc[j][i]);
        };
        fetch(0, 0);
#pragma unroll
        for (int k = 0; k < FEW_K; k += 8) {
            fetch(1, k + 4);
            multiply(0);
            if (k + 8 < FEW_K) fetch(0, k + 8);
            multiply(1);
        }
    }
    if (copies) {
        gf_wait<0>();
        return;
    }
    if (!works) return;                          // (whole warps)
#pragma unroll
    for (int j = 0; j < RN; ++j) {
        const int col = c0 + 8 * j, n = n0 + col;
#pragma unroll
        for (int i = 0; i < RM; ++i) {
            float sum = acc[j][i];
#pragma unroll
            for (int r = 1; r < PARTS; ++r) sum += __shfl_down_sync(0xffffffffu, acc[j][i], 8 * r);
            if (part == 0 && col < cols && n < N && m0 + i < M)
                C[(size_t)(m0 + i) * N + n] = bias ? sum + bias[n] : sum;
        }
    }
}

// ---------------------------------------------------------------------------------------------- rows of any width
constexpr int GB = 64;   // tile of C is GB x GB
constexpr int GK = 16;   // k-step

__global__ void __launch_bounds__(256, 5)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C, int M,
                int N, int K) {
    __shared__ float sa[GK][GB + 4];
    __shared__ float sw[GK][GB + 4];
    __shared__ float done[16][256];     // every thread's sums of the ranges that are done (in registers: a fifth slower in full waves)
    pdl_enter(TR_GEMM_F32);
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;          // 16 x 16 threads, 4 x 4 outputs each
    const int m0 = blockIdx.y * GB, n0 = blockIdx.x * GB;
    const int Kp = part_of(K);
    float acc[4][4] = {};
    const int lr = tid >> 2;            // 0..63: row of the tile this thread loads
    const int lk = (tid & 3) * 4;       // 0,4,8,12: first k of its four elements
    int next = Kp;
    for (int k0 = 0; k0 < K; k0 += GK) {
        if (k0 == next) {               // a range of k begins
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float& sum = acc[i / 4][i % 4];
                done[i][tid] = k0 == Kp ? sum : done[i][tid] + sum;
                sum = 0.f;
            }
            next += Kp;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + lk + j;
            const int am = m0 + lr, wn = n0 + lr;
            sa[lk + j][lr] = (am < M && k < K) ? A[(size_t)am * K + k] : 0.f;
            sw[lk + j][lr] = (wn < N && k < K) ? W[(size_t)wn * K + k] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < GK; ++k) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = sa[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = sw[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            const float sum = K > Kp ? done[4 * i + j][tid] + acc[i][j] : acc[i][j];
            if (n < N) C[(size_t)m * N + n] = bias ? sum + bias[n] : sum;
        }
    }
}

template <int BM, int BN, int TM, int TN, int CL>
static int launch_f32_tiles(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
    auto kernel = gemm_f32_tile_kernel<BM, BN, TM, TN, CL>;
    const int stages = TILE_STAGES * (BM + BN) * TILE_LD * 4, smem = CL > 1 ? max(stages, BM * BN * 4) : stages + BM * BN * 4;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    if constexpr (CL == 1)
        return launch(kernel, dim3((M + BM - 1) / BM, (N + BN - 1) / BN), (BM / TM) * (BN / TN), smem, stream, A, W, bias, C, M, N, K);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((M + BM - 1) / BM * CL, (N + BN - 1) / BN);
    cfg.blockDim = dim3((BM / TM) * (BN / TN));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    return launch_counted(cfg, kernel, A, W, bias, C, M, N, K);
}

template <int RM>
static int launch_f32_few(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int cols, int w_ready,
                          cudaStream_t stream) {
    const int smem = FEW_STAGES * (cols + M) * FEW_LD * 4;
    const int warps = (cols + 15) / 16 * ((M + RM - 1) / RM);
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_few_kernel<RM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    return launch(gemm_f32_few_kernel<RM>, dim3((N + cols - 1) / cols), warps * 32 + COPIERS, smem, stream, A, W, bias, C, M, N, K,
                  cols, w_ready);
}

// How many outputs, over all of k, the fullest SM takes.
static double fullest(int M, int N, int BM, int BN, int CL) {
    const long long blocks = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN) * CL;
    return (double)((blocks + 147) / 148) * BM * BN / CL;
}

// What tiles of BM x 64 take for a short k, in steps of 16 of k of a tile of 64 x 64: the blocks that follow one another on the
// fullest SM, and a block's own way through a step where it has the SM to itself; a cluster's exchange is one step more.
static double tile_cost(int M, int N, int K, int BM, int CL) {
    const long long blocks = (long long)((M + BM - 1) / BM) * ((N + 63) / 64) * CL;
    const int steps = CL > 1 ? part_of(K) / TILE_K : (K + TILE_K - 1) / TILE_K;
    return (steps + (CL > 1 ? 1 : 0)) * ((double)((blocks + 147) / 148) * (BM == 32 ? 0.5625 : 1.0) + (BM == 32 ? 0.7 : 1.0));
}

}  // namespace air

// w_ready: W was complete before the launch ahead of this one was made (a model's weights): it may be read before that one ends.
AIR_API int air_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int w_ready,
                         cudaStream_t stream) {
    using namespace air;
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return AIR_ERR_BAD_ARGUMENT;
    if (K % 4 || (((uintptr_t)A | (uintptr_t)W) & 15) || (N + 63) / 64 > 65535) {
        dim3 grid((N + GB - 1) / GB, (M + GB - 1) / GB);
        if (grid.y > 65535) return AIR_ERR_BAD_ARGUMENT;
        return launch(gemm_f32_kernel, grid, 256, 0, stream, A, W, bias, C, M, N, K);
    }
    // A stream of weights up to 16 rows, unless k is so short that its blocks' ways in and out are all that it has: 4 rows by 4,096 x 16
    // 2.8 us against 2.2 by half tiles, 16 rows by 4,096 x 32 4.3 and 2.6, by 16,384 x 64 14.7 and 6.4 (by 4,096 x 64 4.7 and 4.0, one row
    // by 4,096 x 32 2.2 and 2.6).  As many columns to a block as put every SM to work.  (16 rows by 16,384 x 2,048: 80 us;
    // tiles of 32 rows, half of them empty, would take the 77 us of 32 rows there, and twice as long where N is small: 64
    // blocks at 1,024 columns.)
    if (M <= FEW_ROWS && (K <= 16 || (K <= 32 && M > 8) || (K <= 64 && N > 148 * FEW_COLS)))
        return launch_f32_tiles<32, 64, 4, 4, 1>(A, W, bias, C, M, N, K, stream);
    if (M <= FEW_ROWS) {
        const int cols = max(1, min(FEW_COLS, (N + 147) / 148));
        if (M == 1) return launch_f32_few<1>(A, W, bias, C, M, N, K, cols, w_ready, stream);
        if (M == 2) return launch_f32_few<2>(A, W, bias, C, M, N, K, cols, w_ready, stream);
        return launch_f32_few<4>(A, W, bias, C, M, N, K, cols, w_ready, stream);
    }
    // From 64 steps of k on, a cluster with a block for every range: tiles of 64 x 64 wherever they share out as evenly over the
    // SMs as tiles of 32 x 64 do, whose outputs cost an eighth more to feed.  (32 rows by 16,384 x 2,048: 72 us against 117; 300 by
    // 3,072 x 2,048: 119 against 111.  Tiles of 128 columns or rows were within 3 % of 64 x 64 at 512 and 2,048 rows and slower
    // below.)
    if (K >= 1024) {
        if (fullest(M, N, 32, 64, PARTS) * 1.125 < fullest(M, N, 64, 64, PARTS))
            return launch_f32_tiles<32, 64, 4, 4, PARTS>(A, W, bias, C, M, N, K, stream);
        return launch_f32_tiles<64, 64, 4, 8, PARTS>(A, W, bias, C, M, N, K, stream);
    }
    // Fewer steps: the quickest of the four by tile_cost.  Measured over 1,188 sizes (17 to 2,048 rows, 64 to 16,384 columns, k of
    // 16 to 768): in the mean 2 % above the quickest of the four.  us, by blocks that began their ranges one after the other (17 rows: in
    // a cluster), by the kernel of any width, and now: 2,048 rows by 8,192 x 64 173, 120, 74; 777 by 4,096 x 64 43, 28, 20; 300 by 2,048 x
    // 512 65, 61, 28; 17 by 2,048 x 16 4.0, 2.4, 2.2.
    const double whole = tile_cost(M, N, K, 64, 1), half = tile_cost(M, N, K, 32, 1), whole_cut = tile_cost(M, N, K, 64, PARTS),
                 half_cut = tile_cost(M, N, K, 32, PARTS), least = min(min(whole, half), min(whole_cut, half_cut));
    if (whole == least) return launch_f32_tiles<64, 64, 4, 8, 1>(A, W, bias, C, M, N, K, stream);
    if (whole_cut == least) return launch_f32_tiles<64, 64, 4, 8, PARTS>(A, W, bias, C, M, N, K, stream);
    if (half == least) return launch_f32_tiles<32, 64, 4, 4, 1>(A, W, bias, C, M, N, K, stream);
    return launch_f32_tiles<32, 64, 4, 4, PARTS>(A, W, bias, C, M, N, K, stream);
}

AIR_API int air_trace_set_gemm_f32(unsigned long long* buffer) { return air::set_trace_here(buffer); }
