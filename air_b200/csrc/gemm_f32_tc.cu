// 32-bit matrix product on the fifth-generation tensor cores: C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]), float32 in and out.
//
// Nothing is computed at a lower precision than by fused multiply-adds: a float32 number, times 2^24, is cut into three bfloat16
// numbers that add up to it exactly (x = x1 + x2 + x3, each the rest rounded to nearest: 3 x 8 bits hold the 24, and the factor
// keeps the last of them within bfloat16's range down to the smallest number that 32 bits hold; without it bits were lost below
// 2^-110), a product of two bfloat16 numbers is exact in 32 bits, and of the nine products per pair the six down to 2^-17 of the
// largest are taken (the others together are below 2^-24 of it, without a bias).  The tensor cores add up 64 numbers of k, the small
// products first; every such sum is then added to a 32-bit total in registers, in ascending order over an eighth of k, and the
// eighths' totals are added in ascending order; their sum is multiplied by 2^-48.  So the chain of roundings is K/512 additions of
// sums of 64 where the multiply-add kernels (gemm_f32.cu) have K/4 additions of one product.
// The sum of an element is the same whatever M is and wherever its row stands, as in gemm_f32.cu; which of the two files
// takes a product depends on the matrix W alone.
//
// A result that is not finite (an infinity among the operands, a number from 2^104 or a sum from 2^80 on, which the factors take
// out of range) is worked out again by multiply-adds from memory, in the order of gemm_f32.cu, so that such operands give what they
// give there.
//
//   split_rows_kernel      for more than eight rows: A -> planes of bfloat16 [3][M][Kp], Kp = K up to a multiple of 64
//   gemm_f32_tc_kernel     one block, or several that share out the eighths of k, per tile of 128 rows of W by NT rows of A: a cluster of
//                          four or eight, or (up to eight rows) two, four or eight that leave the eighths' totals in memory;
//                          384 threads a block:
//     warps 0-7   the 128 rows of W (float32, brought by TMA in boxes of 32 k) are cut into planes by the thread that owns
//                 the row and put into tensor memory as the M side of the product, 64 k at a time, two buffers; the same
//                 threads add the finished sums to their totals (warps 0-3 one half of k and of the columns, 4-7 the other);
//     warps 8, 10 issue the copies of W (ahead of the end of the launch before this one where it is a model's weight) and A
//                 (up to eight rows: warps 10 and 11 cut them themselves);
//     warp 9      issues tcgen05.mma, A from tensor memory, B (the planes of the rows of A) from shared memory.
//   ft_add_kernel          adds up the totals that are in memory
// The planes of W stay out of shared memory, which for few rows would be the bound: 32 KB of W would be written, read,
// written as 48 KB and read six times.
// Measured, us a product in a chain of products with different matrices, by gemm_f32.cu and here: 4 rows by 37,888 x 3,584 122
// and 83 (6.5 TB/s: bound by the bytes of W), by 3,584 x 18,944 69 and 48, by 3,584 x 3,584 15.6 and 13.1, by 4,608 x 3,584 16.4 and
// 14.9, by 16,384 x 2,048 40 and 26.5; one row by 16,384 x 2,048 30 and 25.8, by 2,048 x 8,192 18.8 and 16.5, by 2,048 x 2,048 6.2 and 6.9;
// 16 rows by 37,888 x 3,584 230 and 86; 64 rows by 16,384 x 2,048 122 and 33; 300 rows by 2,048 x 2,048 81 and 33, by 16,384 x 2,048
// 529 and 144 (140 TFLOP/s of float32 products, 840 of bfloat16 ones: the tensor pipe, three rounds of 2.6 full), by 37,888 x
// 3,584 2,034 and 445.  Errors against 64 bits (2-norm), normal numbers: k 2,048 2.7e-7 and 7.4e-8, k 18,944 1.2e-6 and 1.8e-7;
// numbers of one sign (truncation inside the tensor cores adds up) 1.7e-7 and 9.1e-8, 4.7e-7 and 1.1e-7.
// What made the difference inside: a wait for a barrier that is long there costs a warp some 100 cycles, so each role waits once
// a chunk (128 rows of A: 1.19 -> 1.04 us a chunk); with all totals of a place asked for before the first is added the clusters'
// exchange fell from 16 to 6 us; rows of A cut by the block instead of a launch ahead are worth 2 us up to eight rows and cost
// 40 % at 16.  Deeper rings for one block per SM were slower (no room for the next product's first copies).
// Every wait on an mbarrier is bounded; on giving up the block sets *status = 4 (as gemm_tc.cu).
#include "common.cuh"
#include "tma.cuh"
#include "umma.cuh"

#include <cooperative_groups.h>

#include <type_traits>

namespace air {

constexpr int FT_BM = 128, FT_BK = 64, FT_PARTS = 8, FT_WORKERS = 256, FT_THREADS = FT_WORKERS + 128;
constexpr int FT_BOX = 128 * 32 * 4;                        // a box of W: 128 rows of 32 numbers
constexpr int FT_A_COLS = 3 * FT_BK / 2;                    // tensor memory of a chunk's planes of W

struct FtArgs {
    const float* a;
    const float* w;
    const float* bias;
    float* c;
    int M, N, K, w_ready;
    int cluster;        // blocks that share a tile: 1, 4 or 8 (a cluster), or 2, 4 or 8 that leave their sums in memory (APART)
    int* status;
    float* sums;        // APART: [FT_PARTS][M][N], the eighths' totals, for ft_add_kernel
};

// Up to 32 rows of A two blocks share an SM; up to FT_CUT rows a warp of the block cuts them into planes itself.  The sum of the eighths that are done is kept in registers where there is room
// for it, else in shared memory (a number of its own per thread).
__host__ __device__ constexpr bool ft_done_in_smem(int nt) { return nt > 64; }
__host__ __device__ constexpr int ft_done(int nt) { return ft_done_in_smem(nt) ? nt * FT_BM * 4 : 0; }
constexpr int FT_CUT = 8;
__host__ __device__ constexpr int ft_x_stage(int nt) { return 3 * nt * FT_BK * 2; }
__host__ __device__ constexpr int ft_x_stages(int nt) { return nt <= 16 ? 5 : nt <= 32 ? 3 : nt <= 64 ? 4 : 2; }
__host__ __device__ constexpr int ft_w_stages(int nt) {     // what is left of an SM, or of half of one
    const int room = (nt <= 32 ? 112 : 224) * 1024 - ft_x_stages(nt) * ft_x_stage(nt) - ft_done(nt);
    return room / FT_BOX > 10 ? 10 : room / FT_BOX;
}
__host__ __device__ constexpr int ft_tmem_cols(int nt) { return 2 * FT_A_COLS + 2 * nt <= 256 ? 256 : 512; }
__host__ __device__ constexpr int ft_smem(int nt) {
    return 1024 + ft_w_stages(nt) * FT_BOX + ft_x_stages(nt) * ft_x_stage(nt) + ft_done(nt) + 128 +
           16 * (ft_w_stages(nt) + ft_x_stages(nt));
}
// k of an eighth: whole chunks
__host__ __device__ __forceinline__ int ft_part(int K) { return ((K + FT_PARTS - 1) / FT_PARTS + FT_BK - 1) / FT_BK * FT_BK; }

// x -= the low half of p, y -= the high half (bfloat16 each): by two operations that take bfloat16 numbers as they are, or TOGETHER by one on
// both, which wants them widened (64 rows by 11,008 x 4,096 53.4 -> 51.4 us, 300 by 16,384 x 2,048 143.5 -> 143.0; where two blocks share an SM
// that is slower: 17 rows 45.2, 12 rows 44.0 -> 45.6).
template <bool TOGETHER> __device__ __forceinline__ void ft_less(float& x, float& y, uint32_t p) {
    if constexpr (TOGETHER)
        asm("{\n\t.reg .b64 v, w;\n\t.reg .b32 l, h;\n\tshl.b32 l, %2, 16;\n\tand.b32 h, %2, 0xffff0000;\n\tmov.b64 v, {%0, %1};\n\t"
            "mov.b64 w, {l, h};\n\tsub.rn.f32x2 v, v, w;\n\tmov.b64 {%0, %1}, v;\n\t}"
            : "+f"(x), "+f"(y) : "r"(p));
    else
        asm("{\n\t.reg .b16 l, h, m;\n\tmov.b16 m, 0xBF80;\n\tmov.b32 {l, h}, %2;\n\tfma.rn.f32.bf16 %0, l, m, %0;\n\tfma.rn.f32.bf16 %1, h, m, %1;\n\t}"
            : "+f"(x), "+f"(y) : "r"(p));
}
// Two neighbouring numbers times FT_SCALE as three pairs of bfloat16, the first in the low half.  (The factor costs 300 rows by
// 16,384 x 2,048 142.8 -> 145.5 us, few rows nothing; as two multiplications one row lost 2 % as well.  Sums taken from tensor
// memory 32 columns at a time instead of 8, and ft_less, bring it back to 143.0; 17 to 32 rows keep a loss of 2 to 4 %.)
constexpr float FT_SCALE = 0x1p24f, FT_UNSCALE = 0x1p-48f;      // (of a number, of a product of two)
template <bool TOGETHER = false> __device__ __forceinline__ void ft_split(float x, float y, uint32_t (&p)[3]) {
    asm("{\n\t.reg .b64 v, f;\n\tmov.b64 v, {%0, %1};\n\tmov.b64 f, {%2, %2};\n\tmul.rn.f32x2 v, v, f;\n\tmov.b64 {%0, %1}, v;\n\t}"
        : "+f"(x), "+f"(y) : "f"(FT_SCALE));
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
        p[i] = *reinterpret_cast<const uint32_t*>(&b);
        if (i < 2) ft_less<TOGETHER>(x, y, p[i]);
    }
}

// a += x, b += y, in one instruction.
__device__ __forceinline__ void ft_add(float& a, float& b, uint32_t x, uint32_t y) {
    asm("{\n\t.reg .b64 u, v;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tadd.rn.f32x2 u, u, v;\n\tmov.b64 {%0, %1}, u;\n\t}"
        : "+f"(a), "+f"(b) : "r"(x), "r"(y));
}

// Waits with a whole warp, every lane for a barrier of its own choice; one try where all are there already.
__device__ __forceinline__ bool ft_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ a, __nv_bfloat16* __restrict__ planes, int M, int K, int Kp, int vec) {
    pdl_enter(TR_CONVERT);
    const long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * 4, plane = (long long)M * Kp;
    if (i >= plane) return;
    const int m = (int)(i / Kp), k = (int)(i % Kp);
    const float* src = a + (size_t)m * K + k;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (vec && k + 4 <= K) load4(src, v);
    else
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (k + e < K) v[e] = src[e];
    uint32_t lo[3], hi[3];
    ft_split(v[0], v[1], lo);
    ft_split(v[2], v[3], hi);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(planes + p * plane + i) = make_uint2(lo[p], hi[p]);
}

__device__ __forceinline__ void ft_store_planes(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// 8, 16, 24 or 32 columns with one wait, which stands in the same statement so that nothing is read ahead of it.
#define FT_R8(r, i) "=r"(r[i]), "=r"(r[i + 1]), "=r"(r[i + 2]), "=r"(r[i + 3]), "=r"(r[i + 4]), "=r"(r[i + 5]), "=r"(r[i + 6]), "=r"(r[i + 7])
#define FT_LD "tcgen05.ld.sync.aligned.32x32b."
#define FT_LD_WAIT "tcgen05.wait::ld.sync.aligned;"
__device__ __forceinline__ void ft_load(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile(FT_LD "x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t" FT_LD_WAIT : FT_R8(r, 0) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void ft_load(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(FT_LD "x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t" FT_LD_WAIT
                 : FT_R8(r, 0), FT_R8(r, 8) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void ft_load(uint32_t taddr, uint32_t (&r)[24]) {
    asm volatile(FT_LD "x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%24];\n\t"
                 FT_LD "x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%25];\n\t" FT_LD_WAIT
                 : FT_R8(r, 0), FT_R8(r, 8), FT_R8(r, 16) : "r"(taddr), "r"(taddr + 16) : "memory");
}
__device__ __forceinline__ void ft_load(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(FT_LD "x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, "
                 "%22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t" FT_LD_WAIT
                 : FT_R8(r, 0), FT_R8(r, 8), FT_R8(r, 16), FT_R8(r, 24) : "r"(taddr) : "memory");
}

// The results of rows m_lo .. m_hi - 1 and columns n0 .. n0 + 127 that are not finite, by multiply-adds from memory in the order of
// gemm_f32.cu, by all threads of the block: R rows at a time (few where registers are few), a thread half of them by one column,
// both operands through a ring of stages of 32 k in shared memory.  A row of A with a NaN is left as it is (its results are NaN).
// 300 rows by 16,384 x 2,048, us: no such results 155, NaN in every row 198, an infinity in one row 460, in every row 2,350 (gemm_f32.cu
// 532 in all cases); 8 rows 34, 36, 134, 135 (47).  Result after result by the thread that had it: 155, 70,700, 548, 70,100.
constexpr int FT_AGAIN_K = 32, FT_AGAIN_LD = FT_AGAIN_K + 4;
__host__ __device__ constexpr int ft_again_rows(int nt) { return nt <= 32 ? 16 : 32; }
__host__ __device__ constexpr int ft_again_stages(int r) { return r <= 16 ? 2 : 3; }
__host__ __device__ constexpr int ft_again_stage(int r) { return (r + FT_BM) * FT_AGAIN_LD; }        // in numbers
__host__ __device__ constexpr int ft_again_numbers(int r) { return ft_again_stages(r) * ft_again_stage(r) + r; }

template <int BYTES> __device__ __forceinline__ void ft_copy(float* to, const float* from, bool in) {
    const int bytes = in ? BYTES : 0;                // (0: zeros, nothing is read)
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(to)), "l"(from), "n"(BYTES), "r"(bytes) : "memory");
}

template <int R>
__device__ __noinline__ void ft_again(const FtArgs& args, int m_lo, int m_hi, int n0, float* smem) {
    constexpr int LD = FT_AGAIN_LD, PARTS = 4, STAGES = ft_again_stages(R), STAGE = ft_again_stage(R);
    const float *const A = args.a, *const W = args.w;
    const int K = args.K, N = args.N, Kp = ((K + PARTS - 1) / PARTS + 15) / 16 * 16, steps_per_part = (Kp + FT_AGAIN_K - 1) / FT_AGAIN_K;
    const int tid = threadIdx.x, lane = tid & 31, col = tid & (FT_BM - 1), row0 = tid / FT_BM * (R / 2);
    int* nan_row = (int*)(smem + STAGES * STAGE);
    for (int m = m_lo; m < m_hi; m += R) {
        const int rows = min(R, m_hi - m), mine = min(R / 2, rows - row0);
        for (int i = tid >> 5; i < rows; i += blockDim.x >> 5) {
            bool none = false;
            for (int k = lane; k < K; k += 32) none |= isnan(A[(size_t)(m + i) * K + k]);
            none = __any_sync(0xffffffffu, none);
            if (lane == 0) nan_row[i] = none;
        }
        __syncthreads();
        unsigned wrong = 0;
        if (n0 + col < N)
            for (int i = 0; i < mine; ++i)
                if (!nan_row[row0 + i] && !isfinite(args.c[(size_t)(m + row0 + i) * N + n0 + col])) wrong |= 1u << i;
        if (!__syncthreads_or(wrong)) continue;
        // step s: 32 k of part s / steps_per_part; zeros beyond the part and beyond the rows and columns
        const int steps = (K + Kp - 1) / Kp * steps_per_part;
        auto bring = [&](int s) {
            float* to = smem + s % STAGES * STAGE;
            const int part = s / steps_per_part, k0 = part * Kp + s % steps_per_part * FT_AGAIN_K, k_hi = min(K, (part + 1) * Kp);
            for (int j = tid; j < R * FT_AGAIN_K; j += blockDim.x) {
                const int r = j / FT_AGAIN_K, k = j % FT_AGAIN_K;
                const bool in = s < steps && r < rows && k0 + k < k_hi;
                ft_copy<4>(to + r * LD + k, in ? A + (size_t)(m + r) * K + k0 + k : A, in);
            }
            for (int j = tid; j < FT_BM * FT_AGAIN_K / 4; j += blockDim.x) {
                const int r = j / (FT_AGAIN_K / 4), k = j % (FT_AGAIN_K / 4) * 4;
                const bool in = s < steps && n0 + r < N && k0 + k < k_hi;       // (K % 4 == 0)
                ft_copy<16>(to + (R + r) * LD + k, in ? W + (size_t)(n0 + r) * K + k0 + k : W, in);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        for (int s = 0; s < STAGES - 1; ++s) bring(s);
        float sum[R / 2], acc[R / 2];
#pragma unroll
        for (int i = 0; i < R / 2; ++i) acc[i] = sum[i] = 0.f;
        for (int s = 0; s < steps; ++s) {
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
            __syncthreads();
            bring(s + STAGES - 1);
            const float* at = smem + s % STAGES * STAGE;
            auto multiply = [&](auto whole) {
#pragma unroll 1
                for (int k = 0; k < FT_AGAIN_K; k += 4) {
                    float w[4], x[4];
                    load4(at + (R + col) * LD + k, w);
#pragma unroll
                    for (int i = 0; i < R / 2; ++i) {
                        if (!decltype(whole)::value && i >= mine) break;
                        load4(at + (row0 + i) * LD + k, x);
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[i] = fmaf(x[e], w[e], acc[i]);
                    }
                }
            };
            if (mine == R / 2) multiply(std::true_type());      // (reads that need not wait for a row's count)
            else if (mine > 0) multiply(std::false_type());
            if ((s + 1) % steps_per_part == 0) {
#pragma unroll
                for (int i = 0; i < R / 2; ++i) {
                    sum[i] = s >= steps_per_part ? sum[i] + acc[i] : acc[i];
                    acc[i] = 0.f;
                }
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
        for (int i = 0; i < R / 2; ++i)
            if (wrong >> i & 1) args.c[(size_t)(m + row0 + i) * N + n0 + col] = args.bias ? sum[i] + args.bias[n0 + col] : sum[i];
        __syncthreads();
    }
}

// APART: the blocks of a tile leave every eighth's totals in memory and ft_add_kernel adds them up: up to FT_CUT rows, where the totals
// are few.  Such blocks need not stand in one GPC, and the SMs take one each before any takes two, which a cluster's do not wait for:
// 4 rows by 4,608 x 3,584 19.3 -> 15.3 us, by 2,048 x 8,192 21.0 -> 17.1, by 16,384 x 2,048 (two blocks) 32.2 -> 27.1; of 9 rows and
// more the second launch and the totals cost what that saves.
template <int NT, bool APART>
__global__ void __launch_bounds__(FT_THREADS, NT <= 32 ? 2 : 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ FtArgs args) {
    constexpr int WS = ft_w_stages(NT), XS = ft_x_stages(NT), XSTAGE = ft_x_stage(NT), XPLANE = XSTAGE / 3, HALF = NT / 2;
    constexpr int TMEM_COLS = ft_tmem_cols(NT);
    constexpr bool DONE_IN_SMEM = ft_done_in_smem(NT);
    static_assert(NT % 16 == 0 && 2 * FT_A_COLS + 2 * NT <= 512, "two sets of accumulators beside two buffers of planes");
    static_assert(WS >= 3 && WS * FT_BOX + XS * XSTAGE >= NT * FT_BM * 4 * 2, "the stages' memory takes a tile's sums twice");
    static_assert(WS * FT_BOX + XS * XSTAGE >= ft_again_numbers(ft_again_rows(NT)) * 4, "and what ft_again stages");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sw = smem;
    uint8_t* sx = smem + WS * FT_BOX;
    float* done_smem = (float*)(sx + XS * XSTAGE) + threadIdx.x;                    // [HALF][FT_WORKERS]
    uint64_t* bars = (uint64_t*)(sx + XS * XSTAGE + ft_done(NT));
    uint64_t *w_full = bars, *w_empty = bars + WS, *x_full = bars + 2 * WS, *x_empty = bars + 2 * WS + XS;
    uint64_t *a_full = bars + 2 * WS + 2 * XS, *d_full = a_full + 2;
    uint32_t* tmem_slot = (uint32_t*)(a_full + 4);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m_tiles = (args.M + NT - 1) / NT;
    const int tile = blockIdx.x / args.cluster, rank = blockIdx.x % args.cluster;
    const int m0 = (tile % m_tiles) * NT, n0 = (tile / m_tiles) * FT_BM;      // (tiles beside one another share their weights)
    const int part = ft_part(args.K), mine = part * (FT_PARTS / args.cluster);
    const int k_lo = min(args.K, rank * mine), k_hi = min(args.K, k_lo + mine);
    const int chunks = (k_hi - k_lo + FT_BK - 1) / FT_BK, chunks_per_part = part / FT_BK;

    if (threadIdx.x == 0) {
        for (int i = 0; i < WS; ++i) {
            mbar_init(&w_full[i], 1);
            mbar_init(&w_empty[i], 4);
        }
        for (int i = 0; i < XS; ++i) {
            mbar_init(&x_full[i], 1);
            mbar_init(&x_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&a_full[i], 8);
            mbar_init(&d_full[i], 1);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) tmem_alloc(tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    float total[HALF], done[DONE_IN_SMEM || APART ? 1 : HALF];
#pragma unroll
    for (int i = 0; i < HALF; ++i) total[i] = 0.f;
    if constexpr (!DONE_IN_SMEM && !APART)
#pragma unroll
        for (int i = 0; i < HALF; ++i) done[i] = 0.f;
    const int quarter = warp & 3, half = warp >> 2, r = quarter * 32 + lane;   // (workers: a row of W, half of k and of the columns)
    if (warp == 8) {
        if (lane == 0) {
            // ------------------------------------------------ the rows of W
            const int boxes = 2 * chunks, first = args.w_ready ? min(WS, boxes) : 0;
            // Read once (rows of one tile), W is first to leave L2, so that the next launches' code stays there (a decoder layer of 2,048 with 1 to 8 requests: 94 -> 86 to
            // 100 -> 94 us; of 3,584 192 -> 189).
            uint64_t once;
            asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
            auto load = [&](int box) {
                const int s = box % WS;
                mbar_expect_tx(&w_full[s], FT_BOX);
                if (args.M <= NT) tma_load_2d_hint(sw + s * FT_BOX, &map_w, k_lo + box * 32, n0, &w_full[s], once);
                else tma_load_2d(sw + s * FT_BOX, &map_w, k_lo + box * 32, n0, &w_full[s]);
            };
            for (int b = 0; b < first; ++b) load(b);
            pdl_wait();
            trace_point(TR_GEMM_F32);
            for (int b = first; b < boxes; ++b) {
                if (b >= WS && !mbar_wait(&w_empty[b % WS], (b / WS - 1) & 1, abort_flag)) break;
                load(b);
            }
        }
    } else if (warp >= 10) {
        if (NT == 16 && (APART || args.M <= FT_CUT)) {
            // ------------------------------------------------ the rows of A, cut here: two warps take the
            // chunks in turn, 16 lanes a row's 64 k
            pdl_wait();
            const int k_mine = (lane & 15) * 4, row0 = lane >> 4;
            const bool vec = ((uintptr_t)args.a & 15) == 0;
            float v[FT_CUT / 2][4];
            auto fetch = [&](int c) {
                const int k = k_lo + c * FT_BK + k_mine;
#pragma unroll
                for (int i = 0; i < FT_CUT / 2; ++i) {
                    const float* src = args.a + (size_t)(row0 + 2 * i) * args.K + k;
                    if (row0 + 2 * i >= args.M || k >= args.K) continue;             // (such columns of the result are nobody's)
                    if (vec) load4(src, v[i]);                                       // (K % 4 == 0)
                    else
#pragma unroll
                        for (int e = 0; e < 4; ++e) v[i][e] = src[e];
                }
            };
#pragma unroll
            for (int i = 0; i < FT_CUT / 2; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) v[i][e] = 0.f;
            if (warp - 10 < chunks) fetch(warp - 10);
            for (int c = warp - 10; c < chunks; c += 2) {
                const int s = c % XS;
                if (c >= XS && !__all_sync(0xffffffffu, mbar_wait(&x_empty[s], (c / XS - 1) & 1, abort_flag))) break;
                uint32_t lo[FT_CUT / 2][3], hi[FT_CUT / 2][3];
                const bool in = k_lo + c * FT_BK + k_mine < args.K;
#pragma unroll
                for (int i = 0; i < FT_CUT / 2; ++i) {
                    ft_split(in ? v[i][0] : 0.f, in ? v[i][1] : 0.f, lo[i]);
                    ft_split(in ? v[i][2] : 0.f, in ? v[i][3] : 0.f, hi[i]);
                }
                if (c + 2 < chunks) fetch(c + 2);
#pragma unroll
                for (int i = 0; i < FT_CUT / 2; ++i) {
                    const int row = row0 + 2 * i;
                    uint8_t* to = sx + s * XSTAGE + row * 128 + (((k_mine >> 3) ^ row) << 4) + (k_mine & 4) * 2;
#pragma unroll
                    for (int p = 0; p < 3; ++p)
                        if (row < args.M) *reinterpret_cast<uint2*>(to + p * XPLANE) = make_uint2(lo[i][p], hi[i][p]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&x_full[s]);
            }
        } else if (warp == 10 && lane == 0) {
            // ------------------------------------------------ the planes of the rows of A
            pdl_wait();
            for (int c = 0; c < chunks; ++c) {
                const int s = c % XS;
                if (c >= XS && !mbar_wait(&x_empty[s], (c / XS - 1) & 1, abort_flag)) break;
                mbar_expect_tx(&x_full[s], XSTAGE);
                for (int p = 0; p < 3; ++p)
                    tma_load_2d(sx + s * XSTAGE + p * XPLANE, &map_x, k_lo + c * FT_BK, p * args.M + m0, &x_full[s]);
            }
        }
    } else if (warp == 9) {
        // ---------------------------------------------------- MMA issuer (see gemm_tc.cu)
        constexpr uint32_t idesc = umma_idesc(FT_BM, NT);
        // the six products, smallest first: (plane of W, plane of A)
        constexpr int PW[6] = {2, 0, 1, 1, 0, 0}, PX[6] = {0, 2, 1, 0, 1, 0};
        const uint64_t dx0 = umma_desc(smem_u32(sx));
        bool ok = true;
        for (int c = 0; c < chunks && ok; ++c) {
            const int buf = c & 1, s = c % XS;
            // (the accumulators are free: a warp says that a chunk's planes are there after it has taken the sums before the last)
            ok = ft_wait(lane & 1 ? &x_full[s] : &a_full[buf], lane & 1 ? (c / XS) & 1 : c >> 1 & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint32_t d = tmem + 2 * FT_A_COLS + buf * NT, a = tmem + buf * FT_A_COLS;
            const uint64_t dx = dx0 + (uint64_t)(s * (XSTAGE >> 4));
            if (elect_one()) {
#pragma unroll
                for (int p = 0; p < 6; ++p)
#pragma unroll
                    for (int k = 0; k < FT_BK / 16; ++k)
                        umma_bf16_ts(d, a + PW[p] * (FT_BK / 2) + 8 * k, dx + (uint64_t)(PX[p] * (XPLANE >> 4)) + 2 * k, idesc,
                                     p + k > 0 ? 1u : 0u);
                umma_commit(&d_full[buf]);
                umma_commit(&x_empty[s]);
            }
            __syncwarp();
        }
    } else {
        // ---------------------------------------------------- workers
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        int left = chunks_per_part;                  // chunks until the eighth is complete
        bool first_part = true;
        auto take = [&](int c) {                     // a finished chunk's sums
            const int buf = c & 1;
            if (!ft_wait(&d_full[buf], c >> 1 & 1, abort_flag)) return false;
            tc_fence_after();
            const uint32_t from = tmem + 2 * FT_A_COLS + buf * NT + half * HALF + lanes;
            auto add = [&](auto first, auto columns) {      // (one wait for as many as there are registers)
                uint32_t v[decltype(columns)::value];
                ft_load(from + decltype(first)::value, v);
#pragma unroll
                for (int e = 0; e < decltype(columns)::value; e += 2)
                    ft_add(total[decltype(first)::value + e], total[decltype(first)::value + e + 1], v[e], v[e + 1]);
            };
            constexpr int AT_ONCE = HALF < 32 ? HALF : 32;
            add(std::integral_constant<int, 0>(), std::integral_constant<int, AT_ONCE>());
            if constexpr (HALF > AT_ONCE) add(std::integral_constant<int, AT_ONCE>(), std::integral_constant<int, HALF - AT_ONCE>());
            tc_fence_before();
            if constexpr (APART) {
                if (--left > 0 && c + 1 < chunks) return true;
                if (first_part) pdl_wait();          // (the memory may be what the predecessor reads)
                const int m1 = m0 + half * HALF, rows = n0 + r < args.N ? args.M - m1 : 0;
                float* to = args.sums + ((size_t)(rank * (FT_PARTS / args.cluster) + c / chunks_per_part) * args.M + m1) * args.N + n0 + r;
#pragma unroll
                for (int i = 0; i < HALF; ++i) {
                    if (i < rows) to[(size_t)i * args.N] = total[i];
                    total[i] = 0.f;
                }
                left = chunks_per_part;
                first_part = false;
            } else if (--left == 0 && c + 1 < chunks) {     // (the last eighth stays in total)
#pragma unroll
                for (int i = 0; i < HALF; ++i) {
                    if constexpr (DONE_IN_SMEM) done_smem[i * FT_WORKERS] = first_part ? total[i] : done_smem[i * FT_WORKERS] + total[i];
                    else done[i] = first_part ? total[i] : done[i] + total[i];
                    total[i] = 0.f;
                }
                left = chunks_per_part;
                first_part = false;
            }
            return true;
        };
        bool ok = true;
        for (int c = 0; c < chunks && ok; ++c) {
            const int buf = c & 1, box = 2 * c + half, s = box % WS;
            // (the buffer for the planes is free: this warp has seen the end of the products before the last)
            ok = ft_wait(&w_full[s], (box / WS) & 1, abort_flag);
            if (!ok) break;
            const float* row = (const float*)(sw + s * FT_BOX + r * 128);
            const uint32_t to = tmem + buf * FT_A_COLS + half * 16 + lanes;
#pragma unroll
            for (int k = 0; k < 2; ++k) {            // 16 k: four pieces of 16 bytes, eight columns of each plane
                uint32_t p[3][8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float v[4];
                    load4(row + (((4 * k + j) ^ (r & 7)) << 2), v);
                    uint32_t lo[3], hi[3];
                    ft_split<(NT > 32)>(v[0], v[1], lo);
                    ft_split<(NT > 32)>(v[2], v[3], hi);
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        p[i][2 * j] = lo[i];
                        p[i][2 * j + 1] = hi[i];
                    }
                }
#pragma unroll
                for (int i = 0; i < 3; ++i) ft_store_planes(to + i * (FT_BK / 2) + 8 * k, p[i]);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&w_empty[s]);
                mbar_arrive(&a_full[buf]);
            }
            if (c > 0) ok = take(c - 1);
        }
        if (ok && chunks > 0) take(chunks - 1);
    }
    pdl_wait();                                      // (nothing is written before the predecessor has completed)
    tc_fence_before();
    __syncthreads();                                 // every copy has landed and every product is done: the stages are free
    const bool gave_up = *abort_flag != 0;
    if (gave_up) {
        // copies that were issued may still be on their way: give them time before their memory is used again
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
        if (threadIdx.x == 0 && args.status) atomicExch(args.status, 4);
    }
    if (warp == 9) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }

    // ---------------------------------------------------------- the eighths' totals
    if constexpr (APART) return;                     // (they are in memory)
    else {
    float* const C = args.c;
    const float* const bias = args.bias;
    const int M = args.M, N = args.N;
    bool odd = false;                                // a result that is not finite was stored
    auto done_at = [&](int i) -> float {
        if constexpr (DONE_IN_SMEM) return done_smem[i * FT_WORKERS];
        else return done[i];
    };
    const bool several = chunks > chunks_per_part;   // (this block has more than one eighth)
    if (args.cluster == 1) {
        if (warp < 8 && !gave_up && n0 + r < N) {
            const float b = bias ? bias[n0 + r] : 0.f;
            const int m1 = m0 + half * HALF, rows = M - m1;
            float* to = C + (size_t)m1 * N + n0 + r;
#pragma unroll
            for (int i = 0; i < HALF; ++i) {
                float sum = (several ? done_at(i) + total[i] : total[i]) * FT_UNSCALE;
                if (bias) sum += b;
                if (i < rows) {
                    odd |= !isfinite(sum);
                    to[(size_t)i * N] = sum;
                }
            }
        }
        if (__syncthreads_or(odd)) ft_again<ft_again_rows(NT)>(args, m0, min(M, m0 + NT), n0, (float*)smem);
        return;
    }
    // A block of several hands on the sum of its eighths if it is the first, else (two of them) one and the other.
    float* sums = (float*)smem;                      // [2][NT][128]
    if (warp < 8 && !gave_up) {
#pragma unroll
        for (int i = 0; i < HALF; ++i) {
            float* to = sums + (half * HALF + i) * FT_BM + r;
            const bool both = rank > 0 && several;
            to[0] = several ? (both ? done_at(i) : done_at(i) + total[i]) : total[i];
            if (args.cluster < FT_PARTS) to[NT * FT_BM] = both ? total[i] : 0.f;
        }
    }
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();
    const bool whole = N % 4 == 0 && ((uintptr_t)C & 15) == 0;      // (n is a multiple of 4)
    // (the rows of A are shared out among the blocks; all of a place's numbers are asked for before the first is added)
    auto add_up = [&](auto blocks) {
        constexpr int CL = decltype(blocks)::value, VALUES = CL == FT_PARTS ? CL : 2 * CL - 1;
        const float* from[VALUES];
#pragma unroll
        for (int q = 0; q < CL; ++q) {
            const float* theirs = cluster.map_shared_rank(sums, q);
            if (CL == FT_PARTS) from[q] = theirs;
            else {
                if (q > 0) from[2 * q - 1] = theirs;
                from[2 * q] = q > 0 ? theirs + NT * FT_BM : theirs;
            }
        }
        for (int i = threadIdx.x * 4; i < NT / CL * FT_BM; i += FT_WORKERS * 4) {
            const int at = rank * (NT / CL) * FT_BM + i, m = m0 + at / FT_BM, n = n0 + at % FT_BM;
            if (m >= M || n >= N) continue;
            float v[VALUES][4];
#pragma unroll
            for (int q = 0; q < VALUES; ++q) load4(from[q] + at, v[q]);
            float* to = C + (size_t)m * N + n;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float sum = v[0][e];
#pragma unroll
                for (int q = 1; q < VALUES; ++q) sum += v[q][e];
                sum *= FT_UNSCALE;
                if (n + e < N) {
                    if (bias) sum += bias[n + e];
                    odd |= !isfinite(sum);
                    v[0][e] = sum;
                    if (!whole) to[e] = sum;
                }
            }
            if (whole) store4(to, v[0]);
        }
    };
    if (warp < 8 && !gave_up) {
        if (args.cluster == FT_PARTS) add_up(std::integral_constant<int, FT_PARTS>());
        else add_up(std::integral_constant<int, 4>());
    }
    cluster.sync();                                  // (nobody's memory is read any more)
    const int m1 = m0 + rank * (NT / args.cluster);
    if (__syncthreads_or(odd)) ft_again<ft_again_rows(NT)>(args, m1, min(M, m1 + NT / args.cluster), n0, (float*)smem);
    }
}

// The eighths' totals of up to FT_CUT rows: 128 columns to a block, a thread four columns of a row.
__global__ void __launch_bounds__(256) ft_add_kernel(const __grid_constant__ FtArgs args) {
    __shared__ __align__(16) float smem[ft_again_numbers(16)];
    pdl_enter(TR_GEMM_F32);
    const int M = args.M, N = args.N, n0 = blockIdx.x * FT_BM, n = n0 + (threadIdx.x & 31) * 4, m = threadIdx.x >> 5;
    const int part = ft_part(args.K), parts = (args.K + part - 1) / part;
    const size_t eighth = (size_t)M * N;
    const bool whole = N % 4 == 0 && ((uintptr_t)args.c & 15) == 0;
    bool odd = false;
    if (m < M && n < N) {
        const float* from = args.sums + (size_t)m * N + n;
        float* to = args.c + (size_t)m * N + n;
        float v[FT_PARTS][4];
#pragma unroll
        for (int p = 0; p < FT_PARTS; ++p) {
            if (p >= parts) continue;
            if (N % 4 == 0) load4(from + p * eighth, v[p]);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e) v[p][e] = n + e < N ? from[p * eighth + e] : 0.f;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float sum = v[0][e];
#pragma unroll
            for (int p = 1; p < FT_PARTS; ++p)
                if (p < parts) sum += v[p][e];
            sum *= FT_UNSCALE;
            if (n + e < N) {
                if (args.bias) sum += args.bias[n + e];
                odd |= !isfinite(sum);
                if (!whole) to[e] = sum;
            }
            v[0][e] = sum;
        }
        if (whole) store4(to, v[0]);
    }
    if (__syncthreads_or(odd)) ft_again<16>(args, 0, M, n0, smem);
}

// A tensor map of a row-major float32 matrix [rows, cols] with boxes of 128 rows x 32 numbers and the 128-byte swizzle.
static int ft_map_w(CUtensorMap* map, const float* base, long long rows, long long cols) {
    EncodeTiled enc = encode_tiled();
    if (!enc) return AIR_ERR_BAD_ARGUMENT;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)cols * 4};
    const cuuint32_t box[2] = {32, 128}, elem[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, elem,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 200000 + (int)r;
}

template <int NT, bool APART = false>
static int ft_launch(const CUtensorMap& mw, const CUtensorMap& mx, const FtArgs& args, cudaStream_t stream) {
    auto kernel = gemm_f32_tc_kernel<NT, APART>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ft_smem(NT));
    if (e != cudaSuccess) return (int)e;
    const unsigned blocks = (unsigned)((args.N + FT_BM - 1) / FT_BM) * ((args.M + NT - 1) / NT) * args.cluster;
    if (args.cluster == 1) return launch(kernel, blocks, FT_THREADS, ft_smem(NT), stream, mw, mx, args);
    if constexpr (APART) {
        const int rc = launch(kernel, blocks, FT_THREADS, ft_smem(NT), stream, mw, mx, args);
        return rc ? rc : launch(ft_add_kernel, (args.N + FT_BM - 1) / FT_BM, 32 * FT_CUT, 0, stream, args);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(FT_THREADS);
    cfg.dynamicSmemBytes = ft_smem(NT);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = args.cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    return launch_counted(cfg, kernel, mw, mx, args);
}

// Width of a tile and blocks that share it, by what they were measured to take, us: a chunk of 64 k (with all SMs at work; tensor
// pipe, power and L2 at widths of 96 and more, the cutting of W below), and the way into and out of a block.  A grid of more
// blocks than fit takes another round; a cluster wants its SMs in one GPC, so that fewer blocks fit.  W itself arrives at 6.3 TB/s.
struct FtShape { int width, cluster, apart; };
// Up to FT_CUT rows: `blocks` blocks of `chunks` chunks.  A block that has an SM to itself takes 0.8 us a chunk, two on one 1.15,
// and 6.3 TB/s are 0.0052 a block.  Measured in a chain of products of one row and here, us: 4,096 x 2,048 8 blocks apart 9.0 (9.3); 2,048 x 8,192
// 16.4 (16.8); 4,608 x 3,584 14.5 (14.5); 16,384 x 2,048 one block to a tile 32.6, two apart 25.9 (25.3); 37,888 x 3,584 82 (89), 87 (93).
// Clusters of eight: their blocks stand two to an SM from some 74 on, and 232 fit.  They are taken where each has its SM (1,024
// x 2,048 5.6 against 5.8 apart), and where they fill the chip, so that there is nothing to spread (a layer of width 3,584 with one
// request, the output product's 224 blocks 176 against 183, its whole; 2 to 8 requests +-1); between (2,048 x 2,048, 128) a whole
// layer of width 2,048 took 83 us with them and 81 apart.
static double ft_few_us(long long blocks, int chunks, bool clustered, bool apart) {
    if (clustered && blocks > 74 && (blocks < 200 || blocks > 232)) return 1e30;
    auto chunk = [&](long long n) { return n <= 0 ? 0. : max(n <= (clustered ? 74 : 148) ? 0.8 : 1.15, n * 0.0052); };
    return chunks * (blocks / 296 * chunk(296) + chunk(blocks % 296)) + (blocks - 1) / 296 * 3 + (clustered ? 2 : apart ? 4 : 3);
}
static FtShape ft_shape(int M, int N, int K) {
    static const struct { int width; float chunk; } widths[] = {{16, 0.6f}, {32, 0.62f}, {64, 0.75f}, {96, 1.15f}, {112, 1.27f}, {128, 1.35f}};
    const int clusters[] = {1, 4, FT_PARTS};
    FtShape best{0, 0, 0};
    double least = 0;
    auto take = [&](const FtShape& shape, double us) {
        if (best.width && us >= least) return;
        best = shape;
        least = us;
    };
    auto chunks_of = [&](int cl) { return min((K + FT_BK - 1) / FT_BK, ft_part(K) / FT_BK * (FT_PARTS / cl)); };
    if (M <= FT_CUT) {
        const long long tiles = ((long long)N + FT_BM - 1) / FT_BM;
        take({16, 1, 0}, ft_few_us(tiles, chunks_of(1), false, false));
        take({16, FT_PARTS, 0}, ft_few_us(tiles * FT_PARTS, chunks_of(FT_PARTS), true, false));
        for (int cl = 2; cl <= FT_PARTS; cl *= 2) take({16, cl, 1}, ft_few_us(tiles * cl, chunks_of(cl), false, true));
        return best;
    }
    for (const auto& w : widths) {
        if (w.width <= 64 && w.width < M) continue;          // (narrow tiles only where one holds all rows)
        const bool two = w.width <= 32;
        for (int cl : clusters) {
            const long long blocks = ((long long)N + FT_BM - 1) / FT_BM * ((M + w.width - 1) / w.width) * cl;
            const int fit = cl == 1 ? (two ? 296 : 148) : cl == 4 ? (two ? 280 : 140) : (two ? 232 : 112);
            const double us = (double)((blocks + fit - 1) / fit) * (chunks_of(cl) * w.chunk + (two ? (cl == 1 ? 5 : 6) : (cl == 1 ? 9 : 8)));
            take({w.width, cl, 0}, max(us, 4.0 * N * K / 6.3e6 + 5));
        }
        if (w.width <= 64) break;                            // (the narrowest that holds all rows)
    }
    return best;
}
static FtShape ft_shape_or(int M, int N, int K, int width, int cluster, int apart) {
    return width && cluster ? FtShape{width, cluster, apart} : ft_shape(M, N, K);
}

}  // namespace air

// How many eighths' totals of M * N numbers air_gemm_f32_tc_apart wants room for: 8 or none.
AIR_API int air_gemm_f32_tc_parts(int M, int N, int K, int width, int cluster, int apart) {
    using namespace air;
    return M > 0 && N > 0 && K > 0 && ft_shape_or(M, N, K, width, cluster, apart).apart ? FT_PARTS : 0;
}

// planes: scratch of 3 * M * (K up to a multiple of 64) bfloat16; null up to FT_CUT rows.  sums: scratch of
// air_gemm_f32_tc_parts * M * N numbers.  W aligned to 16 bytes, K % 4 == 0.
// w_ready as in air_gemm_f32.  width, cluster, apart: rows of A to a tile (16, 32, 64, 96, 112 or 128), blocks that share a tile (1, 4
// or 8), and whether these (2, 4 or 8, for up to FT_CUT rows in tiles of 16) leave their sums in memory, for tests and measurements; 0: by
// ft_shape.
AIR_API int air_gemm_f32_tc_apart(const float* A, const float* W, const float* bias, float* C, void* planes, float* sums, int M, int N,
                                  int K, int w_ready, int width, int cluster, int apart, int* status, cudaStream_t stream) {
    using namespace air;
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 || ((uintptr_t)W & 15)) return AIR_ERR_BAD_ARGUMENT;
    const FtShape shape = ft_shape_or(M, N, K, width, cluster, apart);
    width = shape.width;
    cluster = shape.cluster;
    const bool cut = M <= FT_CUT && width == 16;
    if (width < 16 || (cluster != 1 && cluster != 4 && cluster != FT_PARTS && !(cluster == 2 && shape.apart))) return AIR_ERR_BAD_ARGUMENT;
    if (shape.apart && (!cut || cluster == 1 || !sums || ((uintptr_t)sums & 15))) return AIR_ERR_BAD_ARGUMENT;
    if (!cut && (!planes || ((uintptr_t)planes & 15))) return AIR_ERR_BAD_ARGUMENT;
    const int Kp = (K + FT_BK - 1) / FT_BK * FT_BK;
    const long long blocks = ((long long)M * Kp / 4 + 255) / 256, rows = 3ll * M;
    if (blocks > 0x7fffffff || rows > 0x7fffffff ||
        ((long long)N + FT_BM - 1) / FT_BM * ((M + width - 1) / width) * cluster > 0x7fffffff)
        return AIR_ERR_BAD_ARGUMENT;
    CUtensorMap mw, mx;
    int rc = ft_map_w(&mw, W, N, K);
    if (rc) return rc;
    if (cut) mx = mw;                // (not used)
    else {
        rc = launch(split_rows_kernel, (unsigned)blocks, 256, 0, stream, A, (__nv_bfloat16*)planes, M, K, Kp, ((uintptr_t)A & 15) == 0);
        if (!rc) rc = tensor_map_2d(&mx, planes, rows, Kp, width);
        if (rc) return rc;
    }
    const FtArgs args{A, W, bias, C, M, N, K, w_ready, cluster, status, sums};
    if (shape.apart) return ft_launch<16, true>(mw, mx, args, stream);
    switch (width) {
        case 16: return ft_launch<16>(mw, mx, args, stream);
        case 32: return ft_launch<32>(mw, mx, args, stream);
        case 64: return ft_launch<64>(mw, mx, args, stream);
        case 96: return ft_launch<96>(mw, mx, args, stream);
        case 112: return ft_launch<112>(mw, mx, args, stream);
        case 128: return ft_launch<128>(mw, mx, args, stream);
        default: return AIR_ERR_BAD_ARGUMENT;
    }
}

// The same without that room.
AIR_API int air_gemm_f32_tc(const float* A, const float* W, const float* bias, float* C, void* planes, int M, int N, int K, int w_ready,
                            int width, int cluster, int* status, cudaStream_t stream) {
    using namespace air;
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return AIR_ERR_BAD_ARGUMENT;
    const FtShape shape = ft_shape_or(M, N, K, width, cluster, 0);
    return air_gemm_f32_tc_apart(A, W, bias, C, planes, nullptr, M, N, K, w_ready, shape.width, shape.apart ? FT_PARTS : shape.cluster, 0,
                                 status, stream);
}

AIR_API int air_trace_set_gemm_f32_tc(unsigned long long* buffer) { return air::set_trace_here(buffer); }
