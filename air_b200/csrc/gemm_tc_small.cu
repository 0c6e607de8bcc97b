// bfloat16 matrix product for a few tokens (up to 64) on the fifth-generation tensor cores, with the
// WEIGHTS as the M side of tcgen05.mma: C[T,N] = X[T,K] * W[N,K]^T is computed as its transpose,
// 128 rows of W (the accumulator's lanes) by NT = 16, 32 or 64 tokens (its columns).
//
// gemm_tc.cu puts the tokens on the M side, where an instruction always works on 128 rows: with 8
// tokens a k step of a 256-wide tile takes 128 cycles of the tensor pipe for 8 useful rows, and once
// the weights are in shared memory ahead of time (the block was resident while its predecessor
// ran) those cycles are what a decode step waits for: about 2.6 us per product with ten k-blocks
// per block.  Here a k step takes the time of reading 128 x 16 weights from shared memory (about
// 32 cycles).
//
// One persistent block per SM, 192 or 224 threads, as in gemm_tc.cu: warp 0 issues TMA loads (a tile of
// HALVES x 128 rows of W and the NT-row tile of X per stage, 128-byte swizzle, no multicast), warp 1
// (and warp 6, in turn, where a step is 16 KB) issues tcgen05.mma (M 128, N NT, K 16; per k step one per half of the W tile, sharing the tile of
// X) into one of two sets of accumulators, warps 2-5 read a finished accumulator (thread = output
// feature, columns = tokens) and write the result, coalesced over the features.
//   EPI_F32 / EPI_BF16  store C
//   EPI_SILU            HALVES = 2 and W holds, per 256 rows, 128 rows of the gate projection followed
//                       by the 128 rows of the up projection for the same outputs: silu(gate) * up
//   EPI_SILU, HALVES 1  the same with 64 gate rows and the 64 up rows for the same outputs in one tile of 128 (two copies a
//                       stage): twice as many tiles, for matrices whose tiles of 256 leave more than half of the SMs idle.
//                       The sums go through shared memory, where a thread finds a gate's and its up's
//   EPI_RELU2           store max(C, 0)^2 as bfloat16 (the hidden layer of a feed-forward without a gate)
//   EPI_F32, joined     matrices of few tiles, whose sums are wanted complete: a cluster of two or four blocks shares a tile, a part
//                       of the k range each, and adds the parts up, in order, through one another's shared memory.  A block's
//                       steps pass at some 65 GB/s whatever the tile, so 53 tiles leave half of the memory's rate unused:
//                       8 rows by 6,720 x 4,096 (two blocks) 16.4 -> 13.5 us, by 4,096 x 4,096 (four) 15.2 -> 10.0, by 3,648 x
//                       2,048 (four) 8.7 -> 6.7, 64 rows by 6,720 x 4,096 18.4 -> 15.6.  Tiles of 64 or 32 rows: 20 and 29.
//   EPI_PARTIAL         the k range is split over `splits` blocks; each writes C[split][T][N] (float32)
// Rows of X beyond T and rows of W beyond N are zero-filled by TMA.
// Every wait on an mbarrier is bounded; on giving up the block sets *status = 4 (as gemm_tc.cu).
#include "common.cuh"
#include "tma.cuh"
#include "umma.cuh"

#include <cooperative_groups.h>

namespace air {

constexpr int TS_BK = 64;


enum { TS_F32 = 0, TS_BF16 = 1, TS_SILU = 2, TS_PARTIAL = 3, TS_RELU2 = 4,   // as in gemm_tc.cu
       TS_JOINED = 5 };

struct TsArgs {
    void* out;          // F32/PARTIAL: float [splits][T][N]; BF16: bf16 [T][N]; SILU: bf16 [T][N/2]
    int T, N, K;
    int splits;
    int* status;
    // Optional scale per token, applied to the accumulators before the epilogue: rsqrt(sum over ss_tiles of
    // ss[tile][t] / K + eps), the RMSNorm scale of an input whose rows came as x * weight without it
    // (add_prenorm_kernel in elementwise.cu writes such rows and the sums of squares).  ss == nullptr: none.
    const float* ss;
    int ss_tiles;
    float eps;
    // SILU computes g' * sigmoid(act_alpha * g') * (u' + act_shift) with g' = min(gate, act_limit) and
    // u' = clamp(up, -act_limit, act_limit) where act_limit > 0: (1, 0, 0) is SiLU(gate) * up; act_alpha < 0: max(g', 0) * (u' + act_shift).
    float act_alpha, act_limit, act_shift;
};

// Warps that issue products, each into accumulators of its own: one needs 0.2 us for a step of k, four products and a commit.
__host__ __device__ constexpr int ts_issuers(int halves) { return halves == 1 ? 2 : 1; }
__host__ __device__ constexpr int ts_threads(int halves) { return 160 + 32 * ts_issuers(halves); }
// (a stage always belongs to the same issuer)
__host__ __device__ constexpr int ts_stages(int nt, int halves) {
    const int fit = 196 * 1024 / ((halves * 128 + nt) * TS_BK * 2);
    return (fit > 24 ? 24 : fit) / ts_issuers(halves) * ts_issuers(halves);
}
__host__ __device__ constexpr int ts_tmem_cols(int nt, int halves) {
    return 2 * halves * nt * ts_issuers(halves);             // 64, 128 or 256: a power of two
}

template <int N>
__device__ __forceinline__ void ts_ask(uint32_t taddr, uint32_t (&r)[N]) {
    static_assert(N == 4 || N == 8, "columns of tensor memory at a time");
    if constexpr (N == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr) : "memory");
}
// The sums of N tokens for this thread's feature, of the issuers' accumulators (of one alone, which the only step of k went to,
// where there are no more steps).  taddr: the first token's column of the first accumulator.
template <int NT, int ISSUERS, int N>
__device__ __forceinline__ void ts_sums(uint32_t taddr, int steps, int before, float (&v)[N]) {
    uint32_t a[N], b[N];
    __syncwarp();
    const bool both = ISSUERS > 1 && steps > 1;
    ts_ask<N>(taddr + (ISSUERS > 1 && steps == 1 ? before % ISSUERS * NT : 0), a);
    if (both) ts_ask<N>(taddr + NT, b);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = both ? __uint_as_float(a[i]) + __uint_as_float(b[i]) : __uint_as_float(a[i]);
}

template <int NT, int EPI, int HALVES>
__global__ void __launch_bounds__(ts_threads(HALVES), 1)
gemm_tc_small_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                     const TsArgs args) {
    constexpr bool PAIRED = EPI == TS_SILU && HALVES == 1;      // 64 gate rows and 64 up rows to a tile
    constexpr bool JOINED = EPI == TS_JOINED;                    // (a block is one part of one tile)
    static_assert(!JOINED || HALVES == 1, "a cluster shares a tile of 128 rows");
    constexpr int HALF_W = 128 * TS_BK * 2;           // 16 KB: 128 rows of W, 64 of k
    constexpr int STAGE_W = HALVES * HALF_W;
    constexpr int STAGE_X = NT * TS_BK * 2;
    constexpr int STAGES = ts_stages(NT, HALVES);
    constexpr int ISSUERS = ts_issuers(HALVES);
    constexpr int ACC_COLS = HALVES * NT * ISSUERS;
    constexpr int TMEM_COLS = ts_tmem_cols(NT, HALVES);
    constexpr int TILE_N = HALVES * 128;               // rows of W per tile
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sw = smem;
    uint8_t* sx = smem + STAGES * STAGE_W;
    uint64_t* bars = (uint64_t*)(sx + STAGES * STAGE_X);
    uint64_t* full = bars;
    uint64_t* empty = bars + STAGES;
    uint64_t* acc_full = bars + 2 * STAGES;
    uint64_t* acc_empty = bars + 2 * STAGES + 2;
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * STAGES + 4);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    float* row_scale = (float*)(tmem_slot + 2);       // [NT]
    float* pairs = row_scale + NT;                     // PAIRED: [NT][128], a tile's sums
    // where a tile's rows of W lie (PAIRED: its gate rows; the up rows are 128 further on)
    auto row_of = [](int tile) { return PAIRED ? tile / 2 * 256 + tile % 2 * 64 : tile * TILE_N; };
    // Every byte of W is read once: first to leave L2, so that what the next launches need stays there, their code above all (it is
    // read from memory again otherwise, line after line, while everybody waits).  Without and with it, us: decode steps of one token, 8 layers of
    // 2,048, a prompt of 33 and 15 tokens 5,519 -> 5,130; a layer of 4,096 with 8 requests over 8,192 keys 112.9 -> 110.6.
    uint64_t once;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
    auto load_w = [&](int stage, int k, int n0) {
        tma_load_2d_hint(sw + stage * STAGE_W, &map_w, k, n0, &full[stage], once);
        if (PAIRED) tma_load_2d_hint(sw + stage * STAGE_W + HALF_W / 2, &map_w, k, n0 + 128, &full[stage], once);
    };

    pdl_trigger();
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int n_tiles = (args.N + TILE_N - 1) / TILE_N;
    const int k_tiles = (args.K + TS_BK - 1) / TS_BK;
    const int k_per = (k_tiles + args.splits - 1) / args.splits;
    const int total = n_tiles * args.splits;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], ISSUERS);
            mbar_init(&acc_empty[i], 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // ------------------------------------------------ producer
            const uint32_t bytes = (uint32_t)(STAGE_W + STAGE_X);
            uint32_t stage = 0, phase = 0;
            bool first = true;
            trace_point(TR_GEMM_TC + 100);   // when this block became resident
            for (int tile = blockIdx.x; tile < total && !*abort_flag; tile += gridDim.x) {
                const int split = tile % args.splits;
                const int n0 = row_of(tile / args.splits);
                const int k_begin = split * k_per, k_end = min(k_tiles, k_begin + k_per);
                int kt = k_begin;
                if (first) {
                    // The weights are written by no kernel: the first stages' tiles of W are fetched
                    // while the predecessor in the stream may still be running; the tiles of X (its
                    // output) follow once it has completed.
                    first = false;
                    const int pre = min(STAGES, k_end - k_begin);
                    for (int i = 0; i < pre; ++i) {
                        mbar_expect_tx(&full[i], bytes);
                        load_w(i, (k_begin + i) * TS_BK, n0);
                    }
                    // (Asking further k-tiles into L2 here, as gemm_tc.cu does, was measured to cost 1.7 % of a
                    // decode step with this kernel: the ring is deep, and the requests delay the loads of
                    // the small kernels that run meanwhile.)
                    pdl_wait();
                    trace_point(TR_GEMM_TC);
                    for (int i = 0; i < pre; ++i) tma_load_2d(sx + i * STAGE_X, &map_x, (k_begin + i) * TS_BK, 0, &full[i]);
                    kt = k_begin + pre;
                    if (pre == STAGES) phase = 1; else stage = pre;
                }
                for (; kt < k_end; ++kt) {
                    if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) break;
                    mbar_expect_tx(&full[stage], bytes);
                    load_w(stage, kt * TS_BK, n0);
                    tma_load_2d(sx + stage * STAGE_X, &map_x, kt * TS_BK, 0, &full[stage]);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1 || warp > 5) {
        // ---------------------------------------------------- MMA issuers: each warp runs together, an
        // elected lane issues (see gemm_tc.cu).  Two of them take the stages in turn, each always the same ones: a wait by parity
        // could not tell a round of a stage from the one two later, were a stage to go from one to the other.
        constexpr uint32_t idesc = umma_idesc(128, NT);
        const uint64_t dw0 = umma_desc(smem_u32(sw)), dx0 = umma_desc(smem_u32(sx));
        const int issuer = warp == 1 ? 0 : warp - 5;
        uint32_t before = 0, it = 0;                      // steps of k in the tiles so far
        bool ok = true;
        for (int tile = blockIdx.x; tile < total && ok && !*abort_flag; tile += gridDim.x, ++it) {
            const int split = tile % args.splits;
            const int k_begin = split * k_per, k_end = min(k_tiles, k_begin + k_per);
            const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
            ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[acc], acc_phase ^ 1, abort_flag));
            if (!ok) break;
            tc_fence_after();
            const uint32_t d = tmem_base + acc * ACC_COLS + issuer * NT;
            const int skip = (issuer + before) % ISSUERS;  // (1 - before, 0 - before: the same modulo two)
            uint32_t stage = (before + skip) % STAGES, phase = (before + skip) / STAGES & 1;
            for (int kt = k_begin + skip; kt < k_end; kt += ISSUERS) {
                // (a stage that is already there costs one try; the bounded loop only where the issuer has to wait)
                if (!mbar_try_wait(&full[stage], phase)) ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, abort_flag));
                if (!ok) break;
                tc_fence_after();
                const uint64_t dw = dw0 + (uint64_t)(stage * (STAGE_W >> 4));
                const uint64_t dx = dx0 + (uint64_t)(stage * (STAGE_X >> 4));
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < TS_BK / 16; ++k)
#pragma unroll
                        for (int hf = 0; hf < HALVES; ++hf)
                            umma_bf16(d + hf * ISSUERS * NT, dw + (uint64_t)(hf * (HALF_W >> 4)) + 2 * k, dx + 2 * k, idesc,
                                      (kt >= k_begin + ISSUERS || k > 0) ? 1u : 0u);
                    umma_commit(&empty[stage]);
                }
                __syncwarp();
                if ((stage += ISSUERS) >= STAGES) { stage -= STAGES; phase ^= 1; }
            }
            before += k_end - k_begin;
            if (ok && elect_one()) umma_commit(&acc_full[acc]);
            __syncwarp();
        }
    } else {
        // ---------------------------------------------------- epilogue: warps 2..5, thread = feature
        pdl_wait();   // nothing is written before the predecessor has completed
        const int quarter = warp & 3;                     // the 32 lanes of tensor memory this warp may read
        const int r = quarter * 32 + lane;                // row of the tile's half
        if (args.ss) {
            // the tokens' norm scales, worked out while the weights stream: eight loads in flight at a time,
            // the sums added in the order of the tiles
            if (r < NT) {
                float total = 0.f;
                if (r < args.T) {
                    for (int base = 0; base < args.ss_tiles; base += 8) {
                        float part[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            part[i] = base + i < args.ss_tiles ? args.ss[(size_t)(base + i) * args.T + r] : 0.f;
#pragma unroll
                        for (int i = 0; i < 8; ++i) total += part[i];
                    }
                }
                row_scale[r] = r < args.T ? rsqrtf(total / (float)args.K + args.eps) : 0.f;
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        uint32_t it = 0;
        int done = 0;                                     // steps of k in the tiles so far
        // (PAIRED: the four warps meet at a barrier twice per tile, so all of them go through all tiles, also when a wait has
        // run out: one that left would keep the others there for good)
        for (int tile = blockIdx.x; tile < total && (PAIRED || !*abort_flag); tile += gridDim.x, ++it) {
            const int split = tile % args.splits;
            const int n0 = (tile / args.splits) * TILE_N;
            const int steps = min(k_tiles, (split + 1) * k_per) - split * k_per, before = done;
            done += steps;
            const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
            const bool ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[acc], acc_phase, abort_flag));
            if (!PAIRED && !ok) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + acc * ACC_COLS + ((uint32_t)(quarter * 32) << 16);
            // Loops over a few tokens at a time, as far as there are tokens: this code runs once or twice per launch, from cold
            // instruction caches, and its length is what it costs.  All tokens at once, one after the other in the code, against this, both
            // with two issuers, us a decoder layer of width 2,048: 1 token 55 -> 53, 24 tokens 64.5 -> 60.1, 50 tokens 84 -> 66.
            if constexpr (JOINED) {
                float* mine = (float*)smem;               // [NT][128]: every copy has landed and every product is done
#pragma unroll 1
                for (int t = 0; t < args.T; t += 8) {
                    float v[8];
                    ts_sums<NT, ISSUERS, 8>(taddr + t, steps, before, v);
#pragma unroll
                    for (int i = 0; i < 8; ++i) mine[(t + i) * 128 + r] = v[i];
                }
            } else if constexpr (PAIRED) {
                if (ok) {
#pragma unroll 1
                    for (int t = 0; t < args.T; t += 8) {
                        float v[8];
                        ts_sums<NT, ISSUERS, 8>(taddr + t, steps, before, v);
#pragma unroll
                        for (int i = 0; i < 8; ++i) pairs[(t + i) * 128 + r] = args.ss ? v[i] * row_scale[t + i] : v[i];
                    }
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (ok) {
                    __nv_bfloat16* out = (__nv_bfloat16*)args.out + (size_t)(tile / args.splits) * 64 + (r & 63);
#pragma unroll 2
                    for (int t = r >> 6; t < args.T; t += 2)
                        out[(size_t)t * (args.N / 2)] = __float2bfloat16_rn(
                            gated_activation(pairs[t * 128 + (r & 63)], pairs[t * 128 + 64 + (r & 63)], args.act_alpha, args.act_limit, args.act_shift));
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");      // (read before the next tile's are written)
            } else if constexpr (EPI == TS_SILU) {
                const int col = n0 / 2 + r;
#pragma unroll 1
                for (int t = 0; t < args.T; t += 4) {
                    static_assert(ISSUERS == 1, "gate and up in tiles of 256 rows");
                    // (both behind one wait: 64 rows by 24,576 x 1,024 15.8 us; behind a wait each 18.2)
                    uint32_t gate[4], up[4];
                    __syncwarp();
                    ts_ask<4>(taddr + t, gate);
                    ts_ask<4>(taddr + NT + t, up);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (col < args.N / 2) {
                        __nv_bfloat16* out = (__nv_bfloat16*)args.out + (size_t)t * (args.N / 2) + col;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float scale = args.ss ? row_scale[t + i] : 1.f;
                            if (t + i < args.T)
                                out[(size_t)i * (args.N / 2)] = __float2bfloat16_rn(
                                    gated_activation(__uint_as_float(gate[i]) * scale, __uint_as_float(up[i]) * scale, args.act_alpha, args.act_limit, args.act_shift));
                        }
                    }
                }
            } else {
#pragma unroll 1
                for (int at = 0; at < HALVES * NT; at += 8) {
                    const int hf = at / NT, t = at % NT;
                    if (t >= args.T) continue;
                    float v[8];
                    ts_sums<NT, ISSUERS, 8>(taddr + hf * ISSUERS * NT + t, steps, before, v);
                    const int col = n0 + hf * 128 + r;
                    if (col < args.N) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            if (t + i >= args.T) break;
                            if (args.ss) v[i] *= row_scale[t + i];
                            if constexpr (EPI == TS_BF16) {
                                ((__nv_bfloat16*)args.out)[(size_t)(t + i) * args.N + col] = __float2bfloat16_rn(v[i]);
                            } else if constexpr (EPI == TS_RELU2) {
                                const float x = fmaxf(v[i], 0.f);
                                ((__nv_bfloat16*)args.out)[(size_t)(t + i) * args.N + col] = __float2bfloat16_rn(x * x);
                            } else {
                                ((float*)args.out)[((size_t)split * args.T + t + i) * args.N + col] = v[i];
                            }
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && ok) mbar_arrive(&acc_empty[acc]);
        }
    }

    // ---------------------------------------------------------- leaving
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        // copies that were issued may still be on their way: give them time before the block ends
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
        if (threadIdx.x == 0 && args.status) atomicExch(args.status, 4);
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
    if constexpr (JOINED) {
        cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
        cluster.sync();
        if (warp >= 2 && warp < 6) {                      // the parts in order; the tokens are shared out among the blocks
            // (a warp takes a token's 128 features at once, a lane four of them)
            const int col = (int)blockIdx.x / args.splits * TILE_N + 4 * lane;
            const bool whole = args.N % 4 == 0;
            const float* from[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) from[q] = cluster.map_shared_rank((float*)smem, q < args.splits ? q : 0) + 4 * lane;
#pragma unroll 4
            for (int t = (int)blockIdx.x % args.splits + args.splits * (warp & 3); t < args.T; t += 4 * args.splits) {
                float v[4][4];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (q < args.splits) load4(from[q] + t * 128, v[q]);
                float* to = (float*)args.out + (size_t)t * args.N + col;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float sum = v[0][e] + v[1][e];
                    if (args.splits == 4) sum = (sum + v[2][e]) + v[3][e];
                    if (args.ss) sum *= row_scale[t];
                    v[0][e] = sum;
                    if (!whole && col + e < args.N) to[e] = sum;
                }
                if (whole && col < args.N) store4(to, v[0]);
            }
        }
        cluster.sync();                                   // (nobody leaves while its memory is read)
    }
}

// Blocks that share a tile of complete sums, by what a product takes, us: a block's copies (a step of k is 16 KB at 65 GB/s) or
// the whole matrix at 6.5 TB/s, whichever is longer, and the exchange.  Every block has an SM to itself and eight steps of k in the
// mean (the last one may have fewer); clusters of four do not fit on all SMs (a cluster stands in one GPC).
static int ts_joined_parts(int n_tiles, int k_tiles, int sms) {
    int best = 1;
    double least = 0.95 * max(k_tiles * 0.25, n_tiles * k_tiles * 0.0025);
    for (int parts = 2; parts <= 4; parts *= 2) {
        if (n_tiles * parts > (parts == 4 ? sms - sms / 8 : sms) || k_tiles < 8 * parts ||
            (parts - 1) * ((k_tiles + parts - 1) / parts) >= k_tiles)
            continue;
        const double us = max(k_tiles * 0.25 / parts, n_tiles * k_tiles * 0.0025) + 3;
        if (us < least) {
            best = parts;
            least = us;
        }
    }
    return best;
}

// A tensor map of a row-major bf16 matrix [rows, cols] with boxes of box_rows x 64 and 128-byte swizzle.
static int ts_make_map(CUtensorMap* map, const void* base, long long rows, long long cols, int box_rows) {
    return tensor_map_2d(map, base, rows, cols, box_rows);
}

template <int NT, int EPI, int HALVES>
static int ts_launch(const CUtensorMap& mw, const CUtensorMap& mx, const TsArgs& args, int blocks, cudaStream_t stream) {
    constexpr int STAGES = ts_stages(NT, HALVES);
    // always more than half of an SM's shared memory, so that two blocks never share an SM (and its
    // tensor memory)
    const size_t smem = 1024 + (size_t)STAGES * (HALVES * 128 + NT) * TS_BK * 2 + 16 * STAGES + 256 + 4 * NT +
                        (EPI == TS_SILU && HALVES == 1 ? 512 * NT : 0);
    const size_t request = smem < 120 * 1024 ? 120 * 1024 : smem;
    auto kernel = gemm_tc_small_kernel<NT, EPI, HALVES>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)request);
    if (e != cudaSuccess) return (int)e;
    if constexpr (EPI == TS_JOINED) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(ts_threads(HALVES));
        cfg.dynamicSmemBytes = request;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = args.splits;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = pdl_enabled() ? 2 : 1;
        return launch_counted(cfg, kernel, mw, mx, args);
    }
    return launch(kernel, blocks, ts_threads(HALVES), request, stream, mw, mx, args);
}

template <int NT, int HALVES>
static int ts_dispatch_epi(int epi, const CUtensorMap& mw, const CUtensorMap& mx, const TsArgs& args, int blocks,
                           cudaStream_t stream) {
    switch (epi) {
        case TS_JOINED:
            if constexpr (HALVES == 1) return ts_launch<NT, TS_JOINED, 1>(mw, mx, args, blocks, stream);
            return AIR_ERR_BAD_ARGUMENT;
        case TS_F32: return ts_launch<NT, TS_F32, HALVES>(mw, mx, args, blocks, stream);
        case TS_BF16: return ts_launch<NT, TS_BF16, HALVES>(mw, mx, args, blocks, stream);
        case TS_SILU: return ts_launch<NT, TS_SILU, HALVES>(mw, mx, args, blocks, stream);
        case TS_PARTIAL: return ts_launch<NT, TS_F32, HALVES>(mw, mx, args, blocks, stream);
        case TS_RELU2: return ts_launch<NT, TS_RELU2, HALVES>(mw, mx, args, blocks, stream);
        default: return AIR_ERR_BAD_ARGUMENT;
    }
}

template <int HALVES>
static int ts_dispatch_tokens(int nt, int epi, const CUtensorMap& mw, const CUtensorMap& mx, const TsArgs& args,
                              int blocks, cudaStream_t stream) {
    switch (nt) {
        case 16: return ts_dispatch_epi<16, HALVES>(epi, mw, mx, args, blocks, stream);
        case 32: return ts_dispatch_epi<32, HALVES>(epi, mw, mx, args, blocks, stream);
        default: return ts_dispatch_epi<64, HALVES>(epi, mw, mx, args, blocks, stream);
    }
}

}  // namespace air

// x [T, K] bf16 with T <= 64, w [N, K] bf16 (for epi 2: per 256 rows 128 of gate, then 128 of up), K % 8 == 0.
// out as TsArgs.out.  tile_rows: 128 or 256 rows of W per tile (256 for epi 2).  max_blocks: the number of
// SMs to use (0: all).
AIR_API int air_gemm_tc_small(const void* x, const void* w, void* out, int T, int N, int K, int tile_rows, int epi,
                              int splits, int max_blocks, int* status, const float* ss, int ss_tiles, float eps,
                              float act_alpha, float act_limit, float act_shift, cudaStream_t stream) {
    using namespace air;
    if (T <= 0 || N <= 0) return 0;
    if (T > 64 || K <= 0 || K % 8 || splits < 1 || (splits > 1 && epi != TS_PARTIAL) || ((uintptr_t)x & 15) ||
        ((uintptr_t)w & 15) || ((uintptr_t)out & 15) || (tile_rows != 128 && tile_rows != 256))
        return AIR_ERR_BAD_ARGUMENT;
    if (epi == TS_SILU && (tile_rows != 256 || N % 256)) return AIR_ERR_BAD_ARGUMENT;
    const int k_tiles = (K + TS_BK - 1) / TS_BK;
    // every part of the k range must hold at least one k-tile (an accumulator that no product wrote is not zero)
    if (splits > k_tiles || (long long)(splits - 1) * ((k_tiles + splits - 1) / splits) >= k_tiles)
        return AIR_ERR_BAD_ARGUMENT;
    const int nt = T > 32 ? 64 : (T > 16 ? 32 : 16);
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (max_blocks > 0 && max_blocks < sms) sms = max_blocks;
    // Gate and up rows by 64 where twice as many tiles still are one round of the SMs (16,384 x 2,048, 64 tiles: 13.9 -> 11.1 us
    // inside a decode step of one token; 14,336 x 4,096, 56 tiles: 26 -> 21); beyond, two rounds of
    // half tiles are no shorter than one of whole ones.
    const bool paired = epi == TS_SILU && N / 256 * 2 <= sms;
    if (paired) tile_rows = 128;
    // (by the matrix alone, so that a row's sum does not depend on how many there are)
    if (epi == TS_F32 && tile_rows == 128) {
        const int parts = ts_joined_parts((N + 127) / 128, k_tiles, sms);
        if (parts > 1) {
            epi = TS_JOINED;
            splits = parts;
        }
    }
    CUtensorMap mw, mx;
    int rc = ts_make_map(&mw, w, N, K, paired ? 64 : tile_rows);
    if (rc) return rc;
    rc = ts_make_map(&mx, x, T, K, nt);
    if (rc) return rc;
    const long long tiles = (long long)((N + tile_rows - 1) / tile_rows) * splits;     // (joined: at most one to a block)
    const int blocks = (int)(tiles < sms ? tiles : sms);
    if (ss && ss_tiles < 1) return AIR_ERR_BAD_ARGUMENT;
    TsArgs args{out, T, N, K, splits, status, ss, ss_tiles, eps, act_alpha, act_limit, act_shift};
    if (tile_rows == 256) return ts_dispatch_tokens<2>(nt, epi, mw, mx, args, blocks, stream);
    return ts_dispatch_tokens<1>(nt, epi, mw, mx, args, blocks, stream);
}

AIR_API int air_trace_set_gemm_tc_small(unsigned long long* buffer) { return air::set_trace_here(buffer); }
