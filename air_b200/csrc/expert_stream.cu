// Products of a mixture's experts for steps with few rows per expert, on the fifth-generation tensor cores: C_g = X_g W_g^T,
// where the rows of expert g are the slots start[g] .. start[g + 1] of X [slots, K] (moe_sort_kernel's order; rows in that order
// and with the weights on them come from rows_by_index_kernel, or are the first product's results).
//
// A step of few tokens reads every chosen expert's matrices once and computes next to nothing: it is a stream of weights.  So
// the kernel is gemm_tc_small.cu's, with the weights as the M side of tcgen05.mma and a deep ring of stages that TMA fills,
// and a persistent block walks a list of tiles (row tile of an expert, 128 or 256 rows of its matrix, part of k) that it works
// out from the device's lists: the ring goes on filling across tiles and experts.  The warp-level kernel (grouped_gemm.cu, 64
// x 64 tiles, steps of 32 of k by cp.async) streamed at half the copy rate.
//   EPI 0  float32 rows to planes: p = o_index[slot], plane split * o_div + p % o_div, row p / o_div, times o_scale[p].  With
//          `splits` parts of k every part has planes of its own, which the consumer adds in order: more and shorter tiles
//          to deal out where few experts are reached (parts/experts.py)
//   EPI 1  W_g holds, per 256 rows, 128 of the gate and 128 of the linear branch: bfloat16 [slots, N / 2]
//   EPI 2  max(x, 0)^2 as bfloat16 [slots, N]
// A tile of W may reach into the next expert's rows, a tile of X into the next expert's slots: what they give is not stored.
// Measured, a whole mixture (router, lists, both products, a shared expert half as wide as the dense feed-forward) replayed as
// a graph, us: width 4,096, 16 experts of 3,584, 8 tokens 331 -> 190 (its bytes at the copy rate: 169), 100 tokens 419 by the
// library's grouped product -> 324; width 2,048, experts of 2,048: 8 tokens 94, 100 tokens 169 -> 129.
// What 300 and more tokens take now, and where the library takes over: RoutedExperts.  EPI 0's places and weights are worked out by
// a thread per slot while the products run; row by row in the loop that stores, an index, two divisions and a weight stood
// behind one another: a mixture of width 2,048 with 500 tokens 199 -> 163, with 64 145 -> 140, width 4,096 with 500 406 -> 378.
// Tiles of 256 slots (one set of accumulators, three stages) were slower than the library at any number of rows.
// Every wait on an mbarrier is bounded; on giving up the block sets *status = 4 (as gemm_tc.cu).
#include "common.cuh"
#include "tma.cuh"
#include "umma.cuh"

namespace air {

constexpr int XS_BK = 64;
constexpr int XS_THREADS = 192;
constexpr int XS_ROWS = 64, XS_WIDE = 128;      // slots of a row tile (moe_sort_kernel's): few rows per expert, many

struct XsArgs {
    void* out;
    int slots, N, K, splits;
    const int* start;            // [groups + 1]
    const int* tiles;            // pairs (group, first slot)
    int tile_rows;               // slots to a tile
    const int* num_tiles;
    int lists_ready;             // the lists were complete before this kernel's predecessor let anything start
    const int* o_index; int o_div; long long o_part_stride; int ldo; const float* o_scale;
    int* status;
    float act_alpha, act_limit, act_shift;
};

__host__ __device__ constexpr int xs_stages(int nt, int halves) {
    return 196 * 1024 / ((halves * 128 + nt) * XS_BK * 2) > 24 ? 24 : 196 * 1024 / ((halves * 128 + nt) * XS_BK * 2);
}
__host__ __device__ constexpr int xs_tmem_cols(int nt, int halves) { return 2 * halves * nt < 32 ? 32 : 2 * halves * nt; }

__device__ __forceinline__ void xs_load16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    tmem_ld16(taddr, r);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

template <int NT, int EPI, int HALVES>
__global__ void __launch_bounds__(XS_THREADS, 1)
expert_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const XsArgs args) {
    static_assert(EPI != 1 || HALVES == 2, "the activation needs the gate half and the linear half of a tile");
    constexpr int HALF_W = 128 * XS_BK * 2, STAGE_W = HALVES * HALF_W, STAGE_X = NT * XS_BK * 2;
    constexpr int STAGES = xs_stages(NT, HALVES), ACC_COLS = HALVES * NT, TMEM_COLS = xs_tmem_cols(NT, HALVES);
    constexpr int TILE_N = HALVES * 128;
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
    long long* o_at = (long long*)(tmem_slot + 2);     // EPI 0: where a slot's row goes, and its weight
    float* o_weight = (float*)(o_at + NT);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = (args.N + TILE_N - 1) / TILE_N;
    const int k_tiles = (args.K + XS_BK - 1) / XS_BK;
    const int k_per = (k_tiles + args.splits - 1) / args.splits;
    const int per_tile = n_tiles * args.splits;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
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
    // Whoever comes next may start only when this kernel's predecessors are done: the product behind this one then finds
    // the lists complete and streams its weights without waiting for this one's results (lists_ready).
    if (!args.lists_ready) {
        pdl_wait();
        pdl_trigger();
    }
    // The row tiles are the fastest index: an expert's row tiles stand side by side in the list, so the blocks that read the
    // same part of its matrix do so at the same time.
    const int row_tiles = __ldcg(args.num_tiles), total = row_tiles * per_tile;
    struct Item { int group, slot0, n0, split, k_begin, k_end; };
    auto item_of = [&](int i) {
        Item x;
        const int tile = i % row_tiles, rest = i / row_tiles;
        x.group = __ldcg(args.tiles + 2 * tile);
        x.slot0 = __ldcg(args.tiles + 2 * tile + 1);
        x.split = rest % args.splits;
        x.n0 = rest / args.splits * TILE_N;
        x.k_begin = x.split * k_per;
        x.k_end = min(k_tiles, x.k_begin + k_per);
        return x;
    };

    if (warp == 0) {
        if (lane == 0) {
            // ------------------------------------------------ producer
            const uint32_t bytes = (uint32_t)(STAGE_W + STAGE_X);
            uint32_t stage = 0, phase = 0;
            bool first = true;
            // (a part of an expert's matrix is read once, or by blocks side by side: first to leave L2, so that the next launches' code and
            // lists stay.  Without and with it, us, 16 of 2,048 at 2,048: 8 rows 91.5 -> 84.2, 64 rows 129 -> 119, 1,000 rows 255 -> 248)
            uint64_t once;
            asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
            trace_point(TR_GROUPED_GEMM);
            for (int i = blockIdx.x; i < total && !*abort_flag; i += gridDim.x) {
                const Item x = item_of(i);
                const int row_w = x.group * args.N + x.n0;
                int kt = x.k_begin;
                if (first && args.lists_ready) {
                    // the first stages' weights while the predecessor (the rows' producer) may still be running
                    const int pre = min(STAGES, x.k_end - x.k_begin);
                    for (int s = 0; s < pre; ++s) {
                        mbar_expect_tx(&full[s], bytes);
                        tma_load_2d_hint(sw + s * STAGE_W, &map_w, (x.k_begin + s) * XS_BK, row_w, &full[s], once);
                    }
                    pdl_wait();
                    pdl_trigger();
                    for (int s = 0; s < pre; ++s) tma_load_2d(sx + s * STAGE_X, &map_x, (x.k_begin + s) * XS_BK, x.slot0, &full[s]);
                    kt = x.k_begin + pre;
                    if (pre == STAGES) phase = 1; else stage = pre;
                }
                first = false;
                for (; kt < x.k_end; ++kt) {
                    if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) break;
                    mbar_expect_tx(&full[stage], bytes);
                    tma_load_2d_hint(sw + stage * STAGE_W, &map_w, kt * XS_BK, row_w, &full[stage], once);
                    tma_load_2d(sx + stage * STAGE_X, &map_x, kt * XS_BK, x.slot0, &full[stage]);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------- MMA issuer: the warp runs together, an elected lane issues
        constexpr uint32_t idesc = umma_idesc(128, NT);
        const uint64_t dw0 = umma_desc(smem_u32(sw)), dx0 = umma_desc(smem_u32(sx));
        uint32_t stage = 0, phase = 0, it = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < total && ok && !*abort_flag; i += gridDim.x, ++it) {
            const int split = i / row_tiles % args.splits;
            const int k_begin = split * k_per, k_end = min(k_tiles, k_begin + k_per);
            const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
            ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[acc], acc_phase ^ 1, abort_flag));
            if (!ok) break;
            tc_fence_after();
            const uint32_t d = tmem_base + acc * ACC_COLS;
            for (int kt = k_begin; kt < k_end; ++kt) {
                if (!mbar_try_wait(&full[stage], phase)) ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, abort_flag));
                if (!ok) break;
                tc_fence_after();
                const uint64_t dw = dw0 + (uint64_t)(stage * (STAGE_W >> 4));
                const uint64_t dx = dx0 + (uint64_t)(stage * (STAGE_X >> 4));
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < XS_BK / 16; ++k)
#pragma unroll
                        for (int hf = 0; hf < HALVES; ++hf)
                            umma_bf16(d + hf * NT, dw + (uint64_t)(hf * (HALF_W >> 4)) + 2 * k, dx + 2 * k, idesc,
                                      (kt > k_begin || k > 0) ? 1u : 0u);
                    umma_commit(&empty[stage]);
                }
                __syncwarp();
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
            if (ok && elect_one()) umma_commit(&acc_full[acc]);
            __syncwarp();
        }
    } else {
        // ---------------------------------------------------- epilogue: warps 2..5, thread = feature, columns = slots
        pdl_wait();   // nothing is written before the predecessor has completed
        const int quarter = warp & 3, r = quarter * 32 + lane;
        uint32_t it = 0;
        // (EPI 0: the warps meet at a barrier, so all of them go through all tiles, also when a wait has run out)
        for (int i = blockIdx.x; i < total && (EPI == 0 || !*abort_flag); i += gridDim.x, ++it) {
            const Item x = item_of(i);
            const int rows = min(args.tile_rows, __ldcg(args.start + x.group + 1) - x.slot0);      // (up to NT: see air_expert_stream_tiles)
            const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
            if constexpr (EPI == 0) {
                // (worked out by a thread per slot while the products run, not row by row in the loop below)
                asm volatile("bar.sync 1, 128;" ::: "memory");      // (the last tile's are read)
                for (int t = threadIdx.x - 64; t < min(rows, NT); t += 128) {
                    const int dst = __ldcg(args.o_index + x.slot0 + t);
                    o_at[t] = (x.split * args.o_div + dst % args.o_div) * args.o_part_stride + (long long)(dst / args.o_div) * args.ldo;
                    o_weight[t] = args.o_scale ? args.o_scale[dst] : 1.f;
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
            }
            const bool ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[acc], acc_phase, abort_flag));
            if constexpr (EPI == 0) {
                if (!ok) continue;
            } else if (!ok) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + acc * ACC_COLS + ((uint32_t)(quarter * 32) << 16);
            // (16 slots at a time; a tile of an expert with few rows ends with them)
            for (int t0 = 0; t0 < min(rows, NT); t0 += 16) {
                if constexpr (EPI == 1) {
                    float gate[16], lin[16];
                    xs_load16(taddr + t0, gate);
                    xs_load16(taddr + NT + t0, lin);
                    __nv_bfloat16* out = (__nv_bfloat16*)args.out + (size_t)(x.slot0 + t0) * (args.N / 2) + x.n0 / 2 + r;
#pragma unroll
                    for (int t = 0; t < 16; ++t)
                        if (t0 + t < rows)
                            out[(size_t)t * (args.N / 2)] = __float2bfloat16_rn(
                                gated_activation(gate[t], lin[t], args.act_alpha, args.act_limit, args.act_shift));
                } else {
#pragma unroll
                    for (int hf = 0; hf < HALVES; ++hf) {
                        float v[16];
                        xs_load16(taddr + hf * NT + t0, v);
                        const int col = x.n0 + hf * 128 + r, live = col < args.N ? rows - t0 : 0;
                        if constexpr (EPI == 2) {
                            __nv_bfloat16* out = (__nv_bfloat16*)args.out + (size_t)(x.slot0 + t0) * args.N + col;
#pragma unroll
                            for (int t = 0; t < 16; ++t) {
                                const float y = fmaxf(v[t], 0.f);
                                if (t < live) out[(size_t)t * args.N] = __float2bfloat16_rn(y * y);
                            }
                        } else {
#pragma unroll
                            for (int t = 0; t < 16; ++t)
                                if (t < live) ((float*)args.out)[o_at[t0 + t] + col] = v[t] * o_weight[t0 + t];
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
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
}

template <int NT, int EPI, int HALVES>
static int xs_launch(const CUtensorMap& mw, const CUtensorMap& mx, const XsArgs& args, int blocks, cudaStream_t stream) {
    constexpr int STAGES = xs_stages(NT, HALVES);
    // (more than half of an SM's shared memory: two blocks never share an SM and its tensor memory)
    const size_t smem = 1024 + (size_t)STAGES * (HALVES * 128 + NT) * XS_BK * 2 + 16 * STAGES + 256 + (EPI == 0 ? 12 * NT : 0);
    const size_t request = smem < 120 * 1024 ? 120 * 1024 : smem;
    auto kernel = expert_stream_kernel<NT, EPI, HALVES>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)request);
    if (e != cudaSuccess) return (int)e;
    return launch(kernel, blocks, XS_THREADS, request, stream, mw, mx, args);
}

template <int NT>
static int xs_dispatch(int epi, const CUtensorMap& mw, const CUtensorMap& mx, const XsArgs& args, int blocks, cudaStream_t stream) {
    if (epi == 0) return xs_launch<NT, 0, 1>(mw, mx, args, blocks, stream);
    if (epi == 1) return xs_launch<NT, 1, 2>(mw, mx, args, blocks, stream);
    return xs_launch<NT, 2, 1>(mw, mx, args, blocks, stream);
}

}  // namespace air

// x [slots, K] bf16 in slot order, w [groups, N, K] bf16, K % 8 == 0.  start [groups + 1], tiles and num_tiles as
// moe_sort_kernel leaves them (tile_rows slots to a tile, 64 or 128); no expert has more than most_rows slots.  epi, out: see above (epi 1: N a
// multiple of 256).  lists_ready: the kernel launched right before this one is an expert_stream_kernel that was given the
// same lists without it.
AIR_API int air_expert_stream_tiles(const void* x, int slots, const void* w, int groups, int N, int K, const int* start,
                                    const int* tiles, const int* num_tiles, int max_tiles, int tile_rows, int most_rows, int epi,
                                    void* out, int splits, const int* o_index, int o_div, long long o_part_stride, int ldo,
                                    const float* o_scale, float alpha, float limit, float shift, int lists_ready, int* status,
                                    cudaStream_t stream) {
    using namespace air;
    if (slots <= 0 || N <= 0 || groups <= 0 || max_tiles <= 0) return 0;
    if (K <= 0 || K % 8 || epi < 0 || epi > 2 || splits < 1 || (splits > 1 && epi) || (epi == 1 && N % 256) || !start || !tiles ||
        !num_tiles || (epi == 0 && (!o_index || o_div < 1)) || ((uintptr_t)x & 15) || ((uintptr_t)w & 15) || most_rows < 1 ||
        (tile_rows != XS_ROWS && tile_rows != XS_WIDE) || (long long)groups * N > 0x7fffffff)
        return AIR_ERR_BAD_ARGUMENT;
    const int k_tiles = (K + XS_BK - 1) / XS_BK;
    if (splits > k_tiles || (long long)(splits - 1) * ((k_tiles + splits - 1) / splits) >= k_tiles) return AIR_ERR_BAD_ARGUMENT;
    const int nt = tile_rows == XS_WIDE ? XS_WIDE : most_rows > 32 ? 64 : most_rows > 16 ? 32 : 16;
    CUtensorMap mw, mx;
    int rc = tensor_map_2d(&mw, w, (long long)groups * N, K, epi == 1 ? 256 : 128);
    if (rc) return rc;
    rc = tensor_map_2d(&mx, x, slots, K, nt);
    if (rc) return rc;
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long most = (long long)max_tiles * ((N + (epi == 1 ? 255 : 127)) / (epi == 1 ? 256 : 128)) * splits;
    const int blocks = (int)(most < sms ? most : sms);
    const XsArgs args{out, slots, N, K, splits, start, tiles, tile_rows, num_tiles, lists_ready, o_index, o_div, o_part_stride, ldo, o_scale,
                      status, alpha, limit, shift};
    if (nt == 16) return xs_dispatch<16>(epi, mw, mx, args, blocks, stream);
    if (nt == 32) return xs_dispatch<32>(epi, mw, mx, args, blocks, stream);
    if (nt == 64) return xs_dispatch<64>(epi, mw, mx, args, blocks, stream);
    return xs_dispatch<XS_WIDE>(epi, mw, mx, args, blocks, stream);
}
// The same with 64 slots to a tile.
AIR_API int air_expert_stream(const void* x, int slots, const void* w, int groups, int N, int K, const int* start,
                              const int* tiles, const int* num_tiles, int max_tiles, int most_rows, int epi, void* out, int splits,
                              const int* o_index, int o_div, long long o_part_stride, int ldo, const float* o_scale, float alpha,
                              float limit, float shift, int lists_ready, int* status, cudaStream_t stream) {
    return air_expert_stream_tiles(x, slots, w, groups, N, K, start, tiles, num_tiles, max_tiles, air::XS_ROWS, most_rows, epi, out,
                                   splits, o_index, o_div, o_part_stride, ldo, o_scale, alpha, limit, shift, lists_ready, status, stream);
}

AIR_API int air_trace_set_expert_stream(unsigned long long* buffer) { return air::set_trace_here(buffer); }
