// Attention of single next tokens over a compressed latent (one row per token that every query head reads, its first dv numbers as the
// value too) on the fifth-generation tensor cores.  grouped_attention_tc_kernel (attention_grouped.cu) does the same with 16 heads to a
// block in mma.sync and stays for every other form (other row sizes, keys with values of their own, biases, 16-bit queries).
//
// What bounded that kernel were the instructions of a tile of 64 keys, 5 us; and with 16 heads to a block every key was fetched twice.  Here a
// block takes up to 32 heads, and both products have the KEYS' side, which is the long one, as the rows of tcgen05.mma:
//   S^T [64 keys, 2 HN] = K Q^T      HN heads: their queries' upper halves, then their lower halves (a float32 query is two bfloat16
//                                    numbers, hi + lo, as in the kernel above), both operands with d along the 128-byte rows
//   O^T [dv, 2 HN]     += V^T P      both operands read across their rows: V is the same tile of keys, P's rows are a key's weights, the
//                                    heads' upper halves and then their lower ones, so that the tile is read once for both
// block (token, up to HN heads, split): split s of S takes the tiles of 64 keys whose index is s modulo S.
//   warp 0      a tile's copies (d / 64 boxes, 128-byte swizzle) into one of two stages; asks for the tile after next in L2
//   warp 1      issues S of a tile or O's step of another, whichever has what it needs
//   warps 2, 3  zero the rows of a tile at the edge that the token does not see (they may hold anything)
//   warps 4-19  four to every quarter of the tensor memory's lanes.  Scores: a quarter's first 16 lanes hold 16 keys, a warp takes HN / 4
//               heads, half of them on the 16 lanes behind.  Weights against a reference maximum per head, which moves only where a score
//               exceeds it by more than 5 (a weight of 150 is as good in 32 bits and in two halves as one of 1); then, and with the first
//               tile, the heads' maxima are taken across the threads.  P to shared memory; O rescaled where the reference has moved,
//               and written at the end: part as grouped_attention_tc_kernel leaves it, for the same merge
// All sums are 32-bit.  Every wait on an mbarrier is bounded; on giving up the block sets *status = 5.
//
// What bounds it now: the way of a stage, 2 us a tile (its copy 1.3, S 0.8, weights 0.8, O's step 0.6, in turn; two stages of 74 KB beside
// the queries are what an SM holds), against 1.1 that an SM's copies of the tile take; and 9 us in front of the first and behind the last.
// Measured with the merge, rows of 576 (values 512), 32 heads, us, grouped_attention_tc_kernel and this one: 8 tokens over 100 keys 17.6 and 14.4,
// 1,000 23.8 and 16.4, 4,096 48.3 and 22.9 (its keys at the copy rate: 5.8), 8,000 74.6 and 32.4; 32 tokens over 4,096 149.9 and 55.1 (23); one
// over 8,191 48.3 and 22.9; 16 heads: 8 tokens over 4,096 36.0 and 19.7.  Shorter rows, 32 heads, 32 tokens over 4,000: of 128 (values 128) 65.5 and
// 31.7, 192 (128) 70.8 and 33.3, 256 (256) 80.0 and 37.7, 384 (256) 115 and 44, 512 (512) 131 and 50; 4 heads, 8 over 4,000, rows of 128 19.9 and 12.5; of
// 655 sizes only rows of 128 have slower ones, 8 tokens by up to 20 heads over few keys (10.7 and 11.6 the worst).  Scores in a thread per key (32 heads each, on two of four schedulers): 40.1
// instead of 22.9; rows to be zeroed one after the other by one warp: 29.5.
#include "common.cuh"
#include "umma.cuh"

namespace air {

constexpr int LA_GROUPS = 4;              // warps that share a quarter of the accumulators' lanes
constexpr int LA_THREADS = 32 * (4 + 4 * LA_GROUPS);
constexpr int LA_KT = 64;                  // keys of a tile
constexpr int LA_SUB = LA_KT * 128;        // bytes of a tile's 64 columns
constexpr int LA_MOST_D = 576, LA_MOST_DV = 512;
constexpr float LA_MOVE = 5.f;

struct LatentArgs {
    const float* q;               // [T, H, d]
    const int *block_table, *token_seq, *positions;
    float* part;                  // [T, H, splits, dv + 2]
    int max_blocks, H, d, dv, P, window, mask_mode, splits;
    float scale, softcap;
    int* status;
};

// v[0 .. N): of each the maximum (sum) over the lanes of this half of the warp, number l on its lane l (modulo N)
template <int N, bool SUM>
__device__ __forceinline__ float across(float (&v)[N], int lane) {
    auto both = [](float a, float b) { return SUM ? a + b : fmaxf(a, b); };
#pragma unroll
    for (int o = 8; o >= N; o >>= 1)
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = both(v[i], __shfl_xor_sync(0xffffffffu, v[i], o));
#pragma unroll
    for (int o = N / 2; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const bool upper = lane & o;
            const float mine = upper ? v[i + o] : v[i], other = upper ? v[i] : v[i + o];
            v[i] = both(mine, __shfl_xor_sync(0xffffffffu, other, o));
        }
    return v[0];
}
template <int N> __device__ __forceinline__ void tmem_columns(uint32_t at, float (&v)[N]) {
    static_assert(N == 4 || N == 8, "columns of a thread");
    uint32_t r[N];
    if constexpr (N == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(at) : "memory");
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __uint_as_float(r[i]);
}

// One look at a barrier's phase, without waiting in it.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}

template <int HN>
__global__ void __launch_bounds__(LA_THREADS, 1) latent_attention_kernel(const __grid_constant__ CUtensorMap map_cache, const LatentArgs a) {
    constexpr int QSUB = 2 * HN * 128;                       // bytes of the queries' 64 columns
    constexpr uint32_t S_COLS = 2 * HN, O_COL = 2 * S_COLS;  // tensor memory: S even, S odd, then O by 128 of dv
    constexpr uint32_t TMEM_COLS = 16 * HN;                  // (12 HN are used)
    constexpr int HG = HN / LA_GROUPS, NH = HG / 2, WIDTH = 32 * 4 * LA_GROUPS;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int subs = a.d / 64, stage_bytes = subs * LA_SUB;
    uint8_t* sq = smem;
    uint8_t* sk = sq + subs * QSUB;
    uint8_t* sp = sk + 2 * stage_bytes;                      // P: [hi, lo][HN heads][64 keys], 8 KB kept free
    uint64_t* kv_full = (uint64_t*)(sp + LA_SUB);
    uint64_t *kv_empty = kv_full + 2, *clean = kv_full + 4, *s_full = kv_full + 6, *p_ready = kv_full + 8, *pv_done = kv_full + 9;
    uint32_t* tmem_slot = (uint32_t*)(kv_full + 10);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    float* mref = (float*)(kv_full + 12);                    // [HN] reference maxima, then the factors of a move, then by warp
    float* corr = mref + HN;
    float* wide = corr + HN;                                 // [4][HN]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&kv_full[i], 1);
            mbar_init(&kv_empty[i], 3);                      // the products' end, and warps 2 and 3
            mbar_init(&clean[i], 2);
            mbar_init(&s_full[i], 1);
        }
        mbar_init(p_ready, 4 * LA_GROUPS);
        mbar_init(pv_done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < HN) mref[tid] = -INFINITY;
    if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_enter(TR_ATT_GROUPED);

    const int t = blockIdx.x, head0 = blockIdx.y * HN, nj = min(HN, a.H - head0), split = blockIdx.z;
    const int slot = a.token_seq[t], pos = a.positions[t];
    const int lo = a.window > 0 ? (a.mask_mode == 1 ? pos - pos % a.window : max(0, pos - a.window + 1)) : 0;
    const int* bt = a.block_table + (size_t)max(0, slot) * a.max_blocks;
    const int first = lo / LA_KT + split, n = slot < 0 || first > pos / LA_KT ? 0 : (pos / LA_KT - first) / a.splits + 1;
    auto key_of = [&](int j) { return (first + j * a.splits) * LA_KT; };
    auto edge = [&](int j) { return key_of(j) < lo || key_of(j) + LA_KT - 1 > pos; };
    // (an edge can be the first tile or the last; the last one's wait is its stage's second where both stand in one stage)
    auto edge_phase = [&](int j) { return (uint32_t)(j > 0 && !(j & 1) && edge(0)); };
    const int box_rows = min(a.P, LA_KT);
    auto bring = [&](int j) {                                // (one thread)
        const int stage = j & 1, key0 = key_of(j);
        int valid = 0;
        for (int r = 0; r < LA_KT; r += box_rows) valid += key0 + r <= pos && key0 + r + box_rows - 1 >= lo;
        mbar_expect_tx(&kv_full[stage], (uint32_t)(valid * box_rows * 128 * subs));
        for (int r = 0; r < LA_KT; r += box_rows) {
            const int key = key0 + r;
            if (key > pos || key + box_rows - 1 < lo) continue;
            const int row = bt[key / a.P] * a.P + key % a.P;
            for (int s = 0; s < subs; ++s)
                tma_load_2d(sk + stage * stage_bytes + s * LA_SUB + r * 128, &map_cache, 64 * s, row, &kv_full[stage]);
        }
        // (the tile that will take its place, into L2 meanwhile)
        for (int r = 0; j + 2 < n && r < LA_KT; r += box_rows) {
            const int key = key_of(j + 2) + r;
            if (key > pos) continue;
            const int row = bt[key / a.P] * a.P + key % a.P;
            for (int s = 0; s < subs; ++s) tma_prefetch_l2(&map_cache, 64 * s, row);
        }
    };
    if (tid == 0)
        for (int j = 0; j < min(2, n); ++j) bring(j);
    // the queries as two halves each, rows of 128 bytes with the same swizzle (warp 0 is at the copies meanwhile)
    if (n > 0 && warp > 0) {
        const float* from = a.q + ((size_t)t * a.H + head0) * a.d;
        constexpr int READERS = LA_THREADS / 32 - 1, ROUNDS = (HN + READERS - 1) / READERS, PIECES = (LA_MOST_D / 4 + 31) / 32;
        float v[ROUNDS][PIECES][4];
#pragma unroll
        for (int x = 0; x < ROUNDS; ++x)
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {               // (all of a thread's reads under way at once)
                const int h = warp - 1 + x * READERS, c = (lane + 32 * i) * 4;
                v[x][i][0] = v[x][i][1] = v[x][i][2] = v[x][i][3] = 0.f;
                if (h < nj && c < a.d) load4(from + (size_t)h * a.d + c, v[x][i]);
            }
#pragma unroll
        for (int x = 0; x < ROUNDS; ++x)
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                const int h = warp - 1 + x * READERS, c = (lane + 32 * i) * 4;
                if (h >= HN || c >= a.d) continue;
                uint32_t up[2], rest[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const __nv_bfloat162 b = __floats2bfloat162_rn(v[x][i][2 * e], v[x][i][2 * e + 1]);
                    const __nv_bfloat162 r = __floats2bfloat162_rn(v[x][i][2 * e] - __low2float(b), v[x][i][2 * e + 1] - __high2float(b));
                    up[e] = *reinterpret_cast<const uint32_t*>(&b);
                    rest[e] = *reinterpret_cast<const uint32_t*>(&r);
                }
                uint8_t* to = sq + (c / 64) * QSUB + h * 128 + (((c % 64 / 8) ^ (h & 7)) << 4) + (c & 4) * 2;
                *reinterpret_cast<uint2*>(to) = make_uint2(up[0], up[1]);
                *reinterpret_cast<uint2*>(to + HN * 128) = make_uint2(rest[0], rest[1]);      // (HN is a multiple of 8: the same swizzle)
            }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("bar.sync 2, %0;" ::"n"(LA_THREADS - 32) : "memory");
    }

    if (warp == 0) {
        if (lane == 0)
            for (int j = 2; j < n; ++j) {
                if (!mbar_wait(&kv_empty[j & 1], ((j >> 1) - 1) & 1, abort_flag)) break;
                bring(j);
            }
    } else if (warp == 1) {
        constexpr uint32_t idesc_s = umma_idesc(LA_KT, 2 * HN), idesc_o = umma_idesc(128, 2 * HN, true) | (1u << 15);   // (both across their rows)
        const uint32_t q_at = smem_u32(sq), k_at = smem_u32(sk), p_at = smem_u32(sp);
        // S of tile js, O's step jp: whichever has what it needs.  (S(js) overwrites S(js - 2), whose weights are there once js <= jp + 1.)
        int js = 0, jp = 0;
        for (uint32_t tries = 0; jp < n;) {
            if (js < n && js <= jp + 1 && __all_sync(0xffffffffu, mbar_test(&kv_full[js & 1], (js >> 1) & 1) &&
                                                                      (!edge(js) || mbar_test(&clean[js & 1], edge_phase(js))))) {
                tc_fence_after();
                if (elect_one()) {
                    for (int s = 0; s < subs; ++s) {
                        const uint64_t dk = umma_desc(k_at + (js & 1) * stage_bytes + s * LA_SUB), dq = umma_desc(q_at + s * QSUB);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_bf16(tmem_base + (js & 1) * S_COLS, dk + 2 * k, dq + 2 * k, idesc_s, s > 0 || k > 0 ? 1u : 0u);
                    }
                    umma_commit(&s_full[js & 1]);
                }
                __syncwarp();
                ++js;
                tries = 0;
            } else if (jp < js && __all_sync(0xffffffffu, mbar_test(p_ready, jp & 1))) {
                tc_fence_after();
                const uint32_t v_at = k_at + (jp & 1) * stage_bytes;
                if (elect_one()) {
                    for (int m = 0; m < a.dv / 128; ++m)
#pragma unroll
                        for (int k = 0; k < LA_KT / 16; ++k)
                            umma_bf16(tmem_base + O_COL + m * 2 * HN, umma_desc_mn(v_at + 2 * m * LA_SUB + k * 16 * 128, LA_SUB),
                                      umma_desc_mn(p_at + k * 16 * 128, LA_SUB), idesc_o, jp > 0 || k > 0 ? 1u : 0u);
                    umma_commit(pv_done);
                    umma_commit(&kv_empty[jp & 1]);
                }
                __syncwarp();
                ++jp;
                tries = 0;
            } else if (__any_sync(0xffffffffu, ++tries > 16 * SPIN_LIMIT || ((tries & 1023u) == 1023u && *abort_flag))) {
                *abort_flag = 1;
                break;
            }
        }
    } else if (warp < 4) {
        for (int j = 0; j < n; ++j) {
            // (they look at every tile, and a stage is not filled again before they have: a wait by parity cannot tell a phase from the
            // one two later)
            const int stage = j & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(&kv_full[stage], (j >> 1) & 1, abort_flag))) break;
            if (edge(j)) {
                // the rows ahead of the first key that is seen, and those behind the last one: 16-byte pieces one after the other
                const int ahead = 8 * max(0, min(LA_KT, lo - key_of(j))), behind = 8 * max(0, min(LA_KT, pos + 1 - key_of(j)));
                for (int s = warp - 2; s < subs; s += 2) {
                    uint4* to = reinterpret_cast<uint4*>(sk + stage * stage_bytes + s * LA_SUB);
                    for (int c = lane; c < ahead; c += 32) to[c] = make_uint4(0, 0, 0, 0);
#pragma unroll 4
                    for (int c = behind + lane; c < 8 * LA_KT; c += 32) to[c] = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            __syncwarp();
            if (lane == 0) {
                if (edge(j)) mbar_arrive(&clean[stage]);
                mbar_arrive(&kv_empty[stage]);
            }
        }
    } else if (warp >= 4) {
        const int quarter = warp & 3, group = (warp - 4) >> 2, h0 = group * HG;
        const uint32_t lane_at = tmem_base + ((uint32_t)(quarter * 32) << 16);
        // A quarter's first 16 lanes hold 16 keys of the tile (an instruction of 64 rows); the lanes behind them take half of their heads.
        const int row = 16 * quarter + (lane & 15), h1 = h0 + (lane >> 4) * NH;
        uint8_t* const p_to = sp + row * 128 + (h1 & 7) * 2;
        const int p_hi = ((h1 >> 3) ^ (row & 7)) << 4, p_low = (((HN + h1) >> 3) ^ (row & 7)) << 4;
        float sum[NH];
#pragma unroll
        for (int h = 0; h < NH; ++h) sum[h] = 0.f;
        // group g's part of O: numbers 128 g + row of the values, every head's upper and lower sums
        const uint32_t o_at = lane_at + O_COL + group * 2 * HN;
        const bool holder = group < a.dv / 128;
        // A thread that has given up a wait goes on without waiting, and its warp together: nobody is left at a barrier.  (A vote of the
        // warp on every wait instead: 1 to 4 % of the whole.)
        bool ok = true;
        for (int j = 0; j < n; ++j) {
            if (ok) ok = mbar_wait(&s_full[j & 1], (j >> 1) & 1, abort_flag);
            __syncwarp();
            tc_fence_after();
            float s[NH];
            bool over = false;
            {
                float c[HG], low[HG];
                tmem_columns(lane_at + (j & 1) * S_COLS + h0, c);
                tmem_columns(lane_at + (j & 1) * S_COLS + HN + h0, low);
                const int key = key_of(j) + row;
                const bool seen = key >= lo && key <= pos;
#pragma unroll
                for (int h = 0; h < HG; ++h) c[h] += low[h];
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    const float other = __shfl_sync(0xffffffffu, c[NH + h], lane & 15);
                    s[h] = (lane < 16 ? c[h] : other) * a.scale;
                }
                if (a.softcap > 0.f)
#pragma unroll
                    for (int h = 0; h < NH; ++h) s[h] = a.softcap * tanhf(s[h] / a.softcap);
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    s[h] = seen ? s[h] : -INFINITY;
                    over |= s[h] > mref[h1 + h] + LA_MOVE;
                }
            }
            tc_fence_before();
            int any;
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, %2, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
                         : "=r"(any) : "r"((int)over), "n"(WIDTH) : "memory");
            if (any) {
                float v[NH];
#pragma unroll
                for (int h = 0; h < NH; ++h) v[h] = s[h];
                const float most = across<NH, false>(v, lane);
                if ((lane & 15) < NH) wide[quarter * HN + h1 + (lane & 15)] = most;
                asm volatile("bar.sync 1, %0;" ::"n"(WIDTH) : "memory");
                if (warp == 4 && lane < HN) {
                    const float before = mref[lane], now = fmaxf(before, fmaxf(fmaxf(wide[lane], wide[HN + lane]), fmaxf(wide[2 * HN + lane], wide[3 * HN + lane])));
                    corr[lane] = now == before ? 1.f : expf(before - now);      // (0 when there was none)
                    mref[lane] = now;
                }
                asm volatile("bar.sync 1, %0;" ::"n"(WIDTH) : "memory");
#pragma unroll
                for (int h = 0; h < NH; ++h) sum[h] *= corr[h1 + h];
            }
            // O's step j - 1 has ended: P may be written again, and O rescaled
            if (j > 0 && ok) ok = mbar_wait(pv_done, (j - 1) & 1, abort_flag);
            if (any && j > 0 && holder) {
                __syncwarp();
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < 2 * HN; c += 16) {
                    uint32_t o[16];
                    tmem_ld16(o_at + c, o);
#pragma unroll
                    for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * corr[(c + e) % HN]);
                    tmem_st16(o_at + c, o);
                }
            }
            uint32_t hi[NH / 2], low[NH / 2];
#pragma unroll
            for (int h = 0; h < NH; h += 2) {
                float p[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float m = mref[h1 + h + e];
                    p[e] = m == -INFINITY ? 0.f : expf(s[h + e] - m);
                    sum[h + e] += p[e];
                }
                const __nv_bfloat162 up = __floats2bfloat162_rn(p[0], p[1]);
                const __nv_bfloat162 rest = __floats2bfloat162_rn(p[0] - __low2float(up), p[1] - __high2float(up));
                hi[h / 2] = *reinterpret_cast<const uint32_t*>(&up);
                low[h / 2] = *reinterpret_cast<const uint32_t*>(&rest);
            }
            if constexpr (NH == 4) {
                *reinterpret_cast<uint2*>(p_to + p_hi) = make_uint2(hi[0], hi[1]);
                *reinterpret_cast<uint2*>(p_to + p_low) = make_uint2(low[0], low[1]);
            } else {
                *reinterpret_cast<uint32_t*>(p_to + p_hi) = hi[0];
                *reinterpret_cast<uint32_t*>(p_to + p_low) = low[0];
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_ready);
        }
        ok = __all_sync(0xffffffffu, ok && (n == 0 || mbar_wait(pv_done, (n - 1) & 1, abort_flag)));
        const float total = across<NH, true>(sum, lane);
        if ((lane & 15) < NH) wide[quarter * HN + h1 + (lane & 15)] = total;
        asm volatile("bar.sync 1, %0;" ::"n"(WIDTH) : "memory");
        float* const part = a.part + (((size_t)t * a.H + head0) * a.splits + split) * (a.dv + 2);
        const size_t head_stride = (size_t)a.splits * (a.dv + 2);
        if (slot >= 0 && warp == 4 && lane < nj) {
            part[lane * head_stride + a.dv] = mref[lane];
            part[lane * head_stride + a.dv + 1] = (wide[lane] + wide[HN + lane]) + (wide[2 * HN + lane] + wide[3 * HN + lane]);
        }
        if (n > 0 && ok && holder) {
            tc_fence_after();
            float* to = part + group * 128 + quarter * 32 + lane;
#pragma unroll
            for (int c = 0; c < HN; c += 16) {
                uint32_t o[16], low[16];
                tmem_ld16(o_at + c, o);
                tmem_ld16(o_at + HN + c, low);
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (c + e < nj) to[(c + e) * head_stride] = __uint_as_float(o[e]) + __uint_as_float(low[e]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 32; ++i) __nanosleep(2000);      // copies on their way may still land
        if (tid == 0 && a.status) atomicExch(a.status, 5);
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

template <int HN>
static int launch_latent(const CUtensorMap& map, const LatentArgs& a, int T, cudaStream_t stream) {
    const size_t smem = 1024 + (size_t)(a.d / 64) * (2 * HN * 128 + 2 * LA_SUB) + LA_SUB + 12 * 8 + 6 * HN * sizeof(float);
    auto kernel = latent_attention_kernel<HN>;
    // (never less than half of an SM's memory: one block to an SM, and to its tensor memory)
    const size_t request = smem < 120 * 1024 ? 120 * 1024 : smem;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)request);
    if (e != cudaSuccess) return (int)e;
    return launch(kernel, dim3(T, (a.H + HN - 1) / HN, a.splits), LA_THREADS, request, stream, map, a);
}

}  // namespace air

// The merge of the splits (attention_grouped.cu).
extern "C" int air_grouped_combine(const float* part, const int* token_seq, const float* sink, void* out, int T, int H, int dv, int splits,
                                   const float* gate, int ldg, const double* turn_freq, int turn_rot, int turn_pairing,
                                   const int* positions, cudaStream_t stream);

// As air_grouped_attention with latent rows, for float32 q [T, H, d] (d a multiple of 64 up to 576, on a 16-byte boundary) over a bfloat16
// cache [pages, P, d] (P a divisor or a multiple of 64, at least 8) whose first dv numbers (a multiple of 128 up to 512) are the values.
AIR_API int air_latent_attention(const float* q, const void* cache, long long pages, const int* block_table, int max_blocks,
                                 const int* token_seq, const int* positions, float* part, void* out, int T, int H, int d, int dv, int P,
                                 int window, float scale, int mask_mode, const float* sink, int splits, float softcap,
                                 const float* gate, int ldg, const double* turn_freq, int turn_rot, int turn_pairing, int* status,
                                 cudaStream_t stream) {
    using namespace air;
    if (T <= 0) return 0;
    if (H <= 0 || d <= 0 || d % 64 || d > LA_MOST_D || dv <= 0 || dv % 128 || dv > LA_MOST_DV || dv > d || P < 8 ||
        (P < LA_KT ? LA_KT % P : P % LA_KT) || splits < 1 || splits > 65535 || mask_mode < 0 || mask_mode > 1 || !part || pages <= 0 ||
        pages * P > 0x7fffffffll || (((uintptr_t)q | (uintptr_t)cache) & 15) ||
        (turn_freq && (turn_rot < 0 || turn_rot > dv || (turn_rot & 1) || turn_pairing < 0 || turn_pairing > 1)))
        return AIR_ERR_BAD_ARGUMENT;
    CUtensorMap map;
    int rc = tensor_map_2d(&map, cache, pages * P, d, P < LA_KT ? P : LA_KT);
    if (rc) return rc;
    const LatentArgs a{q, block_table, token_seq, positions, part, max_blocks, H, d, dv, P, window, mask_mode, splits, scale, softcap, status};
    rc = H <= 16 ? launch_latent<16>(map, a, T, stream) : launch_latent<32>(map, a, T, stream);
    if (rc) return rc;
    return air_grouped_combine(part, token_seq, sink, out, T, H, dv, splits, gate, ldg, turn_freq, turn_rot, turn_pairing, positions, stream);
}

AIR_API int air_trace_set_attention_latent(unsigned long long* buffer) { return air::set_trace_here(buffer); }
