// Attention of single next tokens in 32-bit arithmetic, the query heads that share a key/value head together: the sums of
// paged_attention_f32_kernel (attention_ref.cu) for a row by itself, in the same order, bit for bit.
//
// There a block takes a head of a token, its four warps a quarter of the blocks of 32 keys each (block b is warp b modulo 4's: a chain of
// running maximum, sum and weighted values), and the four partial results are merged.  What bounded it: every head of a group read the
// group's keys and values anew, with two blocks of keys in flight.
// Here the four chains are the four blocks of a cluster, and a block takes up to eight heads of a group through its quarter of the
// keys: a warp per head, all of which read the same rows from a ring that two more fill, as far ahead as memory holds.  At the end each
// block merges a quarter of the heads, whose chains the others have written into its shared memory, in the order of the chains.
// What bounds it now: a warp's own chain through 32 keys (a sum over d for the score, the exponentials, 32 sums for the values), 0.9 us,
// and the reads of shared memory by the warps of a block (1.4 us per 32 keys with seven heads).  So a block has fewer heads where SMs
// would be idle, and heads of 128 add up the next 32 keys' scores between the steps of this block's weights and values, whose numbers
// are asked for a step ahead (2,000 keys, 7 heads to a block: 35 us without, 30 with).
//
// q, out: [T, H, d]; cache, block_table, token_seq, positions, window, mask_mode, softcap, sink, gate, bias as in attention_ref.cu.
// Every wait on an mbarrier is bounded; on giving up the block sets *status = 5.
//
// Measured, us, that kernel -> this one (28 heads of 128 in groups of seven): 4 requests over 40 keys 6.1 -> 5.8, over 1,000 26 -> 14.0; 8 over
// 1,000 39 -> 17.9; 64 over 40 36 -> 19.0, over 1,000 288 -> 104; one over 2,000 48 -> 20.6, over 8,000 181 -> 66.  16 heads in groups of four: 64 over
// 1,000 200 -> 86.  16 heads of 64 in pairs: 8 over 1,000 30 -> 15.8, 64 over 100 34 -> 22.  Up to eight requests over 5 to 100 keys differ by
// no more than 0.4, but for 40 and 48 heads in groups of five and six, 6 over 40: 6.6 -> 7.4 and 7.7.  32 heads of 128 in pairs, 64 over 100: 52 -> 60.
// (With blocks that stay although their chain has no keys: 64 over 40, 28 heads 25.7; 40 heads in groups of five 45 instead of 30.)
#include "common.cuh"
#include "tma.cuh"

#include <cooperative_groups.h>
#include <type_traits>

namespace air {

constexpr int FS_CHAINS = 4, FS_HEADS = 8, FS_THREADS = (FS_HEADS + 2) * 32, FS_MOST_STAGES = 6, FS_D = 128;

struct SingleArgs {
    const float* q; const float* cache; const int* block_table; int max_blocks; const int* token_seq; const int* positions;
    float* out; const float* gate; int H, K, d, dv, P, window; float scale, softcap; int mask_mode; const float* sink;
    DistanceBias bias;
    int heads, stages, leave;     // heads of a block, places of the ring, whether blocks without keys leave
    int* status;
};
// Shared memory, in floats: the heads' queries, their weights of a block of keys, per stage 32 keys (rows of d + 4) and 32 values, then the
// results of the heads that this block merges (a share of them, a place for every chain: up to three more than heads).
struct SinglePlaces {
    int d, dv;
    __host__ __device__ int stage() const { return 32 * (d + 4) + 32 * dv; }
    __host__ __device__ int weights() const { return FS_HEADS * d; }
    __host__ __device__ int ring() const { return weights() + FS_HEADS * 32; }
    __host__ __device__ int results(int stages) const { return ring() + stages * stage(); }
    __host__ __device__ size_t bytes(int heads, int stages) const {
        return sizeof(float) * (size_t)(results(stages) + (heads + FS_CHAINS - 1) * (dv + 4));
    }
};

// A warp per head of the block, and two that bring.  D: the size of keys and values where it is known, else 0.
template <int D>
__global__ void __launch_bounds__(FS_THREADS, 2) attention_f32_single_kernel(const SingleArgs a) {
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(8) uint64_t full[FS_MOST_STAGES], empty[FS_MOST_STAGES];
    __shared__ int gave_up;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, d = D ? D : a.d, dv = D ? D : a.dv;
    const SinglePlaces places{d, dv};
    const int chain = blockIdx.x, t = blockIdx.z;
    const int G = a.H / a.K, per_group = (G + a.heads - 1) / a.heads;
    const int kvh = blockIdx.y / per_group, h0 = kvh * G + blockIdx.y % per_group * a.heads, nh = min(a.heads, (kvh + 1) * G - h0);
    if (tid == 0) {
        for (int i = 0; i < FS_MOST_STAGES; ++i) {
            mbar_init(&full[i], 64);                             // (every lane of the two that bring)
            mbar_init(&empty[i], nh);                             // (the warps that have a head)
        }
        gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_enter(TR_ATT_REF);
    const int seq = a.token_seq[t];
    if (seq < 0) return;                         // padding: the same for the whole cluster
    const int pos = a.positions[t];
    const int lo = a.window > 0 ? (a.mask_mode == 1 ? pos - pos % a.window : max(0, pos - a.window + 1)) : 0;
    const int base = (lo / 32 / FS_CHAINS) * FS_CHAINS, first = base + chain;
    // Where blocks wait for SMs, one whose chain has no keys leaves (the cluster's barriers wait for those that have not left): the others
    // merge without it, and nobody writes into its memory.
    if (a.leave && chain > pos / 32 - base) return;
    const int n = first * 32 > pos ? 0 : (pos / 32 - first) / FS_CHAINS + 1;
    float* ring = smem + places.ring();
    float m = -INFINITY, l = 0.f, acc[4] = {};   // of this warp's head: lane x holds numbers 4x..4x+3 of its weighted values
    cluster.barrier_arrive();
    if (warp >= a.heads) {
        // one warp brings the keys, one the values: a row per instruction, sixteen bytes a lane (a copy of the copy engine per row was 37 ns,
        // 2.4 us for 32 keys and values whatever their size); lane j knows where key j's row lies
        const bool values = warp > a.heads;
        const int* bt = a.block_table + (size_t)seq * a.max_blocks;
        const size_t page_stride = (size_t)a.K * a.P * (d + dv), offset = values ? (size_t)a.K * a.P * d : 0;
        const int width = values ? dv : d, ld = values ? dv : d + 4;
        const bool whole = a.P % 32 == 0;        // (32 keys of one page: rows one behind the other)
        auto page_of = [&](int i) {
            const int key = (first + i * FS_CHAINS) * 32 + (whole ? 0 : lane);
            return i < n && key + (whole ? 31 : 0) >= lo && key <= pos ? make_int2(bt[key / a.P], key % a.P) : make_int2(-1, 0);
        };
        int2 next = page_of(0);
        for (int i = 0, stage = 0, phase = 1; i < n; ++i) {
            const int2 page = next;
            next = page_of(i + 1);
            if (i >= a.stages && !__all_sync(0xffffffffu, mbar_wait(&empty[stage], phase, &gave_up))) break;
            const float* from = a.cache + ((size_t)max(page.x, 0) * page_stride + offset + ((size_t)kvh * a.P + page.y) * width);
            const uint32_t to = smem_u32(ring + stage * places.stage() + (values ? 32 * (d + 4) : 0) + lane * 4);
            if (whole) {
                const int key0 = (first + i * FS_CHAINS) * 32, j0 = max(0, lo - key0), j1 = min(32, pos + 1 - key0);
                if (lane * 4 < width)
#pragma unroll 8
                    for (int j = j0; j < j1; ++j)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + j * ld * 4), "l"(from + j * width + lane * 4)
                                     : "memory");
            } else {
                const long long at = page.x < 0 ? -1 : from - a.cache;
#pragma unroll 8
                for (int j = 0; j < 32; ++j) {
                    const long long row = __shfl_sync(0xffffffffu, at, j);        // (-1: not seen, not brought and not used)
                    if (row >= 0 && lane * 4 < width)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + j * ld * 4), "l"(a.cache + row + lane * 4)
                                     : "memory");
                }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[stage])) : "memory");
            if (++stage == a.stages) {
                stage = 0;
                phase ^= 1;
            }
        }
    } else if (warp < nh) {
        const int h = h0 + warp;
        float* sq = smem + warp * d;
        float* sp = smem + places.weights() + warp * 32;
        for (int x = lane; x < d; x += 32) sq[x] = a.q[((size_t)t * a.H + h) * d + x];
        __syncwarp();
        // sixteen more numbers of this lane's key, and four more keys' values: asked for a step before they are used
        struct Keys { float k[4][4], q[4][4]; };
        struct Values { float p[4], v[4][4]; };
        auto ask_keys = [&](Keys& r, const float* sk, int x) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                load4(sk + lane * (d + 4) + x + 4 * e, r.k[e]);
                load4(sq + x + 4 * e, r.q[e]);
            }
        };
        auto add_keys = [&](const Keys& r, float& s, int from, int to) {
#pragma unroll
            for (int e = from; e < to; ++e)
#pragma unroll
                for (int c = 0; c < 4; ++c) s = fmaf(r.q[e][c], r.k[e][c], s);
        };
        auto ask_values = [&](Values& r, const float* sv, int y) {
            load4(sp + y, r.p);
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (D == FS_D || lane * 4 < dv) load4(sv + (y + e) * dv + lane * 4, r.v[e]);
        };
        auto add_values = [&](const Values& r) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    // (a key of weight 0, unseen ones among them, may hold anything; chosen, not jumped over: no read waits for it)
                    const float more = fmaf(r.p[e], r.v[e][c], acc[c]);
                    acc[c] = r.p[e] != 0.f ? more : acc[c];
                }
        };
        auto score = [&](const float* sk, int x, float& s) {         // four more numbers of this lane's key
            float k[4], q[4];
            load4(sk + lane * (d + 4) + x, k);
            load4(sq + x, q);
#pragma unroll
            for (int e = 0; e < 4; ++e) s = fmaf(q[e], k[e], s);
        };
        // Block j: its weights and values from its scores; merged: and the next block's scores, a chain of d sums, between the steps.
        float s = 0.f;
        const float *here = ring, *there = ring;
        auto block = [&](int j, auto merged) {
            constexpr bool M = decltype(merged)::value;
            const float* sv = here + 32 * (d + 4);
            const float* sk = there;
            const int key = (first + j * FS_CHAINS) * 32 + lane;
            const bool valid = key >= lo && key <= pos;
            float x = s * a.scale;
            if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
            x += valid ? distance_bias(a.bias, h, pos - key) : 0.f;
            x = valid ? x : -INFINITY;
            s = 0.f;
            Keys keys[2];
            if constexpr (M) {
                ask_keys(keys[0], sk, 0);
                ask_keys(keys[1], sk, 16);
            }
            float bm = x;
#pragma unroll
            for (int o = 16, i = 0; o > 0; o >>= 1, ++i) {
                const float other = __shfl_xor_sync(0xffffffffu, bm, o);
                if constexpr (M)
                    if (i < 4) add_keys(keys[0], s, i, i + 1);
                bm = fmaxf(bm, other);
            }
            float p = 0.f, corr = 1.f;
            if (bm != -INFINITY) {               // (else the whole block is outside the window)
                const float m_new = fmaxf(m, bm);
                corr = expf(m - m_new);          // 0 when m was -inf
                p = valid ? expf(x - m_new) : 0.f;
                m = m_new;
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[c] *= corr;
            }
            sp[lane] = p;
            __syncwarp();
            Values values[2];
            ask_values(values[0], sv, 0);
            if constexpr (M) ask_keys(keys[0], sk, 32);
#pragma unroll
            for (int o = 16, i = 0; o > 0; o >>= 1, ++i) {
                const float other = __shfl_xor_sync(0xffffffffu, p, o);
                if constexpr (M)
                    if (i < 4) add_keys(keys[1], s, i, i + 1);
                p += other;
            }
            l = fmaf(l, corr, p);                // (1 and 0 where the block is outside)
            if constexpr (M) ask_keys(keys[1], sk, 48);
#pragma unroll
            for (int y = 0; y < 8; ++y) {
                if (y < 7) ask_values(values[(y + 1) % 2], sv, 4 * y + 4);
                if constexpr (M)
                    if (y < 6) add_keys(keys[y % 2], s, 0, 4);
                if constexpr (M)
                    if (y < 4) ask_keys(keys[y % 2], sk, 16 * (y + 4));
                add_values(values[y % 2]);
            }
        };
        bool ok = n == 0 || __all_sync(0xffffffffu, mbar_wait(&full[0], 0, &gave_up));
        if (n > 0 && ok)
#pragma unroll 8
            for (int x = 0; x < d; x += 4) score(here, x, s);
        for (int j = 0, stage = 0, phase = 0; j < n && ok; ++j) {
            uint64_t* const done = &empty[stage];
            const bool more = j + 1 < n;
            if (++stage == a.stages) {
                stage = 0;
                phase ^= 1;
            }
            there = stage ? here + places.stage() : ring;
            if (more) ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, &gave_up));
            if (D == FS_D && more)
                block(j, std::true_type{});
            else {
                block(j, std::false_type{});
                if (more && ok)
#pragma unroll 8
                    for (int x = 0; x < d; x += 4) score(there, x, s);
            }
            __syncwarp();                        // (also: the weights have been read)
            if (lane == 0) mbar_arrive(done);
            here = there;
        }
    }
    cluster.barrier_wait();                      // (all that stay have begun: their memory may be written)
    const int chains = a.leave ? min(FS_CHAINS, pos / 32 - lo / 32 / FS_CHAINS * FS_CHAINS + 1) : FS_CHAINS;
    if (warp < nh) {
        float* results = cluster.map_shared_rank(smem + places.results(a.stages), warp % chains) + (warp / chains * chains + chain) * (dv + 4);
        if (lane * 4 < dv) *(float4*)(results + lane * 4) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        if (lane == 0) {
            results[dv] = m;
            results[dv + 1] = l;
        }
    }
    cluster.sync();                              // (from here on each reads its own memory only)
    for (int x = tid; x < (nh - chain + chains - 1) / chains * dv; x += (int)blockDim.x) {
        const int i = x / dv, c = x % dv, h = h0 + i * chains + chain;
        const float* from = smem + places.results(a.stages) + i * chains * (dv + 4);
        float mm = a.sink ? a.sink[h] : -INFINITY, mw[FS_CHAINS], lw[FS_CHAINS], aw[FS_CHAINS];
#pragma unroll
        for (int w = 0; w < FS_CHAINS; ++w) {
            const float* head = from + w * (dv + 4);
            mw[w] = w < chains ? head[dv] : -INFINITY;
            lw[w] = w < chains ? head[dv + 1] : 0.f;
            aw[w] = w < chains ? head[c] : 0.f;
        }
#pragma unroll
        for (int w = 0; w < FS_CHAINS; ++w) mm = fmaxf(mm, mw[w]);
        float total = a.sink ? expf(a.sink[h] - mm) : 0.f, o = 0.f;
#pragma unroll
        for (int w = 0; w < FS_CHAINS; ++w) {
            const float weight = mw[w] == -INFINITY ? 0.f : expf(mw[w] - mm);
            total += lw[w] * weight;
            o += aw[w] * weight;
        }
        const float inv = (a.gate ? a.gate[(size_t)t * a.H + h] : 1.f) / total;
        a.out[((size_t)t * a.H + h) * dv + c] = o * inv;
    }
    if (gave_up) {
        for (int i = 0; i < 32; ++i) __nanosleep(2000);      // copies on their way may still land
        if (tid == 0 && a.status) atomicExch(a.status, 5);
    }
}

}  // namespace air

// A head to a block, for any batch (attention_ref.cu).
extern "C" int air_paged_attention_ref(const void* q, int q_f32, const void* cache, int dtype, const int* block_table, int max_blocks,
                                       const int* token_seq, const int* positions, void* out, const float* gate, int T, int H, int K, int d,
                                       int dv, int P, int window, float scale, float softcap, int mask_mode, const float* sink, int latent,
                                       const float* bias, int bias_n, cudaStream_t stream);

// Every row of the batch as a token by itself, for a float32 cache [page, K, P, d] keys then [K, P, dv] values on a 16-byte boundary, d and dv
// multiples of 4 up to 128, H a multiple of K.
AIR_API int air_attention_f32_single(const float* q, const float* cache, const int* block_table, int max_blocks, const int* token_seq,
                                     const int* positions, float* out, const float* gate, int T, int H, int K, int d, int dv, int P,
                                     int window, float scale, float softcap, int mask_mode, const float* sink, const float* bias,
                                     int bias_n, int* status, cudaStream_t stream) {
    using namespace air;
    if (T <= 0) return 0;
    if (d <= 0 || d > FS_D || d % 4 || dv <= 0 || dv > FS_D || dv % 4 || H <= 0 || K <= 0 || H % K || P <= 0 || H > 65535 || T > 65535 ||
        mask_mode < 0 || mask_mode > 1 || ((uintptr_t)cache & 15) || (bias && bias_n < 1))
        return AIR_ERR_BAD_ARGUMENT;
    const int G = H / K;
    SingleArgs a{q, cache, block_table, max_blocks, token_seq, positions, out, gate, H, K, d, dv, P, window, scale, softcap, mask_mode, sink,
                 DistanceBias{bias, bias_n}, 0, 0, 0, status};
    // As even shares of a group's heads as blocks of up to eight allow; fewer heads to a block where SMs would be idle (one request over
    // 2,000 keys, 28 heads in groups of seven: 29.7 us with seven to a block, 21.2 with one).
    const int idle = (int)max(1ll, min((long long)G, 128ll / ((long long)FS_CHAINS * K * T)));
    const int most = max((G + FS_HEADS - 1) / FS_HEADS, idle);
    a.heads = (G + most - 1) / most;
    const int shares = (G + a.heads - 1) / a.heads;
    const SinglePlaces places{d, dv};
    // Blocks that all find an SM look far ahead; beyond, as many share one as there are, as registers, five warps to a scheduler, allow and as
    // two places of each find room (512 blocks of 1,000 keys, 16 heads of 64 in pairs: 32 us with three to an SM, 20 with four; 1,024 of 2,000
    // keys, seven heads: 238 with room for three of which registers let two in, 191 with room for two).
    const long long blocks = (long long)FS_CHAINS * K * shares * T;
    const int fit = (int)min((long long)min(4, 20 / (a.heads + 2)), 227 * 1024ll / (long long)(places.bytes(a.heads, 2) + 1280));
    // (heads in pairs gain little by reading keys once: not a second round of the SMs for a few blocks.  16 pairs of 128, 8 requests, 512
    // blocks where 444 fit, over 100 and 1,000 keys: 11.9 and 48 us, one head to a block 8.3 and 42; 24 requests 23 and 28, here and there)
    if (G == 2 && fit < 4 && blocks > 148ll * fit && 2 * blocks < 3 * 148ll * fit)
        return air_paged_attention_ref(q, 1, cache, AIR_F32, block_table, max_blocks, token_seq, positions, out, gate, T, H, K, d, dv, P, window,
                                       scale, softcap, mask_mode, sink, 0, bias, bias_n, stream);
    const int resident = (int)min((blocks + 147) / 148, (long long)fit);
    a.leave = blocks > 148ll * resident;
    const size_t room = (resident == 1 ? 200 : 226 / resident - 1) * 1024;
    a.stages = FS_MOST_STAGES;
    while (a.stages > 2 && places.bytes(a.heads, a.stages) > room) --a.stages;
    const size_t smem = places.bytes(a.heads, a.stages);
    auto kernel = d == FS_D && dv == FS_D ? attention_f32_single_kernel<FS_D> : attention_f32_single_kernel<0>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(FS_CHAINS, K * shares, T);
    cfg.blockDim = dim3((a.heads + 2) * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = FS_CHAINS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    return launch_counted(cfg, kernel, a);
}

AIR_API int air_trace_set_attention_f32(unsigned long long* buffer) { return air::set_trace_here(buffer); }
