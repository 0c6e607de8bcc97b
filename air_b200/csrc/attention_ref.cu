// Paged attention with 32-bit arithmetic for any batch: portions of prompts and single
// decoded tokens alike.  It is the kernel of the float32 path and the fallback of the
// bfloat16 path for head sizes that the tensor-core kernels do not take.
//
// One block per (token, query head), four warps.  Keys are visited in blocks of 32 aligned
// to their absolute position; warp w takes the blocks whose index is w modulo 4, keeps a
// running maximum, sum and weighted value (online softmax), and the four partial results
// are merged in a fixed order.  What a query computes therefore depends only on its
// position and on the cache's contents, not on how the tokens were cut into steps or on
// what else is in the batch.
//
// q: [T, H, d], out: [T, H, dv].  cache: a page holds the keys [K, P, d] and behind them the values [K, P, dv]
// (with dv == d that is [page, 2, K, P, d]).  block_table: [slots, max_blocks], row token_seq[t] for token t
// (negative: padding, skipped).
// A query at position p sees keys max(0, p - window + 1) .. p (window 0: all keys); with mask_mode 1 `window` is the
// size of a chunk instead, and the query sees the keys p - p % window .. p (those of its own chunk, counted from
// position 0 of the request).  With `sink` (float32 [H]) the softmax's denominator holds one more term exp(sink[h]):
// a bare logit that `scale` does not touch and that brings nothing to the output.  With `latent` a page is [P, d] (one row per token, no heads): every
// query head reads the same row as its key, and the row's first dv elements as its value.  q is float32 if q_f32,
// else of the cache's type.
// score = scale * q.k, and with softcap > 0 then softcap * tanh(score / softcap); then, where `bias` is given, plus the
// head's number for the distance (DistanceBias).  With `gate` [T, H] (float32) a
// head's output is multiplied by its token's gate.
#include "common.cuh"

namespace air {

constexpr int ATT_WARPS = 4;

template <typename T, int ATT_MAX_D>
__global__ void __launch_bounds__(ATT_WARPS * 32)
paged_attention_ref_kernel(const void* __restrict__ q_any, int q_f32, const T* __restrict__ cache,
                           const int* __restrict__ block_table, int max_blocks,
                           const int* __restrict__ token_seq, const int* __restrict__ positions,
                           T* __restrict__ out, const float* __restrict__ gate, int H, int K, int d, int dv, int P,
                           int window, float scale, float softcap, int mask_mode, const float* __restrict__ sink,
                           int latent, const DistanceBias bias) {
    __shared__ float sq[ATT_MAX_D];
    __shared__ float sm[ATT_WARPS], sl[ATT_WARPS];
    __shared__ float sacc[ATT_WARPS][ATT_MAX_D];
    pdl_enter(TR_ATT_REF);
    const int t = blockIdx.x, h = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (token_seq[t] < 0) return;  // padding
    const int pos = positions[t];
    const int kvh = (int)(((long long)h * K) / H);
    const int* bt = block_table + (size_t)token_seq[t] * max_blocks;
    const int lo = window > 0 ? (mask_mode == 1 ? pos - pos % window : max(0, pos - window + 1)) : 0;

    if (q_f32)
        for (int i = threadIdx.x; i < d; i += blockDim.x) sq[i] = ((const float*)q_any)[((size_t)t * H + h) * d + i];
    else
        for (int i = threadIdx.x; i < d; i += blockDim.x) sq[i] = to_float(((const T*)q_any)[((size_t)t * H + h) * d + i]);
    __syncthreads();

    const int chunks = (dv + 31) / 32;
    float acc[ATT_MAX_D / 32];
#pragma unroll
    for (int c = 0; c < ATT_MAX_D / 32; ++c) acc[c] = 0.f;
    float m = -INFINITY, l = 0.f;

    const size_t page_stride = latent ? (size_t)P * d : (size_t)K * P * (d + dv);
    const size_t v_offset = latent ? 0 : (size_t)K * P * d;
    const int v_stride = latent ? d : dv;
    for (int b = (lo / 32 / ATT_WARPS) * ATT_WARPS + warp; b * 32 <= pos; b += ATT_WARPS) {
        const int key = b * 32 + lane;
        const bool valid = key >= lo && key <= pos;
        size_t base = 0;      // of the key's value
        float s = -INFINITY;
        if (valid) {
            const int page = bt[key / P];
            const size_t place = (size_t)kvh * P + (size_t)(key % P);
            base = (size_t)page * page_stride + v_offset + place * v_stride;
            const T* kp = cache + (size_t)page * page_stride + place * d;
            float dot = 0.f;
            for (int i = 0; i < d; ++i) dot = fmaf(sq[i], to_float(kp[i]), dot);
            s = dot * scale;
            if (softcap > 0.f) s = softcap * tanhf(s / softcap);
            s += distance_bias(bias, h, pos - key);
        }
        const float bm = warp_max(s);
        if (bm == -INFINITY) continue;  // the whole block is outside the window
        const float m_new = fmaxf(m, bm);
        const float corr = expf(m - m_new);  // 0 when m was -inf
        const float p = valid ? expf(s - m_new) : 0.f;
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int c = 0; c < ATT_MAX_D / 32; ++c) acc[c] *= corr;
        m = m_new;
        for (int j = 0; j < 32; ++j) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const unsigned long long bj = __shfl_sync(0xffffffffu, (unsigned long long)base, j);
            if (pj == 0.f) continue;  // same for the whole warp
            const T* vp = cache + bj;
#pragma unroll
            for (int c = 0; c < ATT_MAX_D / 32; ++c) {
                const int i = c * 32 + lane;
                if (c < chunks && i < dv) acc[c] = fmaf(pj, to_float(vp[i]), acc[c]);
            }
        }
    }
    if (lane == 0) { sm[warp] = m; sl[warp] = l; }
#pragma unroll
    for (int c = 0; c < ATT_MAX_D / 32; ++c) {
        const int i = c * 32 + lane;
        if (c < chunks && i < dv) sacc[warp][i] = acc[c];
    }
    __syncthreads();
    float mm = sink ? sink[h] : -INFINITY;
    for (int w = 0; w < ATT_WARPS; ++w) mm = fmaxf(mm, sm[w]);
    float total = sink ? expf(sink[h] - mm) : 0.f;
    float weight[ATT_WARPS];
    for (int w = 0; w < ATT_WARPS; ++w) {
        weight[w] = sm[w] == -INFINITY ? 0.f : expf(sm[w] - mm);
        total += sl[w] * weight[w];
    }
    const float inv = (gate ? gate[(size_t)t * H + h] : 1.f) / total;
    for (int i = threadIdx.x; i < dv; i += blockDim.x) {
        float o = 0.f;
        for (int w = 0; w < ATT_WARPS; ++w) o += sacc[w][i] * weight[w];
        out[((size_t)t * H + h) * dv + i] = from_float<T>(o * inv);
    }
}

// ---------------------------------------------------------------------------------------------- float32, heads up to 128
// The same sums in the same order (bit for bit), for a float32 cache.  What bounded the kernel above were its reads: a lane
// read its own key number by number, 32 cache lines an instruction.  Here a warp copies its block's 32 keys and values row by
// row into memory of its own (cp.async: the next block's keys while this one's values are added up, and the other way
// round), a lane then reads its key four numbers at a time, and where consecutive rows are consecutive tokens of a request
// (a portion of a prompt) a block takes REF_QUERIES of them, so that a key is fetched once for all of them.
// Measured, us: see air_paged_attention_ref.
constexpr int REF_QUERIES = 8, REF_D = 128;

struct RefArgs {
    const float* q; const float* cache; const int* block_table; int max_blocks; const int* token_seq; const int* positions;
    float* out; const float* gate; int T, H, K, d, dv, P, window; float scale, softcap; int mask_mode; const float* sink;
    int latent; DistanceBias bias;
};
// Shared memory, in floats: the rows' queries, the warps' maxima and sums, then per warp 32 keys (rows of d + 4: eight that
// lie beside one another cover the banks; behind the last block the warp's weighted values), 32 values and the weights.
// SHARED: the values take the keys' memory once the scores are there.
struct RefPlaces {
    int d, dv;
    bool shared;
    __host__ __device__ int keys() const { return max(max(32 * (d + 4), REF_QUERIES * dv), shared ? 32 * dv : 0); }
    __host__ __device__ int of_warp() const { return keys() + (shared ? 0 : 32 * dv) + REF_QUERIES * 32; }
    __host__ __device__ int head() const { return REF_QUERIES * d + 2 * ATT_WARPS * REF_QUERIES; }
    __host__ __device__ size_t bytes() const { return sizeof(float) * (head() + ATT_WARPS * of_warp()); }
};

__device__ __forceinline__ void ref_copy16(void* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void ref_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ref_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
    __syncwarp();
}

// Rows t .. t + n - 1: positions pos .. pos + n - 1 of the request in row `seq` of the table.
// D: the size of keys and values where it is known (the loops over it and the strides are then constants: 100 us against 126 for
// 300 rows of 128), else 0.
template <int N, int D, bool SHARED>
__device__ __forceinline__ void ref_rows(const RefArgs& a, float* smem, int t, int n, int pos, int seq) {
    const int h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d = D ? D : a.d, dv = D ? D : a.dv;
    const int kvh = (int)(((long long)h * a.K) / a.H);
    const int* bt = a.block_table + (size_t)seq * a.max_blocks;
    const size_t page_stride = a.latent ? (size_t)a.P * d : (size_t)a.K * a.P * (d + dv);
    const size_t v_offset = a.latent ? 0 : (size_t)a.K * a.P * d;
    const int v_stride = a.latent ? d : dv;
    auto first = [&](int p) { return a.window > 0 ? (a.mask_mode == 1 ? p - p % a.window : max(0, p - a.window + 1)) : 0; };
    for (int i = threadIdx.x; i < n * d; i += ATT_WARPS * 32) smem[i] = a.q[((size_t)(t + i / d) * a.H + h) * d + i % d];
    __syncthreads();
    const RefPlaces places{d, dv, SHARED};
    const float* sq = smem;
    float* sm = smem + REF_QUERIES * d;
    float* sl = sm + ATT_WARPS * REF_QUERIES;
    float* sk = smem + places.head() + warp * places.of_warp();
    float* sv = SHARED ? sk : sk + places.keys();
    float* sp = sk + places.keys() + (SHARED ? 0 : 32 * dv);
    const int kld = d + 4;
    const int last = pos + n - 1, lo = first(pos);       // (the lowest key of any row is the first row's)
    // lane j knows where key j of a block lies and where its value does; -1: no row sees it, it is not copied and not used
    long long k_at = -1, v_at = -1;
    auto find = [&](int b) {
        const int key = b * 32 + lane;
        k_at = v_at = -1;
        if (key < lo || key > last) return;
        const long long page = (long long)bt[key / a.P] * (long long)page_stride, row = (long long)kvh * a.P + key % a.P;
        k_at = page + row * d;
        v_at = page + (long long)v_offset + row * v_stride;
    };
    auto bring = [&](long long at, float* dst, int ld, int width) {
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            const long long row = __shfl_sync(0xffffffffu, at, j);
            if (row >= 0 && lane * 4 < width) ref_copy16(dst + j * ld + lane * 4, a.cache + row + lane * 4);
        }
        ref_commit();
    };
    float acc[N][REF_D / 32], m[N], l[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < REF_D / 32; ++c) acc[i][c] = 0.f;
    }
    int b = (lo / 32 / ATT_WARPS) * ATT_WARPS + warp;
    if (b * 32 <= last) {
        find(b);
        bring(k_at, sk, kld, d);
        if (!SHARED) bring(v_at, sv, dv, dv);
    }
    for (; b * 32 <= last; b += ATT_WARPS) {
        const int key = b * 32 + lane;
        ref_wait<SHARED ? 0 : 1>();              // the keys are there
        float s[N];
#pragma unroll
        for (int i = 0; i < N; ++i) s[i] = 0.f;
#pragma unroll 4
        for (int x = 0; x < d; x += 4) {
            float k[4];
            load4(sk + lane * kld + x, k);
#pragma unroll
            for (int i = 0; i < N; ++i) {
                float q[4];
                load4(sq + (N > 1 ? min(i, n - 1) : 0) * d + x, q);
#pragma unroll
                for (int e = 0; e < 4; ++e) s[i] = fmaf(q[e], k[e], s[i]);
            }
        }
        __syncwarp();
        const bool more = (b + ATT_WARPS) * 32 <= last;
        if (SHARED) bring(v_at, sv, dv, dv);
        if (more) find(b + ATT_WARPS);
        if (more && !SHARED) {
            bring(k_at, sk, kld, d);
        }
        float corr[N];
        bool any = false;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const bool valid = i < n && key >= first(pos + i) && key <= pos + i;
            float x = s[i] * a.scale;
            if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
            x += valid ? distance_bias(a.bias, h, pos + i - key) : 0.f;
            x = valid ? x : -INFINITY;
            const float bm = warp_max(x);
            corr[i] = 1.f;
            float p = 0.f;
            if (bm != -INFINITY) {               // (else the whole block is outside the row's window)
                const float m_new = fmaxf(m[i], bm);
                corr[i] = expf(m[i] - m_new);    // 0 when m was -inf
                p = valid ? expf(x - m_new) : 0.f;
                l[i] = l[i] * corr[i] + warp_sum(p);
                m[i] = m_new;
                any = true;
            }
            sp[i * 32 + lane] = p;
        }
        if (more && !SHARED) ref_wait<1>();      // the values are there
        else ref_wait<0>();
        if (any) {
#pragma unroll
            for (int i = 0; i < N; ++i)
#pragma unroll
                for (int c = 0; c < REF_D / 32; ++c) acc[i][c] *= corr[i];
#pragma unroll 2
            for (int j = 0; j < 32; j += 4) {
                float p[N][4];
#pragma unroll
                for (int i = 0; i < N; ++i) load4(sp + i * 32 + j, p[i]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float v[REF_D / 32];
#pragma unroll
                    for (int c = 0; c < REF_D / 32; ++c) v[c] = c * 32 + lane < dv ? sv[(j + e) * dv + c * 32 + lane] : 0.f;
#pragma unroll
                    for (int i = 0; i < N; ++i)
                        if (p[i][e] != 0.f)      // same for the whole warp
#pragma unroll
                            for (int c = 0; c < REF_D / 32; ++c) acc[i][c] = fmaf(p[i][e], v[c], acc[i][c]);
                }
            }
        }
        __syncwarp();
        if (more && !SHARED) bring(v_at, sv, dv, dv);
        if (more && SHARED) bring(k_at, sk, kld, d);
    }
    ref_wait<0>();
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (lane == 0) { sm[warp * REF_QUERIES + i] = m[i]; sl[warp * REF_QUERIES + i] = l[i]; }
#pragma unroll
        for (int c = 0; c < REF_D / 32; ++c)
            if (c * 32 + lane < dv) sk[i * dv + c * 32 + lane] = acc[i][c];
    }
    __syncthreads();
    for (int x = threadIdx.x; x < n * dv; x += ATT_WARPS * 32) {
        const int i = x / dv, c = x % dv;
        float mm = a.sink ? a.sink[h] : -INFINITY;
        for (int w = 0; w < ATT_WARPS; ++w) mm = fmaxf(mm, sm[w * REF_QUERIES + i]);
        float total = a.sink ? expf(a.sink[h] - mm) : 0.f, o = 0.f;
        for (int w = 0; w < ATT_WARPS; ++w) {
            const float mw = sm[w * REF_QUERIES + i], weight = mw == -INFINITY ? 0.f : expf(mw - mm);
            total += sl[w * REF_QUERIES + i] * weight;
            o += smem[places.head() + w * places.of_warp() + x] * weight;
        }
        const float inv = (a.gate ? a.gate[(size_t)(t + i) * a.H + h] : 1.f) / total;
        a.out[((size_t)(t + i) * a.H + h) * dv + c] = o * inv;
    }
    __syncthreads();
}

// A block takes `per_block` rows of the batch for one head: runs of consecutive tokens of a request among them together.
// ROOM: how many blocks are to find registers on an SM (0: the compiler takes as many as it likes).
template <int D, bool SHARED, int ROOM>
__global__ void __launch_bounds__(ATT_WARPS * 32, ROOM) paged_attention_f32_kernel(const RefArgs a, int per_block) {
    extern __shared__ __align__(16) float smem[];
    pdl_enter(TR_ATT_REF);
    const int end = min(a.T, (int)(blockIdx.x + 1) * per_block);
    for (int t = blockIdx.x * per_block; t < end;) {
        const int seq = a.token_seq[t], pos = a.positions[t];
        if (seq < 0) { ++t; continue; }          // padding
        int n = 1;
        while (n < REF_QUERIES && t + n < end && a.token_seq[t + n] == seq && a.positions[t + n] == pos + n) ++n;
        if (n == 1) ref_rows<1, D, SHARED>(a, smem, t, 1, pos, seq);
        else if (n <= REF_QUERIES / 2) ref_rows<REF_QUERIES / 2, D, SHARED>(a, smem, t, n, pos, seq);
        else ref_rows<REF_QUERIES, D, SHARED>(a, smem, t, n, pos, seq);
        t += n;
    }
}

}  // namespace air

AIR_API int air_paged_attention_ref(const void* q, int q_f32, const void* cache, int dtype, const int* block_table,
                                    int max_blocks, const int* token_seq, const int* positions, void* out,
                                    const float* gate, int T, int H, int K, int d, int dv, int P, int window,
                                    float scale, float softcap, int mask_mode, const float* sink, int latent,
                                    const float* bias, int bias_n, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (bias && bias_n < 1) return AIR_ERR_BAD_ARGUMENT;
    const air::DistanceBias db{bias, bias_n};
    if (d <= 0 || d > 640 || dv <= 0 || dv > 640 || H <= 0 || K <= 0 || H > 65535 || mask_mode < 0 || mask_mode > 1 ||
        (latent && (dv > d || K != 1)))
        return AIR_ERR_BAD_ARGUMENT;
    dim3 grid(T, H);
    if (dtype == AIR_F32 && d <= air::REF_D && dv <= air::REF_D && d % 4 == 0 && dv % 4 == 0 && ((uintptr_t)cache & 15) == 0) {
        // As many rows to a block, up to REF_QUERIES, as leave a block for every SM.  Measured, us, against the kernel above: 300
        // rows of a prompt, 16 heads of 128: 473 -> 63; 512 rows behind 500: 3,315 -> 247; 4 single tokens over 1,000 keys, 28
        // heads: 317 -> 32; one over 4,000: 1,217 -> 99; 64 over 2,000: 2,409 -> 488.
        // A block waits for its own reads, its shared-memory loads and its chains of sums, one warp to a scheduler.  Where there are
        // more blocks than SMs hold at a time (two, or as many as their memory allows), the values take the keys' memory and three
        // share an SM (300 rows 101 -> 63, 512 401 -> 247, 64 single tokens over 2,000 744 -> 488); else a block keeps both, so that
        // the next keys arrive meanwhile.  Measured, us, both and values in the keys' memory: heads of 128 (one block of both to an SM),
        // 128 blocks of 2,000 keys 49 and 55, 224 95 and 73, 192 of 1,000 50 and 37; heads of 96 (two), 256 blocks of 1,000 keys 37 and 45,
        // 192 in runs of three 104 and 108, 608 of a prompt of 300 60 and 52; of 64 (two), 256 of 1,000 35 and 39, 400 of a portion 102 and 67.
        // Sizes other than 128 have two forms with both: 142 registers where every block has an SM (128 blocks of 1,000 keys, heads of
        // 64: 30.2 us, 31.7 with 194), 194 where two share one (256: 39.5, 34.9).
        const int per_block = (int)min((long long)air::REF_QUERIES, max(1ll, (long long)T * H / 148));
        const air::RefArgs args{(const float*)q, (const float*)cache, block_table, max_blocks, token_seq, positions, (float*)out,
                                gate, T, H, K, d, dv, P, window, scale, softcap, mask_mode, sink, latent, db};
        const long long blocks = (long long)((T + per_block - 1) / per_block) * H;
        const int resident = (int)min((size_t)2, (size_t)(228 * 1024) / (air::RefPlaces{d, dv, false}.bytes() + 1024));
        const bool shared = blocks > 148 * resident;
        const size_t smem = air::RefPlaces{d, dv, shared}.bytes();
        auto kernel = d == 128 && dv == 128 ? (shared ? air::paged_attention_f32_kernel<128, true, 3> : air::paged_attention_f32_kernel<128, false, 1>)
                      : shared              ? air::paged_attention_f32_kernel<0, true, 3>
                      : blocks > 148        ? air::paged_attention_f32_kernel<0, false, 1>
                                            : air::paged_attention_f32_kernel<0, false, 0>;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return (int)e;
        return air::launch(kernel, dim3((T + per_block - 1) / per_block, H), air::ATT_WARPS * 32,
                           smem, stream, args, per_block);
    }
    AIR_DISPATCH(dtype, TT, {
        if (d <= 256 && dv <= 256)
            return air::launch(air::paged_attention_ref_kernel<TT, 256>, grid, air::ATT_WARPS * 32, 0, stream, q, q_f32,
                               (const TT*)cache, block_table, max_blocks, token_seq, positions, (TT*)out, gate, H, K,
                               d, dv, P, window, scale, softcap, mask_mode, sink, latent, db);
        return air::launch(air::paged_attention_ref_kernel<TT, 640>, grid, air::ATT_WARPS * 32, 0, stream, q, q_f32,
                           (const TT*)cache, block_table, max_blocks, token_seq, positions, (TT*)out, gate, H, K, d,
                           dv, P, window, scale, softcap, mask_mode, sink, latent, db);
    });
    return 0;
}

AIR_API int air_trace_set_attention_ref(unsigned long long* buffer) { return air::set_trace_here(buffer); }
