// The delta rule (with a decay per key channel, or one per head) and gated linear attention over whole portions of prompts, in
// chunks of 16 tokens whose rows are computed side by side from the state ahead of them.  Per head, with k, q of length d (k, and q before its scale, of unit length),
// g_t the decays and beta_t the step sizes, the recurrence is
//
//   S_t = diag(g_t) S_(t-1) + k_t u_t^T,   u_t = beta_t (v_t - (diag(g_t) S_(t-1))^T k_t),   o_t = S_t^T q_t.
//
// In a chunk that starts from S_0, with b_t the sum of the decays' logarithms up to token t (so that exp(b_t - b_s) <= 1 for
// s <= t: nothing overflows however fast a channel forgets):
//
//   a_ts = sum_c k_t k_s exp(b_t - b_s)  (s < t),   p_ts = sum_c q_t k_s exp(b_t - b_s)  (s <= t)
//   X_t  = beta_t (r_t - sum_(s < t) a_ts X_s),  solved for r_t = k_t exp(b_t) (-> W, [16, d]) and for r_t = v_t (-> Y, [16, dv])
//   U    = Y - W S_0
//   o_t  = (q_t exp(b_t)) S_0 + sum_(s <= t) p_ts u_s
//   S    = diag(exp(b_last)) S_0 + sum_s (k_s exp(b_last - b_s)) u_s^T
//
// One decay per head is the same with equal b's: a and p are then plain products times exp(b_t - b_s).  Gated linear attention
// is the same with u_t = v_t (q and k as they come, q times its scale): there is no a, W or X, and Y is v.
//
// delta_chunk_prepare_kernel   all that does not depend on the state, 32-bit on the CUDA cores, a block per chunk and head
// delta_chunk_scan_kernel      the last three lines, a block per head, portion and 16 columns of the state.  The state's
//                              columns are the rows of the tensor-core instruction (m16n8k8, TF32 operands, 32-bit sums), its
//                              channels lie across the warps and stay in accumulators from the first chunk to the last:
//                              as a result of one product they are the left operand of the next without a move (the
//                              instruction's k may run in any order that both operands share).  Every 32-bit operand enters as
//                              two TF32 numbers, hi + lo, and every product as lo hi + hi lo + hi hi, which keeps the
//                              operands to 2^-23: what is left out is of the order of 32-bit rounding.  The next chunks'
//                              numbers arrive by the copy engine, in two runs of bytes, while this one's are used.
//
// delta_chunk_scan_together_kernel   the same in half the threads, for many blocks.
//
// Measured, us, against the scan token by token: 2,048 tokens, 16 heads of 128 x 128, one decay per head 432 -> 149 (prepare
// 46, scan 102); gated linear attention, 777 tokens, 16 heads of 128 x 256, 189 -> 83 (29 and 53).  Which portions come here:
// parts/recurrent.py (least).
//
// What bounds the scan is the chain from chunk to chunk: three products of 24 instructions each that a warp issues at 10 cycles an
// instruction, the cutting of 64 numbers into halves, two barriers: 0.80 us a chunk, 0.69 for gated linear attention, which has two
// products.  Half of the warps hold the state and do nothing that the next chunk does not wait for; the sums across warps that give U, and
// the outputs, are the other half's, the latter a chunk behind.  (All of it in four warps: 1.15 us a chunk, 148 and 74 us for the two
// sizes above; the state handed to the other half for q S through shared memory: 136 and 70; barriers in memory instead of bar.sync: 177.)
//
// Errors against 64 bits (2-norm of the difference over that of the result, 2,048 tokens), token by token and here: one decay per
// head, outputs 1.98e-7 and 1.95e-7, states 1.56e-7 and 1.58e-7; gated linear attention 1.60e-7 and 1.60e-7, 1.40e-7 and 1.10e-7; decays
// near 1, where a token's own rounding adds up, 2.9e-6 and 2.5e-7.  (Operands cut instead of rounded to their upper half, the state
// as the products' accumulator, sums of logarithms in one number and 2^x in one instruction: 8.8e-7 and 5.4e-7, at 191 and 86 us.
// The state's update by multiply-adds on the CUDA cores: states 1.48e-7 and 1.01e-7, at 226 and 113 us.)
// An infinity or a NaN reaches what it reaches token by token, and nothing ahead of its token.
//
// What a row is depends on the state and the portion's tokens only.
#include "common.cuh"
#include "tma.cuh"

namespace air {

constexpr int DC = 16;              // tokens of a chunk, and columns of a block of the scan
constexpr int DC_RLD = 24, DC_ULD = 20;      // strides of rows in shared memory: four rows of 8 numbers, eight of 4, fall into different banks
constexpr float DC_FLOOR = -110.f;   // (e^-110 is 0 in 32 bits; differences of the logarithms' sums stay numbers)

// What a chunk and head leave in the scratch memory, DP the channels filled up to 32, 64, 128 or 256 (zeros), in floats:
//   rows [32][DP]     W and q exp b; the eight channels from 8 i on of row t stand at 8 (i ^ (t & 3))
//   keys [DP][16]     (k exp(b_last - b))^T; the eight tokens from 8 i on of channel c stand at 8 (i ^ (c / 2 & 1))
//   last [DP]         exp b_last
//   p    [16][16]     swizzled as the keys are
//   Y^T  [dvp][16]    dvp: dv filled up to a multiple of 16 (zeros)
// (in this arrangement four rows that a warp reads eight bytes at a time fall into different banks)
// (gated linear attention has no W: rows [16][DP] are q exp b alone)
enum { CHUNK_CHANNEL = 0, CHUNK_HEAD = 1, CHUNK_GLA = 2 };
template <int DP, int MODE> struct DeltaChunk {
    static constexpr int ROWS = MODE == CHUNK_GLA ? DC : 2 * DC, KEYS = ROWS * DP, LAST = KEYS + DC * DP, P = LAST + DP, Y = P + DC * DC;
};
__device__ __forceinline__ int dc_row_place(int t, int c) { return c ^ ((t & 3) << 3); }
__device__ __forceinline__ int dc_key_place(int c, int t) { return t ^ (((c >> 1) & 1) << 3); }

struct DeltaChunkArgs {
    const float* q; int ldq;        // [T, ldq]: head g's d numbers at column g * d, before their unit length and scale
    const float* k; int ldk;
    const float* v; int ldv;        // [T, ldv]: head h's dv numbers at column h * dv
    const float* decay; int ldd;    // [T, ldd]: d logits per head (HEAD: one)
    const float* beta; int ldb;     // [T, ldb]: one logit per head (not GLA)
    const float* a_log;             // [H] (not GLA)
    const float* dt_bias;           // [H * d] (HEAD: [H]; not GLA)
    const int* chunks;              // [N, 2]: first row, tokens
    const int* portions;            // [L, 4]: first row, tokens, slot, first chunk
    float* scratch;                 // [N, H, stride]
    float* state;                   // [slots, H, d, dv]
    float* out;                     // [T, H, dv]
    int H, G, d, dv, dvp;
    float q_scale, unit_eps, inv_tau;
    long long stride;
    int* status;
};

__device__ __forceinline__ float softplus_1(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }

// (four blocks to an SM: a block is a chain of short phases between barriers.  With three 49.7 us for 128 chunks of 16 heads, 51.7 with
// a decay per channel and 94 chunks; with four 45.7 and 48.5 for a few spilled registers; five 45.3 and 57.5.  Gated linear attention, 16
// heads, 300, 777, 1,200 and 2,048 tokens: three 13.2, 29.4, 39.2 and 64.2, four 13.5, 29.1, 37.1 and 59.5)
template <int DP, int MODE>
__global__ void __launch_bounds__(256, DP <= 128 ? 4 : 2) delta_chunk_prepare_kernel(const DeltaChunkArgs p) {
    constexpr int ld = DP + 4, PER = DP / 32;
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(16) float sa[DC][DC];
    __shared__ float sbeta[DC], slog[DC], skept[2][DC];       // (HEAD: a token's logarithm; what is left at it
                                                                   // of the state ahead, and of it at the chunk's end)
    pdl_enter(TR_SCAN);
    const int h = blockIdx.y, g = h / (p.H / p.G), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q0 = p.chunks[2 * blockIdx.x], n = p.chunks[2 * blockIdx.x + 1];
    const int d = p.d;
    float* sk = smem;                       // [16][ld]
    float* sq = sk + DC * ld;
    float* sg = sq + DC * ld;               // (not HEAD) the decays,
    float* sb = sg + DC * ld;               // their logarithms, then the logarithms' sums,
    float* sr = sb + DC * ld;               // and what rounding took from the sums
    const float rate = MODE == CHUNK_GLA ? -p.inv_tau : -expf(p.a_log[h]);
    auto log_of = [&](float z) {            // (a NaN stays one)
        const float x = rate * softplus_1(z);
        return x < DC_FLOOR ? DC_FLOOR : x;
    };
    {   // a warp per two tokens: unit lengths, logarithms (both tokens' loads under way at once)
        float x[2][PER], y[2][PER], z[2][PER];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = warp + 8 * r;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int c = lane + 32 * i;
                const bool in = t < n && c < d;
                x[r][i] = in ? p.k[(size_t)(q0 + t) * p.ldk + g * d + c] : 0.f;
                y[r][i] = in ? p.q[(size_t)(q0 + t) * p.ldq + g * d + c] : 0.f;
                // (log sigmoid(z) = -softplus(-z))
                z[r][i] = !in ? 0.f
                    : MODE == CHUNK_GLA ? -p.decay[(size_t)(q0 + t) * p.ldd + h * d + c]
                    : MODE == CHUNK_HEAD ? p.decay[(size_t)(q0 + t) * p.ldd + h] + p.dt_bias[h]
                    : p.decay[(size_t)(q0 + t) * p.ldd + h * d + c] + p.dt_bias[h * d + c];
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = warp + 8 * r;
            float ss = 0.f, qs = 0.f;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                ss = fmaf(x[r][i], x[r][i], ss);
                qs = fmaf(y[r][i], y[r][i], qs);
                if (MODE == CHUNK_HEAD) continue;
                const float left = t < n && lane + 32 * i < d ? log_of(z[r][i]) : 0.f;
                sb[t * ld + lane + 32 * i] = left;
                sg[t * ld + lane + 32 * i] = expf(left);
            }
            float kf = 1.f, qf = p.q_scale;
            if (MODE != CHUNK_GLA) {
                kf = 1.f / sqrtf(warp_sum(ss) + p.unit_eps);
                qf = p.q_scale / sqrtf(warp_sum(qs) + p.unit_eps);
            }
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                sk[t * ld + lane + 32 * i] = x[r][i] * kf;
                sq[t * ld + lane + 32 * i] = y[r][i] * qf;
            }
            if (MODE == CHUNK_HEAD && lane == 0) slog[t] = t < n ? log_of(z[r][0]) : 0.f;
            if (MODE != CHUNK_GLA && lane == 0) sbeta[t] = t < n ? 1.f / (1.f + expf(-p.beta[(size_t)(q0 + t) * p.ldb + h])) : 0.f;
        }
    }
    __syncthreads();
    // the logarithms' sums b_t, as two numbers each: b_t - b_s keeps the 24 bits that the decays between s and t have by
    // themselves, also behind a token that forgets nearly everything
    if (MODE != CHUNK_HEAD && tid < DP) {
        float sum = 0.f, rest = 0.f;
#pragma unroll
        for (int t = 0; t < DC; ++t) {
            const float x = sb[t * ld + tid], next = sum + x, from = next - sum;
            rest += (sum - (next - from)) + (x - from);          // (what the addition has rounded away: Knuth)
            sum = next;
            sb[t * ld + tid] = sum;
            sr[t * ld + tid] = rest;
        }
    }
    auto kept = [&](int s, int t) {                              // HEAD: what is left of token s at token t
        float sum = 0.f;
        for (int i = s + 1; i <= t; ++i) sum += slog[i];
        return expf(sum);
    };
    using Place = DeltaChunk<DP, MODE>;
    float* base = p.scratch + ((size_t)blockIdx.x * p.H + h) * p.stride;
    float* Pm = base + Place::P;
    {
        const int t = tid / DC, s = tid % DC;
        if (s > t) {
            sa[t][s] = 0.f;
            Pm[t * DC + dc_key_place(t, s)] = 0.f;
        }
    }
    __syncthreads();
    if (MODE == CHUNK_HEAD && tid >= 256 - 2 * DC) {
        const int t = tid % DC, end = tid >= 256 - DC;
        skept[end][t] = end ? kept(t, DC - 1) : kept(-1, t);
    }
    // a and p: four threads (a quarter of the channels each) per square of 2 x 2 tokens on or below the diagonal, 36 squares
    if (tid < 160) {
        const int square = min(tid >> 2, 35), part = tid & 3;
        int i = 0;
        while ((i + 1) * (i + 2) / 2 <= square) ++i;
        const int j = square - i * (i + 1) / 2;          // tokens 2 i, 2 i + 1 against 2 j, 2 j + 1
        float a[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, pq[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 2
        for (int c = part * 4; c < DP; c += 16) {
            float xk[2][4], xq[2][4], yk[2][4], late[4], early[4], m[4];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                load4(sk + (2 * i + r) * ld + c, xk[r]);
                load4(sq + (2 * i + r) * ld + c, xq[r]);
                load4(sk + (2 * j + r) * ld + c, yk[r]);
            }
            if (MODE != CHUNK_HEAD) {
                // what is left of token 2 j + 1 at token 2 i, from there the other three by one decay more each
                float b0[4], b1[4], r0[4], r1[4];
                load4(sg + (2 * i + 1) * ld + c, late);
                load4(sg + (2 * j + 1) * ld + c, early);
                load4(sb + (2 * j + 1) * ld + c, b0);
                load4(sb + 2 * i * ld + c, b1);
                load4(sr + (2 * j + 1) * ld + c, r0);
                load4(sr + 2 * i * ld + c, r1);
#pragma unroll
                for (int e = 0; e < 4; ++e) m[e] = i == j ? 0.f : expf((b1[e] - b0[e]) + (r1[e] - r0[e]));
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float w[2][2] = {{yk[0][e], yk[1][e]}, {yk[0][e], yk[1][e]}};
                if (MODE != CHUNK_HEAD) {
                    const float one = i == j ? 1.f : m[e] * early[e];      // (on the diagonal itself nothing has decayed)
                    w[0][0] *= one;
                    w[0][1] *= m[e];
                    w[1][0] *= one * late[e];
                    w[1][1] *= i == j ? 1.f : m[e] * late[e];
                }
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        if (MODE != CHUNK_GLA) a[r][s] = fmaf(xk[r][e], w[r][s], a[r][s]);
                        pq[r][s] = fmaf(xq[r][e], w[r][s], pq[r][s]);
                    }
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                a[r][s] += __shfl_xor_sync(0xffffffffu, a[r][s], 1);
                a[r][s] += __shfl_xor_sync(0xffffffffu, a[r][s], 2);
                pq[r][s] += __shfl_xor_sync(0xffffffffu, pq[r][s], 1);
                pq[r][s] += __shfl_xor_sync(0xffffffffu, pq[r][s], 2);
                const int t = 2 * i + r, u = 2 * j + s;
                if (part == 0 && tid < 144 && u <= t) {
                    if (MODE == CHUNK_HEAD) {
                        const float w = kept(u, t);
                        a[r][s] *= w;
                        pq[r][s] *= w;
                    }
                    if (MODE != CHUNK_GLA) sa[t][u] = u < t ? sbeta[t] * a[r][s] : 0.f;
                    Pm[t * DC + dc_key_place(t, u)] = pq[r][s];
                }
            }
    }
    __syncthreads();
    // W and Y, a thread per column; what else the scan reads of a channel
    for (int j = tid; j < DP + p.dvp; j += 256) {
        float x[DC];
        if (j < DP) {
            float* keys = base + Place::KEYS + j * DC;
#pragma unroll
            for (int t = 0; t < DC; t += 4) {
                float kv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int at = (t + i) * ld + j, end = (DC - 1) * ld + j;
                    const float k = sk[at], here = MODE == CHUNK_HEAD ? skept[0][t + i] : expf(sb[at]);
                    x[t + i] = k * here;
                    base[(Place::ROWS - DC + t + i) * DP + dc_row_place(t + i, j)] = sq[at] * here;
                    kv[i] = k * (MODE == CHUNK_HEAD ? skept[1][t + i] : expf((sb[end] - sb[at]) + (sr[end] - sr[at])));
                    if (t + i == DC - 1) base[Place::LAST + j] = here;
                }
                store4(keys + dc_key_place(j, t), kv);
            }
        } else {
            const int c = j - DP;
#pragma unroll
            for (int t = 0; t < DC; ++t) x[t] = t < n && c < p.dv ? p.v[(size_t)(q0 + t) * p.ldv + h * p.dv + c] : 0.f;
        }
        if (MODE == CHUNK_GLA && j < DP) continue;
        if (MODE != CHUNK_GLA)
#pragma unroll
        for (int t = 0; t < DC; ++t) {
            float sum = sbeta[t] * x[t];
#pragma unroll
            for (int s = 0; s < t; s += 4) {               // (the places on and above the diagonal hold zeros)
                float w[4];
                load4(&sa[t][s], w);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (s + i < t) sum = fmaf(-w[i], x[s + i], sum);
            }
            x[t] = sum;
        }
        if (j < DP) {
#pragma unroll
            for (int t = 0; t < DC; ++t) base[t * DP + dc_row_place(t, j)] = x[t];
        } else {
            float* dst = base + Place::Y + (j - DP) * DC;
#pragma unroll
            for (int t = 0; t < DC; t += 4) {
                const float y[4] = {x[t], x[t + 1], x[t + 2], x[t + 3]};
                store4(dst + t, y);
            }
        }
    }
}

struct Two { uint32_t hi, lo; };
// c = a b (FRESH) or c += a b; with k in the order that the accumulators have: a holds (row g, k 2t), (g + 8, 2t), (g, 2t + 1),
// (g + 8, 2t + 1), b holds (k 2t, column g), (2t + 1, g)
template <bool FRESH>
__device__ __forceinline__ void mma_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (FRESH)        // (zeros as an operand of their own: no register has to be cleared)
        asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                     "{%10, %10, %10, %10};"
                     : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
    else
        asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                     "{%0, %1, %2, %3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The three products of numbers as halves, for N tiles side by side: low += lo hi + hi lo, high = hi hi.  (A product waits 24 cycles
// for the sum that it adds to, one to a sum of its own 12.)
template <int N>
__device__ __forceinline__ void mma_two(bool fresh, float (&low)[N][4], float (&high)[N][4], const Two (&a)[4], const Two (&b)[N][2]) {
#pragma unroll
    for (int x = 0; x < N; ++x) {
        if (fresh) mma_tf32<true>(low[x], a[0].lo, a[1].lo, a[2].lo, a[3].lo, b[x][0].hi, b[x][1].hi);
        else mma_tf32<false>(low[x], a[0].lo, a[1].lo, a[2].lo, a[3].lo, b[x][0].hi, b[x][1].hi);
    }
#pragma unroll
    for (int x = 0; x < N; ++x) mma_tf32<true>(high[x], a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[x][0].hi, b[x][1].hi);
#pragma unroll
    for (int x = 0; x < N; ++x) mma_tf32<false>(low[x], a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[x][0].lo, b[x][1].lo);
}
// Two numbers at a time: the same sums as one by one.
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    asm("{\n\t.reg .b64 u, v;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tadd.rn.f32x2 u, u, v;\n\tmov.b64 {%0, %1}, u;\n\t}"
        : "+f"(a.x), "+f"(a.y) : "f"(b.x), "f"(b.y));
    return a;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    asm("{\n\t.reg .b64 u, v;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tsub.rn.f32x2 u, u, v;\n\tmov.b64 {%0, %1}, u;\n\t}"
        : "+f"(a.x), "+f"(a.y) : "f"(b.x), "f"(b.y));
    return a;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    asm("{\n\t.reg .b64 u, v, w;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tmov.b64 w, {%4, %5};\n\t"
        "fma.rn.f32x2 u, u, v, w;\n\tmov.b64 {%0, %1}, u;\n\t}"
        : "+f"(a.x), "+f"(a.y) : "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return a;
}
// A 32-bit number as two TF32 numbers, for a pair of them: the instruction reads the upper 19 bits of an operand.  The upper one is rounded,
// so that the lower one has 12 bits and a sign of its own, and what it loses is 2^-23 of x at most, to either side.  (Where rounding
// carries a NaN's bits into the sign, x - hi is a NaN all the same.)
__device__ __forceinline__ void two_of_pair(Two& a, Two& b, float2 v) {
    a.hi = (__float_as_uint(v.x) + 0x1000u) & 0xffffe000u;
    b.hi = (__float_as_uint(v.y) + 0x1000u) & 0xffffe000u;
    const float2 rest = sub2(v, make_float2(__uint_as_float(a.hi), __uint_as_float(b.hi)));
    a.lo = __float_as_uint(rest.x);
    b.lo = __float_as_uint(rest.y);
}
__device__ __forceinline__ void two_pair(Two (&b)[2], const float* p) {
    two_of_pair(b[0], b[1], *reinterpret_cast<const float2*>(p));
}

// One warp per scheduler holds the state: the fewer warps share the channels, the fewer sums cross between them (with eight 111 us where
// four take 106: what crosses shared memory doubles).  As many help.
constexpr int DC_WARPS = 4, DC_THREADS = 2 * DC_WARPS * 32;
constexpr int DC_STAGES = 6;        // chunks under way at most

// The scan's two barriers: the holders arrive at SUMS and wait at READY, the helpers the other way round.
enum { DC_SUMS = 1, DC_READY };
template <int ID> __device__ __forceinline__ void dc_sync() { asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(DC_THREADS) : "memory"); }
template <int ID> __device__ __forceinline__ void dc_arrive() { asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(DC_THREADS) : "memory"); }

// Shared memory of a block of the scan, in floats, behind its `stages` buffers.
template <int DP, int MODE> struct DeltaScan {
    static constexpr bool GLA = MODE == CHUNK_GLA;
    static constexpr int BUF = DeltaChunk<DP, MODE>::Y + DC * DC;    // a chunk's numbers and 16 columns of Y
    static constexpr int OUTS = GLA ? 1 : 3;                         // (what a helper reads behind SUMS of the next chunk)
    static constexpr int OUT = 0;                                    // [OUTS][warps][16 tokens][DC_ULD columns]: q S over a warp's channels
    static constexpr int SUMS = OUT + OUTS * DC_WARPS * DC * DC_ULD;    // [warps][16 columns][DC_RLD]: W S over a warp's channels
    static constexpr int U = SUMS + (GLA ? 0 : DC_WARPS * DC * DC_RLD); // [2][16 columns][DC_ULD]: U transposed
    static constexpr int TWO = U + (GLA ? 0 : 2 * DC * DC_ULD);      // [2][16 columns][8 tokens][hi, lo]: the same, cut
    static constexpr int END = TWO + (GLA ? 0 : 2 * DC * DC);
    static constexpr size_t bytes(int stages) { return sizeof(float) * (size_t)(stages * BUF + END); }
};

// 16 rows by NJ tiles of 8 channels times the state's columns: what the tensor cores cut off instead of rounding is kept small, since a
// large product is summed from zero and added up in 32 bits and the small ones have sums of their own.
template <int N>
__device__ __forceinline__ void add_tile(float2 (&sum)[N][2], float (&low)[N][4], int j, const Two (&a)[4], const Two (&b)[N][2]) {
    float high[N][4];
    mma_two<N>(j == 0, low, high, a, b);
#pragma unroll
    for (int x = 0; x < N; ++x)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float2 v = make_float2(high[x][2 * e], high[x][2 * e + 1]);
            sum[x][e] = j ? add2(sum[x][e], v) : v;
        }
}
template <int N> __device__ __forceinline__ void add_low(float2 (&sum)[N][2], const float (&low)[N][4]) {
#pragma unroll
    for (int x = 0; x < N; ++x)
#pragma unroll
        for (int e = 0; e < 2; ++e) sum[x][e] = add2(sum[x][e], make_float2(low[x][2 * e], low[x][2 * e + 1]));
}
template <int NJ>
__device__ __forceinline__ void rows_by_state(float2 (&sum)[2][2], const Two (&a)[NJ][4], const Two (&b)[NJ][2][2]) {
    float low[2][4];
#pragma unroll
    for (int j = 0; j < NJ; ++j) add_tile(sum, low, j, a[j], b[j]);
    add_low(sum, low);
}

// U's numbers of a column and two tokens: Y less the four warps' W S.
__device__ __forceinline__ float2 less_sums(float2 y, const float* from) {
    float2 v[DC_WARPS];
#pragma unroll
    for (int w = 0; w < DC_WARPS; ++w) v[w] = *reinterpret_cast<const float2*>(from + w * DC * DC_RLD);
    return sub2(y, add2(add2(v[0], v[1]), add2(v[2], v[3])));
}
// Of p: what token t (0 .. 7) and its mirror image 15 - t take of the tokens up to them (17 products in all).
__device__ __forceinline__ void rows_of_p(float (&pa)[DC / 2], float (&pb)[DC], const float* p, int t) {
#pragma unroll
    for (int s = 0; s < DC; s += 4) {
        if (s < DC / 2) load4(p + t * DC + dc_key_place(t, s), *reinterpret_cast<float(*)[4]>(&pa[s]));
        load4(p + (DC - 1 - t) * DC + dc_key_place(DC - 1 - t, s), *reinterpret_cast<float(*)[4]>(&pb[s]));
    }
}
// The outputs of these two tokens in a column: q S (the warps' sums [warps][16][DC_ULD], at the column) and what the chunk's tokens add to
// one another, on the CUDA cores: only those up to a token itself, since a product with the zeros of p above the diagonal would carry a
// later token's infinity or NaN into this one's o.
__device__ __forceinline__ float2 outputs_of(const float (&pa)[DC / 2], const float (&pb)[DC], const float* u_at, const float* sums, int t) {
    float u[DC], va[DC_WARPS], vb[DC_WARPS];
#pragma unroll
    for (int s = 0; s < DC; s += 4) load4(u_at + s, *reinterpret_cast<float(*)[4]>(&u[s]));
#pragma unroll
    for (int w = 0; w < DC_WARPS; ++w) {
        va[w] = sums[(w * DC + t) * DC_ULD];
        vb[w] = sums[(w * DC + DC - 1 - t) * DC_ULD];
    }
    float o_a = 0.f, o_b = 0.f, late = 0.f;
#pragma unroll
    for (int s = 0; s < DC / 2; ++s) {
        if (s <= t) o_a = fmaf(pa[s], u[s], o_a);
        o_b = fmaf(pb[s], u[s], o_b);
        if (s < DC / 2 - t) late = fmaf(pb[DC / 2 + s], u[DC / 2 + s], late);
    }
    return make_float2(((va[0] + va[1]) + (va[2] + va[3])) + o_a, ((vb[0] + vb[1]) + (vb[2] + vb[3])) + (o_b + late));
}

// DC_WARPS warps hold the state.  Such a warp holds NJ tiles of 8 channels of it, transposed: S[j] is (column g or g + 8 of the block) x
// (channels 8 j + 2 t, 8 j + 2 t + 1), g = lane / 4, t = lane % 4.  It multiplies W with it, then q while the four helping warps add up
// the holders' W S to U, then takes U into the state.  The helpers complete a chunk's outputs while the holders are at the next one.
// (A warp that has given up a wait goes on through all chunks without waiting: nobody is left at a barrier.)
template <int DP, int MODE, bool ALONE>
__global__ void __launch_bounds__(DC_THREADS, ALONE ? 1 : 2) delta_chunk_scan_kernel(const DeltaChunkArgs p, int stages) {
    constexpr int NJ = DP / (8 * DC_WARPS), GROUP = NJ < 4 ? NJ : 4;
    constexpr bool GLA = MODE == CHUNK_GLA, EARLY = ALONE && NJ <= 4, AHEAD = EARLY && !GLA, BY_TILE = GLA && !ALONE && NJ > 4;
    using Place = DeltaChunk<DP, MODE>;
    using Scan = DeltaScan<DP, MODE>;
    constexpr int BUF = Scan::BUF;
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(8) uint64_t full[DC_STAGES];
    __shared__ int gave_up;
    float* const rest = smem + stages * BUF;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t2 = 2 * (lane & 3);
    const bool holder = warp < DC_WARPS;
    if (tid == 0) {
        for (int i = 0; i < DC_STAGES; ++i) mbar_init(&full[i], 1);
        gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_enter(TR_SCAN);
    const int h = blockIdx.y, col0 = blockIdx.x * DC;
    const int* por = p.portions + 4 * blockIdx.z;
    const int row0 = por[0], tokens = por[1], slot = por[2], chunk0 = por[3];
    if (slot < 0 || tokens <= 0) return;     // (no chunk: nothing to wait for, to add or to write)
    const int chunks = (tokens + DC - 1) / DC;
    auto bring = [&](int i, int stage) {               // (one thread)
        const float* src = p.scratch + ((size_t)(chunk0 + i) * p.H + h) * p.stride;
        float* dst = smem + stage * BUF;
        mbar_expect_tx(&full[stage], BUF * 4);
        bulk_load(dst, src, Place::Y * 4, &full[stage]);
        bulk_load(dst + Place::Y, src + Place::Y + col0 * DC, DC * DC * 4, &full[stage]);
    };
    if (tid == 0)
        for (int i = 0; i < min(stages, chunks); ++i) bring(i, i);
    bool ok = true;
    int stage = 0, phase = 0, slot_out = 0;
    if (holder) {
        const int r0 = warp * 8 * NJ;
        float* st = p.state + ((size_t)slot * p.H + h) * p.d * p.dv;
        float2 S[NJ][2];                     // [column g, g + 8] (channels t2, t2 + 1)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = r0 + 8 * j + t2 + (e & 1), c = col0 + g + 8 * (e >> 1);
                (e & 1 ? S[j][e >> 1].y : S[j][e >> 1].x) = r < p.d && c < p.dv ? st[(size_t)r * p.dv + c] : 0.f;
            }
        const int swap = dc_key_place(g, 0);             // (of rows 8 j + g: the tile does not matter)
        float* const sums_to = rest + Scan::SUMS + (warp * DC + g) * DC_RLD + t2;
        float* const out_to = rest + Scan::OUT + (warp * DC + t2) * DC_ULD + g;
        auto rows = [&](Two (&b)[NJ][2][2], const float* buf, int first) {           // of W or q: rows g and 8 + g
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const float* at = buf + (first + g) * DP + t2 + dc_row_place(g, r0 + 8 * j);
                two_pair(b[j][0], at);
                two_pair(b[j][1], at + 8 * DP);
            }
        };
        Two b[NJ][2][2];
        ok = __all_sync(0xffffffffu, mbar_wait(&full[0], 0, &gave_up));
        if constexpr (AHEAD) rows(b, smem, 0);
        for (int i = 0; i < chunks; ++i) {
            const float* buf = smem + stage * BUF;
            if (++stage == stages) {
                stage = 0;
                phase ^= 1;
            }
            // (the next chunk's numbers are there by now, as a rule)
            const bool there = i + 1 == chunks || mbar_try_wait(&full[stage], phase);
            float2 sum[2][2];
            Two a[NJ][4];
            if constexpr (!BY_TILE)
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    two_of_pair(a[j][0], a[j][2], S[j][0]);
                    two_of_pair(a[j][1], a[j][3], S[j][1]);
                }
            Two c[NJ][2][2];                     // (what is cut ahead of a product is cut between the one before it)
            if constexpr (EARLY) rows(c, buf, Place::ROWS - DC);
            if constexpr (!GLA) {
                if constexpr (!AHEAD) rows(b, buf, 0);
                rows_by_state(sum, a, b);
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int e = 0; e < 2; ++e) *reinterpret_cast<float2*>(sums_to + 8 * e * DC_RLD + 8 * x) = sum[x][e];
                dc_arrive<DC_SUMS>();
            }
            if constexpr (!EARLY && !BY_TILE) rows(c, buf, Place::ROWS - DC);
            Two k[2][GROUP][2], u[2][4];         // keys; U transposed, tokens 0 .. 7 and 8 .. 15
            auto keys = [&](int j0) {
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int j = 0; j < GROUP; ++j)
                        two_pair(k[x][j], buf + Place::KEYS + (r0 + 8 * (j0 + j) + g) * DC + ((8 * x) ^ swap) + t2);
            };
            if constexpr (EARLY) keys(0);
            if constexpr (BY_TILE) {             // (as many registers as two blocks to an SM have)
                float low[2][4];
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    Two at[4], q[2][2];
                    two_of_pair(at[0], at[2], S[j][0]);
                    two_of_pair(at[1], at[3], S[j][1]);
                    const float* row = buf + g * DP + t2 + dc_row_place(g, r0 + 8 * j);
                    two_pair(q[0], row);
                    two_pair(q[1], row + 8 * DP);
                    add_tile(sum, low, j, at, q);
                }
                add_low(sum, low);
            } else {
                rows_by_state(sum, a, c);
            }
            if constexpr (!EARLY) keys(0);
            if constexpr (GLA) {                 // (u is v; the helpers are done with the last chunk's sums)
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        two_of_pair(u[x][e], u[x][2 + e], *reinterpret_cast<const float2*>(buf + Place::Y + (g + 8 * e) * DC + 8 * x + t2));
                if (i > 0) dc_sync<DC_READY>();
            }
            float* const to = out_to + slot_out * DC_WARPS * DC * DC_ULD;
            if (++slot_out == Scan::OUTS) slot_out = 0;
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    to[8 * x * DC_ULD + 8 * e] = sum[x][e].x;
                    to[(8 * x + 1) * DC_ULD + 8 * e] = sum[x][e].y;
                }
            if constexpr (GLA) dc_arrive<DC_SUMS>();
            else {
                dc_sync<DC_READY>();
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const uint4 z = *reinterpret_cast<const uint4*>(rest + Scan::TWO + x * DC * DC + (g + 8 * e) * DC + 2 * t2);
                        u[x][e] = Two{z.x, z.y};
                        u[x][2 + e] = Two{z.z, z.w};
                    }
            }
            if (!there && ok) ok = mbar_wait(&full[stage], phase, &gave_up);
            __syncwarp();
            if constexpr (AHEAD) rows(b, smem + stage * BUF, 0);     // (between the products; of no chunk: what lies there, unused)
#pragma unroll
            for (int j0 = 0; j0 < NJ; j0 += GROUP) {
                if (j0) keys(j0);
                float more[2][GROUP][4], less[GROUP][4];
#pragma unroll
                for (int x = 0; x < 2; ++x) mma_two<GROUP>(x == 0, less, more[x], u[x], k[x]);
#pragma unroll
                for (int j = 0; j < GROUP; ++j) {
                    const float2 left = *reinterpret_cast<const float2*>(buf + Place::LAST + r0 + 8 * (j0 + j) + t2);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float2 x = make_float2(more[0][j][2 * e], more[0][j][2 * e + 1]), y = make_float2(more[1][j][2 * e], more[1][j][2 * e + 1]);
                        S[j0 + j][e] = fma2(S[j0 + j][e], left, add2(x, add2(y, make_float2(less[j][2 * e], less[j][2 * e + 1]))));
                    }
                }
            }
        }
        if constexpr (!GLA) dc_arrive<DC_SUMS>();      // (the last chunk's q S)
        __syncthreads();
        if (!gave_up) {
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int r = r0 + 8 * j + t2 + (e & 1), c = col0 + g + 8 * (e >> 1);
                    if (r < p.d && c < p.dv) st[(size_t)r * p.dv + c] = e & 1 ? S[j][e >> 1].y : S[j][e >> 1].x;
                }
        }
    } else {
        const int mine = warp - DC_WARPS;
        // the numbers of U that this thread completes, a column's tokens u_t and u_t + 1, and the outputs: a token and its mirror image
        const int u_c = 4 * mine + ((lane >> 2) & 3), u_t = 2 * (lane & 3) + 8 * (lane >> 4);
        const int o_c = lane & 15, o_t = mine + 4 * (lane >> 4);
        const float* const sums_from = rest + Scan::SUMS + u_c * DC_RLD + u_t;
        float* const out = p.out + ((size_t)row0 * p.H + h) * p.dv + col0 + o_c;
        const size_t out_row = (size_t)p.H * p.dv;
        const bool in = col0 + o_c < p.dv;
        float pa[DC / 2], pb[DC];
        auto outputs = [&](int i, const float* u_at) {
            const float* sums_of = rest + Scan::OUT + slot_out * DC_WARPS * DC * DC_ULD + o_c;
            if (++slot_out == Scan::OUTS) slot_out = 0;
            const float2 o = outputs_of(pa, pb, u_at, sums_of, o_t);
            if (!in || !ok) return;
            if (i * DC + o_t < tokens) out[(size_t)(i * DC + o_t) * out_row] = o.x;
            if (i * DC + DC - 1 - o_t < tokens) out[(size_t)(i * DC + DC - 1 - o_t) * out_row] = o.y;
        };
        for (int i = 0; i < chunks; ++i) {
            const float* buf = smem + stage * BUF;
            if (ok) ok = mbar_wait(&full[stage], phase, &gave_up);
            __syncwarp();
            float2 y = *reinterpret_cast<const float2*>(buf + Place::Y + u_c * DC + u_t);
            dc_sync<DC_SUMS>();
            if constexpr (!GLA) {
                y = less_sums(y, sums_from);
                if (i * DC + u_t >= tokens) y.x = 0.f;       // (of no token: nothing, also beside a state of infinities)
                if (i * DC + u_t + 1 >= tokens) y.y = 0.f;
                Two one, two;
                two_of_pair(one, two, y);
                *reinterpret_cast<uint4*>(rest + Scan::TWO + (u_t >> 3) * DC * DC + u_c * DC + 2 * (u_t & 7)) = make_uint4(one.hi, one.lo, two.hi, two.lo);
                *reinterpret_cast<float2*>(rest + Scan::U + (i & 1) * DC * DC_ULD + u_c * DC_ULD + u_t) = y;
                dc_arrive<DC_READY>();
            }
            // everybody is done with the chunk before this one: its buffer may be filled again
            if (tid == DC_WARPS * 32 && i > 0 && i - 1 + stages < chunks) bring(i - 1 + stages, stage ? stage - 1 : stages - 1);
            if constexpr (GLA) {
                rows_of_p(pa, pb, buf + Place::P, o_t);
                outputs(i, buf + Place::Y + o_c * DC);
                if (i + 1 < chunks) dc_arrive<DC_READY>();
            } else {
                if (i > 0) outputs(i - 1, rest + Scan::U + ((i - 1) & 1) * DC * DC_ULD + o_c * DC_ULD);
                rows_of_p(pa, pb, buf + Place::P, o_t);
            }
            if (++stage == stages) {
                stage = 0;
                phase ^= 1;
            }
        }
        if constexpr (!GLA) {
            dc_sync<DC_SUMS>();
            outputs(chunks - 1, rest + Scan::U + ((chunks - 1) & 1) * DC * DC_ULD + o_c * DC_ULD);
        }
        __syncthreads();
    }
    if (gave_up) {
        for (int x = 0; x < 32; ++x) __nanosleep(2000);      // (a copy on its way may still land)
        if (tid == 0 && p.status) atomicExch(p.status, 9);
    }
}

// The same scan in four warps, for more blocks than the SMs hold of the other's (launch_delta_chunks says where).  What counts then is not the
// chain but how many of them an SM has: half the threads, one chunk ahead instead of five, nothing cut ahead of its use, three to
// eight blocks to an SM.  Every number is summed as above and in the same order, a chunk's outputs with the chunk: the same bits.
template <int DP, int MODE> struct DeltaTogether {
    static constexpr bool GLA = MODE == CHUNK_GLA;
    static constexpr int BUF = DeltaScan<DP, MODE>::BUF;
    static constexpr int OUT = 0, SUMS = OUT + DC_WARPS * DC * DC_ULD, U = SUMS + (GLA ? 0 : DC_WARPS * DC * DC_RLD), END = U + (GLA ? 0 : DC * DC_ULD);
    static constexpr size_t bytes = sizeof(float) * (size_t)(2 * BUF + END);
};
template <int DP, int MODE>
__global__ void __launch_bounds__(DC_WARPS * 32) delta_chunk_scan_together_kernel(const DeltaChunkArgs p) {
    constexpr int NJ = DP / (8 * DC_WARPS), GROUP = NJ < 4 ? NJ : 4, RG = DeltaChunk<DP, MODE>::ROWS / 8;
    constexpr bool GLA = MODE == CHUNK_GLA;
    using Place = DeltaChunk<DP, MODE>;
    using Scan = DeltaTogether<DP, MODE>;
    constexpr int BUF = Scan::BUF;
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(8) uint64_t full[2];
    __shared__ int gave_up;
    float* const rest = smem + 2 * BUF;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t2 = 2 * (lane & 3);
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) mbar_init(&full[i], 1);
        gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_enter(TR_SCAN);
    const int h = blockIdx.y, col0 = blockIdx.x * DC;
    const int* por = p.portions + 4 * blockIdx.z;
    const int row0 = por[0], tokens = por[1], slot = por[2], chunk0 = por[3];
    if (slot < 0 || tokens <= 0) return;
    const int chunks = (tokens + DC - 1) / DC;
    auto bring = [&](int i) {               // (one thread)
        const float* src = p.scratch + ((size_t)(chunk0 + i) * p.H + h) * p.stride;
        float* dst = smem + (i & 1) * BUF;
        mbar_expect_tx(&full[i & 1], BUF * 4);
        bulk_load(dst, src, Place::Y * 4, &full[i & 1]);
        bulk_load(dst + Place::Y, src + Place::Y + col0 * DC, DC * DC * 4, &full[i & 1]);
    };
    if (tid == 0) bring(0);
    const int r0 = warp * 8 * NJ;
    float* st = p.state + ((size_t)slot * p.H + h) * p.d * p.dv;
    float2 S[NJ][2];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = r0 + 8 * j + t2 + (e & 1), c = col0 + g + 8 * (e >> 1);
            (e & 1 ? S[j][e >> 1].y : S[j][e >> 1].x) = r < p.d && c < p.dv ? st[(size_t)r * p.dv + c] : 0.f;
        }
    const int swap = dc_key_place(g, 0);
    const int u_c = 4 * warp + ((lane >> 2) & 3), u_t = 2 * (lane & 3) + 8 * (lane >> 4);
    const int o_c = lane & 15, o_t = warp + 4 * (lane >> 4);
    float* const out = p.out + ((size_t)row0 * p.H + h) * p.dv + col0 + o_c;
    const size_t out_row = (size_t)p.H * p.dv;
    for (int i = 0; i < chunks; ++i) {
        const float* buf = smem + (i & 1) * BUF;
        // this chunk's numbers are there and everybody is done with the chunk before it
        if (__syncthreads_or(!mbar_wait(&full[i & 1], (i >> 1) & 1, &gave_up))) {
            for (int x = 0; x < 32; ++x) __nanosleep(2000);      // (a copy on its way may still land)
            if (tid == 0 && p.status) atomicExch(p.status, 9);
            return;
        }
        if (tid == 0 && i + 1 < chunks) bring(i + 1);
        float2 sum[RG][2];
        float low[RG][4];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            Two a[4], b[RG][2];
            two_of_pair(a[0], a[2], S[j][0]);
            two_of_pair(a[1], a[3], S[j][1]);
            const float* at = buf + g * DP + t2 + dc_row_place(g, r0 + 8 * j);
#pragma unroll
            for (int x = 0; x < RG; ++x) two_pair(b[x], at + 8 * x * DP);
            add_tile(sum, low, j, a, b);
        }
        add_low(sum, low);
#pragma unroll
        for (int x = 0; x < RG; ++x)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (x < RG - 2) {                // W's rows, then q's
                    *reinterpret_cast<float2*>(rest + Scan::SUMS + (warp * DC + g + 8 * e) * DC_RLD + 8 * x + t2) = sum[x][e];
                } else {
                    float* to = rest + Scan::OUT + (warp * DC + 8 * (x - (RG - 2)) + t2) * DC_ULD + g + 8 * e;
                    to[0] = sum[x][e].x;
                    to[DC_ULD] = sum[x][e].y;
                }
            }
        __syncthreads();
        if constexpr (!GLA) {
            float2 y = less_sums(*reinterpret_cast<const float2*>(buf + Place::Y + u_c * DC + u_t), rest + Scan::SUMS + u_c * DC_RLD + u_t);
            if (i * DC + u_t >= tokens) y.x = 0.f;       // (of no token: nothing, also beside a state of infinities)
            if (i * DC + u_t + 1 >= tokens) y.y = 0.f;
            *reinterpret_cast<float2*>(rest + Scan::U + u_c * DC_ULD + u_t) = y;
            __syncthreads();
        }
        const float* const U = GLA ? buf + Place::Y : rest + Scan::U;
        constexpr int ULD = GLA ? DC : DC_ULD;
        Two u[2][4];                         // U transposed, tokens 0 .. 7 and 8 .. 15
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int e = 0; e < 2; ++e) two_of_pair(u[x][e], u[x][2 + e], *reinterpret_cast<const float2*>(U + (g + 8 * e) * ULD + 8 * x + t2));
#pragma unroll
        for (int j0 = 0; j0 < NJ; j0 += GROUP) {
            float more[2][GROUP][4], less[GROUP][4];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                Two k[GROUP][2];
#pragma unroll
                for (int j = 0; j < GROUP; ++j) two_pair(k[j], buf + Place::KEYS + (r0 + 8 * (j0 + j) + g) * DC + ((8 * x) ^ swap) + t2);
                mma_two<GROUP>(x == 0, less, more[x], u[x], k);
            }
#pragma unroll
            for (int j = 0; j < GROUP; ++j) {
                const float2 left = *reinterpret_cast<const float2*>(buf + Place::LAST + r0 + 8 * (j0 + j) + t2);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float2 x = make_float2(more[0][j][2 * e], more[0][j][2 * e + 1]), y = make_float2(more[1][j][2 * e], more[1][j][2 * e + 1]);
                    S[j0 + j][e] = fma2(S[j0 + j][e], left, add2(x, add2(y, make_float2(less[j][2 * e], less[j][2 * e + 1]))));
                }
            }
        }
        float pa[DC / 2], pb[DC];
        rows_of_p(pa, pb, buf + Place::P, o_t);
        const float2 o = outputs_of(pa, pb, U + o_c * ULD, rest + Scan::OUT + o_c, o_t);
        if (col0 + o_c < p.dv) {
            if (i * DC + o_t < tokens) out[(size_t)(i * DC + o_t) * out_row] = o.x;
            if (i * DC + DC - 1 - o_t < tokens) out[(size_t)(i * DC + DC - 1 - o_t) * out_row] = o.y;
        }
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = r0 + 8 * j + t2 + (e & 1), c = col0 + g + 8 * (e >> 1);
            if (r < p.d && c < p.dv) st[(size_t)r * p.dv + c] = e & 1 ? S[j][e >> 1].y : S[j][e >> 1].x;
        }
}

template <int DP, int MODE, bool ALONE>
static int launch_delta_scan(const DeltaChunkArgs& a, dim3 grid, size_t room, size_t least, cudaStream_t stream) {
    using Scan = DeltaScan<DP, MODE>;
    int stages = DC_STAGES;
    while (stages > 2 && Scan::bytes(stages) > room) --stages;
    const size_t smem = max(Scan::bytes(stages), least);
    auto kernel = delta_chunk_scan_kernel<DP, MODE, ALONE>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(DC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    return launch_counted(cfg, kernel, a, stages);
}

template <int DP, int MODE> static int launch_delta_together(const DeltaChunkArgs& a, dim3 grid, cudaStream_t stream) {
    const size_t smem = DeltaTogether<DP, MODE>::bytes;
    auto kernel = delta_chunk_scan_together_kernel<DP, MODE>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(DC_WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    return launch_counted(cfg, kernel, a);
}

template <int DP, int MODE>
static int launch_delta_chunks(const DeltaChunkArgs& args, int N, int L, cudaStream_t stream) {
    DeltaChunkArgs a = args;
    a.dvp = (a.dv + 15) / 16 * 16;
    a.stride = DeltaChunk<DP, MODE>::Y + (long long)DC * a.dvp;
    const size_t smem1 = sizeof(float) * (MODE == CHUNK_HEAD ? 2 : 5) * DC * (DP + 4);
    if (smem1 > 44 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(delta_chunk_prepare_kernel<DP, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
        if (e != cudaSuccess) return (int)e;
    }
    int rc = launch(delta_chunk_prepare_kernel<DP, MODE>, dim3(N, a.H), 256, smem1, stream, a);
    if (rc) return rc;
    const dim3 grid(a.dvp / DC, a.H, L);
    // (as for the scan token by token: the blocks start when their predecessor has ended, and spread over the SMs)
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long blocks = (long long)grid.x * grid.y * grid.z;
    // Where every block has an SM to itself a warp has the registers to cut what its next product reads between the instructions of the one
    // before, and as many chunks are under way as memory holds; else two blocks share an SM, except where a delta rule's rows of 256 leave
    // no registers for that.  (32 heads of 128 x 128, 256 blocks, 2,048 tokens: 192 us; with one block to an SM they would take two rounds of
    // 102.  Gated linear attention, heads of 256 x 256, two to an SM and one, us with the preparation: 16 heads, 300 tokens 69.3 and 72, 32 heads,
    // 1,000 tokens 342 and 359, 8 portions of 33 tokens 166 and 205.)
    // More blocks than that, and an SM is kept busy by four warps of each of three to eight: delta rule, two to an SM and these, heads of 64 x 128,
    // 512 blocks 3, 7 and 13 chunks long 22.7 / 20.6, 32.2 / 30.5 and 47.5 / 45.8, 4,096 of 7 172 / 152; heads of 128, 512 of 3, 7 and 63 chunks
    // 25.0 / 24.7, 47.1 / 48.5 and 240 / 248 (gated linear attention 22.6 / 20.8, 38.8 / 37.4, 184 / 195), 1,024 of 7 67.6 / 65.7, 4,096 of 3 108 /
    // 98; heads of 256, 4,096 of 13 656 / 734.
    if constexpr (DP <= 128)
        if (blocks > 2 * sms && (DP <= 64 || blocks > 4 * sms || N <= 4 * L)) return launch_delta_together<DP, MODE>(a, grid, stream);
    if constexpr (DP <= 128 || MODE == CHUNK_GLA)
        if (blocks > sms) return launch_delta_scan<DP, MODE, false>(a, grid, 113 * 1024, 0, stream);
    return launch_delta_scan<DP, MODE, true>(a, grid, 226 * 1024, blocks <= sms ? 120 * 1024 : 0, stream);
}

}  // namespace air

namespace air {
template <int MODE> static int launch_chunks_of(const DeltaChunkArgs& a, int N, int L, cudaStream_t stream) {
    if (a.d <= 32) return launch_delta_chunks<32, MODE>(a, N, L, stream);
    if (a.d <= 64) return launch_delta_chunks<64, MODE>(a, N, L, stream);
    if (a.d <= 128) return launch_delta_chunks<128, MODE>(a, N, L, stream);
    return launch_delta_chunks<256, MODE>(a, N, L, stream);
}
}  // namespace air

// mode 0: the delta rule with a decay per key channel, 1: with one per head, 2: gated linear attention (alpha =
// sigmoid(decay)^inv_tau; no beta, a_log, dt_bias, unit lengths).  scratch: float32 [N, H, 49 DP + 256 + 16 dvp] (mode 2: 33
// DP) with DP = d filled up to 32, 64, 128 or 256, dvp = dv to a multiple of 16.  Rows and slots as the lists say; d up to 256.
AIR_API int air_delta_portions(int mode, const float* q, int ldq, const float* k, int ldk, const float* v, int ldv,
                               const float* decay, int ldd, const float* beta, int ldb, const float* a_log,
                               const float* dt_bias, float* state, float* out, const int* portions, int L, const int* chunks,
                               int N, float* scratch, int H, int G, int d, int dv, float q_scale, float unit_eps, float inv_tau,
                               int* status, cudaStream_t stream) {
    using namespace air;
    if (L <= 0 || N <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || d <= 0 || d > 256 || dv <= 0 || H > 65535 || L > 65535 || !scratch ||
        ((uintptr_t)scratch & 15) || mode < 0 || mode > 2 || (mode != CHUNK_GLA && (!beta || !a_log || !dt_bias)))
        return AIR_ERR_BAD_ARGUMENT;
    DeltaChunkArgs a;
    a.q = q; a.ldq = ldq; a.k = k; a.ldk = ldk; a.v = v; a.ldv = ldv; a.decay = decay; a.ldd = ldd; a.beta = beta; a.ldb = ldb;
    a.a_log = a_log; a.dt_bias = dt_bias; a.chunks = chunks; a.portions = portions; a.scratch = scratch; a.state = state;
    a.out = out; a.H = H; a.G = G; a.d = d; a.dv = dv; a.dvp = 0; a.q_scale = q_scale; a.unit_eps = unit_eps; a.stride = 0;
    a.inv_tau = inv_tau;
    a.status = status;
    if (mode == CHUNK_GLA) return launch_chunks_of<CHUNK_GLA>(a, N, L, stream);
    if (mode == CHUNK_HEAD) return launch_chunks_of<CHUNK_HEAD>(a, N, L, stream);
    return launch_chunks_of<CHUNK_CHANNEL>(a, N, L, stream);
}

AIR_API int air_trace_set_delta_chunks(unsigned long long* buffer) { return air::set_trace_here(buffer); }
