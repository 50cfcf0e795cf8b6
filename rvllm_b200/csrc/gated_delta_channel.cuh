// The gated delta rule with one decay per key channel over portions in chunks of 64 tokens, on the
// tensor cores (bfloat16 models; included by gated_delta.cu, whose first comment has the recurrence).
//
// For a head and the tokens 0..63 of a chunk let k_i, q_i be the unit keys and queries (q scaled),
// B_i[c] the sum of channel c's log decays up to and with token i and S_0 the state before the chunk.
// With A_ij = beta_i sum_c k_i[c] k_j[c] e^(B_i[c] - B_j[c]) (j < i), P_ij the same with q_i, without
// beta and with j = i, and T = (I + A)^(-1) diag(beta),
//
//     U = T V - W S_0,   W = T (k e^(B)),       S = diag(e^(B_L)) S_0 + (k e^(B_L - B))^T U
//     o_i = (q_i e^(B_i))^T S_0 + sum_(j <= i) P_ij u_j
//
// A channel may forget by e^-100 within a chunk, so e^(B_i) and e^(-B_j) are never formed apart.  A and P
// are made in blocks of 16 by 16 tokens: below the diagonal blocks the decay from j to i passes the
// first token of i's block, e^(from there to i) and e^(from j to there), neither above 1, go to the two
// operands of a product; within a diagonal block the second eight tokens meet the first eight in the same way, and
// every pair's own power is taken within those.  The sums start anew in
// every block of 16, forwards and backwards.  Only within a diagonal block an exponent is a difference of
// two sums, which are large behind a token that forgets strongly; there a sum is a float32 and what its
// additions lost (a bfloat16: some 2^-33 of it), so that the difference has its own float32 precision.  A
// log decay below -192 counts as -192: either way the power, and every power across the token, is 0.  (One
// token in sixteen with a log decay of -300: error of the state 1.2e-7, as token by token; with plain
// differences 7.9e-6, and NaN behind a decay of -inf.)
//
//   gch_logs    log decays -> [n, H d]
//   conv_silu   q | k | v pass the convolutions and silu -> rows [n, C] float32 (conv_silu.cuh)
//   gch_chunk   block per (chunk, head): unit norms, sums of decays, A, P, the inverse, W, T V, q e^(B) and
//               k e^(B_L - B)
//   gch_scan    block per (head, 16 value columns, request): over the chunks one after another, the two
//               products with S in float32 accumulators; the state before every chunk and U go
//               out, the last state is the record
//   gch_out     warp per (chunk, 16 tokens, head, 32 value columns): o
//
// A value that is not finite must not reach earlier tokens through a product with the zero that stands
// for "later": gch_chunk takes such a value as 0 and notes its token.  From a bad key, value, decay or beta on
// every output of the head is NaN, and so is its state; a bad query's own output is.
//
// Everything is float32: operands enter the bfloat16 products as three parts each (chunks.cuh), six of
// the nine products (the state's error against 64 bits, mean of 16 prompts of 640 tokens with weak / middling / strong
// decays: 3.05e-7 / 1.94e-7 / 1.41e-7; with multiply-adds in the diagonal blocks 3.07e-7 / 1.93e-7 / 1.41e-7).  What one kernel leaves for another's products lies in the order in which a
// warp's fragments hold it, 16 bytes a lane, so that it goes from memory to registers as it is.
//
// The scan by token is a chain of some 360 cycles a token; here it is two products and two barriers a
// chunk (2.4 us, of which the products' issue is 0.8).  gch_chunk has one block of 512 threads a
// multiprocessor (179 KB) and is a row of short phases (thousand cycles: loads 4, norms and sums 4, A and P 14, the
// inverse 7, what scan and out multiply with 7, W and T V 5); 264 such blocks take 57 us.
// 8 heads of 128 by 128, one call: 2,048 tokens 440 -> 201 us, 559 + 1,489 tokens 370 -> 183,
// 4 x 512 tokens of 16 heads 480 -> 315, keys of 64 305 -> 140, 512 tokens beside 31 single ones 261 -> 96.
#pragma once
#include "gated_delta_chunk.cuh"

#define GH_THREADS 512      // threads of a block of gch_chunk
#define GH_LOG2E 1.4426950408889634f
#define GH_NOTHING -192.f   // a power of two that is no float32, whatever it is multiplied by

struct GhArgs {
    const float *proj, *lowrank, *a_log, *dt_bias;
    const float *rows, *logs;                // [n, C], [n, H d]
    const int *q_start, *state_slot;
    int P, LW, C, first_req, n_reqs, H, G, d, dv;
    float unit_eps;
    // per (item, head); pairs of bfloat16, UP = (d / 16 + 1) / 2
    unsigned *W;                             // [3][8 groups of 8 tokens][UP][32][4]
    unsigned *K, *Q;                         // [3][d / 16][4][32][4], [3][4][d / 16][32][4]
    unsigned *S, *U;                         // [dv / 16][3][2][UP][32][4], [dv / 16][3][2][2][32][4]
    float *Pm, *V, *dec;                     // [64][64] (i >= j), [dv][64], [d]
    int4 *bad;                               // the first token that is not finite (64: none), the queries that are not
};

__device__ __forceinline__ float gh_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Whether x can be taken into three parts; if not it is 0 from here on.
__device__ __forceinline__ bool gh_clean(float& x) {
    const bool ok = fabsf(x) <= 3.3895313e38f;            // the largest bfloat16
    if (!ok) x = 0.f;
    return ok;
}
__device__ __forceinline__ bool gh_clean(float4& v) {
    const bool a = gh_clean(v.x), b = gh_clean(v.y), c = gh_clean(v.z), e = gh_clean(v.w);
    return a && b && c && e;
}
// Four of them, on a 4-byte boundary.
__device__ __forceinline__ void gh_lost(const bf16* p, float (&x)[4]) {
    const float2 a = lm_pair(*(const unsigned*)p), b = lm_pair(*(const unsigned*)(p + 2));
    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
}

// The log decays (powers of two) of the portions' tokens, four channels a thread.
__global__ void __launch_bounds__(256) gch_logs_kernel(const GhArgs g, float* __restrict__ logs, int first_token,
                                                       long long count) {
    rv_pdl_launch_dependents();
    const long long x = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
    const int width = g.H * g.d;
    if (x >= count) {
        rv_pdl_wait();
        return;
    }
    const int t = first_token + (int)(x / width), c = (int)(x % width);
    const float rate = -GH_LOG2E * expf(g.a_log[c / g.d]);
    const float4 b = make_float4(g.dt_bias[c], g.dt_bias[c + 1], g.dt_bias[c + 2], g.dt_bias[c + 3]);
    rv_pdl_wait();
    const float4 l = *(const float4*)(g.lowrank + (size_t)t * g.LW + c);
    *(float4*)(logs + (size_t)t * width + c) = make_float4(
        rate * la_softplus(l.x + b.x), rate * la_softplus(l.y + b.y), rate * la_softplus(l.z + b.z), rate * la_softplus(l.w + b.w));
}

template <int UNITS>
__global__ void __launch_bounds__(GH_THREADS) gch_chunk_kernel(const GhArgs g) {
    rv_pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr int d = 16 * UNITS, LD = d + 8, UP = (UNITS + 1) / 2;
    float* As = (float*)smraw;                            // [64][65]
    float* Xs = As + 64 * 65;                             // [64][65]: the inverse; before it
    bf16* ls = (bf16*)Xs;                                 // [64][d + 2]: what the sums bs have lost
    float* tot = Xs + 64 * 65;                            // [4][d]: a block of 16's sum; before it; behind it
    float *pre = tot + 4 * d, *post = pre + 4 * d;
    float* ks = post + 4 * d;                             // [64][LD] each: keys, queries, the sums of the
    float* qs = ks + 64 * LD;                             // logs (powers of two) up to the token and
    float* bs = qs + 64 * LD;                             // behind it within its block
    float* fs = bs + 64 * LD;
    bf16* kt = (bf16*)ks;                                 // then [3][64][LD]: k e^(B)
    bf16* vt = kt + 3 * 64 * LD;                          // and [3][64][LV]: v
    __shared__ float beta[64];
    __shared__ int at[2], bad;                            // the first token with a value that is not finite
    __shared__ unsigned bad_q[2];                         // the tokens whose query is not
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, dv = g.dv, LV = dv + 8;
    const int item = blockIdx.x, h = blockIdx.y, kh = h / (g.H / g.G);
    if (tid == 0) {
        bad = 64;
        bad_q[0] = bad_q[1] = 0u;
    }
    lm_locate(g.q_start, g.state_slot, g.first_req, g.n_reqs, item, at);
    const int t0 = at[0], L = at[1];
    rv_pdl_wait();
    if (t0 < 0) return;
    const size_t ih = (size_t)item * g.H + h;
    const float* base = g.rows + (size_t)t0 * g.C;
    {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        constexpr int EACH = (64 * (d / 4) + GH_THREADS - 1) / GH_THREADS;
        float4 q[EACH], k[EACH], l[EACH];
#pragma unroll
        for (int u = 0; u < EACH; ++u) {
            const int x = tid + u * GH_THREADS, j = x / (d / 4), c = (x - j * (d / 4)) * 4;
            const bool there = j < L;
            q[u] = there ? *(const float4*)(base + (size_t)j * g.C + kh * d + c) : zero;
            k[u] = there ? *(const float4*)(base + (size_t)j * g.C + (g.G + kh) * d + c) : zero;
            l[u] = there ? *(const float4*)(g.logs + ((size_t)(t0 + j) * g.H + h) * d + c) : zero;
        }
#pragma unroll
        for (int u = 0; u < EACH; ++u) {
            const int x = tid + u * GH_THREADS, j = x / (d / 4), c = (x - j * (d / 4)) * 4;
            if (x >= 64 * (d / 4)) continue;
            if (!gh_clean(q[u])) atomicOr(&bad_q[j >> 5], 1u << (j & 31));
            if (!gh_clean(k[u])) atomicMin(&bad, j);
            // (a decay that is -inf forgets all, as it should)
            if (l[u].x != l[u].x || l[u].y != l[u].y || l[u].z != l[u].z || l[u].w != l[u].w) {
                l[u] = zero;
                atomicMin(&bad, j);
            }
            *(float4*)(qs + j * LD + c) = q[u];
            *(float4*)(ks + j * LD + c) = k[u];
            *(float4*)(bs + j * LD + c) = l[u];
        }
        if (tid < 64) {
            float b = tid < L ? 1.f / (1.f + expf(-g.proj[(size_t)(t0 + tid) * g.P + g.C + h])) : 0.f;
            if (!gh_clean(b)) atomicMin(&bad, tid);
            beta[tid] = b;
        }
    }
    __syncthreads();
    {   // unit norms: eight lanes a token
        const int j = tid >> 3;
        float nq = 0.f, nk = 0.f;
        for (int c = (tid & 7) * 4; c < d; c += 32) {
            const float4 q = *(const float4*)(qs + j * LD + c), k = *(const float4*)(ks + j * LD + c);
            nq += q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w;
            nk += k.x * k.x + k.y * k.y + k.z * k.z + k.w * k.w;
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            nq += __shfl_xor_sync(0xffffffffu, nq, o);
            nk += __shfl_xor_sync(0xffffffffu, nk, o);
        }
        float iq = 1.f / sqrtf((float)d) / sqrtf(nq + g.unit_eps), ik = 1.f / sqrtf(nk + g.unit_eps);
        // (a row of zeros without an epsilon: beyond the chunk's end it is no token)
        if (!gh_clean(iq) && j < L && (tid & 7) == 0) atomicOr(&bad_q[j >> 5], 1u << (j & 31));
        if (!gh_clean(ik) && j < L && (tid & 7) == 0) atomicMin(&bad, j);
        for (int c = (tid & 7) * 4; c < d; c += 32) {
            float4 q = *(const float4*)(qs + j * LD + c), k = *(const float4*)(ks + j * LD + c);
            q.x *= iq; q.y *= iq; q.z *= iq; q.w *= iq;
            k.x *= ik; k.y *= ik; k.z *= ik; k.w *= ik;
            *(float4*)(qs + j * LD + c) = q;
            *(float4*)(ks + j * LD + c) = k;
        }
    }
    // the sums, a block of 16 tokens and a channel a thread
    for (int x = tid; x < 4 * d; x += GH_THREADS) {
        const int J = x / d, c = x - J * d;
        float l[16], s = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) l[i] = bs[(16 * J + i) * LD + c];
#pragma unroll
        for (int i = 0; i < 16; ++i) l[i] = l[i] < GH_NOTHING ? GH_NOTHING : l[i];       // (NaN stays)
        float lost = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float t = s + l[i], z = t - s;
            lost += (s - (t - z)) + (l[i] - z);
            s = t;
            bs[(16 * J + i) * LD + c] = s;
            ls[(16 * J + i) * (d + 2) + c] = __float2bfloat16_rn(lost);
        }
        tot[J * d + c] = s;
        s = 0.f;
#pragma unroll
        for (int i = 15; i >= 0; --i) {
            fs[(16 * J + i) * LD + c] = s;
            s += l[i];
        }
    }
    __syncthreads();
    float* Pm = g.Pm + ih * 64 * 64;
    if (warp < 10) {
        // blocks of eight on the diagonal: 10 tiles of two by two tokens each, four lanes a tile, whose
        // loads meet few banks twice (two lanes a tile of blocks of sixteen: 23,000 cycles a chunk beside the products of the other blocks, 13,600 so)
        const int unit = tid >> 2, J = unit / 10, ti = unit - 10 * J;
        int a = 0;
        while ((a + 1) * (a + 2) / 2 <= ti) ++a;
        const int i0 = 8 * J + 2 * a, j0 = 8 * J + 2 * (ti - a * (a + 1) / 2);
        float s[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, p[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 2
        for (int c = (tid & 3) * 4; c < d; c += 16) {
            float ki[2][4], qi[2][4], bi[2][4], kj[2][4], bj[2][4], li[2][4], lj[2][4];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                la_load<float, 4>(ks + (i0 + e) * LD + c, ki[e]);
                la_load<float, 4>(qs + (i0 + e) * LD + c, qi[e]);
                la_load<float, 4>(bs + (i0 + e) * LD + c, bi[e]);
                la_load<float, 4>(ks + (j0 + e) * LD + c, kj[e]);
                la_load<float, 4>(bs + (j0 + e) * LD + c, bj[e]);
                gh_lost(ls + (i0 + e) * (d + 2) + c, li[e]);
                gh_lost(ls + (j0 + e) * (d + 2) + c, lj[e]);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float w = kj[j][x] * gh_exp2((bi[i][x] - bj[j][x]) + (li[i][x] - lj[j][x]));
                        s[i][j] = fmaf(ki[i][x], w, s[i][j]);
                        p[i][j] = fmaf(qi[i][x], w, p[i][j]);
                    }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    s[i][j] += __shfl_xor_sync(0xffffffffu, s[i][j], o);
                    p[i][j] += __shfl_xor_sync(0xffffffffu, p[i][j], o);
                }
                const int r = i0 + i, t = j0 + j;
                if ((tid & 3) == 0) As[r * 65 + t] = t < r ? beta[r] * s[i][j] : 0.f;
                if ((tid & 3) == 1) Pm[r * 64 + t] = t <= r ? p[i][j] : 0.f;        // (beyond the diagonal: no power of a sum)
            }
        // the blocks of eight below those, a pair's a warp: tokens 8 .. 15 of sixteen against 0 .. 7, keys in
        // the product's first eight rows and queries in the others, the decay by way of token 7
        if (warp < 4) {
            const int I = 16 * warp, r = I + 8 + (lane >> 2), j = I + (lane >> 2);
            float y[3][4] = {};
#pragma unroll 2
            for (int kk = 0; kk < UNITS; ++kk) {
                unsigned f[3][4], b[3][2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int c = 16 * kk + e * 8 + (lane & 3) * 2;
                    const float2 m = *(const float2*)(bs + (I + 7) * LD + c), ml = lm_pair(*(const unsigned*)(ls + (I + 7) * (d + 2) + c)),
                                 x = *(const float2*)(bs + r * LD + c), xl = lm_pair(*(const unsigned*)(ls + r * (d + 2) + c)),
                                 z = *(const float2*)(bs + j * LD + c), zl = lm_pair(*(const unsigned*)(ls + j * (d + 2) + c)),
                                 k = *(const float2*)(ks + r * LD + c), q = *(const float2*)(qs + r * LD + c),
                                 kj = *(const float2*)(ks + j * LD + c);
                    const float fx = gh_exp2((x.x - m.x) + (xl.x - ml.x)), fy = gh_exp2((x.y - m.y) + (xl.y - ml.y));
                    lm_split(k.x * fx, k.y * fy, f[0][2 * e], f[1][2 * e], f[2][2 * e]);
                    lm_split(q.x * fx, q.y * fy, f[0][2 * e + 1], f[1][2 * e + 1], f[2][2 * e + 1]);
                    lm_split(kj.x * gh_exp2((m.x - z.x) + (ml.x - zl.x)), kj.y * gh_exp2((m.y - z.y) + (ml.y - zl.y)),
                             b[0][e], b[1][e], b[2][e]);
                }
#pragma unroll
                for (int z = 0; z < 3; ++z)
#pragma unroll
                    for (int x = 2; x >= z; --x) mma_bf16(y[x], f[z], b[x - z][0], b[x - z][1]);
            }
            const int t = I + (lane & 3) * 2;
#pragma unroll
            for (int e = 0; e < 2; ++e) As[r * 65 + t + e] = beta[r] * ((y[2][e] + y[1][e]) + y[0][e]);
            *(float2*)(Pm + r * 64 + t) = make_float2((y[2][2] + y[1][2]) + y[0][2], (y[2][3] + y[1][3]) + y[0][3]);
        }
    } else {
        // a block below the diagonal a warp: (1, 0), (2, 0), (2, 1), (3, 0), (3, 1), (3, 2)
        const int w = warp - 10, I = w == 0 ? 1 : w < 3 ? 2 : 3, J = w - I * (I - 1) / 2;
        const int ra = 16 * I + (lane >> 2), ja = 16 * J + (lane >> 2);
        const float over1 = J < 1 && I > 1, over2 = J < 2 && I > 2;     // whole blocks between the two
        float s[2][4] = {}, p[2][4] = {};
#pragma unroll 2
        for (int kk = 0; kk < UNITS; ++kk) {
            unsigned ak[3][4], aq[3][4], b[3][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = ra + (e & 1) * 8, c = 16 * kk + (e >> 1) * 8 + (lane & 3) * 2;
                const float2 x = *(const float2*)(bs + r * LD + c), k = *(const float2*)(ks + r * LD + c),
                             q = *(const float2*)(qs + r * LD + c);
                const float ex = gh_exp2(x.x), ey = gh_exp2(x.y);
                lm_split(k.x * ex, k.y * ey, ak[0][e], ak[1][e], ak[2][e]);
                lm_split(q.x * ex, q.y * ey, aq[0][e], aq[1][e], aq[2][e]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {                 // tokens ja, ja + 8; a pair of channels, and eight on
                const int j = ja + (e >> 1) * 8, c = 16 * kk + (e & 1) * 8 + (lane & 3) * 2;
                float2 x = *(const float2*)(fs + j * LD + c);
                const float2 m1 = *(const float2*)(tot + d + c), m2 = *(const float2*)(tot + 2 * d + c);
                x = make_float2(fmaf(over2, m2.x, fmaf(over1, m1.x, x.x)), fmaf(over2, m2.y, fmaf(over1, m1.y, x.y)));
                const float2 k = *(const float2*)(ks + j * LD + c);
                lm_split(k.x * gh_exp2(x.x), k.y * gh_exp2(x.y), b[0][e], b[1][e], b[2][e]);
            }
            lm_mma6x2(s[0], s[1], ak, b, p[0], p[1], aq, b);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = ra + 8 * e, t = 16 * J + 8 * i + (lane & 3) * 2;
                As[r * 65 + t] = beta[r] * s[i][2 * e];
                As[r * 65 + t + 1] = beta[r] * s[i][2 * e + 1];
                *(float2*)(Pm + r * 64 + t) = make_float2(p[i][2 * e], p[i][2 * e + 1]);
            }
    }
    for (int c = GH_THREADS - 1 - tid; c < d; c += GH_THREADS) {
        const float t[4] = {tot[c], tot[d + c], tot[2 * d + c], tot[3 * d + c]};
        pre[c] = 0.f; pre[d + c] = t[0]; pre[2 * d + c] = t[0] + t[1]; pre[3 * d + c] = (t[0] + t[1]) + t[2];
        post[3 * d + c] = 0.f; post[2 * d + c] = t[3]; post[d + c] = t[3] + t[2]; post[c] = (t[3] + t[2]) + t[1];
        g.dec[ih * d + c] = gh_exp2(((t[0] + t[1]) + t[2]) + t[3]);
    }
    __syncthreads();
    gc_inverse<GH_THREADS, false>(As, Xs);
    // q e^(B) and k e^(B): a thread has a lane's place in a fragment, rows j, j + 8 and channels c, c + 1,
    // c + 8, c + 9; k e^(B_L - B): channels c, c + 8 and tokens j, j + 1, j + 8, j + 9
    constexpr int SLOTS = 4 * UNITS * 32, OWN = (SLOTS + GH_THREADS - 1) / GH_THREADS;
    unsigned kp[OWN][4][3];
    {
        unsigned *Q = g.Q + ih * 3 * UNITS * 512, *K = g.K + ih * 3 * UNITS * 512;
#pragma unroll
        for (int u = 0; u < OWN; ++u) {
            const int x = tid + u * GH_THREADS, J = x / (UNITS * 32), kk = (x >> 5) - J * UNITS;
            if (x >= SLOTS) continue;
            unsigned w[4][3];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int j = 16 * J + (lane >> 2) + (e & 1) * 8, c = 16 * kk + (e >> 1) * 8 + (lane & 3) * 2;
                const float2 k = *(const float2*)(ks + j * LD + c), q = *(const float2*)(qs + j * LD + c),
                             b = *(const float2*)(bs + j * LD + c), before = *(const float2*)(pre + J * d + c);
                const float ex = gh_exp2(b.x + before.x), ey = gh_exp2(b.y + before.y);
                lm_split(k.x * ex, k.y * ey, kp[u][e][0], kp[u][e][1], kp[u][e][2]);
                lm_split(q.x * ex, q.y * ey, w[e][0], w[e][1], w[e][2]);
            }
#pragma unroll
            for (int s = 0; s < 3; ++s)
                *(uint4*)(Q + ((size_t)s * SLOTS + x) * 4) = make_uint4(w[0][s], w[1][s], w[2][s], w[3][s]);
        }
#pragma unroll
        for (int u = 0; u < OWN; ++u) {
            const int x = tid + u * GH_THREADS, un = x >> 7, J = (x >> 5) & 3;
            if (x >= SLOTS) continue;
            unsigned w[4][3];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int c = 16 * un + (e >> 1) * 8 + (lane >> 2), j = 16 * J + (e & 1) * 8 + (lane & 3) * 2;
                const float behind = post[J * d + c];
                lm_split(ks[j * LD + c] * gh_exp2(fs[j * LD + c] + behind),
                         ks[(j + 1) * LD + c] * gh_exp2(fs[(j + 1) * LD + c] + behind), w[e][0], w[e][1], w[e][2]);
            }
#pragma unroll
            for (int s = 0; s < 3; ++s)
                *(uint4*)(K + ((size_t)s * SLOTS + x) * 4) = make_uint4(w[0][s], w[1][s], w[2][s], w[3][s]);
        }
    }
    __syncthreads();                                      // keys and queries have been read
#pragma unroll
    for (int u = 0; u < OWN; ++u) {
        const int x = tid + u * GH_THREADS, J = x / (UNITS * 32), kk = (x >> 5) - J * UNITS;
        if (x >= SLOTS) continue;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int j = 16 * J + (lane >> 2) + (e & 1) * 8, c = 16 * kk + (e >> 1) * 8 + (lane & 3) * 2;
#pragma unroll
            for (int s = 0; s < 3; ++s) *(unsigned*)(kt + (s * 64 + j) * LD + c) = kp[u][e][s];
        }
    }
    {
        const int vq = dv >> 2;
#pragma unroll 4
        for (int x = tid; x < 64 * vq; x += GH_THREADS) {
            const int j = x / vq, c = (x - j * vq) * 4;
            float4 v = j < L ? *(const float4*)(base + (size_t)j * g.C + 2 * g.G * d + h * dv + c)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
            if (!gh_clean(v)) atomicMin(&bad, j);
            uint2 p[3];
            lm_split(v.x, v.y, p[0].x, p[1].x, p[2].x);
            lm_split(v.z, v.w, p[0].y, p[1].y, p[2].y);
#pragma unroll
            for (int s = 0; s < 3; ++s) *(uint2*)(vt + (s * 64 + j) * LV + c) = p[s];
        }
    }
    __syncthreads();
    if (tid == 0) g.bad[ih] = make_int4(bad, (int)bad_q[0], (int)bad_q[1], 0);
    // W and T V: a warp has 16 tokens and every fourth 16 columns, two of them at a time
    const int rg = warp & 3;
    unsigned a[4][3][4];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        if (kk > rg) continue;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = 16 * rg + (lane >> 2) + (e & 1) * 8, j = 16 * kk + (e >> 1) * 8 + (lane & 3) * 2;
            lm_split(Xs[r * 65 + j] * beta[j], Xs[r * 65 + j + 1] * beta[j + 1], a[kk][0][e], a[kk][1][e], a[kk][2][e]);
        }
    }
    unsigned* W = g.W + ih * 3 * 8 * UP * 128;
    float* V = g.V + ih * dv * 64;
    const int all = UNITS + (dv >> 4);
    for (int u0 = warp >> 2; u0 < all; u0 += 8) {
        const int u1 = u0 + 4 < all ? u0 + 4 : u0;
        const bf16* src[2] = {u0 < UNITS ? kt + 16 * u0 : vt + 16 * (u0 - UNITS),
                              u1 < UNITS ? kt + 16 * u1 : vt + 16 * (u1 - UNITS)};
        const int ld[2] = {u0 < UNITS ? LD : LV, u1 < UNITS ? LD : LV};
        float acc[2][2][4] = {};
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            if (kk > rg) continue;
            unsigned b[2][3][4];
#pragma unroll
            for (int z = 0; z < 2; ++z)
#pragma unroll
                for (int s = 0; s < 3; ++s)
                    ldmatrix_x4_trans(b[z][s], src[z] + (s * 64 + kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * ld[z] + (lane >> 4) * 8);
            lm_mma6x2(acc[0][0], acc[0][1], a[kk], b[0], acc[1][0], acc[1][1], a[kk], b[1]);
        }
#pragma unroll
        for (int z = 0; z < 2; ++z) {
            const int u = z ? u1 : u0;
            const float(&lo)[4] = acc[z][0];
            const float(&hi)[4] = acc[z][1];
            if (z && u1 == u0) continue;
            if (u < UNITS) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    unsigned x[3], y[3];
                    lm_split(lo[2 * e], lo[2 * e + 1], x[0], x[1], x[2]);
                    lm_split(hi[2 * e], hi[2 * e + 1], y[0], y[1], y[2]);
#pragma unroll
                    for (int s = 0; s < 3; ++s)
                        *(uint2*)(W + ((s * 8 + 2 * rg + e) * UP + (u >> 1)) * 128 + lane * 4 + (u & 1) * 2) = make_uint2(x[s], y[s]);
                }
            } else {
                float* o = V + (size_t)(16 * (u - UNITS) + (lane & 3) * 2) * 64 + 16 * rg + (lane >> 2);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    o[8 * e] = lo[2 * e];
                    o[64 + 8 * e] = lo[2 * e + 1];
                    o[8 * 64 + 8 * e] = hi[2 * e];
                    o[9 * 64 + 8 * e] = hi[2 * e + 1];
                }
            }
        }
    }
}

// S^T lies in accumulators, 16 columns by d rows: warp w has rows 16 w.. (and corrects tokens 8 w..).  A
// chunk's operands are requested as soon as the registers of the one before are free: W while the
// state is updated, K and the others while U is formed.
template <int UNITS>
__global__ void __launch_bounds__(256) gch_scan_kernel(const GhArgs g, float* __restrict__ state, long long rec,
                                                       int taps) {
    rv_pdl_launch_dependents();
    constexpr int d = 16 * UNITS, LK = d + 8, UP = (UNITS + 1) / 2;
    __shared__ __align__(16) bf16 ss[3 * GC_COLS * LK];   // the state
    __shared__ __align__(16) bf16 us[3 * GC_COLS * GC_LT];
    __shared__ int first_item;
    const int dv = g.dv, col_blocks = dv / GC_COLS;
    const int h = blockIdx.x / col_blocks, cb = blockIdx.x - h * col_blocks, c0 = cb * GC_COLS;
    const int r = g.first_req + blockIdx.y;
    const int slot = g.state_slot[r], n = la_chunks(g.q_start, g.state_slot, r);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 32) {
        int before = 0;
        for (int b = g.first_req + tid; b < r; b += 32) before += la_chunks(g.q_start, g.state_slot, b);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
        if (tid == 0) first_item = before;
    }
    __syncthreads();
    rv_pdl_wait();
    if (n == 0) return;
    const bool mine = warp < UNITS;                       // this warp has rows of the state
    const int ca = lane >> 2, row = 16 * warp + (lane & 3) * 2, tok = 8 * warp + (lane & 3) * 2;
    float* Sg = state + (size_t)slot * rec + (size_t)(taps - 1) * g.C + ((size_t)h * dv + c0) * d;
    float S[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            S[i][e] = mine ? Sg[(size_t)(ca + (e >> 1) * 8) * d + row + 8 * i + (e & 1)] : 0.f;
    uint4 w[3][UP], k[3][4];
    float2 v[2], keep[2];
    int bad = LA_C;
    auto get_w = [&](size_t ih) {
        const unsigned* W = g.W + ih * 3 * 8 * UP * 128 + lane * 4;
#pragma unroll
        for (int s = 0; s < 3; ++s)
#pragma unroll
            for (int u = 0; u < UP; ++u) w[s][u] = *(const uint4*)(W + ((s * 8 + warp) * UP + u) * 128);
        const float* V = g.V + (ih * dv + c0 + ca) * 64 + tok;
        v[0] = *(const float2*)V;
        v[1] = *(const float2*)(V + 8 * 64);
    };
    auto get_k = [&](size_t ih) {
        if (!mine) return;
        const unsigned* K = g.K + ih * 3 * UNITS * 512 + lane * 4;
#pragma unroll
        for (int s = 0; s < 3; ++s)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) k[s][kk] = *(const uint4*)(K + ((s * UNITS + warp) * 4 + kk) * 128);
        keep[0] = *(const float2*)(g.dec + ih * d + row);
        keep[1] = *(const float2*)(g.dec + ih * d + row + 8);
        bad = g.bad[ih].x;
    };
    const size_t step = g.H;
    size_t ih = (size_t)first_item * g.H + h;
    get_w(ih);
    get_k(ih);
    for (int c = 0; c < n; ++c, ih += step) {
        // the state before the chunk
        if (mine) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                unsigned x[3], y[3];
                lm_split(S[0][2 * e], S[0][2 * e + 1], x[0], x[1], x[2]);
                lm_split(S[1][2 * e], S[1][2 * e + 1], y[0], y[1], y[2]);
#pragma unroll
                for (int s = 0; s < 3; ++s) {
                    bf16* p = ss + (s * GC_COLS + ca + 8 * e) * LK + row;
                    *(unsigned*)p = x[s];
                    *(unsigned*)(p + 8) = y[s];
                }
            }
        }
        __syncthreads();
        // (W S)^T for this warp's eight tokens
        float y[3][4] = {};
        uint4 left[3];
#pragma unroll
        for (int kk = 0; kk < UNITS; ++kk) {
            unsigned a[3][4];
#pragma unroll
            for (int s = 0; s < 3; ++s)
                ldmatrix_x4(a[s], ss + (s * GC_COLS + (lane & 15)) * LK + kk * 16 + (lane >> 4) * 8);
#pragma unroll
            for (int z = 0; z < 3; ++z)
#pragma unroll
                for (int x = 2; x >= z; --x) {
                    const uint4 b = w[x - z][kk >> 1];
                    mma_bf16(y[x], a[z], kk & 1 ? b.z : b.x, kk & 1 ? b.w : b.y);
                }
            // for gch_out: its operand of columns 8 e.. and 32 rows of the state is half of what two such
            // fragments hold, so a warp that has both leaves it, 16 bytes a lane
            const int e = warp & 1;
            if (warp >> 1 == kk >> 1 && kk >> 1 < UP) {
                if (!(kk & 1)) {
#pragma unroll
                    for (int s = 0; s < 3; ++s) left[s] = make_uint4(e ? a[s][1] : a[s][0], e ? a[s][3] : a[s][2], 0u, 0u);
                } else {
#pragma unroll
                    for (int s = 0; s < 3; ++s) {
                        left[s].z = e ? a[s][1] : a[s][0];
                        left[s].w = e ? a[s][3] : a[s][2];
                    }
                }
            }
        }
        if (warp >> 1 < UP) {
            unsigned* to = g.S + (ih * col_blocks + cb) * 3 * 2 * UP * 128 + ((warp & 1) * UP + (warp >> 1)) * 128 + lane * 4;
#pragma unroll
            for (int s = 0; s < 3; ++s) *(uint4*)(to + s * 2 * UP * 128) = left[s];
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            unsigned x[3];
            lm_split(v[e].x - ((y[2][2 * e] + y[1][2 * e]) + y[0][2 * e]),
                     v[e].y - ((y[2][2 * e + 1] + y[1][2 * e + 1]) + y[0][2 * e + 1]), x[0], x[1], x[2]);
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                *(unsigned*)(us + (s * GC_COLS + ca + 8 * e) * GC_LT + tok) = x[s];
            }
        }
        if (c + 1 < n) get_w(ih + step);
        __syncthreads();
        if (warp < 4) {                                   // U in the same way, 32 tokens and 8 columns a warp
            unsigned* to = g.U + (ih * col_blocks + cb) * 3 * 2 * 2 * 128 + ((warp & 1) * 2 + (warp >> 1)) * 128 + lane * 4;
            const bf16* from = us + (8 * (warp & 1) + ca) * GC_LT + 32 * (warp >> 1) + (lane & 3) * 2;
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const bf16* f = from + s * GC_COLS * GC_LT;
                *(uint4*)(to + s * 2 * 2 * 128) = make_uint4(*(const unsigned*)f, *(const unsigned*)(f + 8),
                                                             *(const unsigned*)(f + 16), *(const unsigned*)(f + 24));
            }
        }
        if (mine) {
            float l[3][2][4] = {};
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                unsigned a[3][4];
#pragma unroll
                for (int s = 0; s < 3; ++s)
                    ldmatrix_x4(a[s], us + (s * GC_COLS + (lane & 15)) * GC_LT + kk * 16 + (lane >> 4) * 8);
#pragma unroll
                for (int z = 0; z < 3; ++z)
#pragma unroll
                    for (int x = 2; x >= z; --x) {
                        mma_bf16(l[x][0], a[z], k[x - z][kk].x, k[x - z][kk].y);
                        mma_bf16(l[x][1], a[z], k[x - z][kk].z, k[x - z][kk].w);
                    }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    S[i][e] = bad < LA_C ? __int_as_float(0x7fc00000)
                                         : fmaf(e & 1 ? keep[i].y : keep[i].x, S[i][e], (l[2][i][e] + l[1][i][e]) + l[0][i][e]);
        }
        if (c + 1 < n) get_k(ih + step);
    }
    if (mine)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) Sg[(size_t)(ca + (e >> 1) * 8) * d + row + 8 * i + (e & 1)] = S[i][e];
}

template <int UNITS>
__global__ void __launch_bounds__(128) gch_out_kernel(const GhArgs g, float* __restrict__ o_out) {
    rv_pdl_launch_dependents();
    constexpr int UP = (UNITS + 1) / 2;
    __shared__ int at[2];
    const int lane = threadIdx.x & 31, rg = threadIdx.x >> 5;
    const int item = blockIdx.x, h = blockIdx.y, dv = g.dv, blocks = dv >> 4, cb0 = 2 * blockIdx.z;
    const int nb = min(2, blocks - cb0);                  // (one: it is worked twice, and stored once)
    lm_locate(g.q_start, g.state_slot, g.first_req, g.n_reqs, item, at);
    const int t0 = at[0], L = at[1];
    rv_pdl_wait();
    if (t0 < 0 || 16 * rg >= L) return;
    const size_t ih = (size_t)item * g.H + h;
    const int row_a = 16 * rg + (lane >> 2), row_b = row_a + 8;
    float o[2][2][4] = {};
    // 16 columns' operand `e` of the pair that a lane has 16 bytes of, for both blocks of 16
    auto product = [&](const unsigned (&a)[3][4], const uint4 (&b)[2][3][2], int e) {
        unsigned f[2][3][4];
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                f[x][s][0] = e ? b[x][s][0].z : b[x][s][0].x;
                f[x][s][1] = e ? b[x][s][0].w : b[x][s][0].y;
                f[x][s][2] = e ? b[x][s][1].z : b[x][s][1].x;
                f[x][s][3] = e ? b[x][s][1].w : b[x][s][1].y;
            }
        lm_mma6x2(o[0][0], o[0][1], a, f[0], o[1][0], o[1][1], a, f[1]);
    };
    const unsigned* Q = g.Q + ih * 3 * UNITS * 512 + (size_t)rg * UNITS * 128 + lane * 4;
    const unsigned* S = g.S + (ih * blocks + cb0) * 3 * 2 * UP * 128 + lane * 4;
#pragma unroll 1
    for (int u = 0; u < UP; ++u) {
        uint4 q[2][3], b[2][3][2];
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            q[0][s] = *(const uint4*)(Q + (s * 4 * UNITS + 2 * u) * 128);
            if (2 * u + 1 < UNITS) q[1][s] = *(const uint4*)(Q + (s * 4 * UNITS + 2 * u + 1) * 128);
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    b[x][s][t] = *(const uint4*)(S + (((min(x, nb - 1) * 3 + s) * 2 + t) * UP + u) * 128);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (2 * u + e >= UNITS) continue;
            unsigned a[3][4];
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                a[s][0] = q[e][s].x; a[s][1] = q[e][s].y; a[s][2] = q[e][s].z; a[s][3] = q[e][s].w;
            }
            product(a, b, e);
        }
    }
    const float* Pm = g.Pm + ih * 64 * 64;
    const unsigned* U = g.U + (ih * blocks + cb0) * 3 * 2 * 2 * 128 + lane * 4;
#pragma unroll 1
    for (int u = 0; 2 * u <= rg; ++u) {
        uint4 b[2][3][2];
#pragma unroll
        for (int s = 0; s < 3; ++s)
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    b[x][s][t] = *(const uint4*)(U + (((min(x, nb - 1) * 3 + s) * 2 + t) * 2 + u) * 128);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int kk = 2 * u + e;
            if (kk > rg) continue;
            unsigned a[3][4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int r = x & 1 ? row_b : row_a, j = 16 * kk + (x >> 1) * 8 + (lane & 3) * 2;
                // (what lies above the diagonal's tiles of two by two was never written)
                const float2 p = j <= r ? *(const float2*)(Pm + r * 64 + j) : make_float2(0.f, 0.f);
                lm_split(p.x, j + 1 <= r ? p.y : 0.f, a[0][x], a[1][x], a[2][x]);
            }
            product(a, b, e);
        }
    }
    const int4 bad = g.bad[ih];
    const unsigned bad_q = row_a & 32 ? (unsigned)bad.z : (unsigned)bad.y;
    const float nan = __int_as_float(0x7fc00000);
    if (row_a >= bad.x || (bad_q >> (row_a & 31) & 1u))
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int t = 0; t < 2; ++t) o[x][t][0] = o[x][t][1] = nan;
    if (row_b >= bad.x || (bad_q >> (row_b & 31) & 1u))
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int t = 0; t < 2; ++t) o[x][t][2] = o[x][t][3] = nan;
    float* dst = o_out + ((size_t)t0 * g.H + h) * dv + 16 * cb0 + (lane & 3) * 2;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        if (x >= nb) continue;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            if (row_a < L) *(float2*)(dst + (size_t)row_a * g.H * dv + 16 * x + 8 * t) = make_float2(o[x][t][0], o[x][t][1]);
            if (row_b < L) *(float2*)(dst + (size_t)row_b * g.H * dv + 16 * x + 8 * t) = make_float2(o[x][t][2], o[x][t][3]);
        }
    }
}

// ---------------------------------------------------------------------------------
static size_t gh_chunk_smem(int d, int dv) {
    const size_t in = (size_t)4 * 64 * (d + 8) * 4, parts = (size_t)3 * 64 * (d + 8 + dv + 8) * 2;
    return ((size_t)2 * 64 * 65 + 12 * d) * 4 + (in > parts ? in : parts);
}
// Which sizes the chunk form takes; the rows' alignment is looked at beside the pointers.
static bool gh_sizes_ok(int H, int G, int d, int dv) {
    return d % 16 == 0 && d <= 128 && dv % 16 == 0 && (2 * G * d + H * dv) % 4 == 0 && gh_chunk_smem(d, dv) <= 220 * 1024;
}
// (Some 7.5 KB a token and head of 128 by 128, 3.6 times the form token by token: 490 MB for 8,192 tokens of 8 heads,
// 980 MB of 16.)
struct GhScratch {
    long long rows, logs, W, K, Q, S, U, Pm, V, dec, bad, total;   // in floats, every part a multiple of four
};
static GhScratch gh_layout(int n_tokens, long long items, int H, int d, int dv, int C) {
    const long long ih = items * H, units = d / 16, up = (units + 1) / 2;
    GhScratch s;
    s.rows = 0;
    s.logs = ((long long)n_tokens * C + 3) & ~3LL;
    s.W = s.logs + (long long)n_tokens * H * d;
    s.K = s.W + ih * 3 * 8 * up * 128;
    s.Q = s.K + ih * 3 * units * 512;
    s.S = s.Q + ih * 3 * units * 512;
    s.U = s.S + ih * (dv / 16) * 3 * 2 * up * 128;
    s.Pm = s.U + ih * (dv / 16) * 3 * 2 * 2 * 128;
    s.V = s.Pm + ih * 64 * 64;
    s.dec = s.V + ih * dv * 64;
    s.bad = s.dec + ih * d;
    s.total = s.bad + ih * 4;
    return s;
}

template <int UNITS>
static int gh_launch(const GhArgs& g, long long items, float* state, long long rec, int taps, float* o, cudaStream_t s) {
    const size_t sm = gh_chunk_smem(g.d, g.dv);
    GC_SMEM(gch_chunk_kernel<UNITS>, sm)
    rv_launch(gch_chunk_kernel<UNITS>, dim3((unsigned)items, g.H), dim3(GH_THREADS), sm, s, g);
    RV_CHECK_LAUNCH("gated_delta chunk");
    rv_launch(gch_scan_kernel<UNITS>, dim3(g.H * (g.dv / GC_COLS), g.n_reqs - g.first_req), dim3(256), 0, s, g, state, rec, taps);
    RV_CHECK_LAUNCH("gated_delta scan");
    rv_launch(gch_out_kernel<UNITS>, dim3((unsigned)items, g.H, (g.dv / 16 + 1) / 2), dim3(128), 0, s, g, o);
    RV_CHECK_LAUNCH("gated_delta out");
    return 0;
}

// Portions of requests [first_req, n_reqs), tokens [first_token, n_tokens): o [n, H dv].
static int gh_run(GhArgs g, const float* filt, float* state, long long rec, int taps, const int* token_req,
                  int first_token, int n_tokens, float* scratch, float* o, cudaStream_t s) {
    const long long items = la_items(n_tokens - first_token, g.n_reqs - g.first_req);
    if (items > 65535LL * 32) RV_FAIL("gated_delta: too many tokens");
    const GhScratch lay = gh_layout(n_tokens, items, g.H, g.d, g.dv, g.C);
    g.rows = scratch + lay.rows;
    g.logs = scratch + lay.logs;
    g.W = (unsigned*)(scratch + lay.W);
    g.K = (unsigned*)(scratch + lay.K);
    g.Q = (unsigned*)(scratch + lay.Q);
    g.S = (unsigned*)(scratch + lay.S);
    g.U = (unsigned*)(scratch + lay.U);
    g.Pm = scratch + lay.Pm;
    g.V = scratch + lay.V;
    g.dec = scratch + lay.dec;
    g.bad = (int4*)(scratch + lay.bad);
    const long long count = (long long)(n_tokens - first_token) * g.H * g.d;
    rv_launch(gch_logs_kernel, dim3((unsigned)((count + 1023) / 1024)), dim3(256), 0, s, g, scratch + lay.logs, first_token, count);
    RV_CHECK_LAUNCH("gated_delta decays");
    const ConvSilu conv = {g.proj, filt, nullptr, state, rec, token_req, g.q_start, g.state_slot, g.P, 0,
                           first_token, n_tokens, g.C, taps};
    conv_silu<float>(conv, scratch + lay.rows, s);
    RV_CHECK_LAUNCH("gated_delta conv");
    switch (g.d >> 4) {
        case 1: return gh_launch<1>(g, items, state, rec, taps, o, s);
        case 2: return gh_launch<2>(g, items, state, rec, taps, o, s);
        case 3: return gh_launch<3>(g, items, state, rec, taps, o, s);
        case 4: return gh_launch<4>(g, items, state, rec, taps, o, s);
        case 5: return gh_launch<5>(g, items, state, rec, taps, o, s);
        case 6: return gh_launch<6>(g, items, state, rec, taps, o, s);
        case 7: return gh_launch<7>(g, items, state, rec, taps, o, s);
        default: return gh_launch<8>(g, items, state, rec, taps, o, s);
    }
}
