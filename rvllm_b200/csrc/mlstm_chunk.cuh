// The matrix memory of mlstm.cu over portions in chunks of 64 tokens, on the tensor cores (bfloat16
// output; included by mlstm.cu, whose first comment has the recurrence).
//
// For a head and the tokens 0..63 of a chunk let F_t be the sum of the log forget gates up to and
// with token t, m_t the running maximum, m_0 the one before the chunk and C_0 the memory before it.
// Unrolled, with a_t = F_t - m_t and c_j = F_j - li_j,
//
//     C_t^T q_t = e^(a_t + m_0) C_0^T q_t + sum_(j <= t) e^(a_t - c_j) <q_t, k_j> v_j
//     C_L       = e^(a_L + m_0) C_0       + sum_j        e^(a_L - c_j) k_j v_j^T
//
// and m_t = F_t + max(m_0, max_(j <= t) (li_j - F_j)), so no exponent is above 0.  n is the column
// whose values are 1.
//
//   mlc_gates   block per (request, head): the gates of all tokens, F and m as prefix sums and
//               maxima -> a, c [n, H] float64 (their differences stay exact
//               behind a token that forgets all), m and e^(-m) [n, H]
//   mlc_state   block per (chunk, head): sum_j e^(a_L - c_j) k_j v_j^T and the column of n
//   mlc_scan    over the chunks of a request one after another, elementwise: the memory before every
//               chunk takes the place of the chunk's sum, the last one is the record
//   mlc_out     block per (chunk, head): scores, both terms, the division, the head's norm, weight
//               and gate
//
// The rows are float32 and stay so: operands enter the bfloat16 products as three parts each
// (chunks.cuh), six of the nine products, which reach a float32's last bits.
//
// A value that is not finite reaches no earlier token: mlc_out takes it as 0, and the head's outputs from its
// token on are NaN, as are those of all later chunks by the memory.  (Weights of later tokens are 0 by choice, not
// by a product, so keys and gates need no such care; a bad query is its own row.)
//
// The scan is a chain of some 64 instructions a token; here the only chain is mlc_scan's one
// multiply-add a chunk, and mlc_out, the longest kernel (32 of 53 us for portions of 492 and 1,309
// tokens), waits for its loads (30 % of a scheduler's cycles issue; its products keep the tensor pipe
// 17 % busy).  8 heads of 64 by 128, one call: 2,048 tokens 283 -> 59 us, 492 + 1,309 tokens 182 -> 53,
// 4 x 512 tokens of 16 heads 191 -> 98, keys of 128 442 -> 99.
#pragma once
#include "chunks.cuh"

// Threads of a block of mlc_state (two a value column) and mlc_out (128 for 64 columns) at most: values of
// 256.  Stated as a bound, so that the registers of that many always fit.
#define MLC_THREADS 512

struct MlChunk {
    const float *rows, *bi, *bf, *norm_w;
    const int *q_start, *state_slot;
    float* state;
    double *a, *c;               // [n, H]
    float *m, *em;               // [n, H]: the running maximum and e^-m
    float* m_start;              // [n_reqs, H]: the record's maximum before the step
    float* keep;                 // [items, H]: e^(a_L + m_0)
    float* kv;                   // [items, H, dv + 1, d]
    void* out;
    long long rec;
    int stride, first_req, n_reqs, H, d, dv;
    float cap, eps;
};

// Where a chunk lies: first token, token count (0: no such chunk), request, its number in the request.
// Without a chunk, at[2] is how many chunks there are.
__device__ __forceinline__ void mlc_locate(const MlChunk& g, int item, int* at) {
    if (threadIdx.x < 32) {
        int r = -1, before = 0;
        const bool ok = la_find(g.q_start, g.state_slot, g.first_req, g.n_reqs, item, threadIdx.x, r, before);
        if (threadIdx.x == 0) {
            at[0] = ok ? g.q_start[r] + (item - before) * LA_C : -1;
            at[1] = ok ? min(LA_C, g.q_start[r + 1] - at[0]) : 0;
            at[2] = ok ? r : before;
            at[3] = item - before;
        }
    }
    __syncthreads();
}
__device__ __forceinline__ float mlc_before(const MlChunk& g, const int* at, int h) {
    return at[3] == 0 ? g.m_start[(size_t)at[2] * g.H + h] : g.m[(size_t)(at[0] - 1) * g.H + h];
}

// Two tokens a thread: a block of up to 1,024 threads, a multiple of 32, works so many at a time.
__global__ void __launch_bounds__(1024) mlc_gates_kernel(const MlChunk g) {
    rv_pdl_launch_dependents();
    const int r = g.first_req + blockIdx.x, h = blockIdx.y;
    const int slot = g.state_slot[r], a0 = g.q_start[r], a1 = g.q_start[r + 1];
    const float b_i = g.bi[h], b_f = g.bf[h];
    const int i_off = 2 * g.H * g.d + g.H * g.dv + h, f_off = i_off + g.H;
    __shared__ double part[2][32];               // the warps' sums, then their maxima
    __shared__ double at_chunk[32];              // the sum before every chunk of the round
    __shared__ float m_end;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    rv_pdl_wait();
    if (slot < 0 || a1 <= a0) return;
    float* m_rec = g.state + (size_t)slot * g.rec + g.rec - g.H + h;
    double m0 = *m_rec;
    if (tid == 0) g.m_start[(size_t)r * g.H + h] = (float)m0;
    const int round = 2 * blockDim.x;
    for (int c0 = a0; c0 < a1; c0 += round) {
        const int n = min(round, a1 - c0);
        float li[2], lf[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {            // two neighbouring tokens a thread
            const int t = 2 * tid + e;
            const float* row = g.rows + (size_t)(c0 + min(t, n - 1)) * g.stride;
            li[e] = g.cap * tanhf((row[i_off] + b_i) / g.cap);
            lf[e] = ml_logsigmoid(g.cap * tanhf((row[f_off] + b_f) / g.cap));
        }
        double F[2] = {lf[0], (double)lf[0] + (double)lf[1]};
        double incl = F[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) part[0][warp] = incl;
        // (the sum before this pair, not the sum minus the pair: its second gate may be a NaN)
        double before = __shfl_up_sync(0xffffffffu, incl, 1);
        if (lane == 0) before = 0.;
        __syncthreads();
        for (int w = 0; w < warp; ++w) before += part[0][w];
        F[0] += before;
        F[1] += before;
        if ((2 * tid) % LA_C == 0) at_chunk[2 * tid / LA_C] = before;
        double x[2] = {(double)li[0] - F[0], (double)li[1] - F[1]};
        x[1] = fmax(x[0], x[1]);
        double top = x[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, top, o);
            if (lane >= o) top = fmax(top, up);
        }
        if (lane == 31) part[1][warp] = top;
        double high = __shfl_up_sync(0xffffffffu, top, 1);
        if (lane == 0) high = m0;
        __syncthreads();
        high = fmax(high, m0);
        for (int w = 0; w < warp; ++w) high = fmax(high, part[1][w]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = 2 * tid + e;
            const float m = (float)(F[e] + fmax(high, x[e]));
            if (t < n) {
                const size_t to = (size_t)(c0 + t) * g.H + h;
                const double f = F[e] - at_chunk[t / LA_C];
                g.a[to] = f - (double)m;
                g.c[to] = f - (double)li[e];
                g.m[to] = m;
                g.em[to] = expf(-m);
                if (t == n - 1) m_end = m;
            }
        }
        __syncthreads();
        m0 = m_end;
    }
    if (tid == 0) *m_rec = (float)m0;
}

// Whether all four can be taken into three parts; if not they are 0 from here on.
__device__ __forceinline__ bool mlc_clean(float4& v) {
    const bool ok = fabsf(v.x) <= 3.3895313e38f && fabsf(v.y) <= 3.3895313e38f && fabsf(v.z) <= 3.3895313e38f &&
                    fabsf(v.w) <= 3.3895313e38f;              // the largest bfloat16
    if (!ok) v = make_float4(0.f, 0.f, 0.f, 0.f);
    return ok;
}
// Four neighbouring float32 values times f as three parts, to `dst`, `dst + step` and `dst + 2 step`.
__device__ __forceinline__ void mlc_put4(bf16* dst, int step, float4 x, float f) {
    uint2 p[3];
    lm_split(x.x * f, x.y * f, p[0].x, p[1].x, p[2].x);
    lm_split(x.z * f, x.w * f, p[0].y, p[1].y, p[2].y);
#pragma unroll
    for (int s = 0; s < 3; ++s) *(uint2*)(dst + s * step) = p[s];
}
// A warp has 16 columns of the values by all d rows.
template <int D16>
__global__ void __launch_bounds__(MLC_THREADS) mlc_state_kernel(const MlChunk g) {
    rv_pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr int d = 16 * D16, LK = d + 8;
    const int dv = g.dv, LV = dv + 8, threads = blockDim.x;
    bf16* ks = (bf16*)smraw;                     // [3][64][LK]: k e^(a_L - c_j)
    bf16* vs = ks + 3 * LA_C * LK;               // [3][64][LV]
    __shared__ float w[LA_C];
    __shared__ int at[4];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int item = blockIdx.x, h = blockIdx.y;
    mlc_locate(g, item, at);
    const int t0 = at[0], L = at[1];
    rv_pdl_wait();
    if (t0 < 0) return;
    for (int j = tid; j < LA_C; j += threads)
        w[j] = j < L ? expf((float)(g.a[(size_t)(t0 + L - 1) * g.H + h] - g.c[(size_t)(t0 + j) * g.H + h])) : 0.f;
    if (tid == 0)
        g.keep[(size_t)item * g.H + h] = expf((float)(g.a[(size_t)(t0 + L - 1) * g.H + h] + (double)mlc_before(g, at, h)));
    __syncthreads();
    const float* base = g.rows + (size_t)t0 * g.stride;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int x = tid; x < LA_C * (d / 4); x += threads) {
        const int j = x / (d / 4), c = (x - j * (d / 4)) * 4;
        mlc_put4(ks + j * LK + c, LA_C * LK,
                 j < L ? *(const float4*)(base + (size_t)j * g.stride + (g.H + h) * d + c) : zero, w[j]);
    }
    const int vq = dv >> 2;
#pragma unroll 4
    for (int x = tid; x < LA_C * vq; x += threads) {
        const int j = x / vq, c = (x - j * vq) * 4;
        mlc_put4(vs + j * LV + c, LA_C * LV,
                 j < L ? *(const float4*)(base + (size_t)j * g.stride + 2 * g.H * d + h * dv + c) : zero, 1.f);
    }
    __syncthreads();
    float acc[2 * D16][4];
#pragma unroll
    for (int i = 0; i < 2 * D16; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    const int nk = (L + 15) >> 4;
    for (int kk = 0; kk < nk; ++kk) {
        unsigned a[3][4];
#pragma unroll
        for (int s = 0; s < 3; ++s)
            ldmatrix_x4_trans(a[s], vs + (s * LA_C + kk * 16 + (lane & 7) + (lane >> 4) * 8) * LV + 16 * warp +
                                        ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int nd = 0; nd < D16; ++nd) {
            unsigned b[3][4];
#pragma unroll
            for (int s = 0; s < 3; ++s)
                ldmatrix_x4_trans(b[s], ks + (s * LA_C + kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LK + nd * 16 +
                                            (lane >> 4) * 8);
            lm_mma6(acc[2 * nd], acc[2 * nd + 1], a, b);
        }
    }
    float* kv = g.kv + ((size_t)item * g.H + h) * (dv + 1) * d;
    float* o = kv + (size_t)(16 * warp + (lane >> 2)) * d + (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < 2 * D16; ++i) {
        *(float2*)(o + 8 * i) = make_float2(acc[i][0], acc[i][1]);
        *(float2*)(o + (size_t)8 * d + 8 * i) = make_float2(acc[i][2], acc[i][3]);
    }
    for (int c = tid; c < d; c += threads) {     // the column of n: the parts of a value add up to it
        float s = 0.f;
        for (int j = 0; j < L; ++j)
            s += (__bfloat162float(ks[j * LK + c]) + __bfloat162float(ks[(LA_C + j) * LK + c])) +
                 __bfloat162float(ks[(2 * LA_C + j) * LK + c]);
        kv[(size_t)dv * d + c] = s;
    }
}

__global__ void __launch_bounds__(128) mlc_scan_kernel(const MlChunk g) {
    rv_pdl_launch_dependents();
    const int h = blockIdx.y, r = g.first_req + blockIdx.z;
    const int slot = g.state_slot[r], n = la_chunks(g.q_start, g.state_slot, r);
    __shared__ int first_item;
    if (threadIdx.x < 32) {
        int before = 0;
        for (int b = g.first_req + threadIdx.x; b < r; b += 32) before += la_chunks(g.q_start, g.state_slot, b);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
        if (threadIdx.x == 0) first_item = before;
    }
    __syncthreads();
    rv_pdl_wait();
    const long long size = (long long)(g.dv + 1) * g.d, el = ((long long)blockIdx.x * 128 + threadIdx.x) * 4;
    if (n == 0 || el >= size) return;
    float* rec = g.state + (size_t)slot * g.rec + (size_t)h * size + el;
    float* p = g.kv + ((size_t)first_item * g.H + h) * size + el;
    const size_t step = (size_t)g.H * size;
    const bool wide = ((uintptr_t)rec & 15) == 0;
    float4 S = wide ? *(const float4*)rec : make_float4(rec[0], rec[1], rec[2], rec[3]);
    const float* kp = g.keep + (size_t)first_item * g.H + h;
    constexpr int U = 12;                        // chunks requested together
    for (int c0 = 0; c0 < n; c0 += U) {
        float4 in[U];
        float keep[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c0 + u < n) {
                in[u] = *(const float4*)(p + (size_t)(c0 + u) * step);
                keep[u] = kp[(size_t)(c0 + u) * g.H];
            }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c0 + u < n) {
                *(float4*)(p + (size_t)(c0 + u) * step) = S;
                S.x = fmaf(keep[u], S.x, in[u].x);
                S.y = fmaf(keep[u], S.y, in[u].y);
                S.z = fmaf(keep[u], S.z, in[u].z);
                S.w = fmaf(keep[u], S.w, in[u].w);
            }
    }
    if (wide) {
        *(float4*)rec = S;
    } else {
        rec[0] = S.x; rec[1] = S.y; rec[2] = S.z; rec[3] = S.w;
    }
}

// Four warps have 16 tokens each; as many groups of four as there are 64 columns.  The values take the
// memory's place in shared memory once it has been read.
template <int D16>
__global__ void __launch_bounds__(MLC_THREADS) mlc_out_kernel(const MlChunk g) {
    rv_pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr int d = 16 * D16, LK = d + 8;
    const int dv = g.dv, LV = dv + 8, threads = blockDim.x, groups = threads >> 7;
    bf16* qs = (bf16*)smraw;                     // [3][64][LK]
    bf16* ks = qs + 3 * LA_C * LK;               // [3][64][LK]
    bf16* ss = ks + 3 * LA_C * LK;               // [3][dv][LK]: the memory's columns; then vs [3][64][LV]
    bf16* vs = ss;
    __shared__ double at_[LA_C], ct[LA_C];
    __shared__ float f0[LA_C], em[LA_C], qn[LA_C], sq[4][LA_C], n0[16 * D16];
    __shared__ int at[4], bad;                   // bad: the first token with a value that is not finite
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rg = warp & 3, cg = warp >> 2;
    const int item = blockIdx.x, h = blockIdx.y;
    if (tid == 0) bad = LA_C;
    mlc_locate(g, item, at);
    const int t0 = at[0], L = at[1];
    rv_pdl_wait();
    bf16* out = (bf16*)g.out;
    if (t0 < 0) {
        // a block without a chunk (there is one whenever there are tokens of requests without a slot):
        // such tokens' rows are zeros, dealt out over these blocks
        const int used = at[2], spare = item - used, spares = gridDim.x - used;
        for (int r = g.first_req; r < g.n_reqs; ++r) {
            if (g.state_slot[r] >= 0) continue;
            for (int t = g.q_start[r] + spare; t < g.q_start[r + 1]; t += spares)
                for (int c = tid * 2; c < dv; c += threads * 2)
                    *(unsigned*)(out + ((size_t)t * g.H + h) * dv + c) = 0u;
        }
        return;
    }
    const float* base = g.rows + (size_t)t0 * g.stride;
    const float* S0 = g.kv + ((size_t)item * g.H + h) * (dv + 1) * d;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tid < LA_C) {
        const size_t p = (size_t)(t0 + min(tid, L - 1)) * g.H + h;
        at_[tid] = g.a[p];
        ct[tid] = g.c[p];
        em[tid] = g.em[p];
        f0[tid] = expf((float)(g.a[p] + (double)mlc_before(g, at, h)));
    }
    for (int c = tid; c < d; c += threads) n0[c] = S0[(size_t)dv * d + c];
    // queries, keys and the memory: a quarter of a row's floats a thread and access, eight requested
    // before any is split
    const int rows_all = 2 * LA_C + dv;
    for (int x0 = tid; x0 < rows_all * (d / 4); x0 += 8 * threads) {
        float4 in[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int x = x0 + u * threads, j = x / (d / 4), c = (x - j * (d / 4)) * 4, t = j & (LA_C - 1);
            in[u] = zero;
            if (j < 2 * LA_C) {
                if (t < L) in[u] = *(const float4*)(base + (size_t)t * g.stride + ((j >> 6) * g.H + h) * d + c);
            } else if (j < rows_all) {
                in[u] = *(const float4*)(S0 + (size_t)(j - 2 * LA_C) * d + c);
            }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int x = x0 + u * threads, j = x / (d / 4), c = (x - j * (d / 4)) * 4;
            if (j < 2 * LA_C) mlc_put4((j < LA_C ? qs + j * LK : ks + (j - LA_C) * LK) + c, LA_C * LK, in[u], 1.f);
            else if (j < rows_all) mlc_put4(ss + (j - 2 * LA_C) * LK + c, dv * LK, in[u], 1.f);
        }
    }
    __syncthreads();
    if (tid < 2 * LA_C) {                        // <q, n_0> of every token, two lanes each
        const int j = tid >> 1;
        const float* row = base + (size_t)min(j, L - 1) * g.stride + h * d;
        float s = 0.f;
        for (int c = 4 * (tid & 1); c < d; c += 8) {
            const float4 x = *(const float4*)(row + c);
            s = fmaf(x.x, n0[c], fmaf(x.y, n0[c + 1], fmaf(x.z, n0[c + 2], fmaf(x.w, n0[c + 3], s))));
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if ((tid & 1) == 0) qn[j] = s;
    }
    float p[8][4], o[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) p[i][e] = o[i][e] = 0.f;
#pragma unroll
    for (int kk = 0; kk < D16; ++kk) {
        unsigned a[3][4];
#pragma unroll
        for (int s = 0; s < 3; ++s)
            ldmatrix_x4(a[s], qs + (s * LA_C + 16 * rg + (lane & 15)) * LK + kk * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int nb = 0; nb < 4; ++nb) {         // scores: keys up to the warp's own tokens
            if (nb > rg) continue;
            unsigned b[3][4];
#pragma unroll
            for (int s = 0; s < 3; ++s)
                ldmatrix_x4(b[s], ks + (s * LA_C + nb * 16 + (lane & 7) + (lane >> 4) * 8) * LK + kk * 16 + ((lane >> 3) & 1) * 8);
            lm_mma6(p[2 * nb], p[2 * nb + 1], a, b);
        }
#pragma unroll
        for (int nd = 0; nd < 4; ++nd) {         // the memory's share
            const int c = 64 * cg + 16 * nd;
            if (c >= dv) continue;
            unsigned b[3][4];
#pragma unroll
            for (int s = 0; s < 3; ++s)
                ldmatrix_x4(b[s], ss + (s * dv + c + (lane & 7) + (lane >> 4) * 8) * LK + kk * 16 + ((lane >> 3) & 1) * 8);
            lm_mma6(o[2 * nd], o[2 * nd + 1], a, b);
        }
    }
    __syncthreads();                             // the memory has been read
    {
        const int vq = dv >> 2;
        for (int x0 = tid; x0 < LA_C * vq; x0 += 8 * threads) {
            float4 in[8];
            int to[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int x = x0 + u * threads, j = x / vq, c = (x - j * vq) * 4;
                to[u] = j < LA_C ? j * LV + c : -1;
                in[u] = j < L ? *(const float4*)(base + (size_t)j * g.stride + 2 * g.H * d + h * dv + c) : zero;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (to[u] >= 0) {
                    // (an earlier token's weight of it is 0, and 0 times it must be 0)
                    if (!mlc_clean(in[u])) atomicMin(&bad, to[u] / LV);
                    mlc_put4(vs + to[u], LA_C * LV, in[u], 1.f);
                }
        }
    }
    const int row_a = 16 * rg + (lane >> 2), row_b = row_a + 8;      // this thread's tokens
    const float fa = f0[row_a], fb = f0[row_b];
    float den_a = 0.f, den_b = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        o[i][0] *= fa; o[i][1] *= fa;
        o[i][2] *= fb; o[i][3] *= fb;
        if (i > 2 * rg + 1) continue;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int t = e < 2 ? row_a : row_b, j = 8 * i + (lane & 3) * 2 + (e & 1);
            p[i][e] = j <= t ? p[i][e] * expf((float)(at_[t] - ct[j])) : 0.f;
            (e < 2 ? den_a : den_b) += p[i][e];
        }
    }
    __syncthreads();                             // the values are there
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        if (kk > rg) continue;
        unsigned a[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = 2 * kk + (e >> 1);
            lm_split(p[i][(e & 1) * 2], p[i][(e & 1) * 2 + 1], a[0][e], a[1][e], a[2][e]);
        }
#pragma unroll
        for (int nd = 0; nd < 4; ++nd) {
            const int c = 64 * cg + 16 * nd;
            if (c >= dv) continue;
            unsigned b[3][4];
#pragma unroll
            for (int s = 0; s < 3; ++s)
                ldmatrix_x4_trans(b[s], vs + (s * LA_C + kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LV + c + (lane >> 4) * 8);
            lm_mma6(o[2 * nd], o[2 * nd + 1], a, b);
        }
    }
    // the division, then the norm over the head's columns (a warp has 64 of them)
    const float q_scale = 1.f / sqrtf((float)d);
    float ss_a = 0.f, ss_b = 0.f;
#pragma unroll
    for (int x = 1; x <= 2; x <<= 1) {
        den_a += __shfl_xor_sync(0xffffffffu, den_a, x);
        den_b += __shfl_xor_sync(0xffffffffu, den_b, x);
    }
    // (One division a row and products by it: a float32 rounding more than mlstm_finish's divisions, which
    // the bfloat16 output's error against float64 does not show; dividing every value took mlc_out from 33
    // to 37 us.  The gate is divided: its divisor goes beyond 2^126, where the fast division gives 0.)
    const float by_a = q_scale / (fmaxf(fabsf(fmaf(fa, qn[row_a], den_a) * q_scale), em[row_a]) + 1e-6f);
    const float by_b = q_scale / (fmaxf(fabsf(fmaf(fb, qn[row_b], den_b) * q_scale), em[row_b]) + 1e-6f);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            o[i][e] *= by_a;
            o[i][2 + e] *= by_b;
            ss_a = fmaf(o[i][e], o[i][e], ss_a);
            ss_b = fmaf(o[i][2 + e], o[i][2 + e], ss_b);
        }
#pragma unroll
    for (int x = 1; x <= 2; x <<= 1) {
        ss_a += __shfl_xor_sync(0xffffffffu, ss_a, x);
        ss_b += __shfl_xor_sync(0xffffffffu, ss_b, x);
    }
    if ((lane & 3) == 0) {
        sq[cg][row_a] = ss_a;
        sq[cg][row_b] = ss_b;
    }
    __syncthreads();
    ss_a = ss_b = 0.f;
    for (int x = 0; x < groups; ++x) {
        ss_a += sq[x][row_a];
        ss_b += sq[x][row_b];
    }
    const float ra = 1.f / sqrtf(ss_a / (float)dv + g.eps), rb = 1.f / sqrtf(ss_b / (float)dv + g.eps);
    const float* gate = base + 2 * g.H * d + g.H * dv + 2 * g.H + h * dv;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int c = 64 * cg + 8 * i + (lane & 3) * 2;
        if (c >= dv) continue;
        const float w0 = g.norm_w[h * dv + c], w1 = g.norm_w[h * dv + c + 1];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = e ? row_b : row_a;
            if (t >= L) continue;
            const float2 gt = *(const float2*)(gate + (size_t)t * g.stride + c);
            const float r = t >= bad ? __int_as_float(0x7fc00000) : e ? rb : ra;
            *(unsigned*)(out + ((size_t)(t0 + t) * g.H + h) * dv + c) =
                pack_bf16(o[i][2 * e] * r * w0 / (1.f + expf(-gt.x)), o[i][2 * e + 1] * r * w1 / (1.f + expf(-gt.y)));
        }
    }
}

static size_t mlc_state_smem(int d, int dv) { return (size_t)3 * LA_C * (d + 8 + dv + 8) * 2; }
static size_t mlc_out_smem(int d, int dv) {
    const size_t mem = (size_t)dv * (d + 8), val = (size_t)LA_C * (dv + 8);
    return ((size_t)2 * LA_C * (d + 8) + (mem > val ? mem : val)) * 3 * 2;
}
// Sizes that the chunk form takes: bfloat16 output; heads in multiples of 16, keys up to 128, values up
// to 256, within shared memory; rows and heads on 16-byte boundaries.
static bool mlc_ok(const float* rows, int stride, int out_dtype, int H, int d, int dv, const void* out) {
    return out_dtype == RV_DTYPE_BF16 && d % 16 == 0 && d <= 128 && dv % 16 == 0 && 2 * dv <= MLC_THREADS &&
           stride % 4 == 0 && ((uintptr_t)rows & 15) == 0 && ((uintptr_t)out & 3) == 0 &&
           mlc_out_smem(d, dv) <= 224 * 1024 && mlc_state_smem(d, dv) <= 224 * 1024;
}
// Floats of scratch for portions of n tokens in n_reqs requests.
static long long mlc_scratch(int n, int n_reqs, int H, int d, int dv) {
    return (long long)n * H * 6 + (long long)n_reqs * H + la_items(n, n_reqs) * H * (1 + (dv + 1) * d) + 16;
}

template <int D16>
static int mlc_launch(const MlChunk& g, int n, int items, int threads, int groups, cudaStream_t s) {
    const size_t sm1 = mlc_state_smem(g.d, g.dv), sm2 = mlc_out_smem(g.d, g.dv);
    cudaError_t e = cudaFuncSetAttribute(mlc_state_kernel<D16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm1);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlc_out_kernel<D16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2);
    if (e != cudaSuccess) RV_FAIL("mlstm: %s", cudaGetErrorString(e));
    const int n_reqs = g.n_reqs - g.first_req;
    // as many threads as the longest portion can use
    const int half = (n + 63) / 64 * 32;
    rv_launch(mlc_gates_kernel, dim3(n_reqs, g.H), dim3(half < 1024 ? half : 1024), 0, s, g);
    RV_CHECK_LAUNCH("mlstm_gates");
    rv_launch(mlc_state_kernel<D16>, dim3(items, g.H), dim3(threads), sm1, s, g);
    RV_CHECK_LAUNCH("mlstm_state");
    const long long size = (long long)(g.dv + 1) * g.d;
    rv_launch(mlc_scan_kernel, dim3((unsigned)((size / 4 + 127) / 128), g.H, n_reqs), dim3(128), 0, s, g);
    RV_CHECK_LAUNCH("mlstm_scan");
    rv_launch(mlc_out_kernel<D16>, dim3(items, g.H), dim3(128 * groups), sm2, s, g);
    RV_CHECK_LAUNCH("mlstm_out");
    return 0;
}
static int mlc_run(const MlChunk& g, int n, cudaStream_t s) {
    const int items = (int)la_items(n, g.n_reqs - g.first_req), groups = (g.dv + 63) / 64, threads = 2 * g.dv;
    switch (g.d >> 4) {
        case 1: return mlc_launch<1>(g, n, items, threads, groups, s);
        case 2: return mlc_launch<2>(g, n, items, threads, groups, s);
        case 3: return mlc_launch<3>(g, n, items, threads, groups, s);
        case 4: return mlc_launch<4>(g, n, items, threads, groups, s);
        case 5: return mlc_launch<5>(g, n, items, threads, groups, s);
        case 6: return mlc_launch<6>(g, n, items, threads, groups, s);
        case 7: return mlc_launch<7>(g, n, items, threads, groups, s);
        default: return mlc_launch<8>(g, n, items, threads, groups, s);
    }
}
