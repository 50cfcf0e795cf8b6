// The tensor-core forms of linear_attention.cu's `state` and `out` kernels (bfloat16 rows, d and dv
// in multiples of 16, d up to 128); included by that file, whose first comment explains them.
#pragma once

#define LM_LD 72            // padded row of 64 bfloat16 columns
#define LM_LK 136           // padded row of 128

__device__ __forceinline__ unsigned lm_silu2(unsigned u) {
    const float2 f = lm_pair(u);
    const __nv_bfloat162 r = __floats2bfloat162_rn(la_silu(f.x), la_silu(f.y));
    return *(const unsigned*)&r;
}
// Eight projections of one token, as the recurrence reads them.
__device__ __forceinline__ uint4 lm_in8(const bf16* p, bool there, int act) {
    uint4 v = there ? *(const uint4*)p : make_uint4(0, 0, 0, 0);
    if (act) {
        v.x = lm_silu2(v.x);
        v.y = lm_silu2(v.y);
        v.z = lm_silu2(v.z);
        v.w = lm_silu2(v.w);
    }
    return v;
}
__device__ __forceinline__ float lm_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// z -> B: what the tokens of a chunk up to and with this one keep of a channel, as a power of two
// (sums of log2 a), in place, so that neither of the kernels below repeats it for its tiles.  A
// warp has eight tokens of 32 channels.
#define LM_STRONG -57.7f    // -40 log2 e
__global__ void __launch_bounds__(256) la_decay_kernel(float* __restrict__ z, const float* __restrict__ bias,
                                                       float scale, const int* __restrict__ q_start,
                                                       const int* __restrict__ state_slot, int first_req,
                                                       int n_reqs, int width) {
    rv_pdl_launch_dependents();
    __shared__ float tot[8][32];
    __shared__ int at[2];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, c = blockIdx.y * 32 + lane;
    if (threadIdx.x < 32) {
        int r = -1, before = 0;
        const bool ok = la_find(q_start, state_slot, first_req, n_reqs, blockIdx.x, lane, r, before);
        if (lane == 0) {
            at[0] = ok ? q_start[r] + ((int)blockIdx.x - before) * LA_C : -1;
            at[1] = ok ? min(LA_C, q_start[r + 1] - at[0]) : 0;
        }
    }
    __syncthreads();
    const int t0 = at[0], L = at[1];
    const float b = c < width ? bias[c] : 0.f;
    rv_pdl_wait();
    if (t0 < 0) return;
    float v[8], s = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        v[j] = 8 * g + j < L && c < width ? z[(size_t)(t0 + 8 * g + j) * width + c] : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        s += la_logsigmoid(v[j] + b) * scale;
        v[j] = s;
    }
    tot[g][lane] = s;
    __syncthreads();
    float before = 0.f;
    for (int i = 0; i < g; ++i) before += tot[i][lane];
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (8 * g + j < L && c < width) z[(size_t)(t0 + 8 * g + j) * width + c] = before + v[j];
}

// KV = sum_j (k_j e^(B_L - B_j)) v_j^T for 64 channels by 64 columns: a warp has 16 channels.
// (Decays by channel.)
__global__ void __launch_bounds__(128) la_state_mma_kernel(
    const bf16* __restrict__ rows, int stride, const LaRows lr, const float* __restrict__ zb,
    const int* __restrict__ q_start, const int* __restrict__ state_slot, int first_req, int n_reqs,
    float* __restrict__ kv, float* __restrict__ dec, int H, int d, int dv, int act) {
    rv_pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char smraw[];
    bf16* ks = (bf16*)smraw;                            // [3][64 tokens][LM_LD]
    bf16* vs = ks + 3 * LA_C * LM_LD;                   // [64 tokens][LM_LD]
    __shared__ int at[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int item = blockIdx.x, h = blockIdx.y;
    const int tiles_v = (dv + LA_T - 1) / LA_T;
    const int d0 = (blockIdx.z / tiles_v) * LA_T, v0 = (blockIdx.z % tiles_v) * LA_T;
    lm_locate(q_start, state_slot, first_req, n_reqs, item, at);
    const int t0 = at[0], L = at[1];
    rv_pdl_wait();
    if (t0 < 0) return;
    const int dn = min(LA_T, d - d0), vn = min(LA_T, dv - v0);
    const bf16* base = rows + (size_t)t0 * stride;
    const int kh = h / lr.share;
    // eight columns a thread: 8 chunks a row, 16 rows a round, 4 rounds
    const int ch = tid & 7, jr = tid >> 3;
    uint4 kreg[4], vreg[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int j = jr + 16 * u;
        const bf16* row = base + (size_t)j * stride;
        kreg[u] = lm_in8(row + lr.k + kh * d + d0 + 8 * ch, j < L && 8 * ch < dn, act);
        vreg[u] = lm_in8(row + lr.v + h * dv + v0 + 8 * ch, j < L && 8 * ch < vn, act);
    }
    float bl[8];                                        // B of the chunk's last token
    {
        const float* p = zb + (size_t)(t0 + L - 1) * H * d + h * d + d0;
#pragma unroll
        for (int e = 0; e < 8; ++e) bl[e] = 8 * ch < dn ? p[8 * ch + e] : 0.f;
        if (v0 == 0 && jr == 0 && 8 * ch < dn)
#pragma unroll
            for (int e = 0; e < 8; ++e)
                dec[((size_t)item * H + h) * d + d0 + 8 * ch + e] = lm_exp2(bl[e]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int j = jr + 16 * u;
        *(uint4*)(vs + j * LM_LD + 8 * ch) = vreg[u];
        const unsigned in[4] = {kreg[u].x, kreg[u].y, kreg[u].z, kreg[u].w};
        unsigned o[3][4];
        float bj[8];
        {
            const float* p = zb + (size_t)(t0 + min(j, L - 1)) * H * d + h * d + d0 + 8 * ch;
#pragma unroll
            for (int e = 0; e < 8; e += 4) {
                const float4 x = 8 * ch < dn ? *(const float4*)(p + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                bj[e] = x.x; bj[e + 1] = x.y; bj[e + 2] = x.z; bj[e + 3] = x.w;
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 k2 = lm_pair(in[e]);
            const float fx = lm_exp2(bl[2 * e] - bj[2 * e]), fy = lm_exp2(bl[2 * e + 1] - bj[2 * e + 1]);
            lm_split(k2.x * fx, k2.y * fy, o[0][e], o[1][e], o[2][e]);
        }
#pragma unroll
        for (int s = 0; s < 3; ++s)
            *(uint4*)(ks + (s * LA_C + j) * LM_LD + 8 * ch) = make_uint4(o[s][0], o[s][1], o[s][2], o[s][3]);
    }
    __syncthreads();
    if (16 * warp >= dn) return;
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    const int nk = (L + 15) >> 4;
    for (int kk = 0; kk < nk; ++kk) {
        unsigned a[3][4];
#pragma unroll
        for (int s = 0; s < 3; ++s)
            ldmatrix_x4_trans(a[s], ks + (s * LA_C + kk * 16 + (lane & 7) + (lane >> 4) * 8) * LM_LD +
                                        16 * warp + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int nd = 0; nd < 4; ++nd) {
            if (16 * nd >= vn) continue;
            unsigned b[4];
            ldmatrix_x4_trans(b, vs + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LM_LD + nd * 16 + (lane >> 4) * 8);
#pragma unroll
            for (int s = 2; s >= 0; --s) {
                mma_bf16(acc[2 * nd], a[s], b[0], b[1]);
                mma_bf16(acc[2 * nd + 1], a[s], b[2], b[3]);
            }
        }
    }
    float* o = kv + ((size_t)item * H + h) * d * dv + (size_t)(d0 + 16 * warp + (lane >> 2)) * dv + v0 + (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (8 * i >= vn) continue;
        *(float2*)(o + 8 * i) = make_float2(acc[i][0], acc[i][1]);
        *(float2*)(o + (size_t)8 * dv + 8 * i) = make_float2(acc[i][2], acc[i][3]);
    }
}

// (B in powers of two here: zb is what la_decay left.)
// o = (scores, masked) V + (q e^(B_i)) S for the chunk's 64 tokens by 64 columns: a warp has 16
// tokens.  B is kept whole (bs), q e^(B_i) is formed in fragments, k e^(-B_j) in shared memory.
__global__ void __launch_bounds__(128) la_out_mma_kernel(
    const bf16* __restrict__ rows, int stride, const LaRows lr, const float* __restrict__ zb,
    const int* __restrict__ q_start, const int* __restrict__ state_slot, int first_req, int n_reqs,
    const float* __restrict__ kv, float* __restrict__ num, int H, int d, int dv, int act, float q_scale) {
    rv_pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char smraw[];
    const int LQ = d + 8, LB = d + 2;
    bf16* ss = (bf16*)smraw;                            // [3][d][LM_LD]: the state's columns
    bf16* vs = ss + 3 * d * LM_LD;                      // [64][LM_LD]
    bf16* qs = vs + LA_C * LM_LD;                       // [64][LQ]
    bf16* ks = qs + LA_C * LQ;                          // [3][64][LQ]
    float* bs = (float*)(ks + 3 * LA_C * LQ);           // [64][LB]
    __shared__ int at[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int item = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * LA_T;
    lm_locate(q_start, state_slot, first_req, n_reqs, item, at);
    const int t0 = at[0], L = at[1];
    rv_pdl_wait();
    if (t0 < 0) return;
    const int kh = h / lr.share;
    const int vn = min(LA_T, dv - v0);
    const bf16* base = rows + (size_t)t0 * stride;
    // values, queries, keys: eight columns a thread and access
    {
        const int ch = tid & 7, jr = tid >> 3;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int j = jr + 16 * u;
            *(uint4*)(vs + j * LM_LD + 8 * ch) =
                lm_in8(base + (size_t)j * stride + lr.v + h * dv + v0 + 8 * ch, j < L && 8 * ch < vn, act);
        }
        const int cpr = d >> 3;                         // chunks a row
#pragma unroll 4
        for (int n = tid; n < LA_C * cpr; n += 128) {
            const int j = n / cpr, c = (n - j * cpr) * 8;
            const bf16* row = base + (size_t)j * stride + kh * d + c;
            *(uint4*)(qs + j * LQ + c) = lm_in8(row + lr.q, j < L, act);
            *(uint4*)(ks + j * LQ + c) = lm_in8(row + lr.k, j < L, act);
        }
    }
    // the state before the chunk, in three parts
    {
        const float* S = kv + ((size_t)item * H + h) * d * dv + v0;
        const int c = (tid & 15) * 4;
#pragma unroll 4
        for (int r = tid >> 4; r < d; r += 8) {
            const float4 x = c < vn ? *(const float4*)(S + (size_t)r * dv + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            uint2 p[3];
            lm_split(x.x, x.y, p[0].x, p[1].x, p[2].x);
            lm_split(x.z, x.w, p[0].y, p[1].y, p[2].y);
#pragma unroll
            for (int s = 0; s < 3; ++s) *(uint2*)(ss + (s * d + r) * LM_LD + c) = p[s];
        }
    }
    bool strong;
    {
        const int cpr = d >> 2;
        bool low = false;
#pragma unroll 4
        for (int n = tid; n < LA_C * cpr; n += 128) {
            const int j = n / cpr, c = (n - j * cpr) * 4;
            const float4 x = *(const float4*)(zb + (size_t)(t0 + min(j, L - 1)) * H * d + h * d + c);
            *(float2*)(bs + j * LB + c) = make_float2(x.x, x.y);
            *(float2*)(bs + j * LB + c + 2) = make_float2(x.z, x.w);
            low |= fminf(fminf(x.x, x.y), fminf(x.z, x.w)) < LM_STRONG;
        }
        strong = __syncthreads_or(low);
        if (!strong) {
#pragma unroll 2
            for (int n = tid; n < LA_C * (d >> 1); n += 128) {
                const int j = n / (d >> 1), c = (n - j * (d >> 1)) * 2;
                unsigned* k0 = (unsigned*)(ks + j * LQ + c);
                const float2 k2 = lm_pair(*k0), b2 = *(const float2*)(bs + j * LB + c);
                unsigned p[3];
                lm_split(k2.x * lm_exp2(-b2.x), k2.y * lm_exp2(-b2.y), p[0], p[1], p[2]);
                k0[0] = p[0];
                *(unsigned*)(ks + LA_C * LQ + j * LQ + c) = p[1];
                *(unsigned*)(ks + 2 * LA_C * LQ + j * LQ + c) = p[2];
            }
        }
    }
    __syncthreads();
    const int row_a = 16 * warp + (lane >> 2), row_b = row_a + 8;   // this thread's tokens
    if (16 * warp >= L) return;
    float p[8][4], o[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) p[i][e] = o[i][e] = 0.f;
    for (int kk = 0; kk < (d >> 4); ++kk) {
        unsigned a[3][4];
        ldmatrix_x4(a[0], qs + (16 * warp + (lane & 15)) * LQ + kk * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 q2 = lm_pair(a[0][e]);
            const float2 b2 = *(const float2*)(bs + ((e & 1) ? row_b : row_a) * LB + kk * 16 + (e >> 1) * 8 + (lane & 3) * 2);
            lm_split(q2.x * lm_exp2(b2.x), q2.y * lm_exp2(b2.y), a[0][e], a[1][e], a[2][e]);
        }
        // scores: keys up to the warp's own tokens
        if (!strong) {
#pragma unroll
            for (int nb = 0; nb < 4; ++nb) {
                if (nb > warp) continue;
                unsigned b[3][4];
#pragma unroll
                for (int s = 0; s < 3; ++s)
                    ldmatrix_x4(b[s], ks + (s * LA_C + nb * 16 + (lane & 7) + (lane >> 4) * 8) * LQ + kk * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
                for (int x = 2; x >= 0; --x)                         // smallest products first
#pragma unroll
                    for (int y = 0; y <= x; ++y) {
                        mma_bf16(p[2 * nb], a[y], b[x - y][0], b[x - y][1]);
                        mma_bf16(p[2 * nb + 1], a[y], b[x - y][2], b[x - y][3]);
                    }
            }
        }
        // the state's share
#pragma unroll
        for (int nd = 0; nd < 4; ++nd) {
            if (16 * nd >= vn) continue;
            unsigned b[3][4];
#pragma unroll
            for (int s = 0; s < 3; ++s)
                ldmatrix_x4_trans(b[s], ss + (s * d + kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LM_LD + nd * 16 + (lane >> 4) * 8);
#pragma unroll
            for (int x = 2; x >= 0; --x)
#pragma unroll
                for (int y = 0; y <= x; ++y) {
                    mma_bf16(o[2 * nd], a[y], b[x - y][0], b[x - y][1]);
                    mma_bf16(o[2 * nd + 1], a[y], b[x - y][2], b[x - y][3]);
                }
        }
    }
    // a chunk with strong decays: every pair's own difference
    if (strong) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (i > 2 * warp + 1) continue;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = e < 2 ? row_a : row_b, j = 8 * i + (lane & 3) * 2 + (e & 1);
                float s = 0.f;
                if (j <= r)
                    for (int c = 0; c < d; ++c)
                        s = fmaf(__bfloat162float(qs[r * LQ + c]) * __bfloat162float(ks[j * LQ + c]),
                                 lm_exp2(bs[r * LB + c] - bs[j * LB + c]), s);
                p[i][e] = s;
            }
        }
    }
    // the mask, then the values
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        if (kk > warp) continue;
        unsigned a[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = 2 * kk + (e >> 1), r = (e & 1) ? row_b : row_a, j = 8 * i + (lane & 3) * 2;
            float x = p[i][(e & 1) * 2], y = p[i][(e & 1) * 2 + 1];
            x = j <= r ? x : 0.f;
            y = j + 1 <= r ? y : 0.f;
            lm_split(x, y, a[0][e], a[1][e], a[2][e]);
        }
#pragma unroll
        for (int nd = 0; nd < 4; ++nd) {
            if (16 * nd >= vn) continue;
            unsigned b[4];
            ldmatrix_x4_trans(b, vs + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LM_LD + nd * 16 + (lane >> 4) * 8);
#pragma unroll
            for (int s = 2; s >= 0; --s) {
                mma_bf16(o[2 * nd], a[s], b[0], b[1]);
                mma_bf16(o[2 * nd + 1], a[s], b[2], b[3]);
            }
        }
    }
    float* dst = num + ((size_t)t0 * H + h) * dv + v0 + (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (8 * i >= vn) continue;
        if (row_a < L)
            *(float2*)(dst + (size_t)row_a * H * dv + 8 * i) = make_float2(o[i][0] * q_scale, o[i][1] * q_scale);
        if (row_b < L)
            *(float2*)(dst + (size_t)row_b * H * dv + 8 * i) = make_float2(o[i][2] * q_scale, o[i][3] * q_scale);
    }
}

// ---- one decay per head (a constant, or made by every token) ------------------------------------
// Every token's share of the state is weighed by one factor, so the values carry it and the keys stay
// as they are; and a group's heads share keys, queries and their products.  A block takes `heads` heads
// of one group, one after another, whose keys and queries it reads once.
//
// Bound by mma.sync (1.1 ns a product and multiprocessor, 7 of 19.5 us in `state` and 11 of 32 in `out`) and by
// blocks that load at the same time.  32 heads of 64 columns with one group's keys of 128, 2,048 tokens, against a
// block per head (and 64 channels) with the keys or the state split in shared memory: `state` 22 -> 19.5 us, `out` 53 -> 32.
//
// Values lie in shared memory with the even columns of every sixteen first and the odd ones
// behind them: column n of the first and of the second of two neighbouring products are then columns 2 n and
// 2 n + 1, and a thread's four outputs of a row lie side by side.
__device__ __forceinline__ void lm_store_dealt(bf16* row, int ch, const unsigned (&even)[2], const unsigned (&odd)[2]) {
    bf16* to = row + (ch >> 1) * 16 + (ch & 1) * 4;
    *(uint2*)to = make_uint2(even[0], even[1]);
    *(uint2*)(to + 8) = make_uint2(odd[0], odd[1]);
}

// KV = sum_j k_j (f_j v_j)^T, f_j = e^(B_L - B_j) w_j, for up to 128 channels by 64 columns: a warp has two
// times 16 channels, the scaled values lie in three parts.
template <int MODE>
__global__ void __launch_bounds__(128, 4) la_state_heads_kernel(
    const bf16* __restrict__ rows, int stride, const LaRows lr, const LaToken tk, const float* __restrict__ log_decay,
    const int* __restrict__ q_start, const int* __restrict__ state_slot, int first_req, int n_reqs,
    float* __restrict__ kv, int H, int d, int dv, int act, int heads) {
    constexpr bool TOKEN = MODE == LA_TOKEN;
    rv_pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char smraw[];
    bf16* ks = (bf16*)smraw;                            // [64 tokens][LM_LK]
    bf16* vs = ks + LA_C * LM_LK;                       // [3][64 tokens][LM_LD]
    __shared__ int at[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int item = blockIdx.x, h0 = blockIdx.y * heads;
    const int tiles_v = (dv + LA_T - 1) / LA_T;
    const int d0 = (blockIdx.z / tiles_v) * 128, v0 = (blockIdx.z % tiles_v) * LA_T;
    lm_locate(q_start, state_slot, first_req, n_reqs, item, at);
    const int t0 = at[0], L = at[1];
    rv_pdl_wait();
    if (t0 < 0) return;
    const int dn = min(128, d - d0), vn = min(LA_T, dv - v0);
    const bf16* base = rows + (size_t)t0 * stride;
    {
        const bf16* k = base + lr.k + (h0 / lr.share) * d + d0;
        const int cpr = dn >> 3;
#pragma unroll 8
        for (int n = tid; n < LA_C * cpr; n += 128) {
            const int j = n / cpr, c = (n - j * cpr) * 8;
            *(uint4*)(ks + j * LM_LK + c) = lm_in8(k + (size_t)j * stride + c, j < L, act);
        }
    }
    const int ch = tid & 7, jr = tid >> 3;              // eight columns of a token a thread, four rounds
    uint4 v[4];
    float f[4];
    auto get = [&](int h) {
        const double last = TOKEN ? tk.B[(size_t)(t0 + L - 1) * H + h] : 0.;
        const float ld = TOKEN ? 0.f : log_decay[h];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int j = jr + 16 * u, jj = min(j, L - 1);
            v[u] = lm_in8(base + (size_t)j * stride + lr.v + h * dv + v0 + 8 * ch, j < L && 8 * ch < vn, act);
            const size_t at_j = (size_t)(t0 + jj) * H + h;
            f[u] = TOKEN ? expf((float)(last - tk.B[at_j])) * tk.w[at_j] : expf(ld * (float)(L - 1 - jj));
        }
    };
    get(h0);
    const int nk = (L + 15) >> 4;
    for (int h = h0; h < h0 + heads; ++h) {
        if (h > h0) __syncthreads();                    // the head before has been used
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float2 a = lm_pair(v[u].x), b = lm_pair(v[u].y), c = lm_pair(v[u].z), e = lm_pair(v[u].w);
            unsigned even[3][2], odd[3][2];
            lm_split(a.x * f[u], b.x * f[u], even[0][0], even[1][0], even[2][0]);
            lm_split(c.x * f[u], e.x * f[u], even[0][1], even[1][1], even[2][1]);
            lm_split(a.y * f[u], b.y * f[u], odd[0][0], odd[1][0], odd[2][0]);
            lm_split(c.y * f[u], e.y * f[u], odd[0][1], odd[1][1], odd[2][1]);
#pragma unroll
            for (int s = 0; s < 3; ++s) lm_store_dealt(vs + (s * LA_C + jr + 16 * u) * LM_LD, ch, even[s], odd[s]);
        }
        __syncthreads();
        if (h + 1 < h0 + heads) get(h + 1);
        float acc[2][8][4];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[m][i][0] = acc[m][i][1] = acc[m][i][2] = acc[m][i][3] = 0.f;
        for (int kk = 0; kk < nk; ++kk) {
            unsigned a[2][4];
#pragma unroll
            for (int m = 0; m < 2; ++m)
                if (16 * (warp + 4 * m) < dn)
                    ldmatrix_x4_trans(a[m], ks + (kk * 16 + (lane & 7) + (lane >> 4) * 8) * LM_LK + 16 * (warp + 4 * m) + ((lane >> 3) & 1) * 8);
#pragma unroll
            for (int nd = 0; nd < 4; ++nd) {
                if (16 * nd >= vn) continue;
#pragma unroll
                for (int s = 2; s >= 0; --s) {
                    unsigned b[4];
                    ldmatrix_x4_trans(b, vs + (s * LA_C + kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LM_LD + nd * 16 + (lane >> 4) * 8);
#pragma unroll
                    for (int m = 0; m < 2; ++m)
                        if (16 * (warp + 4 * m) < dn) {
                            mma_bf16(acc[m][2 * nd], a[m], b[0], b[1]);
                            mma_bf16(acc[m][2 * nd + 1], a[m], b[2], b[3]);
                        }
                }
            }
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int c = 16 * (warp + 4 * m);
            if (c >= dn) continue;
            float* o = kv + (((size_t)item * H + h) * d + d0 + c + (lane >> 2)) * dv + v0 + (lane & 3) * 4;
#pragma unroll
            for (int nd = 0; nd < 4; ++nd) {
                if (16 * nd >= vn) continue;
                const float* x = acc[m][2 * nd], *y = acc[m][2 * nd + 1];
                *(float4*)(o + 16 * nd) = make_float4(x[0], y[0], x[1], y[1]);
                *(float4*)(o + (size_t)8 * dv + 16 * nd) = make_float4(x[2], y[2], x[3], y[3]);
            }
        }
    }
}

// o = (scores, weighed and masked) V + e^(B_i) q S for the chunk's 64 tokens by 64 columns.  The
// scores <q_i, k_j>, in blocks of 16 x 16 on and below the diagonal, are formed once and stay in
// registers; for every head their weighed values go to shared memory in three parts.  There a
// warp has 16 columns of all tokens, so that every value of the state is read once, by the thread
// that multiplies with it, and its parts never leave registers.
template <int MODE>
__global__ void __launch_bounds__(128, 4) la_out_heads_kernel(
    const bf16* __restrict__ rows, int stride, const LaRows lr, const LaToken tk, const float* __restrict__ log_decay,
    const int* __restrict__ q_start, const int* __restrict__ state_slot, int first_req, int n_reqs,
    const float* __restrict__ kv, float* __restrict__ num, int H, int d, int dv, int act, float q_scale, int heads) {
    constexpr bool TOKEN = MODE == LA_TOKEN;
    rv_pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char smraw[];
    const int LQ = d + 8;
    bf16* qs = (bf16*)smraw;                            // [64][LQ]
    bf16* vs = qs + LA_C * LQ;                          // [64][LM_LD]
    bf16* ks = vs + LA_C * LM_LD;                       // [64][LQ]; then
    bf16* ps = ks;                                      // [3][64][LM_LD]: the weighed scores
    __shared__ double bt[TOKEN ? 2 : 1][TOKEN ? LA_C : 1];      // TOKEN: B, of this head and of the next one
    __shared__ float pw[2][LA_C + 1];                   // TOKEN: the keys' weights; else the decay's powers
    __shared__ int at[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int item = blockIdx.x, h0 = blockIdx.y * heads, v0 = blockIdx.z * LA_T;
    lm_locate(q_start, state_slot, first_req, n_reqs, item, at);
    const int t0 = at[0], L = at[1];
    rv_pdl_wait();
    if (t0 < 0) return;
    const int vn = min(LA_T, dv - v0), nm = (L + 15) >> 4, nk = d >> 4;
    const bf16* base = rows + (size_t)t0 * stride;
    const int ch = tid & 7, jr = tid >> 3;
    uint4 v[4];
    auto get_v = [&](int h) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            v[u] = lm_in8(base + (size_t)(jr + 16 * u) * stride + lr.v + h * dv + v0 + 8 * ch, jr + 16 * u < L && 8 * ch < vn, act);
    };
    get_v(h0);
    {
        const bf16* row = base + (h0 / lr.share) * d;
        const int cpr = d >> 3;                         // pieces a row
#pragma unroll 4
        for (int n = tid; n < LA_C * cpr; n += 128) {
            const int j = n / cpr, c = (n - j * cpr) * 8;
            *(uint4*)(qs + j * LQ + c) = lm_in8(row + (size_t)j * stride + lr.q + c, j < L, act);
            *(uint4*)(ks + j * LQ + c) = lm_in8(row + (size_t)j * stride + lr.k + c, j < L, act);
        }
    }
    __syncthreads();
    // blocks of scores: warp, warp + 4 and warp + 8 of the ten, row by row of the triangle
    float sc[3][8];
    int bm[3], bn[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int b = warp + 4 * i;
        bm[i] = b >= 6 ? 3 : b >= 3 ? 2 : b >= 1 ? 1 : 0;
        bn[i] = b - bm[i] * (bm[i] + 1) / 2;
        if (b > 9) bm[i] = 4;                           // (none)
#pragma unroll
        for (int e = 0; e < 8; ++e) sc[i][e] = 0.f;
    }
    for (int kk = 0; kk < nk; ++kk) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (bm[i] >= nm) continue;
            unsigned a[4], b[4];
            ldmatrix_x4(a, qs + (16 * bm[i] + (lane & 15)) * LQ + kk * 16 + (lane >> 4) * 8);
            ldmatrix_x4(b, ks + (16 * bn[i] + (lane & 7) + (lane >> 4) * 8) * LQ + kk * 16 + ((lane >> 3) & 1) * 8);
            float lo[4] = {sc[i][0], sc[i][1], sc[i][2], sc[i][3]}, hi[4] = {sc[i][4], sc[i][5], sc[i][6], sc[i][7]};
            mma_bf16(lo, a, b[0], b[1]);
            mma_bf16(hi, a, b[2], b[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                sc[i][e] = lo[e];
                sc[i][4 + e] = hi[e];
            }
        }
    }
    const bool mine = 16 * warp < vn;                   // whether the warp has columns
    for (int h = h0; h < h0 + heads; ++h) {
        const int set = (h - h0) & 1;
        if (TOKEN && tid < LA_C) {
            const size_t at_j = (size_t)(t0 + min(tid, L - 1)) * H + h;
            bt[TOKEN ? set : 0][TOKEN ? tid : 0] = tk.B[at_j];
            pw[set][tid] = tid < L ? tk.w[at_j] : 0.f;
        }
        if (!TOKEN && tid <= LA_C) pw[set][tid] = expf(log_decay[h] * (float)tid);
        // the state: rows 16 kk + 2 t and + 1, + 8 and + 9, two columns, as the products read them; two steps ahead
        const float* S = kv + (((size_t)item * H + h) * d + (lane & 3) * 2) * dv + v0 + 16 * warp + (lane >> 2) * 2;
        auto get_s = [&](float2 (&x)[4], int kk) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (kk < nk && mine) x[e] = *(const float2*)(S + (size_t)(16 * kk + (e & 1) + (e >> 1) * 8) * dv);
        };
        float2 s0[4], s1[4];
        get_s(s0, 0);
        get_s(s1, 1);
        __syncthreads();                                // weights are here; the head before has been used (or the keys)
        auto pair = [&](int r, int j) {
            return TOKEN ? expf((float)(bt[TOKEN ? set : 0][TOKEN ? r : 0] - bt[TOKEN ? set : 0][TOKEN ? j : 0])) * pw[set][j] : pw[set][r - j];
        };
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (bm[i] >= nm) continue;
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                const int r = 16 * bm[i] + (lane >> 2) + (e & 2) * 4, j = 16 * bn[i] + (e >> 2) * 8 + (lane & 3) * 2;
                const float x = j <= r ? sc[i][e] * pair(r, j) : 0.f, y = j + 1 <= r ? sc[i][e + 1] * pair(r, j + 1) : 0.f;
                unsigned p[3];
                lm_split(x, y, p[0], p[1], p[2]);
#pragma unroll
                for (int s = 0; s < 3; ++s) *(unsigned*)(ps + (s * LA_C + r) * LM_LD + j) = p[s];
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const unsigned even[2] = {__byte_perm(v[u].x, v[u].y, 0x5410), __byte_perm(v[u].z, v[u].w, 0x5410)};
            const unsigned odd[2] = {__byte_perm(v[u].x, v[u].y, 0x7632), __byte_perm(v[u].z, v[u].w, 0x7632)};
            lm_store_dealt(vs + (jr + 16 * u) * LM_LD, ch, even, odd);
        }
        if (h + 1 < h0 + heads) get_v(h + 1);
        float o[4][8];
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int e = 0; e < 8; ++e) o[m][e] = 0.f;
        auto add = [&](float (&c)[8], const unsigned (&a)[4], const unsigned (&b)[4]) {
            float lo[4] = {c[0], c[1], c[2], c[3]}, hi[4] = {c[4], c[5], c[6], c[7]};
            mma_bf16(lo, a, b[0], b[1]);
            mma_bf16(hi, a, b[2], b[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                c[e] = lo[e];
                c[4 + e] = hi[e];
            }
        };
        auto share = [&](float2 (&x)[4], int kk) {      // q S of 16 rows of the state, and the next but one
            unsigned b[3][4];
            lm_split(x[0].x, x[1].x, b[0][0], b[1][0], b[2][0]);
            lm_split(x[2].x, x[3].x, b[0][1], b[1][1], b[2][1]);
            lm_split(x[0].y, x[1].y, b[0][2], b[1][2], b[2][2]);
            lm_split(x[2].y, x[3].y, b[0][3], b[1][3], b[2][3]);
            get_s(x, kk + 2);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                if (m >= nm) continue;
                unsigned a[4];
                ldmatrix_x4(a, qs + (16 * m + (lane & 15)) * LQ + kk * 16 + (lane >> 4) * 8);
#pragma unroll
                for (int s = 2; s >= 0; --s) add(o[m], a, b[s]);
            }
        };
        if (mine)
            for (int kk = 0; kk < nk; kk += 2) {
                share(s0, kk);
                if (kk + 1 < nk) share(s1, kk + 1);
            }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int r = 16 * m + (lane >> 2);
            const float fa = TOKEN ? expf((float)bt[TOKEN ? set : 0][TOKEN ? r : 0]) : pw[set][r + 1];
            const float fb = TOKEN ? expf((float)bt[TOKEN ? set : 0][TOKEN ? r + 8 : 0]) : pw[set][r + 9];
#pragma unroll
            for (int e = 0; e < 8; ++e) o[m][e] *= (e & 2) ? fb : fa;
        }
        __syncthreads();                                // scores and values are here
        if (!mine) continue;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            if (kk >= nm) continue;
            unsigned b[4];
            ldmatrix_x4_trans(b, vs + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LM_LD + warp * 16 + (lane >> 4) * 8);
#pragma unroll
            for (int m = kk; m < 4; ++m) {
                if (m >= nm) continue;
#pragma unroll
                for (int s = 2; s >= 0; --s) {
                    unsigned a[4];
                    ldmatrix_x4(a, ps + (s * LA_C + 16 * m + (lane & 15)) * LM_LD + kk * 16 + (lane >> 4) * 8);
                    add(o[m], a, b);
                }
            }
        }
        float* dst = num + ((size_t)t0 * H + h) * dv + v0 + 16 * warp + (lane & 3) * 4;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int r = 16 * m + (lane >> 2);
            const float* x = o[m];
            if (r < L)
                *(float4*)(dst + (size_t)r * H * dv) = make_float4(x[0] * q_scale, x[4] * q_scale, x[1] * q_scale, x[5] * q_scale);
            if (r + 8 < L)
                *(float4*)(dst + (size_t)(r + 8) * H * dv) = make_float4(x[2] * q_scale, x[6] * q_scale, x[3] * q_scale, x[7] * q_scale);
        }
    }
}

static inline size_t lm_state_smem() {
    return (size_t)4 * LA_C * LM_LD * 2;
}
static inline size_t lm_out_smem(int d) {
    return (size_t)(3 * d + LA_C) * LM_LD * 2 + (size_t)4 * LA_C * (d + 8) * 2 + (size_t)LA_C * (d + 2) * 4;
}
static inline size_t lm_state_heads_smem() {
    return (size_t)LA_C * LM_LK * 2 + (size_t)3 * LA_C * LM_LD * 2;
}
static inline size_t lm_out_heads_smem(int d) {
    const size_t keys = (size_t)LA_C * (d + 8) * 2, scores = (size_t)3 * LA_C * LM_LD * 2;
    return (size_t)LA_C * (d + 8) * 2 + (size_t)LA_C * LM_LD * 2 + (keys > scores ? keys : scores);
}
// Heads a block takes one after another: up to four of those that share their keys, as long as there are
// three blocks a multiprocessor (four fit one).
static inline int lm_heads(int share, long long blocks) {
    int n = 1;
    while (n < 4 && share % (2 * n) == 0 && blocks / (2 * n) >= 3 * rv_sm_count()) n *= 2;
    return n;
}
