// y = x . w^T in float32 for few rows or few columns: x [M, K], w [N, K], y [M, N], float32 multiply-adds
// (no TF32 and no split operands).
//
// A block has BM = 8 TMG rows by BN = 4 TNG columns; a thread has 8 rows by 4 columns, spread so that
// neighbouring threads have neighbouring ones.  Tiles of 16 of K arrive by cp.async in a ring of
// GF_STAGES; both operands lie as they do in memory, K innermost, rows of 20 floats, so that the eight
// lanes of an access phase meet no bank twice.  A thread reads four of K at a time and multiplies them
// two by two (fma.rn.f32x2): every output is two sums, over the even and the odd k, added at the end.
// Rows are dealt to as few blocks of up to 64 as there can be, in steps of eight (131 rows: 3 x 48, where
// tiles of 64 would work 192).  Small products have few tiles: their K is split over a cluster of up to
// eight blocks, which leave their tiles in shared memory and add them in rank order.
//
// Bound by the multiply-adds' loads from some 32 rows on (30 - 40 of 74 TFLOP/s).  With fewer rows by
// latency, not by the matrix's bytes: up to 8 rows a block is one warp and K is split eight ways at most, so
// N = 1,536 gives 96 warps to 148 multiprocessors (1 row: 12 % of the bytes' time at 1536 x 6912, 24 %
// at 4608 x 1536, 45 % at 65536 x 1024).  The library's float32 products take tiles of 32 x 32 to 64 x 128
// on the same cores; at equal sizes (us, N x K): 1 row 4608 x 1536 39 -> 18, 13824 x 1536 52 -> 29, 1536 x
// 6912 79 -> 52, 65536 x 1024 113 -> 92; 16 rows 39 -> 19, 52 -> 37, 79 -> 50, 113 -> 84; 64 rows 1536 x 1536
// 38 -> 19, 1536 x 6912 110 -> 68; 144 rows 36 -> 32, 156 -> 127.  With many rows and columns it is the slower
// one (131 rows 13824 x 1536 188 -> 209, 2,048 rows 1,377 -> 2,111), see rv_gemm_f32_better.
// Operands in three bfloat16 parts on mma.sync were measured too: 131 rows 13824 x 1536 147 us, but
// slower than the library below 96 rows and above 144, and than this at N = 1536.
// From 768 of K on gemm_f32_split.cu is the faster one; this one is left with K of 512 to 764.
// Its sums are nearer to float64 (relative error 2 - 4e-7 at these sizes, the library's 3e-7 - 1.5e-6).
// Plain reference: tests/plain_ops.py linear.
#include "common.cuh"
#include "mma_bf16.cuh"

#define GF_BK 16
#define GF_LD 20            // floats of a row of a tile
#define GF_STAGES 4

__device__ __forceinline__ void gf_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float gf_cluster_load(const float* local, unsigned rank) {
    unsigned at = (unsigned)__cvta_generic_to_shared(local), remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}
__device__ __forceinline__ void gf_fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

// The cluster's tiles, each [BM][BN] at the start of its block's shared memory, added in rank order.
template <int BM, int BN, int THREADS>
__device__ __forceinline__ void gf_reduce(const float* sm, float* y, int m0, int n0, int M, int N) {
    const int splits = gridDim.z;
    gf_cluster_sync();                                    // every block's tile is there
    for (int e = blockIdx.z * THREADS + threadIdx.x; e < BM * BN; e += splits * THREADS) {
        const int m = m0 + e / BN, n = n0 + e % BN;
        if (m >= M || n >= N) continue;
        float v[8], sum = 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) v[r] = r < splits ? gf_cluster_load(sm + e, r) : 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) sum += v[r];
        y[(size_t)m * N + n] = sum;
    }
    gf_cluster_sync();                                    // nobody leaves while its tile is read
}

template <int TMG, int TNG>
__global__ void __launch_bounds__(TMG* TNG) gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                            float* __restrict__ y, int M, int N, int K, int per_split) {
    // Neither operand is read before the kernel before has ended: the matrix need not be a weight, it
    // may be what that kernel writes (rows of 32 bits by a matrix of 16 are cast just before).
    rv_pdl_prologue();
    constexpr int TN = 4, BM = 8 * TMG, BN = TN * TNG, THREADS = TMG * TNG, STAGE = (BM + BN) * GF_LD;
    extern __shared__ __align__(16) float sm[];           // [stages][BM rows of x, BN rows of w][GF_LD]
    const int tid = threadIdx.x, ng = tid % TNG, mg = tid / TNG;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const int k0 = blockIdx.z * per_split, k1 = min(K, k0 + per_split);
    const int steps = k1 > k0 ? (k1 - k0 + GF_BK - 1) / GF_BK : 0;
    // a stage's pieces of 16 bytes: rows of w or of x; what lies beyond N, M or K is zero
    auto get = [&](int s, bool weights) {
        float* to = sm + (s % GF_STAGES) * STAGE + (weights ? BM * GF_LD : 0);
        const int rows = weights ? BN : BM, first = weights ? n0 : m0, all = weights ? N : M;
        const float* from = weights ? w : x;
#pragma unroll
        for (int p = tid; p < rows * 4; p += THREADS) {
            const int r = p >> 2, k = k0 + s * GF_BK + (p & 3) * 4;
            const bool there = first + r < all && k < k1;
            cp_async_16(to + r * GF_LD + (p & 3) * 4, from + (size_t)min(first + r, all - 1) * K + (there ? k : 0), there);
        }
    };
#pragma unroll
    for (int s = 0; s < GF_STAGES - 1; ++s) {
        if (s < steps) {
            get(s, true);
            get(s, false);
        }
        cp_async_commit();
    }
    unsigned long long acc[8][TN];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
    for (int s = 0; s < steps; ++s) {
        cp_async_wait<GF_STAGES - 2>();
        __syncthreads();                                  // tile s is here; tile s - 1 has been read
        if (s + GF_STAGES - 1 < steps) {
            get(s + GF_STAGES - 1, true);
            get(s + GF_STAGES - 1, false);
        }
        cp_async_commit();
        const float* xs = sm + (s % GF_STAGES) * STAGE + mg * GF_LD;
        const float* ws = sm + (s % GF_STAGES) * STAGE + (BM + ng) * GF_LD;
#pragma unroll
        for (int k = 0; k < GF_BK; k += 4) {
            ulonglong2 b[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = *(const ulonglong2*)(ws + j * TNG * GF_LD + k);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const ulonglong2 a = *(const ulonglong2*)(xs + i * TMG * GF_LD + k);
#pragma unroll
                for (int j = 0; j < TN; ++j) gf_fma2(acc[i][j], a.x, b[j].x);
#pragma unroll
                for (int j = 0; j < TN; ++j) gf_fma2(acc[i][j], a.y, b[j].y);
            }
        }
    }
    auto value = [&](int i, int j) {
        return __uint_as_float((unsigned)acc[i][j]) + __uint_as_float((unsigned)(acc[i][j] >> 32));
    };
    if (gridDim.z == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int m = m0 + mg + TMG * i, n = n0 + ng + TNG * j;
                if (m < M && n < N) y[(size_t)m * N + n] = value(i, j);
            }
        return;
    }
    cp_async_wait<0>();
    __syncthreads();                                      // the ring is free
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sm[(mg + TMG * i) * BN + ng + TNG * j] = value(i, j);
    gf_reduce<BM, BN, THREADS>(sm, y, m0, n0, M, N);
}

template <int TMG, int TNG>
static cudaError_t gf_launch(const float* x, const float* w, float* y, int M, int N, int K, int m_tiles,
                             cudaStream_t stream) {
    constexpr int BM = 8 * TMG, BN = 4 * TNG;
    const size_t smem = (size_t)GF_STAGES * (BM + BN) * GF_LD * sizeof(float);
    static_assert((size_t)GF_STAGES * (BM + BN) * GF_LD >= (size_t)BM * BN, "the tile fits the ring");
    // (the limit is a device's own: float32 products may be asked on another one than the first)
    static bool raised[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !raised[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<TMG, TNG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) raised[dev] = true;
    }
    // K is split until there are three blocks a multiprocessor, 128 of K at least
    const int n_tiles = (N + BN - 1) / BN;
    int splits = 1;
    while (splits < 8 && (long long)n_tiles * m_tiles * splits < 3 * rv_sm_count() && K / (splits * 2) >= 128) splits *= 2;
    const int per_split = (K + splits * GF_BK - 1) / (splits * GF_BK) * GF_BK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_tiles, m_tiles, splits);
    cfg.blockDim = dim3(TMG * TNG);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = splits;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = rv_pdl_enabled();
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, gemm_f32_kernel<TMG, TNG>, x, w, y, M, N, K, per_split);
}

// Whether this kernel is the faster one.  Both sides were measured at 256 to 6,912 of K, 256 to 65,536
// columns and 1 to 160 rows, and at sizes drawn between them, matrices beyond L2 (us here / the library's):
//   K below 512 (1,024 with fewer than 1,536 or more than 6,144 columns or more than 16 rows): a launch of few steps, whose
//     cluster is not repaid: 256 x 256 8 rows 12 / 7, 64 rows 10 / 7; 1209 x 828 11 rows 14 / 13; 18291 x 780 14 rows 35 / 28.
//   up to 16 rows: 4608 x 512 11 / 15, 1536 x 1536 14 / 27, 4608 x 4096 45 / 102.  K above 2,048 with
//     fewer columns than 1,536 is even with the library, which splits K too (256 x 4096 32 / 30).
//   up to 32 rows: 512 x 1024 9 / 14, 6144 x 1024 17 / 27, but 9216 x 1024 29 / 28.
//   up to 64 rows: 1024 x 1024 12 / 26, 4608 x 1536 37 / 40, 6144 x 1024 32 / 32; 897 x 2164 26 / 23, 9216 x
//     1024 46 / 35.
//   up to 144 rows (three tiles of 48): 1536 x 1024 22 / 25, 1536 x 1536 32 / 36, but 160 rows 27 / 25 and
//     37 / 36; 428 x 3624 119 rows 46 / 34.
//   2,048 columns: to 96 rows 18 / 26 (K 1,024), to 128 rows from K 1,536 on 35 / 37; 2,560: 30 / 30.
extern "C" int rv_gemm_f32_better(int M, int N, int K) {
    if (K % 4 || K < 512 || N < 256) return 0;
    if (K < 1024) return M <= 16 && N >= 1536 && N <= 6144;
    if (M <= 16) return K <= 2048 || N >= 1536;
    if (M <= 32) return N <= 6144;
    if (N < 1024) return 0;
    if (M <= 64) return N <= 6144;
    return (M <= 144 && N <= 1536) || (M <= (K >= 1536 ? 128 : 96) && N <= 2048);
}

// K a multiple of 4, x and w on 16-byte boundaries.
extern "C" int rv_gemm_f32(const float* x, const float* w, float* y, int M, int N, int K, void* stream) {
    if (M == 0 || N == 0) return 0;
    if (M < 0 || N < 0 || K < 4 || K % 4) RV_FAIL("gemm_f32: bad sizes");
    if (((uintptr_t)x | (uintptr_t)w) & 15) RV_FAIL("gemm_f32: the operands must be 16-byte aligned");
    const int m_tiles = (M + 63) / 64, rows = (M + m_tiles - 1) / m_tiles;
    if (m_tiles > 65535) RV_FAIL("gemm_f32: too many rows");
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e;
    // 128 columns a block with few rows, 64 with more: 32 to 128 threads
    switch ((rows + 7) / 8) {
        case 1: e = gf_launch<1, 32>(x, w, y, M, N, K, m_tiles, s); break;
        case 2: e = gf_launch<2, 32>(x, w, y, M, N, K, m_tiles, s); break;
        case 3: e = gf_launch<3, 32>(x, w, y, M, N, K, m_tiles, s); break;
        case 4: e = gf_launch<4, 32>(x, w, y, M, N, K, m_tiles, s); break;
        case 5: e = gf_launch<5, 16>(x, w, y, M, N, K, m_tiles, s); break;
        case 6: e = gf_launch<6, 16>(x, w, y, M, N, K, m_tiles, s); break;
        case 7: e = gf_launch<7, 16>(x, w, y, M, N, K, m_tiles, s); break;
        default: e = gf_launch<8, 16>(x, w, y, M, N, K, m_tiles, s); break;
    }
    if (e != cudaSuccess) RV_FAIL("gemm_f32: %s", cudaGetErrorString(e));
    RV_CHECK_LAUNCH("gemm_f32");
    return 0;
}
