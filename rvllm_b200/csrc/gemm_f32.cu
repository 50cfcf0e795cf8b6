// y = x . w^T in float32 for few rows: x [M, K], w [N, K], y [M, N], float32 multiply-adds
// (no TF32 and no split operands).
//
// A block is one warp with 8 rows by 128 columns; a thread has 8 rows by 4 columns, spread so that
// neighbouring threads have neighbouring ones.  Tiles of 16 of K arrive by cp.async in a ring of
// GF_STAGES; both operands lie as they do in memory, K innermost, rows of 20 floats, so that the eight
// lanes of an access phase meet no bank twice.  A thread reads four of K at a time and multiplies them
// two by two (fma.rn.f32x2): every output is two sums, over the even and the odd k, added at the end.
// K is split over a cluster of up to eight blocks, which leave their tiles in shared memory and add them in rank order.
//
// Bound by latency, not by the matrix's bytes: a block is one warp and K is split eight ways at most, so
// N = 9,216 gives 576 warps to 148 multiprocessors.  gemm_f32_split.cu is the faster one but for the sizes of
// rv_gemm_f32_better, where its tiles fill the chip a little more than once.
// Its sums are nearer to float64 than the library's (relative error 2 - 4e-7, the library's 3e-7 - 1.5e-6).
// Plain reference: tests/plain_ops.py linear.
#include "common.cuh"
#include "mma_bf16.cuh"

#define GF_BK 16
#define GF_LD 20            // floats of a row of a tile
#define GF_STAGES 4
#define GF_BM 8             // rows of a block
#define GF_TN 4             // columns of a thread
#define GF_BN (32 * GF_TN)  // columns of a block

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

// The cluster's tiles, each [GF_BM][GF_BN] at the start of its block's shared memory, added in rank order.
__device__ __forceinline__ void gf_reduce(const float* sm, float* y, int m0, int n0, int M, int N) {
    const int splits = gridDim.z;
    gf_cluster_sync();                                    // every block's tile is there
    for (int e = blockIdx.z * 32 + threadIdx.x; e < GF_BM * GF_BN; e += splits * 32) {
        const int m = m0 + e / GF_BN, n = n0 + e % GF_BN;
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

__global__ void __launch_bounds__(32) gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                      float* __restrict__ y, int M, int N, int K, int per_split) {
    // Neither operand is read before the kernel before has ended: the matrix need not be a weight, it
    // may be what that kernel writes (rows of 32 bits by a matrix of 16 are cast just before).
    rv_pdl_prologue();
    constexpr int TN = GF_TN, BM = GF_BM, BN = GF_BN, STAGE = (BM + BN) * GF_LD;
    extern __shared__ __align__(16) float sm[];           // [stages][BM rows of x, BN rows of w][GF_LD]
    const int tid = threadIdx.x;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const int k0 = blockIdx.z * per_split, k1 = min(K, k0 + per_split);
    const int steps = k1 > k0 ? (k1 - k0 + GF_BK - 1) / GF_BK : 0;
    // a stage's pieces of 16 bytes: rows of w or of x; what lies beyond N, M or K is zero
    auto get = [&](int s, bool weights) {
        float* to = sm + (s % GF_STAGES) * STAGE + (weights ? BM * GF_LD : 0);
        const int rows = weights ? BN : BM, first = weights ? n0 : m0, all = weights ? N : M;
        const float* from = weights ? w : x;
#pragma unroll
        for (int p = tid; p < rows * 4; p += 32) {
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
        const float* xs = sm + (s % GF_STAGES) * STAGE;
        const float* ws = sm + (s % GF_STAGES) * STAGE + (BM + tid) * GF_LD;
#pragma unroll
        for (int k = 0; k < GF_BK; k += 4) {
            ulonglong2 b[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = *(const ulonglong2*)(ws + j * 32 * GF_LD + k);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const ulonglong2 a = *(const ulonglong2*)(xs + i * GF_LD + k);
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
                const int m = m0 + i, n = n0 + tid + 32 * j;
                if (m < M && n < N) y[(size_t)m * N + n] = value(i, j);
            }
        return;
    }
    cp_async_wait<0>();
    __syncthreads();                                      // the ring is free
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) sm[i * BN + tid + 32 * j] = value(i, j);
    gf_reduce(sm, y, m0, n0, M, N);
}

static cudaError_t gf_launch(const float* x, const float* w, float* y, int M, int N, int K, int m_tiles,
                             cudaStream_t stream) {
    const size_t smem = (size_t)GF_STAGES * (GF_BM + GF_BN) * GF_LD * sizeof(float);
    static_assert((size_t)GF_STAGES * (GF_BM + GF_BN) * GF_LD >= (size_t)GF_BM * GF_BN, "the tile fits the ring");
    // (the limit is a device's own: float32 products may be asked on another one than the first)
    static bool raised[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !raised[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) raised[dev] = true;
    }
    // K is split until there are three blocks a multiprocessor, 128 of K at least
    const int n_tiles = (N + GF_BN - 1) / GF_BN;
    int splits = 1;
    while (splits < 8 && (long long)n_tiles * m_tiles * splits < 3 * rv_sm_count() && K / (splits * 2) >= 128) splits *= 2;
    const int per_split = (K + splits * GF_BK - 1) / (splits * GF_BK) * GF_BK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_tiles, m_tiles, splits);
    cfg.blockDim = dim3(32);
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
    return cudaLaunchKernelEx(&cfg, gemm_f32_kernel, x, w, y, M, N, K, per_split);
}

// Whether this kernel is the faster one.  Measured against gemm_f32_split.cu at 512 to 3,072 of K, 2,048 to 65,536
// columns and 1 to 16 rows, replayed, matrices beyond L2 (us here / there): 9216 x 1024 1 row 14.1 / 17.4, 8 rows 15.4 /
// 18.0; 9216 x 1280 17.4 / 19.6, 18.5 / 20.4; 9216 x 1536 20.2 / 21.9, 21.5 / 22.5; 9216 x 2048 25.7 / 26.5, 27.2 / 27.4.  It is the
// slower one at 896 of K and at 6,144 and 12,288 columns, and even or slower with 16 rows and at 3,072 of K; 4608 x 1024 12.6 / 13.4
// is the only other one that it wins by more than 0.3 us.
extern "C" int rv_gemm_f32_better(int M, int N, int K) {
    return K % 4 == 0 && M <= 8 && K >= 1024 && K <= 2048 && N >= 8192 && N <= 10240;
}

// K a multiple of 4, x and w on 16-byte boundaries.
extern "C" int rv_gemm_f32(const float* x, const float* w, float* y, int M, int N, int K, void* stream) {
    if (M == 0 || N == 0) return 0;
    if (M < 0 || N < 0 || K < 4 || K % 4) RV_FAIL("gemm_f32: bad sizes");
    if (((uintptr_t)x | (uintptr_t)w) & 15) RV_FAIL("gemm_f32: the operands must be 16-byte aligned");
    const int m_tiles = (M + GF_BM - 1) / GF_BM;
    if (m_tiles > 65535) RV_FAIL("gemm_f32: too many rows");
    const cudaError_t e = gf_launch(x, w, y, M, N, K, m_tiles, (cudaStream_t)stream);
    if (e != cudaSuccess) RV_FAIL("gemm_f32: %s", cudaGetErrorString(e));
    RV_CHECK_LAUNCH("gemm_f32");
    return 0;
}
