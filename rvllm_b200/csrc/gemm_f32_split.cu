// y = x . w^T in float32 on the 5th-generation tensor cores: x [M, K], w [N, K], y [M, N].
//
// A float32 value is the sum of three bfloat16 values, its bits 1 - 8, 9 - 16 and 17 - 24: x = h + m + l exactly.
// A product of two such sums is formed as eight of the nine products of their parts (l l' is below 2^-30 of it):
// tcgen05.mma of kind::f16, whose products are exact and whose sums are float32.  Where one
// operand's value is a power of two the result is the other's.  The tensor core cuts off what lies below the
// accumulator's last bit, so a sum is not left there for long: a chunk is 32 of K, its small
// products first, and then goes to float32 registers, which add the chunks with round-to-nearest.
// (Two TF32 parts and three products hold 22 bits and leave out 2^-22 of a product.)
//
//   split    x -> parts [row tile][chunk][h, m, l][rows][32], each [rows][32] as the swizzled image that a
//            product's operand has in shared memory, so that a chunk is one contiguous copy
//   product  block per (128 columns, up to 160 rows, share of K).  128 rows of w are the M side, so an
//            output column is a TMEM lane; the rows of x are the N side.
//     warps 0 - 3    w: 32 rows each by cp.async into a ring of its own, split in registers, to TMEM
//                    (the A operand; three chunks): shared memory, which the B operand's reads keep
//                    busy, sees w once in and once out
//     warps 4 - 11   the accumulators (two chunks) to registers, and at the end the outputs
//     warp 12        issues the sixteen products of a chunk
//     warp 13        copies the chunks of x
//   K is shared by a cluster of up to eight blocks, which leave their tiles in shared memory and add
//   them in rank order.
//
// Bound by the tensor cores' reads of shared memory and by the pipeline's meetings with many rows (131 x 13824 x
// 1536: 0.9 us a chunk, of which the sixteen products' own time is some 0.55), by the matrix's bytes with few.  us at N x K,
// a call with its launches, L2 flushed, against the library's kernels on the FP32 cores or gemm_f32.cu's, whichever
// was the faster: 131 rows 4608 x 1536 78 -> 42, 1536 x 1536 37 -> 20, 13824 x 1536 166 -> 56, 1536 x 6912 131 -> 40; 16 rows
// 25 -> 24, 18 -> 15, 45 -> 32, 55 -> 26; 2,048 rows 498 -> 202, 215 -> 103, 1,387 -> 501, 906 -> 327.  Relative error against
// 64 bits there: 0.9 - 2.5e-7 (the library's 1.4e-7 - 1.5e-6, gemm_f32.cu's 1.9e-7 - 1.1e-6).
//
// A sum that is not finite is formed again from x and w by float32 multiply-adds (parts of an infinite value are
// not numbers), and one below 2^-100, whose small products leave float32's range.  Operands below 2^-110
// lose the bits of l that bfloat16 does not have there; that is seen beside operands above 2^10 only.
//
// Every wait is bounded; one that runs out records 41 - 45 in `status` and the block ends.
// Plain reference: tests/plain_ops.py linear.
#include "tcgen05_common.cuh"
#include "mma_bf16.cuh"

#define FS_BK 32            // of K in a chunk: rows of 128 bytes
#define FS_BN 128           // rows of w in a block
#define FS_WS 5             // chunks of w in a ring
#define FS_XS 3             // chunks of x in a ring, and of w in TMEM
#define FS_PARTS 3
#define FS_MAX_ROWS 160     // of x in a block: with three chunks of w and two accumulators 512 columns of TMEM
#define FS_THREADS 448

// Two neighbours' parts, the first in the lower half.
__device__ __forceinline__ void fs_parts(float a, float b, unsigned (&p)[FS_PARTS]) {
#pragma unroll
    for (int i = 0; i < FS_PARTS; ++i) {
        const unsigned ua = __float_as_uint(a), ub = __float_as_uint(b);
        p[i] = __byte_perm(ua, ub, 0x7632);
        a -= __uint_as_float(ua & 0xffff0000u);
        b -= __uint_as_float(ub & 0xffff0000u);
    }
}
__device__ __forceinline__ void fs_mma(unsigned tmem_d, unsigned tmem_a, unsigned long long b_desc, unsigned idesc,
                                       unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Descriptor of a K-major tile with 64-byte swizzle: rows of 64 bytes, eight rows 512 bytes on, layout type 4.
__device__ __forceinline__ unsigned long long fs_desc(const void* tile) {
    const unsigned long long addr = (smem_u32(tile) & 0x3FFFFu) >> 4;
    return addr | (1ull << 16) | (32ull << 32) | (1ull << 46) | (4ull << 61);
}
__device__ __forceinline__ void fs_tmem_store_16(unsigned taddr, const unsigned (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void fs_tmem_load_8(unsigned taddr, unsigned* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void fs_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fs_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float fs_cluster_load(const float* local, unsigned rank) {
    unsigned remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}
// The sum as it is, where its parts did not give it.
__device__ __noinline__ float fs_plain(const float* x, const float* w, int K) {
    float s = 0.f;
    for (int k = 0; k < K; ++k) s = fmaf(x[k], w[k], s);
    return s;
}
__device__ __forceinline__ float fs_checked(float v, const float* x, const float* w, int m, int n, int K) {
    const float a = fabsf(v);
    return v == 0.f || (a >= 7.8886091e-31f && a < INFINITY) ? v : fs_plain(x + (size_t)m * K, w + (size_t)n * K, K);
}

// Block (chunk, row tile).  The next kernel, the product, may begin when all blocks here are past their
// wait: what ran before is then done, and w, which that may have written, can be read.
__global__ void __launch_bounds__(256) fs_split_kernel(const float* __restrict__ x, float* __restrict__ parts, int M, int K,
                                                       int rows) {
    rv_pdl_wait();
    rv_pdl_launch_dependents();
    const int kb = blockIdx.x, m0 = blockIdx.y * rows;
    unsigned char* to = (unsigned char*)parts + ((size_t)blockIdx.y * gridDim.x + kb) * FS_PARTS * rows * FS_BK * 2;
    for (int i = threadIdx.x; i < rows * (FS_BK / 8); i += 256) {
        const int r = i >> 2, c = i & 3, k = kb * FS_BK + c * 8;
        const float* from = x + (size_t)(m0 + r) * K + k;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 a = m0 + r < M && k < K ? *(const float4*)from : zero, b = m0 + r < M && k + 4 < K ? *(const float4*)(from + 4) : zero;
        unsigned p[4][FS_PARTS];
        fs_parts(a.x, a.y, p[0]);
        fs_parts(a.z, a.w, p[1]);
        fs_parts(b.x, b.y, p[2]);
        fs_parts(b.z, b.w, p[3]);
        unsigned char* at = to + r * FS_BK * 2 + ((c ^ ((r >> 1) & 3)) << 4);
#pragma unroll
        for (int s = 0; s < FS_PARTS; ++s) *(uint4*)(at + (size_t)s * rows * FS_BK * 2) = make_uint4(p[0][s], p[1][s], p[2][s], p[3][s]);
    }
}

// grid (row tiles, column tiles, shares of K), clusters of (1, 1, shares)
template <int NT>
__global__ void __launch_bounds__(FS_THREADS, NT <= 32 ? 2 : 1) fs_gemm_kernel(
    const float* __restrict__ parts, const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y,
    int* __restrict__ status, int M, int N, int K) {
    constexpr int XS = FS_XS;
    constexpr int CT = NT / 2;                            // columns of an accumulator that a thread holds
    constexpr unsigned X_PART = NT * FS_BK * 2, X_STAGE = FS_PARTS * X_PART, W_STAGE = FS_BN * FS_BK * 4;
    constexpr unsigned A_PART = FS_BK / 2, A_COLS = FS_PARTS * A_PART, COLS = XS * A_COLS + 2 * NT <= 256 ? 256 : 512;
    static_assert(XS * A_COLS + 2 * NT <= 512, "TMEM holds the chunks and the accumulators");
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* xs = base;
    unsigned char* ws = base + XS * X_STAGE;
    __shared__ __align__(8) unsigned long long full[XS], empty[XS], d_full[2], d_free[2];
    __shared__ unsigned tmem_smem;
    __shared__ volatile int failed;

    rv_pdl_launch_dependents();
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int m0 = blockIdx.x * NT, n0 = blockIdx.y * FS_BN, share = blockIdx.z, shares = gridDim.z;
    const int chunks = (K + FS_BK - 1) / FS_BK;
    const int c0 = (int)((long long)chunks * share / shares), n = (int)((long long)chunks * (share + 1) / shares) - c0;
    if (tid == 0) {
        failed = 0;
        for (int s = 0; s < XS; ++s) {
            mbar_init(&full[s], 5);                       // a chunk of x, and of w by four warps
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&d_full[b], 1);
            mbar_init(&d_free[b], 8);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 12) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_smem)), "r"(COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = __shfl_sync(0xffffffffu, tmem_smem, 0), tmem_d = tmem + XS * A_COLS;
    auto give_up = [&](int code) {
        if (!failed) {
            failed = 1;
            atomicCAS(status, 0, code);
        }
    };

    float acc[CT];
#pragma unroll
    for (int j = 0; j < CT; ++j) acc[j] = 0.f;

    if (warp < 4) {
        // ---- w to TMEM in three parts ---------------------------------------------------------
        unsigned char* ring = ws + warp * (W_STAGE / 4);
        const int first = n0 + warp * 32;
        auto get = [&](int i) {
            unsigned char* to = ring + (i % FS_WS) * W_STAGE;
            const int c = lane & 7, k = (c0 + i) * FS_BK + c * 4;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int r = 4 * j + (lane >> 3);
                const bool there = i < n && first + r < N && k < K;
                cp_async_16(to + r * 128 + ((c ^ (r & 7)) << 4), w + (there ? (size_t)(first + r) * K + k : 0), there);
            }
        };
#pragma unroll
        for (int i = 0; i < FS_WS - 1; ++i) {
            if (i < n) get(i);
            cp_async_commit();
        }
        for (int i = 0; i < n; ++i) {
            cp_async_wait<FS_WS - 2>();
            __syncwarp();                                 // chunk i is here, chunk i - 1 has been read
            if (i + FS_WS - 1 < n) get(i + FS_WS - 1);
            cp_async_commit();
            unsigned p[FS_PARTS][A_PART];
            const unsigned char* row = ring + (i % FS_WS) * W_STAGE + lane * 128;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float4 v = *(const float4*)(row + ((c ^ (lane & 7)) << 4));
                unsigned a[FS_PARTS], e[FS_PARTS];
                fs_parts(v.x, v.y, a);
                fs_parts(v.z, v.w, e);
#pragma unroll
                for (int s = 0; s < FS_PARTS; ++s) {
                    p[s][2 * c] = a[s];
                    p[s][2 * c + 1] = e[s];
                }
            }
            const int b = i % XS;
            bool ok = i < XS || mbar_wait(&empty[b], ((i / XS) - 1) & 1, &failed);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                give_up(41);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned to = tmem + ((unsigned)(warp * 32) << 16) + b * A_COLS;
#pragma unroll
            for (int s = 0; s < FS_PARTS; ++s) fs_tmem_store_16(to + s * A_PART, p[s]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) fs_arrive(&full[b]);
        }
        cp_async_wait<0>();
    } else if (warp < 12) {
        // ---- the chunks' sums to registers -------------------------------------------------------
        const unsigned from = tmem_d + ((unsigned)((warp & 3) * 32) << 16) + ((warp - 4) >> 2) * CT;
        for (int i = 0; i < n; ++i) {
            const int b = i & 1;
            bool ok = mbar_wait(&d_full[b], (i >> 1) & 1, &failed);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                give_up(42);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int j0 = 0; j0 < CT; j0 += 32) {         // up to 32 columns requested together
                unsigned r[32];
#pragma unroll
                for (int j = 0; j < 32; j += 8)
                    if (j0 + j < CT) fs_tmem_load_8(from + b * NT + j0 + j, r + j);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (j0 + 32 >= CT) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) fs_arrive(&d_free[b]);
                }
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (j0 + j < CT) acc[j0 + j] += __uint_as_float(r[j]);
            }
        }
    } else if (warp == 12) {
        // ---- the products: the warp walks the chunks together, one lane issues -----------------------
        rv_pdl_wait();                                    // the bounded waits start when the kernel before is done
        const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(NT >> 3) << 17) |
                               ((unsigned)(FS_BN >> 4) << 24);
        int issued = 0;
        for (int i = 0; i < n; ++i) {
            const int b = i & 1, s = i % XS;
            bool ok = mbar_wait(&full[s], (i / XS) & 1, &failed) &&
                      (i < 2 || mbar_wait(&d_free[b], ((i >> 1) - 1) & 1, &failed));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                give_up(43);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (rv_elect()) {
                const unsigned d = tmem_d + b * NT, a = tmem + s * A_COLS;
                const unsigned long long x0 = fs_desc(xs + s * X_STAGE);
                // parts of w and of x whose numbers add up to 3, 2, 1 and 0: the smallest products first
#pragma unroll
                for (int sum = 3; sum >= 0; --sum)
#pragma unroll
                    for (int p = 0; p < FS_PARTS; ++p)
                        if (sum - p >= 0 && sum - p < FS_PARTS) {
#pragma unroll
                            for (int k = 0; k < FS_BK / 16; ++k)
                                fs_mma(d, a + p * A_PART + 8 * k, x0 + (sum - p) * (X_PART >> 4) + 2 * k, idesc,
                                       sum != 3 || p != 1 || k != 0);
                        }
                tcgen05_commit(&empty[s]);
                tcgen05_commit(&d_full[b]);
            }
            __syncwarp();
            issued = i + 1;
        }
        // nothing of the tensor core's may be under way when TMEM is given back
        if (issued) {
            bool ok = false;
            const long long start = clock64();
            while (!ok && clock64() - start < RV_WAIT_CYCLES)
                ok = mbar_try_wait(&d_full[(issued - 1) & 1], ((issued - 1) >> 1) & 1);
            if (!ok) give_up(44);
        }
    } else if (lane == 0) {
        // ---- the chunks of x ---------------------------------------------------------------------------
        rv_pdl_wait();
        const unsigned char* from = (const unsigned char*)parts + ((size_t)blockIdx.x * chunks + c0) * X_STAGE;
        int issued = 0;
        for (int i = 0; i < n; ++i) {
            const int s = i % XS;
            if (i >= XS && !mbar_wait(&empty[s], ((i / XS) - 1) & 1, &failed)) {
                give_up(45);
                break;
            }
            mbar_expect_tx(&full[s], X_STAGE);
            bulk_load_1d(xs + s * X_STAGE, from + (size_t)i * X_STAGE, X_STAGE, &full[s]);
            issued = i + 1;
        }
        for (int i = max(0, issued - XS); i < issued; ++i) {
            bool ok = false;
            const long long start = clock64();
            while (!ok && clock64() - start < RV_WAIT_CYCLES) ok = mbar_try_wait(&full[i % XS], (i / XS) & 1);
            if (!ok) give_up(45);
        }
    }
    __syncwarp();
    rv_pdl_wait();                                        // before y is written
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();                                      // all copies and products are done
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 12)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS));
    const bool good = !failed;
    const int nl = (warp & 3) * 32 + lane, t0 = ((warp - 4) >> 2) * CT;
    if (shares == 1) {
        if (warp >= 4 && warp < 12 && n0 + nl < N && good) {
#pragma unroll
            for (int j = 0; j < CT; ++j) {
                const int m = m0 + t0 + j;
                if (m < M) y[(size_t)m * N + n0 + nl] = fs_checked(acc[j], x, w, m, n0 + nl, K);
            }
        }
        return;
    }
    float* park = (float*)base;                           // [row][128], over the rings
    if (warp >= 4 && warp < 12) {
#pragma unroll
        for (int j = 0; j < CT; ++j) park[(t0 + j) * FS_BN + nl] = good ? acc[j] : 0.f;
    }
    fs_cluster_sync();                                    // every block's tile is there
    const int rows = min(NT, M - m0);
    for (int e = share * FS_THREADS + tid; e < rows * FS_BN; e += shares * FS_THREADS) {
        const int m = m0 + e / FS_BN, c = n0 + e % FS_BN;
        float v[8], sum = 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) v[r] = r < shares ? fs_cluster_load(park + e, r) : 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) sum += v[r];
        if (c < N) y[(size_t)m * N + c] = fs_checked(sum, x, w, m, c, K);
    }
    __syncwarp();
    fs_cluster_sync();                                    // nobody leaves while its tile is read
}

template <int NT>
static constexpr size_t fs_smem() {
    return (size_t)FS_XS * NT * FS_BK * 2 * FS_PARTS + FS_WS * FS_BN * FS_BK * 4 + 1024;
}
static_assert(fs_smem<FS_MAX_ROWS>() <= 227 * 1024, "the rings fit shared memory");

template <int NT>
static cudaError_t fs_launch(const float* parts, const float* x, const float* w, float* y, int* status, int M, int N,
                             int K, int m_tiles, cudaStream_t stream) {
    static_assert(fs_smem<NT>() >= (size_t)NT * FS_BN * 4, "the tile fits the rings");
    const size_t smem = fs_smem<NT>();
    // (the limit is a device's own)
    static bool raised[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !raised[dev]) {
        cudaError_t e = cudaFuncSetAttribute(fs_gemm_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) raised[dev] = true;
    }
    // K is shared by as many blocks as cost the fewest chunks' times: a block's own chunks, six chunks' time to
    // start and end and four for the cluster, over the blocks that a multiprocessor has one after
    // another (two at a time with up to 32 rows, which then take 0.7 of the time).
    const int n_tiles = (N + FS_BN - 1) / FS_BN, chunks = (K + FS_BK - 1) / FS_BK;
    int shares = 1;
    double least = 0.;
    for (int c = 1; c <= 8 && (c == 1 || chunks / c >= 4); c *= 2) {
        const long long turns = ((long long)m_tiles * n_tiles * c + rv_sm_count() - 1) / rv_sm_count();
        const double each = (double)((chunks + c - 1) / c), fixed = c > 1 ? 10. : 6.;
        const double cost = NT > 32 ? turns * (each + fixed) : turns * each * (turns > 1 ? 0.7 : 1.) + (turns + 1) / 2 * fixed;
        if (c == 1 || cost < least) {
            least = cost;
            shares = c;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(m_tiles, n_tiles, shares);
    cfg.blockDim = dim3(FS_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = shares;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = rv_pdl_enabled();
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, fs_gemm_kernel<NT>, parts, x, w, y, status, M, N, K);
}

// Rows of x that are split at a time: as few tiles as there can be, and 64 MB of parts at the most.
struct FsRows { int tiles, rows; };
static FsRows fs_rows(int M, int K) {
    const long long tile = (long long)FS_MAX_ROWS * ((K + FS_BK - 1) / FS_BK * FS_BK) * 2 * FS_PARTS;
    const int most = (int)((64ll << 20) / tile);
    int tiles = (M + FS_MAX_ROWS - 1) / FS_MAX_ROWS;
    const int rows = (((M + tiles - 1) / tiles + 15) & ~15);
    return {most < 1 ? 1 : tiles < most ? tiles : most, rows};
}
extern "C" long long rv_gemm_f32_split_scratch(int M, int K) {
    if (M <= 0 || K <= 0) return 0;
    const FsRows r = fs_rows(M, K);
    return (long long)r.tiles * r.rows * ((K + FS_BK - 1) / FS_BK) * FS_BK * FS_PARTS / 2;
}

// K a multiple of 4, x, w and scratch (rv_gemm_f32_split_scratch floats) on 16-byte boundaries.
extern "C" int rv_gemm_f32_split(const float* x, const float* w, float* y, float* scratch, int* status, int M, int N,
                                 int K, void* stream) {
    if (M == 0 || N == 0) return 0;
    if (M < 0 || N < 0 || K < 4 || K % 4) RV_FAIL("gemm_f32_split: bad sizes");
    if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)scratch) & 15) RV_FAIL("gemm_f32_split: the operands must be 16-byte aligned");
    const FsRows r = fs_rows(M, K);
    if ((N + FS_BN - 1) / FS_BN > 65535 || (long long)(K + FS_BK - 1) / FS_BK > 0x7fffffffLL) RV_FAIL("gemm_f32_split: too many columns");
    cudaStream_t s = (cudaStream_t)stream;
    for (int m0 = 0; m0 < M; m0 += r.tiles * r.rows) {
        const int m = M - m0 < r.tiles * r.rows ? M - m0 : r.tiles * r.rows, tiles = (m + r.rows - 1) / r.rows;
        const float* xm = x + (size_t)m0 * K;
        float* ym = y + (size_t)m0 * N;
        rv_launch(fs_split_kernel, dim3((K + FS_BK - 1) / FS_BK, tiles), dim3(256), 0, s, xm, scratch, m, K, r.rows);
        RV_CHECK_LAUNCH("gemm_f32_split_parts");
        cudaError_t e = cudaErrorInvalidValue;
        switch (r.rows) {
#define FS_CASE(NT) case NT: e = fs_launch<NT>(scratch, xm, w, ym, status, m, N, K, tiles, s); break;
            FS_CASE(16) FS_CASE(32) FS_CASE(48) FS_CASE(64) FS_CASE(80) FS_CASE(96)
            FS_CASE(112) FS_CASE(128) FS_CASE(144) FS_CASE(160)
#undef FS_CASE
        }
        if (e != cudaSuccess) RV_FAIL("gemm_f32_split: %s", cudaGetErrorString(e));
        RV_CHECK_LAUNCH("gemm_f32_split");
    }
    return 0;
}
