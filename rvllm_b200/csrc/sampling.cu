// Sampling on the device: greedy argmax, and temperature with nucleus (top-p) filtering.
// Rows of float32 logits stay on the device, so only token ids cross to the host.
//
// argmax: the first maximum wins, NaN never wins, a row with nothing above -inf gives
// 0 (the reference's argmax.cu:1-4 and src/sampler.rs:68-78).
//
// sample: a row with T <= 0 is greedy (as argmax).  Otherwise p_i = exp(l_i / T - max)
// (src/sampler.rs:80-91); the nucleus is the set
// {p_i >= tau} for the largest tau whose set has mass >= top_p * total, found by the bit
// pattern of tau (positive floats order like their bits): rows up to 131,072 values by three
// rounds of a histogram, a cluster of blocks a row, longer ones by bisection, a block a row; tokens
// tied with the last kept one are kept (the reference keeps a sorted prefix,
// src/sampler.rs:93-117).  The draw u in [0,1) is a counter-based hash of (seed,
// counter), so a request's stream depends on nothing else in the batch; the token is the
// first in index order whose cumulative kept mass reaches u * kept mass (the reference
// walks in descending-probability order with a stateful generator,
// src/sampler.rs:118-129).  Plain reference: tests/plain_ops.py sample_row.
#include "common.cuh"

// Stage 1: block (row, part) scans its slice of the row; stage 2 combines the parts.
// A candidate is (value, index); the better one has the larger value, or on a tie the
// smaller index, so the result does not depend on how the row is cut.
struct RvBest { float v; int i; };
__device__ __forceinline__ RvBest rv_better(RvBest a, RvBest b) {
    return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}
__device__ __forceinline__ RvBest rv_block_best(RvBest x, float* sv, int* si) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        RvBest y;
        y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
        y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
        x = rv_better(x, y);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sv[warp] = x.v; si[warp] = x.i; }
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        x.v = lane < nw ? sv[lane] : -INFINITY;
        x.i = lane < nw ? si[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            RvBest y;
            y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
            y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
            x = rv_better(x, y);
        }
    }
    return x;   // valid in warp 0
}

__global__ void argmax_parts_kernel(const float* __restrict__ logits, float* __restrict__ part_v,
                                    int* __restrict__ part_i, int vocab, int parts) {
    rv_pdl_prologue();
    __shared__ float sv[32];
    __shared__ int si[32];
    const float* row = logits + (size_t)blockIdx.x * vocab;
    const int per = (vocab + parts - 1) / parts;
    const int a = blockIdx.y * per, b = min(vocab, a + per);
    RvBest best = {-INFINITY, 0x7fffffff};
    // four loads in flight per thread (a load and its compare per iteration would cost one
    // memory latency each); compared in index order, and strict, so the earliest maximum stays
    const int bd = blockDim.x;
    for (int i = a + threadIdx.x; i < b; i += 4 * bd) {
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = i + k * bd < b ? row[i + k * bd] : -INFINITY;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (v[k] > best.v) { best.v = v[k]; best.i = i + k * bd; }   // false for NaN
    }
    best = rv_block_best(best, sv, si);
    if (threadIdx.x == 0) {
        part_v[blockIdx.x * parts + blockIdx.y] = best.v;
        part_i[blockIdx.x * parts + blockIdx.y] = best.i;
    }
}

__global__ void argmax_final_kernel(const float* __restrict__ part_v, const int* __restrict__ part_i,
                                    int* __restrict__ out, int parts) {
    rv_pdl_prologue();
    RvBest best = {-INFINITY, 0x7fffffff};
    for (int p = threadIdx.x; p < parts; p += 32) {
        RvBest c = {part_v[blockIdx.x * parts + p], part_i[blockIdx.x * parts + p]};
        best = rv_better(best, c);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        RvBest y;
        y.v = __shfl_xor_sync(0xffffffffu, best.v, o);
        y.i = __shfl_xor_sync(0xffffffffu, best.i, o);
        best = rv_better(best, y);
    }
    if (threadIdx.x == 0) out[blockIdx.x] = best.i == 0x7fffffff ? 0 : best.i;
}

#define RV_ARGMAX_MAX_PARTS 64

// `scratch` holds rows * parts (value, index) pairs: rows * parts * 8 bytes, parts as
// given by rv_argmax_parts.
extern "C" int rv_argmax_parts(int n_rows, int vocab) {
    int parts = 1;
    const int want = 2 * rv_sm_count();        // two blocks per SM
    while (parts < RV_ARGMAX_MAX_PARTS && n_rows * parts < want && vocab / (parts * 2) >= 1024) parts *= 2;
    return parts;
}

extern "C" int rv_argmax(const float* logits, int* out, void* scratch, long long scratch_bytes,
                         int n_rows, int vocab, void* stream) {
    if (n_rows == 0) return 0;
    if (n_rows < 0 || vocab <= 0) RV_FAIL("argmax: bad sizes");
    if (n_rows > 65535) RV_FAIL("argmax: too many rows for one launch");
    const int parts = rv_argmax_parts(n_rows, vocab);
    if ((long long)n_rows * parts * 8 > scratch_bytes) RV_FAIL("argmax: scratch too small");
    float* part_v = (float*)scratch;
    int* part_i = (int*)((char*)scratch + (size_t)n_rows * parts * 4);
    cudaStream_t s = (cudaStream_t)stream;
    rv_launch(argmax_parts_kernel, dim3(dim3(n_rows, parts)), dim3(256), 0, s, logits, part_v, part_i, vocab, parts);
    RV_CHECK_LAUNCH("argmax");
    rv_launch(argmax_final_kernel, dim3(n_rows), dim3(32), 0, s, part_v, part_i, out, parts);
    RV_CHECK_LAUNCH("argmax");
    return 0;
}

__device__ __forceinline__ float rv_uniform(unsigned long long seed, unsigned long long counter) {
    unsigned long long z = seed + (counter + 1ull) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z = z ^ (z >> 31);
    return (float)(z >> 40) * (1.0f / 16777216.0f);
}

#define RV_SAMPLE_THREADS 1024

// A row whose temperature is not positive is greedy: the first maximum, NaN never wins, nothing
// above -inf gives 0 (as `rv_argmax`).  Every thread of the block calls it.
__device__ __forceinline__ void rv_sample_greedy_row(const float* row, int a, int b, int* out) {
    __shared__ float gv[32];
    __shared__ int gi[32];
    RvBest best = {-INFINITY, 0x7fffffff};
    for (int i = a; i < b; ++i) {
        const float v = row[i];
        if (v > best.v) best = RvBest{v, i};
    }
    best = rv_block_best(best, gv, gi);
    if (threadIdx.x == 0) *out = best.i == 0x7fffffff ? 0 : best.i;
}

__global__ void __launch_bounds__(RV_SAMPLE_THREADS) sample_kernel(
    const float* __restrict__ logits, const float* __restrict__ temperature,
    const float* __restrict__ top_p, const long long* __restrict__ seed,
    const long long* __restrict__ counter, int* __restrict__ out, int vocab) {
    rv_pdl_prologue();
    __shared__ float scratch[33];
    __shared__ float seg_sum[RV_SAMPLE_THREADS];
    __shared__ int chosen_thread;
    const int m = blockIdx.x;
    const float* row = logits + (size_t)m * vocab;
    const float T = temperature[m];
    const float inv_t = 1.f / T;
    // each thread owns a contiguous segment of the vocabulary
    const int seg = (vocab + blockDim.x - 1) / blockDim.x;
    const int a = min(vocab, (int)threadIdx.x * seg), b = min(vocab, a + seg);
    if (!(T > 0.f)) {
        rv_sample_greedy_row(row, a, b, out + m);
        return;
    }

    float mx = -INFINITY;
    for (int i = a; i < b; ++i) mx = fmaxf(mx, row[i] * inv_t);
    mx = rv_block_max(mx, scratch);
    float sum = 0.f;
    for (int i = a; i < b; ++i) sum += expf(row[i] * inv_t - mx);
    const float total = rv_block_sum(sum, scratch);

    // nucleus threshold: the largest tau with mass{p >= tau} >= top_p * total
    float tau = 0.f;
    const float tp = top_p[m];
    if (tp < 1.f) {
        const float need = tp * total;
        unsigned lo = 0u, hi = 0x3f800000u;   // p is in (0, 1]; tau = lo always qualifies
        while (lo < hi) {
            const unsigned mid = lo + (hi - lo + 1) / 2;
            const float cand = __uint_as_float(mid);
            float mass = 0.f;
            for (int i = a; i < b; ++i) {
                const float p = expf(row[i] * inv_t - mx);
                if (p >= cand) mass += p;
            }
            mass = rv_block_sum(mass, scratch);
            if (mass >= need) lo = mid; else hi = mid - 1;
        }
        tau = __uint_as_float(lo);
    }
    float kept = 0.f;
    for (int i = a; i < b; ++i) {
        const float p = expf(row[i] * inv_t - mx);
        if (p >= tau) kept += p;
    }
    seg_sum[threadIdx.x] = kept;
    const float kept_total = rv_block_sum(kept, scratch);   // also orders the seg_sum writes
    const float target = rv_uniform((unsigned long long)seed[m], (unsigned long long)counter[m]) *
                         kept_total;
    if (threadIdx.x == 0) {
        // walk the segment sums in order; 1024 additions
        float acc = 0.f;
        int t = 0, last = 0;
        for (t = 0; t < (int)blockDim.x; ++t) {
            if (seg_sum[t] > 0.f) last = t;
            if (seg_sum[t] > 0.f && acc + seg_sum[t] >= target) break;
            acc += seg_sum[t];
        }
        if (t == (int)blockDim.x) {   // rounding left the target past the end
            t = last;
            acc = -INFINITY;
        }
        chosen_thread = t;
        scratch[0] = acc;
    }
    __syncthreads();
    if ((int)threadIdx.x == chosen_thread) {
        float acc = scratch[0];
        int pick = -1, last = a;
        for (int i = a; i < b; ++i) {
            const float p = expf(row[i] * inv_t - mx);
            if (p >= tau && p > 0.f) {
                last = i;
                acc += p;
                if (acc >= target) {
                    pick = i;
                    break;
                }
            }
        }
        out[m] = pick >= 0 ? pick : last;
    }
}

// The same with the row read from memory once and kept in the registers of a cluster of up to
// eight blocks.  Warp w of the cluster owns the `rows * 32` consecutive values from w * rows * 32
// on, lane l the values j * 32 + l of them: a load of the warp is 128 contiguous bytes.
//
// The nucleus threshold is found by its bit pattern's parts in three rounds of a histogram over the
// values that agree with the parts found so far (for 19, 10 and 9 bits).  Values of a bin share
// their exponent, so a bin's mass is count * (the bin's first mantissa) + the sum of what the
// mantissas have beyond it: two integer additions a value, exact in any order.  After one cluster
// barrier every block adds the blocks' bins, and a suffix sum over them (float64) finds the bin in
// which the mass from the top reaches what is needed; all blocks find the same one.  Values so
// small that all of them together cannot decide have no bins.
//
// The walk to the drawn token follows index order: a prefix over the warps' kept masses finds the
// warp, its rows of 32 the row, a prefix over the lanes the token.  Sums are taken in another
// order than in `sample_kernel`, so a draw that falls within float32 rounding of a boundary may
// pick the neighbouring kept token there; both follow the definition in tests/plain_ops.py
// sample_row.
//
// Bound by latency: seven cluster barriers and the reductions between them (a row of 65,536 logits
// is 256 KB, some 2 us for eight multiprocessors).  65,536 logits, top-p 0.95, against one block of
// 1,024 threads a row that halves the range of patterns thirty times: 8 rows 81 -> 22 us, 64 rows
// 81 -> 40, 256 rows 163 -> 143; without a nucleus 30 -> 10.  Cutting the range into four with a
// cluster barrier per cut (16 of them): 36 us and, at 64 rows, 90.
#define RV_SAMPLE_CT 256                    // threads a block of a cluster
#define RV_SAMPLE_CLUSTER 8                 // the portable cluster size

__device__ __forceinline__ void rv_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// `v` to the same place of block `rank`'s shared memory.
__device__ __forceinline__ void rv_cluster_store(float* local, unsigned rank, float v) {
    unsigned at = (unsigned)__cvta_generic_to_shared(local), remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}
// Sixteen bytes of block `rank`'s copy of `local`.
__device__ __forceinline__ uint4 rv_cluster_load4(const unsigned* local, unsigned rank) {
    unsigned at = (unsigned)__cvta_generic_to_shared(local), remote;
    uint4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(rank));
    asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(remote) : "memory");
    return v;
}

// The bins of the rounds: how many values, and the sum of their mantissas beyond the bin's first.
template <int N1, int N2, int N3>
struct RvBins {
    struct { unsigned count[N1], rest[N1]; } a;
    struct { unsigned count[N2], rest[N2]; } b;
    struct { unsigned count[N3]; } c;
};
struct RvPick { double sums[RV_SAMPLE_CT / 32]; double above; int at; };

// The highest of `n` bins (at most N, a multiple of four) for which the mass of the values in it and
// above it, with `above`, is at least `need` (-1: none); `above` becomes the mass above that bin.
// Bin i holds the values whose bits are first_bits + (i << shift) + anything below.  Every block of
// the cluster reads the bins of all.
template <int N, bool REST>
__device__ __forceinline__ int rv_pick_bin(const unsigned* count, const unsigned* rest, int blocks, int n,
                                           unsigned first_bits, int shift, float need, double& above,
                                           RvPick& pick) {
    constexpr int GROUPS = (N + 4 * RV_SAMPLE_CT - 1) / (4 * RV_SAMPLE_CT), EACH = 4 * GROUPS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double mass[EACH], own = 0.;
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
        const int i0 = threadIdx.x * EACH + 4 * g;
        unsigned num[4] = {0, 0, 0, 0};
        unsigned long long r[4] = {0, 0, 0, 0};
        uint4 q[RV_SAMPLE_CLUSTER];
#pragma unroll
        for (int b = 0; b < RV_SAMPLE_CLUSTER; ++b) {    // all requested before any is used
            q[b] = make_uint4(0u, 0u, 0u, 0u);
            if (b < blocks && i0 < n) q[b] = rv_cluster_load4(count + i0, b);
        }
#pragma unroll
        for (int b = 0; b < RV_SAMPLE_CLUSTER; ++b) {
            num[0] += q[b].x; num[1] += q[b].y; num[2] += q[b].z; num[3] += q[b].w;
        }
        if (REST) {
#pragma unroll
            for (int b = 0; b < RV_SAMPLE_CLUSTER; ++b)
                if (b < blocks && i0 < n) q[b] = rv_cluster_load4(rest + i0, b);
#pragma unroll
            for (int b = 0; b < RV_SAMPLE_CLUSTER; ++b)
                if (b < blocks && i0 < n) { r[0] += q[b].x; r[1] += q[b].y; r[2] += q[b].z; r[3] += q[b].w; }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned bits = first_bits + ((unsigned)(i0 + k) << shift), e = bits >> 23;
            const unsigned long long m0 = (bits & 0x7fffffu) | (e ? 0x800000u : 0u);
            const double unit = __longlong_as_double((long long)((e ? e : 1u) - 150 + 1023) << 52);
            mass[4 * g + k] = num[k] ? (double)(num[k] * m0 + r[k]) * unit : 0.;
            own += mass[4 * g + k];
        }
    }
    double from = own;                                   // this thread's bins and those above, in the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_down_sync(0xffffffffu, from, o);
        if (lane + o < 32) from += up;
    }
    if (lane == 0) pick.sums[warp] = from;
    if (threadIdx.x == 0) pick.at = -1;
    __syncthreads();
    double before = above + (from - own);
    for (int w = warp + 1; w < RV_SAMPLE_CT / 32; ++w) before += pick.sums[w];
    // one thread at the most, but for rounding: then the highest bin counts
    int at = -1;
    double run = before;
    if (before < (double)need && before + own >= (double)need) {
#pragma unroll
        for (int k = EACH - 1; k >= 0; --k)
            if (at < 0) {
                if (run + mass[k] >= (double)need) at = (int)threadIdx.x * EACH + k;
                else run += mass[k];
            }
        if (at >= 0) atomicMax(&pick.at, at);
    }
    __syncthreads();
    const int found = pick.at;
    if (found >= 0 && at == found) pick.above = run;
    __syncthreads();
    if (found >= 0) above = pick.above;
    return found;                                        // (a cluster barrier comes before the next round)
}

// MANY rows (up to 32 values a thread): four blocks a multiprocessor (64 registers), so that more rows are worked at once; few
// rows have registers for all loads in flight (8 rows: 22 against 25 us; 64 rows: 51 against 40).
template <int V, bool MANY>
__global__ void __launch_bounds__(RV_SAMPLE_CT, MANY ? 4 : 2) sample_cluster_kernel(
    const float* __restrict__ logits, const float* __restrict__ temperature,
    const float* __restrict__ top_p, const long long* __restrict__ seed,
    const long long* __restrict__ counter, int* __restrict__ out, int vocab, int rows) {
    constexpr int WARPS = RV_SAMPLE_CT / 32, MOST = WARPS * RV_SAMPLE_CLUSTER;
    // the rounds' bins: bits from S1 up, from S3 up, the rest.  A bin's mantissas beyond its first add
    // up to less than 2^32 in a block (19 bits, 8,192 values); 1.0 is in bin TOP; N1 bins reach
    // from there down over 63 powers of two.
    constexpr int S1 = V <= 32 ? 19 : 18, S3 = S1 / 2;
    constexpr unsigned TOP = 0x3f800000u >> S1, N1 = 64u << (23 - S1), N2 = 1u << (S1 - S3), N3 = 1u << S3;
    // what the cluster's warps tell one another; two sets, so that one barrier a round is enough
    __shared__ float told[2][2][MOST];
    __shared__ __align__(16) RvBins<N1, N2, N3> bins;
    __shared__ RvPick pick;
    rv_pdl_launch_dependents();
    for (int i = threadIdx.x; i < (int)(sizeof(bins) / 16); i += RV_SAMPLE_CT)
        ((uint4*)&bins)[i] = make_uint4(0u, 0u, 0u, 0u);
    rv_pdl_wait();
    const int blocks = gridDim.x, rank = blockIdx.x, m = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = rank * WARPS + (threadIdx.x >> 5);
    const int n_warps = blocks * WARPS;
    const float* row = logits + (size_t)m * vocab;
    const float T = temperature[m], tp = top_p[m];
    const bool greedy = !(T > 0.f);
    const float inv_t = greedy ? 1.f : 1.f / T;
    const int first = warp * rows * 32 + lane;           // this thread's value j is row[first + 32 j]
    float p[V];
#pragma unroll
    for (int j = 0; j < V; ++j)
        p[j] = (j < rows && first + 32 * j < vocab) ? row[first + 32 * j] * inv_t : -INFINITY;
    rv_cluster_sync();                                   // every block has begun: its memory may be written

    int set = 0;
    // lane `to` of the warp leaves (x, y), the same in every lane, with block `to`
    auto tell = [&](float x, float y) {
        if (lane < blocks) {
            rv_cluster_store(&told[set][0][warp], lane, x);
            rv_cluster_store(&told[set][1][warp], lane, y);
        }
        rv_cluster_sync();
        set ^= 1;
    };
    auto heard = [&](int k, int w) { return told[set ^ 1][k][w]; };

    if (greedy) {
        RvBest best = {-INFINITY, 0x7fffffff};
#pragma unroll
        for (int j = 0; j < V; ++j)
            if (p[j] > best.v) best = RvBest{p[j], first + 32 * j};          // false for NaN
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            RvBest y;
            y.v = __shfl_xor_sync(0xffffffffu, best.v, o);
            y.i = __shfl_xor_sync(0xffffffffu, best.i, o);
            best = rv_better(best, y);
        }
        tell(best.v, __int_as_float(best.i));
        if (rank != 0 || threadIdx.x != 0) return;
        for (int w = 0; w < n_warps; ++w)
            best = rv_better(best, RvBest{heard(0, w), __float_as_int(heard(1, w))});
        out[m] = best.i == 0x7fffffff ? 0 : best.i;
        return;
    }

    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < V; ++j) mx = fmaxf(mx, p[j]);
    mx = rv_warp_max(mx);
    tell(mx, 0.f);
    for (int w = lane; w < n_warps; w += 32) mx = fmaxf(mx, heard(0, w));
    mx = rv_warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < V; ++j) {
        p[j] = expf(p[j] - mx);
        sum += p[j];
    }
    tell(rv_warp_sum(sum), 0.f);
    // over the cluster's warps, in the same order in every warp
    float total = 0.f;
    for (int w = lane; w < n_warps; w += 32) total += heard(0, w);
    total = rv_warp_sum(total);

    // the largest tau whose set {p >= tau} has the wanted mass; 0 (all are kept) if no set has it
    float tau = 0.f;
    if (tp < 1.f) {
        const float need = tp * total;
        if (need <= 0.f) {
            tau = 1.f;                                   // the largest alone
        } else {
            // `vocab` values below this one have at most half of the mass that may be missing, or
            // are beyond what float32 sums of at least 1 can hold
            const float least = 1.f - tp > 1e-3f ? fminf(0.5f * (1.f - tp) * total / (float)vocab, 1.f)
                                                 : 1.0842022e-19f;                      // 2^-63
            const unsigned base = max(__float_as_uint(least) >> S1, TOP - (N1 - 4)) & ~3u;
#pragma unroll
            for (int j = 0; j < V; ++j) {
                const unsigned bits = __float_as_uint(p[j]);
                if (p[j] > 0.f && bits >> S1 >= base) {
                    atomicAdd(&bins.a.count[(bits >> S1) - base], 1u);
                    atomicAdd(&bins.a.rest[(bits >> S1) - base], bits & ((1u << S1) - 1u));
                }
            }
            rv_cluster_sync();
            double above = 0.;
            int at = rv_pick_bin<N1, true>(bins.a.count, bins.a.rest, blocks, (int)(TOP - base + 1), base << S1, S1,
                                           need, above, pick);
            if (at >= 0) {
                unsigned found = base + (unsigned)at;
#pragma unroll
                for (int j = 0; j < V; ++j) {
                    const unsigned bits = __float_as_uint(p[j]);
                    if (bits >> S1 == found && p[j] > 0.f) {
                        const unsigned k = (bits >> S3) & (N2 - 1u);
                        atomicAdd(&bins.b.count[k], 1u);
                        atomicAdd(&bins.b.rest[k], bits & (N3 - 1u));
                    }
                }
                rv_cluster_sync();
                // (the lowest bin is taken if rounding of the sums leaves none)
                at = rv_pick_bin<N2, true>(bins.b.count, bins.b.rest, blocks, N2, found << S1, S3, need, above, pick);
                found = found * N2 + (unsigned)max(at, 0);
#pragma unroll
                for (int j = 0; j < V; ++j) {
                    const unsigned bits = __float_as_uint(p[j]);
                    if (bits >> S3 == found && p[j] > 0.f) atomicAdd(&bins.c.count[bits & (N3 - 1u)], 1u);
                }
                rv_cluster_sync();
                at = rv_pick_bin<N3, false>(bins.c.count, nullptr, blocks, N3, found << S3, 0, need, above, pick);
                tau = __uint_as_float(found << S3 | (unsigned)max(at, 0));
            }
        }
    }
    float kept = 0.f;
#pragma unroll
    for (int j = 0; j < V; ++j) {
        p[j] = (p[j] >= tau && p[j] > 0.f) ? p[j] : 0.f;                    // NaN: not kept
        kept += p[j];
    }
    tell(rv_warp_sum(kept), 0.f);

    // the warp in which the cumulative kept mass reaches the target (every warp finds the same one);
    // lane l looks at warps 2 l and 2 l + 1
    const float t0 = 2 * lane < n_warps ? heard(0, 2 * lane) : 0.f;
    const float t1 = 2 * lane + 1 < n_warps ? heard(0, 2 * lane + 1) : 0.f;
    float upto = t0 + t1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += up;
    }
    float before = __shfl_up_sync(0xffffffffu, upto, 1);
    if (lane == 0) before = 0.f;
    const float target = rv_uniform((unsigned long long)seed[m], (unsigned long long)counter[m]) *
                         __shfl_sync(0xffffffffu, upto, 31);
    const unsigned hit0 = __ballot_sync(0xffffffffu, t0 > 0.f && before + t0 >= target);
    const unsigned hit1 = __ballot_sync(0xffffffffu, t1 > 0.f && before + t0 + t1 >= target);
    int chosen;
    bool past_end = false;
    float run = 0.f;
    if (hit0 | hit1) {
        const int l = __ffs((int)(hit0 | hit1)) - 1;
        const bool even = (hit0 >> l) & 1u;
        chosen = 2 * l + (even ? 0 : 1);
        run = __shfl_sync(0xffffffffu, even ? before : before + t0, l);
    } else {                              // rounding left the target past the end: the last kept token
        const unsigned any0 = __ballot_sync(0xffffffffu, t0 > 0.f), any1 = __ballot_sync(0xffffffffu, t1 > 0.f);
        const int l = (any0 | any1) ? 31 - __clz((int)(any0 | any1)) : 0;
        chosen = 2 * l + (int)((any1 >> l) & 1u);
        past_end = true;
    }
    if (warp != chosen) return;
    int token = -1, last = -1;
#pragma unroll
    for (int j = 0; j < V; ++j) {
        const float q = p[j];
        const float rowsum = rv_warp_sum(q);
        const unsigned keepers = __ballot_sync(0xffffffffu, q > 0.f);
        const int at = warp * rows * 32 + j * 32;
        if (keepers) last = at + (31 - __clz((int)keepers));
        if (token < 0 && !past_end && rowsum > 0.f && run + rowsum >= target) {
            // inclusive prefix over the lanes, then the first kept lane that reaches the target
            float pre = q;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float up = __shfl_up_sync(0xffffffffu, pre, o);
                if (lane >= o) pre += up;
            }
            const unsigned hit = __ballot_sync(0xffffffffu, q > 0.f && run + pre >= target);
            token = at + (hit ? __ffs((int)hit) - 1 : 31 - __clz((int)keepers));  // rounding: the row's last
        }
        run += rowsum;
    }
    if (lane == 0) out[m] = token >= 0 ? token : (last >= 0 ? last : 0);
}

// A row over `blocks` blocks of a cluster, V values a thread.
template <int V, bool MANY>
static cudaError_t rv_sample_cluster(const float* logits, const float* temperature, const float* top_p,
                                     const long long* seed, const long long* counter, int* out,
                                     int n_rows, int vocab, int blocks, cudaStream_t stream) {
    const int rows = (vocab + blocks * RV_SAMPLE_CT - 1) / (blocks * RV_SAMPLE_CT);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks, n_rows);
    cfg.blockDim = dim3(RV_SAMPLE_CT);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = rv_pdl_enabled();
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, sample_cluster_kernel<V, MANY>, logits, temperature, top_p, seed, counter,
                              out, vocab, rows);
}

// 1: rows that fit stay on the chip (the default); 0: every pass re-reads the logits
// (RVLLM_SAMPLE_ONCHIP=0).  The switch is for tests and timing.
static int rv_sample_onchip = -1;
extern "C" void rv_sample_set_onchip(int on) { rv_sample_onchip = on ? 1 : 0; }

extern "C" int rv_sample(const float* logits, const float* temperature, const float* top_p,
                         const long long* seed, const long long* counter, int* out, int n_rows,
                         int vocab, void* stream) {
    if (n_rows == 0) return 0;
    if (n_rows < 0 || vocab <= 0) RV_FAIL("sample: bad sizes");
    if (rv_sample_onchip < 0) {
        const char* e = getenv("RVLLM_SAMPLE_ONCHIP");
        rv_sample_onchip = (e && e[0] == '0') ? 0 : 1;
    }
    // Sixteen values a thread (32 with many rows: 64 rows of 32,768 logits take 25 us so, 44 with
    // 16), a block more until the cluster is full, then more values a thread; as many rows as a
    // grid's second dimension has.  Longer rows re-read the logits.
    const bool many = n_rows > 32;
    int blocks = 1;
    while (blocks < RV_SAMPLE_CLUSTER && blocks * RV_SAMPLE_CT * (many ? 32 : 16) < vocab) blocks *= 2;
    const int each = (int)(((long long)vocab + blocks * RV_SAMPLE_CT - 1) / (blocks * RV_SAMPLE_CT));
    if (rv_sample_onchip && each <= 64 && n_rows <= 65535) {
        cudaStream_t s = (cudaStream_t)stream;
#define RV_SAMPLE_CASE(V)                                                                                       \
    (many ? rv_sample_cluster<V, true>(logits, temperature, top_p, seed, counter, out, n_rows, vocab, blocks, s) \
          : rv_sample_cluster<V, false>(logits, temperature, top_p, seed, counter, out, n_rows, vocab, blocks, s))
        const cudaError_t e = each <= 16 ? RV_SAMPLE_CASE(16)
                              : each <= 24 ? RV_SAMPLE_CASE(24)
                              : each <= 32 ? RV_SAMPLE_CASE(32)
                              : each <= 40
                                  ? rv_sample_cluster<40, false>(logits, temperature, top_p, seed, counter, out, n_rows, vocab, blocks, s)
                                  : rv_sample_cluster<64, false>(logits, temperature, top_p, seed, counter, out, n_rows, vocab, blocks, s);
#undef RV_SAMPLE_CASE
        if (e != cudaSuccess) RV_FAIL("sample: %s", cudaGetErrorString(e));
    } else {
        rv_launch(sample_kernel, dim3(n_rows), dim3(RV_SAMPLE_THREADS), 0, (cudaStream_t)stream,
                  logits, temperature, top_p, seed, counter, out, vocab);
    }
    RV_CHECK_LAUNCH("sample");
    return 0;
}
