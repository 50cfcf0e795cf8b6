// How the streaming decode attention (attention_mma.cu) shares a step's key tiles out, for it and for the
// merge of its segments (attention_simt.cu).
//
// The tiles (64 keys) of all requests, one after the other, are cut evenly, to within one tile, into as many
// runs as there are teams of warps; a team has a warp per key/value head (and 16 query heads of it).  What a run
// has of a request is a segment.  From one segment to the next the run's or the request's number grows, so the sum
// of both is a place of its own: a head's segments take `teams + n_reqs` places.  All follows from the contexts'
// lengths, which are there before the launch before has ended.
#pragma once

#define RV_STREAM_TILE 64            // keys
#define RV_STREAM_WARPS 6            // a block, one block a multiprocessor

// Keys that a launch takes of a request: what it was told of, in whole splits of 256 as the other kernels.
static inline int rv_stream_keys(int max_ctx_len) {
    return max_ctx_len > 0 ? (max_ctx_len + 255) / 256 * 256 : 256;
}
static inline int rv_stream_heads(int num_heads, int num_kv_heads) {
    return num_kv_heads * ((num_heads / num_kv_heads + 15) / 16);
}
// Many heads: four runs a warp or so, as a team's size need not divide the warps.
static inline int rv_stream_teams(int num_heads, int num_kv_heads, int n_sms) {
    const int P = rv_stream_heads(num_heads, num_kv_heads), warps = n_sms * RV_STREAM_WARPS;
    return 4 * P <= warps ? warps / P : (4 * warps + P - 1) / P;
}
// Bytes: rows of 64 for every head and place, then an offset and a sum for each.
static inline long long rv_stream_bytes(int n_reqs, int num_heads, int teams) {
    return (long long)num_heads * (teams + n_reqs) * (64 * 4 + 8);
}

// A warp's view of the shares.
struct RvStreamShares {
    const int* ctx_lens;
    int n_reqs, window, max_ctx, total, used;
    bool narrow;
    int grp, grp_len;                // this lane's context length of the 32 requests from `grp` on

    __device__ __forceinline__ int first_tile(int clen) const {
        return window > 0 ? max(0, clen - window) / RV_STREAM_TILE : 0;
    }
    // A request longer than the launch was told of has none: the merge marks its row.
    __device__ __forceinline__ int tiles_of(int clen) const {
        return clen > 0 && clen <= max_ctx ? (clen - 1) / RV_STREAM_TILE - first_tile(clen) + 1 : 0;
    }
    __device__ __forceinline__ void load_group(int at) {
        const int r = at + (threadIdx.x & 31);
        grp = at;
        grp_len = r < n_reqs ? ctx_lens[r] : 0;
    }
    __device__ __forceinline__ RvStreamShares(const int* lens, int reqs, int win, int most, int teams)
        : ctx_lens(lens), n_reqs(reqs), window(win), max_ctx(most), total(0), grp(0), grp_len(0) {
        for (int at = 0; at < n_reqs; at += 32) {
            load_group(at);
            total += __reduce_add_sync(0xffffffffu, tiles_of(grp_len));
        }
        used = min(teams, max(1, total));
        narrow = (unsigned long long)total * used <= 0xffffffffull;
    }
    // (A division of 64 bits takes long enough to be seen: only where 32 do not hold it.)
    __device__ __forceinline__ int mul_div(unsigned a, unsigned b, unsigned less, unsigned by) const {
        return (int)(narrow ? (a * b - less) / by : (unsigned)(((unsigned long long)a * b - less) / by));
    }
    __device__ __forceinline__ int run_start(int run) const { return mul_div(run, total, 0, used); }
    __device__ __forceinline__ int run_of(int tile) const { return mul_div(tile + 1, used, 1, total); }
};
