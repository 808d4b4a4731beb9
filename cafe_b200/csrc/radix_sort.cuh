// radix_sort.cuh -- stable LSD radix sort of lookups on sm_100a, for this library's sorts: lookups by main-table bucket,
// lookups by LRU-table bucket (the order in which the sequential insert of tricks/sketch.cpp:268-296 meets the ids of one
// bucket must be kept, hence stable), and the scatter's lookups by table row.  Keys have 10 to 21 bits, so one to three
// passes of up to 10 bits do.
//
// What moves is one 8-byte pair per lookup: (id, position) for the bucket orders, whose key is recomputed from the id in
// every step (a dozen instructions, cafe_hash with a CafeMod) instead of being carried beside it, and (row, position)
// for the row order.  Writes go to places a few pairs apart at best, so one 8-byte store instead of two or three 4-byte
// ones is what the scatter step is made of.
//
// Up to three independent sorts go in one batch.  A block owns a range of consecutive pairs of one sort; a pass is
//   histogram of the range's digits;
//   per digit, the pairs of the digits before it and of the same digit in the blocks before;
//   every pair to its place: that base + its rank among the range's pairs of the digit, ranks taken in index order
//   (warp match + per-warp counters), so equal keys keep their order.
// After the last pass the bucket ranges are written.
//
// Small batches are bound by launches and by the waits between the steps, large ones by L2 traffic.  So the steps exist
// in two forms: ONE launch with a thread-block cluster per sort, the histograms read from each other's shared memory and
// the hardware's cluster barrier between the steps; or a launch per step over as many blocks as there is work for.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "sketch_core.cuh"

#define CAFE_RS_THREADS 512
#define CAFE_RS_WARPS (CAFE_RS_THREADS / 32)
#define CAFE_RS_ITEMS 8
#define CAFE_RS_TILE (CAFE_RS_THREADS * CAFE_RS_ITEMS)   // pairs ranked at a time by one block
#define CAFE_RS_MAX_BITS 10
#define CAFE_RS_MAX_BINS (1 << CAFE_RS_MAX_BITS)
#define CAFE_RS_MAX_BLOCKS 296
#define CAFE_RS_MAX_SORTS 3
#define CAFE_RS_CLUSTER_MAX 8           // portable cluster size
// A cluster of eight blocks ranks 32 768 pairs at a time; up to four rounds of that cost less than the launches of the
// other form.  The three sorts of a step with 26 x 128 lookups take 17 us in their one launch (the 23 launches of a
// launch per step, sort and bucket index took 84 us one after the other), with 26 x 2048 lookups 49 us (98 us); with
// 26 x 65536, beside the row gather, 0.31 ms of kernel time in 7 launches (0.65 ms in 23).
#define CAFE_RS_CLUSTER_PAIRS (4 * CAFE_RS_CLUSTER_MAX * CAFE_RS_TILE)

struct CafeSortDesc {
    const uint32_t* in;      // ids or keys; the position of entry i is i
    CafeMod mod;             // .n keys; ids are hashed into them
    int32_t hashed;          // 0: `in` holds keys (< mod.n); 1: ids, key = cafe_hash(id, mod); 2: ids, key = id % mod.n
    int32_t n;               // pairs
    uint2* tmp;              // [n] pairs between two passes
    uint2* out;              // [n] sorted (id or key, position)
    int32_t* start;          // [mod.n + 1] first sorted index whose key is >= k, or null
    int32_t* scratch;        // cafe_rs_scratch_elems(n) int32: totals[digit], hist[block][digit]
    int32_t passes, bits, blocks;
};
struct CafeSortBatch {
    CafeSortDesc d[CAFE_RS_MAX_SORTS];
    int32_t count;
};
struct CafeSortShared {
    uint16_t cnt[CAFE_RS_WARPS][CAFE_RS_MAX_BINS];   // per warp: pairs of each digit seen so far, then the prefix over warps
    int32_t hist[CAFE_RS_MAX_BINS];                  // the range's pairs of each digit (read by the other blocks of a cluster)
    int32_t base[CAFE_RS_MAX_BINS];                  // next output index of the range's pairs of each digit
    int32_t warp[CAFE_RS_WARPS];
};

// blocks of a sort of n pairs in the launch-per-step form (a block ranks several tiles, one by one, where there are more)
static inline int cafe_rs_blocks(int64_t n) {
    const int64_t t = (n + CAFE_RS_TILE - 1) / CAFE_RS_TILE;
    return (int)(t < CAFE_RS_MAX_BLOCKS ? t : CAFE_RS_MAX_BLOCKS);
}
// scratch of a sort of at most `cap` pairs
static inline size_t cafe_rs_scratch_elems(int64_t cap) { return (size_t)CAFE_RS_MAX_BINS * (size_t)(cafe_rs_blocks(cap) + 1); }

__device__ __forceinline__ uint32_t cafe_rs_key(const CafeSortDesc& D, uint32_t a) {
    return D.hashed == 1 ? (uint32_t)cafe_hash(a, D.mod) : D.hashed == 2 ? a % (uint32_t)D.mod.n : a;
}
// the passes alternate between the two arrays so that the last one ends in `out`
__device__ __forceinline__ const uint2* cafe_rs_from(const CafeSortDesc& D, int pass) { return ((D.passes - pass) & 1) ? D.tmp : D.out; }
__device__ __forceinline__ uint2* cafe_rs_to(const CafeSortDesc& D, int pass) { return ((D.passes - 1 - pass) & 1) ? D.tmp : D.out; }
__device__ __forceinline__ void cafe_rs_range(const CafeSortDesc& D, int blk, int64_t* lo, int64_t* hi) {
    const int64_t len = (((int64_t)D.n + D.blocks - 1) / D.blocks + 31) & ~(int64_t)31;
    *lo = (int64_t)blk * len;
    *hi = *lo + len < D.n ? *lo + len : (int64_t)D.n;
}
// exclusive prefix of v over the block's threads
__device__ __forceinline__ int cafe_rs_block_exclusive(int v, int32_t* s_warp) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += t;
    }
    if (lane == 31) s_warp[w] = inc;
    __syncthreads();
    int before = 0;
#pragma unroll
    for (int q = 0; q < CAFE_RS_WARPS; ++q) before += q < w ? s_warp[q] : 0;
    return before + inc - v;
}

// step 1: digit histogram of the block's range, in S.hist
__device__ __forceinline__ void cafe_rs_hist(const CafeSortDesc& D, int pass, int blk, CafeSortShared& S) {
    const int bins = 1 << D.bits, shift = pass * D.bits;
    for (int d = threadIdx.x; d < bins; d += CAFE_RS_THREADS) S.hist[d] = 0;
    __syncthreads();
    int64_t lo, hi;
    cafe_rs_range(D, blk, &lo, &hi);
    const uint2* from = cafe_rs_from(D, pass);
    for (int64_t i0 = lo + threadIdx.x; i0 < hi; i0 += 8 * CAFE_RS_THREADS) {
        uint32_t a[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int64_t i = i0 + u * CAFE_RS_THREADS;
            a[u] = i < hi ? (pass == 0 ? D.in[i] : from[i].x) : 0u;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (i0 + u * CAFE_RS_THREADS < hi) atomicAdd(&S.hist[(cafe_rs_key(D, a[u]) >> shift) & (bins - 1)], 1);
    }
    __syncthreads();
}
// step 2's end: loc = totals of this thread's two digits, own = their place among the blocks -> S.base
__device__ __forceinline__ void cafe_rs_set_base(const CafeSortDesc& D, const int (&loc)[2], const int (&own)[2], CafeSortShared& S) {
    const int bins = 1 << D.bits, d = (int)threadIdx.x * 2;
    const int ex = cafe_rs_block_exclusive(loc[0] + loc[1], S.warp);
    if (d < bins) { S.base[d] = ex + own[0]; S.base[d + 1] = ex + loc[0] + own[1]; }
    __syncthreads();
}
// step 3: the block's pairs to their places (S.base set)
__device__ __forceinline__ void cafe_rs_scatter(const CafeSortDesc& D, int pass, int blk, CafeSortShared& S) {
    const int bins = 1 << D.bits, shift = pass * D.bits;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint2* from = cafe_rs_from(D, pass);
    uint2* to = cafe_rs_to(D, pass);
    int64_t lo, hi;
    cafe_rs_range(D, blk, &lo, &hi);
    for (int64_t t0 = lo; t0 < hi; t0 += CAFE_RS_TILE) {
        // a warp owns 32 * CAFE_RS_ITEMS consecutive pairs of the tile and walks them 32 at a time, so (iteration, lane)
        // is index order
        const int64_t base = t0 + (int64_t)w * (32 * CAFE_RS_ITEMS);
        uint2 e[CAFE_RS_ITEMS];
        uint32_t dr[CAFE_RS_ITEMS];   // digit, and rank << 16
#pragma unroll
        for (int it = 0; it < CAFE_RS_ITEMS; ++it) {
            const int64_t i = base + it * 32 + lane;
            e[it] = make_uint2(0u, 0u);
            if (i < hi) e[it] = pass == 0 ? make_uint2(D.in[i], (uint32_t)i) : from[i];
        }
        {
            uint4* z = reinterpret_cast<uint4*>(S.cnt[w]);
            for (int q = lane; q < bins / 8; q += 32) z[q] = make_uint4(0u, 0u, 0u, 0u);
            if (bins < 8 && lane < bins) S.cnt[w][lane] = 0;
        }
        __syncwarp();
#pragma unroll
        for (int it = 0; it < CAFE_RS_ITEMS; ++it) {
            const bool ok = base + it * 32 + lane < hi;
            const uint32_t d = (cafe_rs_key(D, e[it].x) >> shift) & (uint32_t)(bins - 1);
            // lanes beyond the end take digits of their own so that they match nobody
            const unsigned peers = __match_any_sync(0xffffffffu, ok ? d : (uint32_t)(bins + lane));
            const int ahead = __popc(peers & ((1u << lane) - 1u));
            const uint32_t before = ok ? S.cnt[w][d] : 0u;
            __syncwarp();
            if (ok && ahead == 0) S.cnt[w][d] = (uint16_t)(before + __popc(peers));
            __syncwarp();
            dr[it] = d | ((before + ahead) << 16);
        }
        __syncthreads();
        // prefix over the warps, two digits per thread (no carry between the halves: a tile has 4096 pairs)
        uint32_t run = 0;
        if ((int)threadIdx.x * 2 < bins) {
#pragma unroll
            for (int q = 0; q < CAFE_RS_WARPS; ++q) {
                uint32_t* c = reinterpret_cast<uint32_t*>(S.cnt[q]) + threadIdx.x;
                const uint32_t t = *c;
                *c = run;
                run += t;
            }
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < CAFE_RS_ITEMS; ++it) {
            const uint32_t d = dr[it] & 0xffffu;
            if (base + it * 32 + lane < hi) to[(int64_t)S.base[d] + S.cnt[w][d] + (dr[it] >> 16)] = e[it];
        }
        if (t0 + CAFE_RS_TILE < hi) {   // the next tile of the range continues behind this one
            __syncthreads();
            if ((int)threadIdx.x * 2 < bins) {
                S.base[2 * threadIdx.x] += (int)(run & 0xffffu);
                S.base[2 * threadIdx.x + 1] += (int)(run >> 16);
            }
            __syncthreads();
        }
    }
}
// after the last pass: start[k] = first sorted index whose key is >= k, for k in [0, mod.n].  Index i fills the entries
// from the key before it (exclusive) to its own; where a warp meets a wide gap (few lookups, many buckets) its lanes
// fill it together.
__device__ __forceinline__ void cafe_rs_starts(const CafeSortDesc& D, int warp, int nwarps) {
    const int lane = threadIdx.x & 31, M = D.n;
    for (int64_t i0 = (int64_t)warp * 32; i0 <= M; i0 += (int64_t)nwarps * 32) {
        const int64_t i = i0 + lane;
        int lo = 0, hi = -1;
        if (i <= M) {
            lo = (i == 0) ? 0 : (int)cafe_rs_key(D, D.out[i - 1].x) + 1;
            hi = (i == M) ? D.mod.n : (int)cafe_rs_key(D, D.out[i].x);
        }
        const bool wide = hi - lo >= 16;
        if (!wide)
            for (int k = lo; k <= hi; ++k) D.start[k] = (int)i;
        unsigned m = __ballot_sync(0xffffffffu, wide);
        while (m) {
            const int j = __ffs(m) - 1;
            m &= m - 1;
            const int a = __shfl_sync(0xffffffffu, lo, j), b = __shfl_sync(0xffffffffu, hi, j);
            for (int k = a + lane; k <= b; k += 32) D.start[k] = (int)(i0 + j);
        }
    }
}

// All passes of a sort whose blocks have at most a tile of pairs each: ranking the tile counts its digits as well, so there is
// no histogram step, and the pairs are spread over all warps however few they are.
// A sort of 2048 pairs by 18 638 buckets takes 12 us (21 with a histogram step and full tiles per warp), three sorts of 3328
// pairs 17 us (25).  Half-filled blocks in a larger cluster beat full ones (3 x 8547 pairs: 17 us against 22).
template <typename CLUSTER>
__device__ __forceinline__ void cafe_rs_tiles(const CafeSortDesc& D, const CLUSTER& cluster, int nblk, int blk, CafeSortShared& S) {
    const int bins = 1 << D.bits, d2 = (int)threadIdx.x * 2;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t lo, hi;
    cafe_rs_range(D, blk, &lo, &hi);
    const int len = (int)(hi > lo ? hi - lo : 0), items = (len + CAFE_RS_THREADS - 1) / CAFE_RS_THREADS, first = w * 32 * items;
    for (int pass = 0; pass < D.passes; ++pass) {
        const int shift = pass * D.bits;
        const uint2* from = cafe_rs_from(D, pass);
        uint2* to = cafe_rs_to(D, pass);
        uint2 e[CAFE_RS_ITEMS];
        uint32_t dr[CAFE_RS_ITEMS];   // digit, and rank << 16
#pragma unroll
        for (int it = 0; it < CAFE_RS_ITEMS; ++it) {
            const int i = first + it * 32 + lane;
            e[it] = make_uint2(0u, 0u);
            if (it < items && i < len) e[it] = pass == 0 ? make_uint2(D.in[lo + i], (uint32_t)(lo + i)) : from[lo + i];
        }
        {
            uint4* z = reinterpret_cast<uint4*>(S.cnt[w]);
            for (int q = lane; q < bins / 8; q += 32) z[q] = make_uint4(0u, 0u, 0u, 0u);
            if (bins < 8 && lane < bins) S.cnt[w][lane] = 0;
        }
        __syncwarp();
#pragma unroll
        for (int it = 0; it < CAFE_RS_ITEMS; ++it) {
            if (it >= items) break;   // block-uniform
            const bool ok = first + it * 32 + lane < len;
            const uint32_t d = (cafe_rs_key(D, e[it].x) >> shift) & (uint32_t)(bins - 1);
            const unsigned peers = __match_any_sync(0xffffffffu, ok ? d : (uint32_t)(bins + lane));
            const int ahead = __popc(peers & ((1u << lane) - 1u));
            const uint32_t before = ok ? S.cnt[w][d] : 0u;
            __syncwarp();
            if (ok && ahead == 0) S.cnt[w][d] = (uint16_t)(before + __popc(peers));
            __syncwarp();
            dr[it] = d | ((before + ahead) << 16);
        }
        __syncthreads();   // (also: everyone has read its pairs)
        uint32_t run = 0;
        if (d2 < bins) {
#pragma unroll
            for (int q = 0; q < CAFE_RS_WARPS; ++q) {
                uint32_t* c = reinterpret_cast<uint32_t*>(S.cnt[q]) + threadIdx.x;
                const uint32_t t = *c;
                *c = run;
                run += t;
            }
        }
        int loc[2] = {(int)(run & 0xffffu), (int)(run >> 16)}, own[2] = {0, 0};
        if (nblk > 1) {
            if (d2 < bins) { S.hist[d2] = loc[0]; S.hist[d2 + 1] = loc[1]; }
            cluster.sync();
            loc[0] = loc[1] = 0;
            if (d2 < bins) {
                for (int b = 0; b < nblk; ++b) {
                    const int2 h = *reinterpret_cast<const int2*>(cluster.map_shared_rank(S.hist, b) + d2);
                    loc[0] += h.x; loc[1] += h.y;
                    if (b < blk) { own[0] += h.x; own[1] += h.y; }
                }
            }
        }
        cafe_rs_set_base(D, loc, own, S);   // (its barriers also publish the prefixes over the warps)
#pragma unroll
        for (int it = 0; it < CAFE_RS_ITEMS; ++it) {
            if (it >= items) break;
            const uint32_t d = dr[it] & 0xffffu;
            if (first + it * 32 + lane < len) {
                to[(int64_t)S.base[d] + S.cnt[w][d] + (dr[it] >> 16)] = e[it];
            }
        }
        cluster.sync();
    }
}
// a cluster per sort
static __global__ void __launch_bounds__(CAFE_RS_THREADS) k_rs_cluster(const __grid_constant__ CafeSortBatch B) {
    __shared__ __align__(16) CafeSortShared S;
    auto cluster = cooperative_groups::this_cluster();
    const int nblk = (int)cluster.num_blocks(), blk = (int)cluster.block_rank();
    const CafeSortDesc& D = B.d[blockIdx.x / nblk];
    const int bins = 1 << D.bits, d = (int)threadIdx.x * 2;
    const bool tiles = ((((int64_t)D.n + nblk - 1) / nblk + 31) & ~(int64_t)31) <= CAFE_RS_TILE;
    if (tiles) cafe_rs_tiles(D, cluster, nblk, blk, S);
    for (int pass = 0; !tiles && pass < D.passes; ++pass) {
        cafe_rs_hist(D, pass, blk, S);
        cluster.sync();
        int loc[2] = {0, 0}, own[2] = {0, 0};
        if (d < bins) {
            for (int b = 0; b < nblk; ++b) {
                const int2 h = *reinterpret_cast<const int2*>(cluster.map_shared_rank(S.hist, b) + d);
                loc[0] += h.x; loc[1] += h.y;
                if (b < blk) { own[0] += h.x; own[1] += h.y; }
            }
        }
        cafe_rs_set_base(D, loc, own, S);
        cafe_rs_scatter(D, pass, blk, S);
        cluster.sync();   // (also: nobody reads this block's histogram any more)
    }
    if (D.start) cafe_rs_starts(D, blk * CAFE_RS_WARPS + (threadIdx.x >> 5), nblk * CAFE_RS_WARPS);
}
// A launch per step: blockIdx.y = sort, blockIdx.x = block of the sort.
static __global__ void __launch_bounds__(CAFE_RS_THREADS) k_rs_hist(const __grid_constant__ CafeSortBatch B, int pass) {
    __shared__ __align__(16) CafeSortShared S;
    const CafeSortDesc& D = B.d[blockIdx.y];
    if (pass >= D.passes || (int)blockIdx.x >= D.blocks) return;
    cafe_rs_hist(D, pass, blockIdx.x, S);
    int32_t* row = D.scratch + (size_t)(blockIdx.x + 1) * CAFE_RS_MAX_BINS;
    for (int d = threadIdx.x; d < (1 << D.bits); d += CAFE_RS_THREADS) row[d] = S.hist[d];
}
// exclusive prefix over the blocks, in place, and totals: 32 digits per block of the launch, a warp per part of the blocks
static __global__ void __launch_bounds__(CAFE_RS_THREADS) k_rs_scan(const __grid_constant__ CafeSortBatch B, int pass) {
    __shared__ int32_t s_part[CAFE_RS_WARPS][32];
    constexpr int PER = (CAFE_RS_MAX_BLOCKS + CAFE_RS_WARPS - 1) / CAFE_RS_WARPS;
    const CafeSortDesc& D = B.d[blockIdx.y];
    if (pass >= D.passes) return;
    const int d = blockIdx.x * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
    const bool ok = d < (1 << D.bits);
    const int per = (D.blocks + CAFE_RS_WARPS - 1) / CAFE_RS_WARPS;
    int32_t* col = D.scratch + (size_t)(w * per + 1) * CAFE_RS_MAX_BINS + d;
    int v[PER], sum = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) v[q] = (ok && q < per && w * per + q < D.blocks) ? col[(size_t)q * CAFE_RS_MAX_BINS] : 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) sum += v[q];
    s_part[w][threadIdx.x & 31] = sum;
    __syncthreads();
    int run = 0, tot = 0;
#pragma unroll
    for (int q = 0; q < CAFE_RS_WARPS; ++q) { const int t = s_part[q][threadIdx.x & 31]; tot += t; run += q < w ? t : 0; }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        if (ok && q < per && w * per + q < D.blocks) col[(size_t)q * CAFE_RS_MAX_BINS] = run;
        run += v[q];
    }
    if (ok && w == 0) D.scratch[d] = tot;
}
static __global__ void __launch_bounds__(CAFE_RS_THREADS) k_rs_scatter(const __grid_constant__ CafeSortBatch B, int pass) {
    __shared__ __align__(16) CafeSortShared S;
    const CafeSortDesc& D = B.d[blockIdx.y];
    if (pass >= D.passes || (int)blockIdx.x >= D.blocks) return;
    const int32_t* row = D.scratch + (size_t)(blockIdx.x + 1) * CAFE_RS_MAX_BINS;
    const int bins = 1 << D.bits, d = (int)threadIdx.x * 2;
    int loc[2] = {0, 0}, own[2] = {0, 0};
    if (d < bins) { loc[0] = D.scratch[d]; loc[1] = D.scratch[d + 1]; own[0] = row[d]; own[1] = row[d + 1]; }
    cafe_rs_set_base(D, loc, own, S);
    cafe_rs_scatter(D, pass, blockIdx.x, S);
}
static __global__ void __launch_bounds__(CAFE_RS_THREADS) k_rs_starts(const __grid_constant__ CafeSortBatch B) {
    const CafeSortDesc& D = B.d[blockIdx.y];
    if (D.start) cafe_rs_starts(D, blockIdx.x * CAFE_RS_WARPS + (threadIdx.x >> 5), gridDim.x * CAFE_RS_WARPS);
}

static inline int cafe_rs_bits_for(int64_t nb) { int b = 1; while ((1ll << b) < nb) ++b; return b; }

// Sorts every entry of the batch (n > 0 each; passes, bits and blocks are set here), stably.  Returns the first launch
// error, if any.
static inline cudaError_t cafe_radix_sort(CafeSortBatch& B, cudaStream_t st) {
    if (B.count < 1) return cudaSuccess;
    int64_t most = 0, most_nb = 0;
    int passes = 0, blocks = 0;
    bool starts = false;
    for (int s = 0; s < B.count; ++s) {
        CafeSortDesc& D = B.d[s];
        const int total = cafe_rs_bits_for(D.mod.n);
        D.passes = (total + CAFE_RS_MAX_BITS - 1) / CAFE_RS_MAX_BITS;
        D.bits = (total + D.passes - 1) / D.passes;
        most = D.n > most ? D.n : most;
        if (D.start) { starts = true; most_nb = D.mod.n > most_nb ? D.mod.n : most_nb; }
        passes = D.passes > passes ? D.passes : passes;
    }
    if (most <= CAFE_RS_CLUSTER_PAIRS) {
        // enough blocks that each has half a tile of pairs and 16 384 bucket ranges to write at most
        int c = 1;
        while (c < CAFE_RS_CLUSTER_MAX && ((int64_t)c * (CAFE_RS_TILE / 2) < most || (int64_t)c * 16384 < most_nb)) c <<= 1;
        for (int s = 0; s < B.count; ++s) B.d[s].blocks = c;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(B.count * c));
        cfg.blockDim = dim3(CAFE_RS_THREADS);
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)c; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, k_rs_cluster, B);
        const cudaError_t g = cudaGetLastError();
        return e != cudaSuccess ? e : g;
    }
    for (int s = 0; s < B.count; ++s) {
        B.d[s].blocks = cafe_rs_blocks(B.d[s].n);
        blocks = B.d[s].blocks > blocks ? B.d[s].blocks : blocks;
    }
    const dim3 grid((unsigned)blocks, (unsigned)B.count);
    const dim3 scan((unsigned)(CAFE_RS_MAX_BINS / 32), (unsigned)B.count);
    for (int p = 0; p < passes; ++p) {
        k_rs_hist<<<grid, CAFE_RS_THREADS, 0, st>>>(B, p);
        k_rs_scan<<<scan, CAFE_RS_THREADS, 0, st>>>(B, p);
        k_rs_scatter<<<grid, CAFE_RS_THREADS, 0, st>>>(B, p);
    }
    if (starts) k_rs_starts<<<grid, CAFE_RS_THREADS, 0, st>>>(B);
    return cudaGetLastError();
}
