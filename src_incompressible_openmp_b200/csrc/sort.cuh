// Cell index: for every cell, the slots of its particles in ascending particle id.
//
// The reference walks particles in id order whenever it accumulates per-cell sums
// (src/common_grid.cpp:62-67, src/srd_collision.cpp:61-66) or builds per-cell lists
// (src/zone_pass.cpp:112-118). Ordering each cell's slots by particle id makes every
// per-cell FP64 sum on the device run in exactly that order, so sums are bit-identical.
//
// Build: warp-aggregated histogram with atomics (one atomic per run of equal cell ids in a
// warp), exclusive scan of the counts, scatter of (particle id, slot) keys into the cells'
// segments, then a rank sort of each cell's keys: an entry's place in its cell is the number of the
// cell's keys below its own.
#pragma once

#include "common.cuh"

namespace mpcd_dev {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

// ------------------------------------------------------------------ exclusive scan (u64)
__global__ void k_scan_reduce(const uint64_t* __restrict__ in, int64_t n, uint64_t* __restrict__ blockSums) {
    __shared__ uint64_t sh[32];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    uint64_t s = 0;
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t i = base + (int64_t)k * kScanThreads + threadIdx.x;
        if (i < n) s += in[i];
    }
    uint64_t tot;
    block_exclusive_scan(s, sh, &tot);
    if (threadIdx.x == 0) blockSums[blockIdx.x] = tot;
}

// single block: exclusive scan of nb block sums in place
__global__ void k_scan_blocks(uint64_t* __restrict__ blockSums, int nb) {
    __shared__ uint64_t sh[32];
    uint64_t carry = 0;
    for (int base = 0; base < nb; base += kScanThreads) {
        const int i = base + threadIdx.x;
        const uint64_t v = (i < nb) ? blockSums[i] : 0ULL;
        uint64_t tot;
        const uint64_t ex = block_exclusive_scan(v, sh, &tot);
        if (i < nb) blockSums[i] = carry + ex;
        carry += tot;
        __syncthreads();
    }
}

// out[i] = exclusive prefix of in; out[n] = total (out has n+1 entries)
__global__ void k_scan_apply(const uint64_t* __restrict__ in, int64_t n, const uint64_t* __restrict__ blockSums,
                             uint64_t* __restrict__ out) {
    __shared__ uint64_t sh[32];
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    uint64_t v[kScanItems];
    uint64_t s = 0;
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = (base + k < n) ? in[base + k] : 0ULL;
        s += v[k];
    }
    uint64_t tot;
    uint64_t ex = block_exclusive_scan(s, sh, &tot) + blockSums[blockIdx.x];
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) out[base + k] = ex;
        ex += v[k];
    }
    if (base + kScanItems >= n && base < n) out[n] = ex;  // the thread holding the last element
}

// Arrays of at most kSmallScan entries are scanned by one block in one launch (a step of a
// small replica launches many short kernels, so their number counts).
constexpr int kSmallScan = 65536;

// One block: out[i] = exclusive prefix of the values ld(i), out[n] = total (n <= kSmallScan). The
// array goes through in tiles of kScanTile, kScanItems consecutive values per thread, the next
// tile's loads (ld4(base, n, v): the four values from base, 0 past n) in flight during a tile's
// scan. Bound by the tiles' chain of shuffles and barriers; a thread per run of n / 1024 values
// (uncoalesced) took 52 us at 32,301 cells.
template <class Ld4>
__device__ __forceinline__ void scan_small_tiles(int n, uint64_t* __restrict__ out, Ld4 ld4) {
    static_assert(kScanItems == 4, "four values per thread and tile");
    __shared__ uint64_t sh[32];
    const int t = (int)threadIdx.x * kScanItems;
    uint64_t v[4], carry = 0;
    ld4(t, n, v);
    for (int b0 = 0; b0 < n; b0 += kScanTile) {
        uint64_t w[4];
        ld4(b0 + kScanTile + t, n, w);
        uint64_t tot;
        const uint64_t e0 = carry + block_exclusive_scan(v[0] + v[1] + v[2] + v[3], sh, &tot);
        const uint64_t e1 = e0 + v[0], e2 = e1 + v[1], e3 = e2 + v[2];
        const int i = b0 + t;
        if (i + 4 <= n) {
            *reinterpret_cast<ulonglong2*>(out + i) = make_ulonglong2(e0, e1);
            *reinterpret_cast<ulonglong2*>(out + i + 2) = make_ulonglong2(e2, e3);
        } else {
            if (i < n) out[i] = e0;
            if (i + 1 < n) out[i + 1] = e1;
            if (i + 2 < n) out[i + 2] = e2;
        }
        carry += tot;
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = w[k];
    }
    if (threadIdx.x == 0) out[n] = carry;
}

// one block: out[i] = exclusive prefix of in, out[n] = total (n <= kSmallScan)
__device__ __forceinline__ void scan_small_block(const uint64_t* __restrict__ in, int n, uint64_t* __restrict__ out) {
    scan_small_tiles(n, out, [&](int i, int m, uint64_t* v) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = i + k < m ? in[i + k] : 0ULL;
    });
}

__global__ void __launch_bounds__(kScanThreads) k_scan_small(const uint64_t* __restrict__ in, int n,
                                                              uint64_t* __restrict__ out) {
    scan_small_block(in, n, out);
}

// ------------------------------------------------------------------ cell index
// A cell's count is scanned packed as (count, count >= 2), so one scan yields both the segment
// starts and the rank of each cell among cells holding at least two particles (the SRD sign
// stream index). Each count is cleared once read, ready for the next build's histogram.
__device__ __forceinline__ uint64_t pack_count(int k) { return (uint64_t)(uint32_t)k | ((uint64_t)(k >= 2) << 32); }

// k_scan_reduce over the packed counts
__global__ void k_count_scan_reduce(const int* __restrict__ count, int64_t n, uint64_t* __restrict__ blockSums) {
    __shared__ uint64_t sh[32];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    uint64_t s = 0;
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t i = base + (int64_t)k * kScanThreads + threadIdx.x;
        if (i < n) s += pack_count(count[i]);
    }
    uint64_t tot;
    block_exclusive_scan(s, sh, &tot);
    if (threadIdx.x == 0) blockSums[blockIdx.x] = tot;
}

// The packed counts of the four cells from i, whose counts are cleared (count: 16-byte aligned, i a
// multiple of 4; 0 past n)
__device__ __forceinline__ void take_counts4(int* __restrict__ count, int64_t i, int64_t n, uint64_t* v) {
    if (i + 4 <= n) {
        int4* p = reinterpret_cast<int4*>(count + i);
        const int4 c = *p;
        *p = make_int4(0, 0, 0, 0);
        v[0] = pack_count(c.x);
        v[1] = pack_count(c.y);
        v[2] = pack_count(c.z);
        v[3] = pack_count(c.w);
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = 0ULL;
        if (i + k < n) {
            v[k] = pack_count(count[i + k]);
            count[i + k] = 0;
        }
    }
}

// k_scan_apply over the packed counts, clearing them (16-byte loads and stores; 93 us with 4- and
// 8-byte ones at 4,194,304 cells)
__global__ void k_count_scan_apply(int* __restrict__ count, int64_t n, const uint64_t* __restrict__ blockSums,
                                   uint64_t* __restrict__ out) {
    __shared__ uint64_t sh[32];
    static_assert(kScanItems == 4, "four cells per thread");
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    uint64_t v[4];
    take_counts4(count, base, n, v);
    uint64_t tot;
    const uint64_t e0 = block_exclusive_scan(v[0] + v[1] + v[2] + v[3], sh, &tot) + blockSums[blockIdx.x];
    const uint64_t e[4] = {e0, e0 + v[0], e0 + v[0] + v[1], e0 + v[0] + v[1] + v[2]};
    if (base + 4 <= n) {
        *reinterpret_cast<ulonglong2*>(out + base) = make_ulonglong2(e[0], e[1]);
        *reinterpret_cast<ulonglong2*>(out + base + 2) = make_ulonglong2(e[2], e[3]);
    } else {
        for (int k = 0; k < 3; ++k)
            if (base + k < n) out[base + k] = e[k];
    }
    if (base + kScanItems >= n && base < n) out[n] = e[3] + v[3];  // the thread holding the last element
}

// one block: the packed counts' exclusive scan into start (Nc <= kSmallScan), clearing the counts
__device__ __forceinline__ void scan_counts_small_block(int* __restrict__ count, int Nc, uint64_t* __restrict__ start) {
    scan_small_tiles(Nc, start, [&](int i, int n, uint64_t* v) { take_counts4(count, i, n, v); });
}

__global__ void __launch_bounds__(kScanThreads) k_scan_counts_small(int* __restrict__ count, int Nc,
                                                                     uint64_t* __restrict__ start) {
    scan_counts_small_block(count, Nc, start);
}

// pos[s] = arrival order of slot s within its cell (any order; fixed by k_cell_rank).
// One atomic per run of equal cell ids among consecutive lanes: after the end-of-step
// re-sort, slots are ordered by cell, so a warp's lanes form a few long runs. Each warp
// covers kIndexItems runs of 32 consecutive slots, whose atomics are in flight together.
constexpr int kIndexItems = 4;

// The slots in the order of an earlier index: `order`, a permutation of them all, when kOrder. Few
// particles change cells between the two builds around a base pass, so consecutive entries form
// runs of whole cells there, where consecutive slots (ordered by the cells before the streaming) hold
// runs of one or two. pos is by entry then. (The step's two standard-cell builds 2.14 -> 2.04 ms at
// 84 M particles, 0.316 -> 0.311 at 10.5 M, the same at 25,000.)
template <bool kOrder>
__device__ __forceinline__ int slot_of_entry(const int* __restrict__ order, int j) {
    return kOrder ? order[j] : j;
}

template <bool kOrder>
__device__ __forceinline__ void histogram_block(int blk, const int* __restrict__ cid, int n, int* __restrict__ count,
                                                int* __restrict__ pos, const int* __restrict__ order) {
    const int lane = threadIdx.x & 31;
    const int base = ((blk * (int)blockDim.x + (int)threadIdx.x) >> 5) * (32 * kIndexItems) + lane;
    int c[kIndexItems], got[kIndexItems], runStart[kIndexItems];
#pragma unroll
    for (int k = 0; k < kIndexItems; ++k) c[k] = (base + 32 * k < n) ? slot_of_entry<kOrder>(order, base + 32 * k) : -1;
#pragma unroll
    for (int k = 0; k < kIndexItems; ++k) c[k] = c[k] >= 0 ? cid[c[k]] : -1;
#pragma unroll
    for (int k = 0; k < kIndexItems; ++k) {
        const int prev = __shfl_up_sync(0xffffffffu, c[k], 1);
        const bool headOfRun = (lane == 0) || (prev != c[k]);
        const unsigned heads = __ballot_sync(0xffffffffu, headOfRun);
        // run start = highest head lane <= lane; run end = next head lane
        runStart[k] = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
        const unsigned after = heads & ~(0xffffffffu >> (31 - lane));
        const int runEnd = after ? (__ffs(after) - 1) : 32;
        got[k] = (headOfRun && c[k] >= 0) ? atomicAdd(&count[c[k]], runEnd - runStart[k]) : 0;
    }
#pragma unroll
    for (int k = 0; k < kIndexItems; ++k) {
        const int b = __shfl_sync(0xffffffffu, got[k], runStart[k]);
        if (base + 32 * k < n) pos[base + 32 * k] = b + (lane - runStart[k]);
    }
}

template <bool kOrder>
__global__ void k_histogram(const int* __restrict__ cid, int n, int* __restrict__ count, int* __restrict__ pos,
                            const int* __restrict__ order) {
    histogram_block<kOrder>((int)blockIdx.x, cid, n, count, pos, order);
}

// keys[start[cid[s]] + pos[s]] = (pid[s] << 32) | s: each cell's segment holds its
// particles' keys in arrival order (same slot coverage and order as k_histogram)
template <bool kOrder>
__device__ __forceinline__ void scatter_keys_block(int blk, const int* __restrict__ cid, const int* __restrict__ pos,
                                                   const int* __restrict__ pid, int n,
                                                   const uint64_t* __restrict__ start, uint64_t* __restrict__ keys,
                                                   const int* __restrict__ order) {
    const int lane = threadIdx.x & 31;
    const int base = ((blk * (int)blockDim.x + (int)threadIdx.x) >> 5) * (32 * kIndexItems) + lane;
    int t[kIndexItems], c[kIndexItems], p[kIndexItems], q[kIndexItems];
#pragma unroll
    for (int k = 0; k < kIndexItems; ++k) t[k] = base + 32 * k < n ? slot_of_entry<kOrder>(order, base + 32 * k) : -1;
#pragma unroll
    for (int k = 0; k < kIndexItems; ++k) {
        c[k] = t[k] >= 0 ? cid[t[k]] : 0;
        p[k] = t[k] >= 0 ? pos[base + 32 * k] : 0;
        q[k] = t[k] >= 0 ? pid[t[k]] : 0;
    }
    uint32_t at[kIndexItems];
#pragma unroll
    for (int k = 0; k < kIndexItems; ++k) at[k] = (uint32_t)start[c[k]];
#pragma unroll
    for (int k = 0; k < kIndexItems; ++k) {
        if (t[k] >= 0) keys[at[k] + p[k]] = ((uint64_t)(uint32_t)q[k] << 32) | (uint32_t)t[k];
    }
}

template <bool kOrder>
__global__ void k_scatter_keys(const int* __restrict__ cid, const int* __restrict__ pos, const int* __restrict__ pid,
                               int n, const uint64_t* __restrict__ start, uint64_t* __restrict__ keys,
                               const int* __restrict__ order) {
    scatter_keys_block<kOrder>((int)blockIdx.x, cid, pos, pid, n, start, keys, order);
}

// Rank sort of the cells' keys. Eight lanes take a cell of up to 32 entries: their keys stay in
// registers, the cell's ids go through shared memory and are read four at a time, and no block barrier
// is needed; K registers per lane by the fullest such cell of the warp. Larger cells take the whole
// warp. Bound by the latency of start, then keys, and by the m^2 comparisons of a cell (about 400 at 20
// entries). At 84 M particles, 20 per cell, a whole index build took 1.24 ms with a block's ~1,280 keys
// and their segment bounds in shared memory, a thread per key and two barriers, and 1.07-1.11 ms so
// (0.17 -> 0.16 ms at 10.5 M, 10 per cell; 0.024 -> 0.019 ms at 2,500 cells). Sixteen cells per warp:
// 1.13-1.21 ms.
constexpr int kRankThreads = 128;
constexpr int kRankWarpCells = 8;  // consecutive cells of a warp, four at a time
constexpr int kRankCells = kRankThreads / 32 * kRankWarpCells;  // cells per block
constexpr int kRankGroupMax = 32;                               // entries of a cell ranked by eight lanes
constexpr int kRankRow = kRankGroupMax + 4;  // ids of a group (four banks on from the last group's)

__device__ __forceinline__ int seg_lo(uint64_t s) { return (int)(uint32_t)s; }

__device__ __forceinline__ int below4(uint4 q, uint32_t id) {
    return (int)(q.x < id) + (int)(q.y < id) + (int)(q.z < id) + (int)(q.w < id);
}

// Cells [c0, c0 + kRankWarpCells) of a warp by groups of eight lanes, a cell each: a lane holds K of the cell's
// keys (8K >= its entries m), and the group's ids lie padded with the largest id in row `sh`.
// st: lane l <= kRankWarpCells holds the start of cell c0 + l. Cells above 8K entries are left out.
template <int K>
__device__ __forceinline__ void rank_groups(int st, const uint64_t* __restrict__ keys, int* __restrict__ slots,
                                            uint32_t* sh) {
    constexpr int kRounds = kRankWarpCells / 4;
    const int lane = threadIdx.x & 31, k = lane & 7, g = lane >> 3;
    int a[kRounds], m[kRounds];
    uint64_t key[kRounds][K];
#pragma unroll
    for (int q = 0; q < kRounds; ++q) {
        a[q] = __shfl_sync(0xffffffffu, st, 4 * q + g);
        m[q] = __shfl_sync(0xffffffffu, st, 4 * q + g + 1) - a[q];
        if (m[q] > 8 * K) m[q] = 0;
#pragma unroll
        for (int u = 0; u < K; ++u) key[q][u] = k + 8 * u < m[q] ? keys[a[q] + k + 8 * u] : ~0ULL;
    }
#pragma unroll
    for (int q = 0; q < kRounds; ++q) {
        uint32_t id[K];
        int r[K];
#pragma unroll
        for (int u = 0; u < K; ++u) {
            id[u] = (uint32_t)(key[q][u] >> 32);
            r[u] = 0;
            sh[g * kRankRow + k + 8 * u] = id[u];
        }
        __syncwarp();
        const int e = __reduce_max_sync(0xffffffffu, m[q]);
#pragma unroll
        for (int j = 0; j < 8 * K; j += 4) {
            if (j >= e) break;
            const uint4 w = *reinterpret_cast<const uint4*>(sh + g * kRankRow + j);
#pragma unroll
            for (int u = 0; u < K; ++u) r[u] += below4(w, id[u]);
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (k + 8 * u < m[q]) slots[a[q] + r[u]] = (int)(uint32_t)key[q][u];
    }
}

// A cell of m entries from a by a whole warp: 128 keys in registers against 128 ids in sh at a time.
__device__ __noinline__ static void rank_cell_warp(int a, int m, const uint64_t* __restrict__ keys, int* __restrict__ slots,
                                                   uint32_t* sh) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int i0 = 0; i0 < m; i0 += 128) {
        uint64_t key[4];
        int r[4] = {0, 0, 0, 0};
#pragma unroll
        for (int u = 0; u < 4; ++u) key[u] = i0 + lane + 32 * u < m ? keys[a + i0 + lane + 32 * u] : ~0ULL;
#pragma unroll 1
        for (int j0 = 0; j0 < m; j0 += 128) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                sh[lane + 32 * u] = j0 + lane + 32 * u < m ? (uint32_t)(keys[a + j0 + lane + 32 * u] >> 32) : 0xffffffffu;
            __syncwarp();
            const int e = min(128, m - j0);
            for (int j = 0; j < e; j += 4) {
                const uint4 w = *reinterpret_cast<const uint4*>(sh + j);
#pragma unroll
                for (int u = 0; u < 4; ++u) r[u] += below4(w, (uint32_t)(key[u] >> 32));
            }
            __syncwarp();
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i0 + lane + 32 * u < m) slots[a + r[u]] = (int)(uint32_t)key[u];
    }
}

// slots[start[c] + rank] = slot of the key of that rank among cell c's keys (ascending particle id;
// ids are unique, so they alone rank a cell's keys, and none is the padding's 0xffffffff).
__device__ __forceinline__ void cell_rank_block(int blk, const uint64_t* __restrict__ start, int Nc,
                                                const uint64_t* __restrict__ keys, int* __restrict__ slots) {
    static_assert(4 * kRankRow >= 128 && kRankWarpCells < 32, "a warp's row of 128 ids; its starts in one load");
    __shared__ __align__(16) uint32_t ids[kRankThreads / 32][4 * kRankRow];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    uint32_t* sh = ids[wib];
    const int64_t c0 = (int64_t)blk * kRankCells + wib * kRankWarpCells;
    if (c0 >= Nc) return;  // the whole warp; no block barrier follows
    const int st = seg_lo(start[min(c0 + min(lane, kRankWarpCells), (int64_t)Nc)]);
    const int m = __shfl_down_sync(0xffffffffu, st, 1) - st;  // 0 past the warp's cells
    const int most = __reduce_max_sync(0xffffffffu, lane < kRankWarpCells && m <= kRankGroupMax ? m : 0);
    if (most <= 16)
        rank_groups<2>(st, keys, slots, sh);
    else if (most <= 24)
        rank_groups<3>(st, keys, slots, sh);
    else
        rank_groups<4>(st, keys, slots, sh);
    for (unsigned big = __ballot_sync(0xffffffffu, lane < kRankWarpCells && m > kRankGroupMax); big; big &= big - 1) {
        const int l = __ffs(big) - 1;
        rank_cell_warp(__shfl_sync(0xffffffffu, st, l), __shfl_sync(0xffffffffu, m, l), keys, slots, sh);
    }
}

__global__ void __launch_bounds__(kRankThreads) k_cell_rank(const uint64_t* __restrict__ start, int Nc,
                                                            const uint64_t* __restrict__ keys, int* __restrict__ slots) {
    cell_rank_block((int)blockIdx.x, start, Nc, keys, slots);
}

// ------------------------------------------------------------------ batched index builds
// The index builds of many contexts (the replicas of a batch) as one launch per kernel: job r
// is one context's build; blocks [offs[r], offs[r + 1]) of a launch are its blocks.
struct IndexJob {
    const int* cid;
    int* count;
    int* pos;
    uint64_t* start;
    int* slots;
    const int* pid;
    uint64_t* keys;
    int n, Nc;
    const int* order;  // nullable (slot_of_entry)
};

// the job r with offs[r] <= b < offs[r + 1] (offs ascending, offs[0] = 0)
__device__ __forceinline__ int job_of(const int* __restrict__ offs, int nJobs, int b) {
    int lo = 0, hi = nJobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (offs[mid] <= b)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// offs: blocks of kThreads threads covering each job's slots (kIndexItems per thread)
__global__ void k_histogram_batch(const IndexJob* __restrict__ jobs, const int* __restrict__ offs, int nJobs) {
    const int b = (int)blockIdx.x;
    if (nJobs <= 0 || b >= offs[nJobs]) return;
    const int r = job_of(offs, nJobs, b);
    const IndexJob J = jobs[r];
    if (J.order)
        histogram_block<true>(b - offs[r], J.cid, J.n, J.count, J.pos, J.order);
    else
        histogram_block<false>(b - offs[r], J.cid, J.n, J.count, J.pos, nullptr);
}

// one block per job (every job has Nc <= kSmallScan)
__global__ void __launch_bounds__(kScanThreads) k_scan_counts_small_batch(const IndexJob* __restrict__ jobs) {
    const IndexJob J = jobs[blockIdx.x];
    scan_counts_small_block(J.count, J.Nc, J.start);
}

__global__ void k_scatter_keys_batch(const IndexJob* __restrict__ jobs, const int* __restrict__ offs, int nJobs) {
    const int b = (int)blockIdx.x;
    if (nJobs <= 0 || b >= offs[nJobs]) return;
    const int r = job_of(offs, nJobs, b);
    const IndexJob J = jobs[r];
    if (J.order)
        scatter_keys_block<true>(b - offs[r], J.cid, J.pos, J.pid, J.n, J.start, J.keys, J.order);
    else
        scatter_keys_block<false>(b - offs[r], J.cid, J.pos, J.pid, J.n, J.start, J.keys, nullptr);
}

// offs: blocks of each job's rank sort (kRankCells cells per block)
__global__ void __launch_bounds__(kRankThreads) k_cell_rank_batch(const IndexJob* __restrict__ jobs,
                                                                  const int* __restrict__ offs, int nJobs) {
    const int b = (int)blockIdx.x;
    if (nJobs <= 0 || b >= offs[nJobs]) return;
    const int r = job_of(offs, nJobs, b);
    const IndexJob J = jobs[r];
    cell_rank_block(b - offs[r], J.start, J.Nc, J.keys, J.slots);
}

}  // namespace mpcd_dev
