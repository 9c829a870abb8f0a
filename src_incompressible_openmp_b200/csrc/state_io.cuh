// The state in particle-id order from a cell-ordered layout, in two passes.
//
// Neighbours in a cell have unrelated ids, so writing each particle straight to its id's place
// scatters 16-byte pieces over the whole output. Once that is larger than the L2 cache (126 MB)
// every piece costs its own DRAM transaction. Here the particles first go to buckets of
// consecutive ids (a bucket's output window is 32 MB; a block sorts its particles by bucket in
// shared memory, so the buckets fill in runs), then each bucket is written to its window, which
// the L2 cache holds until its lines are whole. The ids are a permutation, so bucket b's
// particles take exactly the places [b << shift, (b + 1) << shift) of the intermediate arrays.
//
// Bound by DRAM bandwidth once the writes are whole lines: 11.7 GB at 84 M particles. Measured
// there, FP64 mpcd_get_state_device: 8.2 ms by the scatter and two copies, 4.2 ms this way; at
// 10.5 M particles 0.95 and 0.57 ms. Fast form: 12.6 (with an allocation per call) and 5.2 ms.
#pragma once

#include "common.cuh"
#include "fast.cuh"

namespace mpcd_dev {

constexpr int kPartThreads = 256;
constexpr int kPartItems = 4;
constexpr int kPartTile = kPartThreads * kPartItems;  // particles sorted together
constexpr int kPartBuckets = 256;                     // bucket limit
constexpr int kPartWindow = 20;                       // log2 of a bucket's ids (32 MB of x and v)

// log2 of the ids per bucket for n particles (at most kPartBuckets buckets)
inline int part_shift(int64_t n) {
    int s = kPartWindow;
    while (((n - 1) >> s) >= kPartBuckets) ++s;
    return s;
}

// The intermediate arrays (n entries each) and the buckets' fill counts (zeroed before).
struct PartBuf {
    double2* x;
    double2* v;
    int* pid;
    int* fill;
};

// Up to kPartTile particles (m of them; load(i, pid, x, v) reads the i-th) into their buckets.
template <class Load>
__device__ __forceinline__ void part_tile(int m, int n, int shift, const PartBuf& B, Load load) {
    __shared__ double2 sx[kPartTile], sv[kPartTile];
    __shared__ int sp[kPartTile];
    __shared__ int cnt[kPartBuckets], off[kPartBuckets], base[kPartBuckets];
    __shared__ uint64_t scan[32];
    const int t = threadIdx.x;
    static_assert(kPartThreads == kPartBuckets, "one thread per bucket");
    cnt[t] = 0;
    __syncthreads();
    double2 x[kPartItems], v[kPartItems];
    int p[kPartItems], r[kPartItems];
#pragma unroll
    for (int k = 0; k < kPartItems; ++k) {
        const int i = t + k * kPartThreads;
        p[k] = -1;
        if (i < m) load(i, p[k], x[k], v[k]);
    }
#pragma unroll
    for (int k = 0; k < kPartItems; ++k)
        if ((unsigned)p[k] < (unsigned)n) r[k] = atomicAdd(cnt + (p[k] >> shift), 1);
    __syncthreads();
    uint64_t tot;
    off[t] = (int)block_exclusive_scan((uint64_t)cnt[t], scan, &tot);
    base[t] = cnt[t] ? (t << shift) + atomicAdd(B.fill + t, cnt[t]) : 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPartItems; ++k)
        if ((unsigned)p[k] < (unsigned)n) {
            const int d = off[p[k] >> shift] + r[k];
            sx[d] = x[k];
            sv[d] = v[k];
            sp[d] = p[k];
        }
    __syncthreads();
    for (int i = t; i < (int)tot; i += kPartThreads) {
        const int b = sp[i] >> shift;
        const int64_t d = (int64_t)base[b] + (i - off[b]);
        if (d >= n || (d >> shift) != b) continue;  // more particles than ids: never on a valid state
        B.x[d] = sx[i];
        B.v[d] = sv[i];
        B.pid[d] = sp[i];
    }
    __syncthreads();
}

// FP64 slots into the buckets
__global__ void __launch_bounds__(kPartThreads) k_part_slots(const double2* __restrict__ x, const double2* __restrict__ v,
                                                             const int* __restrict__ pid, int n, int shift, PartBuf B) {
    const int i0 = blockIdx.x * kPartTile;
    part_tile(min(kPartTile, n - i0), n, shift, B, [&](int i, int& p, double2& X, double2& V) {
        p = pid[i0 + i];
        X = x[i0 + i];
        V = v[i0 + i];
    });
}

// The fast form's bins into the buckets: a block takes cellsPer (at most kPartThreads) cells; the
// pending kick (nullable) is added on the way.
__global__ void __launch_bounds__(kPartThreads) k_part_bins(DevParams P, FastParams F, FastBins b,
                                                            const int2* __restrict__ kick, int cellsPer, int shift,
                                                            PartBuf B) {
    __shared__ int start[kPartThreads + 1];
    __shared__ uint64_t scan[32];
    const int t = threadIdx.x;
    const int c0 = blockIdx.x * cellsPer;
    const int nc = min(cellsPer, P.Nc - c0);
    uint64_t total;
    const int cn = t < nc ? max(0, min(b.cnt[c0 + t], F.K)) : 0;
    start[t] = (int)block_exclusive_scan((uint64_t)cn, scan, &total);
    if (t == 0) start[kPartThreads] = (int)total;
    __syncthreads();
    for (int i0 = 0; i0 < (int)total; i0 += kPartTile)
        part_tile(min(kPartTile, (int)total - i0), P.n, shift, B, [&](int i, int& p, double2& X, double2& V) {
            const int f = i0 + i;
            int g = 0;  // the last cell whose start is at most f
#pragma unroll
            for (int s = kPartThreads / 2; s >= 1; s >>= 1)
                if (start[g + s] <= f) g += s;
            const int c = c0 + g, ix = c / P.Ny, iy = c - ix * P.Ny;
            const size_t s = (size_t)c * F.K + (f - start[g]);
            p = b.pid[s];
            X = fast_position(P, ix, iy, b.off[s]);
            const float2 w = fast_kicked(b.vel[s], kick ? kick[c] : make_int2(0, 0));
            V = make_double2((double)w.x, (double)w.y);
        });
}

// the buckets into particle-id order (x, v nullable)
__global__ void __launch_bounds__(256) k_part_place(PartBuf B, int n, int shift, double2* __restrict__ x,
                                                    double2* __restrict__ v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = i >> shift;
    if (i - (b << shift) >= B.fill[b]) return;
    const int p = B.pid[i];
    if (x) x[p] = B.x[i];
    if (v) v[p] = B.v[i];
}

}  // namespace mpcd_dev
