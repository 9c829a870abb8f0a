// One zone pass of the incompressible redistribution: one warp per zone.
//
// Reference: run_zone_pass_openmp -> run_zone_pass_snapshot_impl
// (src/zone_pass_openmp.cpp:34-172) running run_zone_kernel (src/zone_pass.cpp:669-973)
// on a private copy of the pass input for every zone, then merging zone by zone.
//
// What a zone kernel reads and writes (this is what makes one warp per zone exact):
//   - it moves particles only between cells of its own rectangle (targets and donors are
//     filtered to the zone: src/zone_pass.cpp:611,625,274,819);
//   - outside its rectangle it reads only cell counts of the pass input, up to two cells
//     away (3x3 smoothing of src/zone_pass.cpp:296-319 around the 4-neighbour gradient of
//     :375-411), which never change during the pass;
//   - the particle lists it needs are those of its own cells, in ascending particle id
//     (src/zone_pass.cpp:112-118), and their velocities from the pass input.
// The merge writes each particle from the LAST zone whose rectangle holds the particle's
// input cell (zone ids grow in merge order), i.e. from ownerMap[input cell]. Shifted layouts
// overlap (tiles start at 0 and at tile/2, src/zone_pass.cpp:160-221), so every zone
// processes its full rectangle and writes only the particles it owns. The pass is out of
// place: the output buffers start as a copy of the input, and a zone writes only what it
// changes (positions of moved particles, velocities of corrected cells).
//
// Lists: a cell's list starts as its input segment of the cell index (ascending id) and
// stays implicit -- a head offset into that segment -- until the cell receives particles or
// is shuffled; then it is materialised in a small arena. List entries encode
// (input cell << 20 | position in its input segment), so a particle's slot is read from the
// cell index when needed.
//
// Warp discipline: every lane runs the same control flow with identical scalar values (the
// RNG stream is warp-uniform); lane-parallel sections are candidate evaluation, position
// sampling, list copies and the final momentum correction. Shared-memory scalars written by
// lane 0 are followed by __syncwarp() before any lane reads them.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace mpcd_dev {

// cell flags
constexpr uint8_t kCRecv = 1, kCBulkBulk = 2, kCSkip = 4, kCBulkBefore = 8, kCChanged = 16, kCOwned = 32,
                  kCMat = 64;
constexpr int kEntryShift = 20;  // entry = cell << 20 | position (cells < 4096, positions < 2^20)

struct ZoneArgs {
    DevParams P;
    const int4* rects;        // (xs, xe, ys, ye) per zone, zone id = index + 1
    const int* owner;         // ownerMap of the layout
    const uint64_t* start;    // cell index of the pass input (packed starts)
    const int* slots;
    const double2* vin;
    double2* xout;            // pre-filled with the input positions
    double2* vout;            // pre-filled with the input velocities
    int* cid;                 // standard-grid cell per slot; moved owned particles updated
    const uint64_t* seeds;    // seeded MT19937-64 state per zone (312 words each)
    int nZones;
    int maxCells, winCap, arenaCap, nsmCap;  // capacities of the per-zone working set
    int* overflow;            // zones left to the overflow kernel
    int* nOverflow;
    int2* zoneMoved;          // (dense, sparse) per zone
    double2* zoneCorr;        // (stats[4], stats[5]) per zone
    const int* order;         // launch order of the zones (heaviest first); nullptr = by id
    DevStatus* st;
    // run_zone_pass (serial, in place): zones one after another on the live state. slots[]
    // then holds the pass-input lists followed by an area where each zone appends the new
    // lists (ascending particle id) of the cells it changed; liveStart/liveCnt point to the
    // current list of every cell.
    int serial;
    int* slotsW;              // slots[], writable (the live-list area)
    int* liveCnt;
    int* liveStart;
    int* liveTop;             // next free entry of the live-list area
    int liveEnd;
    const int* pid;           // particle id per slot
    double2* duScratch;       // momentum correction per cell of the running zone
    // single-zone in-place API (serial kernel only; nullptr otherwise): per zone, the kernel-side
    // diagnostics of run_zone_kernel (src/zone_pass.cpp:857-972): sum of uxNow^2, sum of uyNow^2
    // over the zone's non-empty cells, sum and count of the non-zero dPx^2, the same for dPy,
    // the dense cells handled over the passes (nHigh) and the sparse ones (nLow)
    double* zoneDiag;
    // FP32 precision form (f32 != 0): the pass input and output states are these views and
    // vin, xout, vout are unused
    int f32;
    View32 in32, out32;
    // in-place pass (the step's shifted pass; corrSlot nullptr otherwise): corrected velocities go to
    // a list (slot, velocity), written to the input's velocities after the pass (k_apply_corr); at
    // most one entry per particle, since a particle has one owner zone and one final cell
    int* corrSlot;
    double2* corrV;
    int* corrCount;
    // the particles that changed cells in it (moverSlot nullptr: not wanted), as a list per new cell
    // (arrHead, moverNext; -1 ends it) and a flag per old cell: the closure then reads the index of
    // the pass's input with these patches
    int *moverSlot, *moverNext, *moverCount, *arrHead;
    uint8_t* depart;
};

// pass input / output velocities of slot s (kF32: the FP32 views, instantiated separately)
template <bool kF32>
__device__ __forceinline__ double2 zone_vin(const ZoneArgs& A, int s) { return kF32 ? A.in32.vel(s) : A.vin[s]; }
template <bool kF32>
__device__ __forceinline__ void zone_vout(const ZoneArgs& A, int s, double2 w) {
    if (kF32)
        A.out32.set_vel(s, w);
    else
        A.vout[s] = w;
}

// Working set of one zone; carved from shared memory (fast path, I = uint16_t: 16-bit
// per-cell counts and arena offsets) or global memory (overflow path, I = int).
template <typename I>
struct ZoneMem {
    using W = typename std::conditional<sizeof(I) == 2, int16_t, int>::type;
    uint64_t* mt;      // 312: MT19937-64 state
    uint64_t* carry;   // 64: untwisted words of the previous block still to be drawn
    double* nsm;       // (TX+2)(TY+2): smoothed occupancy; reused for dU2 at the end
    W* win;            // (TX+4)(TY+4): pass-input counts around the zone (-1 = outside)
    int* gstart;       // cell: start of its input segment in the cell index
    I* cnt0;           // cell: input count
    I* head;           // cell: list head (implicit: offset into the input segment)
    I* len;            // cell: list length = live count
    I* abase;          // cell: arena start of a materialised list
    I* cap;            // cell: arena capacity of a materialised list
    uint8_t* cflags;   // cell
    uint16_t* list;    // cell: dense / low cell order
    uint16_t* order;   // cell: arena order of materialised lists (compaction)
    uint32_t* arena;   // arenaCap
    int* small;        // 64 ints: ranked targets, donors
    double* smallD;    // 16 doubles: the donors' deviates, polar components and radii

    __host__ __device__ static size_t bytes(int maxCells, int winCap, int arenaCap, int nsmCap) {
        size_t b = 0;
        auto add = [&](size_t n, size_t a) { b = (b + a - 1) / a * a + n; };
        add((size_t)kMtN * 8, 8);
        add(64 * 8, 8);
        add((size_t)nsmCap * 8, 8);
        add((size_t)winCap * sizeof(W), sizeof(W));
        add((size_t)maxCells * 4, 4);
        for (int k = 0; k < 5; ++k) add((size_t)maxCells * sizeof(I), sizeof(I));
        add((size_t)maxCells, 1);
        add((size_t)maxCells * 2, 2);
        add((size_t)maxCells * 2, 2);
        add((size_t)arenaCap * 4, 4);
        add(64 * 4, 4);
        add(16 * 8, 8);
        return (b + 15) / 16 * 16;
    }
    __device__ void carve(char* base, int maxCells, int winCap, int arenaCap, int nsmCap) {
        size_t b = 0;
        auto take = [&](size_t n, size_t a) {
            b = (b + a - 1) / a * a;
            char* p = base + b;
            b += n;
            return p;
        };
        mt = (uint64_t*)take((size_t)kMtN * 8, 8);
        carry = (uint64_t*)take(64 * 8, 8);
        nsm = (double*)take((size_t)nsmCap * 8, 8);
        win = (W*)take((size_t)winCap * sizeof(W), sizeof(W));
        gstart = (int*)take((size_t)maxCells * 4, 4);
        cnt0 = (I*)take((size_t)maxCells * sizeof(I), sizeof(I));
        head = (I*)take((size_t)maxCells * sizeof(I), sizeof(I));
        len = (I*)take((size_t)maxCells * sizeof(I), sizeof(I));
        abase = (I*)take((size_t)maxCells * sizeof(I), sizeof(I));
        cap = (I*)take((size_t)maxCells * sizeof(I), sizeof(I));
        cflags = (uint8_t*)take((size_t)maxCells, 1);
        list = (uint16_t*)take((size_t)maxCells * 2, 2);
        order = (uint16_t*)take((size_t)maxCells * 2, 2);
        arena = (uint32_t*)take((size_t)arenaCap * 4, 4);
        small = (int*)take(64 * 4, 4);
        smallD = (double*)take(16 * 8, 8);
    }
};

// The overflow kernels of many contexts (a batch's replicas) as one launch: job r takes
// blocks [r * perJob, (r + 1) * perJob).
struct OverflowJob {
    ZoneArgs A;  // with the overflow path's capacities
    char* gmem;
    size_t perBlock;
    int* blocksDone;
    double* metricsOut;
};

constexpr int kZoneArgsSmem = (int)((sizeof(ZoneArgs) + 15) / 16 * 16);
constexpr int kF64ZoneWarps = 8;  // zones per block of the batched phase-synchronous kernel

// The zone kernels (zone_body.cuh) are compiled in their own translation unit, zone.cu.
template <bool kF32>
__global__ void k_zone_pass(ZoneArgs A);
template <bool kF32, int kW>
__global__ void k_zone_pass_sync(ZoneArgs A, int perWarp);
template <bool kF32>
__global__ void k_zone_pass_batch(const ZoneArgs* __restrict__ args, const int* __restrict__ offs, int nRep);
__global__ void k_f64_zone_sync(const ZoneArgs* __restrict__ args, const int* __restrict__ offs, int n, int perWarp);
template <bool kF32>
__global__ void k_zone_overflow(ZoneArgs A, char* gmem, size_t perBlock, int* blocksDone, double* metricsOut);
__global__ void k_zone_overflow_batch(const OverflowJob* __restrict__ jobs, int perJob);
__global__ void k_zone_serial(ZoneArgs A, ZoneArgs B, char* gmem);

// Launch order of the zones, heaviest first, so that the last wave of blocks holds the
// cheapest zones. The cost estimate is the number of particles above the bulk high threshold
// in the zone's cells (the dense-phase work); ties keep no particular order, which is fine:
// a zone's result does not depend on when it runs.
constexpr int kCostBuckets = 256;
__device__ __forceinline__ void zone_cost_block(int blk, const DevParams& P, const int4* __restrict__ rects,
                                                const uint64_t* __restrict__ start, int nZones, int* __restrict__ cost,
                                                int* __restrict__ hist) {
    const int z = blk * blockDim.x + threadIdx.x;
    if (z >= nZones) return;
    const int4 R = rects[z];
    double ex = 0.0;
    for (int ix = R.x; ix < R.y; ++ix)
        for (int iy = R.z; iy < R.w; ++iy) {
            const int c = iy + P.Ny * ix;
            const double n = (double)(int)((uint32_t)start[c + 1] - (uint32_t)start[c]);
            if (n > P.highThr) ex += n - P.highThr;
        }
    const int b = min(kCostBuckets - 1, (int)ex);
    cost[z] = b;
    atomicAdd(hist + b, 1);
}
static __global__ void k_zone_cost(DevParams P, const int4* __restrict__ rects, const uint64_t* __restrict__ start, int nZones,
                            int* __restrict__ cost, int* __restrict__ hist) {
    zone_cost_block((int)blockIdx.x, P, rects, start, nZones, cost, hist);
}

// one block: bucket offsets in descending cost, then each zone takes a place in its bucket
__device__ __forceinline__ void zone_order_block(const int* __restrict__ cost, int* __restrict__ hist, int nZones,
                                                 int* __restrict__ order) {
    __shared__ int off[kCostBuckets];
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int b = kCostBuckets - 1; b >= 0; --b) {
            off[b] = acc;
            acc += hist[b];
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < kCostBuckets; b += blockDim.x) hist[b] = 0;  // ready for the next pass
    for (int z = threadIdx.x; z < nZones; z += blockDim.x) order[atomicAdd(&off[cost[z]], 1)] = z;
}
static __global__ void __launch_bounds__(1024) k_zone_order(const int* __restrict__ cost, int* __restrict__ hist, int nZones,
                                                     int* __restrict__ order) {
    zone_order_block(cost, hist, nZones, order);
}

// Seeded MT19937-64 state of every zone: seed = seedBase + 104729 (iz + 1)
// (src/zone_pass_openmp.cpp:78). One thread per zone runs the sequential seeding
// recurrence; states are staged in shared memory and written zone-major, coalesced.
constexpr int kSeedZonesPerBlock = 16;
__device__ __forceinline__ void zone_seeds_block(int blk, uint64_t seedBase, int nZones, uint64_t* out) {
    __shared__ uint64_t st[kSeedZonesPerBlock][kMtN];
    const int t = threadIdx.x;
    const int z0 = blk * kSeedZonesPerBlock;
    if (t < kSeedZonesPerBlock && z0 + t < nZones) {
        uint64_t w = seedBase + 104729ULL * (uint64_t)(z0 + t + 1);
        st[t][0] = w;
        for (int i = 1; i < kMtN; ++i) {
            w = mt_seed_next(w, i);
            st[t][i] = w;
        }
    }
    __syncthreads();
    const int nz = min(kSeedZonesPerBlock, nZones - z0);
    for (int i = t; i < nz * kMtN; i += blockDim.x) out[(size_t)z0 * kMtN + i] = st[i / kMtN][i % kMtN];
}
static __global__ void __launch_bounds__(kSeedZonesPerBlock * 2) k_zone_seeds(uint64_t seedBase, int nZones, uint64_t* out,
                                                                       const uint64_t* seedDev, int which) {
    zone_seeds_block((int)blockIdx.x, seedDev ? seedDev[which] : seedBase, nZones, out);
}

// pass metrics: integer sums and a fixed-order reduction of the per-zone correction stats
// (also clears the overflow-zone counter for the next pass, which starts after this kernel)
static __global__ void k_zone_metrics(const int2* __restrict__ moved, const double2* __restrict__ corr, int nZones,
                               double* __restrict__ out /* movedDense, movedSparse, corrRms, corrMax */,
                               int* __restrict__ nOverflow) {
    if (threadIdx.x == 0 && nOverflow) *nOverflow = 0;
    __shared__ double sa[256], sm[256];
    __shared__ long long sd[256], ss[256];
    __shared__ int sc[256];
    const int t = threadIdx.x;
    double acc = 0.0, mx = 0.0;
    long long d = 0, s = 0;
    int c = 0;
    for (int z = t; z < nZones; z += blockDim.x) {
        const double2 q = corr[z];
        if (q.x > 0.0) {
            acc = __dadd_rn(acc, __dmul_rn(q.x, q.x));
            ++c;
        }
        mx = smax(mx, q.y);
        d += moved[z].x;
        s += moved[z].y;
    }
    sa[t] = acc; sm[t] = mx; sd[t] = d; ss[t] = s; sc[t] = c;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (t < o) {
            sa[t] = __dadd_rn(sa[t], sa[t + o]);
            sm[t] = smax(sm[t], sm[t + o]);
            sd[t] += sd[t + o];
            ss[t] += ss[t + o];
            sc[t] += sc[t + o];
        }
        __syncthreads();
    }
    if (t == 0) {
        out[0] = (double)sd[0];
        out[1] = (double)ss[0];
        out[2] = (sc[0] > 0) ? sqrt(__ddiv_rn(sa[0], (double)sc[0])) : 0.0;
        out[3] = sm[0];
    }
}

}  // namespace mpcd_dev
