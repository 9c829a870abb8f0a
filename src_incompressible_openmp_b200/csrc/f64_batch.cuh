// Batched replicas of the plain (FP64) form: one launch per phase for many independent channels.
// Blocks [offs[r], offs[r + 1]) of a launch run replica r's blocks 0, 1, ... of the single-context
// kernel (the same per-block body, so each replica's state is bit-identical to the replica stepped
// alone). Each block first copies its replica's arguments into shared memory.
//
// A replica's kernels are far too small to fill the GPU, and 30 of them per replica and step made
// the batch launch-bound: 64 replicas of the ensemble family (13.5 M particles) took 10.2 ms per step
// with a stream per replica and a graph of 1,900 launches; the 36 launches of a step here take 4.8 ms.
#pragma once
#include "bc.cuh"
#include "cells.cuh"
#include "closure.cuh"
#include "fast_batch.cuh"
#include "sort.cuh"
#include "zone.cuh"

namespace mpcd_dev {

struct F64Job {
    DevParams P;
    View64 S;          // the state at the step's start (velocities of the base pass's input)
    View64 M;          // after the base pass (the same positions); the shifted pass runs on it in place
    View64 T;          // the step's result
    RedPatch patch;    // the shifted pass's moves
    int* patchCount;
    const int* corrSlot;
    const double2* corrV;
    const int* pid;
    int* pidOut;
    int* cidStd;
    int* cidSrd;
    BcWork W;
    DevStatus* st;
    long long* dStep;
    uint64_t* stepSeeds;
    uint64_t *seeds, *seedsShifted;
    uint8_t *signs0, *signs1;
    const uint64_t *startStd, *startSrd;
    const int *slotsStd, *slotsSrd;
    FieldsOut ref;
    double *pdRaw, *pdrive, *eosX, *eosY, *duRX, *duRY, *cols, *partial, *red;
    const int* mask;
    int* cellOf;
    const int4* rectsBase;
    int *zoneCost, *zoneHist, *zoneOrder;
    int n, nwords, nzBase, nzShifted, anyMask, tileCap, nbRed;
};

// The collision's tile shape unless the members share another: 32 cells by 128 threads. ms per step of the
// ensemble family by shapes 0 to 6: 64 replicas 4.81 4.80 4.91 4.94 4.85 4.84 4.80, 16 replicas 1.76 1.77
// 1.74 1.72 1.75 1.76 1.76, 4 replicas 0.69 0.71 0.70 0.76 0.72 0.71 0.72.
constexpr int kF64CollideShape = 0;
constexpr int kF64WallBlocks = 8;       // blocks per replica of the thermal-wall and correction kernels

#define MPCD_F64_JOB(J, blk)                                            \
    __shared__ __align__(16) char sj[fb_bytes<F64Job>()];               \
    const int rep_ = fb_replica(offs, n, (int)blockIdx.x);              \
    if (rep_ < 0) return;                                               \
    const F64Job& J = fb_stage(jobs, rep_, sj);                         \
    const int blk = (int)blockIdx.x - offs[rep_]

using F64Jobs = const F64Job* __restrict__;
using F64Offs = const int* __restrict__;

// step begin and SRD shift (block 0), wall bitmaps and counters cleared (the others)
__global__ void __launch_bounds__(256) k_f64_head(F64Jobs jobs, F64Offs offs, int n) {
    MPCD_F64_JOB(J, blk);
    if (blk == 0) {
        srd_shift_block(J.P, 0, J.W.srdShift, J.stepSeeds, J.dStep, J.stepSeeds);
        return;
    }
    const int i = (blk - 1) * (int)blockDim.x + (int)threadIdx.x;
    if (i < J.nwords) {
        J.W.bitsX[i] = 0u;
        J.W.bitsY[i] = 0u;
    }
    if (i < 4) J.W.ints[i] = 0;
    if (i == 0) *J.W.nEvents = 0;
    if (i < 2) J.patchCount[i] = 0;
}

// zone generators of the base, then the shifted pass
__global__ void __launch_bounds__(kSeedZonesPerBlock * 2) k_f64_seeds(F64Jobs jobs, F64Offs offs, int n) {
    MPCD_F64_JOB(J, blk);
    const int nb = (J.nzBase + kSeedZonesPerBlock - 1) / kSeedZonesPerBlock;
    if (blk < nb)
        zone_seeds_block(blk, J.stepSeeds[kSeedBase], J.nzBase, J.seeds);
    else
        zone_seeds_block(blk - nb, J.stepSeeds[kSeedShifted], J.nzShifted, J.seedsShifted);
}

__global__ void __launch_bounds__(256) k_f64_stream(F64Jobs jobs, F64Offs offs, int n) {
    MPCD_F64_JOB(J, blk);
    stream_bc_block<false>(blk, J.P, 1, J.S, J.pid, J.cidStd, J.cidSrd, J.W, J.st);
}

__global__ void __launch_bounds__(256) k_f64_word_counts(F64Jobs jobs, F64Offs offs, int n) {
    MPCD_F64_JOB(J, blk);
    word_counts_block(blk, J.W.bitsX, J.W.bitsY, J.nwords, J.W.wordCount);
}

// one block per replica from here on where offs is missing
__global__ void __launch_bounds__(kScanThreads) k_f64_scan_words(F64Jobs jobs) {
    __shared__ __align__(16) char sj[fb_bytes<F64Job>()];
    const F64Job& J = fb_stage(jobs, (int)blockIdx.x, sj);
    scan_small_block(J.W.wordCount, J.nwords, J.W.wordPrefix);
}

__global__ void __launch_bounds__(kNormThreads) k_f64_normals(F64Jobs jobs) {
    __shared__ __align__(16) char sj[fb_bytes<F64Job>()];
    const F64Job& J = fb_stage(jobs, (int)blockIdx.x, sj);
    wall_normals_block(0, J.W.wordPrefix + J.nwords, J.W.normalCap, J.W.normals, J.st, J.stepSeeds);
}

__global__ void __launch_bounds__(256) k_f64_wall_apply(F64Jobs jobs) {
    __shared__ __align__(16) char sj[fb_bytes<F64Job>()];
    const F64Job& J = fb_stage(jobs, (int)blockIdx.x / kF64WallBlocks, sj);
    const int ne = min(*J.W.nEvents, J.W.eventCap);
    for (int blk = (int)blockIdx.x % kF64WallBlocks; blk * (int)blockDim.x < ne; blk += kF64WallBlocks)
        wall_apply_block(blk, J.P, J.S, J.W, J.st);
}

// the rotation signs of step `step` (seed given), or with step < 0 those of the next step
__global__ void __launch_bounds__(kSignThreads) k_f64_signs(F64Jobs jobs, long long step, uint64_t seed) {
    __shared__ __align__(16) char sj[fb_bytes<F64Job>()];
    const F64Job& J = fb_stage(jobs, (int)blockIdx.x, sj);
    if (step >= 0)
        srd_signs_block(seed, J.P.Nc, (step & 1) ? J.signs1 : J.signs0, nullptr, nullptr);
    else
        srd_signs_block(0, J.P.Nc, J.signs0, J.stepSeeds, J.signs1);
}

// tile shape K (kCollideShape); dynamic shared memory: the arguments, then the tile
template <int K>
__global__ void __launch_bounds__(kCollideShape[K].threads) k_f64_collide(F64Jobs jobs, F64Offs offs, int n) {
    extern __shared__ __align__(16) char smem[];
    const int r = fb_replica(offs, n, (int)blockIdx.x);
    if (r < 0) return;
    const F64Job& J = fb_stage(jobs, r, smem);
    srd_collide_block<View64, kCollideShape[K].cells>((int)blockIdx.x - offs[r], smem + fb_bytes<F64Job>(), J.P, J.startSrd,
                                                      J.slotsSrd, J.signs0, J.P.Nc, J.S, J.st, J.stepSeeds, J.signs1,
                                                      J.tileCap);
}

__global__ void __launch_bounds__(256) k_f64_fields(F64Jobs jobs, F64Offs offs, int n) {
    MPCD_F64_JOB(J, blk);
    cell_fields_block(blk, J.P, J.startStd, J.slotsStd, J.S, J.P.rhoTarget, J.ref);
}
__global__ void __launch_bounds__(256) k_f64_blend(F64Jobs jobs, F64Offs offs, int n) {
    MPCD_F64_JOB(J, blk);
    pdrive_blend_block(blk, J.P, J.pdRaw, J.mask, J.anyMask, J.pdrive, nullptr);
}
__global__ void __launch_bounds__(256) k_f64_eos(F64Jobs jobs, F64Offs offs, int n) {
    MPCD_F64_JOB(J, blk);
    eos_block(blk, J.P, J.pdrive, J.eosX, J.eosY);
}

// the base pass's output velocities start as a copy of its input
__global__ void __launch_bounds__(256) k_f64_copy_vel(F64Jobs jobs, F64Offs offs, int n) {
    MPCD_F64_JOB(J, blk);
    const int i = blk * (int)blockDim.x + (int)threadIdx.x;
    if (i < J.n) J.M.v[i] = J.S.v[i];
}
// the shifted pass's corrected velocities
__global__ void __launch_bounds__(256) k_f64_apply_corr(F64Jobs jobs) {
    __shared__ __align__(16) char sj[fb_bytes<F64Job>()];
    const F64Job& J = fb_stage(jobs, (int)blockIdx.x / kF64WallBlocks, sj);
    apply_corr_block((int)blockIdx.x % kF64WallBlocks, kF64WallBlocks, J.M, J.corrSlot, J.corrV, J.patchCount);
}

__global__ void __launch_bounds__(256) k_f64_zone_cost(F64Jobs jobs, F64Offs offs, int n) {
    MPCD_F64_JOB(J, blk);
    zone_cost_block(blk, J.P, J.rectsBase, J.startStd, J.nzBase, J.zoneCost, J.zoneHist);
}
__global__ void __launch_bounds__(1024) k_f64_zone_order(F64Jobs jobs) {
    __shared__ __align__(16) char sj[fb_bytes<F64Job>()];
    const F64Job& J = fb_stage(jobs, (int)blockIdx.x, sj);
    zone_order_block(J.zoneCost, J.zoneHist, J.nzBase, J.zoneOrder);
}

__global__ void __launch_bounds__(256) k_f64_closure(F64Jobs jobs, F64Offs offs, int n) {
    MPCD_F64_JOB(J, blk);
    closure_cells_block(blk, J.P, J.startStd, J.slotsStd, J.M, J.ref.Px, J.ref.Py, J.ref.Ux, J.ref.Uy, RedFields{}, J.duRX,
                        J.duRY, J.cols, J.cellOf, J.patch);
}
__global__ void __launch_bounds__(kRedThreads) k_f64_reduce_partial(F64Jobs jobs, F64Offs offs, int n) {
    __shared__ double sh[2][kRedThreads];
    MPCD_F64_JOB(J, blk);
    reduce_partial_block(blk, J.cols, (int64_t)J.P.Nc, 2, 0u, kFastBatchRedRows, J.partial, sh);
}
__global__ void __launch_bounds__(kRedThreads) k_f64_reduce_final(F64Jobs jobs) {
    __shared__ double sh[2][kRedThreads];
    __shared__ __align__(16) char sj[fb_bytes<F64Job>()];
    const F64Job& J = fb_stage(jobs, (int)blockIdx.x, sj);
    reduce_final_block(J.partial, J.nbRed, 2, 0u, J.red, sh);
}
__global__ void __launch_bounds__(256) k_f64_kick(F64Jobs jobs, F64Offs offs, int n) {
    MPCD_F64_JOB(J, blk);
    kick_flat_block(blk, J.P, J.n, J.cellOf, J.slotsStd, J.red, J.duRX, J.duRY, J.eosX, J.eosY, J.M, J.pid, J.T, J.pidOut,
                    nullptr, nullptr, nullptr, nullptr);
}

// the members' status codes in one array (one copy to the host instead of one per member)
__global__ void k_gather_status(DevStatus* const* __restrict__ st, int n, int* __restrict__ codes) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n) codes[r] = st[r]->code;
}

}  // namespace mpcd_dev
