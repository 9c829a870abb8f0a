// The zone pass's device code: the warp-per-zone body and its kernels (zone.cu).
#pragma once

#include "zone.cuh"

namespace mpcd_dev {

// In-place twist of a 312-word MT19937-64 state by one warp (reads of each half are staged
// in registers before its writes).
__device__ __noinline__ void mt_twist_inplace_warp(uint64_t* A, int lane) {
    uint64_t nv[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int i = lane + k * kWarp;
        nv[k] = (i < kMtN - kMtM) ? (A[i + kMtM] ^ mt_mix(A[i], A[i + 1])) : 0ULL;
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int i = lane + k * kWarp;
        if (i < kMtN - kMtM) A[i] = nv[k];
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int i = kMtN - kMtM + lane + k * kWarp;
        nv[k] = 0ULL;
        if (i < kMtN - 1) nv[k] = A[i - (kMtN - kMtM)] ^ mt_mix(A[i], A[i + 1]);
        else if (i == kMtN - 1) nv[k] = A[kMtM - 1] ^ mt_mix(A[kMtN - 1], A[0]);
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int i = kMtN - kMtM + lane + k * kWarp;
        if (i < kMtN) A[i] = nv[k];
    }
    __syncwarp();
}

// copy a seeded 312-word state from global memory (one warp, 10 loads per lane in flight)
__device__ __noinline__ void mt_load_warp(uint64_t* buf, const uint64_t* seeded, int lane) {
    uint64_t w[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) {
        const int i = lane + k * kWarp;
        w[k] = (i < kMtN) ? seeded[i] : 0ULL;
    }
#pragma unroll
    for (int k = 0; k < 10; ++k) {
        const int i = lane + k * kWarp;
        if (i < kMtN) buf[i] = w[k];
    }
    __syncwarp();
}

// 64-bit division and remainder on rare paths, out of line to keep the zone kernel small
__device__ __noinline__ uint64_t umod64_slow(uint64_t a, uint64_t b) { return a % b; }
__device__ __noinline__ uint64_t udiv64_slow(uint64_t a, uint64_t b) { return a / b; }

// Next block of a zone's stream (out of line, once per 312 draws): loads the seeded state
// on first use, keeps the kMtN - pos words not yet drawn in `carry`, twists in place.
// Returns the number of carried words.
__device__ __noinline__ int mt_refill(uint64_t* buf, uint64_t* carry, const uint64_t* seeded, int pos, int lane) {
    if (seeded) mt_load_warp(buf, seeded, lane);
    const int left = kMtN - pos;  // 0..63 words still to draw from the old block
    for (int i = lane; i < left; i += kWarp) carry[i] = buf[pos + i];
    __syncwarp();
    mt_twist_inplace_warp(buf, lane);
    return left;
}

// Warp-uniform MT19937-64 stream with a single state buffer. Batches of up to 64 draws
// may cross a block boundary: the words left in the old block move to `carry` first.
struct ZoneMt {
    uint64_t* buf;
    uint64_t* carry;
    const uint64_t* seeded;  // the zone's seeded state, loaded at the first draw
    int pos;     // next draw: carry[ncarry + pos] if pos < 0, else buf[pos]
    int ncarry;
    int lane;

    __device__ __forceinline__ void init(uint64_t* b, uint64_t* c, const uint64_t* s, int lane_) {
        buf = b;
        carry = c;
        seeded = s;
        pos = kMtN;
        ncarry = 0;
        lane = lane_;
    }
    __device__ __forceinline__ void ensure(int k) {  // k <= 64
        if (pos + k <= kMtN) return;
        const int left = mt_refill(buf, carry, seeded, pos, lane);
        seeded = nullptr;
        ncarry = left;
        pos = -left;
    }
    __device__ __forceinline__ uint64_t peek(int i) const {
        const int j = pos + i;
        return mt_temper((j < 0) ? carry[ncarry + j] : buf[j]);
    }
    __device__ __forceinline__ void consume(int k) { pos += k; }
    __device__ __forceinline__ uint64_t next() {
        ensure(1);
        const uint64_t u = peek(0);
        consume(1);
        return u;
    }
    __device__ __forceinline__ double u01() { return canon(next()); }
    __device__ __forceinline__ uint64_t uint_in(uint64_t lo, uint64_t hi) {
        const uint64_t range = hi - lo + 1ULL;
        uint64_t u = next();
        uint64_t low = u * range;
        uint64_t high = __umul64hi(u, range);
        if (low < range) {
            const uint64_t thr = umod64_slow(0ULL - range, range);
            while (low < thr) {
                u = next();
                low = u * range;
                high = __umul64hi(u, range);
            }
        }
        return high + lo;
    }
};

// std::shuffle of m entries at a (warp-uniform; lane 0 performs the swaps)
template <typename T>
__device__ __forceinline__ void zone_shuffle(T* a, int m, ZoneMt& r, int lane) {
    if (m <= 0) return;
    int i = 1;
    if ((m % 2) == 0) {
        const int j = (int)r.uint_in(0, 1);
        if (lane == 0) {
            const T t = a[i];
            a[i] = a[j];
            a[j] = t;
        }
        ++i;
    }
    while (i != m) {
        const uint64_t sr = (uint64_t)i + 1ULL;
        const uint64_t x = r.uint_in(0, sr * (sr + 1ULL) - 1ULL);
        // x < sr (sr + 1) < 2^32 for the list sizes here: 32-bit division is exact
        int p1, p2;
        if (sr < 65535ULL) {
            const uint32_t x32 = (uint32_t)x, b1 = (uint32_t)sr + 1u;
            const uint32_t q = x32 / b1;
            p1 = (int)q;
            p2 = (int)(x32 - q * b1);
        } else {
            const uint64_t q = udiv64_slow(x, sr + 1ULL);
            p1 = (int)q;
            p2 = (int)(x - q * (sr + 1ULL));
        }
        if (lane == 0) {
            T t = a[i];
            a[i] = a[p1];
            a[p1] = t;
            t = a[i + 1];
            a[i + 1] = a[p2];
            a[p2] = t;
        }
        i += 2;
    }
    __syncwarp();
}

// The same shuffle for m <= 32 entries, with every draw taken from the stream at once: lane
// k computes draw k, and the swaps are applied in draw order to one value per lane. If some
// draw would need Lemire's rejection step (probability ~ range / 2^64), nothing is consumed
// and the sequential version runs instead.
template <typename T>
__device__ __forceinline__ void zone_shuffle_fast(T* a, int m, ZoneMt& r, int lane) {
    if (m <= 1) return;
    if (m > kWarp) {
        zone_shuffle(a, m, r, lane);
        return;
    }
    const bool even = (m % 2) == 0;
    const int D = (even ? 1 : 0) + (m - (even ? 2 : 1)) / 2;  // <= 16 draws
    r.ensure(D);
    int i = 0, p1 = 0, p2 = -1;
    bool rej = false;
    if (lane < D) {
        const bool first2 = even && lane == 0;
        i = first2 ? 1 : (even ? 2 : 1) + 2 * (lane - (even ? 1 : 0));
        const uint64_t R = first2 ? 2ULL : (uint64_t)(i + 1) * (uint64_t)(i + 2);
        const uint64_t u = r.peek(lane);
        const uint64_t low = u * R;
        if (low < R) rej = low < umod64_slow(0ULL - R, R);
        const uint32_t x = (uint32_t)__umul64hi(u, R);
        if (first2) {
            p1 = (int)x;
        } else {
            const uint32_t b1 = (uint32_t)(i + 2), q = x / b1;
            p1 = (int)q;
            p2 = (int)(x - q * b1);
        }
    }
    if (__any_sync(0xffffffffu, rej)) {
        zone_shuffle(a, m, r, lane);
        return;
    }
    r.consume(D);
    // draw k swaps entry i_k (known from k) with p1 and entry i_k + 1 with p2: one shuffle fetches
    // both places, two move the values
    unsigned v = (lane < m) ? (unsigned)a[lane] : 0u;
    const int pq = p1 | (p2 << 8);  // p2 = -1: no second swap
    const int i0 = even ? 2 : 1;
    for (int k = 0; k < D; ++k) {
        const int w = __shfl_sync(0xffffffffu, pq, k);
        const int a1 = w & 0xff, a2 = w >> 8;
        const int ik = (even && k == 0) ? 1 : i0 + 2 * (k - (even ? 1 : 0));
        v = __shfl_sync(0xffffffffu, v, (lane == ik) ? a1 : ((lane == a1) ? ik : lane));
        if (a2 >= 0) {
            const int i2 = ik + 1;
            v = __shfl_sync(0xffffffffu, v, (lane == i2) ? a2 : ((lane == a2) ? i2 : lane));
        }
    }
    if (lane < m) a[lane] = (T)v;
    __syncwarp();
}

// sqrt(-2 ln r2 / r2) of the polar method, out of line
__device__ __noinline__ double polar_scale(double r2) { return sqrt(__ddiv_rn(__dmul_rn(-2.0, log_cr_dev(r2)), r2)); }

// polar-method normal deviate (libstdc++ normal_distribution), one cached value
struct ZoneNormal {
    double saved;
    int has;
    __device__ __forceinline__ double next(ZoneMt& r) {
        if (has) {
            has = 0;
            return saved;
        }
        double x, y, r2;
        do {
            x = __dsub_rn(__dmul_rn(2.0, r.u01()), 1.0);
            y = __dsub_rn(__dmul_rn(2.0, r.u01()), 1.0);
            r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
        } while (r2 > 1.0 || r2 == 0.0);
        const double mult = polar_scale(r2);
        saved = __dmul_rn(x, mult);
        has = 1;
        return __dmul_rn(y, mult);
    }
};

// Repacks the materialised lists of a zone at the bottom of its arena, in arena order;
// returns the new arena top. Out of line: it runs only when the arena is full.
template <typename I>
__device__ __noinline__ int zone_compact(uint8_t* cflags, I* abase, I* head, const I* len, I* cap,
                                         uint16_t* order, uint32_t* arena, int nl, int lane) {
    for (int l = lane; l < nl; l += kWarp) {
        int r = 0;
        if (cflags[l] & kCMat)
            for (int q = 0; q < nl; ++q)
                if ((cflags[q] & kCMat) && (abase[q] < abase[l] || (abase[q] == abase[l] && q < l))) ++r;
        order[l] = (uint16_t)r;
    }
    __syncwarp();
    int nmat = 0;
    for (int l = 0; l < nl; ++l) nmat += (cflags[l] & kCMat) ? 1 : 0;
    int off = 0;
    for (int r = 0; r < nmat; ++r) {
        int l = 0;
        for (int q = 0; q < nl; ++q)
            if ((cflags[q] & kCMat) && order[q] == r) l = q;
        const int a = abase[l] + head[l], n = len[l];
        // off <= a: copy down in ascending chunks (reads of a chunk precede its writes)
        for (int j0 = 0; j0 < n; j0 += kWarp) {
            const int j = j0 + lane;
            const uint32_t v = (j < n) ? arena[a + j] : 0u;
            __syncwarp();
            if (j < n) arena[off + j] = v;
            __syncwarp();
        }
        if (lane == 0) {
            abase[l] = off;
            head[l] = 0;
            cap[l] = n;
        }
        off += n;
        __syncwarp();
    }
    __syncwarp();
    return off;
}

// smoothed occupancy on the zone plus a one-cell ring (src/zone_pass.cpp:296-319):
// 3x3 binomial weights, renormalised over the in-domain neighbours. Out of line: called at most twice per
// pass, and inlined integer sums came out wrong from ptxas 12.9 in the overflow path's 32-bit working set.
template <typename W, typename I>
__device__ __noinline__ void zone_compute_nsm(double* nsm, const W* win, const I* cnt, int xs, int ys, int TX,
                                              int TY, int Nx, int Ny, int perx, int pery, int lane) {
    const int GX = TX + 2, GY = TY + 2, WY = TY + 4;
    for (int g = lane; g < GX * GY; g += kWarp) {
        int ix = xs - 1 + g / GY, iy = ys - 1 + g % GY;
        if (perx) ix = wrap_index(ix, Nx);
        if (pery) iy = wrap_index(iy, Ny);
        double val = 0.0;
        if (ix >= 0 && ix < Nx && iy >= 0 && iy < Ny) {
            double acc = 0.0, ws = 0.0;
            for (int dy = -1; dy <= 1; ++dy)
                for (int dx = -1; dx <= 1; ++dx) {
                    const int jy = iy + dy, jx = ix + dx;
                    if (jy < 0 || jy >= Ny || jx < 0 || jx >= Nx) continue;
                    const double w = ((dx == 0) ? 2.0 : 1.0) * ((dy == 0) ? 2.0 : 1.0) * 0.0625;
                    int c;
                    if (jx >= xs && jx < xs + TX && jy >= ys && jy < ys + TY) {
                        c = cnt[(jx - xs) * TY + (jy - ys)];
                    } else {
                        int wx = jx - (xs - 2), wy = jy - (ys - 2);
                        if (wx < 0) wx += Nx;
                        else if (wx >= TX + 4) wx -= Nx;
                        if (wy < 0) wy += Ny;
                        else if (wy >= WY) wy -= Ny;
                        c = win[wx * WY + wy];
                    }
                    acc = __dadd_rn(acc, __dmul_rn(w, (double)c));
                    ws = __dadd_rn(ws, w);
                }
            val = __ddiv_rn(acc, smax(ws, 1e-30));
        }
        nsm[g] = val;
    }
    __syncwarp();
}

// A donor's score 100 align + Nsm + 1e-9 N(0,1) with the correctly rounded norm of the gradient
// and deviate (comp, rad: zone_normals_draw), the reference's value. Out of line: it runs only
// where the ranking is not certain without it.
__device__ __noinline__ double zone_exact_score(double gx, double gy, double ddx, double ddy, double nstep, double nsmd,
                                                double comp, double rad) {
    const double ndir = mpcd_dd::hypot_cr(gx, gy);
    double align = 0.0;
    if (ndir >= 1e-14 && nstep >= 1e-14)
        align = __ddiv_rn(__dadd_rn(__dmul_rn(ddx, gx), __dmul_rn(ddy, gy)), __dmul_rn(ndir, nstep));
    const double noise = __dmul_rn(1e-9, __dmul_rn(comp, polar_scale(rad)));
    return __dadd_rn(__dadd_rn(__dmul_rn(100.0, align), nsmd), noise);
}

// cnt deviates of one fresh normal_distribution (polar method: pairs of uniforms in stream
// order until r2 is in (0, 1]; each accepted pair gives y*m, then the cached x*m), drawn but not
// evaluated: comp and rad receive each deviate's polar component and r2, so that the deviate is
// comp * polar_scale(r2). Lane c examines candidate pair c of the batch; the accepted ones are
// ranked by ballot.
__device__ __forceinline__ void zone_normals_draw(double* comp, double* rad, int cnt, ZoneMt& r, int lane) {
    int got = 0;
    while (got < cnt) {
        r.ensure(2 * kWarp);
        const double x = __dsub_rn(__dmul_rn(2.0, canon(r.peek(2 * lane))), 1.0);
        const double y = __dsub_rn(__dmul_rn(2.0, canon(r.peek(2 * lane + 1))), 1.0);
        const double r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
        const bool acc = !(r2 > 1.0 || r2 == 0.0);
        const unsigned am = __ballot_sync(0xffffffffu, acc);
        const int need = (cnt - got + 1) / 2;
        const int rank = __popc(am & lanemask_lt());
        const int used = min(__popc(am), need);
        int last = kWarp - 1;
        if (__popc(am) >= need) last = __ffs(__ballot_sync(0xffffffffu, acc && rank == need - 1)) - 1;
        if (acc && rank < need) {
            const int k0 = got + 2 * rank;
            comp[k0] = y;
            rad[k0] = r2;
            if (k0 + 1 < cnt) {
                comp[k0 + 1] = x;
                rad[k0 + 1] = r2;
            }
        }
        r.consume(2 * (last + 1));
        got += 2 * used;
    }
    __syncwarp();
}

// Scalar (warp-uniform) state of one zone.
template <typename I, bool kF32 = false>
struct ZoneState {
    ZoneMem<I> M;
    ZoneMt rng;
    const ZoneArgs* A;
    int lane, zone;
    int xs, xe, ys, ye, TX, TY, nl, WY;
    // l / TY as (l * tyMagic) >> 32, tyMagic = ceil(2^32 / TY) (2^32 for TY = 1): exact for
    // l * TY < 2^32, which the 16-bit working set guarantees (l, TY < 2^16); the int path divides
    unsigned long long tyMagic;
    int arenaTop, arenaCap;
    int movedDense, movedSparse;
    int atanLane;   // lane k < 25 holds the angular bin of step k (DevParams::atanBin)
    double hypLane; // lane k < 25 holds the length of step k (DevParams::hypotTab)
    bool nbDirect;  // no wrapped neighbour (|offset| <= 2) of a zone cell lies in the zone
    // dense cells by the integer tables (dense_cell_fast): this lane's range-2 neighbour as an
    // offset of the local cell, its step (dx, dy), scan place, and (chebyshev << 4 | distance^2)
    bool fast;
    int nOff, nDx, nDy, nOrig, nKey;
    bool dupNb5;    // a periodic axis shorter than 5 cells: range-2 neighbours can coincide
    bool dupNb3;    // a periodic axis shorter than 3 cells: 8-neighbours can coincide
    bool failed;   // capacity exhausted: the zone is handed to the overflow path
    bool fatal;    // a device error was raised

    __device__ __forceinline__ const DevParams& P() const { return A->P; }
    __device__ __forceinline__ bool in_zone(int ix, int iy) const { return ix >= xs && ix < xe && iy >= ys && iy < ye; }
    __device__ __forceinline__ int loc(int ix, int iy) const { return (ix - xs) * TY + (iy - ys); }
    __device__ __forceinline__ int lx_of(int l) const {
        return (sizeof(I) == 2) ? (int)(((unsigned long long)(unsigned)l * tyMagic) >> 32) : l / TY;
    }
    __device__ __forceinline__ int gx_of(int l) const { return xs + lx_of(l); }
    __device__ __forceinline__ int gy_of(int l) const { return ys + (l - lx_of(l) * TY); }

    __device__ __forceinline__ int nsm_index(int ix, int iy) const {
        int lx = ix - (xs - 1), ly = iy - (ys - 1);
        if (lx < 0) lx += P().Nx;
        if (lx >= TX + 2) lx -= P().Nx;
        if (ly < 0) ly += P().Ny;
        if (ly >= TY + 2) ly -= P().Ny;
        return lx * (TY + 2) + ly;
    }
    __device__ __forceinline__ bool shift_index(int iy, int ix, int dy, int dx, int& jy, int& jx) const {
        jy = iy + dy;
        if (P().pery) jy = wrap_index(jy, P().Ny);
        else if (jy < 0 || jy >= P().Ny) return false;
        jx = ix + dx;
        if (P().perx) jx = wrap_index(jx, P().Nx);
        else if (jx < 0 || jx >= P().Nx) return false;
        return true;
    }
    __device__ __forceinline__ int step_index(int sx, int sy, int tx, int ty, int& ddx, int& ddy) const {
        int a = tx - sx, b = ty - sy;
        if (P().perx) {
            if (a > P().Nx / 2) a -= P().Nx;
            if (a < -P().Nx / 2) a += P().Nx;
        }
        if (P().pery) {
            if (b > P().Ny / 2) b -= P().Ny;
            if (b < -P().Ny / 2) b += P().Ny;
        }
        ddx = a;
        ddy = b;
        if (a < -2 || a > 2 || b < -2 || b > 2) return -1;
        return (a + 2) + 5 * (b + 2);
    }

    // threshold maps (src/zone_pass.cpp:321-345, :715-725) from the cell's bulk flag at
    // the last map build and the smoothed occupancy then
    __device__ __forceinline__ double frac(int l) const {
        const DevParams& p = P();
        if (!p.useLFF) return 1.0;
        const double fraw = __ddiv_rn(M.nsm[nsm_index(gx_of(l), gy_of(l))], smax(p.gamma, 1e-12));
        const double g = __dmul_rn(p.fluidFracGain, fraw);
        return (g < 0.0) ? 0.0 : ((1.0 < g) ? 1.0 : g);
    }
    __device__ __forceinline__ double map_low(int l) const {
        const DevParams& p = P();
        if (M.cflags[l] & kCBulkBefore) return p.lowThrBulk;
        return smax(__dmul_rn(p.lowFrac, __dmul_rn(p.gamma, frac(l))), p.lowThrFloor);
    }
    __device__ __forceinline__ double map_high(int l) const {
        const DevParams& p = P();
        if (M.cflags[l] & kCBulkBefore) return p.highThr;
        return smax(__dmul_rn(p.highFrac, __dmul_rn(p.gamma, frac(l))), p.highThrFloor);
    }
    __device__ __forceinline__ double map_val(int l, bool low) const { return low ? map_low(l) : map_high(l); }

    // ------------------------------------------------------------------ smoothing, maps
    __device__ void compute_nsm() {
        zone_compute_nsm(M.nsm, M.win, M.len, xs, ys, TX, TY, P().Nx, P().Ny, P().perx, P().pery, lane);
    }

    // start of a map build: record which cells are bulk (cnt > 0)
    __device__ void mark_bulk() {
        for (int l = lane; l < nl; l += kWarp) {
            const uint8_t f = M.cflags[l];
            M.cflags[l] = (uint8_t)((f & ~kCBulkBefore) | ((M.len[l] > 0) ? kCBulkBefore : 0));
        }
        __syncwarp();
    }

    template <typename Pred>
    __device__ int collect(Pred pred) {
        int total = 0;
        for (int b = 0; b < nl; b += kWarp) {
            const int l = b + lane;
            const bool ok = (l < nl) && pred(l);
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            if (ok) M.list[total + __popc(m & lanemask_lt())] = (uint16_t)l;
            total += __popc(m);
        }
        __syncwarp();
        return total;
    }

    // ------------------------------------------------------------------ lists
    __device__ __forceinline__ uint32_t elem(int l, int i) const {
        if (M.cflags[l] & kCMat) return M.arena[M.abase[l] + M.head[l] + i];
        return ((uint32_t)l << kEntryShift) | (uint32_t)(M.head[l] + i);
    }

    // repack the materialised lists at the bottom of the arena (rare: out of line)
    __device__ void compact() {
        arenaTop = zone_compact(M.cflags, M.abase, M.head, M.len, M.cap, M.order, M.arena, nl, lane);
    }

    // materialise or grow list t so that `extra` entries can be appended
    __device__ bool ensure_room(int t, int extra) {
        const bool mat = (M.cflags[t] & kCMat) != 0;
        if (mat && M.head[t] + M.len[t] + extra <= M.cap[t]) return true;
        const int n = M.len[t];
        const int want = n + extra + 4;
        if (arenaTop + want > arenaCap) {
            compact();
            if (arenaTop + want > arenaCap) {
                failed = true;
                return false;
            }
        }
        for (int j = lane; j < n; j += kWarp) M.arena[arenaTop + j] = elem(t, j);
        __syncwarp();
        if (lane == 0) {
            M.abase[t] = arenaTop;
            M.head[t] = 0;
            M.cap[t] = want;
            M.cflags[t] |= kCMat;
        }
        arenaTop += want;
        __syncwarp();
        return true;
    }

    // Move `nt` particles from positions srcOff.. of list s into cell t, drawing positions
    // with sample_in_cell (src/zone_pass.cpp:280-294): per particle U for x then U for y.
    // slotPre/preOff: lane k holds the slot of entry preOff + k of list s if it was loaded
    // ahead (owned entries only); entries outside that window are loaded here.
    __device__ bool move_into(int s, int srcOff, int nt, int t, int slotPre = -1, int preOff = 1 << 29) {
        if (!ensure_room(t, nt)) return false;
        const DevParams& p = P();
        const double x0 = __dmul_rn((double)gx_of(t), p.dx), y0 = __dmul_rn((double)gy_of(t), p.dy);
        const int dst = M.abase[t] + M.head[t] + M.len[t];
        for (int q0 = 0; q0 < nt; q0 += kWarp) {
            const int c = min(kWarp, nt - q0);
            rng.ensure(2 * c);
            const int q = q0 + lane;
            const int w = preOff + srcOff + q;  // position in the prefetched window
            const int pre = __shfl_sync(0xffffffffu, slotPre, w & (kWarp - 1));
            if (lane < c) {
                const uint32_t e = elem(s, srcOff + q);
                const double px = __dadd_rn(x0, __dmul_rn(p.dx, canon(rng.peek(2 * lane))));
                const double py = __dadd_rn(y0, __dmul_rn(p.dy, canon(rng.peek(2 * lane + 1))));
                const int lc = (int)(e >> kEntryShift);
                if (M.cflags[lc] & kCOwned) {
                    const int sl = (w < kWarp) ? pre : A->slots[M.gstart[lc] + (int)(e & ((1u << kEntryShift) - 1))];
                    const int cc = cell_of(px, py, p);
                    if (kF32)
                        A->out32.set_pos(sl, make_double2(px, py), cc, p);
                    else
                        A->xout[sl] = make_double2(px, py);
                    A->cid[sl] = cc;
                }
                M.arena[dst + q] = e;
            }
            rng.consume(2 * c);
            __syncwarp();
        }
        if (lane == 0) {
            M.len[t] += nt;
        }
        __syncwarp();
        return true;
    }

    // receivers of a source cell, lane k < nrecv holding the k-th (at most 24 targets)
    __device__ __forceinline__ void push_recv(int& recvReg, int& nrecv, int c) {
        if (!__any_sync(0xffffffffu, lane < nrecv && recvReg == c)) {
            if (lane == nrecv) recvReg = c;
            ++nrecv;
        }
    }

    // update_transfer_correction_masks (src/zone_pass.cpp:492-525), forceSkip = false
    __device__ void update_masks(int src, int recvReg, int nrecv) {
        const bool ok = lane >= nrecv || (M.cflags[recvReg] & kCBulkBefore) != 0;
        const bool allBulk = ((M.cflags[src] & kCBulkBefore) != 0) && __all_sync(0xffffffffu, ok);
        const int prevRecv = __shfl_up_sync(0xffffffffu, recvReg, 1);
        if (lane <= nrecv) {
            const int c = (lane == 0) ? src : prevRecv;
            uint8_t f = M.cflags[c];
            if (allBulk) f |= kCBulkBulk;
            else f = (uint8_t)((f | kCSkip) & ~kCBulkBulk);
            M.cflags[c] = f;
        }
        __syncwarp();
    }

    // ------------------------------------------------------------------ dense phase
    // Targets of dense cell l, ranked, into T[0..m): admissible_dense_targets_rangeR
    // (src/zone_pass.cpp:413-434) with the zone filter, then rank_dense_targets_unified
    // (:436-490, inwardWeight = 0): angular bins, per-bin order on (-deficit, cnt, cheb,
    // dist2, U01) (a stable insertion sort), round robin over the bins from a random start.
    // Lane k < 24 examines neighbour k; the kept ones keep their order (compacted index ci).
    __device__ int select_targets(int l, bool low, int* T) {
        const int ix = gx_of(l), iy = gy_of(l);
        int nb = -1, ddx = 0, ddy = 0, idx = 0;
        if (lane < 24) {
            const int kk = (lane < 12) ? lane : lane + 1;
            const int dy = kk / 5 - 2, dx = kk % 5 - 2;
            int jy, jx;
            if (nbDirect ? in_zone(jx = ix + dx, jy = iy + dy) : (shift_index(iy, ix, dy, dx, jy, jx) && in_zone(jx, jy))) {
                const int t = loc(jx, jy);
                if ((double)M.len[t] < map_val(t, low)) nb = t;
            }
        }
        bool keep = nb >= 0;
        if (dupNb5) {  // wrapped offsets can coincide: keep the first occurrence of each cell
            const unsigned m0 = __ballot_sync(0xffffffffu, nb >= 0);
            const unsigned same = __match_any_sync(0xffffffffu, nb >= 0 ? nb : -1 - lane);
            keep = keep && ((same & m0 & lanemask_lt()) == 0);
        }
        const unsigned mk = __ballot_sync(0xffffffffu, keep);
        const int m = __popc(mk);
        if (m == 0) return 0;
        const int ci = __popc(mk & lanemask_lt());
        // draws: uniform_int(1, 8) for the start bin (range 8: Lemire never rejects), then one
        // U01 per target in compacted order
        rng.ensure(m + 1);
        const int startBin = (int)__umul64hi(rng.peek(0), 8ULL);
        int key2 = 0;
        double dneg = 0.0, tie = 0.0;
        if (keep) {
            idx = step_index(ix, iy, gx_of(nb), gy_of(nb), ddx, ddy);
            if (idx < 0) raise_error(A->st, kErrTableRange, zone);
            dneg = -smax(0.0, __dsub_rn(map_val(nb, low), (double)M.len[nb]));
            const int cheb = max(abs(ddx), abs(ddy)), d2 = ddx * ddx + ddy * ddy;
            key2 = (M.len[nb] << 8) | (cheb << 4) | d2;  // lexicographic (cnt, cheb, dist2)
            tie = canon(rng.peek(1 + ci));
        }
        rng.consume(m + 1);
        // angular bin of the step (table held in lanes 0..24)
        const int tb = __shfl_sync(0xffffffffu, atanLane, idx < 0 ? 0 : idx);
        const int bin = keep ? ((idx < 0) ? 0 : tb) : 8 + lane;
        // rank within the bin: compare only with the other kept lanes of the same bin
        unsigned others = __match_any_sync(0xffffffffu, bin) & ~(1u << lane);
        int r = 0;
        while (__any_sync(0xffffffffu, others != 0u)) {
            const int j = others ? (__ffs(others) - 1) : lane;
            others &= others - 1u;
            const double dj = __shfl_sync(0xffffffffu, dneg, j);
            const int kj = __shfl_sync(0xffffffffu, key2, j);
            const double tj = __shfl_sync(0xffffffffu, tie, j);
            if (j != lane) {
                bool less, eq = false;
                if (dj != dneg) less = dj < dneg;
                else if (kj != key2) less = kj < key2;
                else if (tj != tie) less = tj < tie;
                else { less = false; eq = true; }
                if (less || (eq && j < lane)) ++r;  // lane order = compacted order
            }
        }
        // round robin over the bins from startBin: position = entries of rank < r in every
        // bin, plus the bins before this one (in rotated order) that still hold rank r
        int pos = 0;
        for (int b = 0; b < 8; ++b) {
            const int cb = __popc(__ballot_sync(0xffffffffu, bin == b));
            if (keep) {
                pos += min(cb, r);
                const int rb = (b - startBin + 8) & 7, rq = (bin - startBin + 8) & 7;
                if (rb < rq && cb > r) ++pos;
            }
        }
        if (keep) T[pos] = nb;
        __syncwarp();
        return m;
    }

    // spread_particles_from_dense_source_round_robin (src/zone_pass.cpp:527-589). Lane k holds
    // target k's map value and deficit; a move changes only the deficit of its own target, so
    // each round walks the targets whose deficit was positive at the start of the round.
    __device__ int spread(int s, const int* T, int nT, bool low, int needOut, int& recvReg, int& nrecv, int slotPre,
                          int preOff) {
        if (needOut <= 0 || nT == 0) return 0;
        const int srcLen = M.len[s];
        if (srcLen == 0) return 0;
        int tl = -1, defj = 0;
        double mv = 0.0;
        if (lane < nT) {
            tl = T[lane];
            mv = map_val(tl, low);
            defj = max(0, (int)floor(__dsub_rn(mv, (double)M.len[tl])));
        }
        int taken = 0, moved = 0;
        bool stop = false;
        while (!stop && needOut > 0 && taken < srcLen) {
            const unsigned pm = __ballot_sync(0xffffffffu, lane < nT && defj > 0);
            if (pm == 0) break;  // no target can take a particle: no progress
            unsigned rest = pm;
            while (rest) {
                const int kk = __ffs(rest) - 1;
                rest &= rest - 1;
                const int deficit = __shfl_sync(0xffffffffu, defj, kk);
                const int t = __shfl_sync(0xffffffffu, tl, kk);
                const int remaining = __popc(pm >> kk);
                // ceil(needOut / remaining): integer division gives the same value as the
                // reference's ceil of the double quotient for these magnitudes
                const int rem1 = max(1, remaining);
                const int quota = max(1, (needOut + rem1 - 1) / rem1);
                const int nt = max(1, min(min(quota, deficit), min(needOut, srcLen - taken)));
                if (t == s) {
                    if (lane == 0) raise_error(A->st, kErrTargetIsSource, zone);
                    fatal = true;
                    return moved;
                }
                if (!move_into(s, taken, nt, t, slotPre, preOff)) return moved;
                push_recv(recvReg, nrecv, t);
                if (lane == kk) defj = max(0, (int)floor(__dsub_rn(mv, (double)M.len[tl])));
                taken += nt;
                moved += nt;
                needOut -= nt;
                if (needOut <= 0 || taken >= srcLen) {
                    stop = true;
                    break;
                }
            }
        }
        if (moved > 0 && lane == 0) {
            M.head[s] += taken;
            M.len[s] -= taken;
        }
        __syncwarp();
        return moved;
    }

    // one dense cell (src/zone_pass.cpp:734-753 calling :591-634)
    __device__ void dense_cell(int l) {
        int* T = M.small;
        int recvReg = -1;
        const int ncc = M.len[l];
        if (ncc <= 0) return;
        const double hl = map_high(l);
        if ((double)ncc <= hl) return;
        int nrecv = 0, moved = 0;
        // The two rounds take at most ceil(cnt - high) entries from the front of the list:
        // load the slots of the owned ones now, so the loads overlap the target ranking.
        int slotPre = -1;
        {
            const int take = min(min(M.len[l], max(0, (int)ceil(__dsub_rn((double)ncc, hl)))), kWarp);
            if (lane < take) {
                const uint32_t e = elem(l, lane);
                const int lc = (int)(e >> kEntryShift);
                if (M.cflags[lc] & kCOwned) slotPre = A->slots[M.gstart[lc] + (int)(e & ((1u << kEntryShift) - 1))];
            }
        }
        // first towards the low-threshold map, then whatever is left towards the high one
        // (one copy of the code for both rounds)
#pragma unroll 1
        for (int round = 0; round < 2; ++round) {
            const int need = max(0, (int)ceil(__dsub_rn((double)M.len[l], hl)));
            if (need <= 0) break;
            const bool low = (round == 0);
            const int nT = select_targets(l, low, T);
            moved += spread(l, T, nT, low, need, recvReg, nrecv, slotPre, moved);
            if (failed || fatal) return;
        }
        if (lane < nrecv) M.cflags[recvReg] |= (kCRecv | kCChanged);
        if (lane == 0 && moved > 0) M.cflags[l] |= kCChanged;
        __syncwarp();
        update_masks(l, recvReg, nrecv);
        movedDense += moved;
    }

    // One dense cell, as dense_cell, for zones whose tables hold (fast). Lane 3 b + k examines the
    // k-th neighbour of angular bin b for the whole call: the ranking compares a lane with the two
    // others of its bin, and counts order by ballots over (rank, bin) instead of loops over the
    // bins. All sums and comparisons are on integers (ZoneTables); the tie draw of a target is
    // consumed but never read, since the neighbours of a bin differ in (chebyshev, distance^2).
    // When no more particles leave than targets have a deficit, the round robin's quota stays 1:
    // the first `need` of them take one particle each, in one step with a lane per move (the usual
    // case; the general loop handles the rest). Bound by the latency of its dependent
    // instructions: a call takes 4,300 cycles with one zone per SM (8,600 in the general form),
    // 7,200 with 16 (12,500).
    __device__ void dense_cell_fast(int l) {
        const DevParams& p = P();
        const ZoneTables& z = p.zt;
        const int sCls = (M.cflags[l] & kCBulkBefore) ? 1 : 0;
        const int sFlo = z.flo[1][sCls];
        const int len0 = M.len[l];
        if (len0 <= sFlo) return;
        // ceil(n - high) in FP64, as an integer where the subtraction is exact
        auto excess = [&](int n) {
            return n <= 2 * sFlo ? max(0, n - sFlo) : (int)ceil(__dsub_rn((double)n, z.highThr[sCls]));
        };
        const int lx = lx_of(l), ly = l - lx * TY;
        const int t = l + nOff;
        const bool in = lane < 24 && (unsigned)(lx + nDx) < (unsigned)TX && (unsigned)(ly + nDy) < (unsigned)TY;
        // the slots of the owned entries that may leave, loaded ahead
        int slotPre = -1;
        if (lane < min(len0, excess(len0))) {
            const uint32_t e = elem(l, lane);
            const int lc = (int)(e >> kEntryShift);
            if (M.cflags[lc] & kCOwned) slotPre = A->slots[M.gstart[lc] + (int)(e & ((1u << kEntryShift) - 1))];
        }
        const int tCls = (in && (M.cflags[t] & kCBulkBefore)) ? 1 : 0;
        const int bin = lane / 3, base = 3 * bin;
        bool recv = false;
        int moved = 0;
#pragma unroll 1
        for (int round = 0; round < 2; ++round) {
            const int need = excess(len0 - moved);
            if (need <= 0) break;
            const int tLen = in ? M.len[t] : 0;
            const bool adm = in && tLen < z.cut[round][tCls];
            const unsigned om = __reduce_or_sync(0xffffffffu, adm ? (1u << nOrig) : 0u);
            if (om == 0) continue;
            const int m = __popc(om);
            rng.ensure(m + 1);
            const int startBin = (int)(rng.peek(0) >> 61);  // uniform_int(1, 8) - 1
            rng.consume(m + 1);
            // rank within the bin on (-deficit, cnt, chebyshev, distance^2)
            const int def = z.flo[round][tCls] - tLen;
            const unsigned key =
                adm ? ((unsigned)(255 - (2 * def + z.up[round][tCls])) << 13) | ((unsigned)tLen << 6) | (unsigned)nKey
                    : 0xffffffffu;
            const unsigned ka = __shfl_sync(0xffffffffu, key, base + (lane - base + 1) % 3);
            const unsigned kb = __shfl_sync(0xffffffffu, key, base + (lane - base + 2) % 3);
            // place in the round robin: rank, then bin from the start bin on
            const int q = ((ka < key) + (kb < key)) * 8 + ((bin - startBin) & 7);
            const unsigned below = (1u << (q & 31)) - 1u;
            const unsigned pm = __reduce_or_sync(0xffffffffu, adm && def > 0 ? (1u << q) : 0u);
            if (pm == 0) continue;
            bool one = need <= __popc(pm);
            const int i = __popc(pm & below);  // this target's turn
            const bool act = one && adm && def > 0 && i < need;
            int dst = 0;
            if (one) {
                // room for one entry at the end of each receiving list
                bool grow = act;
                if (act && (M.cflags[t] & kCMat)) {
                    const int hd = M.head[t];
                    dst = M.abase[t] + hd + tLen;
                    grow = hd + tLen >= (int)M.cap[t];
                }
                if (__any_sync(0xffffffffu, grow)) {
                    const int want = grow ? tLen + 5 : 0;
                    int end = want;
#pragma unroll
                    for (int o = 1; o < kWarp; o <<= 1) {
                        const int u = __shfl_up_sync(0xffffffffu, end, o);
                        if (lane >= o) end += u;
                    }
                    const int total = __shfl_sync(0xffffffffu, end, kWarp - 1);
                    one = arenaTop + total <= arenaCap;
                    if (one && grow) {
                        const int a = arenaTop + end - want;
                        const bool mat = (M.cflags[t] & kCMat) != 0;
                        const int from = M.head[t] + (mat ? (int)M.abase[t] : 0);
                        const uint32_t e0 = ((uint32_t)t << kEntryShift) | (uint32_t)from;
                        for (int j = 0; j < tLen; ++j) M.arena[a + j] = mat ? M.arena[from + j] : e0 + (uint32_t)j;
                        M.abase[t] = a;
                        M.head[t] = 0;
                        M.cap[t] = want;
                        M.cflags[t] |= kCMat;
                        dst = a + tLen;
                    }
                    if (one) arenaTop += total;
                    __syncwarp();
                }
            }
            if (!one) {
                int* T = M.small;
                const unsigned am = __reduce_or_sync(0xffffffffu, adm ? (1u << q) : 0u);
                if (adm) T[__popc(am & below)] = t;
                __syncwarp();
                int recvReg = -1, nrecv = 0;
                moved += spread(l, T, m, round == 0, need, recvReg, nrecv, slotPre, moved);
                if (failed || fatal) return;
                for (int k = 0; k < nrecv; ++k)
                    if (__shfl_sync(0xffffffffu, recvReg, k) == t && in) recv = true;
                continue;
            }
            rng.ensure(2 * need);
            const int w = moved + i;
            const int pre = __shfl_sync(0xffffffffu, slotPre, w & (kWarp - 1));
            if (act) {
                const uint32_t e = elem(l, i);
                const double px = __dadd_rn(__dmul_rn((double)(xs + lx + nDx), p.dx), __dmul_rn(p.dx, canon(rng.peek(2 * i))));
                const double py = __dadd_rn(__dmul_rn((double)(ys + ly + nDy), p.dy), __dmul_rn(p.dy, canon(rng.peek(2 * i + 1))));
                const int lc = (int)(e >> kEntryShift);
                if (M.cflags[lc] & kCOwned) {
                    const int sl = (w < kWarp) ? pre : A->slots[M.gstart[lc] + (int)(e & ((1u << kEntryShift) - 1))];
                    const int cc = cell_of(px, py, p);
                    if (kF32)
                        A->out32.set_pos(sl, make_double2(px, py), cc, p);
                    else
                        A->xout[sl] = make_double2(px, py);
                    A->cid[sl] = cc;
                }
                M.arena[dst] = e;
                M.len[t] = tLen + 1;
                recv = true;
            }
            rng.consume(2 * need);
            moved += need;
            __syncwarp();
            if (lane == 0) {
                M.head[l] += need;
                M.len[l] -= need;
            }
            __syncwarp();
        }
        // receivers' flags and update_transfer_correction_masks (src/zone_pass.cpp:492-525) on the
        // source (lane 31) and its receivers
        const bool allBulk = sCls && __all_sync(0xffffffffu, !recv || tCls);
        if (recv || lane == kWarp - 1) {
            const int c = recv ? t : l;
            uint8_t f = M.cflags[c];
            if (recv) f |= kCRecv | kCChanged;
            else if (moved > 0) f |= kCChanged;
            M.cflags[c] = allBulk ? (uint8_t)(f | kCBulkBulk) : (uint8_t)((f | kCSkip) & ~kCBulkBulk);
        }
        __syncwarp();
        movedDense += moved;
    }

    // ------------------------------------------------------------------ sparse phase
    // Gradient of the smoothed occupancy at cell l (src/zone_pass.cpp:375-411). The ring around the
    // zone holds the wrapped neighbours' values, so the map is read at local offsets.
    __device__ __forceinline__ void inward(int l, int at, double& gx, double& gy) const {
        const DevParams& p = P();
        const int ix = gx_of(l), iy = gy_of(l), SY = TY + 2;
        const double* n = M.nsm + at;
        if (!p.perx && ix == 0) gx = __dsub_rn(n[SY], n[0]);
        else if (!p.perx && ix == p.Nx - 1) gx = __dsub_rn(n[0], n[-SY]);
        else gx = __dmul_rn(0.5, __dsub_rn(n[SY], n[-SY]));
        if (!p.pery && iy == 0) gy = __dsub_rn(n[1], n[0]);
        else if (!p.pery && iy == p.Ny - 1) gy = __dsub_rn(n[0], n[-1]);
        else gy = __dmul_rn(0.5, __dsub_rn(n[1], n[-1]));
    }

    // one sparse cell (src/zone_pass.cpp:804-854)
    __device__ void sparse_cell(int l) {
        const DevParams& p = P();
        int* don = M.small + 32;
        const int ncc = M.len[l];
        if (ncc <= 0) return;
        const int lx = lx_of(l), ly = l - lx * TY;
        const int ix = xs + lx, iy = ys + ly;
        int nb = -1;
        if (lane < 8) {
            const int kk = (lane < 4) ? lane : lane + 1;
            const int dy = kk / 3 - 1, dx = kk % 3 - 1;
            if (nbDirect) {
                if ((unsigned)(lx + dx) < (unsigned)TX && (unsigned)(ly + dy) < (unsigned)TY) nb = l + dx * TY + dy;
            } else {
                int jy, jx;
                if (shift_index(iy, ix, dy, dx, jy, jx) && in_zone(jx, jy)) nb = loc(jx, jy);
            }
        }
        const unsigned m0 = __ballot_sync(0xffffffffu, nb >= 0);
        if (m0 == 0) return;
        bool uniq = nb >= 0;
        if (dupNb3) {  // wrapped offsets can coincide: keep the first occurrence of each cell
            const unsigned same = __match_any_sync(0xffffffffu, nb >= 0 ? nb : -1 - lane);
            uniq = uniq && ((same & m0 & lanemask_lt()) == 0);
        }
        const int lowInt = p.lowThrBulkInt;
        int need = max(0, lowInt - ncc);
        if (need <= 0) return;
        const bool isDonor = uniq && M.len[nb] > lowInt;
        const unsigned md = __ballot_sync(0xffffffffu, isDonor);
        const int nd = __popc(md);
        if (nd == 0) return;
        if (isDonor) don[__popc(md & lanemask_lt())] = nb;
        __syncwarp();
        zone_shuffle_fast(don, nd, rng, lane);
        // One N(0,1) per donor in shuffled order, then scores in parallel (lane k = donor k). The
        // score 100 align + Nsm + 1e-9 N(0,1) only ranks the donors, and |N(0,1)| stays below 12.2
        // (r2 >= 2^-106), so the deviates and the last bits of the norm matter only where two
        // scores lie within 3e-8 of each other: the scores come from sqrt(gx^2 + gy^2) (within
        // 1e-12 (1 + |score|) of the reference's) without the deviates, and a ranking with a gap of
        // 1e-7 (1 + |score|) or less between two donors is done again from the exact values.
        zone_normals_draw(M.smallD, M.smallD + 8, nd, rng, lane);
        const int SY = TY + 2, at = (lx + 1) * SY + ly + 1;
        double gx, gy;
        inward(l, at, gx, gy);
        int dk = -1, idx = 0, ddx = 0, ddy = 0;
        double nsmd = 0.0;
        if (lane < nd) {
            dk = don[lane];
            const int dlx = lx_of(dk), dly = dk - dlx * TY;
            idx = step_index(ix, iy, xs + dlx, ys + dly, ddx, ddy);
            nsmd = M.nsm[(dlx + 1) * SY + dly + 1];
        }
        const double hs = __shfl_sync(0xffffffffu, hypLane, idx < 0 ? 0 : idx);
        const double nstep = (idx >= 0) ? hs : 0.0;
        const double ndirF = sqrt(__dadd_rn(__dmul_rn(gx, gx), __dmul_rn(gy, gy)));
        double sc = 0.0;
        if (lane < nd && ndirF >= 1e-14 && nstep >= 1e-14)
            sc = __dmul_rn(100.0, __ddiv_rn(__dadd_rn(__dmul_rn((double)ddx, gx), __dmul_rn((double)ddy, gy)),
                                            __dmul_rn(ndirF, nstep)));
        sc = __dadd_rn(sc, nsmd);
        bool sure = !(ndirF > 0.5e-14 && ndirF < 2e-14);
        int rk = 0;  // descending
        for (int j = 0; j < nd; ++j) {
            const double sj = __shfl_sync(0xffffffffu, sc, j);
            if (lane < nd && j != lane) {
                if (fabs(sj - sc) <= 1e-7 * (1.0 + fabs(sc))) sure = false;
                rk += sj > sc;
            }
        }
        if (!__all_sync(0xffffffffu, sure)) {
            sc = 0.0;
            if (lane < nd)
                sc = zone_exact_score(gx, gy, (double)ddx, (double)ddy, nstep, nsmd, M.smallD[lane], M.smallD[8 + lane]);
            rk = 0;  // ties in shuffled order (std::sort of <= 16 elements is an insertion sort)
            for (int j = 0; j < nd; ++j) {
                const double sj = __shfl_sync(0xffffffffu, sc, j);
                if (lane < nd && j != lane && (sj > sc || (sj == sc && j < lane))) ++rk;
            }
        }
        __syncwarp();
        if (lane < nd) don[rk] = dk;
        __syncwarp();
        for (int k = 0; k < nd; ++k) {
            const int d = don[k];
            const int ld = M.len[d];
            if (ld == 0) continue;
            const int avail = M.len[d] - lowInt;
            if (avail <= 0) continue;
            const int nt = min(min(need, avail), ld);
            if (nt <= 0) continue;
            if (!ensure_room(d, 0)) return;  // materialise the donor list to shuffle it
            zone_shuffle_fast(M.arena + M.abase[d] + M.head[d], ld, rng, lane);
            if (!move_into(d, 0, nt, l)) return;
            if (lane == 0) {
                M.head[d] += nt;
                M.len[d] -= nt;
                M.cflags[l] |= (kCRecv | kCChanged);
                M.cflags[d] |= kCChanged;
            }
            __syncwarp();
            update_masks(d, (lane == 0) ? l : -1, 1);
            movedSparse += nt;
            need -= nt;
            if (need <= 0) break;
        }
    }
};

// global cell of window position w (zone rectangle plus a 2-cell ring, wrapped)
template <typename I, bool kF32>
__device__ __forceinline__ int iy_ix_cell(const ZoneState<I, kF32>& S, int w, const DevParams& p) {
    int ix = S.xs - 2 + w / S.WY, iy = S.ys - 2 + w % S.WY;
    if (p.perx) ix = wrap_index(ix, p.Nx);
    if (p.pery) iy = wrap_index(iy, p.Ny);
    return iy + p.Ny * ix;
}

// End of a zone of the serial pass: apply the deferred momentum corrections, then publish
// the new list (ascending particle id) and count of every cell the zone changed.
template <typename I, bool kF32>
__device__ __forceinline__ void serial_finish(ZoneState<I, kF32>& S, const ZoneArgs& A, const DevParams& p) {
    ZoneMem<I>& M = S.M;
    const int lane = S.lane;
    for (int l = lane; l < S.nl; l += kWarp) {
        const double2 du = A.duScratch[l];
        if (du.x != 0.0 || du.y != 0.0) {
            const int n = M.len[l];
            for (int j = 0; j < n; ++j) {
                const uint32_t e = S.elem(l, j);
                const int sl = A.slots[M.gstart[(int)(e >> kEntryShift)] + (int)(e & ((1u << kEntryShift) - 1))];
                const double2 w = zone_vin<false>(A, sl);
                zone_vout<false>(A, sl, make_double2(__dadd_rn(w.x, du.x), __dadd_rn(w.y, du.y)));
            }
        }
    }
    __syncwarp();
    int top = *A.liveTop;
    for (int b = 0; b < S.nl; b += kWarp) {
        const int l = b + lane;
        const bool ch = l < S.nl && (M.cflags[l] & kCChanged);
        const int n = ch ? M.len[l] : 0;
        int off = n;  // inclusive scan of the list lengths
        for (int o = 1; o < kWarp; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, off, o);
            if (lane >= o) off += t;
        }
        const int total = __shfl_sync(0xffffffffu, off, kWarp - 1);
        off -= n;
        if (top + total > A.liveEnd) {
            if (lane == 0) raise_error(A.st, kErrZoneCapacity, S.zone);
            return;
        }
        if (ch) {
            const int dst = top + off;
            for (int j = 0; j < n; ++j) {
                const uint32_t e = S.elem(l, j);
                A.slotsW[dst + j] = A.slots[M.gstart[(int)(e >> kEntryShift)] + (int)(e & ((1u << kEntryShift) - 1))];
            }
            for (int i = dst + 1; i < dst + n; ++i) {  // insertion sort by particle id
                const int v = A.slotsW[i];
                const int pv = A.pid[v];
                int j = i;
                while (j > dst && A.pid[A.slotsW[j - 1]] > pv) {
                    A.slotsW[j] = A.slotsW[j - 1];
                    --j;
                }
                A.slotsW[j] = v;
            }
            const int gc = S.gy_of(l) + p.Ny * S.gx_of(l);
            A.liveStart[gc] = dst;
            A.liveCnt[gc] = n;
        }
        top += total;
    }
    __syncwarp();
    if (lane == 0) *A.liveTop = top;
    __syncwarp();
}

// ------------------------------------------------------------------ the zone body
// The zone body in four phases: set-up (the pass-input counts around the zone, the cells'
// segments and ownership, the draw stream), one dense pass, the sparse phase, and the output
// (momentum correction and the zone's stats). zone_body runs them back to back; the
// phase-synchronous kernel runs the zones of a block in step, a barrier between phases.

// Set-up; false if the zone must be re-run on the overflow path.
template <bool kSerial, typename I, bool kF32>
__device__ __forceinline__ bool zone_setup(ZoneState<I, kF32>& S, const ZoneArgs& A, int z, char* mem, int maxCells,
                                           int winCap, int arenaCap, int nsmCap) {
    S.A = &A;
    S.lane = threadIdx.x & 31;
    S.zone = z;
    S.failed = false;
    S.fatal = false;
    S.movedDense = S.movedSparse = 0;
    const int lane = S.lane;
    const DevParams& p = A.P;
    const int4 R = A.rects[z];
    S.xs = R.x; S.xe = R.y; S.ys = R.z; S.ye = R.w;
    S.TX = S.xe - S.xs; S.TY = S.ye - S.ys; S.nl = S.TX * S.TY; S.WY = S.TY + 4;
    S.tyMagic = (S.TY > 0) ? (unsigned long long)(0xffffffffu / (unsigned)S.TY) + 1ULL : 0ULL;
    S.atanLane = (lane < 25) ? p.atanBin[lane] : 0;
    S.hypLane = (lane < 25) ? p.hypotTab[lane] : 0.0;
    S.dupNb5 = (p.perx && p.Nx < 5) || (p.pery && p.Ny < 5);
    S.nbDirect = (!p.perx || S.TX < p.Nx - 2) && (!p.pery || S.TY < p.Ny - 2);
    S.dupNb3 = (p.perx && p.Nx < 3) || (p.pery && p.Ny < 3);
    S.fast = p.zt.ok && S.nbDirect;
    S.nDx = S.nDy = S.nOff = S.nOrig = S.nKey = 0;
    if (lane < 24) {
        S.nDx = p.zt.dx[lane];
        S.nDy = p.zt.dy[lane];
        S.nOrig = p.zt.orig[lane];
        S.nOff = S.nDx * S.TY + S.nDy;
        S.nKey = (max(abs(S.nDx), abs(S.nDy)) << 4) | (S.nDx * S.nDx + S.nDy * S.nDy);
    }
    const int W = (S.TX + 4) * S.WY;
    if (S.nl > maxCells || W > winCap || (S.TX + 2) * (S.TY + 2) > nsmCap || S.nl >= (1 << (32 - kEntryShift)) ||
        (sizeof(I) == 2 && S.nl > 65535))
        return false;
    S.M.carve(mem, maxCells, winCap, arenaCap, nsmCap);
    constexpr bool kNarrow = sizeof(I) == 2;  // 16-bit counts: window counts <= 32767, zone total <= 65535
    bool wide = false;
    S.arenaCap = arenaCap;
    S.arenaTop = 0;
    ZoneMem<I>& M = S.M;
    // pass-input counts around the zone
    for (int w0 = 0; w0 < W; w0 += 4 * kWarp) {
        uint64_t a[4], b[4];
        bool ok[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int w = w0 + lane + k * kWarp;
            int ix = S.xs - 2 + w / S.WY, iy = S.ys - 2 + w % S.WY;
            if (p.perx) ix = wrap_index(ix, p.Nx);
            if (p.pery) iy = wrap_index(iy, p.Ny);
            ok[k] = w < W && ix >= 0 && ix < p.Nx && iy >= 0 && iy < p.Ny;
            const int cc = ok[k] ? iy + p.Ny * ix : 0;
            a[k] = ok[k] ? A.start[cc] : 0ULL;
            b[k] = ok[k] ? A.start[cc + 1] : 0ULL;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int w = w0 + lane + k * kWarp;
            if (w < W) {
                int cv = ok[k] ? (int)((uint32_t)b[k] - (uint32_t)a[k]) : -1;
                if (kSerial && ok[k]) cv = A.liveCnt[iy_ix_cell(S, w, p)];
                if (kNarrow && cv > 32767) wide = true;
                M.win[w] = cv;
            }
        }
    }
    // zone cells: segment starts and ownership
    for (int l0 = 0; l0 < S.nl; l0 += 4 * kWarp) {
        int own[4];
        uint64_t st[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int l = l0 + lane + k * kWarp;
            const int c = (l < S.nl) ? S.gy_of(l) + p.Ny * S.gx_of(l) : 0;
            own[k] = (l < S.nl) ? A.owner[c] : 0;
            st[k] = (l < S.nl) ? A.start[c] : 0ULL;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int l = l0 + lane + k * kWarp;
            if (l < S.nl) {
                M.gstart[l] = kSerial ? A.liveStart[S.gy_of(l) + p.Ny * S.gx_of(l)] : (int)(uint32_t)st[k];
                M.cflags[l] = (kSerial || own[k] == z + 1) ? kCOwned : 0;
            }
        }
    }
    __syncwarp();
    int tot = 0;
    for (int l = lane; l < S.nl; l += kWarp) {
        const int c = M.win[(l / S.TY + 2) * S.WY + (l % S.TY + 2)];
        tot += c;
        M.cnt0[l] = c;
        M.len[l] = c;
        M.head[l] = 0;
        M.abase[l] = 0;
        M.cap[l] = 0;
    }
    if (kNarrow) {  // counts too large for the 16-bit working set: the overflow path takes the zone
        for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
        if (__any_sync(0xffffffffu, wide) || tot > 65535) return false;
    }
    __syncwarp();
    S.rng.init(M.mt, M.carry, A.seeds + (size_t)z * kMtN, lane);
    return true;
}

// One dense pass (src/zone_pass.cpp:708-781): the cells above their high map, in shuffled
// order. Returns how many.
template <typename I, bool kF32>
__device__ __forceinline__ int zone_dense_pass(ZoneState<I, kF32>& S) {
    const int lane = S.lane;
    const DevParams& p = S.A->P;
    ZoneMem<I>& M = S.M;
    if (p.useLFF) S.compute_nsm();
    S.mark_bulk();
    const int nd = S.collect([&](int l) {
        return S.fast ? (int)M.len[l] > p.zt.flo[1][(M.cflags[l] & kCBulkBefore) ? 1 : 0]
                      : (double)M.len[l] > S.map_high(l);
    });
    zone_shuffle_fast(M.list, nd, S.rng, lane);
    for (int q = 0; q < nd && !S.failed && !S.fatal; ++q) {
        if (S.fast) S.dense_cell_fast((int)M.list[q]);
        else S.dense_cell((int)M.list[q]);
    }
    return nd;
}

// The sparse phase (src/zone_pass.cpp:783-854). Returns the sparse cells.
template <typename I, bool kF32>
__device__ __forceinline__ int zone_sparse(ZoneState<I, kF32>& S) {
    const int lane = S.lane;
    const DevParams& p = S.A->P;
    ZoneMem<I>& M = S.M;
    // the smoothed occupancy feeds the maps only with local fluid-fraction thresholds;
    // otherwise it is needed only if some cell is sparse (inward gradient, donor scores)
    if (p.useLFF) S.compute_nsm();
    S.mark_bulk();
    const int nlow = S.collect([&](int l) { return M.len[l] > 0 && (double)M.len[l] < S.map_low(l); });
    if (!p.useLFF && nlow > 0) S.compute_nsm();
    zone_shuffle_fast(M.list, nlow, S.rng, lane);
    for (int q = 0; q < nlow && !S.failed && !S.fatal; ++q) S.sparse_cell((int)M.list[q]);
    return nlow;
}

// Output: the momentum correction and the zone's stats; false if the zone must be re-run on the
// overflow path.
template <bool kSerial, typename I, bool kF32>
__device__ __forceinline__ bool zone_finish(ZoneState<I, kF32>& S, const ZoneArgs& A, int z, int nHighAll, int nLowAll) {
    const int lane = S.lane;
    const DevParams& p = A.P;
    ZoneMem<I>& M = S.M;
    if (S.fatal) return true;
    if (S.failed) return false;

    // momentum correction (src/zone_pass.cpp:870-922): per changed cell, the momentum of
    // its input list and of its final list, both in list order; owned particles of
    // corrected cells get v + du
    double* du2 = M.nsm;
    const bool wantDiag = kSerial && A.zoneDiag != nullptr;
    double dgUx2 = 0.0, dgUy2 = 0.0, dgPx2 = 0.0, dgPy2 = 0.0;
    int dgNPx = 0, dgNPy = 0;
    for (int l = lane; l < S.nl; l += kWarp) {
        du2[l] = 0.0;
        if (kSerial) A.duScratch[l] = make_double2(0.0, 0.0);  // cells left unchanged get none
        const int n = M.len[l];
        if (wantDiag && !(M.cflags[l] & kCChanged) && n > 0) {
            // an unchanged cell: uxNow from its input list (ascending id), no momentum error
            double sx = 0.0, sy = 0.0;
            for (int j = 0; j < n; ++j) {
                const double2 w = zone_vin<kF32>(A, A.slots[M.gstart[l] + j]);
                sx = __dadd_rn(sx, w.x);
                sy = __dadd_rn(sy, w.y);
            }
            const double ux = __ddiv_rn(sx, (double)n), uy = __ddiv_rn(sy, (double)n);
            dgUx2 = __dadd_rn(dgUx2, __dmul_rn(ux, ux));
            dgUy2 = __dadd_rn(dgUy2, __dmul_rn(uy, uy));
        }
    }
    // The changed cells, one per lane (listed first: about 70 of a base zone's 100, few of a
    // shifted one's). A lane's chain is slot, then velocity, for each of its
    // particles; the slots of 16 are loaded together, then their velocities in two batches of 8.
    // A materialised list is dead after its sum: its entries are replaced by their slots there
    // (bit 31: not owned), so that the correction finds them without another look-up.
    constexpr int kOwnBit = (int)0x80000000u;
    const int nch = S.collect([&](int l) { return (M.cflags[l] & kCChanged) && M.len[l] > 0; });
    for (int q = lane; q < nch; q += kWarp) {
        const int l = M.list[q];
        const uint8_t f = M.cflags[l];
        const int n = M.len[l], g0 = M.gstart[l];
        const bool mat = (f & kCMat) != 0;
        const int at = (mat ? (int)M.abase[l] : g0) + (int)M.head[l];
        auto sum = [&](int cnt, auto slotAt, double& sx, double& sy) {
            for (int j0 = 0; j0 < cnt; j0 += 16) {
                int sl[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) sl[u] = (j0 + u < cnt) ? slotAt(j0 + u) : 0;
#pragma unroll
                for (int h = 0; h < 16; h += 8) {
                    if (j0 + h >= cnt) break;
                    double2 w[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) w[u] = (j0 + h + u < cnt) ? zone_vin<kF32>(A, sl[h + u]) : make_double2(0.0, 0.0);
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (j0 + h + u < cnt) {
                            sx = __dadd_rn(sx, w[u].x);
                            sy = __dadd_rn(sy, w[u].y);
                        }
                }
            }
        };
        if (!kSerial && mat && A.moverSlot) {
            // the particles of this list that changed cells (a list left implicit has none)
#pragma unroll 1
            for (int j = 0; j < n; ++j) {
                const uint32_t e = M.arena[at + j];
                const int lc = (int)(e >> kEntryShift);
                if (!(M.cflags[lc] & kCOwned)) continue;
                const int sl = A.slots[M.gstart[lc] + (int)(e & ((1u << kEntryShift) - 1))];
                const int from = S.gy_of(lc) + p.Ny * S.gx_of(lc), to = A.cid[sl];
                if (to == from) continue;
                const int m = atomicAdd(A.moverCount, 1);
                A.moverSlot[m] = sl;
                A.moverNext[m] = atomicExch(A.arrHead + to, m);
                A.depart[from] = 1;
            }
        }
        double bx = 0.0, by = 0.0, axs = 0.0, ays = 0.0;
        sum((int)M.cnt0[l], [&](int j) { return A.slots[g0 + j]; }, bx, by);
        sum(n, [&](int j) {
            if (!mat) return A.slots[at + j];
            const uint32_t e = M.arena[at + j];
            const int lc = (int)(e >> kEntryShift);
            const int sl = A.slots[M.gstart[lc] + (int)(e & ((1u << kEntryShift) - 1))];
            if (!kSerial) M.arena[at + j] = (uint32_t)sl | ((M.cflags[lc] & kCOwned) ? 0u : (uint32_t)kOwnBit);
            return sl;
        }, axs, ays);
        const double ux = __ddiv_rn(__dsub_rn(bx, axs), (double)n);
        const double uy = __ddiv_rn(__dsub_rn(by, ays), (double)n);
        du2[l] = __dadd_rn(__dmul_rn(ux, ux), __dmul_rn(uy, uy));
        if (wantDiag) {
            const double ax = __ddiv_rn(axs, (double)n), ay = __ddiv_rn(ays, (double)n);
            dgUx2 = __dadd_rn(dgUx2, __dmul_rn(ax, ax));
            dgUy2 = __dadd_rn(dgUy2, __dmul_rn(ay, ay));
            const double dpx = __dsub_rn(bx, axs), dpy = __dsub_rn(by, ays);
            const double ex = __dmul_rn(dpx, dpx), ey = __dmul_rn(dpy, dpy);
            if (ex > 0.0) { dgPx2 = __dadd_rn(dgPx2, ex); ++dgNPx; }
            if (ey > 0.0) { dgPy2 = __dadd_rn(dgPy2, ey); ++dgNPy; }
        }
        bool doCorr = p.momCorr != 0;
        if (doCorr && (f & kCSkip)) doCorr = false;
        if (doCorr && (f & kCRecv) && !(f & kCBulkBulk)) doCorr = false;
        doCorr = doCorr && (ux != 0.0 || uy != 0.0);
        if (kSerial) {
            // in place: every cell's sums must read the velocities of the zone's start
            if (doCorr) A.duScratch[l] = make_double2(ux, uy);
        } else if (doCorr && A.corrSlot) {  // in place: listed (few cells: one entry at a time)
            if (mat || (f & kCOwned)) {
                int k = n;
                if (mat) {
                    k = 0;
#pragma unroll 1
                    for (int j = 0; j < n; ++j) k += !(M.arena[at + j] >> 31);
                }
                int d = k > 0 ? atomicAdd(A.corrCount, k) : 0;
#pragma unroll 1
                for (int j = 0; j < n; ++j) {
                    const int sl = mat ? (int)M.arena[at + j] : A.slots[at + j];
                    if (sl < 0) continue;
                    const double2 w = zone_vin<kF32>(A, sl);
                    A.corrSlot[d] = sl;
                    A.corrV[d++] = make_double2(__dadd_rn(w.x, ux), __dadd_rn(w.y, uy));
                }
            }
        } else if (doCorr && (mat || (f & kCOwned))) {
            for (int j0 = 0; j0 < n; j0 += 8) {
                int sl[8];
                double2 w[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    sl[u] = (j0 + u >= n) ? kOwnBit : (mat ? (int)M.arena[at + j0 + u] : A.slots[at + j0 + u]);
#pragma unroll
                for (int u = 0; u < 8; ++u) w[u] = sl[u] >= 0 ? zone_vin<kF32>(A, sl[u]) : make_double2(0.0, 0.0);
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (sl[u] >= 0) zone_vout<kF32>(A, sl[u], make_double2(__dadd_rn(w[u].x, ux), __dadd_rn(w[u].y, uy)));
            }
        }
    }
    __syncwarp();
    if (wantDiag) {
        for (int o = 16; o > 0; o >>= 1) {
            dgUx2 = __dadd_rn(dgUx2, __shfl_xor_sync(0xffffffffu, dgUx2, o));
            dgUy2 = __dadd_rn(dgUy2, __shfl_xor_sync(0xffffffffu, dgUy2, o));
            dgPx2 = __dadd_rn(dgPx2, __shfl_xor_sync(0xffffffffu, dgPx2, o));
            dgPy2 = __dadd_rn(dgPy2, __shfl_xor_sync(0xffffffffu, dgPy2, o));
            dgNPx += __shfl_xor_sync(0xffffffffu, dgNPx, o);
            dgNPy += __shfl_xor_sync(0xffffffffu, dgNPy, o);
        }
        if (lane == 0) {
            double* d = A.zoneDiag + 8 * (size_t)z;
            d[0] = dgUx2; d[1] = dgUy2; d[2] = dgPx2; d[3] = (double)dgNPx; d[4] = dgPy2; d[5] = (double)dgNPy;
            d[6] = (double)nHighAll; d[7] = (double)nLowAll;
        }
        __syncwarp();
    }
    // zone stats[4], stats[5] (src/zone_pass.cpp:911-922): the sum of positive dU2 in ascending
    // cell order (adding the zeros changes nothing) and the maximum of their roots (the root of the
    // maximum: a correctly rounded root is monotone).
    double acc = 0.0, top = 0.0;
    int cntDU = 0;
    for (int l = 0; l < S.nl; ++l) {
        const double d2 = du2[l];
        if (d2 > 0.0) {
            acc = __dadd_rn(acc, d2);
            top = smax(top, d2);
            ++cntDU;
        }
    }
    if (kSerial) serial_finish(S, A, p);
    if (lane == 0) {
        A.zoneCorr[z] = make_double2((cntDU > 0) ? sqrt(__ddiv_rn(acc, (double)cntDU)) : 0.0, sqrt(top));
        A.zoneMoved[z] = make_int2(S.movedDense, S.movedSparse);
    }
    return true;
}

// Returns false if the zone must be re-run on the overflow path.
template <bool kSerial, typename I, bool kF32 = false>
__device__ bool zone_body(const ZoneArgs& A, int z, char* mem, int maxCells, int winCap, int arenaCap, int nsmCap) {
    ZoneState<I, kF32> S;
    if (!zone_setup<kSerial>(S, A, z, mem, maxCells, winCap, arenaCap, nsmCap)) return false;
    int nHighAll = 0, nLowAll = 0;  // dense cells over the passes, sparse cells (stats[0], stats[1])
    for (int pass = 0; pass < A.P.maxPasses && !S.failed && !S.fatal; ++pass) nHighAll += zone_dense_pass(S);
    if (!S.failed && !S.fatal) nLowAll = zone_sparse(S);
    return zone_finish<kSerial>(S, A, z, nHighAll, nLowAll);
}

// kF32: the FP32 precision form's state (A.in32, A.out32)
template <bool kF32>
__global__ void __launch_bounds__(32, 20) k_zone_pass(ZoneArgs A) {
    extern __shared__ __align__(16) char smem[];
    if ((int)blockIdx.x >= A.nZones) return;
    const int z = A.order ? A.order[blockIdx.x] : (int)blockIdx.x;
    if (!zone_body<false, uint16_t, kF32>(A, z, smem, A.maxCells, A.winCap, A.arenaCap, A.nsmCap) && (threadIdx.x & 31) == 0)
        A.overflow[atomicAdd(A.nOverflow, 1)] = z;
}

// Phase-synchronous zone pass: kW zones per block, consecutive entries of the launch order
// (heaviest first, so the zones of a block cost about the same), run in step with a block
// barrier after the set-up, after each dense pass and after the sparse phase. The resident
// warps of an SM then execute the same phase's code (the body is too large for the
// instruction cache as a whole). Each warp carves its working set at perWarp bytes.
template <bool kF32, int kW>
__device__ __forceinline__ void zone_sync_block(int blk, const ZoneArgs& A, int perWarp, char* smem) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = blk * kW + w;
    const bool have = slot < A.nZones;
    const int z = have ? (A.order ? A.order[slot] : slot) : 0;
    ZoneState<uint16_t, kF32> S;
    S.failed = S.fatal = false;
    const bool ok = have && zone_setup<false>(S, A, z, smem + (size_t)perWarp * w, A.maxCells, A.winCap, A.arenaCap,
                                               A.nsmCap);
    int nHighAll = 0, nLowAll = 0;
    __syncthreads();
    for (int pass = 0; pass < A.P.maxPasses; ++pass) {
        if (ok && !S.failed && !S.fatal) nHighAll += zone_dense_pass(S);
        __syncthreads();
    }
    if (ok && !S.failed && !S.fatal) nLowAll = zone_sparse(S);
    __syncthreads();
    if (have && !(ok && zone_finish<false>(S, A, z, nHighAll, nLowAll)) && lane == 0)
        A.overflow[atomicAdd(A.nOverflow, 1)] = z;
}
template <bool kF32, int kW>
__global__ void __launch_bounds__(32 * kW) k_zone_pass_sync(ZoneArgs A, int perWarp) {
    extern __shared__ __align__(16) char smem[];
    zone_sync_block<kF32, kW>((int)blockIdx.x, A, perWarp, smem);
}

// The replica r with offs[r] <= block < offs[r + 1] (offs ascending; -1 past the end), its arguments
// copied to smem by the whole block.
__device__ __forceinline__ int stage_zone_args(const ZoneArgs* __restrict__ args, const int* __restrict__ offs, int nRep,
                                               char* smem) {
    const int b = (int)blockIdx.x;
    if (nRep <= 0 || b >= offs[nRep]) return -1;
    int lo = 0, hi = nRep - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (offs[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    static_assert(sizeof(ZoneArgs) % 8 == 0, "ZoneArgs is copied in 8-byte words");
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(args + lo);
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(smem);
    for (int i = (int)threadIdx.x; i < (int)(sizeof(ZoneArgs) / 8); i += (int)blockDim.x) dst[i] = src[i];
    __syncthreads();
    return lo;
}

// The zone pass of several replicas in one launch, one zone per block: the zone at launch position
// b - offs[r] of replica r.
template <bool kF32>
__global__ void __launch_bounds__(32, 20) k_zone_pass_batch(const ZoneArgs* __restrict__ args, const int* __restrict__ offs,
                                                            int nRep) {
    extern __shared__ __align__(16) char smem[];
    const int r = stage_zone_args(args, offs, nRep, smem);
    if (r < 0) return;
    const ZoneArgs& A = *reinterpret_cast<const ZoneArgs*>(smem);
    const int local = (int)blockIdx.x - offs[r];
    const int z = A.order ? A.order[local] : local;
    if (!zone_body<false, uint16_t, kF32>(A, z, smem + kZoneArgsSmem, A.maxCells, A.winCap, A.arenaCap, A.nsmCap) &&
        (threadIdx.x & 31) == 0)
        A.overflow[atomicAdd(A.nOverflow, 1)] = z;
}

// kF64ZoneWarps zones of one replica per block, in step; dynamic shared memory: the arguments, then
// the zones' working sets at perWarp bytes (at least every replica's own)
__global__ void __launch_bounds__(32 * kF64ZoneWarps) k_f64_zone_sync(const ZoneArgs* __restrict__ args, const int* __restrict__ offs, int n,
                                                                      int perWarp) {
    extern __shared__ __align__(16) char smem[];
    const int r = stage_zone_args(args, offs, n, smem);
    if (r < 0) return;
    const ZoneArgs& A = *reinterpret_cast<const ZoneArgs*>(smem);
    zone_sync_block<false, kF64ZoneWarps>((int)blockIdx.x - offs[r], A, perWarp, smem + kZoneArgsSmem);
}

// pass metrics as in k_zone_metrics, by one warp (fixed order: lane stride, then a shuffle tree)
__device__ void zone_metrics_warp(const int2* __restrict__ moved, const double2* __restrict__ corr, int nZones,
                                  double* __restrict__ out) {
    const int t = threadIdx.x & 31;
    double acc = 0.0, mx = 0.0;
    long long d = 0, s = 0;
    int c = 0;
    for (int z = t; z < nZones; z += 32) {
        const double2 q = __ldcg(corr + z);
        const int2 m = __ldcg(moved + z);
        if (q.x > 0.0) {
            acc = __dadd_rn(acc, __dmul_rn(q.x, q.x));
            ++c;
        }
        mx = smax(mx, q.y);
        d += m.x;
        s += m.y;
    }
    for (int o = 16; o > 0; o >>= 1) {
        acc = __dadd_rn(acc, __shfl_down_sync(0xffffffffu, acc, o));
        mx = smax(mx, __shfl_down_sync(0xffffffffu, mx, o));
        d += __shfl_down_sync(0xffffffffu, d, o);
        s += __shfl_down_sync(0xffffffffu, s, o);
        c += __shfl_down_sync(0xffffffffu, c, o);
    }
    if (t == 0) {
        out[0] = (double)d;
        out[1] = (double)s;
        out[2] = (c > 0) ? sqrt(__ddiv_rn(acc, (double)c)) : 0.0;
        out[3] = mx;
    }
}

// zones that did not fit the shared-memory working set, re-run from their seed with a
// global-memory working set per block (deterministic: identical decisions and writes)
// The last of its blocks to finish then computes the pass metrics (zone_metrics_warp) and
// resets the overflow and block counters for the next pass.
// block blk of nblk: the overflow zones blk, blk + nblk, ...; the last block to finish
// computes the pass metrics (when metricsOut is given) and resets the counters
template <bool kF32>
__device__ __forceinline__ void zone_overflow_block(const ZoneArgs& A, char* gmem, size_t perBlock, int* blocksDone,
                                                    double* metricsOut, int blk, int nblk) {
    const int nov = *A.nOverflow;
    for (int i = blk; i < nov; i += nblk)
        if (!zone_body<false, int, kF32>(A, A.overflow[i], gmem + perBlock * blk, A.maxCells, A.winCap, A.arenaCap,
                                         A.nsmCap) &&
            (threadIdx.x & 31) == 0)
            raise_error(A.st, kErrZoneCapacity, A.overflow[i]);
    __syncwarp();
    int last = 0;
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(blocksDone, 1) == nblk - 1;
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    if (!last) return;
    __threadfence();
    if (metricsOut) zone_metrics_warp(A.zoneMoved, A.zoneCorr, A.nZones, metricsOut);
    if (threadIdx.x == 0) {
        *blocksDone = 0;
        *A.nOverflow = 0;
    }
}

template <bool kF32>
__global__ void __launch_bounds__(32) k_zone_overflow(ZoneArgs A, char* gmem, size_t perBlock, int* blocksDone,
                                                      double* metricsOut) {
    zone_overflow_block<kF32>(A, gmem, perBlock, blocksDone, metricsOut, (int)blockIdx.x, (int)gridDim.x);
}

__global__ void __launch_bounds__(32) k_zone_overflow_batch(const OverflowJob* __restrict__ jobs, int perJob) {
    const OverflowJob& J = jobs[blockIdx.x / perJob];
    zone_overflow_block<false>(J.A, J.gmem, J.perBlock, J.blocksDone, J.metricsOut, (int)(blockIdx.x % perJob), perJob);
}

// run_zone_pass (src/zone_pass.cpp:1096-1163): one warp runs the zones in id order on the
// live state; a zone that outgrows the shared-memory working set is re-run at once with the
// global one (B's capacities), which is safe since a failed zone has published nothing.
__global__ void __launch_bounds__(32) k_zone_serial(ZoneArgs A, ZoneArgs B, char* gmem) {
    extern __shared__ __align__(16) char smem[];
    for (int z = 0; z < A.nZones; ++z) {
        bool ok = zone_body<true, uint16_t>(A, z, smem, A.maxCells, A.winCap, A.arenaCap, A.nsmCap);
        if (!ok) ok = zone_body<true, int>(B, z, gmem, B.maxCells, B.winCap, B.arenaCap, B.nsmCap);
        if (!ok) {
            if ((threadIdx.x & 31) == 0) raise_error(A.st, kErrZoneCapacity, z);
            return;
        }
        __syncwarp();
    }
}

}  // namespace mpcd_dev
