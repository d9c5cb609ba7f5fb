// smc_coop.cuh -- the SMC step as one kernel: the exact sequential fold, the
// weight normalisation, the replication counts and the parent indices as
// device phases of a cooperative grid whose CTAs each own one tile of
// consecutive particles (one CTA alone for a small cloud).
//
// What bounds a step of a cloud that fits the chip at once is neither memory
// nor arithmetic but the chain of dependent kernels: the multi-kernel step
// (weight.cu, fold.cu, resample.cu) is about 25 launches of 3-15 us for a few
// microseconds of work each.  Here a tile stays with its CTA (registers and
// shared memory) and a launch boundary becomes an exchange: every CTA
// publishes a few words and reads every other CTA's.  What one thread did
// between two kernels (the walk over a fold's windows) every CTA does for
// itself.  The arithmetic and its order are those of the multi-kernel step, so
// the results are the same bits.
//
// A single call runs its code once, so instruction fetch is a large part of it:
// a tile's values and their grid increments live in shared memory and every
// loop over a thread's elements is rolled (with the loops unrolled and the
// values in registers the weight call of 1001 particles took 56 us).
//
// Tiles: THR threads of PER consecutive elements each, at most one tile per SM:
// the smallest tile that fits the cloud on 148 SMs, in steps of 1024 elements up to
// 8192 (one CTA alone up to 1024 elements, a cluster up to 8192), since more CTAs
// shorten every phase and equal ones wait least for each other.  On a B200, a step
// of the plain systematic and multinomial filters (T = 20):
//   particles   multi-kernel     512 x 2, 1024 x 4, 7, 8   every 1024 elements
//   151,553     157 / 167 us     67 / 110 us (38 tiles)    54 /  92 us (74 tiles)
//   300,000     162 / 174        70 / 117                  58 /  99
//   380,000     165 / 179        71 / 119                  67 / 105
//   500,000     174 / 185        73 / 119                  73 / 120 (the same)
//   606,209     183 / 199        91 / 173 (85 tiles)       81 / 142 (119 tiles)
//   800,000     194 / 214        90 / 175                  84 / 156
//   1,048,576   214 / 232        93 / 177                  92 / 178 (the same)
// (2^20 particles on 256 tiles of 4096, two on most SMs: 97 us a systematic step.)
// Multinomial counts of 606,209 particles alone: 147 us multi-kernel, 144 to 152 on
// 85 tiles, 118 on 119.  Clouds of more tiles than SMs take the multi-kernel step.
#pragma once

#include <cstdint>

#include "block_scan.cuh"
#include "common.cuh"
#include "crmath.cuh"
#include "fold.cuh"
#include "fold_classify.cuh"
#include "transforms.cuh"

namespace mckl_b200 {
namespace coop {

constexpr int kMaxWarps = 32;
constexpr unsigned kMaxTiles = 148;   // one CTA per SM
constexpr unsigned kMaxTile = 8192;   // elements
constexpr unsigned kTileWin = 256;    // windows a tile can list
constexpr unsigned kWinSets = 2;      // sets of window lists: folds take them in turn (fold_grid)
constexpr unsigned kWin = 512;        // windows of a fold the walk takes
constexpr unsigned kSegWin = 64;      // windows of one short fold (seg_fold)
constexpr unsigned kMaxCluster = 8;   // tiles that exchange through distributed shared memory
constexpr int kMaxVals = 2;           // words a tile publishes in one exchange
constexpr int kSpinLimit = 1 << 22;   // polls (each an L2 round trip) before a wait gives up

struct Window {
    double x;       // value
    long long P;    // run increments before it, within the tile
    long long e;    // binade of the run before it
};

// Device working memory of one launch (coop_scratch_bytes).
struct Global {
    ulonglong2 *slots;  // [2][kMaxVals][kMaxTiles]: {value, epoch}
    ulonglong2 *chain;  // [kMaxTiles]: {tile's last value, epoch} of the event-loop fold
    Window *win;        // [kWinSets][tiles][kTileWin]
    double *dots;       // [ceil(N / 1024)] chunk dot products
    int *err;           // set when a wait gave up
};

struct Shared {
    unsigned long long scr[2][2][kMaxWarps];  // warp totals of the scans, alternating
    double tpre, tpmax, total;
    int elast, elast_all, ok;
    uint32_t pw[kMaxTiles + 1];            // windows (or empty slots) before each tile
    long long pq[kMaxTiles + 1];           // run increments (or surplus copies) before each tile
    union {
        struct {
            int we[kWin];                  // the fold's windows in order
            double wx[kWin], wS[kWin];
            long long wP[kWin];
            // short folds: up to eight segments
            int ge[8][kSegWin];
            double gx[8][kSegWin];
            long long gP[8][kSegWin];
        };
        uint4 words[kMaxTile / 4 + 4];     // the filter's noise: a tile's Philox blocks
        uint32_t empties[kMaxTile];        // a tile's empty slots in order
    };
    unsigned long long xs[2][kMaxVals][kMaxCluster];  // exchange slots of a cluster
    long long gq[8];
    unsigned gw[8];
    int gel[8];
    double gtot[8], dots[8];
};

struct Ctx {
    Global g;
    Shared *sh;
    uint32_t T, tile;
    unsigned long long epoch, chain_epoch;
    unsigned folds;  // fold_grid calls so far, the same in every CTA
    unsigned flip;
    bool cluster;  // the T CTAs are one cluster
};

// Element o of a tile in shared memory: one pad word per 16, so that the
// blocked accesses (thread t, elements t PER ..) spread over the banks.
__device__ __forceinline__ uint32_t pad(uint32_t o)
{
    return o + (o >> 4);
}

constexpr uint32_t padded(uint32_t n)
{
    return n + n / 16;
}

__device__ __forceinline__ unsigned long long dbits(double v)
{
    return static_cast<unsigned long long>(__double_as_longlong(v));
}

__device__ __forceinline__ double bitsd(unsigned long long v)
{
    return __longlong_as_double(static_cast<long long>(v));
}

__device__ __forceinline__ void publish(ulonglong2 *p, unsigned long long v, unsigned long long epoch)
{
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p), "l"(v),
                 "l"(epoch)
                 : "memory");
}

// Wait for `epoch` in the NV slots s, s + kMaxTiles, .. and return their values;
// false past the limit.
template <int NV>
__device__ __forceinline__ bool await(ulonglong2 *s, unsigned long long epoch, unsigned long long (&v)[NV])
{
    for (int k = 0; k < kSpinLimit; ++k) {
        unsigned long long e[NV];
        bool all = true;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                         : "=l"(v[q]), "=l"(e[q])
                         : "l"(s + q * kMaxTiles)
                         : "memory");
        }
#pragma unroll
        for (int q = 0; q < NV; ++q) all = all && e[q] == epoch;
        if (all) return true;
    }
    return false;
}

// Store v in word `p` of the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ void store_remote(unsigned long long *p, uint32_t rank, unsigned long long v)
{
    uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p)), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(r), "l"(v) : "memory");
}

// All-gather of NV words per tile: on entry every thread holds this tile's, on
// return thread i < T holds tile i's (0 beyond).  With `data`, what any thread
// of any CTA wrote to global memory before is visible to every thread after
// (read it with __ldcg).  Up to kMaxCluster tiles are one cluster: each CTA
// stores its words into every other's shared memory and the cluster's barrier
// (release, acquire) does the rest; more tiles publish {value, epoch} pairs in
// global memory and read each other's until the epoch appears.  Two slot sets
// alternate: a CTA that publishes exchange n + 2 has seen every CTA publish
// n + 1, which each did after it had read n.  False (in every thread of the
// CTA) when a wait gave up; the caller returns from the kernel.
template <int NV>
__device__ __forceinline__ bool exchange(Ctx &c, unsigned long long (&v)[NV], bool data)
{
    static_assert(NV <= kMaxVals, "slots per tile");
    if (c.T == 1) {
        __syncthreads();
        if (threadIdx.x)
            for (int q = 0; q < NV; ++q) v[q] = 0;
        return true;
    }
    ++c.epoch;
    const unsigned set = c.epoch & 1;
    if (c.cluster) {
        if (threadIdx.x < c.T)
            for (int q = 0; q < NV; ++q) store_remote(&c.sh->xs[set][q][c.tile], threadIdx.x, v[q]);
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] = threadIdx.x < c.T ? c.sh->xs[set][q][threadIdx.x] : 0;
        return true;
    }
    ulonglong2 *s = c.g.slots + set * (kMaxVals * kMaxTiles);
    if (data) __syncthreads();
    if (threadIdx.x == 0) {
        if (data) __threadfence();
#pragma unroll
        for (int q = 0; q < NV; ++q) publish(s + q * kMaxTiles + c.tile, v[q], c.epoch);
    }
    bool ok = true;
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = 0;
    if (threadIdx.x < c.T) {
        ok = await<NV>(s + threadIdx.x, c.epoch, v);
        if (data) __threadfence();
        if (!ok) atomicExch(c.g.err, 1);
    }
    return !__syncthreads_or(!ok);
}

// ---- scans over the CTA, one barrier each (every warp scans the warp totals;
// two scratch sets alternate, so a set is rewritten only behind the other's
// barrier)

// Exclusive sums (formed without a subtraction) and exclusive maxima of
// nonnegative values, and the totals.
template <int THR>
__device__ __forceinline__ void scan_sum_max(Ctx &c, double v, double m, double &es, double &em, double &ts,
    double &tm)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double is = v, im = m;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double us = __shfl_up_sync(0xffffffffu, is, o), um = __shfl_up_sync(0xffffffffu, im, o);
        if (lane >= o) {
            is += us;
            im = fmax(im, um);
        }
    }
    double ps = __shfl_up_sync(0xffffffffu, is, 1), pm = __shfl_up_sync(0xffffffffu, im, 1);
    if (lane == 0) ps = pm = 0.0;
    c.flip ^= 1;
    unsigned long long(*buf)[kMaxWarps] = c.sh->scr[c.flip];
    if (lane == 31) {
        buf[0][warp] = dbits(is);
        buf[1][warp] = dbits(im);
    }
    __syncthreads();
    double ws = lane < THR / 32 ? bitsd(buf[0][lane]) : 0.0, wm = lane < THR / 32 ? bitsd(buf[1][lane]) : 0.0;
#pragma unroll
    for (int o = 1; o < THR / 32; o <<= 1) {
        const double us = __shfl_up_sync(0xffffffffu, ws, o), um = __shfl_up_sync(0xffffffffu, wm, o);
        if (lane >= o) {
            ws += us;
            wm = fmax(wm, um);
        }
    }
    const double bs = __shfl_sync(0xffffffffu, ws, warp > 0 ? warp - 1 : 0);
    const double bm = __shfl_sync(0xffffffffu, wm, warp > 0 ? warp - 1 : 0);
    ts = __shfl_sync(0xffffffffu, ws, THR / 32 - 1);
    tm = __shfl_sync(0xffffffffu, wm, THR / 32 - 1);
    es = warp > 0 ? bs + ps : ps;
    em = warp > 0 ? fmax(bm, pm) : pm;
}

// Maximum over the warp of nonnegative doubles (their bits order as unsigned
// integers: the high words first, then the low words among the largest).
__device__ __forceinline__ double warp_max_nonneg(double v)
{
    const unsigned hi = static_cast<unsigned>(__double2hiint(v)), lo = static_cast<unsigned>(__double2loint(v));
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    return __hiloint2double(static_cast<int>(mh), static_cast<int>(ml));
}

// Exclusive sums of nonnegative values (formed without a subtraction) and the
// total; em: the maximum over the warps before this one, tm over all.
template <int THR>
__device__ __forceinline__ void scan_sum(Ctx &c, double v, double m, double &es, double &em, double &ts, double &tm)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double is = warp_inclusive_sum(v), wmx = warp_max_nonneg(m);
    double ps = __shfl_up_sync(0xffffffffu, is, 1);
    if (lane == 0) ps = 0.0;
    c.flip ^= 1;
    unsigned long long(*buf)[kMaxWarps] = c.sh->scr[c.flip];
    if (lane == 31) {
        buf[0][warp] = dbits(is);
        buf[1][warp] = dbits(wmx);
    }
    __syncthreads();
    double ws = lane < THR / 32 ? bitsd(buf[0][lane]) : 0.0;
    const double wm = lane < THR / 32 ? bitsd(buf[1][lane]) : 0.0;
#pragma unroll
    for (int o = 1; o < THR / 32; o <<= 1) {
        const double us = __shfl_up_sync(0xffffffffu, ws, o);
        if (lane >= o) ws += us;
    }
    const double bs = __shfl_sync(0xffffffffu, ws, warp > 0 ? warp - 1 : 0);
    ts = __shfl_sync(0xffffffffu, ws, THR / 32 - 1);
    tm = warp_max_nonneg(wm);
    em = warp_max_nonneg(lane < warp ? wm : 0.0);
    es = warp > 0 ? bs + ps : ps;
}

// Exclusive sums of two 64-bit integers, and the totals.
template <int THR>
__device__ __forceinline__ void scan_two(Ctx &c, long long a, long long b, long long &ea, long long &eb,
    long long &ta, long long &tb)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long ia = warp_inclusive_sum(a), ib = warp_inclusive_sum(b);
    c.flip ^= 1;
    unsigned long long(*buf)[kMaxWarps] = c.sh->scr[c.flip];
    if (lane == 31) {
        buf[0][warp] = static_cast<unsigned long long>(ia);
        buf[1][warp] = static_cast<unsigned long long>(ib);
    }
    __syncthreads();
    long long wa = lane < THR / 32 ? static_cast<long long>(buf[0][lane]) : 0;
    long long wb = lane < THR / 32 ? static_cast<long long>(buf[1][lane]) : 0;
    wa = warp_inclusive_sum(wa);
    wb = warp_inclusive_sum(wb);
    const long long ba = __shfl_sync(0xffffffffu, wa, warp > 0 ? warp - 1 : 0);
    const long long bb = __shfl_sync(0xffffffffu, wb, warp > 0 ? warp - 1 : 0);
    ta = __shfl_sync(0xffffffffu, wa, THR / 32 - 1);
    tb = __shfl_sync(0xffffffffu, wb, THR / 32 - 1);
    ea = ia - a + (warp > 0 ? ba : 0);
    eb = ib - b + (warp > 0 ? bb : 0);
}

template <int THR>
__device__ __forceinline__ double max_all(Ctx &c, double v)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_max(v);
    c.flip ^= 1;
    unsigned long long(*buf)[kMaxWarps] = c.sh->scr[c.flip];
    if (lane == 0) buf[0][warp] = dbits(v);
    __syncthreads();
    return warp_max(bitsd(buf[0][lane & (THR / 32 - 1)]));
}

template <int THR>
__device__ __forceinline__ uint32_t min_all(Ctx &c, uint32_t v)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = __reduce_min_sync(0xffffffffu, v);
    c.flip ^= 1;
    unsigned long long(*buf)[kMaxWarps] = c.sh->scr[c.flip];
    if (lane == 0) buf[0][warp] = v;
    __syncthreads();
    return __reduce_min_sync(0xffffffffu, static_cast<uint32_t>(buf[0][lane & (THR / 32 - 1)]));
}

// ---- the walk over a fold's windows (fold.cuh): the run before a window is
// one integer step on its binade's grid, the window the reference's own add.
// Within a binade a step of u q is a step of q in the double's own bits, and a
// step past the binade (or from another one) shows in the exponent field: then
// false.  Q: the run increments of the whole fold; elast: the last run's binade.
__device__ __forceinline__ bool walk_windows(unsigned W, const double *wx, const long long *wP, const int *we,
    double *wS, long long Q, int elast, double *total)
{
    long long sb = 0, p = 0;  // the sum's bits, the run increments it includes
    bool ok = true;
#pragma unroll 4
    for (unsigned k = 0; k < W; ++k) {
        const long long P = wP[k], e = we[k];
        const bool run = P != p, in = (sb >> 52) == e;
        sb += P - p;
        ok = ok && (!run || (in && (sb >> 52) == e));
        const double s = __dadd_rn(__longlong_as_double(sb), wx[k]);
        if (wS) wS[k] = s;
        sb = __double_as_longlong(s);
        p = P;
    }
    if (Q != p) {  // the run after the last window
        const bool in = (sb >> 52) == elast;
        sb += Q - p;
        ok = ok && in && (sb >> 52) == elast;
    }
    *total = __longlong_as_double(sb);
    return ok;
}

// grid_increment (fold.cuh) in floating point for the binades whose ulp has a
// reciprocal: x / u is exact, adding 1.5 2^52 rounds it to an integer (ties to
// even) and the remainder is exact.  An increment of 2^51 or more is an event
// too (the walk's own add is always right).
__device__ __forceinline__ long long increment(double x, int e, bool &event)
{
    if (e < 52 || e > 2046) return grid_increment(x, e, event);
    const double y = __dmul_rn(x, __longlong_as_double(static_cast<long long>(2098 - e) << 52));
    event = !(y < 0x1p51);
    const double t = __dadd_rn(y, 0x1.8p52);
    const double r = __dsub_rn(y, __dsub_rn(t, 0x1.8p52));
    if (r == 0.5 || r == -0.5) event = true;
    return __double_as_longlong(t) - 0x4338000000000000ll;
}

// Element k of the calling thread in a padded tile array.
template <int PER>
__device__ __forceinline__ uint32_t at(int k)
{
    return pad(threadIdx.x * PER + k);
}

// fold_classify.cuh's classification with rolled loops: the thread's PER
// values get(k) (0 past n), its increments (or, for a window, the binade
// before it) to s_q, the window bits to *win and the sum of the increments to
// *qs; *elast receives the binade of element n - 1's run (-1: a window) from
// the thread that holds it.
template <int PER, class Get>
__device__ __forceinline__ void classify_tile(const Get &get, long long *s_q, uint64_t i0, uint64_t n, uint64_t T,
    double Abefore, double own, double Mbefore, unsigned *win, long long *qs, int *elast)
{
    int fast = -1;  // the binade of every partial sum of the thread, when certain
    {
        const double Aend = __dadd_rn(Abefore, own);
        const double m = 2.0 * static_cast<double>(i0 + PER) + 2.0 * static_cast<double>(T) + 160.0;
        const double low = __dsub_rn(Abefore, m * ulp_of(Abefore)), hi = __dadd_rn(Aend, m * ulp_of(Aend));
        const auto certain = [hi](double lo) {
            const int e = biased_exp(lo);
            return lo > 0.0 && e != 0x7ff && biased_exp(hi) == e ? e : -1;
        };
        fast = certain(fmax(low, Mbefore));
        if (__any_sync(0xffffffffu, fast < 0)) {
            // the largest term of the warp's threads before this one, too
            const int lane = threadIdx.x & 31;
            double mx = 0.0;
#pragma unroll 1
            for (int k = 0; k < PER; ++k)
                if (i0 + k < n) mx = fmax(mx, get(k));
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double u = __shfl_up_sync(0xffffffffu, mx, o);
                if (lane >= o) mx = fmax(mx, u);
            }
            mx = __shfl_up_sync(0xffffffffu, mx, 1);
            if (lane > 0) Mbefore = fmax(Mbefore, mx);
            fast = certain(fmax(low, Mbefore));
        }
    }
    // A warp whose threads are all certain of their binades, away from the end
    // of the array: the increments alone.  An event sends the warp through the
    // loop below.
    if (__all_sync(0xffffffffu, fast >= 52 && fast <= 2046 && i0 + PER < n)) {
        const double sc = __longlong_as_double(static_cast<long long>(2098 - fast) << 52);
        long long sum = 0;
        bool ev = false;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const double y = __dmul_rn(get(k), sc);
            const double t = __dadd_rn(y, 0x1.8p52);
            const double r = __dsub_rn(y, __dsub_rn(t, 0x1.8p52));
            ev = ev || !(y < 0x1p51) || fabs(r) == 0.5;
            const long long q = __double_as_longlong(t) - 0x4338000000000000ll;
            sum += q;
            s_q[at<PER>(k)] = q;
        }
        if (!__any_sync(0xffffffffu, ev)) {
            *win = 0;
            *qs = sum;
            return;
        }
    }
    int ep = fast;
    if (fast < 0) ep = i0 == 0 ? 0 : certain_binade(Abefore, i0 - 1, T, Mbefore);
    double A = Abefore, M = Mbefore;
    unsigned w = 0;
    long long sum = 0;
#pragma unroll 1
    for (int k = 0; k < PER; ++k) {
        const uint64_t j = i0 + k;
        long long q = 0;
        bool ev = false;
        if (j < n) {
            const double x = get(k);
            int e = fast, en = fast;
            if (fast < 0 && x != 0.0) {
                A = __dadd_rn(A, x);
                M = fmax(M, x);
                en = certain_binade(A, j, T, M);
                e = en >= 0 && en == ep ? en : -1;
            }
            // a zero term leaves the sum unchanged: it keeps the binade before
            // it, certain or not, and is never a window
            if (x != 0.0) {
                ev = true;
                if (e >= 0) q = increment(x, e, ev);
                if (ev) {
                    q = ep;
                    w |= 1u << k;
                } else {
                    sum += q;
                }
            }
            if (j == n - 1) *elast = ev ? -1 : ep;
            if (x != 0.0) ep = en;
        }
        s_q[at<PER>(k)] = q;
    }
    *win = w;
    *qs = sum;
}

// ---- the event-loop fold of one tile (fold.cuh), from the value s before it:
// with PREFIX every partial sum replaces its value in s_v; returns the last.
// len elements of the tile exist.
template <int THR, int PER, bool PREFIX>
__device__ __noinline__ double tile_exact(Ctx &c, double *s_v, long long *s_q, uint32_t len, double s)
{
    constexpr uint32_t kStretch = 256;
    const uint32_t j0 = threadIdx.x * PER;
    uint32_t cur = 0;
    int rounds = 0;
    while (cur < len) {
        if (rounds >= 2 || s == 0.0) {
            // dense events, or nothing accumulated yet: a stretch one at a time
            const uint32_t end = min(len, cur + kStretch);
            if (threadIdx.x == 0) {
                double a = s;
                for (uint32_t j = cur; j < end; ++j) {
                    a = __dadd_rn(a, s_v[pad(j)]);
                    if (PREFIX) s_v[pad(j)] = a;
                }
                c.sh->total = a;
            }
            __syncthreads();
            s = c.sh->total;
            __syncthreads();
            cur = end;
            rounds = 0;
            continue;
        }
        ++rounds;
        const int eb = biased_exp(s);
        const long long K = grid_count(s), top = grid_top(eb);
        long long own = 0;
        unsigned ev = 0;
#pragma unroll 1
        for (int k = 0; k < PER; ++k) {
            long long q = 0;
            if (j0 + k >= cur && j0 + k < len) {
                bool e;
                q = grid_increment(s_v[at<PER>(k)], eb, e);
                if (e) ev |= 1u << k;
            }
            s_q[at<PER>(k)] = q;
            own += q;
        }
        long long before, dummy, t0, t1;
        scan_two<THR>(c, own, 0, before, dummy, t0, t1);
        uint32_t first = 0xffffffffu;
        long long run = before;
#pragma unroll 1
        for (int k = 0; k < PER; ++k) {
            run += s_q[at<PER>(k)];
            if (j0 + k >= cur && j0 + k < len && first == 0xffffffffu && (((ev >> k) & 1u) || K + run >= top))
                first = j0 + k;
        }
        const uint32_t cpos = min_all<THR>(c, first);
        run = before;
#pragma unroll 1
        for (int k = 0; k < PER; ++k) {
            const uint32_t j = j0 + k;
            const long long q = s_q[at<PER>(k)];
            run += q;
            if (j < cur || j >= len || j > cpos) continue;
            double v;
            if (j < cpos) {
                v = from_grid(K + run, eb);
            } else {
                const double prev = cpos == cur ? s : from_grid(K + run - q, eb);
                v = __dadd_rn(prev, s_v[at<PER>(k)]);
            }
            if (PREFIX) s_v[at<PER>(k)] = v;
            if (j == cpos || j + 1 == len) c.sh->total = v;
        }
        __syncthreads();
        s = c.sh->total;
        __syncthreads();
        if (cpos >= len) break;
        cur = cpos + 1;
    }
    return s;
}

// The event-loop fold of the whole array: the tiles in order, each from its
// predecessor's last value; with PREFIX the partial sums replace the values.
// Taken when the windows do not fit their lists (ties everywhere) or a run left
// its binade.
template <int THR, int PER, bool PREFIX>
__device__ __noinline__ bool fold_chain(Ctx &c, double *s_v, long long *s_q, uint64_t n, double *total,
    double *before)
{
    ++c.chain_epoch;
    const uint64_t base = static_cast<uint64_t>(c.tile) * (THR * PER);
    const uint32_t len = base < n ? static_cast<uint32_t>(min(static_cast<uint64_t>(THR * PER), n - base)) : 0u;
    bool ok = true;
    if (threadIdx.x == 0) {
        unsigned long long b[1] = {0};
        if (c.tile > 0) ok = await<1>(c.g.chain + c.tile - 1, c.chain_epoch, b);
        c.sh->tpre = bitsd(b[0]);
    }
    if (!ok) atomicExch(c.g.err, 1);
    if (__syncthreads_or(!ok)) return false;
    const double s_in = c.sh->tpre;
    __syncthreads();
    double s = s_in;
    if (len) s = tile_exact<THR, PER, PREFIX>(c, s_v, s_q, len, s_in);
    if (c.T > 1) {
        if (threadIdx.x == 0) {
            publish(c.g.chain + c.tile, dbits(s), c.chain_epoch);
            unsigned long long b[1] = {0};
            ok = await<1>(c.g.chain + c.T - 1, c.chain_epoch, b);
            c.sh->tpre = bitsd(b[0]);
        }
        if (!ok) atomicExch(c.g.err, 1);
        if (__syncthreads_or(!ok)) return false;
        s = c.sh->tpre;
    }
    *total = s;
    if (PREFIX) {
        *before = threadIdx.x ? s_v[pad(threadIdx.x * PER - 1)] : s_in;
        __syncthreads();
    }
    return true;
}

// What the classification needs of a thread: the approximate sum of the
// elements before its own, its own sum, and a lower bound of the sum before it
// (the largest term of the warps and tiles before).
struct Approx {
    double A, own, M;
};

// The approximate sums of the values in s_v (0 past n).  False when a wait gave up.
template <int THR, int PER>
__device__ __forceinline__ bool fold_approx(Ctx &c, const double *s_v, Approx &ap)
{
    double own = 0.0, mx = 0.0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const double x = s_v[at<PER>(k)];
        own = __dadd_rn(own, x);
        mx = fmax(mx, x);
    }
    double ex, em, ts, tm, tpre = 0.0, tpm = 0.0;
    scan_sum<THR>(c, own, mx, ex, em, ts, tm);
    if (c.T > 1) {
        unsigned long long x[2] = {dbits(ts), dbits(tm)};
        if (!exchange(c, x, false)) return false;
        if (c.cluster) {
            const unsigned long long(*xs)[kMaxCluster] = c.sh->xs[c.epoch & 1];
            for (uint32_t t = 0; t < c.tile; ++t) {
                tpre += bitsd(xs[0][t]);
                tpm = fmax(tpm, bitsd(xs[1][t]));
            }
        } else {
            double e2, m2, t0, t1;
            scan_sum_max<THR>(c, bitsd(x[0]), bitsd(x[1]), e2, m2, t0, t1);
            if (threadIdx.x == c.tile) {
                c.sh->tpre = e2;
                c.sh->tpmax = m2;
            }
            __syncthreads();
            tpre = c.sh->tpre;
            tpm = c.sh->tpmax;
        }
    }
    ap.A = __dadd_rn(tpre, ex);
    ap.own = own;
    ap.M = fmax(tpm, em);
    return true;
}

// ---- the exact left fold of n values, from 0.  The tile's values are in s_v
// (0 past n), each written by its own thread; ap from fold_approx.  The last
// value goes to *total; with PREFIX every partial sum replaces its value in s_v
// and the one before the thread's first element goes to *before.  What was
// written to global memory before the call is visible after it (its exchange
// carries data).  s_q is overwritten.  False when a wait gave up.
//
// A tile writes its window list before the exchange and reads every tile's after
// it, and the next fold may follow with no exchange between (resample_phase with
// known sums).  So folds take two sets of lists in turn: a CTA that writes fold
// n + 2's list is behind the exchange of fold n + 1, which every CTA enters only
// after it has read the lists of fold n.  With one set a CTA that is ahead would
// rewrite its list while another still reads it.
template <int THR, int PER, bool PREFIX>
__device__ __noinline__ bool fold_grid(Ctx &c, double *s_v, long long *s_q, uint64_t n, const Approx ap,
    double *total, double *before)
{
    Shared *sh = c.sh;
    const uint64_t i0 = (static_cast<uint64_t>(c.tile) * THR + threadIdx.x) * PER;
    Window *lists = c.g.win + static_cast<size_t>(++c.folds % kWinSets) * c.T * kTileWin;
    if (threadIdx.x == 0) sh->elast = -1;
    __syncthreads();
    unsigned win;
    long long qs;
    classify_tile<PER>([s_v](int k) { return s_v[at<PER>(k)]; }, s_q, i0, n, c.T, ap.A, ap.own, ap.M, &win, &qs,
        &sh->elast);
    long long P, r, qtot, wtot;
    scan_two<THR>(c, qs, __popc(win), P, r, qtot, wtot);
    bool over = wtot > static_cast<long long>(c.T == 1 ? kWin : kTileWin);
    if (win && !over) {
        long long Pk = P;
        uint32_t rk = static_cast<uint32_t>(r);
#pragma unroll 1
        for (int k = 0; k < PER; ++k) {
            const long long q = s_q[at<PER>(k)];
            if ((win >> k) & 1u) {
                const double x = s_v[at<PER>(k)];
                if (c.T == 1) {
                    sh->we[rk] = static_cast<int>(q);
                    sh->wx[rk] = x;
                    sh->wP[rk] = Pk;
                } else {
                    lists[static_cast<size_t>(c.tile) * kTileWin + rk] = Window{x, Pk, q};
                }
                ++rk;
            } else {
                Pk += q;
            }
        }
    }
    unsigned W;
    long long Q;
    if (c.T == 1) {
        __syncthreads();
        W = static_cast<unsigned>(wtot);
        Q = qtot;
        if (threadIdx.x == 0) {
            sh->pq[0] = 0;
            sh->pw[0] = 0;
            sh->elast_all = sh->elast;
        }
    } else {
        unsigned long long x[2] = {static_cast<unsigned long long>(qtot),
            (static_cast<unsigned long long>(wtot) << 32) | static_cast<uint32_t>(sh->elast + 1)};
        if (!exchange(c, x, true)) return false;
        const long long wi = static_cast<long long>(x[1] >> 32);
        const int el = static_cast<int>(static_cast<uint32_t>(x[1])) - 1;
        long long eq = 0, ew = 0, tq = 0, tw = 0;
        if (c.cluster) {
            const unsigned long long(*xs)[kMaxCluster] = sh->xs[c.epoch & 1];
            for (uint32_t t = 0; t < c.T; ++t) {
                const long long q = static_cast<long long>(xs[0][t]), w = static_cast<long long>(xs[1][t] >> 32);
                if (t < threadIdx.x) {
                    eq += q;
                    ew += w;
                }
                tq += q;
                tw += w;
            }
        } else {
            scan_two<THR>(c, static_cast<long long>(x[0]), wi, eq, ew, tq, tw);
        }
        if (threadIdx.x < c.T) {
            sh->pq[threadIdx.x] = eq;
            sh->pw[threadIdx.x] = static_cast<uint32_t>(ew);
            // the tile that holds element n - 1 tells its run's binade
            if (threadIdx.x == (n - 1) / (THR * PER)) sh->elast_all = el;
        }
        over = __syncthreads_or(wi > static_cast<long long>(kTileWin)) || tw > static_cast<long long>(kWin);
        W = static_cast<unsigned>(tw);
        Q = tq;
        if (!over) {
            for (unsigned k = threadIdx.x; k < W; k += THR) {
                uint32_t lo = 0, hi = c.T;  // the last tile with pw <= k
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (sh->pw[mid] <= k) {
                        lo = mid;
                    } else {
                        hi = mid;
                    }
                }
                const Window *w = lists + static_cast<size_t>(lo) * kTileWin + (k - sh->pw[lo]);
                sh->wx[k] = __ldcg(&w->x);
                sh->wP[k] = sh->pq[lo] + __ldcg(&w->P);
                sh->we[k] = static_cast<int>(__ldcg(&w->e));
            }
        }
    }
    __syncthreads();
    if (!over && threadIdx.x == 0)
        sh->ok = walk_windows(W, sh->wx, sh->wP, sh->we, sh->wS, Q, sh->elast_all, &sh->total) ? 1 : 0;
    __syncthreads();
    // `over` and the walk's outcome come from the same data in every CTA
    if (over || !sh->ok) return fold_chain<THR, PER, PREFIX>(c, s_v, s_q, n, total, before);
    *total = sh->total;
    if constexpr (PREFIX) {
        P += sh->pq[c.tile];
        uint32_t rk = static_cast<uint32_t>(r) + sh->pw[c.tile];
        // the sum's bits: the last window's value plus the run increments since
        long long sb = rk > 0 ? __double_as_longlong(sh->wS[rk - 1]) + (P - sh->wP[rk - 1]) : P;
        *before = __longlong_as_double(sb);
#pragma unroll 2
        for (int k = 0; k < PER; ++k) {
            if ((win >> k) & 1u) {
                sb = __double_as_longlong(sh->wS[rk++]);
            } else {
                sb += s_q[at<PER>(k)];
            }
            s_v[at<PER>(k)] = __longlong_as_double(sb);
        }
        __syncthreads();  // the window lists are rewritten by the next fold
    }
    return true;
}

// ---- short exact folds inside the CTA, one per segment of SEGT threads: the
// fold of the segment's first `len` values get(k) (PER per thread, 0 beyond)
// into sh->gtot[segment].  again(segment, j): value j, for a segment whose
// windows do not fit their list.  s_q is overwritten.
template <int THR, int PER, int SEGT, class Get, class Again>
__device__ void seg_fold(Ctx &c, long long *s_q, uint32_t len, const Get &get, const Again &again)
{
    static_assert(THR / SEGT <= 8 && SEGT % 32 == 0, "segments");
    constexpr int SW = SEGT / 32;  // warps per segment
    Shared *sh = c.sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, seg = threadIdx.x / SEGT;
    const uint32_t i0 = (threadIdx.x % SEGT) * PER;
    double own = 0.0, mx = 0.0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const double x = i0 + k < len ? get(k) : 0.0;
        own = __dadd_rn(own, x);
        mx = fmax(mx, x);
    }
    if (i0 == 0) sh->gel[seg] = -1;
    const double is = warp_inclusive_sum(own), wmx = warp_max_nonneg(mx);
    double ps = __shfl_up_sync(0xffffffffu, is, 1);
    if (lane == 0) ps = 0.0;
    c.flip ^= 1;
    unsigned long long(*buf)[kMaxWarps] = sh->scr[c.flip];
    if (lane == 31) {
        buf[0][warp] = dbits(is);
        buf[1][warp] = dbits(wmx);
    }
    __syncthreads();
    double ws = lane < THR / 32 ? bitsd(buf[0][lane]) : 0.0;
    const double wm = lane < THR / 32 ? bitsd(buf[1][lane]) : 0.0;
#pragma unroll
    for (int o = 1; o < SW; o <<= 1) {
        const double us = __shfl_up_sync(0xffffffffu, ws, o);
        if ((lane & (SW - 1)) >= o) ws += us;
    }
    const bool firstw = (warp & (SW - 1)) == 0;
    const double bs = __shfl_sync(0xffffffffu, ws, firstw ? 0 : warp - 1);
    // the segment's warps before this one
    const double em = warp_max_nonneg(lane < warp && lane >= (warp & ~(SW - 1)) ? wm : 0.0);
    const double ex = firstw ? ps : bs + ps;
    unsigned win;
    long long qs;
    if (len == 0) {  // no segment here (the same for its whole warps)
        win = 0;
        qs = 0;
    } else {
        classify_tile<PER>(get, s_q, i0, len, 1, ex, own, em, &win, &qs, &sh->gel[seg]);
    }
    const long long iq = warp_inclusive_sum(qs);
    const uint32_t iw = warp_inclusive_sum(static_cast<uint32_t>(__popc(win)));
    c.flip ^= 1;
    buf = sh->scr[c.flip];
    if (lane == 31) {
        buf[0][warp] = static_cast<unsigned long long>(iq);
        buf[1][warp] = iw;
    }
    __syncthreads();
    long long wq = lane < THR / 32 ? static_cast<long long>(buf[0][lane]) : 0;
    uint32_t ww = lane < THR / 32 ? static_cast<uint32_t>(buf[1][lane]) : 0;
#pragma unroll
    for (int o = 1; o < SW; o <<= 1) {
        const long long uq = __shfl_up_sync(0xffffffffu, wq, o);
        const uint32_t uw = __shfl_up_sync(0xffffffffu, ww, o);
        if ((lane & (SW - 1)) >= o) {
            wq += uq;
            ww += uw;
        }
    }
    const long long bq = __shfl_sync(0xffffffffu, wq, firstw ? 0 : warp - 1);
    const uint32_t bw = __shfl_sync(0xffffffffu, ww, firstw ? 0 : warp - 1);
    long long P = iq - qs + (firstw ? 0 : bq);
    uint32_t r = iw - __popc(win) + (firstw ? 0 : bw);
    if ((threadIdx.x % SEGT) == SEGT - 1) {
        sh->gq[seg] = P + qs;
        sh->gw[seg] = r + __popc(win);
    }
    if (win) {
#pragma unroll 1
        for (int k = 0; k < PER; ++k) {
            const long long q = s_q[at<PER>(k)];
            if ((win >> k) & 1u) {
                if (r < kSegWin) {
                    sh->ge[seg][r] = static_cast<int>(q);
                    sh->gx[seg][r] = get(k);
                    sh->gP[seg][r] = P;
                }
                ++r;
            } else {
                P += q;
            }
        }
    }
    __syncthreads();
    if (i0 == 0) {
        double t = 0.0;
        const unsigned W = sh->gw[seg];
        if (W > kSegWin ||
            !walk_windows(W, sh->gx[seg], sh->gP[seg], sh->ge[seg], nullptr, sh->gq[seg], sh->gel[seg], &t)) {
            t = 0.0;
            for (uint32_t j = 0; j < len; ++j) t = __dadd_rn(t, again(seg, j));
        }
        sh->gtot[seg] = t;
    }
    __syncthreads();
}

// dd::exp with the accurate phase out of line
__device__ __noinline__ double exp_accurate(double x)
{
    return dd::exp_dd(x);
}

__device__ __forceinline__ double exp_rn(double x)
{
    double y;
    if (!dd::exp_quick(x, &y)) y = exp_accurate(x);
    return y;
}

// ---- Weight::normalize (weight.cu) of the tile's log-weights in s_w (m: the
// thread's maximum of those it wrote).  s_w receives the terms exp(lw - lmax)
// (0 past N), each in its thread's place; the weights are 1 / accw times them.
struct WeightOut {
    double ess, accw, lmax;
};

template <int THR, int PER>
__device__ __forceinline__ bool weight_phase(Ctx &c, double *s_w, long long *s_q, uint64_t N, double m,
    WeightOut &out, Approx &ap)
{
    constexpr uint32_t TILE = THR * PER;
    const uint64_t base = static_cast<uint64_t>(c.tile) * TILE;
    m = max_all<THR>(c, m);
    if (c.T > 1) {
        unsigned long long x[1] = {static_cast<unsigned long long>(ordered_bits(m))};
        if (!exchange(c, x, false)) return false;
        m = max_all<THR>(c, threadIdx.x < c.T ? from_ordered_bits(static_cast<long long>(x[0]))
                                         : -__longlong_as_double(0x7ff0000000000000ll));
    }
    const double lmax = m;
#pragma unroll 2
    for (int k = 0; k < PER; ++k) {
        const bool in = base + threadIdx.x * PER + k < N;
        const double e = in ? exp_rn(__dsub_rn(s_w[at<PER>(k)], lmax)) : 0.0;
        s_w[at<PER>(k)] = e;
    }
    // the ESS's dot products: one short fold per chunk of 1024 particles, by
    // 128 threads of eight consecutive elements (all 512 of two for one chunk)
    constexpr int NSEG = TILE / 1024, SP = NSEG == 1 ? 1024 / THR : 8, SEGT = 1024 / SP;
    if constexpr (SP != PER) __syncthreads();
    const int seg = threadIdx.x / SEGT;
    const uint64_t cb = base + static_cast<uint64_t>(seg) * 1024;
    const uint32_t clen = seg < NSEG && cb < N ? static_cast<uint32_t>(min(static_cast<uint64_t>(1024), N - cb)) : 0u;
    seg_fold<THR, SP, SEGT>(c, s_q, clen,
        [s_w](int k) {
            const double e = s_w[at<SP>(k)];
            return __dmul_rn(e, e);
        },
        [s_w](int sg, uint32_t j) {
            const double e = s_w[pad(sg * 1024 + j)];
            return __dmul_rn(e, e);
        });
    const uint32_t nd = static_cast<uint32_t>((N + 1023) / 1024);
    double *dots = c.T == 1 ? c.sh->dots : c.g.dots;
    if (threadIdx.x < NSEG) {
        const uint32_t d = c.tile * NSEG + threadIdx.x;
        if (d < nd) dots[d] = c.sh->gtot[threadIdx.x];
    }
    double accw, before;
    if (!fold_approx<THR, PER>(c, s_w, ap) || !fold_grid<THR, PER, false>(c, s_w, s_q, N, ap, &accw, &before)) return false;
    constexpr int DP = (kMaxTiles * NSEG + THR - 1) / THR;
    static_assert(DP * THR <= TILE, "the dots' increments fit the tile's");
    if (c.T <= kMaxCluster) {  // a few
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (uint32_t j = 0; j < nd; ++j) t = __dadd_rn(t, c.T == 1 ? dots[j] : __ldcg(dots + j));
            c.sh->gtot[0] = t;
        }
        __syncthreads();
    } else {
        double d[DP];
#pragma unroll
        for (int k = 0; k < DP; ++k) {
            const uint32_t j = threadIdx.x * DP + k;
            d[k] = j < nd ? __ldcg(dots + j) : 0.0;
        }
        seg_fold<THR, DP, THR>(c, s_q, nd,
            [&d](int k) {
                double x = d[0];
#pragma unroll
                for (int q = 1; q < DP; ++q)
                    if (k == q) x = d[q];
                return x;
            },
            [dots](int, uint32_t j) { return __ldcg(dots + j); });
    }
    out.accw = accw;
    out.lmax = lmax;
    out.ess = __ddiv_rn(__dmul_rn(accw, accw), c.sh->gtot[0]);
    return true;
}

// ---- the number of uniforms below v in a nondecreasing sequence u_0..u_{M-1}
// (resample.cu), M < 2^31: galloping out from floor(v M), which is usually
// within a step
template <class U>
__device__ __forceinline__ uint32_t count_below_from(const U &u, uint32_t M, double v, uint32_t g)
{
    uint32_t lo, hi;
    if (g < M && u(g) < v) {
        lo = g + 1;
        hi = M;
        for (uint32_t step = 1; lo - 1 + step < M; step <<= 1) {
            const uint32_t probe = lo - 1 + step;
            if (u(probe) >= v) {
                hi = probe;
                break;
            }
            lo = probe + 1;
        }
    } else {
        lo = 0;
        hi = g;
        for (uint32_t step = 1; step <= hi; step <<= 1) {
            const uint32_t probe = hi - step;
            if (u(probe) < v) {
                lo = probe + 1;
                break;
            }
            hi = probe;
        }
    }
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (u(mid) < v) {
            lo = mid + 1;
        } else {
            hi = mid;
        }
    }
    return lo;
}

template <class U>
__device__ __forceinline__ uint32_t count_below(const U &u, uint32_t M, double v)
{
    const double gx = __dmul_rn(v, static_cast<double>(M));
    return count_below_from(u, M, v, gx > 0.0 ? (gx < static_cast<double>(M) ? static_cast<uint32_t>(gx) : M) : 0);
}

// The replication count of every particle of the thread from the cumulative
// weights in s_v, into s_q.  With ties, *ties grows by the uniforms within one
// representable step of them.
template <int PER, class U>
__device__ __forceinline__ void count_reps(const U &u, uint64_t N, uint32_t R, uint64_t i0, const double *s_v,
    long long *s_q, double before, unsigned long long *ties)
{
    uint32_t prev = i0 == 0 || i0 >= N ? 0 : count_below(u, R, before);
#pragma unroll 2
    for (int k = 0; k < PER; ++k) {
        const uint64_t i = i0 + k;
        uint32_t rep = 0;
        if (i < N) {
            const double v = s_v[at<PER>(k)];
            const uint32_t cur = i + 1 == N ? R : count_below(u, R, v);
            rep = cur - prev;
            prev = cur;
            if (ties && i + 1 < N) {
                const double up = __longlong_as_double(__double_as_longlong(v) + 2);
                const double dn = v > 0.0 ? __longlong_as_double(__double_as_longlong(v) - 1) : v;
                // usually neither neighbour of the bound is that close
                if ((cur < R && u(cur) < up) || (cur > 0 && !(u(cur - 1) < dn)))
                    *ties += count_below_from(u, R, up, cur) - count_below_from(u, R, dn, cur);
            }
        }
        s_q[at<PER>(k)] = static_cast<long long>(rep);
    }
}

// ---- ResampleAlgorithm::operator() (resample.cu) from the tile's weights in
// s_v (0 past N).  canon(j): canonical uniform j of the call's stream; again(i):
// weight i.  ubuf: global memory for the uniforms of the sorted and stratified
// sequences.  known (nullable): fold_approx of the weights.  The counts go to
// s_q (each in its thread's place), the number of uniforms used to *used.
template <int THR, int PER, class Canon, class Again>
__device__ __forceinline__ bool resample_phase(Ctx &c, double *s_v, long long *s_q, uint64_t N, uint64_t M,
    int scheme, const Canon &canon, const Again &again, double *ubuf, const Approx *known, uint64_t *used,
    unsigned long long *ties)
{
    const uint64_t i0 = (static_cast<uint64_t>(c.tile) * THR + threadIdx.x) * PER;
    const int seq = scheme % 3;
    uint64_t R = M;
    double before = 0.0, total, mul = 1.0;
    Approx ap;
    const double coeff = static_cast<double>(M);
    if (scheme >= 3) {
        long long acc = 0;
#pragma unroll 1
        for (int k = 0; k < PER; ++k) {
            double ip;
            s_v[at<PER>(k)] = modf(__dmul_rn(coeff, s_v[at<PER>(k)]), &ip);
            if (i0 + k < N) acc += static_cast<long long>(static_cast<uint64_t>(ip));
        }
        long long e0, e1, t0, t1;
        scan_two<THR>(c, acc, 0, e0, e1, t0, t1);
        if (c.T > 1) {
            unsigned long long x[1] = {static_cast<unsigned long long>(t0)};
            if (!exchange(c, x, false)) return false;
            scan_two<THR>(c, static_cast<long long>(x[0]), 0, e0, e1, t0, t1);
        }
        R = static_cast<uint64_t>(t0) <= M ? M - static_cast<uint64_t>(t0) : 0;
        if (!fold_approx<THR, PER>(c, s_v, ap) || !fold_grid<THR, PER, false>(c, s_v, s_q, N, ap, &total, &before)) return false;
        mul = __ddiv_rn(1.0, total);
    }
    *used = R;
    if (seq == 0 && R > 0) {
#pragma unroll 1
        for (int k = 0; k < PER; ++k) {
            const uint64_t j = i0 + k;
            s_v[at<PER>(k)] = j < R ? -__ddiv_rn(dd::log(canon(j)), static_cast<double>(R - j)) : 0.0;
        }
        if (!fold_approx<THR, PER>(c, s_v, ap) || !fold_grid<THR, PER, true>(c, s_v, s_q, R, ap, &total, &before)) return false;
#pragma unroll 1
        for (int k = 0; k < PER; ++k)
            if (i0 + k < R) ubuf[i0 + k] = __dsub_rn(1.0, exp_rn(-s_v[at<PER>(k)]));
    } else if (seq == 1) {
        const double delta = __ddiv_rn(1.0, static_cast<double>(R));
#pragma unroll 1
        for (int k = 0; k < PER; ++k)
            if (i0 + k < R) ubuf[i0 + k] = __dmul_rn(delta, __dadd_rn(canon(i0 + k), static_cast<double>(i0 + k)));
    }
    const bool draw = N > 1 && R > 0;
    if (draw) {
        // the weights (residuals, scaled) of particles 0 .. N - 2: still in s_v
        // unless the sorted sequence's fold took their place
#pragma unroll 1
        for (int k = 0; k < PER; ++k) {
            if (seq != 0 && scheme < 3 && i0 + k + 1 != N) continue;
            double w = 0.0;
            if (i0 + k + 1 < N) {
                w = seq == 0 ? again(i0 + k) : s_v[at<PER>(k)];
                if (scheme >= 3) {
                    double ip;
                    if (seq == 0) w = modf(__dmul_rn(coeff, w), &ip);
                    w = __dmul_rn(w, mul);
                }
            }
            s_v[at<PER>(k)] = w;
        }
        if (known && scheme < 3) {
            ap = *known;
        } else if (!fold_approx<THR, PER>(c, s_v, ap)) {
            return false;
        }
        if (!fold_grid<THR, PER, true>(c, s_v, s_q, N - 1, ap, &total, &before)) return false;
        if (seq == 2) {
            const double delta = __ddiv_rn(1.0, static_cast<double>(R));
            const double ud = __dmul_rn(canon(0), delta);
            count_reps<PER>([delta, ud](uint32_t j) { return __fma_rn(static_cast<double>(j), delta, ud); }, N,
                static_cast<uint32_t>(R), i0,
                s_v, s_q, before, ties);
        } else {
            count_reps<PER>([ubuf](uint32_t j) { return __ldcg(ubuf + j); }, N, static_cast<uint32_t>(R), i0, s_v, s_q,
                before, ties);
        }
    }
    if (!draw || scheme >= 3) {
#pragma unroll 1
        for (int k = 0; k < PER; ++k) {
            long long rep = draw ? s_q[at<PER>(k)] : (N == 1 && i0 + k == 0 ? static_cast<long long>(R) : 0);
            if (scheme >= 3 && i0 + k < N) {
                double ip;
                modf(__dmul_rn(coeff, again(i0 + k)), &ip);
                rep += static_cast<long long>(static_cast<uint64_t>(ip));
            }
            s_q[at<PER>(k)] = rep;
        }
    }
    return true;
}

// ---- parent indices (resample.cu) from the counts in s_q (0 past N): occupied
// slots keep their particle, the empty slots in ascending order take the
// surplus copies in source order.  keep(d) for every occupied slot d < M of the
// tile, copy(d, parent) for every empty one.  surp: global memory, one word per
// element of the tiles: the surplus copies before it within its tile.  s_q and
// s_v (one array of 2 padded(TILE) 64-bit words, s_v first) are overwritten.
//
// The copies of a tile's empty slots are consecutive, and so are their sources:
// as a rule they lie in the tile itself or its neighbours, whose prefixes are
// staged in shared memory and searched there (a search of the prefixes in L2
// from every empty slot measured 14 us at 2^20 particles against 4).
template <int THR, int PER, class Keep, class Copy>
__device__ __forceinline__ bool index_phase(Ctx &c, double *s_v, long long *s_q, uint64_t N, uint64_t M,
    uint32_t *surp, const Keep &keep, const Copy &copy)
{
    Shared *sh = c.sh;
    constexpr uint32_t TILE = THR * PER;
    constexpr uint32_t kStageTiles = 4 * padded(TILE) / TILE;  // tiles of prefixes that fit the two arrays
    const uint64_t base = static_cast<uint64_t>(c.tile) * TILE, i0 = base + threadIdx.x * PER, K = min(N, M);
    const auto surplus = [K](uint64_t i, long long rep) { return i < K ? (rep != 0 ? rep - 1 : 0) : rep; };
    long long e = 0, s = 0;
    unsigned empty = 0;
#pragma unroll 2
    for (int k = 0; k < PER; ++k) {
        const uint64_t i = i0 + k;
        const long long rep = s_q[at<PER>(k)];
        if (i < M && (i >= K || rep == 0)) {
            empty |= 1u << k;
            ++e;
        }
        if (i < N) s += surplus(i, rep);
    }
    long long E, S, te, ts;
    scan_two<THR>(c, e, s, E, S, te, ts);
#pragma unroll 2
    for (int k = 0; k < PER; ++k) {
        const uint64_t i = i0 + k;
        surp[i] = static_cast<uint32_t>(S);
        if (i < N) S += surplus(i, s_q[at<PER>(k)]);
        if ((empty >> k) & 1u) sh->empties[E++] = threadIdx.x * PER + k;
    }
    unsigned long long x[2] = {static_cast<unsigned long long>(te), static_cast<unsigned long long>(ts)};
    if (!exchange(c, x, true)) return false;
    long long pe = 0, ps = 0, t0, t1;
    if (c.cluster) {
        const unsigned long long(*xs)[kMaxCluster] = sh->xs[c.epoch & 1];
        for (uint32_t t = 0; t < c.T && t < threadIdx.x; ++t) {
            pe += static_cast<long long>(xs[0][t]);
            ps += static_cast<long long>(xs[1][t]);
        }
    } else if (c.T > 1) {
        scan_two<THR>(c, static_cast<long long>(x[0]), static_cast<long long>(x[1]), pe, ps, t0, t1);
    }
    if (threadIdx.x < c.T) {
        sh->pw[threadIdx.x] = static_cast<uint32_t>(pe);
        sh->pq[threadIdx.x] = ps;
    }
#pragma unroll 2
    for (int k = 0; k < PER; ++k) {
        const uint32_t o = k * THR + threadIdx.x;
        if (base + o < K && s_q[pad(o)] != 0) keep(base + o);
    }
    __syncthreads();
    const uint32_t E0 = sh->pw[c.tile], ne = static_cast<uint32_t>(te);
    const uint32_t lastt = static_cast<uint32_t>((N - 1) / TILE);
    // the last tile with at most q surplus copies before it
    const auto tile_of = [sh, lastt](uint32_t q) {
        uint32_t lo = 0, hi = lastt + 1;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sh->pq[mid] <= q) {
                lo = mid;
            } else {
                hi = mid;
            }
        }
        return lo;
    };
    const uint32_t ta = ne ? tile_of(E0) : 0, tb = ne ? tile_of(E0 + ne - 1) : 0;
    uint32_t *st = reinterpret_cast<uint32_t *>(s_v);
    const bool staged = tb - ta < kStageTiles;
    if (staged && ne) {
        const uint4 *src = reinterpret_cast<const uint4 *>(surp + static_cast<size_t>(ta) * TILE);
        uint4 *dst = reinterpret_cast<uint4 *>(st);
        for (uint32_t k = threadIdx.x; k < (tb - ta + 1) * (TILE / 4); k += THR) dst[k] = __ldcg(src + k);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < ne; k += THR) {
        const uint32_t q = E0 + k;
        // the source: the last particle of its tile with surp <= q - (before the tile)
        uint32_t t = ta;
        while (t < tb && sh->pq[t + 1] <= q) t = staged ? t + 1 : tile_of(q);
        const uint32_t r = q - static_cast<uint32_t>(sh->pq[t]);
        uint32_t lo = 0, hi = static_cast<uint32_t>(min(static_cast<uint64_t>(TILE), N - static_cast<uint64_t>(t) * TILE));
        if (staged) {
            const uint32_t *p = st + (t - ta) * TILE;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (p[mid] <= r) {
                    lo = mid;
                } else {
                    hi = mid;
                }
            }
        } else {
            const uint32_t *p = surp + static_cast<size_t>(t) * TILE;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (__ldcg(p + mid) <= r) {
                    lo = mid;
                } else {
                    hi = mid;
                }
            }
        }
        copy(base + sh->empties[k], static_cast<uint64_t>(t) * TILE + lo);
    }
    return true;
}

}  // namespace coop

}  // namespace mckl_b200
